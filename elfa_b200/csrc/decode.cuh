// A decoding step of the EFLA family in one kernel (decode.cu), called by its streaming entry point (stream.cu).
#pragma once
#include "common.cuh"

namespace elfa {

struct EflaDims {
  long long B, T, D, H, d, F, V, layers, L, W, act, kind, prism, tail;
};
struct EflaWork {
  __nv_bfloat16 *x[2], *r, *n, *k, *v, *o, *e, *full, *u, *z, *wc, *q, *h, *g, *f, *nmat;
  float *coef, *segw;
  unsigned int* arrived;                   // DECODE_COUNTERS words
};

// the activation of an MLP by its number: -1 SwiGLU, 0 GELU in the product's epilogue, else an operation of elementwise.cuh
constexpr int ACT_SWIGLU = -1, ACT_GELU = 0;
constexpr int DECODE_COUNTERS = 64;        // barrier counters: one per launch

// Whether a call can take the one-kernel form; if so efla_decode issues it up to and with the final norm, whose rows are left in w.n. ELFA_ERR_UNSUPPORTED:
// the stream has too few SMs for it, and the call is the chain's after all (which writes everything anew).
bool efla_decode_fits(const EflaDims& m);
int efla_decode(const unsigned long long* p, const EflaDims& m, const EflaWork& w, const float* forget, float eps, cudaStream_t s);

}  // namespace elfa
