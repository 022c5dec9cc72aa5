// Coefficient of the EFLA update, c = (1 - exp(-beta lam)) / lam, and its derivatives (series for small lam).
#pragma once
#include "common.cuh"

namespace elfa {

__device__ __forceinline__ void efla_coeff(float beta, float lam, float& c, float& dc_dbeta, float& dc_dlam) {
  if (lam < 1e-6f) {
    c = beta - 0.5f * beta * beta * lam + beta * beta * beta * lam * lam / 6.f;
    dc_dbeta = 1.f - beta * lam + 0.5f * beta * beta * lam * lam;
    dc_dlam = -0.5f * beta * beta + beta * beta * beta * lam / 3.f;
  } else {
    const float ex = __expf(-beta * lam);
    c = (1.f - ex) / lam;
    dc_dbeta = ex;
    dc_dlam = (beta * lam * ex - (1.f - ex)) / (lam * lam);
  }
}

}  // namespace elfa
