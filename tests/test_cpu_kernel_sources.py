"""Rules that the kernels' sources keep and no run can show: what breaks them works until the compiler schedules a warp another way."""
import re

from elfa_b200.build import CSRC


def _function(text, name):
    """The body of the first function called ``name``."""
    at = text.index("{", text.index(f" {name}("))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i]
    raise AssertionError(name)


def test_a_cluster_barrier_brings_the_warp_together_first():
    """``barrier.cluster`` in its ``.aligned`` form wants all threads of a warp at once, and its callers come from loops that some of them leave early."""
    body = _function((CSRC / "common.cuh").read_text(), "cluster_sync_all")
    assert body.index("__syncwarp()") < body.index("barrier.cluster.arrive")
    for f in sorted(CSRC.glob("*.cu*")):                       # and there is no other place that issues it
        if f.name != "common.cuh":
            assert not re.search(r"barrier\.cluster\.\w+[\w.]*\.aligned", f.read_text()), f.name


def test_tensor_memory_is_used_by_whole_warps_after_one_lane_arrived():
    """``tcgen05.ld`` and ``.st`` are ``.sync.aligned``: behind an arrival by one lane the warp is brought together before the next of them."""
    text = (CSRC / "attention_bwd.cu").read_text()
    hand = text[text.index("auto hand_over"):]
    assert hand.index("__syncwarp()") < hand.index("tmem_st")
    text = (CSRC / "gemm_mxfp8.cu").read_text()
    after = text[text.index("if (lane == 0) mbar_arrive_cluster(map_to_cta(over_bar, 0));"):]
    assert after.index("__syncwarp()") < min(after.index("fl & ELFA_EPI_STORE_PREACT"), after.index("tmem_ld32"))


def test_no_kernel_is_given_a_status_word_that_is_not_there():
    """It is allocated on first use, which fails during a stream capture, for one; a kernel that records an error would write to address zero."""
    for f in sorted(CSRC.glob("*.cu")):
        for m in re.finditer(r"(\S+) = (?:elfa::)?status_word\(\);", f.read_text()):
            behind = f.read_text()[m.end():][:160]
            assert re.match(rf"\s*(ELFA_REQUIRE\({re.escape(m[1])}( != nullptr|,)|if \(!{re.escape(m[1])}\))", behind), (f.name, behind)
