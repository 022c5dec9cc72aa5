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
