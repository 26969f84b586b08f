"""The abort path of the tensor-core pair kernel: the warps that go through its loops as a whole
take one decision per warp.  Lanes that read the abort flag or wait on a barrier for themselves
could leave a loop alone, and the others would wait for them in its votes for ever."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "microsn_gb300", "csrc", "pairtc.cu")


def _kernel():
    s = open(SRC).read()
    s = s[s.index("k_pairdiff_tc(const __grid_constant__"):]
    return re.sub(r"//[^\n]*", "", s[:s.index("\n}\n")])


def test_whole_warps_decide_as_one():
    k = _kernel()
    helpers = re.findall(r"auto warp_(?:aborted|wait) = .*?};", k)
    assert len(helpers) == 2 and all("0xffffffffu" in h for h in helpers)
    assert "__shfl_sync" in helpers[0] and "__all_sync" in helpers[1]
    loops = k[k.index("} else if (warp == 1) {"):]  # (the producer before it is one lane)
    assert "if (warp == 0 && lane == 0)" in k
    assert "abort_s" not in loops and "mbar_wait(" not in loops
    assert loops.count("warp_aborted()") >= 3 and loops.count("warp_wait(") >= 4
