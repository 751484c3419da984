"""Rules of the CUDA sources that a run cannot show: what the instruction set
leaves undefined may work on one compiler and hang on the next."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dygrass_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_cluster_barriers_need_no_convergence():
    """barrier.cluster.*.aligned is undefined unless all lanes of a warp execute
    it together.  The phases reach the barrier out of divergent loops, so the
    plain forms are used, or a __syncwarp() stands directly before."""
    found = 0
    for name in sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))):
        code = _code(name)
        for m in re.finditer(r"barrier\.cluster\.(arrive|wait)[\w.]*", code):
            found += 1
            if ".aligned" in m.group(0):
                before = code[:code.rfind("asm", 0, m.start())].rstrip()
                assert before.endswith("__syncwarp();"), f"{name}: {m.group(0)}"
    assert found >= 2
