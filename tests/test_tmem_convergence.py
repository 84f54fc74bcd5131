"""The TMEM instructions in the .sync.aligned form need the whole warp converged.  They are
issued by helpers of tc.cuh that bring the warp together first, and nowhere else: a kernel's
lanes may have left by a `continue` or a predicated store before the next one."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nightstream_b200", "csrc")


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_aligned_instructions_only_in_the_helpers():
    users = [f for f in sorted(os.listdir(CSRC)) if re.search(r'"tcgen05[^"]*\.aligned', _code(f))]
    assert users == ["tc.cuh"]


def test_helpers_converge_the_warp_first():
    bodies = re.findall(r"__device__ __forceinline__ [^;{]*\{(.*?)\n\}", _code("tc.cuh"), flags=re.S)
    aligned = [b for b in bodies if ".aligned" in b]
    assert len(aligned) == 4  # alloc, dealloc, two loads
    for b in aligned:
        assert b.split("asm volatile")[0].strip() == "__syncwarp();"
