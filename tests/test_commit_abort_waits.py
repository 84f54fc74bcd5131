"""A commitment CTA in which a wait ran out still waits (with a limit) for what it started: the
MMAs before its TMEM goes back, the bulk copies before its shared memory does.  The waits
cannot be made to run out without a fault, so the order is read from the source."""
import os
import re

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nightstream_b200", "csrc",
                        "commit_tc.cu")).read()


def _kernel():
    return re.sub(r"//[^\n]*", "", SRC[SRC.index("commit_win_kernel(const"):SRC.index("int commit_ws(")])


def test_mmas_are_waited_for_after_an_abort():
    waits = re.findall(r"okw = \(([^;]*)\) \?", _kernel())
    assert len(waits) == 1
    terms = [t.strip() for t in waits[0].split("&&")]
    assert terms.index("mbar_wait(done, 0)") < terms.index("!s_abort")  # && ends at the first false term


def test_copies_are_waited_for_after_an_abort():
    k = _kernel()
    for bar in ("full_a", "full_g"):
        loop = k[k.index("mbar_expect_tx(&%s[" % bar):]
        loop = loop[:loop.index("} else if")]
        assert "drain(%s," % bar in loop  # behind the loop, whichever way it ended
