"""A round's launch writes its values last: a caller that has them has left nothing of the round
running.  The order inside a kernel does not show in results, so it is read from the source."""
import os
import re

SRC = re.sub(r"//[^\n]*", "", open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                                "nightstream_b200", "csrc", "mem_oracle.cu")).read())


def test_address_lane_writes_what_the_next_round_reads_before_its_values():
    k = SRC[SRC.index("ta_eval_kernel(const TaEval a)"):SRC.index("struct TaFold")]
    after = re.split(r"ta_finish\(a, s_red\);|ta_carries\(a, s_red\);", k)
    assert len(after) > 1
    assert not re.search(r"key_next\[|tab_out\[", after[-1])
    fin = SRC[SRC.index("void ta_finish("):SRC.index("ta_eval_kernel(const TaEval a)")]
    assert fin.index("atomicInc(a.ticket") < fin.index("ta_carries(")


def test_fold_step_waits_for_its_rollover_copy():
    fold = re.sub(r"//[^\n]*", "", open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                                     "nightstream_b200", "csrc", "fold.cu")).read())
    step = fold[fold.index('"fold/step_done"'):]
    step = step[:step.index("return NEO_OK;")]
    assert step.index("cudaMemcpyAsync(sh->valwit.p + ") < step.index("ctx_sync(ctx)")
