"""What the stage kernel's text has to keep, checked without a GPU (a run that broke it
could hang one)."""
import re

from conftest import ROOT

CSRC = ROOT / "glemur_gb300" / "csrc"


def code(name):
    """A source file without its comments."""
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_one_thread_decides_whether_a_block_computes_its_tile():
    """The march's barrier counts every thread of the block.  Another block may set the
    status bits between two reads, so the word is read in one place, by thread 0, in
    front of a __syncthreads, and every thread branches on what that thread found."""
    s = code("gm_stage_tma.cuh")
    assert '"bar.sync 1, %0;"' in s
    assert s.count("GM_ST_TIMEOUT | GM_ST_ALIGN") == 1
    body = re.search(r"int stage_stopped\([^)]*\) \{.*?\n\}", s, re.S).group(0)
    assert "GM_ST_TIMEOUT | GM_ST_ALIGN" in body and "->done" in body
    rest = s.replace(body, "")
    assert "->done" not in rest
    # the single case: the barrier's own reduction of thread 0's word
    one = "if (__syncthreads_or(threadIdx.x == 0 ? stage_stopped(A.a.st) : 0)) return;"
    assert rest.count(one) == 1
    rest = rest.replace(one, "")
    # the batch: thread 0 fetches the item and its run's word, a barrier, all branch on both
    assert rest.count("stage_stopped(") == 1
    assert re.search(r"if \(threadIdx\.x == 0\) \{[^{}]*ctl->skip = [^;]*stage_stopped\([^;]*;\s*\}\s*__syncthreads\(\);\s*"
                     r"const int w = ctl->work, skip = ctl->skip;\s*__syncthreads\(\);", rest)
