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


def test_field_passes_read_step_data_by_ordinary_loads():
    """The passes are launched while the kernel before them still writes.  __ldg, and a
    const pointer that nothing aliases, promise data that no one writes while the grid
    is there: only the uploaded B0 and its scaled copy are that."""
    s = code("gm_fields.cuh")
    assert "launch_next(" in s and "ld.global.nc" not in s
    assert len(re.findall(r'asm volatile\("ld\.global\.f(32|64) ', s)) == 2
    args = re.findall(r"__ldg\(\s*([^),]*)", s)
    assert args and all(re.match(r"(b0s\b|&B0\[)", a) for a in args), args
    assert set(re.findall(r"const T\* __restrict__ (\w+)", s)) <= {"B0"}
    # the launches of this kind are those of the field passes and of the ghost faces,
    # whose pointers are not const
    assert "launch_next(" not in code("gm_stage_tma.cuh")
    k = code("gm_kernels_impl.cuh")
    assert re.findall(r"launch_next\((\w+)", k) == ["k_export_peri"]
    body = re.search(r"void __launch_bounds__\(256\) k_export_peri\(.*?\n\}", k, re.S).group(0)
    assert "__ldg" not in body and "const T*" not in body
