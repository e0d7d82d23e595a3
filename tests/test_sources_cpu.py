"""Rules of the kernels' sources whose breach no test on a GPU may show: it would be a race or a warp that waits without a limit."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen3-27b-thor-runner_b200", "csrc")


def source(name):
    """A source file without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, name)).read(), flags=re.S)


@pytest.mark.parametrize("name", ["prefill_pair.cu", "skinny_umma.cu", "decode_fp4.cu", "decode_fp4_stream.cu"])
def test_warps_are_whole_at_tensor_memory_accesses(name):
    """tcgen05.ld and .st want a converged warp.  Its lanes leave a wait on a barrier, a look at one or a branch on their row one by
    one: between any of these and the access stands a __syncwarp(), or a vote decides for the warp."""
    src = source(name)
    vote = r"if \(!__all_sync\(0xffffffffu, ready\)\) \{\s*ptx::mbar_wait\([^;]*;\s*__syncwarp\(\);\s*\}"
    src = re.sub(vote, "WHOLE", src)
    assert not re.search(r"if \(!ready\)\s*\{\s*ptx::mbar_wait\(&aempty", src)      # a __syncwarp() that only some lanes reach
    calls = [m.start() for m in re.finditer(r"(?<!void )\btmem_(?:st|ld)16\(", src)]
    assert calls
    for at in calls:
        before = src[:at]
        whole = max(before.rfind("__syncwarp();"), before.rfind("WHOLE"))
        assert whole > max(before.rfind(f) for f in ("mbar_wait(", "mbar_test_wait(", "continue;", "elect_one("))
        # a loop whose lanes may leave a turn early meets a __syncwarp() before the next turn's load; so does a function it calls
        turn = re.search(r"(?:for \(int c0 = 0; c0 < p\.NT; c0 \+= 16\)|auto sums = \[&\]\([^{]*\)) \{[^}]*$", before)
        assert not turn or "__syncwarp();" in turn.group(0)


def test_bf16_weight_loader_waits_for_the_stream():
    """The header lets W come from the kernel right before, and the kernels of this library let their successors start early: the
    loading warp waits for them before its first load."""
    src = source("dense_gemv.cu")
    loader = src[src.index("if (warp == 2 * kGroupWarps)"):]
    loader = loader[:loader.index("return;")]
    assert "griddep_wait()" in loader and loader.index("griddep_wait()") < loader.index("tma_load_2d(")


def test_what_the_kernel_before_writes_is_not_read_as_read_only():
    """__ldg() and const __restrict__ parameters promise that nobody writes the memory while the kernel runs.  A kernel that starts
    behind its predecessor runs while that one still writes; what it waits for then needs plain loads.  (A chain's parameter block
    is written once, by the host.)"""
    for name in sorted(os.listdir(CSRC)):
        src = source(name) if name.endswith((".cu", ".cuh")) else ""
        early = "ProgrammaticStreamSerialization" in src
        for part in re.split(r"(?=__global__ )", src) if early else []:
            head = part[:part.index("{")] if part.startswith("__global__") else ""
            reads = [c for c in re.findall(r"__ldg\([^;]*", part) if "ch.params" not in c]
            if head and "griddep_wait()" not in part:      # an ordinary launch in the same file
                continue
            assert "__restrict__" not in head and not reads, (name, head, reads)
