"""The prefill kernel on pairs of SMs, as far as the CPU can check it: its plans, its work lists, and a rule of its source."""
import ctypes
import os
import random
import re
import subprocess

import pytest

import pair_forms

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qwen3-27b-thor-runner_b200", "csrc")
PAIRS = 74


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pair") / "pair_plan_check.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "pair_plan_check.cpp")], check=True)
    return ctypes.CDLL(out)


def plan(lib, M, N, K, dense=False, pairs=PAIRS, stream_k=True):
    out = (ctypes.c_int * 15)()
    lib.pair_plan(M, N, K, pairs, int(stream_k), int(dense), out)
    p = dict(zip(("T", "R", "m_tiles", "row_tiles", "items", "dp_items", "sk_tiles", "w_stages", "x_stages", "units", "accs", "a_col0",
                  "smem", "pairs", "ring"), out))
    p["how"] = ("whole" if not p["sk_tiles"] else "tail" if p["dp_items"] else
                "parts" if p["pairs"] % p["sk_tiles"] == 0 else "straddle")
    return p


@pytest.mark.parametrize("dense,shapes", [(False, pair_forms.FP4), (True, pair_forms.BF16)])
def test_shapes_take_the_form_they_name(lib, dense, shapes):
    for M, N, K, T, R, how in shapes:
        p = plan(lib, M, N, K, dense)
        assert (p["T"], p["R"], p["how"]) == (T, R, how), (M, N, K)


def _shapes(count):
    rng = random.Random(7)
    for _ in range(count):
        M = rng.choice([1, 17, rng.randint(1, 300), rng.randint(1, 9000)])
        N = 8 * rng.randint(1, rng.choice([8, 100, 2000, 4352]))
        yield M, N, 256 * rng.randint(1, rng.choice([1, 4, 20, 72])), rng.random() < 0.5, rng.choice([PAIRS, PAIRS, PAIRS, 73, 66, 16, 2, 1])


def test_every_output_is_summed_once(lib):
    """All pairs' lists together: each stage of each tile once, no partial slot twice, all holders of a tile agree on the others, no whole
    tile among the parts of a plan that is split all over.  Whatever the prices are: they choose among valid plans."""
    for M, N, K, dense, pairs in _shapes(2500):
        for stream_k, prices in ((0, 0), (1, 0), (1, 1)):
            assert lib.pair_walk(M, N, K, pairs, stream_k, int(dense), prices) == 0, (M, N, K, dense, pairs, stream_k, prices)


def test_plans_stay_within_the_chip(lib):
    """Shared memory, tensor memory (512 columns) and what the issuers rely on: an even number of units and accumulators, two token
    stages a turn and one more; a ring of an even number of units that has barriers (16) and, in tensor memory, columns."""
    for M, N, K, dense, pairs in _shapes(4000):
        p = plan(lib, M, N, K, dense, pairs)
        assert p["smem"] <= 225 * 1024 and 3 <= p["x_stages"] <= 8 and p["w_stages"] <= 8
        assert p["units"] in (2, 4, 6, 8) and p["accs"] in (2, 4)
        assert p["T"] % 32 == 0 and 32 <= p["T"] <= (224 if dense else 192) and p["R"] in (1, 2)
        assert p["accs"] * p["T"] <= (512 if dense else p["a_col0"]) and (dense or p["a_col0"] + 64 * p["units"] == 512)
        fine = lib.pair_fine(M, N, K, pairs, int(dense))
        assert p["ring"] % 2 == 0 and p["units"] << fine <= p["ring"] <= 16
        assert dense or p["accs"] * p["T"] + p["ring"] * (32 if fine else 64) <= 512
        assert not dense or p["ring"] * (16384 if fine else 32768) == p["units"] * 32768      # the loaders' blocks fill the ring exactly
        assert 1 <= p["pairs"] <= pairs
        assert not dense or fine or p["dp_items"] > 0               # the kernel has no such form


@pytest.mark.parametrize("M,N,K,dense,at_most", [
    (65, 512, 5120, False, 5), (149, 8, 5120, False, 5), (256, 1024, 8192, False, 8), (32, 512, 8192, False, 5), (100, 1024, 17408, False, 12),
    (256, 512, 5120, True, 5), (17, 512, 8192, True, 5), (100, 1024, 5120, True, 5), (17, 1024, 17408, True, 12),
])
def test_small_weights_are_split(lib, M, N, K, dense, at_most):
    """A few row tiles on a long k: parts of a few stages on most of the chip, not whole tiles on a corner of it (K / 256 stages one
    after the other: 65 x 512 x 5120 25 us whole, 14 split)."""
    p = plan(lib, M, N, K, dense)
    assert p["how"] == "parts"
    assert -(-(K // 256) // (p["pairs"] // p["sk_tiles"])) <= at_most


def elects(src):
    """Functions of the source that elect a lane of the whole warp."""
    functions = re.split(r"(?=__device__ __forceinline__ )", src[:src.index("__global__ ")])
    return sorted({re.match(r"__device__ __forceinline__ \w+ (\w+)\(", f).group(1) for f in functions if "elect.sync" in f})


def test_issuing_warps_decide_as_a_whole():
    """The issuers elect a lane of the full warp for every MMA and commit, so a lane that leaves the loop alone (its wait ran out,
    another lane's did not) would leave the rest waiting without a limit.  No wait on a GPU can be made to run out in some lanes
    only, hence the source: behind the loop's last wait the warp votes, and nothing but the vote decides whether it goes on."""
    src = open(os.path.join(CSRC, "prefill_pair.cu")).read()
    issuer = src[src.index("MMA issuers (leader only)"):src.index("dequantise into TMEM")]
    loop = issuer[issuer.index("for (int turn = 0;"):]
    assert re.match(r"for \(int turn = 0; turn < turns; \+\+turn\)", loop)            # not on the lane's own `ok`
    vote = loop.index("ok = __all_sync(0xffffffffu, ok);")
    assert set(re.findall(r"\b((?:mma|commit)\w*)\(", issuer)) <= set(elects(src))
    elections = [m.start() for m in re.finditer(r"\b(?:%s)\(" % "|".join(elects(src)), loop)]
    # the commit behind the loop stands behind the voted `ok` itself
    assert len(elections) >= 7 and loop.rindex("ptx::mbar_wait(") < vote < loop.index("break;") < min(elections)
    assert re.search(r"if \(ok\) commit_pair\(tfull0", loop) and "ok =" not in loop[loop.index("break;"):]
    assert loop.count("break;") == 1 and "return" not in loop and "continue" not in loop
