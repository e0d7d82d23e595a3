"""The few-token kernel where its two issuing warps, its reduction in chunks of four rows and its token range can go wrong."""
import numpy as np
import pytest

import oracle_binding as ob
import util

pytestmark = pytest.mark.gpu
TOL = 1e-3      # BF16 rounding of sums in another order: last bits flip in a few elements


@pytest.fixture(scope="module")
def handle():
    import nvfp4
    h = nvfp4.Handle(0, 128 << 20)
    yield h
    h.close()


@pytest.fixture
def few(handle):
    """65 to 80 tokens to this kernel whatever the shape."""
    with util.options(handle, skinny_max_m=128):
        yield handle


@pytest.mark.parametrize("M,N,K,res", [
    (17, 128, 256, False),        # one stage: a unit for each issuer
    (33, 130, 512, True),         # two rows in the second tile, N % 4 != 0
    (64, 1001, 5120, True),       # split tiles, odd N: scalar stores in the reduction
    (48, 1004, 5120, True),       # split tiles, N % 4 == 0: eight-byte ones, the last tile cut
    (64, 19200, 1024, True),      # 150 tiles: two items a CTA on the first slots, accumulators in turn
    (65, 512, 5120, True),        # beyond 64 tokens: one item at a time in tensor memory
    (80, 19208, 768, False),      # the same with more tiles than CTAs, the last one cut
    (80, 640, 17408, True),       # deep split
])
def test_against_the_oracle(few, M, N, K, res):
    import torch
    handle = few
    packed, scale = util.make_weight(N, K, seed=M + N, sigma=0.14)
    A, R = util.make_bf16((M, K), seed=M), util.make_bf16((M, N), seed=N)
    dA, dP, dS = util.to_dev(A), util.to_dev(packed), util.to_dev(scale)
    outs = []
    for _ in range(2):
        C = util.to_dev(R) if res else torch.zeros((M, N), dtype=torch.int16, device="cuda")
        handle.linear(dA, M, dP, dS, 1.5, N, K, C, residual=C if res else None)
        torch.cuda.synchronize()
        outs.append(util.to_host_u16(C))
    assert handle.device_status() == 0
    assert np.array_equal(outs[0], outs[1])               # a fixed order of summation
    # the kernel's arithmetic: exact weights, 1 / gs once in FP32 (the oracle's GEMM form rounds the scaled weights to BF16)
    assert ob.rel_frobenius(outs[0], ob.linear(A, packed, scale, 1.5, residual=R if res else None, mode=ob.GEMV, threads=8)) <= TOL


@pytest.mark.parametrize("writer", ["linear", "swiglu"])
@pytest.mark.parametrize("M", [65, 80])
def test_weights_follow_a_kernel_that_lets_its_successor_start(few, M, writer):
    """The codes are the BF16 output of a library call right before, which leaves most SMs idle and lets its successor start early
    (SwiGLU at its first instruction); a copy, as below, never does.  The bits of the synchronised sequence."""
    import torch
    handle = few
    N, K = 2048, 1024                                    # N * K / 2 bytes of codes: an output of [T, 256]
    T, K1 = 2048, 2560
    A, A1 = util.to_dev(util.make_bf16((M, K), seed=M)), util.to_dev(util.make_bf16((T, K1), seed=M + 1))
    w1 = [tuple(util.to_dev(a) for a in util.make_weight(256, K1, seed=M + 2 + i, sigma=0.14)) for i in range(3)]
    gate_up = [util.to_dev(util.make_bf16((T, 512), seed=M + 10 + i)) for i in range(3)]
    scale = util.to_dev(util.make_weight(N, K, seed=M + 20, sigma=0.14)[1])
    made = torch.empty((T, 256), dtype=torch.int16, device="cuda")
    codes = made.view(torch.uint8).view(N, K // 2)

    def step(i, out, wait):
        if writer == "linear":
            handle.linear(A1, T, w1[i][0], w1[i][1], 1.0, 256, K1, made)
        else:
            handle.swiglu(gate_up[i], None, T, 256, made)
        if wait:
            torch.cuda.synchronize()
        handle.linear(A, M, codes, scale, 1.0, N, K, out)
        if wait:
            torch.cuda.synchronize()

    want = [torch.empty((M, N), dtype=torch.int16, device="cuda") for _ in range(3)]
    for i in range(3):
        step(i, want[i], True)
    assert not torch.equal(want[0], want[1])
    for r in range(30):
        got = torch.empty((M, N), dtype=torch.int16, device="cuda")
        step(r % 3, got, False)
        assert torch.equal(got, want[r % 3]), r
    assert handle.device_status() == 0


@pytest.mark.parametrize("M", [65, 80])
def test_weights_follow_the_stream_beyond_64_tokens(few, M):
    """A weight copied into place right before the call, on the same stream, is the one that is used."""
    import torch
    handle = few
    N, K = 4096, 2048
    sets = [tuple(util.to_dev(a) for a in util.make_weight(N, K, seed=s)) for s in (1, 2)]
    A = util.to_dev(util.make_bf16((M, K), seed=3))
    packed, scale = torch.empty_like(sets[0][0]), torch.empty_like(sets[0][1])
    want = []
    for p, s in sets:
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        handle.linear(A, M, p, s, 1.0, N, K, C)
        torch.cuda.synchronize()
        want.append(util.to_host_u16(C))
    for i in range(12):
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        packed.copy_(sets[i % 2][0])
        scale.copy_(sets[i % 2][1])
        handle.linear(A, M, packed, scale, 1.0, N, K, C)
        torch.cuda.synchronize()
        assert np.array_equal(util.to_host_u16(C), want[i % 2]), i


def test_a_workspace_too_small_is_refused_as_before(handle):
    """65 to 80 tokens on a handle sized for fewer: the same refusal as above, before any launch."""
    import ctypes
    import torch
    import nvfp4
    M, N, K = 80, 128, 17408
    size = ctypes.c_size_t(0)
    nvfp4.load().nvfp4_workspace_bytes(17, N, 256, ctypes.byref(size))
    h = nvfp4.Handle(0, size.value)
    try:
        p, s = (util.to_dev(a) for a in util.make_weight(N, K, seed=1))
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        with pytest.raises(nvfp4.Nvfp4Error, match="workspace"):
            h.linear(util.to_dev(util.make_bf16((M, K), seed=2)), M, p, s, 1.0, N, K, C)
        assert h.launch_count() == 0 and not C.any()
    finally:
        h.close()


@pytest.mark.parametrize("M", [65, 80])
@pytest.mark.parametrize("option,value", [("prefill_impl", 2), ("prefill_stream_k", 0)])
def test_options_that_name_the_prefill_kernel_reach_it(handle, M, option, value):
    """Above 64 tokens the few-token kernel is the default, not what a caller gets who names another: the bits are the prefill kernel's,
    and a number of rows that it refuses is refused."""
    import torch
    import nvfp4
    N, K = 640, 5120
    p, s = (util.to_dev(a) for a in util.make_weight(N, K, seed=M))
    A = util.to_dev(util.make_bf16((M, K), seed=M + 1))

    def call(**settings):
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        with util.options(handle, **settings):
            handle.linear(A, M, p, s, 1.0, N, K, C)
        return C

    want = call(skinny_max_m=0, **{option: value})
    assert not torch.equal(want, call())                  # else the comparison below says nothing
    assert torch.equal(want, call(**{option: value}))
    if option == "prefill_impl":
        with util.options(handle, prefill_impl=value), pytest.raises(nvfp4.Nvfp4Error, match="shape"):
            handle.linear(A, M, p, s, 1.0, N - 1, K, torch.zeros((M, N - 1), dtype=torch.int16, device="cuda"))


@pytest.mark.parametrize("N,K,here", [
    (6272, 5120, False), (6400, 5120, True),             # 49 and 50 row tiles on 148 CTAs: the latter three CTAs a tile or fewer
    (640, 17408, False), (2048, 5120, False), (640, 5120, True),      # 2.3, 2.2 and less than one stage a CTA
    (4736, 3072, True), (4608, 3072, False), (4736, 3328, False),     # four CTAs a tile, or a few more; twelve stages, thirteen
    (4096, 9472, True), (4096, 9216, False),             # eight stages a CTA
])
def test_route_at_65_tokens(handle, N, K, here):
    """Which kernel takes the call, by its bits: the limit of 128 names this kernel, 0 the prefill kernel."""
    import torch
    M = 65
    if handle.get_option("sm_count") != 148:
        pytest.skip("shapes chosen for 148 SMs")
    p, s = (util.to_dev(a) for a in util.make_weight(N, K, seed=M))
    A = util.to_dev(util.make_bf16((M, K), seed=M + 1))

    def call(**settings):
        C = torch.zeros((M, N), dtype=torch.bfloat16, device="cuda")
        with util.options(handle, **settings):
            handle.linear(A, M, p, s, 1.0, N, K, C)
        return C

    mine, other = call(skinny_max_m=128), call(skinny_max_m=0)
    assert not torch.equal(mine, other)
    assert torch.equal(call(), mine if here else other)
