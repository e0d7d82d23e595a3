"""The prefill GEMM on pairs of SMs: every form of its work (pair_forms.py: tokens per tile, row tiles per item, whole and split
items) through every output form, and sizes at the edges of its tiles (256 rows a pair, 256-k stages)."""
import ctypes

import numpy as np
import pytest

import nvfp4
import oracle_binding as ob
import pair_forms
import util

pytestmark = pytest.mark.gpu

# Relative Frobenius error against the oracle's exact-weight arithmetic (GEMV mode): both round the same FP32 sums once, in
# another order.  (Its GEMM mode rounds weights / global_scale to BF16, 2^-9 each: 1.5e-3 and more when the scale is not 1.)
TOL = 1e-3


def run(h, A, packed, scale, gs, residual=None):
    import torch
    M, K = A.shape
    N = packed.shape[0]
    dC = torch.full((M, N), 0x7FC0, dtype=torch.int16, device="cuda")   # NaN canary
    dR = util.to_dev(residual) if residual is not None else None
    h.linear(util.to_dev(A), M, util.to_dev(packed), util.to_dev(scale), gs, N, K, dC, residual=dR)
    torch.cuda.synchronize()
    return util.to_host_u16(dC)


def sample(N):
    """Weight rows at the edges of row tiles and CTAs, and some between."""
    edges = [0, 7, 8, 127, 128, 255, 256, 383, 384, N // 256 * 256 - 1, N // 256 * 256, N - 8, N - 1]
    return np.unique([r for r in edges if 0 <= r < N] + list(np.random.default_rng(N).integers(0, N, 48)))


def swiglu_of(plain, N):
    import torch
    slabs = plain.float().view(plain.shape[0], N // 16, 2, 8)
    gate, up = slabs[:, :, 0].reshape(plain.shape[0], -1), slabs[:, :, 1].reshape(plain.shape[0], -1)
    return (gate / (1 + torch.exp(-gate)) * up).to(torch.bfloat16)


@pytest.fixture
def pair_only(handle):
    """17 to 80 tokens to the pair kernel too."""
    with util.options(handle, skinny_max_m=0, gemm_weight_rounding=0):
        yield handle


@pytest.mark.parametrize("M,N,K,T,R,how", pair_forms.FP4)
def test_every_form_through_every_output(pair_only, M, N, K, T, R, how):
    import torch
    h, gs = pair_only, 1.7
    packed, scale = util.make_weight(N, K, seed=M + N, sigma=0.14)
    A, residual = util.make_bf16((M, K), seed=M + 5), util.make_bf16((M, N), seed=N + 6)
    dA, dp, ds, dR = (util.to_dev(x) for x in (A, packed, scale, residual))
    rows = sample(N)
    at = torch.from_numpy(rows).cuda()
    p_s, s_s, r_s = (np.ascontiguousarray(x) for x in (packed[rows], scale[rows], residual[:, rows]))

    def call(res=None, out=None):
        out = torch.full((M, N), 0x7FC0, dtype=torch.int16, device="cuda") if out is None else out      # NaN canary
        h.linear(dA, M, dp, ds, gs, N, K, out, residual=res)
        return out

    def error(out, **how_):
        return ob.rel_frobenius(util.to_host_u16(out[:, at]), ob.linear(A, p_s, s_s, gs, threads=8, **how_))

    plain = call()
    assert error(plain, mode=ob.GEMV) <= TOL
    assert torch.isfinite(plain.view(torch.bfloat16).float()).all()
    added = call(dR)
    assert error(added, residual=r_s, mode=ob.GEMV) <= TOL
    for _ in range(3):
        assert torch.equal(plain, call()) and torch.equal(added, call(dR))           # fixed summation order
    alias = dR.clone()
    assert torch.equal(added, call(alias, alias))                                    # C as its own residual
    f32 = torch.full((M, N), float("nan"), device="cuda")
    h.linear_f32(dA, M, dp, ds, gs, N, K, f32)
    assert torch.equal(f32.to(torch.bfloat16).view(torch.int16), plain)              # the same sums, not rounded
    if N % 32 == 0:
        out = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
        h.linear_ex(dA, M, dp, ds, gs, N, K, out, swiglu_epilogue=True)
        # same sums, so at most one BF16 step where the two exponentials round differently: 2^-8 of the value
        assert torch.allclose(out.float(), swiglu_of(plain.view(torch.bfloat16), N).float(), rtol=2 ** -7, atol=1e-30)
    h.set_option("gemm_weight_rounding", 1)
    rounded = call(dR)
    assert torch.equal(rounded, call(dR))
    assert error(rounded, residual=r_s, mode=ob.GEMM) <= TOL
    assert h.device_status() == 0


@pytest.mark.parametrize("gs", [1.0, 0.37, 2688.0, 3.0e-20, 7.0e25])
def test_rounded_weights_are_the_dequantised_matrix(handle, gs):
    """One-hot tokens pick single weights out: with gemm_weight_rounding each is the bits that nvfp4_dequant_bf16 stores (the
    reference's), over all codes and finite block scales."""
    import torch
    N, K = 2048, 256
    rng = np.random.default_rng(11)
    packed = util.to_dev(rng.integers(0, 256, (N, K // 2), dtype=np.uint8))
    scale = util.to_dev((np.arange(N * K // 16, dtype=np.int64) * 31 % 127).astype(np.uint8).reshape(N, K // 16))      # 0 .. 126, all of them
    want = torch.empty((N, K), dtype=torch.bfloat16, device="cuda")
    handle.dequant(packed, scale, gs, N, K, want)
    out = torch.full((K, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    handle.set_option("gemm_weight_rounding", 1)
    try:
        handle.linear(torch.eye(K, dtype=torch.bfloat16, device="cuda"), K, packed, scale, gs, N, K, out)
    finally:
        handle.set_option("gemm_weight_rounding", 0)
    assert torch.equal(out.T.float(), want.float())                    # by value: -0 and 0 are alike
    assert torch.isfinite(want.float()).all() and handle.device_status() == 0


@pytest.mark.parametrize("M,N,K,T,R,how", [f for f in pair_forms.FP4 if f[3:] in ((160, 2, "whole"), (128, 1, "parts"), (160, 2, "tail"))])
def test_non_finite_tokens_keep_to_themselves(pair_only, M, N, K, T, R, how):
    """Tokens are columns of shared accumulators: an infinity or a NaN in one of them reaches no other."""
    import torch
    packed, scale = util.make_weight(N, K, seed=M, sigma=0.14)
    dA = util.to_dev(util.make_bf16((M, K), seed=M + 1))
    dp, ds = util.to_dev(packed), util.to_dev(scale)
    clean, got = (torch.empty((M, N), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    pair_only.linear(dA, M, dp, ds, 1.0, N, K, clean)
    bad = {0: 0x7F80, M // 2: 0x7FC0, M - 1: 0xFF80 - 0x10000}      # +inf, NaN, -inf
    for m, bits in bad.items():
        dA[m, (37 * m + 5) % K] = bits
    pair_only.linear(dA, M, dp, ds, 1.0, N, K, got)
    finite = torch.ones(M, dtype=torch.bool, device="cuda")
    finite[list(bad)] = False
    assert torch.equal(got[finite], clean[finite])
    assert not torch.isfinite(got[~finite].float()).any()
    assert pair_only.device_status() == 0


@pytest.mark.parametrize("M,N,K,T,R,how", pair_forms.BF16)
def test_every_form_on_bf16_weights(handle, M, N, K, T, R, how):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    W = (0.05 * torch.randn((N, K), device="cuda", generator=gen)).to(torch.bfloat16)
    A, residual = util.make_bf16((M, K), seed=M + 3), util.make_bf16((M, N), seed=N + 4)
    dA, dR = util.to_dev(A), util.to_dev(residual)
    rows = sample(N)
    at = torch.from_numpy(rows).cuda()
    W_s = util.to_host_u16(W[at])

    def call(res=None, out=None):
        out = torch.full((M, N), 0x7FC0, dtype=torch.int16, device="cuda") if out is None else out
        handle.linear_bf16(dA, M, W, N, K, out, residual=res)
        return out

    plain, added = call(), call(dR)
    assert ob.rel_frobenius(util.to_host_u16(plain[:, at]), ob.dense_linear(A, W_s)) <= TOL
    assert ob.rel_frobenius(util.to_host_u16(added[:, at]), ob.dense_linear(A, W_s, residual=np.ascontiguousarray(residual[:, rows]))) <= TOL
    assert torch.isfinite(plain.view(torch.bfloat16).float()).all()
    for _ in range(3):
        assert torch.equal(plain, call()) and torch.equal(added, call(dR))
    alias = dR.clone()
    assert torch.equal(added, call(alias, alias))
    assert handle.device_status() == 0


@pytest.mark.parametrize("M,N,K,res", [
    (65, 8, 256, True),           # one short row tile, one stage: every wait is a first phase
    (96, 264, 512, False),        # two row tiles, the second of 8 rows
    (97, 768, 256, True),         # three row tiles, one token in the last tile
    (160, 5376, 512, False),      # 21 row tiles, two stages
    (161, 1280, 1024, True),      # one token in the last tile
    (193, 2048, 2816, False),     # one token in the last tile, eleven stages
    (385, 520, 4352, True),       # ragged rows, one token in the last tile, split
    (2500, 2816, 256, False),     # many items of one stage: the rings run across items
    (1300, 5120, 768, True),      # items of two row tiles, three stages each
])
def test_pair_kernel_vs_oracle(pair_only, M, N, K, res):
    handle = pair_only
    packed, scale = util.make_weight(N, K, seed=M + N, sigma=0.14)
    A = util.make_bf16((M, K), seed=M + 5)
    R = util.make_bf16((M, N), seed=N + 6) if res else None
    got = run(handle, A, packed, scale, 1.7, residual=R)
    for _ in range(3):
        assert np.array_equal(got, run(handle, A, packed, scale, 1.7, residual=R))   # fixed summation order
    assert ob.rel_frobenius(got, ob.linear(A, packed, scale, 1.7, residual=R, mode=ob.GEMV, threads=8)) <= TOL
    assert handle.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(70, 96, 256), (150, 5120, 2560), (333, 1024, 4352)])
def test_swiglu_output_equals_linear_and_swiglu(pair_only, M, N, K):
    """Interleaved rows (8 gate, 8 up): the SwiGLU of the plain call's rounded outputs."""
    import torch
    handle = pair_only
    packed, scale = util.make_weight(N, K, seed=M, sigma=0.14)
    A = util.make_bf16((M, K), seed=M + 1)
    dA, dp, ds = util.to_dev(A), util.to_dev(packed), util.to_dev(scale)
    plain = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    out = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
    handle.linear(dA, M, dp, ds, 1.0, N, K, plain)
    handle.linear_ex(dA, M, dp, ds, 1.0, N, K, out, swiglu_epilogue=True)
    want = swiglu_of(plain, N)
    # same sums, so at most one BF16 step where the two exponentials round differently: 2^-8 of the value
    assert torch.allclose(out.float(), want.float(), rtol=2 ** -7, atol=1e-30)
    assert handle.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(17, 8, 256), (33, 776, 256), (161, 2816, 512), (512, 5120, 1280), (700, 264, 2560)])
def test_bf16_weights_vs_oracle(handle, M, N, K):
    import torch
    W = util.make_bf16((N, K), seed=N + 1, std=0.05)
    A = util.make_bf16((M, K), seed=M + 3)
    dA, dW = util.to_dev(A), util.to_dev(W)
    outs = []
    for _ in range(8):
        dC = torch.full((M, N), 0x7FC0, dtype=torch.int16, device="cuda")
        handle.linear_bf16(dA, M, dW, N, K, dC)
        outs.append(dC)
    torch.cuda.synchronize()
    got = util.to_host_u16(outs[0])
    assert all(np.array_equal(got, util.to_host_u16(o)) for o in outs[1:])
    assert ob.rel_frobenius(got, ob.dense_linear(A, W)) <= TOL
    assert handle.device_status() == 0


@pytest.mark.parametrize("option,value,M", [("gemm_weight_rounding", 1, 9), ("gemm_weight_rounding", 1, 16), ("decode_max_m", 0, 1),
                                            ("decode_max_m", 8, 12)])
def test_few_tokens_need_the_kernels_whole_scratch(option, value, M):
    """Options send 16 tokens and fewer to the pair kernel: a workspace sized for the GEMV kernels alone is refused before
    anything is launched, through the host-buffer call too; one sized for 17 tokens takes the call."""
    import torch
    N, K = 512, 1024
    lib = nvfp4.load()
    packed, scale = util.make_weight(N, K, seed=M, sigma=0.14)
    A = util.make_bf16((M, K), seed=M + 1)
    dA, dp, ds = util.to_dev(A), util.to_dev(packed), util.to_dev(scale)
    dC = torch.full((M, N), 0x7FC0, dtype=torch.int16, device="cuda")
    hA, hC = torch.from_numpy(A.view(np.int16)), torch.zeros((M, N), dtype=torch.int16)
    for max_m in (16, 17):
        need = ctypes.c_size_t()
        assert lib.nvfp4_workspace_bytes(max_m, N, K, ctypes.byref(need)) == 0
        h = nvfp4.Handle(0, need.value)
        h.set_option(option, value)
        before = h.launch_count()
        st = h.linear(dA, M, dp, ds, 1.0, N, K, dC, check=False)
        if max_m == 16:
            assert st == -4
            assert lib.nvfp4_linear_host(h.h, hA.data_ptr(), M, dp.data_ptr(), ds.data_ptr(), 1.0, N, K, None, hC.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream) == -4
            assert h.launch_count() == before
        else:
            assert st == 0 and h.launch_count() == before + 2
            assert ob.rel_frobenius(util.to_host_u16(dC), ob.linear(A, packed, scale, 1.0, mode=ob.GEMV, threads=8)) <= TOL
            assert h.device_status() == 0
        h.close()


@pytest.mark.parametrize("M", [65, 300])
def test_weights_follow_the_stream(pair_only, M):
    """A weight written by the work right before the call, again and again into the same buffers: by a copy, and by a call of
    this library whose BF16 output serves as the codes (that kernel lets the next one start early)."""
    import torch
    handle = pair_only
    N, K = 2048, 1024                                    # the second weight is the first call's [T, 256] output: N * K / 2 bytes
    T, K1 = 2048, 2560
    A = util.to_dev(util.make_bf16((M, K), seed=M))
    A1 = util.to_dev(util.make_bf16((T, K1), seed=M + 1))
    w1 = [util.make_weight(256, K1, seed=M + 2 + i, sigma=0.14) for i in range(4)]
    w1 = [(util.to_dev(p), util.to_dev(s)) for p, s in w1]
    source = [util.make_weight(N, K, seed=M + 20 + i, sigma=0.14) for i in range(4)]
    source = [(util.to_dev(p), util.to_dev(s)) for p, s in source]
    made = torch.empty((T, 256), dtype=torch.int16, device="cuda")
    packed, scale = torch.empty_like(source[0][0]), torch.empty_like(source[0][1])
    codes = made.view(torch.uint8).view(N, K // 2)

    def step(i, out, wait):
        sync = torch.cuda.synchronize if wait else (lambda: None)
        packed.copy_(source[i][0])
        scale.copy_(source[i][1])
        sync()
        handle.linear(A, M, packed, scale, 1.0, N, K, out[0])
        sync()
        handle.linear(A1, T, w1[i][0], w1[i][1], 1.0, 256, K1, made)
        sync()
        handle.linear(A, M, codes, scale, 1.0, N, K, out[1])
        sync()

    buffers = lambda: [torch.empty((M, N), dtype=torch.int16, device="cuda") for _ in range(2)]
    want = [buffers() for _ in range(4)]
    for i in range(4):
        step(i, want[i], True)
    for r in range(40):
        got = buffers()
        step(r % 4, got, False)
        assert all(torch.equal(g, w) for g, w in zip(got, want[r % 4])), r
    assert handle.device_status() == 0
