"""RMSNorm and SwiGLU at the edges of what a thread keeps in registers, and in a stream of kernels that start behind each other."""
import numpy as np
import pytest

import oracle_binding as ob
import util

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handle():
    import nvfp4
    h = nvfp4.Handle(0, 96 << 20)
    yield h
    h.close()


# 6144 and 8192 columns fit the registers (with a bias, without), one chunk of eight more is read again
@pytest.mark.parametrize("M,K,add", [(2, 6144, True), (3, 6152, True), (2, 8192, False), (3, 8200, False), (1, 8, False), (1, 8, True)])
def test_rmsnorm_register_edges(handle, M, K, add):
    import torch
    x, w, b = util.make_bf16((M, K), seed=K), util.make_bf16((K,), seed=K + 1, std=0.3), util.make_bf16((M, K), seed=K + 2)
    dx, out = util.to_dev(x), torch.zeros((M, K), dtype=torch.int16, device="cuda")
    if add:
        handle.add_rmsnorm(dx, util.to_dev(b), util.to_dev(w), 1e-6, M, K, out)
        want, res = ob.rmsnorm(x, w, 1e-6, bias=b)
    else:
        handle.rmsnorm(dx, util.to_dev(w), 1e-6, M, K, out)
        want, res = ob.rmsnorm(x, w, 1e-6), x
    torch.cuda.synchronize()
    got = util.to_host_u16(out)
    assert np.array_equal(util.to_host_u16(dx), res)
    # the sum of squares is added in another order: at most the last bit, of few elements
    assert util.bf16_ulp_diff(got, want) <= 1 and (got != want).sum() <= max(1, got.size // 50)


# fewer vectors than threads, an odd last step, more than one step of the whole grid (2368 x 256 vectors)
@pytest.mark.parametrize("M,I", [(1, 8), (7, 1000), (149, 17408), (401, 13824)])
def test_swiglu_row_walk(handle, M, I):
    import torch
    merged = util.make_bf16((M, 2 * I), seed=M + I, std=2.0)
    out = torch.zeros(M, I, dtype=torch.int16, device="cuda")
    handle.swiglu(util.to_dev(merged), None, M, I, out)
    torch.cuda.synchronize()
    assert util.bf16_ulp_diff(util.to_host_u16(out), ob.swiglu_merged(merged)) <= 1


@pytest.mark.parametrize("M", [4, 24, 80])
def test_stream_order_of_the_block(handle, M):
    """norm, linear, SwiGLU, linear on one stream, back to back: the bits of the same calls with a synchronisation after each."""
    import torch
    H, I, rounds = 1024, 2048, 4
    gu, gs = (util.to_dev(a) for a in util.make_weight(2 * I, H, seed=3))
    dn, ds = (util.to_dev(a) for a in util.make_weight(H, I, seed=4))
    nw = util.to_dev(util.make_bf16((H,), seed=5, std=0.3))

    def block(wait):
        x = util.to_dev(util.make_bf16((M, H), seed=M))
        n, g, a = (torch.zeros((M, c), dtype=torch.int16, device="cuda") for c in (H, 2 * I, I))
        for _ in range(rounds):
            for step in (lambda: handle.rmsnorm(x, nw, 1e-6, M, H, n), lambda: handle.linear(n, M, gu, gs, 4.0, 2 * I, H, g),
                         lambda: handle.swiglu(g, None, M, I, a), lambda: handle.linear(a, M, dn, ds, 4.0, H, I, x, residual=x)):
                step()
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return util.to_host_u16(x)

    want = block(True)
    for _ in range(3):
        assert np.array_equal(block(False), want)
