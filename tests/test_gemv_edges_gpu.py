"""The tensor-core GEMVs where what they ask for early can go wrong: a CTA's k range of one chunk or wrapping round, split tiles with a
residual that is the output, token factors of every token, ragged rows."""
import numpy as np
import pytest

import oracle_binding as ob
import util

pytestmark = pytest.mark.gpu
TOL = 1e-3      # BF16 rounding of sums in another order, and the expansion's remainder (1e-5 to 8e-5 of a block's largest element)


@pytest.fixture(scope="module")
def handle():
    import nvfp4
    h = nvfp4.Handle(0, 64 << 20)
    yield h
    h.close()


@pytest.mark.parametrize("N,K", [
    (128, 256),        # one half-unit: one CTA, one chunk (the second loading warp has none)
    (136, 1280),       # ten half-units on ten CTAs, every tile split five ways, eight rows in the last
    (6400, 1280),      # 250 half-units on 148 CTAs: k ranges of one and two chunks, some wrapping round
    (3000, 5120),      # 480: wrapping ranges, tiles split over several CTAs, ragged rows
    (512, 17408),      # deep
])
@pytest.mark.parametrize("M", [1, 2, 3, 9, 10, 16])
def test_in_place_residual(handle, M, N, K):
    import torch
    packed, scale = util.make_weight(N, K, seed=N + K, sigma=0.14)
    A, R = util.make_bf16((M, K), seed=M), util.make_bf16((M, N), seed=N)
    A = ob.f32_to_bf16(ob.bf16_to_f32(A) * (2.0 ** np.arange(M, dtype=np.float32))[:, None])      # another factor for every token
    C = util.to_dev(R)
    handle.linear(util.to_dev(A), M, util.to_dev(packed), util.to_dev(scale), 1.5, N, K, C, residual=C)
    torch.cuda.synchronize()
    assert handle.device_status() == 0
    want = ob.linear(A, packed, scale, 1.5, residual=R, mode=ob.GEMV, threads=8)
    got = util.to_host_u16(C)
    for m in range(M):
        assert ob.rel_frobenius(got[m:m + 1], want[m:m + 1]) <= TOL, m


@pytest.mark.parametrize("M", [1, 2, 3, 4, 7, 9, 10, 13, 16])
def test_a_launch_takes_its_own_partial_sums_only(handle, M):
    """Launches with other activations follow each other on the same slots; every tile is split over several CTAs.  An old value beside
    a new tag would show: what a launch gives is compared bit by bit with what the same inputs gave when nothing else ran."""
    import torch
    N, K = 4352, 5120
    p, s = (util.to_dev(a) for a in util.make_weight(N, K, seed=7))
    sets = []
    for i in range(3):
        A = util.to_dev(util.make_bf16((M, K), seed=10 * M + i))
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        handle.linear(A, M, p, s, 1.0, N, K, C)
        handle.linear(A, M, p, s, 1.0, N, K, C)      # the slots hold this very launch's values: right whatever is torn
        torch.cuda.synchronize()
        sets.append((A, C.clone()))
    wrong = torch.zeros(1, dtype=torch.int64, device="cuda")
    for it in range(200):
        A, want = sets[it % 3]
        C = torch.zeros((M, N), dtype=torch.int16, device="cuda")
        handle.linear(A, M, p, s, 1.0, N, K, C)
        wrong += (C != want).sum()
    assert int(wrong) == 0 and handle.device_status() == 0
