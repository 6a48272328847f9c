"""The dynamic projection that prefill runs beside its convolution, against float64."""

import ctypes

import pytest
import torch

from tests.helpers import selftest_lib

pytestmark = pytest.mark.gpu


# one value, one row and one row more than a tile of 128; K below, at and beside steps of 64; columns below, at and beside
# multiples of 16 up to the 192 covered; a cluster of 1, 2, 4 and 8 blocks a tile; a ring that is used again
@pytest.mark.parametrize("B,L,K,N", [
    (1, 1, 8, 1), (1, 5, 40, 3), (1, 128, 64, 16), (1, 129, 128, 36), (2, 127, 136, 33), (1, 397, 1536, 72),
    (4, 1000, 1536, 36), (1, 6000, 1536, 72), (3, 3300, 520, 48), (1, 18950, 1536, 72), (1, 19000, 1544, 191),
    (1, 300, 192, 192), (1, 300, 1536, 192)])
def test_prefill_conv_dyn(B, L, K, N):
    from frac_ssm_b200 import _cabi as C
    g = torch.Generator(device="cuda").manual_seed(L + N)
    xg = torch.randn(B, L, 2 * K, generator=g, device="cuda").bfloat16()
    xg[..., K:] = float("nan")            # the gate beside x takes no part
    x = xg[..., :K]
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    conv_w = torch.randn(K, 1, 4, generator=g, device="cuda").bfloat16()
    mask = (torch.rand(B, L, generator=g, device="cuda") > 0.2).float()
    R = 8
    lib, p = C.lib(), C.ptr

    def outputs():
        return [torch.full(s, float("nan"), device="cuda", dtype=torch.bfloat16)
                for s in ((B, L, K), (B * K // R, L, R), (B, K, 3))]
    conv, alone = outputs(), outputs()
    dyn = torch.full((B * L * N + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    C.check(lib.fracssm_prefill_conv_dyn(p(xg), 2 * K, p(mask), p(conv_w), None, *map(p, conv), p(w), p(dyn), N, R, B, L, K, 4,
                                         C.stream_of(xg)), "prefill_conv_dyn")
    C.check(lib.fracssm_prefill_conv(p(xg), 2 * K, p(mask), p(conv_w), None, *map(p, alone), R, B, L, K, 4, C.stream_of(xg)),
            "prefill_conv")
    for a, b in zip(conv, alone):
        assert torch.equal(a, b)
    assert (dyn[B * L * N:] == 7).all()
    got = dyn[:B * L * N].view(B * L, N).double()
    x64, w64 = x.reshape(B * L, K).double(), w.double()
    exact, size = x64 @ w64.t(), x64.abs() @ w64.abs().t()
    # a bf16 rounding (half of 2^-7), and K float32 additions of at most the sum of the magnitudes
    assert ((got - exact).abs() <= 2 ** -8 * exact.abs() + K * 2 ** -23 * size).all()


def test_prefill_conv_dyn_refuses_what_it_does_not_cover():
    from frac_ssm_b200 import _cabi as C
    x = torch.zeros(8, 64, device="cuda", dtype=torch.bfloat16)
    lib, p = C.lib(), C.ptr
    for cols, K, w in ((193, 64, p(x)), (3, 60, p(x)), (3, 64, x.data_ptr() + 2), (0, 64, p(x))):
        assert lib.fracssm_prefill_conv_dyn(p(x), 64, None, p(x), None, p(x), None, None, w, p(x), cols, 4, 1, 1, K, 4,
                                            C.stream_of(x)) != 0


# a block alone and clusters of 2, 4 and 8, one row and tiles with rows beyond the last
@pytest.mark.parametrize("rows,K,N", [(1, 40, 3), (9000, 1536, 72), (4000, 1536, 36), (397, 1536, 72), (19000, 200, 192)])
def test_a_wait_that_runs_out_marks_every_row(rows, K, N):
    """One load of every 128 rows is left out: its wait gives up after two milliseconds, for all blocks of the cluster."""
    from frac_ssm_b200 import _cabi as C
    fn = selftest_lib().fracssm_selftest_prefill_dyn_wait_limit
    vp, i64 = ctypes.c_void_p, ctypes.c_int64
    fn.argtypes, fn.restype = [vp, i64, vp, vp, i64, i64, i64, ctypes.c_uint64, vp], ctypes.c_int
    x = torch.ones(rows, K, device="cuda", dtype=torch.bfloat16)
    w = torch.ones(N, K, device="cuda", dtype=torch.bfloat16)
    dyn = torch.zeros(rows * N + 8, device="cuda", dtype=torch.bfloat16)
    assert fn(C.ptr(x), K, C.ptr(w), C.ptr(dyn), rows, K, N, 2_000_000, C.stream_of(x)) == 0
    torch.cuda.synchronize()
    assert torch.isnan(dyn[:rows * N]).all() and (dyn[rows * N:] == 0).all()
