"""prefill_mix: zeros written beside the parameter prep, and the state turned around beside the epilogue."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# the single-pass scan with counters, with tags, and on both sides of the 131072 token-heads up to which the prep writes the
# zeros; the stages (more than 128 modes) with tiles of the state that are not full, beside the epilogue and in front of it
@pytest.mark.parametrize("B,L,H,R,M", [
    (1, 2, 1, 64, 128), (1, 397, 24, 64, 128), (2, 130, 3, 64, 128), (1, 2000, 24, 64, 128), (1, 5461, 24, 64, 128),
    (1, 5462, 24, 64, 128), (2, 1500, 70, 64, 128), (2, 40, 3, 40, 130), (1, 40, 2, 33, 161)])
def test_prefill_mix_on_any_workspace(B, L, H, R, M):
    from frac_ssm_b200 import _cabi as C
    g = torch.Generator(device="cuda").manual_seed(L)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda").bfloat16()
    di, T, bf16, f32 = H * R, 64, torch.bfloat16, torch.float32
    dyn, rw, x, gate = randn(B, L, 3 * H), randn(B, L, 2 * H * M), randn(B, L, di), randn(B, L, di)
    u = x.view(B, L, H, R).transpose(1, 2).contiguous()
    small = [randn(H), randn(1), randn(1), randn(M), randn(H, R), randn(di)]
    params = (ctypes.c_void_p * 6)(*(t.data_ptr() for t in small))
    nums = (ctypes.c_float * 9)(1.0, 1e-3, 0.1, 0.1, 0.9, 1e-4, 1.0, 0.0, 1e-6)
    lib, p = C.lib(), C.ptr
    nbytes = max(lib.fracssm_frac_scan_auto_workspace_bytes(B * H, L, R, M, T), 256)

    def run(fill, turn):
        def empty(*shape, dtype=f32):
            return torch.empty(*shape, device="cuda", dtype=dtype).fill_(float("nan"))
        ws = torch.full((nbytes,), fill, device="cuda", dtype=torch.uint8)
        c, kappa, rho = (empty(B * H, L, M) for _ in range(3))
        h, y, fin = empty(B * H, L, R, dtype=bf16), empty(B, L, di, dtype=bf16), empty(B * H, R, M)
        state = empty(B * H, M, R) if turn else None
        C.check(lib.fracssm_prefill_mix(p(dyn), None, p(rw), p(x), p(gate), di, None, params, 0, nums, p(u), p(c), p(kappa),
                                        C.F32, p(rho), p(h), p(fin), p(state), p(y), p(ws), nbytes, B, L, H, R, M, T,
                                        C.stream_of(x)), "prefill_mix")
        return y, fin, state
    y0, fin, _ = run(0, False)
    assert y0.isfinite().all()
    for fill in (0, 255, 1):
        y, _, state = run(fill, True)
        assert torch.equal(y, y0) and torch.equal(state, fin.transpose(1, 2))
