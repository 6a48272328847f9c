"""The segment kernels of the scan (csrc/scan_modes.cu), which path="auto" takes up to 128 modes where the
single-pass kernel does not apply, against the float64 token recurrence and the chunked stages."""

import pytest
import torch

from oracle import frac_oracle as O

pytestmark = pytest.mark.gpu


def _exact(u, c, kappa, rho, init):
    u, c, kappa, rho = (t.double() for t in (u, c, kappa, rho))
    rho = rho.clamp_min(1e-6)
    B, L, R = u.shape
    S = torch.zeros(B, R, c.shape[-1], dtype=torch.float64) if init is None else init.double().clone()
    h = torch.empty(B, L, R, dtype=torch.float64)
    for t in range(L):
        S = S * rho[:, t, None, :] + u[:, t, :, None] * kappa[:, t, None, :]
        h[:, t] = (S * c[:, t, None, :]).sum(-1)
    return h, S


def _rel(x, ref):
    return ((x.double().cpu() - ref).norm() / ref.norm().clamp_min(1e-30)).item()


# edges: one token, one column, columns that are no multiple of 4 or exceed a block, modes that fill no
# group of 8, lengths around a stage of 8 and a segment of 32 tokens, rows that need no segments
CASES = [(1, 1, 1, 1), (1, 7, 3, 5), (2, 33, 20, 8), (3, 64, 128, 8), (2, 65, 130, 9), (1, 300, 64, 16), (5, 97, 192, 17),
         (2, 257, 64, 33), (4, 100, 96, 64), (1, 129, 66, 65), (2, 71, 64, 128), (1200, 9, 8, 8), (400, 40, 128, 100)]


@pytest.mark.parametrize("B,L,R,M", CASES)
@pytest.mark.parametrize("dtype,coeff", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                         (torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
def test_segments_match_recurrence_and_stages(B, L, R, M, dtype, coeff):
    from frac_ssm_b200.ops.b200 import frac_scan
    if (R, M, dtype) == (64, 128, torch.bfloat16):
        pytest.skip("the single-pass kernel's shape")
    u, c, kappa, rho, init = O.scan_inputs(B, L, R, M, dtype=torch.float32, gen="model_like", seed=B + L + R + M)
    u, c, kappa = u.to(dtype), c.to(coeff), kappa.to(coeff)
    rho.view(-1)[::17] = 0.0                                   # below the floor of 1e-6
    keep = slice(0, min(B, 4))
    for start in (None, init):
        g = [t.cuda() for t in (u, c, kappa, rho)]
        ig = None if start is None else start.cuda()
        h, fin = frac_scan(*g, 32, ig, True, final_state_dtype=torch.float32)
        hs, fs = frac_scan(*g, 32, ig, True, final_state_dtype=torch.float32, path="staged")
        h_ref, f_ref = _exact(*(t[keep] for t in (u, c, kappa, rho)), None if start is None else start[keep])
        # outputs are rounded once (2^-9 bfloat16, 2^-12 half); float32: sums of at most L * M terms
        out = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11, torch.float32: 2e-6}[dtype]
        assert _rel(h[keep], h_ref) <= out
        assert _rel(fin[keep], f_ref) <= 2e-6
        assert _rel(h, hs.double().cpu()) <= 2 * out + 1e-5
        assert _rel(fin, fs.double().cpu()) <= 1e-5


# more than 384 segments a row: a share of the carry kernel's 32 warps is then more than the 12 segments it keeps in
# registers, and it reads what it overwrites a batch at a time
@pytest.mark.parametrize("B,L,R,M", [(2, 32768, 128, 16), (1, 20011, 64, 8), (3, 7001, 20, 5)])
@pytest.mark.parametrize("with_start", [False, True])
def test_many_segments(B, L, R, M, with_start):
    from frac_ssm_b200 import _cabi as C
    from frac_ssm_b200.ops.b200 import frac_scan
    Mp = (M + 7) // 8 * 8
    nseg = C.lib().fracssm_frac_scan_auto_workspace_bytes(B, L, R, M, 32) // (4 * B * Mp * (R + 1))
    assert nseg > 384
    u, c, kappa, rho, init = O.scan_inputs(B, L, R, M, dtype=torch.float32, gen="model_like", seed=L)
    start = init if with_start else None
    g = [t.cuda() for t in (u, c, kappa, rho)]
    ig = None if start is None else start.cuda()
    h, fin = frac_scan(*g, 32, ig, True)
    hs, fs = frac_scan(*g, 32, ig, True, path="staged")
    h_ref, f_ref = _exact(u, c, kappa, rho, start)
    bound = 2.0 ** -23 * L ** 0.5         # roundings of at most L steps, of either sign
    for got, staged, ref in ((h, hs, h_ref), (fin, fs, f_ref)):
        assert _rel(got, ref) <= bound
        assert _rel(got, staged.double().cpu()) <= 2 * bound


@pytest.mark.parametrize("B,L,R,M,T,strided", [(8, 8192, 192, 40, 64, False), (16, 4096, 128, 72, 128, False), (8, 8192, 128, 128, 64, True)])
def test_large_calls_that_load_by_element_take_the_stages(B, L, R, M, T, strided):
    """A segment is then the slower way (8 x 8192 tokens, 192 columns x 40 modes: 819 us against 541)."""
    from frac_ssm_b200.ops.b200 import frac_scan
    g = torch.Generator(device="cuda").manual_seed(M)

    def rows(n, lo, hi, dtype):
        x = lo + (hi - lo) * torch.rand(B, L, n + strided, device="cuda", generator=g)
        return x.to(dtype)[:, :, int(strided):]
    bf = torch.bfloat16
    args = rows(R, -1, 1, bf), rows(M, 0, 1 / M, bf), rows(M, 0, 1, bf), rows(M, 0.9, 1, torch.float32)
    auto, staged = (frac_scan(*args, T, None, True, path=path) for path in ("auto", "staged"))
    assert torch.equal(auto[0], staged[0]) and torch.equal(auto[1], staged[1])
    few = frac_scan(*(t[:1, :4000] for t in args), T)      # below the line: the same values by the segments
    want = staged[0][:1, :4000]
    assert not torch.equal(few, want) and _rel(few, want.double().cpu()) <= 2 ** -7


@pytest.mark.parametrize("M,R", [(16, 64), (8, 20)])
def test_segments_take_any_stride_and_alignment(M, R):
    from frac_ssm_b200.ops.b200 import frac_scan
    B, L = 3, 90
    for dtype in (torch.bfloat16, torch.float32):
        u, c, kappa, rho, init = O.scan_inputs(B, L, R, M, dtype=dtype, gen="model_like", seed=5)
        ref = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True)

        def odd(t, pad):       # rows `pad` elements further apart, batch and token strides swapped, base shifted by one
            buf = torch.zeros(L, B, t.shape[-1] + pad, dtype=t.dtype, device="cuda")
            buf[:, :, 1:1 + t.shape[-1]] = t.cuda().transpose(0, 1)
            return buf[:, :, 1:1 + t.shape[-1]].transpose(0, 1)
        got = frac_scan(odd(u, 3), odd(c, 1), odd(kappa, 2), odd(rho, 5), 32, init.cuda(), True)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])   # the same sums in the same order


def test_initial_state_passes_through_masked_tokens():
    from frac_ssm_b200.ops.b200 import frac_scan
    B, L, R, M = 2, 200, 64, 16
    u, c, kappa, rho, init = O.scan_inputs(B, L, R, M, dtype=torch.float32, gen="model_like", seed=1)
    kappa.zero_()
    rho.fill_(1.0)
    _, fin = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 64, init.cuda(), True)
    assert torch.equal(fin.cpu(), init)


@pytest.mark.parametrize("M", [5, 8, 12, 20, 100])      # 8: no padding modes
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_an_infinity_stays_one_where_modes_are_padded(M, dtype):
    from frac_ssm_b200.ops.b200 import frac_scan
    u, c, kappa, rho, init = O.scan_inputs(2, 300, 64, M, dtype=torch.float32, gen="model_like", seed=M)
    u, c, kappa = u.to(dtype), c.abs().add(0.01).to(dtype), kappa.abs().add(0.01).to(dtype)
    u[0, 37, 5], u[1, 200, 63] = float("inf"), float("-inf")
    rho = 0.9 + 0.1 * rho          # 0.9 ** 300 = 2e-14: no product of decays becomes zero, which would make NaN of it too
    h, fin = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True, final_state_dtype=torch.float32)
    h_ref, f_ref = _exact(u, c, kappa, rho, init)
    assert torch.isinf(h_ref).any() and not torch.isnan(h_ref).any()
    for got, ref in ((h, h_ref), (fin, f_ref)):
        got, finite = got.double().cpu(), torch.isfinite(ref)
        assert torch.equal(got[~finite], ref[~finite]) and torch.isfinite(got[finite]).all()
