"""The segment scan's summary by groups of 8 tokens (csrc/scan_modes.cu), with and without 16-byte loads: lengths around a
group and a segment, decays whose product over a group underflows, and the carry over every number of segments' form."""

import pytest
import torch

from oracle import frac_oracle as O
from tests.test_gpu_scan_modes import _exact, _rel

pytestmark = pytest.mark.gpu


# one token more and less than groups and segments of 16 tokens; all numbers of modes' groups; columns of one and two blocks
@pytest.mark.parametrize("B,L,R,M", [(2, 31, 64, 8), (2, 33, 128, 16), (1, 47, 64, 32), (3, 17, 256, 16), (2, 129, 64, 64), (1, 40, 128, 128),
                                     (2, 33, 60, 16), (1, 47, 64, 30)])
@pytest.mark.parametrize("dtype,coeff", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_groups_match_recurrence(B, L, R, M, dtype, coeff):
    from frac_ssm_b200.ops.b200 import frac_scan
    u, c, kappa, rho, init = O.scan_inputs(B, L, R, M, dtype=torch.float32, gen="model_like", seed=L + R + M)
    u, c, kappa = u.to(dtype), c.to(coeff), kappa.to(coeff)
    rho[:, L // 3:2 * L // 3, ::2] = 1e-7        # whole groups at the floor of 1e-6: seven such decays are 1e-42
    h, fin = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True, final_state_dtype=torch.float32)
    h_ref, f_ref = _exact(u, c, kappa, rho, init)
    # outputs are rounded once; float32 sums of at most L * M terms whose roundings are of either sign
    assert _rel(h, h_ref) <= {torch.bfloat16: 2 ** -8, torch.float32: 2e-6}[dtype]
    assert _rel(fin, f_ref) <= 2e-6


# 8, 12, 24, 48 and more segments for each of the carry's 32 warps
@pytest.mark.parametrize("L", [4000, 5000, 10000, 20000, 30000])
def test_carry_over_any_number_of_segments(L):
    from frac_ssm_b200 import _cabi as C
    from frac_ssm_b200.ops.b200 import frac_scan
    R, M = 64, 8
    nseg = C.lib().fracssm_frac_scan_auto_workspace_bytes(1, L, R, M, 32) // (4 * M * (R + 1))
    assert nseg == (L + 15) // 16
    u, c, kappa, rho, init = O.scan_inputs(1, L, R, M, dtype=torch.float32, gen="model_like", seed=L)
    h, fin = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True)
    h_ref, f_ref = _exact(u, c, kappa, rho, init)
    bound = 2.0 ** -23 * L ** 0.5         # roundings of at most L steps, of either sign
    assert _rel(h, h_ref) <= bound and _rel(fin, f_ref) <= bound


def test_an_infinity_stays_one_where_decays_underflow():
    """Eight decays at the floor are 1e-48, which is zero; the state that the recurrence keeps is infinite all the same."""
    from frac_ssm_b200.ops.b200 import frac_scan
    u, c, kappa, rho, init = O.scan_inputs(1, 64, 64, 16, dtype=torch.float32, gen="model_like", seed=3)
    c, kappa = c.abs().add(0.01), kappa.abs().add(0.01)
    u[0, 8, 5] = float("inf")
    rho[:, 8:16] = 1e-6
    rho[:, 16:] = rho[:, 16:].clamp_min(0.5)
    h, _ = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True)
    h_ref, _ = _exact(u, c, kappa, rho, init)
    assert torch.equal(torch.isinf(h.cpu()), torch.isinf(h_ref)) and not torch.isnan(h).any()


# (64, 16), (128, 64) load in 16-byte pieces, (60, 16) and (64, 30) element by element, the last with padded modes
@pytest.mark.parametrize("R,M", [(64, 16), (128, 64), (60, 16), (64, 30)])
@pytest.mark.parametrize("L,where,floored,small", [
    (64, 3, (8, 16), 1.0),         # the group behind the infinity's, within a segment
    (64, 3, (16, 32), 1.0),        # the whole segment behind the infinity's: what the carry multiplies with
    (64, 8, (9, 16), 1e-12),       # a weight whose product with seven decays underflows although neither is zero
    (5000, 5, (6, 5000), 1.0)])    # every segment behind it, over the carry's shares
def test_an_infinity_outlasts_decays_that_underflow(R, M, L, where, floored, small):
    """In the recurrence each decay is 1e-6 or more, and an infinity times that stays one."""
    from frac_ssm_b200.ops.b200 import frac_scan
    u, c, kappa, rho, init = O.scan_inputs(1, L, R, M, dtype=torch.float32, gen="model_like", seed=L + R)
    c, kappa = c.abs().add(0.01), kappa.abs().add(0.01) * small
    u[0, where, 5] = float("inf")
    rho = rho.clamp_min(0.5)
    rho[:, floored[0]:floored[1]] = 1e-6
    h, fin = frac_scan(*(t.cuda() for t in (u, c, kappa, rho)), 32, init.cuda(), True)
    h_ref, f_ref = _exact(u, c, kappa, rho, init)
    assert torch.isinf(h_ref[0, where:, 5]).all()
    assert torch.equal(torch.isinf(h.cpu()), torch.isinf(h_ref)) and not torch.isnan(h).any()
    assert torch.equal(torch.isinf(fin.cpu()), torch.isinf(f_ref)) and not torch.isnan(fin).any()
