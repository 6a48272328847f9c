"""Tags or counter where one wave of 148 blocks just holds all tiles, or just not: the same bits."""

import pytest
import torch

from oracle import frac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,tiles", [(2, 2), (64, 2), (49, 3), (50, 3), (37, 4), (38, 4), (24, 6), (25, 6)])
@pytest.mark.parametrize("coeff", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("ragged", [0, 1, 127])
def test_few_tiles_a_row(B, tiles, coeff, ragged):
    from frac_ssm_b200.ops.b200 import frac_scan
    L = tiles * 128 - ragged
    inputs = O.scan_inputs(B, L, 64, 128, dtype=torch.float32, gen="random", seed=tiles)
    # the reference: more rows than take the tags, whose first ones are these
    u, c, kappa, rho, init = (t.repeat(-(-66 // B), *[1] * (t.dim() - 1)).cuda() for t in inputs)
    u, c, kappa = u.bfloat16(), c.to(coeff), kappa.to(coeff)

    def run(n):
        return frac_scan(u[:n], c[:n], kappa[:n], rho[:n], 256, init[:n], True, final_state_dtype=torch.float32, path="fused",
                         check=True)
    for got, want in zip(run(B), run(u.shape[0])):
        assert torch.equal(got, want[:B])
