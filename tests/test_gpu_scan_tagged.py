"""The single-pass scan's two ways of handing the state from tile to tile: with tags beside the values for few
rows (up to 64; where one wave holds all tiles, or from 4, 12 or 24 tiles on), else through a counter.  The arithmetic is the same, so the results are the same bits."""

import pytest
import torch

from oracle import frac_oracle as O

pytestmark = pytest.mark.gpu


# one tile, edges of tiles, several chains deep; either side of 4, 12 and 24 tiles
@pytest.mark.parametrize("L", [1, 128, 129, 256, 384, 385, 1000, 1408, 1409, 2560, 2944, 2945])
@pytest.mark.parametrize("coeff", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("start,final", [(False, False), (True, True)])
def test_tagged_and_counted_hand_over_give_the_same_bits(L, coeff, start, final):
    from frac_ssm_b200.ops.b200 import frac_scan
    B = 65                                                           # the first count without tags
    u, c, kappa, rho, init = (t.cuda() for t in O.scan_inputs(B, L, 64, 128, dtype=torch.float32, gen="random", seed=L))
    u, c, kappa = u.bfloat16(), c.to(coeff), kappa.to(coeff)

    def run(rows):
        out = frac_scan(u[rows], c[rows], kappa[rows], rho[rows], 256, init[rows] if start else None, final,
                        final_state_dtype=torch.float32, path="fused", check=True)
        return out if final else (out,)
    ref = run(slice(0, B))
    for rows in (slice(0, 1), slice(3, 5), slice(0, 33), slice(16, 64), slice(1, 65)):
        for got, want in zip(run(rows), ref):
            assert torch.equal(got, want[rows])
