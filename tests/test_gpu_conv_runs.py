"""The bfloat16 convolution of width 4 in runs of 8, 16 and 32 tokens a thread, against float32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# run lengths by the size of the grid; sequences that end inside a group of four, a run, or before the history is full
@pytest.mark.parametrize("B,L,C", [(1, 2, 512), (1, 5, 8), (1, 397, 1536), (2, 1001, 1536), (3, 2050, 1032), (4, 4099, 520)])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("w_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("biased", [False, True])
def test_conv_runs(B, L, C, masked, w_dtype, biased):
    from frac_ssm_b200 import _cabi as K
    g = torch.Generator(device="cuda").manual_seed(L)
    xg = torch.randn(B, L, 2 * C, generator=g, device="cuda").bfloat16()
    w = torch.randn(C, 4, generator=g, device="cuda").to(w_dtype)
    bias = torch.randn(C, generator=g, device="cuda").to(w_dtype) if biased else None
    mask = torch.rand(B, L, generator=g, device="cuda") if masked else None
    y, u = (torch.full(s, float("nan"), device="cuda", dtype=torch.bfloat16) for s in ((B, L, C), (B * C // 8, L, 8)))
    K.check(K.lib().fracssm_causal_conv_silu_heads(K.ptr(xg), K.BF16, L * 2 * C, 2 * C, K.ptr(mask), L, 1, K.ptr(w), K.ptr(bias),
                                                   K.dt(w), K.ptr(y), K.BF16, K.ptr(u), 8, B, L, C, 4, K.stream_of(xg)),
            "causal_conv_silu_heads")
    x = xg[..., :C].double()
    if masked:
        x = x * mask.double()[..., None]
    x = torch.nn.functional.pad(x.transpose(1, 2), (3, 0))
    acc = sum(w.double()[:, k:k + 1] * x[..., k:k + L] for k in range(4))
    size = sum((w.double()[:, k:k + 1] * x[..., k:k + L]).abs() for k in range(4))
    if biased:
        acc, size = acc + bias.double()[:, None], size + bias.double().abs()[:, None]
    exact = (acc * torch.sigmoid(acc)).transpose(1, 2)
    # a bf16 rounding (half of 2^-7); silu's slope is below 1.1 and its own error a few 2^-23 of |acc|; six float32 roundings
    bound = 2 ** -8 * exact.abs() + 2 ** -20 * size.transpose(1, 2) + 1e-30
    assert ((y.double() - exact).abs() <= bound).all()
    assert torch.equal(u.view(B, C // 8, L, 8).transpose(1, 2).reshape(B, L, C), y)
