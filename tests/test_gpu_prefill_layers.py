"""The few-calls prefill (models/prefill.py) against the modules' own forward."""

import pytest
import torch

from tests.test_gpu_decode_layers import _Count, _flat, _model

pytestmark = pytest.mark.gpu


def _hooked(model, *args, **kw):
    """The same call with the modules' own forward: a hook keeps the native route away."""
    handle = model.model.layers[0].register_forward_hook(lambda *a: None)
    out = model(*args, **kw)
    handle.remove()
    return out


# lengths around the convolution's history and the scan's tiles; single-pass and segment scans; odd widths; one layer,
# and layers enough for every buffer that they share to be used again
@pytest.mark.parametrize("hidden,H,M,B,L,layers", [
    (64, 2, 128, 1, 2, 2), (128, 4, 128, 2, 3, 2), (256, 8, 128, 2, 129, 2), (96, 3, 7, 3, 50, 2), (768, 12, 8, 2, 200, 2),
    (768, 24, 128, 1, 397, 2), (72, 3, 20, 2, 33, 2), (72, 3, 20, 2, 33, 1), (128, 4, 128, 2, 150, 5), (96, 3, 7, 3, 50, 4)])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("coeff", [None, torch.bfloat16])
def test_prefill_matches_modules(hidden, H, M, B, L, layers, masked, coeff):
    half = _model(hidden, H, M, layers).to(torch.bfloat16)
    exact_model = _model(hidden, H, M, layers)
    for p, q in zip(list(exact_model.parameters()) + list(exact_model.buffers()), list(half.parameters()) + list(half.buffers())):
        p.data.copy_(q.data)
    for layer in half.model.layers:
        layer.mixer.coeff_dtype = coeff
    ids = torch.randint(1, 50, (B, L), generator=torch.Generator().manual_seed(L)).cuda()
    mask = None
    if masked:
        mask = torch.ones(B, L, dtype=torch.long)
        mask[B - 1, : L // 2] = 0
        mask = mask.cuda()
    with _Count("fracssm_prefill_mix") as count:
        native = _flat(half(ids, attention_mask=mask, use_cache=True))
        logits, none = half(ids, attention_mask=mask, use_cache=False)
        assert count.n == 2 * layers
        assert none is None and torch.equal(logits, native[0])
        modules = _flat(_hooked(half, ids, attention_mask=mask, use_cache=True))
        assert count.n == 2 * layers
    exact = _flat(exact_model(ids, attention_mask=mask, use_cache=True))
    for n, m, e in zip(native, modules, exact):
        assert n.shape == m.shape and n.dtype == m.dtype and n.is_contiguous()
        scale = e.float().norm().clamp_min(1e-6)
        err, err_m = ((x.float() - e.float()).norm() / scale for x in (n, m))
        # the same roundings at the same places: the same error up to chance
        assert err <= 1.25 * err_m + 2e-3, (err, err_m)


def test_mixed_parameter_types_and_other_masks():
    half = _model(64, 2, 16).to(torch.bfloat16)
    for layer in half.model.layers:
        layer.mixer.base_log_tau = layer.mixer.base_log_tau.float()
        layer.mixer.D.data = layer.mixer.D.data.float()
        layer.norm.weight.data = layer.norm.weight.data.float()
    ids = torch.ones(2, 40, dtype=torch.long).cuda()
    mask = torch.ones(2, 40, device="cuda", dtype=torch.bool)
    mask[0, 30:] = False
    for m in (mask, mask.float() * 0.3, mask.t().contiguous().t()):
        with _Count("fracssm_prefill_mix") as count:
            native = _flat(half(ids, attention_mask=m, use_cache=True))
            assert count.n == 2
        for a, b in zip(native, _flat(_hooked(half, ids, attention_mask=m, use_cache=True))):
            assert (a.float() - b.float()).norm() <= 2e-2 * b.float().norm() + 1e-3


@pytest.mark.parametrize("H,M,B,L", [(24, 128, 2, 3000), (24, 128, 1, 397), (12, 8, 8, 3000)])
@pytest.mark.parametrize("use_cache", [False, True])
def test_prefill_needs_no_more_memory_than_the_modules(H, M, B, L, use_cache):
    """The modules with the scratch of the chunked stages, which the scan allocated before it had the segment kernels:
    what fitted the GPU then still does."""
    from frac_ssm_b200 import _cabi as C
    half = _model(768, H, M, layers=4).to(torch.bfloat16)
    ids = torch.ones(B, L, dtype=torch.long).cuda()
    lib = C.lib()
    alone = lib.fracssm_frac_scan_auto_workspace_bytes

    def peak(run):
        run(half, ids, use_cache=use_cache)      # (the library GEMMs' own workspace)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        run(half, ids, use_cache=use_cache)
        torch.cuda.synchronize()
        return torch.cuda.max_memory_allocated() - before
    native = peak(lambda m, *a, **k: m(*a, **k))
    lib.fracssm_frac_scan_auto_workspace_bytes = lambda *a: lib.fracssm_frac_scan_workspace_bytes(*a, C.PATH_AUTO)
    try:
        modules = peak(_hooked)
    finally:
        lib.fracssm_frac_scan_auto_workspace_bytes = alone
    assert native <= modules, (native / B / L, modules / B / L)


def test_a_mask_on_another_device_is_refused_with_a_cache_as_by_the_modules():
    half = _model(64, 2, 16).to(torch.bfloat16)
    ids, mask = torch.ones(2, 40, dtype=torch.long).cuda(), torch.ones(2, 40, dtype=torch.long)
    for run in (half, lambda *a, **k: _hooked(half, *a, **k)):
        run(ids, attention_mask=mask, use_cache=False)
        with pytest.raises(RuntimeError, match="same device"):
            run(ids, attention_mask=mask, use_cache=True)


@pytest.mark.parametrize("rows,D", [(1, 8), (5, 768), (4, 2048), (3, 264)])
@pytest.mark.parametrize("w_dtype", [torch.bfloat16, torch.float32])
def test_add_rmsnorm(rows, D, w_dtype):
    from frac_ssm_b200 import _cabi as C
    g = torch.Generator().manual_seed(D)
    x, y = (torch.randn(rows, D, generator=g).bfloat16().cuda() for _ in range(2))
    w = (1 + 0.1 * torch.randn(D, generator=g)).to(w_dtype).cuda()
    total, norm = torch.empty_like(x), torch.empty_like(x)
    C.check(C.lib().fracssm_add_rmsnorm(C.ptr(x), C.ptr(y), C.ptr(w), C.dt(w), 1e-6, C.ptr(total), C.ptr(norm), rows, D,
                                        C.stream_of(x)), "add_rmsnorm")
    x2, y2 = x.clone(), y.clone()          # in place: the sum over x, the norm over y
    C.check(C.lib().fracssm_add_rmsnorm(C.ptr(x2), C.ptr(y2), C.ptr(w), C.dt(w), 1e-6, C.ptr(x2), C.ptr(y2), rows, D,
                                        C.stream_of(x)), "add_rmsnorm")
    assert torch.equal(x2, total) and torch.equal(y2, norm)
    assert torch.equal(total, x + y)
    s = total.double()
    ref = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert (norm.double() - ref).abs().max() <= 2 ** -8 * ref.abs().max()      # one rounding to bfloat16


# runs of 8, 16 and 32 tokens a thread: with the shorter ones the tail is written by the same launch
@pytest.mark.parametrize("B,L,C", [(1, 2, 64), (2, 50, 72), (4, 1000, 1536), (8, 3000, 1536), (64, 200, 520)])
@pytest.mark.parametrize("masked", [False, True])
def test_prefill_conv_and_its_tail(B, L, C, masked):
    from frac_ssm_b200 import _cabi as abi
    from frac_ssm_b200.models.modeling_frac import causal_conv_silu
    g = torch.Generator(device="cuda").manual_seed(L + C)
    xg = torch.randn(B, L, 2 * C, device="cuda", generator=g).bfloat16()
    x, w = xg[..., :C], torch.randn(C, 1, 4, device="cuda", generator=g).bfloat16()
    bias = torch.randn(C, device="cuda", generator=g).bfloat16()
    mask = (torch.rand(B, L, device="cuda", generator=g) > 0.3).float() if masked else None
    y, tail = torch.empty(B, L, C, device="cuda", dtype=torch.bfloat16), torch.empty(B, C, 3, device="cuda", dtype=torch.bfloat16)
    abi.check(abi.lib().fracssm_prefill_conv(abi.ptr(x), 2 * C, abi.ptr(mask), abi.ptr(w), abi.ptr(bias), abi.ptr(y), None,
                                             abi.ptr(tail), 0, B, L, C, 4, abi.stream_of(x)), "prefill_conv")
    assert torch.equal(y, causal_conv_silu(x, w, bias, mask))
    kept = x if mask is None else x * mask[..., None].bfloat16()
    assert torch.equal(tail, torch.nn.functional.pad(kept.transpose(1, 2), (3, 0))[..., -3:])
