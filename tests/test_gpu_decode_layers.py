"""The native decode step over all layers (csrc/decode_layers.cu) against the modules' own token loop."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(hidden, H, M, layers=2, vocab=50):
    from frac_ssm_b200.models import FracConfig, FracForCausalLM
    torch.manual_seed(hidden + H + M)
    m = FracForCausalLM(FracConfig(vocab_size=vocab, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=H,
                                   frac_num_modes=M))
    with torch.no_grad():
        for name, p in m.named_parameters():
            if "conv1d" in name:
                p.uniform_(-0.5, 0.5)
            elif p.dim() == 2 and "embed" not in name:
                p.normal_(0, p.shape[1] ** -0.5)
            elif name.endswith(("dt_bias", "bias")):
                p.normal_(0, 0.3)
            elif "norm" in name:
                p.uniform_(0.8, 1.2)
    return m.cuda().eval()


def _past(model, B, dtype, seed=0):
    cfg = model.config
    g = torch.Generator().manual_seed(seed)
    H, M, R = cfg.num_attention_heads, cfg.frac_num_modes, cfg.frac_head_dim
    return tuple((0.1 * torch.randn(B, H, M, R, generator=g).cuda(),
                  torch.randn(B, cfg.intermediate_size, 3, generator=g).bfloat16().to(dtype).cuda())
                 for _ in range(cfg.num_hidden_layers))


class _Count:
    """Counts the calls of a native function."""

    def __init__(self, name="fracssm_decode_layers"):
        self.name = name

    def __enter__(self):
        from frac_ssm_b200 import _cabi as C
        self.lib, self.n = C.lib(), 0
        self.fn = getattr(self.lib, self.name)

        def counted(*a):
            self.n += 1
            return self.fn(*a)
        setattr(self.lib, self.name, counted)
        return self

    def __exit__(self, *exc):
        setattr(self.lib, self.name, self.fn)


def _flat(out):
    logits, past = out
    return [logits] + ([] if past is None else [t for pair in past for t in pair])


# sequences around the groups of 8; widths that fill the 8 warps' shares unevenly; heads whose projections end
# inside a 16-row tile; modes that are no multiple of 4; one and several column shares per head; layers enough for the
# two buffers of the hidden state to be used again
@pytest.mark.parametrize("hidden,H,M,B,layers", [
    (32, 1, 8, 1, 2), (64, 2, 7, 2, 2), (96, 3, 16, 3, 2), (256, 4, 128, 8, 2), (256, 8, 33, 9, 2), (768, 24, 128, 1, 2),
    (768, 12, 8, 17, 2), (128, 2, 128, 33, 2), (768, 24, 128, 64, 2), (96, 3, 16, 2, 1), (128, 2, 20, 3, 5), (256, 4, 128, 20, 6)])
@pytest.mark.parametrize("first", [False, True])
def test_native_step_matches_modules(hidden, H, M, B, layers, first):
    half = _model(hidden, H, M, layers).to(torch.bfloat16)
    model = _model(hidden, H, M, layers)
    for p, q in zip(list(model.parameters()) + list(model.buffers()), list(half.parameters()) + list(half.buffers())):
        p.data.copy_(q.data)                                    # the same (rounded) weights in float32
    exact_past = None if first else _past(model, B, torch.float32)
    ids = torch.randint(1, 50, (B, 1), generator=torch.Generator().manual_seed(B)).cuda()
    exact = _flat(model(ids, past_key_values=exact_past, use_cache=True))
    past = None if first else _past(half, B, torch.bfloat16)
    kept = None if first else [t.clone() for pair in past for t in pair]
    with _Count() as count:
        native = _flat(half(ids, past_key_values=past, use_cache=True))
        again = _flat(half(ids, past_key_values=past, use_cache=True))
        logits_only, none = half(ids, past_key_values=past, use_cache=False)
        assert count.n == 3 and none is None
        handle = half.model.layers[0].mixer.out_proj.register_forward_hook(lambda *a: None)   # the modules' own loop
        modules = _flat(half(ids, past_key_values=past, use_cache=True))
        handle.remove()
        assert count.n == 3
    if not first:
        assert all(torch.equal(a, b) for a, b in zip(kept, [t for pair in past for t in pair]))   # inputs untouched
    assert torch.equal(logits_only, native[0])
    for n, a, m, e in zip(native, again, modules, exact):
        assert n.shape == m.shape and n.dtype == m.dtype and torch.equal(n, a)
        scale = e.float().norm().clamp_min(1e-6)
        err, err_m = ((x.float() - e.float()).norm() / scale for x in (n, m))
        # the native step rounds at the same places or not at all: no larger error, up to chance
        assert err <= 1.25 * err_m + 2e-3, (err, err_m)


def test_what_the_native_step_does_not_cover_still_runs():
    half = _model(64, 2, 8).to(torch.bfloat16)
    ids = torch.ones(2, 1, dtype=torch.long).cuda()
    past = _past(half, 2, torch.bfloat16)
    with _Count() as count:
        ref = half(ids, past_key_values=past, use_cache=True)
        assert count.n == 1
        masked = half(ids, attention_mask=torch.ones_like(ids), past_key_values=past, use_cache=True)
        strided = tuple((s.transpose(2, 3).contiguous().transpose(2, 3), c) for s, c in past)
        odd = half(ids, past_key_values=strided, use_cache=True)
        many = half(torch.ones(65, 1, dtype=torch.long).cuda(), use_cache=True)
        with torch.autocast("cuda", torch.bfloat16):
            half(ids, past_key_values=past, use_cache=True)
        assert count.n == 1
    assert many[0].shape[0] == 65
    for got in (masked, odd):
        for a, b in zip(_flat(got), _flat(ref)):
            assert (a.float() - b.float()).norm() <= 2e-2 * b.float().norm() + 1e-3


class _Seen(torch.Tensor):
    """A tensor subclass that sees the operations on it."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        _Seen.n += 1
        return super().__torch_function__(func, types, args, kwargs or {})


@pytest.mark.parametrize("which", [0, 1])
def test_cached_tensors_that_observe_operations_keep_the_modules(which):
    half = _model(64, 2, 8).to(torch.bfloat16)
    ids = torch.ones(2, 1, dtype=torch.long).cuda()
    past = _past(half, 2, torch.bfloat16)
    seen = tuple(tuple(t.as_subclass(_Seen) if i == which else t for i, t in enumerate(pair)) for pair in past)
    _Seen.n = 0
    with _Count() as count:
        half(ids, past_key_values=seen, use_cache=False)
        assert count.n == 0
    assert _Seen.n > 0


def test_a_cache_that_can_be_gone_through_once_is_taken_by_the_modules():
    half = _model(64, 2, 8).to(torch.bfloat16)
    ids = torch.ones(2, 1, dtype=torch.long).cuda()
    past = _past(half, 2, torch.bfloat16)
    with _Count() as count:
        got = half(ids, past_key_values=(pair for pair in past), use_cache=True)
        assert count.n == 0
        ref = half(ids, past_key_values=past, use_cache=True)
        with pytest.raises(ValueError):      # as the modules do
            half(ids, past_key_values=tuple((*pair, None) for pair in past), use_cache=True)
        assert count.n == 1
    for a, b in zip(_flat(got), _flat(ref)):
        assert (a.float() - b.float()).norm() <= 2e-2 * b.float().norm() + 1e-3


def test_each_layers_cache_is_a_tensor_of_its_own():
    half = _model(64, 2, 8, layers=3).to(torch.bfloat16)
    ids = torch.ones(2, 1, dtype=torch.long).cuda()
    with _Count() as count:
        first = half(ids, use_cache=True)[1]
        then = half(ids, past_key_values=first, use_cache=True)[1]
        assert count.n == 2
    prompt = half(torch.ones(2, 9, dtype=torch.long).cuda(), use_cache=True)[1]
    for past in (first, then, prompt):
        tensors = [t for pair in past for t in pair]
        assert len({t.untyped_storage().data_ptr() for t in tensors}) == 6
        for t in tensors:
            assert t.untyped_storage().nbytes() == t.numel() * t.element_size() and not t._is_view()


def test_native_step_in_a_cuda_graph():
    half = _model(256, 4, 16).to(torch.bfloat16)
    ids = torch.ones(2, 1, dtype=torch.long).cuda()
    past = _past(half, 2, torch.bfloat16)
    ref = _flat(half(ids, past_key_values=past, use_cache=True))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _flat(half(ids, past_key_values=past, use_cache=True))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, ref))
