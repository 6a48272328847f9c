"""The two forms of the decode step (csrc/decode_layers.cu), one kernel and a kernel a stage: several launches a call, heads
wider than a team, modes beyond a warp's share, captured calls, two streams at a time."""

import pytest
import torch

from tests.test_gpu_decode_layers import _flat, _model, _past

pytestmark = pytest.mark.gpu


# 35 layers are two launches of the one-kernel form; heads of 320 columns, 20, 129 and 600 modes (no warp's multiple, more
# than four items' worth of shared memory); more blocks' worth of items than SMs
@pytest.mark.parametrize("hidden,H,M,B,layers", [(32, 1, 8, 3, 35), (320, 1, 20, 2, 2), (64, 2, 600, 9, 2), (768, 24, 128, 16, 2), (640, 2, 129, 5, 1)])
def test_both_forms_give_the_same_bits(hidden, H, M, B, layers):
    """Up to 16 sequences a plain call is one kernel, a captured one a kernel a stage; both against float32."""
    half, model = _model(hidden, H, M, layers).to(torch.bfloat16), _model(hidden, H, M, layers)
    for p, q in zip(list(model.parameters()) + list(model.buffers()), list(half.parameters()) + list(half.buffers())):
        p.data.copy_(q.data)
    ids = torch.randint(1, 50, (B, 1), generator=torch.Generator().manual_seed(B)).cuda()
    with torch.no_grad():
        exact = _flat(model(ids, past_key_values=_past(model, B, torch.float32), use_cache=True))
        past = _past(half, B, torch.bfloat16)
        plain = [t.clone() for t in _flat(half(ids, past_key_values=past, use_cache=True))]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = _flat(half(ids, past_key_values=past, use_cache=True))
        graph.replay()
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(plain, captured))
    # one rounding of bfloat16 is 2^-9; a layer rounds its activations five times, and errors add up like a walk
    bound = 2 ** -9 * 5 * (2 + layers ** 0.5)
    for a, r in zip(plain, exact):
        assert (a.double() - r.double()).norm() < bound * r.double().norm()


def test_two_streams_at_a_time():
    """Two streams of kernels whose blocks share their work: neither waits for the other's."""
    models = [_model(256, 4, 128, 4).to(torch.bfloat16), _model(768, 12, 8, 3).to(torch.bfloat16)]
    ids = [torch.randint(1, 50, (b, 1)).cuda() for b in (1, 20)]
    pasts = [_past(m, i.shape[0], torch.bfloat16) for m, i in zip(models, ids)]
    with torch.no_grad():
        want = [m(i, past_key_values=p, use_cache=True)[0].clone() for m, i, p in zip(models, ids, pasts)]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in models]
        got = [[], []]
        for _ in range(50):
            for k, stream in enumerate(streams):
                with torch.cuda.stream(stream):
                    got[k].append(models[k](ids[k], past_key_values=pasts[k], use_cache=True)[0])
        torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(g, want[k]) for g in got[k])
