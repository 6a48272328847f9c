"""The one-kernel decode step (csrc/decode_layers.cu) works with the blocks that are there: any number of them gives the bits of
the kernel-per-stage form, and SMs that other streams hold for long stop nothing."""

import ctypes
import time

import pytest
import torch

from tests.helpers import selftest_lib
from tests.test_gpu_decode_layers import _flat, _model, _past

pytestmark = pytest.mark.gpu

ERR_WAIT = 4


class _Form:
    """Calls of fracssm_decode_layers go to a self-test entry with these last arguments; status: what its status call said."""

    def __init__(self, *last, entry="decode_layers", types=(ctypes.c_int, ctypes.c_int)):
        self.last, self.name, self.types, self.status = last, "fracssm_selftest_" + entry, types, None

    def __enter__(self):
        from frac_ssm_b200 import _cabi as C
        self.lib, test = C.lib(), selftest_lib()
        self.fn, form = self.lib.fracssm_decode_layers, getattr(test, self.name)
        form.argtypes, form.restype = [*self.fn.argtypes, *self.types], ctypes.c_int
        test.fracssm_decode_layers_status.argtypes = [ctypes.c_void_p, ctypes.c_void_p]

        def call(*a):
            rc = form(*a, *self.last)
            self.status = test.fracssm_decode_layers_status(a[5], a[13])      # synchronises
            return rc
        self.lib.fracssm_decode_layers = call
        return self

    def __exit__(self, *exc):
        self.lib.fracssm_decode_layers = self.fn


# one block; two, of which one takes dyn_proj; fewer and more blocks than tiles or items; more blocks than run at a time, whose
# last ones find the list closed; groups of 8, 16 and 32 sequences; two launches of the one-kernel form
@pytest.mark.parametrize("hidden,H,M,B,layers", [(256, 4, 128, 1, 3), (768, 12, 8, 9, 2), (768, 24, 128, 17, 2), (320, 5, 20, 29, 2), (64, 2, 8, 32, 35)])
def test_any_number_of_blocks_gives_the_same_bits(hidden, H, M, B, layers):
    model = _model(hidden, H, M, layers).to(torch.bfloat16)
    ids = torch.randint(1, 50, (B, 1), generator=torch.Generator().manual_seed(B)).cuda()
    past = _past(model, B, torch.bfloat16)

    def step():
        return [t.clone() for t in _flat(model(ids, past_key_values=past, use_cache=True))]
    with torch.no_grad():
        with _Form(0, 0):
            want = step()
        for blocks in (1, 2, 3, 37, 147, 0, 300):
            with _Form(1, blocks) as form:
                assert all(torch.equal(a, b) for a, b in zip(step(), want)), blocks
            assert form.status == 0


@pytest.mark.parametrize("B", [1, 20])
def test_a_step_beside_kernels_that_hold_sms(B):
    """Eight kernels of other streams keep eight SMs for half a second: the step neither waits for them nor goes wrong."""
    model = _model(768, 24, 128, 4).to(torch.bfloat16)
    ids = torch.randint(1, 50, (B, 1)).cuda()
    past = _past(model, B, torch.bfloat16)
    with torch.no_grad():
        want = [t.clone() for t in _flat(model(ids, past_key_values=past, use_cache=True))]
        torch.cuda.synchronize()
        held = []
        for _ in range(8):
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                torch.cuda._sleep(1_000_000_000)
                held.append(torch.cuda.Event())
                held[-1].record()
        got = _flat(model(ids, past_key_values=past, use_cache=True))
        torch.cuda.current_stream().synchronize()
        assert not any(e.query() for e in held)
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


# which form a captured call takes: 17 to 32 sequences go by the weights of a layer, 12 MB and more are one kernel
@pytest.mark.parametrize("H,M,B,one", [(24, 128, 17, True), (24, 128, 20, True), (24, 128, 32, True), (24, 128, 16, False), (12, 8, 17, False),
                                       (12, 8, 32, False), (12, 64, 20, False), (24, 33, 20, True)])
def test_captured_steps_give_the_same_bits(H, M, B, one):
    model = _model(768, H, M, 3).to(torch.bfloat16)
    ids = torch.randint(1, 50, (B, 1)).cuda()
    past = _past(model, B, torch.bfloat16)
    with torch.no_grad():
        plain = [t.clone() for t in _flat(model(ids, past_key_values=past, use_cache=True))]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            captured = _flat(model(ids, past_key_values=past, use_cache=True))
        nodes = ctypes.c_size_t()
        handle = ctypes.c_void_p(graph.raw_cuda_graph())
        assert ctypes.CDLL("libcudart.so.12").cudaGraphGetNodes(handle, None, ctypes.byref(nodes)) == 0
        assert (nodes.value < 4 * 3) == one
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(plain, captured))


# the first barrier, after which the others wait in vain too; the last one, after which they finish; one of a first launch of two
@pytest.mark.parametrize("B,layers,barrier", [(1, 2, 1), (1, 2, 7), (20, 2, 7), (3, 35, 127), (3, 35, 60)])
def test_a_wait_that_runs_out_marks_everything(B, layers, barrier):
    """One block waits for an arrival that is not to come, for two milliseconds at most."""
    model = _model(64, 2, 8, layers).to(torch.bfloat16)
    ids = torch.randint(1, 50, (B, 1)).cuda()
    past = _past(model, B, torch.bfloat16)
    with torch.no_grad():
        want = [t.clone() for t in _flat(model(ids, past_key_values=past, use_cache=True))]
        t0 = time.time()
        with _Form(barrier, 2_000_000, entry="decode_wait_limit", types=(ctypes.c_int, ctypes.c_uint64)) as form:
            got = _flat(model(ids, past_key_values=past, use_cache=True))
        assert time.time() - t0 < 5.0 and form.status == ERR_WAIT
        assert all(torch.isnan(t).all() for t in got)
        again = _flat(model(ids, past_key_values=past, use_cache=True))      # the context is usable as before
    assert all(torch.equal(a, b) for a, b in zip(again, want))


def test_the_entries_are_part_of_the_test_library_alone():
    from frac_ssm_b200 import _cabi as C
    product = ctypes.CDLL(C.lib_path())
    assert not any(hasattr(product, "fracssm_selftest_" + n) for n in ("decode_layers", "decode_wait_limit"))
