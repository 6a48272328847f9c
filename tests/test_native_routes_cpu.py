"""What keeps the native model routes from standing in for the modules (no GPU needed: the modules are only looked at)."""

import pytest
import torch

from frac_ssm_b200.models import FracConfig, FracForCausalLM, decode
from frac_ssm_b200.models import modeling_frac as mf

CLASSES = (mf.FracBlock, mf.RMSNorm, mf.FracMixer, mf.RMSNormGated)


def _model(layers=3):
    return FracForCausalLM(FracConfig(vocab_size=16, hidden_size=64, num_hidden_layers=layers, num_attention_heads=2,
                                      frac_num_modes=8)).to(torch.bfloat16).model


def _looked_at(model):
    m = model.layers[0].mixer
    sizes = (m.hidden_size, m.num_heads, m.head_dim, m.num_modes, m.conv_kernel, m.inner_dim)
    return decode.layer_params(model.layers, CLASSES, sizes, -1)


def test_plain_modules_are_covered():
    found = _looked_at(_model())
    assert len(found) == 3 and all(mask == 0 and len(tensors) == 14 and len(nums) == 10 for tensors, mask, nums in found)


@pytest.mark.parametrize("path,name", [
    ("layers.1", "forward"), ("layers.2.norm", "forward"), ("layers.0.mixer", "forward"), ("layers.1.mixer", "_scan_params"),
    ("layers.1.mixer", "_conv_state_after"), ("layers.2.mixer.in_proj", "forward"), ("layers.0.mixer.out_norm", "forward")])
def test_a_method_set_on_an_instance_keeps_the_modules(path, name):
    model = _model()
    module = model.get_submodule(path)
    setattr(module, name, getattr(module, name))
    assert _looked_at(model) is None


@pytest.mark.parametrize("register", ["register_forward_hook", "register_forward_pre_hook"])
@pytest.mark.parametrize("path", ["layers.1", "layers.2.norm", "layers.0.mixer", "layers.1.mixer.rw_proj", "layers.2.mixer.out_norm"])
def test_a_hook_keeps_the_modules(path, register):
    model = _model()
    handle = getattr(model.get_submodule(path), register)(lambda *a: None)
    assert _looked_at(model) is None
    handle.remove()
    assert _looked_at(model) is not None


@pytest.mark.parametrize("owner,name", [
    (mf.FracBlock, "forward"), (mf.RMSNorm, "forward"), (mf.FracMixer, "forward"), (mf.FracMixer, "_scan_params"),
    (mf.FracMixer, "_conv_state_after"), (mf.RMSNormGated, "forward"), (torch.nn.Linear, "forward"),
    (torch.nn.Module, "__call__"), (mf, "causal_conv_silu"), (mf, "decode_step"), (mf, "frac_scan"), (mf, "scan_epilogue"),
    (mf, "rmsnorm_gated_fwd"), (mf, "compute_params_from_projections")])
def test_a_patched_class_or_function_keeps_the_modules(monkeypatch, owner, name):
    assert mf.as_defined()
    original = getattr(owner, name)
    monkeypatch.setattr(owner, name, lambda *a, **k: original(*a, **k))
    assert not mf.as_defined()


@pytest.mark.parametrize("path,name", [("layers.1.norm", "weight"), ("layers.0.mixer.in_proj", "weight"), ("layers.2.mixer", "D"),
                                       ("layers.1.mixer.dyn_proj", "bias"), ("layers.1.mixer", "base_log_tau"),
                                       ("layers.0.mixer.conv1d", "weight"), ("layers.0.mixer.in_proj", "bias")])
def test_a_tensor_kept_as_a_plain_attribute_keeps_the_modules(path, name):
    """(deleted as a parameter or buffer and set again: the modules' own forward finds it all the same)"""
    model = _model()
    module = model.get_submodule(path)
    value = getattr(module, name)
    delattr(module, name)
    object.__setattr__(module, name, None if value is None else value.detach())
    assert _looked_at(model) is None


def test_a_property_in_the_place_of_a_number_keeps_the_modules():
    model = _model()
    del model.layers[1].mixer.__dict__["read_temp"]
    assert _looked_at(model) is None


@pytest.mark.parametrize("path", ["layers.0.mixer.in_proj", "layers.2.mixer.out_proj", "layers.1.mixer.rw_proj", "layers.1.mixer.dyn_proj"])
def test_a_weight_of_another_shape_keeps_the_modules(path):
    """(which refuse it) although it has as many elements"""
    model = _model()
    module = model.get_submodule(path)
    module.weight = torch.nn.Parameter(module.weight.detach().t().contiguous())
    assert _looked_at(model) is None


def test_caches_in_other_containers_go_to_the_modules():
    pair = (torch.ones(1), torch.ones(1))
    for past in (None, (pair, pair), [None, pair], (list(pair), None)):
        assert decode._pairs(past, 2)
    once = (p for p in (pair, pair))
    assert not decode._pairs(once, 2) and len(list(once)) == 2      # not touched
    for past in ((pair,), {0: pair, 1: pair}.values(), (pair, (*pair, None)), (pair, torch.ones(2, 3)), (pair, iter(pair))):
        assert not decode._pairs(past, 2)
