"""One token through all layers in native code (`csrc/decode_layers.cu`): four kernels per layer.

Covers bfloat16 models on one GPU, one token per sequence, up to 64 sequences, no attention mask.  The
parameters are looked up in the modules on every call (nothing is remembered between calls), and whatever
this route would pass by (hooks, replaced or subclassed modules, autocast, tracing, function transforms)
sends the call back to the modules' own forward.
"""

from __future__ import annotations

import array

import torch
from torch import nn
from torch.nn.modules import module as _nn_module

from .. import _cabi as C

_PTRS = 19      # columns of the pointer table of fracssm_decode_layers
_MAY_BE_F32 = 1 << 0 | 0b111111 << 7      # the norm weights and the small parameters
_TENSORS = (nn.Parameter, torch.Tensor)


def _plain(m, cls):
    return type(m) is cls and not m._forward_hooks and not m._forward_pre_hooks and "forward" not in m.__dict__


def transformed():
    """True under anything that has to see the individual operations."""
    return (torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or bool(_nn_module._global_forward_hooks)
            or bool(_nn_module._global_forward_pre_hooks) or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._len_torch_function_stack() > 0 or torch._C._functorch.peek_interpreter_stack() is not None)


def layer_params(layer, classes, sizes, dev):
    """One layer's 14 parameters (None for an absent bias), the bit mask of those that are float32, and its numbers,
    in the order of the tables of fracssm_decode_layers; None when native code does not cover the layer."""
    d, H, R, M, K, di = sizes
    block_cls, norm_cls, mixer_cls, gated_cls = classes
    if not _plain(layer, block_cls):
        return None
    norm, mixer = layer._modules["norm"], layer._modules["mixer"]
    if not _plain(norm, norm_cls) or not _plain(mixer, mixer_cls):
        return None
    mods = mixer._modules
    in_proj, conv1d, dyn, rw = mods["in_proj"], mods["conv1d"], mods["dyn_proj"], mods["rw_proj"]
    out_norm, out_proj = mods["out_norm"], mods["out_proj"]
    if not (_plain(in_proj, nn.Linear) and _plain(conv1d, nn.Conv1d) and _plain(dyn, nn.Linear)
            and _plain(rw, nn.Linear) and _plain(out_norm, gated_cls) and _plain(out_proj, nn.Linear)):
        return None
    if in_proj._parameters["bias"] is not None or out_proj._parameters["bias"] is not None:
        return None        # (a bias of rw_proj is not read by the modules either)
    if mixer.num_heads != H or mixer.head_dim != R or mixer.num_modes != M or mixer.conv_kernel != K:
        return None
    own = mixer._parameters
    tensors = (norm._parameters["weight"], in_proj._parameters["weight"], conv1d._parameters["weight"],
               conv1d._parameters["bias"], dyn._parameters["weight"], dyn._parameters["bias"], rw._parameters["weight"],
               own["dt_bias"], own["read_residual_logit"], own["write_residual_scale"], mixer._buffers["base_log_tau"],
               own["D"], out_norm._parameters["weight"], out_proj._parameters["weight"])
    mask = slot = 0
    bf16, f32 = torch.bfloat16, torch.float32
    for t, n in zip(tensors, (d, 2 * di * d, K * di, di, 3 * H * di, 3 * H, 2 * H * M * di, H, 1, 1, M, di, di, d * di)):
        if t is None:
            if slot != 3 and slot != 5:
                return None
        else:
            if t.dtype is not bf16:
                if t.dtype is not f32 or not _MAY_BE_F32 >> slot & 1:
                    return None
                mask |= 1 << slot
            if t.get_device() != dev or t.numel() != n or not t.is_contiguous() or type(t) not in _TENSORS:
                return None
        slot += 1
    cfg = mixer.config
    return tensors, mask, (norm.variance_epsilon, out_norm.variance_epsilon, mixer.read_temp, cfg.frac_dt_min,
                           cfg.frac_dt_max, cfg.frac_alpha_min, cfg.frac_alpha_max, cfg.frac_lambda_min,
                           cfg.frac_lambda_max, cfg.frac_gate_bias_init)


def _layer_entry(layer, classes, sizes, B, ptrs, nums, dev, state, conv):
    """Appends one layer's row to both tables; False when the layer is not covered."""
    found = layer_params(layer, classes, sizes, dev)
    if found is None:
        return False
    tensors, mask, numbers = found
    d, H, R, M, K, di = sizes
    row = [0 if t is None else t.data_ptr() for t in tensors]
    if row[2] & 7 or (row[1] | row[4] | row[6] | row[13]) & 15:   # conv weight; projection weights
        return False
    ptrs += row
    if state is None:
        ptrs += (0, 0)
    else:
        if (state.dtype is not torch.float32 or state.shape != (B, H, M, R) or not state.is_contiguous()
                or state.get_device() != dev or conv.dtype is not torch.bfloat16 or conv.shape != (B, di, 3)
                or not conv.is_contiguous() or conv.get_device() != dev or state.data_ptr() & 15):
            return False
        ptrs += (state.data_ptr(), conv.data_ptr())
    ptrs += (0, 0, mask)
    nums += numbers
    return True


def decode_layers(layers, h, past, use_cache, classes):
    """h [B, 1, hidden] through `layers` -> (h, new past or None), or None when the call is not covered.
    `past`: per layer (state, conv_state), or None for a first token."""
    if type(h) is not torch.Tensor or h.dtype is not torch.bfloat16 or not h.is_cuda or h.dim() != 3 or h.shape[1] != 1:
        return None
    B, _, d = h.shape
    n = len(layers)
    if B < 1 or n < 1 or (past is not None and len(past) != n) or transformed():
        return None
    if type(layers) is not nn.ModuleList or not h.is_contiguous() or h.data_ptr() & 15:
        return None
    if type(layers[0]) is not classes[0] or type(layers[0].mixer) is not classes[2]:
        return None
    mixer = layers[0].mixer
    H, R, M, K = mixer.num_heads, mixer.head_dim, mixer.num_modes, mixer.conv_kernel
    di = H * R
    lib = C.lib()
    if not lib.fracssm_decode_layers_supported(B, d, H, R, M, K):
        return None
    dev = h.get_device()
    sizes = (d, H, R, M, K, di)
    # every layer is looked at before the first launch: a call is covered as a whole or not at all
    ptrs, nums = [], []
    for i, layer in enumerate(layers):
        state = conv = None
        if past is not None and past[i] is not None:
            state, conv = past[i]
            if state is None or conv is None:
                return None
        if not _layer_entry(layer, classes, sizes, B, ptrs, nums, dev, state, conv):
            return None
    new_past = None
    if use_cache:
        states = torch.empty(n, B, H, M, R, device=h.device, dtype=torch.float32).unbind(0)
        convs = torch.empty(n, B, di, 3, device=h.device, dtype=torch.bfloat16).unbind(0)
        for i in range(n):
            ptrs[i * _PTRS + 16] = states[i].data_ptr()
            ptrs[i * _PTRS + 17] = convs[i].data_ptr()
        new_past = tuple(zip(states, convs))
    table, numbers = array.array("Q", ptrs), array.array("f", nums)
    out = torch.empty(B, 1, d, device=h.device, dtype=torch.bfloat16)
    with C.trace("decode_layers"), torch.cuda.device(dev):
        nbytes = lib.fracssm_decode_layers_workspace_bytes(B, d, H, R, M)
        ws = torch.empty(nbytes, device=h.device, dtype=torch.uint8)
        C.check(lib.fracssm_decode_layers(table.buffer_info()[0], numbers.buffer_info()[0], n, C.ptr(h), C.ptr(out),
                                          C.ptr(ws), nbytes, B, d, H, R, M, K, C.stream_of(h)), "decode_layers")
    return out, new_past
