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


def _plain(m, cls):
    return type(m) is cls and not m._forward_hooks and not m._forward_pre_hooks and "forward" not in m.__dict__


def _transformed():
    """True under anything that has to see the individual operations."""
    return (torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or bool(_nn_module._global_forward_hooks)
            or bool(_nn_module._global_forward_pre_hooks) or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._len_torch_function_stack() > 0 or torch._C._functorch.peek_interpreter_stack() is not None)


def _layer_entry(layer, classes, sizes, ptrs, nums, dev, state, conv):
    """Appends one layer's row to both tables; False when the layer is not covered."""
    B, d, H, R, M, di = sizes
    block_cls, norm_cls, mixer_cls, gated_cls = classes
    if not _plain(layer, block_cls):
        return False
    norm, mixer = layer._modules["norm"], layer._modules["mixer"]
    if not _plain(norm, norm_cls) or not _plain(mixer, mixer_cls):
        return False
    mods = mixer._modules
    in_proj, conv1d, dyn, rw = mods["in_proj"], mods["conv1d"], mods["dyn_proj"], mods["rw_proj"]
    out_norm, out_proj = mods["out_norm"], mods["out_proj"]
    if not (_plain(in_proj, nn.Linear) and _plain(conv1d, nn.Conv1d) and _plain(dyn, nn.Linear)
            and _plain(rw, nn.Linear) and _plain(out_norm, gated_cls) and _plain(out_proj, nn.Linear)):
        return False
    if in_proj._parameters["bias"] is not None or out_proj._parameters["bias"] is not None:
        return False       # (a bias of rw_proj is not read by the modules either)
    if mixer.num_heads != H or mixer.head_dim != R or mixer.num_modes != M or mixer.conv_kernel != 4:
        return False
    own = mixer._parameters
    mask = 0
    bf16, f32 = torch.bfloat16, torch.float32
    for slot, t, n, either in (
            (0, norm._parameters["weight"], d, True), (1, in_proj._parameters["weight"], 2 * di * d, False),
            (2, conv1d._parameters["weight"], 4 * di, False), (3, conv1d._parameters["bias"], di, False),
            (4, dyn._parameters["weight"], 3 * H * di, False), (5, dyn._parameters["bias"], 3 * H, False),
            (6, rw._parameters["weight"], 2 * H * M * di, False), (7, own["dt_bias"], H, True),
            (8, own["read_residual_logit"], 1, True), (9, own["write_residual_scale"], 1, True),
            (10, mixer._buffers["base_log_tau"], M, True), (11, own["D"], di, True),
            (12, out_norm._parameters["weight"], di, True), (13, out_proj._parameters["weight"], d * di, False)):
        if t is None:
            if slot != 3 and slot != 5:
                return False
            ptrs.append(0)
            continue
        if t.dtype is not bf16:
            if not either or t.dtype is not f32:
                return False
            mask |= 1 << slot
        if t.get_device() != dev or t.numel() != n or not t.is_contiguous() or type(t) not in (nn.Parameter, torch.Tensor):
            return False
        ptrs.append(t.data_ptr())
    if ptrs[-12] & 7 or (ptrs[-13] | ptrs[-10] | ptrs[-8] | ptrs[-1]) & 15:   # conv weight; projection weights
        return False
    if state is None:
        ptrs.append(0)
        ptrs.append(0)
    else:
        if (state.dtype is not f32 or state.shape != (B, H, M, R) or not state.is_contiguous() or state.get_device() != dev
                or conv.dtype is not bf16 or conv.shape != (B, di, 3) or not conv.is_contiguous()
                or conv.get_device() != dev or state.data_ptr() & 15):
            return False
        ptrs.append(state.data_ptr())
        ptrs.append(conv.data_ptr())
    ptrs.extend((0, 0, mask))
    cfg = mixer.config
    nums.extend((norm.variance_epsilon, out_norm.variance_epsilon, mixer.read_temp, cfg.frac_dt_min, cfg.frac_dt_max,
                 cfg.frac_alpha_min, cfg.frac_alpha_max, cfg.frac_lambda_min, cfg.frac_lambda_max,
                 cfg.frac_gate_bias_init))
    return True


def decode_layers(layers, h, past, use_cache, classes):
    """h [B, 1, hidden] through `layers` -> (h, new past or None), or None when the call is not covered.
    `past`: per layer (state, conv_state), or None for a first token."""
    if type(h) is not torch.Tensor or h.dtype is not torch.bfloat16 or not h.is_cuda or h.dim() != 3 or h.shape[1] != 1:
        return None
    B, _, d = h.shape
    n = len(layers)
    if B < 1 or n < 1 or (past is not None and len(past) != n) or _transformed():
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
    sizes = (B, d, H, R, M, di)
    # every layer is looked at before the first launch: a call is covered as a whole or not at all
    ptrs, nums = [], []
    for i, layer in enumerate(layers):
        state = conv = None
        if past is not None and past[i] is not None:
            state, conv = past[i]
            if state is None or conv is None:
                return None
        if not _layer_entry(layer, classes, sizes, ptrs, nums, dev, state, conv):
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
