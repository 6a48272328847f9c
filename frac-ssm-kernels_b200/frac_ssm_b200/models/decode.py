"""One token through all layers in native code (`csrc/decode_layers.cu`): one kernel, or four per layer.

Covers bfloat16 models on one GPU, one token per sequence, up to 64 sequences, no attention mask.  The
parameters are looked up in the modules on every call (nothing is remembered between calls), and whatever
this route would pass by (hooks, replaced, patched or subclassed modules, autocast, tracing, function transforms)
sends the call back to the modules' own forward.
"""

from __future__ import annotations

import array
from itertools import chain, repeat
from operator import attrgetter, contains, itemgetter

import torch
from torch import nn
from torch.nn.modules import module as _nn_module

from .. import _cabi as C

_PTRS = 19      # columns of the pointer table of fracssm_decode_layers
_ptr = torch.Tensor.data_ptr
_MAY_BE_F32 = 1 << 0 | 0b111111 << 7      # the norm weights and the small parameters
_parts = itemgetter("in_proj", "conv1d", "dyn_proj", "rw_proj", "out_norm", "out_proj")
_modules, _parameters = itemgetter("_modules"), itemgetter("_parameters")
_TENSORS = frozenset((nn.Parameter, torch.Tensor))


def transformed():
    """True under anything that has to see the individual operations."""
    return (torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or bool(_nn_module._global_forward_hooks)
            or bool(_nn_module._global_forward_pre_hooks) or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._len_torch_function_stack() > 0 or torch._C._functorch.peek_interpreter_stack() is not None
            or torch._C._get_tracing_state() is not None or torch.autograd.forward_ad._current_level >= 0)


def layer_params(layers, classes, sizes, dev):
    """Per layer its 14 parameters (None for an absent bias), the bit mask of those that are float32, and its numbers,
    in the order of the tables of fracssm_decode_layers; None when native code does not cover the layers."""
    try:
        return _layer_params(layers, classes, sizes, dev)
    except (KeyError, AttributeError):      # something is not where the modules' own __init__ puts it
        return None


def _layer_params(layers, classes, sizes, dev):
    """The same question goes to all modules or parameters at once: there are hundreds of each, and asked one by one
    the answers cost as much as the launches."""
    d, H, R, M, K, di = sizes
    block_cls, norm_cls, mixer_cls, gated_cls = classes
    layers = list(layers)
    if set(map(type, layers)) != {block_cls}:
        return None
    inner = [layer.__dict__["_modules"] for layer in layers]
    norms, mixers = [m["norm"] for m in inner], [m["mixer"] for m in inner]
    if set(map(type, mixers)) != {mixer_cls} or set(map(type, norms)) != {norm_cls}:
        return None
    own = list(map(vars, mixers))
    parts = list(chain.from_iterable(map(_parts, map(_modules, own))))      # six a layer
    if list(map(type, parts)) != [nn.Linear, nn.Conv1d, nn.Linear, nn.Linear, gated_cls, nn.Linear] * len(layers):
        return None
    part_dicts = list(map(vars, parts))
    dicts = [*map(vars, layers), *map(vars, norms), *own, *part_dicts]
    if (any(map(itemgetter("_forward_hooks"), dicts)) or any(map(itemgetter("_forward_pre_hooks"), dicts))
            or any(map(contains, dicts, repeat("forward"))) or any(map(contains, own, repeat("_scan_params")))
            or any(map(contains, own, repeat("_conv_state_after")))):
        return None
    counts = (d, 2 * di * d, K * di, di, 3 * H * di, 3 * H, 2 * H * M * di, H, 1, 1, M, di, di, d * di)
    found, every, expected, products = [], [], [], []
    last_cfg = cfg_nums = None
    held = map(_parameters, part_dicts)
    for i, (norm, m, in_proj, conv1d, dyn, rw, out_norm, out_proj) in enumerate(zip(norms, own, held, held, held, held, held,
                                                                                    held)):
        if in_proj["bias"] is not None or out_proj["bias"] is not None:
            return None        # (a bias of rw_proj is not read by the modules either)
        if m["num_heads"] != H or m["head_dim"] != R or m["num_modes"] != M or m["conv_kernel"] != K:
            return None
        p, norm = m["_parameters"], vars(norm)
        tensors = (norm["_parameters"]["weight"], in_proj["weight"], conv1d["weight"], conv1d["bias"], dyn["weight"],
                   dyn["bias"], rw["weight"], p["dt_bias"], p["read_residual_logit"], p["write_residual_scale"],
                   m["_buffers"]["base_log_tau"], p["D"], out_norm["weight"], out_proj["weight"])
        products += (tensors[1], tensors[4], tensors[6], tensors[13])
        if tensors[3] is None or tensors[5] is None:
            every += [t for t in tensors if t is not None]
            expected += [n for t, n in zip(tensors, counts) if t is not None]
        else:
            every += tensors
            expected += counts
        cfg = m["config"]
        if cfg is not last_cfg:
            last_cfg, cfg_nums = cfg, (cfg.frac_dt_min, cfg.frac_dt_max, cfg.frac_alpha_min, cfg.frac_alpha_max,
                                       cfg.frac_lambda_min, cfg.frac_lambda_max, cfg.frac_gate_bias_init)
        found.append((tensors, (norm["variance_epsilon"], part_dicts[6 * i + 4]["variance_epsilon"], m["read_temp"], *cfg_nums)))
    T = torch.Tensor
    if not _TENSORS.issuperset(map(type, every)):      # (a missing weight is no tensor either)
        return None
    if set(map(T.get_device, every)) != {dev} or list(map(T.numel, every)) != expected or not all(map(T.is_contiguous, every)):
        return None
    if list(map(attrgetter("shape"), products)) != [(2 * di, d), (3 * H, di), (2 * H * M, di), (d, di)] * len(layers):
        return None
    bf16 = torch.bfloat16
    if set(map(attrgetter("dtype"), every)) == {bf16}:
        return [(tensors, 0, nums) for tensors, nums in found]
    out = []
    for tensors, nums in found:
        mask = 0
        for slot, t in enumerate(tensors):
            if t is not None and t.dtype is not bf16:
                if t.dtype is not torch.float32 or not _MAY_BE_F32 >> slot & 1:
                    return None
                mask |= 1 << slot
        out.append((tensors, mask, nums))
    return out


def _pairs(past, n):
    """Whether `past` is None or n times None or (state, conv_state), in tuples or lists.  (The modules take it from any
    iterable, also one that can be gone through once only, and refuse other entries.)"""
    if past is None:
        return True
    kinds = (tuple, list)
    return (isinstance(past, kinds) and len(past) == n
            and all(p is None or (isinstance(p, kinds) and len(p) == 2) for p in past))


def decode_layers(layers, h, past, use_cache, classes):
    """h [B, 1, hidden] through `layers` -> (h, new past or None), or None when the call is not covered.
    `past`: per layer (state, conv_state), or None for a first token."""
    if type(h) is not torch.Tensor or h.dtype is not torch.bfloat16 or not h.is_cuda or h.dim() != 3 or h.shape[1] != 1:
        return None
    B, _, d = h.shape
    n = len(layers)
    if B < 1 or n < 1 or transformed() or not _pairs(past, n):
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
    found = layer_params(layers, classes, sizes, dev)
    if found is None:
        return None
    states = convs = None
    if past is None or all(p is None for p in past):
        olds = [(0, 0)] * n
    else:
        if any(p is None or p[0] is None or p[1] is None for p in past):
            return None
        states, convs = [p[0] for p in past], [p[1] for p in past]
        f32, bf16 = torch.float32, torch.bfloat16
        if not _TENSORS.issuperset(map(type, states)) or not _TENSORS.issuperset(map(type, convs)):
            return None        # (a subclass may have to see the operations)
        for ts, dtype, shape in ((states, f32, (B, H, M, R)), (convs, bf16, (B, di, 3))):
            for t in ts:
                if t.dtype is not dtype or t.shape != shape or not t.is_contiguous() or t.get_device() != dev:
                    return None
        olds = [(s.data_ptr(), c.data_ptr()) for s, c in zip(states, convs)]
        if any(s & 15 for s, _ in olds):
            return None
    ptrs, nums = [], []
    for (tensors, mask, numbers), old in zip(found, olds):
        if tensors[3] is not None and tensors[5] is not None:
            row = list(map(_ptr, tensors))
        else:
            row = [0 if t is None else t.data_ptr() for t in tensors]
        if row[2] & 7 or (row[1] | row[4] | row[6] | row[13]) & 15:   # conv weight; projection weights
            return None
        ptrs += row
        ptrs += old
        ptrs += (0, 0, mask)
        nums += numbers
    new_past = None
    if use_cache:
        # (a tensor of its own for each layer: who keeps or saves one keeps no other)
        if states is None:
            states = [torch.empty(B, H, M, R, device=h.device, dtype=torch.float32)] * n
            convs = [torch.empty(B, di, 3, device=h.device, dtype=torch.bfloat16)] * n
        states, convs = list(map(torch.empty_like, states)), list(map(torch.empty_like, convs))
        ptrs[16::_PTRS] = map(_ptr, states)
        ptrs[17::_PTRS] = map(_ptr, convs)
        new_past = tuple(zip(states, convs))
    table, numbers = array.array("Q", ptrs), array.array("f", nums)
    out = torch.empty(B, 1, d, device=h.device, dtype=torch.bfloat16)
    with C.trace("decode_layers"), torch.cuda.device(dev):
        nbytes = lib.fracssm_decode_layers_workspace_bytes(B, d, H, R, M)
        ws = torch.empty(nbytes, device=h.device, dtype=torch.uint8)
        C.check(lib.fracssm_decode_layers(table.buffer_info()[0], numbers.buffer_info()[0], n, C.ptr(h), C.ptr(out),
                                          C.ptr(ws), nbytes, B, d, H, R, M, K, C.stream_of(h)), "decode_layers")
    return out, new_past
