"""A prompt through all layers with few calls per layer: bfloat16 models on one GPU.

Between the three library GEMMs of a layer stand three native calls (residual addition + norm; convolution, the next
token's history and the narrow dynamic projection; parameter prep, scan, state and epilogue), the small parameters are read in their own types
and the intermediates live in buffers that all layers share.  As with `decode.py`, nothing is remembered between
calls and whatever has to see the individual modules or operations keeps the modules' own forward.
"""

from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F
from torch import nn

from .. import _cabi as C
from .. import parallel
from ..modules.rmsnorm_gated import rmsnorm_gated_fwd
from ..ops.b200.frac_scan import taken_whole
from .decode import layer_params, transformed

_MAX_NORM = 2048      # longest row of fracssm_add_rmsnorm


def prefill_layers(layers, h, attention_mask, use_cache, classes):
    """h [B, L, hidden], L > 1, through `layers` from an empty cache -> (h, new past or None), or None when the call
    is not covered."""
    if type(h) is not torch.Tensor or h.dtype is not torch.bfloat16 or not h.is_cuda or h.dim() != 3:
        return None
    B, L, d = h.shape
    n_layers = len(layers)
    if B < 1 or L < 2 or n_layers < 1 or d % 8 or d > _MAX_NORM or transformed() or type(layers) is not nn.ModuleList:
        return None
    if not h.is_contiguous() or h.data_ptr() & 15:
        return None
    if type(layers[0]) is not classes[0] or type(layers[0].mixer) is not classes[2]:
        return None
    mixer = layers[0].mixer
    H, R, M, K, T = mixer.num_heads, mixer.head_dim, mixer.num_modes, mixer.conv_kernel, mixer.chunk_size
    di = H * R
    dev = h.get_device()
    if not 2 <= K <= 8 or not isinstance(T, int) or T < 1 or B * H > 65535:
        return None
    if not taken_whole(B * H, L) and parallel._auto_local_splits(B * H, L, T, 1, h.device) > 1:   # frac_scan cuts them up
        return None
    mask = None
    if attention_mask is not None:
        # (the modules copy a mask over from another device, but refuse one where the cache needs it)
        if type(attention_mask) is not torch.Tensor or attention_mask.shape != (B, L) or attention_mask.get_device() != dev:
            return None
        mask = attention_mask.to(torch.float32).contiguous()
    coeff = mixer.coeff_dtype
    if coeff not in (None, torch.float32, torch.bfloat16):
        return None
    coeff = torch.float32 if coeff is None else coeff
    sizes = (d, H, R, M, K, di)
    # a call is covered as a whole or not at all
    found = layer_params(layers, classes, sizes, dev)
    if found is None:
        return None
    for layer in layers:
        m = layer.mixer
        if m.fuse_gate_into_scan or (torch.float32 if m.coeff_dtype is None else m.coeff_dtype) is not coeff or m.chunk_size != T:
            return None

    lib, bf16, f32 = C.lib(), torch.bfloat16, torch.float32

    def empty(*shape, dtype=bf16):
        return torch.empty(*shape, device=h.device, dtype=dtype)

    rows = B * L
    own_dyn = 3 * H <= 192 and di % 8 == 0 and rows <= 1 << 30      # (what fracssm_prefill_conv_dyn covers)
    with C.trace("prefill_layers"), torch.cuda.device(dev):
        stream = C.stream_of(h)
        nbytes = lib.fracssm_frac_scan_auto_workspace_bytes(B * H, L, R, M, T)
        ws = empty(max(nbytes, 256), dtype=torch.uint8)
        x_conv, u, scan_out = empty(rows, di), empty(B * H, L, R), empty(B * H, L, R)
        y = u.view(rows, di)      # (the epilogue writes it when the scan has read u)
        c, kappa, rho = empty(B * H, L, M, dtype=coeff), empty(B * H, L, M, dtype=coeff), empty(B * H, L, M, dtype=f32)
        total = empty(rows, d) if n_layers > 1 else None      # the residual from the second layer on
        fin = states = tails = None
        if use_cache:
            fin = empty(B * H, R, M, dtype=f32)
            # (a tensor of its own for each layer: who keeps or saves one keeps no other)
            states, tails = [empty(B, H, M, R, dtype=f32)], [empty(B, di, K - 1)]
            for _ in range(n_layers - 1):
                states.append(torch.empty_like(states[0]))
                tails.append(torch.empty_like(tails[0]))
        p_ws, p_conv, p_u, p_h, p_y, p_c, p_k, p_rho, p_fin, p_total, p_mask = (
            0 if t is None else t.data_ptr() for t in (ws, x_conv, u, scan_out, y, c, kappa, rho, fin, total, mask))
        ck = C.dt_of(coeff)
        res, out, n = h.view(rows, d), None, None
        for i, (t, f32_mask, nums) in enumerate(found):
            (norm_w, in_w, conv_w, conv_b, dyn_w, dyn_b, rw_w, dt_bias, read_logit, write_logit, log_tau, D, out_norm_w,
             out_w) = t
            if i == 0:
                n = rmsnorm_gated_fwd(res, norm_w, None, nums[0])[0]
            else:
                p_out = out.data_ptr()      # (the norm takes its place)
                C.check(lib.fracssm_add_rmsnorm(res.data_ptr(), p_out, norm_w.data_ptr(),
                                                C.F32 if f32_mask & 1 else C.BF16, nums[0], p_total, p_out, rows, d,
                                                stream), "add_rmsnorm")
                res, n, out = total, out, None
            xg = F.linear(n, in_w)
            n = None      # (like xg below: what is no longer read makes room)
            p_x = xg.data_ptr()
            conv = (p_x, 2 * di, p_mask, conv_w.data_ptr(), 0 if conv_b is None else conv_b.data_ptr(), p_conv, p_u,
                    tails[i].data_ptr() if use_cache else 0)
            # (the bias of dyn is added where it is read)
            if own_dyn and not dyn_w.data_ptr() & 15:
                dyn = empty(rows, 3 * H)
                C.check(lib.fracssm_prefill_conv_dyn(*conv, dyn_w.data_ptr(), dyn.data_ptr(), 3 * H, R, B, L, di, K, stream),
                        "prefill_conv_dyn")
            else:
                C.check(lib.fracssm_prefill_conv(*conv, R, B, L, di, K, stream), "prefill_conv")
                dyn = F.linear(xg[:, :di], dyn_w)
            rw = F.linear(x_conv, rw_w)
            params = (ctypes.c_void_p * 6)(dt_bias.data_ptr(), read_logit.data_ptr(), write_logit.data_ptr(),
                                           log_tau.data_ptr(), D.data_ptr(), out_norm_w.data_ptr())
            numbers = (ctypes.c_float * 9)(*nums[2:], nums[1])
            C.check(lib.fracssm_prefill_mix(dyn.data_ptr(), 0 if dyn_b is None else dyn_b.data_ptr(), rw.data_ptr(), p_conv,
                                            p_x + 2 * di, 2 * di, p_mask, params, f32_mask >> 7 & 63, numbers, p_u, p_c,
                                            p_k, ck, p_rho, p_h, p_fin, states[i].data_ptr() if use_cache else 0, p_y,
                                            p_ws, ws.numel(), B, L, H, R, M, T, stream), "prefill_mix")
            del xg, dyn, rw      # (or the next layer's would be allocated beside them)
            out = F.linear(y, out_w)
        h = (res + out).view(B, L, d)
    return h, tuple(zip(states, tails)) if use_cache else None
