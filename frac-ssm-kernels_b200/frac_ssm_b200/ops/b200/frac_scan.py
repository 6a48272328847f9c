"""The composed forward scan on the B200 CUDA extension.

Backend-module interface of the reference (`frac_ssm/ops/triton/frac_scan.py:102-130`):
`frac_scan(u, c, kappa, rho, chunk_size, initial_state=None, return_final_state=False)`.
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from ... import _cabi as C
from .stages import _op

# "auto": the single-pass tcgen05 kernel when it covers the shape, else the segment kernels (up to 128 modes, where they
# are the faster ones), else the staged kernels.
_PATHS = {"auto": C.PATH_AUTO, "staged": C.PATH_STAGED, "fused": C.PATH_FUSED}

def frac_scan(u, c, kappa, rho, chunk_size, initial_state=None, return_final_state=False, *,
              final_state_dtype=None, path="auto", check=False):
    """Fractional chunked scan, forward.

    Args:
        u: [B, L, R] input features (bfloat16, float16 or float32); dim 0 is batch*heads.
        c, kappa: [B, L, M] read / write coefficients, same dtype as each other (u's or float32).
        rho: [B, L, M] float32 decay.
        chunk_size: tokens per chunk.
        initial_state: [B, R, M] float32 or None.
        return_final_state: also return the state after the last token.
        final_state_dtype: dtype of the returned state; default follows the reference
            (bfloat16 when u is bfloat16, else float32).  The state is always carried in float32.
        path: "auto", "staged" or "fused".  "auto" takes the single-pass kernel when it covers the
            shape, else up to 128 modes the segment kernels (but for large calls whose rows these
            could not load in 16-byte pieces), else the staged ones.  For very few rows with many
            tokens (fewer than 12 rows from 32768 tokens on, 12 and 13 rows from 131072 on) it cuts
            every row into sub-segments first, because a row is one chain of tiles and 148 SMs want
            more chains than that: one summary pass over u, kappa and rho gives every sub-segment
            its incoming state, then all sub-segments are scanned as rows
            (`parallel.seq_parallel_scan`).
        check: after the launch, synchronise and raise if a bounded device-side wait of the
            single-pass kernel ran out (debugging aid; the default stays asynchronous).
    Returns:
        h [B, L, R] in u.dtype, and final_state [B, R, M] if requested.
    """
    assert rho.dtype == torch.float32, "rho must be float32 for numerical stability"
    if initial_state is not None:
        assert initial_state.dtype == torch.float32, "initial_state must be float32"
    assert u.dim() == 3, f"u must be 3D (B, L, R), got {u.dim()}D"
    assert c.dim() == 3, f"c must be 3D (B, L, M), got {c.dim()}D"
    assert kappa.dim() == 3, f"kappa must be 3D (B, L, M), got {kappa.dim()}D"
    assert rho.dim() == 3, f"rho must be 3D (B, L, M), got {rho.dim()}D"
    assert all(x.is_cuda for x in (u, c, kappa, rho)), "inputs must be on CUDA"
    assert c.dtype == kappa.dtype and c.dtype in (u.dtype, torch.float32), (
        "c and kappa dtype must match u dtype or be float32"
    )
    assert isinstance(chunk_size, int) and chunk_size > 0, (
        f"chunk_size must be a positive integer, got {chunk_size}"
    )
    B, L, R = u.shape
    M = c.shape[-1]
    assert c.shape == (B, L, M) and kappa.shape == (B, L, M) and rho.shape == (B, L, M), (
        "c, kappa and rho shapes must match (B, L, M)"
    )
    if initial_state is not None:
        assert initial_state.shape == (B, R, M), "initial_state shape must be (B, R, M)"
        assert initial_state.is_cuda, "initial_state must be on CUDA"
    if final_state_dtype is None:
        final_state_dtype = torch.bfloat16 if u.dtype == torch.bfloat16 else torch.float32
    assert final_state_dtype in (torch.float32, torch.bfloat16)

    path_code = _PATHS[path]
    if path == "auto" and not check and not torch.compiler.is_compiling():
        splits = _row_splits(u, c, chunk_size)
        if splits > 1:
            from ... import parallel
            h, fin = parallel.seq_parallel_scan(u, c, kappa, rho, chunk_size, initial_state, True,
                                                local_splits=splits, process_local=True)
            return (h, fin.to(final_state_dtype)) if return_final_state else h
    if check:      # the status read-back bypasses the registered op (it needs the scratch)
        h, fin = _launch(u, c, kappa, rho, chunk_size, initial_state, return_final_state,
                         final_state_dtype == torch.float32, path_code, check)
    else:
        h, fin = _frac_scan_fwd_op(u, c, kappa, rho, chunk_size, initial_state, return_final_state,
                                   final_state_dtype == torch.float32, path_code)
    if return_final_state:
        return h, fin
    return h


def taken_whole(B, L):
    """Whether the single-pass kernel takes B rows of L tokens as they are, however long.

    Whole, a row's chain of tiles advances a tile per 1.05 us and a CTA needs some 10 us a tile; cutting the rows costs
    a second read of u, kappa and rho and a step on the host per sub-segment, some 13 us each where nothing hides it.
    Milliseconds whole / cut, bfloat16 coefficients (float32 lies the same way):

                     32768          131072         524288         1048576
         8 rows   0.36 / 1.53    1.21 / 1.34    4.66 / 3.05    9.23 / 5.77
        12 rows   0.42 / 0.68    1.29 / 1.21    4.91 / 4.23    9.75 / 8.23
        13 rows   0.40 / 0.70    1.29 / 1.30    4.95 / 4.56    9.86 / 9.03
        14 rows   0.38 / 0.70    1.33 / 1.39    5.05 / 4.90   10.01 / 10.10
        24 rows   0.50 / 0.65    1.77 / 2.11    6.82 / 8.04   13.74 / 16.59

    Below 12 rows the line stays at the 32768 tokens of `parallel._auto_local_splits`, although fewer than 131072 (and
    up to 4 rows more) would be faster whole: both entry points cut there.
    """
    return B >= 14 or (B >= 12 and L < 131072)


def _row_splits(u, c, chunk_size):
    """Sub-segments per row for the "auto" path: more than 1 only where the single-pass kernel covers
    both the call and the cut-up call, the tensors are dense, and the rows are few and long."""
    from ... import parallel
    B, L, R = u.shape
    if B < 1 or taken_whole(B, L) or not (u.is_contiguous() and c.is_contiguous()) or u.dtype != torch.bfloat16:
        return 1
    splits = parallel._auto_local_splits(B, L, chunk_size, 1, u.device)
    if splits > 1 and not C.lib().fracssm_scan_fused_supported(B * splits, L // splits, R, c.shape[-1],
                                                               chunk_size, C.dt(u), C.dt(c)):
        return 1
    return splits


def _launch(u, c, kappa, rho, chunk_size, initial_state, want_final, final_fp32, path_code, check=False):
    B, L, R = u.shape
    M = c.shape[-1]
    final_state_dtype = torch.float32 if final_fp32 else torch.bfloat16
    u, c, kappa, rho = C.rows(u), C.rows(c), C.rows(kappa), C.rows(rho)
    init = None if initial_state is None else initial_state.contiguous()
    h = torch.empty(B, L, R, device=u.device, dtype=u.dtype)
    fin = torch.empty(B, R, M, device=u.device, dtype=final_state_dtype) if want_final else None
    if L == 0:      # no token: the state passes through unchanged (zeros without an initial state)
        if want_final:
            if init is None:
                fin.zero_()
            else:
                fin.copy_(init)
        return h, fin
    if B > 0:
        lib = C.lib()
        with C.trace("frac_scan"), C.device_of(u):
            su, sc, sk, sr = u.stride(), c.stride(), kappa.stride(), rho.stride()
            # (strided inputs may take the chunked stages where dense ones take the segment kernels)
            if path_code == C.PATH_AUTO and all([t.is_contiguous() for t in (u, c, kappa, rho)]):
                nbytes = lib.fracssm_frac_scan_auto_workspace_bytes(B, L, R, M, chunk_size)
            else:
                nbytes = lib.fracssm_frac_scan_workspace_bytes(B, L, R, M, chunk_size, path_code)
            nbytes = max(nbytes, 256)
            ws = torch.empty(nbytes, device=u.device, dtype=torch.uint8)
            C.check(lib.fracssm_frac_scan_fwd(
                u.data_ptr(), C.dt(u), su[0], su[1], c.data_ptr(), kappa.data_ptr(), C.dt(c), sc[0], sc[1], sk[0], sk[1],
                rho.data_ptr(), sr[0], sr[1], None if init is None else init.data_ptr(), h.data_ptr(),
                None if fin is None else fin.data_ptr(), C.dt_of(final_state_dtype), ws.data_ptr(), nbytes, B, L, R, M,
                chunk_size, path_code, C.raw_stream(u)), "frac_scan")
            if check and L > 0 and path_code != C.PATH_STAGED and u.is_contiguous() and \
                    lib.fracssm_scan_fused_supported(B, L, R, M, chunk_size, C.dt(u), C.dt(c)):
                C.check(lib.fracssm_scan_fused_status(C.ptr(ws), C.stream_of(u)), "frac_scan")
    if fin is None:
        fin = torch.empty(0, device=u.device, dtype=final_state_dtype)
    return h, fin


# Registered as a torch custom op (with a shape-only "fake" implementation) so that callers can put
# the scan inside torch.compile(fullgraph=True), as the reference does for its ops
# (frac_ssm/ops/triton/chunk_state.py:243-302).  Forward only: asking for gradients raises.
@_op("frac_scan_fwd")
def _frac_scan_fwd_op(u: torch.Tensor, c: torch.Tensor, kappa: torch.Tensor, rho: torch.Tensor,
                      chunk_size: int, initial_state: Optional[torch.Tensor], want_final: bool,
                      final_fp32: bool, path_code: int) -> Tuple[torch.Tensor, torch.Tensor]:
    return _launch(u, c, kappa, rho, chunk_size, initial_state, want_final, final_fp32, path_code)


@_frac_scan_fwd_op.register_fake
def _(u, c, kappa, rho, chunk_size, initial_state, want_final, final_fp32, path_code):
    B, L, R = u.shape
    M = c.shape[-1]
    fdt = torch.float32 if final_fp32 else torch.bfloat16
    fin = torch.empty((B, R, M) if want_final else (0,), device=u.device, dtype=fdt)
    return torch.empty(B, L, R, device=u.device, dtype=u.dtype), fin


__all__ = ["frac_scan"]
