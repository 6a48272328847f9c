"""Scratch sizes of the C ABI (no GPU needed)."""

import pytest

from frac_ssm_b200 import _cabi as C

SHAPES = [(1, 1, 1, 1, 1), (2, 32768, 128, 16, 64), (192, 8192, 64, 128, 256), (24, 1048576, 64, 128, 256), (3, 1000, 96, 200, 32),
          (64, 8192, 64, 128, 256), (65, 8192, 64, 128, 256), (48, 1000, 128, 8, 32), (1, 100000, 8, 8, 256)]


@pytest.mark.parametrize("shape", SHAPES)
def test_scratch_sized_for_the_automatic_path_serves_every_path(shape):
    """A caller may size its scratch with path 0 once and call any path with it."""
    size = C.lib().fracssm_frac_scan_workspace_bytes
    assert size(*shape, C.PATH_AUTO) >= max(size(*shape, C.PATH_STAGED), size(*shape, C.PATH_FUSED))


def test_scratch_of_the_automatic_path_alone():
    lib = C.lib()
    for shape in SHAPES:
        need = lib.fracssm_frac_scan_auto_workspace_bytes(*shape)
        assert 0 < need <= lib.fracssm_frac_scan_workspace_bytes(*shape, C.PATH_AUTO)
    # the headline shape: the single-pass kernel's state, not the chunked stages' gigabyte
    assert lib.fracssm_frac_scan_auto_workspace_bytes(192, 8192, 64, 128, 256) < 8 << 20
    assert lib.fracssm_frac_scan_auto_workspace_bytes(0, 8192, 64, 128, 256) == 0


@pytest.mark.parametrize("shape,staged", [((8, 8192, 192, 40, 64), True), ((8, 8192, 192, 40, 32), False), ((8, 8192, 128, 128, 64), False),
                                          ((16, 16384, 64, 72, 128), True), ((2, 32768, 128, 40, 64), False),
                                          ((400, 2048, 192, 40, 64), False), ((16, 16384, 16, 100, 64), False)])
def test_scratch_of_the_automatic_path_holds_the_stages_where_dense_calls_take_them(shape, staged):
    """(they do where the segment kernels would load element by element and were measured to be slower)"""
    lib = C.lib()
    need = lib.fracssm_frac_scan_auto_workspace_bytes(*shape)
    assert (need >= lib.fracssm_frac_scan_workspace_bytes(*shape, C.PATH_STAGED)) == staged
