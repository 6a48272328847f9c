"""When a launch function is called directly and when through its registered op (no GPU needed)."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from frac_ssm_b200.ops.b200 import stages


class _Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Sub(torch.Tensor):
    pass


def test_direct_only_where_nothing_observes_the_op():
    x = torch.ones(2)
    w = torch.ones(2, requires_grad=True)
    assert stages._unobserved((x, 3, 1.0, None, True, torch.bfloat16))
    assert not stages._unobserved((x, w))
    with torch.no_grad():
        assert stages._unobserved((x, w, torch.nn.Parameter(x)))
    assert not stages._unobserved((x.as_subclass(_Sub),))
    negated = torch.complex(x, x).conj().imag       # its memory holds x, its values are -x
    assert negated.is_neg() and not stages._unobserved((x, negated))
    with _Mode():
        assert not stages._unobserved((x,))
    seen = []
    torch.vmap(lambda t: seen.append(stages._unobserved((t,))) or t)(torch.ones(3, 2))
    with torch.autograd.forward_ad.dual_level():
        seen.append(stages._unobserved((x,)))
    torch.jit.trace(lambda t: seen.append(stages._unobserved((t,))) or t + 1, x, check_trace=False)
    assert seen and not any(seen)


def test_few_long_rows_are_cut_where_that_was_measured_to_be_faster():
    import importlib
    fs = importlib.import_module("frac_ssm_b200.ops.b200.frac_scan")

    def splits(B, L):
        u = torch.empty(B, L, 64, dtype=torch.bfloat16, device="meta")
        return fs._row_splits(u, torch.empty(B, L, 128, dtype=torch.bfloat16, device="meta"), 256)
    assert splits(12, 1048576) == 16 and splits(13, 524288) == 16 and splits(12, 131072) == 16
    assert splits(12, 65536) == splits(13, 32768) == 1       # 12 x 32768 tokens: 0.42 ms whole, 0.68 cut
    assert splits(14, 1048576) == splits(24, 1048576) == 1   # 24 rows: 13.7 ms whole, 16.6 cut
    assert splits(8, 1048576) == 32 and splits(3, 32768) == 32


@pytest.fixture(scope="module")
def double():
    """An op like the package's own, and how often its function ran."""
    runs = []

    @stages._op("test_double")
    def _double_op(x: torch.Tensor, times: int) -> torch.Tensor:
        runs.append(times)
        return x * times

    @_double_op.register_fake
    def _(x, times):
        return torch.empty_like(x)
    return _double_op, runs


def test_a_profiled_call_shows_the_registered_op(double):
    op, runs = double
    x = torch.ones(2)
    op(x, 2)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        assert torch.equal(op(x, 3), x * 3)
    assert any(e.key == "frac_ssm_b200::test_double" for e in prof.key_averages())
    assert runs[-2:] == [2, 3]


def test_the_returned_function_has_the_ops_own_methods(double):
    op, runs = double
    assert op._qualname == "frac_ssm_b200::test_double" and op._opoverload is torch.ops.frac_ssm_b200.test_double.default
    assert op(x=torch.ones(2), times=2).sum() == 4
    compiled = torch.compile(lambda t: op(t, 4) + 1, fullgraph=True, backend="eager")
    assert compiled(torch.ones(2)).sum() == 10
    for name in ("register_kernel", "register_fake", "register_autograd", "register_vmap", "register_torch_dispatch",
                 "register_autocast", "set_kernel_enabled"):
        assert callable(getattr(op, name)), name
    x = torch.ones(2)

    @op.register_kernel("cpu")
    def _(x, times):
        return x * times + 1
    n = len(runs)
    assert torch.equal(op(x, 2), x * 2 + 1) and len(runs) == n      # what was registered runs, not the function
    with op.set_kernel_enabled("cpu", False):
        assert torch.equal(op(x, 2), x * 2) and len(runs) == n + 1
    assert torch.equal(op(x, 2), x * 2 + 1) and len(runs) == n + 1


@pytest.mark.parametrize("register", ["register_kernel", "register_vmap", "register_torch_dispatch", "register_autocast"])
def test_what_is_registered_by_the_ops_name_runs(register):
    name = f"frac_ssm_b200::test_by_name_{register}"

    @stages._op(name.split("::")[1])
    def _twice_op(x: torch.Tensor) -> torch.Tensor:
        return x * 2
    assert _twice_op._direct
    if register == "register_kernel":
        torch.library.register_kernel(name, "cpu", lambda x: x * 3)
        assert torch.equal(_twice_op(torch.ones(2)), torch.full((2,), 3.0))
    elif register == "register_vmap":
        torch.library.register_vmap(name, lambda info, dims, x: (x * 5, 0))
        assert torch.equal(torch.vmap(_twice_op)(torch.ones(2)), torch.full((2,), 5.0))
    elif register == "register_torch_dispatch":
        torch.library.register_torch_dispatch(name, _Mode, lambda mode, func, types, args, kwargs: args[0] * 7)
        with _Mode():
            assert torch.equal(_twice_op(torch.ones(2)), torch.full((2,), 7.0))
    else:
        torch.library.register_autocast(name, "cpu", torch.bfloat16)
        with torch.autocast("cpu", torch.bfloat16):
            assert _twice_op(torch.ones(2)).dtype == torch.bfloat16
    assert not _twice_op._direct
