"""MusaAdam.apply_gradients takes any iterable of (grad, var) pairs.  One that makes
its pairs on demand sees every update before the next pair is asked for; a list
or tuple, whose pairs all exist before the call, shares launches."""
import subprocess
import sys

import pytest
import torch

from conftest import ROOT
from tensorflow_musa_extension_b200 import optimizers, raw_ops


class _Device(torch.Tensor):
    """A host tensor that the optimizer takes for a device tensor."""
    is_cuda = True


class _Launcher:
    """Stands in for the native path: an update is var -= grad."""

    def __init__(self):
        self.groups = []

    def adam_kind(self, var, m, v, grad):
        return 0

    def adam_group(self, group, *scalars):
        self.groups.append(len(group))
        for var, _, _, grad in group:
            var -= grad
        return 0


def _host(values):
    return torch.tensor(values, dtype=torch.float32).as_subclass(_Device)


def _refilled(variables, make):
    buf = make([0.0, 0.0])
    for i, var in enumerate(variables):
        buf.fill_(i + 1.0)
        yield buf, var


def _from_the_variable_before(variables, make):
    grad = make([1.0, 1.0])
    for var in variables:
        yield grad, var
        grad = var * 2.0


ITERABLES = {"refilled": _refilled, "from_the_variable_before": _from_the_variable_before,
             "zip": lambda variables, make: zip((g for g, _ in _refilled(variables, make)),
                                                variables)}


@pytest.mark.parametrize("kind", sorted(ITERABLES))
def test_pairs_made_on_demand_host(monkeypatch, kind):
    launcher = _Launcher()
    monkeypatch.setattr(raw_ops, "_native", lambda: launcher)
    got, want = ([_host([0.0, 0.0]) for _ in range(3)] for _ in range(2))
    assert optimizers.MusaAdam().apply_gradients(ITERABLES[kind](got, _host)) == 1
    for grad, var in ITERABLES[kind](want, _host):
        var -= grad
    assert [t.tolist() for t in got] == [t.tolist() for t in want]
    assert launcher.groups == [1, 1, 1]


@pytest.mark.parametrize("form", [list, tuple])
def test_pairs_at_hand_share_a_launch_host(monkeypatch, form):
    launcher = _Launcher()
    monkeypatch.setattr(raw_ops, "_native", lambda: launcher)
    vs = [_host([0.0]) for _ in range(3)]
    optimizers.MusaAdam().apply_gradients(form((_host([i + 1.0]), v) for i, v in enumerate(vs)))
    assert [v.item() for v in vs] == [-1.0, -2.0, -3.0] and launcher.groups == [3]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(ITERABLES))
def test_pairs_made_on_demand(kernel_lib, kind):
    """The bits of one op call per pair."""
    def make(values):
        return torch.tensor(values * 500, device="cuda")

    got, want = ([torch.full((1000,), 0.5 * i, device="cuda") for i in range(3)]
                 for _ in range(2))
    opt = optimizers.MusaAdam()
    opt.apply_gradients(ITERABLES[kind](got, make))
    for grad, var in ITERABLES[kind](want, make):
        m, v = torch.zeros_like(var), torch.zeros_like(var)
        raw_ops.MusaResourceApplyAdamMixed(var, m, v, 0.9, 0.999, 1e-3, 0.9, 0.999, 1e-7, grad)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


WITHOUT_MEMORY = """
import ctypes, resource, sys
sys.path.insert(0, %r)
import tensorflow_musa_extension_b200 as package
from tensorflow_musa_extension_b200 import _capi
lib = _capi.bind(package.get_library())
count = 1 << 22                     # the overlap check asks for 96 bytes of each
null = (ctypes.c_void_p * count)()
sizes = (ctypes.c_int64 * count)()  # empty variables: nothing to launch
pages = int(open("/proc/self/statm").read().split()[0])
limit = pages * resource.getpagesize() + (64 << 20)
resource.setrlimit(resource.RLIMIT_AS, (limit, limit))
sys.exit(lib.LaunchApplyAdamGroupHostTable(0, 0, null, null, null, null, sizes, count, 1e-3, 0.9,
                                           0.999, 1e-7, False, None))
"""


def test_group_launcher_without_host_memory(kernel_lib):
    """The check for variables that share memory needs a host table; without the
    memory for it the update is still made, variable by variable."""
    got = subprocess.run([sys.executable, "-c", WITHOUT_MEMORY % ROOT], capture_output=True,
                         text=True)
    # 35 and 100: the CUDA runtime's own answers on a machine without a device.
    assert got.returncode in (0, 35, 100), (got.returncode, got.stderr)
