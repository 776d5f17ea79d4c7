"""The ops where the extension module of the native host path cannot be loaded:
one warning, then every call takes the general path."""
import logging
import sys

import numpy as np
import pytest
import torch

import tensorflow_musa_extension_b200 as package
from oracle import np_ref
from helpers import assert_close, to_numpy
from tensorflow_musa_extension_b200 import optimizers, raw_ops


@pytest.fixture
def no_extension(monkeypatch):
    monkeypatch.delattr(package, "_native_ops", raising=False)
    monkeypatch.setitem(sys.modules, package.__name__ + "._native_ops", None)
    monkeypatch.setattr(raw_ops, "_bound_native", None)


def test_one_warning_and_every_call_declined(monkeypatch, caplog, no_extension, kernel_lib):
    monkeypatch.setattr(raw_ops, "_require_cuda", lambda: None)
    with caplog.at_level(logging.WARNING, logger=raw_ops.__name__):
        for _ in range(2):
            native = raw_ops._native()
            assert native.adam_kind(1, 2, 3, 4) == -1
            assert native.bn_forward(*range(9)) is None and native.layer_norm(1, 2, 3, 4) is None
    assert len(caplog.records) == 1
    assert "tensorflow_musa_extension_b200.build" in caplog.text


@pytest.mark.gpu
def test_ops_without_the_extension(no_extension, kernel_lib):
    rng = np.random.default_rng(0)
    x = rng.standard_normal((6, 5, 24)).astype(np.float32)
    g, b = (rng.uniform(0.5, 1.5, 24).astype(np.float32) for _ in range(2))
    e = np.empty(0, np.float32)
    want = np_ref.fused_batch_norm(x, g, b, epsilon=1e-3)
    for form in (lambda a: a, lambda a: torch.from_numpy(a).cuda()):   # host and device inputs
        got = raw_ops.FusedBatchNormV3(form(x), form(g), form(b), form(e), form(e), epsilon=1e-3)
        assert_close(to_numpy(got.y), want[0], 1e-4, 1e-4, "y")
        y = raw_ops.MusaLayerNorm(form(x), form(g), form(b))
        assert_close(to_numpy(y), np_ref.layer_norm(x, g, b), 1e-4, 1e-5, "layer norm")
    got, want = torch.from_numpy(x).cuda(), torch.from_numpy(x).cuda()
    grad = torch.full_like(got, 0.25)
    optimizers.MusaAdam().apply_gradients([(grad, got)])
    raw_ops.MusaResourceApplyAdamMixed(want, torch.zeros_like(want), torch.zeros_like(want), 0.9,
                                       0.999, 1e-3, 0.9, 0.999, 1e-7, grad)
    assert torch.equal(got, want)
