"""Outputs of the native host path: tensors of their own, down to the storage."""
import pytest
import torch

from tensorflow_musa_extension_b200 import raw_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 127, 128, 2048])
def test_small_outputs_do_not_overlap(kernel_lib, c):
    x = torch.randn(64, c, device="cuda")
    v, e = torch.rand(c, device="cuda") + 0.5, torch.empty(0, device="cuda")
    f = raw_ops.FusedBatchNormV3(x, v, v, e, e)
    g = raw_ops.FusedBatchNormGradV3(x, x, v, f.reserve_space_1, f.reserve_space_2)
    for out in (f, g):
        spans = []
        for t in out:
            assert t.is_contiguous() and t.device == x.device and not t.requires_grad
            assert t.data_ptr() % 512 == 0
            spans.append((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()))
        spans.sort()
        assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    # A write to one leaves the others alone, and one outlives the rest.
    before, kept = f.batch_mean.clone(), f.batch_mean
    f.batch_variance.fill_(7.0)
    f.reserve_space_3.fill_(7.0)
    del f, g
    torch.cuda.synchronize()
    again = raw_ops.FusedBatchNormV3(x, v, v, e, e)
    assert torch.equal(kept, before) and torch.equal(again.batch_mean, before)


def test_small_outputs_have_their_own_storage(kernel_lib):
    """Growing one output in place, or keeping one, touches and holds none of the others."""
    c = 64
    x = torch.randn(64, c, device="cuda")
    v, e = torch.rand(c, device="cuda") + 0.5, torch.empty(0, device="cuda")
    f = raw_ops.FusedBatchNormV3(x, v, v, e, e)
    g = raw_ops.FusedBatchNormGradV3(x, x, v, f.reserve_space_1, f.reserve_space_2)
    for out in (f, g):
        for t in out:
            assert t.storage_offset() == 0
            assert t.untyped_storage().nbytes() == t.numel() * t.element_size()
        assert len({t.untyped_storage().data_ptr() for t in out if t.numel()}) \
            == sum(1 for t in out if t.numel())
        before = [t.clone() for t in out]
        for k, t in enumerate(out):
            t.resize_(4 * t.numel() + 256).fill_(7.0)
            for a, b in zip(out[k + 1:], before[k + 1:]):
                assert torch.equal(a, b)


def test_strides_and_names_follow_the_input(kernel_lib):
    """Contiguous with odd strides along an axis of one: as empty_like gives it, names
    too."""
    base = torch.randn(4, 5, 6, 64, device="cuda")
    x = base.as_strided((4, 1, 30, 64), (1920, 77, 64, 1))
    v, e = torch.rand(64, device="cuda") + 0.5, torch.empty(0, device="cuda")
    assert x.is_contiguous()
    y = raw_ops.FusedBatchNormV3(x, v, v, e, e).y
    assert y.stride() == torch.empty_like(x).stride()
    want = raw_ops.FusedBatchNormV3(base.reshape(4, 1, 30, 64), v, v, e, e).y
    assert torch.equal(y, want)
    named = base.clone().rename("N", "H", "W", "C")
    got = raw_ops.FusedBatchNormV3(named, v, v, e, e).y
    assert got.names == torch.empty_like(named).names
