"""The native host path of the ops against their general Python path: the same
bits for every call that the native path takes, the same answers and errors for
those that it leaves."""
import threading

import pytest
import torch

from tensorflow_musa_extension_b200 import errors, optimizers, raw_ops

pytestmark = pytest.mark.gpu

F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16


class _Declines:
    def __getattr__(self, name):
        return lambda *a: -1 if name == "adam_kind" else None


def _both(monkeypatch, call):
    """Outputs by the native path, then by the general path."""
    got = call()
    with monkeypatch.context() as m:
        m.setattr(raw_ops, "_native", lambda: _Declines())
        want = call()
    return got, want


def _same(got, want):
    got = got if isinstance(got, tuple) else (got,)
    want = want if isinstance(want, tuple) else (want,)
    assert type(got) is type(want) and len(got) == len(want)
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride()
        assert torch.equal(a, b) and not a.requires_grad


def _rand(shape, dtype, seed=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


# How a tensor reaches the op: as it was made, transposed storage, every second
# row, off a 16-byte boundary, a Parameter.
FORMS = {
    "plain": lambda t: t,
    "transposed": lambda t: t.transpose(0, 1).contiguous().transpose(0, 1),
    "strided": lambda t: torch.stack((t, t), 1).flatten(0, 1)[::2],
    "offset": lambda t: torch.cat((t.new_zeros(1), t.reshape(-1)))[1:].view(t.shape),
    "parameter": lambda t: torch.nn.Parameter(t),
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("shape,layout", [((5, 3, 4, 24), "NHWC"), ((3, 37), "NHWC"),
                                          ((4, 16, 3, 5), "NCHW"), ((2, 3, 4, 8), "NCHW")])
def test_batch_norm(monkeypatch, kernel_lib, form, dtype, shape, layout):
    c = shape[-1] if layout == "NHWC" else shape[1]
    x, dy = FORMS[form](_rand(shape, dtype)), FORMS[form](_rand(shape, dtype, 1))
    s, o, m = (_rand((c,), F32, i) for i in (2, 3, 4))
    v = _rand((c,), F32, 5).abs() + 0.5
    e = torch.empty(0, device="cuda")
    for args in ((e, e, 1e-3, 1.0, layout, True), (m, v, 1e-3, 0.25, layout, True),
                 (m, v, 1e-3, 1.0, layout, False), (m.half(), v, 1e-3, 0.5, layout, True)):
        got, want = _both(monkeypatch, lambda: raw_ops.FusedBatchNormV3(x, s, o, *args))
        _same(got, want)
    for training in (True, False):
        _same(*_both(monkeypatch, lambda: raw_ops.FusedBatchNormGradV3(
            dy, x, s, m, v, None, 1e-3, layout, training)))


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("shape", [(33, 24), (7, 5, 101)])
def test_chains_and_row_norms(monkeypatch, kernel_lib, form, dtype, shape):
    x, dy = FORMS[form](_rand(shape, dtype)), FORMS[form](_rand(shape, dtype, 1))
    b, g = _rand(shape[-1:], dtype, 2), _rand(shape[-1:], dtype, 3)
    for op in (raw_ops.MusaBiasAddRelu, raw_ops.MusaBiasAddSwish, raw_ops.BiasAdd):
        _same(*_both(monkeypatch, lambda: op(x, b)))
    _same(*_both(monkeypatch, lambda: raw_ops.MusaBiasAddReluGrad(dy, x)))
    _same(*_both(monkeypatch, lambda: raw_ops.MusaLayerNorm(x, g, b)))
    _same(*_both(monkeypatch, lambda: raw_ops.MusaLayerNormGrad(dy, x, g, b)))
    if dtype != F16:
        got, want = _both(monkeypatch, lambda: raw_ops.MusaRmsNorm(x, g))
        _same(got, want)
        _same(*_both(monkeypatch, lambda: raw_ops.MusaRmsNormGradDx(x, want.inv_rms, g, dy)))


def test_refusals_are_those_of_the_general_path(monkeypatch, kernel_lib):
    x, s, e = _rand((4, 8), F32), _rand((8,), F32), torch.empty(0, device="cuda")
    calls = [
        lambda: raw_ops.FusedBatchNormV3(x, s[:7], s, e, e),
        lambda: raw_ops.FusedBatchNormV3(x, s, s, e, e, is_training=False),
        lambda: raw_ops.FusedBatchNormV3(x, s, s, e, e, exponential_avg_factor=0.5),
        lambda: raw_ops.FusedBatchNormV3(x, s, s, e, e, data_format="NDHWC"),
        lambda: raw_ops.FusedBatchNormV3(x.double(), s, s, e, e),
        lambda: raw_ops.FusedBatchNormGradV3(x.half(), x, s, s, s),
        lambda: raw_ops.FusedBatchNormGradV3(x[:3], x, s, s, s),
        lambda: raw_ops.MusaBiasAddRelu(x, s[:7]),
        lambda: raw_ops.MusaBiasAddReluGrad(x, x.half()),
        lambda: raw_ops.MusaLayerNorm(x, s.half(), s),
        lambda: raw_ops.MusaRmsNorm(x.half(), s.half()),
    ]
    for call in calls:
        with pytest.raises(errors.InvalidArgumentError) as got:
            call()
        with monkeypatch.context() as m:
            m.setattr(raw_ops, "_native", lambda: _Declines())
            with pytest.raises(errors.InvalidArgumentError) as want:
                call()
        assert str(got.value) == str(want.value)


@pytest.mark.parametrize("state,grad", [(F32, F32), (F32, BF16), (BF16, BF16), (F16, F16)])
def test_adam_step(monkeypatch, kernel_lib, state, grad):
    def step():
        opt = optimizers.MusaAdam(1e-2)
        vs = [_rand(sh, state, i) for i, sh in enumerate(((3, 5), (1,), (1000,), (0,), (64, 33)))]
        gs = [_rand(v.shape, grad, 9 + i) for i, v in enumerate(vs)]
        gs[4] = FORMS["strided"](gs[4])
        pairs = list(zip(gs, vs)) + [(gs[2], vs[2]), (None, vs[0])]   # vs[2] twice, in order
        opt.apply_gradients(pairs)
        opt.apply_gradients(pairs)
        return tuple(t for v in vs for t in (v, opt.get_slot(v, "m"), opt.get_slot(v, "v")))
    _same(*_both(monkeypatch, step))


def _train_step(x, dy, s, o):
    e = torch.empty(0, device="cuda")
    f = raw_ops.FusedBatchNormV3(x, s, o, e, e, 1e-3)
    g = raw_ops.FusedBatchNormGradV3(dy, x, s, f.reserve_space_1, f.reserve_space_2, None, 1e-3)
    b = s.to(x.dtype)
    return (*f, *g, raw_ops.MusaLayerNorm(x, b, b), *raw_ops.MusaLayerNormGrad(dy, x, b, b),
            raw_ops.MusaBiasAddRelu(x, b))


def _step_inputs(seed, c):
    # The first size fits the one-kernel form, the second takes the chain and its scratch.
    rows = 700 if c == 48 else 70000
    return (_rand((rows, c), BF16, seed), _rand((rows, c), BF16, seed + 1),
            _rand((c,), F32, seed + 2), _rand((c,), F32, seed + 3))


@pytest.mark.parametrize("c", [48, 256])
@pytest.mark.parametrize("own_stream", [False, True])
def test_several_threads(kernel_lib, c, own_stream):
    """Calls of four threads at once, on one stream or on one each: the bits of
    the same calls made one after the other (scratch is private to a call)."""
    inputs = [_step_inputs(10 * i, c) for i in range(4)]
    want = [_train_step(*a) for a in inputs]
    torch.cuda.synchronize()
    got, failed = [None] * 4, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream() if own_stream
                                   else torch.cuda.default_stream()):
                for _ in range(20):
                    got[i] = _train_step(*inputs[i])
                torch.cuda.current_stream().synchronize()
        except Exception as e:   # reported by the assertion below
            failed.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for a, b in zip(got, want):
        for u, v in zip(a, b):
            assert torch.equal(u, v)


@pytest.mark.parametrize("c", [48, 256])
def test_graph_capture(kernel_lib, c):
    """A captured step (outputs and scratch from the graph's pool) replayed on new
    inputs: the bits of the eager calls."""
    buffers, other = _step_inputs(3, c), _step_inputs(50, c)
    _train_step(*buffers)      # per-device set-up
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _train_step(*buffers)
    for values in (other, _step_inputs(90, c)):
        for t, v in zip(buffers, values):
            t.copy_(v)
        graph.replay()
        torch.cuda.synchronize()
        for u, v in zip(out, _train_step(*values)):
            assert torch.equal(u, v)
    del graph
