"""What the Python entry points hand to the library for a torch tensor, on the
CPU: the tensors are host tensors that pass for device ones, the library is a
stand-in that reads the pointers it gets."""
import ctypes

import numpy as np
import pytest
import torch

import prc_d2z

N = 8


class _Device(torch.Tensor):
    """A host tensor that says that it lives on a CUDA device."""
    is_cuda = property(lambda self: True)


_Device.__module__ = "torch"


def _dev(x):
    return torch.as_tensor(x).as_subclass(_Device)


def _read(p, dtype=np.float32):
    p = p.value if isinstance(p, ctypes.c_void_p) else p
    return np.frombuffer((ctypes.c_char * (N ** 3 * np.dtype(dtype).itemsize)).from_address(p), dtype).copy()


def _write(p, value, dtype=np.float32):
    p = p.value if isinstance(p, ctypes.c_void_p) else p
    np.frombuffer((ctypes.c_char * (N ** 3 * np.dtype(dtype).itemsize)).from_address(p), dtype)[:] = value


class _Stream:
    """Stands for torch's current stream."""

    def __init__(self, handle):
        self.cuda_stream, self.waits = handle, 0

    def synchronize(self):
        self.waits += 1


class _Library:
    """Records what the pointers hold at the time of the call."""

    def __init__(self):
        self.seen = []

    def prc_d2z_history(self, ctx, z, on_dev, counts, h, hz):
        return 0

    def prc_d2z_smooth(self, ctx, d, in_dev, radius, out, out_dev):
        return 0

    def prc_d2z_forward(self, ctx, d, in_dev, z, am, out_dev, sig):
        _write(z, np.arange(N ** 3))
        if am is not None:
            _write(am, np.arange(N ** 3) % 7, np.uint8)
        return 0

    def prc_d2z_correct(self, ctx, zvz, z, on_dev):
        _write(z, _read(z) + 1)
        return 0

    def prc_d2z_gaussian_field(self, ctx, seed, amp, n, z, on_dev):
        _write(z, np.arange(N ** 3) + 5)
        return 0

    def prc_d2z_backward(self, ctx, g, am, in_dev, out, out_dev, db):
        self.seen += [_read(g), _read(am, np.uint8)]
        _write(out, 4)
        return 0

    def prc_d2z_batch_forward(self, b, dp, zp, ap, mode):
        self.seen += [_read(p) for p in dp]
        for i, p in enumerate(zp):
            _write(p, np.arange(N ** 3) + i)
        return 0


@pytest.fixture
def lib(monkeypatch):
    L = _Library()
    monkeypatch.setattr(prc_d2z, "load", lambda: L)
    L.stream = _Stream(0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: L.stream)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: L.stream.cuda_stream, raising=False)
    return L


def _engine(stream=0):
    e = object.__new__(prc_d2z.Delta2Zreion)
    e.N, e.n3, e.n_radii, e._ctx, e._stream = N, N ** 3, 3, None, stream
    return e


def _batch(n):
    b = object.__new__(prc_d2z.Batch)
    b.n, b.N, b._b = n, [N] * n, None
    return b


def _transposed(seed, dtype=torch.float32):
    return _dev(torch.from_numpy(np.random.default_rng(seed).integers(0, 200, (N, N, N))).to(dtype).permute(2, 1, 0))


def test_copies_of_unordered_inputs_live_until_the_call(lib):
    """The elements of a transposed input reach the library in order, one box's
    copy not overwritten by the next one's."""
    boxes = [_transposed(i) for i in range(4)]
    out = [_dev(torch.zeros(N, N, N)) for _ in boxes]
    _batch(4).forward(boxes, out, mode="loop")
    for x, got in zip(boxes, lib.seen):
        assert np.array_equal(got, x.numpy().ravel())
    lib.seen.clear()
    g, am = _transposed(9), _transposed(10, torch.uint8)
    _engine().backward(g, am, dL_ddelta=_dev(torch.zeros(N, N, N)))
    assert np.array_equal(lib.seen[0], g.numpy().ravel())
    assert np.array_equal(lib.seen[1], am.numpy().ravel())


def test_unordered_outputs_get_the_results(lib):
    """A transposed output tensor holds the result afterwards (reshape gives the
    library a copy of it), in its own element order."""
    count = np.arange(N ** 3, dtype=np.float32).reshape(N, N, N)
    flat = lambda: _dev(torch.zeros(N, N, N))  # noqa: E731
    e = _engine()
    z, am = _transposed(1), _transposed(2, torch.uint8)
    r = e.forward(flat(), zreion=z, argmax=am)
    assert r[0] is z and np.array_equal(z.numpy(), count)
    assert np.array_equal(am.numpy(), count % 7)
    z = _transposed(3)
    before = z.numpy().copy()
    e.correct(z, np.zeros(4, np.float32))
    assert np.array_equal(z.numpy(), before + 1)
    z = _transposed(4)
    e.gaussian_field(1, np.zeros(4, np.float32), out=z)
    assert np.array_equal(z.numpy(), count + 5)
    z = _transposed(5)
    e.backward(flat(), _dev(torch.zeros(N, N, N, dtype=torch.uint8)), dL_ddelta=z)
    assert np.array_equal(z.numpy(), np.full_like(count, 4))
    zs = [_transposed(6), flat(), _transposed(7)]
    _batch(3).forward([flat() for _ in zs], zs, mode="loop")
    for i, z in enumerate(zs):
        assert np.array_equal(z.numpy(), count + i)


def test_what_was_refused_stays_refused(lib):
    """Strided vectors, wrong types and counts, tensors in host memory."""
    e, ok = _engine(), _dev(torch.zeros(N, N, N))
    for bad in (_dev(torch.zeros(2 * N ** 3))[::2], _dev(torch.zeros(N ** 3, dtype=torch.float64)),
                _dev(torch.zeros(N, N, N - 1)), torch.zeros(N, N, N)):
        for a, b in ((bad, ok), (ok, bad)):
            with pytest.raises(ValueError):
                e.forward(a, zreion=b, want_argmax=False)


@pytest.mark.parametrize("torch_stream,ctx_stream,waits", [(0, 0, 0), (7, 7, 0), (7, 0, 1), (0, 7, 1)])
def test_work_of_another_torch_stream_is_waited_for(lib, monkeypatch, torch_stream, ctx_stream, waits):
    """Tensors filled on a stream that the context does not use are complete
    before the library reads them; on the same stream nothing is waited for."""
    lib.stream = _Stream(torch_stream)
    e, x = _engine(ctx_stream), _dev(torch.zeros(N, N, N))
    am, tab = _dev(torch.zeros(N, N, N, dtype=torch.uint8)), np.zeros(4, np.float32)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: x)
    calls = [lambda: e.forward(x, zreion=x, argmax=am), lambda: e.backward(x, am, dL_ddelta=x),
             lambda: e.smooth(x, 0), lambda: e.history(x), lambda: e.correct(x, tab),
             lambda: e.gaussian_field(1, tab, out=x)]
    for k, call in enumerate(calls):
        call()
        assert lib.stream.waits == (k + 1) * waits, k


def test_a_batch_waits_for_torch(lib):
    """A batch's streams are its own: torch's work is always waited for."""
    x = _dev(torch.zeros(N, N, N))
    _batch(2).forward([x, x], [_dev(torch.zeros(N, N, N)) for _ in range(2)], mode="loop")
    assert lib.stream.waits == 1
