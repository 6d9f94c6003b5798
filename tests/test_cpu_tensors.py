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


class _Library:
    """Records what the pointers hold at the time of the call."""

    def __init__(self):
        self.seen = []

    def prc_d2z_backward(self, ctx, g, am, in_dev, out, out_dev, db):
        self.seen += [_read(g), _read(am, np.uint8)]
        _write(out, 4)
        return 0

    def prc_d2z_batch_forward(self, b, dp, zp, ap, mode):
        self.seen += [_read(p) for p in dp]
        return 0


@pytest.fixture
def lib(monkeypatch):
    L = _Library()
    monkeypatch.setattr(prc_d2z, "load", lambda: L)
    return L


def _engine():
    e = object.__new__(prc_d2z.Delta2Zreion)
    e.n3, e.n_radii, e._ctx = N ** 3, 3, None
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
