"""Device memory of contexts and batches: what the radius batch asks for, and
spare slots (the full default width, an odd batch's extra slot) out of one
reserve of 6 GB that all contexts of the process share."""
import numpy as np
import pytest

import prc_d2z

pytestmark = pytest.mark.gpu
RESERVE = 6 << 30


def _slot(N):
    return N * N * (N // 2 + 2) * 8


def _box(N, nr, **kw):
    return dict(N=N, box_mpc=1.5 * N, radii_mpc=np.linspace(3.0, 0.4 * N, nr), barrier_b=np.linspace(2.0, 1.0, nr),
                barrier_a=1.0, **kw)


def _used(make):
    """(what make returned, bytes of device memory it took)."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    made = make()
    return made, before - torch.cuda.mem_get_info()[0]


# 40 boxes at the full default width of 64 slots are 22.5 GB at 128^3; with the
# smallest default, 16 slots and the spectrum, 5.9 GB
COUNT, N, NR = 40, 128, 64
LEAN = COUNT * 17 * _slot(N)


def _warm():
    with prc_d2z.Delta2Zreion(**_box(N, 2)):
        pass


def test_a_default_batch_takes_the_smallest_default_where_the_reserve_is_too_small():
    _warm()
    batch, used = _used(lambda: prc_d2z.Batch([_box(N, NR) for _ in range(COUNT)], n_streams=2))
    assert used <= 1.1 * LEAN + 2 ** 28, used
    batch.close()
    batch, used = _used(lambda: prc_d2z.Batch([_box(N, NR) for _ in range(4)], n_streams=2))
    assert used >= 4 * (NR + 1) * _slot(N), used   # four fit: full width
    batch.close()


def test_default_contexts_share_one_reserve():
    _warm()
    ctx, used = _used(lambda: [prc_d2z.Delta2Zreion(**_box(N, NR)) for _ in range(COUNT)])
    assert used <= 1.1 * LEAN + RESERVE + 2 ** 28, used
    for c in ctx:
        c.close()
    c, used = _used(lambda: prc_d2z.Delta2Zreion(**_box(N, NR)))  # the reserve was given back
    assert used >= (NR + 1) * _slot(N), used
    c.close()


def test_boxes_without_reserve_give_the_same_results():
    """Of thirty contexts of 128^3 x 48, and of a batch beside them, those at the
    smallest default (three sweeps) give what the full width gives."""
    import torch
    _warm()
    delta = torch.randn((N, N, N), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    box = _box(N, 48)
    ctx = [prc_d2z.Delta2Zreion(**box) for _ in range(30)]
    z0, am0, sig0 = ctx[0].forward(delta, want_sigma_grid=True)
    n0, n1 = ctx[0].last_launches(), None
    z, am, sig = ctx[-1].forward(delta, want_sigma_grid=True)
    n1 = ctx[-1].last_launches()
    assert n0 == 6 and n1 == 12   # 3 forward passes, 3 a sweep: one and three sweeps
    assert torch.equal(z, z0) and torch.equal(am, am0)
    np.testing.assert_allclose(sig, sig0, rtol=1e-12)
    batch = prc_d2z.Batch([box, box], n_streams=1)
    out = [torch.empty_like(delta) for _ in range(2)]
    batch.forward([delta, delta], out, mode="grouped")
    assert all(torch.equal(o, z0) for o in out)
    batch.close()
    for c in ctx:
        c.close()
