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


def _warm(n=N):
    """Loads the kernels of a size (device memory that no context owns)."""
    with prc_d2z.Delta2Zreion(**_box(n, 1)):
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


# (N, radius_batch, slots beyond the spectrum's): a batch that bounds the memory of
# a large grid gets the slots it asks for; below 256^3, and up to 512^3 from three on,
# an odd one takes one more, but not for the faithful window, which runs no pairs
@pytest.mark.parametrize("N,B,slots,faithful", [(192, 1, 2, False), (256, 1, 1, False), (256, 3, 4, False), (256, 5, 5, True),
                                                (512, 1, 1, False), (768, 1, 1, False), (768, 3, 3, False),
                                                (1024, 1, 1, False)])
def test_an_odd_radius_batch(N, B, slots, faithful):
    _warm(N)
    c, used = _used(lambda: prc_d2z.Delta2Zreion(**_box(N, 2 * B + 2, radius_batch=B), faithful_window=faithful))
    assert (slots + 1) * _slot(N) <= used <= (slots + 1.5) * _slot(N) + 2 ** 24, used / _slot(N)
    c.close()


# without that slot the sweeps of an odd batch are its pairs and the last radius
# (sweeps counted by launches: 3 forward passes, 3 a sweep)
@pytest.mark.parametrize("N,nr,B,sweeps", [(256, 4, 1, 4), (768, 3, 3, 1), (768, 5, 5, 2), (768, 7, 3, 3), (1024, 3, 1, 3)])
def test_odd_sweeps_without_the_extra_slot(N, nr, B, sweeps):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(N + nr)
    delta = 3.0 * torch.randn((N, N, N), device="cuda", generator=gen)
    with prc_d2z.Delta2Zreion(**_box(N, nr)) as ctx:
        z0, am0, _ = ctx.forward(delta)
        g0, db0 = ctx.backward(delta, am0)
    with prc_d2z.Delta2Zreion(**_box(N, nr, radius_batch=B)) as ctx:
        z, am, _ = ctx.forward(delta)
        assert ctx.last_launches() == 3 + 3 * sweeps
        g, db = ctx.backward(delta, am0)
    assert torch.equal(z, z0) and torch.equal(am, am0)
    # the sums over the radii meet in another order: a few roundings of float sums
    assert float((g - g0).abs().max()) <= 1e-6 * float(g0.abs().max())
    np.testing.assert_allclose(db, db0, rtol=1e-10, atol=1e-10 * N ** 1.5)
