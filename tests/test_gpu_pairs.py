"""The sweep kernels on pairs of radii give the bits of the single-radius ones.

A context of one radius runs the single-radius kernels; a context of several
runs pairs (and fills the last pair of an odd sweep).  zreion is the maximum
of the one-radius results, the argmax the first radius that reaches it, and
sigma_R the one-radius value (whose partial sums are the same: only the order
of the double-precision additions may differ)."""
import numpy as np
import pytest

import prc_d2z

pytestmark = pytest.mark.gpu


# every size with pair kernels; odd and even counts, several sweeps, a last
# sweep of one radius, an odd radius batch, counts on both sides of the lines
# below which larger grids keep the single-radius kernels
@pytest.mark.parametrize("N,nr,batch", [(32, 5, 0), (32, 9, 4), (64, 7, 3), (96, 6, 0), (128, 3, 2), (192, 5, 4),
                                        (256, 4, 3), (256, 11, 0), (384, 3, 0), (384, 7, 0), (512, 3, 0),
                                        (512, 6, 0), (512, 21, 0), (768, 2, 0), (1024, 3, 2)])
def test_pairs_match_single_radius(N, nr, batch):
    import torch
    box = 1.5 * N
    cl = prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9)
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=nr, BoxSize=box), cl)
    box_mpc = float(np.float32(box) / np.float32(0.68))
    gen = torch.Generator(device="cuda").manual_seed(N + nr)
    delta = 3.0 * torch.randn((N, N, N), device="cuda", generator=gen)
    args = dict(barrier_a=t.barrier_a, growth_init=t.DInit)
    with prc_d2z.Delta2Zreion(N, box_mpc, t.radii_mpc, t.barrier_b, radius_batch=batch, **args) as ctx:
        z, am, sig = ctx.forward(delta, want_sigma_grid=True)
        plain, _, _ = ctx.forward(delta, want_argmax=False)
    assert torch.equal(plain, z)
    best = torch.zeros_like(z)
    win = torch.full_like(am, prc_d2z.PRC_ARGMAX_NONE)
    for r in range(nr):
        with prc_d2z.Delta2Zreion(N, box_mpc, t.radii_mpc[r:r + 1], t.barrier_b[r:r + 1], **args) as one:
            zr, _, s = one.forward(delta, want_sigma_grid=True)
        win[zr > best] = r
        best = torch.maximum(best, zr)
        assert abs(sig[r] - s[0]) <= 1e-12 * s[0]
        del zr
    assert torch.equal(z, best)
    assert torch.equal(am, win)


# the adjoint of a context with the faithful float window runs the
# single-radius kernels (with the same accurate window as any other): the same
# sums in the same order, so the same bits (dL/dB_R up to the order of its
# double-precision additions)
@pytest.mark.parametrize("N,nr,batch", [(32, 5, 0), (64, 9, 4), (96, 3, 0), (128, 8, 6), (192, 4, 2), (256, 5, 0),
                                        (384, 3, 0), (512, 3, 2), (512, 5, 0), (768, 2, 0), (1024, 2, 0)])
def test_adjoint_pairs_match_single_radius(N, nr, batch):
    import torch
    box = 1.5 * N
    cl = prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9)
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=nr, BoxSize=box), cl)
    gen = torch.Generator(device="cuda").manual_seed(7 * N + nr)
    g = torch.randn((N, N, N), device="cuda", generator=gen)
    am = torch.randint(0, nr + 1, (N, N, N), device="cuda", generator=gen, dtype=torch.uint8)
    am[am == nr] = prc_d2z.PRC_ARGMAX_NONE
    out = []
    for faithful in (False, True):
        with prc_d2z.Delta2Zreion(N, float(np.float32(box) / np.float32(0.68)), t.radii_mpc, t.barrier_b, t.barrier_a,
                                  t.DInit, radius_batch=batch, faithful_window=faithful) as ctx:
            out.append(ctx.backward(g, am))
    (d, db), (d1, db1) = out
    assert torch.equal(d, d1)
    # sums of about N^3/nr random terms of size A: compared on that scale
    assert np.max(np.abs(db - db1)) <= 1e-12 * t.barrier_a * N ** 1.5
