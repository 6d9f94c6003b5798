"""More of tests/test_gpu_pairs.py: sizes and counts on both sides of the lines
between pairs and single radii, NaN barriers in either half of a pair, and
adjoint sweeps of more radii than a lane keeps one sum for."""
import numpy as np
import pytest

import prc_d2z
import test_gpu_pairs as pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nr,batch", [(128, 3, 0), (192, 3, 0), (512, 2, 0), (512, 4, 0), (512, 17, 17), (768, 7, 0),
                                        (1024, 5, 0)])
def test_lines_between_pairs_and_single_radii(N, nr, batch):
    pairs.test_pairs_match_single_radius(N, nr, batch)


@pytest.mark.parametrize("N,nr,batch", [(192, 3, 0), (1024, 3, 0)])
def test_adjoint_lines(N, nr, batch):
    pairs.test_adjoint_pairs_match_single_radius(N, nr, batch)


def test_a_window_variant_leaves_the_adjoint_alone():
    """The adjoint of a context with a tuned window variant runs as without:
    the same sweeps (eleven radii in pairs by an odd batch of five: six and five,
    where single radii take five, five and one) and the same bits."""
    import torch
    N, nr = 128, 11
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=nr, BoxSize=192.0),
                               prc_d2z.CLParameters(Rmax=60.0, zeta=30.0, M_min=1.47e9))
    gen = torch.Generator(device="cuda").manual_seed(3)
    g = torch.randn((N, N, N), device="cuda", generator=gen)
    am = torch.randint(0, nr, (N, N, N), device="cuda", generator=gen, dtype=torch.uint8)
    assert prc_d2z.win_variants(N) > 1
    out = []
    for variant in (0, 1):
        with prc_d2z.Delta2Zreion(N, 280.0, t.radii_mpc, t.barrier_b, t.barrier_a, radius_batch=5) as ctx:
            ctx.tune(0, variant)
            out.append(ctx.backward(g, am)[0])
            assert ctx.last_launches() == 2 * 3 + 3
    assert torch.equal(*out)


# sums in both of a lane's accumulators (pairs 0..15 and 16..31), a last pair of
# one radius, on 8, 12 and 16 elements a lane
@pytest.mark.parametrize("N,nr", [(32, 64), (64, 63), (64, 33), (128, 64), (192, 63), (192, 64), (256, 63), (256, 64),
                                  (512, 64)])
def test_adjoint_of_more_than_32_radii_in_one_sweep(N, nr):
    """Against FP64: dL/d delta within 1e-5 relative L2, dL/dB_r of every radius
    within the rounding of its float partial sums (256 cells each: at most 16
    sequential additions and 5 levels of a tree, so 21 * 2^-24 of A sum |g|)."""
    import torch
    from fp64_chain import kmag, tophat64
    box = 1.5 * N
    box_mpc = float(np.float32(box) / np.float32(0.68))
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=nr, BoxSize=box),
                               prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9))
    gen = torch.Generator(device="cuda").manual_seed(N + nr)
    g = torch.randn((N, N, N), device="cuda", generator=gen)
    am = torch.randint(0, nr + 1, (N, N, N), device="cuda", generator=gen, dtype=torch.uint8)
    am[am == nr] = prc_d2z.PRC_ARGMAX_NONE
    with prc_d2z.Delta2Zreion(N, box_mpc, t.radii_mpc, t.barrier_b, t.barrier_a, radius_batch=nr) as ctx:
        d, db = ctx.backward(g, am)
        assert ctx.last_launches() == 6   # one sweep
    km = kmag(N, box_mpc, g.device)
    acc = torch.zeros((N, N, N // 2 + 1), dtype=torch.complex128, device="cuda")
    for r in range(nr):
        m = am == r
        w = tophat64(km * t.radii_mpc[r])
        w[0, 0, 0] = 0.0
        acc += w * torch.fft.rfftn(torch.where(m, t.barrier_a * g.double(), 0.0))
        gr = g[m].double()
        assert abs(db[r] - t.barrier_a * float(gr.sum())) <= 21 * 2.0 ** -24 * t.barrier_a * float(gr.abs().sum()), r
    ref = torch.fft.irfftn(acc, s=(N, N, N))
    rel = float(torch.linalg.vector_norm(d.double() - ref) / torch.linalg.vector_norm(ref))
    assert rel < 1e-5, rel


# a NaN barrier never wins: in the first and the second half of a pair, in both,
# in the pair of one radius and everywhere; four warps merge their maxima up to 128
@pytest.mark.parametrize("N", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("where", [(0,), (1,), (2, 3), (6,), (0, 3, 5, 6), tuple(range(7))])
def test_nan_barriers_never_win(N, where):
    import torch
    nr = 7 if N < 192 else 14   # (an odd sweep below 192, an even one above)
    nan = np.array([w + 7 * k for w in where for k in range(nr // 7)])
    box = 1.5 * N
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=nr, BoxSize=box),
                               prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9))
    b = t.barrier_b.copy()
    b[nan] = np.nan
    gen = torch.Generator(device="cuda").manual_seed(N)
    delta = 3.0 * torch.randn((N, N, N), device="cuda", generator=gen)
    box_mpc = float(np.float32(box) / np.float32(0.68))
    args = dict(barrier_a=t.barrier_a, growth_init=t.DInit)
    with prc_d2z.Delta2Zreion(N, box_mpc, t.radii_mpc, b, radius_batch=nr, **args) as ctx:
        z, am, _ = ctx.forward(delta)
        plain, _, _ = ctx.forward(delta, want_argmax=False)
    best = torch.zeros_like(z)
    win = torch.full_like(am, prc_d2z.PRC_ARGMAX_NONE)
    for r in set(range(nr)) - set(nan):
        with prc_d2z.Delta2Zreion(N, box_mpc, t.radii_mpc[r:r + 1], b[r:r + 1], **args) as one:
            zr, _, _ = one.forward(delta)
        win[zr > best] = r
        best = torch.maximum(best, zr)
    assert torch.equal(z, best) and torch.equal(plain, best)
    assert torch.equal(am, win)
