"""More of tests/test_gpu_pairs.py: sizes and counts on both sides of the lines
between pairs and single radii, NaN barriers in either half of a pair, and
adjoint sweeps of more radii than a lane keeps one sum for."""
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
