"""The bounded wait of every inverse z pass, made to run out on purpose (as in
tests/test_gpu_waits.py, whose sweeps are all pairs shared by four warps): pairs
with a warp to itself (from 192^3 on), and the single-radius pass, which a
faithful window, one radius and few odd radii run, on small and large grids;
with argmax and per-radius sums.  The call reports it, the next one is exact."""
import pytest

import prc_d2z
from prc_d2z import _lib, fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nr,faithful", [(192, 4, False), (256, 4, False), (32, 5, True), (64, 1, False), (128, 4, True),
                                           (256, 3, False), (512, 3, False)])
@pytest.mark.parametrize("sums", [False, True])
def test_forward_reports_a_wait_that_ran_out(N, nr, faithful, sums):
    import torch
    box = 1.5 * N
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=max(nr, 2), BoxSize=box),
                               prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9))
    delta = fields.gaussian_field(N, box, seed=31, backend="torch").contiguous()
    L = _lib.load()
    with prc_d2z.Delta2Zreion(N, box, t.radii_mpc[:nr], t.barrier_b[:nr], t.barrier_a, faithful_window=faithful) as ctx:
        z_ref, am_ref, _ = ctx.forward(delta, want_sigma_grid=sums)
        _lib.check(L.prc_d2z_test_withhold_copy(1))
        try:
            with pytest.raises(prc_d2z.PrcError) as ei:
                ctx.forward(delta, want_sigma_grid=sums)
        finally:
            L.prc_d2z_test_withhold_copy(0)
        assert ei.value.code == _lib.PRC_ERR_CUDA
        assert "wait limit" in str(ei.value)
        z, am, _ = ctx.forward(delta, want_sigma_grid=sums)
        assert torch.equal(z, z_ref) and torch.equal(am, am_ref)
