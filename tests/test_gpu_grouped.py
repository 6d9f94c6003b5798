"""Batches on single radii and on pairs: every box of a grouped size joins a
grouped launch, whatever its radius count and batch, and a box gets the per-box
result in grouped and in per-box launches on either side of their lines."""
import numpy as np
import pytest

import prc_d2z

pytestmark = pytest.mark.gpu


def _box(N, nr, radius_batch):
    box = 1.5 * N
    t = prc_d2z.compute_tables(prc_d2z.Parameters(N=N, Nscales=max(nr, 2), BoxSize=box),
                               prc_d2z.CLParameters(Rmax=min(0.4 * box, 60.0), zeta=30.0, M_min=1.47e9))
    return dict(N=N, box_mpc=float(np.float32(box) / np.float32(0.68)), radii_mpc=t.radii_mpc[:nr],
                barrier_b=t.barrier_b[:nr], barrier_a=t.barrier_a, growth_init=t.DInit, radius_batch=radius_batch)


# (N, radii, radius batch): one radius, one slot, counts on both sides of the
# lines between single radii and pairs, several sweeps, a last sweep of one
# radius, boxes of one size in both kinds of group
SPEC = {
    "small": [(32, 1, 0), (32, 2, 1), (64, 1, 0), (64, 3, 0), (96, 3, 0), (96, 5, 4), (96, 4, 1), (64, 9, 4)],
    "128": [(128, 1, 0), (128, 7, 0), (128, 9, 0), (128, 8, 0), (128, 5, 3), (128, 9, 4), (128, 3, 1)],
    "192": [(192, 1, 0), (192, 3, 0), (192, 5, 0), (192, 7, 3), (192, 4, 0)],
    "256": [(256, 1, 0), (256, 2, 0), (256, 9, 0), (256, 11, 0), (256, 13, 0), (256, 9, 4), (256, 3, 1)],
}


@pytest.mark.parametrize("name", list(SPEC))
@pytest.mark.parametrize("mode,with_argmax", [("grouped", False), ("grouped", True), ("graph", True), ("loop", False)])
def test_boxes_match_per_box(name, mode, with_argmax):
    import torch
    boxes = [_box(*s) for s in SPEC[name]]
    gen = torch.Generator(device="cuda").manual_seed(len(name))
    fields = [3.0 * torch.randn((b["N"],) * 3, device="cuda", generator=gen) for b in boxes]
    ref = []
    for b, d in zip(boxes, fields):
        with prc_d2z.Delta2Zreion(**b) as ctx:
            ref.append(ctx.forward(d, want_argmax=with_argmax)[:2])
    batch = prc_d2z.Batch(boxes, n_streams=3)
    for _ in range(2):  # the second call replays the captured graph
        out = [torch.full_like(d, -3.0) for d in fields]
        am = [torch.full(d.shape, 7, dtype=torch.uint8, device="cuda") for d in fields] if with_argmax else None
        batch.forward(fields, out, am, mode=mode)
        for i, (z, a) in enumerate(ref):
            assert torch.equal(out[i], z), SPEC[name][i]
            assert not with_argmax or torch.equal(am[i], a), SPEC[name][i]
    batch.close()


@pytest.mark.parametrize("N,nr", [(32, 1), (64, 1), (128, 3), (192, 1), (256, 5)])
def test_few_radii_keep_grouped_launches(N, nr):
    """Boxes of one radius, or of few odd ones, run in as many launches as one
    box of them does, not in one set a box."""
    import torch
    d = [torch.zeros((N,) * 3, device="cuda") for _ in range(6)]
    counts = []
    for n in (4, 6):
        batch = prc_d2z.Batch([_box(N, nr, 0)] * n, n_streams=2)
        batch.forward(d[:n], [torch.empty_like(x) for x in d[:n]], mode="grouped")
        counts.append(batch.launches())
        batch.close()
    assert counts[0] == counts[1]


@pytest.mark.parametrize("radius_batch,sweeps", [(8, 1), (4, 2)])
def test_grouped_launch_count(radius_batch, sweeps):
    """Three forward passes and three passes a sweep."""
    import torch
    d = [torch.zeros((32, 32, 32), device="cuda") for _ in range(3)]
    batch = prc_d2z.Batch([_box(32, 8, radius_batch)] * 3, n_streams=1)
    batch.forward(d, [torch.empty_like(x) for x in d], mode="grouped")
    assert batch.launches() == 3 + 3 * sweeps
    batch.close()
