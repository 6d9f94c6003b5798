"""The work that users of this framework have it do, as measured cases.

Every case is one call (or one training step) through a public entry point of
`prc_d2z`: `Delta2Zreion.forward` on a device-resident field, `forward_many`
on a stream of pinned host boxes, `Batch.forward` on many boxes, the torch
operation of `prc_d2z.autograd`, and `Delta2Zreion.backward`.  Grid sizes are
the compiled ones from 32 to 1024 (powers of two and three times them), radii
run from a handful to 64, and the radius batch is either the constructor's
default or all radii in one sweep, which the autotuner picks up to 512^3.

A case is a dict:
  kind    forward | stream | batch | grad | backward
  n       grid side (batch: the sizes, comma separated, one per box)
  radii   number of smoothing radii (batch: of the largest count; the boxes
          have between half of that and all of it)
  sweep   radius batch (0: the constructor's default)
  argmax, sigma   optional outputs of forward
  boxes   boxes of a stream
  mode    batch mode

The inputs are made with torch alone: Gaussian fields of a BBKS spectrum, and
the radius and barrier tables of the step from plain numpy.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pr-calc_gb300"))

import prc_d2z  # noqa: E402
from prc_d2z import autograd  # noqa: E402

OMEGAM, H, NS, SIGMA8 = 0.31, 0.68, 0.965, 0.81
CELL = 1.5          # Mpc/h, the batched workload's cell
ZETA, M_MIN = 80.5, 1e9 / 0.68
RMIN_CELLS, RMAX = 2.0, 60.0   # radii from two cells to 60 Mpc/h
ZHIGH, DHIGH, DELTAC = 20.0, 0.0614, 1.686
DEV = "cuda"
SIZES = (32, 48, 64, 96, 128, 192, 256, 384, 512, 768)


def listed():
    def case(name, kind, n, radii, sweep=0, **more):
        return {"name": name, "kind": kind, "n": n, "radii": radii, "sweep": sweep, **more}
    return [
        # the smallest call: a test-sized box, a few radii, argmax as by default
        case("forward 32 x 8", "forward", 32, 8, argmax=True, sigma=False),
        # one small box of a survey of parameters, zreion alone
        case("forward 64 x 64", "forward", 64, 64, argmax=False, sigma=False),
        # the small plain configuration (128^3, 32 radii), all radii in one sweep
        case("forward 128 x 32", "forward", 128, 32, sweep=32, argmax=False, sigma=False),
        # a size with a factor of three and an odd number of radii, with every
        # output the executable writes (argmax for .rbubble, sigma_R)
        case("forward 192 x 41", "forward", 192, 41, argmax=True, sigma=True),
        # a mid-sized box with the constructor's radius batch
        case("forward 384 x 24", "forward", 384, 24, argmax=False, sigma=False),
        # the headline step: 512^3, 64 radii, one sweep (the autotuned batch)
        case("forward 512 x 64", "forward", 512, 64, sweep=64, argmax=False, sigma=False),
        # the largest grid, several sweeps of the autotuned batch
        case("forward 1024 x 32", "forward", 1024, 32, sweep=12, argmax=False, sigma=False),
        # a loop over realisations held on the host, copies included
        case("stream 6 of 256 x 32", "stream", 256, 32, sweep=32, boxes=6),
        # boxes of mixed sizes in grouped launches
        case("batch mixed", "batch", "64,96,128,192,256,64,96,128,192,256,64,96,128,192,256,64", 48, mode="grouped"),
        # many small boxes in grouped launches
        case("batch 48 of 64", "batch", ",".join(["64"] * 48), 40, mode="grouped"),
        # one training step: zreion, the loss's gradient in delta and in the barrier
        case("grad 256 x 64", "grad", 256, 64),
        # the adjoint alone at full size
        case("backward 512 x 32", "backward", 512, 32),
    ]


def draw(rng):
    kind = rng.choice(["forward"] * 5 + ["stream", "batch", "batch", "grad", "backward"])
    radii = int(round(math.exp(rng.uniform(math.log(3), math.log(64)))))
    if kind == "batch":
        count = rng.randint(4, 12)
        sizes = [rng.choice((32, 64, 64, 96, 128, 192, 256)) for _ in range(count)]
        return {"kind": kind, "n": ",".join(map(str, sizes)), "radii": max(4, min(radii, 48)), "sweep": 0,
                "mode": rng.choice(["grouped", "grouped", "graph", "loop"])}
    n = rng.choice({"forward": SIZES, "stream": (64, 96, 128, 192, 256, 384),
                    "grad": (32, 64, 96, 128, 192, 256), "backward": (64, 96, 128, 192, 256, 384, 512)}[kind])
    c = {"kind": kind, "n": n, "radii": radii, "sweep": 0}
    if rng.random() < 0.5 and radii * n ** 3 * 4 < 36e9:
        c["sweep"] = radii
    if kind == "forward":
        c["argmax"] = rng.random() < 0.4
        c["sigma"] = rng.random() < 0.2
    if kind == "stream":
        c["boxes"] = rng.randint(2, 6)
    return c


# ------------------------------------------------------------------ tables
def _bbks(k):
    q = k / (OMEGAM * H)
    return np.log1p(2.34 * q) / (2.34 * q) * (1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3
                                             + (6.71 * q) ** 4) ** -0.25


def _sigma(r):
    """sigma of a top hat of radius r [Mpc/h], normalised to sigma_8."""
    lk = np.linspace(math.log(1e-4), math.log(3e2), 20000)
    k = np.exp(lk)

    def s2(x):
        x = k * x
        w = np.where(x > 1e-2, 3 * (np.sin(x) - x * np.cos(x)) / x ** 3, 1 - x * x / 10)
        return float(np.sum(k ** (3 + NS) * _bbks(k) ** 2 * w * w))
    return SIGMA8 * math.sqrt(s2(r) / s2(8.0))


def _tables(n, radii):
    """(box in Mpc, radii in Mpc, barrier offsets, barrier slope) of one box."""
    box = CELL * n / H
    rmin, rmax = box * RMIN_CELLS / n, min(RMAX / H, 0.4 * box)
    r = np.exp(np.linspace(math.log(rmin), math.log(rmax), radii))
    rho0 = 2.775e11 * OMEGAM * H * H
    smin = _sigma((3 * M_MIN / (4 * math.pi * rho0)) ** (1 / 3) * H)
    erfizeta = float(torch.special.erfinv(torch.tensor(1 - 1 / ZETA, dtype=torch.float64)))
    b = np.array([math.sqrt(2 * (smin ** 2 - _sigma(x * H) ** 2)) * erfizeta for x in r])
    return box, r, b, (1 + ZHIGH) * DHIGH / DELTAC


def _box_of(n, radii, sweep):
    box, r, b, a = _tables(n, radii)
    return dict(N=n, box_mpc=box, radii_mpc=r, barrier_b=b, barrier_a=a, growth_init=1.0, radius_batch=sweep)


def _engine(c):
    return prc_d2z.Delta2Zreion(**_box_of(c["n"], c["radii"], c["sweep"]),
                                argmax=bool(c.get("argmax", c["kind"] in ("grad", "backward"))))


# ------------------------------------------------------------------ inputs
def _rng(seed, k=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + k)


def _m2(n, dtype):
    f = torch.fft.fftfreq(n, d=1.0 / n, device=DEV, dtype=dtype) ** 2
    fz = torch.arange(n // 2 + 1, device=DEV, dtype=dtype) ** 2
    return f[:, None, None] + f[None, :, None] + fz


def _field(n, seed, k=0):
    """A Gaussian random density field of the BBKS spectrum, float32."""
    box = CELL * n
    m = np.sqrt(np.arange(3 * (n // 2) ** 2 + 1, dtype=np.float64))
    kk = 2 * math.pi / box * np.maximum(m, 0.5)
    lk = np.linspace(math.log(1e-4), math.log(3e2), 20000)
    q = np.exp(lk)
    x = 8.0 * q
    w = np.where(x > 1e-2, 3 * (np.sin(x) - x * np.cos(x)) / x ** 3, 1 - x * x / 10)
    norm = SIGMA8 ** 2 / (np.sum(q ** (3 + NS) * _bbks(q) ** 2 * w * w) * (lk[1] - lk[0]) / (2 * math.pi ** 2))
    amp = np.sqrt(n ** 3 * norm * kk ** NS * _bbks(kk) ** 2 / box ** 3)
    amp[0] = 0.0
    amp = torch.from_numpy(amp.astype(np.float32)).to(DEV)
    s = torch.fft.rfftn(torch.randn((n, n, n), device=DEV, generator=_rng(seed, k)))
    s *= amp[_m2(n, torch.float32).to(torch.int32)]
    return torch.fft.irfftn(s, s=(n, n, n)).contiguous()


def _winners(n, radii, seed):
    """An argmax grid: smooth regions of one winning radius, a fifth of the cells never reached."""
    f = _field(n, seed, 3)
    f = f / f.std()
    r = torch.floor((f + 0.85) * (0.45 * radii)).clamp(-1, radii - 1)
    return torch.where(r < 0, torch.full_like(r, 255.0), r).to(torch.uint8)


def _target(n, seed):
    return 6.0 + 6.0 * torch.rand((n, n, n), device=DEV, generator=_rng(seed, 7))


def _batch_boxes(c):
    sizes = [int(x) for x in str(c["n"]).split(",")]
    lo = max(2, c["radii"] // 2)
    counts = [lo + (7 * i) % (c["radii"] - lo + 1) for i in range(len(sizes))]
    return list(zip(sizes, counts))


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "batch":
        boxes = _batch_boxes(case)
        s["batch"] = prc_d2z.Batch([_box_of(n, r, r) for n, r in boxes], n_streams=3)
        s["delta"] = [_field(n, seed, 10 + i) for i, (n, _) in enumerate(boxes)]
        s["z"] = [torch.empty_like(d) for d in s["delta"]]
        return s
    n = case["n"]
    s["engine"] = _engine(case)
    if kind == "stream":
        s["delta"] = [_pinned(_field(n, seed, i)) for i in range(case["boxes"])]
        s["z"] = [_pinned(torch.empty((n, n, n), device=DEV)) for _ in range(case["boxes"])]
    elif kind == "backward":
        s["g"] = torch.randn((n, n, n), device=DEV, generator=_rng(seed, 5))
        s["argmax"] = _winners(n, case["radii"], seed)
        s["out"] = torch.empty_like(s["g"])
    else:
        s["delta"] = _field(n, seed)
        if kind == "grad":
            s["delta"].requires_grad_(True)
            s["target"] = _target(n, seed)
        else:
            s["z"] = torch.empty_like(s["delta"])
            s["am"] = torch.empty(s["delta"].shape, dtype=torch.uint8, device=DEV) if case["argmax"] else None
    return s


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def run(s):
    c = s["case"]
    if c["kind"] == "batch":
        return s["batch"].forward(s["delta"], s["z"], mode=c["mode"])
    e = s["engine"]
    if c["kind"] == "stream":
        return e.forward_many(s["delta"], s["z"])
    if c["kind"] == "backward":
        g, db = e.backward(s["g"], s["argmax"], dL_ddelta=s["out"], want_dB=True)
        return {"delta": g, "barrier": db}
    if c["kind"] == "grad":
        z = autograd.delta2zreion_fn(s["delta"], e)
        loss = ((z - s["target"]) ** 2).mean()
        g, = torch.autograd.grad(loss, s["delta"])
        return {"z": z.detach(), "delta": g, "barrier": e.last_dB}
    z, am, sig = e.forward(s["delta"], zreion=s["z"], argmax=s["am"], want_argmax=c["argmax"],
                           want_sigma_grid=c["sigma"])
    return {"z": z, **({"argmax": am} if c["argmax"] else {}), **({"sigma": sig} if c["sigma"] else {})}


def work(case):
    """Inputs read once, outputs written once; the transforms' operations
    (2.5 n log2 n for a real transform, one forward and one per radius) and the
    window, barrier and maximum (about 20 for each half-spectrum element and 4
    for each cell of a radius)."""
    if case["kind"] == "batch":
        parts = [work({"kind": "forward", "n": n, "radii": r, "argmax": False}) for n, r in _batch_boxes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n3, r = case["n"] ** 3, case["radii"]
    fft = 2.5 * n3 * math.log2(n3)
    one = {"bytes": (8 + bool(case.get("argmax"))) * n3, "flops": (r + 1) * fft + r * 14 * n3}
    back = {"bytes": 9 * n3, "flops": (r + 1) * fft + r * 14 * n3}
    if case["kind"] == "stream":
        return {k: case["boxes"] * v for k, v in one.items()}
    if case["kind"] == "backward":
        return back
    if case["kind"] == "grad":
        return {"bytes": 8 * n3 + 4 * n3 + 4 * n3, "flops": one["flops"] + back["flops"]}
    return one


# ------------------------------------------------------------------ 64 bits
def _window(k, r):
    x = k * r
    w = 3.0 * (torch.sin(x) - x * torch.cos(x)) / x ** 3
    x2 = x * x
    w = torch.where(x < 1e-2, 1.0 - x2 / 10.0 + x2 * x2 / 280.0, w)
    w[0, 0, 0] = 0.0
    return w


def _forward64(delta, box, radii, b, a):
    n = delta.shape[0]
    spec = torch.fft.rfftn(delta.double())
    k = torch.sqrt(_m2(n, torch.float64)) * (2 * math.pi / box)
    z = torch.zeros(delta.shape, dtype=torch.float64, device=DEV)
    am = torch.full(delta.shape, 255, dtype=torch.uint8, device=DEV)
    sig = []
    for i, r in enumerate(radii):
        d = torch.fft.irfftn(spec * _window(k, float(r)), s=(n, n, n))
        sig.append(math.sqrt(float((d * d).mean())))
        d = a * (d + float(b[i])) - 1.0
        am[d > z] = i
        z = torch.maximum(z, d)
        del d
    return z, am, np.array(sig)


def _backward64(g, am, box, radii, a):
    n = g.shape[0]
    k = torch.sqrt(_m2(n, torch.float64)) * (2 * math.pi / box)
    acc, db = None, []
    for i, r in enumerate(radii):
        h = torch.where(am == i, g, torch.zeros_like(g)) * a
        db.append(float(h.sum()))
        h = torch.fft.rfftn(h) * _window(k, float(r))
        acc = h if acc is None else acc.add_(h)
        del h
    return torch.fft.irfftn(acc, s=(n, n, n)), np.array(db)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, (n, r) in enumerate(_batch_boxes(case)):
            box, rr, b, a = _tables(n, r)
            out.append(_forward64(_field(n, seed, 10 + i), box, rr, b, a)[0])
        return out
    n = case["n"]
    box, rr, b, a = _tables(n, case["radii"])
    if kind == "stream":
        return [_forward64(_field(n, seed, i), box, rr, b, a)[0].cpu().numpy() for i in range(case["boxes"])]
    if kind == "backward":
        g = torch.randn((n, n, n), device=DEV, generator=_rng(seed, 5)).double()
        d, db = _backward64(g, _winners(n, case["radii"], seed), box, rr, a)
        return {"delta": d, "barrier": db}
    z, am, sig = _forward64(_field(n, seed), box, rr, b, a)
    if kind == "grad":
        d, db = _backward64(2.0 * (z - _target(n, seed).double()) / n ** 3, am, box, rr, a)
        return {"z": z, "delta": d, "barrier": db}
    return {"z": z, **({"argmax": None} if case["argmax"] else {}), **({"sigma": sig} if case["sigma"] else {})}
