"""The work that a user of this framework has it do, as cases that can be timed.

A case is one pass of the statistics (forward) and of their gradient (VJP) through
the public Python entry points, at sizes from a 16-pixel-a-side sky to the largest
that one card holds: `listed` names twelve, `draw` gives others of the same ranges,
`prepare` makes what a program has in hand before the call, `run` is the pass, `work`
what it cannot do without, `tolerance` how far another correct implementation at
the same precision may be, and `exact` the same outputs from plain torch in 64 bits
(the second half of this file, which uses nothing of the framework).

A program that evaluates many maps keeps one engine and gives it one map after
another, so the states of a case share the engine of their configuration; the engine
of another configuration is let go of.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parent.parent / "stl-dev-mpi_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

L = 4  # orientations of the framework's wavelets


def listed():
    return [
        # one small sky, everything FP64, numpy in and out: the plain single-map evaluation, all latency
        dict(name="sky16_f64_host", kind="sky", nside=16, J=3, batch=1, dtype="float64", io="host"),
        # three maps of a region study: three masks, an odd batch, the variances asked for, numpy in and out
        dict(name="sky64_masks_moments", kind="sky", nside=64, J=5, batch=3, dtype="float32", io="host", masks=3,
             moments=True),
        # a training step's loss term: a batch of four maps through the autograd function
        dict(name="sky256_autograd", kind="sky", nside=256, J=7, batch=4, dtype="float32", io="autograd"),
        # the plain FP64 path on one map
        dict(name="sky512_f64", kind="sky", nside=512, J=8, batch=1, dtype="float64", io="device"),
        # the headline configuration: four FP32 maps, maps and gradients in device memory
        dict(name="sky1024_f32_b4", kind="sky", nside=1024, J=9, batch=4, dtype="float32", io="device"),
        # the largest sky: one map, the wavelet fields recomputed in the VJP instead of kept
        dict(name="sky2048_f32_recompute", kind="sky", nside=2048, J=10, batch=1, dtype="float32", io="device",
             fields="recompute"),
        # the cross statistics of two surveys' maps
        dict(name="cross512_f32", kind="cross", nside=512, J=8, batch=1, dtype="float32", io="device"),
        # polarisation: (Q, U) maps through the spin-2 front end
        dict(name="spin512_f32", kind="spin", nside=512, J=8, batch=1, dtype="float32", io="device"),
        # ragged disc patches of one survey, 1 024 to 65 536 pixels each, in one batch
        dict(name="patches512_f32", kind="patch", nside=512, J=5, discs=512, least=1024, most=65536, core=0.0,
             dtype="float32"),
        # a handful of small FP64 discs whose statistics average a core only, with variances
        dict(name="patches128_core_f64", kind="patch", nside=128, J=4, discs=13, least=500, most=5000, core=0.6,
             dtype="float64", moments=True),
        # the first L-BFGS iterations of a synthesis on the device
        # (FP64: in FP32 a line search takes another step for another rounding, and the iterates part ways)
        dict(name="synthesis256_f64", kind="synthesis", nside=256, J=7, iterations=7, dtype="float64"),
        # the other terms of a synthesis objective: kappa transform, detail pyramid, sorted marginal
        dict(name="terms512", kind="terms", nside=512, depth=8),
    ]


def draw(rng):
    kind = rng.choice(["sky"] * 6 + ["patch"] * 3 + ["cross", "spin", "synthesis", "terms"])
    if kind == "patch":
        nside = rng.choice([128, 256, 512])
        least = int(math.exp(rng.uniform(math.log(400), math.log(2000))))
        most = int(least * math.exp(rng.uniform(0.0, math.log(min(32.0, 1.5 * nside * nside / least)))))
        # the core keeps a quarter of a disc's pixels at least, so it holds some at every level
        return dict(kind=kind, nside=nside, J=rng.choice([3, 4, 5] if nside > 128 else [3, 4]),
                    discs=int(math.exp(rng.uniform(math.log(3), math.log(400)))), least=least, most=most,
                    core=rng.choice([0.0, 0.0, 0.5, 0.7]), dtype=rng.choice(["float32", "float32", "float64"]),
                    moments=rng.random() < 0.3)
    if kind == "terms":
        k = rng.randint(5, 10)
        return dict(kind=kind, nside=1 << k, depth=rng.randint(2, k))
    k = rng.randint(4, 10 if kind == "sky" else 9)
    nside, J = 1 << k, rng.randint(max(2, k - 4), k - 1)  # the last level is nside 4 or more
    dtype = rng.choice(["float32", "float32", "float64"])
    if kind == "synthesis":
        k = min(k, 8)
        return dict(kind=kind, nside=1 << k, J=min(J, k - 1), iterations=rng.randint(3, 9), dtype="float64")
    most = {10: 4, 9: 8}.get(k, 12) if dtype == "float32" else {10: 1, 9: 4}.get(k, 8)
    case = dict(kind=kind, nside=nside, J=J, batch=rng.randint(1, most if kind == "sky" else max(1, most // 4)),
                dtype=dtype, io=rng.choice(["device", "device", "autograd", "host"]) if kind == "sky" else "device")
    if kind == "sky" and case["io"] != "autograd" and k <= 9 and rng.random() < 0.3:
        case.update(masks=rng.randint(1, 4), moments=rng.random() < 0.5)
    return case


# ---- inputs -------------------------------------------------------------------

def _generator(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + what * 7919 + 12345) % (1 << 62))
    return g


def _npix(nside):
    return 12 * nside * nside


def _lognormal(shape, seed, what):
    """exp(g - 1/2), g ~ N(0, 1): the maps of the framework's benchmark."""
    g = torch.randn(shape, generator=_generator(seed, what), device="cuda", dtype=torch.float64)
    return torch.exp(g - 0.5)


def _cotangent(shape, seed):
    """A complex cotangent with every coefficient in it."""
    c = torch.randn(tuple(shape) + (2,), generator=_generator(seed, 99), device="cuda", dtype=torch.float64)
    return torch.view_as_complex(c)


def _map_shape(case):
    n = _npix(case["nside"])
    return (case["batch"], n) if case["kind"] == "sky" else (case["batch"], 2, n)


def _maps(case, seed):
    x = _lognormal(_map_shape(case), seed, 1)
    if case["kind"] == "spin":  # (Q, U) of either sign
        x = torch.randn(x.shape, generator=_generator(seed, 1), device="cuda", dtype=torch.float64)
    # the FP32 paths are given FP32 maps; the same values go to the 64-bit computation
    return x.float().double() if case["dtype"] == "float32" else x


def _mask_ids(case):
    """Pixels of each mask: caps of the sky of different heights, as a part of the NESTED range is."""
    n, out = _npix(case["nside"]), []
    for k in range(case.get("masks", 0)):
        lo, hi = n * k // (case["masks"] + 1), n * (k + 2) // (case["masks"] + 1) + 7 * k
        out.append(np.arange(lo, min(hi, n)))
    return out


def _disc_centres(case):
    """Centres uniform on the sphere and radii whose discs hold least to most pixels, log-uniform."""
    r = np.random.default_rng(3)
    v = r.standard_normal((case["discs"], 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    counts = np.exp(r.uniform(math.log(case["least"]), math.log(case["most"]), case["discs"]))
    radii = np.degrees(np.arccos(1.0 - counts * (4.0 * np.pi / _npix(case["nside"])) / (2.0 * np.pi)))
    return v, radii, (radii * case["core"] if case["core"] else None)


def _disc_values(sizes, case, seed):
    x = torch.randn(int(sum(sizes)), generator=_generator(seed, 1), device="cuda", dtype=torch.float64)
    return x.float().double() if case["dtype"] == "float32" else x


def _synthesis_maps(case, seed):
    """(target map, starting map): lognormal, and N(0, 1) rescaled to the target's mean and deviation."""
    n = _npix(case["nside"])
    t = _lognormal((1, n), seed, 1)
    g = torch.randn((1, n), generator=_generator(seed, 2), device="cuda", dtype=torch.float64)
    return t, (g - g.mean()) / g.std() * t.std() + t.mean()


def _terms_inputs(case, seed):
    n, depth = _npix(case["nside"]), case["depth"]
    kx = np.linspace(-3.0, 4.0, 41)
    r = np.random.default_rng(int(seed) % (1 << 63))
    x = torch.randn(n, generator=_generator(seed, 1), device="cuda", dtype=torch.float64)
    t = torch.randn(n, generator=_generator(seed, 2), device="cuda", dtype=torch.float64).sort().values
    return dict(x=x, t=t, kx=kx, ky=np.tanh(kx) + 0.1 * kx, kd=1.0 / np.cosh(kx) ** 2 + 0.1,
                scale=(0.2, 1.3, 0.05, 0.9), power=r.standard_normal((1, depth)) / n,
                levels=np.arange(depth, dtype=np.int32), kurt=r.uniform(0.5, 1.5, (1, depth, 3)) / np.array([n, 1, 1]))


# ---- states and passes ---------------------------------------------------------

_kept = {"key": None, "engine": None}


def _engine(key, make):
    """The engine of this configuration: the last one, or a new one (one engine is kept)."""
    if _kept["key"] != key:
        if _kept["engine"] is not None:
            _kept["engine"].close()
        _kept.update(key=None, engine=None)
        _kept.update(engine=make(), key=key)
    return _kept["engine"]


def _sky_engine(case):
    import stl_b200

    def make():
        kw = {"sky": {}, "cross": {"cross": True}, "spin": {"spin": 2}, "synthesis": {}}[case["kind"]]
        e = stl_b200.NativeEngine(case["nside"], case["J"], batch=case.get("batch", 1), dtype=case["dtype"],
                                  fields=case.get("fields", "keep"), prepare=True, **kw)
        if case.get("masks"):
            e.set_masks(_mask_ids(case))
        return e

    key = tuple(case.get(k) for k in ("kind", "nside", "J", "batch", "dtype", "fields", "masks"))
    return _engine(key, make)


def _patch_engine(case):
    import stl_b200

    def make():
        e = stl_b200.PatchEngine(case["nside"], case["J"], dtype=case["dtype"])
        e.select(*_disc_centres(case))
        return e

    return _engine(tuple(sorted((k, v) for k, v in case.items() if k != "name")), make)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "terms":
        import stl_b200
        s, n = _terms_inputs(case, seed), _npix(case["nside"])
        s["engine"] = _engine(("terms", n, case["depth"]),
                              lambda: stl_b200.Terms(rows=1, length=n, depth=case["depth"], sort=n))
        s["engine"].kappa_table(s["kx"], s["ky"], s["kd"])
        return dict(s, case=case)
    if kind == "patch":
        e = _patch_engine(case)
        sizes = [i.size for i in e.ids]
        x = _disc_values(sizes, case, seed).cpu().numpy()
        return dict(case=case, engine=e, x=np.split(x, np.cumsum(sizes)[:-1]),
                    cot=_cotangent((len(sizes), e.ncoeff), seed).cpu().numpy(), grad=np.empty(x.size))
    e = _sky_engine(case)
    if kind == "synthesis":
        t, x = _synthesis_maps(case, seed)
        target, var = e.forward(t.cpu().numpy(), moments=True)
        v = var.reshape(-1)
        return dict(case=case, engine=e, x=x, target=target, weights=1.0 / np.maximum(v, 1e-12 * v.max()))
    x = _maps(case, seed)
    c = _cotangent(e._shape(), seed)
    if case["io"] == "host":
        return dict(case=case, engine=e, x=x.cpu().numpy(), cot=c.cpu().numpy(), grad=np.empty(x.numel()))
    x = x.float() if case["dtype"] == "float32" else x
    if case["io"] == "autograd":
        return dict(case=case, engine=e, x=x.requires_grad_(), cot=c)
    return dict(case=case, engine=e, x=x, cot=c.cpu().numpy(), grad=torch.empty_like(x))


def _answer(values, var, grad, moments):
    return dict(values=values, var=var, grad=grad) if moments else dict(values=values, grad=grad)


def run(state):
    case, e = state["case"], state["engine"]
    kind, moments = case["kind"], bool(case.get("moments"))
    if kind == "terms":
        x = state["x"]
        k, dk = e.kappa(x, *state["scale"])
        e.pyramid(k)
        sums = e.moments(k)
        gk = torch.zeros_like(x)
        e.level_power_grad(k, state["power"], gk)
        e.kurtosis_grad(k, state["levels"], state["kurt"], gk)
        g = torch.zeros_like(x)
        e.add_product(g, gk, dk)
        perm = e.sort(x)
        loss = e.marginal(x, perm, state["t"], 2.0 / x.numel(), g)
        return dict(k=k, dk=dk, sums=sums, grad=g, perm=perm, loss=loss)
    if kind == "patch":
        values, var = e.forward(state["x"], moments=moments)
        e.vjp(state["cot"], out=state["grad"])
        return _answer(values, var, state["grad"], moments)
    if kind == "synthesis":
        x = state["x"].clone()
        _, losses = e.synthesize(x, state["target"], weights=state["weights"],
                                 options={"max_iter": case["iterations"], "history_size": 10})
        return dict(x=x, loss=float(losses[-1]))
    if case["io"] == "host":
        values, var = e.forward(state["x"], moments=moments)
        return _answer(values, var, e.vjp(state["cot"], out=state["grad"]), moments)
    if case["io"] == "autograd":
        import stl_b200
        x = state["x"]
        x.grad = None
        values = stl_b200.scattering(e, x)
        values.backward(state["cot"])
        return dict(values=values.detach(), grad=x.grad)
    values, var = e.forward_tensor(state["x"], moments=moments)
    return _answer(values, var, e.vjp_tensor(state["cot"], state["grad"]), moments)


# ---- what a pass cannot do without -----------------------------------------------

def _coefficients(case):
    pairs = sum(n + 1 for n in range(case["J"]))
    pairs2 = sum((n + 1) * (n + 2) // 2 for n in range(case["J"]))
    orders = 2 if case["kind"] == "cross" else 1
    return 2 * (orders == 1) + 2 * L * case["J"] + orders * (L * L * pairs + L ** 3 * pairs2)


def work(case):
    """Bytes: maps in, gradients out, statistics out and cotangents in, each once.  Flops: each pixel of a level
    has L complex wavelet outputs of the map and of the L (n + 1) stored moduli, each over about 44 cells (the
    union of the cells that the L orientations of the 5 x 5 stencil read), and as many in the gradient; the
    products of the level's K = 1 + L (n + 1) operands for each of the L orientations, and twice that in the
    gradient; 28 weights a decimated value, both ways."""
    if case["kind"] == "terms":
        n = _npix(case["nside"])
        # x, targets in; kappa, derivative, gradient, positions out
        return {"bytes": n * (8 + 8 + 8 + 8 + 8 + 4), "flops": n * (40 + 12 * case["depth"])}
    if case["kind"] == "patch":
        _, radii, _ = _disc_centres(case)
        n0 = float(np.sum((1.0 - np.cos(np.radians(radii))) * _npix(case["nside"]) / 2.0))
        fields, stats = 1, case["discs"]
    else:
        n0, stats = float(_npix(case["nside"])), case.get("batch", 1)
        fields = stats * (2 if case["kind"] in ("cross", "spin") else 1)
        stats = (fields if case["kind"] == "spin" else stats) * max(1, case.get("masks", 0))
    flops = 0.0
    for n in range(case["J"]):
        rows, k = 1 + L * (n + 1), 1 + L * (n + 1)
        level = rows * 44 * 2 * 2 * L * 2 + 3 * L * 4 * k * k
        if n + 1 < case["J"]:
            level += rows * 28 * 2 * 2 / 4
        flops += n0 / 4 ** n * fields * level
    if case["kind"] == "spin":
        flops += n0 * fields * 25 * 2 * 2 * 2
    size = 4 if case["dtype"] == "float32" and case.get("io") in ("device", "autograd") else 8
    byte = 2 * n0 * fields * size + 2 * 16 * stats * _coefficients(case)
    if case["kind"] == "synthesis":  # a little more than one evaluation an iteration; start in, result out
        return {"bytes": byte, "flops": flops * case["iterations"]}
    return {"bytes": byte, "flops": flops}


def tolerance(case):
    """About four times the largest distance from `exact` seen over the listed cases and 40 drawn ones.  Gradients pass
    z / |z| (the cross ones steeper powers), so the pixels nearest |z| = 0 are the farthest off, the more so the more
    pixels there are; an L-BFGS iterate carries the rounding of every iteration before."""
    if case["kind"] == "terms":
        return {"rel": 2e-15, "max": 1e-14}
    if case["kind"] == "synthesis":
        return {"rel": 1e-11, "max": 1e-9}
    if case["dtype"] == "float64":
        return {"rel": 1e-11, "max": 1e-8} if case["kind"] == "cross" else {"rel": 1.5e-12, "max": 1e-9}
    return {"rel": 2e-5, "max": 5e-3} if case["kind"] == "cross" else {"rel": 5e-7, "max": 5e-4}


# ---- the same in plain torch, 64 bits -----------------------------------------------
# HEALPix geometry (NESTED), the oriented wavelet bound to the pixels by bilinear
# interpolation, the smooth decimation, the statistics; gradients by autograd.

_JRLL = (2, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 4)
_JPLL = (1, 3, 5, 7, 0, 2, 4, 6, 1, 3, 5, 7)
# the face next to a face in each of the 9 directions (-1: none), and how its axes lie
_NEXT = ((8, 9, 10, 11, -1, -1, -1, -1, 10, 11, 8, 9), (5, 6, 7, 4, 8, 9, 10, 11, 9, 10, 11, 8),
         (-1, -1, -1, -1, 5, 6, 7, 4, -1, -1, -1, -1), (4, 5, 6, 7, 11, 8, 9, 10, 11, 8, 9, 10),
         (0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11), (1, 2, 3, 0, 0, 1, 2, 3, 5, 6, 7, 4),
         (-1, -1, -1, -1, 7, 4, 5, 6, -1, -1, -1, -1), (3, 0, 1, 2, 3, 0, 1, 2, 4, 5, 6, 7),
         (2, 3, 0, 1, -1, -1, -1, -1, 0, 1, 2, 3))
_FLIP = ((0, 0, 3), (0, 0, 6), (0, 0, 0), (0, 0, 5), (0, 0, 0), (5, 0, 0), (0, 0, 0), (6, 0, 0), (3, 0, 0))
_BITS = ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F), (2, 0x3333333333333333),
         (1, 0x5555555555555555))


def _table(t, like):
    return torch.tensor(t, device=like.device)


def _spread(v):
    for s, m in _BITS:
        v = (v | (v << s)) & m
    return v


def _squeeze(v):
    v = v & _BITS[-1][1]
    for (s, _), m in zip(reversed(_BITS), [b[1] for b in reversed(_BITS[:-1])] + [0xFFFFFFFF]):
        v = (v | (v >> s)) & m
    return v


def _nest(x, y, face, nside):
    return face * nside * nside + _spread(x) + 2 * _spread(y)


def _centre(pix, nside):
    """(z, sin theta, phi) of NESTED pixel centres."""
    face, p = pix // (nside * nside), pix % (nside * nside)
    x, y = _squeeze(p), _squeeze(p >> 1)
    jr = _table(_JRLL, pix)[face] * nside - x - y - 1
    cap = (jr < nside) | (jr > 3 * nside)
    nr = torch.where(jr < nside, jr, torch.where(jr > 3 * nside, 4 * nside - jr, nside))
    shift = torch.where(cap, 0, (jr - nside) & 1)
    t = nr.double() ** 2 / (3.0 * nside * nside)
    z = torch.where(cap, torch.where(jr < nside, 1.0 - t, t - 1.0), (2 * nside - jr).double() * 2.0 / (3.0 * nside))
    s = torch.where(cap, torch.sqrt(t * (2.0 - t)), torch.sqrt((1.0 - z) * (1.0 + z)))
    jp = (_table(_JPLL, pix)[face] * nr + x - y + 1 + shift).div(2, rounding_mode="floor")
    jp = torch.where(jp > 4 * nr, jp - 4 * nr, torch.where(jp < 1, jp + 4 * nr, jp))
    return z, s, (jp.double() - (shift.double() + 1.0) * 0.5) * (0.5 * math.pi / nr.double())


def _frame(pix, nside):
    """Centre and the tangent vectors along theta and phi, [..., 3] each."""
    z, s, p = _centre(pix, nside)
    c, d = torch.cos(p), torch.sin(p)
    return (torch.stack([s * c, s * d, z], -1), torch.stack([z * c, z * d, -s], -1),
            torch.stack([-d, c, torch.zeros_like(c)], -1))


def _ring2nest(pix, nside):
    np_, cap = _npix(nside), 2 * nside * (nside - 1)
    north, south = pix < cap, pix >= np_ - cap

    def ring_of(v):  # the ring of the v-th pixel from a pole: the largest r with 2 r (r - 1) <= v
        r = ((1.0 + torch.sqrt(1.0 + 2.0 * v.double())) * 0.5).long()
        r = torch.where(2 * r * (r - 1) > v, r - 1, r)
        return torch.where(2 * r * (r + 1) <= v, r + 1, r)

    a = torch.where(north, pix, 0)
    rn = ring_of(a)
    b = torch.where(south, np_ - 1 - pix, 0)
    rs = ring_of(b)
    e = torch.where(north | south, 0, pix - cap)
    re = e // (4 * nside) + nside
    ring = torch.where(north, rn, torch.where(south, 4 * nside - rs, re))
    nr = torch.where(north, rn, torch.where(south, rs, nside))
    at = torch.where(north, a - 2 * rn * (rn - 1), torch.where(south, 2 * rs * (rs + 1) - 1 - b, e % (4 * nside))) + 1
    shift = torch.where(north | south, 0, (ring + nside) & 1)
    up, down = re - nside + 1, 3 * nside + 1 - re
    fm = (at - up.div(2, rounding_mode="floor") + nside - 1).div(nside, rounding_mode="floor")
    fp = (at - down.div(2, rounding_mode="floor") + nside - 1).div(nside, rounding_mode="floor")
    belt = torch.where(fp == fm, fp | 4, torch.where(fp < fm, fp, fm + 8))
    quarter = (at - 1) // nr.clamp(min=1)
    face = torch.where(north, quarter, torch.where(south, quarter + 8, belt))
    u = ring - _table(_JRLL, pix)[face] * nside + 1
    v = 2 * at - _table(_JPLL, pix)[face] * nr - shift - 1
    v = torch.where(v >= 2 * nside, v - 8 * nside, v)
    return _nest((v - u) >> 1, (-v - u) >> 1, face, nside)


def _interpolate(vec, nside):
    """(NESTED pixels, weights) [..., 4] of the bilinear interpolation at unit vectors."""
    z = vec[..., 2].clamp(-1.0, 1.0)
    theta = torch.atan2(torch.hypot(vec[..., 0], vec[..., 1]), z)
    phi = torch.remainder(torch.atan2(vec[..., 1], vec[..., 0]), 2.0 * math.pi)
    belt = (nside * (2.0 - 1.5 * z)).long()
    pole = (nside * torch.sqrt(3.0 * (1.0 - z.abs()))).long()
    above = torch.where(z.abs() <= 2.0 / 3.0, belt, torch.where(z > 0, pole, 4 * nside - pole - 1))

    def on_ring(ring):
        half = torch.where(ring > 2 * nside, 4 * nside - ring, ring)
        cap = half < nside
        t = half.double() ** 2 / (3.0 * nside * nside)
        th = torch.where(cap, torch.atan2(torch.sqrt(t * (2.0 - t)), 1.0 - t),
                         torch.acos(((2 * nside - half).double() * 2.0 / (3.0 * nside)).clamp(-1.0, 1.0)))
        count = torch.where(cap, 4 * half, 4 * nside)
        off = torch.where(cap | (((half - nside) & 1) == 0), 0.5, 0.0)
        first = torch.where(cap, 2 * half * (half - 1), 2 * nside * (nside - 1) + (half - nside) * 4 * nside)
        mirror = ring != half
        th = torch.where(mirror, math.pi - th, th)
        first = torch.where(mirror, _npix(nside) - first - count, first)
        at = phi * count.double() / (2.0 * math.pi) - off
        i = torch.floor(at)
        w = at - i
        i = i.long()
        return first + torch.remainder(i, count), first + torch.remainder(i + 1, count), 1.0 - w, w, th

    a0, a1, u0, u1, ta = on_ring(above.clamp(min=1))
    b0, b1, v0, v1, tb = on_ring((above + 1).clamp(max=4 * nside - 1))
    north, south = (above == 0)[..., None], (above + 1 == 4 * nside)[..., None]
    t = (theta - ta) / (tb - ta)
    pix = torch.stack([a0, a1, b0, b1], -1)
    w = torch.stack([u0 * (1 - t), u1 * (1 - t), v0 * t, v1 * t], -1)
    # in a polar cap above the first ring the pole's value is the mean of the ring's four pixels
    wn, ws = theta / tb, (theta - ta) / (math.pi - ta)
    fn, fs = (1 - wn) / 4, ws / 4
    pn = torch.stack([(b0 + 2) & 3, (b1 + 2) & 3, b0, b1], -1)
    last = _npix(nside) - 4
    ps = torch.stack([a0, a1, ((a0 - last + 2) & 3) + last, ((a1 - last + 2) & 3) + last], -1)
    pix = torch.where(north, pn, torch.where(south, ps, pix))
    w = torch.where(north, torch.stack([fn, fn, v0 * wn + fn, v1 * wn + fn], -1),
                    torch.where(south, torch.stack([u0 * (1 - ws) + fs, u1 * (1 - ws) + fs, fs, fs], -1), w))
    return _ring2nest(pix, nside), w


def _box(pix, nside, k):
    """The (2k + 1)^2 cells around each pixel [..., cells], -1 where a face corner has none."""
    face, p = pix // (nside * nside), pix % (nside * nside)
    d = torch.arange(-k, k + 1, device=pix.device)
    x = _squeeze(p)[..., None] + d.repeat(2 * k + 1)
    y = _squeeze(p >> 1)[..., None] + d.repeat_interleave(2 * k + 1)
    way = 4 + (x >= nside).long() - (x < 0).long() + 3 * (y >= nside).long() - 3 * (y < 0).long()
    x, y = torch.remainder(x, nside), torch.remainder(y, nside)
    to = _table(_NEXT, pix)[way, face[..., None]]
    flip = _table(_FLIP, pix)[way, (face // 4)[..., None]]
    x = torch.where((flip & 1) > 0, nside - 1 - x, x)
    y = torch.where((flip & 2) > 0, nside - 1 - y, y)
    x, y = torch.where((flip & 4) > 0, y, x), torch.where((flip & 4) > 0, x, y)
    return torch.where(to < 0, -1, _nest(x, y, to.clamp(min=0), nside))


class _Grid:
    """The pixels of a level: the whole sky, or the supports of discs one after another (sorted per disc)."""

    def __init__(self, nside, ids=None, part=None):
        self.nside, self.ids, self.part = nside, ids, part
        self.n = _npix(nside) if ids is None else ids.numel()
        self.keys = None if ids is None else part * _npix(nside) + ids

    def pixels(self, a, b):
        if self.ids is None:
            return torch.arange(a, b, device="cuda"), None
        return self.ids[a:b], self.part[a:b]

    def find(self, pix, part):
        """Positions of pixels (of the given discs), -1 where the grid has none."""
        if self.ids is None:
            return pix
        want = part.reshape(part.shape + (1,) * (pix.dim() - part.dim())) * _npix(self.nside) + pix
        at = torch.searchsorted(self.keys, want).clamp(max=self.n - 1)
        return torch.where((pix >= 0) & (self.keys[at] == want), at, -1)

    def coarser(self):
        if self.ids is None:
            return _Grid(self.nside // 2)
        keys = torch.unique(self.part * (_npix(self.nside) // 4) + self.ids // 4)
        return _Grid(self.nside // 2, keys % (_npix(self.nside) // 4), keys // (_npix(self.nside) // 4))


def _gabor():
    """The 5 x 5 oriented wavelet: zero mean, unit sum of moduli, rounded to 32 bits (the sums in order: a
    last bit of theirs moves the rounding)."""
    k = [(math.cos(0.5 * math.pi * x) * math.exp(-(x * x + y * y) / 2.0),
          math.sin(0.5 * math.pi * x) * math.exp(-(x * x + y * y) / 2.0))
         for y in (-2.0, -1.0, 0.0, 1.0, 2.0) for x in (-2.0, -1.0, 0.0, 1.0, 2.0)]
    re = im = size = 0.0
    for u, v in k:
        re, im = re + u, im + v
    k = [(u - re / 25.0, v - im / 25.0) for u, v in k]
    for u, v in k:
        size += math.hypot(u, v)
    k = np.array([(u / size, v / size) for u, v in k]).T
    return torch.tensor(k.astype(np.float32).astype(np.float64), device="cuda")


def _wavelet_rows(grid):
    """(rows, chunk(a, b)): the wavelet rows of a level, L a pixel: cells [m, 100] and weights [m, 2, 100]."""
    nside, ker = grid.nside, _gabor()
    y, x = torch.meshgrid(torch.arange(-2, 3, device="cuda"), torch.arange(-2, 3, device="cuda"), indexing="ij")
    x, y = x.reshape(-1).double(), y.reshape(-1).double()
    r, turn = torch.hypot(x, y) * math.sqrt(4.0 * math.pi / _npix(nside)), torch.atan2(y, x)
    sx, sy, sz = torch.sin(r) * torch.cos(turn), torch.sin(r) * torch.sin(turn), torch.cos(r)

    def chunk(a, b):
        pix, part = grid.pixels(a, b)
        c, et, ep = _frame(pix, nside)
        z, _, phi = _centre(pix, nside)
        sign = torch.where(z < 0, -1.0, 1.0)  # the orientation's zero turns with longitude, mirrored in the south
        g = torch.arange(L, device="cuda", dtype=torch.float64) * (math.pi / L)
        alpha = -sign[:, None] * phi[:, None] + sign[:, None] * g
        ca, sa = torch.cos(alpha)[:, :, None, None], torch.sin(alpha)[:, :, None, None]
        u, v = et[:, None, None], ep[:, None, None]
        vec = (sx[:, None] * (ca * u + sa * v) + sy[:, None] * (ca * v - sa * u) + sz[:, None] * c[:, None, None])
        cells, w = _interpolate(vec, nside)  # [n, L, 25, 4]
        if grid.ids is not None:
            at = grid.find(cells, part)
            at = torch.where(w > 1e-9, at, -1)  # a disc's wavelet binds no cell of a smaller weight
            none = (at < 0).all(-1, keepdim=True)  # a point off the disc takes the centre's cells
            at = torch.where(none, at[:, :, 12:13], at)
            w = torch.where(none, w[:, :, 12:13], w)
            w = torch.where(at >= 0, w, 0.0)
            w = w / w.sum(-1, keepdim=True).clamp(min=1e-12)
            cells = at.clamp(min=0)
        weights = ker[:, :, None] * w[:, :, None]  # [n, L, 2, 25, 4]
        return cells.reshape(-1, 100), weights.reshape(-1, 2, 100)

    return grid.n, chunk


def _decimation_rows(fine, coarse):
    """The smooth decimation: Gaussian means over the fine pixels within three pixel sizes."""
    nside = fine.nside
    radius = 3.0 * math.sqrt(4.0 * math.pi / _npix(nside))

    def chunk(a, b):
        pix, part = coarse.pixels(a, b)
        box = _box(pix, nside // 2, 2)
        cells = (4 * box[..., None] + torch.arange(4, device="cuda")).reshape(pix.numel(), -1)
        cells = torch.where(box.repeat_interleave(4, 1) < 0, -1, cells)
        at = fine.find(cells, part)
        c, v = _frame(pix, nside // 2)[0][:, None], _frame(cells.clamp(min=0), nside)[0]
        gamma = 2.0 * torch.asin((0.5 * torch.linalg.vector_norm(c - v, dim=-1)).clamp(max=1.0))
        w = torch.where((at >= 0) & (gamma <= radius), torch.exp(-0.5 * (2.0 * gamma / radius) ** 2), 0.0)
        w = w / w.sum(-1, keepdim=True)
        return at.clamp(min=0), w[:, None]

    return coarse.n, chunk


def _spin_rows(nside):
    """-(d_x - i d_y)^2 on the 5 x 5 cells, exact on polynomials of degree 4, of Q + iU carried to the pixel's frame."""
    h = math.sqrt(4.0 * math.pi / _npix(nside))
    powers = [(t - b, b) for t in range(5) for b in range(t + 1)]
    image = torch.zeros(15, 2, device="cuda", dtype=torch.float64)
    image[powers.index((2, 0)), 0], image[powers.index((0, 2)), 0], image[powers.index((1, 1)), 1] = -2.0, 2.0, 2.0

    def chunk(a, b):
        pix = torch.arange(a, b, device="cuda")
        c, et, ep = (t[:, None] for t in _frame(pix, nside))
        cells = _box(pix, nside, 2)
        v, vt, vp = _frame(cells.clamp(min=0), nside)
        z = (v * c).sum(-1)
        px, py = (v * et).sum(-1) / z / h, (v * ep).sum(-1) / z / h
        wt = torch.where(cells >= 0, torch.exp(-(px * px + py * py) / 4.0), 0.0)
        A = torch.stack([px ** i * py ** j for i, j in powers], 1)  # [n, 15, cells]
        gram = (A * wt[:, None]) @ A.transpose(1, 2)
        w = (A.transpose(1, 2) @ torch.linalg.solve(gram, image.expand(b - a, 15, 2))) * wt[..., None]
        w = torch.view_as_complex(w.contiguous())
        axis = torch.linalg.cross(c.expand_as(v), v)  # e_theta of the pixel carried to the cell
        s = torch.linalg.vector_norm(axis, dim=-1, keepdim=True)
        k = axis / s.clamp(min=1e-300)
        e = et.expand_as(v)
        moved = e * z[..., None] + torch.linalg.cross(k, e) * s + k * (k * e).sum(-1, keepdim=True) * (1.0 - z[..., None])
        moved = torch.where(s < 1e-15, e, moved)
        psi = torch.atan2((moved * vp).sum(-1), (moved * vt).sum(-1))
        w = torch.view_as_real(w * torch.polar(torch.ones_like(psi), -2.0 * psi))
        return cells.clamp(min=0), w.transpose(1, 2).contiguous()

    return _npix(nside), chunk


class _Rows(torch.autograd.Function):
    """y[row] = W[row] x[cells of row] for x [n, R], a chunk of rows at a time: [rows, outputs, R]."""

    @staticmethod
    def forward(ctx, x, rows, chunk, each):
        step = max(1024, min(1 << 18, (1 << 27) // (100 * each * max(4, x.shape[1]))))
        ctx.chunk, ctx.cuts, ctx.n = chunk, [(a, min(a + step, rows)) for a in range(0, rows, step)], x.shape[0]
        return torch.cat([w @ x[cells] for cells, w in (chunk(a, b) for a, b in ctx.cuts)])

    @staticmethod
    def backward(ctx, gy):
        gx, at = gy.new_zeros(ctx.n, gy.shape[2]), 0
        for cells, w in (ctx.chunk(a, b) for a, b in ctx.cuts):
            g = w.transpose(1, 2) @ gy[at:at + cells.shape[0]]
            gx.index_add_(0, cells.reshape(-1), g.reshape(-1, gy.shape[2]))
            at += cells.shape[0]
        return gx, None, None, None


def _apply(op, x, each=1):
    return _Rows.apply(x, op[0], op[1], each)


def _model(x, grids, J, split, cross=False, moments=False):
    """Statistics of x [n, fields]: split(n, V) gives, for level n, the parts of V's rows that are averaged.
    Values [averages, fields (or pairs), coefficients], in the plan's order, and variances with moments."""
    wave = [_wavelet_rows(g) for g in grids]
    down = [_decimation_rows(grids[n], grids[n + 1]) for n in range(J - 1)]
    fields = x.shape[1]
    maps, mods, out = x, [], []

    def psi(n, v):  # [n, R] -> complex [n, R, L]
        y = _apply(wave[n], v, L).reshape(grids[n].n, L, 2, -1)
        return torch.complex(y[:, :, 0], y[:, :, 1]).transpose(1, 2)

    first = []  # mean and mean square of the maps
    for p in split(0, x):
        first.append(torch.stack([p.mean(0), (p * p).mean(0)], -1))
    second = [[(p * p).mean(0), (p ** 4).mean(0)] for p in split(0, x)] if moments else None
    columns = [[f.to(torch.complex128)] for f in first]
    squares = [[torch.stack(s, -1)] for s in second] if moments else None
    for n in range(J):
        if n:
            maps = _apply(down[n - 1], maps)[:, 0]
            mods = [_apply(down[n - 1], m.reshape(m.shape[0], -1))[:, 0].reshape(-1, fields, L) for m in mods]
        z = psi(n, maps)  # [n, fields, L]
        mods.append(z.abs())
        br = psi(n, torch.stack(mods, 2).reshape(grids[n].n, -1)).reshape(grids[n].n, fields, L * (n + 1), L)
        V = torch.cat([z[:, :, None], br], 2)  # operands [n, fields, K, l3]
        for a, v in enumerate(split(n, V)):
            count = v.shape[0]
            ends = [(0, 1), (1, 0)] if cross else [(None, None)]
            for p, (c1, c2) in enumerate(ends):
                if cross:
                    u, w = (v.reshape(count, fields // 2, 2, *v.shape[2:])[:, :, c] for c in (c1, c2))
                else:
                    u = w = v
                zu, zw = u[:, :, 0], w[:, :, 0]
                if p == 0:
                    if cross:
                        ru, rw = (t / torch.sqrt(t.abs() + 1e-8) for t in (zu, zw))
                        columns[a] += [(ru * rw.conj()).mean(0), (zu * zw.conj()).mean(0)]
                    else:
                        columns[a] += [zu.abs().mean(0) + 0j, (zu.abs() ** 2).mean(0) + 0j]
                        if moments:
                            squares[a] += [(zu.abs() ** 2).mean(0), (zu.abs() ** 4).mean(0)]
                u, w = u.permute(1, 3, 2, 0), w.permute(1, 3, 2, 0)  # [fields, l3, K, n]
                columns[a] += _triples((u @ w.conj().transpose(2, 3)) / count, n)
                if moments:
                    q = u.abs() ** 2
                    squares[a] += _triples((q @ q.transpose(2, 3)) / count, n)
    if cross:
        columns = [c[1:] for c in columns]
    values = torch.stack([torch.cat(c, -1) for c in columns])
    if not moments:
        return values, None
    return values, (torch.stack([torch.cat(c, -1) for c in squares]) - values.abs() ** 2).clamp(min=0)


def _triples(gram, n):
    """S3 and S4 of a level from the products [fields, l3, K, K], in the plan's order."""
    out = []
    for j2 in range(n + 1):
        two = slice(1 + L * j2, 1 + L * (j2 + 1))
        out.append(gram[:, :, two, 0].permute(0, 2, 1).reshape(gram.shape[0], -1))
        for j1 in range(j2 + 1):
            one = slice(1 + L * j1, 1 + L * (j1 + 1))
            out.append(gram[:, :, one, two].permute(0, 2, 3, 1).reshape(gram.shape[0], -1))
    return out


def _levels(grid, J):
    out = [grid]
    for _ in range(J - 1):
        out.append(out[-1].coarser())
    return out


def _whole(n, v):
    return [v]


def _mask_split(case):
    levels = []
    for ids in _mask_ids(case):
        per = [torch.tensor(ids, device="cuda")]
        for _ in range(case["J"] - 1):
            per.append(torch.unique(per[-1] // 4))
        levels.append(per)
    return lambda n, v: [v[per[n]] for per in levels]


def _host(*tensors):
    return [t.detach().cpu().numpy() for t in tensors]


def _gradient(values, cot, x):
    loss = (cot.conj() * values).real.sum()
    return torch.autograd.grad(loss, x)[0]


def _exact_sky(case, seed):
    x = _maps(case, seed)
    B, n = case["batch"], _npix(case["nside"])
    grids = _levels(_Grid(case["nside"]), case["J"])
    split = _mask_split(case) if case.get("masks") else _whole
    fields = x.reshape(-1, n).t().contiguous().requires_grad_()
    inner = fields
    if case["kind"] == "spin":
        y = _apply(_spin_rows(case["nside"]), fields).reshape(n, 2, B, 2)  # [n, (re, im), maps, (Q, U)]
        inner = torch.stack([y[:, 0, :, 0] - y[:, 1, :, 1], y[:, 0, :, 1] + y[:, 1, :, 0]], -1).reshape(n, 2 * B)
    values, var = _model(inner, grids, case["J"], split, cross=case["kind"] == "cross",
                         moments=bool(case.get("moments")))
    v = values.transpose(0, 1)  # [fields, averages, coefficients]
    head = (B, 2) if case["kind"] == "spin" else (B,)
    shape = head + ((case["masks"],) if case.get("masks") else ()) + (v.shape[-1],)
    v = v.reshape(shape)
    grad = _gradient(v, _cotangent(shape, seed), fields).t().reshape(x.shape)
    if case["io"] == "autograd":
        return dict(values=v.detach(), grad=grad)
    v, grad = _host(v, grad) if case["io"] == "host" else (_host(v)[0], grad)
    return dict(values=v, var=None if var is None else _host(var.transpose(0, 1).reshape(shape))[0], grad=grad)


def _exact_patch(case, seed):
    centres, radii, cores = _disc_centres(case)
    v, _, _ = _frame(torch.arange(_npix(case["nside"]), device="cuda"), case["nside"])
    ids, parts, core_keys = [], [], []
    for i, c in enumerate(torch.tensor(centres, device="cuda")):
        c = c / torch.linalg.vector_norm(c)
        angle = torch.atan2(torch.linalg.vector_norm(torch.linalg.cross(c.expand_as(v), v), dim=-1), v @ c)
        got = torch.nonzero(angle <= math.radians(radii[i])).reshape(-1)
        ids.append(got)
        parts.append(torch.full_like(got, i))
        core_keys.append(got if cores is None else got[angle[got] <= math.radians(cores[i])])
    del v
    sizes = [i.numel() for i in ids]
    grids = _levels(_Grid(case["nside"], torch.cat(ids), torch.cat(parts)), case["J"])
    inside = []  # per level and disc, the rows of the core
    cuts = [torch.bincount(g.part, minlength=len(ids)).tolist() for g in grids]
    for n, g in enumerate(grids):
        inside.append([torch.searchsorted(s, k) for s, k in zip(torch.split(g.ids, cuts[n]), core_keys)])
        core_keys = [torch.unique(k // 4) for k in core_keys]

    def split(n, t):
        pieces = torch.split(t, cuts[n])
        return pieces if cores is None else [p[r] for p, r in zip(pieces, inside[n])]

    x = _disc_values(sizes, case, seed)[:, None].requires_grad_()
    values, var = _model(x, grids, case["J"], split, moments=bool(case.get("moments")))
    values = values[:, 0]
    grad = _gradient(values, _cotangent(values.shape, seed), x)[:, 0]
    v, grad = _host(values, grad)
    return dict(values=v, var=None if var is None else _host(var[:, 0])[0], grad=grad)


def _exact_synthesis(case, seed):
    """torch's L-BFGS of the weighted squared residual of the statistics."""
    t, x = _synthesis_maps(case, seed)
    grids = _levels(_Grid(case["nside"]), case["J"])
    with torch.no_grad():
        target, var = _model(t.t().contiguous(), grids, case["J"], _whole, moments=True)
        weights = 1.0 / var.clamp(min=1e-12 * var.max())
    x = x.t().contiguous().requires_grad_()
    opt = torch.optim.LBFGS([x], lr=1.0, max_iter=case["iterations"], tolerance_grad=1e-12, tolerance_change=1e-15,
                            history_size=10, line_search_fn="strong_wolfe")

    def closure():
        opt.zero_grad()
        r = _model(x, grids, case["J"], _whole)[0] - target
        loss = (weights * (r.real ** 2 + r.imag ** 2)).sum()
        loss.backward()
        return loss

    opt.step(closure)
    return dict(x=x.detach().t().contiguous(), loss=None)


def _exact_terms(case, seed):
    s = _terms_inputs(case, seed)
    x, (gm, gs, km, ks) = s["x"], s["scale"]
    kx, ky, kd = (torch.tensor(s[k], device="cuda") for k in ("kx", "ky", "kd"))
    t = x * gs + gm
    j = (torch.searchsorted(kx, t, right=True) - 1).clamp(0, kx.numel() - 2)
    h = kx[j + 1] - kx[j]
    u = (t - kx[j]) / h
    y0, y1, d0, d1 = ky[j], ky[j + 1], kd[j] * h, kd[j + 1] * h
    v = y0 + u * (d0 + u * (3 * (y1 - y0) - 2 * d0 - d1 + u * (2 * (y0 - y1) + d0 + d1)))
    dv = (d0 + u * (2 * (3 * (y1 - y0) - 2 * d0 - d1) + u * 3 * (2 * (y0 - y1) + d0 + d1))) / h
    for out, end in ((t <= kx[0], 0), (t >= kx[-1], -1)):
        v, dv = torch.where(out, ky[end] + kd[end] * (t - kx[end]), v), torch.where(out, kd[end], dv)
    k, dk = (v - km) / ks, dv * gs / ks
    level, grad, sums = k, torch.zeros_like(k), []
    for n in range(case["depth"]):
        parent = level.reshape(-1, 4).mean(1)
        d = (level.reshape(-1, 4) - parent[:, None])
        sums.append([float((d ** 2).sum()), float((d ** 4).sum())])
        coef, K, V = s["kurt"][0, n]
        g = s["power"][0, n] * d + coef * (d ** 3 - (d ** 3).mean(1, keepdim=True) - K * V * d)
        grad += g.reshape(-1).repeat_interleave(4 ** n)
        level = parent
    order = torch.sort(x, stable=True).indices
    r = x[order] - s["t"]
    grad = grad * dk
    grad[order] += 2.0 / x.numel() * r
    return dict(k=k, dk=dk, sums=np.array([sums]), grad=grad, perm=None, loss=float((r * r).sum()))


def exact(case, seed):
    if case["kind"] == "terms":
        return _exact_terms(case, seed)
    if case["kind"] == "patch":
        return _exact_patch(case, seed)
    if case["kind"] == "synthesis":
        return _exact_synthesis(case, seed)
    if case["nside"] > 512:  # over 20 seconds
        return None
    return _exact_sky(case, seed)
