"""The work that users of the framework have it do, as cases that can be timed and compared.

A case is a dict of plain values; `listed()` gives the fixed ones, `draw(rng)` further ones of the same
ranges.  `prepare` builds what a user's program holds before the call (images, initial level sets, a
workspace), `run` makes one pass through the public entry points, `work` counts what such a pass cannot do
without and `exact` restates it in float64 torch.

Inputs stand for vessel stacks: a mask of smooth winding structures, bright vessels on a dark background
with noise (uint8, or float32 with the same values), and a level set that is a perturbed mask's smooth
distance-like field, clipped to +-3 where a clipped signed distance is what the pipeline hands over.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "paper-rsf-vesselseg_gb300"))

from rsf_gb300 import Params, Workspace, autograd, driver, tiling  # noqa: E402

DEV = "cuda:0"
# lambda 1, mu 1, nu 0.001 * 255^2, eps 1, dt 0.1: the benchmark configurations' parameters
PAPER = dict(dt=0.1, mu=1.0, lambda1=1.0, lambda2=1.0, nu=0.001 * 255.0 ** 2, eps=1.0)
# what the command line takes when no flag is given
DEFAULTS = dict(dt=0.1, mu=1.0, lambda1=0.1, lambda2=0.1, nu=0.0001, eps=0.2)
# the differentiable checks' parameters: gradients that stay within FP32 over several steps
GENTLE = dict(dt=0.1, mu=0.2, lambda1=1e-4, lambda2=2e-4, nu=0.1, eps=1.0)
SETS = {"paper": PAPER, "defaults": DEFAULTS, "gentle": GENTLE}


def _case(call, z, y, x, sigma, iters, dtype="u8", prm="paper", **kw):
    c = dict(call=call, z=z, y=y, x=x, sigma=sigma, iters=iters, dtype=dtype, prm=prm, boundary="reference")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one cropped patch, a few iterations while a user tries parameters; latency counts
        dict(_case("evolve", 20, 26, 30, 1.5, 10), name="patch 30x26x20 sigma1.5"),
        # the plain benchmark volume: 128^3 bytes, sigma 3
        dict(_case("evolve", 128, 128, 128, 3.0, 10), name="volume 128^3 sigma3"),
        # one large volume at the executable's default sigma of 5
        dict(_case("evolve", 512, 512, 512, 5.0, 4), name="volume 512^3 sigma5"),
        # the batch driver's headline: 48 uneven sub-volumes of a 512 x 1024 x 1024 stack, advanced together
        dict(_case("batch", 512, 1024, 1024, 3.0, 4, cores=256, halo=32, first=32), name="batch 48 tiles sigma3"),
        # float32 stack of ragged size in overlapping tiles, sigma 4
        dict(_case("batch", 301, 450, 517, 4.0, 4, dtype="f32", cores=192, halo=32), name="batch f32 ragged sigma4"),
        # another blur width, ragged sizes, one-sided boundary rule: thin vessels in small sub-volumes
        dict(_case("batch", 150, 263, 333, 2.0, 6, cores=128, halo=16, boundary="clamp"), name="batch ragged sigma2"),
        # the executable's call shape and defaults: NumPy arrays in and out, float32 image, 30 iterations
        dict(_case("host", 61, 187, 203, 5.0, 30, dtype="f32", prm="defaults"), name="host arrays defaults"),
        # the executable's --sigma2 box window for the data term
        dict(_case("evolve", 72, 100, 131, 3.0, 4, prm="paper", sigma2=1.0), name="volume box window"),
        # training through the evolution: a batch of equal crops, forward, soft Dice loss, backward
        dict(_case("grad", 96, 112, 96, 3.0, 4, prm="gentle", batch=4, every=2), name="train batch 4 sigma3"),
        # the same for one small float32 crop at another blur width, checkpoint at every step
        dict(_case("grad", 43, 58, 67, 1.5, 3, dtype="f32", prm="gentle", every=1), name="train one crop sigma1.5"),
        # initial level set of a large seed stack
        dict(_case("sdf", 256, 448, 512, 0.0, 0), name="signed distance 256x448x512"),
        # the whole job: cut, initial level sets, evolve, stitch
        dict(_case("segment", 190, 333, 290, 3.0, 5, cores=128, halo=32, mode="blend"), name="segment blend sigma3"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(("evolve", "evolve", "batch", "batch", "host", "grad", "sdf", "segment", "box"))
    sigma = rng.choice((1.5, 2.0, 3.0, 3.0, 4.0, 5.0, 5.0))
    dtype = rng.choice(("u8", "u8", "f32"))
    boundary = rng.choice(("reference", "reference", "clamp"))

    def size(lo, hi):
        """Extents of about the same magnitude, lo to hi voxels along each axis."""
        m = _log(rng, lo, hi)
        return [min(hi, max(lo, int(round(m * rng.uniform(0.6, 1.4))))) for _ in range(3)]

    if call == "evolve":
        z, y, x = size(16, 448)
        return _case("evolve", z, y, x, sigma, rng.randint(3, 10) if z * y * x < 1 << 24 else 4, dtype,
                     boundary=boundary)
    if call == "batch":
        z, y, x = size(100, 640)
        cores = rng.choice((96, 128, 192, 256))
        while -(-z // cores) * -(-y // cores) * -(-x // cores) > 48:
            cores += 32
        return _case("batch", z, y, x, sigma, 4, dtype, cores=cores, halo=rng.choice((16, 32)), boundary=boundary)
    if call == "host":
        z, y, x = size(24, 256)
        return _case("host", z, y, x, sigma, rng.randint(5, 30), rng.choice(("u8", "f32")), "defaults")
    if call == "box":
        z, y, x = size(32, 128)
        return _case("evolve", z, y, x, rng.choice((2.0, 3.0, 5.0)), rng.randint(2, 4), dtype, sigma2=1.0)
    if call == "grad":
        z, y, x = size(32, 128)
        return _case("grad", z, y, x, rng.choice((1.5, 3.0, 3.0, 4.0, 5.0)), rng.randint(2, 4), dtype, "gentle",
                     batch=rng.randint(1, 4), every=rng.randint(1, 3), boundary=boundary)
    if call == "sdf":
        z, y, x = size(40, 512)
        return _case("sdf", z, y, x, 0.0, 0, rng.choice(("u8", "f32")))
    z, y, x = size(96, 352)
    return _case("segment", z, y, x, sigma, rng.randint(2, 6), dtype, cores=rng.choice((96, 128, 192)),
                 halo=rng.choice((16, 32)), mode=rng.choice(("core", "blend")))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _smooth(shape, gen):
    """Three products of sines with random phases and wavelengths of 16 to 45 voxels, slopes around 1."""
    out = None
    for _ in range(3):
        f = [0.14 + 0.26 * v for v in torch.rand(3, generator=gen).tolist()]
        p = [2.0 * math.pi * v for v in torch.rand(3, generator=gen).tolist()]
        z, y, x = (torch.sin(f[a] * torch.arange(n, device=DEV, dtype=torch.float32) + p[a])
                   for a, n in enumerate(shape))
        zy = 3.5 * z[:, None] * y[None, :]
        t = zy[:, :, None] * x
        out = t if out is None else out.add_(t)
    return out


def _inputs(shape, seed, dtype, clip):
    """image, level set (both on the GPU, shape (L, H, W))."""
    gen = torch.Generator()
    gen.manual_seed(int(seed))
    f = _smooth(shape, gen)
    dgen = torch.Generator(device=DEV)
    dgen.manual_seed(int(seed))
    img = torch.randn(shape, generator=dgen, device=DEV)
    img = img.mul_(18.0).add_(torch.where(f > 0.0, 180.0, 40.0)).clamp_(0.0, 255.0).round_()
    # the segmentation that starts the evolution is off by a voxel or so, here more, there less
    phi = f.add_(_smooth(shape, gen).mul_(0.3))
    if clip:
        phi = phi.clamp_(-3.0, 3.0)
    return (img.to(torch.uint8) if dtype == "u8" else img), phi.contiguous()


def _seed_volume(shape, seed, dtype):
    """A seed stack: 255 (or a probability-like value) inside winding structures, about a tenth of the volume."""
    gen = torch.Generator()
    gen.manual_seed(int(seed))
    f = _smooth(shape, gen)
    return torch.where(f > 2.5, 255.0, 0.0).to(torch.uint8 if dtype == "u8" else torch.float32)


def _tiles(c):
    shape = (c["z"], c["y"], c["x"])
    cores = c["cores"]
    if c.get("first"):  # a thin first core along z, as in the uneven benchmark batch
        zs = list(range(c["first"], c["z"], cores))
        return tiling.plan(shape, ([0] + zs + [c["z"]], cores, cores), c["halo"])
    return tiling.plan(shape, cores, c["halo"])


def _params(c):
    return Params(sigma=c["sigma"], boundary=c["boundary"], sigma2=c.get("sigma2", 0.0), **SETS[c["prm"]])


def prepare(case, seed):
    c = dict(case)
    call, shape = c["call"], (c["z"], c["y"], c["x"])
    s = {"case": c}
    if call != "sdf":
        s["params"] = _params(c)
    if call in ("evolve", "host"):
        img, phi0 = _inputs(shape, seed, c["dtype"], c["prm"] == "paper")
        s["ws"] = Workspace(phi0.numel(), 1)
        if call == "host":
            s["image"], s["phi0"] = img.cpu().numpy(), phi0.cpu().numpy()
            s["phi"] = s["phi0"].copy()
        else:
            s["image"], s["phi0"], s["phi"] = img, phi0, phi0.clone()
    elif call == "batch":
        tiles = _tiles(c)
        ins = [_inputs(t.shape, seed * 4096 + i, c["dtype"], True) for i, t in enumerate(tiles)]
        s["phi0"] = [p for _, p in ins]
        s["pairs"] = [(i, p.clone()) for i, p in ins]
        s["ws"] = Workspace(sum(t.voxels for t in tiles), len(tiles))
    elif call == "grad":
        b = c.get("batch", 0)
        ins = [_inputs(shape, seed * 64 + i, c["dtype"], False) for i in range(max(b, 1))]
        img, phi0 = (torch.stack(v) for v in zip(*ins))
        if not b:
            img, phi0 = img[0].contiguous(), phi0[0].contiguous()
        s["image"], s["phi0"] = img, phi0.requires_grad_(True)
        s["mask"] = img.float() > 110.0
        s["ws"] = Workspace(phi0.numel(), max(b, 1))
        s["weights"] = {n: torch.tensor(SETS[c["prm"]][n], dtype=torch.float32, requires_grad=True)
                        for n in ("lambda1", "lambda2", "mu", "nu")}
    elif call == "sdf":
        s["seed"] = _seed_volume(shape, seed, c["dtype"])
        s["ws"] = Workspace(s["seed"].numel(), 1)
    else:
        s["image"], _ = _inputs(shape, seed, c["dtype"], False)
        s["seed"] = _seed_volume(shape, seed, "u8")
    return s


def run(state):
    s, c = state, state["case"]
    call = c["call"]
    if call == "evolve":
        s["phi"].copy_(s["phi0"])
        return s["ws"].evolve(s["image"], s["phi"], s["params"], c["iters"])
    if call == "host":
        np.copyto(s["phi"], s["phi0"])
        return s["ws"].evolve_host(s["image"], s["phi"], s["params"], c["iters"])
    if call == "batch":
        for (_, p), p0 in zip(s["pairs"], s["phi0"]):
            p.copy_(p0)
        return s["ws"].evolve_batched(s["pairs"], s["params"], c["iters"])
    if call == "grad":
        w = s["weights"]
        phi = autograd.evolve(s["phi0"], s["image"], s["params"], c["iters"], checkpoint_every=c["every"],
                              workspace=s["ws"], **w)
        loss = autograd.soft_dice_loss(phi, s["mask"], s["params"].eps)
        grads = torch.autograd.grad(loss, [s["phi0"]] + [w[n] for n in ("lambda1", "lambda2", "mu", "nu")])
        return [phi.detach(), loss.detach(), *grads]
    if call == "sdf":
        return s["ws"].signed_distance(s["seed"])
    return driver.segment(s["image"], s["seed"], s["params"], c["iters"], cores=c["cores"], halo=c["halo"],
                          mode=c["mode"], device=DEV)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = dict(case)
    shape = (c["z"], c["y"], c["x"])
    isz = 1 if c["dtype"] == "u8" else 4
    n = c["z"] * c["y"] * c["x"]
    if c["call"] == "sdf":
        return {"bytes": n * (isz + 4), "flops": 12 * n}
    k = len(_taps(c["sigma"]))
    boxes = [t.shape for t in _tiles(c)] if c["call"] in ("batch", "segment") else [shape] * max(c.get("batch", 1), 1)
    flops = vox = 0
    for b in boxes:
        v = [max(m - k + 1, 0) for m in b]
        v = v if min(v) > 0 else [0, 0, 0]
        m = b[0] * b[1] * b[2]
        # four fields along x, y, z (two flops a tap) and about 120 pointwise
        blur = 8 * k * (b[0] * b[1] * v[2] + b[0] * v[1] * v[2] + v[0] * v[1] * v[2])
        box = 6 * (2 * int(c.get("sigma2", 0.0)) + 1) ** 3 * m if c.get("sigma2", 0.0) >= 1.0 else 0
        # a training step runs each iteration forward and once more backward, at about two and a half times the cost
        flops += (blur + 120 * m + box) * c["iters"] * (3.5 if c["call"] == "grad" else 1)
        vox += m
    if c["call"] == "grad":
        return {"bytes": vox * (4 + isz + 1 + 4 + 4), "flops": flops}  # level set, image, mask; result, gradient
    if c["call"] == "segment":
        return {"bytes": n * (isz + 1 + 4), "flops": flops}
    return {"bytes": vox * (8 + isz), "flops": flops}


# ---------------------------------------------------------------------------
# The same in float64 torch
# ---------------------------------------------------------------------------
def _f32(v):
    return float(np.float32(v))


def _taps(sigma):
    """k = floor(7 sigma) made odd, exp(-(i - k/2)^2 / u) / sqrt(u pi), u = (int)(2 sigma^2), as float32 values."""
    k = int(np.float32(7.0) * np.float32(sigma))
    k += 1 - k % 2
    u = int(np.float32(2.0) * np.float32(sigma) * np.float32(sigma))
    s = np.sqrt(np.float32(u) * np.float32(math.pi))
    d = np.arange(k, dtype=np.float32) - np.float32(k // 2)
    return ((np.float32(1.0) / s) * np.exp(((-d * d) / np.float32(u)).astype(np.float64)).astype(np.float32)).tolist()


def _blur(f, taps):
    for axis in (2, 1, 0):
        n = f.shape[axis] - len(taps) + 1
        if torch.is_grad_enabled() and f.requires_grad:
            f = sum(g * f.narrow(axis, i, n) for i, g in enumerate(taps))
        else:
            out = taps[0] * f.narrow(axis, 0, n)
            for i in range(1, len(taps)):
                out.add_(f.narrow(axis, i, n), alpha=taps[i])
            f = out
    return f


def _dx(f, boundary):
    flat = f.reshape(-1)
    r = torch.cat((f[..., 1:], f[..., -1:]), dim=2)
    if boundary == "reference":  # x = 0 reads the previous element in memory
        l = torch.cat((flat[:1], flat[:-1])).reshape(f.shape)
    else:
        l = torch.cat((f[..., :1], f[..., :-1]), dim=2)
    return 0.5 * (r - l)


def _d(f, axis, boundary):
    if axis == 2:
        return _dx(f, boundary)
    n = f.shape[axis]
    r = torch.cat((f.narrow(axis, 1, n - 1), f.narrow(axis, n - 1, 1)), dim=axis)
    l = torch.cat((f.narrow(axis, 0, 1), f.narrow(axis, 0, n - 1)), dim=axis)
    return 0.5 * (r - l)


def _unit(phi, boundary):
    """Gradient and gradient over its length plus 1e-6, along x, y, z."""
    g = [_d(phi, a, boundary) for a in (2, 1, 0)]
    m2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2]
    zero = m2 == 0
    mag = torch.where(zero, torch.zeros_like(m2), torch.sqrt(torch.where(zero, torch.ones_like(m2), m2)))
    return g, [v / (mag + 1e-6) for v in g]


def _data(phi, img, taps, p, box):
    """e_out, e_in of the data term."""
    h = 0.5 * (1.0 + (2.0 / math.pi) * torch.atan(phi / _f32(p["eps"])))
    k, r = len(taps), len(taps) // 2
    fits = []
    for w in (h, 1.0 - h):
        f = torch.ones_like(phi)
        if min(phi.shape) >= k:
            inner = _blur(img * w, taps) / _blur(w, taps)
            f = torch.nn.functional.pad(inner - 1.0, (r,) * 6) + 1.0
        fits.append(f)
    if box < 1:
        return [(img - f) ** 2 for f in fits]

    def window(v):
        for axis in range(3):
            n = v.shape[axis]
            parts = []
            for o in range(-box, box + 1):
                sh = torch.zeros_like(v)
                m = n - abs(o)
                if m > 0:
                    sh.narrow(axis, max(-o, 0), m).copy_(v.narrow(axis, max(o, 0), m))
                parts.append(sh)
            v = sum(parts)
        return v

    n, s1, s2 = window(torch.ones_like(img)), window(img), window(img * img)
    w = 1.0 / (2 * box + 1) ** 2
    return [w * (s2 - 2.0 * f * s1 + n * f * f) for f in fits]


def _step(phi, img, taps, p, boundary, box=0, weights=None):
    l1, l2, mu, nu = weights if weights is not None else [_f32(p[n]) for n in ("lambda1", "lambda2", "mu", "nu")]
    dt, eps = _f32(p["dt"]), _f32(p["eps"])
    eo, ei = _data(phi, img, taps, p, box)
    g, n = _unit(phi, boundary)
    kappa = sum(_d(v, a, boundary) for v, a in zip(n, (2, 1, 0)))
    lap = sum(_d(v, a, boundary) for v, a in zip(g, (2, 1, 0)))
    delta = (1.0 / math.pi) * eps / (eps * eps + phi * phi)
    return phi - delta * (l1 * eo - l2 * ei) * dt + nu * dt * delta * kappa + mu * dt * (lap - kappa)


def _evolve64(phi, img, c):
    taps, p = _taps(c["sigma"]), SETS[c["prm"]]
    phi, img = phi.double(), img.double()
    with torch.no_grad():
        for _ in range(c["iters"]):
            phi = _step(phi, img, taps, p, c["boundary"], int(c.get("sigma2", 0.0)))
    return phi


def _distance2(feature):
    """Squared distance of every voxel to the nearest feature voxel; a huge value where there is none."""
    big = 1 << 28
    d = torch.where(feature, 0, big).to(torch.int32)
    for axis in range(3):
        n = d.shape[axis]
        at = torch.arange(n, device=d.device, dtype=torch.int32).reshape([-1 if a == axis else 1 for a in range(3)])
        out = torch.full_like(d, big)
        for q in range(n):
            out = torch.minimum(out, d.narrow(axis, q, 1) + (at - q) ** 2)
        d = out
    return d


def _sdf64(seed):
    inside = seed.float() > 13.0
    if inside.all() or not inside.any():
        return torch.full(seed.shape, float(sum(seed.shape)) * (1.0 if inside.all() else -1.0), device=seed.device,
                          dtype=torch.float64)
    return torch.where(inside, _distance2(~inside).double().sqrt(), -_distance2(inside).double().sqrt())


def _stitch64(parts, tiles, shape, mode):
    out = torch.zeros(shape, dtype=torch.float64, device=DEV)
    if mode == "core":
        for part, t in zip(parts, tiles):
            out[t.core_slices()] = part[t.core_in_tile()]
        return out
    total = torch.zeros_like(out)
    for part, t in zip(parts, tiles):
        w = torch.ones((1, 1, 1), dtype=torch.float64, device=DEV)
        for a in range(3):
            at = torch.arange(t.lo[a], t.hi[a], device=DEV, dtype=torch.float64)
            v = torch.ones_like(at)
            for o in tiles:
                if o.chi[a] == t.clo[a] and o.hi[a] > t.lo[a]:  # the tile before: rise across the overlap
                    v = torch.where(at < o.hi[a], (at - t.lo[a]) / max(o.hi[a] - t.lo[a] - 1, 1), v)
                    break
            u = torch.ones_like(at)
            for o in tiles:
                if o.clo[a] == t.chi[a] and o.lo[a] < t.hi[a]:  # the tile after: fall
                    u = torch.where(at >= o.lo[a], (t.hi[a] - 1 - at) / max(t.hi[a] - o.lo[a] - 1, 1), u)
                    break
            w = w * (u * v).reshape([-1 if b == a else 1 for b in range(3)])
        out[t.slices()] += w * part
        total[t.slices()] += w
    return out / total


def exact(case, seed):
    c = dict(case)
    call, shape = c["call"], (c["z"], c["y"], c["x"])
    if call in ("evolve", "host"):
        img, phi = _inputs(shape, seed, c["dtype"], c["prm"] == "paper")
        return _evolve64(phi, img, c)
    if call == "batch":
        out = []
        for i, t in enumerate(_tiles(c)):
            img, phi = _inputs(t.shape, seed * 4096 + i, c["dtype"], True)
            out.append(_evolve64(phi, img, c))
        return out
    if call == "sdf":
        return _sdf64(_seed_volume(shape, seed, c["dtype"]))
    if call == "segment":
        img, _ = _inputs(shape, seed, c["dtype"], False)
        sd = _seed_volume(shape, seed, "u8")
        tiles = _tiles(c)
        parts = [_evolve64(_sdf64(sd[t.slices()]).float(), img[t.slices()], c) for t in tiles]
        return _stitch64(parts, tiles, shape, c["mode"])
    # grad
    b = c.get("batch", 0)
    p, taps = SETS[c["prm"]], _taps(c["sigma"])
    ins = [_inputs(shape, seed * 64 + i, c["dtype"], False) for i in range(max(b, 1))]
    weights = [torch.tensor(_f32(p[n]), dtype=torch.float64, device=DEV, requires_grad=True)
               for n in ("lambda1", "lambda2", "mu", "nu")]
    phi0 = [q.double().requires_grad_(True) for _, q in ins]
    phis = []
    for (img, _), q in zip(ins, phi0):
        img = img.double()
        for _ in range(c["iters"]):
            q = _step(q, img, taps, p, c["boundary"], 0, weights)
        phis.append(q)
    phi = torch.stack(phis) if b else phis[0]
    mask = torch.stack([i.float() > 110.0 for i, _ in ins]) if b else ins[0][0].float() > 110.0
    h = 0.5 * (1.0 + (2.0 / math.pi) * torch.atan(phi / _f32(p["eps"])))
    m = mask.double()
    loss = 1.0 - 2.0 * (h * m).sum() / (h.sum() + m.sum())
    grads = torch.autograd.grad(loss, phi0 + weights)
    g0 = torch.stack(grads[:len(phi0)]) if b else grads[0]
    return [phi.detach(), loss.detach(), g0, *grads[len(phi0):]]
