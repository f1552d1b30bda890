"""The work a user of this library has it do, as timed cases.

The ranges come from the repository's own configurations: images from 64x64x32
to 128x128x159 voxels, sinograms from 64x64 bins x 192 planes to 147x168 x 1293
and 128x160 x 4319, span 3 to 11, 1 to 16 subsets, FP32 and 16-bit storage of
the ratio sinogram, the back projector in both axial forms.  Operators are
called on device buffers (Context.*), whole reconstructions through Recon and
Batch.  Values: ellipsoid phantoms, their Poisson counts and ratios, gain
normalizations with or without dead bins.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gfirst_gb300 as gf

GEO = ("res", "nzs", "nrad", "nang", "span", "nseg", "pitch", "diam", "fov")
SMALL = dict(zip(GEO, (64, 32, 64, 64, 3, 11, 1.6, 84.8772096, 51.2)))
SERVE64 = dict(zip(GEO, (64, 64, 64, 64, 3, 21, 1.6, 84.8772096, 51.2)))
SERVE96 = dict(zip(GEO, (96, 96, 96, 96, 3, 31, 1.6, 127.3158, 76.8)))
REFERENCE = dict(zip(GEO, (128, 159, 147, 168, 11, 15, 1.63, 165.7758, 100.0)))
PRECLINICAL = dict(zip(GEO, (128, 159, 128, 160, 3, 53, 1.6, 165.7758, 100.0)))


def listed():
    return [
        # one subset's projection of a small scanner: a call that latency rules
        dict(name="fp_small", op="fp", **SMALL, nsub=4, subset=1),
        # the whole sinogram of the reference scanner in one call (a bare projection, the normalization)
        dict(name="fp_reference_full", op="fp", **REFERENCE, nsub=1, subset=0),
        # one subset of the full-scale scanner
        dict(name="fp_preclinical", op="fp", **PRECLINICAL, nsub=16, subset=5),
        # the back projector in its default form: small, and the full-scale subset of a first iteration
        dict(name="bp_small", op="bp", **SMALL, nsub=4, subset=2, form="view", gaps=0.02, late=False),
        dict(name="bp_preclinical", op="bp", **PRECLINICAL, nsub=16, subset=3, form="view", gaps=0.0, late=False),
        # the form with the reference's rounding, every angle, dead bins, empty rays outside the body
        dict(name="bp_reference_voxel", op="bp", **REFERENCE, nsub=1, subset=0, form="voxel", gaps=0.02, late=True),
        # the image update and the joint filter on full-scale images
        dict(name="update_preclinical", op="update", **PRECLINICAL, nsub=16),
        dict(name="bilateral_preclinical", op="bilateral", **PRECLINICAL, nsub=16),
        # a served request: host data in, two iterations, image out
        dict(name="request_64", op="recon", **SERVE64, nsub=8, iters=2, storage="f16", gaps=0.0, counts=2e6, load=True),
        # one iteration (16 sub-iterations) of the full-scale reconstruction, data resident
        dict(name="recon_preclinical", op="recon", **PRECLINICAL, nsub=16, iters=1, storage="f32", gaps=0.0,
             counts=5e7, load=False),
        # doubles and triples from a VLOR list, one iteration with the joint filter
        dict(name="triples_reference", op="triples", **REFERENCE, nsub=8, iters=1, storage="bf16", gaps=0.02,
             counts=4e7, events=1000000),
        # dynamic frames of uneven counts and subset counts, fused, from one graph
        dict(name="frames_96", op="frames", **SERVE96, frames=8, iters=1, storage="f16", gaps=0.0, counts=1e7),
    ]


def _geometry(rng, widest=128):
    """A scanner between the small and the full-scale one, odd sizes among them."""
    res = int(round(math.exp(rng.uniform(math.log(48), math.log(widest)))))
    nzs = int(round(math.exp(rng.uniform(math.log(24), math.log(159)))))
    nrad = max(33, min(147, res + rng.randint(-8, 19)))
    nang = rng.randint(48, 160)
    span = rng.choice([1, 3, 5, 7, 9, 11])
    vx = rng.uniform(0.65, 0.95)
    fov = round(res * vx, 4)
    # widest odd number of segments whose outermost still has planes
    most = 1
    while most < 53 and nzs - 2 * ((most + 1) // 2 * span + span // 2 + 1) >= 2:
        most += 2
    nseg = 2 * rng.randint(0, most // 2) + 1
    return dict(res=res, nzs=nzs, nrad=nrad, nang=nang, span=span, nseg=nseg, pitch=round(rng.uniform(1.5, 1.7), 3),
                diam=round(fov * 1.657758, 4), fov=fov)


def draw(rng):
    op = rng.choice(["fp", "fp", "bp", "bp", "bp", "update", "bilateral", "recon", "recon", "triples", "frames"])
    g = _geometry(rng, 96 if op == "frames" else 128)
    nsub = rng.choice([1, 2, 4, 5, 8, 16])
    gaps = rng.choice([0.0, 0.0, 0.02])
    storage = rng.choice(["f32", "f32", "f16", "bf16"])
    counts = float(round(math.exp(rng.uniform(math.log(1e6), math.log(5e7)))))
    if op == "fp":
        return dict(op=op, **g, nsub=nsub, subset=rng.randrange(nsub))
    if op == "bp":
        return dict(op=op, **g, nsub=nsub, subset=rng.randrange(nsub), form=rng.choice(["view", "view", "voxel"]),
                    gaps=gaps, late=rng.choice([False, True]))
    if op in ("update", "bilateral"):
        return dict(op=op, **g, nsub=nsub)
    nsub = rng.choice([2, 4, 5, 8, 16])
    if op == "recon":
        return dict(op=op, **g, nsub=nsub, iters=1, storage=storage, gaps=gaps, counts=counts,
                    load=rng.choice([False, True]))
    if op == "triples":
        return dict(op=op, **g, nsub=nsub, iters=1, storage=storage, gaps=gaps, counts=counts,
                    events=int(round(math.exp(rng.uniform(math.log(1e4), math.log(1e6))))))
    return dict(op=op, **g, frames=rng.randint(2, 6), iters=1, storage=storage, gaps=gaps, counts=counts)


# ---------------------------------------------------------------- inputs
def _geo(case):
    return gf.Geometry(*(case[k] for k in GEO))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _phantom(case, seed, organs=8):
    """Body ellipsoid (activity 1) with hot organs, [NZS][RES][RES]."""
    rs = np.random.RandomState(seed % (1 << 31))
    res, nzs = case["res"], case["nzs"]
    ar = lambda n: torch.arange(n, dtype=torch.float32, device="cuda")  # noqa: E731
    z, y, x = torch.meshgrid(ar(nzs), ar(res), ar(res), indexing="ij")
    c, cz = (res - 1) / 2.0, (nzs - 1) / 2.0
    ax, ay, az = 0.31 * res, 0.23 * res, 0.44 * nzs
    body = ((x - c) / ax) ** 2 + ((y - c) / ay) ** 2 + ((z - cz) / az) ** 2 <= 1.0
    img = body.float()
    for _ in range(organs):
        ox, oy, oz = rs.uniform(-0.6, 0.6) * ax, rs.uniform(-0.6, 0.6) * ay, rs.uniform(-0.7, 0.7) * az
        sx, sy, sz = rs.uniform(0.07, 0.25) * ax, rs.uniform(0.07, 0.25) * ay, rs.uniform(0.05, 0.2) * az
        o = ((x - c - ox) / sx) ** 2 + ((y - c - oy) / sy) ** 2 + ((z - cz - oz) / sz) ** 2 <= 1.0
        img = torch.where(o & body, torch.full_like(img, rs.uniform(2.0, 20.0)), img)
    return img.reshape(-1)


def _view(ctx, t):
    return gf.DeviceArray.view(ctx, t.data_ptr(), t.numel())


def _gains(n, case, gen):
    """Normalization gains U(0.85, 1.15), 0 in the dead bins."""
    gains = 0.85 + 0.3 * torch.rand(n, generator=gen, device="cuda")
    if case["gaps"]:
        gains[torch.rand(n, generator=gen, device="cuda") < case["gaps"]] = 0.0
    return gains


def _project(ctx, img):
    out = torch.zeros(ctx.ndata, device="cuda")
    torch.cuda.synchronize()
    for s in range(ctx.nsub):
        ctx.forward_project(_view(ctx, img), s, _view(ctx, out))
    ctx.sync()
    return out


def _counts(lam, gains, counts, gen):
    """Poisson prompts of lam at the given total, then a low uniform background, as a sinogram file holds them."""
    m = lam * gains
    prompts = torch.poisson(m * (counts / float(m.double().sum())), generator=gen)
    out = np.empty(2 * lam.numel(), np.float32)
    out[: lam.numel()] = prompts.cpu().numpy()
    out[lam.numel():] = 0.0
    return out


def _ratio(case, ctx, gen):
    """A data/projection ratio sinogram and its mask: Poisson counts over their means inside the body;
    outside it 0 (the first iterations: activity there, no counts) or the gap value (later ones)."""
    nrad, nang, P = case["nrad"], case["nang"], ctx.P
    ar = lambda n: torch.arange(n, dtype=torch.float32, device="cuda")  # noqa: E731
    half = 0.5 * case["pitch"]
    r = (ar(nrad) - (nrad - 1) / 2) * half
    th = math.pi * ar(nang) / nang
    width = torch.sqrt((0.31 * case["fov"] * torch.cos(th)) ** 2 + (0.23 * case["fov"] * torch.sin(th)) ** 2)
    chord = torch.sqrt((1 - (r[None, :] / width[:, None]) ** 2).clamp(min=0))
    lam = (40.0 * chord).expand(P, nang, nrad)
    corr = torch.poisson(lam.contiguous(), generator=gen) / lam.clamp(min=1.0)
    corr = torch.where(lam > 0, corr, torch.full_like(corr, -1000.0 if case["late"] else 0.0))
    calib = torch.ones_like(corr)
    if case["gaps"]:
        calib[torch.rand(corr.shape, generator=gen, device="cuda") < case["gaps"]] = -1000.0
    calib[:, :, (r.abs() > 0.5 * case["fov"])] = -1000.0
    return corr.reshape(-1).contiguous(), calib.reshape(-1).contiguous()


def _events(lam, n, gen):
    """VLOR events: one bin drawn from the projection, the other anywhere, 1-based, in either order."""
    cdf = torch.cumsum(lam.double(), 0)
    true = torch.searchsorted(cdf, torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1])
    other = torch.randint(0, lam.numel(), (n,), generator=gen, device="cuda")
    swap = torch.rand(n, generator=gen, device="cuda") < 0.5
    ev = torch.stack([torch.where(swap, other, true), torch.where(swap, true, other)], 1) + 1
    return ev.clamp(max=lam.numel()).int().cpu().numpy()


def prepare(case, seed):
    op, gen = case["op"], _gen(seed)
    s = {"case": case}
    if op == "frames":
        s["ctxs"], s["recs"] = [], []
        rs = np.random.RandomState(seed % (1 << 31))
        lam = None
        for k in range(case["frames"]):
            ctx = gf.Context(_geo(case), nsub=(4, 8, 16)[rs.randint(3)])
            if lam is None:
                lam = _project(ctx, _phantom(case, seed))
                gains = _gains(ctx.ndata, case, gen)
                norm = gains.cpu().numpy()
            rec = gf.Recon(ctx, 1, niter=case["iters"], storage=case["storage"])
            rec.load(dsino=_counts(lam, gains, case["counts"] * rs.uniform(0.02, 1.0), gen), norm=norm)
            rec._keep = None
            s["ctxs"].append(ctx)
            s["recs"].append(rec)
        s["batch"] = gf.Batch(s["recs"])
        s["batch"].set_fused(True)
        torch.cuda.synchronize()
        return s
    ctx = s["ctx"] = gf.Context(_geo(case), nsub=case["nsub"])
    if op == "fp":
        s["img"], s["out"] = _phantom(case, seed), torch.zeros(ctx.ndata, device="cuda")
        s["args"] = (_view(ctx, s["img"]), case["subset"], _view(ctx, s["out"]))
    elif op == "bp":
        ctx.set_bp_form(case["form"])
        s["corr"], s["calib"] = _ratio(case, ctx, gen)
        s["numer"], s["denom"] = torch.empty(ctx.nvox, device="cuda"), torch.empty(ctx.nvox, device="cuda")
        s["args"] = (_view(ctx, s["corr"]), _view(ctx, s["calib"]), case["subset"], _view(ctx, s["numer"]),
                     _view(ctx, s["denom"]))
    elif op == "update":
        # sums of a subset's views: 300 samples of ratio about 1, none in the corners
        s["img"] = _phantom(case, seed) + 0.1
        s["denom"] = torch.floor(300 * torch.rand(ctx.nvox, generator=gen, device="cuda"))
        s["numer"] = s["denom"] * (0.999 + 0.002 * torch.rand(ctx.nvox, generator=gen, device="cuda"))
        s["args"] = (_view(ctx, s["img"]), _view(ctx, s["numer"]), _view(ctx, s["denom"]))
    elif op == "bilateral":
        s["ref"] = _phantom(case, seed)
        s["img"] = _phantom(case, seed + 1) * (0.8 + 0.4 * torch.rand(ctx.nvox, generator=gen, device="cuda"))
        s["out"] = torch.empty(ctx.nvox, device="cuda")
        s["args"] = (_view(ctx, s["img"]), _view(ctx, s["ref"]), float(s["ref"].max()), _view(ctx, s["out"]))
    else:
        lam = _project(ctx, _phantom(case, seed))
        gains = _gains(ctx.ndata, case, gen)
        data = {"dsino": _counts(lam, gains, case["counts"], gen), "norm": gains.cpu().numpy()}
        mode = 3 if op == "triples" else 1
        if mode == 3:
            lam = _project(ctx, _phantom(case, seed + 1, organs=5))
            data["tsino"] = _counts(lam, gains, 0.05 * case["counts"], gen)
            data["events"] = _events(lam, case["events"], gen)
        rec = s["rec"] = gf.Recon(ctx, mode, niter=case["iters"], storage=case["storage"])
        if case.get("load"):  # a client's page-locked buffers
            s["data"] = {k: gf.host_copy(v) for k, v in data.items()}
        else:
            rec.load(**data)
            rec._keep = None
    torch.cuda.synchronize()
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "fp":
        s["ctx"].forward_project(*s["args"])
        return s["out"]
    if op == "bp":
        s["ctx"].back_project(*s["args"])
        return [s["numer"], s["denom"]]
    if op == "update":
        s["ctx"].image_update(*s["args"])
        return s["img"]
    if op == "bilateral":
        s["ctx"].bilateral(*s["args"])
        return s["out"]
    if op == "frames":
        for r in s["recs"]:
            r.restart()
        s["batch"].iterate(case["iters"])
        return [r.image(0) for r in s["recs"]]
    r = s["rec"]
    if case.get("load"):
        r.load(**s["data"])
    else:
        r.restart()
    r.iterate(case["iters"])
    return [r.image(0), r.image(1)] if op == "triples" else [r.image(0)]


# ---------------------------------------------------------------- work
def _zmin(case, k):
    return 0 if k == 0 else ((k + 1) // 2 - 1) * case["span"] + case["span"] // 2 + 1


def _planes(case):
    return sum(case["nzs"] - 2 * _zmin(case, k) for k in range(case["nseg"]))


def work(case):
    """Each input read and each output written once; 4 operations per ray sample (a 1-D
    interpolation added up, the in-plane part shared by all planes) and 10 per voxel and
    view in its range (ratio and mask)."""
    res, op = case["res"], case["op"]
    nvox, P = res * res * case["nzs"], _planes(case)
    bins = P * case["nang"] * case["nrad"]
    if op == "update":
        return {"bytes": 16 * nvox, "flops": 25 * nvox}
    if op == "bilateral":
        return {"bytes": 12 * nvox, "flops": 729 * 8 * nvox}
    pair = 8 if case.get("storage", "f32") == "f32" else 4
    fp = bins * (res + 1) * 4
    bp = P * res * res * case["nang"] * 10
    if op == "fp":
        n = case["nsub"]
        return {"bytes": 4 * nvox + 4 * bins / n, "flops": fp / n}
    if op == "bp":
        n = case["nsub"]
        return {"bytes": 8 * nvox + 8 * bins / n, "flops": bp / n}
    it = {"bytes": bins * (9 + 2 * pair), "flops": fp + bp}  # one iteration: every subset once
    k = case["iters"] * {"recon": 1, "triples": 2, "frames": case.get("frames", 1)}[op]
    w = {"bytes": k * it["bytes"] + 4 * nvox, "flops": k * it["flops"]}
    if case.get("load"):
        w["bytes"] += 12 * bins
    return w


# ---------------------------------------------------------------- in 64 bits
F64 = torch.float64


class _Exact:
    """The path's operators in 64 bits on file layouts, from their formulas."""

    def __init__(self, case):
        self.c = case
        f = lambda v: float(np.float32(v))  # noqa: E731
        self.res, self.nzs, self.nrad, self.nang = case["res"], case["nzs"], case["nrad"], case["nang"]
        self.pitch, self.diam, self.fov = f(case["pitch"]), f(case["diam"]), f(case["fov"])
        self.vx = self.fov / self.res
        self.pi = f(3.1415926)
        self.segs, acc = [], 0
        for k in range(case["nseg"]):
            zmin = _zmin(case, k)
            n = self.nzs - 2 * zmin
            self.segs.append((zmin, n, acc, (0 if k == 0 else 1 - 2 * (k % 2)) * zmin))
            acc += n
        self.P = acc
        self.radm, self.resm = (self.nrad - 1) / 2, (self.res - 1) / 2

    def ar(self, n):
        return torch.arange(n, dtype=F64, device="cuda")

    def trig(self, t):
        a = -t / self.nang * self.pi + self.pi
        return math.sin(a), math.cos(a)

    def fp(self, img, nsub, subset, out):
        res, nzs = self.res, self.nzs
        img = img.to(F64).view(nzs, res, res)
        out = out.view(self.P, self.nang, self.nrad)
        lam = torch.arange(math.floor(-0.5 * res), math.floor(0.5 * res) + 1, dtype=F64, device="cuda")
        for t in range(subset, self.nang, nsub):
            sn, cs = self.trig(t)
            x0 = 0.5 * self.pitch / self.vx * (self.ar(self.nrad) - self.radm)
            x = (self.resm + x0 * cs)[None, :] + lam[:, None] * sn
            y = (self.resm + x0 * sn)[None, :] - lam[:, None] * cs
            fx, fy = x.floor(), y.floor()
            wx, wy = x - fx, y - fy
            i0, i1 = fx.long().clamp(0, res - 1), (fx.long() + 1).clamp(0, res - 1)
            j0, j1 = fy.long().clamp(0, res - 1), (fy.long() + 1).clamp(0, res - 1)
            B = img[:, j0, i0] * ((1 - wx) * (1 - wy)) + img[:, j0, i1] * (wx * (1 - wy)) + \
                img[:, j1, i0] * ((1 - wx) * wy) + img[:, j1, i1] * (wx * wy)  # [nzs, L, nrad]
            for zmin, n, acc, zs in self.segs:
                dz = self.vx * zs / (0.5 * self.diam)
                m = (lam * dz).floor()
                f = (lam * dz - m)[None, :, None]
                k = (self.ar(n)[:, None] + zmin + m[None, :]).long()  # [n, L]
                k0, k1 = k.clamp(0, nzs - 1), (k + 1).clamp(0, nzs - 1)
                L = torch.arange(lam.numel(), device="cuda")[None, :]
                out[acc:acc + n, t] = (B[k0, L] * (1 - f) + B[k1, L] * f).sum(1)
        return out.view(-1)

    def bp(self, corr, calib, nsub, subset):
        res, nzs = self.res, self.nzs
        corr, calib = corr.view(self.P, self.nang, self.nrad), calib.view(self.P, self.nang, self.nrad)
        num, den = (torch.zeros(nzs, res * res, dtype=F64, device="cuda") for _ in range(2))
        xv = (self.ar(res) - self.resm).repeat(res)
        yv = (self.ar(res) - self.resm).repeat_interleave(res)
        z0 = self.ar(nzs)[:, None]
        for t in range(subset, self.nang, nsub):
            sn, cs = self.trig(t)
            x = self.radm + (xv * cs + yv * sn) * (self.vx / (self.pitch / 2))
            yrot = -xv * sn + yv * cs
            fx = x.floor()
            a = x - fx
            i0, i1 = fx.long().clamp(0, self.nrad - 1), (fx.long() + 1).clamp(0, self.nrad - 1)
            for zmin, n, acc, zs in self.segs:
                z = z0 + yrot[None, :] * (self.vx * zs / (self.diam / 2))
                fz = z.floor()
                b = z - fz
                ok = (z + 0.5 >= zmin) & (z + 0.5 < nzs - zmin)
                j0, j1 = fz.long().clamp(0, nzs - 1), (fz.long() + 1).clamp(0, nzs - 1)
                got = []
                for src in (corr, calib):
                    v = torch.full((nzs, self.nrad), -1000.0, dtype=F64, device="cuda")
                    v[zmin:nzs - zmin] = src[acc:acc + n, t]
                    row = torch.lerp(v[:, i0], v[:, i1], a[None, :])  # [nzs, columns]
                    got.append(torch.lerp(row.gather(0, j0), row.gather(0, j1), b))
                ok &= (got[0] >= 0) & (got[1] >= 0)
                num += torch.where(ok, got[0], 0.0)
                den += torch.where(ok, got[1], 0.0)
        return num.view(-1), den.view(-1)

    def taps(self, psf):
        k = np.arange(-4, 5) * float(np.float32(1.662)) / float(np.float32(psf + 0.1))
        w = np.exp(-k * k)
        return w / w.sum()

    def conv_xy(self, img, psf):
        """9 taps along y (zeros outside), then along x; the 4 border columns keep the input."""
        res = self.res
        v, w = img.view(self.nzs, res, res), self.taps(psf)
        p = torch.nn.functional.pad(v, (0, 0, 4, 4))
        yc = sum(p[:, k:k + res] * w[k] for k in range(9))
        out = v.clone()
        out[:, :, 4:res - 4] = sum(yc[:, :, k:k + res - 8] * w[k] for k in range(9))
        return out.reshape(-1)

    def filter_z(self, c):
        """Axial filter; the voxel of column (0, 0) takes the rule of the slice before it."""
        nzs, w = self.nzs, np.exp(-np.arange(-2, 3) ** 2.0)
        w = w / w.sum()
        v = c.view(nzs, -1)
        p = torch.nn.functional.pad(v, (0, 0, 2, 2))
        third = float(np.float32(0.333))
        two_up, two_dn = 0.5 * (v + p[3:nzs + 3]), 0.5 * (p[1:nzs + 1] + v)
        three = third * (p[1:nzs + 1] + v + p[3:nzs + 3])
        five = sum(p[k:k + nzs] * float(w[k]) for k in range(5))
        rule = lambda K: two_up if K == 0 else two_dn if K == nzs - 1 else three if K in (1, nzs - 2) else five  # noqa: E731
        out = torch.stack([rule(z)[z] for z in range(nzs)])
        for z in range(1, nzs):
            out[z, 0] = rule(z - 1)[z, 0]
        return out

    def update(self, img, num, den, psf=1.5):
        ratio = torch.where(den < float(np.float32(0.001)), torch.ones_like(num), num / den)
        f = self.filter_z(self.conv_xy(ratio, psf))
        f[0, 0] = den[0]
        out = img.view(self.nzs, -1) * f
        out[0], out[-1] = out[1].clone(), out[-2].clone()
        return out.reshape(-1)

    def bilateral(self, img, ref, max_ref, r=4, sigma3d=0.75, sigmai=0.025):
        res, nzs = self.res, self.nzs
        s3, si = (2 * float(np.float32(s)) for s in (sigma3d, sigmai))
        ref, img = ref.to(F64).view(nzs, res, res), img.to(F64).view(nzs, res, res)
        num, den = torch.zeros_like(ref), torch.zeros_like(ref)
        for dz in range(-r, r + 1):
            for dy in range(-r, r + 1):
                for dx in range(-r, r + 1):
                    a, b = [], []  # voxel ranges, neighbour ranges
                    for d, n in ((dz, nzs), (dy, res), (dx, res)):
                        a.append(slice(max(0, -d), n - max(0, d)))
                        b.append(slice(max(0, d), n - max(0, -d)))
                    a, b = tuple(a), tuple(b)
                    w = torch.exp(-((ref[b] - ref[a]) / max_ref) ** 2 / si ** 2) * \
                        math.exp(-(dx * dx + dy * dy + dz * dz) / s3 ** 2)
                    den[a] += w
                    num[a] += w * img[b]
        out = torch.where(den > 1e-8, num / den, 0.0)
        out[:r], out[:, :r], out[:, :, :r] = 0.0, 0.0, 0.0
        return out.reshape(-1)

    def recon(self, dsino, norm, nsub, iters):
        """Multiplicative update over ordered subsets from a unit cylinder."""
        res, nzs, nd = self.res, self.nzs, self.P * self.nang * self.nrad
        h = torch.arange(res, device="cuda") - res // 2
        disk = (h[None, :] ** 2 + h[:, None] ** 2 <= (res // 2) ** 2).to(F64)
        img = disk.expand(nzs, res, res).reshape(-1)
        proj = self.fp(img, 1, 0, torch.zeros(nd, dtype=F64, device="cuda"))
        calib = torch.where((proj > 0.01) & (norm > 0.01), 1.0, -1000.0).to(F64)
        data, bg = dsino[:nd] * res, dsino[nd:].clamp(min=0) * res
        for _ in range(iters):
            for s in range(nsub):
                proj = self.fp(self.conv_xy(img, 1.5), nsub, s, proj)
                q = proj + bg
                corr = torch.where(q >= float(np.float32(0.01)), data / q, -1000.0)
                img = self.update(img, *self.bp(corr, calib, nsub, s))
        return img


def exact(case, seed):
    op, e = case["op"], _Exact(case)
    if op in ("triples", "frames"):
        return None
    views = case["nseg"] * case["nang"]
    if op == "recon" and views * case["res"] ** 2 * case["nzs"] * case["iters"] > 1e9:
        return None
    s = prepare(dict(case, load=True) if op == "recon" else case, seed)
    d = lambda v: v.to(F64)  # noqa: E731
    if op == "fp":
        return e.fp(s["img"], case["nsub"], case["subset"], torch.zeros(s["out"].numel(), dtype=F64, device="cuda"))
    if op == "bp":
        return list(e.bp(d(s["corr"]), d(s["calib"]), case["nsub"], case["subset"]))
    if op == "update":
        return e.update(d(s["img"]), d(s["numer"]), d(s["denom"]))
    if op == "bilateral":
        return e.bilateral(s["img"], s["ref"], s["args"][2])
    up = lambda k: torch.from_numpy(np.array(s["data"][k])).cuda().to(F64)  # noqa: E731
    return [e.recon(up("dsino"), up("norm"), case["nsub"], case["iters"])]
