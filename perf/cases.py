"""What a user of spacetimetomography_b200 has it do, as timed cases.

Every case goes through the package's public entry points (Context, Solver,
Batch, Flow, warp, warp_vjp) on inputs made from a seed: ellipsoid phantoms
with their analytic cone-beam sinograms, smooth flow fields and smooth image
pairs.  `exact` restates each path in 64-bit torch.

Layouts are the package's: volumes (nz, ny, nx), projections (views, H, W).
"""
import math
import random

import numpy as np
import torch

import spacetimetomography_b200 as stt

DEV = "cuda:0"
F64 = torch.float64
GOLDEN = math.pi * (3.0 - math.sqrt(5.0))
CUT256 = (8, 8, 8, 45, 8, 8, 30, 20)  # the reference's ROI cut, stated at 256 voxels


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # one small projection: a script that projects a test object view by view (latency and launches count)
        dict(name="project_view_64", kind="fp", nx=64, ny=64, nz=64, W=96, H=80, views=1, dtype="f32", shift=0.0),
        # the scan of one frame at the headline size: 36 views of 512^2 of a 256^3 volume
        dict(name="project_ring_256", kind="fp", nx=256, ny=256, nz=256, W=512, H=512, views=36, dtype="f32", shift=0.0),
        # a BF16-stored volume of odd extents, off-centre, on an odd detector
        dict(name="project_odd_bf16", kind="fp", nx=187, ny=203, nz=171, W=333, H=301, views=15, dtype="bf16",
             shift=1.5),
        # the gradient of a projection loss: the exact adjoint of the projector
        dict(name="adjoint_192", kind="adjoint", nx=192, ny=176, nz=160, W=256, H=240, views=12, shift=0.0),
        # a small scan's SART call: 128 views of 128^2 of a 128^3 volume (the first of the bench's configurations)
        dict(name="sart_128", kind="sart", nx=128, ny=128, nz=128, W=128, H=128, views=128, bp="voxel", dtype="f32"),
        # SART on the largest configuration's sizes, a few views of its 720
        dict(name="sart_512", kind="sart", nx=512, ny=512, nz=512, W=1024, H=1024, views=4, bp="voxel", dtype="f32"),
        # the ray-driven form of SART at the headline size
        dict(name="sart_ray_256", kind="sart", nx=256, ny=256, nz=256, W=512, H=512, views=6, bp="ray", dtype="f32"),
        # the space-time solve: one primal-dual iteration of a short sequence at the headline size
        dict(name="solve_4d_256", kind="solve", nx=256, ny=256, nz=256, W=512, H=512, frames=3, views=36, dtype="f32"),
        # motion compensation in a differentiable program: the warp and its gradient, forward and backward
        dict(name="warp_grad_112", kind="warp", nx=112, ny=128, nz=96, motion=3.0),
        # one level of the optical flow between two frames, odd extents, a fixed number of iterations
        dict(name="flow_level_odd", kind="flow", nx=135, ny=121, nz=147, warps=2, iters=60),
        # the whole multiscale flow with the reference's parameters, which stops on its residual
        dict(name="flow_pyramid_128", kind="pyramid", nx=128, ny=128, nz=128),
        # independent reconstructions of uneven size solved side by side
        dict(name="batch_uneven", kind="batch", count=8, low=64, high=128, det=160, views=60, pick=5),
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        n = size(lo, hi)
        return {a: max(24, int(n * rng.uniform(0.85, 1.0))) for a in ("nx", "ny", "nz")}

    kind = rng.choice(["fp", "fp", "adjoint", "sart", "sart", "solve", "warp", "flow", "pyramid", "batch"])
    if kind == "fp":
        c = box(48, 256)
        m = max(c.values())
        return dict(c, kind=kind, W=int(m * rng.uniform(1.2, 2.0)), H=int(m * rng.uniform(1.0, 2.0)), views=size(1, 30),
                    dtype=rng.choice(["f32", "f32", "bf16"]), shift=rng.choice([0.0, 1.5]))
    if kind == "adjoint":
        c = box(48, 192)
        m = max(c.values())
        return dict(c, kind=kind, W=int(m * rng.uniform(1.0, 1.6)), H=int(m * rng.uniform(1.0, 1.6)), views=size(1, 12),
                    shift=rng.choice([0.0, 1.5]))
    if kind == "sart":
        bp = rng.choice(["voxel", "voxel", "ray"])
        c = box(48, 320 if bp == "voxel" else 224)
        m = max(c.values())
        return dict(c, kind=kind, W=int(m * rng.uniform(1.0, 2.0)), H=int(m * rng.uniform(1.0, 2.0)), views=size(2, 16),
                    bp=bp, dtype=rng.choice(["f32", "f32", "bf16"]))
    if kind == "solve":
        c = box(48, 192)
        m = max(c.values())
        return dict(c, kind=kind, W=int(m * rng.uniform(1.0, 2.0)), H=int(m * rng.uniform(1.0, 2.0)),
                    frames=rng.randint(1, 3), views=rng.randint(6, 24), dtype=rng.choice(["f32", "f32", "bf16"]))
    if kind == "warp":
        return dict(box(48, 112), kind=kind, motion=round(rng.uniform(0.5, 4.0), 2))
    if kind == "flow":
        return dict(box(40, 150), kind=kind, warps=rng.randint(1, 2), iters=rng.randint(20, 60))
    if kind == "pyramid":
        return dict(box(48, 104), kind=kind)
    return dict(kind=kind, count=rng.randint(3, 8), low=48, high=rng.randint(72, 128), det=rng.randint(96, 192),
                views=rng.randint(24, 60), pick=rng.randint(0, 1000))


# ---- inputs -------------------------------------------------------------------

class Scan:
    """A circular cone-beam scan: the volume fills the detector, 1 mm voxels, golden-angle views."""

    def __init__(self, dims, W, H, views, shift=0.0, first=0):
        self.dims, self.W, self.H, self.views = tuple(dims), W, H, views
        m = max(dims)
        self.sid = 600.0 if m <= 256 else 600.0 * m / 256
        self.sdd = self.sid * 5.0 / 3.0
        self.ds = 2.0 * m / W
        self.off = (shift, -shift, 0.5 * shift)
        self.angles = ((np.arange(views) + first) * GOLDEN + 0.3) % (2 * math.pi)

    def context(self):
        ctx = stt.Context(0)
        ctx.set_geometry(self.dims, (1.0, 1.0, 1.0), (self.W, self.H), self.ds, self.sid, self.sdd, self.angles,
                         self.off)
        return ctx

    def frame(self, v):
        """(R, t, centre): camera = R (voxel - centre) + t."""
        c, s = math.cos(self.angles[v]), math.sin(self.angles[v])
        R = torch.tensor([[c, 0, s], [0, 1, 0], [-s, 0, c]], dtype=F64, device=DEV)
        t = torch.tensor([-self.off[0], -self.off[2], -self.sid + self.off[1]], dtype=F64, device=DEV)
        ctr = torch.tensor([(d - 1) * 0.5 for d in self.dims], dtype=F64, device=DEV)
        return R, t, ctr

    def rays(self, v):
        """Source (3,) and unit directions (3, H*W) of view v in voxel coordinates."""
        R, t, ctr = self.frame(v)
        src = ctr + R.T @ (-t)
        i = (torch.arange(self.W, dtype=F64, device=DEV) - (self.W - 1) * 0.5) * self.ds
        j = (torch.arange(self.H, dtype=F64, device=DEV) - (self.H - 1) * 0.5) * self.ds
        cam = torch.stack([i.expand(self.H, -1), j[:, None].expand(-1, self.W),
                           torch.full((self.H, self.W), -self.sdd, dtype=F64, device=DEV)]).reshape(3, -1)
        d = R.T @ cam
        return src, d / d.norm(dim=0)


def zero_shell(v):
    """Measured objects lie inside the field of view: the outermost voxels are empty."""
    v[..., 0, :, :] = v[..., -1, :, :] = 0
    v[..., :, 0, :] = v[..., :, -1, :] = 0
    v[..., :, :, 0] = v[..., :, :, -1] = 0
    return v


def ellipsoids(dims, seed, n=10):
    r = np.random.default_rng(seed)
    d = np.asarray(dims, float)
    out = []
    for _ in range(n):
        q = np.linalg.qr(r.normal(size=(3, 3)))[0]
        out.append((r.uniform(0.25, 0.75, 3) * (d - 1), r.uniform(0.04, 0.22, 3) * d.min(), q, r.uniform(0.1, 1.0)))
    return out


def rasterize(parts, dims):
    v = torch.zeros(tuple(dims[::-1]), device=DEV)
    for c, a, q, rho in parts:
        lo = [max(0, int(c[k] - max(a) - 1)) for k in range(3)]
        hi = [min(dims[k], int(c[k] + max(a) + 2)) for k in range(3)]
        x, y, z = (torch.arange(lo[k], hi[k], device=DEV, dtype=torch.float32) - float(c[k]) for k in range(3))
        s = 0
        for k in range(3):
            u = (q[0, k] * x[None, None, :] + q[1, k] * y[None, :, None] + q[2, k] * z[:, None, None]) / a[k]
            s = s + u * u
        v[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += rho * (s <= 1.0)
    return zero_shell(v)


def sinogram(parts, scan):
    """Analytic line integrals of the ellipsoids (views, H, W)."""
    out = torch.zeros((scan.views, scan.H, scan.W), device=DEV)
    for v in range(scan.views):
        src, d = scan.rays(v)
        for c, a, q, rho in parts:
            m = torch.tensor(q.T / a[:, None], dtype=F64, device=DEV)
            o, w = m @ (src - torch.tensor(c, dtype=F64, device=DEV)), m @ d
            ww, ow = (w * w).sum(0), o @ w
            out[v] += (2.0 * rho * torch.sqrt(torch.clamp(ow * ow - ww * (o @ o - 1.0), min=0)) / ww).view(
                scan.H, scan.W).float()
    return out


def waves(dims, seed, n=6, longest=1.0, shortest=0.12, displaced=None):
    """A smooth field in about [-1, 1]: products of cosines; `displaced` moves the points it is read at."""
    r = np.random.default_rng(seed)
    m = max(dims)
    out = torch.zeros(tuple(dims[::-1]), device=DEV)
    for _ in range(n):
        f = []
        for k in range(3):
            wl = m * math.exp(r.uniform(math.log(shortest), math.log(longest)))
            x = torch.arange(dims[k], device=DEV, dtype=F64) - (0.0 if displaced is None else displaced[k])
            f.append(torch.cos(2 * math.pi * x / wl + r.uniform(0, 2 * math.pi)).float())
        out += r.uniform(0.5, 1.0) / n * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
    return out


def motion(dims, seed, amplitude):
    """A smooth inter-frame motion (3, nz, ny, nx) in voxels."""
    return torch.stack([waves(dims, seed * 31 + k, 3, 1.0, 0.4) for k in range(3)]) * amplitude


def roi_cut(dims):
    return tuple(max(1, c * min(dims) // 256) for c in CUT256)


def gmax_of(b):
    return float(b.max()) / 4.0


def dims_of(case):
    return (case["nx"], case["ny"], case["nz"])


def stored(t, dtype):
    return t.to(torch.bfloat16) if dtype == "bf16" else t


def pd_params(dims, gmax, tp=0.1, bc=0.05):
    sigma = 0.9 / 8.0
    return stt.PdParams(sigma=sigma, tau=1.0, tv_w=0.01, tp_w=tp, bc_w=bc, huber_factor=1.0 / (1.0 + sigma), gmax=gmax,
                        cut=roi_cut(dims))


def start_volume(truth, seed):
    """A reconstruction under way: the object, not yet right."""
    nz, ny, nx = truth.shape
    return truth * (0.8 + 0.2 * waves((nx, ny, nz), seed + 5))


def inputs(case, seed):
    """Everything the call is given, without the package's objects."""
    kind = case["kind"]
    if kind == "batch":
        r = random.Random(case["pick"])
        out = []
        for k in range(case["count"]):
            n = r.randint(case["low"], case["high"])
            det, views = r.randint(case["det"] // 2, case["det"]), r.randint(case["views"] // 2, case["views"])
            scan = Scan((n, n, n), det, det, views)
            parts = ellipsoids(scan.dims, seed * 101 + k)
            out.append(dict(scan=scan, vol=start_volume(rasterize(parts, scan.dims), seed + k),
                            proj=sinogram(parts, scan), seed=seed * 7 + k))
        return out
    dims = dims_of(case)
    if kind == "fp":
        scan = Scan(dims, case["W"], case["H"], case["views"], case["shift"])
        return dict(scan=scan, vol=stored(start_volume(rasterize(ellipsoids(dims, seed), dims), seed), case["dtype"]))
    if kind == "adjoint":
        scan = Scan(dims, case["W"], case["H"], case["views"], case["shift"])
        y = sinogram(ellipsoids(dims, seed), scan)
        for v in range(scan.views):  # a residual: of both signs
            y[v] *= waves((scan.W, scan.H, 1), seed * 977 + v)[0]
        return dict(scan=scan, y=y)
    if kind == "sart":
        scan = Scan(dims, case["W"], case["H"], case["views"])
        parts = ellipsoids(dims, seed)
        b = sinogram(parts, scan)
        perm = np.random.default_rng(seed).permutation(scan.views).astype(np.int32)
        return dict(scan=scan, vol=stored(start_volume(rasterize(parts, dims), seed), case["dtype"]), gmax=gmax_of(b),
                    proj=stored(b, case["dtype"]), perm=perm, cut=roi_cut(dims))
    if kind == "solve":
        F, V = case["frames"], case["views"]
        scan = Scan(dims, case["W"], case["H"], F * V)
        parts, vols, proj = ellipsoids(dims, seed), [], []
        for f in range(F):
            moved = [(c + 1.5 * f * np.sin(c / 40.0 + seed), a, q, rho) for c, a, q, rho in parts]
            vols.append(start_volume(rasterize(moved, dims), seed + f))
            one = Scan(dims, case["W"], case["H"], V, 0.0, f * V)
            proj.append(sinogram(moved, one))
        vols = torch.stack(vols + [vols[-1]])
        proj = torch.stack(proj)
        n = tuple(dims[::-1])
        st = dict(vol=vols, xbar=vols * 1.01, xprev=torch.zeros((F,) + n, device=DEV),
                  ytv=torch.stack([torch.stack([waves(dims, seed + 50 + 3 * f + k) for k in range(3)]) for f in
                                   range(F)]) * 0.01,
                  ytp=torch.stack([waves(dims, seed + 70 + f) for f in range(F)]) * 0.05,
                  ybc=torch.stack([waves(dims, seed + 80 + f) for f in range(F)]) * 0.04,
                  flow=torch.stack([motion(dims, seed + 90 + f, 2.0) for f in range(F)]))
        for k in ("vol", "xbar", "xprev"):
            st[k] = stored(st[k], case["dtype"])
        st["proj"] = stored(proj, case["dtype"])
        return dict(scan=scan, state=st, gmax=gmax_of(proj))
    if kind == "warp":
        return dict(flow=motion(dims, seed, case["motion"]), src=waves(dims, seed + 1, 8, 0.5, 0.06),
                    out_bar=waves(dims, seed + 2, 8, 0.5, 0.06))
    # an image pair: textured frames, the second displaced by a voxel or so
    r = np.random.default_rng(seed)
    u = r.uniform(0.6, 1.4, 3) * r.choice([-1.0, 1.0], 3)
    return dict(i1=0.5 + waves(dims, seed, 8, 0.5, 0.08), i2=0.5 + waves(dims, seed, 8, 0.5, 0.08, u),
                cut=roi_cut(dims)[:6])


# ---- preparation and one pass ----------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = inputs(case, seed)
    if kind == "batch":
        inst = []
        for d in s:
            gmax = gmax_of(d["proj"])
            inst.append(dict(ctx=d["scan"].context(), vol=d["vol"], proj=d["proj"], bp_mode=0, alpha=0.3,
                             pd=pd_params(d["scan"].dims, gmax, 0.0, 0.0), seed=d["seed"],
                             roi_cut=roi_cut(d["scan"].dims)))
        return dict(kind=kind, inst=inst, batch=stt.Batch(inst, mode=stt.SOLVE_GRAPH))
    dims = dims_of(case)
    shape = tuple(dims[::-1])
    s["kind"] = kind
    if kind in ("fp", "adjoint", "sart", "solve"):
        s["ctx"] = s["scan"].context()
    if kind == "fp":
        s["proj"] = torch.zeros((s["scan"].views, s["scan"].H, s["scan"].W), device=DEV)
    elif kind == "adjoint":
        s["vol_bar"] = torch.zeros(shape, device=DEV)
    elif kind == "sart":
        s["raylen"] = torch.zeros((s["scan"].H, s["scan"].W), device=DEV)
        s["mode"] = 1 if case["bp"] == "ray" else 0
    elif kind == "solve":
        s["solver"] = stt.Solver(s["ctx"], s["state"], case["frames"], case["views"], pd_params(dims, s["gmax"]),
                                 alpha=0.3, bp_mode=0, roi_cut=roi_cut(dims), seed=seed, mode=stt.SOLVE_GRAPH,
                                 autotune=True, storage=case["dtype"])
    elif kind == "warp":
        s["out"] = torch.empty(shape, device=DEV)
        s["src_bar"] = torch.empty(shape, device=DEV)
        s["flow_bar"] = torch.empty((3,) + shape, device=DEV)
    else:
        s["V"] = torch.zeros((3,) + shape, device=DEV)
        s["Y"] = torch.zeros((10,) + shape, device=DEV)
        p = dict(cut=s["cut"])
        if kind == "flow":
            p.update(tol=0.0, max_iter=case["iters"] - 1, n_warps=case["warps"], scales=1)
        s["flow"] = stt.Flow(shape, stt.FlowParams(**p))
    return s


def run(s):
    kind = s["kind"]
    if kind == "fp":
        return s["ctx"].fp_typed(s["vol"], s["proj"])
    if kind == "adjoint":
        s["vol_bar"].zero_()
        return s["ctx"].fp_vjp(s["y"], s["vol_bar"])
    if kind == "sart":
        s["ctx"].sart_sweep(s["vol"], s["proj"], s["perm"], 0.3, s["gmax"], s["mode"], s["raylen"], roi_cut=s["cut"])
        return {"vol": s["vol"], "raylen": s["raylen"]}
    if kind == "solve":
        s["solver"].iterate(1)
        return {k: s["state"][k] for k in ("vol", "xbar", "xprev", "ytv", "ytp", "ybc")}
    if kind == "warp":
        s["src_bar"].zero_()
        s["flow_bar"].zero_()
        stt.warp(s["flow"], s["src"], -1.0, out=s["out"])
        stt.warp_vjp(s["flow"], s["src"], -1.0, s["out_bar"], s["src_bar"], s["flow_bar"])
        return {"out": s["out"], "src_bar": s["src_bar"], "flow_bar": s["flow_bar"]}
    if kind == "flow":
        s["V"].zero_()
        s["Y"].zero_()
        s["flow"].level(s["i1"], s["i2"], s["V"], s["Y"], s["cut"])
        return {"V": s["V"], "Y": s["Y"]}
    if kind == "pyramid":
        s["V"].zero_()
        return s["flow"].multiscale(s["i1"], s["i2"], s["V"])
    s["batch"].iterate(1)
    return [d["vol"] for d in s["inst"]]


def work(case):
    """Inputs read once and outputs written once; operations of the samples, taps and updates themselves."""
    kind = case["kind"]
    if kind == "batch":
        r = random.Random(case["pick"])
        b = f = 0
        for _ in range(case["count"]):
            n = r.randint(case["low"], case["high"])
            det, views = r.randint(case["det"] // 2, case["det"]), r.randint(case["views"] // 2, case["views"])
            smp = _samples((n, n, n), det, det)
            b += 4 * (14 * n ** 3 + views * det * det)
            f += views * (28 * smp + 50 * n ** 3) + 60 * n ** 3
        return {"bytes": b, "flops": f}
    dims = dims_of(case)
    n = dims[0] * dims[1] * dims[2]
    if kind in ("fp", "adjoint", "sart", "solve"):
        pix, smp = case["W"] * case["H"], _samples(dims, case["W"], case["H"])
    es = 2 if case.get("dtype") == "bf16" else 4
    if kind == "fp":
        return {"bytes": es * n + 4 * case["views"] * pix, "flops": 28 * case["views"] * smp}
    if kind == "adjoint":
        return {"bytes": 4 * n + 4 * case["views"] * pix, "flops": 28 * case["views"] * smp}
    if kind == "sart":
        per = 28 * smp + (50 * n if case["bp"] == "voxel" else 50 * smp)
        return {"bytes": 2 * es * n + (es * case["views"] + 8) * pix, "flops": case["views"] * per}
    if kind == "solve":
        F, V = case["frames"], case["views"]
        return {"bytes": F * ((5 * es + 4 * (2 * 5 + 3)) * n + es * V * pix),
                "flops": F * (V * (28 * smp + 50 * n) + 2 * 4 * 90 * n + 60 * n)}
    if kind == "warp":
        return {"bytes": 4 * 10 * n, "flops": (4 * 90 + 4 * 250) * n}
    if kind == "flow":
        it = case["warps"] * case["iters"]
        return {"bytes": 4 * n * (2 + 2 * 13 + it * (2 * 13 + 4)), "flops": n * it * 120}
    # the pyramid: some 450 iterations of its three warps on the full size, as many on 0.65 of it, 650 on 0.42
    return {"bytes": 4 * n * 30 * 620, "flops": n * 120 * 620}


def _samples(dims, W, H):
    """Samples of one view: the volume's share of the rays at the isocentre, one per sqrt(3) mm."""
    m = max(dims)
    ds = 2.0 * m / W
    return int(dims[0] * dims[1] * dims[2] * (5.0 / 3.0 / ds) ** 2 / math.sqrt(3.0) * min(1.0, H * ds * 0.6 / dims[1]))


# ---- 64-bit restatements --------------------------------------------------------------

class Marcher:
    """The samples of one view's rays: positions tnear + k sd inside the box, the entry sample twice, and the march's
    restart before the entry where a falling coordinate enters below 0.5."""

    def __init__(self, scan, v):
        src, d = scan.rays(v)
        self.sd = math.sqrt(3.0)
        hi = torch.tensor([n - 1.0 for n in scan.dims], dtype=F64, device=DEV)[:, None]
        t1, t2 = -src[:, None] / d, (hi - src[:, None]) / d
        tn = torch.clamp(torch.minimum(t1, t2).amax(0), min=0.0)
        tf = torch.maximum(t1, t2).amin(0)
        self.hit = tn < tf
        self.at = torch.nonzero(self.hit).view(-1)
        self.src, self.d, self.tn, self.tf = src, d[:, self.at], tn[self.at], tf[self.at]
        self.length = torch.where(self.hit, tf - tn, torch.zeros_like(tf))
        self.n = self.hit.numel()
        self.dims = scan.dims
        self.hi = hi
        p = self.src[:, None] + self.d * self.tn
        back = (0.5 - self.src[:, None]) / self.d
        back = torch.where((self.d < 0) & (p < 0.5), back, torch.full_like(back, math.inf)).amin(0)
        self.k0 = torch.where(back < self.tn, torch.ceil((back - self.tn) / self.sd), torch.zeros_like(back))

    def batches(self, most=3_000_000):
        """(indices into the hit rays, positions (3, k, rays), live (k, rays)); the entry sample comes first."""
        if not self.at.numel():
            return
        yield (self.src[:, None] + self.d * self.tn)[:, None], torch.ones_like(self.tn, dtype=torch.bool)[None]
        last = int(torch.ceil((self.tf - self.tn) / self.sd - self.k0).max())
        step = max(1, most // self.at.numel())
        for m in range(0, last + 1, step):
            k = self.k0 + torch.arange(m, min(m + step, last + 1), device=DEV, dtype=F64)[:, None]
            t = self.tn + k * self.sd
            yield self.src[:, None, None] + self.d[:, None] * t, t < self.tf

    def corners(self, p):
        """Flat index of the base voxel, the strides, and the 8 (offset, weight) pairs of the positions."""
        nx, ny, nz = self.dims
        q = torch.minimum(torch.clamp(p, min=0.0), self.hi.view(3, 1, 1))
        b = torch.minimum(q.floor(), self.hi.view(3, 1, 1) - 1)
        f = q - b
        i = b.long()
        base = i[0] + nx * (i[1] + ny * i[2])
        return base, [(dx + nx * (dy + ny * dz), (f[0] if dx else 1 - f[0]) * (f[1] if dy else 1 - f[1]) *
                       (f[2] if dz else 1 - f[2])) for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]

    def project(self, vol):
        flat, out = vol.reshape(-1), torch.zeros(self.n, dtype=F64, device=DEV)
        acc = torch.zeros(self.at.numel(), dtype=F64, device=DEV)
        for p, live in self.batches():
            base, taps = self.corners(p)
            v = sum(w * flat[base + o] for o, w in taps)
            acc += torch.where(live, v, torch.zeros_like(v)).sum(0)
        out[self.at] = acc * self.sd
        return out

    def scatter(self, y, scale, into, weights=None):
        """into += scale y w over every sample's corners; weights += w."""
        c = y.reshape(-1)[self.at] * scale
        for p, live in self.batches():
            base, taps = self.corners(p)
            for o, w in taps:
                w = torch.where(live, w, torch.zeros_like(w))
                into.index_add_(0, (base + o).view(-1), (c * w).reshape(-1))
                if weights is not None:
                    weights.index_add_(0, (base + o).view(-1), w.reshape(-1))


def cr_weights(d):
    return [0.5 * (-d + 2 * d ** 2 - d ** 3), 1 + 0.5 * (-5 * d ** 2 + 3 * d ** 3), 0.5 * (d + 4 * d ** 2 - 3 * d ** 3),
            0.5 * (-d ** 2 + d ** 3)]


def bp_voxel(scan, v, corr, vol, alpha, gmax):
    nx, ny, nz = scan.dims
    R, t, ctr = scan.frame(v)
    c = corr.reshape(-1)
    x = torch.arange(nx, dtype=F64, device=DEV) - ctr[0]
    y = (torch.arange(ny, dtype=F64, device=DEV) - ctr[1])[:, None]
    for z0 in range(0, nz, 64):
        z = (torch.arange(z0, min(nz, z0 + 64), dtype=F64, device=DEV) - ctr[2])[:, None, None]
        depth = -(R[2, 0] * x + R[2, 2] * z + t[2])
        ux = (scan.W - 1) * 0.5 + (R[0, 0] * x + R[0, 2] * z + t[0]) / depth * (scan.sdd / scan.ds)
        uy = (scan.H - 1) * 0.5 + (y + t[1]) / depth * (scan.sdd / scan.ds)
        ux = ux.expand_as(uy)
        ok = (ux >= 2) & (ux < scan.W - 2) & (uy >= 2) & (uy < scan.H - 2)
        px, py = ux[ok].floor(), uy[ok].floor()
        wx, wy = cr_weights(ux[ok] - px), cr_weights(uy[ok] - py)
        base = (py.long() - 1) * scan.W + px.long() - 1
        val = sum(wx[a] * sum(wy[b] * c[base + (a + b * scan.W)] for b in range(4)) for a in range(4))
        part = vol[z0:z0 + 64]
        part[ok] = torch.clamp(part[ok] + alpha * val, 0.0, gmax)


def roi_mask(dims, cut):
    nx, ny, nz = dims
    i = torch.arange(nx, device=DEV)[None, None, :]
    j = torch.arange(ny, device=DEV)[None, :, None]
    k = torch.arange(nz, device=DEV)[:, None, None]
    a, b = cut[6], cut[7]
    out = ((i < a) & ((k < b) | (k > nz - b))) | ((i > nx - a) & ((k < b) | (k > nz - b)))
    out = out | ((k < a) & ((i < b) | (i > nx - b))) | ((k > nz - a) & ((i < b) | (i > nx - b)))
    out = out | (i < cut[0]) | (i > nx - cut[1]) | (j < cut[2]) | (j > ny - 7) | (k < cut[4]) | (k > nz - cut[5])
    return (~out).to(F64)


def roi_box(dims, cut):
    nx, ny, nz = dims
    i = torch.arange(nx, device=DEV)[None, None, :]
    j = torch.arange(ny, device=DEV)[None, :, None]
    k = torch.arange(nz, device=DEV)[:, None, None]
    return (i >= cut[0]) & (i <= nx - cut[1]) & (j >= cut[2]) & (j <= ny - cut[3]) & (k >= cut[4]) & (k <= nz - cut[5])


def sart(scan, views, vol, proj, alpha, gmax, ray, raylen, cut):
    """One SART call, in place on vol; views: (index in the scan, index in proj) in order."""
    n = vol.numel()
    for v, k in views:
        m = Marcher(scan, v)
        ax = m.project(vol)
        if ray:
            L = m.length
        else:
            raylen[m.hit] = m.length[m.hit]
            L = raylen
        corr = (proj[k].reshape(-1).to(F64) - ax) / (L + 1.0)
        if ray:
            c, w = torch.zeros(n, dtype=F64, device=DEV), torch.zeros(n, dtype=F64, device=DEV)
            m.scatter(corr, 1.0, c, w)
            new = torch.clamp(vol.view(-1) + c / w, 0.0, gmax)
            vol.view(-1).copy_(torch.where(w > 0, new, torch.zeros_like(new)))
        else:
            bp_voxel(scan, v, corr, vol, alpha, gmax)
    if ray:
        raylen.zero_()
    if cut is not None:
        vol *= roi_mask(scan.dims, cut)


def view_order(seed, iteration, frames, f, views):
    """SplitMix64 and Fisher-Yates: the solver's documented view order."""
    mask = (1 << 64) - 1
    s = (seed + 0x9E3779B97F4A7C15 * (iteration * frames + f + 1)) & mask
    p = list(range(views))
    for i in range(views - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        p[i], p[j] = p[j], p[i]
    return p


def sample(img, g):
    """Clamped tricubic samples of img (nz, ny, nx) at grid positions g (3 tensors in [1, dim-2])."""
    nz, ny, nx = img.shape
    flat, ax = img.reshape(-1), []
    for q, n, stride in zip(g, (nx, ny, nz), (1, nx, nx * ny)):
        i = q.detach().floor().long()
        ax.append(([(i - 1) * stride, i * stride, torch.clamp(i + 1, max=n - 1) * stride,
                    torch.clamp(i + 2, max=n - 1) * stride], cr_weights(q - i)))
    val, corners, at = 0.0, [], []
    for c in range(4):
        for b in range(4):
            row = ax[1][0][b] + ax[2][0][c]
            tap = [flat[row + ax[0][0][a]] for a in range(4)]
            val = val + ax[2][1][c] * ax[1][1][b] * sum(ax[0][1][a] * tap[a] for a in range(4))
            if b in (1, 2) and c in (1, 2):
                corners += [tap[1].detach(), tap[2].detach()]
                at += [row + ax[0][0][1], row + ax[0][0][2]]
    corners, at = torch.stack(corners), torch.stack(at)
    (mx, imx), (mn, imn) = corners.max(0), corners.min(0)
    top, low = flat[at.gather(0, imx[None])[0]], flat[at.gather(0, imn[None])[0]]
    return torch.where(val > mx, top, torch.where(val < mn, low, val))


def warp(flow, src, dt, z0=0, z1=None):
    """The semi-Lagrangian warp of planes [z0, z1)."""
    nz, ny, nx = src.shape
    z1 = nz if z1 is None else z1
    dims = (nx, ny, nz)
    p = torch.meshgrid(*[torch.arange(a, b, dtype=F64, device=DEV) + 0.5 for a, b in ((z0, z1), (0, ny), (0, nx))],
                       indexing="ij")[::-1]

    def grid(q):
        return [torch.clamp(q[a] - 0.5, 1.0, dims[a] - 2.0) for a in range(3)]

    c = [torch.clamp((p[a] - 0.5).long(), 1, dims[a] - 2) for a in range(3)]
    h = -dt
    p2 = [p[a] + h * flow[a][c[2], c[1], c[0]] for a in range(3)]
    g2 = grid(p2)
    q = [p2[a] + 0.5 * (p[a] - (p2[a] - h * sample(flow[a], g2))) for a in range(3)]
    return sample(src, grid(q))


def warp_all(flow, src, dt):
    nz = src.shape[0]
    flow, src = flow.to(F64), src.to(F64)
    return torch.cat([warp(flow, src, dt, z, min(nz, z + 48)) for z in range(0, nz, 48)])


def shifted(x, axis, by):
    """x at the neighbour `by` along an axis (wrapping; callers mask the border)."""
    return torch.roll(x, -by, axis)


def pd_iteration(scan, st, F, V, gmax, dims, seed, tp, bc):
    """One space-time primal-dual iteration on 64-bit state, in place."""
    sigma, tau, tv, cut = 0.9 / 8.0, 1.0, 0.01, roi_cut(dims)
    hf = 1.0 / (1.0 + sigma)
    inner = roi_box(dims, cut).clone()
    for a in range(3):
        inner.select(a, 0).fill_(False)
        inner.select(a, -1).fill_(False)
    for f in range(F):
        x, x1 = st["xbar"][f], st["xbar"][f + 1]
        bw = warp_all(st["flow"][f], x1, -1.0)
        ytp = st["ytp"][f] + sigma * (x1 - x)
        ybc = st["ybc"][f] + sigma * (bw - x)
        for k, a in enumerate((2, 1, 0)):
            y = torch.clamp(st["ytv"][f][k] + sigma * (shifted(x, a, 1) - x) * hf, -tv, tv)
            st["ytv"][f][k] = torch.where(inner, y, st["ytv"][f][k])
        st["ytp"][f] = torch.where(inner, ytp * tp / (tp + 2 * sigma), ytp)
        st["ybc"][f] = torch.where(inner, torch.clamp(ybc, -bc, bc), ybc)
    for f in range(F):
        v = st["vol"][f].clone()
        st["xprev"][f] = v
        if f == 0:
            v = v + tau * (st["ytp"][f] + st["ybc"][f])
        else:
            v = v - tau * (st["ytp"][f - 1] - st["ytp"][f])
            v = v - tau * (warp_all(st["flow"][f - 1], st["ybc"][f - 1], 1.0) - st["ybc"][f])
        div = sum(st["ytv"][f][k] - shifted(st["ytv"][f][k], a, -1) for k, a in enumerate((2, 1, 0)))
        v = torch.where(inner, torch.clamp(v + tau * div, 0.0, gmax), v)
        order = view_order(seed, 0, F, f, V)
        raylen = torch.zeros(scan.W * scan.H, dtype=F64, device=DEV)
        sart(scan, [(f * V + k, k) for k in order], v, st["proj"][f], 0.3, gmax, False, raylen, cut)
        st["vol"][f] = v
        st["xbar"][f] = torch.where(roi_box(dims, cut), 2 * v - st["xprev"][f], st["xbar"][f])


def flow_level(i1, i2, cut, warps, iters):
    """One level of the Huber-regularised flow from zero, a fixed number of iterations."""
    nz, ny, nx = i1.shape
    lam, sigma1 = 1.2, 1.0 / 3.0
    hf = 1.0 / (1.0 + sigma1 * 1.0 / lam)
    i1, i2 = i1.to(F64), i2.to(F64)
    V = torch.zeros((3,) + i1.shape, dtype=F64, device=DEV)
    y = torch.zeros((10,) + i1.shape, dtype=F64, device=DEV)
    kx = torch.zeros_like(y)
    roi = torch.zeros(i1.shape, dtype=torch.bool, device=DEV)
    roi[cut[4]:nz - cut[5], cut[2]:ny - cut[3], cut[0]:nx - cut[1]] = True

    def down(q, a):  # backward difference: first q, last minus the one below
        out = q - shifted(q, a, -1)
        out.select(a, 0).copy_(q.select(a, 0))
        out.select(a, -1).copy_(-q.select(a, -2))
        return out

    def up(q, a):
        out = shifted(q, a, 1) - q
        out.select(a, -1).zero_()
        return out

    for _ in range(warps):
        w = warp_all(V, i2, -1.0)
        g = []
        for a in (2, 1, 0):
            n = w.shape[a]
            idx = torch.arange(n, device=DEV)
            d = (w.index_select(a, torch.clamp(idx + 1, max=n - 1)) - w.index_select(a, torch.clamp(idx - 1, min=0))) / 2
            g.append(torch.where(roi, d, torch.zeros_like(d)))
        ut = torch.where(roi, w - i1 - sum(g[c] * V[c] for c in range(3)), torch.zeros_like(w))
        tau = [1.0 / (4.0 + q.abs()) for q in g]
        sig2 = 1.0 / (g[0].abs() + g[1].abs() + g[2].abs())
        for _ in range(iters):
            for c in range(3):
                kt = -down(y[3 * c], 2) - down(y[3 * c + 1], 1) - down(y[3 * c + 2], 0) + g[c] * y[9]
                V[c] = torch.where(roi, V[c] - tau[c] * kt, V[c])
            for c in range(3):
                t = []
                for k, a in enumerate((2, 1, 0)):
                    kn = up(V[c], a)
                    t.append((y[3 * c + k] + sigma1 * (2 * kn - kx[3 * c + k])) * hf)
                    kx[3 * c + k] = kn
                dv = torch.clamp(torch.sqrt(t[0] ** 2 + t[1] ** 2 + t[2] ** 2) / lam, min=1.0)
                for k in range(3):
                    y[3 * c + k] = t[k] / dv
            k4 = sum(g[c] * V[c] for c in range(3))
            q = y[9] + sig2 * (2 * k4 - kx[9] + ut)
            y[9] = torch.where(q.isnan(), torch.ones_like(q), torch.clamp(q, -1.0, 1.0))
            kx[9] = k4
    return V, torch.where(roi, y, torch.zeros_like(y))


def exact(case, seed):
    kind = case["kind"]
    if kind == "pyramid":  # when a warp stops hangs on a residual summed in 32 bits: no such value
        return None
    s = inputs(case, seed)
    if kind == "fp":
        vol = s["vol"].to(F64)
        return torch.stack([Marcher(s["scan"], v).project(vol).view(s["scan"].H, s["scan"].W) for v in
                            range(s["scan"].views)])
    if kind == "adjoint":
        out = torch.zeros(s["scan"].dims[::-1], dtype=F64, device=DEV)
        for v in range(s["scan"].views):
            m = Marcher(s["scan"], v)
            m.scatter(s["y"][v].to(F64), m.sd, out.view(-1))
        return out
    if kind == "sart":
        vol = s["vol"].to(F64)
        raylen = torch.zeros(case["W"] * case["H"], dtype=F64, device=DEV)
        sart(s["scan"], [(int(k), int(k)) for k in s["perm"]], vol, s["proj"], 0.3, s["gmax"], case["bp"] == "ray",
             raylen, s["cut"])
        return {"vol": vol, "raylen": raylen.view(case["H"], case["W"])}
    if kind == "solve":
        st = {k: v if k in ("proj", "flow") else v.to(F64) for k, v in s["state"].items()}
        pd_iteration(s["scan"], st, case["frames"], case["views"], s["gmax"], dims_of(case), seed, 0.1, 0.05)
        return {k: st[k] for k in ("vol", "xbar", "xprev", "ytv", "ytp", "ybc")}
    if kind == "warp":
        flow, src = s["flow"].to(F64).requires_grad_(), s["src"].to(F64).requires_grad_()
        out = warp(flow, src, -1.0)
        out.backward(s["out_bar"].to(F64))
        return {"out": out.detach(), "src_bar": src.grad, "flow_bar": flow.grad}
    if kind == "flow":
        V, Y = flow_level(s["i1"], s["i2"], s["cut"], case["warps"], case["iters"])
        return {"V": V, "Y": Y}
    out = []
    for d in s:
        scan, n = d["scan"], d["vol"].shape
        vol = d["vol"].to(F64)
        z = torch.zeros((1,) + tuple(n), dtype=F64, device=DEV)
        st = dict(vol=torch.stack([vol, vol]), xbar=torch.stack([vol, vol]), xprev=z.clone(),
                  ytv=torch.zeros((1, 3) + tuple(n), dtype=F64, device=DEV), ytp=z.clone(), ybc=z.clone(),
                  flow=torch.zeros((1, 3) + tuple(n), dtype=F64, device=DEV), proj=d["proj"][None])
        pd_iteration(scan, st, 1, scan.views, gmax_of(d["proj"]), scan.dims, d["seed"], 0.0, 0.0)
        out.append(st["vol"][0])
    return out
