"""The work that is timed: the projector pair, ordered-subset EM, penalized
gradients and FBP through the public entry points, over the sizes, angles,
pitches and storage types that users of the framework run.

``listed()`` are fixed cases, ``draw(rng)`` gives more of the same ranges.
``exact(case, seed)`` computes a case's outputs in 64 bits with plain torch
from the definition of the operators (separable footprints: box overlaps of
voxels and bins along u0 and u1), independently of the library.  Inputs come
from the seed alone: ellipsoid phantoms, and Poisson counts whose means are
the ellipsoids' analytic line integrals.
"""
import math

import numpy as np
import torch

from petl_b200 import Geometry, autograd, ops, penalized, recon

DEV = "cuda"
# the PET/X scanner's two panel pairs (psi, D, L, H) and bin pitch; its slope
# limits are the defaults of add_planogram
PETX = ((0.0, 101.0, 251.52, 156.72), (90.0, 266.6, 125.12, 156.72))
PETX_PITCH = 1.6
RD = (2.0, 0.01)              # relative differences: gamma, beta
TV = (1e-4, 0.01, 1.0, 26)    # Huber TV: delta, beta, p, neighbours
ELLIPSOIDS = 10


# ----------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------
def _panel(kind, n, T, D, name=None, psi=0.0, **more):
    """A dual-panel case: an n x n x n/2 volume at pitch T between panels of
    n T / 2 mm at a distance of D mm (v0 up to 0.5, v1 up to 0.25)."""
    c = dict(kind=kind, psi=psi, D=D, L=n * T / 2, H=n * T / 2, T=T, v_m0=0.5, v_m1=0.25, nx=n, ny=n, nz=n // 2, w=T,
             h=T, counts=5e6)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the projector pair at the size the framework quotes its throughput on:
        # planogram (65, 129, 128, 256)
        _panel("project", 256, 1.0, 256.0, "project_256", counts=5e7),
        _panel("backproject", 256, 1.0, 256.0, "backproject_256", counts=5e7),
        # served reconstructions: the smallest volume, where each launch counts
        # (one iteration of 8 subsets), and an ordinary one (4 subsets)
        _panel("osem", 64, 1.5, 250.0, "osem_64", subsets=8, counts=1e5),
        _panel("osem", 192, 1.5, 200.0, "osem_192", subsets=4),
        # planogram-sized arrays stored in bfloat16, one iteration of 8 subsets
        _panel("osem_bf16", 256, 1.0, 256.0, "osem_bf16_256", subsets=8, counts=5e7),
        # differentiable penalized reconstruction: objective and gradient of a
        # batch of 4 volumes through autograd
        _panel("penalized", 128, 2.0, 256.0, "penalized_128", batch=4, counts=1e6),
        # rebinning, ramp filter and 2-D backprojection of a full-size scan
        _panel("fbp", 256, 1.0, 256.0, "fbp_256", counts=5e7),
        # the PET/X scanner: both panel pairs into 0.5 mm voxels (a bin is 1.6
        # mm), analytically and by one ordered-subset step
        dict(name="fbp_petx", kind="fbp", petx=True, nx=120, ny=120, nz=120, w=0.5, h=0.5, counts=2e7),
        dict(name="step_petx", kind="step", petx=True, nx=120, ny=120, nz=120, w=0.5, h=0.5, subsets=8, counts=2e7),
        # a rotated panel pair: forward, and backward in both forms (the
        # reference's weights in OSEM, the exact transpose in autograd)
        _panel("project", 256, 1.0, 256.0, "project_psi30_256", psi=30.0, counts=5e7),
        _panel("step", 192, 1.5, 250.0, "step_psi30_192", psi=30.0, subsets=4),
        # ragged sizes, planogram rows that are no multiple of 16 bytes and an
        # off-centre volume, psi = 90: forward and gradient through autograd
        dict(name="vjp_ragged", kind="vjp", psi=90.0, D=230.0, L=141.0, H=129.0, T=1.5, v_m0=0.45, v_m1=0.2, nx=150,
             ny=141, nz=75, w=1.5, h=1.5, ox=3.0, oy=-4.5, oz=1.5, counts=5e6),
    ]


def draw(rng):
    kind = rng.choice(["project", "backproject", "osem", "osem", "osem_bf16", "penalized", "fbp", "step", "step", "vjp"])
    counts = math.exp(rng.uniform(math.log(1e5), math.log(5e7)))
    if kind in ("fbp", "step") and rng.random() < 0.35:  # PET/X, other fields of view
        n = int(round(math.exp(rng.uniform(math.log(48), math.log(120)))))
        nz = int(round(n * rng.uniform(0.5, 1.0)))
        w = round(rng.uniform(0.5, 1.6), 2)
        return dict(kind=kind, petx=True, nx=n, ny=n, nz=nz, w=w, h=rng.choice([w, 1.6]), subsets=8, counts=counts)
    # BF16 storage takes panels at psi = 0 only
    psi = 0.0 if kind == "osem_bf16" else rng.choice([0.0, 0.0, 90.0, round(rng.uniform(-80.0, 170.0), 1)])
    axis = psi in (0.0, 90.0)
    top = 256 if axis and kind not in ("penalized", "osem") else 192 if kind != "penalized" else 128
    n = int(round(math.exp(rng.uniform(math.log(48), math.log(top)))))
    if kind == "osem_bf16":
        n = min(top, max(64, (n + 7) // 8 * 8))  # rows of whole 16-byte granules
    T = round(rng.uniform(1.0, 2.0), 2)
    D = max(round(rng.uniform(200.0, 300.0), 1), n * T * 0.8)
    c = _panel(kind, n, T, D, psi=psi, counts=counts)
    if kind not in ("osem_bf16",):  # ragged volumes and panels
        c.update(ny=max(32, n - rng.randrange(0, n // 4)), nz=max(16, n // 2 - rng.randrange(0, n // 8)))
        c["H"] = round(c["H"] * rng.uniform(0.8, 1.2), 2)
    if kind in ("osem", "osem_bf16", "step"):
        c["subsets"] = rng.choice([4, 8])
    if kind == "backproject":
        c["adjoint"] = rng.random() < 0.4
    if kind == "penalized":
        c["batch"] = rng.choice([1, 2, 4])
    return c


# ----------------------------------------------------------------------------
# geometry (float32 values as the planogram set-up rounds them)
# ----------------------------------------------------------------------------
def _planogram_args(c):
    if c.get("petx"):
        return [(p, D, L, H, PETX_PITCH, 1.0, min(1.0, (H - 1.5 * PETX_PITCH) / D)) for p, D, L, H in PETX]
    return [(c["psi"], c["D"], c["L"], c["H"], c["T"], c["v_m0"], c["v_m1"])]


def _volume_args(c):
    return (c["nx"], c["ny"], c["nz"], c["w"], c["h"], c.get("ox", 0.0), c.get("oy", 0.0), c.get("oz", 0.0))


def _geometries(c):
    return [Geometry(*a, volume=_volume_args(c)) for a in _planogram_args(c)]


class _Scan:
    """One planogram and volume as numbers: double values of the float32
    geometry, and the float32 visibility decisions."""

    def __init__(self, args, vol):
        f4 = np.float32
        psi, D, L, H, T, m0, m1 = (float(f4(a)) for a in args)
        psi = float(f4(psi * math.pi / 180.0))
        self.R, self.L, self.H = float(f4(0.5 * D)), float(f4(0.5 * L)), float(f4(0.5 * H))
        m1 = min(float(f4(f4(self.H) / f4(self.R))), m1)
        self.Tu, tv0 = T, float(f4(f4(T) / f4(self.R)))
        self.m0, self.Tv1 = m0, tv0
        self.NU0 = 2 * int(f4(f4(f4(self.L) + f4(f4(self.R) * f4(m0))) / f4(T)))
        self.NU1 = 2 * int(f4(f4(self.H) / f4(T)))
        self.NV0 = 2 * int(f4(f4(m0) / f4(tv0))) + 1
        self.NV1 = 2 * int(f4(f4(m1) / f4(self.Tv1))) + 1
        self.Tv0 = float(f4(m0 * 2.0 / self.NV0))
        start = lambda T_, n: float(f4(float(f4(f4(-T_) * f4(n - 1))) / 2.0))  # noqa: E731
        self.u0_0, self.u1_0 = start(T, self.NU0), start(T, self.NU1)
        self.v0_0, self.v1_0 = start(self.Tv0, self.NV0), start(self.Tv1, self.NV1)
        self.cos, self.sin = float(f4(math.cos(psi))), float(f4(math.sin(psi)))
        nx, ny, nz, w, h, ox, oy, oz = vol
        self.nx, self.ny, self.nz, self.Tx, self.Tz = nx, ny, nz, float(f4(w)), float(f4(h))
        org = lambda n, t, o: float(f4(-0.5 * (n - 1) * t + float(f4(o))))  # noqa: E731
        self.x0, self.y0, self.z0 = org(nx, self.Tx, ox), org(ny, self.Tx, oy), org(nz, self.Tz, oz)
        if psi != 0.0 and abs(self.cos) < 1e-6:
            self.cos = 0.0
        v0, v1 = self.at32(self.NV0, self.Tv0, self.v0_0), self.at32(self.NV1, self.Tv1, self.v1_0)
        u0, u1 = self.at32(self.NU0, T, self.u0_0), self.at32(self.NU1, T, self.u1_0)
        half = f4(0.5) * f4(T)
        lim0 = (self.R * np.abs(v0).astype(np.float64) + self.L).astype(f4)
        lim1 = (-self.R * np.abs(v1).astype(np.float64) + self.H).astype(f4)
        self.vis0 = ~((np.abs(u0) - half)[None, :] > lim0[:, None])   # [v0][u0]
        self.vis1 = ~((np.abs(u1) - half)[None, :] > lim1[:, None])   # [v1][u1]
        self.v1f, self.lim1, self.half = v1, lim1, half
        # driving axis of each view, and the corner pair of the voxel's extent
        vd = v0.astype(np.float64)
        self.rxf = -(vd * self.cos + self.sin).astype(f4)
        self.ryf = -(vd * self.sin - self.cos).astype(f4)

    @staticmethod
    def at32(n, T, start):
        return (np.arange(n, dtype=np.float64) * T + start).astype(np.float32)

    @property
    def shape(self):
        return (self.NV1, self.NV0, self.NU1, self.NU0)

    @property
    def vol_shape(self):
        return (self.nz, self.ny, self.nx)

    def v(self, n, T, start, dt=torch.float64):
        return (torch.arange(n, device=DEV, dtype=torch.float64) * T + start).to(dt)


def _scans(c):
    return [_Scan(a, _volume_args(c)) for a in _planogram_args(c)]


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _ellipsoids(c, seed):
    """Centres, radii and activities of seeded ellipsoids inside the volume."""
    rng = np.random.default_rng(seed)
    ext = np.array([c["nx"] * c["w"], c["ny"] * c["w"], c["nz"] * c["h"]]) * 0.5
    off = np.array([c.get("ox", 0.0), c.get("oy", 0.0), c.get("oz", 0.0)])
    out = []
    for _ in range(ELLIPSOIDS):
        r = ext * rng.uniform(0.06, 0.45, 3)
        out.append((off + rng.uniform(-1, 1, 3) * (ext - r) * 0.95, r, float(rng.uniform(0.1, 1.0))))
    return out


def _phantom(c, s, seed, background=0.01):
    """The ellipsoids on the voxel grid, with a uniform background."""
    x, y, z = s.v(s.nx, s.Tx, s.x0), s.v(s.ny, s.Tx, s.y0), s.v(s.nz, s.Tz, s.z0)
    f = torch.full(s.vol_shape, background, device=DEV)
    for ctr, r, val in _ellipsoids(c, seed):
        inside = (((x - ctr[0]) / r[0]) ** 2)[None, None, :] + (((y - ctr[1]) / r[1]) ** 2)[None, :, None] + \
            (((z - ctr[2]) / r[2]) ** 2)[:, None, None] <= 1.0
        f += inside.float() * val
    return f


def _counts(c, scans, seed):
    """Poisson counts of each planogram: mean = the ellipsoids' line integrals
    on the visible bins, scaled to the case's total."""
    means = []
    for s in scans:
        f32 = torch.float32
        v0, v1 = s.v(s.NV0, s.Tv0, s.v0_0, f32).view(-1, 1, 1), s.v(s.NV1, s.Tv1, s.v1_0, f32)
        u0, u1 = s.v(s.NU0, s.Tu, s.u0_0, f32).view(1, 1, -1), s.v(s.NU1, s.Tu, s.u1_0, f32).view(1, -1, 1)
        dx, dy = -(v0 * s.cos + s.sin), -(v0 * s.sin - s.cos)
        vis0 = torch.from_numpy(s.vis0).to(DEV)[:, None, :]
        mean = torch.empty(s.shape, device=DEV)
        for i in range(s.NV1):
            dz = -v1[i]
            tot = torch.zeros(s.shape[1:], device=DEV)
            for ctr, r, val in _ellipsoids(c, seed):
                px, py, pz = (u0 * s.cos - ctr[0]) / r[0], (u0 * s.sin - ctr[1]) / r[1], (u1 - ctr[2]) / r[2]
                qx, qy, qz = dx / r[0], dy / r[1], dz / r[2]
                a = qx * qx + qy * qy + qz * qz
                b = px * qx + py * qy + pz * qz
                disc = b * b - a * (px * px + py * py + pz * pz - 1.0)
                tot += val * disc.clamp_(min=0.0).sqrt_() / a
            mean[i] = tot * vis0 * torch.from_numpy(s.vis1[i]).to(DEV)[None, :, None]
        means.append(mean)
    scale = c["counts"] / float(sum(m.sum(dtype=torch.float64) for m in means))
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.poisson(m.mul_(scale), generator=gen) for m in means]


def _inputs(c, seed):
    """The arrays a user's program holds before the call."""
    scans, kind = _scans(c), c["kind"]
    if kind == "project":
        return dict(f=_phantom(c, scans[0], seed))
    if kind == "vjp":
        w = torch.rand(scans[0].shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)) + 0.5
        return dict(f=_phantom(c, scans[0], seed), w=w)
    if kind == "penalized":
        B = c["batch"]
        g = torch.stack([_counts(c, scans, seed * 16 + b)[0] for b in range(B)])
        # an iterate: the phantoms on the scale of the counts
        f = torch.stack([_phantom(c, scans[0], seed * 16 + b, 0.05) for b in range(B)])
        return dict(f=f * 0.02, g=g)
    g = _counts(c, scans, seed)
    if kind == "step":
        return dict(f=_phantom(c, scans[0], seed, 0.2), g=g)
    if kind == "osem_bf16":
        return dict(g=[g[0].to(torch.bfloat16)])
    return dict(g=g)


def prepare(case, seed):
    st = dict(case=case, G=_geometries(case), **_inputs(case, seed))
    kind, S = case["kind"], case.get("subsets", 1)
    if kind == "osem":
        st["sens"] = [recon.sensitivity(st["G"], st["g"], subset=(i, S)) for i in range(S)]
    elif kind == "osem_bf16":
        ones = torch.ones_like(st["g"][0])
        st["sens"] = [ops.backproject_bf16(st["G"][0], ones, subset=(i, S)) for i in range(S)]
        for x in st["sens"]:
            x[x == 0.0] = 1.0
    elif kind == "step":
        st["sens"] = recon.sensitivity(st["G"], st["g"], subset=(1, S))
        st["ratio"] = [torch.zeros_like(x) for x in st["g"]]
        st["d"] = torch.empty_like(st["f"])
    elif kind == "penalized":
        st["g"] = st["g"].contiguous()
    return st


def run(state):
    c, G = state["case"], state["G"]
    kind, S = c["kind"], c.get("subsets", 1)
    if kind == "project":
        return ops.project(G[0], state["f"])
    if kind == "backproject":
        return ops.backproject(G[0], state["g"][0], mode="adjoint" if c.get("adjoint") else "reference")
    if kind == "osem":
        return recon.osem(G, state["g"], 1, S, sens=state["sens"])[0]
    if kind == "osem_bf16":
        return recon.osem_bf16(G[0], state["g"][0], 1, S, sens=state["sens"])
    if kind == "penalized":
        return penalized.gradient(state["f"], G[0], state["g"], RD, TV)
    if kind == "fbp":
        return ops.fbp(G, state["g"])
    if kind == "step":  # one subset of an OSEM iteration: data ratio, backprojection, update factor
        sub = (1, S)
        ops.project_ratio(G, state["f"], state["g"], out=state["ratio"], subset=sub)
        ops.backproject(G, state["ratio"], f=state["d"], subset=sub)
        return state["ratio"] + [ops.divide_(state["d"], state["sens"])]
    if kind == "vjp":
        x = state["f"].detach().requires_grad_(True)
        y = autograd.project(x, G[0])
        y.backward(state["w"])
        return y.detach(), x.grad
    raise ValueError(kind)


# ----------------------------------------------------------------------------
# what a case needs at least
# ----------------------------------------------------------------------------
def _pair_flops(s, first=0, step=1):
    """Multiply-adds of one projection of the views: each visible ray meets
    every driving plane with the u1 taps of its footprint, and the u0 taps
    are applied once per (view, plane, slice, visible column)."""
    cols, rows = float(s.vis0[first::step].sum()), float(s.vis1.sum())
    planes = max(s.nx, s.ny) if s.sin and s.cos else s.nx if s.sin else s.ny
    taps = lambda T, V: max(1.0, T / V) + min(1.0, T / V)  # noqa: E731
    return 2.0 * planes * cols * (rows * taps(s.Tu, s.Tz) + s.nz * taps(s.Tu, s.Tx))


def work(case):
    kind, S = case["kind"], case.get("subsets", 1)
    b = fl = 0.0
    for s in _scans(case):
        ng, nf = float(np.prod(s.shape)), float(s.nx * s.ny * s.nz)
        if kind in ("project", "backproject"):
            b, fl = b + 4 * (ng + nf), fl + _pair_flops(s)
        elif kind in ("osem", "osem_bf16"):
            e = 2 if kind == "osem_bf16" else 4
            # the data in, the image out; each subset's sensitivity in and its image through
            b += e * ng + 4 * nf * 2 * S
            fl += 2 * sum(_pair_flops(s, i, S) for i in range(S))
        elif kind == "step":
            b += 4 * (2 * ng * len(range(1, s.NV0, S)) / s.NV0 + 3 * nf)
            fl += 2 * _pair_flops(s, 1, S)
        elif kind == "vjp":
            b, fl = b + 4 * (2 * ng + 2 * nf), fl + 2 * _pair_flops(s)
        elif kind == "penalized":
            b += 4 * case["batch"] * (ng + 2 * nf)
            fl += case["batch"] * (2 * _pair_flops(s) + nf * 26 * 20)
        elif kind == "fbp":
            nr = ng / s.NV1
            n = 2.0 ** math.ceil(math.log2(s.NU0))
            b += 4 * (ng + nf)
            fl += ng * (2 + 2.5 * math.log2(n)) + nr * 5 * math.log2(2 * n) * 2 + nf * s.NV0 * 8
    return {"bytes": b, "flops": fl}


def tolerance(case):
    """About four times the error against the 64-bit result."""
    if case["kind"] == "osem_bf16":
        return {"rel": 1e-3}  # the data ratio and the projector's input are rounded to bfloat16
    if case.get("petx") or case["psi"] not in (0.0, 90.0):
        return {"rel": 4e-5}  # ray positions in float32, weights from their differences
    return {"rel": 1e-5}


# ----------------------------------------------------------------------------
# the operators in 64 bits
# ----------------------------------------------------------------------------
def _view(s, iv0, f):
    """Ray quantities of view iv0 and the volume as [plane][in-plane][z]."""
    v0 = iv0 * s.Tv0 + s.v0_0
    rx, ry = -(v0 * s.cos + s.sin), -(v0 * s.sin - s.cos)
    u0 = s.v(s.NU0, s.Tu, s.u0_0)
    x, y = s.v(s.nx, s.Tx, s.x0), s.v(s.ny, s.Tx, s.y0)
    if abs(s.rxf[iv0]) >= abs(s.ryf[iv0]):  # planes of constant x
        sp, rp, pp, ra, pa, trig, a0, na = x, rx, u0 * s.cos, ry, u0 * s.sin, s.sin, s.y0, s.ny
        F = f.permute(2, 1, 0)
    else:
        sp, rp, pp, ra, pa, trig, a0, na = y, ry, u0 * s.sin, rx, u0 * s.cos, s.cos, s.x0, s.nx
        F = f.permute(1, 2, 0)
    t = (sp[:, None] - pp[None, :]) / rp                      # [plane][u0]
    half = 0.5 * s.Tu * abs(trig) + 0.5 * s.Tx
    lo = torch.ceil((pa[None, :] + t * ra - half - a0) / s.Tx)
    iu = torch.arange(s.NU0, device=DEV, dtype=torch.float64)
    fw = 0.5 * s.Tx / abs(trig) / s.Tu
    taps = []
    for j in range(int(math.ceil(2 * half / s.Tx - 1e-9))):
        ia = lo + j
        cc = ((ia * s.Tx + a0 - t * ra) / trig - s.u0_0) / s.Tu
        w = (torch.minimum(iu + 0.5, cc + fw) - torch.maximum(iu - 0.5, cc - fw)).clamp_(min=0.0)
        w = w * ((ia >= 0) & (ia < na))
        taps.append((ia.clamp(0, na - 1).long(), w))
    return v0, t, F, taps, s.Tx / abs(trig)


def _z_taps(s, t, v1):
    """(slice index, weight) of the u1 footprint of rays [plane][u0][u1]."""
    tv = (t * v1)[:, :, None]
    iu1 = torch.arange(s.NU1, device=DEV, dtype=torch.float64)
    half = 0.5 * (s.Tu + s.Tz)
    lo = torch.ceil((iu1 * s.Tu + (s.u1_0 - half - s.z0) - tv) / s.Tz)
    fw = 0.5 * s.Tz / s.Tu
    for j in range(int(math.ceil(2 * half / s.Tz - 1e-9))):
        iz = lo + j
        cc = (iz * s.Tz + (s.z0 - s.u1_0) + tv) / s.Tu
        w = (torch.minimum(iu1 + 0.5, cc + fw) - torch.maximum(iu1 - 0.5, cc - fw)).clamp_(min=0.0)
        w.mul_((iz >= 0) & (iz < s.nz))
        yield iz.clamp_(0, s.nz - 1).long(), w


def _forward(s, f, views):
    """P f in 64 bits on the given views; the others stay zero."""
    f = f.double()
    g = torch.zeros(s.shape, device=DEV, dtype=torch.float64)
    v1 = [i * s.Tv1 + s.v1_0 for i in range(s.NV1)]
    vis1 = torch.from_numpy(s.vis1).to(DEV)
    for iv0 in views:
        v0, t, F, taps, l_phi = _view(s, iv0, f)
        p = torch.arange(F.shape[0], device=DEV)[:, None]
        X = sum(F[p, ia] * w[:, :, None] for ia, w in taps)    # [plane][u0][z]
        vis0 = torch.from_numpy(s.vis0[iv0]).to(DEV)
        for i in range(s.NV1):
            rows = sum((X.gather(2, iz).mul_(w)).sum(0) for iz, w in _z_taps(s, t, v1[i]))
            rows = rows * (l_phi / math.sqrt(1.0 + v0 * v0 + v1[i] ** 2))
            g[i, iv0] = (rows * vis0[:, None] * vis1[i][None, :]).t()
    return g


def _adjoint(s, g, views):
    """The transpose of _forward."""
    out = torch.zeros(s.vol_shape, device=DEV, dtype=torch.float64)
    v1 = [i * s.Tv1 + s.v1_0 for i in range(s.NV1)]
    vis1 = torch.from_numpy(s.vis1).to(DEV)
    for iv0 in views:
        v0, t, F, taps, l_phi = _view(s, iv0, out)
        P = F.shape[0]
        Y = torch.zeros((P, s.NU0, s.nz), device=DEV, dtype=torch.float64)
        vis0 = torch.from_numpy(s.vis0[iv0]).to(DEV)
        for i in range(s.NV1):
            rows = g[i, iv0].double().t() * vis0[:, None] * vis1[i][None, :]
            rows = rows * (l_phi / math.sqrt(1.0 + v0 * v0 + v1[i] ** 2))
            for iz, w in _z_taps(s, t, v1[i]):
                Y.scatter_add_(2, iz, w.mul_(rows[None]))
        p = torch.arange(P, device=DEV)[:, None].expand(P, s.NU0)
        for ia, w in taps:
            F.index_put_((p, ia), Y * w[:, :, None], accumulate=True)
    return out


def _backproject(s, g, views):
    """The voxel-driven backprojection in 64 bits: u0 extent of the voxel from
    its corners, u1 extent from its height, rays of slopes for which the
    voxel centre is visible.  g: [v1][v0][u1][u0]."""
    NV1 = g.shape[0]
    x, y = s.v(s.nx, s.Tx, s.x0)[None, :], s.v(s.ny, s.Tx, s.y0)[:, None]
    t = (y * s.cos - x * s.sin).reshape(-1)
    xd = (x * s.cos + y * s.sin).reshape(-1)
    one = NV1 == 1
    v1 = torch.zeros(1, device=DEV, dtype=torch.float64) if one else s.v(s.NV1, s.Tv1, s.v1_0)
    v1f = np.zeros(1, np.float32) if one else s.v1f
    lim1 = np.array([s.H], np.float32) if one else s.lim1
    P = torch.zeros((NV1, s.NU1, s.ny * s.nx), device=DEV, dtype=torch.float64)
    for iv0 in views:
        v0 = iv0 * s.Tv0 + s.v0_0
        wy, wx = -float(s.rxf[iv0]), float(s.ryf[iv0])         # v0 cos + sin, cos - v0 sin
        if abs(wy) > abs(wx):
            e, sign = 0.5 * s.Tx * (s.sin + v0 * s.cos), wy >= 0
        else:
            e, sign = 0.5 * s.Tx * (s.cos - v0 * s.sin), wx >= 0
        mid = (xd + v0 * t - s.u0_0) / s.Tu
        e = (e if sign else -e) / s.Tu
        A, B = mid - e, mid + e
        lo = torch.ceil(A - 0.5)
        gv = g[:, iv0].double()
        lphi = 1.0 / max(abs(v0 * s.cos + s.sin), abs(s.cos - v0 * s.sin)) / torch.sqrt(1.0 + v0 * v0 + v1 * v1)
        gv = gv * lphi[:, None, None]
        for j in range(int(math.floor(2 * e + 1.0)) + 1):
            iu = lo + j
            w = (torch.minimum(iu + 0.5, B) - torch.maximum(iu - 0.5, A)).clamp_(min=0.0)
            w = w * ((iu >= 0) & (iu < s.NU0))
            P.addcmul_(gv.index_select(2, iu.clamp_(0, s.NU0 - 1).long()), w)
    z = s.v(s.nz, s.Tz, s.z0)
    f4 = np.float32
    xf, yf = _Scan.at32(s.nx, s.Tx, s.x0)[None, :], _Scan.at32(s.ny, s.Tx, s.y0)[:, None]
    zf = _Scan.at32(s.nz, s.Tz, s.z0)
    tf = (yf.astype(np.float64) * s.cos - (xf * f4(s.sin)).astype(np.float64)).astype(f4).reshape(-1)
    tf, zf = torch.from_numpy(tf).to(DEV).double(), torch.from_numpy(zf).to(DEV).double()
    f = torch.zeros((s.nz, s.ny * s.nx), device=DEV, dtype=torch.float64)
    hw = 0.5 * s.Tz / s.Tu
    for i in range(NV1):
        u1f = (float(v1f[i]) * tf[None, :] + zf[:, None]).float()
        vis = (u1f.abs() - float(s.half)) <= float(lim1[i])
        mid = (z[:, None] + float(v1[i]) * t[None, :] - s.u1_0) / s.Tu
        lo = torch.ceil(mid - hw - 0.5)
        for j in range(int(math.floor(2 * hw + 1.0)) + 1):
            iu = lo + j
            w = (torch.minimum(iu + 0.5, mid + hw) - torch.maximum(iu - 0.5, mid - hw)).clamp_(min=0.0)
            w = w * ((iu >= 0) & (iu < s.NU1) & vis)
            f += P[i].gather(0, iu.clamp_(0, s.NU1 - 1).long()) * w
    return (f * s.Tx).view(s.vol_shape)


def _fft_size(n):
    """Smallest 2^(a+1) 3^b that holds n samples."""
    return min(2 ** a * 3 ** b for a in range(1, 24) for b in range(0, 14) if 2 ** a * 3 ** b >= n)


def _fbp(s, g):
    """Fourier rebinning along u0, ramp filter and 2-D backprojection."""
    N, f4 = _fft_size(s.NU0), np.float32
    K = N // 2 + 1
    Tf = f4(1.0 / (N * s.Tu))
    U = np.where(np.arange(K) < N // 2, np.arange(K), np.arange(K) - N).astype(f4) * Tf
    ap = f4(1.0 / (2.0 * s.Tu * 2.0 * s.m0))
    v0 = s.v(s.NV0, s.Tv0, s.v0_0)
    spec = torch.zeros((s.NV0, s.NU1, K), device=DEV, dtype=torch.complex128)
    cnt = np.zeros(K)
    for i in range(s.NV1):
        av1 = f4(abs(float(f4(f4(f4(i) * f4(s.Tv1)) + f4(s.v1_0)))))
        flat = av1 <= f4(0.5) * f4(s.Tv1)
        m = np.ones(K, bool) if flat else np.abs(U) > av1 * ap
        wgt = 1.0 / torch.sqrt(1.0 + float(av1) ** 2 + v0 * v0)
        row = torch.fft.rfft(g[i].double() * wgt[:, None, None], n=N, dim=2)
        spec += row * torch.from_numpy(m.astype(np.float64)).to(DEV)
        cnt += m
    norm = np.where((cnt > 0) & (np.arange(K) > 0), 1.0 / np.maximum(cnt, 1.0), 1.0)
    reb = torch.fft.irfft(spec * torch.from_numpy(norm).to(DEV), n=N, dim=2)[:, :, :s.NU0]
    reb = reb * torch.sqrt(1.0 + v0 * v0)[:, None, None]
    M = _fft_size(2 * s.NU0)
    k = np.arange(M)
    k = np.where(k < M // 2, k, k - M).astype(np.float64)
    h = torch.from_numpy((1.0 / (s.Tu * math.pi * (0.25 - k * k))).astype(f4).astype(np.float64)).to(DEV)
    reb = torch.fft.irfft(torch.fft.rfft(reb, n=M, dim=2) * torch.fft.rfft(h).real, n=M, dim=2)[:, :, :s.NU0]
    reb = reb * torch.sqrt(1.0 + v0 * v0)[:, None, None]
    scale = float(f4(f4(f4(s.Tv0) * f4(s.Tu)) / f4(s.Tx)))
    return _backproject(s, reb[None], range(s.NV0)) * scale


def _osem(scans, g, S, f, steps, sens=None):
    """Ordered subsets: f *= P^T(g / P f) / P^T 1 for each subset of steps."""
    ones = [torch.ones(s.shape, device=DEV) for s in scans]
    for i in steps:
        ratio, d, sn = _ratio(scans, g, f, i, S), 0.0, 0.0
        for s, r, o in zip(scans, ratio, ones):
            d = d + _backproject(s, r, range(i, s.NV0, S))
            sn = sn + _backproject(s, o, range(i, s.NV0, S))
        f = f * (d / torch.where(sn == 0, torch.ones_like(sn), sn))
    return f


def _ratio(scans, g, f, i, S):
    out = []
    for s, x in zip(scans, g):
        Pf = _forward(s, f, range(i, s.NV0, S))
        out.append(torch.where(Pf == 0, torch.zeros_like(Pf), x.double() / Pf))
    return out


def _neighbours(f):
    """(neighbour volume, weight) of the 26 neighbours, clamped at the faces."""
    pad = torch.nn.functional.pad(f[None, None], (1,) * 6, mode="replicate")[0, 0]
    n = f.shape
    for a in range(3):
        for b in range(3):
            for c in range(3):
                k = abs(a - 1) + abs(b - 1) + abs(c - 1)
                if k:
                    yield pad[a:a + n[0], b:b + n[1], c:c + n[2]], float(np.float32(1.0 / math.sqrt(k)))


def _penalties(f):
    """Costs and gradients of the relative-difference and Huber (p = 1)
    penalties, every pair counted from both sides."""
    (gam, brd), (dl, btv) = RD, TV[:2]
    brd, btv, dl = float(np.float32(brd)), float(np.float32(btv)), float(np.float32(dl))
    x = torch.where(f < float(np.float32(1e-8)), torch.zeros_like(f), f)
    cost, grad = 0.0, torch.zeros_like(f)
    for (y, w), (yt, _) in zip(_neighbours(x), _neighbours(f)):
        d, a = x - y, (x - y).abs()
        den = x + y + gam * a
        ok = den != 0
        den = torch.where(ok, den, torch.ones_like(den))
        cost = cost + w * brd * (d * d / den).sum()
        grad += 2.0 * w * brd * (d * (gam * a + x + 3.0 * y) / (den * den))
        d = f - yt
        a = d.abs()
        quad = a <= dl
        cost = cost + w * btv * torch.where(quad, 0.5 * d * d, dl * a - 0.5 * dl * dl).sum()
        grad += 2.0 * w * btv * torch.where(quad, d, dl * d.sign())
    return cost, grad


def _cost_s(case):
    """Rough seconds of exact(): one gather pass moves about 40 bytes a tap."""
    kind, S, t = case["kind"], case.get("subsets", 1), 0.0
    for s in _scans(case):
        views = s.NV0 if kind != "step" else s.NV0 / S
        taps = math.ceil(1.0 + s.Tu / s.Tz)
        fwd = s.NV1 * views * taps * (12e-5 + max(s.nx, s.ny) * s.NU0 * s.NU1 * 1.2e-11 * 4)
        t += fwd * {"project": 1, "backproject": 1, "fbp": 0.2, "penalized": 3 * case.get("batch", 1), "vjp": 3}.get(kind, 1.6)
    return t


def exact(case, seed):
    if _cost_s(case) > 20.0:
        return None
    scans, inp = _scans(case), _inputs(case, seed)
    s, kind, S = scans[0], case["kind"], case.get("subsets", 1)
    allv = range(s.NV0)
    if kind == "project":
        return _forward(s, inp["f"], allv)
    if kind == "backproject":
        return (_adjoint if case.get("adjoint") else _backproject)(s, inp["g"][0], allv)
    if kind in ("osem", "osem_bf16"):
        return _osem(scans, inp["g"], S, torch.ones(s.vol_shape, device=DEV, dtype=torch.float64), range(S))
    if kind == "step":
        ratio, d, sn = _ratio(scans, inp["g"], inp["f"], 1, S), 0.0, 0.0
        for p, r in zip(scans, ratio):
            d = d + _backproject(p, r, range(1, p.NV0, S))
            sn = sn + _backproject(p, torch.ones(p.shape, device=DEV), range(1, p.NV0, S))
        return ratio + [d / torch.where(sn == 0, torch.ones_like(sn), sn)]
    if kind == "fbp":
        return sum(_fbp(p, g) for p, g in zip(scans, inp["g"]))
    if kind == "vjp":
        return _forward(s, inp["f"], allv), _adjoint(s, inp["w"], allv)
    if kind == "penalized":
        vals, grads = [], []
        for f, g in zip(inp["f"].double(), inp["g"].double()):
            Pf = _forward(s, f, allv)
            on = Pf > 0
            safe = torch.where(on, Pf, torch.ones_like(Pf))
            val = torch.where(on, Pf - g * safe.log(), torch.zeros_like(Pf)).sum()
            cost, grad = _penalties(f)
            vals.append(val + cost)
            grads.append(grad + _adjoint(s, torch.where(on, 1.0 - g / safe, torch.zeros_like(Pf)), allv))
        return torch.stack(vals), torch.stack(grads)
    return None
