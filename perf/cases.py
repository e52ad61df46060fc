"""The calls a user of this framework has it do, as cases that can be timed and compared.

Every case is a dict of plain values.  ``prepare`` makes what a program has in hand before the call (geometry handle,
image, measurements, network), ``run`` makes one pass through the public entry points, ``exact`` computes the same
outputs in 64 bits with plain torch operations.  The ray end points, the voxel grid and the TOF bins are inputs of the
computation and are read from the geometry object; everything after them is computed here on its own.
"""
import ctypes
import math

import numpy as np
import torch

from omega_b200 import _native
from omega_b200 import reconstruction as rec
from omega_b200.learned import LAYERS, UNet3D
from omega_b200.projector import geometry as geo
from omega_b200.projector import proj

C_MM = 2.99792458e11  # mm / s
DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _pet(**k):
    c = dict(kind="pet", projector=1, crystals=384, rings=32, diameter=600.0, fov=300.0, nx=128, nz=63, ndist=256,
             nang=192, nsinos=63, subsets=16, tof=1, atomics="float", read="fp32")
    c.update(k)
    return c


def _ct(kind, **k):
    c = dict(kind=kind, rows=512, cols=512, pitch=0.4, views=360, subsets=1, nx=256, nz=256, voxel=0.25, sod=500.0,
             sdd=1000.0)
    c.update(k)
    return c


def listed():
    return [
        # the smallest call a custom reconstruction loop makes: one subset forward and back on the 288 x 16 scanner
        # (64 x 64 x 16 image, 8 subsets); launch latency and a nearly empty chip count here
        _pet(name="pet64_pair", crystals=288, rings=16, nx=64, nz=16, ndist=144, nang=144, nsinos=31, subsets=8),
        # the ordinary sub-iteration of a custom loop: one of 16 subsets forward and back, improved Siddon
        _pet(name="pet128_pair"),
        # dynamic study: one OSEM iteration (all 16 subsets) of 24 frames that share one geometry
        dict(_pet(name="pet_osem_24f"), kind="frames", frames=24),
        # TOF Siddon with the deterministic int64 backprojection, odd sizes
        _pet(name="pet_tof_int64", crystals=480, rings=21, diameter=700.0, fov=420.0, nx=147, nz=41, ndist=281,
             nang=240, nsinos=41, subsets=7, tof=11, atomics="int64"),
        # the precision configuration: interpolation projector, 15 TOF bins, 200 x 200 x 109 image, one of 16 subsets
        _pet(name="interp_tof_pair", projector=4, crystals=672, rings=55, diameter=856.0, fov=600.0, nx=200, nz=109,
             ndist=400, nang=336, nsinos=109, tof=15),
        # interpolation projector without TOF, BF16 image reads, ragged sizes
        _pet(name="interp_bf16_pair", projector=4, crystals=384, nx=121, nz=55, ndist=219, nang=192, nsinos=59,
             subsets=9, read="bf16"),
        # cone-beam CT with the interpolation projector (ray-driven forward, voxel-driven back), ragged sizes
        _ct("ct4", name="ct_interp_pair", rows=301, cols=218, pitch=0.7, views=90, nx=170, nz=121, voxel=0.4),
        # cone-beam CT, distance-driven: one of 4 subsets (90 of 360 views) of the 512 x 512 panel, forward ...
        _ct("bdd_fp", name="ct_bdd_fp", subsets=4),
        # ... and back
        _ct("bdd_bp", name="ct_bdd_bp", subsets=4),
        # cone-beam CT, the whole PDHG + TV iteration on all 360 views (forward, dual, back, TV and primal step)
        _ct("pdhg", name="ct_pdhg"),
        # one convolution layer of the learned warm start's network, ragged volume
        dict(name="unet_conv", kind="conv", cin=32, cout=32, X=62, Y=58, Z=31, batch=4, mode="relu"),
        # one training step of the network: forward, loss and all gradients, batch of 4 studies
        dict(name="unet_train", kind="unet", X=128, Y=128, Zs=63, batch=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pet", "pet", "pet4", "pet4", "frames", "ct4", "bdd_fp", "bdd_bp", "pdhg", "conv", "conv",
                       "unet"])
    if kind in ("pet", "pet4", "frames"):
        crystals = 32 * rng.randint(9, 21)   # an even number of blocks of 16
        rings = _log(rng, 8, 40)
        diameter = 1.55 * crystals
        nsinos = 2 * rings - 1
        c = _pet(projector=4 if kind == "pet4" else 1, crystals=crystals, rings=rings, diameter=diameter,
                 fov=round(diameter * rng.uniform(0.4, 0.65), 1), nx=_log(rng, 64, 200), nz=_log(rng, 11, 80),
                 ndist=rng.randint(crystals // 3, crystals // 2), nang=crystals // 2, nsinos=nsinos, subsets=min(rng.randint(4, 16), nsinos))
        if kind == "frames":
            c.update(kind="frames", frames=rng.choice([2, 3, 5, 8, 12]), nx=_log(rng, 64, 128), nz=_log(rng, 11, 40),
                     rings=min(rings, 20))
            c.update(nsinos=2 * c["rings"] - 1, subsets=min(c["subsets"], 2 * c["rings"] - 1))
        else:
            c["tof"] = rng.choice([1, 1, 5, 9, 11, 13, 15])
            c["atomics"] = rng.choice(["float", "float", "int64"])
            if c["tof"] == 1:
                c["read"] = rng.choice(["fp32", "fp32", "bf16"])
        return c
    if kind in ("ct4", "bdd_fp", "bdd_bp", "pdhg"):
        nx = _log(rng, 64, 256)
        if kind != "ct4" and rng.random() < 0.6:
            nx = nx // 4 * 4
        rows = int(nx * rng.uniform(1.2, 2.2))
        if kind != "ct4" and rng.random() < 0.6:
            rows = rows // 4 * 4
        nz = int(nx * rng.uniform(0.3, 1.0)) + 1
        voxel = 64.0 / nx
        return _ct(kind, rows=rows, cols=int(rows * rng.uniform(0.4, 1.0)) + 1,
                   pitch=round(2.0 * 1.35 * nx * voxel / rows, 4), views=_log(rng, 24, 120),
                   subsets=1, nx=nx, nz=nz, voxel=round(voxel, 4))
    if kind == "conv":
        cin, cout = rng.choice([(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16), (32, 16),
                                (64, 32), (32, 96), (16, 48)])
        return dict(kind="conv", cin=cin, cout=cout, X=_log(rng, 12, 130), Y=_log(rng, 12, 130), Z=_log(rng, 5, 64),
                    batch=rng.choice([1, 2, 4]), mode=rng.choice(["relu", "mask", "plain"]))
    return dict(kind="unet", X=4 * _log(rng, 6, 32), Y=4 * _log(rng, 6, 32), Zs=_log(rng, 9, 63),
                batch=rng.choice([1, 2, 3]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _pet_options(c):
    o = proj.projectorClass()
    o.cryst_per_block = 16
    o.blocks_per_ring = c["crystals"] // 16
    o.cryst_per_block_axial, o.linear_multip = c["rings"], 1
    o.rings = c["rings"]
    o.det_per_ring = o.det_w_pseudo = c["crystals"]
    o.diameter = c["diameter"]
    o.cr_p = math.pi * c["diameter"] / c["crystals"]
    o.cr_pz = 4.0
    o.FOVa_x = o.FOVa_y = c["fov"]
    o.axial_fov = 4.0 * c["rings"]
    o.Nx = o.Ny = c["nx"]
    o.Nz = c["nz"]
    o.span, o.ring_difference = 3, c["rings"] - 1
    o.Ndist, o.Nang = c["ndist"], c["nang"]
    o.NSinos = c["nsinos"]
    o.TotSinos = int(np.sum(geo.default_segment_table(c["rings"], 3, c["rings"] - 1, c["nsinos"])))
    o.projector_type = c["projector"]
    o.subsets, o.subsetType = c["subsets"], 8
    if c["tof"] > 1:
        o.TOF_bins = o.TOF_bins_used = c["tof"]
        o.TOF_FWHM = 200e-12
        o.TOF_width = 1.42 * c["fov"] / c["tof"] / (C_MM / 2)
    o.use_64bit_atomics = c["atomics"] == "int64"
    o.imageReadPrecision = c["read"]
    o.verbose = 0
    o.addProjector()
    return o


def _ct_options(c):
    o = proj.projectorClass()
    o.CT = True
    o.nRowsD, o.nColsD = c["rows"], c["cols"]
    o.nProjections = c["views"]
    o.dPitchX = o.dPitchY = c["pitch"]
    o.sourceToCRot, o.sourceToDetector = c["sod"], c["sdd"]
    o.Nx = o.Ny = c["nx"]
    o.Nz = c["nz"]
    o.FOVa_x = o.FOVa_y = c["voxel"] * c["nx"]
    o.axial_fov = c["voxel"] * c["nz"]
    o.angles = np.linspace(0, 2 * np.pi, c["views"], endpoint=False).astype(np.float32)
    o.projector_type = 4 if c["kind"] == "ct4" else 5
    o.subsets, o.subsetType = c["subsets"], 8
    o.verbose = 0
    o.SinM = np.zeros((c["rows"], c["cols"], c["views"]), dtype=np.float32)  # marks projection data
    o.addProjector()
    o.SinM = np.empty(0, dtype=np.float32)
    return o


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _phantom(nx, ny, nz, seed, scale, noise):
    """An elliptic body with hot and cold ellipsoids and the texture of an iterate, x fastest, positive."""
    g = _gen(seed)
    r = np.random.default_rng(seed)
    ax = [(torch.arange(n, device=DEV, dtype=torch.float32) + 0.5) / n * 2 - 1 for n in (nz, ny, nx)]
    z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    v = torch.full((nz, ny, nx), 0.02, device=DEV)
    v[((x / .72) ** 2 + (y / .55) ** 2 + 0 * z < 1)] = 1.0
    for k in range(8):
        p = r.uniform(-.45, .45, 3)
        q = r.uniform(.05, .22, 3)
        v[((x - p[0]) / q[0]) ** 2 + ((y - p[1]) / q[1]) ** 2 + ((z - p[2]) / (2 * q[2])) ** 2 < 1] = \
            (4.0, 0.3, 2.0)[k % 3]
    v *= 1 + noise * (torch.rand(v.shape, generator=g, device=DEV) - 0.5)
    return (v * scale).reshape(-1)


def _subset(c):
    return c["subsets"] // 2


def _pet_measurement(m, seed):
    """Measured over estimated counts of a low-count scan: around 1, with zeros."""
    return torch.poisson(torch.full((m,), 6.0, device=DEV), generator=_gen(seed + 1)) / 6.0


def _ct_measurement(m, seed):
    """A dual variable / residual: of both signs."""
    return torch.randn(m, generator=_gen(seed + 1), device=DEV) * 0.1 + 0.05


def _frame_measurements(c, n_proj, seed):
    lam = torch.linspace(2.0, 30.0, c["frames"], device=DEV)[:, None].expand(c["frames"],
                                                                              c["ndist"] * c["nang"] * n_proj)
    return torch.poisson(lam, generator=_gen(seed + 1))


def _frame_images(c, seed):
    base = _phantom(c["nx"], c["nx"], c["nz"], seed, 1.0, 0.6)
    k = torch.linspace(0.01, 0.15, c["frames"], device=DEV)[:, None]
    return (base[None] * k).contiguous()


def _pdhg_start(c, seed):
    x0 = _phantom(c["nx"], c["nx"], c["nz"], seed, 0.005, 0.4)
    y = torch.rand(c["rows"] * c["cols"] * c["views"], generator=_gen(seed + 1), device=DEV) * 0.6
    chord = c["voxel"] * c["nx"]
    mag = c["sdd"] / c["sod"]
    tau = 0.5 / (chord * (mag * c["voxel"] / c["pitch"]) ** 2 * c["voxel"] * c["views"])
    return x0, y, tau


def _conv_inputs(c, seed):
    g = _gen(seed)
    nv = c["batch"] * c["Z"] * c["Y"] * c["X"]
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    x = torch.relu(rnd(nv * c["cin"])).bfloat16()
    w = (rnd(27, c["cout"], c["cin"]) * math.sqrt(2.0 / (27 * c["cin"]))).bfloat16()
    b = rnd(c["cout"]) * 0.1 if c["mode"] == "relu" else None
    mask = torch.relu(rnd(nv * c["cout"])).bfloat16() if c["mode"] == "mask" else None
    return x, w, b, mask


def _unet_inputs(c, seed):
    n = c["X"] * c["Y"] * c["Zs"]
    osem = torch.stack([_phantom(c["X"], c["Y"], c["Zs"], seed + 100 * b, 0.5 + b, 0.5) for b in range(c["batch"])])
    target = torch.stack([_phantom(c["X"], c["Y"], c["Zs"], seed + 100 * b, 0.5 + b, 0.1) for b in range(c["batch"])])
    sens = torch.rand(n, generator=_gen(seed + 7), device=DEV) + 0.5
    r = np.random.default_rng(seed)
    sd = {"head_w": r.normal(0, .2, 16).astype(np.float32), "head_b": np.zeros(1, dtype=np.float32)}
    for i, (ci, co) in enumerate(LAYERS):
        fan = 2 if i == 0 else ci
        w = r.normal(0.0, math.sqrt(2.0 / (27 * fan)), (27, co, ci)).astype(np.float32)
        if i == 0:
            w[:, :, 2:] = 0
        sd[f"w{i}"] = torch.from_numpy(w).bfloat16().float().numpy()
        sd[f"b{i}"] = r.normal(0, .05, co).astype(np.float32)
    return osem, target, sens, sd


def prepare(case, seed):
    c, k = case, case["kind"]
    if k in ("pet", "frames", "ct4", "bdd_fp", "bdd_bp", "pdhg"):
        o = _pet_options(c) if k in ("pet", "frames") else _ct_options(c)
        o.initProj()
    if k == "pet":
        s = _subset(c)
        return dict(kind=k, o=o, s=s, x=_phantom(c["nx"], c["nx"], c["nz"], seed, 0.05, 0.6),
                    y=_pet_measurement(o.measurementCount(s), seed))
    if k == "frames":
        return dict(kind=k, loop=rec.OSEMBatch(o, _frame_measurements(c, c["nsinos"], seed), x0=_frame_images(c, seed)))
    if k in ("ct4", "bdd_fp", "bdd_bp"):
        s = _subset(c)
        return dict(kind=k, o=o, s=s, x=_phantom(c["nx"], c["nx"], c["nz"], seed, 0.01, 0.2),
                    y=_ct_measurement(o.measurementCount(s), seed))
    if k == "pdhg":
        x0, y, tau = _pdhg_start(c, seed)
        return dict(kind=k, loop=rec.PDHG(o, y, 0.05, tv_smooth=1e-4, tau=tau, x0=x0))
    if k == "conv":
        x, w, b, mask = _conv_inputs(c, seed)
        out = torch.empty(x.numel() // c["cin"] * c["cout"], dtype=torch.bfloat16, device=DEV)
        return dict(kind=k, c=c, x=x, w=w, b=b, mask=mask, out=out)
    osem, target, sens, sd = _unet_inputs(c, seed)
    net = UNet3D(c["X"], c["Y"], c["Zs"], c["batch"], DEV)
    net.load_state_dict(sd)
    return dict(kind=k, net=net, osem=osem, target=target, sens=sens, n=c["X"] * c["Y"] * c["Zs"])


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def run(state):
    k = state["kind"]
    if k in ("pet", "ct4"):
        o, s = state["o"], state["s"]
        return o.forwardProject(state["x"], s), o.backwardProject(state["y"], s)
    if k == "bdd_fp":
        return state["o"].forwardProject(state["x"], state["s"])
    if k == "bdd_bp":
        return state["o"].backwardProject(state["y"], state["s"])
    if k == "frames":
        return state["loop"].iterate(1)
    if k == "pdhg":
        loop = state["loop"]
        return loop.iterate(1), loop.u, loop.p
    if k == "conv":
        c = state["c"]
        _native.call("omb_unet_conv_tc", c["cin"], c["cout"], _ptr(state["x"]), _ptr(state["w"]), _ptr(state["b"]),
                     _ptr(state["out"]), _ptr(state["mask"]), 1 if c["mode"] == "relu" else 0, c["X"], c["Y"], c["Z"],
                     c["batch"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return state["out"]
    net = state["net"]
    pred = net.forward(state["osem"], state["n"], state["sens"], 1.0)
    net.backward(state["target"], state["n"])
    return pred, [p["gw"] for p in net.params], [p["gb"] for p in net.params], net.gw_head, net.gb_head


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    c, k = case, case["kind"]
    if k in ("pet", "frames"):
        n = c["nx"] * c["nx"] * c["nz"]
        views = c["nsinos"] if k == "frames" else -(-c["nsinos"] // c["subsets"])
        rays = c["ndist"] * c["nang"] * views
        steps = 1.1 * c["nx"] * (1 if c["projector"] == 1 else 0.9)   # crossings / samples of a mean chord
        per = (2 if c["projector"] == 1 else 16) + 2                  # forward, back
        f = c.get("frames", 1)
        flops = rays * steps * (per * f if c["tof"] == 1 else per + 14.0 * c["tof"])
        return {"bytes": 4.0 * f * 2 * (n + rays * c["tof"]), "flops": flops}
    if k in ("ct4", "bdd_fp", "bdd_bp", "pdhg"):
        n = c["nx"] * c["nx"] * c["nz"]
        views = c["views"] // c["subsets"]
        rays = c["rows"] * c["cols"] * views
        # a footprint covers about 2 x 2 voxels of each slice, about 2 x 2 pixels of each view
        fp, bp = rays * c["nx"] * (8.0 if k != "ct4" else 16.0), float(n) * views * 12.0
        return {"bdd_fp": {"bytes": 4.0 * (n + rays), "flops": fp}, "bdd_bp": {"bytes": 4.0 * (n + rays), "flops": bp},
                "ct4": {"bytes": 8.0 * (n + rays), "flops": fp + bp},
                "pdhg": {"bytes": 4.0 * (4 * n + 3 * rays), "flops": fp + bp + 60.0 * n}}[k]
    if k == "conv":
        nv = c["batch"] * c["Z"] * c["Y"] * c["X"]
        return {"bytes": 2.0 * nv * (c["cin"] + c["cout"] * (2 if c["mode"] == "mask" else 1)),
                "flops": 54.0 * nv * c["cin"] * c["cout"]}
    nv = c["batch"] * c["X"] * c["Y"] * (-(-c["Zs"] // 4) * 4)
    level = [1, 1, 8, 8, 64, 64, 8, 8, 1, 1]
    mac = sum(27.0 * ci * co * nv / lv for (ci, co), lv in zip(LAYERS, level))
    act = sum(2.0 * (ci + co) * nv / lv for (ci, co), lv in zip(LAYERS, level))
    return {"bytes": 3 * act, "flops": 6 * mac}


def tolerance(case):
    k = case["kind"]
    if k == "conv":
        return {"rel": 5e-3}   # BF16 outputs: half a unit in the last place is 2^-9 of a value
    if k == "unet":
        return {"rel": 2e-2}   # BF16 activations and activation gradients through ten layers
    if k in ("ct4", "bdd_fp"):
        return {"rel": 2.5e-5}  # footprint edges / sample positions along oblique rays in FP32: 6e-6 to 2e-5 seen
    return {"rel": 1e-5}       # FP32 geometry and sums


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

class _Grid:
    def __init__(self, o):
        f = lambda v: float(np.ravel(v)[0])  # noqa: E731
        self.n = [int(np.ravel(v)[0]) for v in (o.Nx, o.Ny, o.Nz)]
        self.d = [f(v) for v in (o.dx, o.dy, o.dz)]
        self.b = [f(v) for v in (o.bx, o.by, o.bz)]
        self.m = [float(np.float32(b) + np.float32(n) * np.float32(d)) for b, n, d in zip(self.b, self.n, self.d)]
        self.voxels = self.n[0] * self.n[1] * self.n[2]
        self.eps = float(np.float32(o.epps))


def _pet_rays(o, c, s):
    """End points of a subset's rays, (R, 3) each."""
    xy = torch.from_numpy(np.asarray(o.x, dtype=np.float32).reshape(-1, 4)).to(DEV, F64)
    z = torch.from_numpy(np.asarray(o.z, dtype=np.float32).reshape(-1, 2)).to(DEV, F64)
    lo, hi = int(o.nMeas[s]), int(o.nMeas[s + 1])
    nb, nv = xy.shape[0], hi - lo
    xy = xy[None].expand(nv, nb, 4)
    z = z[lo:hi, None, :].expand(nv, nb, 2)
    return (torch.stack([xy[..., 0], xy[..., 1], z[..., 0]], -1).reshape(-1, 3),
            torch.stack([xy[..., 2], xy[..., 3], z[..., 1]], -1).reshape(-1, 3))


def _tof_of(o, c):
    if c["tof"] == 1:
        return None
    return [float(np.float32(v)) for v in np.ravel(o.TOFCenter)], float(np.float32(o.sigma_x))


def _tof_weights(tof, eps, sign, ele, D):
    """Trapezoid of the TOF Gaussian over an element, per bin, and their sum (at least eps)."""
    centers, sigma = tof
    dx = ele / 3.0
    w = []
    for c in centers:
        t = [torch.exp(-0.5 * ((D - c - a) / sigma) ** 2) for a in (0.0, dx * sign, 2 * dx * sign, ele * sign)]
        w.append((t[0] + t[3] + 2 * (t[1] + t[2])) * dx * (0.3989423 / sigma))
    total = sum(w)
    return w, torch.where(total < eps, torch.full_like(total, eps), total)


def _siddon(g, p, q):
    """Voxel, length and (for TOF) signed distance data of every crossing of rays p -> q: (R, A) each."""
    v = q - p
    L = v.norm(dim=1)
    R = p.shape[0]
    t_lo = torch.zeros(R, device=DEV, dtype=F64)
    t_hi = torch.ones(R, device=DEV, dtype=F64)
    enter = torch.full((R,), -1e300, device=DEV, dtype=F64)
    planes, hit = [], torch.ones(R, device=DEV, dtype=torch.bool)
    for a in range(3):
        still = v[:, a].abs() < 1e-6
        va = torch.where(still, torch.ones_like(L), v[:, a])
        al = (g.b[a] + torch.arange(g.n[a] + 1, device=DEV, dtype=F64)[None] * g.d[a] - p[:, a:a + 1]) / va[:, None]
        first, last = torch.minimum(al[:, 0], al[:, -1]), torch.maximum(al[:, 0], al[:, -1])
        inside = (q[:, a] >= g.b[a]) & (q[:, a] <= g.m[a])
        hit &= ~still | inside
        enter = torch.where(still, enter, torch.maximum(enter, first))
        t_lo = torch.where(still, t_lo, torch.maximum(t_lo, first))
        t_hi = torch.where(still, t_hi, torch.minimum(t_hi, last))
        planes.append(torch.where(still[:, None], t_lo[:, None].expand_as(al), al))
    hit &= t_hi > t_lo
    al = torch.cat(planes, 1)
    al = torch.minimum(torch.maximum(al, t_lo[:, None]), torch.maximum(t_hi, t_lo)[:, None]).sort(1)[0]
    ele = (al[:, 1:] - al[:, :-1]) * L[:, None]
    ele = torch.where(hit[:, None], ele, torch.zeros_like(ele))
    mid = 0.5 * (al[:, 1:] + al[:, :-1])
    ijk = []
    for a in range(3):
        at = p[:, a:a + 1] + v[:, a:a + 1] * mid
        at = torch.where(v[:, a:a + 1].abs() < 1e-6, q[:, a:a + 1], at)   # a ray along this face stays in one row
        ijk.append(((at - g.b[a]) / torch.full_like(at, g.d[a])).floor().clamp(0, g.n[a] - 1).long())
    ind = ijk[0] + g.n[0] * (ijk[1] + g.n[1] * ijk[2])
    # distance of an element's start from the middle of the ray
    D0 = enter.abs() * L - L / 2
    sign = torch.sign(D0)
    D = D0[:, None] - sign[:, None] * (torch.cumsum(ele, 1) - ele)
    for a, b in ((0, 1), (1, 0)):   # rays along an image row: voxels counted from the row's start
        row = (v[:, 2].abs() < 1e-6) & (v[:, b].abs() < 1e-6)
        half = torch.copysign(torch.full_like(L, g.n[a] * g.d[a] / 2), v[:, b])
        sg = torch.sign(half)
        sign = torch.where(row, sg, sign)
        D = torch.where(row[:, None], half[:, None] - sg[:, None] * g.d[a] * ijk[a], D)
    return ind, ele, 1.0 / L, D, sign


def _siddon_pair(g, p, q, x, y, tof):
    """Forward projection of x and backprojection of y, improved Siddon."""
    R = p.shape[0]
    nb = 1 if tof is None else len(tof[0])
    fp = torch.zeros(nb, R, device=DEV, dtype=F64)
    bp = torch.zeros(g.voxels, device=DEV, dtype=F64)
    y = y.reshape(nb, R)
    step = max(1, int(3e7 / (sum(g.n) + 3)))
    for r in range(0, R, step):
        at = slice(r, min(r + step, R))
        ind, ele, inv, D, sign = _siddon(g, p[at], q[at])
        le = ele * inv[:, None]
        if tof is None:
            fp[0, at] = (le * x[ind]).sum(1)
            bp.index_add_(0, ind.reshape(-1), (le * y[0, at, None]).reshape(-1))
        else:
            w, total = _tof_weights(tof, g.eps, sign[:, None], ele, D)
            le = le / total
            xv, back = x[ind] * le, torch.zeros_like(le)
            for t in range(nb):
                fp[t, at] = (w[t] * xv).sum(1)
                back += w[t] * y[t, at, None]
            bp.index_add_(0, ind.reshape(-1), (back * le).reshape(-1))
    return fp.reshape(-1), bp


def _march(g, p, q, dL):
    """First parameter, step, sample count and length of rays sampled every dL."""
    v = q - p
    lo = torch.full_like(p[:, 0], -math.inf)
    hi = torch.full_like(p[:, 0], math.inf)
    for a in range(3):
        t0, t1 = (g.b[a] - p[:, a]) / v[:, a], (g.m[a] - p[:, a]) / v[:, a]
        lo, hi = torch.maximum(lo, torch.fmin(t0, t1)), torch.minimum(hi, torch.fmax(t0, t1))
    L = (v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2]).sqrt()
    step = torch.full_like(L, dL) / L   # (a number over a tensor would be taken as its reciprocal's multiple)
    n = torch.where(lo < hi, ((hi - lo) / step).floor() + 1, torch.zeros_like(lo))
    return v, torch.where(lo < hi, lo, torch.zeros_like(lo)), step, n, L


def _trilinear(g, x, pos):
    i0, w = [], []
    for a in range(3):
        t = ((pos[a] - g.b[a]) / g.d[a] - 0.5).clamp(-1, g.n[a])
        f = t.floor()
        w.append(t - f)
        i0.append(f.long())
    out = 0
    for k in range(8):
        ind, ww, mul = 0, 1, 1
        for a in range(3):
            e = k >> a & 1
            ind = ind + (i0[a] + e).clamp(0, g.n[a] - 1) * mul
            ww = ww * (w[a] if e else 1 - w[a])
            mul *= g.n[a]
        out = out + ww * x[ind]
    return out


def _interp_forward(g, p, q, x, dL, tof, pet):
    R = p.shape[0]
    nb = 1 if tof is None else len(tof[0])
    fp = torch.zeros(nb, R, device=DEV, dtype=F64)
    most = int(math.sqrt(sum((n * d) ** 2 for n, d in zip(g.n, g.d))) / dL) + 2
    chunk = max(1, int(2e7 / most))
    for r in range(0, R, chunk):
        at = slice(r, min(r + chunk, R))
        v, ts, st, n, L = _march(g, p[at], q[at], dL)
        m = int(n.max())
        if m == 0:
            continue
        i = torch.arange(m, device=DEV, dtype=F64)[None]
        t = ts[:, None] + i * st[:, None]
        val = dL * _trilinear(g, x, [p[at, a:a + 1] + v[:, a:a + 1] * t for a in range(3)])
        val = torch.where(i < n[:, None], val, torch.zeros_like(val))
        if pet:
            val = val / L[:, None]
        if tof is None:
            fp[0, at] = val.sum(1)
        else:
            D0 = ts.abs() * L - 0.5 * L
            sg = torch.sign(D0)
            w, total = _tof_weights(tof, g.eps, sg[:, None], torch.full_like(val, dL), D0[:, None] - sg[:, None] * i * dL)
            for b in range(nb):
                fp[b, at] = (w[b] * val / total).sum(1)
    return fp.reshape(-1)


def _interp_backward(g, p, q, y, dL, tof):
    R = p.shape[0]
    nb = 1 if tof is None else len(tof[0])
    y = y.reshape(nb, R)
    bp = torch.zeros(g.voxels, device=DEV, dtype=F64)
    most = int(math.sqrt(sum((n * d) ** 2 for n, d in zip(g.n, g.d))) / dL) + 2
    chunk = max(1, int(2e7 / most))
    for r in range(0, R, chunk):
        at = slice(r, min(r + chunk, R))
        v, ts, st, n, L = _march(g, p[at], q[at], dL)
        m = int(n.max())
        if m == 0:
            continue
        i = torch.arange(m, device=DEV, dtype=F64)[None]
        t = ts[:, None] + i * st[:, None]
        ind, mul = 0, 1
        for a in range(3):
            ind = ind + ((p[at, a:a + 1] + v[:, a:a + 1] * t - g.b[a]) * (1.0 / g.d[a])).clamp_min(0).long() * mul
            mul *= g.n[a]
        good = (i < n[:, None]) & (ind > 0) & (ind < g.voxels)   # voxel 0 takes no samples
        le = (dL / L)[:, None].expand_as(t)
        if tof is None:
            val = le * y[0, at, None]
        else:
            kd = torch.cumsum(good.to(F64), 1) - good.to(F64)
            D0 = ts.abs() * L - 0.5 * L
            sg = torch.sign(D0)
            w, total = _tof_weights(tof, g.eps, sg[:, None], torch.full_like(t, dL), D0[:, None] - sg[:, None] * kd * dL)
            val = sum(w[b] * y[b, at, None] for b in range(nb)) * le / total
        bp.index_add_(0, ind[good], val[good])
    return bp


class _Panel:
    """Source, panel centre and pixel step of every view of a subset."""

    def __init__(self, o, c, s):
        lo, hi = int(o.nMeas[s]), int(o.nMeas[s + 1])
        self.xy = np.asarray(o.x, dtype=np.float32).reshape(-1, 6)[lo:hi].astype(np.float64)
        self.uv = np.asarray(o.z, dtype=np.float32).reshape(-1, 2)[lo:hi].astype(np.float64)
        self.nr, self.nc = c["rows"], c["cols"]
        self.pitch = float(np.float32(c["pitch"]))
        self.views = hi - lo


def _ct_rays(P, v):
    s, d, u = P.xy[v, :3], P.xy[v, 3:], P.uv[v]
    ia = torch.arange(P.nr, device=DEV, dtype=F64) - P.nr / 2 + .5
    ib = torch.arange(P.nc, device=DEV, dtype=F64) - P.nc / 2 + .5
    q = torch.stack([(d[0] + ia * u[0])[None].expand(P.nc, P.nr), (d[1] + ia * u[1])[None].expand(P.nc, P.nr),
                     (d[2] + ib * P.pitch)[:, None].expand(P.nc, P.nr)], -1).reshape(-1, 3)
    return torch.tensor(s, device=DEV, dtype=F64)[None].expand_as(q), q


def _onto_panel(P, v, x, y, z):
    """Panel coordinates (pixel edges at whole numbers) of the projections of points, and the parameter of the hit."""
    s, d, u = P.xy[v, :3], P.xy[v, 3:], P.uv[v]
    lu = math.hypot(u[0], u[1])
    e, n = (u[0] / lu, u[1] / lu), (-u[1] / lu, u[0] / lu)
    t = (n[0] * (d[0] - s[0]) + n[1] * (d[1] - s[1])) / (n[0] * (x - s[0]) + n[1] * (y - s[1]))
    pu = (e[0] * (s[0] + t * (x - s[0]) - d[0]) + e[1] * (s[1] + t * (y - s[1]) - d[1])) / P.pitch + P.nr / 2
    pv = (s[2] + t * (z - s[2]) - d[2]) / P.pitch + P.nc / 2
    return pu, pv, t


def _prefix_at(P, V, e, dim):
    """Integral of the piecewise constant V along dim from 0 to e (P: its exclusive prefix sums), e within [0, n]."""
    n = V.shape[dim]
    i = e.floor().clamp(0, n - 1).long()
    return P.gather(dim, i) + (e - i) * V.gather(dim, i)


def _prefix(V, dim):
    return torch.cumsum(V, dim) - V


def _bdd_forward(g, P, x):
    nx, ny, nz = g.n
    img = x.reshape(nz, ny, nx)
    out = torch.zeros(P.views, P.nc, P.nr, device=DEV, dtype=F64)
    ia = torch.arange(P.nr, device=DEV, dtype=F64) - P.nr / 2 + .5
    for v in range(P.views):
        s, d, u = P.xy[v, :3], P.xy[v, 3:], P.uv[v]
        a = 1 if abs(s[0]) <= abs(s[1]) else 0      # slices along this axis
        l = 1 - a                                   # noqa: E741  lateral axis
        V = (img.permute(1, 0, 2) if a == 1 else img.permute(2, 0, 1)).contiguous()   # slice, z, lateral
        dist = g.b[a] - s[a] + (torch.arange(g.n[a], device=DEV, dtype=F64) + .5) * g.d[a]
        cen = [d[k] + ia * u[k] for k in (0, 1)]
        edge = []
        for h in (0.5, -0.5):
            slope = (cen[l] + h * u[l] - s[l]) / (cen[a] + h * u[a] - s[a])
            edge.append((dist[:, None] * slope[None] - (g.b[l] - s[l])) / g.d[l])      # slice, row
        lo, hi = torch.minimum(*edge), torch.maximum(*edge)
        width = (edge[1] - edge[0]).abs()
        pre = _prefix(V, 2)
        ex = lambda e: e.clamp(0, g.n[l])[:, None, :].expand(-1, nz, -1).contiguous()  # noqa: E731
        lat = _prefix_at(pre, V, ex(hi), 2) - _prefix_at(pre, V, ex(lo), 2)            # slice, z, row
        zpre = _prefix(lat, 1)
        zb = d[2] + (torch.arange(P.nc + 1, device=DEV, dtype=F64) - P.nc / 2) * P.pitch
        ze = (dist[:, None, None] * ((zb - s[2])[None, :, None] / (cen[a] - s[a])[None, None, :])
              - (g.b[2] - s[2])) / g.d[2]                                             # slice, column edge, row
        I = _prefix_at(zpre, lat, ze.clamp(0, nz), 1)                                 # noqa: E741
        dz = ze[:, 1:] - ze[:, :-1]
        I = (I[:, 1:] - I[:, :-1]) / dz                                               # noqa: E741
        mean = (I / (width[:, None, :] * g.d[l] * g.d[2])).sum(0)
        ib = (torch.arange(P.nc, device=DEV) // 8 * 8).to(F64) - P.nc / 2 + .5         # weights of groups of 8 columns
        w = [(cen[k] - s[k])[None, :] for k in (0, 1)] + [(d[2] + ib * P.pitch - s[2])[:, None]]
        L = (w[0] ** 2 + w[1] ** 2 + w[2] ** 2).sqrt()
        out[v] = mean * g.d[0] * g.d[1] * g.d[2] * L / w[a].abs()
    return out.reshape(-1)


def _centres(g, a):
    return g.b[a] + (torch.arange(g.n[a], device=DEV, dtype=F64) + .5) * g.d[a]


def _bdd_backward(g, P, y):
    nx, ny, nz = g.n
    y = y.reshape(P.views, P.nc, P.nr)
    out = torch.zeros(nz, ny * nx, device=DEV, dtype=F64)
    qx = _centres(g, 0)[None, :].expand(ny, nx).reshape(-1)
    qy = _centres(g, 1)[:, None].expand(ny, nx).reshape(-1)
    qz = _centres(g, 2)[:, None]
    for v in range(P.views):
        s = P.xy[v, :3]
        ysl = abs(s[0]) <= abs(s[1])
        sg = 1.0 if (s[1] if ysl else s[0]) > 0 else -1.0
        hx, hy = (0.5 * g.d[0] * sg, 0.0) if ysl else (0.0, -0.5 * g.d[1] * sg)
        ul, vl, _ = _onto_panel(P, v, qx - hx, qy - hy, qz - 0.5 * g.d[2])
        ur, vr, _ = _onto_panel(P, v, qx + hx, qy + hy, qz + 0.5 * g.d[2])
        ua, ub = torch.minimum(ul, ur).clamp(0, P.nr), torch.maximum(ul, ur).clamp(0, P.nr)
        va, vb = torch.minimum(vl, vr).clamp(0, P.nc), torch.maximum(vl, vr).clamp(0, P.nc)
        Y = y[v]
        pre = _prefix(Y, 1)
        ex = lambda e: e[None].expand(P.nc, -1).contiguous()  # noqa: E731
        row = _prefix_at(pre, Y, ex(ub), 1) - _prefix_at(pre, Y, ex(ua), 1)   # column, voxel column
        cp = _prefix(row, 0)
        I = _prefix_at(cp, row, vb, 0) - _prefix_at(cp, row, va, 0)           # noqa: E741
        axis = (qy - s[1] if ysl else qx - s[0]).abs()
        out += I * (g.d[1] if ysl else g.d[0]) / axis * ((qx - s[0]) ** 2 + (qy - s[1]) ** 2 + (qz - s[2]) ** 2).sqrt()
    return out.reshape(-1)


def _ct4_backward(g, P, y, kerroin):
    nx, ny, nz = g.n
    y = y.reshape(P.views, P.nc * P.nr)
    out = torch.zeros(nz, ny, nx, device=DEV, dtype=F64)
    qx, qy, qz = _centres(g, 0)[None, None, :], _centres(g, 1)[None, :, None], _centres(g, 2)[:, None, None]
    for v in range(P.views):
        s = P.xy[v, :3]
        u, w, t = _onto_panel(P, v, qx, qy, qz)
        u = u.expand_as(w)
        good = (u >= 0) & (u <= P.nr) & (w >= 0) & (w <= P.nc)
        fu, fw = (u - .5).floor(), (w - .5).floor()
        au, aw = u - .5 - fu, w - .5 - fw
        val = 0
        for e in (0, 1):
            for f in (0, 1):
                at = (fu.long() + e).clamp(0, P.nr - 1) + (fw.long() + f).clamp(0, P.nc - 1) * P.nr
                val = val + y[v][at] * (au if e else 1 - au) * (aw if f else 1 - aw)
        out += torch.where(good, val * ((qx - s[0]) ** 2 + (qy - s[1]) ** 2 + (qz - s[2]) ** 2).sqrt() * t ** 3,
                           torch.zeros_like(val))
    return out.reshape(-1) * kerroin


def _tv_gradient(x, smooth):
    """x: (z, y, x); neighbours outside read the edge voxel."""
    p = torch.nn.functional.pad(x[None, None], (1,) * 6, mode="replicate")[0, 0]

    def at(i, j, k):
        nz, ny, nx = x.shape
        return p[1 + k:1 + k + nz, 1 + j:1 + j + ny, 1 + i:1 + i + nx]

    c, px, py, pz = at(0, 0, 0), at(1, 0, 0), at(0, 1, 0), at(0, 0, 1)
    mx, my, mz = at(-1, 0, 0), at(0, -1, 0), at(0, 0, -1)
    n = lambda a, b, d: (a * a + b * b + d * d + smooth).sqrt()  # noqa: E731
    return ((3 * c - px - py - pz) / n(px - c, py - c, pz - c) +
            (c - mx) / n(c - mx, at(-1, 1, 0) - mx, at(-1, 0, 1) - mx) +
            (c - my) / n(at(1, -1, 0) - my, c - my, at(0, -1, 1) - my) +
            (c - mz) / n(at(1, 0, -1) - mz, at(0, 1, -1) - mz, c - mz) + 1e-7)


def _conv(x, w):
    """3 x 3 x 3 convolution of (B, Z, Y, X, ci) with (27, co, ci), zero outside."""
    B, Z, Y, X, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = 0
    for t in range(27):
        k, j, i = t // 9, t // 3 % 3, t % 3
        out = out + p[:, k:k + Z, j:j + Y, i:i + X] @ w[t].T
    return out


class _Conv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b):
        ctx.save_for_backward(x, w)
        return _conv(x, w) + b

    @staticmethod
    def backward(ctx, dz):
        x, w = ctx.saved_tensors
        B, Z, Y, X, ci = x.shape
        dx = _conv(dz, w.flip(0).transpose(1, 2))
        p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        d = dz.reshape(-1, dz.shape[-1])
        dw = torch.stack([d.T @ p[:, t // 9:t // 9 + Z, t // 3 % 3:t // 3 % 3 + Y, t % 3:t % 3 + X].reshape(-1, ci)
                          for t in range(27)])
        return dx, dw, d.sum(0)


def _pool(x):
    B, Z, Y, X, C = x.shape
    return x.reshape(B, Z // 2, 2, Y // 2, 2, X // 2, 2, C).mean((2, 4, 6))


def _up(x):
    for d in (1, 2, 3):
        x = x.repeat_interleave(2, d)
    return x


def _unet_exact(c, seed):
    osem, target, sens, sd = _unet_inputs(c, seed)
    B, X, Y, Zs = c["batch"], c["X"], c["Y"], c["Zs"]
    Z = (Zs + 3) // 4 * 4
    vol = lambda t: torch.nn.functional.pad(t.to(F64).reshape(-1, Zs, Y, X), (0, 0, 0, 0, 0, Z - Zs))  # noqa: E731
    scale = 1.0 / osem.to(F64).mean(1)[:, None, None, None]
    x0 = torch.zeros(B, Z, Y, X, 16, device=DEV, dtype=F64)
    x0[..., 0] = vol(osem) * scale
    x0[..., 1] = vol(sens)
    par = {k: torch.from_numpy(np.asarray(v)).to(DEV, F64).requires_grad_() for k, v in sd.items()}
    f = lambda i, t: torch.relu(_Conv.apply(t, par[f"w{i}"], par[f"b{i}"]))  # noqa: E731
    with torch.enable_grad():
        a2 = f(1, f(0, x0))
        a4 = f(3, f(2, _pool(a2)))
        a6 = f(5, f(4, _pool(a4)))
        a8 = f(7, f(6, torch.cat([_up(a6), a4], -1)))
        a10 = f(9, f(8, torch.cat([_up(a8), a2], -1)))
        pred = x0[..., 0] + par["head_b"] + a10 @ par["head_w"]
        r = (pred - vol(target) * scale)[:, :Zs]
        (r * r).mean().backward()
    return (pred.detach().reshape(-1), [par[f"w{i}"].grad.reshape(-1) for i in range(10)],
            [par[f"b{i}"].grad for i in range(10)], par["head_w"].grad, par["head_b"].grad)


def _osem_exact(o, c, seed):
    g = _Grid(o)
    x = _frame_images(c, seed).to(F64)
    m = _frame_measurements(c, c["nsinos"], seed)
    rays0 = 0
    for s in range(c["subsets"]):
        p, q = _pet_rays(o, c, s)
        y = m[:, rays0:rays0 + p.shape[0]].to(F64)
        rays0 += p.shape[0]
        back = torch.zeros_like(x)
        sens = torch.zeros(g.voxels, device=DEV, dtype=F64)
        step = max(1, int(3e7 / (sum(g.n) + 3)))
        for r in range(0, p.shape[0], step):
            at = slice(r, min(r + step, p.shape[0]))
            ind, ele, inv, _, _ = _siddon(g, p[at], q[at])
            le = ele * inv[:, None]
            ray, col = (le > 0).nonzero(as_tuple=True)
            vox, le = ind[ray, col], le[ray, col]
            sens.index_add_(0, vox, le)
            for f in range(c["frames"]):
                fp = torch.zeros(at.stop - at.start, device=DEV, dtype=F64).index_add_(0, ray, le * x[f, vox])
                ratio = y[f, at] / (fp + g.eps)
                back[f].index_add_(0, vox, le * ratio[ray])
        x = x / sens.clamp_min(g.eps) * (back + g.eps)
    return x


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "conv":
        x, w, b, mask = _conv_inputs(c, seed)
        out = _conv(x.to(F64).reshape(c["batch"], c["Z"], c["Y"], c["X"], c["cin"]), w.to(F64))
        if b is not None:
            out = torch.relu(out + b.to(F64))
        out = out.reshape(-1)
        return out if mask is None else torch.where(mask > 0, out, torch.zeros_like(out))
    if k == "unet":
        return _unet_exact(c, seed)
    o = _pet_options(c) if k in ("pet", "frames") else _ct_options(c)
    o.nMeas = np.asarray(o.nMeas).ravel()
    g = _Grid(o)
    if k == "frames":
        return _osem_exact(o, c, seed)
    s = _subset(c)
    if k == "pet":
        p, q = _pet_rays(o, c, s)
        x = _phantom(c["nx"], c["nx"], c["nz"], seed, 0.05, 0.6)
        x = (x.bfloat16() if c["read"] == "bf16" else x).to(F64)   # the option's reads, rounded once
        y = _pet_measurement(p.shape[0] * c["tof"], seed).to(F64)
        tof = _tof_of(o, c)
        if c["projector"] == 1:
            return _siddon_pair(g, p, q, x, y, tof)
        dL = float(np.float32(o.dL))
        return _interp_forward(g, p, q, x, dL, tof, True), _interp_backward(g, p, q, y, dL, tof)
    if k == "pdhg":
        P = _Panel(o, c, 0)
        x0, y, tau = _pdhg_start(c, seed)
        x0, y = x0.to(F64), y.to(F64)
        dual = (_bdd_forward(g, P, x0) - y) / 2.0
        n = g.n
        rhs = _bdd_backward(g, P, dual) + 0.05 * _tv_gradient(x0.reshape(n[2], n[1], n[0]), 1e-4).reshape(-1)
        u = (x0 - float(tau) * rhs).clamp_min(g.eps)
        return 2 * u - x0, u, dual
    P = _Panel(o, c, s)
    x = _phantom(c["nx"], c["nx"], c["nz"], seed, 0.01, 0.2).to(F64)
    y = _ct_measurement(P.views * P.nr * P.nc, seed).to(F64)
    if k == "bdd_fp":
        return _bdd_forward(g, P, x)
    if k == "bdd_bp":
        return _bdd_backward(g, P, y)
    dL = float(np.float32(o.dL))
    fp = torch.cat([_interp_forward(g, *_ct_rays(P, v), x, dL, None, False) for v in range(P.views)])
    return fp, _ct4_backward(g, P, y, float(np.ravel(o.kerroin)[0]))
