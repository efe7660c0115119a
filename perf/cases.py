"""Performance cases of the D3Q19 framework: what users have it do, from one
cavity step to a batched ensemble, through the public API of `lbm`.

listed() names the standing cases, draw() gives further ones of the same
ranges, prepare() builds what a program holds before the call, run() is one
pass, work() the bytes and operations that pass cannot do without, exact() the
same outputs in 64-bit torch arithmetic.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path.cwd() / "gpu-sims_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lbm  # noqa: E402

PREC = {"f32": lbm.PREC_F32, "f16s": lbm.PREC_F16S, "bf16s": lbm.PREC_BF16S}
EDGES = (32, 48, 64, 80, 96)  # cavity edges of the ensemble (lbm.configs)
SPHERE_TAU = 0.55


def listed():
    return [
        # one call of a small viewer or coupled solver: a single step of a lid
        # cavity, where launch and call latency are most of the time
        {"name": "cavity64_one_step", "kind": "box", "flow": "cavity", "nx": 64, "ny": 64, "nz": 64,
         "prec": "f32", "trt": False, "cs": 0.0, "steps": 1},
        # odd, ragged box with walls, an obstacle and Smagorinsky: sizes as
        # they come from a user's geometry
        {"name": "ragged_les_f32", "kind": "box", "flow": "channel", "nx": 161, "ny": 97, "nz": 75,
         "prec": "f32", "trt": False, "cs": 0.1, "steps": 32},
        # periodic Taylor-Green vortex with the wall-free TRT collision
        {"name": "tgv256_trt_f16", "kind": "box", "flow": "tgv", "nx": 256, "ny": 256, "nz": 256,
         "prec": "f16s", "trt": True, "cs": 0.0, "steps": 32},
        # the body-forced channel with a sphere, the framework's benchmark, in
        # fp32 and in 16-bit storage
        {"name": "channel_f32", "kind": "box", "flow": "channel", "nx": 512, "ny": 128, "nz": 128,
         "prec": "f32", "trt": False, "cs": 0.0, "steps": 20},
        {"name": "channel_f16", "kind": "box", "flow": "channel", "nx": 512, "ny": 128, "nz": 128,
         "prec": "f16s", "trt": False, "cs": 0.0, "steps": 20},
        # the same channel with a velocity inlet and a pressure outlet
        {"name": "duct_f16", "kind": "box", "flow": "duct", "nx": 512, "ny": 128, "nz": 128,
         "prec": "f16s", "trt": False, "cs": 0.0, "steps": 20},
        # training-data generation: lid cavities of mixed size advanced
        # together, every domain's moments read back at the end
        {"name": "ensemble32_f16", "kind": "ensemble", "domains": 32, "prec": "f16s", "steps": 1000},
        # large-eddy run with the learned closure at its default settings
        {"name": "closure128_f32", "kind": "closure", "n": 128, "prec": "f32", "variant": 0, "steps": 16},
        # the reference's wind tunnel at its desktop tier, a burst of substeps
        {"name": "tunnel_desktop", "kind": "tunnel", "nx": 256, "ny": 128, "nz": 128, "steps": 16},
        # a viewer's whole frame at the laptop tier: substeps, streamlines,
        # the raymarched image
        {"name": "frame_laptop", "kind": "frame", "nx": 128, "ny": 128, "nz": 128, "steps": 4,
         "count": 10000, "width": 1280, "height": 720},
        # one snapshot of the closure's training data: filtered moments and
        # samples of a fine field
        {"name": "snapshot256", "kind": "snapshot", "n": 256, "factor": 4, "samples": 4096},
        # the gradient of the closure network over one training batch
        {"name": "closure_grad_4k", "kind": "grad", "samples": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box"] * 5 + ["ensemble", "closure", "tunnel", "tunnel", "frame", "snapshot", "grad"])
    if kind == "box":
        flow = rng.choice(["cavity", "channel", "tgv", "duct"])
        nodes = 10.0 ** rng.uniform(4.7, 7.0)
        edge = nodes ** (1.0 / 3.0)
        long = rng.uniform(1.0, 3.0) if flow in ("channel", "duct") else rng.uniform(0.8, 1.25)
        nx = max(24, int(edge * long ** (2.0 / 3.0)))
        nx = rng.choice([nx, nx // 8 * 8, nx // 2 * 2 + 1])
        ny = max(16, int(edge * long ** (-1.0 / 3.0) * rng.uniform(0.8, 1.2)))
        nz = max(16, int(nodes / (nx * ny)))
        return {"kind": "box", "flow": flow, "nx": nx, "ny": ny, "nz": nz,
                "prec": rng.choice(["f32", "f16s", "f16s", "bf16s"]), "trt": rng.random() < 0.5,
                "cs": rng.choice([0.0, 0.0, 0.0, 0.1]), "steps": rng.choice([1, 4, 16, 20, 32, 50])}
    if kind == "ensemble":
        return {"kind": "ensemble", "domains": rng.randint(4, 32), "prec": rng.choice(["f32", "f16s", "bf16s"]),
                "steps": _log_int(rng, 50, 600)}
    if kind == "closure":
        return {"kind": "closure", "n": rng.choice([64, 96, 128, 100, 160, 75]), "prec": rng.choice(["f32", "f16s"]),
                "variant": rng.choice([0, 0, 8]), "steps": rng.randint(2, 24)}
    if kind == "tunnel":
        return {"kind": "tunnel", "nx": _log_int(rng, 64, 384), "ny": _log_int(rng, 48, 192),
                "nz": _log_int(rng, 32, 160), "steps": rng.randint(1, 24)}
    if kind == "frame":
        return {"kind": "frame", "nx": rng.randint(96, 256), "ny": rng.randint(64, 128), "nz": rng.randint(64, 128),
                "steps": rng.randint(1, 8), "count": _log_int(rng, 1000, 20000),
                "width": rng.randint(320, 1920), "height": rng.randint(200, 1080)}
    if kind == "snapshot":
        f = rng.choice([2, 3, 4, 8])
        return {"kind": "snapshot", "n": f * rng.randint(48 // f, 288 // f), "factor": f,
                "samples": _log_int(rng, 512, 65536)}
    return {"kind": "grad", "samples": _log_int(rng, 500, 300000)}


# ---- inputs ------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _axes(nx, ny, nz):
    ar = lambda n: torch.arange(n, device="cuda", dtype=torch.float64)  # noqa: E731
    return ar(nx)[None, None, :], ar(ny)[None, :, None], ar(nz)[:, None, None]


def _sphere(nx, ny, nz):
    """Solid sphere a quarter down the channel, its radius an eighth of the height."""
    x, y, z = _axes(nx, ny, nz)
    r = min(ny, nz) // 8
    inside = (x - nx // 4) ** 2 + (y - ny // 2) ** 2 + (z - nz // 2) ** 2 <= float(r * r)
    return inside.to(torch.uint8).contiguous()


def _airfoil(nx, ny, nz, aoa_deg, thickness=0.12):
    """Symmetric four-digit section, chord nx/4 at x = nx/4, extruded in z."""
    x, y, _ = _axes(nx, ny, 1)
    chord, a = 0.25 * nx, math.radians(aoa_deg)
    dx, dy = x + 0.5 - 0.25 * nx, y + 0.5 - 0.5 * ny
    s = (dx * math.cos(a) - dy * math.sin(a)) / chord + 0.5
    t = (dx * math.sin(a) + dy * math.cos(a)) / chord
    c = s.clamp(0.0, 1.0)
    half = 5.0 * thickness * (0.2969 * c.sqrt() - 0.126 * c - 0.3516 * c ** 2 + 0.2843 * c ** 3 - 0.1036 * c ** 4)
    inside = (s >= 0) & (s <= 1) & (t.abs() <= half)
    return inside.to(torch.uint8).expand(nz, ny, nx).contiguous()


def _box_fields(case, seed):
    """Initial density [nz, ny, nx] and velocity [3, nz, ny, nx], fp32."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _gen(seed)
    rho = torch.ones((nz, ny, nx), device="cuda")
    u = 1e-4 * torch.randn((3, nz, ny, nx), generator=g, device="cuda")
    if case["flow"] == "tgv":
        x, y, z = _axes(nx, ny, nz)
        x, y, z = (2.0 * math.pi * a / n for a, n in ((x, nx), (y, ny), (z, nz)))
        u[0] += (0.05 * torch.sin(x) * torch.cos(y) * torch.cos(z)).float()
        u[1] -= (0.05 * torch.cos(x) * torch.sin(y) * torch.cos(z)).float()
        rho += (3.0 * 0.05 ** 2 / 16.0 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)).float()
    if case["flow"] in ("channel", "duct"):
        u *= 1.0 - _sphere(nx, ny, nz).float()
    return rho, u


def _box_desc(case):
    """Keyword description of a box, shared by the lattice and exact()."""
    wall = np.zeros((6, 3))
    d = {"periodic": (0, 0, 0), "body_accel": (0.0, 0.0, 0.0), "open_x": (0, 0), "open_rho": (0.0, 0.0)}
    if case["flow"] == "cavity":
        wall[lbm.FACE_ZP] = (0.05, 0.0, 0.0)
        d["tau"] = 0.6
    elif case["flow"] == "channel":
        d.update(periodic=(1, 0, 0), body_accel=(1e-6, 0.0, 0.0), tau=SPHERE_TAU)
    elif case["flow"] == "duct":
        wall[lbm.FACE_XM] = (0.05, 0.0, 0.0)
        d.update(open_x=(lbm.OPEN_VELOCITY, lbm.OPEN_PRESSURE), open_rho=(0.0, 1.0), tau=SPHERE_TAU)
    else:
        d.update(periodic=(1, 1, 1), tau=0.52)
    d.update(wall_velocity=wall, smagorinsky_cs=case["cs"],
             collision=lbm.COLL_TRT if case["trt"] else lbm.COLL_BGK)
    return d


def _ensemble(case, seed):
    """Edges (fixed by the case), relaxation times (from the seed)."""
    edges = np.random.default_rng(2024).choice(EDGES, size=case["domains"])
    re = np.random.default_rng(seed).uniform(100.0, 1000.0, size=case["domains"])
    return edges, 0.5 + 3.0 * 0.05 * edges / re


def _network(seed):
    """A He-initialised closure network around plain Smagorinsky."""
    rng = np.random.default_rng(seed)
    nin, nh = lbm.CLOSURE_INPUTS, lbm.CLOSURE_HIDDEN
    w1 = rng.standard_normal(nh * nin) * math.sqrt(2.0 / nin)
    w2 = rng.standard_normal(nh * nh) * math.sqrt(2.0 / nh)
    w3 = 0.1 * rng.standard_normal(nh) * math.sqrt(1.0 / nh)
    mean = np.array([0.0] * 6 + [-8.0, 0.0, 0.0])
    scale = np.array([2.0] * 6 + [0.6, 2.0, 50.0])
    return np.concatenate([w1, 0.1 * rng.standard_normal(nh), w2, 0.1 * rng.standard_normal(nh), w3,
                           [math.log(math.e - 1.0)], mean, scale]).astype(np.float32)


def _turbulence(n, seed, rms=0.04):
    """Smooth random velocity [3, n, n, n], energy around wavenumber 4."""
    g = _gen(seed)
    k = torch.fft.fftfreq(n, d=1.0 / n, device="cuda")
    kr = torch.fft.rfftfreq(n, d=1.0 / n, device="cuda")
    kk = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2).sqrt()
    amp = kk * torch.exp(-((kk / 4.0) ** 2))
    u = torch.empty((3, n, n, n), device="cuda")
    for c in range(3):
        xi = torch.complex(torch.randn(kk.shape, generator=g, device="cuda"),
                           torch.randn(kk.shape, generator=g, device="cuda"))
        u[c] = torch.fft.irfftn(amp * xi, s=(n, n, n), dim=(0, 1, 2))
        u[c] *= rms / u[c].std()
    return u


def _samples(case, seed):
    """Training rows as closure_samples makes them: features of a random
    non-equilibrium flux, the Cs^2 ratio and the |S|^3 weight."""
    n, g = case["samples"], _gen(seed)
    s = torch.randn((n, 6), generator=g, device="cuda", dtype=torch.float64)
    s[:, :3] -= s[:, :3].mean(1, keepdim=True)
    mag = 10.0 ** (-3.5 + 0.3 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    rho = 1.0 + 0.005 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    x = _features(list((mag[:, None] * s).T), rho).T.float().contiguous()
    target = (torch.randn(n, generator=g, device="cuda") * 2.0 + 0.8).clamp(-50.0, 50.0)
    weight = (mag ** 3).float()
    return x, target, (weight / weight.mean()).contiguous()


def _tunnel(case, seed):
    rng = np.random.default_rng(seed)
    aoa = 4.0 + rng.uniform(-2.0, 2.0)
    speed, a = 0.04 * rng.uniform(0.9, 1.1), math.radians(aoa)
    u = tuple(float(np.float32(v)) for v in (speed * math.cos(a), speed * math.sin(a), 0.0))
    return aoa, u


def _ring(case, seed):
    """Streamline positions [count, 64, 4]: seeded over the whole domain."""
    g = _gen(seed + 5)
    size = torch.tensor([case["nx"], case["ny"], case["nz"], 128.0], device="cuda")
    p = torch.rand((case["count"], 1, 4), generator=g, device="cuda") * size
    p[..., 3] = p[..., 3].floor()
    return p.expand(-1, lbm.STREAMLINE_HISTORY, -1).contiguous()


def _camera(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    eye = (0.5 * nx, 0.8 * ny, 2.2 * max(nx, nz))
    return eye, lbm.camera(eye, (0.5 * nx, 0.5 * ny, 0.5 * nz), aspect=case["width"] / case["height"])


# ---- the pass ------------------------------------------------------------------

class _Device:
    """Device memory of a lattice as torch sees it (keeps the lattice alive)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": "<f4", "version": 3}


def _moments(lat):
    r, u = lat.device_moments()
    nx, ny, nz = lat.shape
    return (torch.as_tensor(_Device(lat, r, (nz, ny, nx)), device="cuda"),
            torch.as_tensor(_Device(lat, u, (3, nz, ny, nx)), device="cuda"))


def _host(rho, u):
    return rho.reshape(-1).cpu().numpy(), u.reshape(3, -1).T.contiguous().cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.Stream()
    st = {"kind": kind, "stream": stream, "case": case}
    ptr = stream.cuda_stream
    if kind == "box":
        d = _box_desc(case)
        lat = lbm.Lattice(nx=case["nx"], ny=case["ny"], nz=case["nz"], mode=lbm.MODE_PHYSICS,
                          precision=PREC[case["prec"]], **d)
        lat.set_stream(ptr)
        if case["flow"] in ("channel", "duct"):
            lat.set_flags(_sphere(case["nx"], case["ny"], case["nz"]).cpu().numpy())
        lat.init_from_moments(*_host(*_box_fields(case, seed)))
        st.update(lat=lat, out=_moments(lat))
    elif kind == "ensemble":
        edges, taus = _ensemble(case, seed)
        wall = np.zeros((6, 3))
        wall[lbm.FACE_ZP] = (0.05, 0.0, 0.0)
        b = lbm.Batch([lbm.default_desc(nx=int(e), ny=int(e), nz=int(e), mode=lbm.MODE_PHYSICS,
                                        precision=PREC[case["prec"]], collision=lbm.COLL_TRT, tau=float(t),
                                        wall_velocity=wall) for e, t in zip(edges, taus)])
        b.set_stream(ptr)
        b.init_equilibrium(-1, 1.0, (0.0, 0.0, 0.0))
        b.autotune(10)
        st.update(batch=b)
    elif kind == "closure":
        n = case["n"]
        lat = lbm.Lattice(nx=n, ny=n, nz=n, mode=lbm.MODE_PHYSICS, precision=PREC[case["prec"]],
                          periodic=(1, 1, 1), tau=0.502, smagorinsky_cs=0.1)
        lat.set_stream(ptr)
        lat.set_closure(_network(seed))
        lat.init_from_moments(*_host(torch.ones((n, n, n), device="cuda"), _turbulence(n, seed)))
        if case["variant"]:
            lat.set_step_variant(case["variant"])
        st.update(lat=lat, out=_moments(lat))
    elif kind in ("tunnel", "frame"):
        aoa, u = _tunnel(case, seed)
        lat = lbm.Lattice(nx=case["nx"], ny=case["ny"], nz=case["nz"], tau=0.6, u_inf=u)
        lat.set_stream(ptr)
        lat.set_flags(_airfoil(case["nx"], case["ny"], case["nz"], aoa).cpu().numpy())
        lat.init_equilibrium(1.0, u)
        st.update(lat=lat, out=_moments(lat))
        if kind == "frame":
            eye, inv = _camera(case)
            st.update(ring=_ring(case, seed), head=0, frame=1, d_u=lat.device_moments()[1],
                      view=lbm.velmag_params(inv_view_proj=inv, camera_pos=eye),
                      image=torch.empty((case["height"], case["width"], 4), device="cuda"))
    elif kind == "snapshot":
        n, f, m = case["n"], case["factor"], case["samples"]
        u = _turbulence(n, seed).contiguous()
        rho = (1.0 + 0.01 * torch.randn((n, n, n), generator=_gen(seed + 9), device="cuda")).contiguous()
        st.update(rho=rho, u=u, filt=torch.empty((10, (n // f) ** 3), device="cuda"),
                  x=torch.empty((m, lbm.CLOSURE_INPUTS), device="cuda"), t=torch.empty(m, device="cuda"),
                  w=torch.empty(m, device="cuda"))
    else:
        x, t, w = _samples(case, seed)
        tr = lbm.Trainer(_network(seed), lbm.adam_default())
        tr.set_stream(ptr)
        st.update(x=x, t=t, w=w, trainer=tr)
    torch.cuda.synchronize()
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind in ("box", "closure", "tunnel"):
        st["lat"].step(case["steps"])
        return st["out"]
    if kind == "ensemble":
        st["batch"].step(case["steps"])
        return [st["batch"].read_moments(d) for d in range(case["domains"])]
    ptr = st["stream"].cuda_stream
    if kind == "frame":
        shape = (case["nx"], case["ny"], case["nz"])
        st["lat"].step(case["steps"])
        lbm.streamline_advect(st["d_u"], shape, st["ring"].data_ptr(), case["count"], lbm.STREAMLINE_HISTORY,
                              st["head"], st["frame"], float(case["steps"]), stream=ptr)
        st["head"] = (st["head"] + 1) % lbm.STREAMLINE_HISTORY
        st["frame"] += 1
        lbm.render_velmag(st["d_u"], shape, st["view"], case["width"], case["height"],
                          st["image"].data_ptr(), stream=ptr)
        return (*st["out"], st["ring"], st["image"])
    if kind == "snapshot":
        n, f = case["n"], case["factor"]
        lbm.box_filter(st["rho"].data_ptr(), st["u"].data_ptr(), (n, n, n), f, st["filt"].data_ptr(), ptr)
        lbm.closure_samples(st["filt"].data_ptr(), (n // f,) * 3, 0.502, 0.1, 7, case["samples"],
                            st["x"].data_ptr(), st["t"].data_ptr(), st["w"].data_ptr(), ptr)
        return st["filt"], st["x"], st["t"], st["w"]
    n = case["samples"]
    return st["trainer"].grad(st["x"].data_ptr(), st["t"].data_ptr(), st["w"].data_ptr(), n, 1.0 / n)


def work(case):
    kind = case["kind"]
    if kind in ("box", "closure", "tunnel", "frame"):
        n = case["n"] ** 3 if kind == "closure" else case["nx"] * case["ny"] * case["nz"]
        eb = 4 if case.get("prec", "f32") == "f32" else 2
        per = 260 + (150 if case.get("cs") or kind == "closure" else 0) + (2 * 1344 if kind == "closure" else 0)
        w = {"bytes": n * ((38 * eb + 1) * case["steps"] + 16), "flops": n * per * case["steps"]}
        if kind == "frame":
            w["bytes"] += 12 * n + 16 * case["width"] * case["height"] + 2 * 16 * case["count"]
            w["flops"] += 128 * 90 * case["width"] * case["height"] // 2
        return w
    if kind == "ensemble":
        n = int((_ensemble(case, 0)[0].astype(np.int64) ** 3).sum())
        eb = 4 if case["prec"] == "f32" else 2
        return {"bytes": n * ((38 * eb + 1) * case["steps"] + 16), "flops": n * 300 * case["steps"]}
    if kind == "snapshot":
        n = case["n"] ** 3
        return {"bytes": 16 * n + 40 * n // case["factor"] ** 3 + 44 * case["samples"], "flops": 25 * n}
    return {"bytes": 44 * case["samples"] + 4 * 1409, "flops": 6 * 1344 * case["samples"]}


# ---- 64-bit results --------------------------------------------------------------

_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (1, -1, 0),
      (-1, 1, 0), (-1, -1, 0), (1, 0, 1), (1, 0, -1), (-1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1),
      (0, -1, -1)]
_OPP = [_C.index((-a, -b, -c)) for a, b, c in _C]
_W = [1.0 / 3.0] + [1.0 / 18.0] * 6 + [1.0 / 36.0] * 12


def _f32(v):
    return float(np.float32(v))


def _feq(rho, u):
    """Equilibrium [19, ...] of rho [...] and u [3, ...]."""
    c = torch.tensor(_C, device="cuda", dtype=torch.float64)
    w = torch.tensor(_W, device="cuda", dtype=torch.float64).reshape(-1, *[1] * rho.dim())
    cu = torch.tensordot(c, u, 1)
    return w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * (u * u).sum(0))


def _features(P, rho):
    xx, yy, zz, xy, xz, yz = P
    n = (xx * xx + yy * yy + zz * zz + 2.0 * (xy * xy + xz * xz + yz * yz)).sqrt() + 1e-30
    a, b, c, d, e, f = (v / n for v in P)
    t3 = (a ** 3 + b ** 3 + c ** 3 + 3.0 * (d * d * (a + b) + e * e * (a + c) + f * f * (b + c)) + 6.0 * d * e * f)
    return torch.stack([a, b, c, d, e, f, n.log(), t3, rho - 1.0])


def _net64(net):
    """Parameters of a network as the kernels use them: bf16 weights."""
    w = torch.tensor(net, device="cuda")
    r = w.bfloat16().double()
    w = w.double()
    return {"w1": r[:288].reshape(32, 9), "b1": w[288:320], "w2": r[320:1344].reshape(32, 32), "b2": w[1344:1376],
            "w3": r[1376:1408], "b3": w[1408], "mean": w[1409:1418], "scale": w[1418:1427]}


def _mlp(p, x):
    """Network output of features x [9, m]."""
    x = (x - p["mean"][:, None]) * p["scale"][:, None]
    h = (p["w1"] @ x + p["b1"][:, None]).clamp(min=0.0)
    h = (p["w2"] @ h + p["b2"][:, None]).clamp(min=0.0)
    return torch.nn.functional.softplus(p["w3"] @ h + p["b3"])


def _open_face(v, side, d):
    """Zou-He populations entering through x face `side` of v [19, nz, ny, nx]."""
    x, s = (0, 1) if side == 0 else (v.shape[-1] - 1, -1)
    at = [v[i, ..., x] for i in range(19)]
    m = sum(at[i] for i in range(19) if _C[i][0] == 0) + 2.0 * sum(at[i] for i in range(19) if _C[i][0] == -s)
    if d["open_x"][side] == lbm.OPEN_VELOCITY:
        u = [_f32(a) for a in d["wall_velocity"][side]]
        rho = m / (1.0 - s * u[0])
    else:
        rho = torch.full_like(m, _f32(d["open_rho"][side]))
        u = [s * (1.0 - m / rho), 0.0, 0.0]
    ny, nz = (0.5 * sum(_C[i][k] * at[i] for i in range(19) if _C[i][0] == 0) - rho * u[k] / 3.0 for k in (1, 2))
    new = {i: at[_OPP[i]] + 6.0 * _W[i] * rho * (s * u[0] + _C[i][1] * u[1] + _C[i][2] * u[2])
           - _C[i][1] * ny - _C[i][2] * nz for i in range(19) if _C[i][0] == s}
    for i, a in new.items():
        v[i, ..., x] = a


def _physics(rho, u, steps, d, tau, mask=None, net=None):
    """rho [B, nz, ny, nx] and u [3, B, ...] after `steps` textbook steps."""
    nz, ny, nx = rho.shape[-3:]
    solid = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda") if mask is None else mask.bool()
    f = _feq(rho, u)
    tau = tau if torch.is_tensor(tau) else torch.tensor(tau, device="cuda", dtype=torch.float64)
    tau = tau.reshape(-1, 1, 1, 1)
    acc = torch.tensor([_f32(a) for a in d["body_accel"]], device="cuda", dtype=torch.float64).reshape(3, 1, 1, 1, 1)
    forced = bool(acc.any())
    trt, cs, magic = d["collision"] == lbm.COLL_TRT, _f32(d["smagorinsky_cs"]), 3.0 / 16.0
    x, y, z = _axes(nx, ny, nz)
    links = []  # per direction: where the population bounces back, and the moving wall's term
    for i in range(1, 19):
        c = _C[i]
        out, term = torch.roll(solid, (c[2], c[1], c[0]), (0, 1, 2)), 0.0
        for axis, (pos, n) in enumerate(((x, nx), (y, ny), (z, nz))):
            if d["periodic"][axis] or not c[axis]:
                continue
            beyond = (pos == 0 if c[axis] > 0 else pos == n - 1).expand(nz, ny, nx)
            out = out & ~beyond | beyond
            wall = d["wall_velocity"][2 * axis + (0 if c[axis] > 0 else 1)]
            cu = 6.0 * _W[i] * sum(c[k] * _f32(wall[k]) for k in range(3))
            # a link through several faces takes z's velocity, then y's, then x's
            term = torch.where(beyond, cu, term) if cu or torch.is_tensor(term) else term
        links.append((out if bool(out.any()) else None, term))
    wt = torch.tensor(_W, device="cuda", dtype=torch.float64).reshape(-1, 1, 1, 1, 1)
    ct = torch.tensor(_C, device="cuda", dtype=torch.float64)
    opp = torch.tensor(_OPP, device="cuda")
    for _ in range(steps):
        v = torch.empty_like(f)
        v[0] = f[0]
        for i in range(1, 19):
            c, (out, term) = _C[i], links[i - 1]
            v[i] = torch.roll(f[i], (c[2], c[1], c[0]), (-3, -2, -1))
            if out is not None:
                v[i] = torch.where(out, f[_OPP[i]] + term, v[i])
        for side in range(2):
            if d["open_x"][side]:
                _open_face(v[:, 0], side, d)
        rho = v.sum(0)
        u = torch.tensordot(ct.T, v, 1) / rho + 0.5 * acc
        eq = _feq(rho, u)
        t = tau
        if cs > 0.0:
            ne = v - eq
            P = [sum(_C[i][a] * _C[i][b] * ne[i] for i in range(19) if _C[i][a] * _C[i][b])
                 for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
            q = (P[0] ** 2 + P[1] ** 2 + P[2] ** 2 + 2.0 * (P[3] ** 2 + P[4] ** 2 + P[5] ** 2)).sqrt()
            cs2 = cs * cs
            if net is not None:
                feats = _features([p.reshape(-1) for p in P], rho.reshape(-1))
                cs2 = cs2 * torch.cat([_mlp(net, x) for x in feats.split(1 << 20, 1)]).reshape(rho.shape)
            t = 0.5 * (t + (t * t + 18.0 * math.sqrt(2.0) * cs2 * q / rho).sqrt())
        om = 1.0 / t
        om_m = 1.0 / (magic / (t - 0.5) + 0.5) if trt else om
        src = 0.0
        if forced:
            cu, ca = torch.tensordot(ct, u, 1), torch.tensordot(ct, acc, 1)
            src = wt * rho * (3.0 * (ca - (u * acc).sum(0)) + 9.0 * cu * ca)
        if trt:
            w = v - eq
            wo = w[opp]
            f = v - 0.5 * om * (w + wo) - 0.5 * om_m * (w - wo)
            if forced:
                so = src[opp]
                f += (1.0 - 0.5 * om) * 0.5 * (src + so) + (1.0 - 0.5 * om_m) * 0.5 * (src - so)
        else:
            f = v - om * (v - eq) + (1.0 - 0.5 * om) * src
        del eq
    if mask is not None:
        rho, u = torch.where(solid, 0.0, rho), torch.where(solid, 0.0, u)
    return rho, u


def _tunnel_steps(case, seed):
    """rho, u of the reference's four-pass step (collide with u in binary16,
    clamped pull, boundaries, moments)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    aoa, ui = _tunnel(case, seed)
    solid = _airfoil(nx, ny, nz, aoa).bool()
    one = torch.ones((nz, ny, nx), device="cuda", dtype=torch.float64)
    inlet = torch.tensor(ui, device="cuda", dtype=torch.float64).reshape(3, 1, 1, 1)
    rho, u = one, inlet * one
    f = _feq(rho, u)
    ti = 1.0 / _f32(0.6)
    ar = [torch.arange(n, device="cuda") for n in (nx, ny, nz)]
    pad = torch.nn.functional.pad(solid[None, None].float(), (1,) * 6, value=1.0)[0, 0].bool()
    for _ in range(case["steps"]):
        f = (1.0 - ti) * f + ti * _feq(rho, u.float().half().double())
        g = torch.empty_like(f)
        for i, c in enumerate(_C):
            xi, yi, zi = ((ar[a] - c[a]).clamp(0, n - 1) for a, n in enumerate((nx, ny, nz)))
            g[i] = f[i].index_select(0, zi).index_select(1, yi).index_select(2, xi)
        f = g.clone()
        for i in range(1, 19):
            c = _C[i]
            hit = pad[1 + c[2]:nz + 1 + c[2], 1 + c[1]:ny + 1 + c[1], 1 + c[0]:nx + 1 + c[0]]
            f[_OPP[i]] = torch.where(hit, f[i], f[_OPP[i]])
        f[..., 0] = _feq(one[..., 0], u.new_tensor(ui).reshape(3, 1, 1) * one[..., 0])
        up = g[..., nx - 2]
        r = up.sum(0)
        vu = torch.tensordot(u.new_tensor(_C).T, up, 1) / r
        vu = torch.where(solid[..., nx - 2] | (r <= 1e-12), inlet[..., 0], vu)
        f[..., nx - 1] = _feq(one[..., 0], vu)
        for at, pairs in ((f[:, :, 0], ((4, 3), (8, 7), (10, 9), (17, 15), (18, 16))),
                          (f[:, :, ny - 1], ((3, 4), (7, 8), (9, 10), (15, 17), (16, 18))),
                          (f[:, 0], ((6, 5), (12, 11), (14, 13), (16, 15), (18, 17))),
                          (f[:, nz - 1], ((5, 6), (11, 12), (13, 14), (15, 16), (17, 18)))):
            for a, b in pairs:
                at[a] = at[b].clone()
        f *= ~solid
        rho = f.sum(0)
        u = torch.where(rho > 1e-12, torch.tensordot(u.new_tensor(_C).T, f, 1) / rho, 0.0)
    return rho, u


def _filter64(case, seed):
    """Favre box filter [10, nc] of the snapshot's fields."""
    n, f = case["n"], case["factor"]
    m = n // f
    box = lambda a: a.reshape(m, f, m, f, m, f).mean((1, 3, 5)).reshape(-1)  # noqa: E731
    u = _turbulence(n, seed).double()
    rho = (1.0 + 0.01 * torch.randn((n, n, n), generator=_gen(seed + 9), device="cuda")).double()
    r = box(rho)
    v = [box(rho * u[k]) / r for k in range(3)]
    tau = [box(rho * u[a] * u[b]) / r - v[a] * v[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    return torch.stack([r, *v, *tau])


def _grad64(case, seed):
    x, t, w = (a.double() for a in _samples(case, seed))
    p = _net64(_network(seed))
    leaves = [p[k].requires_grad_() for k in ("w1", "b1", "w2", "b2", "w3", "b3")]
    loss = (w * (_mlp(p, x.T) - t) ** 2).sum() / case["samples"]
    loss.backward()
    return torch.cat([a.grad.reshape(-1) for a in leaves]), float(loss.detach())


def exact(case, seed):
    """What run() returns for a new state, in 64 bits."""
    kind = case["kind"]
    if kind == "box":
        d = _box_desc(case)
        rho, u = _box_fields(case, seed)
        mask = _sphere(case["nx"], case["ny"], case["nz"]) if case["flow"] in ("channel", "duct") else None
        rho, u = _physics(rho.double()[None], u.double()[:, None], case["steps"], d, _f32(d["tau"]), mask)
        return rho[0], u[:, 0]
    if kind == "ensemble":
        edges, taus = _ensemble(case, seed)
        wall = np.zeros((6, 3))
        wall[lbm.FACE_ZP] = (0.05, 0.0, 0.0)
        d = {"periodic": (0, 0, 0), "body_accel": (0.0, 0.0, 0.0), "open_x": (0, 0), "wall_velocity": wall,
             "smagorinsky_cs": 0.0, "collision": lbm.COLL_TRT}
        got = [None] * len(edges)
        for e in sorted(set(int(v) for v in edges)):
            ids = [i for i, v in enumerate(edges) if v == e]
            rho = torch.ones((len(ids), e, e, e), device="cuda", dtype=torch.float64)
            tau = torch.tensor([_f32(taus[i]) for i in ids], device="cuda", dtype=torch.float64)
            rho, u = _physics(rho, torch.zeros((3, *rho.shape), device="cuda", dtype=torch.float64), case["steps"],
                              d, tau)
            for k, i in enumerate(ids):
                got[i] = (rho[k].reshape(-1), u[:, k].reshape(3, -1).T.contiguous())
        return got
    if kind == "closure":
        n = case["n"]
        d = {"periodic": (1, 1, 1), "body_accel": (0.0, 0.0, 0.0), "open_x": (0, 0), "wall_velocity": np.zeros((6, 3)),
             "smagorinsky_cs": 0.1, "collision": lbm.COLL_BGK}
        rho = torch.ones((1, n, n, n), device="cuda", dtype=torch.float64)
        rho, u = _physics(rho, _turbulence(n, seed).double()[:, None], case["steps"], d, _f32(0.502),
                          net=_net64(_network(seed)))
        return rho[0], u[:, 0]
    if kind == "tunnel":
        return _tunnel_steps(case, seed)
    if kind == "frame":
        # positions and image follow binary16 velocities and cut off at
        # thresholds: they have no value of their own in 64 bits
        return (*_tunnel_steps(case, seed), None, None)
    if kind == "snapshot":
        return _filter64(case, seed), None, None, None
    return _grad64(case, seed)
