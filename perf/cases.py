"""Performance cases: the work a user of seismic_engine has it do, through its
public entry points, from a small modelling call to a checkpointed gradient of
a large grid.

Operations (case["op"]):
  shot        shot_forward: one forward shot, seismograms and final wavefield
  rtm         rtm_shot: forward shot with snapshots, exact adjoint with imaging
  fwi         fwi.modeling and its backward (torch.autograd) for several shots
  fwi_ckpt    fwi.fwi_gradient with checkpointing: misfit and gradient
  ray_setup   CSRMatrix.build_ray_matrix, the starting model's times A m and the right-hand side A^T d
  tomo_cg     normal_cg_device: Jacobi-CG on the damped ray normal equations
  update_cg   normal_cg_device: the model update (I + L^T L) x = g
  inversion   AdjointStateInversion.run: one iteration on sampled-ray picks
  net_apply   LearnedPreconditioner: z = M r
  net_train   LearnedPreconditioner: z = M r and the weights' gradients

`exact` restates each operation in FP64 with plain torch.
"""
import math
import os
import sys
from types import SimpleNamespace

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "03-seismic-tomography-compute_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import seismic_engine as se  # noqa: E402
from seismic_engine import _lib, fwi, precond  # noqa: E402
from seismic_engine.inversion import AdjointStateInversion  # noqa: E402
from seismic_engine.workloads import ReceiverGrid, ShotSpec, ricker  # noqa: E402

DEV = "cuda"
SNAP = {"bf16": _lib.ST_SNAP_BF16, "fp16": _lib.ST_SNAP_FP16, "fp32": _lib.ST_SNAP_FP32}
D_CELL = 10.0   # cell size of the wave cases, m
DT = 0.0009     # s: Courant number 0.45 at 5000 m/s
LAM = 1e-2      # damping of the tomography systems


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a quick modelling call on a small box with the default sponge rule: launches and latency decide
        _wave("shot_small", "shot", 48, 40, 56, 200, sponge="reference", width=6),
        # the 128^3 plain forward modelling workload, 64 x 64 receivers
        _wave("shot_128", "shot", 128, 128, 128, 500),
        # the 256^3 single-shot RTM with BF16 snapshots (the headline workload), fewer steps
        _wave("rtm_256", "rtm", 256, 256, 256, 200, snap="bf16"),
        # a migration on a survey-shaped box whose extents divide by nothing
        _wave("rtm_ragged", "rtm", 150, 203, 171, 160, snap="fp16"),
        # the 192^3 FWI workload through torch.autograd with FP32 snapshots: two of its shots
        _wave("fwi_192", "fwi", 192, 192, 192, 150, snap="fp32", shots=2),
        # one shot of a large adjoint step: more history than is stored, recomputed from checkpoints
        _wave("fwi_ckpt_384", "fwi_ckpt", 384, 384, 320, 96, snap="bf16", segment=16, slots=4),
        # setting up a tomography system: the ray matrix of 500k rays on 50^3 cells, A m and A^T d
        dict(name="ray_setup_50", op="ray_setup", n=50, rays=500_000),
        # the first iterations of the traveltime tomography solve, 2M rays on 100^3 cells (a solve to 1e-6 takes
        # thousands; FP32 iterates of more than about ten are no longer the FP64 ones)
        dict(name="tomo_cg_100", op="tomo_cg", n=100, rays=2_000_000, iters=10),
        # iterations of the model update on the 256^3 inversion grid (7 entries per row)
        dict(name="update_cg_256", op="update_cg", nx=256, ny=256, nz=256, iters=40),
        # one iteration of the inversion driver: 2000 sources x 1000 ocean-bottom stations on 100^3 cells
        dict(name="inversion_100", op="inversion", n=100, sources=2000, stations=1000),
        # the learned preconditioner inside a solve on 100^3 cells
        dict(name="net_apply_100", op="net_apply", nx=100, ny=100, nz=100, layers=2),
        # one sample of its training on 32^3 cells: forward and backward
        dict(name="net_train_32", op="net_train", nx=32, ny=32, nz=32, layers=2),
    ]


def _wave(name, op, nx, ny, nz, nt, snap=None, sponge="stable", width=20, shots=1, segment=0, slots=0):
    c = dict(op=op, nx=nx, ny=ny, nz=nz, nt=nt, sponge=sponge, width=width)
    if name is not None:
        c["name"] = name
    if snap is not None:
        c["snap"] = snap
    if op == "fwi":
        c["shots"] = shots
    if op == "fwi_ckpt":
        c["segment"], c["slots"] = segment, slots
    return c


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    op = rng.choice(["shot", "shot", "rtm", "rtm", "fwi", "fwi_ckpt", "ray_setup", "tomo_cg", "update_cg",
                     "inversion", "net_apply", "net_train"])
    if op in ("shot", "rtm", "fwi", "fwi_ckpt"):
        lo = {"shot": 40, "rtm": 64, "fwi": 64, "fwi_ckpt": 128}[op]
        hi = {"shot": 320, "rtm": 300, "fwi": 224, "fwi_ckpt": 384}[op]
        n = log_int(lo, hi)
        nx, ny, nz = (max(lo, min(hi, int(n * rng.uniform(0.7, 1.3)))) for _ in range(3))
        snap = None if op == "shot" else rng.choice(["bf16", "bf16", "fp16", "fp32"])
        if op in ("fwi", "fwi_ckpt"):  # gradients need snapshot rows of a multiple of 16 bytes
            nz -= nz % 8
        elif rng.random() < 0.5:
            nz -= nz % 4
        # steps: a pass no longer than the listed ones', a snapshot store of at most 12 GB
        cost = {"shot": 1, "rtm": 3, "fwi": 4, "fwi_ckpt": 5}[op]
        most = 5e9 / cost / (nx * ny * nz)
        if op in ("rtm", "fwi"):
            most = min(most, 12e9 / (nx * ny * nz * (4 if snap == "fp32" else 2)))
        nt = max(9, min(int(most), log_int(40, 400)))
        width = min(20, min(nx, ny, nz) // 6)
        sponge = "reference" if op == "shot" and nt <= 200 and rng.random() < 0.5 else "stable"
        return _wave(None, op, nx, ny, nz, nt, snap=snap, sponge=sponge, width=width if sponge == "stable" else 6,
                     shots=rng.randint(1, 2), segment=rng.choice([8, 15, 16, 24]), slots=rng.randint(2, 6))
    if op in ("ray_setup", "tomo_cg"):
        n = log_int(20, 64 if op == "ray_setup" else 100)
        c = dict(op=op, n=n, rays=int(n ** 3 * rng.uniform(1.5, 4.0 if n < 64 else 2.0)))
        if op == "tomo_cg":
            c["iters"] = rng.randint(5, 10)
        return c
    if op == "update_cg":
        nx, ny, nz = (log_int(32, 256) for _ in range(3))
        return dict(op=op, nx=nx, ny=ny, nz=nz, iters=rng.randint(15, 40))
    if op == "inversion":
        return dict(op=op, n=log_int(24, 100), sources=log_int(50, 2000), stations=log_int(50, 1000))
    nx, ny, nz = (log_int(16, 110 if op == "net_apply" else 48) for _ in range(3))
    return dict(op=op, nx=nx, ny=ny, nz=nz, layers=rng.randint(1, 3))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _smooth(shape, coarse, g, dtype=torch.float32):
    """A smooth random field of unit scale: coarse normal values, interpolated."""
    size = [max(2, -(-s // coarse)) for s in shape]
    c = torch.randn([1, 1] + size, generator=g, device=DEV, dtype=dtype)
    return torch.nn.functional.interpolate(c, size=list(shape), mode="trilinear", align_corners=True)[0, 0]


def _velocity(case, g):
    """Four layers 1500 .. 4500 m/s with a smooth perturbation of a few percent (FP32, below 5000 m/s)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    layer = torch.arange(nz, device=DEV) * 4 // nz
    v = 1500.0 + 1000.0 * layer.to(torch.float32)
    return (v * (1.0 + 0.03 * _smooth((nx, ny, nz), 16, g).clamp(-3, 3))).contiguous()


def _receivers(case):
    step = 3 if min(case["nx"], case["ny"]) < 64 else 2
    return ReceiverGrid(0, step, case["nx"] // step, 0, step, case["ny"] // step, 5)


def _shots(case, seed):
    r = np.random.default_rng(seed)
    w = ricker(15.0 if case["nt"] > 100 else 30.0, DT, case["nt"])
    nx, ny = case["nx"], case["ny"]
    src = [(int(nx * r.uniform(0.3, 0.7)), int(ny * r.uniform(0.3, 0.7)), 5) for _ in range(case.get("shots", 1))]
    return [ShotSpec(s, w, _receivers(case)) for s in src]


def _arrivals(case, shot, g):
    """Receiver data FP32 [nt, nrec]: Ricker arrivals with moveout, plus a little noise."""
    xyz = torch.from_numpy(shot.rec.coords()).to(DEV, torch.float32)
    off = torch.hypot(xyz[:, 0] - shot.src[0], xyz[:, 1] - shot.src[1]) * D_CELL
    t = torch.arange(case["nt"], device=DEV, dtype=torch.float32)[:, None] * DT
    out = 0.01 * torch.randn((case["nt"], off.numel()), generator=g, device=DEV)
    for depth, amp in ((0.0, 1.0), (400.0, 0.5), (900.0, -0.3)):
        arrive = 0.04 + torch.sqrt(off * off + 4 * depth * depth) / 2200.0
        a = (math.pi * 15.0 * (t - arrive)) ** 2
        out += amp * (1 - 2 * a) * torch.exp(-a)
    return out.contiguous()


def _wave_inputs(case, seed):
    g = _gen(seed)
    v = _velocity(case, g)
    shots = _shots(case, seed)
    return v, shots, [_arrivals(case, s, g) for s in shots]


def _ray_inputs(case, seed):
    """Ray endpoints (FP64, device), data d (traveltimes of a smooth model sampled along the rays, 1% noise) and
    that model."""
    n = case["n"]
    ends = torch.from_numpy(se.workloads.ray_endpoints(case["rays"], n, seed)).to(DEV)
    g = _gen(seed)
    model = _smooth((n, n, n), 8, g).reshape(-1)
    d = torch.zeros(case["rays"], device=DEV)
    for k in range(32):
        p = ends[:, :3] + (k + 0.5) / 32 * (ends[:, 3:] - ends[:, :3])
        c = p.floor().clamp_(0, n - 1).long()
        d += model[(c[:, 0] * n + c[:, 1]) * n + c[:, 2]]
    d *= ((ends[:, 3:] - ends[:, :3]).norm(dim=1) / 32).float()
    return ends, d + 0.01 * d.std() * torch.randn(d.shape, generator=g, device=DEV), model


def _pick_inputs(case, seed):
    """Sources below an ocean-bottom station array, one pick per pair; vp = water over a gradient, perturbed 5%."""
    n, d = case["n"], 200.0
    r = np.random.default_rng(seed)
    ext = n * d
    floor = min(4000.0, 0.25 * ext)
    src = np.stack([r.uniform(0, ext, case["sources"]), r.uniform(0, ext, case["sources"]),
                    r.uniform(floor, ext, case["sources"])], axis=1)
    sta = np.stack([r.uniform(0, ext, case["stations"]), r.uniform(0, ext, case["stations"]),
                    np.full(case["stations"], floor)], axis=1)
    src_xyz = np.repeat(src, case["stations"], axis=0)
    sta_xyz = np.tile(sta, (case["sources"], 1))
    weight = r.uniform(0.5, 1.5, src_xyz.shape[0])
    z = torch.arange(n, device=DEV, dtype=torch.float64) * d
    col = torch.where(z < floor, 1500.0, (3000.0 * (1.0 + 0.3 * (z - floor) / 5000.0)).clamp(max=8500.0))
    vp = col * (1.0 + 0.05 * _smooth((n, n, n), 8, _gen(seed), torch.float64).clamp(-3, 3))
    straight = np.sqrt(((src_xyz - sta_xyz) ** 2).sum(axis=1))
    observed = straight / 4000.0 * (1.0 + 0.02 * r.standard_normal(straight.size))
    return (n, n, n, d, d, d, 0.0, 0.0, 0.0), src_xyz, sta_xyz, weight, vp.cpu().numpy(), observed


def _net_inputs(case, seed):
    g = _gen(seed)
    n = case["nx"] * case["ny"] * case["nz"]
    dinv = 1.0 / (torch.exp(1.5 * torch.randn(n, generator=g, device=DEV) + 4.0) + LAM)
    r = torch.randn(n, generator=g, device=DEV) / dinv.sqrt()
    return r, dinv, torch.randn(n, generator=g, device=DEV)


def _driver(model, rays, observed, weights):
    return AdjointStateInversion(model, None, None, max_iterations=1, step_length=10.0, smoothing_sigma=2.0,
                                 misfit_type="l2", rays=rays, observed=observed, weights=weights)


class _DeviceArray:
    """A device array of `owner` as seen by torch.as_tensor (no copy; the tensor keeps this object, and so the
    owner, alive)."""

    def __init__(self, owner, ptr, shape, typestr, strides=None):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False),
                                         "version": 3, "strides": strides}


def prepare(case, seed):
    op = case["op"]
    st = {"case": case}
    if op in ("shot", "rtm", "fwi", "fwi_ckpt"):
        v, shots, data = _wave_inputs(case, seed)
        nx, ny, nz = v.shape
        solver = se.WaveEquationSolver(
            se.GridParams(nx, ny, nz, D_CELL, D_CELL, D_CELL),
            se.SolverConfig(dt=DT, nt=case["nt"], sponge_width=case["width"], sponge_mode=case["sponge"]))
        fwi.set_velocity_device(solver, v)
        st.update(solver=solver, shots=shots, data=data)
        if op == "shot":
            st["seis"] = torch.zeros((case["nt"], shots[0].rec.count), device=DEV)
        elif op == "rtm":
            st["out"] = [torch.zeros(v.numel(), device=DEV) for _ in range(3)]
        elif op == "fwi":
            st["v"] = v
            st["data"] = torch.stack(data)
        elif op == "fwi_ckpt":
            st["v"] = v
    elif op in ("ray_setup", "tomo_cg"):
        st["ends"], st["d"], st["model"] = _ray_inputs(case, seed)
        st["x"] = torch.zeros(case["n"] ** 3, device=DEV)
        if op == "ray_setup":
            st["times"] = torch.zeros(case["rays"], device=DEV)
        else:
            st["A"] = se.CSRMatrix()
            st["A"].build_ray_matrix(st.pop("ends"), case["n"], case["n"], case["n"])
    elif op == "update_cg":
        shape = case["nx"], case["ny"], case["nz"]
        n = shape[0] * shape[1] * shape[2]
        L = se.CSRMatrix()
        L.build_fd_stencil_7point(*shape, np.full(n, 1.0), 1.0, 1.0, 1.0, 1.0)
        L.add_diagonal(-2.0)  # the 7-point Laplacian
        st.update(L=L, g=_smooth(shape, 4, _gen(seed)).reshape(-1).contiguous(), x=torch.zeros(n, device=DEV))
    elif op == "inversion":
        m, src, sta, weight, vp, observed = _pick_inputs(case, seed)
        rays = se.SampledRays(m, src, sta, weight)
        model = SimpleNamespace(nx=m[0], ny=m[1], nz=m[2], dx=m[3], dy=m[4], dz=m[5], origin_x=0.0, origin_y=0.0,
                                origin_z=0.0, vp=vp, vp_min=1450.0, vp_max=8500.0)
        st.update(model=model, vp=vp, driver=_driver(model, rays, observed, weight))
    else:
        net = precond.LearnedPreconditioner(case["nx"], case["ny"], case["nz"], layers=case["layers"], seed=seed % 1000)
        st["r"], st["dinv"], st["dz"] = _net_inputs(case, seed)
        st.update(net=net, z=torch.zeros_like(st["r"]))
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case = st["case"]
    op = case["op"]
    nt = case.get("nt")
    if op == "shot":
        s, sh = st["solver"], st["shots"][0]
        se.shot_forward(s, sh.src, sh.wavelet, nt, sh.rec, seis=st["seis"])
        L = se.field_layout(s.nx, s.ny, s.nz)
        strides = (4 * L["plane"], 4 * L["NZP"], 4)
        ptr = s.device_field_ptr(_lib.ST_FIELD_CURRENT) + 4 * (L["plane"] + L["NZP"] + L["ZOFF"])
        field = torch.as_tensor(_DeviceArray(s, ptr, (s.nx, s.ny, s.nz), "<f4", strides), device=DEV)
        return {"seis": st["seis"], "field": field}
    if op == "rtm":
        sh = st["shots"][0]
        image, illum, refl = st["out"]
        se.rtm_shot(st["solver"], sh.src, sh.wavelet, nt, sh.rec, st["data"][0], image, illum, refl,
                    snap_kind=SNAP[case["snap"]])
        return {"image": image, "illum": illum, "refl": refl}
    if op == "fwi":
        v = st["v"].clone().requires_grad_(True)
        seis = fwi.modeling(v, st["solver"], st["shots"], nt, snap_kind=SNAP[case["snap"]])
        loss = 0.5 * ((seis - st["data"]) ** 2).sum()
        loss.backward()
        return {"seis": seis.detach(), "grad": v.grad}
    if op == "fwi_ckpt":
        sh = st["shots"][0]
        grad = torch.zeros(st["v"].numel(), device=DEV)
        torch.cuda.current_stream().synchronize()  # the solver works on a stream of its own
        misfit = fwi.fwi_gradient(st["solver"], sh.src, sh.wavelet, nt, sh.rec, st["data"][0], grad,
                                  snap_kind=SNAP[case["snap"]], checkpoint=(case["segment"], case["slots"]))
        return {"misfit": misfit, "grad": grad}
    if op == "ray_setup":
        n = case["n"]
        A = st["A"] = se.CSRMatrix()
        A.build_ray_matrix(st["ends"], n, n, n)
        A.spmv_device(st["model"], st["times"])
        A.spmv_device(st["d"], st["x"], transpose=True)
        row_ptr = _DeviceArray(A, A.device_arrays()[0], (case["rays"] + 1,), "<i8")
        return {"row_ptr": torch.as_tensor(row_ptr, device=DEV), "times": st["times"], "rhs": st["x"]}
    if op == "tomo_cg":
        se.normal_cg_device(st["A"], st["d"], LAM, st["x"], case["iters"], 1e-30, True)
        return {"x": st["x"]}
    if op == "update_cg":
        se.normal_cg_device(st["L"], None, 1.0, st["x"], case["iters"], 1e-30, True, rhs=st["g"])
        return {"x": st["x"]}
    if op == "inversion":
        seen = {}
        st["model"].vp = st["vp"].copy()
        res = st["driver"].run(lambda it, misfit, gradient, step: seen.update(gradient=gradient, step=step))
        return {"vp": st["model"].vp, "gradient": seen["gradient"], "step": seen["step"],
                "misfit": res["final_misfit"]}
    net, r, dinv, z = st["net"], st["r"], st["dinv"], st["z"]
    net.forward(r, dinv, z)
    if op == "net_apply":
        return {"z": z}
    grads = [torch.zeros_like(p) for p in net.params]
    net.backward(st["dz"], r, dinv, grads)
    return {"z": z, "grads": grads}


# ------------------------------------------------------------------ work
def work(case):
    """Inputs once, outputs once; snapshots (history the adjoint needs) written and read once."""
    op = case["op"]
    if op in ("shot", "rtm", "fwi", "fwi_ckpt"):
        pts, nt = case["nx"] * case["ny"] * case["nz"], case["nt"]
        rec = _receivers(case).count * nt * 4
        step = 16.0 * pts * nt  # update of one point: 16 operations
        es = 4 if case.get("snap") == "fp32" else 2
        if op == "shot":
            return {"bytes": 8.0 * pts + rec, "flops": step}
        if op == "rtm":
            return {"bytes": 16.0 * pts + rec + 2.0 * es * pts * nt, "flops": 2 * step + 6.0 * pts * nt}
        shots = case.get("shots", 1)
        hist = es * pts * (nt if op == "fwi" else case["segment"])
        return {"bytes": shots * (8.0 * pts + 2 * rec + 2.0 * hist), "flops": shots * (3 * step + 15.0 * pts * nt)}
    if op in ("ray_setup", "tomo_cg"):
        n = case["n"]
        nnz = 1.8 * n * case["rays"]  # cells crossed by the rays
        if op == "ray_setup":
            return {"bytes": 8.0 * nnz + 48.0 * case["rays"] + 4.0 * (3 * case["rays"] + n ** 3), "flops": 12.0 * nnz}
        # one read of the matrix per iteration: it exceeds the caches
        return {"bytes": case["iters"] * 8.0 * nnz, "flops": case["iters"] * 4.0 * nnz}
    if op == "update_cg":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": case["iters"] * (7 * 8.0 + 8 + 4 * 8.0) * n, "flops": case["iters"] * 38.0 * n}
    if op == "inversion":
        samples = case["sources"] * case["stations"] * max(2.0, 0.13 * case["n"])
        picks = case["sources"] * case["stations"]
        return {"bytes": 12.0 * 4.0 * samples + 8.0 * (12 * picks + 6 * case["n"] ** 3), "flops": 12 * 2.0 * samples}
    n = case["nx"] * case["ny"] * case["nz"]
    conv = 2.0 * 27 * 32 * 32 * n * 2 * case["layers"] + 2.0 * 2 * 27 * 32 * n
    act = 64.0 * n * (2 * case["layers"] + 1)  # BF16 activations, kept for the backward pass
    if op == "net_apply":
        return {"bytes": 12.0 * n, "flops": conv}
    return {"bytes": 24.0 * n + 2 * act, "flops": 3 * conv}


# ------------------------------------------------------------------ FP64 restatements
def _sponge(case):
    """D of every point: 1 - 0.015 (w - d)^2 / w^2 within w cells of the nearest face."""
    w = case["width"]

    def dist(n):
        i = torch.arange(n, device=DEV)
        return torch.minimum(i, n - 1 - i)

    d = torch.minimum(torch.minimum(dist(case["nx"])[:, None, None], dist(case["ny"])[None, :, None]),
                      dist(case["nz"])[None, None, :])
    tab = torch.ones(w + 1, device=DEV, dtype=torch.float64)
    tab[:w] = 1.0 - 0.015 * (w - torch.arange(w, device=DEV, dtype=torch.float64)) ** 2 / (w * w)
    return tab[d.clamp(max=w)]


def _lap(u):
    """7-point Laplacian, zero outside."""
    out = -6.0 * u
    out[1:] += u[:-1]
    out[:-1] += u[1:]
    out[:, 1:] += u[:, :-1]
    out[:, :-1] += u[:, 1:]
    out[:, :, 1:] += u[:, :, :-1]
    out[:, :, :-1] += u[:, :, 1:]
    return out


class _Wave64:
    def __init__(self, case, v):
        self.case, self.nt = case, case["nt"]
        self.c = (v.double() * DT / D_CELL) ** 2  # cell size folded in
        self.D = _sponge(case)
        self.stable = case["sponge"] == "stable"
        R = _receivers(case)
        xyz = torch.from_numpy(R.coords()).to(DEV)
        self.rec = (xyz[:, 0] * case["ny"] + xyz[:, 1]) * case["nz"] + xyz[:, 2]

    def step(self, u, prev, force=None):
        out = 2.0 * u - self.D * prev + self.c * _lap(u)
        if force is not None:
            f = out.view(-1)
            f[self.rec] += self._weight()[self.rec] * force
        return out.mul_(self.D) if self.stable else out

    def _weight(self):
        # forcing enters the undamped update as c r (cell size squared restored)
        return self.c.view(-1) * D_CELL ** 2

    def forward(self, shot, keep=False):
        """Seismograms, final field and (keep) every field V_t before step t."""
        u = torch.zeros_like(self.c)
        prev = torch.zeros_like(u)
        w = shot.wavelet
        u[shot.src] += w[0]
        seis = torch.zeros((self.nt, self.rec.numel()), device=DEV, dtype=torch.float64)
        hist = []
        for t in range(self.nt):
            if keep:
                hist.append(u)
            out = self.step(u, prev)
            seis[t] = out.view(-1)[self.rec]
            if t + 1 < self.nt:
                out[shot.src] += w[t + 1]
            u, prev = out, u
        return seis, u, hist

    def backward(self, data, visit):
        """The adjoint from data [nt, nrec]; visit(t, mu_t) for every step."""
        mu = torch.zeros_like(self.c)
        nxt = torch.zeros_like(mu)
        f = mu.view(-1)
        f[self.rec] += self._weight()[self.rec] * (self.D.view(-1)[self.rec] if self.stable else 1.0) * data[-1]
        for t in range(self.nt - 1, -1, -1):
            visit(t, mu)
            mu, nxt = self.step(mu, nxt, data[t - 1] if t >= 1 else None), mu

    def gradient(self, shot, adj, hist):
        g = torch.zeros_like(self.c)

        def visit(t, mu):
            g.add_(mu / self.c * _lap(hist[t]))

        self.backward(adj, visit)
        # the cell size folded into c, d^2 in mu / c, d^2 in L, d in dc/dv = 2 v dt^2, comes back as d^-3
        return g * 2.0 * self.c.sqrt() * DT / D_CELL ** 3


def _ray_entries(ends, n, chunk=100_000):
    """(row, col, length) of every crossed cell, by sorting the face crossings of each ray."""
    rows, cols, vals = [], [], []
    for a in range(0, ends.shape[0], chunk):
        p0, d = ends[a:a + chunk, :3], ends[a:a + chunk, 3:] - ends[a:a + chunk, :3]
        face = torch.arange(n + 1, device=DEV, dtype=torch.float64)
        t = torch.cat([((face - p0[:, k:k + 1]) / d[:, k:k + 1]).nan_to_num_(1.0, 1.0, 1.0) for k in range(3)], dim=1)
        edge = torch.zeros((t.shape[0], 1), device=DEV, dtype=torch.float64)
        t = torch.cat([edge, t.clamp_(0.0, 1.0), edge + 1.0], dim=1).sort(dim=1).values
        mid = 0.5 * (t[:, 1:] + t[:, :-1])
        seg = (t[:, 1:] - t[:, :-1]) * d.norm(dim=1, keepdim=True)
        col = torch.zeros_like(mid, dtype=torch.int64)
        for k in range(3):
            col = col * n + (p0[:, k:k + 1] + mid * d[:, k:k + 1]).floor().clamp_(0, n - 1).long()
        i, j = torch.nonzero(seg > 0, as_tuple=True)
        rows.append((i + a).int())
        cols.append(col[i, j].int())
        vals.append(seg[i, j])
    return torch.cat(rows), torch.cat(cols), torch.cat(vals)


class _Rays64:
    def __init__(self, ends, n):
        self.row, self.col, self.val = _ray_entries(ends, n)
        self.shape = ends.shape[0], n ** 3

    def _sum(self, out_idx, in_idx, x, size, square=False):
        y = torch.zeros(size, device=DEV, dtype=torch.float64)
        for a in range(0, self.val.numel(), 1 << 26):
            b = slice(a, a + (1 << 26))
            v = self.val[b]
            y.index_add_(0, out_idx[b].long(), v * v if square else v * x[in_idx[b].long()])
        return y

    def mul(self, x):
        return self._sum(self.row, self.col, x, self.shape[0])

    def tmul(self, y):
        return self._sum(self.col, self.row, y, self.shape[1])

    def diag(self):
        return self._sum(self.col, None, None, self.shape[1], square=True)


def _cg64(op, b, dinv, iters):
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(iters):
        q = op(p)
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        z = dinv * r
        rz, old = torch.dot(r, z), rz
        p = z + rz / old * p
    return x


def _inversion64(case, seed):
    m, src, sta, weight, vp, observed = _pick_inputs(case, seed)
    n, h = m[0], m[3]
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    src, sta, w, obs, v0 = to(src), to(sta), to(weight), to(observed), to(vp).reshape(-1)
    cs = (src / h).clamp(0, n - 1).floor()
    cr = (sta / h).clamp(0, n - 1).floor()
    dist = (src - sta).norm(dim=1)
    steps = (dist / (5.0 * h)).floor().clamp(min=2).long()
    ds = dist / steps
    pick = torch.repeat_interleave(torch.arange(dist.numel(), device=DEV), steps)
    k = torch.arange(pick.numel(), device=DEV) - (steps.cumsum(0) - steps)[pick]
    frac = (k.double() + 0.5) / steps[pick]
    cell = torch.zeros_like(pick)
    for a in range(3):
        cell = cell * n + (cs[pick, a] + frac * (cr[pick, a] - cs[pick, a])).floor().long()

    def times(v):
        return torch.zeros_like(dist).index_add_(0, pick, ds[pick] / v[cell])

    def misfit(t):
        return float(0.5 * (w * (obs - t) ** 2).sum())

    t0 = times(v0)
    first = misfit(t0)
    res = (obs - t0) * w
    g = torch.zeros_like(v0).index_add_(0, cell, res[pick] * (-ds[pick] / v0[cell] ** 2) * w[pick]).view(n, n, n)
    i = torch.arange(n, device=DEV)
    off = (i[:, None] - i[None, :]).abs()
    G = torch.where(off <= 6, torch.exp(-(off.double() ** 2) / 8.0), 0.0)  # sigma 2, radius 6
    G = G / G.sum(dim=1, keepdim=True)
    for axis in range(3):
        g = torch.tensordot(g, G, dims=([0], [1]))  # the smoothed axis goes last: three turns restore the order
    v = v0.view(n, n, n)
    lap = torch.zeros_like(v)
    lap[1:-1] += v[2:] - 2 * v[1:-1] + v[:-2]
    lap[:, 1:-1] += v[:, 2:] - 2 * v[:, 1:-1] + v[:, :-2]
    lap[:, :, 1:-1] += v[:, :, 2:] - 2 * v[:, :, 1:-1] + v[:, :, :-2]
    g = (g - 1e-4 * lap).reshape(-1)
    g = g / g.abs().max()
    step = 10.0
    for _ in range(10):
        if misfit(times((v0 - step * g).clamp(1450.0, 8500.0))) < first:
            break
        step *= 0.5
    return {"vp": (v0 - step * g).clamp(1450.0, 8500.0).view(n, n, n), "gradient": g, "step": step, "misfit": first}


def _net64(case, seed, train):
    net = precond.LearnedPreconditioner(case["nx"], case["ny"], case["nz"], layers=case["layers"], seed=seed % 1000)
    r, dinv, dz = (t.double() for t in _net_inputs(case, seed))
    params = [p.detach().double().requires_grad_(train) for p in net.params]
    shape = case["nx"], case["ny"], case["nz"]

    def taps(x, w, sign):
        """out[v] = sum over taps of x[v + sign * tap] w[tap]; x [nx, ny, nz, ci], w [27, ci, co]."""
        pad = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        out = 0.0
        for t in range(27):
            o = [1 + sign * q for q in (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)]
            out = out + pad[o[0]:o[0] + shape[0], o[1]:o[1] + shape[1], o[2]:o[2] + shape[2]] @ w[t]
        return out

    wc = params[0].t()[:, None, :]  # [27, 1, 32]
    s = 1.0 / r.square().mean().sqrt()
    u = taps((s * dinv.sqrt() * r).view(*shape, 1), wc, -1)
    for w in params[1:]:
        u = u + taps(u, w.permute(2, 1, 0), 1)
    for w in reversed(params[1:]):
        u = u + taps(u, w.permute(2, 0, 1), -1)
    y = taps(u, wc.transpose(1, 2), 1).reshape(-1)
    z = dinv * r + dinv.sqrt() / s * y
    if not train:
        return {"z": z}
    z.backward(dz)
    return {"z": z.detach(), "grads": [p.grad for p in params]}


def exact(case, seed):
    op = case["op"]
    if op in ("shot", "rtm", "fwi", "fwi_ckpt"):
        v, shots, data = _wave_inputs(case, seed)
        W = _Wave64(case, v)
        data = [d.double() for d in data]
        if op == "shot":
            seis, field, _ = W.forward(shots[0])
            return {"seis": seis, "field": field}
        if op == "rtm":
            _, _, hist = W.forward(shots[0], keep=True)
            image, illum = torch.zeros_like(W.c), torch.zeros_like(W.c)
            scale = W._weight().view_as(W.c) * (W.D if W.stable else 1.0)

            def visit(t, mu):
                image.add_(hist[t] * mu / scale)
                illum.add_(hist[t] ** 2)

            W.backward(data[0], visit)
            refl = torch.where(illum > 1e-10, image / illum, 0.0)
            return {"image": image.view(-1), "illum": illum.view(-1), "refl": refl.view(-1)}
        if op == "fwi":
            grad, seis = torch.zeros_like(W.c), []
            for sh, d in zip(shots, data):
                s, _, hist = W.forward(sh, keep=True)
                seis.append(s)
                grad += W.gradient(sh, s - d, hist)
            return {"seis": torch.stack(seis), "grad": grad}
        s, _, hist = W.forward(shots[0], keep=True)
        res = s - data[0]
        return {"misfit": float(0.5 * res.square().sum()), "grad": W.gradient(shots[0], res, hist).view(-1)}
    if op == "ray_setup":
        ends, d, model = _ray_inputs(case, seed)
        A = _Rays64(ends, case["n"])
        return {"row_ptr": None, "times": A.mul(model.double()), "rhs": A.tmul(d.double())}
    if op == "tomo_cg":
        ends, d, _ = _ray_inputs(case, seed)
        A = _Rays64(ends, case["n"])
        return {"x": _cg64(lambda p: A.tmul(A.mul(p)) + LAM * p, A.tmul(d.double()), 1.0 / (A.diag() + LAM),
                           case["iters"])}
    if op == "update_cg":
        shape = case["nx"], case["ny"], case["nz"]
        b = _smooth(shape, 4, _gen(seed)).reshape(-1).double()
        n_at = 37.0 + _lap(torch.ones(shape, device=DEV, dtype=torch.float64)).view(-1) + 6.0  # 36 + neighbours + 1
        return {"x": _cg64(lambda p: _lap(_lap(p.view(shape))).view(-1) + p, b, 1.0 / n_at, case["iters"])}
    if op == "inversion":
        return _inversion64(case, seed)
    return _net64(case, seed, op == "net_train")
