"""The calls a user of the library makes, as cases that can be timed and compared.

A case is one flow and one way of stepping it: a single domain (``run``), the
same with its residual checked every few steps (``converge``), a restart from
populations in host memory that are read back at the end (``restart``), or
many domains stepped together (``batch``).  Every state starts from a smooth
flow of the size such a simulation has once it has developed, so that all
components of the velocity are well above the rounding of the storage, as a
restart from a checkpoint is.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the domain(s), holding the seed's initial flow
    run(state)          one pass: the steps of the case, then its fields
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the same fields from plain torch in 64 bits
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.getcwd()


def _package():
    name = "nflow_red_poplar_b200"
    if name not in sys.modules:
        path = os.path.join(ROOT, "nflow-red-poplar_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path)
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ------------------------------------------------------------------ cases
def _case(name=None, kind="run", nx=64, ny=64, nz=64, geometry="cavity", model="mrt_les",
          re=1000.0, storage="f32", streaming="ab", rounding="nearest", steps=100, check_every=0,
          members=0, mix=0):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, geometry=geometry, model=model, re=re,
             storage=storage, streaming=streaming, rounding=rounding, steps=steps,
             check_every=check_every, members=members, mix=mix)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small box stepped one call per time step: coupling to another
        # code, probes every step
        _case("cavity 24 one step", nx=24, ny=24, nz=24, re=100.0, steps=1),
        # the 64^3 SRT cavity at tau 0.6 (the benchmark's smallest box), default options
        _case("cavity 64 srt", nx=64, ny=64, nz=64, model="srt", re=192.0, steps=100),
        # the headline box and scheme: 256^3, MRT + LES, Re 5000, in place
        _case("cavity 256 aa", nx=256, ny=256, nz=256, re=5000.0, streaming="aa", steps=100),
        # a box whose sides are no powers of two, default options
        _case("cavity 173x141x119", nx=173, ny=141, nz=119, re=1000.0, steps=60),
        # the precision channel in FP16, in place
        _case("channel 512x128x128 f16 aa", nx=512, ny=128, nz=128, geometry="channel",
              re=1000.0, storage="f16", streaming="aa", steps=100),
        # BF16 with stochastic rounding, the unbiased 16-bit form, on a mid-size channel
        _case("channel 256x72x64 bf16 sr aa", nx=256, ny=72, nz=64, geometry="channel", re=500.0,
              storage="bf16", streaming="aa", rounding="stochastic", steps=60),
        # FP16 with the default (pull) streaming
        _case("cavity 200x104x96 f16", nx=200, ny=104, nz=96, re=2000.0, storage="f16", steps=60),
        # the FP64 build, used to judge the other formats
        _case("cavity 96 f64", nx=96, ny=96, nz=96, re=1000.0, storage="f64", steps=40),
        # a channel around solid voxels
        _case("obstacles 180x60x68", nx=180, ny=60, nz=68, geometry="obstacles", model="srt_les",
              re=200.0, steps=60),
        # stepping until the residual is small, checked every 50 steps
        _case("converge 96x64x80", kind="converge", nx=96, ny=64, nz=80, re=400.0, steps=200,
              check_every=50),
        # the program of the reference: populations in, steps, populations out
        _case("restart 128", kind="restart", nx=128, ny=128, nz=128, re=1000.0, streaming="aa",
              steps=100),
        # the mixed batch (edges 32 to 128, cavities and channels), one chunk of 32 steps
        _case("batch of 16", kind="batch", members=16, mix=1, steps=32),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


LARGEST = 256 ** 3 * 100  # node updates of a pass


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["converge", "restart", "batch"])
    storage = rng.choice(["f32", "f32", "f32", "f16", "f16", "bf16", "f64"])
    model = rng.choice(["mrt_les", "mrt_les", "mrt_les", "srt", "srt_les", "mrt"])
    re = round(_log(rng, 100, 250 if model == "srt" else 2000), 1)
    streaming = rng.choice(["ab", "aa"])
    if kind == "batch":
        # 4 to 16 members, all of one storage and streaming
        return _case(None, kind, 0, 0, 0, "mixed", "mixed", 0.0,
                     "f32" if storage == "f64" else storage, streaming,
                     steps=rng.choice([16, 32, 33, 64]), members=rng.randint(4, 16),
                     mix=rng.randint(1, 10 ** 6))
    geometry = rng.choice(["cavity", "cavity", "cavity", "channel", "channel", "obstacles"])
    if geometry == "obstacles":
        streaming = "ab"
    nodes = _log(rng, 16 ** 3, 1.3e7 if storage != "f64" else 4e6)
    if kind == "restart":
        nodes = min(nodes, 2.2e6)
    e = nodes ** (1.0 / 3.0)
    long_ = _log(rng, 0.8, 1.8)
    wide = _log(rng, 0.8, 1.25)
    nx = max(16, round(e * long_))
    ny = max(16, round(e * wide / math.sqrt(long_)))
    nz = max(16, round(e / wide / math.sqrt(long_)))
    rounding = "nearest"
    if rng.random() < 0.5:
        nx = (nx + 7) // 8 * 8
        if storage in ("f16", "bf16") and geometry != "obstacles" and rng.random() < 0.4:
            rounding = "stochastic"
    weight = 4 if storage == "f64" else 1
    most = LARGEST // (weight * nx * ny * nz)
    steps = max(1, min(most, round(_log(rng, 1, 200))))
    if kind == "converge":
        steps = max(2, steps)
    return _case(None, kind, nx, ny, nz, geometry, model, re, storage, streaming, rounding, steps,
                 check_every=max(1, steps // rng.randint(1, 5)) if kind == "converge" else 0)


def _parts(case):
    """The single domains of a case (a batch: its members, fixed by `mix`)."""
    if case["kind"] != "batch":
        return [case]
    rng = np.random.default_rng(case["mix"])
    parts = []
    for _ in range(case["members"]):
        e = int(rng.choice([32, 40, 48, 64, 80, 96, 128], p=[.2, .1, .2, .2, .1, .1, .1]))
        channel = bool(rng.random() < 0.5)
        model = "srt" if rng.random() < 0.5 else "mrt_les"
        re = float(np.exp(rng.uniform(np.log(100.0), np.log(250.0 if model == "srt" else 2000.0))))
        nx = min(4 * e, 256) if channel else e
        parts.append(dict(case, kind="run", nx=nx, ny=e, nz=e, model=model, re=re,
                          geometry="channel" if channel else "cavity"))
    return parts


# ------------------------------------------------------- parameters, flow
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1]
CZ = [0, 0, 0, -1, 1, 0, 0, -1, -1, 1, 1, 0, 0, 0, 0, -1, 1, -1, 1]
OPP = [0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15]


def _speed(case):
    return 0.1 if case["geometry"] == "cavity" else 0.05


def _tau(case):
    h = case["nx"] if case["geometry"] == "cavity" else min(case["ny"], case["nz"])
    return float(np.float32(3.0 * _speed(case) * h / case["re"] + 0.5))


def _flow(case, seed):
    """Populations [ny][nz][nx][19] (float32, on the GPU) in equilibrium with a
    smooth random flow: three long waves per velocity component over the mean
    flow, the density within 0.1 %."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator().manual_seed(int(seed) * 1000003 + nx * 7 + ny * 5 + nz * 3)
    dev = torch.device("cuda")
    y = (torch.arange(ny, device=dev, dtype=torch.float32) / (ny - 1)).view(ny, 1, 1)
    z = (torch.arange(nz, device=dev, dtype=torch.float32) / (nz - 1)).view(1, nz, 1)
    x = (torch.arange(nx, device=dev, dtype=torch.float32) / (nx - 1)).view(1, 1, nx)

    def waves(amp):
        out = torch.zeros(ny, nz, nx, device=dev)
        for _ in range(3):
            k = torch.randint(1, 4, (3,), generator=g).tolist()
            p = (torch.rand(3, generator=g) * 2 * math.pi).tolist()
            out += amp * torch.sin(math.pi * k[0] * x + p[0]) * \
                torch.sin(math.pi * k[1] * y + p[1]) * torch.sin(math.pi * k[2] * z + p[2])
        return out

    u0 = _speed(case)
    u = [waves(0.25 * u0) for _ in range(3)]
    if case["geometry"] != "cavity":
        u[0] += u0 * 16 * y * (1 - y) * z * (1 - z)
    rho = 1 + waves(3e-4)
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    f = torch.empty(ny, nz, nx, 19, device=dev)
    for q in range(19):
        eu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
        f[..., q] = W[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq)
    return f


def _solid(case):
    """Two spheres on the channel's axis, well inside the box."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    y, z, x = np.meshgrid(np.arange(ny), np.arange(nz), np.arange(nx), indexing="ij", sparse=True)
    r = max(1, min(nx, ny, nz) // 6)
    near = lambda cx: (x - cx) ** 2 + (y - ny // 2) ** 2 + (z - nz // 2) ** 2 <= r * r  # noqa: E731
    return near(nx // 3) | near(2 * nx // 3)


# ---------------------------------------------------------------- the path
class _Wrapped:
    """Device memory of the library for torch; holds its owner, so that the
    memory outlives the tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4",
                                         "version": 3}


class _Fields:
    """rho, ux, uy, uz of a domain as torch tensors over the library's arrays."""

    def __init__(self, pkg, dom, owner):
        self.lib, self.dom, self.owner, self.known = pkg.lib(), dom, owner, {}
        self.p = [ctypes.c_void_p() for _ in range(5)]
        self.ref = [ctypes.byref(v) for v in self.p]

    def now(self):
        self.lib.lbm_device_fields(self.dom.h, *self.ref)
        out = []
        for i in (0, 2, 3, 4):
            a = self.p[i].value
            if a not in self.known:
                self.known[a] = torch.as_tensor(_Wrapped(a, self.dom.shape, self.owner),
                                                device="cuda")
            out.append(self.known[a])
        return tuple(out)


def _inputs(pkg, case):
    mrt, les = case["model"].startswith("mrt"), case["model"].endswith("les")
    iv = pkg.make_inputval(case["nx"], case["ny"], case["nz"], u=_speed(case), tau=_tau(case),
                           casetype=pkg.CAVITY if case["geometry"] == "cavity" else pkg.CHANNEL,
                           mrt=mrt, les=les, cs=0.1)
    opt = pkg.default_options(
        storage={"f32": pkg.STORE_F32, "f16": pkg.STORE_F16_SHIFT, "bf16": pkg.STORE_BF16_SHIFT,
                 "f64": pkg.STORE_F64}[case["storage"]],
        stream_mode=pkg.STREAM_AA if case["streaming"] == "aa" else pkg.STREAM_AB)
    if case["rounding"] == "stochastic":
        # the in-place form rounds stochastically over rows of whole words
        # only; elsewhere such a user takes the pull form
        if case["nx"] % 8 or case["nx"] < 16:
            opt.stream_mode = pkg.STREAM_AB
        opt.rounding = pkg.ROUND_STOCHASTIC
    return iv, opt


def prepare(case, seed):
    pkg = _package()
    if case["kind"] == "batch":
        parts = [(_inputs(pkg, c), c) for c in _parts(case)]
        need = sum(pkg.batch_domain_bytes(iv, o) for (iv, o), _ in parts)
        b = pkg.Batch(hbm_budget=need + (len(parts) << 16), chunk_steps=32)
        fields = []
        for n, ((iv, o), c) in enumerate(parts):
            m = b.member(b.add(iv, o, steps=1 << 40))
            m.import_arF(_flow(c, seed + 1000 * n).cpu().numpy())
            fields.append(_Fields(pkg, m, b))
        b.sync()
        return dict(case=case, batch=b, fields=fields)
    iv, opt = _inputs(pkg, case)
    d = pkg.Domain(iv, opt)
    if case["geometry"] == "obstacles":
        d.set_solid_mask(_solid(case))
    f = _flow(case, seed)
    s = dict(case=case, dom=d, fields=_Fields(pkg, d, d))
    if case["kind"] == "restart":
        ny, nz, nx = d.shape
        host = torch.zeros(ny + 2, nz + 2, nx + 2, 19, pin_memory=True)
        host[1:-1, 1:-1, 1:-1] = f.cpu()
        s["in"] = host.numpy()
        s["back"] = torch.empty(ny + 2, nz + 2, nx + 2, 19, pin_memory=True)
        s["out"] = s["back"].numpy()
    else:
        d.import_arF(f.cpu().numpy())
    d.sync()
    return s


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "run":
        state["dom"].run(steps)
        return state["fields"].now()
    if kind == "converge":
        done, _ = state["dom"].run_until_converged(steps, case["check_every"], 1e-12)
        return (done,) + state["fields"].now()
    if kind == "restart":
        d = state["dom"]
        d.import_arF(state["in"], padded=True)
        d.run(steps)
        d.export_arF(padded=True, out=state["out"])
        return (state["back"],) + state["fields"].now()
    state["batch"].step(steps)
    return [f.now() for f in state["fields"]]


# ------------------------------------------------------------ what it needs
SIZE = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}
# additions and multiplications of one node update (moments, relaxation,
# back transform in opposite pairs; the stress and tau of the LES)
FLOPS = {"srt": 170, "srt_les": 240, "mrt": 260, "mrt_les": 330}


def work(case):
    """Each population read once and written once over the pass, however many
    steps it takes, the four fields written once, and every update's
    operations."""
    b = f = 0
    for c in _parts(case):
        n = c["nx"] * c["ny"] * c["nz"]
        b += n * (2 * 19 * SIZE[c["storage"]] + 16)
        f += n * c["steps"] * FLOPS[c["model"]]
        if c["kind"] == "restart":  # the host's populations in and out
            b += 2 * 19 * 4 * (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------- in 64 bits
def _moments():
    """The 19 moments of D3Q19 (rows), from the velocities."""
    c = np.array([CX, CY, CZ], dtype=np.float64)
    x, y, z = c
    n2 = (c * c).sum(0)
    one = np.ones(19)
    return np.stack([
        one, 19 * n2 - 30, (21 * n2 * n2 - 53 * n2 + 24) / 2,
        x, (5 * n2 - 9) * x, y, (5 * n2 - 9) * y, z, (5 * n2 - 9) * z,
        3 * x * x - n2, (3 * n2 - 5) * (3 * x * x - n2),
        y * y - z * z, (3 * n2 - 5) * (y * y - z * z),
        x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z])


def _exact_run(case, seed):
    dev, f64 = torch.device("cuda"), torch.float64
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f = _flow(case, seed).permute(3, 0, 1, 2).to(f64).contiguous()
    r32 = lambda v: float(np.float32(v))  # noqa: E731
    tau, u0, cs = _tau(case), r32(_speed(case)), r32(0.1)
    les_c = r32(np.float32(18.0) * np.float32(1.41421356237)) * cs * cs
    M = torch.tensor(_moments(), device=dev)
    Minv = torch.linalg.inv(M)
    y = torch.arange(ny, device=dev).view(ny, 1, 1)
    z = torch.arange(nz, device=dev).view(1, nz, 1)
    x = torch.arange(nx, device=dev).view(1, 1, nx)
    side = (z == 0) | (z == nz - 1)
    cavity = case["geometry"] == "cavity"
    if cavity:
        lid = (y == ny - 1) & ~side & (x > 0) & (x < nx - 1)
    else:
        side = side | (y == 0) | (y == ny - 1)
        inlet, outlet = (x == 0) & ~side, (x == nx - 1) & ~side
        eta, zeta = y.to(f64) / (ny - 1), z.to(f64) / (nz - 1)
        uin = (u0 * 16 * eta * (1 - eta) * zeta * (1 - zeta)).float().to(f64)
    solid = None
    if case["geometry"] == "obstacles":
        solid = torch.tensor(_solid(case), device=dev)

    def macro():
        rho = f.sum(0)
        j = [sum(s[q] * f[q] for q in range(19) if s[q]) for s in (CX, CY, CZ)]
        return rho, [v / rho for v in j]

    rho, u = macro()
    for _ in range(case["steps"]):
        jx, jy, jz = (rho * v for v in u)
        te = 0.0
        if case["model"].endswith("les"):
            qq, cc = 0.0, (CX, CY, CZ)
            for a in range(3):
                for b in range(a, 3):
                    p = sum(cc[a][q] * cc[b][q] * f[q] for q in range(19) if cc[a][q] * cc[b][q])
                    t = p - rho * u[a] * u[b] - (rho / 3 if a == b else 0)
                    qq = qq + (1 if a == b else 2) * t * t
            te = 0.5 * (torch.sqrt(tau * tau + les_c * torch.sqrt(qq) / rho) - tau)
            del qq, p, t
        nu = 1.0 / (tau + te)
        if case["model"].startswith("mrt"):
            d = torch.einsum("kq,qyzx->kyzx", M, f)
            jj = jx * jx + jy * jy + jz * jz
            m9, m11 = 2 * jx * jx - jy * jy - jz * jz, jy * jy - jz * jz
            for k, eq, s in ((0, rho, 0), (1, 19 * jj - 11 * rho, 1.19),
                             (2, 3 * rho - 5.5 * jj, 1.4), (3, jx, 0), (4, -2 / 3 * jx, 1.2),
                             (5, jy, 0), (6, -2 / 3 * jy, 1.2), (7, jz, 0), (8, -2 / 3 * jz, 1.2),
                             (9, m9, nu), (10, -0.5 * m9, 1.4), (11, m11, nu),
                             (12, -0.5 * m11, 1.4), (13, jx * jy, nu), (14, jy * jz, nu),
                             (15, jx * jz, nu), (16, 0, 1.98), (17, 0, 1.98), (18, 0, 1.98)):
                d[k] = (d[k] - eq) * s
            fs = torch.einsum("qk,kyzx->qyzx", Minv, d).neg_().add_(f)
            del d, jj, m9, m11
        else:
            fs = torch.empty_like(f)
            usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
            for q in range(19):
                eu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
                fs[q] = f[q] + (W[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq) - f[q]) * nu
        del jx, jy, jz, te, nu
        if not cavity:
            near = rho[:, :, 1:2].clone()
            ub = [(v[:, :, -1:] + 0.5 * (v[:, :, -1:] - v[:, :, -2:-1])) for v in u]
            ubsq = sum(v * v for v in ub)
        for q in range(19):
            o = OPP[q]
            f[q] = torch.roll(fs[q], (CY[q], CZ[q], CX[q]), (0, 1, 2))
            out = torch.zeros(ny, nz, nx, dtype=torch.bool, device=dev)
            for c, n, dim in ((CY[q], ny, 0), (CZ[q], nz, 1), (CX[q], nx, 2)):
                if c:
                    out.select(dim, 0 if c > 0 else n - 1)[:] = True
            if q == 0:
                continue
            wall = fs[o]
            if cavity:
                wall = torch.where(lid, wall - 6 * W[q] * CX[o] * u0, wall)
            else:
                wall = torch.where(inlet, wall - 6 * W[q] * near * CX[o] * uin, wall)
                eu = CX[o] * ub[0] + CY[o] * ub[1] + CZ[o] * ub[2]
                wall = torch.where(outlet, 2 * W[q] * (1 + 4.5 * eu * eu - 1.5 * ubsq) - wall, wall)
            f[q] = torch.where(out, wall, f[q])
            if solid is not None:
                behind = torch.roll(solid, (CY[q], CZ[q], CX[q]), (0, 1, 2)) & ~out
                f[q] = torch.where(behind, fs[o], f[q])
        del fs
        rho, u = macro()
    if solid is not None:
        rho = torch.where(solid, torch.zeros_like(rho), rho)
        u = [torch.where(solid, torch.zeros_like(v), v) for v in u]
    return f, (rho, u[0], u[1], u[2])


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_run(c, seed + 1000 * n)[1] for n, c in enumerate(_parts(case))]
    f, fields = _exact_run(case, seed)
    if case["kind"] == "converge":
        return (case["steps"],) + fields
    if case["kind"] == "restart":
        ny, nz, nx = case["ny"], case["nz"], case["nx"]
        back = torch.zeros(ny + 2, nz + 2, nx + 2, 19, dtype=torch.float64)
        back[1:-1, 1:-1, 1:-1] = f.permute(1, 2, 3, 0).cpu()
        return (back,) + fields
    return fields
