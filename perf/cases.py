"""The work that programs built on this framework have it do, as cases to be timed and compared.

A case is one of:

* ``plain``  -- time steps of one domain without MHD, periodic, a Taylor-Green-like flow;
* ``mhd``    -- time steps of one MHD domain: wall shell, finite-plasma start, an external static field,
  with the exact field (BITWISE, the default, or FAST) or the learned far field (SURROGATE);
* ``batch``  -- time steps of many uneven MHD domains advanced together;
* ``magnet`` -- the setup of a box with a disk magnet: voxelisation and the static field.

``prepare`` gives a program's state before the call (handles created, fields uploaded, initialized), ``run``
one pass through the public entry points.  Outputs are the device buffers themselves: density and velocity,
the dynamic fields, the net charge (with 32-bit storage; 16-bit storage does not resolve this difference of
two lattices, so there the lattices themselves come back) and the distribution functions.  16-bit FP16S
distributions are seen as the half-precision values that they are; FP16C codes are not a type of torch, so
there the moments stand for them.

``exact`` is the same first pass in 64 bits with plain torch: the Esoteric-Pull step, the LOD bin sums, the
Coulomb/Biot-Savart sums over the bins, and the magnet's potential.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ionsolver_gb300 as I

FLOAT_TYPES = {"FP16S": 0, "FP16C": 1, "FP32": 2}
FIELD_MODES = {"BITWISE": 0, "FAST": 1, "SURROGATE": 2}
SETS = {"D2Q9": 0, "D3Q19": 2}
NU = 1.0 / 30.0
# the finite-plasma units: cells of 6.46 cm, steps of 1 ns, gas 1e-3 kg/m^3, current unit 1 A
UNITS = dict(m=0.0646, kg=2.7e-7, s=1e-9, a=1.0, k=1.0, prop=0)
RHO_E0 = 0.01          # background electron density
MAGNETIZATION = 300.0  # A/m


def listed():
    return [
        # the reference's default configuration (D2Q9, FP16S) on a small plane: a step is launch latency
        dict(name="plane-d2q9-fp16s", kind="plain", vset="D2Q9", nx=300, ny=200, nz=1, ft="FP16S", trt=False, steps=1),
        # the small periodic box of the Taylor-Green configuration, stepped in a loop; it stays in L2
        dict(name="tgv64-fp32", kind="plain", vset="D3Q19", nx=64, ny=64, nz=64, ft="FP32", trt=False, steps=10),
        # the same flow at a size bound by memory
        dict(name="tgv256-fp32", kind="plain", vset="D3Q19", nx=256, ny=256, nz=256, ft="FP32", trt=False, steps=2),
        # a channel of no round size with the two-relaxation-time collision and 16-bit storage
        dict(name="ragged-trt-fp16s", kind="plain", vset="D3Q19", nx=150, ny=101, nz=70, ft="FP16S", trt=True, steps=2),
        # the smallest MHD box in use, in the default field mode
        dict(name="mhd32-bitwise", kind="mhd", nx=32, ny=32, nz=32, depth=4, ft="FP32", mode="BITWISE"),
        # an ordinary MHD box in the default field mode
        dict(name="mhd96-bitwise", kind="mhd", nx=96, ny=96, nz=96, depth=4, ft="FP32", mode="BITWISE"),
        # the headline configuration: 128^3, FP32, the FAST field
        dict(name="mhd128-fast", kind="mhd", nx=128, ny=128, nz=128, depth=4, ft="FP32", mode="FAST"),
        # the large box with 16-bit storage
        dict(name="mhd256-fast-fp16s", kind="mhd", nx=256, ny=256, nz=256, depth=4, ft="FP16S", mode="FAST"),
        # an uneven box with the custom 16-bit codec: LOD bins of 12 x 10 x 8 cells
        dict(name="mhd-uneven-fast-fp16c", kind="mhd", nx=192, ny=160, nz=128, depth=4, ft="FP16C", mode="FAST"),
        # a parameter sweep: uneven domains of 32 to 96 cells an edge advanced together
        dict(name="batch24-fast", kind="batch", count=24, lo=32, hi=96, ft="FP32"),
        # the learned far field on the two-ring configuration's storage, at half its edge
        dict(name="learned192-fp16s", kind="mhd", nx=192, ny=192, nz=192, depth=4, ft="FP16S", mode="SURROGATE"),
        # the setup of the headline box: voxelise the disk magnet, precompute its field
        dict(name="magnet128", kind="magnet", n=128, radius=16, thickness=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plane", "plain", "plain", "bitwise", "fast", "fast", "fast", "fast", "batch", "learned", "magnet"])
    if kind == "plane":
        return dict(kind="plain", vset="D2Q9", nx=_log_int(rng, 64, 2048), ny=_log_int(rng, 64, 2048), nz=1,
                    ft=rng.choice(list(FLOAT_TYPES)), trt=rng.random() < 0.3, steps=rng.choice([1, 2, 10]))
    if kind == "plain":
        nx = _log_int(rng, 24, 256)
        if rng.random() < 0.5:
            nx = max(16, nx // 16 * 16)
        return dict(kind="plain", vset="D3Q19", nx=nx, ny=_log_int(rng, 24, 256), nz=_log_int(rng, 24, 256),
                    ft=rng.choice(list(FLOAT_TYPES)), trt=rng.random() < 0.3, steps=rng.choice([1, 2, 10]))
    if kind == "batch":
        lo = rng.choice([32, 48])
        return dict(kind="batch", count=rng.randint(3, 24), lo=lo, hi=rng.choice([64, 80, 96]), ft=rng.choice(["FP32", "FP16S"]))
    if kind == "magnet":
        return dict(kind="magnet", n=_log_int(rng, 40, 128), radius=rng.randint(4, 16), thickness=rng.randint(2, 8))
    depth = rng.choice([3, 4, 4, 4])
    step = 1 << depth
    top = {"bitwise": 96, "fast": 256, "learned": 192}[kind]
    n = _log_int(rng, 32 if kind != "learned" else 64, top)
    edges = [max(32, int(n * rng.choice([1.0, 1.0, 0.75, 0.6])) // step * step) for _ in range(3)]
    mode = {"bitwise": "BITWISE", "fast": "FAST", "learned": "SURROGATE"}[kind]
    return dict(kind="mhd", nx=edges[0], ny=edges[1], nz=edges[2], depth=depth, ft=rng.choice(list(FLOAT_TYPES)), mode=mode)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _flow(nx, ny, nz, seed):
    """A periodic vortex with a phase from the seed and a little noise: u [3][N], rho [N]."""
    g = _generator(seed)
    phase = torch.rand(3, generator=g, device="cuda") * (2.0 * math.pi)
    x = torch.arange(nx, device="cuda", dtype=torch.float32) * (2.0 * math.pi / nx) + phase[0]
    y = torch.arange(ny, device="cuda", dtype=torch.float32) * (2.0 * math.pi / ny) + phase[1]
    z = torch.arange(nz, device="cuda", dtype=torch.float32) * (2.0 * math.pi / nz) + phase[2]
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    shape = (nz, ny, nx)
    ux = 0.05 * torch.cos(x) * torch.sin(y) * torch.sin(z)
    uy = -0.05 * torch.sin(x) * torch.cos(y) * torch.sin(z)
    u = torch.stack([ux.expand(shape), uy.expand(shape), torch.zeros(shape, device="cuda")])
    noise = torch.randn((3,) + shape, generator=g, device="cuda") * 1e-3
    if nz == 1:
        noise[2] = 0.0
    rho = 1.0 + torch.randn(shape, generator=g, device="cuda") * 1e-3
    return (u + noise).reshape(3, -1), rho.reshape(-1)


def _plasma(nx, ny, nz, seed):
    """Charge, velocity, static field and wall flags of an MHD box, as [N] and [3][N] tensors."""
    g = _generator(seed)
    N = nx * ny * nz
    q = torch.rand(N, generator=g, device="cuda") * 2e-3 - 1e-3
    u = torch.randn(3, N, generator=g, device="cuda") * 1e-3
    flags = torch.zeros(nz, ny, nx, dtype=torch.uint8, device="cuda")
    flags[0] = flags[-1] = 1
    flags[:, 0] = flags[:, -1] = 1
    flags[:, :, 0] = flags[:, :, -1] = 1
    # an axial dipole below the floor and a weak guide field, of the disk magnet's strength in these units
    x = torch.arange(nx, device="cuda", dtype=torch.float32)[None, None, :] - 0.5 * nx
    y = torch.arange(ny, device="cuda", dtype=torch.float32)[None, :, None] - 0.5 * ny
    z = torch.arange(nz, device="cuda", dtype=torch.float32)[:, None, None] + 0.25 * nz
    r2 = x * x + y * y + z * z
    a = B_SCALE * (0.25 * nz) ** 3 / (r2 * torch.sqrt(r2))
    b = torch.stack([(a * 3.0 * x * z / r2), (a * 3.0 * y * z / r2), (a * (3.0 * z * z / r2 - 1.0)) + 0.1 * B_SCALE])
    return dict(q=q, u=u, flags=flags.reshape(-1), b_stat=b.reshape(3, -1))


def _constants():
    m, kg, s, a = (UNITS[k] for k in ("m", "kg", "s", "a"))
    eps0 = 8.8541878128e-12 / ((a * a * s ** 4) / (kg * m ** 3))
    mu0 = 1.256637062e-6 / ((kg * m) / (a * a * s * s))
    kkge = (9.1093837139e-31 / -1.602176634e-19) / (kg / (a * s))
    return dict(ke=1.0 / (4.0 * math.pi * eps0), kmu=mu0 / (4.0 * math.pi), kmu0=mu0, kkge=kkge, wq=0.4)


B_SCALE = 1e-2 * abs(2.0 * _constants()["kkge"])  # a cyclotron rotation of about 1e-2 a step


class _Buffer:
    """A device buffer of a handle for torch; holds the handle for as long as a tensor sees it."""

    def __init__(self, lbm, ptr, count, typestr):
        self.owner = lbm
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(lbm, name, count, ft=None):
    ptr, _ = lbm.device_ptr(name)
    typestr = "|u1" if name == "flags" else "<f2" if ft == "FP16S" else "<f4"
    return torch.as_tensor(_Buffer(lbm, ptr, count, typestr), device="cuda")


def _outputs(lbm, ft, mhd, planar=False):
    N = lbm.n
    out = {"rho": _view(lbm, "rho", N), "u": _view(lbm, "u", 3 * N)}
    if ft != "FP16C":
        out["fi"] = _view(lbm, "fi", (9 if planar else 19) * N, ft)
    if mhd:
        out["e_dyn"] = _view(lbm, "e_dyn", 3 * N)
        out["b_dyn"] = _view(lbm, "b_dyn", 3 * N)
        if ft == "FP32":
            out["q"] = _view(lbm, "q", N)
        if ft != "FP16C":
            out["ei"] = _view(lbm, "ei", 19 * N, ft)
            out["fqi"] = _view(lbm, "fqi", 7 * N, ft)
    return out


def _host(t):
    return t.cpu().numpy().reshape(-1)


def _mhd_lbm(nx, ny, nz, depth, ft, mode, seed):
    cfg = I.LbmConfig(velocity_set=2, float_type=FLOAT_TYPES[ft], units=I.Units(**UNITS), n_x=nx, n_y=ny, n_z=nz, nu=NU,
                      ext_volume_force=True, ext_magneto_hydro=True, mhd_lod_depth=depth, field_mode=FIELD_MODES[mode])
    lbm = I.Lbm(cfg)
    for name, value in _plasma(nx, ny, nz, seed).items():
        lbm.write(name, _host(value))
    lbm.set_electron_background(RHO_E0)
    if mode == "SURROGATE":
        rng = np.random.Generator(np.random.PCG64(int(seed) + 11))
        count = lbm.surrogate_weights().size
        lbm.surrogate_weights((rng.standard_normal(count) * 0.02).astype(np.float32))
        # the sampled check runs every step; untrained weights must not make it fall back
        lbm.surrogate_configure(tolerance=1e6)
    lbm.initialize()
    return lbm


def _domains(case, seed):
    """The edges of a batch's domains: multiples of 16, spread over [lo, hi]; the sizes are the sweep's, not the seed's."""
    rng = np.random.Generator(np.random.PCG64(3))
    edges = np.arange(case["lo"], case["hi"] + 1, 16)
    return [(int(rng.choice(edges)), int(seed) * 100 + i) for i in range(case["count"])]


def _disk(case):
    n, r, t = case["n"], float(case["radius"]), float(case["thickness"])
    return (0.5 * n + 0.13, 0.5 * n - 0.21, 1.3 + 0.5 * t), min(r, 0.5 * n - 4.0), t


def _magnetization(seed):
    m = np.random.Generator(np.random.PCG64(int(seed))).normal(size=3)
    return (m / np.linalg.norm(m) * MAGNETIZATION).tolist()


def prepare(case, seed):
    if case["kind"] == "plain":
        cfg = I.LbmConfig(velocity_set=SETS[case["vset"]], relaxation_time=int(case["trt"]), float_type=FLOAT_TYPES[case["ft"]],
                          n_x=case["nx"], n_y=case["ny"], n_z=case["nz"], nu=NU)
        lbm = I.Lbm(cfg)
        u, rho = _flow(case["nx"], case["ny"], case["nz"], seed)
        lbm.write("u", _host(u))
        lbm.write("rho", _host(rho))
        lbm.initialize()
        return dict(case=case, lbm=lbm, out=_outputs(lbm, case["ft"], False, planar=case["vset"] == "D2Q9"))
    if case["kind"] == "mhd":
        lbm = _mhd_lbm(case["nx"], case["ny"], case["nz"], case["depth"], case["ft"], case["mode"], seed)
        return dict(case=case, lbm=lbm, out=_outputs(lbm, case["ft"], True))
    if case["kind"] == "batch":
        doms = [_mhd_lbm(n, n, n, 4, case["ft"], "FAST", s) for n, s in _domains(case, seed)]
        outs = [{k: v for k, v in _outputs(d, case["ft"], True).items() if k in ("u", "e_dyn")} for d in doms]
        return dict(case=case, batch=I.Batch(doms), out=outs)
    n = case["n"]
    cfg = I.LbmConfig(velocity_set=2, float_type=2, units=I.Units(**UNITS), n_x=n // 4 * 4, n_y=n // 4 * 4, n_z=n // 4 * 4, nu=NU,
                      ext_volume_force=True, ext_magneto_hydro=True, mhd_lod_depth=2)
    lbm = I.Lbm(cfg)
    c, r, t = _disk(case)
    mesh = lbm.add_mesh(*I.cylinder(c, r, t, axis=2))
    return dict(case=case, lbm=lbm, mesh=mesh, model=I.ModelType.Magnet(_magnetization(seed)),
                out={"flags": _view(lbm, "flags", lbm.n), "b_stat": _view(lbm, "b_stat", 3 * lbm.n)})


def run(state):
    case = state["case"]
    if case["kind"] == "plain":
        if case["steps"] == 1:
            state["lbm"].do_time_step()
        else:
            state["lbm"].run(case["steps"])
    elif case["kind"] == "mhd":
        state["lbm"].do_time_step()
    elif case["kind"] == "batch":
        state["batch"].run(1)
    else:
        state["lbm"].voxelise_mesh(state["mesh"], state["model"])
        state["lbm"].precompute_B()
    return state["out"]


def work(case):
    if case["kind"] == "plain":
        N, q, w = case["nx"] * case["ny"] * case["nz"], 9 if case["vset"] == "D2Q9" else 19, 4 if case["ft"] == "FP32" else 2
        return {"bytes": case["steps"] * N * (2 * q * w + 1 + 16), "flops": case["steps"] * N * 22 * q}
    if case["kind"] in ("mhd", "batch"):
        cells = [n ** 3 for n, _ in _domains(case, 0)] if case["kind"] == "batch" else [case["nx"] * case["ny"] * case["nz"]]
        depth = case.get("depth", 4)
        w = 4 if case["ft"] == "FP32" else 2
        # lattices read and written, flags, E/B read by the step and written from the static fields, rho, u, q
        nbytes = sum(cells) * (2 * 45 * w + 1 + 24 + 24 + 24 + 16 + 4)
        # the exact sum in the reference's order takes every source for every cell; the other modes at least the nearest bins
        sources = 8 ** depth if case.get("mode") == "BITWISE" else min(27, 8 ** depth)
        return {"bytes": nbytes, "flops": sum(cells) * (1000 + 34 * sources)}
    n, (_, r, t) = case["n"], _disk(case)
    cells = math.pi * r * r * t
    return {"bytes": n ** 3 * (1 + 24) + cells * 13, "flops": (n + 2) ** 3 * cells * 15}


# ---------------------------------------------------------------------------
# the same pass in 64 bits
# ---------------------------------------------------------------------------
_D2Q9 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0)]
_D3Q19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
          (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]
_D3Q7 = _D3Q19[:7]


def _weights(c):
    if len(c) == 9:
        return [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
    return [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _from(a, c):
    """a at the neighbour in direction c, periodic; arrays are [z][y][x]."""
    shifts = [(-c[2], 0), (-c[1], 1), (-c[0], 2)]
    shifts = [s for s in shifts if s[0]]
    return torch.roll(a, [s[0] for s in shifts], [s[1] for s in shifts]) if shifts else a


def _load(f, c, odd):
    v = [f[0]]
    for i in range(1, len(c), 2):
        v += [f[i if odd else i + 1], _from(f[i + 1 if odd else i], c[i])]
    return [x.clone() for x in v]


def _store(f, c, odd, v, act):
    f[0] = torch.where(act, v[0], f[0])
    for i in range(1, len(c), 2):
        own, nbr, back = (i if odd else i + 1), (i + 1 if odd else i), tuple(-k for k in c[i])
        f[own] = torch.where(act, v[i + 1], f[own])
        f[nbr] = torch.where(_from(act, back), _from(v[i], back), f[nbr])


def _feq(c, rho, u):
    """Equilibrium less the rest weights."""
    w, uu = _weights(c), 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = []
    for i, ci in enumerate(c):
        p = 3.0 * (ci[0] * u[0] + ci[1] * u[1] + ci[2] * u[2])
        out.append(w[i] * (rho * (0.5 * p * p + p - uu) + (rho - 1.0)))
    return out


def _aeq(Q, u):
    e = [0.25 * (Q - 1.0)]
    for a in range(3):
        e += [0.125 * (Q - 1.0) + 0.5 * Q * u[a], 0.125 * (Q - 1.0) - 0.5 * Q * u[a]]
    return e


def _moments(c, f):
    rho = sum(f) + 1.0
    u = [sum(ci[a] * fi for ci, fi in zip(c, f) if ci[a]) if any(ci[a] for ci in c) else torch.zeros_like(rho) for a in range(3)]
    return rho, [x / rho for x in u]


def _guo(c, u, force):
    """Guo's forcing terms of every direction."""
    w = _weights(c)
    uf = -(u[0] * force[0] + u[1] * force[1] + u[2] * force[2]) / 3.0
    out = []
    for i, ci in enumerate(c):
        cf = ci[0] * force[0] + ci[1] * force[1] + ci[2] * force[2]
        cu = ci[0] * u[0] + ci[1] * u[1] + ci[2] * u[2] + 1.0 / 3.0
        out.append(9.0 * w[i] * ((cf * cu if i else 0.0) + uf))
    return out


def _collide(c, f, rho, u, w, trt, force=None):
    eq = _feq(c, rho, u)
    F = [x * (1.0 - 0.5 * w) for x in _guo(c, u, force)] if force is not None else [0.0] * len(c)
    if not trt:
        return [(1.0 - w) * a + w * e + g for a, e, g in zip(f, eq, F)]
    wm = 1.0 / (0.1875 / (1.0 / w - 0.5) + 0.5)
    out = [f[0] + w * (eq[0] - f[0])]
    for i in range(1, len(c), 2):
        s, d = (eq[i] + eq[i + 1]) - (f[i] + f[i + 1]), (eq[i] - eq[i + 1]) - (f[i] - f[i + 1])
        out += [f[i] + 0.5 * w * s + 0.5 * wm * d, f[i + 1] + 0.5 * w * s - 0.5 * wm * d]
    return out


def _clamp(u):
    return [torch.clamp(x, -0.57735027, 0.57735027) for x in u]


def _plain_exact(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    c = _D2Q9 if case["vset"] == "D2Q9" else _D3Q19
    shape = (nz, ny, nx)
    u, rho = _flow(nx, ny, nz, seed)
    u, rho = [x.double().reshape(shape) for x in u], rho.double().reshape(shape)
    act = torch.ones(shape, dtype=torch.bool, device="cuda")
    f = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in c]
    _store(f, c, True, _feq(c, rho, u), act)
    w = 1.0 / (3.0 * NU + 0.5)
    for t in range(case["steps"]):
        v = _load(f, c, bool(t & 1))
        rho, u = _moments(c, v)
        u = _clamp(u)
        _store(f, c, bool(t & 1), _collide(c, v, rho, u, w, case["trt"]), act)
    out = {"rho": rho.reshape(-1), "u": torch.stack(u).reshape(-1)}
    if case["ft"] != "FP16C":
        scale = 32768.0 if case["ft"] == "FP16S" else 1.0
        out["fi"] = torch.stack(f).reshape(-1) * scale
    return out


def _field(nx, ny, nz, depth, q, vel, act):
    """The sums over the LOD bins of charge (added) and velocity (averaged) for every cell, without its own bin."""
    nd = 1 << depth
    bs = (nx // nd, ny // nd, nz // nd)
    cells = bs[0] * bs[1] * bs[2]

    def bins(a):
        return torch.where(act, a, torch.zeros_like(a)).reshape(nd, bs[2], nd, bs[1], nd, bs[0]).sum((1, 3, 5)).reshape(-1)

    Q, V = bins(q), [bins(v) / cells for v in vel]
    first = sum(8 ** i for i in range(depth + 1)) - nd ** 3  # the sources begin where the finest level's table begins
    axes = [torch.arange(n, dtype=torch.float64, device="cuda") for n in (nx, ny, nz)]
    own = [torch.arange(n, device="cuda") // b for n, b in zip((nx, ny, nz), bs)]
    own = own[0][None, None, :] + (own[1][None, :, None] + own[2][:, None, None] * nd) * nd
    N = nx * ny * nz
    e, b = torch.zeros(3, nz, ny, nx, dtype=torch.float64, device="cuda"), torch.zeros(3, nz, ny, nx, dtype=torch.float64, device="cuda")
    chunk = max(1, (1 << 22) // N)
    for lo in range(first, nd ** 3, chunk):
        d = torch.arange(lo, min(lo + chunk, nd ** 3), device="cuda")
        pos = [((d // nd ** a % nd).double() + 0.5) * bs[a] for a in range(3)]
        rx = axes[0][None, None, None, :] - pos[0][:, None, None, None]
        ry = axes[1][None, None, :, None] - pos[1][:, None, None, None]
        rz = axes[2][None, :, None, None] - pos[2][:, None, None, None]
        r2 = (rx * rx + ry * ry) + rz * rz
        inv = torch.where(own[None] == d[:, None, None, None], 0.0, r2.pow(-1.5))
        s = [x[d][:, None, None, None] for x in (Q, Q * V[0], Q * V[1], Q * V[2])]
        E = [inv * rx, inv * ry, inv * rz]
        for a in range(3):
            e[a] += (s[0] * E[a]).sum(0)
            i, j = (a + 1) % 3, (a + 2) % 3
            b[a] += (s[1 + i] * E[j] - s[1 + j] * E[i]).sum(0)
    return e, b


def _mhd_exact(nx, ny, nz, depth, ft, mode, seed):
    k = _constants()
    shape = (nz, ny, nx)
    p = _plasma(nx, ny, nz, seed)
    act = (p["flags"] == 0).reshape(shape)
    zero = torch.zeros(shape, dtype=torch.float64, device="cuda")
    u = [torch.where(act, x.double().reshape(shape), zero) for x in p["u"]]
    q0 = torch.where(act, p["q"].double().reshape(shape), zero)
    bs = [x.double().reshape(shape) for x in p["b_stat"]]
    rho = torch.ones_like(zero)
    everywhere = torch.ones_like(act)
    lattices = []
    for c, v in ((_D3Q19, _feq(_D3Q19, rho, u)), (_D3Q19, _feq(_D3Q19, rho * RHO_E0, u)), (_D3Q7, _aeq(q0 + RHO_E0, u))):
        f = [zero.clone() for _ in c]
        _store(f, c, True, v, everywhere)
        lattices.append(f)
    fi, ei, fqi = lattices
    w = 1.0 / (3.0 * NU + 0.5)
    # the electron gas: Lorentz force of the static field, Guo half step
    v = _load(ei, _D3Q19, False)
    rhoe, ue = _moments(_D3Q19, v)
    cross = [ue[1] * bs[2] - ue[2] * bs[1], ue[2] * bs[0] - ue[0] * bs[2], ue[0] * bs[1] - ue[1] * bs[0]]
    fe = [-rhoe * x for x in cross]
    ue = _clamp([x + y * (0.5 / (rhoe * k["kkge"])) for x, y in zip(ue, fe)])
    _store(ei, _D3Q19, False, _collide(_D3Q19, v, rhoe, ue, w, False, fe), act)
    # the gas and the charge that it carries
    v = _load(fi, _D3Q19, False)
    rho1, ug = _moments(_D3Q19, v)
    a = _load(fqi, _D3Q7, False)
    rhoq = sum(a) + 1.0
    _store(fqi, _D3Q7, False, [(1.0 - k["wq"]) * x + k["wq"] * y for x, y in zip(a, _aeq(rhoq, ug))], act)
    q = rhoq - rhoe
    cross = [ug[1] * bs[2] - ug[2] * bs[1], ug[2] * bs[0] - ug[0] * bs[2], ug[0] * bs[1] - ug[1] * bs[0]]
    fg = [rhoq * x for x in cross]
    un = _clamp([x + y * (0.5 / rho1) for x, y in zip(ug, fg)])
    _store(fi, _D3Q19, False, _collide(_D3Q19, v, rho1, un, w, False, fg), act)
    out = {"rho": torch.where(act, rho1, rho).reshape(-1),
           "u": torch.stack([torch.where(act, x, y) for x, y in zip(un, u)]).reshape(-1)}
    scale = 32768.0 if ft == "FP16S" else 1.0
    if ft != "FP16C":
        out.update(fi=torch.stack(fi).reshape(-1) * scale, ei=torch.stack(ei).reshape(-1) * scale,
                   fqi=torch.stack(fqi).reshape(-1) * scale)
    if ft == "FP32":
        out["q"] = torch.where(act, q, q0).reshape(-1)
    # 16-bit storage leaves its own rounding in the net charge, and a learned field has no exact value
    near = any(n // (1 << (1 << depth)) > 1 for n in (nx, ny, nz))
    if ft != "FP32" or mode == "SURROGATE" or near:
        out["e_dyn"] = out["b_dyn"] = None
    else:
        e, b = _field(nx, ny, nz, depth, q, ug, act)
        out["e_dyn"] = torch.where(act[None], k["ke"] * e, torch.zeros_like(e)).reshape(-1)
        stat = torch.stack(bs)
        out["b_dyn"] = torch.where(act[None], stat + k["kmu"] * b, stat).reshape(-1)
    return out


def _disk_cells(n, mesh):
    """Cells (x, y, z) inside a convex mesh as the voxeliser has them: rays along the axis of the box's smallest face
    (the mesh grown by 2 cells) through the cell centres, distances from the first cell whole numbers; a ray's cells lie
    above its first hit and below its last."""
    p = [torch.from_numpy(np.asarray(v, np.float64)) for v in mesh]
    lo, hi = torch.stack(p).amin((0, 1)) - 2.0, torch.stack(p).amax((0, 1)) + 2.0
    d = hi - lo
    face = [float(d[1] * d[2]), float(d[2] * d[0]), float(d[0] * d[1])]
    axis = 0 if face[0] < face[1] and face[0] < face[2] else 1 if face[1] < face[2] else 2
    i, j = [a for a in range(3) if a != axis]
    start = float(min(max(int(lo[axis]), 0), n - 1))
    g = torch.arange(n, dtype=torch.float64)
    a, b = g[:, None].expand(n, n), g[None, :].expand(n, n)
    first, last = torch.full((n, n), math.inf, dtype=torch.float64), torch.full((n, n), -math.inf, dtype=torch.float64)
    for v0, v1, v2 in zip(*p):
        det = (v1[i] - v0[i]) * (v2[j] - v0[j]) - (v2[i] - v0[i]) * (v1[j] - v0[j])
        if det == 0.0:
            continue
        s = ((a - v0[i]) * (v2[j] - v0[j]) - (v2[i] - v0[i]) * (b - v0[j])) / det
        t = ((v1[i] - v0[i]) * (b - v0[j]) - (a - v0[i]) * (v1[j] - v0[j])) / det
        hit = (s >= 0) & (t >= 0) & (s + t < 1)
        at = torch.floor(v0[axis] + s * (v1[axis] - v0[axis]) + t * (v2[axis] - v0[axis]) - start)
        first = torch.where(hit, torch.minimum(first, at), first)
        last = torch.where(hit, torch.maximum(last, at), last)
    h = g[None, None, :] - start
    inside = (h > first[..., None]) & (h < last[..., None])
    where = torch.nonzero(inside)
    out = torch.empty_like(where)
    out[:, i], out[:, j], out[:, axis] = where[:, 0], where[:, 1], where[:, 2]
    return out


def _magnet_exact(case, seed):
    m = torch.tensor(_magnetization(seed), dtype=torch.float64, device="cuda") / (UNITS["a"] / UNITS["m"])
    n = case["n"] // 4 * 4
    c, r, t = _disk(case)
    cells = _disk_cells(n, I.cylinder(c, r, t, axis=2)).double().cuda() + 1.0
    ax = torch.arange(n + 2, dtype=torch.float64, device="cuda")
    psi = torch.zeros(n + 2, n + 2, n + 2, dtype=torch.float64, device="cuda")
    chunk = max(1, (1 << 23) // (n + 2) ** 3)
    for lo in range(0, cells.shape[0], chunk):
        at = cells[lo:lo + chunk]
        dx = ax[None, None, None, :] - at[:, 0, None, None, None]
        dy = ax[None, None, :, None] - at[:, 1, None, None, None]
        dz = ax[None, :, None, None] - at[:, 2, None, None, None]
        r2 = (dx * dx + dy * dy) + dz * dz
        inv = torch.where(r2 == 0.0, 0.0, r2.pow(-1.5))
        psi += (((dx * m[0] + dy * m[1]) + dz * m[2]) * inv).sum(0)
    psi /= 4.0 * math.pi
    grad = [(psi[1:-1, 1:-1, 2:] - psi[1:-1, 1:-1, :-2]) / 2, (psi[1:-1, 2:, 1:-1] - psi[1:-1, :-2, 1:-1]) / 2,
            (psi[2:, 1:-1, 1:-1] - psi[:-2, 1:-1, 1:-1]) / 2]
    b = torch.stack(grad) * -_constants()["kmu0"]
    magnet = torch.zeros(n, n, n, dtype=torch.bool, device="cuda")
    i = (cells - 1.0).long()
    magnet[i[:, 2], i[:, 1], i[:, 0]] = True
    return {"flags": None, "b_stat": torch.where(magnet[None], torch.zeros_like(b), b).reshape(-1)}


def exact(case, seed):
    if case["kind"] == "plain":
        return _plain_exact(case, seed)
    if case["kind"] == "mhd":
        return _mhd_exact(case["nx"], case["ny"], case["nz"], case["depth"], case["ft"], case["mode"], seed)
    if case["kind"] == "batch":
        outs = [_mhd_exact(n, n, n, 4, case["ft"], "FAST", s) for n, s in _domains(case, seed)]
        return [{k: o[k] for k in ("u", "e_dyn")} for o in outs]
    return _magnet_exact(case, seed)
