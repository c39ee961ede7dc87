"""The work that programs built on this package have it do, as measurable cases.

Every case is one call sequence through the public entry points: structured boxes (``Box``), levels
in the reference layout (``Simulation``) and domain pools (``Pool``), advanced some time steps, with
the fields a program reads afterwards. ``exact`` restates the same physics in plain torch, in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

from virtualfluids_b200 import BoundaryConditionFactory as BCF
from virtualfluids_b200 import Box, GridScalingFactory, ListGrid, MultiLevelGrid, Parameter, Pool, Simulation
from virtualfluids_b200 import _native as N
from virtualfluids_b200 import workloads

DEV = "cuda"
BYTES = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2, "e3m12": 2}
STORAGE = {"f64": N.STORAGE_F64, "f32": N.STORAGE_F32, "f16": N.STORAGE_F16, "bf16": N.STORAGE_BF16,
           "e3m12": N.STORAGE_E3M12}


def listed():
    return [
        # the benchmark of the package: Taylor-Green box in the reference's arithmetic, energy every step
        {"name": "box_f64_exact_256", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "storage": "f64",
         "arith": "exact", "steps": 4, "energy": True, "solve": False},
        # a periodic turbulence box of sizes nobody tuned for, in the default double arithmetic
        {"name": "box_f64_ragged", "kind": "box", "nx": 201, "ny": 135, "nz": 170, "storage": "f64", "arith": "fast",
         "steps": 8, "energy": False, "solve": False},
        # a large single-precision box, the storage most production runs use
        {"name": "box_f32_large", "kind": "box", "nx": 320, "ny": 256, "nz": 192, "storage": "f32", "arith": "fast",
         "steps": 8, "energy": True, "solve": False},
        # a compressed box: 16-bit populations, stochastic rounding
        {"name": "box_f16_ragged", "kind": "box", "nx": 250, "ny": 190, "nz": 230, "storage": "f16", "arith": "fast",
         "steps": 8, "energy": False, "solve": False},
        # one small solve of a parameter sweep: initialise, advance, read the fields; launches count
        {"name": "box_f32_small_solve", "kind": "box", "nx": 32, "ny": 32, "nz": 32, "storage": "f32",
         "arith": "fast", "steps": 64, "energy": False, "solve": True},
        # setting a level up and writing it out: initial fields in, macroscopic fields out
        {"name": "box_f64_set_up_and_output", "kind": "box", "nx": 192, "ny": 160, "nz": 144, "storage": "f64",
         "arith": "fast", "steps": 0, "energy": False, "solve": True},
        # the lid-driven cavity of the reference's application, reference layout and arithmetic
        {"name": "cavity_f64_exact_64", "kind": "cavity", "nx": 64, "ny": 64, "nz": 64, "storage": "f64",
         "arith": "exact", "steps": 20},
        # a channel past a cube on the reference layout: interpolated walls, inlet, pressure outlet
        {"name": "channel_list_f32", "kind": "channel", "path": "list", "nx": 131, "ny": 67, "nz": 75, "cube": 9,
         "storage": "f32", "arith": "fast", "steps": 32},
        # the duct past a wall-mounted cube on a structured box, with the drag of every step
        {"name": "channel_box_f32", "kind": "channel", "path": "box", "nx": 256, "ny": 128, "nz": 128, "cube": 16,
         "storage": "f32", "arith": "fast", "steps": 16},
        # two nested levels: the fine level takes two steps per coarse one, interpolation both ways
        {"name": "refined_f64", "kind": "refined", "n": 48, "lo": 13, "hi": 35, "storage": "f64", "arith": "fast",
         "steps": 10},
        # a batch of ducts of uneven sizes in one pool, as a sweep over shapes and Reynolds numbers
        {"name": "pool_ducts_f16", "kind": "ducts", "count": 192, "storage": "f16", "arith": "fast", "steps": 48},
        # porous blocks with exact sphere distances between pressure planes, as the serving loop steps them
        {"name": "pool_porous_f32", "kind": "porous", "sides": "96,64,81", "porosity": 0.75, "storage": "f32",
         "arith": "fast", "steps": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "box", "cavity", "channel", "channel", "refined", "ducts", "porous"])
    if kind == "box":
        nx, ny, nz = _log(rng, 17, 320), _log(rng, 17, 256), _log(rng, 17, 256)
        while nx * ny * nz > 1 << 24:
            nx, ny, nz = nx - nx // 8, ny - ny // 8, nz - nz // 8
        storage = rng.choice(["f64", "f64", "f32", "f32", "f16", "bf16", "e3m12"])
        arith = rng.choice(["fast", "exact"]) if BYTES[storage] == 8 else "fast"
        solve = rng.random() < 0.3
        steps = max(4, min(64, int(6e7 / (nx * ny * nz) / (BYTES[storage] / 4 if BYTES[storage] > 4 else 1))))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "storage": storage, "arith": arith, "steps": steps,
                "energy": rng.random() < 0.3, "solve": solve}
    if kind == "cavity":
        storage = rng.choice(["f64", "f32"])
        return {"kind": kind, "nx": _log(rng, 20, 96), "ny": _log(rng, 20, 96), "nz": _log(rng, 20, 96),
                "storage": storage, "arith": rng.choice(["exact", "fast"]), "steps": 20}
    if kind == "channel":
        ny, nz = _log(rng, 32, 128), _log(rng, 32, 128)
        return {"kind": kind, "path": rng.choice(["list", "box"]), "nx": _log(rng, 64, 256), "ny": ny, "nz": nz,
                "cube": rng.randrange(5, min(ny, nz) // 3), "storage": rng.choice(["f32", "f64"]), "arith": "fast",
                "steps": 16}
    if kind == "refined":
        n = rng.randrange(24, 60)
        lo = rng.randrange(5, n // 3)
        return {"kind": kind, "n": n, "lo": lo, "hi": rng.randrange(lo + 8, n - 5), "storage": rng.choice(["f64", "f32"]),
                "arith": "fast", "steps": 10}
    if kind == "ducts":
        storage = rng.choice(["f32", "f16"])
        return {"kind": kind, "count": _log(rng, 12, 192) // (2 if storage == "f32" else 1), "storage": storage,
                "arith": "fast", "steps": 48}
    return {"kind": kind, "sides": ",".join(str(_log(rng, 32, 96)) for _ in range(rng.randrange(1, 4))),
            "porosity": round(rng.uniform(0.72, 0.85), 3), "storage": rng.choice(["f32", "f16"]), "arith": "fast",
            "steps": 32}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _real(case):
    return torch.float64 if case["storage"] == "f64" else torch.float32


def _modes(shape, seed, positions=None, periods=None, amp_rho=1e-2, amp_u=0.03):
    """drho, ux, uy, uz: a large-scale vortex field of seeded wave vectors and phases (three product
    modes per component), x fastest; float64 on the device."""
    g = np.random.default_rng(seed)
    if positions is None:
        nx, ny, nz = shape
        ax = [torch.arange(n, dtype=torch.float64, device=DEV) for n in (nx, ny, nz)]
        x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
        periods = shape
    else:
        x, y, z = positions
    out = []
    for amp in (amp_rho, amp_u, amp_u, amp_u):
        f = 0.0
        for _ in range(3):
            k, ph = g.integers(1, 3, 3), g.uniform(0, 2 * np.pi, 3)
            f = f + amp / 3 * (torch.cos(2 * np.pi * k[0] / periods[0] * x + ph[0])
                               * torch.cos(2 * np.pi * k[1] / periods[1] * y + ph[1])
                               * torch.cos(2 * np.pi * k[2] / periods[2] * z + ph[2]))
        out.append(f.reshape(-1).contiguous())
    return out


def _box_inputs(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    g = np.random.default_rng(seed + 7)
    return {"shape": shape, "omega": float(g.uniform(1.85, 1.95)),
            "fields": [f.to(_real(case)) for f in _modes(shape, seed)]}


def _cavity_inputs(case, seed):
    g = np.random.default_rng(seed + 7)
    grid = ListGrid(case["nx"], case["ny"], case["nz"])
    for side in ("PX", "MX", "PY", "MY", "MZ"):
        grid.add_side(side, "noslip")
    lid = float(g.uniform(0.04, 0.06))
    grid.add_side("PZ", "velocity", velocity=(lid, 0.3 * lid, 0.0))
    return grid, float(g.uniform(0.008, 0.012))


def _channel_inputs(case, seed):
    g = np.random.default_rng(seed + 7)
    u = float(g.uniform(0.04, 0.05))
    nu = float(g.uniform(0.006, 0.010))
    grid, omega, _ = workloads.cube_duct(case["nx"], case["ny"], case["nz"], cube=case["cube"], x0=case["nx"] // 4,
                                         u_max=u, re=u * case["cube"] / nu)
    # started at the inlet's profile with a seeded perturbation
    x, y, z = (torch.from_numpy(grid.coords[a].astype(np.float64)).to(DEV) for a in range(3))
    eta, zeta = (y + 0.5) / grid.ny, (z + 0.5) / grid.nz
    env = 16 * eta * (1 - eta) * zeta * (1 - zeta)
    inside = torch.from_numpy(grid.geo == N.GEO_FLUID).to(DEV)
    env = torch.where(inside, env, torch.zeros_like(env))
    m = _modes(None, seed, (x, y, z), (grid.nx, grid.ny, grid.nz), amp_rho=2e-3, amp_u=0.3 * u)
    fields = [m[0] * env, (u + m[1]) * env, m[2] * env, m[3] * env]
    return grid, float(omega), fields


def _refined_inputs(case, seed):
    m = MultiLevelGrid.uniform(ListGrid(case["n"], case["n"], case["n"], periodic=(True, True, True)))
    m.refine((case["lo"],) * 3, (case["hi"],) * 3)
    return m


def _ducts_inputs(case, seed):
    ducts = workloads.duct_batch(case["count"], seed=case["count"])     # the sweep; the seed makes its start
    out = []
    for i, d in enumerate(ducts):
        nx, ny, nz = d["shape"]
        fields = _modes(d["shape"], seed + 1000 + i, amp_rho=5e-3, amp_u=0.01)
        eta = (torch.arange(ny, dtype=torch.float64, device=DEV) - 0.5) / (ny - 2)
        zeta = (torch.arange(nz, dtype=torch.float64, device=DEV) - 0.5) / (nz - 2)
        env = (16 * eta * (1 - eta))[None, :, None] * (zeta * (1 - zeta))[:, None, None]
        env = env.clamp(min=0).expand(nz, ny, nx).reshape(-1)
        fields = [f * env for f in fields]
        fields[1] = fields[1] + 0.03 * env
        out.append((d, [f.to(_real(case)) for f in fields]))
    return out


def _porous_inputs(case, seed):
    out = []
    for i, side in enumerate(int(v) for v in case["sides"].split(",")):
        b = workloads.porous_block_bcs(side, seed + 31 * i, porosity=case["porosity"])
        g = np.random.default_rng(seed + 7 + i)
        m = torch.from_numpy(b["mask"]).to(DEV).double()
        fields = [f * m for f in _modes(b["shape"], seed + 100 + i, amp_rho=2e-3, amp_u=5e-3)]
        out.append((b, 1.0 / (3.0 * float(g.uniform(0.012, 0.0167)) + 0.5), [f.to(_real(case)) for f in fields]))
    return out


def _parameter(case, nu):
    p = Parameter()
    p.set_viscosity_lb(nu)
    p.configure_main_kernel("K17CompressibleNavierStokes")
    p.storage = STORAGE[case["storage"]]
    p.arith = N.ARITH_EXACT if case["arith"] == "exact" else N.ARITH_FAST
    return p


def _interpolated_factory():
    bcf = BCF()
    bcf.set_no_slip_boundary_condition(BCF.NoSlipBC.NoSlipInterpolatedCompressible)
    bcf.set_geometry_boundary_condition(BCF.NoSlipBC.NoSlipInterpolatedCompressible)
    bcf.set_velocity_boundary_condition(BCF.VelocityBC.VelocityInterpolatedCompressible)
    bcf.set_pressure_boundary_condition(BCF.PressureBC.PressureNonEquilibriumCompressible)
    return bcf


def _empty(n, like, count=4):
    return [torch.empty(n, dtype=like, device=DEV) for _ in range(count)]


def prepare(case, seed):
    kind, real = case["kind"], _real(case)
    if kind == "box":
        i = _box_inputs(case, seed)
        box = Box(*i["shape"], i["omega"], storage=case["storage"], arith=case["arith"])
        if not case["solve"]:
            box.init(*i["fields"])
        energy = torch.empty(2 * case["steps"], dtype=torch.float64, device=DEV) if case["energy"] else None
        return {"case": case, "box": box, "fields": i["fields"], "energy": energy, "out": _empty(box.n, real)}
    if kind == "cavity":
        grid, nu = _cavity_inputs(case, seed)
        bcf = BCF()
        bcf.set_no_slip_boundary_condition(BCF.NoSlipBC.NoSlipBounceBack)
        bcf.set_velocity_boundary_condition(BCF.VelocityBC.VelocityBounceBack)
        sim = Simulation(_parameter(case, nu), grid, bcf)
        sim.init()
        return {"case": case, "sim": sim}
    if kind == "channel":
        grid, omega, fields = _channel_inputs(case, seed)
        if case["path"] == "list":
            sim = Simulation(_parameter(case, (1 / omega - 0.5) / 3), grid, _interpolated_factory())
            sim.init(*(f.cpu().numpy() for f in fields))
            sim.set_graph(16)
            return {"case": case, "sim": sim}
        box = Box.from_grid(grid, omega, _interpolated_factory(), storage=case["storage"], arith=case["arith"])
        f0 = grid.first_node
        box.init(*(f[f0:f0 + box.n].to(real).contiguous() for f in fields))
        box.enable_drag_lift(case["steps"])
        return {"case": case, "box": box, "energy": None, "out": _empty(box.n, real)}
    if kind == "refined":
        m = _refined_inputs(case, seed)
        scaling = GridScalingFactory()
        scaling.set_scaling_factory(GridScalingFactory.GridScaling.ScaleCompressible)
        sim = Simulation(_parameter(case, 0.01), m, BCF(), scaling)
        for level in range(2):
            pos = [torch.from_numpy(p).to(DEV) for p in m.positions(level)]
            f = _modes(None, seed, pos, (case["n"],) * 3, amp_rho=5e-3, amp_u=0.02)
            f = [v.cpu().numpy() for v in f]
            for v in f:
                v[0] = 0.0
            sim.init(*f, level=level)
        return {"case": case, "sim": sim}
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    domains = _ducts_inputs(case, seed) if kind == "ducts" else _porous_inputs(case, seed)
    args = []
    for d in domains:
        if kind == "ducts":
            args.append(dict(shape=d[0]["shape"], omega=d[0]["omega"], periodic=(True, False, False),
                             forces=(d[0]["g"], 0.0, 0.0)))
        else:
            args.append(dict(shape=d[0]["shape"], omega=d[1], periodic=(False, True, True), mask=d[0]["mask"],
                             bcs=d[0]["bcs"]))
    need = 0
    probe = Pool(1 << 20, storage=case["storage"], max_domains=4)
    for a in args:
        need += probe.domain_bytes(a["shape"], a["omega"], a["periodic"], has_mask=True, bcs=a.get("bcs"))
    probe.close()
    pool = Pool(need + (1 << 20), storage=case["storage"], max_domains=max(8, len(args)))
    ids, at, total = [], [], 0
    for a, d in zip(args, domains):
        ids.append(pool.add(**a))
        pool.init(ids[-1], *d[-1], stream=stream)
        at.append(total)
        total += math.prod(a["shape"])
    torch.cuda.synchronize()
    return {"case": case, "pool": pool, "ids": ids, "at": at, "stream": stream, "out": _empty(total, real)}


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _macroscopic(sim, level):
    """The level's macroscopic output, left in its device arrays (rho, vx, vy, vz)."""
    s = sim.levels[level]
    N.check(N.lib().vfb_calc_macroscopic_compressible(ctypes.byref(s.level), None))
    return [s.rho, s.vx, s.vy, s.vz]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("box", "channel") and "box" in state:
        box = state["box"]
        if kind == "box" and case["solve"]:
            box.init(*state["fields"])
        if case["steps"]:
            box.step(case["steps"], energy=state["energy"])
        out = {"fields": box.fields(out=state["out"])}
        if state["energy"] is not None:
            out["energy"] = state["energy"]
        if kind == "channel":
            out["force"] = box.drag_lift_history()
        return out
    if "sim" in state:
        sim = state["sim"]
        sim.run(case["steps"])
        return [_macroscopic(sim, level) for level in range(len(sim.levels))]
    pool, stream = state["pool"], state["stream"]
    pool.step(case["steps"], stream=stream)
    lib, size = N.lib(), state["out"][0].element_size()
    base = [o.data_ptr() for o in state["out"]]
    handle = ctypes.c_void_p(stream.cuda_stream)
    for i, at in zip(state["ids"], state["at"]):
        N.check(lib.vfb_pool_domain_fields(pool._h, i, *(ctypes.c_void_p(b + at * size) for b in base), 0, handle))
    torch.cuda.current_stream().wait_stream(stream)
    return state["out"]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    """Per node update 27 populations read and 27 written and about 830 operations (K17 with fused
    multiply-adds; 1250 as the reference spells it); fields out, and in for a solve."""
    s, real = BYTES[case["storage"]], 8 if case["storage"] == "f64" else 4
    ops = 1250 if case["arith"] == "exact" else 830
    kind = case["kind"]
    if kind in ("box", "cavity", "channel"):
        n = case["nx"] * case["ny"] * case["nz"]
        updates = n * case["steps"]
    elif kind == "refined":
        fine = 8 * (case["hi"] - case["lo"]) ** 3
        n = case["n"] ** 3 + fine
        updates = (case["n"] ** 3 + 2 * fine) * case["steps"]
    elif kind == "ducts":
        n = case["count"] * 80000       # mean of the batch's log-uniform sides, walls left out
        updates = n * case["steps"]
    else:
        n = sum(int(v) ** 3 for v in case["sides"].split(","))
        updates = int(n * case["porosity"]) * case["steps"]
    b = updates * 54 * s + n * (27 * s + 4 * real)
    if case.get("solve"):
        b += n * (27 * s + 4 * real)
    return {"bytes": b, "flops": updates * ops + n * 120}


def tolerance(case):
    """Four times what two orders of the same sums showed on B200 (FP64 up to 6e-15 from ``exact``, FP32 up to
    2.6e-6). The 16-bit forms round stochastically with bits hashed from the value, so a last-bit
    change of one value draws other bits in all that follow: two runs differ by the rounding noise
    (FP16 up to 3e-3 from ``exact``, in the ducts' drho)."""
    s = case["storage"]
    if s == "f64":
        return {"rel": 1e-13, "max": 1e-11}
    if s == "f32":
        return {"rel": 2e-5, "max": 2e-3}
    return {"rel": {"f16": 1.2e-2, "bf16": 1.6e-2, "e3m12": 4e-3}[s], "max": 0.9}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
     (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
     (0, -1, 1), (1, 1, 1), (-1, 1, 1), (1, -1, 1), (-1, -1, 1), (1, 1, -1), (-1, 1, -1), (1, -1, -1), (-1, -1, -1)]
INV = [C.index((-a, -b, -c)) for a, b, c in C]
WEIGHT = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[abs(a) + abs(b) + abs(c)] for a, b, c in C]
LINE = (1 / 6, 2 / 3, 1 / 6)    # weights along one axis
MU = (1.0, 0.0, 1 / 3)          # their moments


def _moments(f):
    """drho and the momenta of f (27 tensors)."""
    drho = sum(f)
    return (drho,) + tuple(sum(C[d][a] * f[d] for d in range(27) if C[d][a]) for a in range(3))


def _equilibrium(drho, u):
    usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = []
    for d in range(27):
        cu = sum(C[d][a] * u[a] for a in range(3))
        out.append(WEIGHT[d] * (drho + (1 + drho) * (3 * cu + 4.5 * cu * cu - usq)))
    return out


def _collide(f, w, force, lim=0.01):
    """The K17 cumulant collision (Geier et al., J. Comput. Phys. 348, 2017) of f - w: the
    post-collision populations, drho and the velocity with half the force."""
    drho, jx, jy, jz = _moments(f)
    r = 1 / (1 + drho)
    v = [j * r + 0.5 * g for j, g in zip((jx, jy, jz), force)]
    m = {(C[d][0] + 1, C[d][1] + 1, C[d][2] + 1): f[d] for d in range(27)}

    def lines(axis):
        for p in range(3):
            for q in range(3):
                at = [p, q]
                yield p, q, [tuple(at[:axis] + [t] + at[axis:]) for t in range(3)]

    # K of a line: the weights of the axes still in velocity space, the moments of the others
    offset = {2: lambda a, b: LINE[a] * LINE[b], 1: lambda a, c: LINE[a] * MU[c], 0: lambda b, c: MU[b] * MU[c]}
    for axis in (2, 1, 0):
        u = v[axis]
        for p, q, (i, j, k) in lines(axis):
            s, t = m[i] + m[k], m[k] - m[i]
            m0 = s + m[j]
            g = m0 + offset[axis](p, q)
            m[i], m[j], m[k] = m0, t - u * g, s - 2 * u * t + u * u * g
    vx2, vy2, vz2 = (u * u for u in v)
    op = 8 * (w - 2) * (1 + 2 * w) / (-8 - 14 * w + 7 * w * w)
    om = 8 * (w - 2) * (-7 + 4 * w) / (56 - 50 * w + 9 * w * w)
    oxyz = 24 * (w - 2) * (-2 - 7 * w + 3 * w * w) / (48 + 152 * w - 130 * w * w + 29 * w ** 3)
    fa = (4 + 2 * w - 3 * w * w) / (2 - 7 * w + 5 * w * w)
    fb = (4 + 28 * w - 14 * w * w) / (6 - 21 * w + 15 * w * w)
    trace = m[2, 0, 0] + m[0, 2, 0] + m[0, 0, 2]
    dy, dz = m[2, 0, 0] - m[0, 2, 0], m[2, 0, 0] - m[0, 0, 2]
    gxy, gxz, gyz = (-3 * w * m[i] for i in ((1, 1, 0), (1, 0, 1), (0, 1, 1)))
    gx = -w / 2 * (dy + dz) + (m[0, 0, 0] - trace) / 2
    gy, gz = gx + 1.5 * w * dy, gx + 1.5 * w * dz
    trace = m[0, 0, 0] - 1.5 * (vx2 * gx + vy2 * gy + vz2 * gz)
    dy = (1 - w) * dy - 3 * (1 - w / 2) * (vx2 * gx - vy2 * gy)
    dz = (1 - w) * dz - 3 * (1 - w / 2) * (vx2 * gx - vz2 * gz)
    b, c, a = (1 - w) * m[0, 1, 1], (1 - w) * m[1, 0, 1], (1 - w) * m[1, 1, 0]     # yz, xz, xy

    def relax(x, rate):
        return x - (rate + (1 - rate) * x.abs() / (x.abs() + lim)) * x

    xyz = relax(m[1, 1, 1], oxyz)
    plus, minus = {}, {}
    for i, j in (((2, 1, 0), (0, 1, 2)), ((2, 0, 1), (0, 2, 1)), ((1, 2, 0), (1, 0, 2))):
        plus[i], minus[i] = relax(m[i] + m[j], op), relax(m[i] - m[j], om)
        m[i], m[j] = (plus[i] + minus[i]) / 2, (plus[i] - minus[i]) / 2
    xx, yy, zz = (dy + dz + trace) / 3, (trace - 2 * dy + dz) / 3, (trace + dy - 2 * dz) / 3
    k = -(1 / w - 0.5)
    q220, q202, q022 = (k * s * (2 / 3) * fa for s in (gy + gx, gx + gz, gy + gz))
    q112, q121, q211 = (k * s / 3 * fb for s in (gxy, gxz, gyz))
    q211 = q211 + ((3 * xx + 1) * b + 6 * a * c) * r / 3
    q121 = q121 + ((3 * yy + 1) * c + 6 * a * b) * r / 3
    q112 = q112 + ((3 * zz + 1) * a + 6 * c * b) * r / 3

    def fourth(q, x, y, s):
        return q + ((9 * (x * y + 2 * s * s) + 3 * (x + y)) * r - drho * r) / 9

    q220, q202, q022 = fourth(q220, xx, yy, a), fourth(q202, xx, zz, c), fourth(q022, yy, zz, b)

    def fifth(p, x, q, y, s, t, p1, u, p2):
        return (3 * (p * x + q * y + 4 * s * xyz + 2 * (t * p1 + u * p2)) + x + y) * r / 3

    q122 = fifth(zz, m[1, 2, 0], yy, m[1, 0, 2], b, c, m[0, 2, 1], a, m[0, 1, 2])
    q212 = fifth(zz, m[2, 1, 0], xx, m[0, 1, 2], c, b, m[2, 0, 1], a, m[1, 0, 2])
    q221 = fifth(xx, m[0, 2, 1], yy, m[2, 0, 1], a, c, m[1, 2, 0], b, m[2, 1, 0])
    q222 = -(-(4 * xyz * xyz + xx * q022 + yy * q202 + zz * q220 + 4 * (b * q211 + c * q121 + a * q112)
               + 2 * (m[1, 2, 0] * m[1, 0, 2] + m[2, 1, 0] * m[0, 1, 2] + m[2, 0, 1] * m[0, 2, 1])) * r
             + (4 * (c * c * yy + b * b * xx + a * a * zz) + 2 * xx * yy * zz + 16 * a * b * c) * r * r
             - ((q022 + q202 + q220) / 3 + trace_of(xx, yy, zz) / 9) * r
             + (2 * (c * c + b * b + a * a) + zz * yy + zz * xx + yy * xx + trace_of(xx, yy, zz) / 3) * r * r * (2 / 3)
             + (drho * drho - drho) * r * r / 27)
    m.update({(2, 0, 0): xx, (0, 2, 0): yy, (0, 0, 2): zz, (1, 1, 0): a, (1, 0, 1): c, (0, 1, 1): b, (1, 1, 1): xyz,
              (2, 2, 0): q220, (2, 0, 2): q202, (0, 2, 2): q022, (1, 1, 2): q112, (1, 2, 1): q121, (2, 1, 1): q211,
              (1, 2, 2): q122, (2, 1, 2): q212, (2, 2, 1): q221, (2, 2, 2): q222, (1, 0, 0): -m[1, 0, 0],
              (0, 1, 0): -m[0, 1, 0], (0, 0, 1): -m[0, 0, 1]})
    for axis in (0, 1, 2):
        u = v[axis]
        for p, q, (i, j, k3) in lines(axis):
            g, bv = m[i] + offset[axis](p, q), m[j] * u
            m[i], m[j], m[k3] = ((m[k3] - m[j] + g * (u * u - u)) / 2 + bv, m[i] - m[k3] - 2 * bv - g * u * u,
                                 (m[k3] + m[j] + g * (u * u + u)) / 2 + bv)
    return [m[C[d][0] + 1, C[d][1] + 1, C[d][2] + 1] for d in range(27)], drho, v


def trace_of(xx, yy, zz):
    return xx + yy + zz


class _Plain:
    """Boxes of nodes, x fastest, one behind the other in flat 64-bit arrays: collide, stream,
    boundary lists; links into solid nodes without a list bounce back one step late (the value waits
    at the solid node). domains: (shape, omega, fields, forces, fluid or None) each."""

    def __init__(self, domains):
        one = len(domains) == 1
        self.at, n = [], 0
        for shape, *_ in domains:
            self.at.append(n)
            n += math.prod(shape)
        drho, *u = (torch.cat([d[2][i].double().reshape(-1) for d in domains]) for i in range(4))
        self.f = _equilibrium(drho, u)

        def per_node(values):
            if one:
                return values[0]
            return torch.cat([torch.full((math.prod(d[0]),), v, dtype=torch.float64, device=DEV)
                              for d, v in zip(domains, values)])

        self.omega = per_node([d[1] for d in domains])
        self.forces = [per_node([d[3][i] for d in domains]) for i in range(3)]
        self.fluid = self.held = None
        # the node that direction d comes from
        self.source = []
        for c in C:
            parts = []
            for (shape, *_), at in zip(domains, self.at):
                nx, ny, nz = shape
                x, y, z = ((torch.arange(m, device=DEV) - c[i]) % m for i, m in enumerate((nx, ny, nz)))
                parts.append((at + x[None, None, :] + nx * (y[None, :, None] + ny * z[:, None, None])).reshape(-1))
            self.source.append(torch.cat(parts))
        if domains[0][4] is not None:
            self.fluid = torch.cat([d[4].reshape(-1) for d in domains])
            self.f = [x * self.fluid for x in self.f]
            self.from_solid = [~self.fluid[i] & self.fluid for i in self.source]
            self.held = list(self.f)

    def step(self, lists=(), pressure=(), drag=None, bounce_back=False):
        n = self.f[0].numel()
        post, energy = [torch.empty_like(self.f[0]) for _ in range(27)], [0.0, 0.0]

        def part(x, at):
            return x[at] if torch.is_tensor(x) else x

        for at in range(0, n, 1 << 22):
            at = slice(at, min(n, at + (1 << 22)))
            p, drho, v = _collide([x[at] for x in self.f], part(self.omega, at), [part(x, at) for x in self.forces])
            for d in range(27):
                post[d][at] = p[d]
            energy[0] = energy[0] + (1 + drho).sum()
            energy[1] = energy[1] + (0.5 * (1 + drho) * sum(u * u for u in v)).sum()
        new = [post[d][self.source[d]] for d in range(27)]
        if self.held is not None:
            new = [torch.where(self.from_solid[d], self.held[d], new[d]) * self.fluid for d in range(27)]
            self.held = [post[INV[d]] for d in range(27)]
        force = torch.zeros(3, dtype=torch.float64, device=DEV)
        for kind, k, q, vel in lists:
            p = [x[k] for x in post]
            for d in range(1, 27):
                cut = (q[d] >= 0) & (q[d] <= 1)
                if drag is not None and kind == "geometry":
                    force += torch.tensor(C[d], dtype=torch.float64, device=DEV) * (p[d] * cut).sum()
                e, wall = INV[d], None
                if vel is not None:
                    wall = sum(C[e if bounce_back else d][a] * vel[a] for a in range(3))
                if bounce_back:
                    val = p[d] if wall is None else p[d] + 6 * WEIGHT[d] * wall
                else:
                    val = _interpolated(p, d, q[d], wall, part(self.omega, k))
                new[e][k[cut]] = val[cut]
        if drag is not None:
            _, k, q, _ = next(x for x in lists if x[0] == "geometry")
            for d in range(1, 27):
                cut = (q[INV[d]] >= 0) & (q[INV[d]] <= 1)
                force -= torch.tensor(C[d], dtype=torch.float64, device=DEV) * (new[d][k] * cut).sum()
            drag.append(force)
        for k, kn, rho, axis, sign in pressure:
            p = [x[kn] for x in new]
            drho, *j = _moments(p)
            u = [x / (1 + drho) for x in j]
            was, now = _equilibrium(drho, u), _equilibrium(rho, u)
            for d in range(27):
                if C[d][axis] != sign:
                    new[d][k] = p[d] - was[d] + now[d]
        self.f = new
        return torch.stack(energy)

    def fields(self):
        drho, *j = _moments(self.f)
        out = [drho] + [x / (1 + drho) for x in j]
        return out if self.fluid is None else [x * self.fluid for x in out]


def _interpolated(p, d, q, wall, omega):
    """Interpolated bounce-back of one direction (Bouzidi-type, with the collision's equilibrium)."""
    drho, *j = _moments(p)
    u = [x / (1 + drho) for x in j]
    cu = sum(C[d][a] * u[a] for a in range(3))
    usq = 1.5 * sum(x * x for x in u) * (1 + drho)
    feq = WEIGHT[d] * (drho + 4.5 * cu * cu * (1 + drho) - usq)
    f, g = p[d], p[INV[d]]
    moved = 0.0 if wall is None else 6 * WEIGHT[d] * wall
    return (1 - q) / (1 + q) * (f - g + (f + g - 2 * feq * omega) / (1 - omega)) / 2 + (q * (f + g) - moved) / (1 + q)


def _grid_lists(grid, real):
    """The grid's boundary lists in box indices, q and velocities rounded to the level's real type."""
    lists, pressure, f0 = [], [], grid.first_node
    for kind in ("velocity", "noslip", "geometry"):
        m = grid.merged(kind)
        if m is None:
            continue
        k, q, vel = (torch.from_numpy(np.ascontiguousarray(x)).to(DEV) for x in m)
        lists.append((kind, k.long() - f0, q.to(real).double(), vel.to(real).double() if kind == "velocity" else None))
    for b in grid.bcs:
        if b.kind == "pressure":
            k, kn = (torch.from_numpy(x.astype(np.int64) - f0).to(DEV) for x in (b.k, b.k_neighbor))
            axis, sign = {"MX": (0, -1), "PX": (0, 1)}[b.side]
            pressure.append((k, kn, torch.full(k.shape, float(b.rho), dtype=torch.float64, device=DEV), axis, sign))
    return lists, pressure


def exact(case, seed):
    kind, real = case["kind"], _real(case)
    if kind == "refined":
        return None     # no plain form of the two-level coupling short enough to be its own check
    if kind == "box":
        i = _box_inputs(case, seed)
        p = _Plain([(i["shape"], i["omega"], i["fields"], (0.0, 0.0, 0.0), None)])
        energy = [p.step() for _ in range(case["steps"])]
        out = {"fields": p.fields()}
        if case["energy"]:
            out["energy"] = torch.cat(energy)
        return out
    if kind in ("cavity", "channel"):
        if kind == "cavity":
            grid, nu = _cavity_inputs(case, seed)
            omega, fields = 1 / (3 * nu + 0.5), [torch.zeros(grid.number_of_nodes, dtype=torch.float64, device=DEV)] * 4
        else:
            grid, omega, fields = _channel_inputs(case, seed)
        f0, n = grid.first_node, math.prod(grid.dims)
        fluid = torch.from_numpy(grid.geo[f0:f0 + n] == N.GEO_FLUID).to(DEV)
        lists, pressure = _grid_lists(grid, real)
        p = _Plain([(grid.dims, omega, [f[f0:f0 + n].to(real) for f in fields], (0.0, 0.0, 0.0), fluid)])
        drag = [] if case.get("path") == "box" else None
        for _ in range(case["steps"]):
            p.step(lists, pressure, drag, bounce_back=kind == "cavity")
        if drag is not None:
            return {"fields": p.fields(), "force": torch.stack(drag)}
        out = []
        for x in p.fields():
            full = torch.zeros(grid.number_of_nodes, dtype=torch.float64, device=DEV)
            full[f0:f0 + n] = x
            out.append(full)
        return [out]
    domains, blocks = [], []
    if kind == "ducts":
        for d, fields in _ducts_inputs(case, seed):
            nx, ny, nz = d["shape"]
            fluid = torch.zeros((nz, ny, nx), dtype=torch.bool, device=DEV)
            fluid[1:-1, 1:-1] = True
            domains.append((d["shape"], d["omega"], fields, (d["g"], 0.0, 0.0), fluid))
    else:
        blocks = _porous_inputs(case, seed)
        for b, omega, fields in blocks:
            domains.append((b["shape"], omega, fields, (0.0, 0.0, 0.0), torch.from_numpy(b["mask"] != 0).to(DEV)))
    p = _Plain(domains)
    lists, pressure = [], []
    for (b, _, _), at in zip(blocks, p.at):
        k, q = (torch.from_numpy(np.ascontiguousarray(x)).to(DEV) for x in b["bcs"]["noslip"])
        lists.append(("noslip", k.long() + at, q.to(real).double(), None))
        pk, pn, rho, direction = (torch.from_numpy(x).to(DEV) for x in b["bcs"]["pressure"])
        for code, sign in ((N.DIR_M00, -1), (N.DIR_P00, 1)):
            i = direction == code
            pressure.append((pk[i].long() + at, pn[i].long() + at, rho[i].to(real).double(), 0, sign))
    for _ in range(case["steps"]):
        p.step(lists, pressure)
    return p.fields()
