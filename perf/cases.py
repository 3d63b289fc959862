"""Timed work of the framework, through its public entry points.

listed() names the cases and draw(rng) gives more of the same ranges. prepare(case, seed) builds
what a user's program holds before the call (a solver with its state, bodies and poses),
run(state) is one pass, work(case) the bytes and operations that a pass cannot do without, and
exact(case, seed) the first pass's result in binary64, computed with torch alone.

States are smooth random flows: a few long Fourier modes of velocity at the speeds that the
configurations use (0.02 to 0.05 lattice units), the matching density fluctuation, S = u u plus a
small non-equilibrium part, and noise of a few per cent of the speed in every cell.
"""
import math

import numpy as np
import torch

from openhomelbm_b200 import _lib, coupling
from openhomelbm_b200.batching import CapsuleChain, SwimmerBatch2D, SwimmerSpec, TileAutotuner
from openhomelbm_b200.lbm import LBM_Solver
from openhomelbm_b200.lbm3d import LBM_Solver3D
from openhomelbm_b200.serving import Domain, PlainDomain, Request

U_REF, S_REF = 0.05, 2.5e-3  # storage scales of the reduced types: the flow's speed and its square
SIZE = {"float64": 8, "float32": 4, "float16": 2, "bfloat16": 2}


def listed():
    return [
        # One step of the Karman wake: the smallest call, where the launches and the host count.
        {"name": "wake2d_512x128", "kind": "wake2d", "nx": 512, "ny": 128, "storage": "float32"},
        # A control step of a 2D learning environment: 24 same-size worlds of odd sides, two moving
        # bodies each, 8 LBM steps with poses in and loads out.
        {"name": "env2d_24x203x117", "kind": "env2d", "worlds": 24, "nx": 203, "ny": 117, "bodies": 2, "substeps": 8,
         "storage": "float32"},
        # The batching form: 60 uneven worlds with a capsule swimmer each, float16 storage, one
        # control step of 8 LBM steps.
        {"name": "batch2d_60_f16", "kind": "batch2d", "worlds": 60, "substeps": 8, "storage": "float16"},
        # One step of the periodic box of the headline benchmark.
        {"name": "box3d_256_f32", "kind": "box3d", "nx": 256, "ny": 256, "nz": 256, "storage": "float32"},
        # The same box in the reduced storage that the serving and precision forms use.
        {"name": "box3d_256_f16", "kind": "box3d", "nx": 256, "ny": 256, "nz": 256, "storage": "float16"},
        # The precision study's box, the largest field: 512^3 in bfloat16.
        {"name": "box3d_512_bf16", "kind": "box3d", "nx": 512, "ny": 512, "nz": 512, "storage": "bfloat16"},
        # The accuracy reference of that study (binary64 throughout).
        {"name": "box3d_192_f64", "kind": "box3d", "nx": 192, "ny": 192, "nz": 192, "storage": "float64"},
        # A channel of odd sides with an inlet, its flag field and outer boundaries.
        {"name": "duct3d_181x103x91", "kind": "duct3d", "nx": 181, "ny": 103, "nz": 91, "storage": "float32",
         "force": False, "diagnostics": False},
        # A channel with a body force and the mass and health diagnostics on.
        {"name": "duct3d_force_diag", "kind": "duct3d", "nx": 160, "ny": 96, "nz": 128, "storage": "float32",
         "force": True, "diagnostics": True},
        # A control step of one swimmer alone on the plain solver: 8 LBM steps with five moving
        # meshes, poses in and loads out. A small domain, where the launches follow one another.
        {"name": "swimmer3d_64_f32", "kind": "swimmer3d", "side": 64, "substeps": 8, "storage": "float32"},
        # The same at a size that fills the GPU.
        {"name": "swimmer3d_160_f32", "kind": "swimmer3d", "side": 160, "substeps": 8, "storage": "float32"},
        # A tick of the serving form: domains of different sides resident in float16, a control
        # step of 8 LBM steps of each, their kernels overlapping on the device.
        {"name": "served3d_mix_f16", "kind": "served3d", "sides": "64,64,96,96,96,128,128,160,192", "substeps": 8,
         "storage": "float16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wake2d", "env2d", "batch2d", "box3d", "box3d", "duct3d", "duct3d", "swimmer3d", "served3d"])
    if kind == "wake2d":
        return {"kind": kind, "nx": _log_int(rng, 96, 1500), "ny": _log_int(rng, 48, 400),
                "storage": rng.choice(["float32", "float16"])}
    if kind == "env2d":
        return {"kind": kind, "worlds": _log_int(rng, 1, 32), "nx": _log_int(rng, 64, 320), "ny": _log_int(rng, 48, 200),
                "bodies": rng.randint(1, 3), "substeps": rng.choice([4, 8, 10]), "storage": "float32"}
    if kind == "batch2d":
        return {"kind": kind, "worlds": _log_int(rng, 8, 60), "substeps": rng.choice([4, 8]),
                "storage": rng.choice(["float16", "float32", "bfloat16"])}
    if kind == "box3d":
        storage = rng.choice(["float32", "float16", "bfloat16", "float64"])
        # the reduced types are stored only in the sides the tensor copies take (y 16, z 32); the
        # others take any, and users choose both kinds
        even = storage in ("float16", "bfloat16") or rng.random() < 0.5
        hi = {"float32": 288, "float64": 192}.get(storage, 352)
        n = [_log_int(rng, 32, hi) for _ in range(3)]
        if even:
            n[1], n[2] = max(16, n[1] // 16 * 16), max(32, n[2] // 32 * 32)
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "storage": storage}
    if kind == "duct3d":
        storage = rng.choice(["float32", "float32", "float64", "float16"])
        n = [_log_int(rng, 24, 192) for _ in range(3)]
        if storage == "float16" or rng.random() < 0.4:
            n[1], n[2] = max(16, n[1] // 16 * 16), max(32, n[2] // 32 * 32)
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "storage": storage, "force": rng.random() < 0.4,
                "diagnostics": rng.random() < 0.4}
    if kind == "swimmer3d":
        side = _log_int(rng, 48, 176)
        if rng.random() < 0.6:
            side = max(64, side // 32 * 32)
        return {"kind": kind, "side": side, "substeps": rng.choice([4, 8]), "storage": "float32"}
    sides, room = [], 18_000_000  # cells: no more than the listed mix
    for _ in range(rng.randint(1, 9)):
        side = rng.choice([64, 64, 96, 96, 128, 128, 160, 192])
        if side ** 3 <= room:
            sides.append(side)
            room -= side ** 3
    return {"kind": kind, "sides": ",".join(str(s) for s in sides), "substeps": 8,
            "storage": rng.choice(["float16", "float16", "bfloat16"])}


# ----------------------------------------------------------------------------- states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31))


def _smooth(shape, rng, modes=3):
    """A sum of long Fourier modes of the box, amplitude about 1 (binary64, on the GPU)."""
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    axes = [torch.arange(n, dtype=torch.float64, device="cuda") * (2 * math.pi / n) for n in shape]
    for _ in range(modes):
        term = None
        for d, x in enumerate(axes):
            w = torch.cos(int(rng.integers(0, 4)) * x + float(rng.uniform(0, 2 * math.pi)))
            w = w.reshape([-1 if k == d else 1 for k in range(len(shape))])
            term = w if term is None else term * w
        out += term * float(rng.uniform(0.3, 0.7))
    return out


def _physical(shape, seed, mean=(0.0, 0.0, 0.0), speed=0.03):
    """Moments of a smooth random flow: rho, u, S (2D: 6 planes, 3D: 10), float32 values."""
    rng, g = np.random.default_rng(int(seed)), _gen(seed)
    dim = len(shape)
    pairs = [(0, 0), (1, 1), (0, 1)] if dim == 2 else [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    m = torch.empty((1 + dim + len(pairs),) + tuple(shape), dtype=torch.float32, device="cuda")

    def noise():
        return torch.rand(shape, generator=g, device="cuda") - 0.5

    u = []
    for a in range(dim):
        u.append((mean[a] + speed * _smooth(shape, rng)).float() + 0.05 * speed * noise())
        m[1 + a] = u[a]
    m[0] = (1.0 + 1.5 * speed * speed * _smooth(shape, rng)).float() + 1e-4 * noise()
    for k, (a, b) in enumerate(pairs):
        neq = (0.05 * speed * speed) * (_smooth(shape, rng, 1).float() + 0.2 * noise())
        m[1 + dim + k] = u[a] * u[b] + neq
    return m


def _stored(m, storage):
    """The moments as a buffer of that storage type holds them."""
    if storage not in ("float16", "bfloat16"):
        return m.to(torch.float64 if storage == "float64" else torch.float32)
    dim = 2 if m.shape[0] == 6 else 3
    pairs = [(0, 0), (1, 1), (0, 1)] if dim == 2 else [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    r = torch.empty(m.shape, dtype=torch.float16 if storage == "float16" else torch.bfloat16, device=m.device)
    r[0] = (m[0].double() - 1.0).to(r.dtype)
    r[1:1 + dim] = (m[1:1 + dim] / U_REF).to(r.dtype)
    for k, (a, b) in enumerate(pairs):
        r[1 + dim + k] = ((m[1 + dim + k] - m[1 + a] * m[1 + b]) / S_REF).to(r.dtype)
    return r


def _load(flow, seed, mean=(0.0, 0.0, 0.0), speed=0.03):
    t = _stored(_physical(tuple(flow.cur.shape[1:]), seed, mean, speed), flow.storage)
    flow.moments[0].copy_(t)
    flow.moments[1].copy_(t)


def _ngon(n, aspect=1.0):
    th = np.linspace(0, 2 * np.pi, n, endpoint=False)
    return np.stack([np.cos(th), aspect * np.sin(th)], 1).astype(np.float32)


def _scales(storage):
    return dict(u_scale=U_REF, s_scale=S_REF) if storage in ("float16", "bfloat16") else {}


# ----------------------------------------------------------------------------- prepare
def _prepare_wake2d(c, seed):
    nx, ny = c["nx"], c["ny"]
    s = LBM_Solver(nx, ny, solid_num=1, storage=c["storage"], **_scales(c["storage"]))
    f = s.flows[0]
    f.vis_shear = 0.012
    f.bc_type = [0, 1, 1, 1]
    f.bc_value = np.array([[0.05, 0.0], [0, 0], [0, 0], [0, 0]], np.float32)
    _load(f, seed, mean=(0.04, 0.0), speed=0.01)
    r = max(4.0, 0.09 * ny)
    f.configure_solid(0, _ngon(96), (0.25 * nx, 0.5 * ny), scale=r / nx)
    return {"solver": s}


def _prepare_env2d(c, seed):
    rng = np.random.default_rng(seed)
    W, nx, ny, n, S = c["worlds"], c["nx"], c["ny"], c["bodies"], c["substeps"]
    s = LBM_Solver(nx, ny, solid_num=n, nworld=W, storage=c["storage"])
    r = 0.09 * ny
    centres = np.array([[(0.25 + 0.5 * (k + 0.5) / n) * nx, 0.5 * ny] for k in range(n)])
    for w, f in enumerate(s.flows):
        f.vis_shear = 0.02
        f.bc_type = [0, 1, 1, 1]
        f.bc_value = np.array([[0.03, 0.0], [0, 0], [0, 0], [0, 0]], np.float32)
        _load(f, seed * 1000 + w, mean=(0.03, 0.0), speed=0.01)
    for k in range(n):
        s.create_solid_from_polygon(k, _ngon(32, 0.4), tuple(centres[k]), r / nx)
    s.finalize_mappings(list(range(n)))
    # bodies that sway and turn slowly; positions are given in body radii from each origin
    t = np.arange(1, S + 1)[:, None, None] / S
    ph = rng.uniform(0, 2 * np.pi, (1, W, n))
    pos = np.zeros((S, W, n, 3), np.float32)
    pos[..., 0], pos[..., 1] = 0.02 * np.sin(t + ph), 0.02 * np.cos(t + ph)
    ang = 0.1 * np.sin(0.3 * t + ph)
    quat = np.zeros((S, W, n, 4), np.float32)
    quat[..., 0], quat[..., 3] = np.cos(ang / 2), np.sin(ang / 2)
    f32 = dict(dtype=torch.float32, device="cuda")
    return {"solver": s, "substeps": S, "ids": s.solid_ids_wp, "pos": torch.tensor(pos, **f32),
            "quat": torch.tensor(quat, **f32), "scales": s.scales_wp, "forces": torch.zeros((S, W, n, 3), **f32),
            "torques": torch.zeros((S, W, n, 3), **f32)}


def _prepare_batch2d(c, seed):
    rng = np.random.default_rng(seed)
    size_rng = np.random.default_rng(c["worlds"])  # the sizes are the case's, not the seed's
    specs = []
    for _ in range(c["worlds"]):
        nx = int(round(math.exp(size_rng.uniform(math.log(256), math.log(1024)))))
        ny = int(round(math.exp(size_rng.uniform(math.log(128), math.log(512)))))
        specs.append(SwimmerSpec(nx, ny, CapsuleChain(head=(0.25 * nx, 0.5 * ny + float(rng.uniform(-2, 2))),
                                                      freq=float(rng.uniform(0.002, 0.01)))))
    b = SwimmerBatch2D(specs, storage=c["storage"], substeps=c["substeps"], autotuner=TileAutotuner())
    # the worlds' storage scales are SwimmerBatch2D's own (0.02 and its square)
    for w, f in enumerate(b.flows):
        m = _physical((f.nx, f.ny), seed * 1000 + w, speed=0.01)
        if f.encoded:
            for mom in f.moments:
                mom[0] = (m[0].double() - 1.0).to(mom.dtype)
                mom[1:3] = (m[1:3] / f.u_scale).to(mom.dtype)
                for k, (a, e) in enumerate([(0, 0), (1, 1), (0, 1)]):
                    mom[3 + k] = ((m[3 + k] - m[1 + a] * m[1 + e]) / f.s_scale).to(mom.dtype)
        else:
            for mom in f.moments:
                mom.copy_(m)
    return {"batch": b}


def _prepare_box3d(c, seed):
    s = LBM_Solver3D(c["nx"], c["ny"], c["nz"], periodic=True, storage=c["storage"], with_flag=False, with_force=False,
                     **_scales(c["storage"]))
    s.set_viscosity(1e-3)
    _load(s.flows[0], seed)
    return {"solver": s}


DUCT_IN = (0.04, 0.0, 0.0)


def _duct_force(c, seed):
    if not c["force"]:
        return None
    rng = np.random.default_rng(seed + 7)
    shape = (c["nx"], c["ny"], c["nz"])
    return torch.stack([1e-5 * _smooth(shape, rng, 2).float() for _ in range(3)])


def _prepare_duct3d(c, seed):
    s = LBM_Solver3D(c["nx"], c["ny"], c["nz"], storage=c["storage"], with_force=c["force"], **_scales(c["storage"]))
    f = s.flows[0]
    s.set_viscosity(0.01)
    f.bc_type = [0, 1, 1, 1, 1, 1]
    f.bc_value = np.array([DUCT_IN] + [(0, 0, 0)] * 5, np.float32)
    _load(f, seed, mean=DUCT_IN, speed=0.01)
    if c["force"]:
        f.force.copy_(_duct_force(c, seed))
        f.use_force = True
    s.diagnostics = c["diagnostics"]
    return {"solver": s}


def _prepare_swimmer3d(c, seed):
    d = PlainDomain(Request(0, c["side"], int(seed), substeps=c["substeps"]), c["storage"], 0.01, torch.device("cuda"))
    _load(d.solver.flows[0], seed, speed=0.02)
    return {"domain": d}


def _prepare_served3d(c, seed):
    sides = [int(v) for v in c["sides"].split(",")]
    # the launch settings that ServeEngine applies while it serves
    prev = {k: _lib.get_tuning(k) for k in ("d3q27_chunks", "d3q27_link_blocks")}
    _lib.set_tuning("d3q27_chunks", 1)
    _lib.set_tuning("d3q27_link_blocks", torch.cuda.get_device_properties(0).multi_processor_count // 4)
    try:
        doms = [Domain(Request(i, n, int(seed) * 100 + i, substeps=c["substeps"]), c["storage"], 0.01,
                       torch.device("cuda")) for i, n in enumerate(sides)]
    finally:
        for k, v in prev.items():
            _lib.set_tuning(k, v)
    for i, d in enumerate(doms):
        f = d.solver.flows[0]
        m = _physical((f.nx, f.ny, f.nz), int(seed) * 100 + i, speed=0.01)
        pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        for mom in f.moments:  # the domain's own storage scales
            mom[0] = (m[0].double() - 1.0).to(mom.dtype)
            mom[1:4] = (m[1:4] / f.u_scale).to(mom.dtype)
            for k, (a, b) in enumerate(pairs):
                mom[4 + k] = ((m[4 + k] - m[1 + a] * m[1 + b]) / f.s_scale).to(mom.dtype)
        d.stage_poses(0)
    torch.cuda.synchronize()
    return {"domains": doms}


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, int(seed))
    state["kind"] = case["kind"]
    return state


# ----------------------------------------------------------------------------- run
# The reduced storages round stochastically, and a body's load is what its cells' stored moments
# make it: those cases return the stored moments, the binary32 cases the loads too.
def _run_wake2d(st):
    s = st["solver"]
    s.step()
    f = s.flows[0]
    return {"moments": f.cur} if f.encoded else {"moments": f.cur, "loads": s.solid_loads_all}


def _run_env2d(st):
    s = st["solver"]
    for k in range(st["substeps"]):
        coupling.convert_and_update_solid_batch_2d(s, st["ids"], st["pos"][k], st["quat"][k])
        s.step()
        coupling.extract_forces_torques_batch(s, st["ids"], st["scales"], st["forces"][k], st["torques"][k])
    return {"moments": [f.cur for f in s.flows], "forces": st["forces"], "torques": st["torques"]}


def _run_batch2d(st):
    b = st["batch"]
    loads = b.control_step()
    out = {"moments": [f.cur for f in b.flows]}
    if not b.flows[0].encoded:
        out["loads"] = loads
    return out


def _run_box3d(st):
    st["solver"].step()
    return {"moments": st["solver"].flows[0].cur}


def _run_duct3d(st):
    s = st["solver"]
    s.step()
    out = {"moments": s.flows[0].cur}
    if s.diagnostics:
        out["mass"], out["health"] = s.mass, s.health
    return out


def _run_swimmer3d(st):
    d = st["domain"]
    d.control_step()
    return {"moments": d.solver.flows[0].cur, "loads": d.loads.pop()}


def _run_served3d(st):
    doms = st["domains"]
    for d in doms:
        d.launch()
    for d in doms:
        d.stage_poses(d.done + 1)
    for d in doms:
        d.event.synchronize()
    for d in doms:
        d.finish(0.0)
        d.loads.pop()
    return {"moments": [d.solver.flows[0].moments[0] for d in doms]}


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ----------------------------------------------------------------------------- work
def work(case):
    """Moments read and written once per step (and force where it is used), and the operations of
    the source-side rebuild and the moment-space collision: about 420 a cell in 3D, 170 in 2D."""
    k, b = case["kind"], SIZE[case["storage"]]
    if k == "wake2d":
        n, steps = case["nx"] * case["ny"], 1
    elif k == "env2d":
        n, steps = case["worlds"] * case["nx"] * case["ny"], case["substeps"]
    elif k == "batch2d":
        r, n = np.random.default_rng(case["worlds"]), 0
        for _ in range(case["worlds"]):
            n += (int(round(math.exp(r.uniform(math.log(256), math.log(1024)))))
                  * int(round(math.exp(r.uniform(math.log(128), math.log(512))))))
        steps = case["substeps"]
    elif k == "swimmer3d":
        n, steps = case["side"] ** 3, case["substeps"]
    elif k == "served3d":
        n, steps = sum(int(v) ** 3 for v in case["sides"].split(",")), case["substeps"]
    else:
        n, steps = case["nx"] * case["ny"] * case["nz"], 1
    if k.endswith("2d"):
        return {"bytes": 12.0 * b * n * steps, "flops": 170.0 * n * steps}
    extra = 12 if case.get("force") else 0
    return {"bytes": (20.0 * b + extra) * n * steps, "flops": 420.0 * n * steps}


# ----------------------------------------------------------------------------- exact
def _decode64(t, storage, us=U_REF, ss=S_REF):
    d = t.double()
    if storage not in ("float16", "bfloat16"):
        return d
    out = torch.empty_like(d)
    out[0] = d[0] + 1.0
    out[1:4] = d[1:4] * us
    for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        out[4 + k] = d[4 + k] * ss + out[1 + a] * out[1 + b]
    return out


def _encode64(m, storage, us=U_REF, ss=S_REF):
    if storage not in ("float16", "bfloat16"):
        return m
    out = torch.empty_like(m)
    out[0] = m[0] - 1.0
    out[1:4] = m[1:4] / us
    for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        out[4 + k] = (m[4 + k] - m[1 + a] * m[1 + b]) / ss
    return out


def _step64(m, vis, periodic, force=None):
    """One D3Q27 step in binary64 from moments m (10, nx, ny, nz): every population rebuilt from
    its upwind cell by the second-order expansion, clamped at zero, then the regularised
    collision. Walled domains: populations from outside are zero, and the border cells' values
    are not meaningful."""
    rho, ux, uy, uz, sxx, syy, szz, sxy, sxz, syz = m
    usq = ux * ux + uy * uy + uz * uz
    tr = (sxx + syy + szz) / 3.0
    acc = {k: torch.zeros_like(rho) for k in ("r", "x", "y", "z", "xx", "yy", "zz", "xy", "xz", "yz")}
    for cx in (-1, 0, 1):
        for cy in (-1, 0, 1):
            for cz in (-1, 0, 1):
                n = (cx != 0) + (cy != 0) + (cz != 0)
                w = (8 / 27, 2 / 27, 1 / 54, 1 / 216)[n]
                cu = cx * ux + cy * uy + cz * uz
                q = (cx * cx * sxx + cy * cy * syy + cz * cz * szz
                     + 2.0 * (cx * cy * sxy + cx * cz * sxz + cy * cz * syz)) - tr
                f = (w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq + 1.5 * q)).clamp_(min=0.0)
                f = torch.roll(f, (cx, cy, cz), (0, 1, 2))
                if not periodic:
                    for d, c in enumerate((cx, cy, cz)):
                        if c:
                            f.select(d, 0 if c > 0 else -1).zero_()
                acc["r"] += f
                for name, v in (("x", cx), ("y", cy), ("z", cz), ("xx", cx * cx), ("yy", cy * cy), ("zz", cz * cz),
                                ("xy", cx * cy), ("xz", cx * cz), ("yz", cy * cz)):
                    if v:
                        acc[name].add_(f, alpha=v)
    F = force.double() if force is not None else [0.0, 0.0, 0.0]
    om = 1.0 / (3.0 * vis + 0.5)
    out = torch.empty_like(m)
    r = acc["r"]
    u = [(acc[a] + 0.5 * F[i]) / r for i, a in enumerate("xyz")]
    R = [r * v * v for v in u]
    p = [acc["xx"] - r / 3.0, acc["yy"] - r / 3.0, acc["zz"] - r / 3.0]
    trp, trr = (p[0] + p[1] + p[2]) / 3.0, (R[0] + R[1] + R[2]) / 3.0
    out[0] = r
    for a in range(3):
        out[1 + a] = u[a] + 0.5 * F[a] / r
        out[4 + a] = ((1.0 - om) * (p[a] - trp + trr) + om * R[a] + F[a] * u[a]) / r
    for k, (a, b, name) in enumerate(((0, 1, "xy"), (0, 2, "xz"), (1, 2, "yz"))):
        out[7 + k] = ((1.0 - om) * acc[name] + om * r * u[a] * u[b] + 0.5 * (F[a] * u[b] + F[b] * u[a])) / r
    return out


def _boundary64(old, new, bc_type, bc_value):
    """The outer boundaries of a walled box: ``old`` the buffer before the pass (its border cells
    hold earlier values), ``new`` the stepped interior. A face cell takes its inward neighbour's
    density and velocity (or the face's own velocity) and its stress moved to that velocity;
    edges and corners apply their faces in axis order, reading a neighbour on a low face as it
    was before the pass and one on a high face as the pass left it."""
    n = new.shape[1:]
    out = new.clone()
    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    faces = {(0, 0): 0, (0, 1): 1, (1, 1): 2, (1, 0): 3, (2, 1): 4, (2, 0): 5}

    def core(face, t, nb):
        r = t.clone()
        r[0] = nb[0]
        for a in range(3):
            r[1 + a] = float(bc_value[face][a]) if bc_type[face] == 0 else nb[1 + a]
        for k, (a, b) in enumerate(pairs):
            r[4 + k] = r[1 + a] * r[1 + b] - nb[1 + a] * nb[1 + b] + nb[4 + k]
        return r

    def at(buf, where):
        return buf[(slice(None),) + where]

    def place(sides, shift=None):
        w = []
        for a in range(3):
            if a in sides:
                i = (n[a] - 1 if sides[a] else 0) if a != shift else (n[a] - 2 if sides[a] else 1)
                w.append(slice(i, i + 1))
            else:
                w.append(slice(1, n[a] - 1))
        return tuple(w)

    for count in (1, 2, 3):
        done = out.clone()
        for mask in range(27):
            sides = {a: (mask // 3 ** a) % 3 - 1 for a in range(3)}
            sides = {a: v for a, v in sides.items() if v >= 0}
            if len(sides) != count:
                continue
            t = at(old, place(sides)).clone()
            for a in sorted(sides):
                src = place(sides, a)
                nb = at(old if (count > 1 and sides[a] == 0) else out, src)
                t = core(faces[(a, sides[a])], t, nb)
            done[(slice(None),) + place(sides)] = t
        out = done
    return out


def exact(case, seed):
    k = case["kind"]
    if k not in ("box3d", "duct3d"):
        return None  # moving polygons and meshes, or several steps: no short independent form
    shape = (case["nx"], case["ny"], case["nz"])
    sto = case["storage"]
    if k == "box3d":
        raw = _stored(_physical(shape, int(seed)), sto)
        m = _decode64(raw, sto)
        return {"moments": _encode64(_step64(m, 1e-3, True), sto)}
    raw = _stored(_physical(shape, int(seed), DUCT_IN, 0.01), sto)
    m = _decode64(raw, sto)
    new = _step64(m, 0.01, False, _duct_force(case, int(seed)))
    inside = (slice(None),) + (slice(1, -1),) * 3
    post = m.clone()
    post[inside] = new[inside]
    mass = post[(0,) + (slice(1, -1),) * 3].sum()
    value = np.array([DUCT_IN] + [(0, 0, 0)] * 5, np.float32)
    post = _boundary64(m, post, [0, 1, 1, 1, 1, 1], value)
    out = {"moments": _encode64(post, sto)}
    if case["diagnostics"]:
        out["mass"] = mass.reshape(1)
        out["health"] = None
    return out
