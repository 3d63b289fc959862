"""The D2Q9 boundary and stream launches at small and uneven sizes, against the binary64 oracle.

Two steps from random states: sides of three cells (every border cell next to a corner, some next to
two), sides around the blocks of the boundary pass and the strips of the stream phase, all
boundary types.

Tolerance, before any run: a stored moment is at most about 40 rounded operations on terms whose
magnitudes sum to 2, divided by rho >= 0.8, a step: below 2 * 40 * 2 / 0.8 eps = 200 eps (2^-24).
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _state(nx, ny, seed):
    rng = np.random.default_rng(seed)
    m = np.zeros((6, nx, ny))
    m[0] = 1.0 + 0.02 * rng.uniform(-1, 1, (nx, ny))
    m[1:3] = 0.05 * rng.uniform(-1, 1, (2, nx, ny))
    for k, (a, b) in enumerate([(0, 0), (1, 1), (0, 1)]):
        m[3 + k] = m[1 + a] * m[1 + b] + 1e-3 * rng.uniform(-1, 1, (nx, ny))
    return m.astype(np.float32)


@pytest.mark.parametrize("nx,ny", [(3, 3), (3, 40), (41, 3), (4, 5), (31, 33), (8, 61), (130, 47), (97, 150), (9, 600)])
@pytest.mark.parametrize("bc", [(0, 1, 1, 1), (1, 0, 0, 1), (0, 0, 0, 0), (1, 1, 1, 1)])
def test_two_steps_match_the_binary64_oracle(nx, ny, bc):
    from openhomelbm_b200.lbm import LBM_Solver

    s = LBM_Solver(nx, ny, solid_num=1, use_graph=False)
    f = s.flows[0]
    f.vis_shear = 0.05
    f.bc_type = list(bc)
    f.bc_value = np.array([[0.03, 0.01], [-0.02, 0.0], [0.01, 0.02], [0.0, -0.01]], np.float32)
    m, p = _state(nx, ny, 1), _state(nx, ny, 2)
    f.moments[0].copy_(torch.tensor(m))
    f.moments[1].copy_(torch.tensor(p))
    m, p = m.astype(np.float64), p.astype(np.float64)
    for _ in range(2):
        s.step()
        new, _ = orc.step_2d(m, p, vis_shear=0.05, bc_type=bc, bc_value=f.bc_value, flag=orc.border_flags_2d(nx, ny),
                             dtype=np.float64)
        m, p = new, m
    assert np.abs(f.cur.double().cpu().numpy() - m).max() <= 200 * 2.0 ** -24


@pytest.mark.parametrize("n_solids,n_seg,radius", [(1, 3, 5.0), (2, 40, 6.0), (1, 400, 4.0), (5, 230, 6.0)])
def test_cut_links_of_few_and_many_segments(n_solids, n_seg, radius):
    """Outlines with few, many (more candidate segments per cell than a block keeps) and very many
    segments (more than a block stages), moving, two steps against the binary32 oracle, which takes
    the same cut-link decisions. Tolerance: both sides round, 2 x 200 eps a step, and the loads are
    sums of at most 600 links of magnitude below 1: 600 x 200 eps."""
    from openhomelbm_b200.lbm import LBM_Solver

    nx, ny = 90, 64
    s = LBM_Solver(nx, ny, solid_num=n_solids, use_graph=False)
    f = s.flows[0]
    f.vis_shear = 0.05
    f.bc_type = [0, 1, 1, 1]
    f.bc_value = np.array([[0.03, 0.0], [0, 0], [0, 0], [0, 0]], np.float32)
    m, p = _state(nx, ny, 3), _state(nx, ny, 4)
    f.moments[0].copy_(torch.tensor(m))
    f.moments[1].copy_(torch.tensor(p))
    th = np.linspace(0, 2 * np.pi, n_seg, endpoint=False) + 0.1
    poly = np.stack([np.cos(th), 0.8 * np.sin(th)], 1).astype(np.float32)
    pos = np.array([[14.3 + 15.1 * k, 30.7 + 1.3 * k] for k in range(n_solids)], np.float32)
    for k in range(n_solids):
        f.configure_solid(k, poly, tuple(pos[k]), scale=radius / nx)
    sol = orc.Solids2D(line=np.stack([poly] * n_solids), line_num=np.full(n_solids, n_seg), position=pos.copy(),
                       angle=np.zeros(n_solids), scale=np.full(n_solids, np.float32(radius / nx)),
                       mass_center=np.zeros((n_solids, 2)),
                       max_radius=f.solid_max_radius.cpu().numpy()).cast(np.float32)
    eps = 2.0 ** -24
    for step in range(2):
        for k in range(n_solids):
            f.solid_position[k] += torch.tensor([0.02, -0.01], device=f.device)
            sol.position[k] += np.array([0.02, -0.01], np.float32)
        s.step()
        new, loads = orc.step_2d(m, p, vis_shear=np.float32(0.05), bc_type=f.bc_type, bc_value=f.bc_value,
                                 flag=orc.border_flags_2d(nx, ny), solids=sol)
        m, p = new, m
        assert np.abs(f.cur.cpu().numpy() - m).max() <= (step + 1) * 400 * eps
        got = np.stack([f.solid_forcex.cpu().numpy(), f.solid_forcey.cpu().numpy()], 1)
        assert np.abs(got).max() > 0
        assert np.abs(got - loads[:, :2]).max() <= 600 * 200 * eps


def test_parameters_changed_in_place_reach_the_next_step():
    """Viscosity, a boundary type or value, the body-force switch and an outline changed between
    steps, in place or by assignment: the same bits as when the parameters are packed on every step."""
    from openhomelbm_b200.lbm import LBM_Solver

    def changes(s):
        f = s.flows[1]
        yield lambda: setattr(f, "vis_shear", 0.05)
        yield lambda: f.bc_value.__setitem__((0, 0), 0.05)
        yield lambda: f.bc_type.__setitem__(3, 0)
        yield lambda: setattr(f, "bc_type", (0, 0, 1, 1))
        yield lambda: setattr(f, "bc_value", [[0.02, 0.01], [0, 0], [0, 0], [0, 0]])
        yield lambda: (f.force.fill_(1e-4), setattr(f, "use_force", True))
        yield lambda: f.configure_solid(0, [(0.3, 0.0), (0.0, 0.3), (-0.3, 0.0), (0.0, -0.3)], (20.0, 15.0), scale=0.2)
        yield lambda: setattr(f, "solid_line", f.solid_line.clone().mul_(0.5))

    out = []
    for always in (False, True):
        s = LBM_Solver(48, 32, solid_num=1, nworld=2)
        s.create_solid_from_polygon(0, [(0.2, 0.0), (0.0, 0.2), (-0.2, 0.0), (0.0, -0.2)], (24.0, 16.0), 0.2)
        s.flows[1].bc_type = [0, 1, 1, 1]
        seen = []
        for change in changes(s):
            change()
            for _ in range(2):
                if always:
                    s._desc_key = None
                s.step()
            seen.append([f.cur.clone() for f in s.flows])
        out.append(seen)
    torch.cuda.synchronize()
    for k, (a, b) in enumerate(zip(*out)):
        for x, y in zip(a, b):
            assert torch.equal(x, y), k
        if k:
            assert not torch.equal(a[1], out[0][k - 1][1]), k


@pytest.mark.parametrize("storage", ["float32", "float16", "float64"])
@pytest.mark.parametrize("nworld,nx,ny", [(1, 1501, 179), (1, 1499, 401), (1, 2003, 631), (1, 2111, 1097), (90, 61, 47),
                                          (600, 33, 31), (1, 9001, 7)])
def test_stream_without_a_work_list_equals_the_tiles(nworld, nx, ny, storage):
    """The stream phase over a grid (a thread per cell, or strips of 4 to 32 planes by size) stores the
    bits of the 8 x 32 tiles: walled worlds with solid cells inside and a body force, and periodic ones."""
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.batching import TileConfig, WorldBatch2D
    from openhomelbm_b200.lbm import LBM_Solver

    torch.manual_seed(5)
    for periodic in (False, True):
        s = LBM_Solver(nx, ny, solid_num=1, nworld=nworld, storage=storage, periodic=periodic, u_scale=0.05, s_scale=2.5e-3)
        for f in s.flows[:3] + s.flows[-1:]:
            m = torch.rand((6, nx, ny), device="cuda", dtype=torch.float64) - 0.5
            m[0] *= 0.1
            if f.encoded:
                f.moments[0].copy_(m)
            else:
                m[1:3] *= 0.1
                m[3:] *= 0.02
                f.moments[0].copy_(m)
                f.moments[0][0] += 1.0
            if not periodic:
                f.flag[nx // 2 : nx // 2 + 3, ny // 3 : ny // 3 + 2] = 1
                f.force.uniform_(-1e-4, 1e-4)
                f.use_force = True
        s._upload_descriptors()
        st = _lib.stream_ptr()
        _lib.check(_lib.lib().hl_d2q9_step_batch(_lib.ptr(s._desc_dev), nworld, 0, s.flows[0].storage_code, nx, ny, 0, 2, st))
        got = [f.moments[1].clone() for f in s.flows]
        for f in s.flows:
            f.moments[1].zero_()
            f.moments[1][0] = 0.0 if f.encoded else 1.0
        b = WorldBatch2D(s.flows)
        b.launch(0, st, TileConfig(8, 32, 1184), phases=2, any_solid=False)
        torch.cuda.synchronize()
        for k, f in enumerate(s.flows):
            inner = got[k] if periodic else got[k][:, 1:-1, 1:-1]
            want = f.moments[1] if periodic else f.moments[1][:, 1:-1, 1:-1]
            assert torch.equal(inner, want), (periodic, k)
        assert got[0].double().std() > 0


@pytest.mark.parametrize("nworld", [11, 16, 49])
def test_cut_links_of_many_worlds_equal_one(nworld):
    """The cut links of a world among many (fewer, smaller blocks each) store the bits that it gets alone;
    its loads are the same binary64 sums in another order, within 64 links * 2^-52 of their magnitude,
    rounded to binary32 (2^-23)."""
    from openhomelbm_b200.lbm import LBM_Solver

    def run(n):
        s = LBM_Solver(150, 97, solid_num=2, nworld=n)
        m = torch.tensor(_state(150, 97, 3), device="cuda")
        for f in s.flows:
            for buf in f.moments:
                buf.copy_(m)
        ang = np.linspace(0, 2 * np.pi, 40, endpoint=False)
        ring = [(0.5 * np.cos(a), 0.5 * np.sin(a)) for a in ang]
        s.create_solid_from_polygon(0, ring, (50.3, 48.6), 0.3)
        s.create_solid_from_polygon(1, ring, (100.2, 47.1), 0.2)
        for _ in range(3):
            s.step()
        torch.cuda.synchronize()
        return s

    one, many = run(1), run(nworld)
    loads = one.solid_loads_all[0].double()
    assert loads.abs().max() > 0
    for w, f in enumerate(many.flows):
        assert torch.equal(f.cur, one.flows[0].cur), w
        assert (many.solid_loads_all[w].double() - loads).abs().max() <= loads.abs().max() * 2.0 ** -22, w
