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
