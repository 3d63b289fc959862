"""Mass over many binary32 steps of the sweep kernel (d3q27_sweep.cuh).

A periodic box keeps its mass but for roundings, which fall to either side: n steps of N cells whose
densities are each stored within 2^-25 of 1 drift by about 2^-25 sqrt(n / N), 9e-10 for 200 steps of 48 x 64
x 64 cells, and ten times that is allowed. A term that is systematically off, by a rounded constant times
|u|^2 for one, adds up instead: 200 x 6 |u|^2 x 1e-8 = 2.5e-7 for the flow here.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(48, 64, 64), (49, 80, 32)])
def test_mass_of_a_mean_flow(shape):
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    rng = np.random.default_rng(1)
    axes = np.meshgrid(*[2 * np.pi * np.arange(n) / n for n in shape], indexing="ij")

    def smooth():
        out = 0.0
        for _ in range(6):
            term = rng.uniform(0.2, 0.6)
            for x in axes:
                term = term * np.cos(int(rng.integers(0, 5)) * x + rng.uniform(0, 2 * np.pi))
            out = out + term
        return out

    m = np.zeros((10, *shape))
    m[0] = 1.0 + 4e-4 * smooth()
    for a, mean in enumerate((0.1, 0.06, -0.08)):
        m[1 + a] = mean + 0.02 * smooth()
    for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        m[4 + k] = m[1 + a] * m[1 + b]
    s = LBM_Solver3D(*shape, periodic=True, use_graph=False, with_flag=False, with_force=False)
    f = s.flows[0]
    s.set_viscosity(2e-3)
    f.moments[0].copy_(torch.tensor(m))
    before = float(f.cur[0].double().mean())
    for _ in range(200):
        s.step()
    assert abs(float(f.cur[0].double().mean()) / before - 1) <= 9e-9
