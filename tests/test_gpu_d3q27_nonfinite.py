"""Non-finite cells in the binary64 sweep kernel (d3q27_sweep.cuh).

A cell with a NaN in u or in a diagonal stress sends populations that are all NaN, and the clamp at
zero takes each as f = 0: the step is that of a cell of zero density. The NaNs here have the largest
bit patterns, the one that a binary32 NaN of GPU arithmetic becomes in binary64 among them.

Tolerance as in test_gpu_d3q27_sweep.py: 320 eps, eps = 2^-53.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from test_gpu_d3q27_sweep import _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7FFFFFFFE0000000, 0x7FFFFFFFFFFFFFFF, 0x7FF8000000000000, -1])
@pytest.mark.parametrize("shape", [(5, 16, 64), (5, 9, 33)])  # rows by tensor copies, by 8-byte copies
@pytest.mark.parametrize("regime", ["calm", "clamped"])
def test_binary64_cells_with_nan_send_nothing(bits, shape, regime):
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    cells = [(2, 2, 7, 30), (5, 4, 0, 0), (4, 0, 8, 31)]  # moment (u_y, S_yy, S_xx), x, y, z
    m = _state(shape, regime, 9)
    s = LBM_Solver3D(*shape, periodic=True, storage="float64", use_graph=False)
    f = s.flows[0]
    t = torch.tensor(m)
    for k, x, y, z in cells:
        t.view(torch.int64)[k, x, y, z] = bits
        m[:, x, y, z] = 0.0
    f.moments[0].copy_(t)
    assert (f.moments[0].view(torch.int64).cpu() == t.view(torch.int64)).all()
    _lib.check(_lib.lib().hl_d3q27_stream_collide(f.world_struct(0), 0.02, None, _lib.stream_ptr()), "step")
    want, _ = orc.step_3d(m, np.zeros_like(m), vis_shear=0.02, periodic=True, dtype=np.float64)
    got = f.moments[1].cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= 320 * 2.0 ** -53


@pytest.mark.parametrize("storage", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(8, 16, 64), (8, 17, 36), (8, 11, 33)])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("state", ["nan", "empty"])
def test_cells_that_nothing_reaches_are_counted(storage, shape, periodic, state):
    """A flow that has blown up (NaN everywhere) or a cavity without fluid sends no population: the
    density of the cells inside is zero, and each counts as unhealthy."""
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    s = LBM_Solver3D(*shape, periodic=periodic, storage=storage, use_graph=False)
    f = s.flows[0]
    s.set_viscosity(0.01)
    t = torch.tensor(_state(shape, "calm", 4))
    inside = (slice(2, 6), slice(3, 9), slice(4, 30))  # its inner 2 x 4 x 24 cells hear from no other
    if state == "nan":
        t[1:] = float("nan")
    else:
        t[(slice(None),) + inside] = 0.0
    for m in f.moments:
        m.copy_(t)
    s.diagnostics = True
    s.step()
    nx, ny, nz = shape
    cells = nx * ny * nz if periodic else (nx - 2) * (ny - 2) * (nz - 2)
    want = cells if state == "nan" else 2 * 4 * 24
    assert int(s.health[0]) == want
    rho = f.cur[0, 3:5, 4:8, 5:29]
    assert (rho == 0).all(), rho.flatten()[:4]
