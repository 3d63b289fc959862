"""Every cell that a walled stream-collide stores, border cells included, and a world without a flag field.

The reference reads a cell outside the domain as zero populations. Here the domain lies in a periodic
one of the oracle, one layer of cells of zero density around it, which send nothing: the oracle's new
values of all cells of the domain are those that the walled step stores where its flags say fluid.

Tolerance as in test_gpu_d3q27_sweep.py: 320 eps (2^-24 or 2^-53).
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from test_gpu_d3q27_sweep import _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,shape", [("float32", (5, 16, 32)), ("float32", (4, 17, 36)), ("float32", (5, 13, 31)),
                                           ("float64", (5, 8, 32)), ("float64", (4, 9, 34)), ("float64", (5, 11, 33))])
@pytest.mark.parametrize("regime", ["calm", "clamped"])
@pytest.mark.parametrize("flags", ["borders fluid", "some", None])
@pytest.mark.parametrize("diagnostics", [False, True])
def test_all_stored_cells(storage, shape, regime, flags, diagnostics):
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    s = LBM_Solver3D(*shape, storage=storage, use_graph=False, with_flag=flags is not None)
    f = s.flows[0]
    t = torch.tensor(_state(shape, regime, 21)).to(torch.float32 if storage == "float32" else torch.float64)
    m = t.double().numpy()
    f.moments[0].copy_(t)
    f.moments[1].fill_(7)
    fluid = np.zeros(shape, bool)
    fluid[1:-1, 1:-1, 1:-1] = True
    if flags == "borders fluid":
        fluid[:] = True
    elif flags == "some":
        flip = np.random.default_rng(2).random(shape) < 0.3
        fluid[flip] = ~fluid[flip]
    if flags is not None:
        f.flag.copy_(torch.tensor(np.where(fluid, 0, 2).astype(np.int32)))
    rng = np.random.default_rng(12)
    force = (1e-3 * rng.uniform(-1, 1, (3, *shape))).astype(np.float32)
    f.force.copy_(torch.tensor(force))
    f.use_force = True
    mass, health = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(1 << 14, dtype=torch.uint8, device="cuda")
    d = _lib.hl_diag(scratch.data_ptr(), 1 << 14, mass.data_ptr(), health.data_ptr()) if diagnostics else None
    _lib.check(_lib.lib().hl_d3q27_stream_collide(f.world_struct(0), 0.02, d, _lib.stream_ptr()), "step")
    got = f.moments[1].double().cpu().numpy()

    pad = ((0, 0), (1, 1), (1, 1), (1, 1))
    big = np.pad(m, pad)
    with np.errstate(all="ignore"):
        new, _ = orc.step_3d(big, np.zeros_like(big), vis_shear=0.02, periodic=True, dtype=np.float64,
                             force=np.pad(force.astype(np.float64), pad))
    want = new[:, 1:-1, 1:-1, 1:-1]
    eps = 2.0 ** (-24 if storage == "float32" else -53)
    assert np.isfinite(want[:, fluid]).all()
    assert np.abs(got[:, fluid] - want[:, fluid]).max() <= 320 * eps
    assert (got[:, ~fluid] == 7).all()
    if diagnostics:
        assert int(health) == 0
        assert abs(float(mass) - want[0][fluid].sum()) <= 320 * eps * fluid.sum()


@pytest.mark.parametrize("storage,shape", [("float32", (700, 16, 32)), ("float32", (300, 3, 4)), ("float64", (515, 9, 33))])
def test_a_long_column_in_many_chunks(storage, shape):
    """A domain of one or two tiles is cut into as many chunks along x as there are blocks: the bits of
    one chunk."""
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    out = []
    for chunks in (0, 1):
        s = LBM_Solver3D(*shape, storage=storage, use_graph=False, with_flag=False)
        f = s.flows[0]
        f.moments[0].copy_(torch.tensor(_state(shape, "clamped", 8)))
        f.moments[1].fill_(7)
        _lib.set_tuning("d3q27_chunks", chunks)
        try:
            _lib.check(_lib.lib().hl_d3q27_stream_collide(f.world_struct(0), 0.02, None, _lib.stream_ptr()), "step")
        finally:
            _lib.set_tuning("d3q27_chunks", 0)
        out.append(f.moments[1].clone())
    assert torch.equal(*out)
    assert (out[0][0] != 7).sum() == np.prod([n - 2 for n in shape])
