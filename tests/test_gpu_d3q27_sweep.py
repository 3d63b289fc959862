"""The sweep kernel (d3q27_sweep.cuh) at the edges of its tiles and on both of its paths.

One step from random states against the binary64 oracle: sides around the tile (16 rows of
binary32, 8 of binary64, 32 along z, 2 and 3 planes), periodic and walled, with flag fields that
make border cells fluid and inner cells walls, with force. The "calm" states stay inside the bound
under which no population can be negative; the "clamped" ones leave it in part of the box, where
many populations are negative and the clamp at zero acts.

Tolerance, before any run: a stored moment is at most about 64 rounded operations on terms whose
magnitudes sum to 2, divided by rho >= 0.4, so its error is below 64 * 2 * eps / 0.4 = 320 eps
(eps = 2^-24 or 2^-53); a 16-bit store adds up to one spacing.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
U_SCALE, S_SCALE = 0.5, 0.25


def _state(shape, regime, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    m = np.zeros((10, *shape))
    amp = 0.04 * np.ones(shape)
    if regime == "clamped":  # strong in a slab of x and in a patch at one z end
        amp[nx // 2:] = 0.5
        amp[:, : max(1, ny // 3), -1:] = 0.5
    m[0] = 1.0 + 0.3 * amp * rng.uniform(-1, 1, shape)
    for k in range(1, 4):
        m[k] = amp * rng.uniform(-1, 1, shape)
    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    for k, (a, b) in enumerate(pairs):
        m[4 + k] = m[1 + a] * m[1 + b] + 0.1 * amp * rng.uniform(-1, 1, shape)
    return m


def _encode(m, storage):
    if storage == "float16":
        r = m.copy()
        r[0] -= 1.0
        r[1:4] /= U_SCALE
        for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            r[4 + k] = (m[4 + k] - m[1 + a] * m[1 + b]) / S_SCALE
        return torch.tensor(r).to(torch.float16)
    return torch.tensor(m).to(torch.float32 if storage == "float32" else torch.float64)


def _decode(t, storage):
    r = t.double().cpu().numpy()
    if storage != "float16":
        return r
    m = r.copy()
    m[0] = r[0] + 1.0
    m[1:4] = r[1:4] * U_SCALE
    for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        m[4 + k] = r[4 + k] * S_SCALE + m[1 + a] * m[1 + b]
    return m


SHAPES = {
    "float32": [(5, 16, 32), (4, 17, 36), (7, 33, 64), (3, 15, 28), (6, 48, 32), (2, 16, 32)],
    "float64": [(5, 8, 32), (4, 9, 34), (3, 7, 30), (6, 16, 64), (5, 17, 33), (7, 11, 31)],
    "float16": [(5, 16, 32), (4, 32, 64)],
}
CASES = [(s, sh) for s in SHAPES for sh in SHAPES[s]]


@pytest.mark.parametrize("storage,shape", CASES)
@pytest.mark.parametrize("regime", ["calm", "clamped"])
@pytest.mark.parametrize("periodic", [True, False])
def test_one_step_matches_the_binary64_oracle(storage, shape, regime, periodic):
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    kw = dict(u_scale=U_SCALE, s_scale=S_SCALE) if storage == "float16" else {}
    s = LBM_Solver3D(*shape, periodic=periodic, storage=storage, use_graph=False, **kw)
    f = s.flows[0]
    raw = _encode(_state(shape, regime, 3 + len(regime)), storage)
    cur = _decode(raw, storage)
    f.moments[0].copy_(raw)
    f.moments[1].fill_(7)
    rng = np.random.default_rng(11)
    flag = None
    if not periodic:  # borders mostly walls, some fluid; some inner walls
        flag = orc.border_flags_3d(*shape)
        flip = rng.random(shape) < 0.1
        flag[flip] = np.where(flag[flip] == 0, 2, 0)
        f.flag.copy_(torch.tensor(flag))
    force = (1e-3 * rng.uniform(-1, 1, (3, *shape))).astype(np.float32)
    f.force.copy_(torch.tensor(force))
    f.use_force = True
    vis = 0.02
    L = _lib.lib()
    _lib.check(L.hl_d3q27_stream_collide(f.world_struct(0), vis, None, _lib.stream_ptr()), "step")
    got_raw = f.moments[1].double().cpu().numpy()

    # the oracle steps and applies the outer boundaries: only the cells that the step itself stores
    # (and no boundary pass touches) are compared
    new, _ = orc.step_3d(cur, np.full_like(cur, 7.0), vis_shear=vis, flag=flag, force=force.astype(np.float64),
                         periodic=periodic, dtype=np.float64)
    fluid = np.ones(shape, bool) if periodic else flag == 0
    inner = np.zeros(shape, bool)
    inner[1:-1, 1:-1, 1:-1] = True
    check = fluid if periodic else fluid & inner
    eps = 2.0 ** (-53 if storage == "float64" else -24)
    ref_raw = new
    if storage == "float16":
        ref_raw = new.copy()
        ref_raw[0] -= 1.0
        ref_raw[1:4] /= U_SCALE
        for k, (a, b) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            ref_raw[4 + k] = (new[4 + k] - new[1 + a] * new[1 + b]) / S_SCALE
    tol = 320 * eps * np.ones_like(ref_raw)
    if storage == "float16":
        tol = tol / S_SCALE + np.spacing(np.abs(ref_raw).astype(np.float16)).astype(np.float64) * 1.01
    err = np.abs(got_raw - ref_raw)
    assert (err[:, check] <= tol[:, check]).all(), float((err / tol)[:, check].max())
    # cells that are not fluid keep their value
    assert (got_raw[:, ~fluid] == 7).all()


def test_non_finite_cells_act_as_in_the_other_kernel():
    """A NaN or infinite cell's populations are clamped to zero (fmax drops a NaN), in both kernels:
    the same cells stay finite, with the same values."""
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    shape = (6, 32, 64)
    out = []
    for kernel in (1, 2):
        s = LBM_Solver3D(*shape, periodic=True, use_graph=False)
        f = s.flows[0]
        t = _encode(_state(shape, "calm", 5), "float32")
        t[0, 2, 15, 31] = float("nan")
        t[2, 4, 0, 0] = float("inf")
        t[7, 1, 20, 40] = float("nan")
        f.moments[0].copy_(t)
        _lib.set_tuning("d3q27_kernel", kernel)
        try:
            _lib.check(_lib.lib().hl_d3q27_stream_collide(f.world_struct(0), 0.02, None, _lib.stream_ptr()), "step")
        finally:
            _lib.set_tuning("d3q27_kernel", 0)
        out.append(f.moments[1].double().cpu().numpy())
    ok = np.isfinite(out[0])
    assert (np.isfinite(out[1]) == ok).all()
    assert np.abs(out[0][ok] - out[1][ok]).max() <= 2 * 320 * 2.0 ** -24
