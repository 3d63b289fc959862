"""The stream phase of hl_d2q9_step_batch over worlds of different sizes.

The launch knows the largest sides only: it may not take strips that would be long and few in the worlds
that there are, unless the caller says that all have the same size. Whichever form runs, the bits are
those of the 8 x 32 tiles of a work list.
"""
import re

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

rng = np.random.default_rng(2)
MIXED = [(int(np.exp(rng.uniform(np.log(64), np.log(512)))), int(np.exp(rng.uniform(np.log(48), np.log(400))))) for _ in range(7)]
SETS = {  # sizes: planes of a strip where 148 SMs choose (0: a thread per cell), without and with the hint
    "one_large": ([(512, 512)] + [(33, 31)] * 23, 8, None),
    "mixed": (MIXED + [(512, 400)], 0, None),
    "thin": ([(2048, 16), (16, 1024), (3, 3)], 8, None),
    "small": ([(3 + k % 37, 3 + k % 31) for k in range(200)], 0, None),
    "wide_range": ([(1024, 500)] * 12 + [(257, 129)] * 30, 32, None),
    "same": ([(203, 117)] * 24, 0, 8),
}


@pytest.mark.parametrize("name", list(SETS))
@pytest.mark.parametrize("storage", ["float32", "float16"])
def test_uneven_worlds(name, storage):
    from torch.profiler import ProfilerActivity, profile

    from openhomelbm_b200 import _lib
    from openhomelbm_b200.batching import TileConfig, WorldBatch2D
    from openhomelbm_b200.lbm import LBM_Solver

    sizes, planes, planes_same = SETS[name]
    torch.manual_seed(4)
    flows = []
    for nx, ny in sizes:
        s = LBM_Solver(nx, ny, solid_num=1, storage=storage, u_scale=0.05, s_scale=2.5e-3)
        f = s.flows[0]
        m = torch.rand((6, nx, ny), device="cuda") - 0.5
        if f.encoded:
            m[0] *= 0.1
        else:
            m[1:3] *= 0.1
            m[3:] *= 0.02
            m[0] = 1.0 + 0.1 * m[0]
        f.moments[0].copy_(m)
        flows.append(f)
    b = WorldBatch2D(flows)
    st = _lib.stream_ptr()

    def launch(phases):
        for f in flows:
            f.moments[1].zero_()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            _lib.check(_lib.lib().hl_d2q9_step_batch(_lib.ptr(b.desc), b.n, 0, b.storage_code, max(n[0] for n in sizes),
                                                     max(n[1] for n in sizes), 0, phases, st))
            torch.cuda.synchronize()
        names = [e.key for e in p.key_averages() if "stream" in e.key and "kernel" in e.key]
        strips = [int(m.group(1)) for m in (re.search(r"stream_strips_kernel<[^,]*, (\d+)>", n) for n in names) if m]
        return [f.moments[1].clone() for f in flows], (strips + [0])[0] if names else None

    got, tx = launch(_lib.HL_PHASE_STREAM)
    for f in flows:
        f.moments[1].zero_()
    b.launch(0, st, TileConfig(8, 32, 1184), phases=_lib.HL_PHASE_STREAM, any_solid=False)
    torch.cuda.synchronize()
    for f, g in zip(flows, got):
        assert torch.equal(f.moments[1], g), (f.nx, f.ny)
    assert got[0].double().std() > 0
    b200 = torch.cuda.get_device_properties(0).multi_processor_count == 148
    if b200 and tx is not None:  # None: the profiler records nothing here
        assert tx == planes
    if planes_same is not None:
        again, tx = launch(_lib.HL_PHASE_STREAM | _lib.HL_PHASE_SAME_SIZE)
        for g, h in zip(again, got):
            assert torch.equal(g, h)
        if b200 and tx is not None:
            assert tx == planes_same
