"""Diagnostics scratch of one partial sum per SM, the size that hl_d3q27_stream_collide has always taken.

The sweep kernel runs two blocks per SM, which share this scratch's partial sums. The field is the same, the health
count too, and the mass is a binary64 sum of the same positive terms in another order. A term passes
through at most 4000 additions (a thread's cells, the block's tree, the blocks' sums), each within 2^-53:
4000 x 2^-53 on either side, below 1e-12 of the mass.
"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,shape", [("float32", (96, 64, 64)), ("float32", (96, 50, 44)), ("float32", (60, 47, 53)),
                                           ("float64", (96, 64, 64)), ("float64", (70, 41, 33)), ("float16", (96, 64, 64)),
                                           ("bfloat16", (64, 48, 96))])
def test_scratch_of_one_block_per_sm(storage, shape):
    from openhomelbm_b200 import _lib
    from openhomelbm_b200.lbm3d import LBM_Solver3D

    L = _lib.lib()
    least = torch.cuda.get_device_properties(0).multi_processor_count * 12 + 64
    kw = dict(u_scale=0.05, s_scale=2.5e-3) if "16" in storage else {}
    s = LBM_Solver3D(*shape, periodic="16" in storage, storage=storage, use_graph=False, **kw)
    f = s.flows[0]
    g = torch.Generator(device="cuda").manual_seed(3)
    for m in f.moments:
        m.copy_(0.02 * (torch.rand(m.shape, generator=g, device="cuda") - 0.5))
        if not kw:
            m[0] += 1.0
    w = f.world_struct(0)
    out = []
    for size in (least, int(L.hl_d3q27_scratch_bytes(ctypes.byref(w)))):
        buf = torch.zeros(size + 256, dtype=torch.uint8, device="cuda")
        buf[size:] = 0x5A
        mass = torch.zeros(1, dtype=torch.float64, device="cuda")
        health = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        f.moments[1].fill_(1)
        d = _lib.hl_diag(buf.data_ptr(), size, mass.data_ptr(), health.data_ptr())
        for _ in range(2):  # the counter is back at zero for the next call
            mass.zero_()
            _lib.check(L.hl_d3q27_stream_collide(w, 0.02, ctypes.byref(d), _lib.stream_ptr()), "step")
        torch.cuda.synchronize()
        assert (buf[size:] == 0x5A).all()
        out.append((f.moments[1].clone(), float(mass), int(health)))
    assert torch.equal(out[0][0], out[1][0])
    assert out[0][2] == out[1][2] == 0
    assert out[0][1] > 0 and abs(out[0][1] - out[1][1]) <= 1e-12 * out[1][1]
    d = _lib.hl_diag(buf.data_ptr(), least - 1, mass.data_ptr(), health.data_ptr())
    assert L.hl_d3q27_stream_collide(w, 0.02, ctypes.byref(d), _lib.stream_ptr()) == _lib.HL_ERR_ARG
