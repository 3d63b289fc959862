"""D3Q27 outer boundaries: the one-launch pass against the three waves.

A batch that holds a world with a side of three cells runs in waves, a lone world of larger sides in
one pass: both write the same values, to the bit, since each cell's arithmetic is the same.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["float64", "float32", "bfloat16"])
@pytest.mark.parametrize("shape", [(4, 4, 4), (4, 5, 6), (5, 4, 33), (7, 130, 4), (4, 4, 300), (37, 19, 6)])
def test_one_pass_equals_waves(shape, storage):
    from openhomelbm_b200 import _lib

    L = _lib.lib()
    st = _lib.stream_ptr()
    code = _lib.DTYPES[storage]
    sto = _lib.hl_storage(code, 0.05, 2e-3) if storage == "bfloat16" else _lib.hl_storage(code, 1.0, 1.0)
    rng = np.random.default_rng(17)

    def world(sh, types):
        m = [torch.tensor(rng.uniform(-0.5, 0.5, (10, *sh)), dtype=_lib.torch_dtype(code), device="cuda") for _ in range(2)]
        if storage != "bfloat16":
            m[0][0] += 1.0
            m[1][0] += 1.0
        bc = _lib.hl_bc3d()
        for f in range(6):
            bc.bc_type[f] = int(types[f])
            for k in range(3):
                bc.bc_value[f][k] = float(rng.uniform(-0.03, 0.03))
        w = _lib.hl_world3d(*sh, sto, m[0].data_ptr(), m[1].data_ptr(), None, None, 0)
        scratch = torch.zeros(int(L.hl_d3q27_bc_scratch_bytes(ctypes.byref(w))), dtype=torch.uint8, device="cuda")
        return m, bc, w, scratch

    for types in ((1, 0, 1, 0, 2, 1), (0, 2, 2, 1, 0, 0), (2, 1, 0, 2, 1, 2)):
        doms = [world(shape, types), world((3, 3, 3), types)]
        n = len(doms)
        nbytes = int(L.hl_d3q27_bc_batch_bytes(n))
        desc = torch.empty(nbytes + 16, dtype=torch.uint8, device="cuda")
        ptr = (desc.data_ptr() + 15) // 16 * 16
        worlds = (_lib.hl_world3d * n)(*[d[2] for d in doms])
        bcs = (_lib.hl_bc3d * n)(*[d[1] for d in doms])
        scr = (ctypes.c_void_p * n)(*[d[3].data_ptr() for d in doms])
        _lib.check(L.hl_d3q27_bc_batch_prepare(worlds, bcs, scr, n, ptr, nbytes, st), "prepare")
        m, bc, w, scratch = doms[0]
        start = m[1].clone()
        _lib.check(L.hl_d3q27_apply_bc(ctypes.byref(w), ctypes.byref(bc), scratch.data_ptr(), st), "pass")
        got = m[1].clone()
        m[1].copy_(start)
        _lib.check(L.hl_d3q27_apply_bc_batch(ptr, n, 0, st), "waves")
        torch.cuda.synchronize()
        assert not torch.equal(got, start)
        assert torch.equal(got, m[1]), types
