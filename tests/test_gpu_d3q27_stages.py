"""The tuning key "d3q27_stages": the depth of the 16-bit storages' staging, with the same field at each."""
import pytest
import torch

from test_gpu_stored_bits import STEP, step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stages", [3, 4, 5])
@pytest.mark.parametrize("storage", ["float16", "bfloat16"])
def test_staging_depth_is_the_one_asked_for(storage, stages):
    from torch.profiler import ProfilerActivity, profile

    from openhomelbm_b200 import _lib

    _lib.set_tuning("d3q27_stages", stages)
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            got = step((20, 32, 64), storage, True, False, False)
            torch.cuda.synchronize()
    finally:
        _lib.set_tuning("d3q27_stages", 0)
    assert got == STEP[(20, 32, 64), storage, True, False]
    names = [e.key for e in p.key_averages()]
    if not names:
        pytest.skip("the profiler records nothing here")
    names = [n for n in names if "step_kernel_tma" in n]
    assert names and all(f"{storage.replace('bfloat', 'BF').replace('float', 'F')}, {stages}," in n for n in names), names
