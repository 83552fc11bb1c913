"""The library's scratch pool keeps memory between calls and gives it back: destroying a plan or
closing a server leaves nothing of a fit's scratch behind for other users of the GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(fs, torch, n=1024):
    """A fit whose scratch is some hundred MiB (its result does not matter here)."""
    N_ = fs.native
    sp = fs.synth.synthetic_params(n)
    c = N_.to_c_param(sp)
    d = torch.rand((9, n, n), device="cuda")
    torch.cuda.synchronize()
    peaks = np.zeros((3, 4))
    N_.check(N_.lib().fsim_estimate_raw(C.byref(c), C.c_void_p(d.data_ptr()), N_.INPUT_F32, 10, 1, C.c_double(0.6),
                                        peaks.ctypes.data_as(C.c_void_p)))


@pytest.mark.parametrize("how", ["plan", "server"])
def test_idle_scratch_is_given_back(fs, torch_cuda, how):
    torch = torch_cuda
    N_ = fs.native
    sp = fs.synth.synthetic_params(64)
    if how == "plan":
        held = fs.plan.ReconPlan(sp, path=N_.PATH_OFFLINE, input_type=N_.INPUT_F32, fade_px=10)
    else:
        held = fs.plan.Server([sp], max_batch=1, max_inflight=1, streams=1, refit_every=0)
    torch.cuda.empty_cache()
    _fit(fs, torch)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held.close()
    torch.cuda.synchronize()
    # 3 x 1024^2: planes of 16 bytes, spectra of 9 frames: at least 100 MiB
    assert torch.cuda.mem_get_info()[0] - before >= 100 << 20
    _fit(fs, torch)  # and the pool serves the next call
