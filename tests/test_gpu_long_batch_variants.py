"""Launch-shape variants in batches long enough for the form without dependent launches: every variant
of every pass gives the oracle's image (relative L2 <= 1e-4 against the single-precision oracle, the
bound of the single-stack variant test)."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(384, 27), (512, 11), (1024, 6)])
def test_every_variant_in_a_long_batch(fs, oracle, torch_cuda, n, count):
    torch = torch_cuda
    N_, lib = fs.native, fs.native.lib()
    raw, truth = fs.synth.make_dataset(n=n, seed=200 + n)
    sp = fs.synth.sim_param_for(truth, n)
    exp = oracle.recon_raw(sp, raw, fade=10)
    plan = fs.plan.ReconPlan(sp, path=N_.PATH_OFFLINE, input_type=N_.INPUT_F32, fade_px=10)
    d_raw = torch.from_numpy(np.ascontiguousarray(raw, np.float32)).cuda()
    d_out = torch.empty((count, 2 * n, 2 * n), dtype=torch.float32, device="cuda")
    ws = torch.empty(fs.plan.batch_workspace_bytes([plan] * count), dtype=torch.uint8, device="cuda")
    jobs = [(plan, d_raw.data_ptr(), o.data_ptr()) for o in d_out]
    torch.cuda.synchronize()
    v, cnt, saved = C.c_int(), C.c_int(), []
    for p in range(3):
        N_.check(lib.fsim_tune_get(n, N_.PATH_OFFLINE, p, C.byref(v), C.byref(cnt)))
        saved.append((v.value, cnt.value))
    try:
        for p in range(3):
            for var in range(saved[p][1]):
                N_.check(lib.fsim_tune_set(n, N_.PATH_OFFLINE, p, var))
                d_out.zero_()
                torch.cuda.synchronize()
                fs.plan.recon_batch(jobs, ws.data_ptr(), ws.numel())
                torch.cuda.synchronize()
                assert rel_l2(d_out[0].cpu().numpy(), exp) < 1e-4, (p, var)
                assert torch.equal(d_out[0], d_out[-1]) and torch.equal(d_out[0], d_out[count // 2]), (p, var)
            N_.check(lib.fsim_tune_set(n, N_.PATH_OFFLINE, p, saved[p][0]))
    finally:
        for p in range(3):
            N_.check(lib.fsim_tune_set(n, N_.PATH_OFFLINE, p, saved[p][0]))
