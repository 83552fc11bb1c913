"""Short offline batches run their passes as dependent launches, long ones do not: both give the
same bits, also when short batches with other inputs follow one another on one workspace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,per_call", [(64, 640, 1), (64, 640, 7), (256, 48, 1), (192, 112, 3)])
def test_short_batches_match_one_long_batch(fs, n, count, per_call):
    import torch
    raw, truth = fs.synth.make_dataset(n=n, seed=n, na=1.49, em_wavelength=488.0, pxl_um=0.08)
    sp = fs.synth.sim_param_for(truth, n, n_phases=3, n_bands=2)
    plan = fs.plan.ReconPlan(sp, path=fs.native.PATH_OFFLINE, input_type=fs.native.INPUT_F32, fade_px=10)
    gain = torch.linspace(0.5, 2.0, count, device="cuda").view(-1, 1, 1, 1)
    d_raw = (torch.as_tensor(np.asarray(raw, np.float32), device="cuda").reshape(1, -1, n, n) * gain).contiguous()
    out = torch.empty((2, count, 2 * n, 2 * n), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()

    def run(first, number, dst, ws):
        fs.plan.recon_batch([(plan, d_raw[k].data_ptr(), dst[k].data_ptr()) for k in range(first, first + number)],
                            ws.data_ptr(), ws.numel())

    ws = torch.empty(fs.plan.batch_workspace_bytes([plan] * count), dtype=torch.uint8, device="cuda")
    run(0, count, out[0], ws)
    for k in range(0, count, per_call):
        run(k, min(per_call, count - k), out[1], ws)
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
