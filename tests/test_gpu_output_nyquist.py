"""Offline reconstructions whose shifted OTF supports reach the output grid's Nyquist column and row
under an apodization that reaches them too. Both lines are their own mirror images, but masks,
Wiener denominator and apodization are evaluated at one coordinate of the two (-N along x, +N
along y). Tolerance: relative L2 <= 1e-5 against the FP64 oracle, the bound of the other fused
tests (single precision through 12 transforms of length <= 2^10: about 1e-6)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _make(fs, n, seed, pixel, bands=2, apo=2.0, measured=False, att=False):
    kw = dict(n_bands=3, n_phases=5) if bands == 3 else {}
    raw, truth = fs.synth.make_dataset(n=n, seed=seed, na=1.49, em_wavelength=488.0, pxl_um=pixel,
                                       k0_frac=0.85 / (bands - 1), **kw)
    sp = fs.synth.sim_param_for(truth, n, n_phases=kw.get("n_phases", 3), n_bands=bands)
    if measured:
        from test_gpu_vector_api import measured_otf
        sp.setOtf(measured_otf(fs, samples=300, bands=bands, na=1.49, lam=488.0))
    if att:
        sp.otf().setAttenuation(0.97, 1.1)
        sp.otf().switchAttenuation(True)
    sp.setApoCutoff(apo)
    return raw, sp


def _plan(fs, sp):
    return fs.plan.ReconPlan(sp, path=fs.native.PATH_OFFLINE, input_type=fs.native.INPUT_F32, fade_px=10)


def _exact(oracle, sp, raw):
    return oracle.recon_raw(sp, raw.astype(np.float64), fade=10, dtype=np.float64)


# the cutoff radius is 6.107 * pixel * n pixels, the shifts 0.85 of it
@pytest.mark.parametrize("n,pixel,bands,measured,att", [
    (64, 0.09, 2, False, False), (64, 0.12, 3, False, False), (128, 0.09, 2, False, False),
    (128, 0.10, 2, False, False), (128, 0.12, 2, False, False), (128, 0.165, 2, False, False),
    (192, 0.10, 3, False, False), (256, 0.085, 2, False, False), (256, 0.12, 2, False, True),
    (384, 0.10, 2, False, False), (512, 0.10, 2, False, False), (64, 0.12, 2, True, False),
    (128, 0.10, 2, True, True), (128, 0.12, 3, True, False), (192, 0.12, 2, True, False)])
def test_offline_output_nyquist_vs_fp64(fs, oracle, n, pixel, bands, measured, att):
    raw, sp = _make(fs, n, n + bands, pixel, bands, 2.0, measured, att)
    assert rel_l2(_plan(fs, sp).reconstruct_host(raw), _exact(oracle, sp, raw)) < 1e-5


@pytest.mark.parametrize("n", [64, 192])
def test_output_nyquist_in_mixed_batches(fs, oracle, torch_cuda, n):
    """One batch with supports inside and beyond the output grid and complex masks, alone and as a
    graph: every job gives the bits of its own single-job batch."""
    torch = torch_cuda
    made = [_make(fs, n, 11, 0.08), _make(fs, n, 12, 0.12), _make(fs, n, 13, 0.10, measured=True),
            _make(fs, n, 14, 0.10, bands=3)]
    plans = [_plan(fs, sp) for _, sp in made]
    alone = [p.reconstruct_host(raw) for p, (raw, _) in zip(plans, made)]
    for got, (raw, sp) in zip(alone, made):
        assert rel_l2(got, _exact(oracle, sp, raw)) < 1e-5
    d_raw = [torch.from_numpy(raw).cuda() for raw, _ in made]
    d_out = torch.zeros((2, len(made), 2 * n, 2 * n), dtype=torch.float32, device="cuda")
    ws = torch.empty(fs.plan.batch_workspace_bytes(plans), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    jobs = [[(p, r.data_ptr(), o.data_ptr()) for p, r, o in zip(plans, d_raw, out)] for out in d_out]
    fs.plan.recon_batch(jobs[0], ws.data_ptr(), ws.numel())
    torch.cuda.synchronize()
    g = fs.plan.BatchGraph(jobs[1], ws.data_ptr(), ws.numel())
    g.launch()
    torch.cuda.synchronize()
    for out in d_out:
        for got, exp in zip(out.cpu().numpy(), alone):
            assert np.array_equal(got, exp)


def test_output_nyquist_after_plan_update(fs, oracle, torch_cuda):
    """A plan built for an apodization that ends inside the output grid, updated to one that
    reaches the Nyquist lines and back: new batches and a graph recorded before the updates."""
    torch = torch_cuda
    raw, inside = _make(fs, 128, 3, 0.10, apo=1.5)
    beyond = _make(fs, 128, 3, 0.10, apo=2.0)[1]
    plan = _plan(fs, inside)
    d_raw = torch.from_numpy(raw).cuda()
    d_out = torch.zeros((256, 256), dtype=torch.float32, device="cuda")
    ws = torch.empty(fs.plan.batch_workspace_bytes([plan]), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    g = fs.plan.BatchGraph([(plan, d_raw.data_ptr(), d_out.data_ptr())], ws.data_ptr(), ws.numel())
    for sp in (beyond, inside):
        plan.update(sp)
        exp = _exact(oracle, sp, raw)
        assert rel_l2(plan.reconstruct_host(raw), exp) < 1e-5
        g.launch()
        torch.cuda.synchronize()
        assert rel_l2(d_out.cpu().numpy(), exp) < 1e-5


@pytest.mark.parametrize("pixel,measured", [(0.08, True), (0.12, False), (0.10, True)])
def test_short_and_long_batches_same_bits(fs, torch_cuda, pixel, measured):
    """Short batches run band 0 and the pairs as one dependent launch behind passes A and G, long ones as
    two launches: the same bits with complex masks and edge weights too (real masks inside the grid
    in test_gpu_short_batches.py)."""
    torch = torch_cuda
    n, count = 64, 640
    raw, sp = _make(fs, n, 21, pixel, measured=measured)
    plan = _plan(fs, sp)
    gain = torch.linspace(0.5, 2.0, count, device="cuda").view(-1, 1, 1, 1)
    d_raw = (torch.from_numpy(raw).cuda().reshape(1, -1, n, n) * gain).contiguous()
    out = torch.empty((2, count, 2 * n, 2 * n), dtype=torch.float32, device="cuda")
    ws = torch.empty(fs.plan.batch_workspace_bytes([plan] * count), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for dst, step in zip(out, (count, 5)):
        for k in range(0, count, step):
            fs.plan.recon_batch([(plan, d_raw[i].data_ptr(), dst[i].data_ptr()) for i in range(k, k + step)],
                                ws.data_ptr(), ws.numel())
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
