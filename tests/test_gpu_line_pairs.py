"""The fused passes on line pairs where their index rules change: OTF windows wider than the raw
spectrum (each transform element then holds two window columns or rows), windows as wide as the
output grid, real and complex masks, every radix plan. Tolerance: relative L2 <= 1e-5 against
the FP64 oracle, the bound of the other fused tests (single precision through 12 transforms of
length <= 2^10: about 1e-6)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _make(fs, n, seed, pixel, apo=2.0, **kw):
    raw, truth = fs.synth.make_dataset(n=n, seed=seed, na=1.49, em_wavelength=488.0, pxl_um=pixel, **kw)
    sp = fs.synth.sim_param_for(truth, n, n_phases=kw.get("n_phases", 3), n_bands=kw.get("n_bands", 2))
    sp.setApoCutoff(apo)
    return raw, sp


# the cutoff radius is 6.107 * pixel * n pixels; the apodization ends inside the output grid
@pytest.mark.parametrize("n,pixel,apo", [(64, 0.1, 1.5), (192, 0.1, 1.5), (256, 0.09, 1.7), (512, 0.1, 1.5),
                                         (128, 0.165, 0.9), (384, 0.165, 0.9)])
@pytest.mark.parametrize("bands", [2, 3])
def test_offline_wide_windows_vs_fp64(fs, oracle, n, pixel, apo, bands):
    kw = dict(n_bands=3, n_phases=5) if bands == 3 else {}
    raw, sp = _make(fs, n, n + bands, pixel, apo, k0_frac=(0.3 if bands == 3 else 0.45), **kw)
    plan = fs.plan.ReconPlan(sp, path=fs.native.PATH_OFFLINE, input_type=fs.native.INPUT_F32, fade_px=10)
    got = plan.reconstruct_host(raw)
    assert rel_l2(got, oracle.recon_raw(sp, raw.astype(np.float64), fade=10, dtype=np.float64)) < 1e-5


@pytest.mark.parametrize("n,pixel,apo", [(64, 0.1, 1.5), (192, 0.08, 2.0), (256, 0.1, 1.5)])
def test_offline_complex_masks_vs_fp64(fs, oracle, n, pixel, apo):
    from test_gpu_vector_api import measured_otf
    raw, sp = _make(fs, n, n + 7, pixel, apo, k0_frac=0.5)
    sp.setOtf(measured_otf(fs, samples=300))
    plan = fs.plan.ReconPlan(sp, path=fs.native.PATH_OFFLINE, input_type=fs.native.INPUT_F32, fade_px=10)
    got = plan.reconstruct_host(raw)
    assert rel_l2(got, oracle.recon_raw(sp, raw.astype(np.float64), fade=10, dtype=np.float64)) < 1e-5


@pytest.mark.parametrize("n,pixel", [(64, 0.08), (64, 0.1), (128, 0.165), (256, 0.1), (384, 0.08), (512, 0.09)])
@pytest.mark.parametrize("shift", ["fraction", "whole", "mixed"])
def test_live_edges_vs_fp64(fs, oracle, n, pixel, shift):
    """The live path's mirrored halves: fractional, whole-pixel and mixed shifts (the edge bins
    of the pasted ranges differ), supports inside and beyond the raw spectrum, apodization that
    reaches the Nyquist row and column of the output."""
    raw, sp = _make(fs, n, n + 3, pixel, k0_frac=0.45, as_u16=True)
    for d in range(3):
        v = sp.dir(d)
        x, y = v.px(1), v.py(1)
        if shift == "whole" or (shift == "mixed" and d == 0):
            x, y = round(x), round(y)
        elif shift == "mixed" and d == 1:
            x = round(x)
        v.setPxPy(x, y)
    plan = fs.plan.ReconPlan(sp, path=fs.native.PATH_LIVE, input_type=fs.native.INPUT_U16, fade_px=10)
    got = plan.reconstruct_host(raw)
    exp, _ = oracle.live_recon(sp, raw, dtype=np.float64)
    assert rel_l2(got, exp[0]) < 1e-5


def test_live_three_bands_vs_fp64(fs, oracle):
    raw, sp = _make(fs, 128, 5, 0.08, k0_frac=0.45, as_u16=True, n_bands=3, n_phases=5)
    plan = fs.plan.ReconPlan(sp, path=fs.native.PATH_LIVE, input_type=fs.native.INPUT_U16, fade_px=10)
    got = plan.reconstruct_host(raw)
    exp, _ = oracle.live_recon(sp, raw, dtype=np.float64)
    assert rel_l2(got, exp[0]) < 1e-5
