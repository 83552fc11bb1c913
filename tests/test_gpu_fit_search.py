"""The parameter search's own phase and magnitude (the third and fourth value of every reported peak)
against the FP64 oracle, at every number of threads per row of the search's sums. Bound 5e-7:
four times what the single-precision oracle differs from the FP64 one on such stacks (1.3e-7)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,u16", [(128, False), (256, True), (384, False), (512, False), (1024, True)])
def test_search_phase_and_magnitude_vs_fp64(fs, oracle, torch_cuda, n, u16):
    N_ = fs.native
    raw, truth = fs.synth.make_dataset(n=n, seed=70 + n, k0_frac=0.85, as_u16=u16)
    sp = fs.synth.sim_param_for(truth, n, known=False)
    spec = oracle.prepare_raw(sp, raw.astype(np.float64), fade=10, dtype=np.float64)
    _, exp, _ = oracle.estimate(sp, spec, fit_band=1, dtype=np.float64)
    c = N_.to_c_param(sp)
    d = torch_cuda.from_numpy(raw.view(np.int16) if u16 else raw).cuda()
    torch_cuda.cuda.synchronize()
    got = np.zeros((sp.nrDirs, 4))
    N_.check(N_.lib().fsim_estimate_raw(C.byref(c), C.c_void_p(d.data_ptr()), N_.INPUT_U16 if u16 else N_.INPUT_F32, 10, 1,
                                        C.c_double(0.6), got.ctypes.data_as(C.c_void_p)))
    assert np.abs(got[:, :2] - exp[:, :2]).max() < 1e-9
    assert np.abs(np.angle(np.exp(1j * (got[:, 2] - exp[:, 2])))).max() < 5e-7
    assert np.abs(got[:, 3] - exp[:, 3]).max() < 5e-7


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_bins_beyond_the_otf_may_hold_anything(fs, oracle, torch_cuda, bad):
    """Spectra whose bins beyond the OTF support are not finite (as after a division by the OTF): the
    coarse correlation finds no peak, and the search from its fallback start zeroes those bins as the
    oracle does. Bounds as for finite spectra (single-precision spectra, 1e-4 in the reported value)."""
    n = 128
    raw, truth = fs.synth.make_dataset(n=n, seed=8, pxl_um=0.06, k0_frac=0.85)
    sp = fs.synth.sim_param_for(truth, n, known=False)
    spec = oracle.prepare_raw(sp, raw, fade=10).astype(np.complex64)
    f = np.fft.fftfreq(n) * n
    spec[:, np.hypot(f[None, :], f[:, None]) > truth["cutoff_px"] + 2] = bad
    _, exp, _ = oracle.estimate(sp, spec, fit_band=1)
    V = fs.vectors
    vecs = [[V.Vec2dCplx(n, n) for _ in range(3)] for _ in range(3)]
    for a in range(3):
        for p in range(3):
            vecs[a][p].setData(spec[3 * a + p])
    got = fs.algorithm.SimAlgorithm.estimateParameters(sp, vecs, 1, 0.6)
    assert np.isfinite(exp).all()
    assert np.abs(got[:, :2] - exp[:, :2]).max() < 1e-9
    assert np.abs(got[:, 3] - exp[:, 3]).max() < 1e-4
