"""The parameter fit on line pairs (every size it has transforms for, from raw frames and from
spectra, two and three bands) against the oracle, and the paired 2D FFT at its edges."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _estimate_raw(fs, sp, raw, fade, band):
    import torch
    N_ = fs.native
    c = N_.to_c_param(sp)
    u16 = raw.dtype == np.uint16
    d = torch.from_numpy(raw.view(np.int16) if u16 else raw).cuda()
    torch.cuda.synchronize()
    peaks = np.zeros((sp.nrDirs, 4))
    N_.check(N_.lib().fsim_estimate_raw(C.byref(c), C.c_void_p(d.data_ptr()), N_.INPUT_U16 if u16 else N_.INPUT_F32,
                                        fade, band, C.c_double(0.6), peaks.ctypes.data_as(C.c_void_p)))
    return N_.from_c_param(c), peaks


@pytest.mark.parametrize("n,bands,band,u16,fade", [(128, 2, 1, False, 10), (256, 2, 1, True, 0), (384, 2, 1, False, 10),
                                                   (384, 3, 2, False, 10), (256, 3, 2, True, 7), (512, 3, 1, False, 10),
                                                   (768, 2, 1, True, 10), (192, 2, 1, False, 10)])
def test_fit_vs_oracle(fs, oracle, torch_cuda, n, bands, band, u16, fade):
    """Shifts equal the oracle's grid points to 1e-9 px (192 runs the op-by-op form); phases and
    modulations within 1e-4: single-precision spectra, summed over at least 10^3 bins."""
    nph = 5 if bands == 3 else 3
    # band 1 of a three-band fit is searched beyond 0.6 of the cutoff: a pattern it can find there
    k0 = {(2, 1): 0.85, (3, 2): 0.43, (3, 1): 0.7}[(bands, band)]
    raw, truth = fs.synth.make_dataset(n=n, seed=900 + n + bands, n_phases=nph, n_bands=bands, k0_frac=k0, as_u16=u16)
    sp = fs.synth.sim_param_for(truth, n, n_phases=nph, n_bands=bands, known=False)
    spec = oracle.prepare_raw(sp, raw.astype(np.float32), fade=fade)
    par, peaks, _ = oracle.estimate(sp, spec, fit_band=band)
    got, gp = _estimate_raw(fs, sp, raw, fade, band)
    assert np.abs(gp[:, :2] - peaks[:, :2]).max() < 1e-9
    assert np.abs(gp[:, 3] - peaks[:, 3]).max() < 1e-4
    assert np.abs(np.array(got["pX"]) - np.array(par["pX"])).max() < 1e-9
    assert np.abs(np.angle(np.exp(1j * (np.array(got["phaOff"]) - np.array(par["phaOff"]))))).max() < 1e-4
    for d in range(3):
        assert np.abs(np.array(got["modulations"][d]) - np.array(par["modulations"][d])).max() < 1e-4
    # the same from spectra through the vector API
    V = fs.vectors
    vecs = [[V.Vec2dCplx(n, n) for _ in range(nph)] for _ in range(3)]
    for a in range(3):
        for p in range(nph):
            vecs[a][p].setData(spec[a * nph + p].astype(np.complex64))
    sp2 = sp.duplicate()
    vp = fs.algorithm.SimAlgorithm.estimateParameters(sp2, vecs, band, 0.6)
    assert np.abs(vp[:, :2] - peaks[:, :2]).max() < 1e-9


@pytest.mark.parametrize("w,h,batch,off", [(32, 64, 3, 0), (64, 32, 2, 1), (48, 96, 5, 0), (1024, 48, 1, 1), (512, 512, 3, 1),
                                           (3072, 32, 1, 0), (64, 4096, 1, 0), (256, 2048, 2, 1)])
@pytest.mark.parametrize("inverse", [0, 1])
def test_fft2d_pairs(fs, torch_cuda, w, h, batch, off, inverse):
    """Shortest and longest lines, 3*2^k lengths, blocks only partly filled, and planes whose base
    is 8-byte but not 16-byte aligned; 1e-6 relative L2: about 2^-24 per level of the transform."""
    torch = torch_cuda
    N_ = fs.native
    N_.init(0)
    g = torch.Generator(device="cuda").manual_seed(w + h)
    buf = torch.randn(batch * h * w + 2, dtype=torch.complex64, device="cuda", generator=g)
    x = buf[off:off + batch * h * w].view(batch, h, w)
    f = torch.fft.ifft2 if inverse else torch.fft.fft2
    ref = f(x.to(torch.complex128)).cpu().numpy()
    edge = buf[[0, -1, -2]].cpu().numpy()
    torch.cuda.synchronize()
    N_.check(N_.lib().fsim_fft2d_batch(C.c_void_p(x.data_ptr()), w, h, batch, inverse, None))
    N_.check(N_.lib().fsim_sync())
    assert rel_l2(x.cpu().numpy(), ref) < 1e-6
    after = buf[[0, -1, -2]].cpu().numpy()
    if off:
        assert after[0] == edge[0] and after[1] == edge[1]  # nothing outside the planes is written
    else:
        assert after[1] == edge[1] and after[2] == edge[2]


@pytest.mark.parametrize("w,h", [(48, 192), (96, 384), (192, 1536), (384, 768), (768, 96), (1536, 48)])
@pytest.mark.parametrize("inverse", [0, 1])
def test_fft2d_radix12_plans(fs, torch_cuda, w, h, inverse):
    """Every 3*2^k plan that ends in a radix-12 stage, along rows and along columns; 1e-6 relative
    L2 as above."""
    torch = torch_cuda
    N_ = fs.native
    N_.init(0)
    g = torch.Generator(device="cuda").manual_seed(w + h)
    x = torch.randn(2, h, w, dtype=torch.complex64, device="cuda", generator=g)
    f = torch.fft.ifft2 if inverse else torch.fft.fft2
    ref = f(x.to(torch.complex128)).cpu().numpy()
    torch.cuda.synchronize()
    N_.check(N_.lib().fsim_fft2d_batch(C.c_void_p(x.data_ptr()), w, h, 2, inverse, None))
    N_.check(N_.lib().fsim_sync())
    assert rel_l2(x.cpu().numpy(), ref) < 1e-6
