"""The 2D FFT on both sides of the size where it goes from single lines to line pairs (powers of
two: 2^19 elements, 2^20 with lines of 1024 and beyond), at the shortest and longest lines, and
4096-point columns; 1e-6 relative L2 against a 64-bit FFT: about 2^-24 per level of the transform."""
import ctypes as C

import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,batch,off", [(64, 64, 1, 0), (64, 64, 128, 1), (64, 64, 129, 0), (1024, 1024, 1, 1),
                                           (1024, 1024, 2, 1), (4096, 64, 4, 0), (64, 4096, 5, 1), (4096, 256, 1, 0),
                                           (2048, 512, 1, 0), (2048, 1024, 1, 0), (128, 256, 3, 0), (96, 64, 1, 0),
                                           (256, 4096, 2, 0)])
@pytest.mark.parametrize("inverse", [0, 1])
def test_fft2d_lines_and_pairs(fs, torch_cuda, w, h, batch, off, inverse):
    torch = torch_cuda
    N_ = fs.native
    N_.init(0)
    g = torch.Generator(device="cuda").manual_seed(w * batch + h)
    buf = torch.randn(batch * h * w + 2, dtype=torch.complex64, device="cuda", generator=g)
    x = buf[off:off + batch * h * w].view(batch, h, w)
    f = torch.fft.ifft2 if inverse else torch.fft.fft2
    ref = f(x.to(torch.complex128)).cpu().numpy()
    edge = buf[[0, -1]].cpu().numpy()
    torch.cuda.synchronize()
    N_.check(N_.lib().fsim_fft2d_batch(C.c_void_p(x.data_ptr()), w, h, batch, inverse, None))
    N_.check(N_.lib().fsim_sync())
    assert rel_l2(x.cpu().numpy(), ref) < 1e-6
    after = buf[[0, -1]].cpu().numpy()
    assert after[1] == edge[1] and (not off or after[0] == edge[0])  # nothing outside the arrays is written
