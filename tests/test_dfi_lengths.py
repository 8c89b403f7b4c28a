"""DFI's row transform at the convolution lengths whose last radix is 2, 4 and 8
(``atb_dfi_rows``), the smallest and the largest among them, against NumPy's
FP64 transform (algotom/rec/reconstruction.py:774-776).

The FP64 convolution's error is a few 1e-16 of the row's norm per stage, ten
stages with the products: below 1e-12 of the largest output.
"""
import numpy as np
import pytest

from algotom_b200 import _native as nat
from algotom_b200.rec import dfi
from algotom_b200.rec import reconstruction as R


@pytest.mark.gpu
@pytest.mark.parametrize("w,m", [(3, 16), (9, 32), (31, 64), (65, 256),
                                 (201, 512), (511, 1024), (1601, 4096),
                                 (4095, 8192)])
def test_row_transform(cuda, w, m):
    import torch
    assert nat.load().atb_dfi_fft_length(w) == m
    rng = np.random.default_rng(w)
    nrow, nslice = 3, 2
    x = rng.random((nrow, nslice, w)).astype(np.float32) + 0.1
    t = torch.as_tensor(x, device="cuda")
    chirp, tw, bfwd, binv = dfi._fft_tables(w, t.device)
    out = torch.empty((nrow, nslice, w), dtype=torch.complex128,
                      device="cuda")
    nat.call("atb_dfi_rows", t.data_ptr(), nslice * w, w, nrow, nslice, w, 0,
             nat.PAD_MODES["edge"], 0, None, None, chirp.data_ptr(),
             tw.data_ptr(), bfwd.data_ptr(), binv.data_ptr(), out.data_ptr(),
             nslice * w, w, R._stream_ptr())
    got = out.cpu().numpy()
    ref = np.fft.fftshift(np.fft.fft(np.fft.ifftshift(
        x.astype(np.float64), axes=2), axis=2), axes=2)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
