"""The 2-D filter of BPF at the transform lengths where its kernels differ:
one stage only, with and without the radices 11 and 13, and lengths of which
many, three, two and one fit an SM.

Reference: ``apply_circular_ramp_filter`` (algotom/rec/reconstruction.py
:527-560).  A window that shifts by whole pixels must return the padded image's
own samples, a ramp window the FP64 oracle's.  The device transforms are FP64
(errors of 1e-15 of the image's largest sample per stage, ten stages at most,
summed over both axes: below 1e-12 of it) and round the result once to float32
(2^-24 of it).
"""
import numpy as np
import pytest

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R
from oracle import fbp_oracle as O

SIZES = [(1, 0, 1), (4, 0, 4), (8, 0, 8), (11, 0, 11), (13, 0, 13),
         (64, 0, 64), (105, 0, 105), (143, 0, 143), (110, 33, 176),
         (127, 0, 256), (1536, 0, 1536), (2304, 0, 2304), (1280, 150, 2880),
         (3600, 0, 3600), (3640, 0, 3640)]


def _close(got, ref, top):
    tol = 1.01 * 2.0 ** -24 * np.abs(ref) + 1e-12 * top
    assert (np.abs(got.astype(np.float64) - ref) <= tol).all()


@pytest.mark.gpu
@pytest.mark.parametrize("ncol,pad,t", SIZES)
def test_lengths(cuda, ncol, pad, t):
    import torch
    assert nat.load().atb_bpf_filter2d_length(ncol, pad) == t
    rng = np.random.default_rng(ncol + pad)
    x = rng.standard_normal((ncol, 3, ncol)).astype(np.float32)
    dev = torch.from_numpy(x).cuda()
    n = ncol + 2 * pad
    k = np.fft.fftfreq(n) * n
    sy, sx = min(2, n - 1), min(3, n - 1)
    win = np.fft.fftshift(np.exp(-2j * np.pi * (k[:, None] * sy
                                                + k[None, :] * sx) / n))
    for w, name in ((win, None), (None, "hann")):
        if w is None and ncol < 4:
            continue
        got = R._circular_filter(dev, w, name, pad, "edge").cpu().numpy()
        # one of a pair, and the last one alone
        for s in (0, 2) if ncol < 3000 else (2,):
            img = x[:, s].astype(np.float64)
            if w is None:
                ref = O.apply_circular_ramp_filter(img, None, name, pad,
                                                   "edge")
            else:
                ref = np.roll(np.pad(img, pad, mode="edge"), (sy, sx),
                              axis=(0, 1))[pad:pad + ncol, pad:pad + ncol]
            _close(got[:, s], ref, np.abs(img).max())
