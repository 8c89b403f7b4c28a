"""Error of the tensor-core back-projector against FP64, beside the gather
kernel's on the same stack, where angles are many for the image (the gather
kernel's position errors average out over the angles, truncated sums do not).

Both errors are root mean squares over thousands of pixels with independent
roundings, known to a few per cent, so 10 % more than the gather's is allowed.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200 import phantom
from algotom_b200.rec import reconstruction as R
from oracle import cpu_port

pytestmark = pytest.mark.gpu


def _filtered(nrow, nslice, ncol, cen, cuda):
    s = np.stack([phantom.ellipse_sinogram(40 + k, nrow, ncol, cen,
                                           photons=1e4)[0]
                  for k in range(3)], axis=1)
    s = s[:, np.arange(nslice) % 3]
    return R.filter_sinograms(torch.from_numpy(s).to(cuda), ncol // 7)


def _both(f, ang, cen):
    got = R.backproject(f, ang, cen)
    ref = torch.empty_like(got)
    nrow, nslice, ncol = f.shape
    nat.call("atb_backproject", f.data_ptr(), nat.F32, f.stride(0),
             f.stride(1), nrow, nslice, ncol,
             R._trig(ang, f.device).data_ptr(), float(np.float32(cen)), 0,
             -1.0, 1.0, ref.data_ptr(), ref.stride(0), ref.stride(1), 0,
             R._stream_ptr(f.device))
    return got, ref


@pytest.mark.parametrize("nrow,nslice,ncol", [
    (361, 16, 128), (901, 16, 64), (901, 24, 200), (1201, 32, 160),
    (1801, 16, 96), (1801, 15, 320), (901, 16, 512)])
def test_no_further_off_than_the_gather_kernel(cuda, nrow, nslice, ncol):
    cen, ang = ncol / 2 - 1.2, np.linspace(0.0, np.pi, nrow)
    f = _filtered(nrow, nslice, ncol, cen, cuda)
    got, ref = _both(f, ang, cen)
    assert not torch.equal(got, ref)  # two kernels
    err = np.zeros(2)
    for k in range(3):
        exact = cpu_port.back_projection(f[:, k].cpu().numpy(), ang, cen,
                                         ref_arith=False)
        for n, img in enumerate((got, ref)):
            d = img[:, k].cpu().numpy().astype(np.float64) - exact
            err[n] += np.sum(d * d)
    assert err[0] ** 0.5 <= 1.1 * err[1] ** 0.5


@pytest.mark.parametrize("nrow,ncol", [(4001, 64), (8193, 48)])
def test_very_many_angles_take_the_gather_kernel(cuda, nrow, ncol):
    cen, ang = ncol / 2 - 1.2, np.linspace(0.0, np.pi, nrow)
    f = _filtered(nrow, 16, ncol, cen, cuda)
    got, ref = _both(f, ang, cen)
    # (angle groups, which few tiles take, change the last bit only)
    assert float((got - ref).abs().max()) <= 2e-7 * float(ref.abs().max())
