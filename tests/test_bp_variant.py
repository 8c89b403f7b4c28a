"""``backproject(variant=...)`` is ``atb_backproject`` with that tile variant, and
the angle groups on the samples and tiles that the rule takes them to."""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R
from oracle import cpu_port
from oracle import fbp_oracle as O

pytestmark = pytest.mark.gpu


def _plain(t, ang, cen, flags):
    nrow, nslice, ncol = t.shape
    out = torch.empty((ncol, nslice, ncol), device=t.device)
    nat.call("atb_backproject", t.data_ptr(), R._CODES[t.dtype], t.stride(0),
             t.stride(1), nrow, nslice, ncol,
             R._trig(ang, t.device).data_ptr(), float(np.float32(cen)), 0,
             -1.0, 1.0, out.data_ptr(), out.stride(0), out.stride(1), flags,
             R._stream_ptr(t.device))
    return out


def _samples(nrow, nslice, ncol, cuda, dtype=torch.float32):
    x = np.random.default_rng(ncol).uniform(0.1, 1.0, (nrow, nslice, ncol))
    return torch.from_numpy(x.astype(np.float32)).to(cuda, dtype)


@pytest.mark.parametrize("nslice", [1, 3, 7, 16])
@pytest.mark.parametrize("variant", [0, 1])
def test_variant_is_taken(cuda, variant, nslice):
    nrow, ncol, cen = 200, 130, 63.4
    ang = np.linspace(0.0, np.pi, nrow)
    t = _samples(nrow, nslice, ncol, cuda)
    for staging, flag in (("tma", 0), ("cp.async", 16)):
        got = R.backproject(t, ang, cen, variant=variant, staging=staging)
        want = _plain(t, ang, cen, variant << 2 | flag)
        assert torch.equal(got, want)
    assert not torch.equal(R.backproject(t, ang, cen), got)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("nrow,nslice,ncol", [(200, 1, 64), (97, 2, 65),
                                              (181, 7, 96)])
def test_groups_of_16_bit_samples(cuda, dtype, nrow, nslice, ncol):
    """As without groups but for the FP32 sums' grouping: the 3e-7 of
    test_bp_stack.py's float32 groups."""
    assert R._stack_need(R._CODES[dtype], nrow, nslice, ncol) > 0
    ang = np.linspace(0.0, np.pi, nrow)
    t = _samples(nrow, nslice, ncol, cuda, dtype)
    got = R.backproject(t, ang, 30.7).cpu().numpy()
    assert O.rel_l2(got, _plain(t, ang, 30.7, 0).cpu().numpy()) < 3e-7


@pytest.mark.parametrize("nrow,ncol", [(310, 1400), (330, 1411)])
def test_groups_of_large_tiles_against_fp64(cuda, nrow, ncol):
    """Single slices of 1400 pixels and more split their 64 x 64 tiles' angles;
    tolerance of the gather kernel's other tests."""
    assert R._stack_need(nat.F32, nrow, 1, ncol) > 0
    ang, cen = np.linspace(0.0, np.pi, nrow), ncol / 2 - 3.3
    t = _samples(nrow, 1, ncol, cuda)
    got = R.backproject(t, ang, cen)[:, 0].cpu().numpy()
    ref = cpu_port.back_projection(t[:, 0].cpu().numpy(), ang, cen,
                                   ref_arith=False)
    assert O.rel_l2(got, ref) < 1e-6
