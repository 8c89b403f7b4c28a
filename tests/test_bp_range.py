"""Stacks whose slices hold samples of very different sizes: the tensor cores'
two float16 terms hold a sample relative to its slice's largest, so slices with
an outlier (or a faint band) have to give ``atb_backproject``'s results.

Tolerance off the outlier's rays, pixel by pixel: samples of 0.1 to 1 have slopes
up to 0.9 per bin and positions carry up to 3e-5 bins, 2.7e-5 of a sample; the
mean is 0.55, so 5e-5 relative.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R
from oracle import fbp_oracle as O

pytestmark = pytest.mark.gpu
NROW, NCOL, CEN = 101, 97, 47.3
ANG = np.linspace(0.0, np.pi, NROW)


def _stack(nslice, seed=0):
    return np.random.default_rng(seed).uniform(
        0.1, 1.0, (NROW, nslice, NCOL)).astype(np.float32)


def _gather(t, edge_pad):
    out = torch.empty((NCOL, t.shape[1], NCOL), device=t.device)
    nat.call("atb_backproject", t.data_ptr(), R._CODES[t.dtype], t.stride(0),
             t.stride(1), NROW, t.shape[1], NCOL,
             R._trig(ANG, t.device).data_ptr(), float(np.float32(CEN)),
             int(edge_pad), -1.0, 1.0, out.data_ptr(), out.stride(0),
             out.stride(1), 0, R._stream_ptr(t.device))
    return out


def _same(a, b):
    """The same bits (3e38 overflows to NaN in both, where it is read)."""
    return torch.equal(a.contiguous().view(torch.int32),
                       b.contiguous().view(torch.int32))


@pytest.mark.parametrize("edge_pad", [False, True])
@pytest.mark.parametrize("nslice", [15, 33])
@pytest.mark.parametrize("big", [1e6, -1e9, 3e38])
def test_outlier_reaches_only_its_pixels(cuda, nslice, edge_pad, big):
    x = _stack(nslice)
    x[20, 7, 40] = big
    t = torch.from_numpy(x).to(cuda)
    got = R.back_projection_gpu_chunk(t, ANG, CEN, edge_pad=edge_pad)
    assert _same(got[:, :15], _gather(t, edge_pad)[:, :15])
    ref = O.back_projection(np.where(x == np.float32(big), 0, x)[:, 7], ANG,
                            CEN, edge_pad)
    one = np.zeros((NROW, NCOL), np.float32)
    one[20, 40] = 1.0
    off = O.back_projection(one, ANG, CEN, edge_pad) == 0.0
    g = got[:, 7].cpu().numpy()
    assert off.sum() > 0.9 * off.size
    live = off & (ref > 0.0)
    assert np.max(np.abs(g - ref)[live] / ref[live]) < 5e-5


@pytest.mark.parametrize("lo,hi", [(0, 97), (30, 33), (31, 33)])
def test_faint_samples_keep_their_bits(cuda, lo, hi):
    """A slice, or a band of its bins, 1e-9 of the largest sample."""
    x = _stack(16, 1)
    x[:, 3, lo:hi] *= 1e-9
    x[40, 3, 96] = 1.0
    t = torch.from_numpy(x).to(cuda)
    assert torch.equal(R.backproject(t, ANG, CEN), _gather(t, False))


def test_ordinary_stacks_stay_on_the_tensor_cores(cuda):
    """Zeros, isolated faint samples and float16's own range change nothing."""
    x = _stack(16, 2)
    x[:, 2, 20:50] = 0.0
    x[::2, 4, 60] = 1e-9
    t = torch.from_numpy(x).to(cuda)
    got = R.backproject(t, ANG, CEN)
    assert not torch.equal(got, _gather(t, False))
    for k in (2, 4, 15):
        assert O.rel_l2(got[:, k].cpu().numpy(),
                        O.back_projection(x[:, k], ANG, CEN, False)) < 1e-6


@pytest.mark.parametrize("big", [1e6, 3e38])
@pytest.mark.parametrize("n", [16, 47])
def test_outlier_in_a_centre_search(cuda, n, big):
    x = _stack(1, 3)[:, 0]
    x[20, 40] = big
    t = torch.from_numpy(np.ascontiguousarray(x)).to(cuda)
    trig = R._trig(ANG, cuda)
    need = nat.call("atb_backproject_centers_workspace", NROW, NCOL, n)
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)
    out = [torch.full((n, NCOL, NCOL), np.nan, device=cuda) for _ in range(2)]
    for o, name, extra in ((out[0], "atb_backproject_centers_stack",
                            (ws.data_ptr(), need)),
                           (out[1], "atb_backproject_centers", ())):
        nat.call(name, t.data_ptr(), t.stride(0), NROW, NCOL, trig.data_ptr(),
                 25.25, 1, n, 1, -1.0, 1.0, o.data_ptr(), o.stride(1),
                 o.stride(0), 0, *extra, R._stream_ptr(cuda))
    # (atb_backproject_centers takes the last three of 47 in other tiles)
    assert _same(out[0][:44], out[1][:44])
    if n > 44:
        off = out[1][44:].abs() < 1e3
        diff = (out[0][44:] - out[1][44:])[off].abs()
        assert bool(diff.max() < 5e-5 * 35)
