"""The tensor-core back-projector of slice stacks (``atb_backproject_stack``)
against the FP64 oracle, at the edges of its tiles (8 x 8 pixels in regions of
16 x 16), angle chunks (4, 8 and 16) and slice groups (16, 24, 32).

Tolerance: positions are rounded to 2^-21 bins and samples to 2^-22, and the
tensor cores truncate up to 16 additions at 2^-24 each, 8 2^-24 = 4.8e-7 of a
sum on average in the worst case; with samples of one sign nothing cancels, so
1e-6 relative L2 holds them all.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R
from oracle import fbp_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _stack(nrow, nslice, ncol, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.1, 1.0, (nrow, nslice, ncol)).astype(np.float32)
    return x * 10.0 ** rng.integers(-3, 4, (1, nslice, 1)).astype(np.float32)


def _check(x, ang, cen, edge_pad, cuda, **kw):
    got = R.backproject(torch.from_numpy(x).to(cuda), ang, cen,
                        edge_pad=edge_pad, **kw).cpu().numpy()
    assert nat.call("atb_backproject_status", 0) == 0
    for k in sorted({0, x.shape[1] // 2, x.shape[1] - 1}):
        ref = O.back_projection(x[:, k], ang, cen, edge_pad)
        assert O.rel_l2(got[:, k], ref) < TOL, k
    return got


@pytest.mark.parametrize("edge_pad", [False, True])
@pytest.mark.parametrize("nrow,nslice,ncol,cen", [
    (1, 15, 16, 7.5), (3, 16, 8, 3.0), (4, 17, 15, 9.25), (7, 24, 17, 0.0),
    (8, 25, 31, 30.0), (9, 31, 33, 16.0), (16, 32, 48, 20.7),
    (17, 33, 40, 19.5), (33, 47, 65, 33.3), (40, 64, 100, 12.1)])
def test_stack_against_oracle(cuda, nrow, nslice, ncol, cen, edge_pad):
    assert nat.call("atb_backproject_stack_workspace", nrow, nslice, ncol) > 0
    ang = np.linspace(0.0, np.pi, nrow)  # 0, 90 and 180 degrees among them
    _check(_stack(nrow, nslice, ncol, nrow), ang, cen, edge_pad, cuda)


def test_small_stacks_take_the_gather_kernel():
    assert nat.call("atb_backproject_stack_workspace", 181, 14, 256) == 0
    assert nat.call("atb_backproject_stack_workspace", 181, 15, 256) > 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_stack_of_16_bit_samples_with_mask_and_strides(cuda, dtype):
    nrow, nslice, ncol = 21, 18, 50
    x = torch.from_numpy(_stack(nrow, nslice, ncol)).clamp(1e-3, 1e3)
    wide = torch.zeros((nslice, nrow, ncol + 3), dtype=dtype, device=cuda)
    wide[:, :, 1:ncol + 1] = x.transpose(0, 1).to(cuda, dtype)
    view = wide.transpose(0, 1)[:, :, 1:ncol + 1]
    ang = np.linspace(0.0, np.pi, nrow)
    r2 = 20.0 ** 2
    got = R.backproject(view, ang, 24.2, mask_r2=r2, scale=0.5).cpu().numpy()
    d = np.arange(ncol) - ncol // 2
    keep = (d[None] ** 2 + d[:, None] ** 2 <= r2)
    host = view.float().cpu().numpy()
    for k in (0, nslice - 1):
        ref = 0.5 * keep * O.back_projection(host[:, k], ang, 24.2, False)
        assert O.rel_l2(got[:, k], ref) < TOL
        assert not np.any(got[:, k][~keep])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_samples_reach_only_their_pixels(cuda, bad):
    nrow, nslice, ncol = 24, 20, 64
    x = _stack(nrow, nslice, ncol)
    x[11, 3, 30] = bad
    ang = np.linspace(0.0, np.pi, nrow)
    t = torch.from_numpy(x).to(cuda)
    got = R.backproject(t, ang, 31.2)
    ref = R.backproject(t, ang, 31.2, staging="cp.async")
    assert torch.equal(got.isnan(), ref.isnan())
    assert torch.equal(got.isinf(), ref.isinf())
    assert bool(got[:, 4].isfinite().all()) and not bool(
        got[:, 3].isfinite().all())


def test_same_bits_twice_and_under_capture(cuda):
    nrow, nslice, ncol = 40, 32, 96
    t = torch.from_numpy(_stack(nrow, nslice, ncol)).to(cuda)
    ang = np.linspace(0.0, np.pi, nrow)
    a = R.backproject(t, ang, 47.0)
    out = torch.empty_like(a)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        R.backproject(t, ang, 47.0, out=out)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, out)
