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


def _gather(t, ang, cen, edge_pad=False):
    """``atb_backproject`` itself: no tensor cores, no angle groups."""
    nrow, nslice, ncol = t.shape
    out = torch.empty((ncol, nslice, ncol), device=t.device)
    nat.call("atb_backproject", t.data_ptr(), nat.F32, t.stride(0),
             t.stride(1), nrow, nslice, ncol,
             R._trig(ang, t.device).data_ptr(), float(np.float32(cen)),
             int(edge_pad), -1.0, 1.0, out.data_ptr(), out.stride(0),
             out.stride(1), 0, R._stream_ptr(t.device))
    return out


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
    assert nat.call("atb_backproject_stack_workspace", nat.F32, nrow, nslice,
                    ncol) > 0
    ang = np.linspace(0.0, np.pi, nrow)  # 0, 90 and 180 degrees among them
    _check(_stack(nrow, nslice, ncol, nrow), ang, cen, edge_pad, cuda)


def test_small_stacks_take_the_gather_kernel():
    def need(code, nslice):
        return nat.call("atb_backproject_stack_workspace", code, 181, nslice,
                        2560)
    assert need(nat.F32, 14) == need(nat.BF16, 32) == 0
    assert need(nat.F32, 15) > 0 and need(nat.F16, 15) > 0


def test_stack_of_16_bit_samples_with_mask_and_strides(cuda):
    dtype = torch.float16
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
    ref = _gather(t, ang, 31.2)
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


@pytest.mark.parametrize("edge_pad", [False, True])
@pytest.mark.parametrize("nrow,nslice,ncol", [
    (64, 1, 33), (65, 1, 100), (200, 1, 64), (97, 2, 65), (70, 3, 130),
    (131, 4, 40), (181, 7, 96), (300, 14, 50)])
def test_angle_groups_against_oracle(cuda, nrow, nslice, ncol, edge_pad):
    """Few tiles: the angles are split over CTAs, the groups' compensated
    totals are added in FP64 and rounded once (positions carry the gather
    kernel's 1e-5 bins, as without groups)."""
    assert nat.call("atb_backproject_stack_workspace", nat.F32, nrow, nslice,
                    ncol) > 0
    ang = np.linspace(0.0, np.pi, nrow)
    x = _stack(nrow, nslice, ncol, nrow)
    got = _check(x, ang, ncol / 2 - 1.3, edge_pad, cuda)
    one = _gather(torch.from_numpy(x).to(cuda), ang, ncol / 2 - 1.3,
                  edge_pad).cpu().numpy()
    assert O.rel_l2(got, one) < 3e-7


def test_tiles_outside_the_mask_are_zero(cuda):
    nrow, ncol = 90, 200
    ang = np.linspace(0.0, np.pi, nrow)
    d = np.arange(ncol) - ncol // 2
    for nslice in (1, 2, 5):
        x = _stack(nrow, nslice, ncol)
        t = torch.from_numpy(x).to(cuda)
        for r in (3.0, 60.0, 100.0):
            keep = d[None] ** 2 + d[:, None] ** 2 <= r * r
            for staging in ("tma", "cp.async"):
                out = torch.full((ncol, nslice, ncol), np.nan, device=cuda)
                R.backproject(t, ang, 99.0, mask_r2=r * r, out=out,
                              staging=staging)
                got = out.cpu().numpy()
                ref = O.back_projection(x[:, 0], ang, 99.0, False) * keep
                assert O.rel_l2(got[:, 0], ref) < TOL
                assert not np.any(got[:, nslice - 1][~keep])


@pytest.mark.parametrize("edge_pad", [0, 1])
@pytest.mark.parametrize("n,spacing,c0", [(15, 1, 140.25), (24, 2, 130.0),
                                          (33, 1, 150.5), (47, 3, 20.75),
                                          (20, 9, 1.0)])
def test_centre_groups_against_oracle(cuda, n, spacing, c0, edge_pad):
    """Groups of candidate centres: blocks inside every centre's detector on
    the tensor cores, the others on the gather kernel."""
    nrow, ncol = 41, 301
    ang = np.linspace(0.0, np.pi, nrow)
    x = _stack(nrow, 1, ncol)
    t = torch.from_numpy(x[:, 0]).to(cuda)
    need = nat.call("atb_backproject_centers_workspace", nrow, ncol, n)
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)
    out = torch.full((n, ncol, ncol), np.nan, device=cuda)
    nat.call("atb_backproject_centers_stack", t.data_ptr(), t.stride(0), nrow,
             ncol, R._trig(ang, cuda).data_ptr(), c0, spacing, n, edge_pad,
             -1.0, 1.0, out.data_ptr(), out.stride(1), out.stride(0), 0,
             ws.data_ptr(), need, R._stream_ptr(cuda))
    got = out.cpu().numpy()
    for m in (0, n // 2, n - 1):
        ref = O.back_projection(x[:, 0], ang, c0 + m * spacing, edge_pad)
        assert O.rel_l2(got[m], ref) < TOL, m
