"""The tensor-core back-projector at sizes where the gather kernel is the faster
(flags bit 6 of the stack entry points takes it there all the same): few angles
and small images, the edges of its tiles, angle chunks and slice groups; and the
rule that leaves such calls to the gather kernel.

Tolerance as in test_bp_stack.py: 1e-6 relative L2 holds the roundings of
positions (2^-21 bins) and samples (2^-22) and the truncation of up to 16
additions at 2^-24 each.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R
from oracle import fbp_oracle as O

pytestmark = pytest.mark.gpu
TOL, FORCE = 1e-6, 64


def _stack(nrow, nslice, ncol):
    rng = np.random.default_rng(nrow)
    x = rng.uniform(0.1, 1.0, (nrow, nslice, ncol)).astype(np.float32)
    return x * 10.0 ** rng.integers(-3, 4, (1, nslice, 1)).astype(np.float32)


def _bp(name, t, ang, cen, edge_pad, flags=0):
    nrow, nslice, ncol = t.shape
    out = torch.full((ncol, nslice, ncol), np.nan, device=t.device)
    args = ()
    if name == "atb_backproject_stack":
        need = nat.call(name + "_workspace", nat.F32, nrow, nslice, ncol)
        ws = torch.empty(max(1, need), dtype=torch.uint8, device=t.device)
        args = (ws.data_ptr(), need)
    nat.call(name, t.data_ptr(), nat.F32, t.stride(0), t.stride(1), nrow,
             nslice, ncol, R._trig(ang, t.device).data_ptr(), cen,
             int(edge_pad), -1.0, 1.0, out.data_ptr(), out.stride(0),
             out.stride(1), flags, *args, R._stream_ptr(t.device))
    return out


def _centres(name, t, ang, c0, spacing, n, edge_pad, flags=0):
    nrow, ncol = t.shape
    out = torch.full((n, ncol, ncol), np.nan, device=t.device)
    args = ()
    if name == "atb_backproject_centers_stack":
        need = nat.call("atb_backproject_centers_workspace", nrow, ncol, n)
        ws = torch.empty(need, dtype=torch.uint8, device=t.device)
        args = (ws.data_ptr(), need)
    nat.call(name, t.data_ptr(), t.stride(0), nrow, ncol,
             R._trig(ang, t.device).data_ptr(), c0, spacing, n, edge_pad,
             -1.0, 1.0, out.data_ptr(), out.stride(1), out.stride(0), flags,
             *args, R._stream_ptr(t.device))
    return out


@pytest.mark.parametrize("edge_pad", [False, True])
@pytest.mark.parametrize("nrow,nslice,ncol,cen", [
    (1, 15, 16, 7.5), (3, 16, 8, 3.0), (4, 17, 15, 9.25), (7, 24, 17, 0.0),
    (8, 25, 31, 30.0), (9, 31, 33, 16.0), (16, 32, 48, 20.75),
    (17, 33, 40, 19.5), (33, 47, 65, 33.25), (40, 64, 170, 12.125),
    (5, 16, 1, 0.0), (6, 16, 2, 0.5), (7, 17, 3, 1.0), (9, 15, 5, 2.25)])
def test_forced_stack_against_oracle(cuda, nrow, nslice, ncol, cen, edge_pad):
    ang = np.linspace(0.0, np.pi, nrow)
    x = _stack(nrow, nslice, ncol)
    t = torch.from_numpy(x).to(cuda)
    got = _bp("atb_backproject_stack", t, ang, cen, edge_pad, FORCE)
    assert nat.call("atb_backproject_status", 0) == 0
    for k in sorted({0, nslice // 2, nslice - 1}):
        ref = O.back_projection(x[:, k], ang, cen, edge_pad)
        assert O.rel_l2(got[:, k].cpu().numpy(), ref) < TOL, k


@pytest.mark.parametrize("edge_pad", [0, 1])
@pytest.mark.parametrize("n,spacing,c0", [(15, 1, 140.25), (24, 2, 130.0),
                                          (33, 1, 150.5), (47, 3, 20.75),
                                          (20, 9, 1.0)])
def test_forced_centres_against_oracle(cuda, n, spacing, c0, edge_pad):
    nrow, ncol = 41, 301
    ang = np.linspace(0.0, np.pi, nrow)
    x = _stack(nrow, 1, ncol)[:, 0]
    got = _centres("atb_backproject_centers_stack",
                   torch.from_numpy(x).to(cuda), ang, c0, spacing, n,
                   edge_pad, FORCE).cpu().numpy()
    for m in (0, n // 2, n - 1):
        ref = O.back_projection(x, ang, c0 + m * spacing, bool(edge_pad))
        assert O.rel_l2(got[m], ref) < TOL, m


@pytest.mark.parametrize("nrow,nslice,ncol,tensor", [
    (63, 16, 100, 0), (64, 16, 100, 16), (47, 32, 161, 0), (48, 32, 161, 32),
    (56, 24, 161, 24), (71, 21, 200, 0), (72, 21, 200, 21), (119, 18, 200, 0),
    (120, 18, 200, 18), (65, 16, 320, 0), (66, 16, 320, 16),
    (34, 15, 512, 0), (35, 15, 512, 15), (55, 24, 161, 0),
    (63, 17, 160, 0), (64, 17, 160, 17), (50, 47, 1000, 32)])
def test_groups_with_few_angles_take_the_gather_kernel(cuda, nrow, nslice,
                                                       ncol, tensor):
    """The first ``tensor`` slices run on the tensor cores, whose bits do not
    depend on the group, the others are ``atb_backproject``'s."""
    ang, cen = np.linspace(0.0, np.pi, nrow), ncol / 2 - 1.25
    t = torch.from_numpy(_stack(nrow, nslice, ncol)).to(cuda)
    got = _bp("atb_backproject_stack", t, ang, cen, False)
    forced = _bp("atb_backproject_stack", t, ang, cen, False, FORCE)
    assert torch.equal(got[:, :tensor], forced[:, :tensor])
    rest = t[:, tensor:].contiguous()
    if nslice > tensor:
        gather = _bp("atb_backproject", rest, ang, cen, False)
        assert torch.equal(got[:, tensor:], gather)


def test_without_tensor_maps_the_gather_kernel_runs(cuda):
    """(bit 7: the driver's encoder is not there)"""
    nrow, nslice, ncol = 90, 32, 100
    ang = np.linspace(0.0, np.pi, nrow)
    t = torch.from_numpy(_stack(nrow, nslice, ncol)).to(cuda)
    got = _bp("atb_backproject_stack", t, ang, 48.75, True, 128)
    assert torch.equal(got, _bp("atb_backproject", t, ang, 48.75, True))


@pytest.mark.parametrize("nrow,ncol,n,c0,tensor", [
    (400, 96, 16, 40.5, 0), (23, 96, 15, 40.5, 0), (24, 96, 15, 40.5, 15),
    (127, 400, 20, 190.5, 0), (128, 400, 20, 190.5, 20),
    (128, 400, 20, 30.5, 0), (255, 640, 16, 310.5, 0)])
def test_centre_groups_that_stay_on_the_gather_kernel(cuda, nrow, ncol, n, c0,
                                                      tensor):
    ang = np.linspace(0.0, np.pi, nrow)
    t = torch.from_numpy(_stack(nrow, 1, ncol)[:, 0].copy()).to(cuda)
    got = _centres("atb_backproject_centers_stack", t, ang, c0, 1, n, 0)
    want = _centres("atb_backproject_centers_stack", t, ang, c0, 1, n, 0,
                    FORCE) if tensor else \
        _centres("atb_backproject_centers", t, ang, c0, 1, n, 0)
    assert torch.equal(got, want)
