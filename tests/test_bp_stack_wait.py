"""The tensor-core back-projector's bounded waits, made to run out on purpose.

``atb_backproject_stack`` flags bit 5 (tests only) arms the first CTA's first
copies for 16 bytes more than they deliver: every copy completes, nothing is
withheld, and the waits for them run out after their second.  The CTA then
requests nothing more (a ring slot short of bytes must not be armed again) and
walks to its end (bit 6: whatever the angles); the call returns, the status word says so, only that region of
16 x 16 pixels is missing, and the next call is right.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrow,nslice,edge_pad", [
    (5, 16, 0),     # one chunk of angles: nothing is in flight behind it
    (64, 24, 1),    # the ring fills while the waits run
    (200, 32, 0)])  # staging waits for a free ring slot too
def test_wait_runs_out_and_is_reported(cuda, nrow, nslice, edge_pad):
    ncol = 80
    s3 = torch.from_numpy(np.random.default_rng(5).standard_normal(
        (nrow, nslice, ncol)).astype(np.float32)).to(cuda)
    trig = R._trig(np.linspace(0, np.pi, nrow, endpoint=False), cuda)
    need = nat.call("atb_backproject_stack_workspace", nat.F32, nrow, nslice,
                    ncol)
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)

    def launch(flags):
        out = torch.full((ncol, nslice, ncol), np.nan, device=cuda)
        nat.call("atb_backproject_stack", s3.data_ptr(), nat.F32,
                 s3.stride(0), s3.stride(1), nrow, nslice, ncol,
                 trig.data_ptr(), 39.25, edge_pad, -1.0, 1.0, out.data_ptr(),
                 out.stride(0), out.stride(1), flags | 64, ws.data_ptr(), need,
                 R._stream_ptr(cuda))
        torch.cuda.synchronize()
        return out

    nat.call("atb_backproject_status", 1)  # start clean
    ref = launch(0)
    assert nat.call("atb_backproject_status", 0) == 0
    assert bool(ref.isfinite().all())
    out = launch(1 << 5)
    assert nat.call("atb_backproject_status", 1) == 1  # read and reset
    region = torch.zeros((ncol, nslice, ncol), dtype=torch.bool, device=cuda)
    region[:16, :, :16] = True
    assert bool(out[region].isnan().all())
    assert torch.equal(out[~region], ref[~region])
    assert torch.equal(launch(0), ref)
    assert nat.call("atb_backproject_status", 0) == 0
