"""The flat-field / -log pre-step of vertical reconstructions in one launch for
several chunks: rows of four samples at a time and the general form, counters
per chunk.  The arithmetic is float32 with correctly rounded subtraction and
division; logf is within 1 ulp, so 3e-7 relative (plus 1e-7 absolute near
log 1) holds it."""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat
from algotom_b200.rec import reconstruction as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.uint16])
@pytest.mark.parametrize("field", [False, True])
@pytest.mark.parametrize("n,height,width,chunk", [
    (1, 1, 1, 1), (3, 2, 3, 2), (7, 3, 4, 3), (5, 9, 129, 5), (11, 4, 132, 4),
    (4, 2, 260, 30)])
def test_chunks_against_numpy(cuda, n, height, width, chunk, field, dtype):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 900, (n, height, width)).astype(dtype)
    dark = flat = None
    if field:
        dark = rng.integers(0, 20, (height, width)).astype(np.float32)
        flat = rng.integers(500, 900, (height, width)).astype(np.float32)
    v = x.astype(np.float32)
    v = (v - dark) / flat if field else v
    bad = v <= 0
    want = -np.log(np.where(bad, np.float32(1), v).astype(np.float64))
    counts = [int(bad[a:a + chunk].sum()) for a in range(0, n, chunk)]
    for shift in (0, 1):  # an odd base takes the general form
        code = nat.F32 if dtype == np.float32 else nat.U16
        raw = torch.zeros(x.size + shift, dtype=torch.float32 if dtype ==
                          np.float32 else torch.uint16, device=cuda)
        raw[shift:] = torch.from_numpy(x.ravel()).to(cuda)
        src = raw[shift:].view(n, height, width)
        out = torch.empty((n, height, width), device=cuda)
        non = torch.zeros(len(counts), dtype=torch.int32, device=cuda)
        d = [torch.from_numpy(f).to(cuda) if field else None
             for f in (dark, flat)]
        nat.call("atb_flat_log_chunks", src.data_ptr(), code, src.stride(0),
                 src.stride(1), n, height, width, chunk,
                 *(t.data_ptr() if field else None for t in d), width, 1,
                 out.data_ptr(), out.stride(0), out.stride(1),
                 non.data_ptr(), R._stream_ptr(cuda))
        assert non.tolist() == counts
        assert np.allclose(out.cpu().numpy(), want, rtol=3e-7, atol=1e-7)
