"""``atb_radon_adjoint`` reads nothing beside an image line.

Rays whose run of 32 lines ends exactly on the first or last pixel: the end of
the run, rounded as ``(xf + 31 r) - span``, is one pixel further in than as
``(xf - span) + 31 r``, so that bounds formed the one way do not hold a walk
formed the other.  The pixel beside the line carries next to no weight, so NaN
around the image shows a read of it.
"""
import numpy as np
import pytest
import torch

from algotom_b200 import _native as nat

NCOL = 288
# angle, centre, bin, first line of the run
CASES = [(0.7553517346258771, 142.6171879066859, 151, 252),
         (0.6972972450338121, 142.9911856614644, 186, 216),
         (0.6972972450338121, 143.10851924909855, 163, 252),
         (0.6616862921639072, 143.07806922120255, 170, 252),
         (0.6784457776456341, 142.7902247737047, 189, 216),
         (-0.43459620383329917, 143.33163676016486, 72, 252),
         (-0.3190045807988174, 142.74986978222145, 39, 216),
         (-0.3299277979919403, 143.17511563920868, 41, 216)]


@pytest.mark.parametrize("theta,center,d,line", CASES)
def test_cases_end_on_the_border(theta, center, d, line):
    """The two roundings differ there, and only one stays on the line."""
    f32, fma = np.float32, lambda j, r, x: np.float32(j * np.float64(r) +
                                                      np.float64(x))
    c, s = np.cos(-theta), np.sin(-theta)
    ic, r, span = 0.5 * (NCOL - 1), f32(-s / c), f32(abs(1.0 / c))
    x0 = line * (-s / c) + (d - center + ic * s) / c + ic
    xi, xf = int(np.floor(x0)), f32(x0 - np.floor(x0))
    one = xi + int(np.floor(f32(fma(31, r, xf) - span)))
    two = xi + int(np.floor(fma(31, r, f32(xf - span))))
    assert abs(one - two) == 1
    assert one + 1 >= 0 and one + 3 <= NCOL - 1
    assert two + 1 < 0 or two + 3 > NCOL - 1


@pytest.mark.gpu
@pytest.mark.parametrize("theta,center,d,line", CASES)
def test_nothing_beside_a_line_is_read(cuda, theta, center, d, line):
    wide = torch.zeros((NCOL + 2, 1, NCOL + 2), device=cuda)
    wide[1:-1, :, 1:-1] = torch.from_numpy(
        np.random.default_rng(3).uniform(0.1, 1.0, (NCOL, 1, NCOL))).to(cuda)
    trig = torch.tensor([[np.cos(-theta), np.sin(-theta)]],
                        dtype=torch.float64, device=cuda)
    need = nat.call("atb_radon_workspace", 1, NCOL)
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)
    got = []
    for fill in (0.0, np.nan):
        for edge in (wide[:1], wide[-1:], wide[..., :1], wide[..., -1:]):
            edge.fill_(fill)
        img = wide[1:-1, :, 1:-1]
        out = torch.empty((1, 1, NCOL), device=cuda)
        nat.call("atb_radon_adjoint", img.data_ptr(), img.stride(0),
                 img.stride(1), 1, 1, NCOL, trig.data_ptr(), center,
                 out.data_ptr(), out.stride(0), out.stride(1), ws.data_ptr(),
                 need, torch.cuda.current_stream(cuda).cuda_stream)
        got.append(out)
    assert bool(got[1].isfinite().all())
    assert torch.equal(*got)
