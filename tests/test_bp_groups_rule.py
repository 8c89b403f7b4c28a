"""Which launches of few tiles split their angles over CTAs: a group's partial
image is written and read whatever its angles, so few angles bear none."""
import pytest

from algotom_b200 import _native as nat


@pytest.mark.parametrize("nrow,nslice,ncol,split", [
    (181, 1, 256, True), (900, 1, 1024, True), (361, 1, 1024, True),
    (120, 1, 1024, False), (181, 1, 1390, False), (720, 1, 1390, False),
    (181, 1, 2560, False), (1801, 1, 2560, True), (120, 2, 256, True),
    (120, 2, 1024, False), (720, 2, 1024, True), (181, 2, 1536, False),
    (33, 4, 640, False), (181, 4, 800, True), (65, 4, 1024, False),
    (65, 8, 640, False), (720, 8, 640, True), (120, 12, 400, False),
    (720, 12, 400, True), (181, 4, 1024, False),
    (720, 14, 2560, False)])
def test_few_angles_are_not_split(nrow, nslice, ncol, split):
    need = nat.call("atb_backproject_stack_workspace", nat.F32, nrow, nslice,
                    ncol)
    assert (need > 0) == split
