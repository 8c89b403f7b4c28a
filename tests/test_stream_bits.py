"""A stack streamed from the host has the bits of the device-resident one: the
streamed launches end at the same slices, whichever kernel takes them.  (Even
numbers of slices: the row filter transforms a projection's rows in pairs.)"""
import json

import numpy as np
import pytest
import torch

from algotom_b200.rec import reconstruction as R


@pytest.mark.parametrize("nrow,ncol,storage,kahan,joined", [
    (901, 1280, "float32", "chunk", True),    # tensor cores
    (901, 1280, "float16", "chunk", True),
    (181, 200, "bfloat16", "chunk", True),    # angle groups
    (1801, 2560, "bfloat16", "chunk", False),
    (901, 1280, "float32", "angle", False)])
@pytest.mark.parametrize("nslice", [1, 32, 70, 127, 128, 130, 257])
def test_groups_cover_the_spans(nslice, nrow, ncol, storage, kahan, joined):
    spans = R._slab_spans(nslice, 32)
    groups = R._slab_groups(spans, 32, nrow, ncol, storage, kahan)
    assert [sp for g in groups for sp in g] == spans
    sizes = [sum(n for _, n in g) for g in groups]
    full, left = divmod(nslice, 32)
    if joined:
        assert sizes == [32] * full + ([left] if left else [])
    else:
        assert all(len(g) == 1 for g in groups)


@pytest.mark.gpu
@pytest.mark.parametrize("nslice,nrow,ncol,storage,kahan", [
    (128, 101, 96, "float32", "chunk"), (138, 91, 200, "float32", "chunk"),
    (144, 100, 64, "float16", "chunk"), (134, 20, 170, "float32", "chunk"),
    (134, 181, 64, "bfloat16", "chunk"), (70, 181, 128, "bfloat16", "chunk"),
    (132, 61, 64, "float32", "angle"), (38, 2100, 48, "float32", "chunk")])
def test_streamed_bits_are_the_resident_ones(cuda, nslice, nrow, ncol,
                                             storage, kahan):
    x = np.random.default_rng(nslice).uniform(
        0.1, 1.0, (nrow, nslice, ncol)).astype(np.float32)
    ang, cen = np.linspace(0.0, np.pi, nrow), ncol / 2 - 1.3
    kw = dict(angles=ang, apply_log=False, storage=storage, kahan=kahan)
    got = R.fbp_reconstruction(x, cen, **kw)
    dev = R.fbp_reconstruction(torch.from_numpy(x).to(cuda), cen, **kw)
    assert np.array_equal(got, dev.cpu().numpy())


@pytest.mark.gpu
def test_a_half_finished_group_is_completed(cuda, tmp_path):
    nrow, nslice, ncol, cen = 64, 130, 64, 30.2
    x = np.random.default_rng(1).uniform(
        0.1, 1.0, (nrow, nslice, ncol)).astype(np.float32)
    out = np.full((ncol, nslice, ncol), np.nan, np.float32)
    man = str(tmp_path / "rec.json")
    kw = dict(angles=np.linspace(0.0, np.pi, nrow), apply_log=False, out=out,
              resume=man)
    R.fbp_reconstruction(x, cen, **kw)
    want = out.copy()
    d = json.load(open(man))
    assert sorted(map(tuple, d["done"])) == R._slab_spans(nslice, 32)
    d["done"] = [[0, 8], [32, 32], [128, 2]]
    json.dump(d, open(man, "w"))
    out[:, 8:32] = out[:, 64:128] = np.nan
    R.fbp_reconstruction(x, cen, **kw)
    assert np.array_equal(out, want)
    assert sorted(map(tuple, json.load(open(man))["done"])) == \
        R._slab_spans(nslice, 32)
