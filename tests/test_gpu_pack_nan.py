"""Tiled packers with NaN and infinite residuals: a NaN comes behind every number of its 16-coordinate tile, each tile keeps its
fixed count all the same, and the other tiles are what they are without it."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("structured,nnz", [(True, 32), (False, 64), (False, 32)])
@pytest.mark.parametrize("nans", [1, 2, 5, 8, 11, 13, 16])
def test_tiles_with_nans_keep_their_count_and_their_neighbours(structured, nnz, nans):
    from oracle.encode import encode_tiled_fp16
    from reskv_b200._extension import load_extension

    rng = np.random.default_rng(100 * nnz + nans)
    t, count = 131, 3
    x = rng.standard_normal((1, 2, t, 128)).astype(np.float16)
    x[:, 1] = np.round(x[:, 1])  # many equal keys
    cen = np.zeros((1, 2, count, 128), np.float16)
    ids = rng.integers(0, count, (1, 2, t)).astype(np.int32)
    for h in range(2):
        for token in range(t):
            tile = token % 8
            where = 16 * tile + rng.permutation(16)
            x[0, h, token, where[:nans]] = np.nan
            if token % 3 == 0 and nans < 15:
                x[0, h, token, where[nans]] = -np.inf
    want, want_meta = encode_tiled_fp16(x, cen, ids, nnz, structured)
    gpu = [torch.from_numpy(a).to(DEV) for a in (x, cen, ids)]
    values, meta = (a.cpu().numpy() for a in load_extension("compression").compress_fp16(*gpu, nnz, structured))
    assert np.array_equal(meta, want_meta)
    assert np.array_equal(np.isnan(values), np.isnan(want))
    numbers = ~np.isnan(want)
    assert np.array_equal(values.view(np.uint16)[numbers], want.view(np.uint16)[numbers])
