"""K and V clustered in the same launches against one call each, at the edges of the 128-token tiles and of the share of a
CTA, with token slices of longer buffers; given ids of every integer width."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("iterations", [1, 4])
@pytest.mark.parametrize("b,h,t,count", [(1, 1, 32, 32), (1, 2, 127, 8), (2, 3, 129, 32), (1, 1, 8193, 20), (5, 8, 700, 32), (3, 8, 4500, 1)])
def test_pair_equals_single_calls(b, h, t, count, iterations):
    from reskv_b200._extension import load_extension
    from reskv_b200.compression import cluster
    from reskv_b200.synthetic import mixture

    bufs = [torch.full((b, h, t + 70, 128), float("nan"), dtype=torch.float16, device=DEV) for _ in range(2)]
    sides = []
    for i, buf in enumerate(bufs):
        buf[:, :, 7 : 7 + t] = mixture(b, h, t, seed=10 + i, device=DEV)
        sides.append(buf[:, :, 7 : 7 + t])
    pair = load_extension("compression").kmeans_pair(*sides, count, iterations)
    for value, (x, (centres, ids, ids8)) in enumerate(zip(sides, pair)):
        want_c, want_i = cluster(x.contiguous(), count, iterations, value=bool(value))
        assert torch.equal(ids8.int(), ids)
        if iterations == 1:  # the first assignment is exact
            assert torch.equal(ids, want_i)
        moved = (ids != want_i).sum().item()
        assert moved <= 1e-3 * ids.numel()  # FP32 sums of another order: tokens between two centres
        if moved == 0:  # the last sums are of the same pieces
            assert torch.equal(centres, want_c)


@pytest.mark.parametrize("dtype", [torch.int8, torch.int16, torch.int32, torch.int64])
def test_given_ids_of_every_width(dtype):
    from reskv_b200 import ResKVKernelConfig, compress
    from reskv_b200.synthetic import gaussian

    b, h, t, count = 1, 2, 333, 9
    x = gaussian(b, h, t, 128, seed=1, device=DEV)
    cen = gaussian(b, h, count, 128, seed=2, device=DEV)
    ids = torch.randint(count, (b, h, t), generator=torch.Generator().manual_seed(3)).to(DEV)
    want = compress(x, x, ResKVKernelConfig(), clustering=((cen, ids.int()), (cen, ids.int())))
    got = compress(x, x, ResKVKernelConfig(), clustering=((cen, ids.to(dtype)), (cen, ids.transpose(1, 2).contiguous().transpose(1, 2).to(dtype))))
    for a, w in ((got.key, want.key), (got.value, want.value)):
        assert torch.equal(a.cluster_ids, w.cluster_ids) and torch.equal(a.payload, w.payload)
    for bad in (-1, count):
        wrong = ids.clone()
        wrong[0, 1, -1] = bad
        with pytest.raises(ValueError, match="out of range"):
            compress(x, x, ResKVKernelConfig(), clustering=((cen, ids), (cen, wrong.to(dtype))))
