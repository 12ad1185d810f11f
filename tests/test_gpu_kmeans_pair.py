"""K and V clustered in the same launches: bit for bit what one call each gives, at the edges of the 128-token tiles, of the
pieces and of the share of a CTA, with token slices of longer buffers; given ids of every integer width."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("iterations", [1, 4])
@pytest.mark.parametrize("b,h,t,count", [(1, 1, 32, 32), (1, 2, 127, 8), (2, 3, 129, 32), (1, 1, 8193, 20), (5, 8, 700, 32), (3, 8, 4500, 1),
                                       (1, 8, 1152, 32), (16, 8, 3000, 32), (32, 8, 2050, 32), (5, 4, 17000, 32)])
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
        assert torch.equal(ids, want_i) and torch.equal(centres, want_c)


@pytest.mark.parametrize("b,t", [(1, 300), (3, 4870), (8, 8128)])
def test_compress_equals_compress_with_its_own_clustering(b, t):
    from reskv_b200 import ResKVKernelConfig, compress
    from reskv_b200.compression import cluster

    def between_centres(seed):
        """Few distinct values and a little noise: the last bits of a centre decide where many tokens go."""
        gen = torch.Generator(device=DEV).manual_seed(seed)
        steps = torch.randint(-1, 2, (b, 8, t, 128), device=DEV, generator=gen)
        return (0.37 * steps + 0.001 * torch.randn(b, 8, t, 128, device=DEV, generator=gen)).half()

    key, value = between_centres(1), between_centres(2)
    cfg = ResKVKernelConfig(sparsity=0.75, layout="unstructured")
    n, iterations = cfg.num_clusters, cfg.kmeans_iterations
    want = compress(key, value, cfg, clustering=(cluster(key, n, iterations), cluster(value, n, iterations, value=True)))
    got = compress(key, value, cfg)
    for a, w in ((got.key, want.key), (got.value, want.value)):
        for name in ("centroids", "cluster_ids", "payload", "metadata"):
            assert torch.equal(getattr(a, name), getattr(w, name))


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
