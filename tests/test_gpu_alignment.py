"""Views that start off a 16-byte boundary: clustering reads them piece by piece, the compact packer (the one that takes them)
writes rows of 64-bit words wherever they lie."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _starting_at(x, elements):
    """``x`` in a buffer of its own, ``elements`` behind a 16-byte boundary."""
    buf = torch.zeros(x.numel() + elements, dtype=x.dtype, device=x.device)
    buf[elements:] = x.flatten()
    return buf[elements:].view(x.shape)


@pytest.mark.parametrize("value", [False, True])
@pytest.mark.parametrize("options", [{}, {"exact": True}, {"warp_mma": True}, {"count": 40}])
@pytest.mark.parametrize("b,h,t,offset", [(1, 1, 64, 1), (2, 3, 333, 4), (1, 2, 1030, 7)])
def test_clustering_of_a_misaligned_view(b, h, t, offset, options, value):
    from reskv_b200.compression import cluster
    from reskv_b200.synthetic import mixture

    x = mixture(b, h, t, seed=t, device=DEV)
    options = {"count": 32, "iterations": 3, "value": value, **options}
    got = cluster(_starting_at(x, offset), **options)
    # such input takes the integer sums, whose means are the correctly rounded ones: the same call on aligned rows
    want = cluster(x, **{**options, "exact": True, "warp_mma": False})
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_compressing_a_misaligned_prompt():
    from reskv_b200 import ResKVKernelConfig, compress
    from reskv_b200.synthetic import mixture

    k, v = (mixture(2, 2, 300, seed=i, device=DEV) for i in range(2))
    cfg = ResKVKernelConfig(bits=4, layout="compact", kmeans_iterations=2)
    got = compress(_starting_at(k, 1), _starting_at(v, 3), cfg)
    for side, x in ((got.key, k), (got.value, v)):
        given = ((side.centroids, side.cluster_ids),) * 2
        want = compress(x, x, cfg, clustering=given).key
        assert all(torch.equal(getattr(side, name), getattr(want, name)) for name in ("cluster_ids", "payload", "metadata", "scale"))


@pytest.mark.parametrize("bits,nnz", [(4, 32), (4, 64), (2, 64)])
def test_compact_bitmap_rows_on_eight_byte_boundaries(bits, nnz):
    from reskv_b200._extension import _stream, check, library, load_extension
    from reskv_b200.synthetic import gaussian, mixture

    x, cen = mixture(1, 2, 77, seed=1, device=DEV), gaussian(1, 2, 16, 128, seed=2, device=DEV)
    ids = torch.randint(16, (1, 2, 77), device=DEV, dtype=torch.int32)
    words, bitmap, scale = load_extension("compression").compress_compact(x, cen, ids, nnz, bits)
    buf = torch.zeros(bitmap.numel() + 1, dtype=torch.int64, device=DEV)
    words2, scale2 = torch.empty_like(words), torch.empty_like(scale)
    check(library().reskv_encode_compact(x.data_ptr(), cen.data_ptr(), ids.data_ptr(), 1, 2, 77, 77, 16, nnz, bits, words2.data_ptr(),
                                         buf[1:].data_ptr(), scale2.data_ptr(), 77, _stream(x.device)))
    assert torch.equal(buf[1:].view(bitmap.shape), bitmap) and torch.equal(words2, words) and torch.equal(scale2, scale)
