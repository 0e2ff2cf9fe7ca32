"""Selection stage of the exhaustive search (linear_select.cuh) against a stable sort:
ties at the k-th distance by id, sizes at the edges of its blocks and digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(tmp_path, x):
    from ngt_gb300 import Index
    from ngt_gb300.graph_build import write_index
    n = len(x)
    ring = np.concatenate([np.arange(2, n + 1), [1]]).astype(np.uint32)
    offsets = np.concatenate([[0, 0], np.arange(1, n + 1)]).astype(np.int64)
    path = str(tmp_path / "ix")
    write_index(path, x, offsets, ring, np.zeros(n, np.float32), extra_prf={"EdgeSizeForSearch": "10"})
    return Index(path, read_only=True)


# 1,023 ids need one id digit and 1,025 two; a selection block takes 4,096 rows; 40,001 rows
# take ten blocks.  Values 0..1 over 3 dimensions: 4 distances in all, so nearly every cut
# falls among ties.  All sums are small whole numbers: the distances are exact.
@pytest.mark.parametrize("n,dim,top,ks", [
    (2, 3, 1, (1, 2)),
    (1023, 3, 1, (1, 100, 1022, 1023)),
    (1025, 3, 1, (1, 1024, 2000)),
    (4095, 20, 3, (10, 4095)),
    (4097, 129, 255, (7, 4096)),
    (40001, 3, 1, (1, 33, 5000, 12288)),
    (40001, 520, 255, (20,)),
])
def test_selection_equals_a_stable_sort(tmp_path, n, dim, top, ks):
    rng = np.random.default_rng(n + dim)
    x = rng.integers(0, top + 1, (n, dim)).astype(np.float32)
    q = rng.integers(0, top + 1, (3, dim)).astype(np.float32)
    with _index(tmp_path, x) as ix:
        for k in ks:
            for v in q:
                d = np.sqrt(((x - v) ** 2).sum(1, dtype=np.float64)).astype(np.float32)
                order = np.argsort(d, kind="stable")[:k]
                got = ix.linear_search(v, k=k)
                assert [r.id for r in got] == (order + 1).tolist()
                assert np.array_equal(np.array([r.distance for r in got], np.float32), d[order])


def test_selection_leaves_out_what_is_not_finite(tmp_path):
    """Objects at a distance of +inf or NaN are no results, whatever k."""
    x = np.zeros((300, 4), np.float32)
    x[:, 0] = np.arange(300) % 7
    x[5, 1] = np.inf
    x[9, 2] = np.nan
    with _index(tmp_path, x) as ix:
        for k in (10, 300):
            got = ix.linear_search(np.zeros(4, np.float32), k=k)
            d = np.where(np.isfinite(x).all(1), x[:, 0], np.inf)
            order = [i for i in np.argsort(d, kind="stable") if np.isfinite(d[i])][:k]
            assert [r.id for r in got] == [i + 1 for i in order]


def test_many_queries_over_a_small_index(tmp_path):
    """The autotuner's ground truth is the exhaustive search of all its sample queries: 65,000
    over 100 objects run in several blocks, whose buffers stay within the engine's limits (64 MB
    here and 64 MB of its memory pool) however many queries there are."""
    import torch
    from ngt_gb300 import Index
    from test_gpu_exact_shapes import _index as random_index
    path = str(tmp_path / "ix")
    random_index(path, 100, 128, 60, 4, bytes_=True)
    q = np.random.default_rng(5).integers(0, 60, (65_000, 128)).astype(np.float32)
    with Index(path, read_only=True) as ix:
        # the search kernels' own buffers: as large as they get
        ix.autotune(q[:6000], k=99, epsilon=0.5, recall_floor=1.0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ix.autotune(q, k=99, epsilon=0.6, recall_floor=1.0)
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= 160 << 20
