"""The CTA-per-query kernel's row batches at their edges: a step of m new rows, m around
multiples of a batch (threads / lanes of a row x rows in flight), for one to 32 lanes a row
and for 8-bit codes by dot products, 8-bit codes in floats and bf16 rows.  Every node links
to all others, so that one step sees every row; whole-number data, so that the result is the
sorted list of exact distances (by distance, then id)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [3, 24, 60, 128, 130, 257])
@pytest.mark.parametrize("m", [1, 2, 33, 127, 128, 129, 256, 300, 1023, 1025])
def test_steps_of_m_rows(tmp_path, dim, m):
    from ngt_gb300 import Index
    from ngt_gb300.base import KERNEL_WIDE
    from ngt_gb300.graph_build import write_index
    rng = np.random.default_rng(dim * 7 + m)
    n = m + 1
    x = rng.integers(0, 17, (n, dim)).astype(np.float32)
    to = (np.arange(n)[:, None] + np.arange(1, n)) % n + 1
    path = str(tmp_path / "ix")
    write_index(path, x, np.concatenate([[0, 0], np.cumsum(np.full(n, m))]).astype(np.int64),
                to.reshape(-1).astype(np.uint32), np.zeros(n * m, np.float32))
    q = rng.integers(0, 17, (40, dim)).astype(np.float32)
    half = q + 0.5                                   # exact in 8-bit steps of 1/256
    k = min(n, 20)
    with Index(path, read_only=True) as ix:
        for v, rows in ((q, 2), (half, 2), (q, 1)):
            d = ((x[None].astype(np.float64) - v[:, None, :]) ** 2).sum(2)
            order = np.lexsort((np.broadcast_to(np.arange(n), d.shape), d), axis=1)[:, :k]
            for threads in (64, 128, 256, 0):
                ix.set_batched_tuning(list_capacity=64, parents=1, neighbour_capacity=2048, cta_threads=threads,
                                      search_rows=rows)
                ids, ds, cnt = ix.batch_search(v, k=k, epsilon=10.0, edge_size=m, kernel=KERNEL_WIDE)
                assert (cnt == k).all()
                assert np.array_equal(ids, order + 1), (threads, rows)
                assert np.allclose(ds, np.sqrt(np.take_along_axis(d, order, 1)), rtol=1e-6)
