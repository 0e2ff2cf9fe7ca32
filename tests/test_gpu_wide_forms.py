"""The CTA-per-query kernel's forms give the same results: threads per query chosen by the
number of queries (512 up to one per SM, on large indexes two; 256; 128 from six per SM),
the visited bitmap in shared or global memory, 8-bit rows scored by integer dot products or
in floats."""
import numpy as np
import pytest

from golden_util import materialize
from test_gpu_exact_shapes import _index

pytestmark = pytest.mark.gpu


def _wide(ix, q, k, eps, **tuning):
    from ngt_gb300.base import KERNEL_WIDE
    ix.set_batched_tuning(**tuning)
    ids, ds, n, st = ix.batch_search(q, k=k, epsilon=eps, kernel=KERNEL_WIDE, with_stats=True)
    return ids, ds, n, st["distance_computations"]


# 262,143 slots: a 32 KB bitmap, the last size of one query per SM; 262,200: two per SM
@pytest.mark.parametrize("n", [2000, 262_142, 262_200])
def test_threads_by_number_of_queries(tmp_path, n):
    from ngt_gb300 import Index
    path = str(tmp_path / "ix")
    q = np.concatenate([_index(path, n, 20, 16, n)] * 3)[:915]
    with Index(path, read_only=True) as ix:
        ref = _wide(ix, q, 10, 0.2, cta_threads=64, search_rows=1)
        for rows in (1, 2):
            for nq in (1, 152, 153, 304, 305, 911, 912):
                got = _wide(ix, q[:nq], 10, 0.2, search_rows=rows)
                for a, b in zip(ref, got):
                    assert np.array_equal(a[:nq], b), (rows, nq)


@pytest.mark.parametrize("name", ["f32_cosine", "f32_l1", "u8_l2", "u8_hamming", "u8_jaccard", "f16_l2", "qs8_l2",
                                  "f32_poincare", "f32_lorentz"])
def test_other_distances(tmp_path, name):
    from ngt_gb300 import Index
    path, meta, queries, _ = materialize(name, str(tmp_path))
    q = np.concatenate([queries] * 8)[:320]
    with Index(path, read_only=True) as ix:
        ref = _wide(ix, q, 10, 0.1, cta_threads=256)
        for nq in (1, 152, 320):
            got = _wide(ix, q[:nq], 10, 0.1)
            for a, b in zip(ref, got):
                assert np.array_equal(a[:nq], b), nq


# The dot products hold squared distances below 2^24: 256 dimensions of differences of 255
# reach 16,646,400; 257 dimensions are scored in floats.
@pytest.mark.parametrize("dim", [1, 15, 17, 128, 256, 257, 600])
def test_integer_dot_products(tmp_path, dim):
    from ngt_gb300 import Index
    from ngt_gb300.graph_build import write_index
    rng = np.random.default_rng(dim)
    n = 3000
    x = rng.choice([0.0, 1.0, 128.0, 254.0, 255.0], (n, dim)).astype(np.float32)
    x[0], x[1] = 0.0, 255.0
    to = np.concatenate([(np.arange(n)[:, None] + np.arange(1, 9)) % n, rng.integers(0, n, (n, 8))], 1)
    path = str(tmp_path / "ix")
    write_index(path, x, np.concatenate([[0, 0], np.cumsum(np.full(n, 16))]).astype(np.int64),
                (to + 1).reshape(-1).astype(np.uint32), np.zeros(n * 16, np.float32))
    q = rng.choice([0.0, 255.0, 3.0], (60, dim)).astype(np.float32)
    q[0], q[1] = 0.0, 255.0
    mixed = q.copy()
    mixed[::2, 0] += 0.5                     # every other query in floats
    mixed[1::4, 0] = 300.0                   # or out of the codes' range
    with Index(path, read_only=True) as ix:
        assert ix.wide_search_rows() == "u8"
        for v in (q, mixed):
            a, b = _wide(ix, v, 10, 0.3, search_rows=2), _wide(ix, v, 10, 0.3, search_rows=1)
            whole = (v == np.rint(v)).all(1) & (dim <= 257)       # bf16 sums are exact for these
            whole &= (v <= 255).all(1)
            for r, s in zip(a, b):
                assert np.array_equal(r[whole], s[whole])
            d = np.sqrt(((x[a[0].astype(np.int64) - 1].astype(np.float64) - v[:, None, :]) ** 2).sum(2))
            assert np.allclose(a[1], d, rtol=1e-6)
        one = _wide(ix, q, 10, 0.3, search_rows=2)
        for j in (1, 3):                     # a query's form does not depend on the others'
            alone = _wide(ix, q[j:j + 1], 10, 0.3, search_rows=2)
            assert np.array_equal(alone[0][0], one[0][j]) and np.array_equal(alone[1][0], one[1][j])


# The rule's other line: 128 threads only while a step has at most 1,024 neighbour slots (10
# parents, or as many slots as the caller sets).
@pytest.mark.parametrize("tuning", [dict(parents=10), dict(parents=11), dict(parents=16), dict(parents=17),
                                    dict(parents=16, neighbour_capacity=1024),
                                    dict(parents=4, neighbour_capacity=2048)])
def test_threads_by_neighbour_slots(tmp_path, tuning):
    from ngt_gb300 import Index
    path = str(tmp_path / "ix")
    q = np.concatenate([_index(path, 5000, 20, 40, 3)] * 3)[:920]
    with Index(path, read_only=True) as ix:
        for rows in (1, 2):
            got = _wide(ix, q, 10, 0.2, search_rows=rows, **tuning)
            for threads in (128, 256):
                ref = _wide(ix, q, 10, 0.2, search_rows=rows, cta_threads=threads, **tuning)
                for a, b in zip(ref, got):
                    assert np.array_equal(a, b), (rows, threads)
