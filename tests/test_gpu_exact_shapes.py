"""The exact-order graph kernel where its forms meet: 512 threads per query up to one CTA
per SM (152 on this chip), 128 above; the visited set as a bitmap or a hash in shared
memory; rows of every lane-group width.  Results and counters against the oracle on random
graphs; coordinates are whole numbers, so the distances are exact."""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _index(path, n, dim, degree, seed, bytes_=False):
    from ngt_gb300.graph_build import write_index
    rng = np.random.default_rng(seed)
    x = rng.integers(0, 60, (n, dim)).astype(np.float32)
    # neighbours near in id and far ones; ascending by distance as an index has them
    near = (np.arange(n)[:, None] + rng.integers(1, 20, (n, degree // 2))) % n
    to = np.concatenate([near, rng.integers(0, n, (n, degree - degree // 2))], 1)
    d = np.sqrt(sum((x[:, None, c] - x[to, c]) ** 2 for c in range(dim)))
    order = np.argsort(d, axis=1, kind="stable")
    to, d = np.take_along_axis(to, order, 1), np.take_along_axis(d, order, 1)
    offsets = np.concatenate([[0, 0], np.cumsum(np.full(n, degree))]).astype(np.int64)
    write_index(path, x, offsets, (to + 1).reshape(-1).astype(np.uint32), d.reshape(-1).astype(np.float32))
    if bytes_:
        prf = open(os.path.join(path, "prf")).read().replace("ObjectType\tFloat-4", "ObjectType\tInteger-1")
        open(os.path.join(path, "prf"), "w").write(prf)
        rec = np.empty((n, 1 + dim), np.uint8)
        rec[:, 0] = ord("+")
        rec[:, 1:] = x
        with open(os.path.join(path, "obj"), "wb") as f:
            f.write(np.uint64(n + 1).tobytes() + b"-" + rec.tobytes())
    return rng.integers(0, 60, (310, dim)).astype(np.float32)


def _same(path, q, nqs, k, eps, mode="read_only"):
    from ngt_gb300 import Index
    o = oracle.Oracle(oracle.IndexFiles(path))
    oi, od, on, dc = o.search(q, k=k, epsilon=eps, mode=mode, threads=8)
    with Index(path, read_only=mode == "read_only") as ix:
        for nq in nqs:
            ids, ds, n, st = ix.batch_search(q[:nq], k=k, epsilon=eps, with_stats=True)
            assert np.array_equal(n, on[:nq])
            assert np.array_equal(st["distance_computations"], dc[:nq])
            assert (st["status"] & 1 == 0).all()
            for j in range(nq):
                assert np.array_equal(ids[j, :n[j]], oi[j, :n[j]]), (nq, j)
                assert np.array_equal(ds[j, :n[j]], od[j, :n[j]]), (nq, j)


# the 128-thread kernel's visited bitmap in shared memory holds 262,144 ids (with id 0)
@pytest.mark.parametrize("n", [300, 262_143, 262_144])
def test_batch_sizes_and_visited_sets(tmp_path, n):
    path = str(tmp_path / "ix")
    q = _index(path, n, 4, 12, n)
    _same(path, q, (1, 152, 153, 310), 10, 0.4)


@pytest.mark.parametrize("dim,bytes_", [(10, True), (20, True), (40, True), (70, True), (3, False), (20, False),
                                        (70, False), (129, False), (600, False)])
def test_row_widths(tmp_path, dim, bytes_):
    path = str(tmp_path / "ix")
    q = _index(path, 2000, dim, 40, dim, bytes_)
    for mode in ("read_only", "updatable"):
        _same(path, q, (7, 310), 30, 0.1, mode)


def test_long_edge_lists_and_refills(tmp_path):
    """300 edges a node: several rounds per expansion, in either kernel; epsilon wide enough
    that the overflow tier refills the shared list many times."""
    path = str(tmp_path / "ix")
    q = _index(path, 20_000, 8, 300, 5)
    from ngt_gb300 import Index
    o = oracle.Oracle(oracle.IndexFiles(path))
    oi, od, on, dc = o.search(q[:160], k=50, epsilon=0.6, edge_size=0, threads=8)
    with Index(path, read_only=True) as ix:
        for nq in (5, 160):
            ids, ds, n, st = ix.batch_search(q[:nq], k=50, epsilon=0.6, edge_size=0, with_stats=True)
            assert np.array_equal(ids, oi[:nq, :50]) and np.array_equal(ds, od[:nq, :50])
            assert np.array_equal(st["distance_computations"], dc[:nq])


def test_large_index_without_a_shared_bitmap(tmp_path):
    """1.9M objects: the 512-thread kernel falls back to its hash and the global bitmap."""
    from ngt_gb300 import Index
    path = str(tmp_path / "ix")
    q = _index(path, 1_900_000, 2, 8, 9)
    with Index(path, read_only=True) as ix:
        a = ix.batch_search(q, k=10, epsilon=0.3, with_stats=True)
        b = ix.batch_search(q[:20], k=10, epsilon=0.3, with_stats=True)
    assert np.array_equal(a[0][:20], b[0]) and np.array_equal(a[1][:20], b[1])
    assert np.array_equal(a[3]["distance_computations"][:20], b[3]["distance_computations"])


# The result set's merge: sets that fill slowly (k beyond a node's neighbours), ties at the
# last result everywhere (coordinates 0..2), a search radius that is reached at once.
@pytest.mark.parametrize("mode", ["read_only", "updatable"])
@pytest.mark.parametrize("k", [1, 2, 15, 130, 400])
def test_result_sets_with_ties(tmp_path, k, mode):
    path = str(tmp_path / "ix")
    _index(path, 3000, 6, 24, 77)
    x = np.random.default_rng(1).integers(0, 3, (3000, 6)).astype(np.float32)
    rec = np.empty((3000, 25), np.uint8)
    rec[:, 0] = ord("+")
    rec[:, 1:] = x.view(np.uint8).reshape(3000, -1)
    with open(os.path.join(path, "obj"), "wb") as f:      # other coordinates over the same graph
        f.write(np.uint64(3001).tobytes() + b"-" + rec.tobytes())
    q = np.random.default_rng(2).integers(0, 3, (160, 6)).astype(np.float32)
    for eps in (0.0, 0.5):
        _same(path, q, (9, 160), k, eps, mode)
    from ngt_gb300 import Index
    o = oracle.Oracle(oracle.IndexFiles(path))
    oi, od, on, dc = o.search(q, k=k, epsilon=0.2, radius=1.5, mode=mode, threads=8)
    with Index(path, read_only=mode == "read_only") as ix:
        ids, ds, n = ix.batch_search(q, k=k, epsilon=0.2, radius=1.5)
    assert np.array_equal(n, on)
    for j in range(len(q)):
        assert np.array_equal(ids[j, :n[j]], oi[j, :n[j]]) and np.array_equal(ds[j, :n[j]], od[j, :n[j]])


# Distances below zero (int8 codes under the inner product: whole numbers of either sign,
# exact in a float), where the updates of the result set are replayed one by one.  With size 1
# and a radius a read-only search may hold one negative result and a round of neighbours none
# of which is negative.
@pytest.mark.parametrize("mode", ["read_only", "updatable"])
@pytest.mark.parametrize("k", [1, 2, 30])
def test_negative_distances(tmp_path, k, mode):
    from ngt_gb300 import Index
    path = str(tmp_path / "ix")
    n, dim = 2000, 15                                     # 16 elements a row with the inner product's own
    _index(path, n, dim, 24, 11)
    prf = open(os.path.join(path, "prf")).read()
    for old, new in (("ObjectType\tFloat-4", "ObjectType\tQSUInteger-8B"), ("DistanceType\tL2",
                     "DistanceType\tInnerProduct\nMaxMagnitude\t1\nQuantizationOffset\t0\nQuantizationScale\t127.5")):
        prf = prf.replace(old, new)
    open(os.path.join(path, "prf"), "w").write(prf)
    rng = np.random.default_rng(12)
    rec = np.empty((n, 2 + dim), np.uint8)
    rec[:, 0] = ord("+")
    rec[:, 1:] = rng.integers(0, 256, (n, dim + 1))       # 127 * 127 * 16 - sum of products: of either sign
    with open(os.path.join(path, "obj"), "wb") as f:
        f.write(np.uint64(n + 1).tobytes() + b"-" + rec.tobytes())
    q = (rng.integers(75, 128, (160, 1)) - rng.integers(0, 50, (160, dim))).astype(np.float32)
    o = oracle.Oracle(oracle.IndexFiles(path))
    signs = set()
    with Index(path, read_only=mode == "read_only") as ix:
        for eps in (-0.2, 0.0, 0.3, 4.0):
            for radius in (-1.0, 0.0, 20000.0):
                oi, od, on, dc = o.search(q, k=k, epsilon=eps, radius=radius, mode=mode, threads=8)
                for nq in (9, 160):                       # 512 and 128 threads a query
                    ids, ds, c, st = ix.batch_search(q[:nq], k=k, epsilon=eps, radius=radius, with_stats=True)
                    assert np.array_equal(c, on[:nq]), (eps, radius, nq)
                    assert np.array_equal(st["distance_computations"], dc[:nq]), (eps, radius, nq)
                    for j in range(nq):
                        assert np.array_equal(ids[j, :c[j]], oi[j, :c[j]]), (eps, radius, nq, j)
                        assert np.array_equal(ds[j, :c[j]], od[j, :c[j]]), (eps, radius, nq, j)
                        signs.update(np.sign(ds[j, :c[j]]).tolist())
    assert -1.0 in signs and 1.0 in signs


# Result sets that leave no room for a visited bitmap in shared memory: the hash takes its
# place, then smaller ones, then (one query an SM) 128 threads instead of 512.  26,981 is what
# 232,448 bytes held beside a row of four chunks, 256 keys of the list twice, a round's keys
# and a hash of 2,048 words.
@pytest.mark.parametrize("n", [30_000, 200_000, 262_143])
def test_largest_result_sizes(tmp_path, n):
    import ctypes

    import torch
    from ngt_gb300 import Index
    from ngt_gb300.base import QUERY_STATS_DTYPE
    from test_zz_no_alloc import _noalloc
    path = str(tmp_path / "ix")
    q = _index(path, n, 4, 12, n)[:153]
    files = oracle.IndexFiles(path)
    for k in (23_900, 26_981):
        oi, od, on, dc = oracle.Oracle(files).search(q[:12], k=k, epsilon=0.0, threads=8)
        with Index(path, read_only=True) as ix:
            for nq in (1, 153):
                ids, ds, c, st = ix.batch_search(q[:nq], k=k, epsilon=0.0, with_stats=True)
                for j in range(min(nq, 12)):
                    assert c[j] == on[j] and st["distance_computations"][j] == dc[j]
                    assert np.array_equal(ids[j, :c[j]], oi[j, :c[j]]) and np.array_equal(ds[j, :c[j]], od[j, :c[j]])
            rows = torch.from_numpy(ix.convert_queries(q[:12])).cuda()
            params, nparams = ix.make_params(k, 0.0)
            r = torch.zeros((12, k, 2), dtype=torch.int32, device="cuda")
            c = torch.zeros(12, dtype=torch.int32, device="cuda")
            st = torch.zeros((12, QUERY_STATS_DTYPE.itemsize // 4), dtype=torch.int32, device="cuda")
            ix._check(_noalloc(ix._lib)(ix._index, rows.data_ptr(), 12, ctypes.cast(params, ctypes.c_void_p), nparams,
                                        r.data_ptr(), k, c.data_ptr(), st.data_ptr(), None, ix._err))
            torch.cuda.synchronize()
            c, r = c.cpu().numpy(), r.cpu().numpy()
            for j in range(12):
                assert c[j] == on[j] and np.array_equal(r[j, :c[j], 0].view(np.uint32), oi[j, :c[j]])
