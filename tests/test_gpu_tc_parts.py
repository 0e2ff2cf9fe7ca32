"""Tensor-core exhaustive search: query tiles of 64 and 256, growing parts, and the second
pass after a candidate list overflowed, against the plain exhaustive search."""
import numpy as np
import pytest

from test_gpu_linear_select import _index

pytestmark = pytest.mark.gpu


def _plain(ix, q, k):
    r = [ix.linear_search(v, k=k) for v in q]
    return (np.array([[o.id for o in x] for x in r], np.uint32),
            np.array([[o.distance for o in x] for x in r], np.float32))


@pytest.mark.parametrize("dim", [3, 64, 65, 200])
@pytest.mark.parametrize("n", [100, 8193, 70_001])
def test_tile_widths_and_parts(tmp_path, n, dim):
    rng = np.random.default_rng(n + dim)
    x = rng.integers(0, 100, (n, dim)).astype(np.float32)       # whole numbers: bf16 scores are exact
    q = rng.integers(0, 100, (260, dim)).astype(np.float32)
    k = 10
    with _index(tmp_path, x) as ix:
        ids, ds, cnt, st = ix.linear_search_tc(q, k=k, candidates=64)
        assert (st == 0).all()
        pi, pd = _plain(ix, q[:20], k)
        assert np.array_equal(ids[:20], pi) and np.array_equal(ds[:20], pd)
        for nq in (1, 63, 64, 65, 256, 257):                    # one tile of 64, of 256, two
            for fp8 in ("bf16", "fp8"):
                a = ix.linear_search_tc(q[:nq], k=k, candidates=64 if fp8 == "bf16" else 2000 if n > 2000 else 64,
                                        precision=fp8)
                if fp8 == "bf16":
                    assert np.array_equal(a[0], ids[:nq]) and np.array_equal(a[1], ds[:nq]), nq
                elif nq <= 64:
                    b = ix.linear_search_tc(np.concatenate([q[:nq]] * 70)[:65 * nq], k=k, precision=fp8,
                                            candidates=2000 if n > 2000 else 64)
                    assert np.array_equal(a[0], b[0][:nq]) and np.array_equal(a[1], b[1][:nq]), nq
        s64, s256 = ix.tc_scores(q[:64]), ix.tc_scores(q)
        assert np.array_equal(s64, s256[:64])


def test_rows_sorted_by_nearness_are_searched_again(tmp_path):
    """Each doubling part opens with 5,000 rows nearer than all before: a list holds one
    part's, but not those of a part sixteen times the rows before it."""
    n = 150_000
    rng = np.random.default_rng(3)
    x = rng.integers(90, 100, (n, 4)).astype(np.float32)
    row, near = 8192 - 1, 80                                     # objects have ids from 1
    while row < n:
        x[row:row + 5000] = rng.integers(near - 10, near, (min(5000, n - row), 4))
        row, near = 2 * (row + 1) - 1, near - 15
    q = rng.integers(0, 3, (40, 4)).astype(np.float32)
    with _index(tmp_path, x) as ix:
        pi, pd = _plain(ix, q, 10)
        for graphs in (False, True):
            ix.set_tc_graphs(graphs)
            for _ in range(2):
                ids, ds, cnt, st = ix.linear_search_tc(q, k=10, candidates=64)
                assert (st == 0).all() and (cnt == 10).all()
                assert np.array_equal(ids, pi) and np.array_equal(ds, pd)


def test_a_part_beyond_the_list_still_reports_overflow(tmp_path):
    """Rows that come nearer one by one overflow any schedule: status bit 1, as before."""
    n = 120_000
    x = np.zeros((n, 2), np.float32)
    x[:, 0] = np.arange(n, 0, -1) // 2
    with _index(tmp_path, x) as ix:
        ids, ds, cnt, st = ix.linear_search_tc(np.zeros((3, 2), np.float32), k=10, candidates=64)
        assert (st & 1 != 0).all()


def test_an_overflow_in_a_replayed_capture_is_not_the_next_search_s(tmp_path):
    """A search inside a caller's capture cannot read its overflow word; a later search that
    overflows no list runs once, as it does on a fresh index."""
    import torch
    n = 120_000
    x = np.zeros((n, 2), np.float32)
    x[:, 0] = np.arange(n, 0, -1) // 2                           # comes nearer to 0, farther from n
    with _index(tmp_path, x) as ix:
        def buffers(v):
            rows = torch.from_numpy(ix.convert_queries(v)).cuda()
            return (rows, torch.zeros((3, 10, 2), dtype=torch.int32, device="cuda"),
                    torch.zeros(3, dtype=torch.int32, device="cuda"), torch.zeros(3, dtype=torch.int32, device="cuda"))

        def search(b, stream=None):
            ix._check(ix._lib.ngtgpu_linear_search_tc_ex(ix._index, b[0].data_ptr(), 3, 10, 64, 0, 0, b[1].data_ptr(),
                                                         10, b[2].data_ptr(), b[3].data_ptr(), stream, ix._err))

        near, far = buffers(np.zeros((3, 2), np.float32)), buffers(np.full((3, 2), n, np.float32))
        search(far)
        torch.cuda.synchronize()
        assert (far[3] == 0).all()
        first = ix.kernel_launches()
        search(far)
        once = ix.kernel_launches() - first
        want = far[1].clone()
        side = torch.cuda.Stream()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side, capture_error_mode="thread_local"):
            search(near, side.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        assert (near[3] & 1 != 0).all()
        before = ix.kernel_launches()
        search(far)
        torch.cuda.synchronize()
        assert ix.kernel_launches() - before == once
        assert (far[3] == 0).all() and torch.equal(far[1], want)


def test_sorted_rows_are_not_searched_twice_every_time(tmp_path):
    """Where fast-growing parts overflow, the next searches take doubling parts at once: 1 of
    them, then 2, 4 ..; a search whose lists hold ends that."""
    n = 150_000
    rng = np.random.default_rng(3)
    x = rng.integers(90, 100, (n, 4)).astype(np.float32)
    row, near = 8192 - 1, 80
    while row < n:
        x[row:row + 5000] = rng.integers(near - 10, near, (min(5000, n - row), 4))
        row, near = 2 * (row + 1) - 1, near - 15
    toward = rng.integers(0, 3, (40, 4)).astype(np.float32)      # nearer and nearer rows
    away = np.full((40, 4), 95, np.float32)                      # the first rows are the nearest
    for graphs in (False, True):
        with _index(tmp_path / str(graphs), x) as ix:
            pi, pd = _plain(ix, toward, 10)
            ix.set_tc_graphs(graphs)

            def launches(q):
                before = ix.kernel_launches()
                ids, ds, cnt, st = ix.linear_search_tc(q, k=10, candidates=64)
                assert (st == 0).all() and (cnt == 10).all()
                if q is toward:
                    assert np.array_equal(ids, pi) and np.array_equal(ds, pd)
                return ix.kernel_launches() - before

            launches(away)                                       # converts the rows too
            fast = launches(away)
            twice, once = launches(toward), launches(toward)
            assert fast < once and twice == fast + once
            assert [launches(toward) for _ in range(3)] == [twice, once, once]
            assert [launches(toward) for _ in range(5)] == [twice] + [once] * 4
            assert launches(away) == fast                        # a try that holds: all is as at first
            assert [launches(toward) for _ in range(2)] == [twice, once]
