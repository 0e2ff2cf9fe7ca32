"""The quantized-graph kernel's queue at its limits: a visited hash that moves to the global
bitmap (more than 1,024 neighbours within the exploration radius), a shared list of 256
keys refilled from the overflow tier, result sets of up to 1,023, and launches larger than
the grid, whose CTAs take their queries from a counter."""
import numpy as np
import pytest

import oracle
from golden_util import materialize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,eps,expansion", [(10, 1.0, 3.0), (100, 0.4, 5.0), (341, 0.1, 3.0), (50, -0.3, 5.0)])
def test_queue_limits_equal_oracle(tmp_path, k, eps, expansion):
    from ngt_gb300 import QuantizedIndex
    path, meta, queries, _ = materialize("qg_f32_l2_d32", str(tmp_path))
    o = oracle.Oracle(oracle.IndexFiles(path))
    q = queries[:60]
    oi, od, on, _ = o.qg_search(q, k=k, epsilon=eps, result_expansion=expansion, threads=8)
    with QuantizedIndex(path, zero_based_numbering=False) as ix:
        ids, ds, n, st = ix.batch_search(q, size=k, epsilon=eps, result_expansion=expansion, with_stats=True)
        many = ix.batch_search(np.concatenate([q] * 40), size=k, epsilon=eps, result_expansion=expansion)
    assert np.array_equal(n, on) and (st["status"] & 1 == 0).all()
    w = ids.shape[1]
    assert np.array_equal(ids, oi[:, :w]) and np.array_equal(ds, od[:, :w])
    if eps == 1.0:
        assert (st["status"] & 2 != 0).any()
    for j in range(40):
        assert np.array_equal(many[0][j * 60:(j + 1) * 60], ids) and np.array_equal(many[1][j * 60:(j + 1) * 60], ds)
