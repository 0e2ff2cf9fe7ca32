"""The two-step QBG search's blob phase at the edges of its batches: 63 to 65 and more
probed blobs, result sets on both sides of the batch selection's limit (224) and of its
shared memory rule (1,024), blobs larger than a batch's distances, and ties across the
end of the result set, where the blobs' order decides.  Ids, distances, counts and judged
blobs equal the oracle's."""
import os

import numpy as np
import pytest

import oracle
from golden_util import materialize

pytestmark = pytest.mark.gpu


def _check(path, queries, k, expansion, blobs, refine):
    from ngt_gb300 import QBGIndex
    o = oracle.Oracle(oracle.IndexFiles(os.path.join(path, "global")))
    oi, od, on, ob = o.qbg_search(queries, path, k=k, epsilon=0.1, blob_epsilon=0.0, result_expansion=expansion,
                                  explored_blobs=blobs, threads=8, two_step=True,
                                  **({"refinement_expansion": expansion} if refine else {}))
    with QBGIndex(path) as ix:
        ids, ds, n, st = ix.batch_search(queries, k=k, epsilon=0.1, blob_epsilon=0.0, result_expansion=expansion,
                                         explored_blobs=blobs, with_stats=True, two_step=True, refine=refine)
    assert np.array_equal(n, on)
    w = ids.shape[1]
    assert np.array_equal(ids, oi[:, :w])
    assert np.array_equal(ds.view(np.uint32), od[:, :w].view(np.uint32))
    assert np.array_equal(st["visited"], ob)
    assert (st["status"] == 0).all()


@pytest.mark.parametrize("k,expansion,blobs", [(1, 1.0, 1), (1, 1.0, 64), (2, 1.0, 65), (10, 10.0, 63),
                                               (100, 2.24, 64), (100, 2.25, 64), (512, 2.0, 200), (600, 2.0, 64)])
def test_scan_batches_equal_oracle(k, expansion, blobs, tmp_path):
    path, _, queries, _ = materialize("qbg_u8_l2_d64", str(tmp_path))
    _check(path, queries, k, expansion, blobs, refine=True)


@pytest.fixture(scope="module")
def repeated(tmp_path_factory):
    """14,000 equal rows, 60 further rows repeated 50 times each and 3,000 single ones: a blob
    beyond a batch's distances, and ties of every kind; subvectors of 1, 2 and 4 elements."""
    from ngt_gb300.qbg_build import build_qbg
    rng = np.random.default_rng(17)
    x = np.concatenate([np.repeat(rng.integers(0, 40, (1, 32)), 14000, 0),
                        np.repeat(rng.integers(0, 40, (60, 32)), 50, 0),
                        rng.integers(0, 40, (3000, 32))]).astype(np.uint8)
    rng.shuffle(x)
    out = {}
    for dsv in (1, 2, 4):
        out[dsv] = str(tmp_path_factory.mktemp("qbg%d" % dsv))
        build_qbg(out[dsv], x, nblobs=160, nsid=6, dsv=dsv, iters=3, log=lambda *a: None)
    near = x[rng.integers(0, len(x), 150)].astype(np.float32)
    return out, np.concatenate([near, rng.integers(0, 40, (150, 32)).astype(np.float32)])


@pytest.mark.parametrize("dsv", [1, 2, 4])
@pytest.mark.parametrize("k,expansion,blobs", [(1, 1.0, 100), (3, 1.0, 64), (10, 3.0, 100), (10, 10.0, 64),
                                               (200, 3.0, 120)])
def test_scan_ties_and_large_blobs_equal_oracle(dsv, k, expansion, blobs, repeated):
    paths, queries = repeated
    _check(paths[dsv], queries, k, expansion, blobs, refine=False)
