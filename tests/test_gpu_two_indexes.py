"""Open indexes of one type searched from several threads at once: the kernels are shared by
the whole process, their shared-memory sizes are each index's own."""
import threading

import numpy as np
import pytest

from test_gpu_exact_shapes import _index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["exact", "wide"])
def test_threads_with_different_sizes(tmp_path, kernel):
    """Three small indexes' launches beside those of one whose visited bitmap of 75 KB lies in
    shared memory.  The device call returns before its kernel ends, so that launches of all
    indexes follow one another closely."""
    import torch
    from ngt_gb300 import Index
    from ngt_gb300.base import KERNEL_EXACT, KERNEL_WIDE
    kern = {"exact": KERNEL_EXACT, "wide": KERNEL_WIDE}[kernel]
    sizes = (600_000, 2000, 2000, 2000)
    paths = {n: str(tmp_path / str(n)) for n in set(sizes)}
    queries = {n: _index(p, n, 2, 8, n)[:1] for n, p in paths.items()}
    opened, rows, out, errors = [], [], [], []
    for n in sizes:
        ix = Index(paths[n], read_only=True)
        opened.append(ix)
        rows.append(torch.from_numpy(ix.convert_queries(queries[n])).cuda())
        out.append((torch.zeros((1, 5, 2), dtype=torch.int32, device="cuda"),
                    torch.zeros(1, dtype=torch.int32, device="cuda"),
                    torch.zeros((1, 5), dtype=torch.int32, device="cuda")))
    params, nparams = Index.make_params(5, 0.1)
    torch.cuda.synchronize()

    def work(t, rounds):
        try:
            r, c, s = out[t]
            for _ in range(rounds):
                opened[t].search_device(rows[t].data_ptr(), 1, params, nparams, r.data_ptr(), 5, c.data_ptr(),
                                        s.data_ptr(), kernel=kern)
        except Exception as e:          # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))

    for t in range(len(sizes)):         # alone: what each must return
        work(t, 1)
    torch.cuda.synchronize()
    alone = [[x.cpu().numpy() for x in o] for o in out]
    threads = [threading.Thread(target=work, args=(t, 1500)) for t in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for a, o in zip(alone, out):
        assert all(np.array_equal(x, y.cpu().numpy()) for x, y in zip(a, o))
    for ix in opened:
        ix.close()
    assert not errors, errors[:3]
