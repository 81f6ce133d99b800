"""PageRank's set-up and its last-block finish: stored zeroes (out-degrees are
counted, not the row lengths), hub rows, dangling rows, a given initial guess,
on the single kernel and on the per-step launches, against the restatement.

Both stop at an L1 change of 1e-9 and contract by 0.85 per iteration, so one
iteration more or less moves pr by at most 1e-9 / 0.15 in all; rounding of the
column sums (at most 1e5 terms) stays far below that."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zeros", [0.0, 0.3])
@pytest.mark.parametrize("given", [0, 1])
@pytest.mark.parametrize("n,edges", [(300, 900), (5000, 60000), (40000, 1300000)])
def test_setup_and_finish(cuda, oracle, n, edges, zeros, given):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    rng = np.random.default_rng([n, given, int(10 * zeros)])
    key = np.unique((rng.integers(0, n, edges) * rng.random(edges) ** 2).astype(np.int64) * n +
                    (rng.integers(0, n, edges) * rng.random(edges) ** 3).astype(np.int64))
    I, J = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    V = (rng.random(len(key)) >= zeros).astype(np.float64)
    rp, col, vals = oracle.coo_to_crs(n, I, J, V, abi.FP64)
    cp, row, tv = oracle.coo_to_crs(n, J, I, V, abi.FP64)
    L, LT = dev.from_host(n, n, rp, col, vals), dev.from_host(n, n, cp, row, tv)
    pr0 = rng.random(n)
    pr0 /= pr0.sum()
    pr = torch.from_numpy(pr0.copy()).cuda()
    it, res = C.c_int64(), C.c_double()
    abi.call("alpb_pagerank", n, *L.p(), *LT.p(), dev.ptr(pr), given, 0.85, 1e-9, 1000,
             C.byref(it), C.byref(res), dev.stream_ptr())
    rc, want, it2, _ = oracle.pagerank(rp, col, vals, cp, row, tv, pr0=pr0 if given else None)
    assert rc == 0 and abs(it.value - it2) <= 1
    assert np.abs(pr.cpu().numpy() - want).sum() <= 1e-9 / 0.15
