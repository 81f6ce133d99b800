"""The row-streaming product of short regular rows: chunk edges, the last
chunk's ragged copy, every value size, arrays that start off a 16-byte boundary
(another kernel) and rows of 1 to 64 nonzeroes, against the restatement.

FP64: rows of at most 64 terms in another order, each order off by at most
64 * 2^-53 of the sum of magnitudes; values are positive, so 2e-14 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [2, 1])
@pytest.mark.parametrize("ring", [0, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("maxlen,m", [(1, 5), (3, 31), (5, 33), (5, 5000), (8, 64), (9, 16),
                                      (27, 17), (27, 20001), (33, 1000), (64, 300)])
def test_rowstream(cuda, oracle, maxlen, m, ring, form):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    from oracle.oracle import NP
    rng = np.random.default_rng([maxlen, m, ring])
    n = m + 70
    lens = np.full(m, maxlen)
    if m > 20:      # a few shorter rows keep the profile regular
        lens[rng.integers(0, m, m // 10)] = maxlen // 2
        lens[rng.integers(0, m, m // 30)] = 0
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.uint32)
    vtype = abi.RING_TYPE[ring]
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 3, k)).astype(NP[vtype])  # noqa: E731
    vals, u, v = value(len(col)), value(m), value(n)
    for pattern in (False, True):
        want = u.copy()
        assert oracle.mxv(ring, 0, form, m, n, rp, col, None if pattern else vals,
                          abi.VOID if pattern else vtype, want, v=v)[0] == 0
        for shift in (0, 1):
            A = dev.from_host(m, n, rp, col, None if pattern else vals,
                              abi.VOID if pattern else vtype)
            keep = torch.empty(len(col) + 1, dtype=torch.int32, device="cuda")
            keep[shift:shift + len(col)] = A.indices
            A.indices = keep[shift:shift + len(col)]
            plan = dev.Plan(A)
            assert plan.info()[0] == abi.SCHED_VECTOR
            got = torch.from_numpy(u.copy()).cuda()
            dev.mxv(ring, A, got, torch.from_numpy(v).cuda(), form=form, plan=plan)
            if vtype == 3:
                np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2e-14, atol=0)
            else:
                np.testing.assert_array_equal(got.cpu().numpy(), want)
            plan.close()
