"""The row-streaming product of short regular rows: chunk edges, the last
chunk's ragged copy, every value size, arrays that start off a 16-byte boundary
(another kernel) and rows of 1 to 64 nonzeroes, against the restatement; and
which of the two kernels a product takes.

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


def streamed_sums(rp, x):
    """row sums in k_spmv_rows' order: one lane a row up to 8 entries, five at a
    time, else two lanes, seven at a time"""
    lens = np.diff(rp)
    L, U = (1, 5) if lens.max() <= 8 else (2, 7)
    acc = np.zeros((len(lens), L))
    for q0 in range(0, -(-int(lens.max()) // L), U):
        part = np.zeros_like(acc)
        for q in range(q0, q0 + U):
            for k in range(L):
                on = lens > q * L + k
                part[on, k] += x[rp[:-1][on] + q * L + k]
        acc += part
    return acc.sum(1)


def lane_sums(rp, x, W):
    """row sums in k_spmv_vector_dense's order: W lanes, then by halves"""
    lens = np.diff(rp)
    acc = np.zeros((len(lens), W))
    for k in range(int(lens.max())):
        on = lens > k
        acc[on, k % W] += x[rp[:-1][on] + k]
    while acc.shape[1] > 1:
        h = acc.shape[1] // 2
        acc = acc[:, :h] + acc[:, h:]
    return acc[:, 0]


@pytest.mark.parametrize("maxlen,m,valued,streamed", [
    (1, 100, True, True), (2, 1001, True, True), (5, 33, True, False), (5, 5000, False, True),
    (7, 4099, True, False), (7, 4099, False, True), (8, 4000, True, False), (8, 4000, False, False),
    (9, 2000, False, False), (11, 2000, False, True), (15, 2000, True, False), (17, 15, True, True),
    (27, 20001, True, True), (27, 20001, False, True), (32, 1000, True, False), (33, 1000, True, True),
    (63, 300, True, True), (64, 300, True, False), (5, 4200000, True, True)])
def test_which_kernel_sums_rows_of_one_length(cuda, maxlen, m, valued, streamed):
    """Streamed or by lanes, told by the bits of the FP64 sums (matrix values of
    one, so only the order of the adds rounds)."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    rng = np.random.default_rng([maxlen, m])
    lens = np.full(m, maxlen)
    if m > 200 and maxlen > 2:      # boundary rows
        lens[rng.integers(0, m, m // 200)] = maxlen // 2
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    n = m + 70
    col = rng.integers(0, n, int(rp[-1])).astype(np.uint32)
    x, u = rng.random(n), rng.random(m)
    A = dev.from_host(m, n, rp, col, np.ones(len(col)) if valued else None, abi.FP64 if valued else abi.VOID)
    got = torch.from_numpy(u.copy()).cuda()
    plan = dev.Plan(A)
    dev.mxv(0, A, got, torch.from_numpy(x).cuda(), plan=plan)
    sums = streamed_sums(rp, x[col]) if streamed else lane_sums(rp, x[col], plan.info()[1])
    assert np.array_equal(got.cpu().numpy(), u + sums)


def test_rows_of_differing_lengths_by_lanes(cuda):
    import torch
    from alp_b200 import device as dev
    rng = np.random.default_rng(5)
    m = 20000
    lens = rng.integers(8, 25, m)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = rng.integers(0, m, int(rp[-1])).astype(np.uint32)
    x, u = rng.random(m), rng.random(m)
    A = dev.from_host(m, m, rp, col, np.ones(len(col)))
    got = torch.from_numpy(u.copy()).cuda()
    plan = dev.Plan(A)
    dev.mxv(0, A, got, torch.from_numpy(x).cuda(), plan=plan)
    assert np.array_equal(got.cpu().numpy(), u + lane_sums(rp, x[col], plan.info()[1]))


@pytest.mark.parametrize("ring", [0, 2, 4, 5])
@pytest.mark.parametrize("maxlen,m", [(1, 31), (2, 33), (3, 4000), (5, 63), (5, 64), (5, 65), (7, 999),
                                      (17, 15), (17, 16), (27, 17), (63, 301)])
def test_streamed_rows_of_one_length(cuda, oracle, maxlen, m, ring):
    """Rows of one length, odd: streamed under every value size where the type
    and the size let them be; edges of a chunk of 64 rows (up to 8 nonzeroes) and
    of 16."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    from oracle.oracle import NP
    rng = np.random.default_rng([maxlen, m, ring])
    n = m + 70
    rp = (np.arange(m + 1) * maxlen).astype(np.int64)
    col = np.concatenate([rng.choice(n, maxlen, replace=False) for _ in range(m)]).astype(np.uint32)
    vtype = abi.RING_TYPE[ring]
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 3, k)).astype(NP[vtype])  # noqa: E731
    vals, u, v = value(len(col)), value(m), value(n)
    for pattern in (False, True):
        want = u.copy()
        kind = abi.VOID if pattern else vtype
        assert oracle.mxv(ring, 0, 2, m, n, rp, col, None if pattern else vals, kind, want, v=v)[0] == 0
        A = dev.from_host(m, n, rp, col, None if pattern else vals, kind)
        got = torch.from_numpy(u.copy()).cuda()
        dev.mxv(ring, A, got, torch.from_numpy(v).cuda(), plan=dev.Plan(A))
        if vtype == 3:
            np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2e-14, atol=0)
        else:
            np.testing.assert_array_equal(got.cpu().numpy(), want)
