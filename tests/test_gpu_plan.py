"""Products with a plan that does not describe their storage, and what a plan
remembers from one tuning to the next.  Results are compared with the plain
sums in numpy: rows of up to n positive FP64 terms in two orders agree to
2 n 2^-53 relative, whole numbers exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lengths(kind, m, rng):
    if kind == "regular":
        return np.full(m, 5)
    k = np.minimum(rng.zipf(1.6, m), 4000)
    k[:3] = 4000, 300, 65
    return k


def reshaped(lens, rng):
    """another structure of the same number of rows and nonzeroes: its rows in
    another order, then half of each of the first rows moved to one of them"""
    other = rng.permutation(lens)
    cut = other[:400] // 2
    other[:400] -= cut
    other[401] += cut.sum()
    return other


def storage(lens, n, rng):
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return rp, rng.integers(0, n, int(rp[-1])).astype(np.uint32)


def check(A, rp, col, vals, plan, rng, sparse):
    import torch
    from alp_b200 import device as dev
    m, n = A.m, A.n
    x, u = rng.random(n), rng.random(m)
    xa = (rng.random(n) < 0.4).astype(np.uint8)
    got = torch.from_numpy(u.copy()).cuda()
    kw = {"v_assigned": torch.from_numpy(xa).cuda()} if sparse else {}
    dev.mxv(0, A, got, torch.from_numpy(x).cuda(), plan=plan, **kw)
    terms = vals * x[col] * (xa[col] if sparse else 1)
    want = u.copy()
    np.add.at(want, np.repeat(np.arange(m), np.diff(rp)), terms)
    tol = 2 * np.diff(rp).max() * 2.0 ** -53
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=tol, atol=0)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("kind,m", [("regular", 4000), ("regular", 500000), ("skewed", 4000),
                                    ("skewed", 500000)])
def test_plan_of_another_storage(cuda, kind, m, sparse):
    from alp_b200 import device as dev
    rng = np.random.default_rng([m, sparse])
    n, lens = 70001, lengths(kind, m, rng)
    rp, col = storage(lens, n, rng)
    rp2, col2 = storage(reshaped(lens, rng), n, rng)
    vals = rng.random(len(col))
    A, B = dev.from_host(m, n, rp, col, vals), dev.from_host(m, n, rp2, col2, vals)
    assert A.nnz == B.nnz
    for sched in (0, 1, 2):
        plan = dev.Plan(A, sched=sched)
        check(A, rp, col, vals, plan, rng, sparse)
        check(B, rp2, col2, vals, plan, rng, sparse)
        check(A, rp, col, vals, plan, rng, sparse)


def test_boolean_plan_of_another_storage(cuda):
    import torch
    from alp_b200 import device as dev
    rng = np.random.default_rng(2)
    m, n, lens = 4000, 70001, lengths("skewed", 4000, rng)
    rp, col = storage(lens, n, rng)
    rp2, col2 = storage(reshaped(lens, rng), n, rng)
    A, B = dev.from_host(m, n, rp, col, None, 0), dev.from_host(m, n, rp2, col2, None, 0)
    plan = dev.Plan(A)
    x = (rng.random(n) < 0.01).astype(np.uint8)
    for M, o, c in ((A, rp, col), (B, rp2, col2)):
        u = torch.zeros(m, dtype=torch.uint8, device="cuda")
        dev.mxv(1, M, u, torch.from_numpy(x).cuda(), plan=plan)
        want = np.zeros(m, np.uint8)
        np.maximum.at(want, np.repeat(np.arange(m), np.diff(o)), x[c])
        assert np.array_equal(u.cpu().numpy(), want)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("kind,m", [("regular", 4000), ("regular", 500000), ("skewed", 500000)])
def test_structure_changed_in_place(cuda, kind, m, sparse):
    """The offsets a plan was made from get another structure of as many
    nonzeroes.  Products that ran on the plan's lane width alone (the vector
    schedule, the general path) stay right: no row is lost to a list of long
    rows, and no row outgrows its stage in shared memory."""
    from alp_b200 import device as dev
    if kind == "skewed" and not sparse:
        pytest.skip("a merge-path plan's tile table is the structure")
    rng = np.random.default_rng([m, sparse, 7])
    n, lens = 70001, lengths(kind, m, rng)
    rp, col = storage(lens, n, rng)
    rp2, col2 = storage(reshaped(lens, rng), n, rng)
    vals = rng.random(len(col))
    A, B = dev.from_host(m, n, rp, col, vals), dev.from_host(m, n, rp2, col2, vals)
    for sched in (0, 2):
        plan = dev.Plan(A, sched=sched)
        check(A, rp, col, vals, plan, rng, sparse)
        old = A.offsets.clone(), A.indices.clone()
        A.offsets.copy_(B.offsets)
        A.indices.copy_(B.indices)
        check(A, rp2, col2, vals, plan, rng, sparse)
        A.offsets.copy_(old[0])
        A.indices.copy_(old[1])


@pytest.mark.parametrize("kind,m,n", [("skewed", 3000, 3000), ("skewed", 60, 20000), ("regular", 40, 500),
                                      ("regular", 3000, 3000), ("regular", 200000, 200000)])
def test_tuning_again_tries_the_same_kernels(cuda, kind, m, n):
    """Whatever a tuning chose, the next one of the same plan, for another ring
    too, launches the same candidates, and products stay right."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    rng = np.random.default_rng([m, n])
    if kind == "skewed":
        lens = np.minimum(rng.zipf(1.6, m), 4000)
        lens[:3] = 4000, 300, 65
    else:
        lens = np.full(m, 5)
    rp, col = storage(lens, n, rng)
    vals = rng.random(len(col))
    A = dev.from_host(m, n, rp, col, vals)
    P = dev.CRS(m, n, A.nnz, A.offsets, A.indices, None, abi.VOID)
    plan, counts = dev.Plan(A), []
    for ring, M, dt in ((0, A, torch.float64), (2, P, torch.int32), (0, A, torch.float64)) * 3:
        x, y = torch.ones(n, dtype=dt, device="cuda"), torch.zeros(m, dtype=dt, device="cuda")
        before = abi.launches()
        abi.call("alpb_spmv_autotune", plan.h, ring, n, dev.ptr(M.indices), dev.ptr(M.values), M.vtype,
                 dev.ptr(x), dev.ptr(y), dev.stream_ptr())
        counts.append(abi.launches() - before)
        check(A, rp, col, vals, plan, rng, False)
    assert len(set(counts)) == 1, counts
