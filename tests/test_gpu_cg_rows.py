"""CG on short regular rows (fixed rows per block): grids of fewer rows than
blocks, ragged grids, every lane split, vectors in shared and in global memory,
items resident and streamed, work spaces that are not 16-byte aligned.

What the solver promises: it stops at ||r|| < tol ||b||, x carries that
residual, and the work space holds r.  r is updated, not recomputed; the two
differ by rounding of at most a few steps' 2^-53 |A| |x| each, far below the
1e-13 ||b|| allowed for these well conditioned systems."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(A, b, max_iter, tol, shift=0, plan=None):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    x = torch.zeros_like(b)
    work = torch.empty(4 * A.m + 1, dtype=torch.float64, device="cuda")[shift:]
    it, res = C.c_int64(), C.c_double()
    rc = abi.lib().alpb_cg_solve(A.m, *A.p(), dev.ptr(b), dev.ptr(x), max_iter, tol, C.byref(it),
                                 C.byref(res), dev.ptr(work), plan.h if plan else None,
                                 dev.stream_ptr())
    torch.cuda.synchronize()
    return rc, x, it.value, res.value, work[:A.m]


def residual(A, b, x):
    import torch
    o, i = A.offsets, A.indices.to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(A.m, device="cuda"), o[1:] - o[:-1])
    return b - torch.zeros_like(b).index_add_(0, rows, A.values * x[i])


@pytest.mark.parametrize("sizes", [(3, 3, 3), (3, 4, 5), (5, 5, 5), (10, 11, 9), (16, 16, 16),
                                   (24, 25, 26), (32, 32, 32), (41, 40, 39), (64, 48, 50),
                                   (70, 71, 72), (3000,), (37, 900)])
def test_cg_rows_stencils(cuda, oracle, sizes):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    A = dev.stencil(sizes, 3.0 ** len(sizes), -1.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(len(sizes))
    b = torch.randn(A.m, generator=g, device="cuda", dtype=torch.float64)
    nb = float(b.norm())
    for tol, plan in ((1e-10, dev.Plan(A, sched=abi.SCHED_MERGE_PATH)), (1e-6, None)):
        rc, x, it, rr, _ = solve(A, b, 3000, tol, plan=plan)
        assert rc == abi.SUCCESS, abi.last_error()
        r = float(residual(A, b, x).norm())
        assert r <= tol * nb + 1e-13 * nb
        assert abs(np.sqrt(rr) - r) <= 1e-13 * nb
    if A.m <= 60000:
        o, i, v = A.to_host()
        rc, x2, it2, _ = oracle.cg(o, i, v, b.cpu().numpy(), np.zeros(A.m), 3000, 1e-6)
        assert rc == 0 and abs(it - it2) <= 1


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("L", [2, 3, 33, 300, 1100])
def test_cg_rows_budget_and_work_space(cuda, L, shift):
    """A fixed number of iterations on 5-point systems (1100^2: vectors stay in
    global memory): not converged, and r and the residual are x's."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    A = dev.poisson2d(L, 0.01)
    g = torch.Generator(device="cuda")
    g.manual_seed(L)
    b = torch.randn(A.m, generator=g, device="cuda", dtype=torch.float64)
    rc, x, it, rr, work = solve(A, b, 25, 1e-14, shift)
    assert it <= 25 and rc == (abi.FAILED if L > 3 else abi.SUCCESS)
    r = residual(A, b, x)
    assert abs(np.sqrt(rr) - float(r.norm())) <= 1e-13 * float(b.norm())
    if shift == 0:
        assert float((work - r).norm()) <= 1e-13 * float(b.norm())


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("sizes", [(40, 40, 40), (64, 64, 64), (80, 80, 80)])
def test_few_iterations(cuda, sizes, steps):
    """A handful of iterations runs on the matrix as it stands where rewriting it
    would cost more than it saves: on both sides of that line the residual
    belongs to x."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    A = dev.stencil(sizes, 27.0, -1.0)
    b = dev.gen_values(A.m, abi.FP64, 7)
    rc, x, it, rr, work = solve(A, b, steps, 1e-14)
    assert rc == abi.FAILED and it == steps
    r, nb = residual(A, b, x), float(b.norm())
    assert abs(np.sqrt(rr) - float(r.norm())) <= 1e-13 * nb
    assert float((work - r).norm()) <= 1e-13 * nb


@pytest.mark.parametrize("sizes,rewritten", [((80, 80, 80), True), ((300, 300, 300), False)])
def test_workspace_is_bounded(cuda, sizes, rewritten):
    """The rewritten rows of an 80^3 grid come from the device's pool; those of
    300^3 would be 8.7 GB, more than the 8 GiB that the solver takes, and it runs
    without them."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    cu, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    A = dev.stencil(sizes, 27.0, -1.0)
    b = dev.gen_values(A.m, abi.FP64, 7)
    plan = dev.Plan(A, sched=abi.SCHED_MERGE_PATH)
    torch.cuda.synchronize()
    high = C.c_uint64(0)
    assert cu.cuMemPoolTrimTo(pool, C.c_size_t(0)) == 0
    assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(high)) == 0    # USED_MEM_HIGH
    rc, x, it, rr, work = solve(A, b, 8, 1e-14, plan=plan)
    assert rc == abi.FAILED and it == 8
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(high)) == 0
    assert (high.value > 12 * A.nnz // 2) == rewritten
    assert abs(np.sqrt(rr) - float(work.norm())) <= 1e-13 * float(b.norm())
