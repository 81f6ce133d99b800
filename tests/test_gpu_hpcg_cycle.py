"""The persistent V-cycle of the device HPCG against a numpy restatement of
multigrid_v_cycle.hpp and red_black_gauss_seidel.hpp: one cluster or the whole
grid, levels of fewer rows than warps, rows in several rounds per step, colour
counts whose neighbours share a colour (the two-pass step), none to two
smoothing steps, 1 to 8 right-hand sides.

After a few iterations the two differ by the rounding of each: sums of 27 terms,
a few hundred colour steps per iteration, each a contraction (diagonal 26, 26
entries of -1), so errors of 2^-53 per step add up to at most 1e-12 of x."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def stencil(nx, ny, nz):
    t = lambda n: sp.diags([np.ones(n - 1), np.ones(n), np.ones(n - 1)], [-1, 0, 1])  # noqa: E731
    n = nx * ny * nz
    return (27 * sp.identity(n) - sp.kron(t(nz), sp.kron(t(ny), t(nx)))).tocsr()


def restated(dims, levels, colors, pre, post, b, iterations):
    lv, d = [], dims
    for l in range(levels + 1):
        if l and min(d) < 4:
            break
        c = np.arange(np.prod(d) // 8)
        cx, cy = d[0] // 2, d[1] // 2
        inj = 2 * (c % cx) + 2 * ((c // cx) % cy) * d[0] + 2 * (c // (cx * cy)) * d[0] * d[1]
        A = stencil(*d)
        lv.append((A, [A[k::colors] for k in range(min(colors, A.shape[0]))], inj))
        d = tuple(s // 2 for s in d)

    def smooth(l, r, z):
        rows = lv[l][1]
        for order in (range(len(rows)), range(len(rows) - 1, -1, -1)):
            for k in order:
                z[k::colors] = (r[k::colors] - rows[k] @ z + z[k::colors] * 26.0) / 26.0

    def cycle(l, r):
        A, _, inj = lv[l]
        z = np.zeros_like(r)
        if l + 1 == len(lv):
            smooth(l, r, z)
            return z
        for _ in range(pre):
            smooth(l, r, z)
        z[inj] += cycle(l + 1, (r - A @ z)[inj])
        for _ in range(post):
            smooth(l, r, z)
        return z

    x, r, p, rz = np.zeros_like(b), b.copy(), None, None
    for _ in range(iterations):
        z = cycle(0, r)
        new = (r * z).sum(0)
        p = z if p is None else (new / rz) * p + z
        rz = new
        ap = lv[0][0] @ p
        alpha = rz / (p * ap).sum(0)
        x += alpha * p
        r -= alpha * ap
    return x, np.sqrt((r * r).sum(0)) / np.sqrt((b * b).sum(0))


@pytest.mark.parametrize("nrhs", [1, 2, 4, 8])
@pytest.mark.parametrize("dims,levels,colors,pre,post", [
    ((8, 8, 8), 1, 27, 1, 1), ((4, 6, 10), 0, 27, 1, 1), ((16, 12, 20), 1, 27, 2, 0),
    ((16, 16, 16), 1, 16, 1, 1), ((32, 32, 32), 3, 27, 1, 1), ((8, 16, 8), 1, 5, 0, 1),
    ((64, 32, 40), 2, 27, 1, 1), ((8, 8, 8), 1, 300, 1, 1)])
def test_cycle_matches_restatement(cuda, dims, levels, colors, pre, post, nrhs):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    n = int(np.prod(dims))
    b = np.random.default_rng([n, nrhs]).standard_normal((n, nrhs))
    h = C.c_void_p()
    abi.call("alpb_hpcg_create", C.byref(h), *dims, 26.0, -1.0, colors, 2, levels, nrhs,
             dev.stream_ptr())
    tb = torch.from_numpy(b.reshape(-1).copy()).cuda()
    x = torch.zeros_like(tb)
    it, res = (C.c_int64 * nrhs)(), (C.c_double * nrhs)()
    abi.call("alpb_hpcg_solve", h, dev.ptr(tb), dev.ptr(x), 1, pre, post, 6, 1e-30, it, res,
             dev.stream_ptr())
    abi.lib().alpb_hpcg_destroy(h)
    assert list(it) == [6] * nrhs
    want, rel = restated(dims, levels, colors, pre, post, b, 6)
    got = x.cpu().numpy().reshape(n, nrhs)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("colors", [27, 16])
def test_large_level_by_launches(cuda, colors):
    """A finest level of more than 100,000 warps' worth of rows per colour step (a
    launch per step), its coarse level in the cycle kernel; in place (27 colours), and with neighbours of one
    colour (16)."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    dims, nrhs = (164, 164, 164), 8
    n = int(np.prod(dims))
    b = np.random.default_rng(colors).standard_normal((n, nrhs))
    h = C.c_void_p()
    abi.call("alpb_hpcg_create", C.byref(h), *dims, 26.0, -1.0, colors, 2, 1, nrhs,
             dev.stream_ptr())
    tb = torch.from_numpy(b.reshape(-1).copy()).cuda()
    x = torch.zeros_like(tb)
    it, res = (C.c_int64 * nrhs)(), (C.c_double * nrhs)()
    abi.call("alpb_hpcg_solve", h, dev.ptr(tb), dev.ptr(x), 1, 1, 0, 1, 1e-30, it, res,
             dev.stream_ptr())
    abi.lib().alpb_hpcg_destroy(h)
    want, _ = restated(dims, 1, colors, 1, 0, b, 1)
    assert list(it) == [1] * nrhs
    assert np.abs(x.cpu().numpy().reshape(n, nrhs) - want).max() <= 1e-12 * np.abs(want).max()


def test_right_hand_sides_stop_on_their_own(cuda):
    """More iterations than are queued at a time; a right-hand side of a
    scaled unit vector and zero-free noise stop at their own steps, and x no
    longer changes after that."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    n, nrhs = 16 ** 3, 2
    rng = np.random.default_rng(4)
    b = np.stack([stencil(16, 16, 16) @ np.ones(n), rng.standard_normal(n)], 1)
    out = []
    for cols in ([0, 1], [0, 0], [1, 1]):
        h = C.c_void_p()
        abi.call("alpb_hpcg_create", C.byref(h), 16, 16, 16, 26.0, -1.0, 27, 4, 1, nrhs,
                 dev.stream_ptr())
        tb = torch.from_numpy(b[:, cols].reshape(-1).copy()).cuda()
        x = torch.zeros_like(tb)
        it, res = (C.c_int64 * nrhs)(), (C.c_double * nrhs)()
        abi.call("alpb_hpcg_solve", h, dev.ptr(tb), dev.ptr(x), 1, 1, 1, 100, 1e-10, it, res,
                 dev.stream_ptr())
        abi.lib().alpb_hpcg_destroy(h)
        out.append((list(it), x.cpu().numpy().reshape(n, nrhs)))
    (mixed, xm), (first, xf), (second, xs) = out
    assert mixed == [first[0], second[1]] and max(mixed) > 4
    assert np.array_equal(xm[:, 0], xf[:, 0]) and np.array_equal(xm[:, 1], xs[:, 1])


@pytest.mark.parametrize("nrhs,dims", [(8, (48, 48, 48)), (8, (51, 51, 53)), (4, (80, 80, 81)),
                                       (4, (81, 81, 81)), (2, (20, 21, 22)), (1, (20, 21, 22))])
def test_plain_iterations(cuda, nrhs, dims):
    """Without the preconditioner, on both sides of the size from which A p is a
    walk over the rows with a pass for the dot product (rows times right-hand
    sides squared above 2^23).  Six iterations of a contraction, sums of 27 terms
    and of n products: 1e-12 of x as above."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    n = int(np.prod(dims))
    b = np.random.default_rng([n, nrhs]).standard_normal((n, nrhs))
    h = C.c_void_p()
    abi.call("alpb_hpcg_create", C.byref(h), *dims, 26.0, -1.0, 27, 4, 0, nrhs, dev.stream_ptr())
    tb = torch.from_numpy(b.reshape(-1).copy()).cuda()
    x = torch.zeros_like(tb)
    it, res = (C.c_int64 * nrhs)(), (C.c_double * nrhs)()
    abi.call("alpb_hpcg_solve", h, dev.ptr(tb), dev.ptr(x), 0, 1, 1, 6, 1e-30, it, res,
             dev.stream_ptr())
    abi.lib().alpb_hpcg_destroy(h)
    A, want, r = stencil(*dims), np.zeros_like(b), b.copy()
    p, rr = r.copy(), (r * r).sum(0)
    for _ in range(6):
        ap = A @ p
        alpha = rr / (p * ap).sum(0)
        want += alpha * p
        r -= alpha * ap
        new = (r * r).sum(0)
        p, rr = r + new / rr * p, new
    assert list(it) == [6] * nrhs
    assert np.abs(x.cpu().numpy().reshape(n, nrhs) - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("precondition", [0, 1])
@pytest.mark.parametrize("last", [1, 2, 3, 5])
def test_solve_ends_where_it_converges(cuda, last, precondition):
    """A solve that converges on iteration `last` leaves what that many iterations
    leave, whatever was queued behind it."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    dims, nrhs = (24, 16, 32), 4
    n = int(np.prod(dims))
    b = torch.from_numpy(np.repeat(np.random.default_rng(last).standard_normal(n), nrhs)).cuda()

    def solve(max_iter, tol):
        h, x = C.c_void_p(), torch.zeros_like(b)
        abi.call("alpb_hpcg_create", C.byref(h), *dims, 26.0, -1.0, 27, 4, 1, nrhs, dev.stream_ptr())
        it, res = (C.c_int64 * nrhs)(), (C.c_double * nrhs)()
        abi.call("alpb_hpcg_solve", h, dev.ptr(b), dev.ptr(x), precondition, 1, 1, max_iter, tol, it,
                 res, dev.stream_ptr())
        abi.lib().alpb_hpcg_destroy(h)
        return x, list(it), list(res)

    want = solve(last, 1e-30)
    norm = float(b.view(n, nrhs)[:, 0].norm())
    tol = want[2][0] / norm * 1.0001
    for k in range(1, last):
        assert solve(k, 1e-30)[2][0] / norm > tol
    got = solve(100, tol)
    assert got[1] == want[1] == [last] * nrhs
    assert torch.equal(got[0], want[0]) and got[2] == want[2]
