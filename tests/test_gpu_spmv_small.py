"""Small skewed matrices in one launch: rows at the edges of a lane group and of
a block's batch, empty rows, matrices without long rows, both lane widths,
against the restatement.

FP64 (positive terms): orders of at most 8192 terms agree to 2 * 8192 * 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = {"long": [0, 1, 63, 64, 65, 255, 256, 257, 1023, 1025, 8192] + [3] * 150,
        "short_only": [0, 64, 1, 2] * 3 + [2] * 61,
        "many": [20] * 700 + [500] * 9 + [0] * 300,
        "one": [9, 0, 0, 0, 0]}


@pytest.mark.parametrize("form", [2, 1])
@pytest.mark.parametrize("ring", [0, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("rows", sorted(ROWS))
def test_small_products(cuda, oracle, rows, ring, form):
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    from oracle.oracle import NP
    rng = np.random.default_rng([len(rows), ring])
    lens = np.array(ROWS[rows])
    m, n = len(lens), 9000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.uint32)
    vtype = abi.RING_TYPE[ring]
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 3, k)).astype(NP[vtype])  # noqa: E731
    vals, u, v = value(len(col)), value(m), value(n)
    if ring == 7:       # products of many factors above one: keep them finite
        vals, v = vals * 1e-3, v * 1e-3 + 1.0
    for pattern in (False, True):
        want = u.copy()
        t = abi.VOID if pattern else vtype
        w = None if pattern else vals
        assert oracle.mxv(ring, 0, form, m, n, rp, col, w, t, want, v=v)[0] == 0
        A = dev.from_host(m, n, rp, col, w, t)
        plan = dev.Plan(A)
        assert plan.info()[0] == abi.SCHED_MERGE_PATH
        got = torch.from_numpy(u.copy()).cuda()
        dev.mxv(ring, A, got, torch.from_numpy(v).cuda(), form=form, plan=plan)
        if vtype == 3:
            np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2 * 8192 * 2.0 ** -53, atol=0)
        else:
            np.testing.assert_array_equal(got.cpu().numpy(), want)
        plan.close()
