"""The general mxv path (masks, sparse vectors, descriptors) on rows cut in
chunks: row lengths at the edges of a row group, of a chunk and of the warp
that sums a row's chunks, against the restatement.

Integer and boolean rings must agree bit for bit.  FP64 sums n <= 9000
positive terms in another order: each of the two orders is off by at most
(n - 1) 2^-53 relative, so entries agree to 2 * 9000 * 2^-53 = 2e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 31, 32, 33, 63, 64, 65, 66, 255, 256, 257, 511, 513, 8191, 8193, 8449, 9000, 2]
DESCR = {"none": 0, "invert": 1, "structural": 8, "invert_structural": 9, "add_identity": 32,
         "use_index": 64, "explicit_zero": 512}


def storage(rng, vtype):
    from oracle.oracle import NP, VOID
    n = 9001
    lens = np.array(LENGTHS * 3)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.uint32)
    if vtype == 3:
        vals = rng.random(len(col))
    elif vtype == 2:
        vals = rng.integers(1, 101, len(col)).astype(np.int32)
    else:
        vals = (rng.random(len(col)) < 0.5).astype(NP[vtype])
    return len(lens), n, rp, col, vals


@pytest.mark.parametrize("frontier", [0.02, 0.5, 1.0])
@pytest.mark.parametrize("descr", sorted(DESCR))
@pytest.mark.parametrize("ring", [0, 1, 2])
def test_general_path_long_rows(cuda, oracle, ring, descr, frontier):
    import torch
    from alp_b200 import device as dev
    vtype = {0: 3, 1: 1, 2: 2}[ring]
    rng = np.random.default_rng([ring, DESCR[descr], int(100 * frontier)])
    m, n, rp, col, vals = storage(rng, vtype)
    npt = {3: np.float64, 2: np.int32, 1: np.uint8}[vtype]
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 2 if vtype == 1 else 1000, k)).astype(npt)  # noqa: E731
    u, v = value(m), value(n)
    ua = (rng.random(m) < 0.5).astype(np.uint8)
    va = (rng.random(n) < frontier).astype(np.uint8)
    mask, mask_a = (rng.random(m) < 0.7).astype(np.uint8), (rng.random(m) < 0.8).astype(np.uint8)
    A = dev.from_host(m, n, rp, col, vals, vtype)
    plan = dev.Plan(A, sched=1)
    for form in (0, 1, 2):
        wu, wa = u.copy(), ua.copy()
        rc, wn = oracle.mxv(ring, DESCR[descr], form, m, n, rp, col, vals, vtype, wu, wa,
                            u_mask=mask, u_mask_assigned=mask_a, u_mask_count=int(mask_a.sum()),
                            v=v, v_assigned=va)
        assert rc == 0
        T = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
        gu, ga = T(u), T(ua)
        gn = torch.tensor([int(ua.sum())], dtype=torch.int64, device="cuda")
        dev.mxv(ring, A, gu, T(v), descr=DESCR[descr], form=form, u_assigned=ga, u_nnz=gn,
                u_mask=T(mask), u_mask_assigned=T(mask_a), u_mask_count=int(mask_a.sum()),
                v_assigned=T(va), plan=plan)
        np.testing.assert_array_equal(ga.cpu().numpy() != 0, wa != 0)
        assert int(gn) == wn
        got, want = gu.cpu().numpy()[wa != 0], wu[wa != 0]
        if vtype == 3:
            np.testing.assert_allclose(got, want, rtol=2e-12, atol=0)
        else:
            np.testing.assert_array_equal(got, want)
    plan.close()


@pytest.mark.parametrize("n", [65537, 1638400, 1638401])
@pytest.mark.parametrize("case", ["sparse", "input_mask", "both_inverted"])
@pytest.mark.parametrize("ring", [0, 1, 2])
def test_general_path_input_bits(cuda, oracle, ring, case, n):
    """From 2^21 nonzeroes on the inputs that take part are asked as bits in
    shared memory, up to 1,638,400 of them (one more: in memory, as below);
    the last word is ragged for most n.  Rows of up to 2e5 terms: FP64 orders
    agree to 2 * 2e5 * 2^-53 = 5e-11."""
    import torch
    from alp_b200 import device as dev
    vtype = {0: 3, 1: 1, 2: 2}[ring]
    npt = {3: np.float64, 2: np.int32, 1: np.uint8}[vtype]
    rng = np.random.default_rng([ring, n])
    lens = rng.integers(0, 70, 60000)
    lens[[5, 77]] = 200000, 300
    m, nnz = len(lens), int(lens.sum())
    assert nnz >= 1 << 21
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = rng.integers(0, n, nnz).astype(np.uint32)
    col[-1] = n - 1
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 2 if vtype == 1 else 1000, k)).astype(npt)  # noqa: E731
    vals, u, v = value(nnz), value(m), value(n)
    va = (rng.random(n) < 0.1).astype(np.uint8)
    vm, vma = (rng.random(n) < 0.5).astype(np.uint8), (rng.random(n) < 0.6).astype(np.uint8)
    kw, gkw, descr = {}, {}, 0
    T = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    if case != "input_mask":
        kw["v_assigned"], gkw["v_assigned"] = va, T(va)
    if case != "sparse":
        kw.update(v_mask=vm, v_mask_assigned=vma, v_mask_count=int(vma.sum()))
        gkw.update(v_mask=T(vm), v_mask_assigned=T(vma), v_mask_count=int(vma.sum()))
        descr = 1 if case == "both_inverted" else 0
    want = u.copy()
    assert oracle.mxv(ring, descr, 0, m, n, rp, col, vals, vtype, want, v=v, **kw)[0] == 0
    A = dev.from_host(m, n, rp, col, vals, vtype)
    for plan in (dev.Plan(A), None):
        got = T(u)
        dev.mxv(ring, A, got, T(v), descr=descr, form=0, plan=plan, **gkw)
        if vtype == 3:
            np.testing.assert_allclose(got.cpu().numpy(), want, rtol=5e-11, atol=0)
        else:
            np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("path", ["general", "rows", "small", "merge"])
def test_products_under_capture(cuda, path):
    """A captured product, replayed on new inputs, gives the direct call's bits
    (the general path takes its scratch from the stream-ordered pool)."""
    import torch
    from alp_b200 import _abi as abi
    from alp_b200 import device as dev
    rng = np.random.default_rng(11)
    m = n = 40000 if path == "merge" else 5000
    lens = np.full(m, 5) if path == "rows" else np.minimum(rng.zipf(1.7, m) * 8, 2000)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = rng.integers(0, n, int(lens.sum())).astype(np.uint32)
    A = dev.from_host(m, n, rp, col, rng.random(len(col)))
    plan = dev.Plan(A, sched=abi.SCHED_MERGE_PATH if path == "merge" else abi.SCHED_AUTO)
    x, u = (torch.empty(k, dtype=torch.float64, device="cuda") for k in (n, m))
    xa = torch.from_numpy((rng.random(n) < 0.3).astype(np.uint8)).cuda()
    kw = {"v_assigned": xa, "v_count": int(xa.sum())} if path == "general" else {}
    call = lambda: dev.mxv(0, A, u, x, plan=plan, **kw)  # noqa: E731
    x.fill_(1.0)
    u.fill_(0.0)
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for k in range(3):
        x.copy_(torch.from_numpy(rng.random(n)))
        u.fill_(float(k))
        g.replay()
        got = u.clone()
        u.fill_(float(k))
        call()
        assert torch.equal(got, u)


def lane_sums(rp, x, W):
    """Row sums of x as W lanes take them: lane l the entries l, l + W, ... in
    order, then the lanes by halves."""
    lens = np.diff(rp)
    acc = np.zeros((len(lens), W))
    for k in range(0, int(lens.max(initial=0)), W):
        for lane in range(W):
            on = lens > k + lane
            acc[on, lane] = x[rp[:-1][on] + k + lane] + acc[on, lane]
    while acc.shape[1] > 1:
        h = acc.shape[1] // 2
        acc = acc[:, :h] + acc[:, h:]
    return acc[:, 0]


@pytest.mark.parametrize("case", ["no_plan", "steady", "given", "given_hubs", "narrow"])
def test_general_path_lane_width(cuda, case):
    """Which lanes sum a row, in the bits of an FP64 product by a pattern matrix
    of more than 2^20 nonzeroes: the default width without a plan, the plan's on
    rows of one length, the caller's where one was given, a quarter of the
    plan's own where lengths differ.  Rows in the plan's list of long rows (more
    than 64 nonzeroes, beside hub rows) are left out."""
    import torch
    from alp_b200 import device as dev
    rng = np.random.default_rng(17)
    m, n = 60000, 30011
    if case == "steady":
        lens, kw, W = np.full(m, 27), {}, 4
    elif case == "no_plan":
        lens, kw, W = rng.integers(10, 45, m), None, 16
    else:
        lens = rng.integers(0, 61, m)
        kw, W = ({}, 4) if case == "narrow" else ({"vector_width": 8}, 8)
        if case == "given_hubs":
            lens[[3, 40000]] = 5000, 90
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    nnz = int(rp[-1])
    assert nnz > 1 << 20
    col = rng.integers(0, n, nnz).astype(np.uint32)
    A = dev.from_host(m, n, rp, col, None, 0)
    plan = None if kw is None else dev.Plan(A, **kw)
    x, u = rng.random(n), rng.random(m)
    xa = np.ones(n, np.uint8)
    got = torch.from_numpy(u.copy()).cuda()
    dev.mxv(0, A, got, torch.from_numpy(x).cuda(), plan=plan, v_assigned=torch.from_numpy(xa).cuda())
    want = np.where(lens > 0, u + lane_sums(rp, x[col], W), u)
    ok = got.cpu().numpy() == want
    if case == "given_hubs":
        ok |= lens > 64
    assert ok.all(), np.flatnonzero(~ok)[:5]


@pytest.mark.parametrize("vertices", [3000, 200000])
def test_captured_general_product_holds_no_allocation(cuda, vertices):
    """Under capture the general path takes no scratch: the graph has only
    kernels, so it can be a child of another graph; hub rows, with and without
    the size that asks input bits in shared memory, give the direct bits."""
    import ctypes as C

    import torch
    from alp_b200 import device as dev
    cu = C.CDLL("libcuda.so.1")
    rng = np.random.default_rng(vertices)
    m = n = vertices
    lens = np.minimum(rng.zipf(1.7, m) * 8, 3000)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    A = dev.from_host(m, n, rp, rng.integers(0, n, int(rp[-1])).astype(np.uint32), rng.random(int(rp[-1])))
    assert vertices < 10000 or A.nnz > 1 << 21
    plan = dev.Plan(A)
    x = torch.from_numpy(rng.random(n)).cuda()
    xa = torch.from_numpy((rng.random(n) < 0.3).astype(np.uint8)).cuda()
    u, count = torch.zeros(m, dtype=torch.float64, device="cuda"), int(xa.sum())

    def call():
        dev.mxv(0, A, u, x, plan=plan, v_assigned=xa, v_count=count)

    call()
    want = u.clone()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    raw, k = C.c_void_p(g.raw_cuda_graph()), C.c_size_t()
    assert cu.cuGraphGetNodes(raw, None, C.byref(k)) == 0 and k.value >= 1
    nodes = (C.c_void_p * k.value)()
    assert cu.cuGraphGetNodes(raw, nodes, C.byref(k)) == 0
    for node in nodes:
        kind = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        assert kind.value == 0      # CU_GRAPH_NODE_TYPE_KERNEL
    parent, child, run = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert cu.cuGraphCreate(C.byref(parent), 0) == 0
    assert cu.cuGraphAddChildGraphNode(C.byref(child), parent, None, C.c_size_t(0), raw) == 0
    assert cu.cuGraphInstantiateWithFlags(C.byref(run), parent, C.c_ulonglong(0)) == 0
    for _ in range(2):
        u.zero_()
        torch.cuda.synchronize()
        assert cu.cuGraphLaunch(run, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert torch.equal(u, want)
    assert cu.cuGraphExecDestroy(run) == 0 and cu.cuGraphDestroy(parent) == 0


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("density", [0.3, 1.0])
@pytest.mark.parametrize("true", [0.0, 0.02, 1.0])
def test_boolean_rows_of_many_inputs(cuda, oracle, true, density, masked):
    """From a quarter of the inputs on a boolean row is looked at by its first
    nonzeroes alone before the rest: whichever nonzero decides it, and whether it
    is assigned at all when none does."""
    import torch
    from alp_b200 import device as dev
    rng = np.random.default_rng([int(100 * true), int(10 * density), masked])
    n = 9001
    lens = np.array(LENGTHS * 3)
    lens = np.concatenate([lens, rng.integers(0, 60, 40000 if masked else 400)])
    m = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = rng.integers(0, n, int(rp[-1])).astype(np.uint32)
    v = (rng.random(n) < true).astype(np.uint8)
    va = (rng.random(n) < density).astype(np.uint8)
    u, ua = (rng.random(m) < 0.1).astype(np.uint8), (rng.random(m) < 0.5).astype(np.uint8)
    mask = (rng.random(m) < 0.6).astype(np.uint8)
    T = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    kw = dict(u_mask=mask, u_mask_assigned=mask, u_mask_count=int(mask.sum())) if masked else {}
    wu, wa = u.copy(), ua.copy()
    rc, wn = oracle.mxv(1, 0, 0, m, n, rp, col, None, 0, wu, wa, v=v, v_assigned=va, **kw)
    assert rc == 0
    A = dev.from_host(m, n, rp, col, None, 0)
    for plan in (dev.Plan(A), dev.Plan(A, vector_width=8), None):
        gu, ga = T(u), T(ua)
        gn = torch.tensor([int(ua.sum())], dtype=torch.int64, device="cuda")
        dev.mxv(1, A, gu, T(v), form=0, u_assigned=ga, u_nnz=gn, v_assigned=T(va), plan=plan,
                **{k: T(a) if isinstance(a, np.ndarray) else a for k, a in kw.items()})
        assert np.array_equal(ga.cpu().numpy() != 0, wa != 0) and int(gn) == wn
        assert np.array_equal(gu.cpu().numpy()[wa != 0], wu[wa != 0])


@pytest.mark.parametrize("ring", [0, 1, 2])
def test_dense_descriptor_ignores_flags_at_every_size(cuda, oracle, ring):
    """Under the dense descriptor the input's flags are not read, also where an
    input mask is asked as bits (more than 2^21 nonzeroes).  Sums of up to 100
    positive terms: FP64 orders agree to 2 * 100 * 2^-53."""
    import torch
    from alp_b200 import device as dev
    vtype = {0: 3, 1: 1, 2: 2}[ring]
    npt = {3: np.float64, 2: np.int32, 1: np.uint8}[vtype]
    rng = np.random.default_rng(ring)
    m, n = 60000, 20000
    lens = rng.integers(0, 100, m)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    nnz = int(rp[-1])
    assert nnz >= 1 << 21
    col = rng.integers(0, n, nnz).astype(np.uint32)
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 2 if vtype == 1 else 1000, k)).astype(npt)  # noqa: E731
    vals, u, v = value(nnz), value(m), value(n)
    vm = (rng.random(n) < 0.5).astype(np.uint8)
    stale, full = np.zeros(n, np.uint8), np.ones(n, np.uint8)
    A = dev.from_host(m, n, rp, col, vals, vtype)
    T = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    want = u.copy()
    assert oracle.mxv(ring, 16, 0, m, n, rp, col, vals, vtype, want, v=v, v_assigned=full, v_mask=vm,
                      v_mask_assigned=full, v_mask_count=n)[0] == 0
    got = T(u)
    dev.mxv(ring, A, got, T(v), descr=16, form=0, plan=dev.Plan(A), v_assigned=T(stale), v_count=n,
            v_mask=T(vm), v_mask_assigned=T(full), v_mask_count=n)
    if vtype == 3:
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=3e-14, atol=0)
    else:
        np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("ring", [0, 1, 2])
@pytest.mark.parametrize("m,length", [(4, 100000), (16, 1000), (64, 6144), (64, 6145), (2000, 767),
                                      (2000, 768), (40, 256), (40, 257), (9000, 129)])
def test_few_or_long_rows(cuda, oracle, ring, m, length):
    """Long rows of one length: walked, a block each, or in chunks, at the edges
    of those rules.  FP64 sums of n positive terms: 2 n 2^-53 relative."""
    import torch
    from alp_b200 import device as dev
    vtype = {0: 3, 1: 1, 2: 2}[ring]
    npt = {3: np.float64, 2: np.int32, 1: np.uint8}[vtype]
    rng = np.random.default_rng([ring, m, length])
    n = 30011
    rp = (np.arange(m + 1) * length).astype(np.int64)
    col = rng.integers(0, n, int(rp[-1])).astype(np.uint32)
    value = lambda k: (rng.random(k) if vtype == 3 else rng.integers(0, 2 if vtype == 1 else 1000, k)).astype(npt)  # noqa: E731
    vals, u, v = value(len(col)), value(m), value(n)
    T = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    A = dev.from_host(m, n, rp, col, vals, vtype)
    plan = dev.Plan(A)
    mask = (rng.random(m) < 0.7).astype(np.uint8)
    for frontier in (0.001, 0.3):
        va, ua = (rng.random(n) < frontier).astype(np.uint8), (rng.random(m) < 0.5).astype(np.uint8)
        wu, wa = u.copy(), ua.copy()
        kw = dict(u_mask_count=int(mask.sum()))
        rc, wn = oracle.mxv(ring, 0, 0, m, n, rp, col, vals, vtype, wu, wa, v=v, v_assigned=va,
                            u_mask=mask, u_mask_assigned=mask, **kw)
        assert rc == 0
        gu, ga, gn = T(u), T(ua), torch.tensor([int(ua.sum())], dtype=torch.int64, device="cuda")
        dev.mxv(ring, A, gu, T(v), form=0, u_assigned=ga, u_nnz=gn, v_assigned=T(va), plan=plan,
                u_mask=T(mask), u_mask_assigned=T(mask), **kw)
        assert np.array_equal(ga.cpu().numpy() != 0, wa != 0) and int(gn) == wn
        got, want = gu.cpu().numpy()[wa != 0], wu[wa != 0]
        if vtype == 3:
            np.testing.assert_allclose(got, want, rtol=2 * length * 2.0 ** -53, atol=0)
        else:
            np.testing.assert_array_equal(got, want)
