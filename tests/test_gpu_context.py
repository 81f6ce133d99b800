"""What the library remembers between calls belongs to one CUDA context: the
same calls in a second context of the device, and after the device's context
has been reset, give the first one's bits.  Each program runs in a process of
its own, without torch (which does not outlive a reset)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

HEAD = """
import ctypes as C
import numpy as np
from alp_b200 import _abi as abi
cu = C.CDLL("libcuda.so.1")
rng = np.random.default_rng(5)

def up(a):
    p = C.c_void_p()
    abi.call("alpb_malloc", C.byref(p), max(a.nbytes, 1))
    abi.call("alpb_memcpy_h2d", p, a.ctypes.data_as(C.c_void_p), a.nbytes, None)
    abi.call("alpb_stream_sync", None)
    return p

def down(p, a):
    abi.call("alpb_memcpy_d2h", a.ctypes.data_as(C.c_void_p), p, a.nbytes, None)
    abi.call("alpb_stream_sync", None)
    return a.tobytes()

X, Y = rng.random(70001), rng.random(70001)

def reductions():
    n, x, y = len(X), up(X), up(Y)
    d, r, v, c = C.c_double(0.5), C.c_double(0.0), C.c_double(1.0), C.c_double(2.0)
    abi.call("alpb_dot_f64", C.byref(d), abi.OP_ADD, abi.OP_MUL, n, x, None, y, None, None)
    abi.call("alpb_reduce_f64", C.byref(r), abi.OP_MAX, n, x, None, None)
    abi.call("alpb_vec_reduce", C.byref(v), abi.OP_ADD, 0.0, abi.OP_MUL, 0, n, x, abi.FP64, None,
             y, abi.FP64, None, None, None, abi.BOOL, 0, None)
    S = abi.VecStep
    steps = (S * 2)(S(kind=abi.VEC_FOLDL, op=abi.OP_ADD, z=0, x=1, y=-1),
                    S(kind=abi.VEC_REDUCE, op=abi.OP_ADD, mul_op=abi.OP_MUL, z=-1, x=0, y=1))
    abi.call("alpb_vec_chain", abi.FP64, n, 2, (C.c_void_p * 2)(x, y),
             (C.c_int * 2)(abi.FP64, abi.FP64), 2, steps, C.byref(c), None)
    assert abs(d.value - 0.5 - X @ Y) < 1e-9 and r.value == X.max()
    assert abs(v.value - 1.0 - X @ Y) < 1e-9 and abs(c.value - 2.0 - (X + Y) @ Y) < 1e-9
    return [t.value for t in (d, r, v, c)]
"""

SOLVERS = """
def stencil(sizes):
    sz, nnz, m = (C.c_int64 * 4)(*sizes), C.c_int64(), int(np.prod(sizes))
    off = up(np.zeros(m + 1, np.int64))
    abi.call("alpb_gen_stencil_crs", 3, sz, 26.0, -1.0, 1, off, None, None, C.byref(nnz), None)
    idx, val = up(np.zeros(nnz.value, np.uint32)), up(np.zeros(nnz.value))
    abi.call("alpb_gen_stencil_crs", 3, sz, 26.0, -1.0, 1, off, idx, val, C.byref(nnz), None)
    return m, nnz.value, off, idx, val

def solvers():
    out = []
    m, nnz, off, idx, val = stencil((21, 17, 19))
    for sched in (abi.SCHED_AUTO, abi.SCHED_MERGE_PATH):    # rows streamed; merge path
        plan = C.c_void_p()
        abi.call("alpb_spmv_plan_create", C.byref(plan), m, nnz, off, sched, 0, None)
        y = up(np.zeros(m))
        abi.call("alpb_mxv", 0, 0, 2, m, m, nnz, off, idx, val, abi.FP64, y, None, None, None, None,
                 abi.BOOL, -1, up(X[:m].copy()), None, m, None, None, abi.BOOL, -1, plan, None)
        out.append(down(y, np.zeros(m)))
    x, it, res = up(np.zeros(m)), C.c_int64(), C.c_double()
    abi.call("alpb_cg_solve", m, off, idx, val, up(X[:m].copy()), x, 1000, 1e-8, C.byref(it),
             C.byref(res), None, plan, None)
    out += [down(x, np.zeros(m)), it.value, res.value]
    abi.lib().alpb_spmv_plan_destroy(plan)
    # the stencil is symmetric: its CRS is its CCS
    p = up(np.zeros(m))
    abi.call("alpb_pagerank", m, off, idx, None, off, idx, None, p, 0, 0.85, 1e-3, 200, C.byref(it),
             C.byref(res), None)
    out += [down(p, np.zeros(m)), it.value, res.value]
    # a sparse input over more than 2^21 nonzeroes, its flags asked in shared memory
    m, nnz, off, idx, val = stencil((48, 48, 48))
    va = (np.arange(m) % 3 == 0).astype(np.uint8)
    plan, y = C.c_void_p(), up(np.zeros(m))
    abi.call("alpb_spmv_plan_create", C.byref(plan), m, nnz, off, abi.SCHED_AUTO, 0, None)
    abi.call("alpb_mxv", 0, 0, 2, m, m, nnz, off, idx, val, abi.FP64, y, None, None, None, None,
             abi.BOOL, -1, up(np.arange(m) / 7.0), up(va), int(va.sum()), None, None, abi.BOOL, -1,
             plan, None)
    abi.lib().alpb_spmv_plan_destroy(plan)
    return out + [down(y, np.zeros(m))]
"""

SECOND = """
abi.call("alpb_init", 0)
first = work()
ctx, old = C.c_void_p(), C.c_void_p()
assert cu.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0
for _ in range(2):
    assert work() == first
assert cu.cuCtxPopCurrent_v2(C.byref(old)) == 0
assert work() == first
assert cu.cuCtxDestroy_v2(ctx) == 0
assert work() == first
print("contexts ok")
"""

RESET = """
abi.call("alpb_init", 0)
first = work()
for _ in range(2):
    assert cu.cuDevicePrimaryCtxReset_v2(0) == 0
    abi.call("alpb_init", 0)
    hold = up(np.zeros(1 << 20))   # so that old addresses belong to somebody
    assert work() == first
    assert down(hold, np.ones(1 << 20)) == bytes(8 << 20)
print("contexts ok")
"""


def run(work, program):
    p = subprocess.run([sys.executable, "-c", HEAD + work + program], capture_output=True,
                       text=True, timeout=300, cwd=ROOT)
    assert p.returncode == 0 and "contexts ok" in p.stdout, p.stdout + p.stderr


@pytest.mark.parametrize("program", [SECOND, RESET], ids=["second", "reset"])
def test_reductions(cuda, program):
    run("work = reductions\n", program)


@pytest.mark.parametrize("program", [SECOND, RESET], ids=["second", "reset"])
def test_products_and_solvers(cuda, program):
    run(SOLVERS + "work = solvers\n", program)
