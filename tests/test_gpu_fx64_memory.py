"""The fixed-point copies that an FP64 operator keeps beside its links cost no call its memory: where a field, a
workspace or an inner operator's workspace finds none, they are given back and the hopping term runs on
the FP64 kernel.  Each case runs in a process of its own whose device memory pool has a small bound, so the
device itself is never short."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

CHILD = r"""
import ctypes as C, sys
import numpy as np
import grid_gb300 as g
from oracle import oracle as o

class Props(C.Structure):  # CUmemPoolProps
    _fields_ = [("type", C.c_int), ("handles", C.c_int), ("location", C.c_int * 2), ("security", C.c_void_p),
                ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]

def pool_of(max_size):
    p = Props(type=1, max_size=max_size)  # CU_MEM_ALLOCATION_TYPE_PINNED on device 0
    p.location[0] = 1
    pool = C.c_void_p()
    assert cu.cuMemPoolCreate(C.byref(pool), C.byref(p)) == 0
    assert cu.cuDeviceSetMemPool(0, pool) == 0
    return pool

what, bound, taken, flags, graphs = sys.argv[1], *(int(a) for a in sys.argv[2:])
cu = C.CDLL("libcuda.so.1")
dims, Ls, par = (8, 8, 8, 16), 8, (0.1, 1.8, 1.5, 0.5)
U, x = g.random_gauge(dims, 0.5, 1), g.random_gaussian(4096 * Ls * 12, 2)
small = g.MobiusFermion(g.random_gauge((2, 2, 2, 2), 0.5, 1), (2, 2, 2, 2), 4, *par)  # context and module
pool = pool_of(bound)
if taken:
    held = C.c_void_p()
    assert cu.cuMemAllocAsync(C.byref(held), C.c_size_t(taken), None) == 0
ref = o.OracleOp(1, 0, dims, Ls, list(par), U, g.antiperiodic_t())

if what == "fields":
    op = g.MobiusFermion(U, dims, Ls, *par, flags=flags)
    a, b = op.FermionRedBlackField(g.ODD).import_(x), op.FermionRedBlackField(g.EVEN)
    op.DhopEO(a, b, 0)
    before, more = b.export(), []
    try:
        while len(more) < 1000:
            more.append(op.FermionRedBlackField(g.ODD))
    except g.GridError:
        pass
    op.DhopEO(a, b, 0)
    after = b.export()
    assert o.rel_l2(after, ref.dhop_cb(x, 1, 0)) < 2e-14 and o.rel_l2(after, before) < 2e-14  # 2e-14: double-float
    n = len(more)
    del more
    op.ImportGauge(U)  # takes the copies again where there are any
    op.DhopEO(a, b, 0)
    assert (b.export() == before).all()
    print("RESULT", n)
else:
    od = g.MobiusFermion(U, dims, Ls, *par, flags=flags)
    of = g.MobiusFermion(U, dims, Ls, *par, precision=g.F32)
    src, sol = od.FermionField().import_(np.concatenate([x, x])), od.FermionField().zero()
    cg = g.ConjugateGradientReliableUpdate(1e-9, 2000, 1e-3, g.SchurDiagMooeeOperator(of), g.SchurDiagMooeeOperator(od),
                                           use_graphs=graphs)
    s = g.SchurRedBlackDiagMooeeSolve(cg)
    s(od, src, sol)
    assert o.rel_l2(ref.apply(o.OP_M, sol.export()), np.concatenate([x, x])) < 1e-7
    high = C.c_uint64()
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(high)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    print("RESULT", high.value)
"""


def child(what, bound, flags, graphs=0, taken=0):
    args = [str(v) for v in (bound, taken, flags, graphs)]
    r = subprocess.run([sys.executable, "-c", CHILD, what] + args, cwd=ROOT, timeout=240,
                       env=dict(os.environ, PYTHONPATH=str(ROOT)), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return int(r.stdout.split("RESULT")[1])


def test_fields_take_the_copies_memory(gpu_available):
    """Under one bound an operator with copies has room for as many fields as one without, and its
    hopping term stays right after they are gone and after they are back."""
    assert child("fields", 160 << 20, 0) >= child("fields", 160 << 20, 2)


@pytest.mark.parametrize("graphs", [0, 1])
def test_mixed_solve_in_the_memory_of_one_without_copies(gpu_available, graphs):
    """A mixed-precision solve in less than the copies' 21 MiB above what it takes without them.  (The hole that they
    leave is not all of use: a full FP64 field of 12 MiB fits once.)  The pool is bounded in steps of 32 MiB:
    what is left of the last one is taken before."""
    used = child("solve", 0, 2, graphs) + (14 << 20)
    taken = -used % (32 << 20)
    child("solve", used + taken, 0, graphs, taken)
