"""The solve with one launch per colour (FAS_MODE_SOR_COLOUR), which also serves
meshes that the persistent solve does not take: FP64 against
fas_gpu_facsls_noalloc (the same kernels, so the same bits) and the checker, the
FP32 form against the persistent solve to the bit (both sum a row's products in
slot order on the same lanes), whole increments as one graph, and a change of
mode between assembly and solve.  Sizes lie on both sides of the persistent
solve's limits between one tile, a cluster and a tile per SM, with rows of every
element family.
"""
import ctypes as C

import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator
from cpfem_code_b200.solver import load_library
from oracle import OracleSolver

pytestmark = pytest.mark.gpu
GRID, COLOUR, FP32, GRAPH = abi.FAS_MODE_SOR_GRID, abi.FAS_MODE_SOR_COLOUR, abi.FAS_MODE_SOR_FP32, abi.FAS_MODE_GRAPH

CASES = [((3, 4, 3), 8, {}), ((5, 5, 5), 8, {}), ((13, 13, 13), 8, {}), ((13, 13, 14), 8, {}), ((25, 24, 26), 8, {}),
         ((2, 1, 1), 20, {}), ((3, 2, 2), 20, {}), ((6, 6, 6), 20, {}), ((7, 9, 8), 20, {}), ((5, 4, 6), 10, {}),
         ((5, 6, 4), 15, {}), ((6, 5, 7), 8, dict(ties=(True, True, True)))]


def _assembled(p, mode):
    g = GpuSolver(p.copy(), mode=mode)
    g.update_node()
    g.elvals(1, 1)
    g.suvals(1)
    return g


def _solved(p, mode, then=None):
    g = _assembled(p, mode)
    try:
        if then is not None:
            g.set_mode(then)
        sweeps, err = g.facsls()
        return sweeps, err, g.download(p.copy()).ddx
    finally:
        g.close()


@pytest.mark.parametrize("n,nodes,extra", CASES)
def test_fp64_equals_noalloc(n, nodes, extra):
    p = generator.structured_cube(n=n, ninc=1, seed=11, nodes=nodes, **extra)
    sweeps, err, ddx = _solved(p, GRID | COLOUR)
    g = _assembled(p, GRID)
    try:
        s, e = C.c_int32(0), C.c_double(0.0)
        fn = load_library().fas_gpu_facsls_noalloc
        fn.restype, fn.argtypes = C.c_int32, [C.c_void_p, C.POINTER(C.c_int32), C.POINTER(C.c_double)]
        abi.check(fn(g._h, C.byref(s), C.byref(e)), "fas_gpu_facsls_noalloc")
        assert (s.value, e.value) == (sweeps, err)
        np.testing.assert_array_equal(g.download(p.copy()).ddx, ddx)
    finally:
        g.close()


@pytest.mark.parametrize("n,nodes,extra", CASES)
def test_fp32_persistent_equals_colour_launches(n, nodes, extra):
    p = generator.structured_cube(n=n, ninc=1, seed=11, nodes=nodes, **extra)
    a, b = _solved(p, GRID | FP32), _solved(p, GRID | FP32 | COLOUR)
    assert a[0] == b[0]
    np.testing.assert_array_equal(a[2], b[2])


@pytest.mark.parametrize("n,nodes,fp32", [((4, 3, 4), 8, 0), ((9, 8, 10), 8, 0), ((9, 8, 10), 8, FP32), ((4, 3, 3), 20, 0),
                                          ((4, 3, 3), 20, FP32)])
def test_increments(n, nodes, fp32):
    p = generator.structured_cube(n=n, ninc=2, grain=2, seed=3, xfree=1, nodes=nodes)
    out = []
    for mode in (COLOUR, COLOUR | GRAPH):
        g = GpuSolver(p.copy(), mode=mode | GRID | fp32)
        try:
            sw = [[r["sor_sweeps"] for r in g.increment(inc)[0]] for inc in (1, 2)]
            out.append((sw, g.download(p.copy())))
        finally:
            g.close()
    (sa, a), (sb, b) = out
    assert sa == sb
    for name in ("x", "dx", "st", "sv"):
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name))
    if not fp32:
        po = p.copy()
        o = OracleSolver(po, 8, threads=8)
        for inc in (1, 2):
            o.increment(inc)
        o.download()
        for name in ("x", "st"):
            ref = getattr(po, name)
            assert np.abs(getattr(a, name) - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("nodes", [8, 20])
def test_mode_set_after_assembly(nodes):
    p = generator.structured_cube(n=(6, 7, 5), ninc=1, seed=2, nodes=nodes)
    ref = _solved(p, GRID | FP32)
    for first, then in ((GRID | FP32, GRID | FP32 | COLOUR), (GRID | FP32 | COLOUR, GRID | FP32)):
        got = _solved(p, first, then)
        assert got[0] == ref[0]
        np.testing.assert_array_equal(got[2], ref[2])
