"""The persistent solve (k_sor_flow, the default FACSLS) against one launch per
colour (fas_gpu_facsls_noalloc) on the same assembled system.

Both run the same multicolour iteration; a row's products are summed in
another order (8 or 16 lanes and late columns last, against 4 or 16 lanes) and
the point update's constants are taken out in advance, so iterates differ by
rounding.  Every sweep adds at most a few units of 2^-53 of the iterate's
largest value per row, and the sweeps contract errors of earlier ones, so
1e-12 bounds a few hundred sweeps with two orders to spare.  Sizes lie at the
edges of the layout: one tile and the first mesh of several, tiles of a few
rows, of partial groups and chunks, tiles that stay in shared memory and tiles
that stream, rows of every element family, ties to far nodes.
"""
import ctypes as C

import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator
from cpfem_code_b200.solver import load_library

pytestmark = pytest.mark.gpu
RTOL = 1e-12
RTOL32 = 1e-5      # the tuned form's bound against the FP64 path

CASES = [((1, 1, 1), 8, {}), ((3, 4, 3), 8, {}), ((4, 4, 5), 8, {}), ((7, 6, 6), 8, {}), ((9, 11, 8), 8, {}),
         ((17, 13, 19), 8, {}), ((25, 24, 26), 8, {}), ((33, 29, 35), 8, {}), ((40, 60, 37), 8, {}),
         ((2, 1, 1), 20, {}), ((3, 3, 2), 20, {}), ((7, 9, 8), 20, {}), ((16, 15, 17), 20, {}),
         ((5, 4, 6), 10, {}), ((5, 6, 4), 15, {}), ((6, 5, 7), 8, dict(ties=(True, True, True))),
         ((3, 4, 3), 20, dict(ties=(True, False, True)))]


def _assembled(p, mode):
    g = GpuSolver(p.copy(), mode=mode)
    g.update_node()
    g.elvals(1, 1)
    g.suvals(1)
    return g


def _noalloc(g):
    fn = load_library().fas_gpu_facsls_noalloc
    fn.restype = C.c_int32
    fn.argtypes = [C.c_void_p, C.POINTER(C.c_int32), C.POINTER(C.c_double)]
    sweeps, err = C.c_int32(0), C.c_double(0.0)
    abi.check(fn(g._h, C.byref(sweeps), C.byref(err)), "fas_gpu_facsls_noalloc")
    return sweeps.value, err.value


@pytest.mark.parametrize("n,nodes,extra", CASES)
@pytest.mark.parametrize("fp32", [False, True])
def test_flow_equals_colour_launches(n, nodes, extra, fp32):
    p = generator.structured_cube(n=n, ninc=1, seed=11, nodes=nodes, **extra)
    g = _assembled(p, abi.FAS_MODE_SOR_GRID | (abi.FAS_MODE_SOR_FP32 if fp32 else 0))
    try:
        start = g.download(p.copy())
        sweeps, err = _noalloc(g)
        ref = g.download(p.copy()).ddx
        got = []
        for _ in range(2):                 # the second solve finds the first one's published values
            g.upload(start)
            s, e = g.facsls()
            got.append(g.download(p.copy()).ddx)
            if fp32:
                assert abs(s - sweeps) <= 1
            else:
                assert s == sweeps
                assert abs(e - err) <= 1e-10 * err
        scale = np.abs(ref).max()
        assert np.abs(got[0] - ref).max() <= (RTOL32 if fp32 else RTOL) * scale
        np.testing.assert_array_equal(got[0], got[1])
    finally:
        g.close()


# both sides of the limits between one tile, a cluster of 16 tiles and a tile
# per SM (180 and 2,906 rows of 27 slots; 350 KB and 5.5 MB of 81-slot rows), and
# far ties inside a cluster; each size also as a whole increment in one graph
CLUSTER = [((4, 4, 5), 8, {}), ((5, 5, 5), 8, {}), ((13, 13, 13), 8, {}), ((13, 13, 14), 8, {}), ((3, 2, 2), 20, {}),
           ((6, 6, 6), 20, {}), ((7, 7, 6), 20, {}), ((5, 4, 4), 8, dict(ties=(True, True, True)))]


@pytest.mark.parametrize("n,nodes,extra", CLUSTER)
@pytest.mark.parametrize("fp32", [False, True])
def test_flow_at_the_limits_of_its_forms(n, nodes, extra, fp32):
    test_flow_equals_colour_launches(n, nodes, extra, fp32)


@pytest.mark.parametrize("n", [(2, 3, 2), (6, 5, 6)])
def test_flow_forms_in_graphs(n):
    p = generator.structured_cube(n=n, ninc=1, seed=5, xfree=1)
    out = []
    for mode in (abi.FAS_MODE_PLAIN, abi.FAS_MODE_GRAPH):
        g = GpuSolver(p.copy(), mode=mode)
        g.increment(1)
        out.append(g.download(p.copy()))
        g.close()
    np.testing.assert_array_equal(out[0].x, out[1].x)
    np.testing.assert_array_equal(out[0].st, out[1].st)
