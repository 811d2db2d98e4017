"""Which solve serves meshes near the upper limit of the persistent one: it takes
a mesh while its tiles leave the copy ring enough chunk slots to be faster than one
launch per colour (a solve of few launches), and both solve it alike."""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator

pytestmark = pytest.mark.gpu
FP32 = abi.FAS_MODE_SOR_FP32


@pytest.mark.parametrize("n,nodes,mode,persistent", [(80, 8, 0, True), (82, 8, 0, False), (78, 8, FP32, True), (80, 8, FP32, False),
                                                     (44, 20, 0, True), (46, 20, 0, False), (42, 20, FP32, True),
                                                     (44, 20, FP32, False)])
def test_limit(n, nodes, mode, persistent):
    _check(generator.cube_config(n=n, ninc=1, grain=2, seed=1, nodes=nodes), mode, persistent)


@pytest.mark.parametrize("n,nodes", [((400, 400, 1), 8), ((1, 300, 400), 8), ((160, 160, 1), 20), ((2, 20000, 2), 8)])
def test_sheets_and_rods_of_long_elements(n, nodes):
    """Tiles are cut by the number of elements along an axis, not by their length:
    cut between the layers, these meshes' halos left no room for the ring."""
    _check(generator.structured_cube(n=n, ninc=1, seed=1, nodes=nodes, xfree=1), 0, True)


def _check(p, mode, persistent):
    p.ctrl.toler = 3e-3                        # some tens of sweeps
    out = []
    for m in (mode, mode | abi.FAS_MODE_SOR_COLOUR):
        g = GpuSolver(p.copy(), mode=m)
        try:
            g.update_node()
            g.elvals(1, 1)
            g.suvals(1)
            g.profile(1)
            sweeps, _ = g.facsls()
            out.append((sweeps, g.profile(0)["n_launches"], g.download(p.copy()).ddx))
        finally:
            g.close()
    (sweeps, launches, x), (ref_sweeps, ref_launches, ref) = out
    assert sweeps == ref_sweeps
    assert (launches < ref_launches // 4) == persistent
    assert np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()
