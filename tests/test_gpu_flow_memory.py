"""A handle with room for the assembled rows but not for the persistent solve's
copy of them (as large again) solves with one launch per colour."""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [abi.FAS_MODE_PLAIN, abi.FAS_MODE_GRAPH])
def test_no_room_for_the_tiles(mode):
    import torch
    p = generator.structured_cube(n=(40, 40, 40), ninc=1, seed=6, xfree=1)
    p.ctrl.maxit = 2

    def solved(mode):
        free = torch.cuda.mem_get_info()[0]
        g = GpuSolver(p.copy(), mode=mode)
        try:
            sweeps = [r["sor_sweeps"] for r in g.increment(1)[0]]
            return sweeps, g.download(p.copy()).x, free - torch.cuda.mem_get_info()[0]
        finally:
            g.close()

    torch.cuda.empty_cache()
    solved(mode)                                   # what the process allocates once
    solved(mode | abi.FAS_MODE_SOR_COLOUR)
    _, _, most = solved(mode)
    sweeps, x, least = solved(mode | abi.FAS_MODE_SOR_COLOUR)
    assert most - least > 100 << 20                # 68,921 rows of 1,984 bytes and more
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (most + least) // 2, dtype=torch.uint8, device="cuda")
    try:
        got = solved(mode)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert got[0] == sweeps
    np.testing.assert_array_equal(got[1], x)
    assert solved(mode)[2] >= most                 # with room again, a new handle takes the tiles
