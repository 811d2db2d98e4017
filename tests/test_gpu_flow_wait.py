"""The persistent solve beside a kernel of another stream that sits on one SM.

Each tile needs a whole SM, and every tile waits for its neighbours' values with
bounded waits.  The tiles of a cooperative launch start together, so the solve
starts when the SM is free and no wait runs out; one launch per colour
(FAS_MODE_SOR_COLOUR) runs on the SMs that are free.
"""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator

pytestmark = pytest.mark.gpu
COLOUR, FP32 = abi.FAS_MODE_SOR_COLOUR, abi.FAS_MODE_SOR_FP32


def _assembled(p, mode):
    g = GpuSolver(p.copy(), mode=mode)
    g.update_node()
    g.elvals(1, 1)
    g.suvals(1)
    return g


@pytest.mark.parametrize("n,nodes,mode", [((16, 15, 17), 8, 0), ((16, 15, 17), 8, FP32), ((9, 10, 8), 20, 0),
                                          ((16, 15, 17), 8, COLOUR)])
def test_an_sm_held_by_another_stream(n, nodes, mode):
    import torch
    p = generator.structured_cube(n=n, ninc=1, seed=4, nodes=nodes)
    g = _assembled(p, mode)
    try:
        start = g.download(p.copy())
        ref = g.facsls()
        ddx = g.download(p.copy()).ddx
        g.upload(start)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            torch.cuda._sleep(int(0.5 * 1.9e9))        # one block for about half a second
            done = torch.cuda.Event()
            done.record()
        got = g.facsls()
        assert done.query() == (mode != COLOUR)        # the persistent solve needed the SM that the sleeper held
        assert got == ref
        np.testing.assert_array_equal(g.download(p.copy()).ddx, ddx)
        side.synchronize()
    finally:
        g.close()
