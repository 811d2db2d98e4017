"""The general constitutive kernels (one thread or one warp per Gauss point, in
work-sorted order or from the device queue), which serve materials without a
single latent hardening number, against the CPU checker; bounds are those of
the parity tests (1e-11 of a pass, 1e-10 after increments)."""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator
from oracle import OracleSolver

pytestmark = pytest.mark.gpu
MODES = [abi.FAS_MODE_PLAIN, abi.FAS_MODE_CP_WARP, abi.FAS_MODE_CP_QUEUE]


def _general(p):
    p.smatrx = p.smatrx.copy()
    p.smatrx[:, 0, 1] += 0.1
    return p


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("mixed", [False, True])
def test_points(mode, mixed):
    hcp = generator.hcp_zirconium()
    p = generator.point_batch(1500, seed=11, **(dict(material=hcp) if mixed else {}))
    if mixed:
        p.nss, p.e, p.ssang, p.ab, p.an, p.ampar, p.smatrx = generator.pack_materials([generator.fcc_aluminium(), hcp])
        p.le[:] = 1 + np.random.default_rng(2).integers(0, 2, p.ngps)
    p = _general(p)
    pg, po = p.copy(), p.copy()
    g, o = GpuSolver(pg, mode=mode), OracleSolver(po, 8, threads=8)
    for s in (g, o):
        s.constitutive(1, 1)
        s.download()
    for name in ("ds", "dsv", "srate", "dep"):
        assert rel(getattr(pg, name), getattr(po, name)) < 1e-11, name
    assert rel(g.tangent(), o.tangent()) < 1e-11
    np.testing.assert_array_equal(g.cp_ops(), o.cp_ops())


@pytest.mark.parametrize("mode", MODES)
def test_mixed_mesh(mode):
    p = _general(generator.mixed_config(n=6, ninc=2))
    pg, po = p.copy(), p.copy()
    g, o = GpuSolver(pg, mode=mode), OracleSolver(po, 8, threads=8)
    for inc in (1, 2):
        rg, evg = g.increment(inc)
        ro, evo = o.increment(inc)
        assert [r["sor_sweeps"] for r in rg] == [r["sor_sweeps"] for r in ro]
        assert [(e["gp"], e["sys"]) for e in evg] == [(e["gp"], e["sys"]) for e in evo]
    g.download()
    o.download()
    assert rel(pg.st, po.st) < 1e-10
    assert rel(pg.sv[:, :33], po.sv[:, :33]) < 1e-10


@pytest.mark.parametrize("n,nodes", [((6, 6, 6), 8), ((3, 3, 3), 20), ((3, 2, 3), 10), ((2, 3, 3), 15)])
def test_queue_and_graph(n, nodes):
    p = _general(generator.structured_cube(n=n, ninc=2, grain=1, seed=5, xfree=1, nodes=nodes))
    out = []
    for mode in (abi.FAS_MODE_PLAIN, abi.FAS_MODE_CP_QUEUE, abi.FAS_MODE_CP_QUEUE | abi.FAS_MODE_GRAPH):
        g = GpuSolver(p.copy(), mode=mode)
        rep = [g.increment(inc)[0] for inc in (1, 2)]
        out.append((rep, g.download(p.copy())))
        g.close()
    for rep, q in out[1:]:
        assert rep == out[0][0]
        for name in ("x", "st", "sv"):
            np.testing.assert_array_equal(getattr(q, name), getattr(out[0][1], name))
    o = OracleSolver(p, 8, threads=8)
    for inc in (1, 2):
        o.increment(inc)
    o.download()
    for name in ("x", "st"):
        assert rel(getattr(out[0][1], name), getattr(p, name)) < 1e-10
