"""The group pass (k_cp, several lanes per Gauss point) against the CPU checker
where its layout or its rule can go wrong: slip-system counts at the edges of
the three shapes (4, 8 and 16 lanes, full and partly empty), point counts at
the edges of warps and CTAs, every hardening option of PLASTC, self hardening
above the latent one, two materials of different shapes, elastic points, and
materials that the rule leaves to the general kernels.

A point takes at most ten outer iterations of six inner ones; each sums at
most 60 products in another order than the checker, and the power law
amplifies a relative error of the stress 1 / am = 20 times: 20 * 60 * 60 *
1.1e-16 = 8e-12 of the largest value.  1e-10 leaves one order.
"""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, abi, generator
from oracle import OracleSolver

pytestmark = pytest.mark.gpu
RTOL = 1e-10


def _material(ns, latent=1.0, self_=None, a3=0.0, a4=1.0, a6=0.0, matrix=None):
    """`ns` slip systems: the twelve of FCC, then random ones."""
    m = generator.fcc_aluminium()
    rng = np.random.default_rng(ns)
    an = rng.standard_normal((60, 3))
    an /= np.linalg.norm(an, axis=1)[:, None]
    ab = np.cross(an, rng.standard_normal((60, 3)))
    ab /= np.linalg.norm(ab, axis=1)[:, None]
    ab[:12], an[:12] = m["ab"], m["an"]
    ampar = np.zeros((ns, 10))
    ampar[:, :6] = (0.05, 150.0, a3, a4, 80.0, a6)
    s = np.full((ns, ns), latent)
    np.fill_diagonal(s, latent if self_ is None else self_)
    return dict(name=f"m{ns}", ns=ns, e=m["e"], ssang=np.zeros(ns), ab=ab[:ns], an=an[:ns], ampar=ampar,
                smatrx=s if matrix is None else matrix)


def _check(p, inc=1):
    pg, po = p.copy(), p.copy()
    g, o = GpuSolver(pg), OracleSolver(po, 8, threads=8)
    for s in (g, o):
        s.constitutive(inc, 1)
        s.download()
    for name in ("ds", "dsv", "srate", "dep", "erepmd"):
        a, b = getattr(pg, name, None), getattr(po, name, None)
        if a is None:
            continue
        scale = np.abs(b).max()
        if name == "erepmd":       # an error measure below the tolerance: its scale is the tolerance
            scale = max(scale, p.ctrl.toler)
        assert np.abs(a - b).max() <= RTOL * scale, name
    t, r = g.tangent(), o.tangent()
    assert np.abs(t - r).max() <= RTOL * np.abs(r).max()
    np.testing.assert_array_equal(g.cp_stats()[0], o.cp_stats()[0])
    np.testing.assert_array_equal(g.cp_ops(), o.cp_ops())


@pytest.mark.parametrize("ns,npts", [(3, 1), (4, 31), (5, 33), (8, 129), (11, 257), (12, 1000), (13, 5), (16, 127), (24, 300),
                                     (31, 65), (32, 129), (33, 9), (47, 100), (59, 33), (60, 257)])
def test_shapes(ns, npts):
    _check(generator.point_batch(npts, seed=ns, material=_material(ns)))


@pytest.mark.parametrize("ns", [12, 17, 40])
@pytest.mark.parametrize("opts", [dict(latent=0.0, self_=1.0), dict(latent=1.0, self_=1.4), dict(a3=7.0), dict(a4=1.7),
                                  dict(a6=0.02), dict(latent=1.2, self_=1.3, a3=3.0, a4=2.0, a6=0.05)])
def test_hardening(ns, opts):
    _check(generator.point_batch(150, seed=ns + 1, material=_material(ns, **opts)))


@pytest.mark.parametrize("opts", [dict(latent=1.4, self_=1.0), dict(matrix=np.ones((12, 12)) + 0.1 * np.tri(12))])
def test_left_to_the_general_kernels(opts):
    _check(generator.point_batch(150, seed=9, material=_material(12, **opts)))


@pytest.mark.parametrize("pair", [(12, 30), (12, 60), (30, 60), (12, 12)])
def test_two_materials_and_elastic_points(pair):
    a, b = (_material(n) for n in pair)
    p = generator.point_batch(333, seed=3, material=b if b["ns"] > a["ns"] else a)
    p.nss, p.e, p.ssang, p.ab, p.an, p.ampar, p.smatrx = generator.pack_materials([a, b])
    which = np.random.default_rng(5).integers(0, 2, p.ngps)
    p.le[:] = which + 1
    p.le[::7] *= -1                      # elastic by its sign
    p.de[::11] = 0.0                     # elastic for lack of strain
    p.ds[::13] = 0.0                     # elastic for lack of stress
    _check(p)
