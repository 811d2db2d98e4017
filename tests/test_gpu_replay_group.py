"""The replay and its adjoint by groups of lanes (k_replay_step, k_replay_seed,
k_replay_rev) against the general kernels with their dual passes.

A handle whose materials all qualify takes the groups.  The same points with
one more point of a material whose latent hardening is no single number take
the general kernels, and their objective weights leave that point out.  Sizes
lie at the edges of the lane shapes, of warps and of segments; every hardening
parameter that PLASTC reads is given a value of its own.

States of the two replays agree to 1e-10 (the bound of the constitutive parity
tests); an adjoint is a function of the states whose derivative the power law
scales by at most 1 / am = 20 an increment, damped by the elastic predictor's
restart: 1e-8 of a gradient block's largest entry leaves a factor of five.
"""
import numpy as np
import pytest

from cpfem_code_b200 import GpuSolver, ReplayHistory, generator

pytestmark = pytest.mark.gpu
RTOL = 1e-8


def _material(ns, latent=1.0, self_=None, a3=5.0, a4=1.0, a6=0.0):
    m = generator.fcc_aluminium()
    rng = np.random.default_rng(ns)
    an = rng.standard_normal((32, 3))
    an /= np.linalg.norm(an, axis=1)[:, None]
    ab = np.cross(an, rng.standard_normal((32, 3)))
    ab /= np.linalg.norm(ab, axis=1)[:, None]
    ab[:12], an[:12] = m["ab"], m["an"]
    ampar = np.zeros((ns, 10))
    ampar[:, :6] = (0.05, 150.0, a3, a4, 80.0, a6)
    s = np.full((ns, ns), latent)
    np.fill_diagonal(s, latent if self_ is None else self_)
    return dict(name=f"m{ns}", ns=ns, e=m["e"], ssang=np.zeros(ns), ab=ab[:ns], an=an[:ns], ampar=ampar, smatrx=s)


def _history(p, ninc, chk, seed):
    rng = np.random.default_rng(seed)
    de = np.stack([p.de * (1.0 + 0.2 * rng.standard_normal(p.de.shape)) for _ in range(ninc)])
    de[:, ::9] *= 1e-4                                       # points that hardly slip
    if ninc > 1:
        de[1, ::5] = 0.0                                     # the elastic branch for lack of strain
    dr = 2e-4 * rng.standard_normal((ninc, p.ngps, 3))
    w = 1e6 * (0.5 + rng.random(p.ngps))
    w[-1] = 0.0                                              # the extra point
    return de, dr, np.full(ninc, p.tiem[0]), w, 1e-3 * rng.standard_normal(p.ngps)


@pytest.mark.parametrize("ns,npts,ninc,chk,opts", [
    (3, 1, 1, 1, {}), (12, 15, 5, 2, {}), (12, 64, 4, 4, dict(latent=0.0, self_=1.0)), (12, 33, 3, 1, dict(a4=1.7)),
    (11, 129, 4, 3, dict(latent=1.0, self_=1.4)), (13, 31, 4, 2, dict(a6=0.02)), (24, 17, 3, 5, {}),
    (30, 65, 5, 2, dict(latent=1.2, self_=1.3, a4=2.0, a6=0.05)), (32, 40, 3, 2, dict(a4=0.0))])
def test_groups_equal_dual_passes(ns, npts, ninc, chk, opts):
    mat = _material(ns, **opts)
    other = _material(ns)                                    # as many systems as the state has
    other["smatrx"] = np.ones((ns, ns)) + 0.1 * np.tri(ns)   # no single latent number
    p = generator.point_batch(npts + 1, seed=ns + npts, material=mat)
    p.ctrl.toler = 1e-11
    p.nss, p.e, p.ssang, p.ab, p.an, p.ampar, p.smatrx = generator.pack_materials([mat, other])
    p.le[2::7] *= -1                                         # elastic by its sign
    p.le[-1] = 1
    h = _history(p, ninc, chk, 3)
    out = []
    for last in (1, 2):
        q = p.copy()
        q.le[-1] = last
        g = GpuSolver(q)
        try:
            out.append(g.adjoint_grad(ReplayHistory(*h, q=(0.3, 0.5, 0.8), chk_every=chk)))
            J, _ = g.adjoint_forward(ReplayHistory(*h, q=(0.3, 0.5, 0.8), chk_every=chk))
            assert J == out[-1]["J"]
        finally:
            g.close()
    a, b = out
    assert abs(a["J"] - b["J"]) <= RTOL * abs(b["J"])
    for key, sl in (("st", slice(0, npts)), ("sv", slice(0, npts)), ("ampar", slice(0, 1))):
        x, y = a[key][sl], b[key][sl]
        assert np.isfinite(x).all()
        # Euler angles and slip resistances have scales of their own
        for u, v in ((x[:, :3], y[:, :3]), (x[:, 3:], y[:, 3:])) if key == "sv" else ((x, y),):
            assert np.abs(u - v).max() <= RTOL * np.abs(v).max(), key
