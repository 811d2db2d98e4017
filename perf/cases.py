"""The calls whose time and results are watched, over the range they are used in.

Three kinds of call, each through the Python face of the C ABI:

``points``   the constitutive update of independent material points (a
             material-point driver, or a solver that keeps its own mesh and
             hands strain increments over): strain increments and the stress
             guess go up from pinned host memory, the stress, the state
             variables' increments, slip rates and (where asked for) the
             tangents come back;
``step``     Newton iterations of an increment on a structured mesh
             (UPDATE_NODE, then passes of NRITER's loop body: element pass,
             assembly, boundary conditions, SOR solve, correction), for a
             driver that keeps its own Newton loop (its third pass is the first
             with plastic points); with ``steps`` 0 the whole increment in one
             call, as the reference's main loop has it;
``adjoint``  the gradient of a lattice-strain objective over a recorded
             strain history (calibration of hardening and orientations).

The state that a pass changes goes up before it, so that every pass does the
same work.
"""
import functools
import math

import numpy as np
import torch

from cpfem_code_b200 import GpuSolver, ReplayHistory, abi, generator

MODES = {"plain": abi.FAS_MODE_PLAIN, "tuned": abi.FAS_MODE_SOR_FP32, "graph": abi.FAS_MODE_GRAPH}


def listed():
    return [
        # the smallest material-point batch of a calibration loop: one
        # specimen's grains, tangents wanted; launches and copies count
        dict(name="points_fcc_4k", kind="points", material="fcc", n=4099, strain=1e-3, tangent=True),
        # 30 slip systems, several families: the heavy local systems
        dict(name="points_hcp_100k", kind="points", material="hcp", n=100003, strain=1e-3, tangent=False),
        # the constitutive micro-benchmark's 2^20 points
        dict(name="points_fcc_1m", kind="points", material="fcc", n=1 << 20, strain=1e-3, tangent=False),
        # 64 nodes: the smallest mesh in use, nothing but latency
        dict(name="step_cube_3", kind="step", nx=3, ny=3, nz=3, nodes=8, mixed=False, grain=1,
             xfree=3, mode="plain", steps=3),
        # a whole increment of a small cube in one call, every face held
        dict(name="increment_cube_12", kind="step", nx=12, ny=12, nz=12, nodes=8, mixed=False, grain=2, xfree=1,
             mode="plain", steps=0),
        # the 16^3 cube of the differentiation workload
        dict(name="step_cube_16", kind="step", nx=16, ny=16, nz=16, nodes=8, mixed=False, grain=1,
             xfree=3, mode="plain", steps=4),
        # half HCP, half FCC with twinning: uneven local work, solver in L2
        dict(name="step_mixed_32", kind="step", nx=32, ny=32, nz=32, nodes=8, mixed=True, grain=2,
             xfree=3, mode="plain", steps=3),
        # the headline cube, in FP64 and with the FP32-matrix sweeps
        dict(name="step_cube_64", kind="step", nx=64, ny=64, nz=64, nodes=8, mixed=False, grain=2,
             xfree=3, mode="plain", steps=3),
        dict(name="step_cube_64_tuned", kind="step", nx=64, ny=64, nz=64, nodes=8, mixed=False, grain=2, xfree=3,
             mode="tuned", steps=3),
        # the reference sample's mesh: 10^3 20-node bricks
        dict(name="step_brick20_10", kind="step", nx=10, ny=10, nz=10, nodes=20, mixed=False, grain=1, xfree=3,
             mode="plain", steps=3),
        # 20-node bricks with uneven edges, solver streamed from memory
        dict(name="step_brick20_21", kind="step", nx=21, ny=17, nz=23, nodes=20, mixed=False, grain=2, xfree=3,
             mode="plain", steps=3),
        # the gradient over the 16^3 cube's points and 20 increments
        dict(name="adjoint_4k", kind="adjoint", n=4096, ninc=20, chk=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("points", "step", "step", "step", "adjoint"))
    if kind == "points":
        material = rng.choice(("fcc", "fcc", "hcp"))
        n = _log_int(rng, 500, (1 << 20) if material == "fcc" else 100000)
        return dict(kind=kind, material=material, n=n, strain=rng.choice((5e-4, 1e-3, 2e-3)),
                    tangent=n <= 20000 and rng.random() < 0.5)
    if kind == "adjoint":
        ninc = rng.randint(2, 20)
        return dict(kind=kind, n=_log_int(rng, 300, 4096 * 20 // ninc), ninc=ninc, chk=rng.randint(1, ninc))
    nodes = rng.choice((8, 8, 20))
    steps = rng.choice((0, 2, 3))
    top = {8: (1728 if steps == 0 else 64 ** 3), 20: (216 if steps == 0 else 8000)}[nodes]
    edge = _log_int(rng, 8, top) ** (1.0 / 3.0)
    a, b = rng.uniform(0.8, 1.25), rng.uniform(0.8, 1.25)
    mesh = [max(2, int(round(edge * f))) for f in (a, b, 1.0 / (a * b))]
    while mesh[0] * mesh[1] * mesh[2] > top:
        mesh[mesh.index(max(mesh))] -= 1
    return dict(kind=kind, nx=mesh[0], ny=mesh[1], nz=mesh[2], nodes=nodes, mixed=nodes == 8 and rng.random() < 0.25,
                grain=rng.choice((1, 2)), xfree=1 if steps == 0 else 3,
                mode=rng.choice(("plain", "plain", "tuned") if steps else ("plain", "tuned", "graph")), steps=steps)


# ------------------------------------------------------------------- inputs
def _pinned(a):
    t = torch.empty(a.shape, dtype=getattr(torch, str(a.dtype)), pin_memory=True)
    b = t.numpy()
    b[...] = a
    return b


class _Host:
    """Host arrays of a state transfer: what is named goes across, the rest stays."""

    def __init__(self, nsv, ns, **arrays):
        self.nsv, self.ns = nsv, ns
        self.arrays = {k: _pinned(np.ascontiguousarray(v)) for k, v in arrays.items()}

    def state_descriptor(self):
        d = abi.FasState(real_bytes=8, nsv=self.nsv, ld_sv=self.nsv, ld_slip=self.ns)
        for k, a in self.arrays.items():
            setattr(d, k, abi.iptr(a) if a.dtype == np.int32 else abi.ptr(a))
        return d


def _mesh(case):
    return case["nx"], case["ny"], case["nz"]


def _materials(case):
    if case["kind"] == "step" and case["mixed"]:
        return [generator.hcp_zirconium(), generator.fcc_aluminium()]
    if case["kind"] == "points" and case["material"] == "hcp":
        return [generator.hcp_zirconium()]
    return [generator.fcc_aluminium()]


def _problem(case, seed):
    if case["kind"] == "step":
        two = dict(fractions=[0.5, 0.5], twinlim=1, twinprob=1.0) if case["mixed"] else {}
        return generator.structured_cube(n=_mesh(case), xfree=case["xfree"], eps_inc=(1e-3, 0.0, 0.0), ninc=2,
                                         grain=case["grain"], seed=seed, nodes=case["nodes"],
                                         materials=_materials(case), **two)
    p = generator.point_batch(case["n"], seed=seed, strain_norm=case.get("strain", 1e-3),
                              material=_materials(case)[0])
    if case.get("material") == "hcp":
        ns = int(p.nss[0])
        spread = 1.0 + np.random.default_rng(seed + 1).random((case["n"], ns))
        p.sv[:, 3:3 + ns] = generator.hcp_zirconium()["tau0"] * spread
    return p


def _history(case, seed):
    """A monotonic path per point with a little scatter and spin."""
    n, ninc = case["n"], case["ninc"]
    rng = np.random.default_rng(seed + 7)
    path = rng.standard_normal((1, n, 6)) + 0.1 * rng.standard_normal((ninc, n, 6))
    path *= 1e-3 / np.linalg.norm(path, axis=2, keepdims=True)
    return dict(de=path, dr=2e-4 * rng.standard_normal((ninc, n, 3)), dt=np.full(ninc, 1e-3),
                w=rng.random(n) / n, y=1e-4 * rng.standard_normal(n), q=(1.0, 0.0, 0.0))


def prepare(case, seed):
    p = _problem(case, seed)
    nsv, ns, g = int(p.nsv), int(p.nss.max()), p.ngps
    z = np.zeros
    st = dict(case=case, solver=GpuSolver(p, mode=MODES[case.get("mode", "plain")]))
    if case["kind"] == "points":
        st["up"] = _Host(nsv, ns, de=p.de, dr=p.dr, ds=p.ds, dsv=z((g, nsv)), twinsys=z(g, np.int32))
        st["down"] = _Host(nsv, ns, ds=z((g, 6)), dsv=z((g, nsv)), dep=z(g), srate=z((g, ns)),
                           twinsys=z(g, np.int32))
    elif case["kind"] == "adjoint":
        st["hist"] = ReplayHistory(chk_every=case["chk"], **_history(case, seed))
    else:
        n3 = p.x.size
        up = dict(x=p.x, dx=z(n3), ds=z((g, 6)), dsv=z((g, nsv)), timestwinned=z(g, np.int32),
                  twinsys=z(g, np.int32))
        down = dict(x=z(n3), dx=z(n3), ddx=z(n3), fc=z(n3), ds=z((g, 6)), dsv=z((g, nsv)), de=z((g, 6)),
                    dr=z((g, 3)), dep=z(g), srate=z((g, ns)), twinsys=z(g, np.int32))
        if case["steps"] == 0:   # the whole increment also commits
            up.update(st=z((g, 6)), ep=z((g, 6)), eps=z(g), rt=z((g, 3)), sv=p.sv[:, :nsv], cumslip=z((g, ns)))
            down.update(st=z((g, 6)), ep=z((g, 6)), eps=z(g), rt=z((g, 3)), sv=z((g, nsv)), cumslip=z((g, ns)),
                        timestwinned=z(g, np.int32))
        st["up"], st["down"] = _Host(nsv, ns, **up), _Host(nsv, ns, **down)
    return st


def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "adjoint":
        return s.adjoint_grad(state["hist"])
    s.upload(state["up"])
    out = {}
    if case["kind"] == "points":
        s.constitutive(1, 1)
        if case["tangent"]:
            out["tangent"] = s.tangent()
    else:
        if case["steps"] == 0:
            reports, _ = s.increment(1)
        else:
            s.update_node()
            reports = [s.nr_step(1, k + 1)[0] for k in range(case["steps"])]
        out["sor_sweeps"] = np.array([r["sor_sweeps"] for r in reports], np.int64)
        out["norms"] = np.array([[r["sdx"], r["sfc"], r["cp_err"], r["alp2"]] for r in reports])
    s.download(state["down"])
    out.update(state["down"].arrays)
    return out


def work(case):
    per = {12: 1.6e4, 30: 8.0e4}    # counted operations of one plastic update by slip systems
    if case["kind"] == "points":
        ns = 30 if case["material"] == "hcp" else 12
        gp = 6 + 3 + 6 + 6 + 2 * (3 + ns)            # de, dr, st, ds, sv, dsv in
        gp += 6 + (3 + ns) + 1 + ns + (36 if case["tangent"] else 0)
        return dict(bytes=8.0 * gp * case["n"], flops=per[ns] * case["n"])
    if case["kind"] == "adjoint":
        n, ninc = case["n"], case["ninc"]
        return dict(bytes=8.0 * n * (9 * ninc + 2 + 2 * 21), flops=n * ninc * (per[12] + 3 * 4.0e3))
    nx, ny, nz = _mesh(case)
    el = nx * ny * nz
    corners = (nx + 1) * (ny + 1) * (nz + 1)
    edges = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    nnod, npg, blocks = (corners, 1, 27.0 * corners) if case["nodes"] == 8 else \
        (corners + edges, 8, 81.0 * corners + 51.0 * edges)
    ns = 30 if case["mixed"] else 12
    steps = case["steps"] or 6
    # state in and out once, about 300 sweeps of the solver per Newton iteration
    return dict(bytes=8.0 * (3 * nnod * 6 + el * npg * (6 * 5 + 2 * (3 + ns) + 3 + ns)),
                flops=steps * (300.0 * 18.0 * blocks + el * npg * per[ns] / 2))


# ------------------------------------------------- the same in plain 64 bits
F8 = torch.float64
PI, PJ = (0, 1, 2, 1, 2, 0), (0, 1, 2, 2, 0, 1)      # Voigt 11 22 33 23 31 12


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F8, device=_dev())


def _material(m):
    amp = _t(np.asarray(m["ampar"], float)[:, :6])
    return dict(ns=int(m["ns"]), e=_t(m["e"]), ab=_t(m["ab"]), an=_t(m["an"]), am=amp[:, 0], amp=amp,
                sm=_t(m["smatrx"]), ssang=_t(m["ssang"]))


def _euler(ph):
    s1, c1, s2, c2, s, c = (f(ph[..., k]) for k in (0, 2, 1) for f in (torch.sin, torch.cos))
    a = torch.stack([c1 * c2 - s1 * s2 * c, s1 * c2 + c1 * s2 * c, s2 * s,
                     -c1 * s2 - s1 * c2 * c, -s1 * s2 + c1 * c2 * c, c2 * s,
                     s1 * s, -c1 * s, c], -1)
    return a.reshape(a.shape[:-1] + (3, 3)), torch.stack([s2, c2, s], -1)


def _compliance(e, a):
    """Rotated compliance as the reference's ELASTC has it."""
    rows = []
    b = [[a[..., q, p] for q in range(3)] for p in range(3)]
    for I in range(6):
        for J in range(6):
            i, j, k, l = PI[min(I, J)], PJ[min(I, J)], PI[max(I, J)], PJ[max(I, J)]
            pr = lambda p, q, r, s: b[i][p] * b[j][q] * b[k][r] * b[l][s]
            v = sum(pr(p, p, p, p) * e[p] for p in range(3))
            for m, (p, q) in enumerate(((1, 2), (2, 0), (0, 1))):
                v = v + (pr(p, p, q, q) + pr(q, q, p, p)) * e[3 + m]
                v = v + 0.5 * (pr(p, q, p, q) + pr(q, p, q, p)) * e[6 + m]
            rows.append((1.0 if min(I, J) < 3 else 2.0) * v)
    return torch.stack(rows, -1).reshape(a.shape[:-2] + (6, 6))


def _rotate(r, v):
    d = lambda i: torch.sqrt(1.0 - r[..., (i + 1) % 3] ** 2 - r[..., (i + 2) % 3] ** 2)
    R = torch.stack([d(0), r[..., 2], -r[..., 1], -r[..., 2], d(1), r[..., 0], r[..., 1], -r[..., 0], d(2)],
                    -1).reshape(r.shape[:-1] + (3, 3))
    A = v[..., [0, 5, 4, 5, 1, 3, 4, 3, 2]].reshape(v.shape[:-1] + (3, 3))
    B = R.transpose(-1, -2) @ A @ R
    return torch.stack([B[..., PI[k], PJ[k]] for k in range(6)], -1)


def _mises(v, stress):
    m = 6.0 if stress else 1.5
    q = sum((v[..., i] - v[..., (i + 1) % 3]) ** 2 + m * v[..., i + 3] ** 2 for i in range(3))
    return torch.sqrt(q / 4.5)


def _systems(mat, a):
    d, n = mat["ab"] @ a, mat["an"] @ a              # a^T v for every system
    b = torch.stack([d[..., 0] * n[..., 0], d[..., 1] * n[..., 1], d[..., 2] * n[..., 2],
                     d[..., 1] * n[..., 2] + d[..., 2] * n[..., 1], d[..., 2] * n[..., 0] + d[..., 0] * n[..., 2],
                     d[..., 0] * n[..., 1] + d[..., 1] * n[..., 0]], -1)
    return b, torch.linalg.cross(d, n) / 2.0


def _spower(a, p):
    big = a.abs() >= 1e-35
    v = torch.exp(torch.clamp(p * torch.log(torch.where(big, a.abs(), 1.0)), -80.0, 80.0))
    return torch.where(big, torch.copysign(v, a), 0.0)


def _harden(mat, s0, gam, p=None):
    """Hardened resistances and the rates h_ij = s_ij gradh_j (saturating
    Voce hardening, exponents 1 and 0)."""
    amp = mat["amp"]
    a2, a3, a5 = (amp[:, k] + (p[j] if p is not None else 0.0) for k, j in ((1, 1), (2, 2), (4, 3)))
    arg = torch.clamp(torch.where(a5 != 0.0, 1.0 - s0 / a5, 0.0), min=0.0)
    h = mat["sm"] * (a3 + a2 * arg).unsqueeze(-2)
    return s0 + (h @ gam.abs().unsqueeze(-1)).squeeze(-1), h


def _scale(mat, act, s, gam, tau, cap, afactor):
    first = act.to(torch.int8).argmax(1, keepdim=True)
    ga = torch.where(act, gam.abs(), -1.0)
    top = ga.max(1).values
    at = ga.argmax(1, keepdim=True)
    am = torch.where((at == first).squeeze(1), mat["am"][0], mat["am"][at.squeeze(1)])
    over = top > cap
    sc = torch.where(over, cap / torch.where(over, top, 1.0), 1.0)
    sm = _spower(0.9 * sc, afactor * am)
    sm = torch.where(over, torch.where(sm == 0.0, 0.004 / am, sm), 1.0)
    return s * sm[:, None], gam * sc[:, None], tau * sm[:, None]


def _slips(mat, act, s0, gam, tau, dt, c):
    """Newton on the logarithms of the active slips, then the matrix of the
    local system."""
    am, n = mat["am"], gam.shape[1]
    conv = c.toler * float(am.max())
    both = act[:, :, None] & act[:, None, :]
    eye = torch.eye(n, dtype=F8, device=gam.device)

    def rates(k, g):
        s1, h = _harden(mat, s0[k], g)
        ah = torch.where(g.abs()[:, None, :] > 1e-14, torch.sign(g)[:, None, :] * h / s1[:, :, None], 0.0)
        return s1, torch.where(both[k], ah, 0.0)

    gam = gam.clone()
    todo = torch.arange(gam.shape[0], device=gam.device)
    for _ in range(c.maxit):
        g = gam[todo]
        s1, ah = rates(todo, g)
        A = ah * g[:, None, :] + eye * torch.where(act[todo], am, 1.0)[:, None, :]
        fg = s1 * _spower(g / dt, am)
        ok = act[todo] & (tau[todo] * fg > 0.0)
        err = torch.where(ok, torch.log(torch.where(ok, tau[todo] / torch.where(ok, fg, 1.0), 1.0)), 0.0)
        size = err.norm(dim=1)
        dg = torch.linalg.solve(A, err)
        big = dg.abs().max(1).values
        gam[todo] = g * torch.exp(torch.where(big > 5.0, 5.0 / big, 1.0)[:, None] * dg)
        todo = todo[size > conv]
        if todo.numel() == 0:
            break
    s1, ah = rates(slice(None), gam)
    X = ah * tau[:, :, None]
    dia = torch.where(gam.abs() > 1e-12, am * tau / torch.where(gam.abs() > 1e-12, gam, 1.0), am / 1e-12)
    return gam, s1, torch.where(both, X, 0.0) + eye * torch.where(act, dia, 1.0)[:, None, :]


def _update(mat, c, sv, dsv, de, r, st, ds, dt, twins=None):
    """The stress update of points of one material, plastic branch:
    dict of ds, dsv, dep, srate, chi, twinsys, xg (signed slips)."""
    ns, ph = mat["ns"], sv[:, :3] + dsv[:, :3]
    a, aug = _euler(ph)
    S, (b, rot) = _compliance(mat["e"], a), _systems(mat, a)
    t, s0 = _rotate(r, st), sv[:, 3:3 + ns]
    s, cap = t + ds, 6.0 * _mises(de, False)
    n = sv.shape[0]
    o = {k: torch.zeros((n,) + d, dtype=F8, device=sv.device)
         for k, d in (("ds", (6,)), ("dsv", (3 + ns,)), ("dep", ()), ("srate", (ns,)), ("chi", (6, 6)), ("xg", (ns,)),
                      ("err", ()))}
    o["twinsys"] = torch.zeros(n, dtype=torch.int64, device=sv.device)
    twin = mat["ssang"].abs() > 1.5
    todo = torch.arange(n, device=sv.device)
    for it in range(c.maxit):
        B, s_, s0_ = b[todo], s[todo], s0[todo]
        tau = (B @ s_.unsqueeze(-1)).squeeze(-1)
        if twins:
            fires = (twin & (tau > s0_)) & (o["twinsys"][todo] == 0)[:, None]
            o["twinsys"][todo] += torch.where(fires.any(1), fires.to(torch.int8).argmax(1) + 1, 0)
        gam = dt * _spower(tau / s0_, 1.0 / mat["am"])
        gam = torch.where(twin | (mat["ssang"] * tau / s0_ < 0.0), 0.0, gam)
        act = ~(gam.abs() < 1e-6 * gam.abs().max(1, keepdim=True).values)
        gam = torch.where(act, gam, 0.0)
        s_, gam, tau = _scale(mat, act, s_, gam, tau, cap[todo], c.afactor)
        gam, s1, X = _slips(mat, act, s0_, gam, tau, dt, c)
        s_, gam, tau = _scale(mat, act, s_, gam, tau, cap[todo], c.afactor)
        epl = (B.transpose(1, 2) @ gam.unsqueeze(-1)).squeeze(-1)
        err = de[todo] - epl - (S[todo] @ (s_ - t[todo]).unsqueeze(-1)).squeeze(-1)
        Ba = torch.where(act[:, :, None], B, 0.0)
        jac = Ba.transpose(1, 2) @ torch.linalg.solve(X, Ba) + S[todo]
        err = torch.linalg.solve(jac, err)
        em = _mises(err, True) / _mises(s_, True)
        s_ = s_ + err / (1.0 + c.alpha * em)[:, None]
        s[todo] = s_
        fin = ~(em > c.toler) | (it + 1 >= c.maxit)
        k = todo[fin]
        if k.numel():
            g = gam[fin]
            rtn = (rot[k].transpose(1, 2) @ g.unsqueeze(-1)).squeeze(-1) - r[k]
            rx, ag = (a[k] @ rtn.unsqueeze(-1)).squeeze(-1), aug[k]
            d1 = torch.where(ag[:, 2].abs() < 1e-5, rtn[:, 2], (ag[:, 0] * rx[:, 0] + ag[:, 1] * rx[:, 1]) / ag[:, 2])
            dph = ag[:, 1] * rx[:, 0] - ag[:, 0] * rx[:, 1]
            d2 = rx[:, 2] - d1 * a[k][:, 2, 2]
            o["dsv"][k] = torch.cat([torch.stack([d1, dph, d2], 1), s1[fin] - s0_[fin]], 1)
            o["ds"][k], o["err"][k], o["srate"][k] = s_[fin] - st[k], em[fin], (g / dt).abs()
            o["dep"][k] = _mises(epl[fin], False)
            inv = torch.linalg.inv(jac[fin])
            o["chi"][k] = (inv + inv.transpose(1, 2)) / 2.0
            tk = (b[k] @ s_[fin].unsqueeze(-1)).squeeze(-1)
            o["xg"][k] = torch.where(g != 0.0, torch.copysign(g.abs(), tk), 0.0)
        todo = todo[~fin]
        if todo.numel() == 0:
            break
    return o


def _exact_points(case, seed):
    p = _problem(case, seed)
    mat, outs = _material(_materials(case)[0]), []
    ns, step = mat["ns"], 1 << 16
    for i in range(0, p.ngps, step):
        k = slice(i, i + step)
        sv = _t(p.sv[k, :3 + ns])
        o = _update(mat, p.ctrl, sv, torch.zeros_like(sv), _t(p.de[k]), _t(p.dr[k]), _t(p.st[k]), _t(p.ds[k]),
                    float(p.tiem[0]))
        outs.append({n: o[n].cpu().numpy() for n in ("ds", "dsv", "dep", "srate", "chi")})
    out = {n: np.concatenate([o[n] for o in outs]) for n in outs[0]}
    chi = out.pop("chi")
    return dict(({"tangent": chi} if case["tangent"] else {}), **out, twinsys=np.zeros(p.ngps, np.int32))


def _local(case):
    """Local derivatives [gp, 3, node] of the element and its weight factor:
    the one-point brick, or the 20-node brick tabulated to six decimals."""
    if case["nodes"] == 8:
        c = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1),
                      (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], float)
        return 0.125 * c.T[None], 8.0
    c = generator.BRICK20_HALF.astype(float) - 1.0
    signs = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
    t = np.zeros((8, 3, 20))
    for g, sg in enumerate(signs):
        q = 0.57735 * np.array(sg, float)
        for i, ci in enumerate(c):
            f = 1.0 + q * ci
            zero = np.flatnonzero(ci == 0)
            for j in range(3):
                u, v = (j + 1) % 3, (j + 2) % 3
                if zero.size == 0:
                    t[g, j, i] = 0.125 * ci[j] * f[u] * f[v] * (q @ ci - 2.0 + f[j])
                elif j == zero[0]:
                    t[g, j, i] = -0.5 * q[j] * f[u] * f[v]
                else:
                    m = zero[0]
                    t[g, j, i] = 0.25 * ci[j] * (1.0 - q[m] ** 2) * f[3 - j - m]
    return np.round(t, 6), 1.0


def _colours(case, p):
    """Greedy node colours in ascending (z, y, x) order."""
    if case["nodes"] == 8:
        at = np.rint(p.x.reshape(-1, 3) * np.array(_mesh(case))).astype(np.int64) & 1
        return at @ np.array([1, 2, 4])
    ln = p.ln - 1
    order = np.lexsort((np.arange(p.nnod),) + tuple(p.x.reshape(-1, 3).T))
    el = [[] for _ in range(p.nnod)]
    for e, nodes in enumerate(ln.tolist()):
        for n in nodes:
            el[n].append(e)
    col = np.full(p.nnod, -1)
    for n in order:
        used = set(col[ln[el[n]].ravel()].tolist())
        col[n] = next(c for c in range(len(used) + 1) if c not in used)
    return col


def _geometry(d, s):
    """gaussm[r, c, p, q] of tangents d and stresses s: block entry (r, c) is
    its contraction with the derivatives of the two nodes."""
    vo = [[0, 5, 4], [5, 1, 3], [4, 3, 2]]
    S = lambda p, q: s[:, vo[p][q]]
    M = torch.zeros((d.shape[0], 3, 3, 3, 3), dtype=F8, device=d.device)
    for r in range(3):
        for c in range(3):
            for p in range(3):
                for q in range(3):
                    v = d[:, vo[r][p], vo[c][q]]
                    if r == c:
                        if p == q:
                            v = v - (S(r, r) if p == r else (S(r, r) - S(p, p)) / 2.0)
                        elif r not in (p, q):
                            v = v + S(p, q) / 2.0
                    else:
                        k = 3 - r - c
                        if p == q:
                            v = v - (S(r, c) / 2.0 if p == k else S(r, c))
                        elif k not in (p, q):
                            v = v - (S(r, r) + S(c, c)) / 4.0
                        else:
                            v = v - S(c if r in (p, q) else r, k) / 4.0
                    M[:, r, c, p, q] = v
    return M


def _exact_steps(case, seed):
    p = _problem(case, seed)
    dev, c = _dev(), p.ctrl
    tab, wf = _local(case)
    tab = _t(tab)
    ln = torch.as_tensor(p.ln.astype(np.int64) - 1, device=dev)
    ne, nn = ln.shape
    npg, N = tab.shape[0], p.nnod
    le = np.repeat(p.le, npg)
    mats = [_material(m) for m in _materials(case)]
    groups = [torch.as_tensor(np.flatnonzero(le == k + 1), device=dev) for k in range(len(mats))]
    ns, nsv, G, dt = int(p.nss.max()), int(p.nsv), p.ngps, float(p.tiem[0])
    x, dx = _t(p.x).reshape(N, 3), torch.zeros((N, 3), dtype=F8, device=dev)
    sv, st = _t(p.sv[:, :nsv]), torch.zeros((G, 6), dtype=F8, device=dev)
    z = lambda *s: torch.zeros(s, dtype=F8, device=dev)
    ds, dsv, dep, srate = z(G, 6), z(G, nsv), z(G), z(G, ns)
    twin = torch.zeros(G, dtype=torch.int64, device=dev)
    # the block pattern: one entry per pair of nodes that share an element
    pair = (ln[:, :, None] * N + ln[:, None, :]).reshape(-1)
    keys, where = torch.unique(pair, return_inverse=True)
    row, col = keys // N, keys % N
    colour = torch.as_tensor(_colours(case, p), device=dev)
    plan = []
    start = torch.searchsorted(row, torch.arange(N + 1, device=dev))
    for k in range(int(colour.max()) + 1):
        rows = torch.nonzero(colour == k).squeeze(1)
        cnt = start[rows + 1] - start[rows]
        at = torch.arange(int(cnt.max()), device=dev)[None]
        idx = torch.where(at < cnt[:, None], start[rows][:, None] + at, 0)
        plan.append((rows, idx, (at < cnt[:, None]) & (col[idx] != rows[:, None]),
                     torch.searchsorted(keys, rows * N + rows)))
    xs = _t(p.x_spec[0])
    kin = torch.as_tensor((p.ib.astype(np.int64) // 100) % 100, device=dev)
    held = torch.nonzero(kin > 0).squeeze(1)
    pen = c.efix * xs[kin[held] - 1][:, [0, 1, 3, 1, 2, 4, 3, 4, 5]].reshape(-1, 3, 3)
    goal = xs[kin[held] - 1][:, [6, 10, 14]]
    free = torch.as_tensor(p.ib < 10, device=dev)
    # UPDATE_NODE adds dx = 0
    sweeps, norms = [], []
    for step in range(case["steps"]):
        J = torch.einsum("gji,eik->egjk", tab, x[ln])
        sfd = torch.einsum("egkj,gji->egik", torch.linalg.inv(J), tab).reshape(ne * npg, nn, 3)
        w = (wf * torch.linalg.det(J)).reshape(-1)
        gr = torch.einsum("qia,qib->qab", sfd, dx[ln].repeat_interleave(npg, 0))
        de = torch.stack([gr[:, 0, 0], gr[:, 1, 1], gr[:, 2, 2], gr[:, 2, 1] + gr[:, 1, 2], gr[:, 0, 2] + gr[:, 2, 0],
                          gr[:, 1, 0] + gr[:, 0, 1]], 1)
        r = torch.stack([gr[:, 2, 1] - gr[:, 1, 2], gr[:, 0, 2] - gr[:, 2, 0], gr[:, 1, 0] - gr[:, 0, 1]], 1) / 2.0
        chi, t, cp = z(G, 6, 6), z(G, 6), z(G)
        for m, gi in zip(mats, groups):
            plastic = (_mises(_rotate(r[gi], st[gi]) + ds[gi], True) > 0) & (_mises(de[gi], False) > 0)
            k = gi[~plastic]
            if k.numel():
                inv = torch.linalg.inv(_compliance(m["e"], _euler(sv[k, :3] + dsv[k, :3])[0]))
                chi[k], dep[k] = inv, 0.0
                t[k] = (inv @ de[k].unsqueeze(-1)).squeeze(-1)
            for k in torch.split(gi[plastic], 1 << 16):
                if k.numel() == 0:
                    continue
                o = _update(m, c, sv[k], dsv[k], de[k], r[k], st[k], ds[k], dt, case["mixed"])
                n1 = m["ns"]
                chi[k], t[k], dep[k], cp[k] = o["chi"], o["ds"] + st[k], o["dep"], o["err"]
                dsv[k, :3 + n1], srate[k, :n1] = o["dsv"], o["srate"]
                twin[k] = torch.where(twin[k] == 0, o["twinsys"], twin[k])
        ds = t - st
        vals, f = z(keys.numel(), 3, 3), z(N, 3)
        sg = t[:, [0, 5, 4, 5, 1, 3, 4, 3, 2]].reshape(-1, 3, 3)
        f.index_add_(0, ln.reshape(-1), torch.einsum("q,qij,qaj->qai", w, sg, sfd).reshape(ne, npg, nn, 3).sum(1)
                     .reshape(-1, 3))
        wh = where.reshape(ne, -1)
        for e0 in range(0, ne, 1 << 13):
            e1 = min(ne, e0 + (1 << 13))
            q = slice(e0 * npg, e1 * npg)
            M = _geometry(chi[q], t[q]) * w[q, None, None, None, None]
            T = torch.einsum("qrcps,qbs->qrcpb", M, sfd[q])
            Ke = torch.einsum("qap,qrcpb->qabrc", sfd[q], T).reshape(e1 - e0, npg, nn * nn, 3, 3).sum(1)
            vals.index_add_(0, wh[e0:e1].reshape(-1), Ke.reshape(-1, 3, 3))
        fc = f.clone()
        dia = torch.searchsorted(keys, held * N + held)
        vals[dia] += pen
        f[held] += (pen @ (dx[held] - goal).unsqueeze(-1)).squeeze(-1)
        sol, tol = z(N, 3), c.toler ** 2
        ready = []
        for rows, idx, off, d in plan:
            A = torch.where(off[:, :, None, None], vals[idx], 0.0).permute(0, 2, 1, 3)
            ready.append((rows, col[idx], A.reshape(len(rows), 3, -1), vals[d], f[rows]))
        for sweep in range(1, 1001):
            old = sol.clone()
            for rows, cols, A, D, rhs in ready:
                acc = (A @ sol[cols].reshape(len(rows), -1, 1)).squeeze(-1)
                v = list(sol[rows].unbind(1))
                for i in range(3):
                    rest = acc[:, i] + sum(D[:, i, j] * v[j] for j in range(3) if j != i)
                    v[i] = v[i] + 1.2 * ((rhs[:, i] - rest) / D[:, i, i] - v[i])
                sol[rows] = torch.stack(v, 1)
            if float(((sol - old) ** 2).sum() / (sol ** 2).sum()) < tol:
                break
        size = float(dx.norm())
        sdx = c.toler if size == 0.0 else float(sol.norm()) / size
        alp = 1.0 / (1.0 + c.alpha * sdx)
        sweeps.append(sweep)
        norms.append([sdx, float(f[free].norm()), float(cp.mean()), alp])
        x, dx = x - alp * sol, dx - alp * sol
    host = dict(x=x.reshape(-1), dx=dx.reshape(-1), ddx=sol.reshape(-1), fc=fc.reshape(-1), ds=ds, dsv=dsv, de=de,
                dr=r, dep=dep, srate=srate)
    out = dict(sor_sweeps=np.array(sweeps, np.int64), norms=np.array(norms))
    out.update({k: v.cpu().numpy() for k, v in host.items()}, twinsys=twin.cpu().numpy().astype(np.int32))
    return out


def _exact_adjoint(case, seed):
    p, h = _problem(case, seed), _history(case, seed)
    mat, n, ninc = _material(_materials(case)[0]), case["n"], case["ninc"]
    ns, q = mat["ns"], _t(np.array(h["q"]) / np.linalg.norm(h["q"]))
    sv, st = _t(p.sv[:, :3 + ns]), _t(p.st)
    de, dr, w, y = (_t(h[k]) for k in ("de", "dr", "w", "y"))
    kept = []
    for i in range(ninc):
        S = _compliance(mat["e"], _euler(sv[:, :3])[0])
        o = _update(mat, p.ctrl, sv, torch.zeros_like(sv), de[i], dr[i], st, torch.linalg.solve(S, de[i]),
                    float(h["dt"][i]))
        kept.append((st, sv, st + o["ds"], o["xg"]))
        st, sv = st + o["ds"], sv + o["dsv"]
    qq = torch.stack([q[PI[k]] * q[PJ[k]] for k in range(6)])

    def strain(v):
        return (qq * (_compliance(mat["e"], _euler(v[6:9])[0]) @ v[:6])).sum()

    end = torch.cat([st, sv[:, :3]], 1)
    e = torch.func.vmap(strain)(end)
    J = float((0.5 * w * (e - y) ** 2).sum())
    seed_ = (w * (e - y))[:, None] * torch.func.vmap(torch.func.grad(strain))(end)
    bar = torch.cat([seed_, torch.zeros((n, ns), dtype=F8, device=q.device)], 1)   # stress, angles, resistances
    pbar = torch.zeros(4, dtype=F8, device=q.device)

    def system(v, act, dei, ri, dt):
        """Residuals of the local system and the increment's outputs from
        v = (stress, slips, old stress, angles, resistances, parameters)."""
        s, g, s_old, ph, s0, pr = torch.split(v, [6, ns, 6, 3, ns, 4])
        a, aug = _euler(ph)
        (b, rot), gz = _systems(mat, a), torch.where(act, g, 0.0)
        s1, _ = _harden(mat, s0, gz, pr)
        tau = torch.where(act, b @ s, 1.0)
        Ra = torch.log(tau.abs()) - torch.log(s1) - (mat["am"] + pr[0]) * torch.log(torch.where(act, g, 1.0).abs() / dt)
        Rs = dei - gz @ b - _compliance(mat["e"], a) @ (s - _rotate(ri, s_old))
        rtn = gz @ rot - ri
        rx = a @ rtn
        d1 = torch.where(aug[2].abs() < 1e-5, rtn[2], (aug[0] * rx[0] + aug[1] * rx[1]) / aug[2])
        turn = torch.stack([d1, aug[1] * rx[0] - aug[0] * rx[1], rx[2] - d1 * a[2, 2]])
        return torch.cat([Rs, torch.where(act, Ra, g), s, ph + turn, s1])

    nx, jac = 6 + ns, torch.func.vmap(torch.func.jacfwd(system), in_dims=(0, 0, 0, 0, None), chunk_size=4096)
    for i in reversed(range(ninc)):
        zst, zsv, s, g = kept[i]
        v = torch.cat([s, g, zst, zsv, torch.zeros((n, 4), dtype=F8, device=q.device)], 1)
        D = jac(v, g != 0.0, de[i], dr[i], float(h["dt"][i]))
        R, Y = D[:, :nx], D[:, nx:]
        rhs = (Y.transpose(1, 2) @ bar.unsqueeze(-1)).squeeze(-1)
        lam = torch.linalg.solve(R[:, :, :nx].transpose(1, 2), rhs[:, :nx])
        full = rhs[:, nx:] - (R[:, :, nx:].transpose(1, 2) @ lam.unsqueeze(-1)).squeeze(-1)
        bar, pbar = full[:, :9 + ns], pbar + full[:, 9 + ns:].sum(0)
    g_sv, g_amp = np.zeros((n, abi.FAS_MAXSVS)), np.zeros((1, 10))
    g_sv[:, :3 + ns] = bar[:, 6:].cpu().numpy()
    g_amp[0, [0, 1, 2, 4]] = pbar.cpu().numpy()
    return dict(st=bar[:, :6].cpu().numpy(), sv=g_sv, ampar=g_amp, J=J)


@functools.lru_cache(maxsize=1)
def _exact(key, seed):
    case = dict(key)
    if case["kind"] == "points":
        return _exact_points(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    # a whole increment is many solves one after the other: minutes here
    return _exact_steps(case, seed) if case["steps"] else None


def exact(case, seed):
    return _exact(tuple((k, v) for k, v in sorted(case.items()) if k != "name"), seed)
