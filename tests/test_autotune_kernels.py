"""The autotuner times the kernels that its defines act on (CPU: a recording
stand-in for the solver): solves with one launch per colour, and materials that
the general constitutive kernels serve."""
import numpy as np

from cpfem_code_b200 import abi, autotune, generator, solver


def _group_rule(p):
    """Whether every material has one latent hardening number (the rule of the group pass)."""
    out = []
    for m, ns in enumerate(p.nss):
        s = p.smatrx[m, :ns, :ns].T
        out.append(len(np.unique(s[~np.eye(ns, dtype=bool)])) == 1)
    return all(out)


def test_measure_runs_the_tuned_kernels(monkeypatch, tmp_path):
    solves, passes = [], []

    class Recorder:
        def __init__(self, p, mode=0):
            self.p, self.mode = p, mode

        def facsls(self):
            solves.append(self.mode)
            return 10, 0.0

        def constitutive(self, inc, nit):
            passes.append(self.p)

        def elvals(self, inc, nit):
            if inc == 2:
                passes.append(self.p)

        def download(self, p):
            return p

        def profile(self, k):
            return dict(ms_total=1.0, ms_constitutive=1.0)

        def __getattr__(self, name):
            return lambda *a, **k: None

    monkeypatch.setattr(autotune, "n_libs", lambda: 1)
    monkeypatch.setattr(autotune, "_load", lambda path: None)
    monkeypatch.setattr(autotune, "TUNE_DIR", str(tmp_path))
    monkeypatch.setattr(autotune, "MEASURE", str(tmp_path / "measure.json"))
    monkeypatch.setattr(solver, "GpuSolver", Recorder)
    batch = generator.point_batch
    monkeypatch.setattr(generator, "workload", lambda name: batch(4, seed=2))
    monkeypatch.setattr(generator, "point_batch", lambda n, seed: batch(4, seed=seed))
    autotune.measure()
    assert solves and all(m & abi.FAS_MODE_SOR_COLOUR for m in solves)
    assert {m & abi.FAS_MODE_SOR_FP32 for m in solves} == {0, abi.FAS_MODE_SOR_FP32}
    assert passes and not any(_group_rule(p) for p in passes)
    assert _group_rule(batch(4, seed=1))
