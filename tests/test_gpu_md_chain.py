"""The MD step with one list and no reciprocal sum: its graph is a chain of
pairs and updates alone, where the pair kernel's wait is all that orders an
update's early loads of the state after the stores of the update before it."""

import numpy as np
import pytest
import torch

from mdir_b200 import NonbondedTerm, systems
from mdir_b200.md import Integrator

pytestmark = pytest.mark.gpu


def run(s, waters, temperature, tau, steps, unroll):
    n = len(s["charges"])
    t = NonbondedTerm(n)
    t.set_particles(np.zeros(n), s["types"], s["sigma"], s["epsilon"])
    if waters is not None:
        t.set_exclusions(pairs=s["excluded_pairs"])
    t.set_interaction(s["cutoff"], s["reach"], 0.0)
    t.set_deterministic(True)
    md = Integrator(t, s["masses"], waters)
    md.thermostat(temperature, tau, 1)
    x = torch.tensor(s["positions"], dtype=torch.float64, device="cuda")
    v = torch.tensor(systems.maxwell_velocities(s, temperature, seed=2), device="cuda")
    md.build(x, s["box"])
    md.run(x, v, s["box"], 0.002, steps, unroll=unroll)
    return x, v, md.thermo()


# free atoms in one wave of blocks and in several, with and without the
# thermostat's scaling (read early too); rigid waters
@pytest.mark.parametrize("kind,tau,steps", [("argon", 0.0, 3000), ("argon", 0.1, 3000), ("argon-large", 0.0, 400),
                                            ("waters", 0.1, 1000)])
def test_the_chain_without_pruning_or_pme_is_the_step_by_step_run(cuda, kind, tau, steps):
    if kind == "waters":
        s = systems.tip3p(waters=500, seed=31)
        args = (s, s["waters"], 300.0)
    else:
        s = systems.argon() if kind == "argon" else systems.argon(cells=16, length=3.47 * 16 / 6)
        args = (s, None, 120.0)
    x1, v1, t1 = run(*args, tau, steps, 10)  # the graphs
    x2, v2, t2 = run(*args, tau, steps, 0)  # a step at a time, the host waiting for each
    assert t1["steps"] == t2["steps"] == steps and t1["builds"] == t2["builds"] > 1
    assert torch.equal(x1, x2) and torch.equal(v1, v2)


@pytest.mark.parametrize("factor", [1.5, 3.0, 0.75])
@pytest.mark.parametrize("window_drift", [0.0071, 0.0113, 0.0197, 0.0411])
def test_the_rebuild_decision_counts_the_first_window_two_thirds(cuda, factor, window_drift):
    """Atoms without forces, all of one speed: the drift grows by the same
    amount in every window, and the builds are those of the rule's own
    arithmetic (the largest drift so far, plus its growth over the last window
    times the factor, two thirds of it after a build's first window, plus
    0.002 nm, against half the skin)."""
    s = systems.argon(skin=0.2)
    n, dt, unroll, windows = len(s["charges"]), 0.002, 10, 60
    t = NonbondedTerm(n)
    t.set_particles(np.zeros(n), s["types"], s["sigma"], np.zeros_like(s["epsilon"]))
    t.set_interaction(s["cutoff"], s["reach"], 0.0)
    md = Integrator(t, s["masses"])
    md.thermostat(120.0, 0.0, 1)
    md.lookahead(factor)
    x = torch.tensor(s["positions"], dtype=torch.float64, device="cuda")
    d = np.random.default_rng(3).normal(size=(n, 3))
    d *= window_drift / (dt * unroll) / np.linalg.norm(d, axis=1)[:, None]
    v = torch.tensor(d, device="cuda")
    md.build(x, s["box"])
    before = md.thermo()["builds"]
    md.run(x, v, s["box"], dt, windows * unroll, unroll=unroll)
    builds, drift, last = 0, 0.0, 0.0
    for _ in range(windows):
        drift += window_drift
        growth = (drift - last) * factor * (2.0 / 3.0 if last == 0.0 else 1.0)
        if drift + growth + 0.002 > 0.1:
            builds, drift, last = builds + 1, 0.0, 0.0
        else:
            last = drift
    th = md.thermo()
    assert th["redone"] == 0 and th["builds"] - before == builds > 0
