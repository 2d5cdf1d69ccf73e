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
