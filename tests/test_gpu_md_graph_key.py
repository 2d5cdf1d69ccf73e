"""The step graph is captured again when a parameter that its launches take
changes: a run after the change is, bit for bit in the deterministic mode, the
run of an integrator made with the new parameters."""

import numpy as np
import pytest
import torch

from mdir_b200 import NonbondedTerm, systems
from mdir_b200.md import Integrator

pytestmark = pytest.mark.gpu


def made(s):
    t = NonbondedTerm(len(s["charges"]))
    t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
    t.set_exclusions(pairs=s["excluded_pairs"])
    t.set_interaction(s["cutoff"], 1.3, s["beta"])
    t.set_pme(s["grid"], s["order"])
    t.set_deterministic(True)
    t.set_pruned_reach(0.95)
    md = Integrator(t, s["masses"], s["waters"])
    md.thermostat(300.0, 0.0, 1)
    return t, md


def change(t, s, what):
    if what == "reach":
        t.set_reach(1.02)
    elif what == "interaction":
        t.set_interaction(0.8, 1.3, 1.1 * s["beta"])
    elif what == "coulomb":
        t.set_interaction(s["cutoff"], 1.3, s["beta"], coulomb=100.0)
    elif what == "types":  # the same atoms in four types, a mixed table instead of one that factorizes
        types = np.asarray(s["types"]) + 2 * (np.arange(len(s["types"])) % 2)
        sigma = np.tile(np.asarray(s["sigma"]), (2, 2)) * np.array([1.0, 1.0, 1.01, 1.0])[:, None]
        sigma = 0.5 * (sigma + sigma.T)
        t.set_particles(s["charges"], types, sigma, np.tile(np.asarray(s["epsilon"]), (2, 2)))
    elif what == "exclusions":  # the same, in new buffers
        t.set_exclusions(pairs=s["excluded_pairs"])
    elif what == "grid":
        t.set_pme([k + 8 for k in s["grid"]], s["order"])


@pytest.mark.parametrize("what", ["reach", "interaction", "coulomb", "types", "exclusions", "grid"])
def test_a_run_after_a_change_is_a_fresh_integrators(cuda, what):
    s = systems.tip3p(waters=500, seed=33)
    v0 = systems.maxwell_velocities(s, 300.0, seed=2)
    seen = []
    for runs_before in (True, False):
        t, md = made(s)
        x = torch.tensor(s["positions"], dtype=torch.float64, device="cuda")
        v = torch.tensor(v0, device="cuda")
        if runs_before:
            md.build(x, s["box"])
            md.run(x, v, s["box"], 0.002, 20, unroll=10)
            x.copy_(torch.as_tensor(s["positions"]))
            v.copy_(torch.as_tensor(v0))
        change(t, s, what)
        before = md.thermo()["builds"]
        md.build(x, s["box"])
        md.run(x, v, s["box"], 0.002, 100, unroll=10)
        seen.append((x.clone(), v.clone(), md.thermo()["builds"] - before))
        md.close()
        t.close()
    (x1, v1, b1), (x2, v2, b2) = seen
    assert torch.equal(x1, x2) and torch.equal(v1, v2) and b1 == b2
