"""The energy sums over the units' rows at the edges of their tiles: the sums
do not depend on the room of the buffers, and are the FP64 oracle's."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# 300 waters: under one tile of 2,048 rows; 1,500: units around it; 4,000: several
@pytest.mark.parametrize("waters", [300, 1500, 1700, 4000])
def test_energies_are_the_oracles_and_reproducible(cuda, waters):
    from mdir_b200 import NonbondedTerm, systems
    s = systems.tip3p(waters=waters, seed=5)
    x = torch.tensor(s["positions"], device=cuda)
    seen = []
    for reach in (s["reach"], s["reach"], 1.3):  # the last: more room than its lists at the reach below need
        t = NonbondedTerm(len(s["charges"]))
        t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
        t.set_exclusions(pairs=s["excluded_pairs"])
        t.set_interaction(s["cutoff"], min(reach, 0.95 * float(s["box"][0])), s["beta"])
        t.set_pme(s["grid"], s["order"])
        t.build(x, s["box"])
        t.set_reach(s["reach"])
        sizes = t.build(x, s["box"])
        for _ in range(2):  # the sums replace rows: a second evaluation writes them again
            t.force(x, energy=True)
            e = t.energies()
            seen.append([e[k] for k in ("lj", "coulomb", "excluded")] + list(e["virial_pair"].reshape(-1)))
        assert sizes[2] > 0
        t.close()
    for row in seen[1:]:
        np.testing.assert_array_equal(seen[0], row)
    ref = O.evaluate(s, s["positions"])["terms"]
    scale = sum(abs(ref[k]) for k in ("lj", "coulomb", "excluded"))
    for value, k in zip(seen[0], ("lj", "coulomb", "excluded")):
        assert abs(value - ref[k]) <= 1e-6 * scale


def test_batch_constants_follow_the_charges(cuda):
    from mdir_b200 import systems
    from mdir_b200.batch import BatchEvaluator
    frames = systems.batch_frames(count=5, low=1000, high=2000, seed=8)
    ev = BatchEvaluator(frames)
    ev.force(energy=True)
    e = ev.energies()
    for k, f in enumerate(frames):
        q = np.asarray(f["charges"])
        want = -systems.COULOMB * f["beta"] / np.sqrt(np.pi) * np.sum(q * q)
        assert abs(e["self"][k] - want) <= 1e-12 * abs(want)
    ev.close()
