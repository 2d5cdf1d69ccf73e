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


def test_constants_follow_the_charges_set_again(cuda):
    """The sums of the charges are kept where they are set: a second set of
    charges (here of a net charge of 0.8 a system) replaces them, in a batch and
    in a context, in the constants and in the energy gradient's background."""
    from mdir_b200 import NonbondedTerm, systems
    from mdir_b200 import _lib as L
    from mdir_b200.batch import BatchEvaluator
    from mdir_b200.term import _hp
    frames = systems.batch_frames(count=5, low=1000, high=2000, seed=8)

    def wanted(f, q):
        V = float(np.prod(f["box"]))
        return (-systems.COULOMB * f["beta"] / np.sqrt(np.pi) * np.sum(q * q),
                -systems.COULOMB * np.pi * np.sum(q) ** 2 / (2 * V * f["beta"] ** 2))

    ev = BatchEvaluator(frames)
    old = [np.asarray(f["charges"]) for f in frames]
    new = [1.1 * q + 0.8 / len(q) for q in old]
    types = np.ascontiguousarray(np.concatenate([f["types"] for f in frames]), dtype=np.int32)
    sigma, epsilon = (np.ascontiguousarray(frames[0][k], dtype=np.float64) for k in ("sigma", "epsilon"))
    for charges in (old, new, old):
        q = np.ascontiguousarray(np.concatenate(charges), dtype=np.float64)
        L.check(L.lib().mdrtNbBatchSetParticles(ev._h, _hp(q), _hp(types), len(sigma), _hp(sigma), _hp(epsilon)),
                "mdrtNbBatchSetParticles")
        ev.force(energy=True)
        e = ev.energies()
        for k, (f, q) in enumerate(zip(frames, charges)):
            for got, want in zip((e["self"][k], e["background"][k]), wanted(f, q)):
                assert abs(got - want) <= 1e-12 * abs(want) + 1e-15, (k, got, want)
    ev.close()
    f, q0, q1 = frames[0], old[0], new[0]
    x = torch.tensor(f["positions"], device=cuda)

    seen = []
    for sequence in ((q0, q1), (q1,)):
        t = NonbondedTerm(len(q0))
        t.set_exclusions(pairs=f["excluded_pairs"])
        t.set_interaction(f["cutoff"], f["reach"], f["beta"])
        t.set_pme(f["grid"], f["order"])
        for q in sequence:
            t.set_particles(q, f["types"], f["sigma"], f["epsilon"])
            t.build(x, f["box"])
            c = t.constants(f["box"])
            for got, want in zip((c["self"], c["background"]), wanted(f, q)):
                assert abs(got - want) <= 1e-12 * abs(want) + 1e-15
            dq, _ = t.parameter_gradient(x)
        seen.append(dq)
        t.close()
    # f32 pair terms summed by atomics in two orders: 1e-6 of the norm
    assert float((seen[0] - seen[1]).norm()) <= 1e-6 * float(seen[1].norm())
