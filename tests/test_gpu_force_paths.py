"""A force call's routes: the reciprocal chain beside the pairs or after them
(by size), the finish that gathers (orders 4 and 8) and the one that does not,
accumulated and fresh forces, atoms with no place, streams."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def term(s, order, deterministic, grid=None):
    from mdir_b200 import NonbondedTerm
    t = NonbondedTerm(len(s["charges"]))
    t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
    t.set_exclusions(pairs=s["excluded_pairs"])
    t.set_interaction(s["cutoff"], s["reach"], s["beta"])
    t.set_pme(grid if grid is not None else s["grid"], order)
    t.set_deterministic(deterministic)
    return t


def close(a, b, tol):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    return np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


# below and above the sizes from which the chain runs beside (2,000 atoms with
# energies, 6,000 without) and the units of a warp are whole (about 4,000)
@pytest.mark.parametrize("waters", [300, 1300, 1999, 2000, 2700])
@pytest.mark.parametrize("order", [4, 5, 6, 8])
@pytest.mark.parametrize("deterministic", [False, True])
def test_the_call_is_the_sum_of_its_parts(cuda, waters, order, deterministic):
    from mdir_b200 import systems
    s = systems.tip3p(waters=waters, seed=2, order=order)
    t = term(s, order, deterministic)
    x = torch.tensor(s["positions"], device=cuda)
    t.build(x, s["box"])
    parts = [t.force(x, pairs=p, pme=q, excluded=e) for p, q, e in
             ((True, False, False), (False, True, False), (False, False, True))]
    total = sum(parts)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        moved = x + 0.0
        for energy in (False, True):
            f = t.force(moved, energy=energy, potential=True)
            # f32 accumulators of the parts against their sum: each term rounds by 2^-24 of it
            assert close(f, total, 2e-6)
            base = torch.full_like(f, 3.0)
            t.force(moved, energy=energy, forces=base, accumulate=True)
            assert close(base - 3.0, total, 2e-6)
        pot = t.potential(side)
    side.synchronize()
    e_rec = 0.5 * float((torch.as_tensor(s["charges"], device=cuda) * pot).sum())
    t.force(x, energy=True)
    # the reciprocal energy is half the charges' potential
    assert abs(e_rec - t.energies()["reciprocal"]) <= 1e-5 * abs(e_rec) + 1e-6 * abs(t.energies()["excluded"])
    t.close()


@pytest.mark.parametrize("pme", [True, False])
@pytest.mark.parametrize("order", [4, 6])
def test_an_atom_with_no_place_gets_zeros(cuda, pme, order):
    from mdir_b200 import systems
    s = systems.tip3p(waters=2200, seed=2, order=order)
    t = term(s, order, False)
    x = torch.tensor(s["positions"], device=cuda)
    bad = x.clone()
    bad[[5, 4000]] = float("nan")
    t.build(bad, s["box"], allow_nan=True)
    f = torch.full_like(x, 7.0)
    t.force(bad, forces=f, pme=pme)
    assert torch.equal(f[[5, 4000]], torch.zeros(2, 3, dtype=torch.float64, device=cuda))
    assert bool(torch.isfinite(f).all())
    kept = torch.full_like(x, 7.0)
    t.force(bad, forces=kept, pme=pme, accumulate=True)
    assert torch.equal(kept[[5, 4000]], torch.full((2, 3), 7.0, dtype=torch.float64, device=cuda))
    t.close()


def test_calls_captured_in_a_graph_replay(cuda):
    from mdir_b200 import systems
    s = systems.tip3p(waters=2200, seed=2)
    t = term(s, 4, True)
    x = torch.tensor(s["positions"], device=cuda)
    t.build(x, s["box"])
    out = torch.empty_like(x)
    t.force(x, forces=out)  # its lazy tables, outside the capture
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t.force(x, forces=out)
    want = []
    for shift in (0.0, 0.002):
        x += shift
        want.append(t.force(x).clone())
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[-1])  # fixed-point sums: the same bits
    t.close()


@pytest.mark.parametrize("waters", [600, 2200])  # without and with a stream of its own for the chain
def test_a_first_call_in_a_graph_and_a_sum_set_after_the_build(cuda, waters):
    from mdir_b200 import systems
    s = systems.tip3p(waters=waters, seed=2)
    x = torch.tensor(s["positions"], device=cuda)
    t = term(s, 4, True)
    t.build(x, s["box"])
    t.force(x, energy=True)
    want = t.force(x).clone()  # fixed-point sums: the same bits on every route
    late = term(s, 4, True)
    late.set_pme((0, 0, 0), 4)
    late.build(x, s["box"])
    late.set_pme(s["grid"], 4)
    assert torch.equal(late.force(x), want)
    first = term(s, 4, True)
    first.build(x, s["box"])
    out = torch.empty_like(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        first.force(x, forces=out)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    for k in (t, late, first):
        k.close()
