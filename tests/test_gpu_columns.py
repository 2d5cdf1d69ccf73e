"""The columns' first groups by one block and, past 8,192 columns, by a count
and a scan: flat boxes and batches on both sides of that edge."""

import numpy as np
import pytest
import torch

from mdir_b200 import _lib as L
from tests.test_gpu_search import canon5, near

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 65), (90, 91), (91, 91), (130, 127)])
def test_flat_boxes_hold_every_pair(cuda, nx, ny):
    from mdir_b200 import NonbondedTerm
    d, R = 0.5, 0.18  # a column's edge: the side of 16 atoms' cube
    box = np.array([nx * d * 1.003, ny * d * 1.003, 0.6])
    n = int(16 * box.prod() / d ** 3)
    x = np.random.default_rng(nx).uniform(0, 1, (n, 3)) * box
    t = NonbondedTerm(n)
    t.set_interaction(R, R, 0.0)
    sizes = t.build(torch.tensor(x, device=cuda), box)
    got = canon5(t.pair_images(sizes))
    order = t.buffer(L.SLOT_ORDER, np.int32)[: 16 * sizes[6]]
    t.close()
    np.testing.assert_array_equal(np.sort(order[order >= 0]), np.arange(n))  # every atom has one place
    # the lists' reach is R' = R + 3e-6 (the edges) in f32: every pair well
    # inside is there, none well outside (1e-5 nm: several f32 spacings)
    rows = lambda r: set(map(bytes, np.ascontiguousarray(r)))  # noqa: E731
    wide = R + 3e-6 * box.sum()
    have = rows(got)
    assert len(have) == len(got)
    assert rows(near(x, list(box), wide - 1e-5)) <= have <= rows(near(x, list(box), wide + 1e-5))


def test_a_batch_is_its_halves(cuda):
    from mdir_b200 import systems
    from mdir_b200.batch import BatchEvaluator
    frames = systems.batch_frames(count=520, low=1026, high=1100, seed=12)  # 16 columns a frame
    energies = []
    for part in (frames, frames[:260], frames[260:]):
        ev = BatchEvaluator(part)
        ev.force(energy=True)
        energies.append(ev.energies())
        ev.close()
    whole, *halves = energies
    # the same lists entry for entry: each frame's units sum to the same bits
    for term in ("lj", "coulomb"):
        np.testing.assert_array_equal(whole[term], np.concatenate([h[term] for h in halves]))
