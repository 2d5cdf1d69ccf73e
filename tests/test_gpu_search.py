"""The search of the neighbor build at the sizes and positions where its
window, chunks and warps a group change: places on column and bin edges, one
warp a group (large systems) and four, images through tilted cells."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_neighbors import canon, device_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,spacing,R", [(4.0, 0.5, 1.0), (4.0, 0.25, 0.75), (3.0, 0.5, 2.9), (2.4, 0.3, 0.6)])
def test_places_on_column_and_bin_edges(cuda, L, spacing, R):
    g = np.arange(int(round(L / spacing))) * spacing
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(3)
    x = x + L * rng.integers(-1, 2, size=x.shape)  # whole cells: 0 and L alike
    x[::7] = np.nextafter(x[::7], -10.0)  # and just below an edge
    t, sizes, pairs = device_pairs(x, L, R, None)
    count, ref = O.pairset(x, [L, L, L], R, None)
    assert len(pairs) == count
    np.testing.assert_array_equal(canon(pairs), canon(ref))
    t.close()


def near(x, cell, R):
    """Sorted rows (i, j, na, nb, nc), i < j, with |x_i - x_j - n H| <= R in f64."""
    from scipy.spatial import cKDTree
    H = O.cell_matrix(cell) if len(cell) == 6 else np.diag(cell)
    n = len(x)
    f = np.floor(x @ np.linalg.inv(H))  # x = home + f H
    home = x - f @ H
    inv = np.linalg.inv(H)
    margin = R * np.linalg.norm(inv, axis=0)
    rows = []
    tree = cKDTree(home)
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                s = np.array([a, b, c])
                fr = (home @ inv) + s
                keep = np.nonzero(np.all((fr > -margin) & (fr < 1 + margin), axis=1))[0]
                if len(keep) == 0:
                    continue
                hits = tree.query_ball_point(home[keep] + s @ H, R)
                j = np.repeat(keep, [len(h) for h in hits])
                i = np.concatenate([np.asarray(h, dtype=np.int64) for h in hits]) if len(j) else j
                sel = i < j
                i, j = i[sel], j[sel]
                # x_j's image: home_j + s H = x_j + (s - f_j) H, seen from x_i = home_i + f_i H
                rows.append(np.concatenate([i[:, None], j[:, None], s - f[j] + f[i]], axis=1))
    return canon5(np.concatenate(rows))


def canon5(r):
    r = np.asarray(r).astype(np.int64)
    return r[np.lexsort(tuple(r[:, k] for k in range(4, -1, -1)))]


@pytest.mark.parametrize("n", [63984, 64016, 70001])  # the last groups with four warps each, the first with one
@pytest.mark.parametrize("tilts", [(), (2.8, -2.7, 2.2)])
def test_large_lists_hold_every_pair(cuda, n, tilts):
    from mdir_b200 import NonbondedTerm
    rng = np.random.default_rng(n)
    edge = (n / 100.0) ** (1 / 3)
    cell = [edge, 1.01 * edge, 0.99 * edge, *[v * edge / 8.7 for v in tilts]]
    H = O.cell_matrix(cell) if tilts else np.diag(cell)
    x = rng.uniform(0, 1, (n, 3)) @ H + rng.integers(-1, 2, (n, 3)) @ H
    R = 0.45
    t = NonbondedTerm(n)
    t.set_interaction(cutoff=R, reach=R, beta=0.0)
    excluded = np.stack([np.arange(0, n - 1, 2), np.arange(1, n, 2)], 1)
    t.set_exclusions(pairs=excluded)
    sizes = t.build(torch.tensor(x, dtype=torch.float64, device="cuda"), cell)
    got = canon5(t.pair_images(sizes))
    t.close()
    assert len(np.unique(got, axis=0)) == len(got)
    # the lists' reach is R' = R + 3e-6 (the cell's numbers) in f32: every pair
    # well inside is there, none well outside (1e-5 nm: ten f32 spacings)
    wide = 3e-6 * sum(abs(v) for v in cell)
    key = lambda r: set(map(tuple, r.tolist()))  # noqa: E731
    free = lambda r: r[~((r[:, 0] % 2 == 0) & (r[:, 1] == r[:, 0] + 1))]  # noqa: E731
    have = key(got)
    assert key(free(near(x, cell, R + wide - 1e-5))) <= have
    assert have <= key(free(near(x, cell, R + wide + 1e-5)))


def test_lists_of_one_and_four_warps_a_group_sum_to_the_same_bits(cuda):
    from mdir_b200 import systems
    from mdir_b200.batch import BatchEvaluator
    frames = systems.batch_frames(count=7, low=1000, high=4000, seed=11)
    lists = []
    for warps in (1, 4):
        ev = BatchEvaluator(frames)
        ev.set_tuning(search_warps=warps)
        ev.build()
        ev.force(energy=True)
        lists.append(ev.energies())
        ev.close()
    # a batch shows no lists; a unit's energies and virial are f32 sums over its
    # entries in their order, so that another entry or order would change bits
    for term in ("lj", "coulomb"):
        np.testing.assert_array_equal(lists[0][term], lists[1][term])


@pytest.mark.parametrize("waters,reach", [(300, 1.0), (1200, 1.0), (1200, 1.6), (2671, 1.2)])
@pytest.mark.parametrize("seldom", [False, True])
def test_lj_partners_first_is_the_stable_partition(cuda, waters, reach, seldom):
    """Without a pruned reach a group's entries of a partner with LJ terms come
    first, each part in the order found (the lists of a context with a pruned
    reach); `seldom`: one atom in 30 has them, so the part that moves down
    overlaps where it lies in a row that is more than half full."""
    from mdir_b200 import NonbondedTerm, systems
    from mdir_b200 import _lib as Lb
    s = systems.tip3p(waters=waters, seed=9)
    types = np.asarray(s["types"]).copy()
    if seldom:
        types[:] = 1
        types[::30] = 0
    x = torch.tensor(s["positions"], device="cuda")
    rows = []
    for dual in (True, False):
        t = NonbondedTerm(len(s["charges"]))
        t.set_particles(s["charges"], types, s["sigma"], s["epsilon"])
        t.set_exclusions(pairs=s["excluded_pairs"])
        t.set_interaction(s["cutoff"], min(reach, 0.99 * float(s["box"][0])), s["beta"])
        if dual:
            t.set_pruned_reach(0.95)
        sizes = t.build(x, s["box"])
        G, cap = sizes[6], t.info()["list_capacity"]
        e = t.buffer(Lb.SLOT_ENTRIES, np.int32, 2)[: G * cap].reshape(G, cap, 2)
        c = t.buffer(Lb.SLOT_COUNTS, np.int32)[:G]
        order = t.buffer(Lb.SLOT_ORDER, np.int32)
        rows.append([e[g, : c[g]].copy() for g in range(G)])
        t.close()
    for found, first in zip(*rows):
        lj = types[order[found[:, 0]]] == 0
        np.testing.assert_array_equal(np.concatenate([found[lj], found[~lj]]), first)
