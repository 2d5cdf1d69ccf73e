"""The pairs' virial in the deterministic mode on systems whose groups of 16
places are long (a few clusters in a wide box): as accurate as pair by pair in
f32, whatever the distance between the clusters."""

import numpy as np
import pytest
import torch
from scipy.special import erfc

from mdir_b200 import NonbondedTerm

pytestmark = pytest.mark.gpu

COULOMB, SIGMA, EPSILON, CHARGE = 138.935457644, 0.3405, 0.996, 0.5


def clusters(n, L, seed):
    """n / 4 tetrahedra at contact distances, one a cell of a coarse lattice."""
    rng = np.random.default_rng(seed)
    m = n // 4
    k = int(np.ceil(m ** (1 / 3)))
    at = rng.permutation(k ** 3)[:m]
    c = np.stack([at // (k * k), at // k % k, at % k], -1) + rng.uniform(0.3, 0.7, (m, 3))
    tet = 0.27 * np.array([[0, 0, 0], [1, 1, 0], [1, 0, 1], [0, 1, 1]])
    return (c[:, None] * (L / k) + tet + rng.uniform(-0.02, 0.02, (m, 4, 3))).reshape(-1, 3)


@pytest.mark.parametrize("n,L", [(32, 60.0), (32, 150.0), (256, 20.0), (256, 150.0), (4096, 60.0)])
@pytest.mark.parametrize("coulomb", [False, True])
def test_the_virial_keeps_its_digits_in_long_groups(cuda, n, L, coulomb):
    beta = 3.0 if coulomb else 0.0
    eps = 0.0 if coulomb else EPSILON
    a, b = np.triu_indices(4, 1)  # the clusters are out of each other's reach
    i, j = [(4 * np.arange(n // 4)[:, None] + side).reshape(-1) for side in (a, b)]
    errors = []
    for seed in range(8):
        x = clusters(n, L, seed)
        # 0.5 is exact in f32
        q = np.random.default_rng(seed + 100).choice([-CHARGE, CHARGE], n) if coulomb else np.zeros(n)
        t = NonbondedTerm(n)
        t.set_particles(q, np.zeros(n, dtype=np.int32), np.array([[SIGMA]]), np.array([[eps]]))
        t.set_interaction(1.0, 1.1, beta)
        t.set_deterministic(True)
        xd = torch.tensor(x, device=cuda)
        t.build(xd, [L] * 3)
        t.force(xd, energy=True)
        got = np.asarray(t.energies()["virial_pair"])
        t.close()
        d = x[i] - x[j]
        r2 = np.sum(d * d, 1)
        r, s6 = np.sqrt(r2), (SIGMA ** 2 / r2) ** 3
        fs = 24 * eps * (2 * s6 * s6 - s6) / r2
        if coulomb:
            fs = COULOMB * q[i] * q[j] * (erfc(beta * r) / r + 2 * beta / np.sqrt(np.pi) * np.exp(-beta ** 2 * r2)) / r2
        want = np.einsum("p,pa,pb->ab", fs, d, d)
        errors.append(np.abs(got - want).max() / np.sum(np.abs(fs) * r2))
    # a pair: three roundings of 2^-24 in r^2, made up to 7 times larger by
    # 1/r^14, and some of the products: 40 of them at most, of either sign, so
    # their mean falls with the root of the pairs; 1.5 for the approximate 1/r
    # and erfc, which may lean one way.  Sums of forces over a group of 150 nm
    # were off by some 20 of 2^-24.
    assert np.sqrt(np.mean(np.square(errors))) <= (40 / np.sqrt(len(i)) + 1.5) * 2.0 ** -24
