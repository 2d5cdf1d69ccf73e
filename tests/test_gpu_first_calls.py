"""First calls on a non-blocking stream while the null stream is busy: the
scratch they allocate is cleared in the order of their own stream."""

import numpy as np
import pytest

from mdir_b200 import NonbondedTerm, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("busy_ms", [0.5, 1.0, 2.0])
def test_the_first_gradient_beside_a_busy_null_stream(cuda, busy_ms):
    import torch
    s, X, _ = systems.force_matching(frames=100, waters=2000)
    t = NonbondedTerm(len(s["charges"]))
    t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
    t.set_exclusions(pairs=s["excluded_pairs"])
    t.set_interaction(s["cutoff"], s["reach"], s["beta"])
    t.set_pme(s["grid"], s["order"])
    x = torch.as_tensor(X, device=cuda)
    g = torch.randn(x.shape, dtype=torch.float64, device=cuda, generator=torch.Generator(cuda).manual_seed(3))
    nt = len(s["type_sigma"])
    side = torch.cuda.Stream()
    t.build(x[0], s["box"], stream=side)
    sums = []
    for call in range(2):
        dq = torch.zeros(t.n, dtype=torch.float64, device=cuda)
        dtable = torch.zeros((2, nt, nt), dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        if call == 0:
            torch.cuda._sleep(int(1.9e6 * busy_ms))  # some ms of the null stream, then it ends by itself
        t.parameter_gradient_frames(x, 0, 1, g, dq, dtable, stream=side)
        side.synchronize()
        sums.append((dq.cpu().numpy(), dtable.cpu().numpy()))
    torch.cuda.synchronize()
    for a, b in zip(*sums):
        # f32 pair terms summed by atomics in two orders: 1e-6 of the norm
        assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
