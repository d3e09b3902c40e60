"""Batched CP-ALS: a tensor's result must not depend on how many CTAs share
it.  The batch's size chooses the cluster (8 CTAs a tensor for a few tensors,
4, 2, then 1), so the same ragged tensors are run in batches of every size,
and a few of them against the oracle's ALS."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

# edges: 1 to 3 row chunks of 32, outer extents below a group of 4 and a
# cluster, inner extents around multiples of 4, ranks around 4, 8 and 16
TENSORS = [((16, 16, 16), 4), ((96, 17, 31), 16), ((1, 40, 23), 3), ((33, 1, 9), 1), ((96, 96, 96), 8),
           ((20, 30, 1), 5), ((32, 3, 2), 2), ((65, 50, 19), 9), ((64, 7, 61), 12), ((31, 2, 96), 16)]


def _batch(cd, copies):
    b = cd.Batch([d for d, _ in TENSORS] * copies, [r for _, r in TENSORS] * copies)
    for t in range(b.n):
        d, r = TENSORS[t % len(TENSORS)]
        rng = np.random.default_rng(100 + t % len(TENSORS))
        true = [rng.standard_normal(x * r) for x in d]
        X = oracle.gencp(d, true, r) + 1e-2 * rng.standard_normal(int(np.prod(d)))
        b.x_view(t).copy_(torch.from_numpy(X.astype(np.float32)))
        for m in range(3):
            b.u_view(t, m).copy_(torch.from_numpy(rng.standard_normal(d[m] * r).astype(np.float32)))
    return b


def test_result_does_not_depend_on_the_cluster(cd, dev):
    ref = None
    for copies in (1, 12, 40, 100):  # 10, 120, 400 and 1000 tensors
        b = _batch(cd, copies)
        fits, sweeps, _ = cd.cp_als_batched(b, max_sweeps=4, tol=0.0)
        assert all(s == 4 for s in sweeps)
        n = len(TENSORS)
        got = [[b.u_view(t, m).clone() for m in range(3)] for t in range(n)]
        if ref is None:
            ref = (got, fits[:n])
        for t in range(b.n):
            for m in range(3):
                assert torch.equal(b.u_view(t, m), ref[0][t % n][m]), (copies, t, m)
            assert fits[t] == ref[1][t % n]


def test_ragged_tensors_match_oracle(cd, dev):
    b = _batch(cd, 1)
    start = b.U.clone()
    fits, _, _ = cd.cp_als_batched(b, max_sweeps=3, tol=0.0)
    for t in (0, 1, 7, 8):
        d, r = TENSORS[t]
        init = []
        for m in range(3):
            o = b.u_offsets[3 * t + m]
            init.append(start[o: o + d[m] * r].cpu().numpy())
        _, want, _ = oracle.cp_als(b.x_view(t).cpu().numpy(), d, r, init, 3)
        # FP32 MTTKRPs of well-conditioned (Gaussian) factors
        assert abs(fits[t] - want[-1]) <= 1e-4
