"""Batched CP-ALS of small tensors, which a CTA each sweeps alone however few
they are: the same bits as in a batch whose large tensors bring clusters, and
the oracle's fit."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

SMALL = [((4, 5, 6), 2), ((16, 16, 16), 4), ((1, 40, 23), 3), ((34, 34, 34), 8), ((32, 3, 2), 2), ((20, 30, 17), 16)]


def _batch(cd, tensors):
    b = cd.Batch([d for d, _ in tensors], [r for _, r in tensors])
    for t, (d, r) in enumerate(tensors):
        rng = np.random.default_rng(7 * sum(d) + r)
        true = [rng.standard_normal(x * r) for x in d]
        X = oracle.gencp(d, true, r) + 1e-2 * rng.standard_normal(int(np.prod(d)))
        b.x_view(t).copy_(torch.from_numpy(X.astype(np.float32)))
        for m in range(3):
            b.u_view(t, m).copy_(torch.from_numpy(rng.standard_normal(d[m] * r).astype(np.float32)))
    return b


def test_small_tensors_alone_and_beside_large_ones(cd, dev):
    alone, beside = _batch(cd, SMALL), _batch(cd, SMALL + [((96, 96, 90), 16)])
    start = alone.U.clone()
    f1, s1, _ = cd.cp_als_batched(alone, max_sweeps=12, tol=0.0)
    f2, s2, _ = cd.cp_als_batched(beside, max_sweeps=12, tol=0.0)
    assert list(s1) == [12] * len(SMALL) and list(f2)[: len(SMALL)] == list(f1)
    for t in range(len(SMALL)):
        for m in range(3):
            assert torch.equal(alone.u_view(t, m), beside.u_view(t, m))
    d, r = SMALL[3]
    init = [start[o: o + d[m] * r].cpu().numpy() for m in range(3) for o in [alone.u_offsets[9 + m]]]
    _, want, _ = oracle.cp_als(alone.x_view(3).cpu().numpy(), d, r, init, 12)
    assert abs(f1[3] - want[-1]) <= 1e-4


def test_tuned_shape_gives_the_same_bits(cd, dev):
    a, b = _batch(cd, SMALL * 3), _batch(cd, SMALL * 3)
    cd.cp_als_batched(a, max_sweeps=3, tol=0.0)
    start = b.U.clone()
    threads, ctas = cd.cp_batched_tune(b)[:2]
    assert (threads, ctas) == (192, 2)
    b.U.copy_(start)
    cd.cp_als_batched(b, max_sweeps=3, tol=0.0)
    assert torch.equal(a.U, b.U)
