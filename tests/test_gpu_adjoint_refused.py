"""Adjoints whose cheapest chain has more leg groups than a plan takes: they run along another one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# operands as (label, dimension) legs, and the slot
NETWORKS = [
    ([[(12, 2), (18, 2), (6, 2), (7, 2), (13, 2), (1, 2), (16, 3), (11, 2), (3, 2), (20, 2), (-1, 2), (14, 1), (15, 2),
       (9, 2), (4, 3)],
      [(13, 2), (20, 2), (1, 2), (-2, 2), (19, 3), (10, 3), (5, 1), (18, 2), (4, 3), (8, 1)],
      [(11, 2), (9, 2), (6, 2), (17, 2), (15, 2), (-3, 2), (-4, 2), (7, 2), (2, 1), (8, 1)],
      [(12, 2), (14, 1), (19, 3), (3, 2), (16, 3), (10, 3), (5, 1), (17, 2), (2, 1)]], 0),
    ([[(13, 1), (11, 2), (5, 3), (16, 2), (18, 3), (-2, 2), (8, 2), (-4, 2), (17, 3), (9, 3), (15, 3), (-1, 2),
       (-3, 2)],
      [(4, 2), (12, 2), (10, 2)],
      [(3, 2), (16, 2), (15, 3), (12, 2), (14, 2), (11, 2), (5, 3), (4, 2), (10, 2), (2, 2), (1, 2), (13, 1), (7, 2),
       (6, 2), (-5, 2)],
      [(1, 2), (-7, 2), (9, 3), (17, 3), (7, 2), (-9, 2), (2, 2), (-6, 2), (8, 2), (-8, 2), (3, 2), (14, 2), (18, 3),
       (6, 2)]], 1),
]


@pytest.mark.parametrize("legs,slot", NETWORKS)
def test_refused_chain(ctx, legs, slot):
    rng = np.random.default_rng(7)

    def randn(shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    ops = [randn([d for _, d in op]) for op in legs]
    labels = [[l for l, _ in op] for op in legs]
    outd = {l: d for op in legs for l, d in op if l < 0}
    out = sorted(outd, reverse=True)
    ybar = randn([outd[l] for l in out])
    got = ctx.download(ctx.contract_vjp([ctx.upload(a) for a in ops], labels, ctx.upload(ybar), slot))
    args = [ybar, [40 + l for l in out]]
    for i, (a, lab) in enumerate(zip(ops, labels)):
        if i != slot:
            args += [a.conj(), [l if l > 0 else 40 + l for l in lab]]
    ref = np.einsum(*args, [l if l > 0 else 40 + l for l in labels[slot]], optimize="greedy")
    assert np.linalg.norm(got - ref) <= 1e-13 * np.linalg.norm(ref)
