"""A system's answer in a batch does not depend on the systems beside it, nor on the grid: its sums are added in chunks
of eight slices counted from its own first slice.  Systems of 1 to 30 chunks and more than the 32 that a block
holds, in a batch of their own, among others in several orders, and with tuned launch shapes: the same bits and
iterations."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu

HEXES = [3, 5, 8, 9, 13, 17, 22, 27, 6, 34]  # 32 to 40,425 rows


@pytest.fixture(scope="module")
def systems():
    return [O.assemble_heat(W.heat_cube(n, sigma=1.0, seed=n, source="random")) for n in HEXES]


def solve(ctx, systems, order, precision, tuned=False, use_graph=True):
    batch = rsg.Batch(ctx, [(systems[i][0].rp, systems[i][0].ci, systems[i][0].val) for i in order])
    if tuned:
        batch.autotune()
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision, use_graph=use_graph)
    x, per, summ = batch.solve(np.concatenate([systems[i][1] for i in order]), conf=conf)
    assert summ.status == rsg.OK and summ.converged == 1
    return {i: (s.iterations, xi) for i, xi, s in zip(order, batch.split(x), per)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_bits_alone_and_among_others(ctx, systems, precision):
    n = len(HEXES)
    want = {}
    for i in range(n):
        want.update(solve(ctx, systems, [i], precision))
    for i, (_, x) in want.items():
        assert O.true_relres(systems[i][0], systems[i][1], x) <= 1e-10 * 1.01
    orders = [list(range(n)), list(range(n))[::-1], [9, 0, 9 - 1, 1, 7, 2, 6, 3, 5, 4], [4, 9]]
    runs = [solve(ctx, systems, o, precision) for o in orders]
    runs.append(solve(ctx, systems, orders[0], precision, tuned=True))
    runs.append(solve(ctx, systems, orders[2], precision, use_graph=False))
    for got in runs:
        for i, (it, x) in got.items():
            assert it == want[i][0] and np.array_equal(x, want[i][1])
