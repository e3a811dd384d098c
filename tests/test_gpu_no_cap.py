"""The largest iteration cap (2^32 - 1: none) and its neighbours in every CG loop: the solve ends by its own stopping
rule with the iterations and bits of an ordinary cap.  The heat cubes need more than 60 (cluster), 120 (one block per
SM, graph, host loop) and 60 (batch) iterations."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu

CAPS = [2 ** 32 - 1, 2 ** 32 - 16, 2 ** 32 - 17]


@pytest.mark.parametrize("n_hex,kw", [(12, {}), (26, {}), (26, dict(persistent=-1)), (26, dict(use_graph=False))])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "auto"])
def test_solve_without_a_cap(ctx, n_hex, kw, precision):
    A, b = O.assemble_heat(W.heat_cube(n_hex, sigma=1.5, seed=2, source="random"))
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = dict(stop_rule="true", rtol=1e-10, precision=precision, **kw)
    x, s = ctx.solve(M, b, conf=rsg.make_conf(n_outer=20000, **conf))
    assert s.iterations > (60 if n_hex == 12 else 120)
    for cap in CAPS:
        y, t = ctx.solve(M, b, conf=rsg.make_conf(n_outer=cap, **conf))
        assert t.status == rsg.OK and t.converged == 1 and t.iterations == s.iterations and np.array_equal(x, y)


def test_auto_precision_continues_without_a_cap(ctx):
    # the beam leaves mixed precision at its first refresh: the FP64 continuation has its own limit
    p = W.stress_beam(16, 8, 8)
    A, b = O.assemble_stress(p)
    M = ctx.matrix(A.rp, A.ci, A.val)
    for kw in ({}, dict(persistent=-1)):
        x, s = ctx.solve(M, b, conf=rsg.make_conf(n_outer=2 ** 32 - 1, stop_rule="true", rtol=1e-10, precision="auto", **kw))
        assert s.status == rsg.OK and s.converged == 1 and O.true_relres(A, b, x) <= 1e-10 * 1.01


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("use_graph", [True, False])
def test_batch_without_a_cap(ctx, precision, use_graph):
    pairs = [O.assemble_heat(W.heat_cube(n, sigma=1.5, seed=n, source="random")) for n in (5, 22, 13)]
    batch = rsg.Batch(ctx, [(A.rp, A.ci, A.val) for A, _ in pairs])
    b = np.concatenate([b for _, b in pairs])
    conf = dict(stop_rule="true", rtol=1e-10, precision=precision, use_graph=use_graph)
    x, per, _ = batch.solve(b, conf=rsg.make_conf(n_outer=20000, **conf))
    assert max(s.iterations for s in per) > 60
    for cap in CAPS:
        y, per_cap, summ = batch.solve(b, conf=rsg.make_conf(n_outer=cap, **conf))
        assert summ.status == rsg.OK and summ.converged == 1 and np.array_equal(x, y)
        assert [s.iterations for s in per_cap] == [s.iterations for s in per]
