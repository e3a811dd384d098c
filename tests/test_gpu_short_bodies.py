"""Solves that ask for a residual check after nearly every iteration (a tolerance below what FP64 attains): the loop's
graph of several iterations a body ends and one with a check after every iteration goes on.  Iterations, checks and
bits are those of the host loop, which launches the same kernels in bodies of two (the batch: four)."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


def heat(n_hex, seed=4):
    return O.assemble_heat(W.heat_cube(n_hex, sigma=1.2, seed=seed, source="random"))


@pytest.mark.parametrize("precision,rtol", [("fp64", 3e-16), ("mixed", 3e-16), ("mixed", 1e-10)])
@pytest.mark.parametrize("prec", [rsg.PREC_JACOBI, rsg.PREC_BLOCK_JACOBI])
def test_single_solve(ctx, precision, rtol, prec):
    A, b = heat(14)
    M = ctx.matrix(A.rp, A.ci, A.val)
    got = []
    for use_graph in (True, False):
        conf = rsg.make_conf(n_outer=700, stop_rule="true", rtol=rtol, precision=precision, persistent=-1,
                             use_graph=use_graph, reliable_delta=0.9 if rtol == 1e-10 else 1e-3)
        got.append(ctx.solve(M, b, conf=conf, prec=prec, block_size=3))
    (x, s), (y, t) = got
    assert (s.status, s.iterations, s.outer, s.true_relres) == (t.status, t.iterations, t.outer, t.true_relres)
    assert np.array_equal(x, y)
    if rtol == 1e-10:
        assert s.status == rsg.OK
    else:
        assert s.iterations == 700 and s.true_relres <= 1e-13
        if precision == "fp64":
            assert s.outer > 100  # most of the iterations past the attainable accuracy


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch(ctx, precision):
    pairs = [heat(n, n) for n in (5, 12, 9)]
    batch = rsg.Batch(ctx, [(A.rp, A.ci, A.val) for A, _ in pairs])
    b = np.concatenate([b for _, b in pairs])
    got = []
    for use_graph in (True, False):
        conf = rsg.make_conf(n_outer=500, stop_rule="true", rtol=3e-16, precision=precision, use_graph=use_graph)
        got.append(batch.solve(b, conf=conf))
    (x, per, s), (y, per2, t) = got
    assert [(p.status, p.iterations, p.outer) for p in per] == [(p.status, p.iterations, p.outer) for p in per2]
    assert np.array_equal(x, y) and max(p.iterations for p in per) == 500 and max(p.true_relres for p in per) <= 1e-13
