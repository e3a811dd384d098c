"""The batch loop's lists and tickets: more systems than a block has threads, systems that share a block and
systems that span many, systems that are done at the start; every system against its dense or oracle
solution (condition numbers below 1e3 at a true relative residual of 1e-10: 1e-7)."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W
from conftest import rel_err

pytestmark = pytest.mark.gpu


def small(n, seed):
    rng = np.random.default_rng(seed)
    D = np.where(rng.random((n, n)) < 0.3, -rng.random((n, n)), 0.0)
    D = D + D.T
    np.fill_diagonal(D, 0.0)
    np.fill_diagonal(D, np.abs(D).sum(axis=1) + 0.1)
    return D, rng.standard_normal(n)


@pytest.mark.parametrize("count,big", [(1, None), (3, 14), (257, None), (300, 20), (600, 24)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_many_uneven_systems(ctx, count, big, precision):
    systems, rhs, want = [], [], []
    for i in range(count):
        D, b = small(1 + (7 * i) % 70, i)
        if i % 11 == 3:
            b[:] = 0.0  # solved before the loop starts
        A = O.csr_from_dense(D)
        systems.append((A.rp, A.ci, A.val))
        rhs.append(b)
        want.append(np.linalg.solve(D, b))
    if big:
        A, b = O.assemble_heat(W.heat_cube(big, sigma=0.5, seed=1, source="random"))
        at = count // 2
        systems.insert(at, (A.rp, A.ci, A.val))
        rhs.insert(at, b)
        x, st = O.solve(A, b, prec=1, n_outer=20000, stop_rule="true", rtol=1e-12)
        want.insert(at, x)
    batch = rsg.Batch(ctx, systems)
    for use_graph in (True, False):
        conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision, use_graph=use_graph)
        x, per, summ = batch.solve(np.concatenate(rhs), conf=conf)
        assert summ.status == rsg.OK and summ.converged == 1
        for xi, w, st in zip(batch.split(x), want, per):
            assert st.true_relres <= 1e-10 * 1.01
            assert rel_err(xi, w) <= 1e-7 if np.any(w) else not np.any(xi)
