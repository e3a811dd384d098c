"""The FP64 direction kernel's forms for SELL-32 matrices (all of the matrix kept in L2, its offsets, nothing; five or
six blocks per SM) against the CSR stream of the same system: both add a row's entries in the same order, so the
iterations agree to the grids' order of the sums and the solutions to the tolerance solved to."""
import numpy as np
import pytest

import rsg
from conftest import rel_err
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hex", [52, 62, 70, 92])
def test_sell_forms_match_csr_stream(ctx, n_hex, monkeypatch):
    A, b = O.assemble_heat(W.heat_cube(n_hex, sigma=1.0, seed=2, source="random"))
    M = ctx.matrix(A.rp, A.ci, A.val)
    monkeypatch.setenv("RSG_NO_SELL", "1")
    C = ctx.matrix(A.rp, A.ci, A.val)
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, persistent=-1)
    x, s = ctx.solve(M, b, conf=conf)
    y, t = ctx.solve(C, b, conf=conf)
    assert s.converged == 1 and O.true_relres(A, b, x) <= 1e-10 * 1.01
    assert abs(int(s.iterations) - int(t.iterations)) <= 2
    assert rel_err(x, y) < 1e-7  # two residuals of 1e-10 and a condition number of some 1e3
