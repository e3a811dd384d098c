"""The Arnoldi step kernels of GMRES at the edges of their tiles (256 rows) and accumulator counts
(8 basis vectors per warp slot): sizes around a tile, restart lengths around 8, 16, 32, 64 and 128, both
matrix layouts, FP64 and mixed precision.

1-D convection-diffusion with a shifted diagonal: condition number below 100, so a true relative
residual of 1e-10 bounds the error by 1e-8; the FP64 run follows the oracle's inner-step count.
"""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu


def system(n):
    D = np.diag(np.full(n, 2.05)) + np.diag(np.full(n - 1, -0.8), 1) + np.diag(np.full(n - 1, -1.2), -1)
    rng = np.random.default_rng(n)
    return D, O.csr_from_dense(D), rng.standard_normal(n)


@pytest.mark.parametrize("n,m", [(1, 5), (31, 8), (255, 9), (256, 16), (257, 17), (513, 33), (1000, 65), (300, 128)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sell", [True, False])
def test_gmres_restart_lengths_and_tiles(ctx, monkeypatch, n, m, precision, sell):
    D, A, b = system(n)
    if not sell:
        monkeypatch.setenv("RSG_NO_SELL", "1")
    M = ctx.matrix(A.rp, A.ci, A.val)
    kw = dict(solver="gmres", n_outer=2000, n_inner=m, stop_rule="true", rtol=1e-10)
    x, st = ctx.solve(M, b, conf=rsg.make_conf(precision=precision, **kw), prec=rsg.PREC_JACOBI)
    assert st.status == rsg.OK and O.true_relres(A, b, x) <= 1e-10 * 1.01
    assert rel_err(x, np.linalg.solve(D, b)) <= 1e-8
    if precision == "fp64":
        _, so = O.solve(A, b, prec=1, **kw)
        assert abs(int(st.iterations) - int(so.iterations)) <= 3
