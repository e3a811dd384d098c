"""GMRES on matrices of extreme scale (powers of two, so that scaling alone rounds nothing): the FP32 basis of mixed
precision is stored unnormalised, and its products have to keep to the size of A v all the same.  Without a
preconditioner, where nothing cancels the scale, and with Jacobi; both matrix layouts.  1-D convection-diffusion
with a condition number below 100: a true relative residual of 1e-10 in the unscaled matrix's inner steps, two
more or less for entries that FP32 denormals round."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(257, 12), (1000, 30)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("prec", [rsg.PREC_NONE, rsg.PREC_JACOBI])
@pytest.mark.parametrize("sell", [True, False])
def test_gmres_extreme_scales(ctx, monkeypatch, n, m, precision, prec, sell):
    if not sell:
        monkeypatch.setenv("RSG_NO_SELL", "1")
    D = np.diag(np.full(n, 2.05)) + np.diag(np.full(n - 1, -0.8), 1) + np.diag(np.full(n - 1, -1.2), -1)
    A, b = O.csr_from_dense(D), np.random.default_rng(n).standard_normal(n)
    conf = rsg.make_conf(solver="gmres", n_outer=2000, n_inner=m, stop_rule="true", rtol=1e-10, precision=precision)
    want, s0 = ctx.solve(ctx.matrix(A.rp, A.ci, A.val), b, conf=conf, prec=prec)
    assert s0.status == rsg.OK
    for p in (-90, -66, 66, 90):
        x, s = ctx.solve(ctx.matrix(A.rp, A.ci, A.val * 2.0 ** p), b, conf=conf, prec=prec)
        assert s.status == rsg.OK and O.true_relres(A, b, x * 2.0 ** p) <= 1e-10 * 1.01
        assert abs(int(s.iterations) - int(s0.iterations)) <= 2
        assert rel_err(x * 2.0 ** p, want) <= 1e-8
