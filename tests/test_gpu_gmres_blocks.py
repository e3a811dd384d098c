"""GMRES with block-Jacobi at the edges of the correction's tiles (the largest number of whole blocks and 16-byte packs
in 256 threads: 512 rows or a few less in FP64, 1024 in FP32): one block, a tile, a block more or less, sizes that
leave half a pack, widths 1 to 8 (3, 5, 6 and 7 do not divide the tile), restart lengths around the eight
vectors in flight, both matrix layouts.

1-D convection-diffusion with a shifted diagonal and blocks that couple: condition number below 100, so a true
relative residual of 1e-10 bounds the error by 1e-8; the FP64 run follows the oracle's inner-step count."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,blocks", [(1, 513), (2, 1), (2, 257), (3, 170), (3, 171), (3, 341), (5, 102), (5, 103), (5, 206),
                                      (6, 86), (7, 73), (7, 147), (8, 64), (8, 65), (8, 129)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,sell", [(7, True), (25, False)])
def test_block_jacobi_tiles(ctx, monkeypatch, w, blocks, precision, m, sell):
    n = w * blocks
    rng = np.random.default_rng(n)
    D = np.diag(2.05 + rng.random(n)) + np.diag(np.full(n - 1, -0.8), 1) + np.diag(np.full(n - 1, -1.2), -1)
    if not sell:
        monkeypatch.setenv("RSG_NO_SELL", "1")
    A, b = O.csr_from_dense(D), rng.standard_normal(n)
    M = ctx.matrix(A.rp, A.ci, A.val)
    kw = dict(solver="gmres", n_outer=2000, n_inner=m, stop_rule="true", rtol=1e-10)
    x, st = ctx.solve(M, b, conf=rsg.make_conf(precision=precision, **kw), prec=rsg.PREC_BLOCK_JACOBI, block_size=w)
    assert st.status == rsg.OK and O.true_relres(A, b, x) <= 1e-10 * 1.01
    assert rel_err(x, np.linalg.solve(D, b)) <= 1e-8
    if precision == "fp64":
        _, so = O.solve(A, b, prec=2, block_size=w, **kw)
        assert abs(int(st.iterations) - int(so.iterations)) <= 3
