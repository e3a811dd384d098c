"""Multi-right-hand-side CG on rows of 1 to 40 entries (trips of 1, 2, 4 and 8 lanes with every remainder) and
row counts that leave part of a warp empty: each column reaches its residual and agrees with the oracle's
tight solution; a column with an infinite right-hand side leaves the others as they are."""
import numpy as np
import pytest
import scipy.sparse as sp

import rsg
from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 4, 7, 16])
@pytest.mark.parametrize("n", [1, 33, 1001])
def test_multi_ragged_rows(ctx, n, k):
    rng = np.random.default_rng(n + k)
    S = sp.lil_matrix((n, n))
    for i in range(0, n, 2):  # symmetric, half of the rows longer than the rest
        for j in rng.choice(n, min(n - 1, int(rng.integers(0, 21))), replace=False) if n > 1 else []:
            if i != j:
                S[i, j] = S[j, i] = -rng.uniform(0.1, 1.0)
    S = sp.csr_matrix(S)
    S = (S + sp.diags(np.asarray(abs(S).sum(axis=1)).ravel() + 0.5)).tocsr().sorted_indices()
    A = O.CSR(n, S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)
    B = rng.standard_normal((k, n))
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = rsg.make_conf(n_outer=2000, stop_rule="true", rtol=1e-10)
    X, per, summ = ctx.solve_multi(M, B, conf=conf)
    for j in range(k):
        assert per[j].converged == 1 and O.true_relres(A, B[j], X[j]) <= 1e-10 * 1.01
        xt, _ = O.solve(A, B[j], prec=1, n_outer=200000, stop_rule="true", rtol=1e-12)
        assert rel_err(X[j], xt) < 1e-8
    if k > 1:
        B[k // 2, n // 2] = np.inf
        Y, per, summ = ctx.solve_multi(M, B, conf=conf)
        others = [j for j in range(k) if j != k // 2]
        assert np.array_equal(Y[others], X[others])
