"""The coarse levels from the second K-cycle level on as one thread-block cluster (k_amg_cluster, taken with
one sweep and at most 7168 rows on that level) against the same levels by the persistent kernel, which adds
in the same order: the same iterations and the same solution bit for bit.  Sizes without such a level, with
one, two and three smoothed levels in the cluster, on both sides of the row limit, and a numbering that
makes every CTA's window the whole level."""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hex,shuffle,cluster", [(6, False, False), (14, False, False), (20, False, True), (31, False, True),
                                                   (45, True, True), (74, False, True), (86, False, False)])
def test_cluster_levels_match_persistent_bitwise(ctx, n_hex, shuffle, cluster):
    A, b = O.assemble_heat(W.heat_cube(n_hex, sigma=1.5, seed=5, source="random"))
    n = len(b)
    if shuffle:
        import scipy.sparse as sp
        p = np.random.default_rng(7).permutation(n)
        S = sp.csr_matrix((A.val, A.ci, A.rp), shape=(n, n))[p][:, p].sorted_indices()
        A, b = O.CSR(n, S.indptr, S.indices, S.data), b[p]
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = [rsg.make_conf(n_outer=2000, stop_rule="true", rtol=1e-10, precision="mixed", persistent=q) for q in (0, 1)]
    rows = ctx.amg_setup(M)["rows"]
    assert (len(rows) > 3 and rows[2] <= 7168) == cluster
    x0, s0 = ctx.solve(M, b, conf=conf[0], prec=rsg.PREC_AMG)
    x1, s1 = ctx.solve(M, b, conf=conf[1], prec=rsg.PREC_AMG)
    assert s0.status == rsg.OK and O.true_relres(A, b, x0) <= 1e-10 * 1.01
    assert s0.iterations == s1.iterations and np.array_equal(x0, x1)
