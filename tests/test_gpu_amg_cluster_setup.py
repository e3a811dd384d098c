"""The packing of the cluster's coarse levels, done anew in every solve: row pointers and places come from a running
scan over tiles of 512 values, so it is run many times at sizes whose blocks own less than a tile of rows, about one
and (through a shuffled numbering) windows of several tiles.  A row pointer left over from another scan would
change the preconditioner: every solve has the iterations and the bits of the persistent kernel's."""
import numpy as np
import pytest
import scipy.sparse as sp

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hex,shuffle,repeats", [(20, False, 40), (33, True, 20), (57, False, 20), (74, False, 8)])
def test_repeated_setups_give_one_result(ctx, n_hex, shuffle, repeats):
    A, b = O.assemble_heat(W.heat_cube(n_hex, sigma=1.5, seed=6, source="random"))
    if shuffle:
        p = np.random.default_rng(8).permutation(len(b))
        S = sp.csr_matrix((A.val, A.ci, A.rp), shape=(len(b), len(b)))[p][:, p].sorted_indices()
        A, b = O.CSR(len(b), S.indptr, S.indices, S.data), b[p]
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = [rsg.make_conf(n_outer=2000, stop_rule="true", rtol=1e-10, precision="mixed", persistent=q) for q in (1, 0)]
    want, s0 = ctx.solve(M, b, conf=conf[0], prec=rsg.PREC_AMG)
    assert s0.status == rsg.OK and O.true_relres(A, b, want) <= 1e-10 * 1.01
    for _ in range(repeats):
        x, s = ctx.solve(M, b, conf=conf[1], prec=rsg.PREC_AMG)
        assert s.iterations == s0.iterations and np.array_equal(x, want)
