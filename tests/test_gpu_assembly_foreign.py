"""A heat re-assembly into a matrix that was not made from its plan: a renumbered mesh has the same numbers of rows
and entries but other rows.  The values land in CSR order, as they always did, and every copy of the matrix (FP32,
SELL-32, norm) follows its own CSR arrays; with the same numbering the result is the plan's own matrix."""
import copy

import numpy as np
import pytest

import rsg
from rsg import workloads as W

pytestmark = pytest.mark.gpu


def renumbered(p):
    q = copy.copy(p)
    perm = np.random.default_rng(1).permutation(p.mesh.n_nodes)
    inv = np.argsort(perm)
    q.mesh = copy.copy(p.mesh)
    q.mesh.xyz = np.ascontiguousarray(p.mesh.xyz[inv])
    q.mesh.tets = np.ascontiguousarray(perm[p.mesh.tets].astype(np.uint32))
    q.disabled, q.node_t = p.disabled[inv], np.ascontiguousarray(p.node_t[inv])
    q.book, q.n_free = W.node_book(q.disabled)
    return q


@pytest.mark.parametrize("n,other", [(5, True), (12, True), (12, False)])
def test_reassembly_into_another_plans_matrix(ctx, torch_cuda, n, other):
    torch = torch_cuda
    p = W.heat_cube(n, sigma=1.0, seed=3, source="random")
    q = renumbered(p) if other else p
    b = torch.empty(p.n_free, dtype=torch.float64, device="cuda")
    own = rsg.Assembly.heat(ctx, q)
    want = own.assemble(q, b).to_host()[2]
    first = rsg.Assembly.heat(ctx, p)
    M = first.assemble(p, b)
    rp, ci, _ = M.to_host()
    own.A = M  # the handle that the caller passes back
    own.assemble(q, b)
    ctx.sync()
    got = M.to_host()
    assert np.array_equal(got[0], rp) and np.array_equal(got[1], ci) and np.array_equal(got[2], want)
    val = got[2]
    assert M.frobenius == pytest.approx(np.linalg.norm(val), rel=1e-13)
    x = np.random.default_rng(2).standard_normal(p.n_free)
    xd = torch.from_numpy(x).cuda()
    y, y32 = torch.empty_like(xd), torch.empty(p.n_free, dtype=torch.float32, device="cuda")
    ctx.spmv(M, xd, y)
    ctx.spmv_f32(M, xd.float(), y32)
    ctx.sync()
    start = rp[:-1].astype(np.int64)
    y_want, size = np.add.reduceat(val * x[ci], start), np.add.reduceat(np.abs(val * x[ci]), start)
    assert np.all(np.abs(y.cpu().numpy() - y_want) <= 1e-13 * size)
    assert np.all(np.abs(y32.cpu().numpy() - y_want) <= 1e-5 * size)
