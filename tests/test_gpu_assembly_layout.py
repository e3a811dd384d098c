"""The packed (row, tet) pairs of the heat assembly: the near form (neighbour nodes numbered within 32767
of the row's), the wide form (a shuffled numbering of 39k nodes) and the global-memory kernel, and the
copies a re-assembly writes itself (CSR FP32, SELL-32 in both precisions, Frobenius norm).

Entries and right-hand side against the oracle at the assembly's 1e-13; the copies are checked through
matrix-vector products, FP64 against the entries read back (1e-13) and FP32 within 2^-23 per product
(1e-5 of the row sum of magnitudes).
"""
import copy

import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


def problem(n, shuffle, transient):
    p = W.heat_cube(n, sigma=1.0, seed=3, source="random", transient=transient)
    if transient:
        p.node_t = np.where(p.disabled, p.node_t, W.uniform(3, 8, p.mesh.n_nodes))
    if not shuffle:
        return p
    q = copy.copy(p)
    perm = np.random.default_rng(1).permutation(p.mesh.n_nodes)  # new number of each node
    inv = np.argsort(perm)
    q.mesh = copy.copy(p.mesh)
    q.mesh.xyz = np.ascontiguousarray(p.mesh.xyz[inv])
    q.mesh.tets = np.ascontiguousarray(perm[p.mesh.tets].astype(np.uint32))
    q.disabled, q.node_t = p.disabled[inv], np.ascontiguousarray(p.node_t[inv])
    q.book, q.n_free = W.node_book(q.disabled)
    return q


@pytest.mark.parametrize("n,shuffle", [(2, False), (3, False), (9, False), (33, False), (33, True)])
@pytest.mark.parametrize("transient", [False, True])
@pytest.mark.parametrize("rows", ["0", "1"])
def test_pair_layouts_and_refreshed_copies(ctx, torch_cuda, monkeypatch, n, shuffle, transient, rows):
    torch = torch_cuda
    monkeypatch.setenv("RSG_ASM_ROW_THREADS", rows)
    p = problem(n, shuffle, transient)
    asm = rsg.Assembly.heat(ctx, p)
    b = torch.empty(p.n_free, dtype=torch.float64, device="cuda")
    first = copy.copy(p)
    first.k_e = 2.0 * p.k_e
    asm.assemble(first, b)
    M = asm.assemble(p, b)  # the re-assembly writes every copy
    ctx.sync()
    Ao, bo = O.assemble_heat(p)
    rp, ci, val = M.to_host()
    assert np.array_equal(rp, Ao.rp) and np.array_equal(ci, Ao.ci)
    rowmax = np.repeat(np.maximum.reduceat(np.abs(Ao.val), Ao.rp[:-1].astype(np.int64)), np.diff(Ao.rp.astype(np.int64)))
    assert np.all(np.abs(val - Ao.val) <= 1e-13 * rowmax)
    assert np.all(np.abs(b.cpu().numpy() - bo) <= 1e-13 * np.abs(bo).max())
    assert M.frobenius == pytest.approx(np.linalg.norm(val), rel=1e-13)
    x = np.random.default_rng(2).standard_normal(p.n_free)
    xd = torch.from_numpy(x).cuda()
    y, y32 = torch.empty_like(xd), torch.empty(p.n_free, dtype=torch.float32, device="cuda")
    ctx.spmv(M, xd, y)
    ctx.spmv_f32(M, xd.float(), y32)
    ctx.sync()
    start = rp[:-1].astype(np.int64)
    want = np.add.reduceat(val * x[ci], start)
    size = np.add.reduceat(np.abs(val * x[ci]), start)
    assert np.all(np.abs(y.cpu().numpy() - want) <= 1e-13 * size)
    assert np.all(np.abs(y32.cpu().numpy() - want) <= 1e-5 * size)
