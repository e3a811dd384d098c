"""RSG_NO_PDL=1 (plain launches) in the loops besides the single solve's: several right-hand sides, the batch, the
learned preconditioner's layers and GMRES with them.  Dependent launch changes only when a kernel's blocks are
scheduled, so the results are the same bits."""
import numpy as np
import pytest

import rsg
import rsg.learned as RL
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    return O.assemble_heat(W.heat_cube(14, sigma=1.0, seed=4, source="random"))


def both(monkeypatch, f):
    a = f()
    monkeypatch.setenv("RSG_NO_PDL", "1")
    b = f()
    assert np.array_equal(a, b)
    return a


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("k", [1, 3, 8])
def test_multi(ctx, system, monkeypatch, k, use_graph):
    A, b = system
    M = ctx.matrix(A.rp, A.ci, A.val)
    B = np.random.default_rng(k).standard_normal((k, A.n))
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, use_graph=use_graph)
    X = both(monkeypatch, lambda: ctx.solve_multi(M, B, conf=conf)[0])
    for j in range(k):
        assert O.true_relres(A, B[j], X[j]) <= 1e-10 * 1.01


@pytest.mark.parametrize("use_graph", [True, False])
def test_batch(ctx, system, monkeypatch, use_graph):
    A, b = system
    batch = rsg.Batch(ctx, [(A.rp, A.ci, A.val)] * 3)
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision="mixed", use_graph=use_graph)
    x = both(monkeypatch, lambda: batch.solve(np.concatenate([b, 2.0 * b, -b]), conf=conf)[0])
    for xi, s in zip(batch.split(x), (1.0, 2.0, -1.0)):
        assert O.true_relres(A, s * b, xi) <= 1e-10 * 1.01


def test_learned(ctx, system, torch_cuda, monkeypatch):
    A, b = system
    M = ctx.matrix(A.rp, A.ci, A.val)
    model = RL.Learned(ctx, layers=3, seed=7)
    r = torch_cuda.from_numpy(b).cuda()
    torch_cuda.cuda.synchronize()

    def apply():
        z = torch_cuda.empty_like(r)
        torch_cuda.cuda.synchronize()
        model.apply(M, r, z, None, tensor_cores=True)
        ctx.sync()
        return z.cpu().numpy()

    def gmres():
        conf = RL.learned_conf(model, rsg.make_conf(solver="gmres", n_outer=300, n_inner=20, stop_rule="true", rtol=1e-8))
        x, st = ctx.solve(M, b, conf=conf, prec=rsg.PREC_LEARNED)
        assert st.converged == 1 and O.true_relres(A, b, x) <= 1e-8 * 1.01
        return x

    both(monkeypatch, apply)
    monkeypatch.delenv("RSG_NO_PDL")
    both(monkeypatch, gmres)
    model.close()
