"""The CG loop with the matrix resident in shared memory (the default for small systems) against the
graph-driven loop (persistent=-1): solution, iteration counts and statistics bit for bit.

Sizes around its units (64 rows in FP64, 128 in mixed precision), with every remainder of the two- and
four-row groups, one to sixteen CTAs of a cluster and one CTA per SM; a shuffled numbering whose band is
the whole matrix; rows longer than 16 entries; a slice padded to more than 1.25 times its entries.
"""
import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


def banded(n, reach, seed=0, shuffle=False):
    """Symmetric diagonally dominant matrix with random couplings up to `reach` rows away."""
    rng = np.random.default_rng(seed + n)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.zeros(n)]
    for k in range(1, reach + 1):
        i = np.arange(n - k) if k < n else np.arange(0)
        i = i[rng.random(i.size) < 0.7]
        v = -rng.random(i.size)
        rows += [i, i + k]
        cols += [i + k, i]
        vals += [v, v]
    r, c, v = (np.concatenate(a) for a in (rows, cols, vals))
    np.add.at(v, np.arange(n), np.bincount(r, weights=np.abs(v), minlength=n) + 0.02)
    if shuffle:
        perm = rng.permutation(n)
        r, c = perm[r], perm[c]
    order = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    return rp, c[order].astype(np.uint32), v[order], rng.standard_normal(n)


def same_bits(ctx, M, b, precision, prec=rsg.PREC_JACOBI, **kw):
    base = dict(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision, **kw)
    xg, sg = ctx.solve(M, b, conf=rsg.make_conf(persistent=-1, **base), prec=prec)
    xr, sr = ctx.solve(M, b, conf=rsg.make_conf(**base), prec=prec)
    assert sg.status == sr.status == rsg.OK
    assert np.array_equal(xg, xr)
    assert (sg.iterations, sg.outer, sg.error, sg.true_relres) == (sr.iterations, sr.outer, sr.error, sr.true_relres)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 63, 64, 65, 127, 129, 193, 577, 1000, 1001, 1002, 1003, 3073, 20000])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sizes(ctx, n, precision):
    rp, ci, val, b = banded(n, 6)
    same_bits(ctx, ctx.matrix(rp, ci, val), b, precision)


@pytest.mark.parametrize("n,reach,shuffle", [(2000, 8, True), (1500, 40, False), (5001, 25, False)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("prec", [rsg.PREC_NONE, rsg.PREC_JACOBI])
def test_wide_bands_and_long_rows(ctx, n, reach, shuffle, precision, prec):
    rp, ci, val, b = banded(n, reach, shuffle=shuffle)
    same_bits(ctx, ctx.matrix(rp, ci, val), b, precision, prec)


@pytest.mark.parametrize("hexes", [4, 8, 14, 20, 27, 41])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "auto"])
def test_heat_cubes(ctx, hexes, precision):
    A, b = O.assemble_heat(W.heat_cube(hexes, sigma=1.2, seed=4, source="random"))
    same_bits(ctx, ctx.matrix(A.rp, A.ci, A.val), b, precision)
