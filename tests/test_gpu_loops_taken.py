"""Which kernels a call launches, and with which grids: several loops give one result bit for bit, so that only the
launches show whether the one meant for a size ran.  Seen through torch's profiler; skipped where it sees none."""
import json

import numpy as np
import pytest

import rsg
from oracle import oracle as O
from rsg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def launches(ctx, torch_cuda, tmp_path):
    torch = torch_cuda

    def run(f):
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
            f()
            ctx.sync()
            torch.cuda.synchronize()
        path = tmp_path / "trace.json"
        prof.export_chrome_trace(str(path))
        events = json.loads(path.read_text())["traceEvents"]
        got = [(e["name"], tuple(e["args"]["grid"])) for e in events if e.get("cat") == "kernel"]
        if not got:
            pytest.skip("the profiler sees no kernels here")
        return got

    return run


def named(got, name):
    return [(n, g) for n, g in got if name in n]


def heat(n_hex):
    return O.assemble_heat(W.heat_cube(n_hex, sigma=1.2, seed=4, source="random"))


@pytest.mark.parametrize("precision,kernel,kid", [("fp64", "k_cg_update<", 2),
                                                  ("mixed", "k_mx_update<", 3)])
def test_profiled_update_has_the_loops_grid(ctx, launches, precision, kernel, kid):
    A, b = heat(60)  # 215,940 rows: more than three blocks an SM with one thread per row
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = rsg.make_conf(n_outer=4, stop_rule="true", rtol=1e-10, precision=precision, use_graph=False)
    loop = {g for _, g in named(launches(lambda: ctx.solve(M, b, conf=conf)), kernel)}
    prof = {g for _, g in named(launches(lambda: ctx.profile_kernel(M, kid, reps=2)), kernel)}
    assert len(loop) == 1 and loop == prof


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_tuned_grids_keep_the_resident_loop(ctx, launches, tmp_path, precision):
    # a tuning cache of one block per kernel: shapes that the resident loop's sums cannot stand for
    A, b = heat(20)
    path = tmp_path / "tune.txt"
    M = ctx.matrix(A.rp, A.ci, A.val)
    ctx.autotune(M, str(path))
    key = path.read_text().split(" : ")[0]
    path.write_text(key + " : sell=1 rpw=0 dir64=1 dir32=1 upd64=1 upd32=1 pdl64=-1 pdl32=-1 it_us=1.000,1.000\n")
    T = ctx.matrix(A.rp, A.ci, A.val)
    assert ctx.autotune(T, str(path))["from_cache"] == 1
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision)
    U = ctx.matrix(A.rp, A.ci, A.val)
    x, s = ctx.solve(U, b, conf=conf)
    y, t = ctx.solve(T, b, conf=conf)
    assert t.iterations == s.iterations and np.array_equal(x, y)
    assert named(launches(lambda: ctx.solve(T, b, conf=conf)), "k_cg_resident")


@pytest.mark.parametrize("precision,n_hex,transport", [(p, n, t) for n, f, m in [
    (4, "true", "true"), (8, "true", "true"), (20, "true", "true"), (27, "false", "true"), (41, "false", "false"),
    (54, None, None)] for p, t in (("fp64", f), ("mixed", m))])
def test_small_systems_take_the_resident_loop(ctx, launches, precision, n_hex, transport):
    # 75 to 70,560 rows: one cluster (true), as far as its shared memory holds the matrix, or one block per SM
    # (false); 160,325 rows: neither
    A, b = heat(n_hex)
    M = ctx.matrix(A.rp, A.ci, A.val)
    conf = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision)
    loop = named(launches(lambda: ctx.solve(M, b, conf=conf)), "k_cg_resident<")
    assert [n.split("k_cg_resident<")[1].split(">")[0].split(", ")[2] for n, _ in loop] == [transport] * bool(transport)
    graph = rsg.make_conf(n_outer=20000, stop_rule="true", rtol=1e-10, precision=precision, persistent=-1)
    assert not named(launches(lambda: ctx.solve(M, b, conf=graph)), "k_cg_resident<")


@pytest.mark.parametrize("n_hex,cluster", [(14, False), (24, True), (45, True), (74, True), (86, False)])
def test_coarse_levels_take_the_cluster(ctx, launches, n_hex, cluster):
    A, b = heat(n_hex)
    M = ctx.matrix(A.rp, A.ci, A.val)
    info = ctx.amg_setup(M)
    assert (len(info["rows"]) > 3 and info["rows"][2] <= 7168) == cluster
    conf = rsg.make_conf(n_outer=2, stop_rule="true", rtol=1e-10, precision="mixed", use_graph=False)
    got = launches(lambda: ctx.solve(M, b, conf=conf, prec=rsg.PREC_AMG))
    visits = named(got, "k_amg_cluster")
    assert bool(visits) == cluster and all(g == (16, 1, 1) for _, g in visits)
    # two visits a cycle in place of the dozen launches or more that each takes without the cluster
    assert (info["cycle_launches"][0] <= 14) == (cluster or len(info["rows"]) <= 3)
