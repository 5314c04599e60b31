"""Requests on a solve service's lanes whose linear solves each take most of
the GPU: they run in turns, a short one beside long ones ends soon, and every
result is the one of the request alone, bit for bit."""
import numpy as np
import pytest

import cudaplasticity_b200 as cp
from cudaplasticity_b200 import workload

pytestmark = pytest.mark.gpu

KW = dict(cg_tol=1e-10, outer_tol=1e-6, max_outer=300, max_cg=2_000_000, precond=1, aitken=1, adaptive_cg=2, recycle=6)


@pytest.fixture(scope="module")
def ctx():
    c = cp.Context(0)
    yield c
    c.close()


def solve(ctx, w, **kw):
    inst = cp.Instance(ctx, w["mesh"], w["material"])
    inst.set_loads(w["rp"], w["mask"], w["uv"])
    rep = inst.solve(allow_not_converged=True, levels=w["levels"], **kw)
    st = inst.state()
    inst.close()
    return st, rep


def served(srv, ws, **kw):
    rids = [srv.submit(w["mesh"], w["material"], w["rp"], w["mask"], w["uv"], levels=w["levels"], **kw) for w in ws]
    out = []
    for rid in rids:
        inst, rep, latency = srv.wait(rid, timeout=120.0)
        out.append((inst.state(), rep, latency))
        inst.close()
    return out


def same(got, want):
    (a, ra, *_), (b, rb) = got, want
    assert all(np.array_equal(a[f], b[f], equal_nan=True) for f in b)
    assert all(ra[k] == rb[k] for k in ("status", "outer_iters", "cg_iters", "cg_rel_res", "rel_err"))


# one node per thread, two, wide rows; more than one turn per linear solve
@pytest.mark.parametrize("precision", [cp.CP_PREC_FP64, cp.CP_PREC_FLOAT_BOOST])
def test_results_do_not_depend_on_the_turns(precision, ctx):
    ws = [workload.instance(i, dof_min=20000, dof_max=40000) for i in range(3)]
    ws.append(workload.instance(4, dof_min=170000, dof_max=200000))
    q8 = dict(workload.instance(5, dof_min=20000, dof_max=40000))
    mesh = cp.Mesh.ring(50.0, 100.0, 72, 71, order=2)
    q8["mesh"], q8["uv"] = mesh.arrays(), None
    q8["rp"], q8["mask"], _ = cp.Loads().set_force(0, 60.0, 0.0, True).fix_border(1).build(mesh)
    ws.append(q8)
    kw = dict(KW, precision=precision, max_outer=6, cg_tol=1e-11, adaptive_cg=0, inner_tol=1e-4)
    alone = [solve(ctx, w, **kw) for w in ws]
    assert sum(r["cg_iters"] / r["outer_iters"] > 256 for _, r in alone) >= 3
    srv = cp.Server(fp64_lanes=5)
    try:
        for got, want in zip(served(srv, ws, **kw), alone):
            same(got, want)
    finally:
        srv.close()


def test_short_requests_beside_long_ones(ctx):
    """The first requests of the service's benchmark as one burst: three of 1 to 2 s alone (0, 4, 6) and five of 9 to 50
    ms, which end long before the long ones do."""
    ws = [workload.instance(i) for i in range(8)]
    kw = dict(KW, precision=cp.CP_PREC_FP64, adaptive_cg=1)
    alone = [solve(ctx, w, **kw) for w in ws]
    srv = cp.Server(fp64_lanes=8)
    try:
        got = served(srv, ws, **kw)
    finally:
        srv.close()
    for g, a in zip(got, alone):
        same(g, a)
    latency = [g[2] for g in got]
    assert max(latency[i] for i in (1, 2, 3, 5, 7)) <= max(latency) / 4, latency
