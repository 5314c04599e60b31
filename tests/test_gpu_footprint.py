"""cp_instance_footprint, by which the solve service admits requests, covers
what an instance of each form of the linear solve holds on the device, and is
not far above it."""
import pytest

import cudaplasticity_b200 as cp
from cudaplasticity_b200 import workload
from test_gpu_chip import ctx, strip  # noqa: F401
from test_gpu_room import pool_bytes

pytestmark = pytest.mark.gpu

KW = dict(cg_tol=1e-6, outer_tol=1e-300, inner_tol=1e-3, max_outer=2, levels=1, max_cg=20000, precond=1)


def ring8(n_c, n_r):
    mesh = cp.Mesh.ring(50.0, 100.0, n_c, n_r, order=2)
    rp, mask, _ = cp.Loads().set_force(0, 100.0, 0.0, True).fix_border(1).build(mesh)
    return mesh.arrays(), rp, mask


# a cluster, a grid, a grid of two nodes per thread, the loop, the loop on the half of K; triangles in a shuffled
# numbering; 8-node quads
@pytest.mark.parametrize("make", [
    lambda: strip(64, 65), lambda: strip(160, 120), lambda: strip(320, 300), lambda: strip(360, 350),
    lambda: strip(500, 500), lambda: strip(160, 120, "t3", 3), lambda: strip(500, 500, "t3"), lambda: ring8(48, 32),
    lambda: ring8(160, 100), lambda: ring8(300, 250)])
@pytest.mark.parametrize("precision", [cp.CP_PREC_FP64, cp.CP_PREC_MIXED, cp.CP_PREC_FLOAT_BOOST])
def test_footprint(make, precision, ctx):  # noqa: F811
    arrays, rp, mask = make()
    base = pool_bytes(ctx)
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    inst.solve(allow_not_converged=True, precision=precision, **dict(KW, recycle=6, predict=1, levels=2, outer_tol=1e300))
    if precision == cp.CP_PREC_MIXED:
        batch = cp.Batch(ctx, max_instances=1, max_width=32)
        other = pool_bytes(ctx)
        batch.add(inst, **KW)
        batch.run()
        batch.harvest()
        assert pool_bytes(ctx) > other
    held = pool_bytes(ctx) - base
    said = cp.footprint(arrays, precision)
    inst.close()
    assert held <= said <= 2.0 * held + (2 << 20), (held, said, said / held)


@pytest.mark.parametrize("lanes", [2])
def test_footprint_of_requests_in_turns(lanes, ctx):  # noqa: F811
    """On a lane a grid's solve keeps its vectors between turns."""
    ws = [workload.instance(i, dof_min=20000, dof_max=40000) for i in range(lanes)]
    said = sum(cp.footprint(w["mesh"], cp.CP_PREC_FP64) for w in ws)
    srv = cp.Server(fp64_lanes=lanes)
    base = pool_bytes(ctx)
    kw = dict(KW, precision=cp.CP_PREC_FP64, cg_tol=1e-11, max_outer=6, max_cg=3000, recycle=6)
    rids = [srv.submit(w["mesh"], w["material"], w["rp"], w["mask"], w["uv"], **kw) for w in ws]
    insts = [srv.wait(rid, timeout=60.0)[0] for rid in rids]
    held = pool_bytes(ctx) - base
    for i in insts:
        i.close()
    srv.close()
    assert held <= said
