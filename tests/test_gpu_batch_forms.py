"""Which form of the linear solve a batch takes: 8-node meshes, whose rows take
more shared memory, go on to the next cluster size until 8,192 nodes."""
import numpy as np
import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import EPS64, ctx, residual, strip  # noqa: F401

pytestmark = pytest.mark.gpu


def solve(ctx, problem):  # noqa: F811
    arrays, rp, mask = problem
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    batch = cp.Batch(ctx, max_instances=1, max_width=32)
    batch.add(inst, cg_tol=1e-11, outer_tol=1e300, inner_tol=1e-3, max_outer=1, max_cg=100000, precond=1)
    batch.run()
    rep = batch.harvest()[0][2]
    u = inst.field("uv")
    res, gap = residual(problem, u, inst.csr())
    # (the bound of the on-chip CG's tests, with rows of up to 42 products)
    assert rep["status"] == 0 and rep["cg_rel_res"] <= 1e-11 and abs(res - rep["cg_rel_res"]) <= 2 * 44 * EPS64 * gap
    inst.close()
    batch.close()
    return u


# 112 and 1,960 nodes (a cluster of 4), 2,352, 3,528 (8), 4,704, 7,840 (16), 8,232 (the tile kernels)
@pytest.mark.parametrize("n_c, n_r, on_chip", [(8, 4, True), (20, 32, True), (24, 32, True), (36, 32, True),
                                               (48, 32, True), (80, 32, True), (84, 32, False)])
def test_8_node_meshes(n_c, n_r, on_chip, ctx, monkeypatch):  # noqa: F811
    mesh = cp.Mesh.ring(50.0, 100.0, n_c, n_r, order=2)
    rp, mask, _ = cp.Loads().set_force(0, 100.0, 0.0, True).fix_border(1).build(mesh)
    p = (mesh.arrays(), rp, mask)
    u = solve(ctx, p)
    monkeypatch.setenv("CUPLAST_BATCH_CHIP", "0")
    tiles = solve(ctx, p)
    # another order of the sums: equal bits only from the same form
    assert np.array_equal(u, tiles) != on_chip
    assert np.linalg.norm(u - tiles) <= 1e-6 * np.linalg.norm(tiles)


def test_launches_per_trip(ctx):  # noqa: F811
    """Runs without an instance on chip leave its launches out (three cluster sizes beside 3 + 1 + 16 + 1 others); a
    batch takes both kinds of run in turn."""
    batch, trips, launches = cp.Batch(ctx, max_instances=2), 0, 0
    for sizes, per_trip in (([(140, 100)], 21), ([(64, 26)], 24), ([(140, 100), (64, 26)], 24), ([(140, 100)], 21)):
        insts = []
        for nx, ny in sizes:
            arrays, rp, mask = strip(nx, ny)
            insts.append(cp.Instance(ctx, arrays, cp.material(210000.0, 0.3)))
            insts[-1].set_loads(rp, mask)
            batch.add(insts[-1], cg_tol=1e-6, outer_tol=1e300, inner_tol=1e-3, max_outer=1, max_cg=20000, precond=1)
        batch.run()
        assert [r["status"] for _, _, r in batch.harvest()] == [0] * len(sizes)
        s = batch.stats()
        assert s["kernel_launches"] - launches == per_trip * (s["trips"] - trips)
        trips, launches = s["trips"], s["kernel_launches"]
        for i in insts:
            i.close()
    batch.close()
