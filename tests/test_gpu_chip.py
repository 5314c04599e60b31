"""The on-chip CG (csrc/cg_chip.cu) at the sizes where its partition can go
wrong: one node short of and past a slice, a CTA and the cluster's and the
grid's largest shapes, rows wider than its registers hold, node numberings
with nothing in common with the mesh's geometry, and every CTA shape.

Each linear solve is checked against the matrix itself (the exported CSR, in
numpy): the residual of the returned displacements may exceed the tolerance of
the recursively computed one by at most the residual gap of a k-step CG,
k eps || |K| |u| || / ||b|| with eps the precision of the recurrences."""
import numpy as np
import pytest

import cudaplasticity_b200 as cp

pytestmark = pytest.mark.gpu

EPS64 = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def ctx():
    c = cp.Context(0)
    yield c
    c.close()


def strip(nx, ny, elem="q4", shuffle=None):
    """A strip of nx x ny nodes, clamped along its bottom and sheared along its top (well conditioned at every aspect)."""
    x, y = np.meshgrid(np.linspace(0.0, 10.0 * nx / max(ny, 1), nx), np.linspace(0.0, 10.0, ny))
    xy = np.stack([x.ravel(), y.ravel()], axis=1)
    q = np.array([[j * nx + i, j * nx + i + 1, (j + 1) * nx + i + 1, (j + 1) * nx + i]
                  for j in range(ny - 1) for i in range(nx - 1)], np.int32)
    q = q[:, [2, 3, 0, 1]]  # the reference's corner order
    arrays = dict(node_xy=xy, elem4=q)
    if elem == "t3":
        arrays = dict(node_xy=xy, elem3=np.concatenate([q[:, [0, 1, 2]], q[:, [0, 2, 3]]]))
    if shuffle is not None:
        to = np.random.default_rng(shuffle).permutation(len(xy)).astype(np.int32)
        back = np.argsort(to)
        arrays = {k: (v[back] if k == "node_xy" else to[v]) for k, v in arrays.items()}
    xy = arrays["node_xy"]
    bottom, top = np.flatnonzero(xy[:, 1] < 1e-9), np.flatnonzero(xy[:, 1] > xy[:, 1].max() - 1e-9)
    rp, mask = np.zeros(2 * len(xy)), np.ones(2 * len(xy), np.uint8)
    mask[2 * bottom] = mask[2 * bottom + 1] = 0
    rp[2 * top], rp[2 * top + 1] = 1.0, 0.2 * np.sin(xy[top, 0])
    return arrays, rp, mask


def solve(ctx, problem, eps=1e-11, precond=1, precision=cp.CP_PREC_FP64, **kw):
    arrays, rp, mask = problem
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    rep = inst.solve(cg_tol=eps, outer_tol=1e300, max_outer=1, precond=precond, max_cg=100000, precision=precision, **kw)
    u, csr = inst.field("uv"), inst.csr()
    inst.close()
    return u, rep, csr


def residual(problem, u, csr):
    """||m.(b - K u)|| / ||b|| and || |K| |u| || / ||b||."""
    _, rp, mask = problem
    rows, cols, val = csr["rows"], csr["cols"], csr["k_data"]
    at = np.repeat(np.arange(len(rows) - 1), np.diff(rows))
    ku = np.bincount(at, weights=val * u[cols], minlength=len(rp))
    ab = np.bincount(at, weights=np.abs(val * u[cols]), minlength=len(rp))
    b = np.linalg.norm(rp)
    return np.linalg.norm(np.where(mask, rp - ku, 0.0)) / b, np.linalg.norm(ab) / b


def check(problem, u, rep, csr, eps, unit=EPS64):
    res, gap = residual(problem, u, csr)
    assert rep["status"] == 0 and rep["cg_iters"] > 0 and rep["cg_rel_res"] <= eps
    assert res <= eps + rep["cg_iters"] * unit * gap, (res, eps, rep["cg_iters"] * unit * gap)


# nodes: 4, 32 and around (a slice), 127..129 x 2 (a CTA), 1664, 1665 (13 CTAs of 4), 6144, 6145 (16 CTAs of 12: the cluster's
# largest, then the grid), 32768, 32769 (128 CTAs of 8, then 9), 56448, 56560 (147 CTAs of 12, then two nodes per
# thread), 112896, 113008 (the largest, then the graph loop)
@pytest.mark.parametrize("nx, ny", [(2, 2), (31, 2), (16, 2), (11, 3), (127, 2), (43, 3), (64, 26),
                                    (555, 3), (96, 64), (2048, 3), (1229, 5), (256, 128), (331, 99), (504, 112), (505, 112),
                                    (1008, 112), (1009, 112)])
def test_sizes(nx, ny, ctx):
    p = strip(nx, ny)
    for precond in (0, 1):
        check(p, *solve(ctx, p, precond=precond), 1e-11)


@pytest.mark.parametrize("form", ["c1", "c3", "c12", "g1", "g3", "g8", "g12"])
@pytest.mark.parametrize("elem, shuffle", [("q4", None), ("q4", 7), ("t3", 3)])
def test_forms_and_numberings(form, elem, shuffle, ctx, monkeypatch):
    """The same system in every CTA shape (forms that do not hold it take the graph loop)."""
    monkeypatch.setenv("CUPLAST_CHIP_FORM", form)
    p = strip(37, 29, elem, shuffle)
    check(p, *solve(ctx, p), 1e-11)


@pytest.mark.parametrize("n_c, n_r", [(8, 4), (24, 24), (48, 47)])
@pytest.mark.parametrize("form", [None, "c12", "g8"])
def test_wide_rows(n_c, n_r, form, ctx, monkeypatch):
    """8-node quads: rows of up to 21 blocks, more than the registers hold."""
    if form:
        monkeypatch.setenv("CUPLAST_CHIP_FORM", form)
    mesh = cp.Mesh.ring(50.0, 100.0, n_c, n_r, order=2)
    rp, mask, _ = cp.Loads().set_force(0, 100.0, 0.0, True).fix_border(1).build(mesh)
    p = (mesh.arrays(), rp, mask)
    check(p, *solve(ctx, p), 1e-11)


@pytest.mark.parametrize("nx, ny", [(2, 2), (16, 2), (127, 2), (64, 26), (96, 64), (1229, 5), (331, 99), (505, 112)])
def test_mixed_precision(nx, ny, ctx):
    """FP32 recurrences inside FP64 defect correction: the solve ends on the FP64 residual itself."""
    p = strip(nx, ny)
    for precond in (0, 1):
        u, rep, csr = solve(ctx, p, precond=precond, precision=cp.CP_PREC_MIXED, inner_tol=1e-3)
        res, gap = residual(p, u, csr)
        # one evaluation of b - K u in each arithmetic order: the rounding of a row's at most 18 products
        assert rep["cg_rel_res"] <= 1e-11 and abs(res - rep["cg_rel_res"]) <= 2 * 20 * EPS64 * gap


# nodes: tiny, 3072, 3075 (clusters of 4, then 8), 6144, 6145, 12288, 12291 (16, then the tile kernels)
@pytest.mark.parametrize("nx, ny", [(2, 2), (16, 2), (96, 32), (1025, 3), (96, 64), (1229, 5), (128, 96), (4097, 3)])
def test_batch(nx, ny, ctx):
    """A batch's linear solves on chip, alone and beside another instance: they end on the FP64 residual, and the
    result is the same bit for bit."""
    p = strip(nx, ny)
    kw = dict(cg_tol=1e-11, outer_tol=1e300, inner_tol=1e-3, max_outer=1, max_cg=100000)
    for precond in (0, 1):
        batch, out = cp.Batch(ctx, max_instances=2), []
        for other in (False, True):
            insts = [cp.Instance(ctx, a, cp.material(210000.0, 0.3)) for a, _, _ in ([strip(40, 30)] * other + [p])]
            for i, (_, rp, mask) in zip(insts, [strip(40, 30)] * other + [p]):
                i.set_loads(rp, mask)
                batch.add(i, precond=precond, **kw)
            batch.run()
            rep = {i._h.value: r for _, i, r in batch.harvest()}[insts[-1]._h.value]
            u, csr = insts[-1].field("uv"), insts[-1].csr()
            res, gap = residual(p, u, csr)
            assert rep["status"] == 0 and rep["cg_rel_res"] <= 1e-11
            assert abs(res - rep["cg_rel_res"]) <= 2 * 20 * EPS64 * gap
            out.append(u)
            for i in insts:
                i.close()
        assert np.array_equal(out[0], out[1])
        batch.close()


def test_mixed_precision_falls_back(ctx, monkeypatch):
    """Where FP32 cannot carry the system (a column 900 elements high and two wide, kappa eps32 >> 1), the on-chip form
    hands over to the two-kernel loop from the same start: the same outcome as that loop alone."""
    p = strip(3, 900)
    out = []
    for form in ("classic", "cluster"):
        monkeypatch.setenv("CUPLAST_FP64_CG", form)
        with pytest.raises(cp.CuplastError) as e:
            solve(ctx, p, precision=cp.CP_PREC_MIXED, inner_tol=1e-3)
        out.append(e.value.status)
    assert out == [cp._capi.CP_ERR_BREAKDOWN] * 2


def test_result_is_reproducible_and_independent_of_the_instance(ctx):
    p = strip(120, 80)
    a, b = solve(ctx, p)[0], solve(ctx, p)[0]
    assert np.array_equal(a, b)


def test_exchange_time_out_is_reported(ctx, monkeypatch):
    """Every poll of the grid form is bounded: with CUPLAST_TEST_BARRIER_NS set the CTAs post sequence numbers that
    none of them waits for, so every poll runs out, the solve returns CP_ERR_TIMEOUT and the context stays usable."""
    p = strip(120, 80)
    monkeypatch.setenv("CUPLAST_TEST_BARRIER_NS", "1000000")
    with pytest.raises(cp.CuplastError) as e:
        solve(ctx, p)
    assert e.value.status == cp._capi.CP_ERR_TIMEOUT
    monkeypatch.delenv("CUPLAST_TEST_BARRIER_NS")
    check(p, *solve(ctx, p), 1e-11)


def test_iteration_cap_and_zero_load(ctx):
    p = strip(64, 26)
    arrays, rp, mask = p
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    rep = inst.solve(allow_not_converged=True, cg_tol=1e-14, outer_tol=1e-30, max_outer=1, precond=1, max_cg=7)
    assert rep["cg_iters"] == 7
    inst.set_loads(np.zeros_like(rp), mask)
    inst.reset_state()  # elements that seven iterations left without strain have no secant modulus
    inst.assemble()
    iters, _ = inst.cg_solve(1e-10)
    assert iters == 0 and not inst.field("uv").any()
    inst.close()
