"""Which meshes the one-launch FP64 CG runs on the upper half of K: those
numbered along rows, from 150,000 nodes, without rows far wider than the rest
(cp_bench_cg_fused reports the bytes of the form that ran). And what the form
rests on: K is its transpose bit for bit, in any numbering."""
import ctypes

import numpy as np
import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import check, ctx, solve, strip  # noqa: F401

pytestmark = pytest.mark.gpu


def runs_on_the_half(ctx, problem):  # noqa: F811
    arrays, rp, mask = problem
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    ms, nbytes = ctypes.c_double(), ctypes.c_double()
    ctx.check(cp._capi.lib().cp_bench_cg_fused(inst._h, 1, 2, ctypes.byref(ms), ctypes.byref(nbytes)))
    nnz, n = inst.csr()["k_data"].size, len(mask) / 2
    inst.close()
    rest = nnz + n * (256 + 34)  # columns, vectors
    values = (nbytes.value - rest) / 8
    assert values in (nnz, (nnz + 4 * n) / 2)
    return values != nnz


def renumber(problem, to):
    """Node i becomes node to[i]."""
    arrays, rp, mask = problem
    back = np.argsort(to)
    out = {k: (v[back] if k == "node_xy" else to[v].astype(np.int32)) for k, v in arrays.items()}
    dof = np.stack([2 * back, 2 * back + 1], axis=1).ravel()
    return out, rp[dof], mask[dof]


def order(kind, nx, ny):
    n = nx * ny
    rng = np.random.default_rng(1)
    if kind == "columns":
        return (np.arange(n) % nx) * ny + np.arange(n) // nx
    if kind == "reversed":
        return np.arange(n)[::-1]
    if kind == "twentieth":  # the first twentieth of the nodes at random
        return np.concatenate([rng.permutation(n // 20), np.arange(n // 20, n)])
    if kind == "rows":  # whole rows in random order
        return rng.permutation(ny)[np.arange(n) // nx] * nx + np.arange(n) % nx
    return rng.permutation(n)


@pytest.mark.parametrize("elem", ["q4", "t3"])
@pytest.mark.parametrize("kind, want", [(None, True), ("columns", True), ("reversed", True), ("twentieth", True),
                                        ("rows", False), ("random", False)])
def test_numbering(elem, kind, want, ctx):  # noqa: F811
    p = strip(500, 400, elem)
    if kind:
        p = renumber(p, order(kind, 500, 400))
    assert runs_on_the_half(ctx, p) == want


def test_size(ctx):  # noqa: F811
    assert not runs_on_the_half(ctx, strip(375, 399))
    assert runs_on_the_half(ctx, strip(375, 400))


def test_one_wide_row(ctx):  # noqa: F811
    """A fan of triangles about one node of a large mesh: its row would widen every node's slots."""
    arrays, rp, mask = strip(500, 400)
    n, f = len(mask) // 2, 12
    a = np.linspace(0.0, 2.0, f)
    fan = np.array([[0, n + i + 1, n + i] for i in range(f - 1)], np.int32)
    xy = np.concatenate([arrays["node_xy"], arrays["node_xy"][0] - np.stack([np.cos(a), np.sin(a)], axis=1)])
    p = (dict(node_xy=xy, elem4=arrays["elem4"], elem3=fan), np.concatenate([rp, np.zeros(2 * f)]),
         np.concatenate([mask, np.ones(2 * f, np.uint8)]))
    assert not runs_on_the_half(ctx, p)


@pytest.mark.parametrize("nx, ny, elem, shuffle", [(64, 26, "q4", None), (64, 26, "q4", 3), (64, 26, "t3", 4),
                                                   (40, 30, "t3", None)])
def test_k_is_symmetric_and_the_forms_agree(nx, ny, elem, shuffle, ctx, monkeypatch):  # noqa: F811
    monkeypatch.setenv("CUPLAST_FP64_CG", "fused")
    p, out = strip(nx, ny, elem, shuffle), []
    for half in ("0", "1"):
        monkeypatch.setenv("CUPLAST_HALF_K", half)
        u, rep, csr = solve(ctx, p)
        check(p, u, rep, csr, 1e-11)
        out.append(u)
    at = np.repeat(np.arange(len(csr["rows"]) - 1), np.diff(csr["rows"]))
    there = np.lexsort((csr["cols"], at))
    back = np.lexsort((at, csr["cols"]))
    assert np.array_equal(csr["k_data"][there], csr["k_data"][back])
    assert np.linalg.norm(out[0] - out[1]) <= 1e-7 * np.linalg.norm(out[0])
    assert not np.array_equal(out[0], out[1])  # (another order of the sums: another kernel)


def test_k_is_symmetric_8_node(ctx):  # noqa: F811
    mesh = cp.Mesh.ring(50.0, 100.0, 24, 24, order=2)
    inst = cp.Instance(ctx, mesh.arrays(), cp.material(210000.0, 0.3))
    inst.assemble()
    csr = inst.csr()
    inst.close()
    at = np.repeat(np.arange(len(csr["rows"]) - 1), np.diff(csr["rows"]))
    there, back = np.lexsort((csr["cols"], at)), np.lexsort((at, csr["cols"]))
    assert np.array_equal(csr["k_data"][there], csr["k_data"][back])
