"""The one-launch FP64 CG on the upper half of K (csrc/cg_fused.cu): meshes of
less than a slice, a slice, one node more, and many; rows with more blocks on
one side than a thread takes at once (shuffled numberings, 8-node quads). The
residual bound is the one of the on-chip CG's tests."""
import numpy as np
import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import check, ctx, solve, strip  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny, elem, shuffle", [
    (2, 2, "q4", None), (16, 2, "q4", None), (11, 3, "q4", None), (96, 64, "q4", None), (505, 112, "q4", None),
    (40, 30, "t3", None), (64, 26, "q4", 3), (64, 26, "t3", 4)])
@pytest.mark.parametrize("precond", [0, 1])
def test_half(nx, ny, elem, shuffle, precond, ctx, monkeypatch):  # noqa: F811
    monkeypatch.setenv("CUPLAST_FP64_CG", "fused")
    p, out = strip(nx, ny, elem, shuffle), []
    for half in ("0", "1"):
        monkeypatch.setenv("CUPLAST_HALF_K", half)
        u, rep, csr = solve(ctx, p, precond=precond)
        check(p, u, rep, csr, 1e-11)
        out.append(csr["k_data"])
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("n_c, n_r", [(8, 4), (24, 24)])
def test_half_wide_rows(n_c, n_r, ctx, monkeypatch):  # noqa: F811
    monkeypatch.setenv("CUPLAST_FP64_CG", "fused")
    monkeypatch.setenv("CUPLAST_HALF_K", "1")
    mesh = cp.Mesh.ring(50.0, 100.0, n_c, n_r, order=2)
    rp, mask, _ = cp.Loads().set_force(0, 100.0, 0.0, True).fix_border(1).build(mesh)
    p = (mesh.arrays(), rp, mask)
    check(p, *solve(ctx, p), 1e-11)
