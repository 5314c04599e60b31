"""The element kernels at the sizes where their tiles end and on distorted
quads: K against 2x2 Gauss quadrature in numpy (1e-13 of
the row's largest value, the bar of the reference fixtures), bitwise symmetry,
and the Hollomon diagram's inverse against its own equation."""
import ctypes

import numpy as np
import pytest

import cudaplasticity_b200 as cp
from cudaplasticity_b200 import _capi

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3
GP = 0.577350269189626


@pytest.fixture(scope="module")
def ctx():
    c = cp.Context(0)
    yield c
    c.close()


def quads(nx, ny, seed):
    """nx x ny nodes, inner positions moved by up to 0.3 of a cell, cells of aspect 7, local numbering rotated."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx) * 7.0, np.arange(ny) * 1.0)
    xy = np.stack([x.ravel(), y.ravel()], axis=1) + rng.uniform(-0.3, 0.3, (nx * ny, 2)) * [7.0, 1.0]
    el = np.array([[(j + 1) * nx + i + 1, (j + 1) * nx + i, j * nx + i, j * nx + i + 1]
                   for j in range(ny - 1) for i in range(nx - 1)], np.int32)
    return xy, np.array([np.roll(e, rng.integers(4)) for e in el], np.int32)


def gauss_k(xy, el, plane):
    """Dense K (unit thickness) by 2x2 Gauss quadrature."""
    n = len(xy)
    if plane == cp.CP_PLANE_STRESS:
        D = E / (1 - NU * NU) * np.array([[1, NU, 0], [NU, 1, 0], [0, 0, (1 - NU) / 2]])
    else:
        D = E / ((1 + NU) * (1 - 2 * NU)) * np.array([[1 - NU, NU, 0], [NU, 1 - NU, 0], [0, 0, (1 - 2 * NU) / 2]])
    K = np.zeros((2 * n, 2 * n))
    ri, si = np.array([1.0, -1, -1, 1]), np.array([1.0, 1, -1, -1])
    for e in el:
        P = xy[e]
        ke = np.zeros((8, 8))
        for r in (-GP, GP):
            for s in (-GP, GP):
                dn = 0.25 * np.stack([ri * (1 + s * si), si * (1 + r * ri)])
                J = dn @ P
                g = np.linalg.solve(J, dn)
                B = np.zeros((3, 8))
                B[0, 0::2], B[1, 1::2], B[2, 0::2], B[2, 1::2] = g[0], g[1], g[1], g[0]
                ke += B.T @ D @ B * np.linalg.det(J)
        at = np.stack([2 * e, 2 * e + 1], axis=1).ravel()
        K[np.ix_(at, at)] += ke
    return K


# nodes: one quad, 127..129 (the tile of 128), 31..33 (a slice), several tiles
@pytest.mark.parametrize("nx, ny", [(2, 2), (31, 2), (11, 3), (43, 3), (64, 2), (32, 4), (16, 8), (27, 19)])
@pytest.mark.parametrize("plane", [cp.CP_PLANE_STRESS, cp.CP_PLANE_STRAIN])
def test_quad_assembly(nx, ny, plane, ctx):
    xy, el = quads(nx, ny, nx * 100 + ny)
    inst = cp.Instance(ctx, dict(node_xy=xy, elem4=el), cp.material(E, NU, plane=plane))
    inst.assemble()
    c = inst.csr()
    inst.close()
    n = 2 * len(xy)
    K = np.zeros((n, n))
    for i in range(n):
        K[i, c["cols"][c["rows"][i]:c["rows"][i + 1]]] = c["k_data"][c["rows"][i]:c["rows"][i + 1]]
    assert np.array_equal(K, K.T)
    ref = gauss_k(xy, el, plane)
    assert np.max(np.abs(K - ref) / np.abs(ref).max(axis=1, keepdims=True)) < 1e-13


@pytest.mark.parametrize("n_exp, eps0", [(0.2, 0.002), (0.05, 1e-4), (0.5, 0.01), (1.0, 0.002)])
@pytest.mark.parametrize("count", [1, 63, 64, 65, 20000])
def test_hollomon_inverse(count, n_exp, eps0, ctx):
    """Unit quads in uniaxial tension, strains from just below yield to 10: table_s solves
    eps = s/E + eps0 ((s/sy)^(1/n) - 1) to the rounding of y = ln(s/sy) and of the powers."""
    import torch

    sy = 250.0
    eps = sy / E * np.geomspace(0.5, 8000.0, count)
    corners = np.array([[1.0, 1.0], [0.0, 1.0], [0.0, 0.0], [1.0, 0.0]])
    xy = np.tile(corners, (count, 1))
    u = xy * np.repeat(eps, 4)[:, None] * np.array([1.0, -NU])
    dev = torch.device("cuda:0")
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v).ravel()).to(dev)  # noqa: E731
    el = torch.arange(4 * count, dtype=torch.int32, device=dev)
    X, U, Ec, nc = t(xy), t(u), t(np.full(count, E)), t(np.full(count, NU))
    psi, f, err = t(np.zeros(count)), t(np.zeros(9 * count)), ctypes.c_double()
    mat = cp.material(E, NU, diagram="hollomon", sigma_y=sy, eps0=eps0, n=n_exp)
    torch.cuda.synchronize()
    st = _capi.lib().cp_secant_update_noalloc(None, ctypes.byref(mat), 4 * count, X.data_ptr(), count, el.data_ptr(),
                                              U.data_ptr(), Ec.data_ptr(), nc.data_ptr(), psi.data_ptr(), f.data_ptr(),
                                              ctypes.byref(err))
    assert st == 0
    f = f.cpu().numpy().reshape(9, count)
    e, s = f[3], f[8]
    assert np.max(np.abs(e / eps - 1.0)) < 1e-13
    plastic = e >= sy / E
    a, b = s / E, eps0 * (s / sy) ** (1.0 / n_exp)
    g = np.where(plastic, a + b - eps0 - e, s - E * e)
    assert np.all(np.abs(g) <= 32 * np.finfo(float).eps * np.where(plastic, a + b / n_exp + e + eps0, E * e))
