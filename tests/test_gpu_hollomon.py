"""Inverse of the Hollomon diagram over the exponents that the API accepts
(every n > 0, not those of metals alone), without a plastic reference strain
(eps0 = 0: the elastic line) and at an infinite strain."""
import ctypes

import numpy as np
import pytest

import cudaplasticity_b200 as cp
from cudaplasticity_b200 import _capi

pytestmark = pytest.mark.gpu

E, NU, SY = 210000.0, 0.3, 250.0
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def ctx():
    c = cp.Context(0)
    yield c
    c.close()


def update(eps, eps0, n_exp):
    """One secant update of unit quads in uniaxial tension: their strain intensity and diagram value."""
    import torch

    count = len(eps)
    corners = np.array([[1.0, 1.0], [0.0, 1.0], [0.0, 0.0], [1.0, 0.0]])
    xy = np.tile(corners, (count, 1))
    u = xy * np.repeat(eps, 4)[:, None] * np.array([1.0, -NU])
    dev = torch.device("cuda:0")
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v).ravel()).to(dev)  # noqa: E731
    el = torch.arange(4 * count, dtype=torch.int32, device=dev)
    X, U, Ec, nc = t(xy), t(u), t(np.full(count, E)), t(np.full(count, NU))
    psi, f, err = t(np.zeros(count)), t(np.zeros(9 * count)), ctypes.c_double()
    mat = cp.material(E, NU, diagram="hollomon", sigma_y=SY, eps0=eps0, n=n_exp)
    torch.cuda.synchronize()
    st = _capi.lib().cp_secant_update_noalloc(None, ctypes.byref(mat), 4 * count, X.data_ptr(), count, el.data_ptr(),
                                              U.data_ptr(), Ec.data_ptr(), nc.data_ptr(), psi.data_ptr(), f.data_ptr(),
                                              ctypes.byref(err))
    assert st == 0
    f = f.cpu().numpy().reshape(9, count)
    return f[3], f[8]


@pytest.mark.parametrize("n_exp", [0.003, 0.05, 0.5, 1.0, 2.0, 5.0, 20.0, 50.0, 100.0, 1000.0])
@pytest.mark.parametrize("eps0", [1e-8, 1e-4, 0.002, 0.1, 100.0])
def test_every_exponent(n_exp, eps0, ctx):
    """table_s solves eps = s/E + eps0 ((s/sy)^(1/n) - 1) to the rounding of y = ln(s/sy) (at most 9) and of the
    powers, from just below yield to a strain of 10."""
    e, s = update(SY / E * np.geomspace(0.5, 8000.0, 400), eps0, n_exp)
    a, b = s / E, eps0 * (s / SY) ** (1.0 / n_exp)
    plastic = e >= SY / E
    g = np.where(plastic, a + b - eps0 - e, s - E * e)
    assert np.all(np.abs(g) <= 32 * EPS * np.where(plastic, a + b / n_exp + e + eps0, E * e))


def test_without_a_plastic_reference_strain(ctx):
    e, s = update(SY / E * np.geomspace(0.5, 8000.0, 400), 0.0, 0.2)
    assert np.all(np.abs(s - E * e) <= 32 * EPS * E * e)


@pytest.mark.parametrize("n_exp, eps0", [(0.2, 0.002), (50.0, 0.002)])
def test_infinite_strain(n_exp, eps0, ctx):
    e, s = update(np.array([1e-3, 1e200]), eps0, n_exp)
    assert e[1] == np.inf and s[1] == np.inf and np.isfinite(s[0])
