"""A linear solve that fails leaves the elements as they were: the update that
follows it on the stream, before the host has seen how it ended, does
nothing, and neither does the relaxation after it."""
import numpy as np
import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import ctx, strip  # noqa: F401

pytestmark = pytest.mark.gpu

FIELDS = [f for f in cp.FIELDS if f != "uv"]


def fields(inst):
    return {f: inst.field(f) for f in FIELDS}


def same(a, b):
    return all(np.array_equal(a[f], b[f], equal_nan=True) for f in FIELDS)


# a cluster, a grid, the graph loop
@pytest.mark.parametrize("nx, ny", [(64, 26), (120, 80), (1009, 112)])
@pytest.mark.parametrize("precond, aitken", [(1, 0), (1, 1), (2, 1)])
def test_breakdown(nx, ny, precond, aitken, ctx):  # noqa: F811
    arrays, rp, mask = strip(nx, ny)
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3, diagram="linear", sigma_t=2.0, k_t=2000.0))
    inst.set_loads(rp, mask)
    kw = dict(cg_tol=1e-8, outer_tol=1e-6, max_outer=3, max_cg=20000, precond=precond, aitken=aitken)
    inst.solve(allow_not_converged=True, **kw)
    before = fields(inst)
    assert not same(before, {f: np.zeros_like(v) for f, v in before.items()})
    bad = rp.copy()
    bad[np.flatnonzero(rp)[3]] = np.nan
    inst.set_loads(bad, mask)
    with pytest.raises(cp.CuplastError) as e:
        inst.solve(**kw)
    assert e.value.status == cp._capi.CP_ERR_BREAKDOWN
    assert same(fields(inst), before)
    inst.close()


@pytest.mark.parametrize("nx, ny", [(64, 26), (120, 80)])
@pytest.mark.parametrize("aitken", [0, 1])
def test_time_out(nx, ny, aitken, ctx, monkeypatch):  # noqa: F811
    arrays, rp, mask = strip(nx, ny)
    monkeypatch.setenv("CUPLAST_TEST_BARRIER_NS", "10000000")
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3, diagram="linear", sigma_t=2.0, k_t=2000.0))
    inst.set_loads(rp, mask)
    before = fields(inst)
    with pytest.raises(cp.CuplastError) as e:
        inst.solve(cg_tol=1e-8, outer_tol=1e-6, max_outer=3, precond=1, aitken=aitken)
    assert e.value.status == cp._capi.CP_ERR_TIMEOUT
    assert same(fields(inst), before)
    inst.close()
