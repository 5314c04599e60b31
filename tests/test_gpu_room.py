"""Device memory: where there is no room for what a faster form of the linear
solve needs, the solve takes the form without it, and keeps nothing of the
parts that did fit."""
import ctypes

import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import EPS64, check, ctx, residual, strip  # noqa: F401

pytestmark = pytest.mark.gpu


def pool_bytes(ctx):  # noqa: F811
    """Bytes in use in the device's default memory pool, which every instance allocates from."""
    rt = ctypes.CDLL("libcudart.so.12")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert cp._capi.lib().cp_context_synchronize(ctx._h) == 0
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0  # cudaMemPoolAttrUsedMemCurrent
    return used.value


def instance(ctx, problem):  # noqa: F811
    arrays, rp, mask = problem
    inst = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
    inst.set_loads(rp, mask)
    return inst


# the allocations of each form: a cluster's plan and scratch; a grid's, its exchange buffers too; u before a mixed solve;
# the half-K loop's widths (2), columns, mirrors and values
@pytest.mark.parametrize("env, nx, ny, precision, needs", [
    ({}, 64, 26, cp.CP_PREC_FP64, 2), ({}, 120, 80, cp.CP_PREC_FP64, 4), ({}, 64, 26, cp.CP_PREC_MIXED, 3),
    ({}, 120, 80, cp.CP_PREC_MIXED, 5),
    ({"CUPLAST_FP64_CG": "fused", "CUPLAST_HALF_K": "1"}, 120, 80, cp.CP_PREC_FP64, 5)])
def test_without_room(env, nx, ny, precision, needs, ctx, monkeypatch):  # noqa: F811
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    p = strip(nx, ny)
    kw = dict(cg_tol=1e-11, outer_tol=1e300, max_outer=1, precond=1, max_cg=100000, precision=precision, inner_tol=1e-3)
    base, held, launches = pool_bytes(ctx), [], []
    for k in [*range(1, needs + 2), 0]:
        monkeypatch.setenv("CUPLAST_TEST_NO_ROOM", str(k))
        inst = instance(ctx, p)
        rep = inst.solve(**kw)
        u, csr = inst.field("uv"), inst.csr()
        res, gap = residual(p, u, csr)
        if precision == cp.CP_PREC_FP64:
            check(p, u, rep, csr, 1e-11)
        else:
            assert rep["status"] == 0 and res <= 1e-11 + 2 * 20 * EPS64 * gap
        held.append(pool_bytes(ctx) - base)
        launches.append(rep["kernel_launches"])
        inst.close()
    assert pool_bytes(ctx) == base
    assert len(set(launches[:needs])) == 1 and launches[needs] == launches[needs + 1]
    if env:  # the iterations' kernel is another one, not their number of launches
        assert held[needs] > held[0]
    else:
        assert launches[needs] < launches[0] / 10
    # (a mixed solve without room for u keeps the plan that its FP64 solves use)
    want = held[:needs] if precision == cp.CP_PREC_FP64 else held[:needs - 1]
    assert len(set(want)) == 1 and held[needs] == held[needs + 1]


@pytest.mark.parametrize("nx, ny", [(64, 26), (96, 60), (120, 80)])
def test_batch_without_room(nx, ny, ctx, monkeypatch):  # noqa: F811
    p = strip(nx, ny)
    base, held = pool_bytes(ctx), []
    for k in (1, 2, 3, 0):
        monkeypatch.setenv("CUPLAST_TEST_NO_ROOM", str(k))
        inst = instance(ctx, p)
        batch = cp.Batch(ctx, max_instances=1)
        batch.add(inst, cg_tol=1e-11, outer_tol=1e300, inner_tol=1e-3, max_outer=1, max_cg=100000, precond=1)
        batch.run()
        rep = batch.harvest()[0][2]
        res, gap = residual(p, inst.field("uv"), inst.csr())
        assert rep["status"] == 0 and res <= 1e-11 + 2 * 20 * EPS64 * gap
        held.append(pool_bytes(ctx) - base)
        inst.close()
        batch.close()
    assert held[0] == held[1] < held[2] == held[3]
