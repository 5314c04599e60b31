"""The cluster exchange of the on-chip CG: every halo record that a CTA reads
is the one its owner wrote for this iteration. A record of an earlier
iteration would change the sums, so a solve is run again and again, beside
other work on the GPU, in clusters of every size and in node orders that make
nearly all neighbours remote: it has to end the same bit for bit each time,
within the residual bound of the on-chip CG's tests."""
import threading
import time

import numpy as np
import pytest

import cudaplasticity_b200 as cp
from test_gpu_chip import EPS64, check, ctx, residual, solve, strip  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form, nx, ny", [("c1", 16, 30), ("c2", 32, 31), ("c4", 64, 26), ("c4", 96, 21),
                                          ("c10", 64, 65), ("c12", 96, 64)])
@pytest.mark.parametrize("elem, shuffle", [("q4", None), ("t3", 5)])
def test_records_are_current(form, nx, ny, elem, shuffle, ctx, monkeypatch):  # noqa: F811
    monkeypatch.setenv("CUPLAST_CHIP_FORM", form)
    p = strip(nx, ny, elem, shuffle)
    want, rep, csr = solve(ctx, p)
    check(p, want, rep, csr, 1e-11)
    stop = threading.Event()

    def other():
        c = cp.Context(0)
        while not stop.is_set():
            solve(c, strip(60, 50))
        c.close()

    beside = threading.Thread(target=other)
    beside.start()
    try:
        for _ in range(20):
            u, again, _ = solve(ctx, p)
            assert again["cg_iters"] == rep["cg_iters"] and np.array_equal(u, want)
    finally:
        stop.set()
        beside.join()


@pytest.mark.parametrize("nx, ny", [(2, 2), (64, 26), (96, 64), (120, 80)])
@pytest.mark.parametrize("precision", [cp.CP_PREC_FP64, cp.CP_PREC_MIXED])
def test_waits_are_limited_in_time(nx, ny, precision, ctx, monkeypatch):  # noqa: F811
    """With CUPLAST_TEST_BARRIER_NS set no CTA of a cluster sends its sums (of a grid: under the number that is waited
    for), so every wait runs out, after that time and not a number of rounds: the solve returns CP_ERR_TIMEOUT within
    a few of them, the kernel ends by itself and the context stays usable."""
    p = strip(nx, ny)
    solve(ctx, p, precision=precision)
    monkeypatch.setenv("CUPLAST_TEST_BARRIER_NS", "300000000")
    t = time.monotonic()
    with pytest.raises(cp.CuplastError) as e:
        solve(ctx, p, precision=precision)
    t = time.monotonic() - t
    assert e.value.status == cp._capi.CP_ERR_TIMEOUT
    assert 0.3 <= t <= 5.0  # a wait of each side of the exchange, and the set-up
    monkeypatch.delenv("CUPLAST_TEST_BARRIER_NS")
    check(p, *solve(ctx, p), 1e-11)


# a cluster of 4, of 8 and of 16 CTAs
@pytest.mark.parametrize("nx, ny", [(64, 26), (96, 60), (120, 80)])
def test_batch_that_gives_up(nx, ny, ctx, monkeypatch):  # noqa: F811
    """The same in a batch: each of its on-chip solves ends by itself with CP_ERR_TIMEOUT, and the context stays
    usable."""
    p = strip(nx, ny)
    arrays, rp, mask = p
    kw = dict(cg_tol=1e-11, outer_tol=1e300, inner_tol=1e-3, max_outer=1, max_cg=100000, precond=1)
    for withheld in (True, False):
        if withheld:
            monkeypatch.setenv("CUPLAST_TEST_BARRIER_NS", "50000000")
        batch = cp.Batch(ctx, max_instances=3)
        monkeypatch.delenv("CUPLAST_TEST_BARRIER_NS", raising=False)
        insts = [cp.Instance(ctx, arrays, cp.material(210000.0, 0.3)) for _ in range(3)]
        for i in insts:
            i.set_loads(rp, mask)
            batch.add(i, **kw)
        t = time.monotonic()
        batch.run()
        t = time.monotonic() - t
        reps = [r for _, _, r in batch.harvest()]
        assert len(reps) == 3
        if withheld:
            assert [r["status"] for r in reps] == [cp._capi.CP_ERR_TIMEOUT] * 3 and t <= 5.0
        else:
            for i, r in zip(insts, reps):
                res, gap = residual(p, i.field("uv"), i.csr())
                assert r["status"] == 0 and res <= 1e-11 + 2 * 20 * EPS64 * gap
        for i in insts:
            i.close()
        batch.close()


@pytest.mark.parametrize("nx, ny", [(64, 26), (96, 60), (120, 80)])
def test_batch_residuals_are_of_the_whole_x(nx, ny, ctx):  # noqa: F811
    """The FP64 residual of a batch's solve reads every CTA's x: with an inner tolerance that replaces it every few
    iterations the result is the same bit for bit, alone and again."""
    arrays, rp, mask = strip(nx, ny, "q4", 11)
    out = []
    for _ in range(6):
        batch = cp.Batch(ctx, max_instances=1)
        i = cp.Instance(ctx, arrays, cp.material(210000.0, 0.3))
        i.set_loads(rp, mask)
        batch.add(i, cg_tol=1e-10, outer_tol=1e300, inner_tol=0.3, max_outer=1, max_cg=100000, precond=1)
        batch.run()
        rep = batch.harvest()[0][2]
        assert rep["status"] == 0 and rep["cg_rel_res"] <= 1e-10
        out.append(i.field("uv"))
        i.close()
        batch.close()
    assert all(np.array_equal(u, out[0]) for u in out)
