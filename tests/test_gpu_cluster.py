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
from test_gpu_chip import check, ctx, solve, strip  # noqa: F401

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
    assert 0.3 <= t <= 0.3 * 3 + 0.5  # a wait of each side of the exchange, and the set-up
    monkeypatch.delenv("CUPLAST_TEST_BARRIER_NS")
    check(p, *solve(ctx, p), 1e-11)
