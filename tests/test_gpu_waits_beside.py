"""Solves beside another context's: a launch whose CTAs wait for one another
starts with all of them or with none, so the time it waits for SMs that another
context's solves hold is not part of its waits.

The other context runs solves to their iteration limit (about 30 ms each) on 140
CTAs of an SM each; the solves beside need more CTAs than the SMs left, with a
bound of 3 ms for their waits."""
import threading

import numpy as np
import pytest

from mfem_euler2d_cpp_b200 import capi

pytestmark = pytest.mark.gpu


def _context(nx, ny, k, **opts):
    ctx = capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0), capi.default_opts(**opts))
    ctx.initial()
    u = ctx.download("U").reshape(-1, 4)
    ctx.upload("U", (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel())
    dt = 0.24 / ctx.freeze(1e-3)
    ctx.freeze(dt)
    ctx.upload("OLD", ctx.download("U") * 0.999)
    ctx.set_dt(dt)
    ctx.residual()
    ctx.condense()
    return ctx


@pytest.mark.parametrize("precond,others", [(capi.PC_JACOBI, 1), (capi.PC_JACOBI, 3), (capi.PC_ILU0, 1)])
def test_short_bounds_hold_beside_long_solves(precond, others):
    stop, started = threading.Event(), threading.Semaphore(0)
    statuses = []

    def long_solves():
        with _context(20, 14, 8, linear_tol=1e-30) as ctx:
            rhs = np.cos(0.3 * np.arange(ctx.nl)) + 0.2
            first = True
            while not stop.is_set():
                try:
                    ctx.linear_solve(rhs)
                    statuses.append(0)
                except capi.EngineError as e:
                    statuses.append(e.status)
                if first:
                    started.release()
                    first = False

    with _context(12, 10, 3, precond=precond) as ctx:
        rhs = np.cos(0.3 * np.arange(ctx.nl)) + 0.2
        want, _, _ = ctx.linear_solve(rhs)
        ctx.set_ilu_wait(3_000_000)
        threads = [threading.Thread(target=long_solves) for _ in range(others)]
        for t in threads:
            t.start()
        try:
            for _ in threads:
                assert started.acquire(timeout=120)
            for _ in range(8):
                got, _, _ = ctx.linear_solve(rhs)
                assert np.array_equal(got, want)
        finally:
            stop.set()
            for t in threads:
                t.join()
    assert set(statuses) == {12}
