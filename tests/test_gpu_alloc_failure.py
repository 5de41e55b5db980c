"""Every device allocation of a Newton update refused in turn: the call returns
EG_ERR_OUT_OF_MEMORY, and the same call on the same context, memory being there
again, gives bit for bit what a context that was never refused gives."""
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
    return ctx


def _update(ctx):
    ctx.residual()
    ctx.newton_update(ctx.cell_norm("R"), ctx.cell_norm("OLD"))
    return ctx.download("DU")


CASES = {
    "hdg": (6, 5, 2, dict()),
    "hdg_k7": (3, 2, 7, dict()),
    "hdg_mixed": (6, 5, 2, dict(precision=capi.PRECISION_MIXED)),
    "hdg_ilu": (6, 5, 2, dict(precond=capi.PC_ILU0)),
    "dg": (6, 5, 2, dict(form=capi.FORM_DG)),
    "dg_ilu": (6, 5, 1, dict(form=capi.FORM_DG, precond=capi.PC_ILU0)),
    "dg_full": (6, 5, 1, dict(form=capi.FORM_DG, assembly=capi.ASSEMBLY_FULL)),
    "hdg_dense": (4, 3, 1, dict(assembly=capi.ASSEMBLY_FULL, solver=capi.SOLVER_DENSE)),
}


@pytest.mark.parametrize("name", CASES)
def test_update_after_each_refused_allocation(name):
    nx, ny, k, opts = CASES[name]
    with _context(nx, ny, k, **opts) as ctx:
        want = _update(ctx)
    for nth in range(1, 64):
        with _context(nx, ny, k, **opts) as ctx:
            ctx.set_alloc_failure(nth)
            try:
                got = _update(ctx)
            except capi.EngineError as e:
                assert e.status == 17
                got = None
            ctx.set_alloc_failure(0)
            if got is not None:  # fewer allocations than nth
                assert nth > 1 and np.array_equal(got, want)
                return
            assert np.array_equal(_update(ctx), want)
    raise AssertionError("more allocations than expected")


@pytest.mark.parametrize("form", [capi.FORM_DG, capi.FORM_HDG])
def test_solve_without_refresh_needs_an_earlier_one(form):
    with _context(5, 4, 2, form=form) as ctx:
        ctx.residual()
        if form == capi.FORM_HDG:
            ctx.condense()
        rhs = np.cos(0.3 * np.arange(ctx.nl if form == capi.FORM_HDG else ctx.nu)) + 0.2
        with pytest.raises(capi.EngineError) as e:
            ctx.linear_solve(rhs, x0=0.5 * rhs, refresh=False)
        assert e.value.status == 1
        x, _, _ = ctx.linear_solve(rhs)
        y, _, _ = ctx.linear_solve(rhs, x0=x, refresh=False)
        assert np.allclose(x, y, rtol=1e-8, atol=1e-10)
