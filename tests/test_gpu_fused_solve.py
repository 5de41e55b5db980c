"""The one-launch GMRES of the block-Jacobi solves: sizes where its split can
go wrong (fewer cells than SMs, one cell more than a whole number per CTA,
slices of a cell shared by warps, the lowest and highest degree), a restart
inside the solve, a non-zero guess and the bounded waits.

The solve stops when the weighted residual is below 1e-12 of the weighted
right-hand side. The weights len / ew_j differ by less than 1e2 within a
mesh used here (the DG form: the Gauss weights), so the plain 2-norm ratio, formed with the separate operator
kernels, is below 1e-10."""
import numpy as np
import pytest

from mfem_euler2d_cpp_b200 import capi

pytestmark = pytest.mark.gpu


def _context(nx, ny, k, form=capi.FORM_HDG, **opts):
    d = capi.simple_wave_desc(nx, ny, k, 37.0)
    ctx = capi.Context(d, capi.default_opts(form=form, **opts))
    ctx.initial()
    # the wave at a fifth of its amplitude: its traces stay admissible on meshes of a few cells
    u = ctx.download("U").reshape(-1, 4)
    ctx.upload("U", (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel())
    dt = 0.24 / ctx.freeze(1e-3)
    ctx.freeze(dt)
    ctx.upload("OLD", ctx.download("U") * 0.999)
    ctx.set_dt(dt)
    ctx.residual()
    if form == capi.FORM_HDG:
        ctx.condense()
    return ctx


def _rel_residual(ctx, form, x, rhs):
    ax = ctx.schur_apply(x) if form == capi.FORM_HDG else ctx.dg_apply(x)
    return np.linalg.norm(ax - rhs) / np.linalg.norm(rhs)


HDG_SIZES = [(2, 2, 0), (5, 3, 1), (149, 2, 1), (13, 11, 2), (12, 12, 3), (37, 9, 3), (7, 5, 4), (20, 15, 4),
             (3, 2, 8), (15, 11, 7)]


@pytest.mark.parametrize("precision", [capi.PRECISION_FP64, capi.PRECISION_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,k", HDG_SIZES)
def test_hdg_solution_satisfies_the_separate_operator(nx, ny, k, precision):
    with _context(nx, ny, k, precision=precision) as ctx:
        rhs = np.cos(0.3 * np.arange(ctx.nl)) + 0.2
        x, eq, st = ctx.linear_solve(rhs)
        assert st.count > 0 and st.residual <= 1e-12
        assert _rel_residual(ctx, capi.FORM_HDG, x, rhs) < 1e-10
        # from a perturbed solution (non-zero guess), without a new factor
        y, _, _ = ctx.linear_solve(rhs, x0=x * (1 + 1e-6), refresh=False)
        assert _rel_residual(ctx, capi.FORM_HDG, y, rhs) < 1e-10


@pytest.mark.parametrize("nx,ny,k", [(2, 2, 0), (63, 45, 1), (13, 11, 2), (37, 9, 3), (7, 5, 4), (11, 7, 6), (3, 2, 8)])
def test_dg_solution_satisfies_the_separate_operator(nx, ny, k):
    with _context(nx, ny, k, form=capi.FORM_DG) as ctx:
        rhs = np.cos(0.3 * np.arange(ctx.nu)) + 0.2
        x, _, st = ctx.linear_solve(rhs)
        assert st.count > 0 and st.residual <= 1e-12
        assert _rel_residual(ctx, capi.FORM_DG, x, rhs) < 1e-10
        y, _, _ = ctx.linear_solve(rhs, x0=x * (1 + 1e-6), refresh=False)
        assert _rel_residual(ctx, capi.FORM_DG, y, rhs) < 1e-10


@pytest.mark.parametrize("restart", [1, 5, 24, 30])
def test_restart_lengths(restart):
    """Several cycles inside one launch (restart 1, 5), the longest the launch
    takes (24) and one that runs in the host-driven loop (30)."""
    with _context(9, 8, 2, restart=restart, linear_tol=1e-10) as ctx:
        rhs = np.sin(0.7 * np.arange(ctx.nl))
        x, _, st = ctx.linear_solve(rhs, linear_tol=1e-10)
        assert st.residual <= 1e-10
        assert _rel_residual(ctx, capi.FORM_HDG, x, rhs) < 1e-8


def test_iteration_limit_and_reuse():
    with _context(9, 8, 2, max_krylov=3) as ctx:
        rhs = np.sin(0.7 * np.arange(ctx.nl))
        with pytest.raises(capi.EngineError) as e:
            ctx.linear_solve(rhs)
        assert e.value.status == 12


def test_bounded_waits_report_and_leave_the_context_usable():
    with _context(12, 10, 3) as ctx:
        rhs = np.sin(0.7 * np.arange(ctx.nl))
        want, _, _ = ctx.linear_solve(rhs)
        ctx.set_ilu_wait(2_000_000, starve=True)
        with pytest.raises(capi.EngineError) as e:
            ctx.linear_solve(rhs)
        assert e.value.status == 24
        ctx.set_ilu_wait(0, starve=False)
        got, _, _ = ctx.linear_solve(rhs)
        assert np.array_equal(got, want)
