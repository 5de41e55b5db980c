"""eg_newton_update with a residual_norm that is not the norm of EG_SLOT_R: the
increment is solved for the right-hand side in the slot, to that one's own
norm, so it is bit for bit the one of the consistent call. (The validation and
line-search criteria do take the number: a small one may end the call there,
with the increment formed.)"""
import ctypes as C

import numpy as np
import pytest

from mfem_euler2d_cpp_b200 import capi

pytestmark = pytest.mark.gpu

KINDS = {
    "dg": dict(form=capi.FORM_DG),
    "dg_ilu": dict(form=capi.FORM_DG, precond=capi.PC_ILU0),
    "dg_full": dict(form=capi.FORM_DG, assembly=capi.ASSEMBLY_FULL),
    "dg_dense": dict(form=capi.FORM_DG, assembly=capi.ASSEMBLY_FULL, solver=capi.SOLVER_DENSE),
    "hdg": dict(),
    "hdg_ilu": dict(precond=capi.PC_ILU0),
}


def _increment(factor, **opts):
    with capi.Context(capi.simple_wave_desc(6, 5, 2, 37.0), capi.default_opts(**opts)) as ctx:
        ctx.initial()
        u = ctx.download("U").reshape(-1, 4)
        ctx.upload("U", (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel())
        dt = 0.24 / ctx.freeze(1e-3)
        ctx.freeze(dt)
        ctx.upload("OLD", ctx.download("U") * 0.999)
        ctx.set_dt(dt)
        ctx.residual()
        iterations = None
        try:
            st = ctx.newton_update(factor * ctx.cell_norm("R"), ctx.cell_norm("OLD"))
            iterations = st.krylov_iterations
        except capi.EngineError as e:
            assert factor < 1 and e.status in (14, 15, 16)
        return ctx.download("DU"), iterations


@pytest.mark.parametrize("kind", KINDS)
def test_the_increment_does_not_depend_on_the_number(kind):
    want, iterations = _increment(1.0, **KINDS[kind])
    assert np.linalg.norm(want) > 0
    for factor in (1e4, 0.5, 0.0):
        got, its = _increment(factor, **KINDS[kind])
        # HDG refines its solve until the recovered residual meets the criterion, so
        # a smaller number may take further solves; DG has one solve
        if factor >= 1 or kind.startswith("dg"):
            assert np.array_equal(got, want)
            assert its is None or its == iterations
        else:
            assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("form", [capi.FORM_DG, capi.FORM_HDG])
def test_a_zero_right_hand_side_is_a_zero_increment(form):
    with capi.Context(capi.simple_wave_desc(6, 5, 2, 37.0), capi.default_opts(form=form)) as ctx:
        ctx.initial()
        u = ctx.download("U").reshape(-1, 4)
        ctx.upload("U", np.tile(u.mean(axis=0), len(u)))  # a uniform state: the residual at OLD = U
        ctx.freeze(1e-3)
        ctx.set_dt(1e-3)
        ctx.upload("R", np.zeros(ctx.nu))
        for number in (0.0, 1.0):
            ctx.newton_update(number, ctx.cell_norm("OLD"))
            assert not np.any(ctx.download("DU"))
            ctx.upload("R", np.zeros(ctx.nu))


@pytest.mark.parametrize("change", ["none", "upload", "residual", "desc"])
def test_the_norm_kept_from_the_residual_call_is_of_the_residual_in_the_slot(change):
    """EG_SLOT_R or the metric written between the residual call and the update."""
    results = []
    for kept in (True, False):
        d = capi.simple_wave_desc(6, 5, 2, 37.0)
        with capi.Context(d, capi.default_opts(form=capi.FORM_DG)) as ctx:
            ctx.initial()
            u = ctx.download("U").reshape(-1, 4)
            u = (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel()
            ctx.upload("U", u)
            dt = 0.24 / ctx.freeze(1e-3)
            ctx.freeze(dt)
            ctx.upload("OLD", u * 0.999)
            ctx.set_dt(dt)
            if kept:
                ctx.newton_residual()
            else:
                ctx.residual()
            if change == "upload":
                ctx.upload("R", 1e-3 * ctx.download("R"))
            elif change == "residual":
                ctx.upload("OLD", u * 0.9995)
                ctx.residual()
            elif change == "desc":
                d2 = capi.simple_wave_desc(6, 5, 2, 20.0)
                assert ctx.lib.eg_set_desc(ctx.h, C.byref(d2)) == capi.OK
            ctx.newton_update(1.0, ctx.cell_norm("OLD"))
            results.append(ctx.download("DU"))
    assert np.array_equal(results[0], results[1])
