"""Block ILU(0) sweeps whose rows read rows of their own CTA that have left its
shared-memory ring, and CTAs with more than one grid row, against the numpy
restatement; applied three times in a row, so that values of an earlier sweep
would show.

A CTA walks a grid row of 2 nx faces and keeps the last ring - W of them in
shared memory (ring: the largest power of two whose rows fit 48 KB; W <= 8
warps). The last cell of a periodic row depends on the first one, 2 nx rows
back: gone from 256 rows at B = 20 (nx = 130), from 128 at B = 28 and 36 (nx =
70), from 512 at B = 8 and 12 (nx = 260); a DG row has nx cells (64 at B = 64). With 300 grid rows the 296 CTAs of a
sweep at most take more than one.

Tolerance as in the other ILU tests: explicit inverses against LU solves."""
import numpy as np
import pytest

from conftest import rel_err
from mfem_euler2d_cpp_b200 import capi
from oracle import euler_oracle as eo

pytestmark = pytest.mark.gpu


def _problem(nx, ny, k, form):
    hdg = form == "hdg"
    pb = eo.Problem(nx, ny, k, 37.0)
    u = pb.initial().reshape(-1, 4)
    u = (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel()
    dt = 0.05 * min(pb.hx, pb.hy)
    ctx = capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0),
                       capi.default_opts(form=capi.FORM_HDG if hdg else capi.FORM_DG, precond=capi.PC_ILU0))
    ctx.upload("U", u)
    ctx.freeze(dt)
    ctx.upload("OLD", u * 0.999)
    ctx.set_dt(dt)
    ctx.residual()
    if hdg:
        ctx.condense()
    ctx.pc_factor(True)
    pb.freeze(u, dt, True)
    pb.old = u * 0.999
    return pb, u, ctx, hdg


@pytest.mark.parametrize("nx,ny,k,form", [(130, 3, 4, "hdg"), (70, 3, 6, "hdg"), (70, 3, 8, "hdg"), (260, 2, 1, "hdg"),
                                          (260, 2, 2, "hdg"), (3, 300, 1, "hdg"), (2, 300, 0, "hdg"), (200, 3, 2, "dg"),
                                          (3, 300, 2, "dg"), (70, 3, 3, "dg")])
def test_apply_against_the_restatement(nx, ny, k, form):
    pb, u, ctx, hdg = _problem(nx, ny, k, form)
    with ctx:
        ilu = eo.BlockILU0(eo.solver_graph(pb, hdg), pb.t if hdg else pb.m)
        if hdg:
            pb.condense(u, pb.residual(u))
            eo.fill_hdg_ilu(pb, ilu)
        else:
            eo.fill_dg_ilu(pb, ilu, u)
        ilu.factor()
        n = ctx.nl if hdg else ctx.nu
        for f in (0.37, 0.11, 0.73):
            b = np.cos(f * np.arange(n))
            assert rel_err(ctx.pc_apply(b), ilu(b)) < 1e-10


@pytest.mark.parametrize("nx,ny,k,form", [(130, 3, 4, "hdg"), (70, 3, 3, "dg")])
def test_waits_that_run_out_leave_the_context_usable(nx, ny, k, form):
    _, _, ctx, hdg = _problem(nx, ny, k, form)
    with ctx:
        b = np.cos(0.37 * np.arange(ctx.nl if hdg else ctx.nu))
        want = ctx.pc_apply(b)
        ctx.set_ilu_wait(limit_ns=1_000_000, starve=True)
        with pytest.raises(capi.EngineError) as e:
            ctx.pc_apply(b)
        assert e.value.status == 24
        ctx.set_ilu_wait()
        assert np.array_equal(ctx.pc_apply(b), want)
