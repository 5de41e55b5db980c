"""Block ILU(0) factors and sweeps that take longer than the bound of their
waits: the bound is on time without a finished row, so the CTAs at the end of
the wavefront may wait for all of it."""
import numpy as np
import pytest

from conftest import rel_err
from mfem_euler2d_cpp_b200 import capi
from oracle import euler_oracle as eo

pytestmark = pytest.mark.gpu


def _context(nx, ny, k, form):
    pb = eo.Problem(nx, ny, k, 37.0)
    u = pb.initial().reshape(-1, 4)
    u = (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel()
    dt = 0.05 * min(pb.hx, pb.hy)
    ctx = capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0), capi.default_opts(form=form, precond=capi.PC_ILU0))
    ctx.upload("U", u)
    ctx.freeze(dt)
    ctx.upload("OLD", u * 0.999)
    ctx.set_dt(dt)
    ctx.residual()
    if form == capi.FORM_HDG:
        ctx.condense()
    pb.freeze(u, dt, True)
    pb.old = u * 0.999
    return pb, u, ctx


def test_large_blocks_at_the_default_bound():
    """324 x 324 blocks: the factor takes about a second. Tolerance as in the other ILU
    tests (explicit inverses against LU solves)."""
    pb, u, ctx = _context(3, 12, 8, capi.FORM_DG)
    with ctx:
        ctx.pc_factor(True)
        b = np.cos(0.37 * np.arange(ctx.nu))
        x = ctx.pc_apply(b)
        ilu = eo.BlockILU0(eo.solver_graph(pb, False), pb.m)
        eo.fill_dg_ilu(pb, ilu, u)
        ilu.factor()
        assert rel_err(x, ilu(b)) < 1e-10


@pytest.mark.parametrize("nx,ny,k,form,limit", [(40, 60, 3, capi.FORM_HDG, 100_000), (16, 24, 4, capi.FORM_DG, 10_000_000)])
def test_a_bound_below_the_whole_sweep(nx, ny, k, form, limit):
    """Bounds several times a row's time (about 20 us and 2 ms in the factor) and
    a fraction of the whole factor's (about 2 ms and 80 ms)."""
    _, _, ctx = _context(nx, ny, k, form)
    with ctx:
        b = np.cos(0.37 * np.arange(ctx.nl if form == capi.FORM_HDG else ctx.nu))
        ctx.pc_factor(True)
        want = ctx.pc_apply(b)
        ctx.set_ilu_wait(limit)
        ctx.pc_factor(True)
        assert np.array_equal(ctx.pc_apply(b), want)
