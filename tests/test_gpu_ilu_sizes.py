"""Block ILU(0) of the condensed system at every block size (8 to 36) against
the numpy restatement: the compile-time factor with the next row's blocks
fetched ahead (up to 28), without (32) and the run-time factor (36), products
on tiles that B does and does not fill.

Tolerance: the apply is a chain of at most nf block products and solves with
blocks whose condition is below 1e3 here; explicit inverses differ from LU
solves by a few eps cond per block, 1e-10 leaves room for the chain."""
import numpy as np
import pytest

from conftest import rel_err
from mfem_euler2d_cpp_b200 import capi
from oracle import euler_oracle as eo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", range(1, 9))
def test_ilu_apply_at_every_block_size(k):
    nx, ny = 5, 4  # periodic: the last rows have lower entries on every side
    pb = eo.Problem(nx, ny, k, 37.0)
    u = pb.initial().reshape(-1, 4)
    u = (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel()
    dt = 0.02
    opts = capi.default_opts(form=capi.FORM_HDG, precond=capi.PC_ILU0)
    with capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0), opts) as ctx:
        ctx.upload("U", u)
        ctx.freeze(dt)
        ctx.upload("OLD", u * 0.999)
        ctx.set_dt(dt)
        ctx.residual()
        ctx.condense()
        ctx.pc_factor(True)
        b = np.cos(0.37 * np.arange(ctx.nl))
        x = ctx.pc_apply(b)
    pb.freeze(u, dt, True)
    pb.old = u * 0.999
    ilu = eo.BlockILU0(eo.solver_graph(pb, True), pb.t)
    pb.condense(u, pb.residual(u))
    eo.fill_hdg_ilu(pb, ilu)
    ilu.factor()
    assert rel_err(x, ilu(b)) < 1e-10
