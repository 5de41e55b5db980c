"""Block ILU(0) contexts of one block size on meshes whose rows differ in
length, factored in turn: a context's factor does not depend on which other
contexts the process has built since."""
import numpy as np
import pytest

from mfem_euler2d_cpp_b200 import capi

pytestmark = pytest.mark.gpu


def _context(nx, ny, k, form):
    ctx = capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0), capi.default_opts(form=form, precond=capi.PC_ILU0))
    ctx.initial()
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


# 3 x 3 cells: the longest rows and most updates (the last faces depend on all sides); 2 x 2: the shortest
@pytest.mark.parametrize("k,form", [(4, capi.FORM_HDG), (6, capi.FORM_HDG), (7, capi.FORM_HDG), (8, capi.FORM_HDG),
                                    (1, capi.FORM_DG), (2, capi.FORM_DG)])
def test_factor_after_a_smaller_one(k, form):
    with _context(3, 3, k, form) as a, _context(12, 10 if k < 6 else 4, k, form) as b, _context(2, 2, k, form) as c:
        n = a.nl if form == capi.FORM_HDG else a.nu
        rhs = np.cos(0.37 * np.arange(n))
        a.pc_factor(True)
        want = a.pc_apply(rhs)
        for other in (b, c):
            other.pc_factor(True)
            a.pc_factor(True)
            assert np.array_equal(a.pc_apply(rhs), want)
