"""The cell inverses of the HDG condensation and the DG block Jacobi at every
degree, against numpy's pivoted solves of the oracle's cell matrices.

A step of positive size is the ordinary case. A negative one makes I minus a
dissipative operator, whose natural-order pivot blocks are badly scaled: those
cells must be found by the elimination's own check and solved again with row
pivoting. Both sides solve with backward error of a few eps, so each cell's
result may differ by a small multiple of eps cond(A); 64 covers the m <= 324
rows (the constant grows like sqrt(m)), 256 the trace sums over two cells."""
import sys

import numpy as np
import pytest

from conftest import ROOT
from mfem_euler2d_cpp_b200 import capi

sys.path.insert(0, str(ROOT / "oracle"))
import euler_oracle as oracle  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
MESHES = {0: (7, 3), 1: (6, 5), 2: (5, 4), 3: (5, 4), 4: (4, 3), 5: (3, 3), 6: (3, 2), 7: (3, 2), 8: (2, 2)}


def _setup(k, factor, form):
    nx, ny = MESHES[k]
    p = oracle.Problem(nx, ny, k, 37.0)
    u = p.initial().reshape(-1, 4)
    u = (u.mean(axis=0) + 0.2 * (u - u.mean(axis=0))).ravel()
    p.freeze(u, 1.0)
    p.dt = factor * 0.24 / p.wave_rate()
    ctx = capi.Context(capi.simple_wave_desc(nx, ny, k, 37.0), capi.default_opts(form=form))
    ctx.upload("U", u)
    ctx.freeze(p.dt)
    ctx.set_dt(p.dt)
    return p, u, ctx


@pytest.mark.parametrize("factor", [1.0, -1.0, -2.0])
@pytest.mark.parametrize("k", range(9))
def test_condensation(k, factor):
    p, u, ctx = _setup(k, factor, capi.FORM_HDG)
    with ctx:
        rng = np.random.default_rng(k)
        r, v, lam = rng.standard_normal(p.nu), rng.standard_normal(p.nl), rng.standard_normal(p.nl)
        A = p.hdg_cell_pieces(u)[0]
        cond = np.linalg.cond(A)
        X, y, rhs, D = p.condense(u, r)
        ctx.upload("R", r)
        for _ in range(2):  # a second condensation starts from an empty list of cells to solve again
            ctx.condense()
        got = ctx.download("X").reshape(p.n, 4 * p.t, p.m).transpose(0, 2, 1)
        err = np.linalg.norm(got - X, axis=(1, 2)) / np.linalg.norm(X, axis=(1, 2))
        assert np.all(err < 64 * EPS * cond)
        got = ctx.download("Y").reshape(p.n, p.m)
        err = np.linalg.norm(got - y, axis=1) / np.linalg.norm(y, axis=1)
        assert np.all(err < 64 * EPS * cond)
        tol = 256 * EPS * cond.max()
        for a, b in ((ctx.download("RHS"), rhs), (ctx.schur_apply(v), p.schur_apply(v)), (ctx.recover(lam), p.recover(lam))):
            assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


@pytest.mark.parametrize("factor", [1.0, -1.0, -2.0])
@pytest.mark.parametrize("k", range(9))
def test_dg_block_jacobi(k, factor):
    p, u, ctx = _setup(k, factor, capi.FORM_DG)
    with ctx:
        J = p.dg_jacobi_blocks(u)
        cond = np.linalg.cond(J)
        b = np.random.default_rng(k).standard_normal(p.nu)
        want = np.linalg.solve(J, b.reshape(p.n, p.m, 1))[..., 0]
        for _ in range(2):
            ctx.pc_factor(True)
        got = ctx.pc_apply(b).reshape(p.n, p.m)
        err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert np.all(err < 64 * EPS * cond)
