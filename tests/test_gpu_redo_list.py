"""The list of cells that a condensation or DG factor solves again, after a call
that ended between filling it and reading it: the next call starts an empty one.

The calls end on a refused allocation. A step of negative size makes every cell
one to be solved again (a list of n entries, so a second one behind it would
leave the buffer). Each cell's result is compared with numpy's pivoted solve of
the oracle's matrix; both have a backward error of a few eps, 64 eps cond(A)
covers the m <= 324 rows."""
import sys

import numpy as np
import pytest

from conftest import ROOT
from mfem_euler2d_cpp_b200 import capi

sys.path.insert(0, str(ROOT / "oracle"))
import euler_oracle as oracle  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
MESHES = {3: (4, 3), 6: (3, 2), 8: (2, 2)}


def _setup(k, form, factor=-1.0):
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


def _refused(ctx, nth, call):
    ctx.set_alloc_failure(nth)
    with pytest.raises(capi.EngineError) as e:
        call()
    assert e.value.status == 17
    ctx.set_alloc_failure(0)


def _check_condensation(ctx, p, u, r):
    ctx.upload("R", r)
    ctx.condense()
    X = p.condense(u, r)[0]
    cond = np.linalg.cond(p.hdg_cell_pieces(u)[0])
    got = ctx.download("X").reshape(p.n, 4 * p.t, p.m).transpose(0, 2, 1)
    err = np.linalg.norm(got - X, axis=(1, 2)) / np.linalg.norm(X, axis=(1, 2))
    assert np.all(err < 64 * EPS * cond)


@pytest.mark.parametrize("k", [6, 8])
def test_condensation_after_a_refused_slab(k):
    """The cluster scratch is the first allocation, the LU slab the second."""
    p, u, ctx = _setup(k, capi.FORM_HDG)
    with ctx:
        r = np.random.default_rng(k).standard_normal(p.nu)
        ctx.upload("R", r)
        _refused(ctx, 2, ctx.condense)
        _check_condensation(ctx, p, u, r)
        held = ctx.device_bytes()
        _check_condensation(ctx, p, u, r)
        assert ctx.device_bytes() == held


def test_condensation_after_an_update_refused_behind_it():
    """The Schur preconditioner's blocks, allocated behind the condensation
    that filled the list."""
    p, u, ctx = _setup(3, capi.FORM_HDG)
    with ctx:
        r = np.random.default_rng(3).standard_normal(p.nu)
        ctx.upload("R", r)
        _refused(ctx, 1, lambda: ctx.newton_update(float(ctx.cell_norm("R")), float(ctx.cell_norm("OLD"))))
        _check_condensation(ctx, p, u, r)


@pytest.mark.parametrize("k", [3, 8])
def test_dg_factor_after_a_refused_slab(k):
    """Blocks and list are the first two allocations, the LU slab the third."""
    p, u, ctx = _setup(k, capi.FORM_DG)
    with ctx:
        _refused(ctx, 3, lambda: ctx.pc_factor(True))
        ctx.pc_factor(True)
        J = p.dg_jacobi_blocks(u)
        b = np.random.default_rng(k).standard_normal(p.nu)
        want = np.linalg.solve(J, b.reshape(p.n, p.m, 1))[..., 0]
        err = np.linalg.norm(ctx.pc_apply(b).reshape(p.n, p.m) - want, axis=1) / np.linalg.norm(want, axis=1)
        assert np.all(err < 64 * EPS * np.linalg.cond(J))
