"""The adjoint step on grids of unequal and odd extents: against central differences of
the FP64 oracle, and the two forms of the face gather (csrc/fl_adjoint.cu) against each
other.

A lone particle with a NaN gradient sends the whole step through the general form; no
other particle shares a face with it.  The two forms' weights are the same numbers (a
fraction of a cell and its distance from a half are exact from the first cell on) added
in the same order, so every other gradient is the same to the bit."""
import numpy as np
import pytest

from fluidgb import FL_CG_F64, scenes

from test_gpu_adjoint import adjoint_grads, fd_errors
from test_gpu_adjoint_reach import gradient

pytestmark = pytest.mark.gpu


def filled(dims, lo, hi, per_cell, seed):
    """`per_cell` particles at random in every interior cell between the fractions lo and hi of the tank."""
    rng = np.random.default_rng(seed)
    d = np.array(dims)
    a, b = np.maximum(1, (np.array(lo) * d).astype(int)), np.minimum(d - 1, (np.array(hi) * d).astype(int))
    cells = np.stack(np.meshgrid(*[np.arange(s, e) for s, e in zip(a, b)], indexing="ij"), -1).reshape(-1, 3)
    pos = np.repeat(cells, per_cell, 0) + rng.uniform(0.06, 0.94, (cells.shape[0] * per_cell, 3))
    parts = np.zeros((pos.shape[0], 8), np.float32)
    parts[:, :3] = pos / dims[0]
    parts[:, 4:7] = 0.1 * rng.standard_normal((pos.shape[0], 3))
    return parts[rng.permutation(pos.shape[0])]


@pytest.mark.parametrize("dims,order", [((21, 19, 23), 1), ((20, 25, 17), 2), ((17, 22, 19), 1)])
def test_matches_finite_differences(oracle, dims, order):
    pytest.importorskip("torch")
    p = scenes.params_for(dims[0], ny=dims[1], nz=dims[2], iters=500, tol=1e-6, precision=FL_CG_F64, stiffness=0.0, advect_order=order)
    parts = filled(dims, (0.3, 0.35, 0.3), (0.7, 0.65, 0.7), 8, sum(dims))
    gv, gg = adjoint_grads(p, parts, 1, 1)
    errs = fd_errors(oracle, p, parts, 1, gv, gg)
    print("%s order %d: rel errors %s" % (dims, order, ["%.2e" % e for e in errs]))
    assert len(errs) >= 2 and max(errs) < 1e-3, errs


@pytest.mark.parametrize("dims", [(9, 11, 10), (12, 7, 9), (33, 17, 18), (31, 30, 29), (40, 37, 22)])
@pytest.mark.parametrize("order", [1, 2])
def test_both_gathers_give_the_same_bits(fluidlib, dims, order):
    pytest.importorskip("torch")
    p = scenes.params_for(dims[0], ny=dims[1], nz=dims[2], iters=30, tol=1e-5, advect_order=order)
    p.cls[0] = 2.0  # the lone particle's cell is air
    parts = filled(dims, (0.62, 0, 0), (1, 1, 1), 3, sum(dims))  # up to the high sides
    lone = np.zeros((1, 8), np.float32)
    lone[0, :3] = np.float32(2.25 / dims[0])
    parts = np.concatenate([parts, lone, parts[:1]])
    want, want_grav = gradient(p, parts, 0.0)
    got, grav = gradient(p, parts, np.float32([np.nan, 0, 0, 0, np.nan, 0, 0, 0]))
    others = np.arange(parts.shape[0]) != parts.shape[0] - 2
    assert np.isfinite(want).all() and not np.isfinite(got[~others]).all()
    assert np.array_equal(got[others], want[others]) and np.array_equal(grav, want_grav)
