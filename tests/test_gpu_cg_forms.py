"""The CG's ways of dividing a solve, against the oracle: chunks in registers or
in turn, whole segments, heads with tails, split segments, and rows that are not
a multiple of four cells (scalar loads)."""
import numpy as np
import pytest

from fluidgb import FL_CG_F32, FL_CG_F64, FL_CG_F64_IEEE, solve_pressure

pytestmark = pytest.mark.gpu

# (grid, filled fraction of x, y, z) -> what the plan does with its 256-cell chunks
CASES = [
    ((5, 5, 5), (1, 1, 1)),              # one chunk, partly past the grid's end
    ((16, 16, 16), (1, 1, 1)),           # one block
    ((13, 3, 90), (1, 1, 1)),            # ragged rows, a single interior layer
    ((33, 30, 31), (0.9, 0.7, 1)),       # several segments per block, scalar loads
    ((64, 64, 64), (0.5, 0.4, 1)),       # half of the warps
    ((128, 128, 128), (0.5, 0.5, 0.5)),  # one segment per block, one chunk per warp
    ((128, 128, 72), (0.3, 0.2, 1)),     # heads and tails
    ((126, 128, 130), (0.5, 0.5, 0.52)),  # the same with scalar loads
    ((128, 64, 72), (1, 1, 1)),          # two chunks per warp
    ((250, 120, 250), (1, 1, 1)),        # split segments, scalar loads
    ((256, 120, 250), (0.4, 1, 1)),      # split segments, half-empty chunks
]


def field(dims, fill, seed=7):
    nx, ny, nz = dims
    rs = np.random.RandomState(seed)
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    ct = np.where((i < fill[0] * nx) & (j < fill[1] * ny) & (k < fill[2] * nz), 1, 2).astype(np.uint8)
    ct[rs.uniform(size=ct.shape) < 0.02] = 0
    ct[rs.uniform(size=ct.shape) < 0.02] = 2
    ct[0], ct[-1], ct[:, 0], ct[:, -1], ct[:, :, 0], ct[:, :, -1] = 0, 0, 0, 0, 0, 0
    div = np.where(ct == 1, rs.standard_normal(ct.shape), 0).astype(np.float32)
    p0 = np.where(ct == 1, rs.standard_normal(ct.shape), 0).astype(np.float32)
    return ct, div, p0


@pytest.mark.parametrize("dims,fill", CASES)
def test_f32_equals_the_oracle(oracle, dims, fill):
    ct, div, p0 = field(dims, fill)
    for iters, warm in ((1, False), (4, True)):
        args = (ct, div, dims, 1.0, 1.0, 1.0, iters, warm, p0)
        got, sg = solve_pressure(*args, tolerance=0.0, precision=FL_CG_F32)
        want, so = oracle.solve_pressure(*args, tolerance=0.0, precision=FL_CG_F32)
        assert np.array_equal(got, want)
        assert sg["cg_iterations"] == so["cg_iterations"] and sg["rs_final"] == so["rs_final"]


@pytest.mark.parametrize("precision", [FL_CG_F64, FL_CG_F64_IEEE])
@pytest.mark.parametrize("dims,fill", CASES[:-2])
def test_extended_forms_follow_the_oracle(oracle, dims, fill, precision):
    # The vectors are the same f32 arithmetic; the dot products agree to about
    # 1e-14, so alpha and beta differ by at most one f32 rounding (6e-8) each
    # and eight iterations by less than 1e-5 of the largest pressure.
    ct, div, p0 = field(dims, fill)
    args = (ct, div, dims, 1.0, 1.0, 1.0, 8, True, p0)
    got, _ = solve_pressure(*args, tolerance=0.0, precision=precision)
    want, _ = oracle.solve_pressure(*args, tolerance=0.0, precision=FL_CG_F64)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
