"""The CG's general form in all precisions, against the oracle: blocks with more chunks
than warps, with operands resident for all of them, for some and for few, rows that are
not a multiple of four cells, and more chunks per block than its table holds (512)."""
import numpy as np
import pytest

from fluidgb import FL_CG_F32, FL_CG_F64, FL_CG_F64_IEEE, solve_pressure

from test_gpu_cg_forms import field

pytestmark = pytest.mark.gpu

# (grid, filled fraction of x, y, z) -> chunks of a block on 152 SMs
CASES = [
    ((97, 91, 90), (1, 1, 1)),        # 20, all resident, scalar loads
    ((128, 120, 90), (1, 1, 1)),      # 35, the last of them not resident
    ((250, 120, 250), (1, 1, 1)),     # 192, scalar loads
    ((256, 120, 250), (0.4, 1, 1)),   # 192 of half-empty chunks
]
LARGE = [(288, 284, 288), (287, 286, 290)]  # 600 and more


@pytest.mark.parametrize("precision", [FL_CG_F64, FL_CG_F64_IEEE])
@pytest.mark.parametrize("dims,fill", CASES)
def test_extended_forms_follow_the_oracle(oracle, dims, fill, precision):
    # alpha and beta differ from the oracle's by at most one f32 rounding (6e-8) each: eight
    # iterations by less than 1e-5 of the largest pressure
    ct, div, p0 = field(dims, fill)
    args = (ct, div, dims, 1.0, 1.0, 1.0, 8, True, p0)
    got, _ = solve_pressure(*args, tolerance=0.0, precision=precision)
    want, _ = oracle.solve_pressure(*args, tolerance=0.0, precision=FL_CG_F64)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("dims,fill", CASES[:2])
def test_f32_equals_the_oracle(oracle, dims, fill):
    ct, div, p0 = field(dims, fill)
    args = (ct, div, dims, 1.0, 1.0, 1.0, 8, True, p0)
    got, _ = solve_pressure(*args, tolerance=0.0, precision=FL_CG_F32)
    want, _ = oracle.solve_pressure(*args, tolerance=0.0, precision=FL_CG_F32)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dims", [(33, 30, 31), (128, 40, 30)])
def test_subnormal_terms(oracle, dims):
    # FL_CG_F64_IEEE converts such terms in another way than normal ones
    ct, div, p0 = field(dims, (1, 1, 1))
    div = np.where(np.random.default_rng(8).uniform(size=div.shape) < 0.3, div * np.float32(1e-40), div).astype(np.float32)
    assert ((div != 0) & (np.abs(div) < 1e-38)).any()
    for iters in (1, 8):
        args = (ct, div, dims, 1.0, 1.0, 1.0, iters, False, p0)
        got, sg = solve_pressure(*args, tolerance=0.0, precision=FL_CG_F64_IEEE)
        want, so = oracle.solve_pressure(*args, tolerance=0.0, precision=FL_CG_F64)
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("dims", LARGE)
def test_more_chunks_than_the_table_holds(oracle, dims):
    ct, div, p0 = field(dims, (1, 1, 1))
    args = (ct, div, dims, 1.0, 1.0, 1.0, 3, True, p0)
    for precision in (FL_CG_F32, FL_CG_F64, FL_CG_F64_IEEE):
        got, sg = solve_pressure(*args, tolerance=0.0, precision=precision)
        if precision != FL_CG_F64_IEEE:  # one oracle for both extended forms
            want, so = oracle.solve_pressure(*args, tolerance=0.0, precision=precision)
        if precision == FL_CG_F32:
            assert np.array_equal(got, want) and sg["rs_final"] == so["rs_final"]
        else:
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
