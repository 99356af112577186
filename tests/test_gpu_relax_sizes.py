"""fl_relax_pressure over the forms of its launch: fewer blocks than the chip has,
one group of 32 cells and a remainder, all blocks, the last size that fits the
blocks' lists and the first one that does not, and more sweeps than one launch
takes.  Cells of all three types at random; bit for bit against the oracle."""
import numpy as np
import pytest

from fluidgb import FL_RELAX_JACOBI, FL_RELAX_RBGS, _abi

pytestmark = pytest.mark.gpu

SOLID, LIQUID, AIR = 0, 1, 2


def random_field(dims, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    ct = np.full((nz, ny, nx), SOLID, np.uint8)
    inner = ct[1:-1, 1:-1, 1:-1]
    inner[:] = rng.choice(np.array([SOLID, LIQUID, AIR], np.uint8), size=inner.shape, p=[0.25, 0.5, 0.25])
    return ct.reshape(-1), rng.standard_normal(nx * ny * nz).astype(np.float32)


@pytest.mark.parametrize("method", [FL_RELAX_JACOBI, FL_RELAX_RBGS])
@pytest.mark.parametrize("dims,iters", [((3, 3, 3), 4), ((4, 5, 3), 9), ((33, 7, 10), 5), ((31, 67, 45), 6),
                                        ((67, 70, 69), 3), ((152, 149, 137), 2), ((153, 149, 137), 2),
                                        ((6, 5, 4), 8193)])
def test_relax_sizes(fluidlib, oracle, method, dims, iters):
    ref = oracle.ref_jacobi_solve if method == FL_RELAX_JACOBI else oracle.ref_rbgs_solve
    ct, div = random_field(dims, sum(dims) + iters)
    got = _abi.relax_pressure(ct, div, dims, 0.5, 1.0, 0.25, method, iters)
    assert np.array_equal(got, ref(dims, 0.5, 1.0, 0.25, ct, div, iters))
