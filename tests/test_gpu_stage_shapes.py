"""The stages around the solver at sizes that cut their blocks and tiles short:
both P2G tile shapes (8 x 8 x 2 below some 1,200 tiles of 8^3), rows that are no
multiple of a vector, bins from empty to crowded, and particles on the walls.
Every array of the state against the oracle, exactly, after one and two steps."""
import numpy as np
import pytest

from fluidgb import scenes

from test_gpu_parity import assert_same_state, make_pair

pytestmark = pytest.mark.gpu


def scatter_particles(dims, per_cell, seed):
    """Uniform particles in the lower two thirds, 300 more in one cell, some on the walls."""
    rng = np.random.default_rng(seed)
    h = np.float32(1.0) / np.float32(dims[0])
    ext = np.array(dims, np.float32) * h
    n = int(per_cell * dims[0] * dims[1] * dims[2])
    pos = rng.random((n, 3), dtype=np.float32) * (ext * np.float32([1.0, 0.66, 1.0]) - 2 * h) + h
    crowd = ((np.array(dims) // 2 + rng.random((300, 3))) * h).astype(np.float32)
    wall = (rng.random((40, 3), dtype=np.float32) * (ext - 2 * h) + h).astype(np.float32)
    wall[:20, 0] = h
    wall[20:, 1] = ext[1] - h
    parts = np.zeros((n + 340, 8), np.float32)
    parts[:, :3] = np.concatenate([pos, crowd, wall])
    parts[:, 4:7] = rng.standard_normal((n + 340, 3)).astype(np.float32) * np.float32(0.5)
    return parts[rng.permutation(n + 340)]


@pytest.mark.parametrize("dims,per_cell", [((5, 5, 5), 1.0), ((9, 11, 10), 4.0), ((33, 17, 18), 2.0), ((40, 37, 21), 5.0),
                                           ((64, 48, 30), 3.0), ((97, 88, 90), 1.5), ((96, 104, 88), 1.0)])
def test_stages_match_oracle(fluidlib, oracle, dims, per_cell):
    p = scenes.params_for(dims[0], ny=dims[1], nz=dims[2], iters=8, stiffness=0.45)
    g, o = make_pair(oracle, p, scatter_particles(dims, per_cell, sum(dims)))
    for step in (1, 2):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, "%s step %d" % (dims, step))
    g.close()
    o.close()
