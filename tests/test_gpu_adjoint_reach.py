"""How far a particle's gradient reaches in fl_step_adjoint: no further than the faces
that it has a weight on, also when it is infinite or NaN."""
import numpy as np
import pytest

from fluidgb import Fluid, scenes

pytestmark = pytest.mark.gpu

N = 32
LONE = (26.25, 26.25, 26.25)  # in cells; x taps 25..27


def case(neighbour):
    """A block of liquid, and two single particles far above it (cells of one particle
    count as air here): the lone one and one that shares no tap with it."""
    p = scenes.params_for(N, iters=60, tol=1e-5)
    p.cls[0] = 2.0  # cells are liquid from two particles on
    block = scenes.seed_particles(N, lambda x, y, z: (x > 0.2) & (x < 0.5) & (y > 0.1) & (y < 0.4) & (z > 0.2) & (z < 0.5),
                                  seed=5, vel_sigma=0.1)
    single = np.zeros((2, 8), np.float32)
    single[:, :3] = np.array([LONE, neighbour]) / N + p.origin[0]
    single[:, 4:7] = 0.1
    return p, np.concatenate([block, single]).astype(np.float32)


def gradient(p, parts, lone):
    import torch
    n = parts.shape[0]
    f = Fluid(p, n)
    f.set_particles(parts)
    tape = f.tape(1)
    tape.record()
    _, ids = f.get_particles()
    g = np.random.default_rng(3).standard_normal((n, 8)).astype(np.float32)
    g[:, 3] = g[:, 7] = 0
    g[n - 2] = lone
    g_out = torch.from_numpy(g[ids]).cuda()
    g_in = torch.empty_like(g_out)
    grav = tape.adjoint(g_out.data_ptr(), g_in.data_ptr(), 300, 1e-6)
    out = g_in.cpu().numpy().copy(), np.array(grav, np.float32)
    tape.close()
    f.close()
    return out


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("neighbour", [(28.25, 26.25, 26.25), (26.25, 24.25, 26.25), (26.25, 26.25, 28.3), (28.2, 28.2, 24.3)])
def test_no_further_than_its_faces(fluidlib, value, neighbour):
    pytest.importorskip("torch")
    p, parts = case(neighbour)
    want, want_grav = gradient(p, parts, 0.0)
    lone = np.zeros(8, np.float32)
    lone[0] = lone[4] = value
    got, grav = gradient(p, parts, lone)
    others = np.arange(parts.shape[0]) != parts.shape[0] - 2
    assert np.isfinite(want).all() and np.isfinite(want_grav).all()
    assert not np.isfinite(got[~others]).all()
    assert np.abs(got[others] - want[others]).max() <= 1e-6 * np.abs(want[others]).max()
    assert np.abs(grav - want_grav).max() <= 1e-6 * np.abs(want_grav).max()
