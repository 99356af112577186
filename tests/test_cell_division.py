"""Division of a cell index by a grid extent as multiply and shift (cell_coords,
fl_device.cuh; division_by, fl_host.cpp): exact for every index below 2^31."""
import numpy as np


def division_by(d):
    L = 1
    while (1 << L) < d:
        L += 1
    return ((1 << (31 + L)) + d - 1) // d, L - 1


def test_quotients_are_exact():
    rng = np.random.default_rng(3)
    top = np.uint64(2**31 - 1)
    for d in list(range(2, 300)) + [511, 512, 513, 1000, 1023, 1024, 1025, 65535, 2**20 + 7, 2**30]:
        mul, shift = division_by(d)
        assert mul < 2**32
        near = (rng.integers(0, 2**31 // d, 200, dtype=np.uint64) * np.uint64(d))[:, None] + np.arange(-1, 2).astype(np.int64)
        n = np.concatenate([near.astype(np.int64).ravel(), rng.integers(0, 2**31, 500), [0, 1, d - 1, d, 2**31 - 1]])
        n = np.clip(n, 0, int(top)).astype(np.uint64)
        q = (n * np.uint64(mul) >> np.uint64(32)) >> np.uint64(shift)
        assert np.array_equal(q, n // np.uint64(d)), d
