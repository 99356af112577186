"""The tile order in which the CG plan lists chunks (k_cg_plan, fl_cg.cu), as
arithmetic: every chunk of a grid comes up exactly once, whatever the planes."""
import pytest

CHUNK, TILE_Y, TILE_Z = 256, 4, 4


def tile_order(nx, ny, nz):
    nchunks = (nx * ny * nz + CHUNK - 1) // CHUNK
    Z = max(1, nx * ny // CHUNK)
    planes = -(-nchunks // Z)
    ty = -(-Z // TILE_Y)
    for t in range(ty * -(-planes // TILE_Z)):
        y0 = TILE_Y * (t % ty)
        c0 = TILE_Z * (t // ty) * Z + y0
        for i in range(16):
            c = c0 + (i // TILE_Y) * Z + i % TILE_Y
            if y0 + i % TILE_Y < Z and c < nchunks:
                yield c


@pytest.mark.parametrize("dims", [(3, 3, 3), (16, 16, 16), (33, 17, 18), (10, 10, 999), (121, 112, 110), (97, 88, 90),
                                  (64, 64, 64), (256, 100, 30)])
def test_every_chunk_once(dims):
    nx, ny, nz = dims
    assert sorted(tile_order(*dims)) == list(range((nx * ny * nz + CHUNK - 1) // CHUNK))
