"""The FP32 advection with two columns per thread (jx even) at the edges of its
tiles and loops.  Vertical (one field per thread): columns of the smallest
height, of fewer levels than its turned loop, of one, two and three levels
left over; rows of one pair, of less and more than a block, of a block and one
pair; rows left over of a block.  Horizontal (strips of 16 rows or more): rows
of less than a strip, of one, of one and one pair, of two; strips of one row.

Reference: the one-column kernels (two fields per thread; shared-memory
tiles), which round every operation the same: the fields are the same bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "pai", "tetav", "qv", "t")


def _advected(dm, jx, iy, kz, rows, fields_per_thread, rotllr):
    g = dm.Moloch(jx, iy, kz, mode="fp32_mixed", rotllr=rotllr)
    g.setup_idealized(hills=((1500.0, jx / 2, iy / 2, 2.0),), u0=25.0, v0=-15.0, pert_amp=5.0, pert_levels=kz)
    g.set_tuning([1, 0, 2, 8, 0])
    for n in range(1, 9):
        g.moloch(n)
    g.set_tuning([rows, 0, fields_per_thread, 8, 0])
    for phase in (0, 1, 2):
        g.phase(phase)
    out = {f: g.get(f) for f in FIELDS}
    g.close()
    return out


@pytest.mark.parametrize("jx,iy,kz", [(4, 4, 4), (62, 5, 5), (64, 7, 8), (66, 6, 11), (130, 9, 12), (46, 10, 13),
                                      (65, 6, 9)])
def test_column_pairs_have_the_bits_of_single_columns(gpu_lib, jx, iy, kz):
    one, pair = (_advected(gpu_lib, jx, iy, kz, 1, f, 1) for f in (2, 1))
    for f in FIELDS:
        assert np.array_equal(one[f], pair[f], equal_nan=True), f


@pytest.mark.parametrize("rotllr", [1, 0])
@pytest.mark.parametrize("jx,iy,kz,rows", [(4, 4, 4, 16), (58, 16, 5, 16), (60, 17, 6, 16), (62, 33, 7, 32),
                                           (120, 31, 4, 16), (122, 40, 6, 64), (61, 20, 5, 16)])
def test_strip_pairs_have_the_bits_of_tiles(gpu_lib, jx, iy, kz, rows, rotllr):
    tiles, strips = (_advected(gpu_lib, jx, iy, kz, r, 2, rotllr) for r in (1, rows))
    for f in FIELDS:
        assert np.array_equal(tiles[f], strips[f], equal_nan=True), f
