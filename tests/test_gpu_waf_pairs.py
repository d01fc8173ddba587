"""The FP32 vertical advection with two columns per thread (jx even, one field
per thread) at the edges of its tiles and loops: columns of the smallest
height, of fewer levels than its turned loop, of one, two and three levels
left over; rows of one pair, of less and more than a block, of a block and one
pair; rows left over of a block.

Reference: the one-column kernel (two fields per thread), which rounds every
operation the same: the fields are the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "pai", "tetav", "qv", "t")


@pytest.mark.parametrize("jx,iy,kz", [(4, 4, 4), (62, 5, 5), (64, 7, 8), (66, 6, 11), (130, 9, 12), (46, 10, 13),
                                      (65, 6, 9)])
def test_column_pairs_have_the_bits_of_single_columns(gpu_lib, jx, iy, kz):
    def advected(fields_per_thread):
        g = gpu_lib.Moloch(jx, iy, kz, mode="fp32_mixed")
        g.setup_idealized(hills=((1500.0, jx / 2, iy / 2, 2.0),), u0=25.0, v0=-15.0, pert_amp=5.0, pert_levels=kz)
        g.set_tuning([1, 0, 2, 8, 0])
        for n in range(1, 9):
            g.moloch(n)
        g.set_tuning([1, 0, fields_per_thread, 8, 0])
        for phase in (0, 1, 2):
            g.phase(phase)
        out = {f: g.get(f) for f in FIELDS}
        g.close()
        return out

    one, pair = advected(2), advected(1)
    for f in FIELDS:
        assert np.array_equal(one[f], pair[f], equal_nan=True), f
