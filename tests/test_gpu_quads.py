"""The FP32 kernels with four columns per thread (momentum: tuning bits 8 +
64; divergence and damping: 16 + 512; jx a multiple of 4) against the
one-column warp strips (8 + 16): the same expressions per column, so the same
bits.  Sizes cover one quad a row, rows ending inside a warp's 128 columns, at
them and just past them, rows not a multiple of the blocks (4 and 13), fewer
levels than CTAs' shares and more, tiles cut between CTAs, and the non-ROTLLR
branch with map factors other than 1."""
import numpy as np
import pytest

from tests.test_gpu_parity_production import periodic_map_factors

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "pai", "tetav", "s", "deltaw", "qv", "t")


def run(dm, jx, iy, kz, tuning, rotllr, graph):
    g = dm.Moloch(jx, iy, kz, mode="fp32_mixed", rotllr=rotllr)
    g.setup_idealized(hills=((400.0, jx / 2.0, iy / 2.0, 4.0),), u0=6.0, v0=-3.0, pert_amp=0.5, pert_levels=kz)
    if not rotllr:
        for name, a in zip(("msfu", "msfv", "msfx"), periodic_map_factors(jx, iy, 9)):
            g.upload(name, a.T)
        g.init()
    g.set_tuning(tuning)
    if graph:
        g.run(3)
    else:
        for s in (1, 2, 3):
            g.moloch(s)
    out = {f: g.get(f) for f in FIELDS}
    g.close()
    return out


@pytest.mark.parametrize("rotllr", [1, 0])
@pytest.mark.parametrize("jx,iy,kz", [(4, 4, 4), (4, 5, 7), (24, 20, 8), (64, 48, 13), (128, 8, 12), (132, 33, 10),
                                      (260, 17, 14), (96, 130, 66)])
def test_quads_match_strips(gpu_lib, jx, iy, kz, rotllr):
    a = run(gpu_lib, jx, iy, kz, [4, 8 | 16, 1, 8], rotllr, False)
    for sound in (8 | 16 | 64, 8 | 16 | 512, 8 | 16 | 64 | 512):
        b = run(gpu_lib, jx, iy, kz, [4, sound, 1, 8], rotllr, sound & 512)
        for f in FIELDS:
            assert np.array_equal(a[f], b[f]), (sound, f, float(np.max(np.abs(a[f] - b[f]))))
