"""FP64 kernels that take the points of a level in order (4096 points or more,
rows that leave a tenth of whole warps idle), on both sides of those lines,
with a last block that is not full, every optional kernel on, both map-factor
branches; horizontal advection in tiles and in strips of one warp a block.

Reference: the oracle, two steps.  Tolerance: 1e-12 for the exact build
(rounding of pow and exp, 1e-13 a phase), 1e-9 for the contracting one (its
bound on a run)."""
import pytest

from tests.test_gpu_parity import DIAG, PROG, compare, pair

pytestmark = pytest.mark.gpu

TOL = {"fp64_exact": 1e-12, "fp64": 1e-9}


@pytest.mark.parametrize("mode", ["fp64_exact", "fp64"])
@pytest.mark.parametrize("rotllr", [1, 0])
@pytest.mark.parametrize("jx,iy,kz", [(67, 62, 5), (65, 63, 5), (70, 60, 6), (91, 46, 7)])
def test_points_in_order(oracle_mod, gpu_lib, mode, rotllr, jx, iy, kz):
    on = dict(divfilter=1, filterpai=1, filtertheta=1) if rotllr else {}
    o, g = pair(oracle_mod, gpu_lib, jx, iy, kz, mode=mode, hills=((300.0, jx / 2, iy / 2, 4.0),), pert_levels=kz,
                rotllr=rotllr, **on)
    if mode == "fp64":
        g.set_tuning([16 if rotllr else 1, 7 if rotllr else 0, 2, 32, 0])
    for _ in range(2):
        for phase in (0, 1, 2, 1, 2, 1, 2, 3):
            o.phase(phase)
            g.phase(phase)
    compare(o, g, PROG + DIAG, TOL[mode])
    o.close()
    g.close()
