"""The FP64 column solve split over a block, on both sides of each of its lines:
columns that do not fill the last block, 3000 and 16000 columns, 64, 128 and
256 levels, the smallest and fewer levels than thread groups; with the
divergence filter (the pressure update is then a kernel of its own) and the
last substep's vertical motion.

Reference: the oracle's sound phase.  Tolerance: 1e-13 for the exact build, as
where its phases are compared at other sizes, 1e-9 for the contracting one
(its bound on a run)."""
import pytest

from tests.test_gpu_parity import compare, pair

pytestmark = pytest.mark.gpu

TOL = {"fp64_exact": 1e-13, "fp64": 1e-9}


@pytest.mark.parametrize("mode", ["fp64_exact", "fp64"])
@pytest.mark.parametrize("jx,iy,kz", [(9, 7, 4), (10, 9, 33), (9, 8, 256), (9, 8, 257), (61, 50, 20), (61, 50, 64),
                                      (56, 55, 65), (56, 55, 129), (127, 126, 12)])
def test_split_columns_match_the_oracle(oracle_mod, gpu_lib, mode, jx, iy, kz):
    o, g = pair(oracle_mod, gpu_lib, jx, iy, kz, mode=mode, hills=((300.0, jx / 2, iy / 2, 3.0),), pert_levels=kz)
    for x in (o, g):
        x.phase(0)
        x.phase(1)
    compare(o, g, ("u", "v", "w", "pai", "tetav", "s", "deltaw"), TOL[mode])
    o.close()
    g.close()


@pytest.mark.parametrize("mode", ["fp64_exact", "fp64"])
def test_split_columns_with_the_divergence_filter(oracle_mod, gpu_lib, mode):
    o, g = pair(oracle_mod, gpu_lib, 21, 19, 13, mode=mode, hills=((300.0, 10.0, 9.0, 3.0),), rotllr=0, divfilter=1)
    for x in (o, g):
        x.phase(0)
        x.phase(1)
    compare(o, g, ("u", "v", "w", "pai", "tetav", "s", "deltaw"), TOL[mode])
    o.close()
    g.close()
