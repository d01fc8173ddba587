"""The one-field advection on the smallest domains the call accepts, four and
five rows and columns and four levels, where the periodic wraps of rows and
columns meet; reference and tolerance as in test_gpu_advect_one."""
import pytest

from tests import test_gpu_advect_one as edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotllr", [1, 0])
@pytest.mark.parametrize("jx,iy,kz", [(4, 4, 4), (5, 4, 4), (4, 5, 4), (5, 5, 5)])
def test_advect_one_on_the_smallest_domains(oracle_mod, gpu_lib, jx, iy, kz, rotllr):
    edges.test_advect_one_at_the_edges(oracle_mod, gpu_lib, jx, iy, kz, rotllr)
