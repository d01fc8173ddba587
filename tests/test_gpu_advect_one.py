"""The one-field advection at the edges of its kernels: the smallest domain,
columns of one warp, of several with a remainder and deeper than a block
holds, rows of less than a block, of a block and of several segments, rows of
a march left over.

Reference: the oracle's wafone on periodic map factors, both map-factor
branches, two calls in a row.  Tolerance: relative L2 <= 1e-13, as where the
same call is compared at its usual sizes (the same FP64 expressions without
contraction on both sides; the quotients round as IEEE)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotllr", [1, 0])
@pytest.mark.parametrize("jx,iy,kz", [(8, 8, 4), (33, 10, 7), (255, 9, 13), (256, 8, 12), (300, 7, 12), (16, 11, 73)])
def test_advect_one_at_the_edges(oracle_mod, gpu_lib, jx, iy, kz, rotllr):
    torch = pytest.importorskip("torch")
    from tests.test_gpu_parity_production import periodic_map_factors
    L = gpu_lib.lib()
    o = oracle_mod.Oracle(oracle_mod.make_cfg(jx, iy, kz, hills=((300.0, jx / 2, iy / 2, 3.0),), u0=5.0, v0=-3.0,
                                              rotllr=bool(rotllr)))
    msfu, msfv, msfx = periodic_map_factors(jx, iy, 5)
    o.set_map_factors(msfu[None], msfv[None], msfx[None])
    o.phase(0)
    o.phase(1)
    o.stagger(1)  # u and v rings become periodic images
    scal = (ctypes.c_double * 9)()
    oracle_mod.lib().oracle_scalars(o.h, scal)
    dta, dx, dzita = scal[0] / scal[6], scal[1], scal[2]
    dev = torch.device("cuda", 0)
    ro = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
          for a in (o.get("s"), o.get("u"), o.get("v"), o.get("fmz"), o.get("fmzf"),
                    msfu[:, 1:-1], msfv[1:-1, :], msfx)]
    pp = torch.from_numpy(np.ascontiguousarray(o.get("tetav"), dtype=np.float64)).to(dev)
    for _ in range(2):
        assert L.moloch_gpu_wafone_noalloc(*[ctypes.c_void_p(t.data_ptr()) for t in [pp] + ro], jx, iy, kz,
                                           dta, dx, dzita, rotllr, None) == 0, L.moloch_gpu_last_error()
        torch.cuda.synchronize()
        o.wafone("tetav")
        want, got = o.get("tetav"), pp.cpu().numpy()
        assert np.linalg.norm((got - want).ravel()) <= 1e-13 * np.linalg.norm(want.ravel())
    o.close()
