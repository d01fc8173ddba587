"""The launch shapes a handle or an ensemble starts with (chosen by size and
mode) against one level, field and tile level a thread, [1, 0, 1, 32, 0]: the
same bits in every mode that allows none to move (FP32 storage and the exact
build), 1e-11 in FP64, whose kernels contract differently.  Sizes on both
sides of each rule's line (jx a multiple of 4 or not, 2e5 and 2^20 points,
4000, 8000 and 20000 columns), both map-factor branches, and the filters."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_gpu_parity_production import periodic_map_factors

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "pai", "t", "qv", "ps", "tetav", "s", "deltaw")
BASE = [1, 0, 1, 32, 0]


def domain(dm, jx, iy, kz, mode, rotllr=1, stream=None, **opts):
    g = dm.Moloch(jx, iy, kz, mode=mode, rotllr=rotllr, stream=stream, **opts)
    g.setup_idealized(hills=((300.0, jx / 2.0, iy / 2.0, 4.0),), u0=6.0, v0=-3.0, pert_levels=kz)
    if not rotllr:
        for name, a in zip(("msfu", "msfv", "msfx"), periodic_map_factors(jx, iy, 9)):
            g.upload(name, a.T)
        g.init()
    return g


@pytest.mark.parametrize("mode", ["fp32_mixed", "fp64_exact", "fp64"])
@pytest.mark.parametrize("jx,iy,kz", [(40, 33, 16), (61, 70, 47), (68, 60, 52), (101, 90, 23), (150, 140, 50), (151, 140, 50)])
@pytest.mark.parametrize("rotllr", [1, 0])
def test_default_shapes_match_the_base_kernels(gpu_lib, mode, jx, iy, kz, rotllr):
    a, b = domain(gpu_lib, jx, iy, kz, mode, rotllr), domain(gpu_lib, jx, iy, kz, mode, rotllr)
    b.set_tuning(BASE)
    for g in (a, b):
        g.moloch(1)
        g.run(2)
    for f in FIELDS:
        x, y = a.get(f), b.get(f)
        assert (rel_l2(x, y) <= 1e-11) if mode == "fp64" else np.array_equal(x, y), (f, rel_l2(x, y))
    a.close()
    b.close()


@pytest.mark.parametrize("mode", ["fp32_mixed", "fp64"])
def test_default_shapes_with_the_filters(gpu_lib, mode):
    opts = dict(mo_divfilter=1, do_filterpai=1, do_filtertheta=1)
    a, b = (domain(gpu_lib, 68, 60, 52, mode, 0, **opts) for _ in range(2))
    b.set_tuning(BASE)
    a.run(3)
    b.run(3)
    for f in FIELDS:
        x, y = a.get(f), b.get(f)
        assert (rel_l2(x, y) <= 1e-11) if mode == "fp64" else np.array_equal(x, y), (f, rel_l2(x, y))
    a.close()
    b.close()


@pytest.mark.parametrize("mode", ["fp32_mixed", "fp64"])
def test_default_shapes_of_an_ensemble(gpu_lib, mode):
    """2^20 points and more; afterwards the persistent kernel, which carries
    only the base shapes, is accepted as before."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    shapes = [(96, 80, 60), (101, 70, 47), (128, 64, 40)]
    ms = [domain(gpu_lib, *q, mode, stream=stream.cuda_stream) for q in shapes]
    solo = [domain(gpu_lib, *q, mode) for q in shapes]
    e = gpu_lib.Ensemble(ms)
    e.run(2)
    e.set_persistent(True)
    assert e.persistent
    e.run(1)
    e.sync()
    e.set_persistent(False)
    e.run(1)
    e.sync()
    for m, s in zip(ms, solo):
        s.set_tuning(BASE)
        s.run(4)
        for f in FIELDS:
            x, y = m.get(f), s.get(f)
            assert (rel_l2(x, y) <= 1e-11) if mode == "fp64" else np.array_equal(x, y), (f, rel_l2(x, y))
    e.close()
    for m in ms + solo:
        m.close()
