"""A bounded wait of the staged column solve that gave up is reported by every
call that hands state to the host, not by sync and lprint steps alone: an
untuned FP32 handle starts with that solve, and a program that steps and
downloads (or takes the output path) calls neither.

The wait is made to run out as in the staged solve's own tests: a hook leaves
one staged chunk unissued, the wait on it gives up after 2e6 SM cycles (about
a millisecond) and the kernel returns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JX, IY, KZ = 64, 48, 20
HILLS = ((400.0, 32.0, 24.0, 4.0),)
TIMEOUT = 6


def failed_step(dm):
    g = dm.Moloch(JX, IY, KZ, mode="fp32_mixed")
    g.setup_idealized(hills=HILLS, u0=4.0)
    g.set_wait_limit(2_000_000, 3)
    g.moloch(1)
    return g


def recovered(dm, g):
    """a fresh state at the default limit: the handle's steps are right again"""
    g.set_wait_limit(0, -1)
    g.setup_idealized(hills=HILLS, u0=4.0)
    ref = dm.Moloch(JX, IY, KZ, mode="fp32_mixed")
    ref.setup_idealized(hills=HILLS, u0=4.0)
    for x in (g, ref):
        x.run(2)
    g.output_start()
    t, _ = g.output_finish()
    assert np.array_equal(t, ref.download("t"))
    for n in ("u", "w", "pai"):
        assert np.array_equal(g.get(n), ref.get(n)), n
    g.sync()
    ref.close()
    g.close()


@pytest.mark.parametrize("field", ["t", "ps", "qx"])
def test_download_reports_it_once(gpu_lib, field):
    g = failed_step(gpu_lib)
    with pytest.raises(gpu_lib.MolochError) as e:
        g.download(field)
    assert e.value.code == TIMEOUT
    g.download(field)  # reported and cleared
    recovered(gpu_lib, g)


@pytest.mark.parametrize("registered", [False, True])
def test_output_reports_it_once(gpu_lib, registered):
    g = failed_step(gpu_lib)
    t, ps = (np.zeros([u - l + 1 for l, u in gpu_lib.field_bounds(n, JX, IY, KZ)], order="F") for n in ("t", "ps"))
    if registered:
        g.host_register(t)
        g.host_register(ps)
    g.output_start()
    with pytest.raises(gpu_lib.MolochError) as e:
        g.output_finish(t, ps)
    assert e.value.code == TIMEOUT
    g.output_start()  # reported and cleared
    g.output_finish(t, ps)
    recovered(gpu_lib, g)


def test_a_snapshot_taken_before_it_is_good(gpu_lib):
    g = gpu_lib.Moloch(JX, IY, KZ, mode="fp32_mixed")
    g.setup_idealized(hills=HILLS, u0=4.0)
    g.moloch(1)
    want = g.download("t")
    g.output_start()
    g.set_wait_limit(2_000_000, 3)
    g.moloch(2)
    t, _ = g.output_finish()
    assert np.array_equal(t, want)
    with pytest.raises(gpu_lib.MolochError) as e:
        g.download("u")
    assert e.value.code == TIMEOUT
    recovered(gpu_lib, g)
