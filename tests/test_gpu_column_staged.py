"""The staged column solve (tuning bit 32) against the one-thread solve, bit for
bit, in every width of its tiles: 32, 64, 128 and 256 columns side by side,
full and ragged, a second tile along the row, fewer and more tiles than CTAs
fit on the GPU, the fewest levels, levels that do not fill the last chunk and
the most that fit.  Both solves evaluate the same expressions a level with
every contraction fixed, so no bit may differ.

The state is saturated and rising in places, so that the latent-heat term is
taken and left, with cloud and rain for the moist factors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "pai", "tetav", "s", "deltaw")
STAGED, ONE = 24 | 32 | 128, 24


def tile_width(jx, iy):
    """warps of 32 columns side by side: the fewest tiles of eight warps, the widest of equals"""
    tiles = {w: -(-jx // (32 * w)) * -(-iy * w // 8) for w in (8, 4, 2, 1)}
    return min(tiles, key=lambda w: (tiles[w], -w))


def moist_state(dm, jx, iy, kz, stream=None):
    g = dm.Moloch(jx, iy, kz, mode="fp32_mixed", stream=stream)
    g.setup_idealized(hills=((500.0, jx / 2.0, iy / 2.0, 5.0),), u0=6.0, v0=-4.0, pert_levels=kz)
    g.phase(0)
    r = np.random.default_rng(jx + 7 * iy + 11 * kz)
    sat = g.get("qsat").transpose(2, 1, 0)
    qx = np.zeros_like(g.download("qx"))
    qx[1:-1, 1:-1, :, 0] = sat * r.uniform(0.8, 1.1, sat.shape)
    for n in range(1, 5):
        qx[1:-1, 1:-1, :, n] = 1e-3 * r.uniform(-1, 1, sat.shape).clip(0)
    g.upload("qx", qx)
    g.upload("w", r.uniform(-0.4, 0.6, g.download("w").shape))
    return g


@pytest.mark.parametrize("jx,iy,kz,wide", [
    (28, 29, 64, 1), (96, 40, 33, 1), (4, 4, 4, 2), (60, 37, 30, 2), (64, 41, 64, 2), (124, 37, 41, 4), (128, 34, 13, 4),
    (252, 40, 30, 8), (480, 33, 41, 8), (228, 320, 16, 8), (512, 160, 64, 8)])
def test_staged_solve_has_the_bits_of_the_one_thread_solve(gpu_lib, jx, iy, kz, wide):
    assert tile_width(jx, iy) == wide
    a, b = moist_state(gpu_lib, jx, iy, kz), moist_state(gpu_lib, jx, iy, kz)
    a.set_tuning([16, ONE])
    b.set_tuning([16, STAGED])
    for g in (a, b):
        g.phase(0)
        g.phase(1)  # five substeps, the last completing s
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f
    for g in (a, b):
        g.run(2)
        g.sync()
    for f in FIELDS + ("t", "qv"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


def test_batched_staged_solve_has_the_bits_of_the_one_thread_solve(gpu_lib):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    shapes = [(252, 40, 30), (28, 29, 64), (37, 20, 12), (124, 37, 41), (64, 41, 64), (480, 33, 16)]
    ms = [moist_state(gpu_lib, *q, stream=stream.cuda_stream) for q in shapes]
    solo = [moist_state(gpu_lib, *q) for q in shapes]
    e = gpu_lib.Ensemble(ms)
    e.set_tuning([16, 24 | 32, 1, 32, 0])
    e.run(3)
    e.sync()
    for m, s in zip(ms, solo):
        s.set_tuning([16, ONE, 1, 32, 0])
        s.run(3)
        for f in FIELDS:
            assert np.array_equal(m.get(f), s.get(f)), f
    e.close()
    for m in ms + solo:
        m.close()
