"""Tuning slots a caller leaves out, and what giving them does to rounding.

  * set_tuning on a handle nothing was chosen for starts from one level, field
    and tile level a thread, [1, 0, 1, 32, 0]: the slots not given stay there,
    whatever the size (in FP64 other variants of the sound kernels round
    differently, so the result shows it).
  * The Coriolis term of the FP32 momentum quads and strips: a handle on the
    shapes it starts with rounds it as the one-point kernel (the results of an
    untuned handle do not depend on its size); a handle given any tuning fuses
    it.  Giving a handle the shapes it already runs therefore moves u and v,
    by the one rounding of a product and what the two subtractions after it
    make of that: 2^-24 of the product and three roundings of 2^-24 of u on
    either side, at most 8 x 2^-24 of the largest wind.
"""
import numpy as np
import pytest

from tests.test_gpu_default_shapes import BASE, FIELDS, domain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,jx,iy,kz", [("fp64", 151, 140, 12), ("fp32_mixed", 100, 60, 40)])
@pytest.mark.parametrize("given", [0, 1, 2, 3, 4])
def test_slots_left_out_keep_the_base_shapes(gpu_lib, mode, jx, iy, kz, given):
    choice = [16, 8, 1, 8][:given]
    a, b = domain(gpu_lib, jx, iy, kz, mode), domain(gpu_lib, jx, iy, kz, mode)
    a.set_tuning(choice)
    b.set_tuning(choice + BASE[given:])
    for g in (a, b):
        g.run(2)
    assert set(a.profile_step()) == set(b.profile_step())  # the same kernels
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


def test_a_tuning_fuses_the_coriolis_term(gpu_lib):
    jx, iy, kz = 100, 60, 40
    a, b, c = (domain(gpu_lib, jx, iy, kz, "fp32_mixed", mo_nsound=1) for _ in range(3))
    b.set_tuning([16, 16 | 512 | 32 | 128 | 8 | 64, 1, 8, 1])  # the shapes a runs
    c.set_tuning([16, 16 | 512 | 32 | 128 | 8 | 64])
    for g in (a, b, c):
        g.phase(0)
        g.phase(1)
    assert set(a.profile_step()) == set(b.profile_step())
    for g in (a, b, c):
        g.setup_idealized(hills=((300.0, jx / 2.0, iy / 2.0, 4.0),), u0=6.0, v0=-3.0, pert_levels=kz)
        g.phase(0)
        g.phase(1)
    wind = max(np.max(np.abs(a.get("u"))), np.max(np.abs(a.get("v"))))
    for f in ("w", "pai", "tetav", "s", "deltaw"):  # formed before the momentum
        assert np.array_equal(a.get(f), b.get(f)), f
    for f in ("u", "v"):
        assert np.max(np.abs(a.get(f) - b.get(f))) <= 8 * 2.0 ** -24 * wind, f
        assert np.array_equal(b.get(f), c.get(f)), f
    for g in (a, b, c):
        g.close()


@pytest.mark.parametrize("jx,iy,kz", [(24, 20, 12), (61, 70, 23), (151, 140, 12)])
@pytest.mark.parametrize("tuning,same", [([4], True), ([32], True), ([1, 0, 2], True), ([1, 0, 5], True), ([1, 0, 10], True),
                                         ([1, 2], True), ([1, 8], True), ([1, 1], False), ([1, 4], False)])
def test_fp64_variants_that_move_no_bit(gpu_lib, jx, iy, kz, tuning, same):
    """All but the k-marching divergence and momentum; those by rounding, 1e-11
    as where the shapes a handle starts with are compared."""
    a, b = domain(gpu_lib, jx, iy, kz, "fp64"), domain(gpu_lib, jx, iy, kz, "fp64")
    a.set_tuning(tuning)
    b.set_tuning(BASE)
    for g in (a, b):
        g.run(3)
    for f in FIELDS:
        x, y = a.get(f), b.get(f)
        assert np.array_equal(x, y) if same else np.linalg.norm(x - y) <= 1e-11 * np.linalg.norm(y), f
    a.close()
    b.close()
