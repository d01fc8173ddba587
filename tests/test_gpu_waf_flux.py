"""The contracting builds' WAF advection (FP64: limiter in flux form) against
the exact build's (slope ratio), one advection phase from the same state:
fields with flat runs, steps of both signs, alternating extrema, differences
far below the ratio form's denominator guard and values that are not finite;
winds of both signs; kz = 4 (no interior level range), sizes with partial
tiles and strips, both launch shapes and every number of fields a thread.

Tolerance: both forms evaluate the same continuous, piecewise linear function
of the neighbours; each rounds under 40 operations a point in each of four
passes on values of the field's size, and a difference enters with slope 2 at
most: 500 eps of the field's largest value bounds the two together (in FP32
that holds the rounding of the uploaded field and winds too)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TRACERS = ("qv", "qc", "qi", "qr", "qs")


def fields(jx, iy, kz, seed):
    r = np.random.default_rng(seed)
    k, i, j = np.meshgrid(np.arange(kz), np.arange(iy), np.arange(jx), indexing="ij")
    smooth = 1.0 + 0.3 * np.sin(2 * np.pi * j / jx) * np.cos(2 * np.pi * i / iy) + 0.02 * k
    return {
        "u": 8.0 * r.uniform(-1, 1, k.shape), "v": 8.0 * r.uniform(-1, 1, k.shape),
        "qv": 1e-2 * smooth,
        "qc": np.where((i + j + k) % 7 < 3, 1e-3, 0.0),                 # steps between flat runs
        "qi": 1e-3 * ((i + j + k) % 2) * r.uniform(0, 1, k.shape),      # alternating extrema
        "qr": 1e-35 * r.integers(0, 3, k.shape),                        # differences below the guard
        "qs": 1e-4 * r.standard_normal(k.shape),
    }


def advected(dm, jx, iy, kz, mode, seed, tuning=None, plant=None):
    g = dm.Moloch(jx, iy, kz, mode=mode)
    g.setup_idealized(hills=((300.0, jx / 2.0, iy / 2.0, 3.0),), u0=2.0, v0=-1.0, pert_levels=kz)
    g.moloch(1)  # s and w of a developed state
    f = fields(jx, iy, kz, seed)
    if plant is not None:
        f["qv"][kz // 2, iy // 2, jx // 2] = plant
    full = {n: g.download(n) for n in ("u", "v", "qx")}
    for n in ("u", "v"):
        b = dm.field_bounds(n, jx, iy, kz)
        full[n][1 - b[0][0]:1 - b[0][0] + jx, 1 - b[1][0]:1 - b[1][0] + iy] = f[n].transpose(2, 1, 0)
    for q, n in enumerate(TRACERS):
        full["qx"][1:jx + 1, 1:iy + 1, :, q] = f[n].transpose(2, 1, 0)
    for n, a in full.items():
        g.upload(n, a)
    if tuning:
        g.set_tuning(tuning)
    g.phase(2)
    out = {n: g.get(n) for n in TRACERS + ("tetav",)}
    g.close()
    return out


@pytest.mark.parametrize("mode,eps", [("fp64", 2.2e-16), ("fp32_mixed", 1.2e-7)])
@pytest.mark.parametrize("jx,iy,kz", [(4, 4, 4), (29, 9, 5), (33, 65, 7), (64, 24, 12)])
@pytest.mark.parametrize("tuning", [[1, 0, 1], [2, 0, 2], [16, 0, 5], [32, 0, 10]])
def test_flux_form_matches_ratio_form(gpu_lib, mode, eps, jx, iy, kz, tuning):
    a = advected(gpu_lib, jx, iy, kz, "fp64_exact", 3)
    b = advected(gpu_lib, jx, iy, kz, mode, 3, tuning)
    for n in TRACERS:
        if n == "qr":  # below the guard the two forms may differ by the field's own size
            assert np.max(np.abs(b[n])) <= 8e-35
            continue
        top = np.max(np.abs(a[n]))
        assert np.max(np.abs(a[n] - b[n])) <= 500 * eps * top, (n, np.max(np.abs(a[n] - b[n])) / top)


@pytest.mark.parametrize("mode", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("plant", [np.nan, np.inf])
@pytest.mark.parametrize("tuning", [[1, 0, 1], [16, 0, 2]])
def test_values_that_are_not_finite_spread_alike(gpu_lib, mode, plant, tuning):
    """The cells of qv that one advection leaves not finite around a planted
    value are those of the ratio form, in every build and launch shape."""
    a = advected(gpu_lib, 33, 27, 9, "fp64_exact", 5, plant=plant)
    b = advected(gpu_lib, 33, 27, 9, mode, 5, tuning, plant=plant)
    assert np.array_equal(np.isfinite(a["qv"]), np.isfinite(b["qv"]))
    for n in ("qc", "qi", "tetav"):
        assert np.isfinite(b[n]).all(), n
