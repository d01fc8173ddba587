"""The FP64 operations the kernels write out themselves, against CUDA's.

Quotients and reciprocals -- the diagnostics' and the moist factors' (the
contracting build), the column pivots' reciprocal, the shared-reciprocal
quotient of the exact build's WAF values and of the one-field advection --
round as IEEE: the same bits (any NaN for a NaN) on seeded values, on
denominators with mantissas on both sides of the cut below 2 where the short
form ends, numerators beside multiples of them, the ends of the exponent
ranges, zeros of both signs, subnormals, infinities and NaN.

pai^(cp/R): cp/R is 3.5, so the exact value is the square root of an integer
power, formed here in integers.  pai^3 and the root are carried in two words,
whose neglected terms lie below 2^-80, so what is left is the last rounding:
0.5 ulp, and no more than pow's largest error on the same values.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUOT, INV, PIVOT, POW = range(4)
POW35_ULP = 0.5 + 2.0 ** -20


def check(dm, op, a, b):
    """(the kernels' values, CUDA's); op None: the diagnostics' quotient"""
    torch = pytest.importorskip("torch")
    L = dm.lib()
    ta, tb = (torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).to("cuda") for x in (a, b))
    out, ref = torch.empty_like(ta), torch.empty_like(ta)
    P = [ctypes.c_void_p(t.data_ptr()) for t in (ta, tb, out, ref)]
    rc = (L.moloch_gpu_check_division_f64(*P, ta.numel(), None) if op is None else
          L.moloch_gpu_check_math_f64(op, *P, ta.numel(), None))
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy(), ref.cpu().numpy()


def denominators():
    r = np.random.default_rng(31)
    mant = np.concatenate([
        np.arange(-40, 41) + 0xffe0000000000,           # both sides of the cut 2 (1 - 2^-12)
        0xfffffffffffff - np.arange(40),                # next to 2
        np.arange(40),                                  # next to 1
        0xffdffffffffff - r.integers(0, 1 << 40, 200),  # below the cut, where the margin is smallest
        r.integers(0, 1 << 52, 400)]).astype(np.uint64)
    expo = np.array([1, 1023 - 1000, 1023 - 101, 1023 - 100, 1023 - 99, 1022, 1023, 1024, 1023 + 99, 1023 + 100,
                     1023 + 101, 2046], dtype=np.uint64)
    b = ((expo[:, None] << np.uint64(52)) | mant[None, :]).ravel().view(np.float64)
    return np.concatenate([b, -b])


def numerators(b):
    r = np.random.default_rng(32)
    out = [np.ones_like(b), r.uniform(1.0, 2.0, b.size) * 2.0 ** r.integers(-60, 60, b.size)]
    q = r.integers(1 << 52, 1 << 53, b.size).astype(np.float64) * 2.0 ** -52
    with np.errstate(over="ignore", under="ignore"):
        near = b * q  # beside a multiple of b, so that the quotient lies beside a double
        out += [near, np.nextafter(near, 0.0), np.nextafter(near, np.inf * np.sign(near)), b, np.nextafter(b, 0.0),
                np.nextafter(b, np.inf * np.sign(b))]
        for e in (-801, -800, -799, 799, 800, 801):
            out.append(r.uniform(1.0, 2.0, b.size) * 2.0 ** e)
    return out


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308, 1e-310, 1.0, -1.0,
                    3.0, 1e300, -1e300, 1.7976931348623157e308, 1e-300, 1e-30, 1e30])


def same_bits(x, y):
    nan = np.isnan(x) & np.isnan(y)
    return nan | (x.view(np.int64) == y.view(np.int64))


def report(x, y, a, b):
    bad = np.flatnonzero(~same_bits(x, y))
    return f"{bad.size} of {x.size}; first: {a[bad[:3]]} / {b[bad[:3]]} -> {x[bad[:3]]}, IEEE {y[bad[:3]]}"


@pytest.mark.parametrize("op", [None, QUOT])
def test_quotients_round_as_ieee(gpu_lib, op):
    b = denominators()
    for a in numerators(b):
        x, y = check(gpu_lib, op, a, b)
        assert same_bits(x, y).all(), report(x, y, a, b)
    r = np.random.default_rng(33)
    n = 1 << 21
    a = r.standard_normal(n) * 10.0 ** r.uniform(-12, 6, n)
    for lo, hi in ((0.3, 1.3), (1.0, 1.2), (1e-30, 1e3)):  # pai, the moist factors, field differences
        b = r.uniform(0.5, 1.0, n) * (r.uniform(lo, hi, n) if lo > 1e-9 else 10.0 ** r.uniform(-30, 3, n))
        x, y = check(gpu_lib, op, a, b)
        assert same_bits(x, y).all(), report(x, y, a, b)


@pytest.mark.parametrize("op", [None, QUOT])
def test_quotients_of_zeros_infinities_and_nan(gpu_lib, op):
    a, b = (x.ravel() for x in np.meshgrid(SPECIAL, SPECIAL))
    x, y = check(gpu_lib, op, a, b)
    assert same_bits(x, y).all(), report(x, y, a, b)


@pytest.mark.parametrize("op", [INV, PIVOT])
def test_reciprocals_round_as_ieee(gpu_lib, op):
    r = np.random.default_rng(34)
    n = 1 << 21
    for b in (denominators(), SPECIAL, 1.0 + 10.0 ** r.uniform(-3, 3, n), 2.0 ** r.uniform(-99, 99, n)):
        x, y = check(gpu_lib, op, b, b)
        assert same_bits(x, y).all(), report(x, y, np.ones_like(b), b)


def ulps_of_pow35(a, y):
    """|y - a^3.5| in units of y's last place, from integers"""
    m, e = math.frexp(a)
    m, e = int(m * 2 ** 53), 7 * (e - 53)  # a^7 = m^7 2^e
    k = 400 + (e & 1)
    s, es = math.isqrt(m ** 7 << k), (e - k) // 2  # a^3.5 = s 2^es
    my, ey = math.frexp(y)
    my, ey = int(my * 2 ** 53), ey - 53
    d = (my << (ey - es)) - s
    return abs(d) / 2.0 ** (ey - es) if abs(d) < 2 ** 900 else abs(d) // 2 ** (ey - es)


@pytest.mark.parametrize("lo,hi", [(0.02, 1.3), (0.95, 1.02), (2.0 ** -99, 2.0 ** 99)])
def test_exner_power_error(gpu_lib, lo, hi):
    r = np.random.default_rng(35)
    n = 20000
    a = np.exp(r.uniform(math.log(lo), math.log(hi), n))
    x, y = check(gpu_lib, POW, a, a)
    ours = max(ulps_of_pow35(float(p), float(q)) for p, q in zip(a, x))
    cuda = max(ulps_of_pow35(float(p), float(q)) for p, q in zip(a, y))
    print(f"pai in [{lo:.3g}, {hi:.3g}]: {ours:.6f} ulp, pow {cuda:.6f} ulp")
    assert ours <= POW35_ULP
    assert ours <= cuda


def test_exner_power_outside_its_range(gpu_lib):
    a = np.concatenate([SPECIAL, 2.0 ** np.array([-101.0, 101.0, -290.0, 290.0])])
    x, y = check(gpu_lib, POW, a, a)
    pow_path = (a <= 0) | ~np.isfinite(a) | (np.abs(a) < 2.0 ** -100) | (np.abs(a) >= 2.0 ** 100)
    assert same_bits(x, y)[pow_path].all()


@pytest.mark.parametrize("plant", [np.inf, -np.inf])
def test_an_infinite_temperature_gives_the_quotient_ieee_gives(gpu_lib, plant):
    """tetav = tvirt / pai of the pre-diagnostics, exact and contracting build"""
    out = {}
    for mode in ("fp64_exact", "fp64"):
        g = gpu_lib.Moloch(9, 8, 5, mode=mode)
        g.setup_idealized(hills=((300.0, 4.0, 4.0, 3.0),))
        t = g.download("t")
        t[3, 4, 2] = plant
        g.upload("t", t)
        g.phase(0)
        out[mode] = g.get("tetav")
        g.close()
    assert np.isinf(out["fp64_exact"]).sum() == 1
    assert np.array_equal(np.isinf(out["fp64"]), np.isinf(out["fp64_exact"]))
    assert not np.isnan(out["fp64"]).any()
