"""The quotients, square roots and float pairs that the sweeps take on the
integer pipes (csrc/int64math.cuh, csrc/pair32.cuh), evaluated on the GPU with the
hardware's own estimates: bit for bit IEEE's values (as numpy gives them), over
random significands and those of all ones, zeros and runs of either, ties,
signed zeros, subnormal and non-finite values and the ends of the exponent range;
and the fast precisions' reciprocal and root within the scheme's bounds:
half an ulp of rounding plus two units of the 62- and 60-bit estimates (1/256 and
1/128 ulp) and 2^-10 for the reference's own rounding."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")

pytestmark = pytest.mark.gpu
N = 1_000_000
SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 2.2250738585072014e-308, 1.79e308, 1.0, -1.0])


def significands(rng, n):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = rng.integers(0, 8, n)
    top, low = np.uint64((1 << 52) - 1), np.uint64((1 << 29) - 1)
    runs = (np.uint64(0xFFFFFFFFFFFFFFFF) << rng.integers(0, 52, n, dtype=np.uint64)) & top
    small = rng.integers(0, 64, n, dtype=np.uint64)
    return np.choose(k, [small * (rng.integers(0, 3, n, dtype=np.uint64)), top - small, m & ~low, m | low, runs, m, m, m])


def numbers(rng, n, lo, hi, signs=True):
    b = (rng.integers(lo, hi, n, dtype=np.uint64) << np.uint64(52)) | significands(rng, n)
    if signs:
        b |= rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    return b.view(np.float64)


def same_bits(a, b):
    return ((a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))).all()


def test_quotients_are_ieee():
    rng = np.random.default_rng(1)
    a, b = numbers(rng, N, 1000, 1040), numbers(rng, N, 1000, 1040)
    a[::2], b[::4] = numbers(rng, N // 2, 0, 2048), numbers(rng, N // 4, 0, 2048)
    a[3::16], b[5::16] = rng.choice(SPECIAL, len(a[3::16])), rng.choice(SPECIAL, len(b[5::16]))
    # dividends next to a divisor times a value half way between two doubles
    half = np.longdouble(1) + np.ldexp(np.longdouble(rng.integers(0, 1 << 52, len(b[7::16]))) + np.longdouble(0.5), -52)
    with np.errstate(all="ignore"):
        a[7::16] = (half * b[7::16].astype(np.longdouble)).astype(np.float64)
        want = a / b
    assert same_bits(ib.fast_math_eval("divide_rn_f64", np.concatenate([a, b])), want)


def test_roots_are_ieee():
    rng = np.random.default_rng(2)
    x = np.concatenate([numbers(rng, N, 1, 2047, signs=False), numbers(rng, 4096, 0, 1), SPECIAL])
    s = numbers(rng, N, 1000, 1040, signs=False)
    x = np.concatenate([x, s * s, np.nextafter(s * s, 0), np.nextafter(s * s, np.inf)])
    with np.errstate(all="ignore"):
        assert same_bits(ib.fast_math_eval("sqrt_rn_f64", x), np.sqrt(x))


def test_pairs_are_the_conversions():
    rng = np.random.default_rng(3)
    x = np.concatenate([numbers(rng, N, 0, 2048), numbers(rng, N, 940, 1160), SPECIAL])
    x[::5] = (x[::5].view(np.uint64) & ~np.uint64((1 << 28) - 1)).view(np.float64)  # ties
    with np.errstate(all="ignore"):
        hi = x.astype(np.float32)
        lo = (x - hi.astype(np.float64)).astype(np.float32)
        assert same_bits(ib.fast_math_eval("pair_hi", x), hi.astype(np.float64))
        assert same_bits(ib.fast_math_eval("pair_lo", x), lo.astype(np.float64))
        assert same_bits(ib.fast_math_eval("widen", x), hi.astype(np.float64))


def test_fast_reciprocal_and_root():
    rng = np.random.default_rng(4)
    x = numbers(rng, N, 2, 2043)
    err = np.abs(ib.fast_math_eval("rcp_f64", x).astype(np.longdouble) - 1 / x.astype(np.longdouble))
    assert (err / np.spacing(np.abs(1 / x))).max() <= 0.5 + 1 / 256 + 2 ** -10
    x = numbers(rng, N, 1, 2047, signs=False)
    err = np.abs(ib.fast_math_eval("sqrt_f64", x).astype(np.longdouble) - np.sqrt(x.astype(np.longdouble)))
    assert (err / np.spacing(np.sqrt(x))).max() <= 0.5 + 1 / 128 + 2 ** -10
