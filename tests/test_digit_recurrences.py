"""The digit recurrences of aph_math.cuh -- quotients, square roots, products and multiples by constants
in integer arithmetic -- on the CPU (tests/host_math.py), against IEEE arithmetic: equality of every
bit, with the FP32 approximations they start from in the middle and at both ends of their documented
error, and the bounds on the reciprocal word that their comments derive."""
import ctypes

import numpy as np
import pytest

import host_math
from quotient_cases import midpoint_cases

pytestmark = pytest.mark.skipif(host_math.compiler() is None, reason="no C++ compiler")

BODY = r"""
static uint64_t bits(double x) { return bits_as<uint64_t>(x); }
extern "C" void quotients(const double *a, const double *b, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = quot_bits(bits(a[i]), bits(b[i]), rcp_word(aph::significand(bits(b[i]))));
}
extern "C" void roots(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = sqrt_bits(bits(a[i]));
}
extern "C" void products(const double *a, const double *b, double *out, long long n) {
  IntOps o;
  for (long long i = 0; i < n; ++i) out[i] = o.mul(a[i], b[i]);
}
extern "C" void sixths(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = div6_x(a[i]);
}
extern "C" void triples(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = mulk_x<3, 0>(a[i]);
}
extern "C" void six_times(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = mulk_x<3, 1>(a[i]);
}
extern "C" void five_quarters(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = mulk_x<5, -2>(a[i]);
}
// words outside 2^84 / b - d, 1 <= d < 5
extern "C" long long bad_words(const double *b, long long n) {
  long long bad = 0;
  for (long long i = 0; i < n; ++i) {
    const unsigned __int128 B = aph::significand(bits(b[i])), Y = (unsigned __int128)1 << 84, R = rcp_word((uint64_t)B);
    bad += !((R + 1) * B <= Y && Y < (R + 5) * B);
  }
  return bad;
}
// the same calls for any operands: the digits, or the IEEE instruction
extern "C" void any_quotients(const double *a, const double *b, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = div_x(a[i], b[i]);
}
extern "C" void any_roots(const double *a, const double *, double *out, long long n) {
  for (long long i = 0; i < n; ++i) out[i] = sqrt_x(a[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return ctypes.CDLL(host_math.build(tmp_path_factory.mktemp("digits"), 1, BODY))


@pytest.fixture(params=[-1.0, 0.0, 1.0], ids=["low", "middle", "high"])
def approx(request, lib):
    lib.set_approx(ctypes.c_double(request.param))
    yield request.param
    lib.set_approx(ctypes.c_double(0.0))


def _values(rng, n, lo, hi, signed=True):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    sig = np.array([0, 1, 2, 3, (1 << 52) - 1, (1 << 52) - 2, 1 << 51, (1 << 51) - 1, (1 << 51) + 1, (1 << 29) - 1, 1 << 29,
                    (1 << 28) - 1, 1 << 28, (1 << 21) - 1, 1 << 21], np.uint64)
    edge = rng.integers(0, 3, n) == 0
    m[edge] = sig[rng.integers(0, sig.size, int(edge.sum()))]
    e = rng.integers(lo + 1023, hi + 1024, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64) if signed else np.zeros(n, np.uint64)
    return (m | (e << np.uint64(52)) | (s << np.uint64(63))).view(np.float64)


def _p(a):
    return np.ascontiguousarray(a).ctypes.data_as(ctypes.c_void_p)


def _check(lib, name, a, b, want):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    out = np.empty_like(a)
    getattr(lib, name)(_p(a), _p(b), _p(out), ctypes.c_longlong(a.size))
    bad = (out.view(np.uint64) != want.view(np.uint64)) & ~(np.isnan(out) & np.isnan(want))
    assert not bad.any(), (name, int(bad.sum()), a[bad][0].hex(), b[bad][0].hex())


N = 1_000_000


def test_quotients(lib, approx):
    rng = np.random.default_rng(31)
    a, b = _values(rng, N, -400, 400), _values(rng, N, -400, 400)
    q = _values(rng, N, 0, 0)
    near = (b * q).view(np.int64) + rng.integers(-4, 5, N)  # quotients next to representable numbers
    ma, mb = midpoint_cases(rng, 50_000)                    # and next to the middles between two
    a, b = np.concatenate([a, near.view(np.float64), ma]), np.concatenate([b, b, mb])
    assert lib.bad_words(_p(b), ctypes.c_longlong(b.size)) == 0
    _check(lib, "quotients", a, b, a / b)


def test_roots(lib, approx):
    rng = np.random.default_rng(32)
    x = _values(rng, N, -400, 400, signed=False)
    r = _values(rng, N, -200, 200, signed=False)
    near = (r * r).view(np.int64) + rng.integers(-4, 5, N)
    half = (r + 0.5 * np.spacing(r)) * (r + 0.5 * np.spacing(r))
    x = np.concatenate([x, near.view(np.float64), half])
    _check(lib, "roots", x, x, np.sqrt(x))


def test_products_and_multiples(lib):
    rng = np.random.default_rng(33)
    zero = np.array([0.0, -0.0, 1.0, -3.0, 2.0 ** 300, 2.0 ** -300])
    a = np.concatenate([_values(rng, N, -400, 400), np.repeat(zero, zero.size)])
    b = np.concatenate([_values(rng, N, -400, 400), np.tile(zero, zero.size)])
    a[:200_000] = 1.0 + rng.integers(0, 1 << 26, 200_000) * 2.0 ** -26  # products half-way between numbers
    b[:200_000] = 1.0 + (2 * rng.integers(0, 1 << 26, 200_000) + 1) * 2.0 ** -27
    _check(lib, "products", a, b, a * b)
    for name, want in (("sixths", a / 6.0), ("triples", 3.0 * a), ("six_times", 6.0 * a), ("five_quarters", 1.25 * a)):
        _check(lib, name, a, b, want)


def test_any_operands(lib, approx):
    """Zeros, infinities, NaN and exponents over the whole range go to the IEEE instruction."""
    rng = np.random.default_rng(34)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.2e-308, 1.7e308, 1.0, 3.0])
    a = np.concatenate([_values(rng, N // 2, -1022, 1023), np.repeat(special, special.size)])
    b = np.concatenate([_values(rng, N // 2, -1022, 1023), np.tile(special, special.size)])
    with np.errstate(all="ignore"):
        _check(lib, "any_quotients", a, b, a / b)
        _check(lib, "any_roots", a, b, np.sqrt(a))
