"""Which faces the integer-pipe solvers may keep, on the CPU (tests/host_math.py): a face they accept
has the bits of the same solver with IEEE operations, NaN for NaN, whatever the signs and zeros of its
state; faces of ordinary states are accepted.  Equality of every bit, so no tolerance."""
import ctypes

import numpy as np
import pytest

import host_math

pytestmark = pytest.mark.skipif(host_math.compiler() is None, reason="no C++ compiler")

COUNT = r"""
static bool same_bits(const double *a, const double *b, int n) {
  for (int k = 0; k < n; ++k)
    if (std::memcmp(a + k, b + k, 8) != 0 && !(a[k] != a[k] && b[k] != b[k])) return false;
  return true;
}
// s: n rows of wl, wr (rho, three velocities, p) and gamma_c, gamma_e left, then right, then whatever
// the solver takes beside; res: faces accepted, accepted and different, the first of those
template <int W, int N, class F>
static void count(const double *s, long long n, long long *res, F f) {
  res[0] = res[1] = 0;
  res[2] = -1;
  for (long long i = 0; i < n; ++i) {
    double got[N] = {0}, want[N] = {0};
    if (!f(s + W * i, got, want)) continue;
    ++res[0];
    if (same_bits(got, want, N)) continue;
    ++res[1];
    if (res[2] < 0) res[2] = i;
  }
}
"""

EXACT = COUNT + r"""
template <int RS>
static void run(const double *s, long long n, long long *res) {
  const GasConsts none{};
  count<14, 5>(s, n, res, [&](const double *w, double *got, double *want) {
    const double *g = w + 10;
    IntOps o;
    riemann<RS, false>(w, w + 5, g[0], g[1], g[2], g[3], none, got, o);
    IeeeOps i;
    riemann<RS, false>(w, w + 5, g[0], g[1], g[2], g[3], none, want, i);
    return o.ok();
  });
}
extern "C" void faces(int rs, const double *s, long long n, long long *res) {
  if (rs == RS_HLLE) run<RS_HLLE>(s, n, res);
  else if (rs == RS_HLLC) run<RS_HLLC>(s, n, res);
  else run<RS_LHLLC>(s, n, res);
}
// PPM states of positive windows of eight cells, as a tame window forms them: the faces between cells 3 and 4
extern "C" void ppm_faces(const double *q, long long n, double *ql, double *qr) {
  for (long long i = 0; i < n; ++i) {
    const double *w = q + 8 * i;
    double dd[8], d2[8], f[8], l[8], r[8];
    for (int c = 1; c < 7; ++c) dd[c] = ppm_dd<true>(w[c - 1], w[c], w[c + 1]), d2[c] = ppm_d2<true>(w[c - 1], w[c], w[c + 1]);
    for (int c = 2; c < 7; ++c) f[c] = ppm_face<true>(w[c - 1], w[c], dd[c - 1], dd[c], d2[c - 1], d2[c]);
    for (int c = 3; c < 5; ++c)
      ppm_cell<true>(w[c - 2], w[c - 1], w[c], w[c + 1], w[c + 2], d2[c - 1], d2[c], d2[c + 1], f[c], f[c + 1], l[c], r[c]);
    ql[i] = l[3];
    qr[i] = r[4];
  }
}
"""

HLLE, HLLC, LHLLC = 2, 3, 4


@pytest.fixture(scope="module")
def exact(tmp_path_factory):
    return ctypes.CDLL(host_math.build(tmp_path_factory.mktemp("exact"), 1, EXACT))


def _ptr(a):
    assert a.dtype == np.float64 and a.flags.c_contiguous
    return a.ctypes.data_as(ctypes.c_void_p)


def _count(fn, which, s):
    res = (ctypes.c_longlong * 3)()
    fn(which, _ptr(s), ctypes.c_longlong(len(s)), res)
    return res[0], res[1], ([x.hex() for x in s[res[2]]] if res[1] else None)


def _states(rng, n, spread):
    """n pairs of face states with densities and pressures log-uniform over 2^+-spread."""
    s = np.empty((n, 14))
    for side in (0, 5):
        s[:, side] = 2.0 ** rng.uniform(-spread, spread, n)
        s[:, side + 1:side + 4] = rng.normal(0.0, 2.0, (n, 3))
        s[:, side + 4] = 2.0 ** rng.uniform(-spread, spread, n)
    s[:, 10:14] = np.array([1.4, 1.4, 1.4, 1.4]) + rng.integers(-100, 101, (n, 4)) * 2.0 ** -52
    return s


@pytest.mark.parametrize("solver", [HLLE, HLLC, LHLLC])
def test_exact_faces_of_any_sign(exact, solver):
    rng = np.random.default_rng(400 + solver)
    n = 200_000
    s = _states(rng, n, 3)
    assert _count(exact.faces, solver, s)[:2] == (n, 0)  # ordinary states: all of them, the same bits
    # one or more of the densities, pressures and adiabatic indices negative, zero or (gamma_e) below 1
    col = np.array([0, 4, 5, 9, 10, 11, 12, 13])
    pick = rng.integers(0, 2, (n, col.size)) & rng.integers(0, 2, (n, col.size))
    pick[np.arange(n), rng.integers(0, col.size, n)] = 1
    x = s[:, col]
    how = rng.integers(0, 5, (n, col.size))
    x = np.where(pick == 1, np.choose(how, [-x, -x * 2.0 ** -4, 0.0 * x, -0.0 * x, x - 1.0]), x)
    s[:, col] = x
    rest = rng.integers(0, 4, n) == 0  # velocities at rest, where sums cancel to zeros
    s[rest, 1:4] = s[rest, 6:9] = 0.0
    got, wrong, first = _count(exact.faces, solver, s)
    assert wrong == 0, (got, wrong, first)


@pytest.mark.parametrize("solver", [HLLE, HLLC, LHLLC])
def test_exact_faces_of_positive_cells_with_troughs(exact, solver):
    """PPM overshoots below zero at a deep trough of positive cells."""
    rng = np.random.default_rng(410 + solver)
    n = 300_000
    ql, qr = np.empty(n), np.empty(n)
    s = _states(rng, n, 3)
    for v in (0, 4):
        q = np.ascontiguousarray(2.0 ** rng.uniform(-8, 0, (n, 8)))
        exact.ppm_faces(_ptr(q), ctypes.c_longlong(n), _ptr(ql), _ptr(qr))
        s[:, v], s[:, v + 5] = ql, qr
    assert (s[:, [0, 4, 5, 9]] < 0).any(axis=1).mean() > 0.05
    got, wrong, first = _count(exact.faces, solver, s)
    assert wrong == 0, (got, wrong, first)
    assert got >= (s[:, [0, 4, 5, 9]] > 0).all(axis=1).sum() * 0.999


FAST = COUNT + r"""
static GasConsts gas() {
  const double gm1 = 0.4, g = gm1 + 1.0;
  return GasConsts{gm1, 1.0 / gm1, g, C_LIGHT2 * g, 1.0 + 1.0 / gm1, (g + 1.0) / std::sqrt(2.0 * g), (g + 1.0) / (2.0 * g)};
}
template <int RS, bool CONSTG>
static void run(const double *s, long long n, long long *res) {
  const GasConsts gc = gas();
  count<14, 5>(s, n, res, [&](const double *w, double *got, double *want) {
    const double *g = w + 10;
    FaceOps o;
    riemann<RS, CONSTG>(w, w + 5, g[0], g[1], g[2], g[3], gc, got, o);
    IeeeOps i;
    riemann<RS, CONSTG>(w, w + 5, g[0], g[1], g[2], g[3], gc, want, i);
    return o.ok();
  });
}
extern "C" void faces(int rs, const double *s, long long n, long long *res) {
  if (rs == RS_HLLE) run<RS_HLLE, false>(s, n, res);
  else if (rs == RS_HLLC) run<RS_HLLC, false>(s, n, res);
  else run<RS_LHLLC, false>(s, n, res);
}
extern "C" void gas_faces(int rs, const double *s, long long n, long long *res) {
  if (rs == RS_HLLE) run<RS_HLLE, true>(s, n, res);
  else if (rs == RS_HLLC) run<RS_HLLC, true>(s, n, res);
  else run<RS_LHLLC, true>(s, n, res);
}
// the reverse of a face: states, then the adjoint of its fluxes
extern "C" void adjoints(int rs, const double *s, long long n, long long *res) {
  const GasConsts gc = gas();
  count<15, 10>(s, n, res, [&](const double *w, double *got, double *want) {
    FaceOps o;
    IeeeOps i;
    for (int k = 0; k < 10; ++k) o.see(w[k]);
    for (int k = 10; k < 15; ++k) o.see(w[k]);
    if (rs == RS_HLLE) hlle_vjp(w, w + 5, gc, 1.0 / gc.c2g, w + 10, got, got + 5, o), hlle_vjp(w, w + 5, gc, 1.0 / gc.c2g, w + 10, want, want + 5, i);
    else hllc_vjp(w, w + 5, gc, 1.0 / gc.c2g, w + 10, got, got + 5, o), hllc_vjp(w, w + 5, gc, 1.0 / gc.c2g, w + 10, want, want + 5, i);
    return o.ok();
  });
}
"""


@pytest.fixture(scope="module")
def fast(tmp_path_factory):
    return ctypes.CDLL(host_math.build(tmp_path_factory.mktemp("fast"), 0, FAST, ("aph_math.cuh", "aph_adjoint_math.cuh")))


def _any_sign(rng, s, col):
    """One or more of the columns negative, zero or lowered by 1 in each row."""
    n = len(s)
    pick = rng.integers(0, 2, (n, col.size)) & rng.integers(0, 2, (n, col.size))
    pick[np.arange(n), rng.integers(0, col.size, n)] = 1
    x = s[:, col]
    s[:, col] = np.where(pick == 1, np.choose(rng.integers(0, 5, x.shape), [-x, -x * 2.0 ** -4, 0.0 * x, -0.0 * x, x - 1.0]), x)
    rest = rng.integers(0, 4, n) == 0
    s[rest, 1:4] = s[rest, 6:9] = 0.0
    return s


@pytest.mark.parametrize("which", ["faces", "gas_faces"])
@pytest.mark.parametrize("solver", [HLLE, HLLC, LHLLC])
def test_fast_faces_of_any_sign(fast, solver, which):
    """Zero pressures above all: 0 x rsqrt(0) is NaN."""
    rng = np.random.default_rng(420 + solver)
    n = 200_000
    fn = getattr(fast, which)
    s = _states(rng, n, 3)
    assert _count(fn, solver, s)[:2] == (n, 0)
    col = np.array([0, 4, 5, 9, 10, 11, 12, 13] if which == "faces" else [0, 4, 5, 9])
    got, wrong, first = _count(fn, solver, _any_sign(rng, s, col))
    assert wrong == 0, (got, wrong, first)


@pytest.mark.parametrize("solver", [HLLE, HLLC])
def test_adjoint_faces_of_any_sign(fast, solver):
    rng = np.random.default_rng(430 + solver)
    n = 200_000
    s = np.concatenate([_states(rng, n, 3)[:, :10], rng.normal(0.0, 1.0, (n, 5))], axis=1)
    assert _count(fast.adjoints, solver, s)[:2] == (n, 0)
    got, wrong, first = _count(fast.adjoints, solver, _any_sign(rng, s, np.array([0, 4, 5, 9])))
    assert wrong == 0, (got, wrong, first)
