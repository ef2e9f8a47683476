// aph_diag.cu -- device evaluation of the exact-mode integer-pipe operations (aph_math.cuh),
// so that tests can compare them bit for bit with the IEEE operations they replace.
#include "../../include/aph_hydro.h"
#include "aph_capi_internal.h"
#define APH_EXACT 1
#include "aph_math.cuh"

using namespace aph;

namespace {

// Round-to-nearest-even sums in 64-bit integer arithmetic (the textbook alignment with a sticky bit,
// guard bits, renormalisation and rounding), for operands that are zero or normal with
// 2^-900 < |x| < 2^900 and results that stay so.  A probe only: 30 SM-cycles a warp, where the
// FP64 instruction takes 17.

// Pack a positive significand S (leading 1 at bit 62, sticky bits below bit 10) with biased
// exponent e and sign bit sg, rounding to nearest even.
__device__ __forceinline__ double round_pack_x(unsigned long long sg, long long e, unsigned long long S) {
  const unsigned long long r = S & 0x3ffULL;
  unsigned long long m = S >> 10;  // 53 bits, leading 1 at bit 52
  if (r > 0x200ULL || (r == 0x200ULL && (m & 1ULL))) ++m;
  if (m >> 53) {  // rounding carried into bit 53
    m >>= 1;
    ++e;
  }
  return __longlong_as_double((long long)(sg | ((unsigned long long)e << 52) | (m & 0xfffffffffffffULL)));
}

// RN(a + b)
__device__ __forceinline__ double add_x(double a, double b) {
  unsigned long long ua = (unsigned long long)__double_as_longlong(a);
  unsigned long long ub = (unsigned long long)__double_as_longlong(b);
  unsigned long long ma = ua & 0x7fffffffffffffffULL, mb = ub & 0x7fffffffffffffffULL;
  if (mb > ma) {  // |a| >= |b| from here on
    const unsigned long long t = ua;
    ua = ub;
    ub = t;
    const unsigned long long tm = ma;
    ma = mb;
    mb = tm;
  }
  const unsigned long long sg = ua & 0x8000000000000000ULL;
  if (mb == 0) {  // b is a zero: a, or the sum of two zeros (-0 only for -0 + -0)
    if (ma != 0) return __longlong_as_double((long long)ua);
    return __longlong_as_double((long long)(ua & ub));
  }
  const long long ea = (long long)(ma >> 52), eb = (long long)(mb >> 52);
  const long long d = ea - eb;
  if (d > 55) return __longlong_as_double((long long)ua);  // |b| below a quarter ulp of a
  // significands with 9 guard bits (leading 1 at bit 61); b's shifted out bits as a sticky bit
  const unsigned long long A = ((ma & 0xfffffffffffffULL) | 0x10000000000000ULL) << 9;
  const unsigned long long Bf = ((mb & 0xfffffffffffffULL) | 0x10000000000000ULL) << 9;
  const unsigned long long Bt = Bf >> d;
  const unsigned long long st = ((Bf << (63 - d)) << 1) != 0 ? 1ULL : 0ULL;  // only for d >= 10
  long long e = ea;
  unsigned long long S;
  if (((ua ^ ub) >> 63) == 0) {  // same signs: the sum's floor, sticky; leading 1 at bit 61 or 62
    S = (A + Bt) | st;
    if (S >> 62) {
      S = (S >> 1) | (S & 1ULL);
      ++e;
    }
    S <<= 1;  // leading 1 at bit 62
  } else {  // the difference's floor (sticky: b was truncated, subtract one more), then sticky
    S = A - Bt - st;
    if (S == 0) return 0.0;  // x - x = +0 (st is 0 then)
    const int sh = __clzll((long long)S) - 1;  // bring the leading 1 to bit 62 (sh <= 2 if st)
    S = (S << sh) | st;
    e -= sh - 1;
  }
  return round_pack_x(sg, e, S);
}
__device__ __forceinline__ double sub_x(double a, double b) {
  return add_x(a, __longlong_as_double(__double_as_longlong(b) ^ (long long)0x8000000000000000ULL));
}

__global__ void k_exact_ops(int op, const double *x, double *out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double v = x[i];
    double r;
    if (op == 0) r = div6_x(v);
    else if (op == 1) r = half_x(v);
    else if (op == 2) r = twice_x(v);
    else r = tame(v) ? 1.0 : 0.0;
    out[i] = r;
  }
}

__global__ void k_exact_ops2(int op, const double *x, const double *y, double *out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double a = x[i], b = y[i];
    double r;
    if (op == 0) r = add_x(a, b);
    else if (op == 1) r = sub_x(a, b);
    else if (op == 2) r = mulk_x<3, 0>(a);
    else if (op == 3) r = mulk_x<3, 1>(a);
    else if (op == 4) r = mulk_x<5, -2>(a);
    else if (op == 5) r = a / b;
    else if (op == 6) r = __drcp_rn(b);
    else if (op == 7) r = sqrt(a);
    else if (op == 8) r = div_x(a, b);
    else if (op == 9) r = rcp_x(b);
    else if (op == 10) r = sqrt_x(a);
    else {
      FaceOps o;
      r = o.mul(a, b);
      if (!o.ok()) r = __dmul_rn(a, b);
    }
    out[i] = r;
  }
}

}  // namespace

extern "C" aph_status aph_diag_exact_ops2(int op, const double *x, const double *y, double *out,
                                          long long n, void *stream) {
  clear_error();
  if (op < 0 || op > 11) return fail(APH_ERR_INVALID, "op %d not in 0..11", op);
  if (n < 0 || (n > 0 && (!x || !y || !out))) return fail(APH_ERR_INVALID, "NULL argument");
  if (n == 0) return APH_OK;
  const long long blocks = (n + 255) / 256;
  k_exact_ops2<<<(unsigned)(blocks < 152 * 16 ? blocks : 152 * 16), 256, 0, (cudaStream_t)stream>>>(
      op, x, y, out, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? APH_OK : cuda_fail(e, "diag_exact_ops2");
}

extern "C" aph_status aph_diag_exact_ops(int op, const double *x, double *out, long long n,
                                         void *stream) {
  clear_error();
  if (op < 0 || op > 3) return fail(APH_ERR_INVALID, "op %d not in 0..3", op);
  if (n < 0 || (n > 0 && (!x || !out))) return fail(APH_ERR_INVALID, "NULL argument");
  if (n == 0) return APH_OK;
  const long long blocks = (n + 255) / 256;
  k_exact_ops<<<(unsigned)(blocks < 152 * 16 ? blocks : 152 * 16), 256, 0, (cudaStream_t)stream>>>(
      op, x, out, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? APH_OK : cuda_fail(e, "diag_exact_ops");
}
