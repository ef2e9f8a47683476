// aph_window.cuh -- lines of cells staged in shared memory, reconstructed to face states: the
// common part of the batched stage kernel's pass items and the per-pack flux kernels.
//
// A window is V variables x T lines of n cells with the reconstruction's halo on both ends.  PPM
// forms per-cell differences, then each limited face value once (two cells share it), then the
// cells' two states.  In the exact build the two adiabatic indices of ordinary windows are not
// slabs of doubles but small-integer offsets from gamma (aph_math.cuh, gam_face).
#pragma once
#include "aph_internal.h"
#include "aph_math.cuh"

#ifndef APH_NS
#error "APH_NS must name the namespace of this translation unit"
#endif

namespace APH_NS {

using namespace aph;

// x / w for 0 <= x, x w < 2^32, with inv = ceil(2^32 / w).
__device__ __forceinline__ int quick_div(int x, int w, unsigned inv) {
  return w == 1 ? x : (int)__umulhi((unsigned)x, inv);
}
// x / w for any x >= 0: inv is less than 1 above 2^32 / w, so the high word of x inv is the quotient
// or one more.  (A division instead: the pack of kh3d 256^3 takes 0.2 % longer, the 512^2 one 0.6 %.)
__device__ __forceinline__ int wide_div(int x, int w, unsigned inv) {
  if (w == 1) return x;
  const unsigned q = __umulhi((unsigned)x, inv);
  return (int)(q - (q * (unsigned)w > (unsigned)x ? 1u : 0u));
}

template <int RECON>
struct Halo {
  static constexpr int G = RECON == RECON_PPM ? 3 : RECON == RECON_PLM ? 2 : 1;
};

// Shared-memory doubles needed by one pass item of T lines of n cells with V
// reconstructed variables.
__host__ __device__ constexpr size_t pass_smem_doubles(int recon, int n, int T, int V) {
  return recon == RECON_PPM
             ? (size_t)V * T * ((n + 6) + 2 * (n + 4) + (n + 3) + (n + 2))
             : (size_t)V * T * ((n + 2 * (recon == RECON_PLM ? 2 : 1)) + 2 * (n + 2));
}

// The adiabatic-index offsets of an item (exact build), two 16-bit values a cell: the window,
// the PPM face values, and the left and right states.
__host__ __device__ constexpr size_t gamma_smem_doubles(int recon, int n, int T) {
#if APH_EXACT
  return ((size_t)T * ((n + 2 * (recon == RECON_PPM ? 3 : recon == RECON_PLM ? 2 : 1)) + 2 * (n + 2) +
                       (recon == RECON_PPM ? n + 3 : 0)) +
          1) / 2;
#else
  return 0;
#endif
}

// What ARITH_MAIN needs for T lines.
__host__ __device__ constexpr size_t main_smem_doubles(int recon, int n, int T, int nvar) {
  return pass_smem_doubles(recon, n, T, nvar) + gamma_smem_doubles(recon, n, T);
}

// Offsets of gamma_c and gamma_e in one word.
__device__ __forceinline__ int gam_pack(int c, int e) { return (int)((unsigned)(c & 0xffff) | ((unsigned)e << 16)); }
__device__ __forceinline__ int gam_c(int x) { return (int)(short)(x & 0xffff); }
__device__ __forceinline__ int gam_e(int x) { return x >> 16; }
#if APH_EXACT
__device__ __forceinline__ bool gam_near(long long k) { return (unsigned long long)(k + kGamMax) <= 2u * kGamMax; }
// gamma far enough from the ends of its binade for the offsets of all face values
__device__ __forceinline__ bool gamma_inside(double gamma) {
  const unsigned long long m = (unsigned long long)__double_as_longlong(gamma) & 0xfffffffffffffULL;
  return m >= 4096 && m <= 0xfffffffffffffULL - 4096;
}
#endif

// The regions of a window in shared memory (V x T x width doubles each): W cells -G..n+G-1; PPM's
// second and centred differences D2 and DD (cells -2..n+1) and face values DPH (faces -1..n+1); the
// right states SR and the left states SL (in DD's place for PPM); exact: the offsets' window GW,
// states GL and GR and PPM face values GD.
struct Window {
  double *W, *D2, *DD, *DPH, *SL, *SR;
  int *GW, *GL, *GR, *GD;
};
template <int RECON>
__device__ __forceinline__ Window window_regions(double *sm, int n, int T, int V, int nvar) {
  constexpr bool P = RECON == RECON_PPM;
  const int NW = n + 2 * Halo<RECON>::G;
  Window w;
  w.W = sm;
  w.D2 = w.W + V * T * NW;
  w.DD = w.D2 + (P ? V * T * (n + 4) : 0);
  w.DPH = w.DD + (P ? V * T * (n + 4) : 0);
  w.SR = w.DPH + (P ? V * T * (n + 3) : 0);
  w.SL = P ? w.DD : w.SR + V * T * (n + 2);
  w.GW = (int *)(sm + pass_smem_doubles(RECON, n, T, nvar));
  w.GL = w.GW + T * NW;
  w.GR = w.GL + T * (n + 2);
  w.GD = w.GR + T * (n + 2);
  return w;
}

// PPM of a window: W holds V x T lines of cells -G..n+G-1 (row width n + 2G);
// per cell the second differences D2 and centred differences DD (cells -2..n+1), per face
// the limited value DPH once (faces -1..n+1), then per cell the parabola limiter writes the
// left state of face c+1 to SL[c+1] and the right state of face c to SR[c+1] (cells -1..n).
// also(0) and also(1) run beside the face and the cell phase (the adiabatic-index offsets).
// inv: the block's quick_div factors for the widths n + k.
template <bool TAME, class ALSO>
__device__ __forceinline__ void ppm_window(const double *W, double *D2, double *DD, double *DPH,
                                           double *SL, double *SR, int V, int nl, int T, int n,
                                           const unsigned *inv, ALSO also) {
  constexpr int G = 3;
  const int NW = n + 2 * G;
  const int tid = threadIdx.x, nth = blockDim.x;
  // row v * T + t of the slabs, position i in it and index o = row * w + i, for element it of rows
  // of width w (o is it where the item fills its T lines, as plain-load items do)
  const bool full = nl == T;
  auto decode = [&](int it, int w, unsigned iw, int &row, int &i, int &o) {
    row = quick_div(it, w, iw);
    i = it - row * w;
    o = it;
    if (!full) {
      const int v = row / nl;
      row += v * (T - nl);
      o = row * w + i;
    }
  };
  const int w4 = n + 4, w3 = n + 3, w2 = n + 2;
  for (int it = tid; it < V * nl * w4; it += nth) {  // cells -2..n+1
    int row, i, o;
    decode(it, w4, inv[4], row, i, o);
    const double *q = W + row * NW + i + 1;
    const double qm = q[-1], q0 = q[0], qp = q[1];
    D2[o] = ppm_d2<TAME>(qm, q0, qp);
    DD[o] = ppm_dd<TAME>(qm, q0, qp);
  }
  __syncthreads();
  for (int it = tid; it < V * nl * w3; it += nth) {  // faces -1..n+1
    int row, i, o;
    decode(it, w3, inv[3], row, i, o);
    const double *q = W + row * NW + i + 2;
    const double *d = DD + row * w4 + i, *e = D2 + row * w4 + i;
    DPH[o] = ppm_face<TAME>(q[-1], q[0], d[0], d[1], e[0], e[1]);
  }
  also(0);
  __syncthreads();
  for (int it = tid; it < V * nl * w2; it += nth) {  // cells -1..n
    int row, i, o;
    decode(it, w2, inv[2], row, i, o);
    const double *q = W + row * NW + i + 2;
    const double *e = D2 + row * w4 + i, *f = DPH + row * w3 + i;
    double ql, qr;
    ppm_cell<TAME>(q[-2], q[-1], q[0], q[1], q[2], e[0], e[1], e[2], f[0], f[1], ql, qr);
    SL[o] = ql;
    SR[o] = qr;
  }
  also(1);
}

// Reconstruction of a window (nl of its T lines): the left state of face c+1 to SL[c+1], the right
// state of face c to SR[c+1], cells c = -1..n.  TAME: every window value is tame; OFFSETS: the
// adiabatic indices are offsets (odd: gamma's last bit).  Ends without a barrier.
template <int RECON, bool TAME, bool OFFSETS>
__device__ __forceinline__ void window_states(const Window &w, int V, int nl, int T, int n, const unsigned *inv,
                                              int odd) {
  constexpr int G = Halo<RECON>::G;
  const int NW = n + 2 * G, w2 = n + 2;
  const int tid = threadIdx.x, nth = blockDim.x;
  if (RECON == RECON_PPM) {
    ppm_window<TAME>(w.W, w.D2, w.DD, w.DPH, w.SL, w.SR, V, nl, T, n, inv, [&](int phase) {
#if APH_EXACT
      if (!OFFSETS) return;
      if (phase == 0) {
        for (int it = tid; it < nl * (n + 3); it += nth) {  // faces -1..n+1
          const int t = quick_div(it, n + 3, inv[3]), f = it - t * (n + 3) - 1;
          const int *g = w.GW + t * NW + f + G;
          w.GD[it] = gam_pack(gam_face(gam_c(g[-2]), gam_c(g[-1]), gam_c(g[0]), gam_c(g[1]), odd),
                              gam_face(gam_e(g[-2]), gam_e(g[-1]), gam_e(g[0]), gam_e(g[1]), odd));
        }
      } else {
        for (int it = tid; it < nl * w2; it += nth) {  // cells -1..n
          const int t = quick_div(it, w2, inv[2]), c = it - t * w2 - 1;
          const int *g = w.GW + t * NW + c + G, *f = w.GD + t * (n + 3) + c + 1;
          int lc, rc, le, re;
          gam_cell(gam_c(g[-1]), gam_c(g[0]), gam_c(g[1]), gam_c(f[0]), gam_c(f[1]), lc, rc);
          gam_cell(gam_e(g[-1]), gam_e(g[0]), gam_e(g[1]), gam_e(f[0]), gam_e(f[1]), le, re);
          w.GL[it] = gam_pack(lc, le);
          w.GR[it] = gam_pack(rc, re);
        }
      }
#endif
    });
    return;
  }
  for (int it = tid; it < V * nl * w2; it += nth) {
    int row = quick_div(it, w2, inv[2]);
    const int i = it - row * w2;  // cell i - 1
    int o = it;
    if (nl != T) {
      row += row / nl * (T - nl);
      o = row * w2 + i;
    }
    const double *q = w.W + row * NW + i + G - 1;
    double ql, qr;
    if (RECON == RECON_PLM) plm(q[-1], q[0], q[1], ql, qr);
    else ql = qr = q[0];
    w.SL[o] = ql;
    w.SR[o] = qr;
  }
#if APH_EXACT
  if (OFFSETS) {
    for (int it = tid; it < nl * w2; it += nth) {
      const int t = quick_div(it, w2, inv[2]), c = it - t * w2 - 1;
      const int *g = w.GW + t * NW + c + G;
      int lc = gam_c(g[0]), le = gam_e(g[0]), rc = lc, re = le;
      if (RECON == RECON_PLM) {
        gam_plm(gam_c(g[-1]), gam_c(g[0]), gam_c(g[1]), odd, lc, rc);
        gam_plm(gam_e(g[-1]), gam_e(g[0]), gam_e(g[1]), odd, le, re);
      }
      w.GL[it] = gam_pack(lc, le);
      w.GR[it] = gam_pack(rc, re);
    }
  }
#endif
}

// The states (rho, v normal, v transverse, p) on both sides of a face along DIR, the left one at
// slot oL of variables vs apart, and the adiabatic indices g: gamma_c, gamma_e left, then right
// (0 where the gas is constant-gamma: V == nvar and no offsets).
template <int DIR, bool OFFSETS>
__device__ __forceinline__ void face_states(const Window &w, int oL, int vs, int V, int nvar, double gamma, double *wl,
                                            double *wr, double *g) {
  constexpr int ivx = DIR;
  constexpr int ivy = IV1 + ((ivx - IV1) + 1) % 3;
  constexpr int ivz = IV1 + ((ivx - IV1) + 2) % 3;
  const int oR = oL + 1;
  const double *SL = w.SL, *SR = w.SR;
  wl[IDN] = SL[IDN * vs + oL]; wl[IV1] = SL[ivx * vs + oL]; wl[IV2] = SL[ivy * vs + oL];
  wl[IV3] = SL[ivz * vs + oL]; wl[IPR] = SL[IPR * vs + oL];
  wr[IDN] = SR[IDN * vs + oR]; wr[IV1] = SR[ivx * vs + oR]; wr[IV2] = SR[ivy * vs + oR];
  wr[IV3] = SR[ivz * vs + oR]; wr[IPR] = SR[IPR * vs + oR];
  g[0] = g[1] = g[2] = g[3] = 0.0;
  if (OFFSETS) {
    const long long base = __double_as_longlong(gamma);
    const int l = w.GL[oL], r = w.GR[oR];
    g[0] = __longlong_as_double(base + gam_c(l));
    g[1] = __longlong_as_double(base + gam_e(l));
    g[2] = __longlong_as_double(base + gam_c(r));
    g[3] = __longlong_as_double(base + gam_e(r));
  } else if (V > nvar) {
    g[0] = SL[nvar * vs + oL];
    g[1] = SL[(nvar + 1) * vs + oL];
    g[2] = SR[nvar * vs + oR];
    g[3] = SR[(nvar + 1) * vs + oR];
  }
}

}  // namespace APH_NS
