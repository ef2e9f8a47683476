// aph_kernels.cuh -- per-pack kernels of the hydro path (the reference-style launch
// granularity: one kernel per operation over all meshblocks of a pack).
//
// Included once per arithmetic mode with APH_NS naming the namespace
// (aph_fast.cu, aph_exact.cu).
#pragma once
#include "aph_amr.cuh"
#include "aph_internal.h"
#include "aph_math.cuh"
#include "aph_window.cuh"

#ifndef APH_NS
#error "APH_NS must name the namespace of this translation unit"
#endif

namespace APH_NS {

using namespace aph;

constexpr int kThreads = 256;

__device__ __forceinline__ int dim_start(int d, int ndim, int ng) { return d < ndim ? ng : 0; }

// ---------------------------------------------------------------------------------------
// ConsToPrim over the entire domain of every block (hydro.cpp:450-532)
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_cons_to_prim(PackDev p, const BlockDev *blocks,
                                                           int *floor_flag) {
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= B.ncell) return;
  const long long nc = B.ncell;
  double u[NHYDRO], w[NHYDRO], g_c, g_e;
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) u[n] = B.cons[n * nc + c];
  const bool fl = cons_to_prim_cell(u, w, g_c, g_e, p.gm1, p.dfloor, p.pfloor);
  B.cons[IDN * nc + c] = u[IDN];
  B.cons[IEN * nc + c] = u[IEN];
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) B.prim[n * nc + c] = w[n];
  if (B.gamma) {
#if !APH_EXACT
    // the flux kernels reconstruct these fields: the reference's values, not the constants
    // the fast ConsToPrim leaves where no floor fired
    if (!fl) gamma_ref(u, p.gm1, g_c, g_e);
#endif
    B.gamma[c] = g_c;
    B.gamma[nc + c] = g_e;
  }
  if (p.nvar > NHYDRO) {
    const double di = rcp_x(u[IDN]);
    for (int n = NHYDRO; n < p.nvar; ++n) B.prim[n * nc + c] = B.cons[n * nc + c] * di;
  }
  if (B.eos_lambda && B.eos_lambda[2 * nc + c] == 0.0) B.eos_lambda[2 * nc + c] = 7.0;  // hydro.cpp:491-493
  if (fl && floor_flag) atomicOr(floor_flag, 1);
}

// ---------------------------------------------------------------------------------------
// CalculateFluxes for one direction (hydro.cpp:580-740): reconstruction of every
// primitive and both adiabatic indices on the cells s-1..e+1 of each line, then the
// Riemann solve on the faces s..e+1.  A CTA takes a segment of M cells of T lines as a window in
// shared memory (aph_window.cuh), so each face value is formed once and no state reaches HBM;
// long lines are cut so that any length fits and a pack of few lines still spreads over the SMs.
// Only lines through the interior are computed (the reference also fills the unused fluxes on
// ghost rows).  The FP64 pipe and integer issue bound it, as the stage kernel.
// ---------------------------------------------------------------------------------------
template <int DIR>
__device__ __forceinline__ void line_geometry(const BlockDev &B, int ndim, int ng, int line,
                                              int &i0, int &j0, int &k0) {
  const int si = ng, sj = dim_start(1, ndim, ng), sk = dim_start(2, ndim, ng);
  const int w = DIR == 1 ? B.nx[1] : B.nx[0], q = line / w, r = line - q * w;
  if (DIR == 1) {
    j0 = sj + r;
    k0 = sk + q;
    i0 = si;
  } else if (DIR == 2) {
    i0 = si + r;
    k0 = sk + q;
    j0 = sj;
  } else {
    i0 = si + r;
    j0 = sj + q;
    k0 = sk;
  }
}

// Where a CTA's lines lie: cells c0..c0+n-1 of lines l0..l0+nl-1.
struct Segment {
  int l0, nl, c0, n;
  bool last;  // up to the lines' ends: the high face of the last cell is the segment's too
};

// How a segment is solved: exact build, gamma offsets (kFluxMain), then double slabs on tame windows
// (kFluxSlabs); fast build, kFluxSlabs; last, any window with the IEEE instructions.  Returns kFluxDone,
// or how to take the segment instead where the window or an operand is out of range (nothing but
// fluxes to be rewritten was stored): kFluxSlabs where only the adiabatic indices are.
constexpr int kFluxMain = 0, kFluxSlabs = 1, kFluxIeee = 2, kFluxDone = 3;

template <int DIR, int RECON, int RS, int HOW>
__device__ __forceinline__ int flux_segment(const PackDev &p, const BlockDev &B, const Segment &g, int T,
                                             const unsigned *inv, double *sm) {
  constexpr int G = Halo<RECON>::G;
  constexpr bool kTame = (APH_EXACT || RECON == RECON_PPM) && HOW != kFluxIeee, kOffsets = HOW == kFluxMain;
  const int nvar = p.nvar, V = kOffsets ? nvar : nvar + 2, n = g.n, nl = g.nl, NW = n + 2 * G;
  const int tid = threadIdx.x, nth = blockDim.x;
  const long long nc = B.ncell;
  const long long stride = DIR == 1 ? 1 : DIR == 2 ? B.ni : (long long)B.ni * B.nj;
  const Window w = window_regions<RECON>(sm, n, T, V, nvar);
  bool tame_ok = true, offset_ok = true;
#if APH_EXACT
  const long long gbase = __double_as_longlong(p.gamma);
  const int odd = (int)gbase & 1;
#else
  const int odd = 0;
#endif
  for (int it = tid; it < nl * NW; it += nth) {
    int t, x0;
    if (DIR == 1) { t = it / NW; x0 = it - t * NW; }
    else { x0 = it / nl; t = it - x0 * nl; }
    int i0, j0, k0;
    line_geometry<DIR>(B, p.ndim, p.ng, g.l0 + t, i0, j0, k0);
    const long long cell = ((long long)k0 * B.nj + j0) * B.ni + i0 + (long long)(g.c0 + x0 - G) * stride;
    double x[NHYDRO];  // (loads before stores: they would wait for one another)
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v) x[v] = B.prim[v * nc + cell];
    const double gc = B.gamma[cell], ge = B.gamma[nc + cell];
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v) {
      w.W[(v * T + t) * NW + x0] = x[v];
      if (kTame) tame_ok = tame_ok & snug(x[v]);
    }
    for (int v = NHYDRO; v < nvar; ++v) {
      const double y = B.prim[v * nc + cell];
      w.W[(v * T + t) * NW + x0] = y;
      if (kTame) tame_ok = tame_ok & tame(y);
    }
#if APH_EXACT
    if (kOffsets) {
      const long long kc = __double_as_longlong(gc) - gbase, ke = __double_as_longlong(ge) - gbase;
      offset_ok = offset_ok & gam_near(kc) & gam_near(ke);
      w.GW[t * NW + x0] = gam_pack((int)kc, (int)ke);
    }
#endif
    if (!kOffsets) {
      w.W[(nvar * T + t) * NW + x0] = gc;
      w.W[((nvar + 1) * T + t) * NW + x0] = ge;
      if (kTame) tame_ok = tame_ok & snug(gc) & snug(ge);
    }
  }
#if APH_EXACT
  if (kOffsets) offset_ok = offset_ok && gamma_inside(p.gamma);
#endif
  if (kTame) {
    if (!__syncthreads_and(tame_ok & offset_ok)) return kOffsets && __syncthreads_and(tame_ok) ? kFluxSlabs : kFluxIeee;
  } else {
    __syncthreads();
  }
  window_states<RECON, kTame, kOffsets>(w, V, nl, T, n, inv, odd);
  __syncthreads();

  // Riemann solve, one item per (line, face); face f in [0, n]
  constexpr int ivx = DIR;
  constexpr int ivy = IV1 + ((ivx - IV1) + 1) % 3;
  constexpr int ivz = IV1 + ((ivx - IV1) + 2) % 3;
  const GasConsts none{};
  double *flux = B.flux[DIR - 1];
  const int nf = g.last ? n + 1 : n, w2 = n + 2, vs = T * w2;
  bool in_range = true;
  for (int it = tid; it < nl * nf; it += nth) {
    int t, f;
    if (DIR == 1) { t = it / nf; f = it - t * nf; }
    else { f = it / nl; t = it - f * nl; }
    double wl[NHYDRO], wr[NHYDRO], gm[4], flx[NHYDRO];
    const int oL = t * w2 + f;
    face_states<DIR, kOffsets>(w, oL, vs, V, nvar, p.gamma, wl, wr, gm);
    if (HOW == kFluxIeee) {
      IeeeOps o;
      riemann<RS, false>(wl, wr, gm[0], gm[1], gm[2], gm[3], none, flx, o);
    } else {
      SolveOps o;
      riemann<RS, false>(wl, wr, gm[0], gm[1], gm[2], gm[3], none, flx, o);
      in_range = in_range & o.ok();
    }
    int i0, j0, k0;
    line_geometry<DIR>(B, p.ndim, p.ng, g.l0 + t, i0, j0, k0);
    // face f of the segment: cell (k0, j0, i0) moved c0 + f cells along DIR, in flux's layout
    const long long *fs = B.fs[DIR - 1];
    const int m = g.c0 + f;
    double *out = flux + (long long)(k0 + (DIR == 3 ? m : 0)) * fs[1] + (long long)(j0 + (DIR == 2 ? m : 0)) * fs[2] +
                  (i0 + (DIR == 1 ? m : 0));
    const long long fn = fs[0];
    out[IDN * fn] = flx[IDN];
    out[ivx * fn] = flx[IV1];
    out[ivy * fn] = flx[IV2];
    out[ivz * fn] = flx[IV3];
    out[IEN * fn] = flx[IEN];
    // passive scalars: upwind by the mass flux (hydro.cpp:607-615)
    for (int v = NHYDRO; v < nvar; ++v)
      out[v * fn] = flx[IDN] * (!is_neg(flx[IDN]) ? w.SL[v * vs + oL] : w.SR[v * vs + oL + 1]);
  }
  return HOW == kFluxIeee || __syncthreads_and(in_range) ? kFluxDone : kFluxIeee;
}

// A segment whose window left the first arithmetic's range, in chunks of lines that fit the slabs of
// the adiabatic indices (out of line: it is rare).
template <int DIR, int RECON, int RS>
static __device__ __noinline__ void flux_general(const PackDev &p, const BlockDev &B, Segment g, int T,
                                                 const unsigned *inv, double *sm, int how) {
  const int l0 = g.l0, nl = g.nl;
  const int Tc = APH_EXACT ? max(1, p.nvar * T / (p.nvar + 2)) : T;
  for (int o = 0; o < nl; o += Tc) {
    g.l0 = l0 + o;
    g.nl = min(Tc, nl - o);
    __syncthreads();
    if (APH_EXACT && how == kFluxSlabs && flux_segment<DIR, RECON, RS, kFluxSlabs>(p, B, g, Tc, inv, sm) == kFluxDone)
      continue;
    __syncthreads();
    flux_segment<DIR, RECON, RS, kFluxIeee>(p, B, g, Tc, inv, sm);
  }
}

template <int DIR, int RECON, int RS, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_fluxes(const __grid_constant__ PackDev p, const BlockDev *blocks,
                                                        int T, int M, int nseg) {
  extern __shared__ __align__(16) double sm[];
  __shared__ unsigned inv[7];
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  const int ntrans = (DIR == 1) ? B.nx[1] * B.nx[2] : (DIR == 2) ? B.nx[0] * B.nx[2] : B.nx[0] * B.nx[1];
  const int N = B.nx[DIR - 1];
  Segment g;
  g.l0 = (int)(blockIdx.x / nseg) * T;
  g.c0 = (int)(blockIdx.x % nseg) * M;
  if (g.l0 >= ntrans || g.c0 >= N) return;
  g.nl = min(T, ntrans - g.l0);
  g.n = min(M, N - g.c0);
  g.last = g.c0 + g.n == N;
  if (threadIdx.x < 7) inv[threadIdx.x] = 0xffffffffu / (unsigned)(g.n + threadIdx.x) + 1u;
  __syncthreads();
  const int how = flux_segment<DIR, RECON, RS, APH_EXACT ? kFluxMain : kFluxSlabs>(p, B, g, T, inv, sm);
  if (how != kFluxDone) flux_general<DIR, RECON, RS>(p, B, g, T, inv, sm, how);
}

// ---------------------------------------------------------------------------------------
// UpdateWithFluxDivergence over the interior: u0 = gam0 u0 + gam1 u1 + beta_dt (-div F)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ bool interior_cell(const BlockDev &B, int ndim, int ng, int idx,
                                              long long &cell, int &ci, int &cj, int &ck) {
  const int n0 = B.nx[0], n1 = B.nx[1], n2 = B.nx[2];
  if (idx >= n0 * n1 * n2) return false;
  const int i = idx % n0, j = (idx / n0) % n1, k = idx / (n0 * n1);
  const int si = ng, sj = dim_start(1, ndim, ng), sk = dim_start(2, ndim, ng);
  ci = i + si;
  cj = j + sj;
  ck = k + sk;
  cell = ((long long)ck * B.nj + cj) * B.ni + ci;
  return true;
}
// Index of face (k, j, i) of component n in flux[d] (face i on the low side of cell i).
__device__ __forceinline__ long long flux_index(const BlockDev &B, int d, int n, int k, int j, int i) {
  return n * B.fs[d][0] + k * B.fs[d][1] + j * B.fs[d][2] + i;
}

__global__ void __launch_bounds__(kThreads) k_update(PackDev p, const BlockDev *blocks,
                                                     double gam0, double gam1, double beta,
                                                     double beta_dt_host, const double *dt_dev) {
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  long long c;
  int ci, cj, ck;
  if (!interior_cell(B, p.ndim, p.ng, blockIdx.x * blockDim.x + threadIdx.x, c, ci, cj, ck)) return;
  const double beta_dt = dt_dev ? beta * dt_dev[0] : beta_dt_host;
  const double a1 = B.dx[1] * B.dx[2], a2 = B.dx[0] * B.dx[2], a3 = B.dx[0] * B.dx[1];
  const long long nc = B.ncell;
#if APH_EXACT
  // areas, the volume and RK factors that are powers of two (every mesh of such widths) are
  // exponent steps: the FP64 pipe is what this kernel waits for (KH 128^3: 517 us with products
  // and a division per variable)
  const double vol = B.dx[0] * B.dx[1] * B.dx[2];
  const double ivol = rcp_x(vol);
  const bool p2 = pow2_normal(vol);
  const int k1 = pow2_step(a1), k2 = pow2_step(a2), k3 = pow2_step(a3);
  const RkForm rk = rk_form(gam0, gam1);
  auto times = [](double f, double area, int k) { return k != kNoStep ? scale_x(f, area, k) : f * area; };
#else
  const Den vol_den = den(B.dx[0] * B.dx[1] * B.dx[2]);
#endif
  // five variables at a time, every load before the first store (they would wait for one another)
  const long long f0 = flux_index(B, 0, 0, ck, cj, ci), s0 = B.fs[0][0];
  const long long f1 = p.ndim >= 2 ? flux_index(B, 1, 0, ck, cj, ci) : 0, s1 = B.fs[1][0];
  const long long f2 = p.ndim == 3 ? flux_index(B, 2, 0, ck, cj, ci) : 0, s2 = B.fs[2][0];
  constexpr int K = 5;
  for (int m = 0; m < p.nvar; m += K) {
    double x[K][8];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int n = m + k;
      if (n >= p.nvar) break;
      x[k][0] = B.flux[0][f0 + n * s0 + 1];
      x[k][1] = B.flux[0][f0 + n * s0];
      if (p.ndim >= 2) {
        x[k][2] = B.flux[1][f1 + n * s1 + B.fs[1][2]];
        x[k][3] = B.flux[1][f1 + n * s1];
      }
      if (p.ndim == 3) {
        x[k][4] = B.flux[2][f2 + n * s2 + B.fs[2][1]];
        x[k][5] = B.flux[2][f2 + n * s2];
      }
      x[k][6] = B.cons[n * nc + c];
      x[k][7] = B.u1[n * nc + c];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (m + k >= p.nvar) break;
#if APH_EXACT
      double du = times(x[k][0], a1, k1) - times(x[k][1], a1, k1);
      if (p.ndim >= 2) du += times(x[k][2], a2, k2) - times(x[k][3], a2, k2);
      if (p.ndim == 3) du += times(x[k][4], a3, k3) - times(x[k][5], a3, k3);
#else
      double du = (a1 * x[k][0] - a1 * x[k][1]);
      if (p.ndim >= 2) du += (a2 * x[k][2] - a2 * x[k][3]);
      if (p.ndim == 3) du += (a3 * x[k][4] - a3 * x[k][5]);
#endif
#if APH_EXACT
      B.cons[(m + k) * nc + c] = rk_sum(rk, x[k][6], x[k][7]) + beta_dt * div_vol(-du, vol, ivol, p2);
#else
      const double div = div_x(-du, vol_den);
      B.cons[(m + k) * nc + c] = gam0 * x[k][6] + gam1 * x[k][7] + beta_dt * div;
#endif
    }
  }
}

// Face (a along d, t across) of component n of flux[d] of a 2D block (as amr_cell).
__device__ __forceinline__ long long amr_face(const BlockDev &B, int ng, int d, int n, int a, int t) {
  const int i = d == 0 ? ng + a : ng + t;
  const int j = d == 0 ? ng + t : ng + a;
  return flux_index(B, d, n, 0, j, i);
}

// Refined 2D meshes: the same update with the coarse-fine correction of each coarse
// boundary cell's flux difference to the mean of the fine face fluxes (faces x-, x+, y-, y+).
__global__ void __launch_bounds__(kThreads) k_update_amr(PackDev p, const BlockDev *blocks,
                                                         double gam0, double gam1, double beta,
                                                         double beta_dt_host, const double *dt_dev) {
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  long long c;
  int ci, cj, ck;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (!interior_cell(B, p.ndim, p.ng, idx, c, ci, cj, ck)) return;
  const int ii = idx % B.nx[0], jj = idx / B.nx[0];
  const double beta_dt = dt_dev ? beta * dt_dev[0] : beta_dt_host;
  const double a1 = B.dx[1] * B.dx[2], a2 = B.dx[0] * B.dx[2];
  const Den vol = den(B.dx[0] * B.dx[1] * B.dx[2]);
  const long long nc = B.ncell;
  for (int n = 0; n < p.nvar; ++n) {
    const long long q = n * nc + c;
    const long long f1 = flux_index(B, 0, n, 0, cj, ci), f2 = flux_index(B, 1, n, 0, cj, ci);
    double du = (a1 * B.flux[0][f1 + 1] - a1 * B.flux[0][f1]);
    du += (a2 * B.flux[1][f2 + B.fs[1][2]] - a2 * B.flux[1][f2]);
    for (int face = 0; face < 4; ++face) {
      if (B.amr.kind[face] != FACE_FINER) continue;
      const int d = face / 2, s = face % 2, td = 1 - d;
      const int a = d == 0 ? ii : jj, t = d == 0 ? jj : ii;
      if (a != (s == 0 ? 0 : B.nx[d] - 1)) continue;
      const double area = d == 0 ? a1 : a2;
      const int tg2 = 2 * (B.amr.origin[td] + t);
      const BlockDev &F = amr_fine_nbr(blocks, B, face, td, tg2);
      const int ft = tg2 - F.amr.origin[td];
      const long long fo = amr_face(B, p.ng, d, n, s == 0 ? 0 : B.nx[d], t);
      const int ffa = s == 0 ? F.nx[d] : 0;
      const long long g0 = amr_face(F, p.ng, d, n, ffa, ft);
      const long long g1 = amr_face(F, p.ng, d, n, ffa, ft + 1);
      const double Fold = B.flux[d][fo];
      const double Fnew = 0.5 * (F.flux[d][g0] + F.flux[d][g1]);
      du = s == 0 ? du + (area * Fold - area * Fnew) : du + (area * Fnew - area * Fold);
    }
    const double div = div_x(-du, vol);
    B.cons[q] = gam0 * B.cons[q] + gam1 * B.u1[q] + beta_dt * div;
  }
}

// ---------------------------------------------------------------------------------------
// EstimateTimestep (hydro.cpp:369-417): per-cell candidate, warp-shuffle min, one
// atomic per CTA on the bit pattern (positive doubles order like unsigned integers,
// NaN candidates sort above +inf and are ignored as fmin ignores them).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long block_min_bits(unsigned long long v) {
  __shared__ unsigned long long red[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, v, o);
    v = x < v ? x : v;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : ~0ULL;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, v, o);
      v = x < v ? x : v;
    }
  }
  return v;
}

__global__ void __launch_bounds__(kThreads) k_estimate_dt(PackDev p, const BlockDev *blocks,
                                                          unsigned long long *min_bits) {
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  long long c;
  unsigned long long v = ~0ULL;
  int ci, cj, ck;
  if (interior_cell(B, p.ndim, p.ng, blockIdx.x * blockDim.x + threadIdx.x, c, ci, cj, ck)) {
    const long long nc = B.ncell;
    double w[NHYDRO];
#pragma unroll
    for (int n = 0; n < NHYDRO; ++n) w[n] = B.prim[n * nc + c];
    const double m = dt_candidate(w, B.cons[IEN * nc + c], B.dx, p.ndim, p.gm1);
    v = (unsigned long long)__double_as_longlong(m);
    if (is_neg(m)) v = ~0ULL;
  }
  v = block_min_bits(v);
  if (threadIdx.x == 0 && v != ~0ULL) atomicMin(min_bits, v);
}

// ---------------------------------------------------------------------------------------
// ApplyGravity, constant field (gravity.cpp:386-407); prim is the state of the previous
// FillDerived, as in the reference.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_apply_gravity(PackDev p, const BlockDev *blocks,
                                                            double g0, double g1, double g2,
                                                            double beta, double beta_dt_host,
                                                            const double *dt_dev) {
  const BlockDev &B = blocks[p.block0 + blockIdx.y];
  long long c;
  int ci, cj, ck;
  if (!interior_cell(B, p.ndim, p.ng, blockIdx.x * blockDim.x + threadIdx.x, c, ci, cj, ck)) return;
  const double dt = dt_dev ? beta * dt_dev[0] : beta_dt_host;
  const long long nc = B.ncell;
  const double rho = B.prim[IDN * nc + c];
  B.cons[IM1 * nc + c] += g0 * rho * dt;
  double de = g0 * B.prim[IV1 * nc + c];
  if (p.ndim >= 2) {
    B.cons[IM2 * nc + c] += g1 * rho * dt;
    de += g1 * B.prim[IV2 * nc + c];
  }
  if (p.ndim >= 3) {
    B.cons[IM3 * nc + c] += g2 * rho * dt;
    de += g2 * B.prim[IV3 * nc + c];
  }
  B.cons[IEN * nc + c] += de * rho * dt;
}

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// Launch shapes.  FP64 issue is a per-SM resource (a few lanes per clock), so a launch
// that covers few SMs -- one small meshblock at a time -- is bound by the latency of its
// longest thread.  Small launches therefore use fewer threads (or lines) per CTA, down to
// one warp, until the grid spans about two CTAs per SM; launches over a whole pack keep the
// full CTA.  The arithmetic of every cell is the same for any shape.
static int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 152;
    cached[dev] = n;
  }
  return cached[dev];
}

static int launch_threads(long long work, int nblocks) {
  const long long want = 2LL * sm_count();
  int t = kThreads;
  while (t > 32 && (long long)cdiv(work, t) * nblocks < want) t >>= 1;
  return t;
}

cudaError_t launch_cons_to_prim(const PackDev &p, const BlockDev *blocks, int max_ncell,
                                int *floor_flag, cudaStream_t s) {
  const int nt = launch_threads(max_ncell, p.nblocks);
  dim3 grid(cdiv(max_ncell, nt), p.nblocks);
  k_cons_to_prim<<<grid, nt, 0, s>>>(p, blocks, floor_flag);
  return cudaGetLastError();
}

constexpr size_t kSegmentBytes = 200 * 1024;  // the most shared memory of a segment

template <int DIR, int RECON, int RS, int MINB>
static cudaError_t launch_segments(const PackDev &p, const BlockDev *blocks, dim3 grid, int nt, size_t smem,
                                   int T, int n, int nseg, cudaStream_t s) {
  if (smem > 48 * 1024) {  // the attribute belongs to the device and its context: not kept from one call for the next
    cudaError_t e = cudaFuncSetAttribute(k_fluxes<DIR, RECON, RS, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSegmentBytes);
    if (e != cudaSuccess) return e;
  }
  k_fluxes<DIR, RECON, RS, MINB><<<grid, nt, smem, s>>>(p, blocks, T, n, nseg);
  return cudaGetLastError();
}

template <int DIR, int RECON, int RS>
static cudaError_t launch_fluxes_t(const PackDev &p, const BlockDev *blocks, cudaStream_t s) {
  // segments of at most kSegment cells (fewer where many scalars would not fit), evenly cut: their
  // halo costs 2 G cells of window each
  constexpr int kSegment = 160;
  const int N = p.max_nx[DIR - 1];
  int nseg = (N + kSegment - 1) / kSegment, n = (N + nseg - 1) / nseg;
  auto bytes = [&](int T) {
    const size_t general = pass_smem_doubles(RECON, n, APH_EXACT ? 1 : T, p.nvar + 2);
    const size_t main = APH_EXACT ? main_smem_doubles(RECON, n, T, p.nvar) : 0;
    return sizeof(double) * (general > main ? general : main);
  };
  while (bytes(1) > kSegmentBytes && n > 1) {
    ++nseg;
    n = (N + nseg - 1) / nseg;
  }
  if (bytes(1) > kSegmentBytes) return cudaErrorInvalidValue;
  long long ntrans;
  if (DIR == 1) ntrans = (long long)p.max_nx[1] * p.max_nx[2];
  else if (DIR == 2) ntrans = (long long)p.max_nx[0] * p.max_nx[2];
  else ntrans = (long long)p.max_nx[0] * p.max_nx[1];
  int T = std::max(1, kThreads / (n + 2));
  while (T > 1 && (bytes(T) > kSegmentBytes / 2 || (long long)cdiv(ntrans, T) * nseg * p.nblocks < 2LL * sm_count()))
    T = (T + 1) / 2;
  const int nt = (int)std::min<long long>(kThreads, 32LL * cdiv((long long)p.nvar * T * (n + 2), 32));
  const size_t smem = bytes(T);
  dim3 grid(cdiv(ntrans, T) * nseg, p.nblocks);
  // Exact mode, more segments than two CTAs an SM: three (80 registers and some spills; 128^3 in blocks of 64^3
  // take 5.57 ms a step where two take 5.94), or else two, whose segments end sooner (meshblocks one
  // by one, 32^2 cells each: 1.425 ms a step against 1.46)
  constexpr int kMost3 = APH_EXACT ? 3 : 2;
  if ((long long)grid.x * grid.y > 2LL * sm_count())
    return launch_segments<DIR, RECON, RS, kMost3>(p, blocks, grid, nt, smem, T, n, nseg, s);
  return launch_segments<DIR, RECON, RS, 2>(p, blocks, grid, nt, smem, T, n, nseg, s);
}

template <int DIR>
static cudaError_t launch_fluxes_dir(const PackDev &p, const BlockDev *blocks, int recon,
                                     int rsolver, cudaStream_t s) {
#define APH_RS_CASES(RC)                                                      \
  switch (rsolver) {                                                          \
    case RS_HLLE: return launch_fluxes_t<DIR, RC, RS_HLLE>(p, blocks, s);     \
    case RS_HLLC: return launch_fluxes_t<DIR, RC, RS_HLLC>(p, blocks, s);     \
    case RS_LHLLC: return launch_fluxes_t<DIR, RC, RS_LHLLC>(p, blocks, s);   \
    default: break;                                                           \
  }
  if (recon == RECON_DC) {
    if (rsolver == RS_NONE) return launch_fluxes_t<DIR, RECON_DC, RS_NONE>(p, blocks, s);
    APH_RS_CASES(RECON_DC)
  } else if (recon == RECON_PLM) {
    APH_RS_CASES(RECON_PLM)
  } else if (recon == RECON_PPM) {
    APH_RS_CASES(RECON_PPM)
  }
#undef APH_RS_CASES
  return cudaErrorInvalidValue;
}

cudaError_t launch_fluxes(const PackDev &p, const BlockDev *blocks, int dir, int recon,
                          int rsolver, cudaStream_t s) {
  if (dir == 1) return launch_fluxes_dir<1>(p, blocks, recon, rsolver, s);
  if (dir == 2) return launch_fluxes_dir<2>(p, blocks, recon, rsolver, s);
  if (dir == 3) return launch_fluxes_dir<3>(p, blocks, recon, rsolver, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_update(const PackDev &p, const BlockDev *blocks, double gam0, double gam1,
                          double beta, double beta_dt_host, const double *dt_dev,
                          int max_interior, cudaStream_t s) {
  const int nt = launch_threads(max_interior, p.nblocks);
  dim3 grid(cdiv(max_interior, nt), p.nblocks);
  if (p.amr)
    k_update_amr<<<grid, nt, 0, s>>>(p, blocks, gam0, gam1, beta, beta_dt_host, dt_dev);
  else
    k_update<<<grid, nt, 0, s>>>(p, blocks, gam0, gam1, beta, beta_dt_host, dt_dev);
  return cudaGetLastError();
}

cudaError_t launch_estimate_dt(const PackDev &p, const BlockDev *blocks, int max_interior,
                               unsigned long long *min_bits, cudaStream_t s) {
  const int nt = launch_threads(max_interior, p.nblocks);
  dim3 grid(cdiv(max_interior, nt), p.nblocks);
  k_estimate_dt<<<grid, nt, 0, s>>>(p, blocks, min_bits);
  return cudaGetLastError();
}

cudaError_t launch_apply_gravity(const PackDev &p, const BlockDev *blocks, double g0, double g1,
                                 double g2, double beta, double beta_dt_host,
                                 const double *dt_dev, int max_interior, cudaStream_t s) {
  const int nt = launch_threads(max_interior, p.nblocks);
  dim3 grid(cdiv(max_interior, nt), p.nblocks);
  k_apply_gravity<<<grid, nt, 0, s>>>(p, blocks, g0, g1, g2, beta, beta_dt_host, dt_dev);
  return cudaGetLastError();
}

}  // namespace APH_NS
