// lh_kernels.cuh — CUDA kernels of the RK3 substep outside its transform passes, which are in
// lh_fxpass.cuh (FP64 form, fixed point) and lh_xpass2.cuh (mixed form, FP32).
//
// Per substep (littleharsh.f90:174-217):
//   k_zinv_fx, k_zinv2  : stagger interpolation (FOU3D.f90:427-474) fused into the inverse z
//                 transforms of the six velocity planes of every level (cft, iopt>=0)
//   k_xpass_fx, k_xpass2 / k_xpass3 : inverse x transforms (rft, iopt>=0), physical products
//                 (ops_in_planes2, FOU3D.f90:2090-2251), CFL maxima (dtc_calc), forward x
//                 transforms (rft, iopt<0) of the products
//   k_zfwd_fx, k_zfwd2  : forward z transforms (cft, iopt<0) + der_x/der_z (FOU3D.f90:476-593):
//                 N_xz of u, v, w and the y-flux products uv, vv, wv
//   k_dt        : dt = min(2.5 dtv, CFL dtc) on the device (FOU3D.f90:291-297)
//   k_helm64    : RHS0 + der_y_h + du += -gRK N + solveU_W / solveV of the FP64 form, both parts of
//                 a column in a lane; channels of few columns: k_helm_rhs, k_helm_sweep64
//   k_meanflow  : flowrate_corr on mode (0,0) (constant flow rate)
//   k_press3 (k_press2), or k_press_rhs, k_press_sweep, k_press_corr : divergence + solveP (LUsolP with the stored factors, k_build_dg) + v_corr
//                 + divergence of the corrected field in the third substep (max |div| -> err)
//   k_ib_du(_mx), k_spec_zinv(_fx, 2), k_ib_xforce(_fx), k_zfwd_spec(_fx, 2) : immersed-boundary
//                 forcing of du (imm_bounds_u/v, FOU3D.f90:806-998) when the geometry has posts
//   Mixed form (LH_PREC_MIXED): FP32 transforms, and k_helm_u_mx2 / k_helm_v_mx2 (staged: _mx3; few
//   columns: k_helm_rhs_mx, k_helm_sweep_mx) solve the Helmholtz systems for the increment in FP32
//   on top of the FP64 state.
// On request: k_xstats, k_wx_stats, k_spectra, k_slip (statistics), k_band_io, k_transpose
// (state I/O).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "lh_internal.cuh"

#define NTHR 256
// blocks per SM the compiler leaves registers for in the immersed-boundary kernels (sweep knobs)
#ifndef LH_IBDU_MINB
#define LH_IBDU_MINB 1
#endif
#ifndef LH_IBX_MINB
#define LH_IBX_MINB 1
#endif

__device__ __forceinline__ void atomic_max_pos(unsigned long long *addr, double v) {
  atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// max that keeps a NaN (fmax drops it): the CFL and divergence maxima must carry a
// non-finite state to dt and err, where the blow-up guard sees it
template <typename T>
__device__ __forceinline__ T nmax(T a, T b) { return (b > a || b != b) ? b : a; }
// running maximum of non-negative doubles (or NaN) kept as their bit patterns: the integer
// order of those patterns is the order of the values, a NaN above every number, so the
// comparisons stay off the FP64 pipe; warp_max_bits reduces it over the warp
__device__ __forceinline__ void bits_max(unsigned long long &m, double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  m = b > m ? b : m;
}
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long m) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, m, o);
    m = w > m ? w : m;
  }
  return m;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
  for (int o = 16; o > 0; o >>= 1) {
    T w = __shfl_xor_sync(0xffffffffu, v, o);
    v = (w > v || isnan((double)w)) ? w : v;
  }
  return v;
}

// Lines per block of the transform kernels, from a shared-memory budget per
// kernel (same values on the host and the device). The budgets set how many
// blocks share an SM; the defaults are the fastest of a sweep on GB300 at C1.
#ifndef LH_BUDGET_ZINV
#define LH_BUDGET_ZINV 49152
#endif
#ifndef LH_BUDGET_XPASS
#define LH_BUDGET_XPASS 24576
#endif
__host__ __device__ constexpr int lh_clamp(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
template <typename V> __host__ __device__ constexpr int kb_zinv(int n) {
  return lh_clamp(LH_BUDGET_ZINV / (2 * n * (int)sizeof(V)), 1, 16);
}
template <typename V> __host__ __device__ constexpr int pb_xpass(int n) {
  return lh_clamp(LH_BUDGET_XPASS / (8 * n * (int)sizeof(V)), 1, 8);
}

// Transform intermediates. A (after the inverse z pass): [(slot*3 + f)][l][kx], l = 0..G2-1,
// kx = 0..N1h-1. B (after the x pass): [pslot][l/2][kx][l%2] (the two rows of a pair interleaved,
// so that the z pass reads a few columns of a row pair as one contiguous run); pslot = slot*4 + p
// (u levels), nuI*4 + (slot-nuI)*2 + p (v). The x pass carries each pair of rows (l, l+1) of a
// field in one complex line (row l in .x, row l+1 in .y after the transform). Optional capture:
// physical velocities of selected levels, [cap][f][l][m].

// Levels loaded ahead in the y sweeps of the column solves (0: a plain loop). Without it
// a sweep's loads wait for the previous level's stores (the compiler cannot separate the
// addresses), one memory latency per level. Deeper prefetch costs registers, i.e. resident
// warps; the depths below were the fastest of a sweep at 256x256x301 (mixed form).
#ifndef LH_PF_PRESS
#define LH_PF_PRESS 1
#endif
#ifndef LH_PF_HU
#define LH_PF_HU 1
#endif
#ifndef LH_PF_HU_BACK
#define LH_PF_HU_BACK 2
#endif
#ifndef LH_PF_HV
#define LH_PF_HV 4
#endif
#ifndef LH_PF_HV_BACK
#define LH_PF_HV_BACK 2
#endif
#ifndef LH_PRESS_MINB
#define LH_PRESS_MINB 1
#endif
// ============================================================================
// Statistics (stats.f90:1-250) of one plane class: the x pass's gather and inverse
// transform, then the plane sums (per level) and the tile-conditioned sums (wall-band
// planes: conddown1/2 at the bottom, condup1/2 mirrored at the top with V's sign
// flipped). u slots hold (u, v interpolated, w), v slots (u interpolated, v, w
// interpolated). Sums: block reduction, one FP64 atomic per quantity and block; the
// conditioned sums add the ntilex tiles of a row in registers first.
// pl: [11][nu] (quantities 0-8 here); cd: [9][ncl][dnz][dnx].
// ============================================================================
template <int N, int PB, typename V>
__device__ __forceinline__ void xstats_sums(const V *__restrict__ res, const Geo &g, double *__restrict__ pl,
                                            double *__restrict__ cd, int ncl, int dnx, int dnz, int ntx, bool isU, int q,
                                            int l0, int npairs) {
  constexpr int G1 = N;
  __shared__ double red[16][6];
  // plane sums
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (int idx = threadIdx.x; idx < PB * G1; idx += blockDim.x) {
    const int pb = idx / G1, m = idx - pb * G1;
    if (pb >= npairs) continue;
    const V u = res[(0 * PB + pb) * G1 + m], v = res[(1 * PB + pb) * G1 + m], w = res[(2 * PB + pb) * G1 + m];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double a = to_d(h ? u.y : u.x), b = to_d(h ? v.y : v.x), c = to_d(h ? w.y : w.x);
      if (isU) { s[0] += a; s[1] += a * a; s[2] += c; s[3] += c * c; s[4] += a * b; s[5] += a * c; }
      else { s[0] += b; s[1] += b * b; s[2] += b * c; }
    }
  }
  const int nq = isU ? 6 : 3, qb = isU ? 0 : 6;
  for (int t = 0; t < nq; ++t) {
    double x = s[t];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][t] = x;
  }
  __syncthreads();
  if (threadIdx.x < nq) {
    double x = 0;
    for (int wi = 0; wi < (int)(blockDim.x >> 5); ++wi) x += red[wi][threadIdx.x];
    atomicAdd(&pl[(size_t)(qb + threadIdx.x) * g.nu + q], x);
  }
  // tile-conditioned sums on the wall-band planes
  if (!dnx) return;
  const int j = q - g.dny;
  const int *NN = isU ? g.N4 : g.N3;
  int j1, sv;
  if (j <= NN[1]) { j1 = j - NN[0]; sv = 1; }
  else if (j > NN[2]) { j1 = NN[3] + 1 - j; sv = -1; }
  else return;
  for (int idx = threadIdx.x; idx < 2 * npairs * dnx; idx += blockDim.x) {
    const int rr = idx / dnx, i = idx - rr * dnx;
    const int pb = rr >> 1, h = rr & 1;
    const int k = (l0 + rr) % dnz;
    double c[6] = {0, 0, 0, 0, 0, 0};
    for (int ix = 0; ix < ntx; ++ix) {
      const int m = i + dnx * ix;
      const V u = res[(0 * PB + pb) * G1 + m], v = res[(1 * PB + pb) * G1 + m], w = res[(2 * PB + pb) * G1 + m];
      const double a = to_d(h ? u.y : u.x), b = to_d(h ? v.y : v.x) * sv, cc = to_d(h ? w.y : w.x);
      if (isU) { c[0] += a; c[1] += a * a; c[2] += cc; c[3] += cc * cc; c[4] += a * b; c[5] += a * cc; }
      else { c[0] += b; c[1] += b * b; c[2] += b * cc; }
    }
    for (int t = 0; t < nq; ++t)
      atomicAdd(&cd[(((size_t)(qb + t) * ncl + (j1 - 1)) * dnz + k) * dnx + i], c[t]);
  }
}

// mixed form (FP64 form: k_xstats_fx)
template <int N>
__global__ void __launch_bounds__(NTHR) k_xstats(const float2 *__restrict__ A, Geo g, const float2 *__restrict__ twx,
                                                 double *__restrict__ pl, double *__restrict__ cd, int ncl, int dnx,
                                                 int dnz, int ntx) {
  typedef float2 V;
  constexpr int PB = pb_xpass<V>(N);
  constexpr int G1 = N, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G2 = g.G2, N1h = g.N1h;
  V *b0 = reinterpret_cast<V *>(smem_raw);
  V *b1 = b0 + 4 * PB * G1;
  const int slot = blockIdx.y;
  const bool isU = slot < g.nuI;
  const int q = slot_level(g, slot, isU);
  const int l0 = blockIdx.x * PB * 2;
  const int npairs = min(PB, (G2 - l0) / 2);
  const size_t fstride = (size_t)G2 * N1h;
  const V *Af = A + (size_t)slot * 3 * fstride;
  for (int idx = threadIdx.x; idx < 3 * PB * G1; idx += blockDim.x) {
    const int line = idx / G1, m = idx - line * G1;
    const int f = line / PB, pb = line - f * PB;
    V z = czero<V>();
    if (pb < npairs) {
      const int l = l0 + 2 * pb;
      int k = m;
      bool conjpart = false;
      if (m > H) { k = G1 - m; conjpart = true; }
      if (k < N1h) {
        V a = Af[f * fstride + (size_t)l * N1h + k];
        V b = Af[f * fstride + (size_t)(l + 1) * N1h + k];
        if (k == 0 || k == H) { a.y = 0; b.y = 0; }
        if (!conjpart) { z.x = a.x - b.y; z.y = a.y + b.x; }
        else { z.x = a.x + b.y; z.y = -a.y + b.x; }
      }
    }
    b0[idx] = z;
  }
  __syncthreads();
  const V *res = line_fft<true, N, 3 * PB, false>(b0, b1, twx);
  xstats_sums<N, PB>(res, g, pl, cd, ncl, dnx, dnz, ntx, isU, q, l0, npairs);
}

// ============================================================================
// dt (kRK = 1): dtc_calc + MPI_ALLREDUCE(MIN) + dt = min(2.5 dtv, CFL dtc)
// ============================================================================
__global__ void k_dt(Geo g, DevScalars *sc) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double u1m = __longlong_as_double((long long)sc->u1m);
  const double u3m = __longlong_as_double((long long)sc->u3m);
  double u2m = __longlong_as_double((long long)sc->u2m);
  if (!(u2m > 1e-6)) u2m = (u2m != u2m) ? u2m : 1e-6;
  const double a = 1.0 / (g.alp * (double)(g.N1 / 2) * u1m);
  const double b = 1.0 / (g.bet * (double)(g.N2 / 2) * u3m);
  const double cv = 1.0 / (u2m * g.dthetavi);
  double d = fmin(a, b);
  d = fmin(d, cv);
  if (a != a || b != b || cv != cv) d = a + b + cv;  // propagate a NaN of any of the three maxima
  sc->dtc = d;
  const double lim = 2.5 * g.dtv, cfl = g.CFL * d;
  const double dt = (cfl != cfl) ? cfl : fmin(lim, cfl);
  sc->dt = dt;
  sc->dti = 1.0 / dt;
  sc->t = sc->t + dt;
  if (!(dt == dt)) sc->status = LH_ENONFINITE;  // the guard fires in the substep that forms dt
}

__global__ void k_reset_cfl(DevScalars *sc) {
  if (threadIdx.x == 0 && blockIdx.x == 0) { sc->u1m = 0ull; sc->u2m = 0ull; sc->u3m = 0ull; }
}

template <typename VN>
__device__ __forceinline__ double2 ld2(const VN &v) { return make_double2((double)v.x, (double)v.y); }

// cp.async copies from global to shared memory (16, 8 and 4 bytes), their commit groups and waits
__device__ __forceinline__ void cpa16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa8(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa4(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
// the same on a 32-bit shared address
__device__ __forceinline__ void cpa8s(unsigned dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa4s(unsigned dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ============================================================================
// Helmholtz solves of the FP64 form (RHS0 + N assembly + LU + both sweeps of one column
// segment). For interior q the right-hand side is u + dt * du with du = RHS0 (laplacian,
// -cRK Nu_old, -dRK grad p, -dRK mpgx on (0,0)) - gRK Nu_new, Nu_new = N_xz + d/dy(flux);
// Nu_new replaces Nu. The forward sweep stores y in the field and the upper factor in a3s; the
// backward sweep writes the solution in place. At immersed-boundary levels du is read from
// `duib` (assembled and forced beforehand) instead of being formed here.
//
// A lane carries a column segment's fields (u and w share their matrix; v) and both parts. The
// FP64 pipe (2 operations a clock and SM) bounds the kernel, so one lane does everything that
// shares the factorisation, and the operations are few: the row l of -dt / Re L serves the matrix
// (I + bRK l) and the right-hand side (-aRK l u), and dt is folded into the other coefficients.
// u/w 93 -> 66 and v 65 -> 42 operations a column level. The level's inputs come D levels ahead
// through a cp.async ring in shared memory. 32-thread blocks spread the columns evenly over the
// 152 SMs (1032 blocks at 256 x 256: 6.8 a SM). Small channels: k_helm_rhs and k_helm_sweep64.
// Measured at 256 x 256 x 301 with posts, ms per step, against one lane per column with all
// operations in the reference's order: u/w 5.63 -> 4.32, v 3.94 -> 2.89 (both run together in the
// step: FP64 pipe 82-86 % busy).
// ============================================================================
#define LH_H64_D 2   // levels ahead
#define LH_H64_T 32  // threads per block
__device__ __forceinline__ double &comp(double2 &v, int s) { return s ? v.y : v.x; }

struct Helm64Args {
  double *u[2];          // the fields (v: [0])
  double *Nu[2];         // previous nonlinear terms
  const double *X[2];    // N_xz
  const double *F[2];    // y-flux
  const double *p;
  double *a3s;           // upper factors [level][column]
  const int *ibslot;
  const double *duib;
  int kRK;
};
__host__ __device__ constexpr int helm64_entries(bool V) { return V ? 5 : 9; }
// bytes: the level tables (row of -dt / Re L without k^2, d/dy factor, immersed slot) and the ring
__host__ __device__ constexpr size_t helm64_smem(bool V, int nlev) {
  return (((size_t)nlev * 36 + 15) & ~(size_t)15) + (size_t)helm64_entries(V) * (LH_H64_D + 1) * LH_H64_T * 16;
}

// V: the wall-normal velocity (levels at the faces; gradient and flux differences across them)
template <bool V>
__global__ void __launch_bounds__(LH_H64_T) k_helm64(Helm64Args a, Geo g, const DevScalars *__restrict__ sc) {
  typedef double2 T;
  constexpr int NF = V ? 1 : 2, NP = 2;  // fields, parts
  constexpr int D = LH_H64_D, NS = D + 1, NT = LH_H64_T, NE = helm64_entries(V);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nlev = V ? g.nv : g.nu, kRK = a.kRK;
  double *t1 = reinterpret_cast<double *>(smem_raw), *t2 = t1 + nlev, *t3 = t2 + nlev, *tth = t3 + nlev;
  int *tib = reinterpret_cast<int *>(tth + nlev);
  T *ring = reinterpret_cast<T *>(smem_raw + (((size_t)nlev * 36 + 15) & ~(size_t)15));
  const double dt = sc->dt;
  const double unit = -dt / g.Re;  // the tables hold -dt / Re L
  {
    const double *d2 = V ? g.d2v : g.d2u, *th = V ? g.thv : g.thu;
    for (int i = threadIdx.x; i < nlev; i += NT) {
      t1[i] = unit * d2[i]; t2[i] = unit * d2[nlev + i]; t3[i] = unit * d2[2 * nlev + i];
      tth[i] = th[i] * g.dd;
      tib[i] = a.ibslot ? a.ibslot[i] : -1;
    }
  }
  __syncthreads();
  const int vc = blockIdx.x * NT + threadIdx.x;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int qlo = g.bq[bd][V ? 2 : 0], qhi = g.bq[bd][V ? 3 : 1];
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const double uk = unit * (g.k2x[kx] + g.k2z[r]);
  const double aR = g.aRK[kRK - 1], bR = g.bRK[kRK - 1];
  const double c2 = -dt * g.cRK[kRK - 1], cg = -dt * g.gRK[kRK - 1], cp = -dt * g.dRK[kRK - 1];
  const double mp = (!V && c == 0) ? cp * sc->mpgx : 0.0;  // u only, real part
  const double gw0 = V ? 0.0 : g.gw[bd][0], gw1 = V ? 0.0 : g.gw[bd][1];
  const size_t ls = (size_t)nc * 2, ci = (size_t)c * 2;
  double *u[NF], *No[NF];
  const double *X[NF], *F[NF];
  double ck[NF];  // -dt dRK k of the field's gradient
  int fd[NF];     // field in duib
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    u[f] = a.u[f] + ci; No[f] = a.Nu[f] + ci;
    X[f] = a.X[f] + ci; F[f] = a.F[f] + ci;
    ck[f] = V ? 0.0 : cp * (f ? g.k1z[r] : g.k1x[kx]);
    fd[f] = V ? 1 : 2 * f;
  }
  double *a3 = a.a3s + c;
#define RS(s_, k_) ring[((s_) * NE + (k_)) * NT + threadIdx.x]
  // slot of level q: the fields one level up, p, Nu, X, flux (v: v one level up, p at q, Nu, X, vv one up)
  auto fetch = [&](int q) {
    const int s_ = (q - qlo - 1) % NS;
    const size_t o = (size_t)q * ls;
    if (V) {
      cpa16(&RS(s_, 0), u[0] + o + ls); cpa16(&RS(s_, 1), a.p + o + ci);
      cpa16(&RS(s_, 2), No[0] + o); cpa16(&RS(s_, 3), X[0] + o); cpa16(&RS(s_, 4), F[0] + o + ls);
    } else {
      cpa16(&RS(s_, 0), a.p + o - ls + ci);
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        cpa16(&RS(s_, 1 + 4 * f), u[f] + o + ls); cpa16(&RS(s_, 2 + 4 * f), No[f] + o);
        cpa16(&RS(s_, 3 + 4 * f), X[f] + o); cpa16(&RS(s_, 4 + 4 * f), F[f] + o);
      }
    }
  };
  T um[NF], u0[NF], fl[NF], y[NF], pm;
  const size_t e0 = (size_t)qlo * ls;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    um[f] = *reinterpret_cast<const T *>(u[f] + e0);
    u0[f] = *reinterpret_cast<const T *>(u[f] + e0 + ls);
    fl[f] = *reinterpret_cast<const T *>(F[f] + e0 + (V ? ls : 0));
  }
  if (V) pm = *reinterpret_cast<const T *>(a.p + e0 + ci);
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    if (qlo + 1 + s_ <= qhi - 1) fetch(qlo + 1 + s_);
    cpa_commit();
  }
  double a3raw = gw0, a2p = 1.0;  // first row: [1, gw(b,1)], rhs 0
#pragma unroll
  for (int f = 0; f < NF; ++f) {
#pragma unroll
    for (int s = 0; s < NP; ++s) comp(y[f], s) = 0.0;
    *reinterpret_cast<T *>(u[f] + e0) = y[f];
  }
  for (int q = qlo + 1; q <= qhi - 1; ++q) {
    cpa_wait<D - 1>();
    const int s_ = (q - qlo - 1) % NS;
    T w[NE];
#pragma unroll
    for (int k = 0; k < NE; ++k) w[k] = RS(s_, k);
    if (q + D <= qhi - 1) fetch(q + D);
    cpa_commit();
    const double l1 = t1[q], l2 = t2[q] + uk, l3 = t3[q], th = tth[q], a1 = bR * l1;
    const int ibs = tib[q];
    const double a3p = a3raw * a2p;
    a3[(size_t)(q - 1) * nc] = a3p;
    a2p = 1.0 / ((1.0 + bR * l2) - a1 * a3p);
    const size_t o = (size_t)q * ls;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      T &up = w[V ? 0 : 1 + 4 * f];
      T rhs;
      if (ibs < 0) {
        T &no = w[2 + 4 * f], &x = w[3 + 4 * f], &fq = w[4 + 4 * f];
        T n;
#pragma unroll
        for (int s = 0; s < NP; ++s) {
          const double t = l1 * comp(um[f], s) + (l2 * comp(u0[f], s) + l3 * comp(up, s));
          const double nn = comp(x, s) + (comp(fq, s) - comp(fl[f], s)) * th;
          comp(n, s) = nn;
          double v = c2 * comp(no, s) - aR * t;  // the increment first: u's rounding enters once
          v += cg * nn;
          if (V) {
            v += (cp * th) * (comp(w[1], s) - comp(pm, s));
          } else {  // i k p: the other part, with its sign
            v += (s ? ck[f] : -ck[f]) * comp(w[0], s ^ 1);
            if (f == 0 && s == 0) v += mp;
          }
          comp(rhs, s) = comp(u0[f], s) + v;
        }
        *reinterpret_cast<T *>(No[f] + o) = n;
      } else {
        T di = *reinterpret_cast<const T *>(a.duib + ((size_t)ibs * 3 + fd[f]) * ls + ci);
#pragma unroll
        for (int s = 0; s < NP; ++s) comp(rhs, s) = comp(u0[f], s) + dt * comp(di, s);
      }
#pragma unroll
      for (int s = 0; s < NP; ++s) comp(y[f], s) = (comp(rhs, s) - a1 * comp(y[f], s)) * a2p;
      *reinterpret_cast<T *>(u[f] + o) = y[f];
      um[f] = u0[f]; u0[f] = up; fl[f] = w[4 + 4 * f];
    }
    if (V) pm = w[1];
    a3raw = bR * l3;
  }
  cpa_wait<0>();
  {  // last row: [gw(b,2), 1], rhs 0
    const double a3p = a3raw * a2p;
    a3[(size_t)(qhi - 1) * nc] = a3p;
    a2p = 1.0 / (1.0 - gw1 * a3p);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
#pragma unroll
      for (int s = 0; s < NP; ++s) comp(y[f], s) = (0.0 - gw1 * comp(y[f], s)) * a2p;
      *reinterpret_cast<T *>(u[f] + (size_t)qhi * ls) = y[f];
    }
  }
  __threadfence();  // the copies below read what this thread stored above
  double *ra = reinterpret_cast<double *>(ring + (size_t)NF * NS * NT);  // factors beside the fields' slots
  auto fetch_b = [&](int q) {
    const int s_ = (qhi - 1 - q) % NS;
#pragma unroll
    for (int f = 0; f < NF; ++f) cpa16(&ring[(s_ * NF + f) * NT + threadIdx.x], u[f] + (size_t)q * ls);
    cpa8(&ra[s_ * NT + threadIdx.x], a3 + (size_t)q * nc);
  };
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    if (qhi - 1 - s_ >= qlo) fetch_b(qhi - 1 - s_);
    cpa_commit();
  }
  for (int q = qhi - 1; q >= qlo; --q) {
    cpa_wait<D - 1>();
    const int s_ = (qhi - 1 - q) % NS;
    T yy[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) yy[f] = ring[(s_ * NF + f) * NT + threadIdx.x];
    const double a3p = ra[s_ * NT + threadIdx.x];
    if (q - D >= qlo) fetch_b(q - D);
    cpa_commit();
#pragma unroll
    for (int f = 0; f < NF; ++f) {
#pragma unroll
      for (int s = 0; s < NP; ++s) comp(y[f], s) = comp(yy[f], s) - a3p * comp(y[f], s);
      *reinterpret_cast<T *>(u[f] + (size_t)q * ls) = y[f];
    }
  }
  cpa_wait<0>();
#undef RS
}

// ============================================================================
// Mixed form of the Helmholtz solves: the same equations written for the
// increment d = u_new - u, (I - beta L) d = dt du + beta L(u), with the BC rows
// d(0) + gw1 d(1) = -(u(0) + gw1 u(1)) (and the top row alike). d is small, so
// the right-hand side, the factorisation and both sweeps run in FP32; L(u) is
// formed from FP64 neighbour differences (u(j+-1) - u(j)); u_new = u + d in FP64.
// ============================================================================
__device__ __forceinline__ float2 f2d(double2 a) { return make_float2((float)a.x, (float)a.y); }
__device__ __forceinline__ float2 f2sub(double2 a, double2 b) { return make_float2((float)(a.x - b.x), (float)(a.y - b.y)); }

// Backward sweep of the mixed-form solves: x(q) = y(q) - a3'(q) x(q+1), u(q) += x(q) for
// q = qhi-1 .. qlo, with ys(q) = (y(q), a3'(q)). The loads of level q are issued
// D levels ahead, before the stores of the levels in between (D = 0: a plain loop).
template <int D>
__device__ __forceinline__ void back_sweep_mx(double *__restrict__ u, const float2 *__restrict__ ys, size_t lstride,
                                              size_t ci, int qlo, int qhi, float x) {
  if constexpr (D == 0) {
#pragma unroll 4
    for (int q = qhi - 1; q >= qlo; --q) {
      const size_t e = (size_t)q * lstride + ci;
      const float2 ya = ys[e];
      x = ya.x - ya.y * x;
      u[e] = u[e] + f2d_alu(x);
    }
    return;
  } else {
  float2 bys[D];
  double bu[D];
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    const int q = qhi - 1 - s_;
    if (q >= qlo) { const size_t e = (size_t)q * lstride + ci; bys[s_] = ys[e]; bu[s_] = u[e]; }
  }
  for (int qb = qhi - 1; qb >= qlo; qb -= D) {
#pragma unroll
    for (int s_ = 0; s_ < D; ++s_) {
      const int q = qb - s_;
      if (q < qlo) break;
      const float2 ya = bys[s_];
      const double uq = bu[s_];
      if (q - D >= qlo) { const size_t en = (size_t)(q - D) * lstride + ci; bys[s_] = ys[en]; bu[s_] = u[en]; }
      x = ya.x - ya.y * x;
      u[(size_t)q * lstride + ci] = uq + f2d_alu(x);
    }
  }
  }
}

// ============================================================================
// Mode (0,0) of the mixed form in FP64. The mean flow and its -dRK mpgx forcing live in
// column 0, so its Helmholtz systems are solved in FP64 as the plain form solves them
// (LUsolU_W / LUsolV, tridLU_3D.f90:55-189, right-hand sides of RHS0_u1/u2/u3,
// littleharsh.f90:635-788): FP64 right-hand side, FP64 solve, the column's previous
// nonlinear term kept in FP64. Only the transforms' products (X, Fl) are the form's FP32
// values. k = 0, so there are no i*k couplings and the real and imaginary parts are six
// independent real systems (u, w, v x 2 parts): one block each, rows built in parallel and
// solved by parallel cyclic reduction (log2(levels) steps) so that the column costs a few
// microseconds instead of a serial FP64 recurrence over the levels. The mixed solve
// kernels skip column 0.
// Scalar views as the mixed kernels': element (q, col, part) at (q*ncol + col)*2 + part.
// nuo: the previous nonlinear term of the column, [u re, u im, w re, w im, v re, v im][nu].
// Shared memory: 8 (nu + 1) doubles.
// ============================================================================
__device__ __forceinline__ int fw2f(int fw) { return fw == 0 ? 0 : (fw == 1 ? 2 : 1); }
__global__ void __launch_bounds__(512) k_helm00_pcr(double *__restrict__ u1, double *__restrict__ u3,
                                                    double *__restrict__ u2, const float *__restrict__ N1xz,
                                                    const float *__restrict__ N3xz, const float *__restrict__ N2xz,
                                                    const float *__restrict__ uvf, const float *__restrict__ wvf,
                                                    const float *__restrict__ vvc, const double *__restrict__ p,
                                                    const float2 *__restrict__ duib, const int *__restrict__ ibslot_u,
                                                    const int *__restrict__ ibslot_v, Geo g,
                                                    const DevScalars *__restrict__ sc, int kRK,
                                                    double *__restrict__ nuo_all) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int fw = blockIdx.x >> 1, part = blockIdx.x & 1;  // fw 0: u, 1: w, 2: v
  const bool isv = fw == 2;
  const int qlo = isv ? g.bq[1][2] : g.bq[1][0], qhi = isv ? g.bq[1][3] : g.bq[1][1];
  const int n = qhi - qlo + 1, ny = isv ? g.nv : g.nu;
  double *A = reinterpret_cast<double *>(smem_raw), *B = A + n, *Cc = B + n, *D = Cc + n;
  double *A2 = D + n, *B2 = A2 + n, *C2b = B2 + n, *D2 = C2b + n;
  const size_t ls = (size_t)g.ncol * 2;
  double *u = fw == 0 ? u1 : (fw == 1 ? u3 : u2);
  const float *X = fw == 0 ? N1xz : (fw == 1 ? N3xz : N2xz);
  const float *Fl = fw == 0 ? uvf : (fw == 1 ? wvf : vvc);
  const int *ibslot = isv ? ibslot_v : ibslot_u;
  double *nuo = nuo_all + (size_t)blockIdx.x * g.nu;
  const double *d2 = isv ? g.d2v : g.d2u;
  const double dt = sc->dt;
  const double C1 = g.aRK[kRK - 1] / g.Re, C2 = -g.cRK[kRK - 1], dR = g.dRK[kRK - 1], G = -g.gRK[kRK - 1];
  const double beta = g.bRK[kRK - 1] * dt / g.Re;
  const double mp = (fw == 0 && part == 0) ? -dR * sc->mpgx : 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int q = qlo + i;
    double a, b, c, d;
    if (q == qlo || q == qhi) {  // boundary rows: [1, gw(b,1)] / [gw(b,2), 1] (u, w); v = 0 (v)
      a = 0.0; b = 1.0; c = 0.0; d = 0.0;
      if (!isv) { if (q == qlo) c = g.gw[1][0]; else a = g.gw[1][1]; }
    } else {
      const size_t e = q * ls + part;
      const double um = u[e - ls], u0 = u[e], up = u[e + ls];
      const double d0q = d2[q], d1q = d2[ny + q], d2q = d2[2 * ny + q];
      const int ibs = ibslot ? ibslot[q] : -1;
      double du;
      if (ibs < 0) {
        const double L = (d0q * um + d1q * u0) + d2q * up;
        double nq, rest;
        if (!isv) {
          nq = (double)X[e] + ((double)Fl[e] - (double)Fl[e - ls]) * g.thu[q] * g.dd;
          rest = mp;
        } else {
          nq = (double)X[e] + ((double)Fl[e + ls] - (double)Fl[e]) * g.thv[q] * g.dd;
          rest = (-dR * g.dd * g.thv[q]) * (p[e] - p[e - ls]);
        }
        du = ((C1 * L + C2 * nuo[q]) + rest) + G * nq;
        nuo[q] = nq;
      } else {
        const float2 di = duib[((size_t)ibs * 3 + fw2f(fw)) * g.ncol];
        du = f2d_alu(part ? di.y : di.x);
      }
      a = -beta * d0q; b = 1.0 - beta * d1q; c = -beta * d2q;
      d = u0 + dt * du;
    }
    A[i] = a; B[i] = b; Cc[i] = c; D[i] = d;
  }
  __syncthreads();
  for (int st = 1; st < n; st *= 2) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int im = i - st, ip = i + st;
      double a = 0.0, b = B[i], c = 0.0, d = D[i];
      if (im >= 0) {
        const double al = -A[i] / B[im];
        a = al * A[im];
        b += al * Cc[im];
        d += al * D[im];
      }
      if (ip < n) {
        const double ga = -Cc[i] / B[ip];
        c = ga * Cc[ip];
        b += ga * A[ip];
        d += ga * D[ip];
      }
      A2[i] = a; B2[i] = b; C2b[i] = c; D2[i] = d;
    }
    __syncthreads();
    double *t;
    t = A; A = A2; A2 = t;
    t = B; B = B2; B2 = t;
    t = Cc; Cc = C2b; C2b = t;
    t = D; D = D2; D2 = t;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) u[(qlo + i) * ls + part] = D[i] / B[i];
}


// ============================================================================
// The sums of products of a level, for every kernel that solves for the mixed form. Which product of
// a b + c d is rounded would be the compiler's choice, and it chose otherwise in one of the kernels
// (k_helm_v_mx2: 1 value in 300 off by a rounding); written out, all give the same bits.
__device__ __forceinline__ float mx_lap(float a, float fdm, float c, float fdp, float sdg, float u) {
  return __fmaf_rn(sdg, u, __fmaf_rn(a, fdm, __fmul_rn(c, fdp)));
}
__device__ __forceinline__ float mx_du(float C1, float L, float C2, float nu, float C3, float pt) {
  return __fmaf_rn(C3, pt, __fmaf_rn(C1, L, __fmul_rn(C2, nu)));
}
__device__ __forceinline__ float mx_rhs(float beta, float L, float dt, float du) { return __fmaf_rn(beta, L, __fmul_rn(dt, du)); }

// ============================================================================
// Mixed-form solves with one lane per (column, real/imaginary part): the matrix
// is real, so the two parts are independent systems; each lane repeats the FP32
// factorisation. Scalar views: element (q, col, part) at (q*ncol + col)*2 + part.
// ys2 holds (y(q), upper factor(q)) per lane.
// k_helm_u_mx2: one field (u when F == 0, w when F == 2) per launch row (blockIdx.y).
// ============================================================================
__global__ void __launch_bounds__(NTHR) k_helm_u_mx2(double *__restrict__ u1, double *__restrict__ u3,
                                                     float *__restrict__ Nu1, float *__restrict__ Nu3,
                                                     const float *__restrict__ N1xz, const float *__restrict__ N3xz,
                                                     const float *__restrict__ uvf, const float *__restrict__ wvf,
                                                     const double2 *__restrict__ p, float2 *__restrict__ ys2, Geo g,
                                                     const DevScalars *__restrict__ sc, int kRK,
                                                     const int *__restrict__ ibslot_u, const float2 *__restrict__ duib) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int qlo = g.bq[bd][0], qhi = g.bq[bd][1];
  const int fw = blockIdx.y;  // 0: u, 1: w
  double *u = fw ? u3 : u1;
  float *Nu = fw ? Nu3 : Nu1;
  const float *X = fw ? N3xz : N1xz;
  const float *Fl = fw ? wvf : uvf;
  if (c == 0) return;  // mode (0,0): k_helm00_pcr (FP64)
  float2 *ys = ys2 + (size_t)fw * g.nu * nc * 2;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float G = (float)(-g.gRK[kRK - 1]);
  const double dt = sc->dt;
  const float dtf = (float)dt;
  const float beta = (float)(g.bRK[kRK - 1] * dt / g.Re);
  const float C3 = (float)(-dR * (fw ? g.k1z[r] : g.k1x[kx]));
  const float dd = (float)g.dd;
  const int nu = g.nu;
  const double gw1 = g.gw[bd][0], gw2 = g.gw[bd][1];
  const size_t lstride = (size_t)nc * 2;
  const size_t ci = (size_t)c * 2 + part;
  const size_t e0 = (size_t)qlo * lstride + ci;
  double um = u[e0], u0 = u[e0 + lstride];
  float y = d2f_alu(-(um + gw1 * u0));  // first row
  // um - u0 at level q is -(up1 - u0) of level q-1: one FP64 difference per level
  float fdm = d2f_alu(um - u0);
  float yprev = y;
  float a3raw = (float)gw1, a2p = 1.f;
  float flm = Fl[e0];
  // the inputs of level q are loaded LH_PF_HU levels ahead of their use, before the
  // stores of the levels in between (the sweep's own stores would otherwise order them)
#if LH_PF_HU > 0
  constexpr int D = LH_PF_HU;
  double fu[D];
  float ffl[D], fa[D], fb[D], fc[D], fsd[D], fth[D], fnu[D], fx[D];
  int fib[D];
  double fp[D];                       // the other part of p: i*C3*p = (-C3 p.y, C3 p.x)
  const double *pc = reinterpret_cast<const double *>(p);
#define HU_FETCH(s_, qq_)                                                        \
  {                                                                              \
    const int q_ = (qq_);                                                        \
    const size_t e_ = (size_t)q_ * lstride + ci;                                 \
    fu[s_] = u[e_ + lstride];                                                    \
    ffl[s_] = Fl[e_];                                                            \
    fa[s_] = g.d2uf[q_]; fb[s_] = g.d2uf[nu + q_]; fc[s_] = g.d2uf[2 * nu + q_]; \
    fsd[s_] = g.sdgu[q_]; fth[s_] = g.thuf[q_];                                  \
    fib[s_] = ibslot_u ? ibslot_u[q_] : -1;                                      \
    fp[s_] = pc[((size_t)(q_ - 1) * nc + c) * 2 + (part ^ 1)];                   \
    fnu[s_] = Nu[e_]; fx[s_] = X[e_];                                            \
  }
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_)
    if (qlo + 1 + s_ <= qhi - 1) HU_FETCH(s_, qlo + 1 + s_)
  for (int qb = qlo + 1; qb <= qhi - 1; qb += D) {
#pragma unroll
    for (int s_ = 0; s_ < D; ++s_) {
      const int q = qb + s_;
      if (q > qhi - 1) break;
      const size_t e = (size_t)q * lstride + ci;
      const double up1 = fu[s_];
      const float flq = ffl[s_], a = fa[s_], b = fb[s_], cc = fc[s_], sdg = fsd[s_] + k2f, thq = fth[s_];
      const float nuq = fnu[s_], xq = fx[s_];
      const int ibs = fib[s_];
      const double po = fp[s_];
      if (q + D <= qhi - 1) HU_FETCH(s_, q + D)
      const float fdp = d2f_alu(up1 - u0);
      const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(u0));
      fdm = -fdp;
      float du;
      if (ibs < 0) {
        const float pt = part ? d2f_alu(po) : -d2f_alu(po);
        du = mx_du(C1, L, C2, nuq, C3, pt);
        const float n = xq + (flq - flm) * thq * dd;
        Nu[e] = n;
        du += G * n;
      } else {
        const float2 di = duib[((size_t)ibs * 3 + (fw ? 2 : 0)) * nc + c];
        du = part ? di.y : di.x;
      }
      const float rr = mx_rhs(beta, L, dtf, du);
      const float a1 = -beta * a;
      const float a2 = 1.f - beta * (b + k2f);
      const float a3p = a3raw * a2p;
      ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
      a2p = 1.f / (a2 - a1 * a3p);
      y = (rr - a1 * y) * a2p;
      yprev = y;
      a3raw = -beta * cc;
      um = u0; u0 = up1;
      flm = flq;
    }
  }
#undef HU_FETCH
#else
#pragma unroll 4
  for (int q = qlo + 1; q <= qhi - 1; ++q) {
    const size_t e = (size_t)q * lstride + ci;
    const double up1 = u[e + lstride];
    const float flq = Fl[e];
    const float a = g.d2uf[q], b = g.d2uf[nu + q], cc = g.d2uf[2 * nu + q];
    const float sdg = g.sdgu[q] + k2f;
    const float fdp = d2f_alu(up1 - u0);
    const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(u0));
    fdm = -fdp;
    float du;
    const int ibs = ibslot_u ? ibslot_u[q] : -1;
    if (ibs < 0) {
      const double2 pj = p[(size_t)(q - 1) * nc + c];
      const float pt = part ? d2f_alu(pj.x) : -d2f_alu(pj.y);  // i*C3*p: (-C3 p.y, C3 p.x)
      du = mx_du(C1, L, C2, Nu[e], C3, pt);
      const float n = X[e] + (flq - flm) * g.thuf[q] * dd;
      Nu[e] = n;
      du += G * n;
    } else {
      const float2 di = duib[((size_t)ibs * 3 + (fw ? 2 : 0)) * nc + c];
      du = part ? di.y : di.x;
    }
    const float rr = mx_rhs(beta, L, dtf, du);
    const float a1 = -beta * a;
    const float a2 = 1.f - beta * (b + k2f);
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    a2p = 1.f / (a2 - a1 * a3p);
    y = (rr - a1 * y) * a2p;
    yprev = y;
    a3raw = -beta * cc;
    um = u0; u0 = up1;
    flm = flq;
  }
#endif
  {  // last row: gw2 d(n-2) + d(n-1) = -(gw2 u(n-2) + u(n-1))
    const int q = qhi;
    const float a1 = (float)gw2;
    const float rl = d2f_alu(-(gw2 * um + u0));
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    a2p = 1.f / (1.f - a1 * a3p);
    y = (rl - a1 * y) * a2p;
    u[(size_t)q * lstride + ci] = u0 + f2d_alu(y);
  }
  back_sweep_mx<LH_PF_HU_BACK>(u, ys, lstride, ci, qlo, qhi, y);
}

__global__ void __launch_bounds__(NTHR) k_helm_v_mx2(double *__restrict__ u2, float *__restrict__ Nu2,
                                                     const float *__restrict__ N2xz, const float *__restrict__ vvc,
                                                     const double *__restrict__ p, float2 *__restrict__ ys, Geo g,
                                                     const DevScalars *__restrict__ sc, int kRK,
                                                     const int *__restrict__ ibslot_v, const float2 *__restrict__ duib) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  if (c == 0) return;  // mode (0,0): k_helm00_pcr (FP64)
  const int qlo = g.bq[bd][2], qhi = g.bq[bd][3];
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float G = (float)(-g.gRK[kRK - 1]);
  const double dt = sc->dt;
  const float dtf = (float)dt;
  const float beta = (float)(g.bRK[kRK - 1] * dt / g.Re);
  const float dd = (float)g.dd;
  const int nv = g.nv;
  const size_t ci = (size_t)c * 2 + part;
  const size_t lstride = (size_t)nc * 2;
  const size_t e0 = (size_t)qlo * lstride + ci;
  double vm = u2[e0], v0 = u2[e0 + lstride];
  const float dRf = (float)dR;
  float y = d2f_alu(-vm);
  float fdm = d2f_alu(vm - v0);  // carried as -(vp1 - v0) of the level below
  float yprev = y;
  float a3raw = 0.f, a2p = 1.f;
  float vvq = vvc[e0 + lstride];
  constexpr int D = LH_PF_HV > 0 ? LH_PF_HV : 1;
  double fv[D];
  float fvv[D], fa[D], fb[D], fc[D], fsd[D], fth[D], fnu[D], fx[D], fpd[D];
  int fib[D];
#define HV_FETCH(s_, qq_)                                                        \
  {                                                                              \
    const int q_ = (qq_);                                                        \
    const size_t e_ = (size_t)q_ * lstride + ci;                                 \
    fv[s_] = u2[e_ + lstride];                                                   \
    fvv[s_] = vvc[e_ + lstride];                                                 \
    fa[s_] = g.d2vf[q_]; fb[s_] = g.d2vf[nv + q_]; fc[s_] = g.d2vf[2 * nv + q_]; \
    fsd[s_] = g.sdgv[q_]; fth[s_] = g.thvf[q_];                                  \
    fib[s_] = ibslot_v ? ibslot_v[q_] : -1;                                      \
    fpd[s_] = d2f_alu(p[e_]) - d2f_alu(p[e_ - lstride]);                         \
    fnu[s_] = Nu2[e_]; fx[s_] = N2xz[e_];                                        \
  }
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_)
    if (qlo + 1 + s_ <= qhi - 1) HV_FETCH(s_, qlo + 1 + s_)
  for (int qb = qlo + 1; qb <= qhi - 1; qb += D) {
#pragma unroll
    for (int s_ = 0; s_ < D; ++s_) {
      const int q = qb + s_;
      if (q > qhi - 1) break;
      const size_t e = (size_t)q * lstride + ci;
      const double vp1 = fv[s_];
      const float vvp = fvv[s_], a = fa[s_], b = fb[s_], cc = fc[s_], sdg = fsd[s_] + k2f, thq = fth[s_];
      const float nuq = fnu[s_], xq = fx[s_], pd = fpd[s_];
      const int ibs = fib[s_];
      if (q + D <= qhi - 1) HV_FETCH(s_, q + D)
      const float fdp = d2f_alu(vp1 - v0);
      const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(v0));
      fdm = -fdp;
      float du;
      if (ibs < 0) {
        const float C3 = -dRf * dd * thq;
        du = mx_du(C1, L, C2, nuq, C3, pd);
        const float n = xq + (vvp - vvq) * thq * dd;
        Nu2[e] = n;
        du += G * n;
      } else {
        const float2 di = duib[((size_t)ibs * 3 + 1) * nc + c];
        du = part ? di.y : di.x;
      }
      const float rr = mx_rhs(beta, L, dtf, du);
      const float a1 = -beta * a;
      const float a2 = 1.f - beta * (b + k2f);
      const float a3p = a3raw * a2p;
      ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
      a2p = 1.f / (a2 - a1 * a3p);
      y = (rr - a1 * y) * a2p;
      yprev = y;
      a3raw = -beta * cc;
      vm = v0; v0 = vp1; vvq = vvp;
    }
  }
#undef HV_FETCH
  {  // last row: d(n-1) = -v(n-1)
    const int q = qhi;
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    y = d2f_alu(-v0);
    u2[(size_t)q * lstride + ci] = v0 + f2d_alu(y);
  }
  back_sweep_mx<LH_PF_HV_BACK>(u2, ys, lstride, ci, qlo, qhi, y);
}

// ============================================================================
// The mixed-form solves with their y-columns staged through shared memory (the arithmetic of
// k_helm_u_mx2 / k_helm_v_mx2, so the same results bit for bit): every lane keeps a ring of
// D + 1 levels of its inputs, filled by cp.async copies D levels ahead (into the slot not being
// read), and the per-level coefficient tables sit in shared memory; the backward sweep stages
// (y, upper factor) and the state the same way. Shared memory: 6 nu tables + the ring,
// 24 (D + 1) bytes per thread.
// ============================================================================
template <int D>
__device__ __forceinline__ void back_sweep_staged(double *__restrict__ u, const float2 *__restrict__ ys, size_t lstride,
                                                  size_t ci, int qlo, int qhi, float x, unsigned char *ring, int nt) {
  constexpr int NS = D + 1;
  float2 *ry = reinterpret_cast<float2 *>(ring);          // [NS][nt]
  double *ru = reinterpret_cast<double *>(ring) + NS * nt;  // [NS][nt]
  auto fetch = [&](int q) {
    const int s_ = (qhi - 1 - q) % NS;
    const size_t e = (size_t)q * lstride + ci;
    cpa8(&ry[s_ * nt + threadIdx.x], ys + e);
    cpa8(&ru[s_ * nt + threadIdx.x], u + e);
  };
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    if (qhi - 1 - s_ >= qlo) fetch(qhi - 1 - s_);
    cpa_commit();
  }
  for (int q = qhi - 1; q >= qlo; --q) {
    cpa_wait<D - 1>();
    const int s_ = (qhi - 1 - q) % NS;
    const float2 ya = ry[s_ * nt + threadIdx.x];
    const double uq = ru[s_ * nt + threadIdx.x];
    if (q - D >= qlo) fetch(q - D);
    cpa_commit();
    x = ya.x - ya.y * x;
    u[(size_t)q * lstride + ci] = uq + f2d_alu(x);
  }
  cpa_wait<0>();
}

template <int D>
__global__ void __launch_bounds__(NTHR) k_helm_u_mx3(double *__restrict__ u1, double *__restrict__ u3,
                                                     float *__restrict__ Nu1, float *__restrict__ Nu3,
                                                     const float *__restrict__ N1xz, const float *__restrict__ N3xz,
                                                     const float *__restrict__ uvf, const float *__restrict__ wvf,
                                                     const double2 *__restrict__ p, float2 *__restrict__ ys2, Geo g,
                                                     const DevScalars *__restrict__ sc, int kRK,
                                                     const int *__restrict__ ibslot_u, const float2 *__restrict__ duib) {
  constexpr int NS = D + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nu = g.nu, nt = blockDim.x;
  float *ta = reinterpret_cast<float *>(smem_raw), *tb = ta + nu, *tc = tb + nu, *tsd = tc + nu, *tth = tsd + nu;
  int *tib = reinterpret_cast<int *>(tth + nu);
  unsigned char *ring = smem_raw + (((size_t)6 * nu * 4 + 15) & ~(size_t)15);
  for (int i = threadIdx.x; i < nu; i += nt) {
    ta[i] = g.d2uf[i]; tb[i] = g.d2uf[nu + i]; tc[i] = g.d2uf[2 * nu + i]; tsd[i] = g.sdgu[i]; tth[i] = g.thuf[i];
    tib[i] = ibslot_u ? ibslot_u[i] : -1;
  }
  __syncthreads();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  if (c == 0) return;  // mode (0,0): k_helm00_pcr (FP64)
  const int qlo = g.bq[bd][0], qhi = g.bq[bd][1];
  const int fw = blockIdx.y;  // 0: u, 1: w
  double *u = fw ? u3 : u1;
  float *Nu = fw ? Nu3 : Nu1;
  const float *X = fw ? N3xz : N1xz;
  const float *Fl = fw ? wvf : uvf;
  float2 *ys = ys2 + (size_t)fw * g.nu * nc * 2;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float G = (float)(-g.gRK[kRK - 1]);
  const double dt = sc->dt;
  const float dtf = (float)dt;
  const float beta = (float)(g.bRK[kRK - 1] * dt / g.Re);
  const float C3 = (float)(-dR * (fw ? g.k1z[r] : g.k1x[kx]));
  const float dd = (float)g.dd;
  const double gw1 = g.gw[bd][0], gw2 = g.gw[bd][1];
  const size_t lstride = (size_t)nc * 2;
  const size_t ci = (size_t)c * 2 + part;
  const size_t e0 = (size_t)qlo * lstride + ci;
  const double *pc = reinterpret_cast<const double *>(p);
  double um = u[e0], u0 = u[e0 + lstride];
  float y = d2f_alu(-(um + gw1 * u0));  // first row
  float fdm = d2f_alu(um - u0);
  float yprev = y;
  float a3raw = (float)gw1, a2p = 1.f;
  float flm = Fl[e0];
  // ring: doubles [NS][2][nt] (u of the level above, p of the other part), floats [NS][3][nt] (Fl, Nu, X)
  double *rd = reinterpret_cast<double *>(ring);
  float *rf = reinterpret_cast<float *>(rd + 2 * NS * nt);
  auto fetch = [&](int q) {
    const int s_ = (q - qlo - 1) % NS;
    const size_t e = (size_t)q * lstride + ci;
    cpa8(&rd[(s_ * 2 + 0) * nt + threadIdx.x], u + e + lstride);
    cpa8(&rd[(s_ * 2 + 1) * nt + threadIdx.x], pc + ((size_t)(q - 1) * nc + c) * 2 + (part ^ 1));
    cpa4(&rf[(s_ * 3 + 0) * nt + threadIdx.x], Fl + e);
    cpa4(&rf[(s_ * 3 + 1) * nt + threadIdx.x], Nu + e);
    cpa4(&rf[(s_ * 3 + 2) * nt + threadIdx.x], X + e);
  };
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    if (qlo + 1 + s_ <= qhi - 1) fetch(qlo + 1 + s_);
    cpa_commit();
  }
  for (int q = qlo + 1; q <= qhi - 1; ++q) {
    cpa_wait<D - 1>();
    const int s_ = (q - qlo - 1) % NS;
    const size_t e = (size_t)q * lstride + ci;
    const double up1 = rd[(s_ * 2 + 0) * nt + threadIdx.x], po = rd[(s_ * 2 + 1) * nt + threadIdx.x];
    const float flq = rf[(s_ * 3 + 0) * nt + threadIdx.x], nuq = rf[(s_ * 3 + 1) * nt + threadIdx.x],
                xq = rf[(s_ * 3 + 2) * nt + threadIdx.x];
    if (q + D <= qhi - 1) fetch(q + D);
    cpa_commit();
    const float a = ta[q], b = tb[q], cc = tc[q], sdg = tsd[q] + k2f, thq = tth[q];
    const int ibs = tib[q];
    const float fdp = d2f_alu(up1 - u0);
    const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(u0));
    fdm = -fdp;
    float du;
    if (ibs < 0) {
      const float pt = part ? d2f_alu(po) : -d2f_alu(po);
      du = mx_du(C1, L, C2, nuq, C3, pt);
      const float n = xq + (flq - flm) * thq * dd;
      Nu[e] = n;
      du += G * n;
    } else {
      const float2 di = duib[((size_t)ibs * 3 + (fw ? 2 : 0)) * nc + c];
      du = part ? di.y : di.x;
    }
    const float rr = mx_rhs(beta, L, dtf, du);
    const float a1 = -beta * a;
    const float a2 = 1.f - beta * (b + k2f);
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    a2p = 1.f / (a2 - a1 * a3p);
    y = (rr - a1 * y) * a2p;
    yprev = y;
    a3raw = -beta * cc;
    um = u0; u0 = up1;
    flm = flq;
  }
  cpa_wait<0>();
  {  // last row: gw2 d(n-2) + d(n-1) = -(gw2 u(n-2) + u(n-1))
    const int q = qhi;
    const float a1 = (float)gw2;
    const float rl = d2f_alu(-(gw2 * um + u0));
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    a2p = 1.f / (1.f - a1 * a3p);
    y = (rl - a1 * y) * a2p;
    u[(size_t)q * lstride + ci] = u0 + f2d_alu(y);
  }
  __threadfence_block();  // the backward sweep's copies read ys written above by this thread
  back_sweep_staged<D>(u, ys, lstride, ci, qlo, qhi, y, ring, nt);
}

template <int D>
__global__ void __launch_bounds__(NTHR) k_helm_v_mx3(double *__restrict__ u2, float *__restrict__ Nu2,
                                                     const float *__restrict__ N2xz, const float *__restrict__ vvc,
                                                     const double *__restrict__ p, float2 *__restrict__ ys, Geo g,
                                                     const DevScalars *__restrict__ sc, int kRK,
                                                     const int *__restrict__ ibslot_v, const float2 *__restrict__ duib) {
  constexpr int NS = D + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nv = g.nv, nt = blockDim.x;
  float *ta = reinterpret_cast<float *>(smem_raw), *tb = ta + nv, *tc = tb + nv, *tsd = tc + nv, *tth = tsd + nv;
  int *tib = reinterpret_cast<int *>(tth + nv);
  unsigned char *ring = smem_raw + (((size_t)6 * nv * 4 + 15) & ~(size_t)15);
  for (int i = threadIdx.x; i < nv; i += nt) {
    ta[i] = g.d2vf[i]; tb[i] = g.d2vf[nv + i]; tc[i] = g.d2vf[2 * nv + i]; tsd[i] = g.sdgv[i]; tth[i] = g.thvf[i];
    tib[i] = ibslot_v ? ibslot_v[i] : -1;
  }
  __syncthreads();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  if (c == 0) return;  // mode (0,0): k_helm00_pcr (FP64)
  const int qlo = g.bq[bd][2], qhi = g.bq[bd][3];
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float G = (float)(-g.gRK[kRK - 1]);
  const double dt = sc->dt;
  const float dtf = (float)dt;
  const float beta = (float)(g.bRK[kRK - 1] * dt / g.Re);
  const float dd = (float)g.dd;
  const size_t ci = (size_t)c * 2 + part;
  const size_t lstride = (size_t)nc * 2;
  const size_t e0 = (size_t)qlo * lstride + ci;
  double vm = u2[e0], v0 = u2[e0 + lstride];
  const float dRf = (float)dR;
  float y = d2f_alu(-vm);
  float fdm = d2f_alu(vm - v0);
  float yprev = y;
  float a3raw = 0.f, a2p = 1.f;
  float vvq = vvc[e0 + lstride];
  float pprev = d2f_alu(p[e0]);  // p of the level below (the pressure difference of level q)
  // ring: doubles [NS][2][nt] (v of the level above, p), floats [NS][3][nt] (vv above, Nu, X)
  double *rd = reinterpret_cast<double *>(ring);
  float *rf = reinterpret_cast<float *>(rd + 2 * NS * nt);
  auto fetch = [&](int q) {
    const int s_ = (q - qlo - 1) % NS;
    const size_t e = (size_t)q * lstride + ci;
    cpa8(&rd[(s_ * 2 + 0) * nt + threadIdx.x], u2 + e + lstride);
    cpa8(&rd[(s_ * 2 + 1) * nt + threadIdx.x], p + e);
    cpa4(&rf[(s_ * 3 + 0) * nt + threadIdx.x], vvc + e + lstride);
    cpa4(&rf[(s_ * 3 + 1) * nt + threadIdx.x], Nu2 + e);
    cpa4(&rf[(s_ * 3 + 2) * nt + threadIdx.x], N2xz + e);
  };
#pragma unroll
  for (int s_ = 0; s_ < D; ++s_) {
    if (qlo + 1 + s_ <= qhi - 1) fetch(qlo + 1 + s_);
    cpa_commit();
  }
  for (int q = qlo + 1; q <= qhi - 1; ++q) {
    cpa_wait<D - 1>();
    const int s_ = (q - qlo - 1) % NS;
    const size_t e = (size_t)q * lstride + ci;
    const double vp1 = rd[(s_ * 2 + 0) * nt + threadIdx.x];
    const float pq = d2f_alu(rd[(s_ * 2 + 1) * nt + threadIdx.x]);
    const float vvp = rf[(s_ * 3 + 0) * nt + threadIdx.x], nuq = rf[(s_ * 3 + 1) * nt + threadIdx.x],
                xq = rf[(s_ * 3 + 2) * nt + threadIdx.x];
    if (q + D <= qhi - 1) fetch(q + D);
    cpa_commit();
    const float a = ta[q], b = tb[q], cc = tc[q], sdg = tsd[q] + k2f, thq = tth[q];
    const int ibs = tib[q];
    const float pd = pq - pprev;
    pprev = pq;
    const float fdp = d2f_alu(vp1 - v0);
    const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(v0));
    fdm = -fdp;
    float du;
    if (ibs < 0) {
      const float C3 = -dRf * dd * thq;
      du = mx_du(C1, L, C2, nuq, C3, pd);
      const float n = xq + (vvp - vvq) * thq * dd;
      Nu2[e] = n;
      du += G * n;
    } else {
      const float2 di = duib[((size_t)ibs * 3 + 1) * nc + c];
      du = part ? di.y : di.x;
    }
    const float rr = mx_rhs(beta, L, dtf, du);
    const float a1 = -beta * a;
    const float a2 = 1.f - beta * (b + k2f);
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    a2p = 1.f / (a2 - a1 * a3p);
    y = (rr - a1 * y) * a2p;
    yprev = y;
    a3raw = -beta * cc;
    vm = v0; v0 = vp1; vvq = vvp;
  }
  cpa_wait<0>();
  {  // last row: d(n-1) = -v(n-1)
    const int q = qhi;
    const float a3p = a3raw * a2p;
    ys[(size_t)(q - 1) * lstride + ci] = make_float2(yprev, a3p);
    y = d2f_alu(-v0);
    u2[(size_t)q * lstride + ci] = v0 + f2d_alu(y);
  }
  __threadfence_block();
  back_sweep_staged<D>(u2, ys, lstride, ci, qlo, qhi, y, ring, nt);
}

// ============================================================================
// Helmholtz solves of the FP64 form below LH_HELM_SPLIT columns (two lanes a column and field: two
// warps a scheduler): the right-hand sides element-wise over (column, chunk of levels), then the
// sweeps alone. An FP64 warp instruction holds its scheduler's half lane a clock for 64 cycles;
// a fused sweep with a lane per component held 26 of them a level, alone it holds the
// factorisation and three. The right-hand side takes
// the place of N_xz, which nothing reads after it, and the sweep's y that of the right-hand side.
// 32 x 32 x 153, us a launch of the fused sweep u/w 165, v 164 (side by side) -> 23 + 76.
// ============================================================================
#define LH_HL 8  // levels of a thread of the right-hand sides
#define LH_HELM_SPLIT 2432
struct HelmArgs {
  double2 *u[3];           // u, w, v
  double2 *Nu[3], *X[3];   // previous nonlinear terms; N_xz, then the right-hand side, then y
  const double2 *F[3];     // y-flux: uv, wv, vv
  const double2 *p;
  double *a3[3];           // upper factors [level][column][part]
  const int *ibslot[3];
  const double2 *duib;     // [slot][field u, v, w][column]
  int kRK;
};

// Right-hand side u + dt du of one field at the interior levels q0 .. q1 - 1 of a column segment
// (both parts), as k_helm64 forms it; V: v
template <bool V>
__device__ __forceinline__ void helm_rhs_field(const HelmArgs &a, const Geo &g, const DevScalars *__restrict__ sc, int f,
                                               int c, int q0, int q1) {
  const int kRK = a.kRK, nc = g.ncol, r = c / g.N1h, kx = c - r * g.N1h, nl = V ? g.nv : g.nu;
  double2 *u = a.u[f];
  double2 *Nu = a.Nu[f], *X = a.X[f];
  const double2 *F = a.F[f];
  const int *ibslot = a.ibslot[f];
  const int fd = V ? 1 : 2 * f;
  const double dt = sc->dt, dR = g.dRK[kRK - 1];
  size_t e = (size_t)q0 * nc + c;
  double2 um = u[e - nc], u0 = u[e];
  double2 fl = V ? F[e] : F[e - nc];
  double2 pm;
  if (V) pm = a.p[e - nc];
  const double unit = -dt / g.Re * g.aRK[kRK - 1], k2 = g.k2x[kx] + g.k2z[r];
  const double c2 = -dt * g.cRK[kRK - 1], cg = -dt * g.gRK[kRK - 1], cp = -dt * dR;
  const double ck = V ? 0.0 : cp * (f ? g.k1z[r] : g.k1x[kx]);
  const double mp = (f == 0 && c == 0) ? cp * sc->mpgx : 0.0;  // u only, real part
  const double *d2 = V ? g.d2v : g.d2u, *th = V ? g.thv : g.thu;
#pragma unroll 2
  for (int q = q0; q < q1; ++q, e += nc) {
    const double2 up1 = u[e + nc], pq = a.p[V ? e : e - nc];
    const double2 fq = V ? F[e + nc] : F[e], nuq = Nu[e], xq = X[e];
    const double l1 = unit * d2[q], l2 = unit * (d2[nl + q] + k2), l3 = unit * d2[2 * nl + q], thq = th[q] * g.dd;
    const int ibs = ibslot ? ibslot[q] : -1;
    double2 rr, nn;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const double upt = t ? up1.y : up1.x, u0t = t ? u0.y : u0.x, umt = t ? um.y : um.x;
      const double flq = t ? fq.y : fq.x, flm = t ? fl.y : fl.x, nu = t ? nuq.y : nuq.x, x = t ? xq.y : xq.x;
      double v;
      if (ibs < 0) {
        const double n = x + (flq - flm) * thq;
        (t ? nn.y : nn.x) = n;
        v = c2 * nu - (l1 * umt + (l2 * u0t + l3 * upt));  // the increment first: u's rounding enters once
        v += cg * n;
        if (V) {
          v += (cp * thq) * (t ? pq.y - pm.y : pq.x - pm.x);
        } else {
          v += t ? ck * pq.x : -ck * pq.y;
          if (t == 0) v += mp;
        }
      } else {
        const double2 di = a.duib[((size_t)ibs * 3 + fd) * nc + c];
        v = dt * (t ? di.y : di.x);
      }
      (t ? rr.y : rr.x) = u0t + v;
    }
    if (ibs < 0) { Nu[e].x = nn.x; Nu[e].y = nn.y; }
    X[e].x = rr.x; X[e].y = rr.y;
    um = u0; u0 = up1; fl = fq;
    if (V) pm = pq;
  }
}
// grid: x = (column block, field), y = chunk of levels
__global__ void __launch_bounds__(128) k_helm_rhs(HelmArgs a, Geo g, const DevScalars *__restrict__ sc) {
  const int f = blockIdx.x % 3, vc = (blockIdx.x / 3) * 128 + threadIdx.x;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int qlo = g.bq[bd][f == 2 ? 2 : 0], qhi = g.bq[bd][f == 2 ? 3 : 1];
  const int q0 = qlo + 1 + blockIdx.y * LH_HL, q1 = min(q0 + LH_HL, qhi);
  if (q0 >= q1) return;
  if (f == 2) helm_rhs_field<true>(a, g, sc, 2, c, q0, q1);
  else helm_rhs_field<false>(a, g, sc, f, c, q0, q1);
}

// The sweeps of one field: lane = (column segment, part), field blockIdx.y. U levels a batch, two
// batches ahead. The level tables are the matrix rows without k^2.
#define LH_HS_U 4
#define LH_HS_T 64
__host__ __device__ constexpr int hsweep_region() { return (3 * LH_HS_U * 2) | 1; }  // doubles of a thread's ring
__host__ __device__ constexpr size_t hsweep_smem(int nlev) { return 8 * ((size_t)3 * nlev + LH_HS_T * hsweep_region()); }
__global__ void __launch_bounds__(LH_HS_T) k_helm_sweep64(HelmArgs a, Geo g, const DevScalars *__restrict__ sc) {
  constexpr int U = LH_HS_U, EL = 2, BE = U * EL;  // a level: y, factor (backward)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int f = blockIdx.y, kRK = a.kRK, nlev = f == 2 ? g.nv : g.nu;
  double *ring_all = reinterpret_cast<double *>(smem_raw), *ta = ring_all + LH_HS_T * hsweep_region(), *tb = ta + nlev,
         *tc = tb + nlev;
  const double beta = g.bRK[kRK - 1] * sc->dt / g.Re;
  {
    const double *d2 = f == 2 ? g.d2v : g.d2u;
    for (int i = threadIdx.x; i < nlev; i += LH_HS_T) {
      ta[i] = -beta * d2[i]; tb[i] = 1.0 - beta * d2[nlev + i]; tc[i] = -beta * d2[2 * nlev + i];
    }
  }
  __syncthreads();
  double *ring = ring_all + threadIdx.x * hsweep_region();
  const unsigned rs = (unsigned)__cvta_generic_to_shared(ring);
  const int tid = blockIdx.x * LH_HS_T + threadIdx.x, vc = tid >> 1, part = tid & 1;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const bool V = f == 2;
  const int qlo = g.bq[bd][V ? 2 : 0], qhi = g.bq[bd][V ? 3 : 1];
  const size_t ls = 2 * (size_t)g.ncol, ci = 2 * (size_t)c + part;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const double bk = beta * (g.k2x[kx] + g.k2z[r]);
  const double gw1 = V ? 0.0 : g.gw[bd][0], gw2 = V ? 0.0 : g.gw[bd][1];
  double *u = reinterpret_cast<double *>(a.u[f]) + ci, *X = reinterpret_cast<double *>(a.X[f]) + ci, *A = a.a3[f] + ci;
  double y = 0.0, a3raw = gw1, a2p = 1.0;  // first row: [1, gw(b,1)], rhs 0
  {
    const double *fx = X + (size_t)(qlo + 1) * ls;
    int left = qhi - qlo - 1;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (left > i) { cpa8s(dst + 8 * i, fx); fx += ls; }
      left -= U;
      dst = dst == rs + 8 * 2 * BE ? rs : dst + 8 * BE;
      cpa_commit();
    };
    fetch();
    fetch();
    double *oy = X + (size_t)(qlo + 1) * ls, *oa = A + (size_t)qlo * ls;
    const double *h = ring;
    int q = qlo + 1;
    for (int n = qhi - qlo - 1; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        const double rr = h[i], a1 = ta[q + i], a2 = tb[q + i] - bk;
        const double a3p = a3raw * a2p;
        *oa = a3p;
        oa += ls;
        a2p = 1.0 / (a2 - a1 * a3p);
        y = (rr - a1 * y) * a2p;
        *oy = y;
        oy += ls;
        a3raw = tc[q + i];
      }
      q += U;
      h = h == ring + 2 * BE ? ring : h + BE;
    }
  }
  cpa_wait<0>();
  {  // last row: [gw(b,2), 1], rhs 0
    const double a3p = a3raw * a2p;
    A[(size_t)(qhi - 1) * ls] = a3p;
    a2p = 1.0 / (1.0 - gw2 * a3p);
    y = (0.0 - gw2 * y) * a2p;
    u[(size_t)qhi * ls] = y;
  }
  __threadfence();  // the copies below read what this thread stored above
  {
    const double *fy = X + (size_t)(qhi - 1) * ls, *fa = A + (size_t)(qhi - 1) * ls;
    double *ou = u + (size_t)(qhi - 1) * ls;
    int left = qhi - qlo;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (left > i) { cpa8s(dst + 16 * i, fy); cpa8s(dst + 16 * i + 8, fa); fy -= ls; fa -= ls; }
      left -= U;
      dst = dst == rs + 8 * 2 * BE ? rs : dst + 8 * BE;
      cpa_commit();
    };
    fetch();
    fetch();
    const double *h = ring;
    for (int n = qhi - qlo; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        const double ya = n == i + 1 ? 0.0 : h[2 * i], a3p = h[2 * i + 1];
        y = ya - a3p * y;
        *ou = y;
        ou -= ls;
      }
      h = h == ring + 2 * BE ? ring : h + BE;
    }
  }
  cpa_wait<0>();
}

// ============================================================================
// The mixed form's solves below LH_HELM_SPLIT_MX columns (of the channel and those beside it in a
// batch): as above, the right-hand sides element-wise, then the sweeps of all three fields in one
// launch. The operations and roundings are those of k_helm_u_mx2 / k_helm_v_mx2 (the fused
// multiply-adds are written out), so the results are the same bit for bit. The right-hand side
// takes the place of N_xz.
// us a step, fused -> split, among others / alone: 32 x 32 x 153 (544 columns) 203 / 479 -> 162 / 345,
// 64 x 64 x 129 (2112) 300 / 534 -> 301 / 466, 96 x 64 x 129 (3136) 380 / 600 -> 404 / 567,
// 96 x 96 x 129 (4704) 511 / 722 -> 572 / 709, 128 x 128 x 201 (8320) 1257 / 1544 -> 1491 / 1695.
// ============================================================================
#define LH_HELM_SPLIT_MX 2432
struct HelmMxArgs {
  double *u[3];            // u, w, v
  float *Nu[3];
  float *X[3];             // N_xz, then the right-hand side
  const float *F[3];
  const double *p;
  float2 *ys[3];           // y, upper factor
  const int *ibslot[3];
  const float2 *duib;
  int kRK;
};
// grid: x = (lane block, field), y = chunk of levels
__global__ void __launch_bounds__(128) k_helm_rhs_mx(HelmMxArgs ar, Geo g, const DevScalars *__restrict__ sc) {
  const int f = blockIdx.x % 3, tid = (blockIdx.x / 3) * 128 + threadIdx.x, vc = tid >> 1, part = tid & 1;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  if (c == 0) return;  // mode (0,0): k_helm00_pcr (FP64)
  const bool V = f == 2;
  const int qlo = g.bq[bd][V ? 2 : 0], qhi = g.bq[bd][V ? 3 : 1], kRK = ar.kRK, nc = g.ncol;
  const int q0 = qlo + 1 + blockIdx.y * LH_HL, q1 = min(q0 + LH_HL, qhi);
  if (q0 >= q1) return;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float G = (float)(-g.gRK[kRK - 1]);
  const float dd = (float)g.dd, dRf = (float)dR;
  const float dtf = (float)sc->dt, beta = (float)(g.bRK[kRK - 1] * sc->dt / g.Re);
  const float C3u = (float)(-dR * (f ? g.k1z[r] : g.k1x[kx]));
  const int nl = V ? g.nv : g.nu;
  const float *d2f = V ? g.d2vf : g.d2uf, *sdgt = V ? g.sdgv : g.sdgu, *tht = V ? g.thvf : g.thuf;
  const int *ibslot = ar.ibslot[f];
  const size_t ls = (size_t)nc * 2, ci = (size_t)c * 2 + part;
  const double *u = ar.u[f] + ci;
  const float *F = ar.F[f] + ci;
  float *Nu = ar.Nu[f] + ci, *X = ar.X[f] + ci;
  size_t e = (size_t)q0 * ls;
  const double um = u[e - ls];
  double u0 = u[e];
  float fdm = q0 == qlo + 1 ? d2f_alu(um - u0) : -d2f_alu(u0 - um);
  float flm = V ? F[e] : F[e - ls];
  float pm = V ? d2f_alu(ar.p[ci + e - ls]) : 0.f;
#pragma unroll 2
  for (int q = q0; q < q1; ++q, e += ls) {
    const double up1 = u[e + ls];
    const float flq = V ? F[e + ls] : F[e], nuq = Nu[e], xq = X[e];
    const float a = d2f[q], cc = d2f[2 * nl + q], sdg = sdgt[q] + k2f, thq = tht[q];
    const int ibs = ibslot ? ibslot[q] : -1;
    const float fdp = d2f_alu(up1 - u0);
    const float L = mx_lap(a, fdm, cc, fdp, sdg, d2f_alu(u0));
    fdm = -fdp;
    float pt, C3;
    if (V) {
      const float pq = d2f_alu(ar.p[ci + e]);
      pt = pq - pm;
      pm = pq;
      C3 = -dRf * dd * thq;
    } else {
      const double po = ar.p[((size_t)(q - 1) * nc + c) * 2 + (part ^ 1)];  // i*C3*p: (-C3 p.y, C3 p.x)
      pt = part ? d2f_alu(po) : -d2f_alu(po);
      C3 = C3u;
    }
    float du;
    if (ibs < 0) {
      du = mx_du(C1, L, C2, nuq, C3, pt);
      const float n = __fmaf_rn(__fmul_rn(__fsub_rn(flq, flm), thq), dd, xq);
      Nu[e] = n;
      du = __fmaf_rn(G, n, du);
    } else {
      const float2 di = ar.duib[((size_t)ibs * 3 + (V ? 1 : 2 * f)) * nc + c];
      du = part ? di.y : di.x;
    }
    X[e] = mx_rhs(beta, L, dtf, du);
    u0 = up1;
    flm = flq;
  }
}
// The sweeps of one field: lane = (column segment, part), field blockIdx.y; the inputs of two batches
// of U levels are on their way while one is worked on.
__host__ __device__ constexpr int hsweep_mx_region() { return (3 * LH_HS_U * 2) | 1; }  // doubles of a thread's ring
__host__ __device__ constexpr size_t hsweep_mx_smem(int nlev) {
  return 8 * (size_t)LH_HS_T * hsweep_mx_region() + 4 * (size_t)3 * nlev;
}
__global__ void __launch_bounds__(LH_HS_T) k_helm_sweep_mx(HelmMxArgs ar, Geo g, const DevScalars *__restrict__ sc) {
  constexpr int U = LH_HS_U;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int f = blockIdx.y, kRK = ar.kRK;
  const bool V = f == 2;
  const int nl = V ? g.nv : g.nu;
  double *ring = reinterpret_cast<double *>(smem_raw) + threadIdx.x * hsweep_mx_region();
  float *ta = reinterpret_cast<float *>(reinterpret_cast<double *>(smem_raw) + LH_HS_T * hsweep_mx_region()), *tb = ta + nl,
        *tc = tb + nl;
  {
    const float *d2f = V ? g.d2vf : g.d2uf;
    for (int i = threadIdx.x; i < nl; i += LH_HS_T) { ta[i] = d2f[i]; tb[i] = d2f[nl + i]; tc[i] = d2f[2 * nl + i]; }
  }
  __syncthreads();
  const int tid = blockIdx.x * LH_HS_T + threadIdx.x, vc = tid >> 1, part = tid & 1;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  if (c == 0) return;
  const int qlo = g.bq[bd][V ? 2 : 0], qhi = g.bq[bd][V ? 3 : 1];
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float beta = (float)(g.bRK[kRK - 1] * sc->dt / g.Re);
  const double gw1 = g.gw[bd][0], gw2 = g.gw[bd][1];
  const size_t ls = (size_t)g.ncol * 2, ci = (size_t)c * 2 + part;
  double *u = ar.u[f] + ci;
  float2 *ys = ar.ys[f] + ci;
  const unsigned rs = (unsigned)__cvta_generic_to_shared(ring);
  const double ulo = u[(size_t)qlo * ls], uhi = u[(size_t)qhi * ls], uhm = u[(size_t)(qhi - 1) * ls];
  float y = V ? d2f_alu(-ulo) : d2f_alu(-(ulo + gw1 * u[(size_t)(qlo + 1) * ls]));  // first row
  float a3raw = V ? 0.f : (float)gw1, a2p = 1.f;
  {
    const float *in = ar.X[f] + ci + (size_t)(qlo + 1) * ls;
    int left = qhi - qlo - 1;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (left > i) { cpa4s(dst + 4 * i, in); in += ls; }
      left -= U;
      dst = dst == rs + 8 * U ? rs : dst + 4 * U;
      cpa_commit();
    };
    fetch();
    fetch();
    float2 *o = ys + (size_t)qlo * ls;
    const float *r0 = reinterpret_cast<const float *>(ring), *h = r0;
    int q = qlo + 1;
    for (int n = qhi - qlo - 1; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        const float a = ta[q + i], b = tb[q + i], cc = tc[q + i], rr = h[i];
        const float a1 = -beta * a;
        const float a2 = __fmaf_rn(-beta, __fadd_rn(b, k2f), 1.f);
        const float a3p = a3raw * a2p;
        *o = make_float2(y, a3p);
        o += ls;
        a2p = 1.f / __fmaf_rn(-a1, a3p, a2);
        y = __fmul_rn(__fmaf_rn(-a1, y, rr), a2p);
        a3raw = -beta * cc;
      }
      q += U;
      h = h == r0 + 2 * U ? r0 : h + U;
    }
  }
  cpa_wait<0>();
  {
    const float a3p = a3raw * a2p;
    ys[(size_t)(qhi - 1) * ls] = make_float2(y, a3p);
    if (V) {  // last row: d(n-1) = -v(n-1)
      y = d2f_alu(-uhi);
    } else {  // last row: gw2 d(n-2) + d(n-1) = -(gw2 u(n-2) + u(n-1))
      const float a1 = (float)gw2;
      const float rl = d2f_alu(-(gw2 * uhm + uhi));
      a2p = 1.f / (1.f - a1 * a3p);
      y = (rl - a1 * y) * a2p;
    }
    u[(size_t)qhi * ls] = uhi + f2d_alu(y);
  }
  __threadfence();  // the copies below read what this thread stored above
  {
    const float2 *fy = ys + (size_t)(qhi - 1) * ls;
    const double *fu = u + (size_t)(qhi - 1) * ls;
    double *ou = u + (size_t)(qhi - 1) * ls;
    int left = qhi - qlo;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (left > i) { cpa8s(dst + 16 * i, fy); cpa8s(dst + 16 * i + 8, fu); fy -= ls; fu -= ls; }
      left -= U;
      dst = dst == rs + 32 * U ? rs : dst + 16 * U;
      cpa_commit();
    };
    fetch();
    fetch();
    const double *h = ring;
    for (int n = qhi - qlo; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        const float2 ya = reinterpret_cast<const float2 *>(h)[2 * i];
        y = ya.x - ya.y * y;
        *ou = h[2 * i + 1] + f2d_alu(y);
        ou -= ls;
      }
      h = h == ring + 4 * U ? ring : h + 2 * U;
    }
  }
  cpa_wait<0>();
}

// ============================================================================
// flowrate_corr (littleharsh.f90:476-509) on mode (0,0) of u1. The block stages the
// coefficients, the level widths and u(0,0) in `w` (shared memory when it fits,
// else global scratch); thread 0 runs the recurrence and the sums in the
// reference's order; the block applies the correction.
// w: 6*(nn+3) doubles: u11, a1, a2, a3, dy, ur
// ============================================================================
__global__ void k_meanflow(double2 *__restrict__ u1, Geo g, DevScalars *sc, int kRK, double *__restrict__ wg,
                           int use_smem) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nn = g.nn, n = nn + 3, dny = g.dny, nc = g.ncol, nu = g.nu;
  double *w = use_smem ? reinterpret_cast<double *>(smem_raw) : wg;
  double *u11 = w, *a1 = w + n, *a2 = w + 2 * n, *a3 = w + 3 * n, *dy = w + 4 * n, *ur = w + 5 * n;
  __shared__ double gg_sh;
  const double dt = sc->dt;
  const double bdt = -g.dRK[kRK - 1] * dt;
  const double beta = g.bRK[kRK - 1] * dt / g.Re;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    if (j == 0) { a1[j] = 0.0; a2[j] = 1.0; a3[j] = g.gw[1][0]; u11[j] = 0.0; }
    else if (j == nn + 2) { a1[j] = g.gw[1][1]; a2[j] = 1.0; a3[j] = 0.0; u11[j] = 0.0; }
    else {
      a1[j] = -beta * g.d2u[j + dny];
      a2[j] = 1.0 - beta * g.d2u[nu + j + dny];
      a3[j] = -beta * g.d2u[2 * nu + j + dny];
      u11[j] = bdt;
    }
    dy[j] = (j >= 1 && j <= nn + 1) ? (g.yv[j + dny] - g.yv[j - 1 + dny]) : 0.0;
    ur[j] = u1[(size_t)(j + dny) * nc].x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a2[0] = 1.0 / a2[0];
    for (int j = 1; j < n; ++j) {
      a3[j - 1] = a3[j - 1] * a2[j - 1];
      a2[j] = 1.0 / (a2[j] - a1[j] * a3[j - 1]);
    }
    u11[0] = u11[0] * a2[0];
    for (int j = 1; j < n; ++j) u11[j] = (u11[j] - a1[j] * u11[j - 1]) * a2[j];
    for (int j = n - 2; j >= 0; --j) u11[j] = u11[j] - a3[j] * u11[j + 1];
    double Qx1 = 0.0, Qx0 = 0.0;
    for (int j = 1; j <= nn + 1; ++j) Qx1 = Qx1 + dy[j] * u11[j];
    for (int j = 1; j <= nn + 1; ++j) Qx0 = Qx0 + dy[j] * ur[j];
    const double gg = (sc->QxT - Qx0) / Qx1;
    sc->mpgx = sc->mpgx + gg;
    sc->dgx = gg;
    gg_sh = gg;
  }
  __syncthreads();
  const double gg = gg_sh;
  for (int j = threadIdx.x; j <= nn + 2; j += blockDim.x) u1[(size_t)(j + dny) * nc].x = ur[j] + gg * u11[j];
}

// flowrate_corr with the tridiagonal system solved by parallel cyclic reduction in one
// block (log2(n) steps) instead of k_meanflow's serial recurrence (its FP64 divisions
// were the latency); same system and correction, the solution's rounding differs.
// Shared memory: 8 n doubles (two copies of the four diagonals/rhs).
__global__ void __launch_bounds__(512) k_meanflow_pcr(double2 *__restrict__ u1, Geo g, DevScalars *sc, int kRK) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double gg_sh;
  const int nn = g.nn, n = nn + 3, dny = g.dny, nc = g.ncol, nu = g.nu;
  double *A = reinterpret_cast<double *>(smem_raw), *B = A + n, *Cc = B + n, *D = Cc + n;
  double *A2 = D + n, *B2 = A2 + n, *C2b = B2 + n, *D2 = C2b + n;
  const double dt = sc->dt;
  const double bdt = -g.dRK[kRK - 1] * dt;
  const double beta = g.bRK[kRK - 1] * dt / g.Re;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    if (j == 0) { A[j] = 0.0; B[j] = 1.0; Cc[j] = g.gw[1][0]; D[j] = 0.0; }
    else if (j == nn + 2) { A[j] = g.gw[1][1]; B[j] = 1.0; Cc[j] = 0.0; D[j] = 0.0; }
    else {
      A[j] = -beta * g.d2u[j + dny];
      B[j] = 1.0 - beta * g.d2u[nu + j + dny];
      Cc[j] = -beta * g.d2u[2 * nu + j + dny];
      D[j] = bdt;
    }
  }
  __syncthreads();
  for (int st = 1; st < n; st *= 2) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int im = i - st, ip = i + st;
      double a = 0.0, b = B[i], c = 0.0, d = D[i];
      if (im >= 0) {
        const double al = -A[i] / B[im];
        a = al * A[im];
        b += al * Cc[im];
        d += al * D[im];
      }
      if (ip < n) {
        const double ga = -Cc[i] / B[ip];
        c = ga * Cc[ip];
        b += ga * A[ip];
        d += ga * D[ip];
      }
      A2[i] = a; B2[i] = b; C2b[i] = c; D2[i] = d;
    }
    __syncthreads();
    double *t;
    t = A; A = A2; A2 = t;
    t = B; B = B2; B2 = t;
    t = Cc; Cc = C2b; C2b = t;
    t = D; D = D2; D2 = t;
  }
  // u11 = D / B; the flow-rate sums Qx1 = sum dy u11, Qx0 = sum dy u(0,0) (j = 1..nn+1)
  // run serially in the reference's order: QxT - Qx0 cancels, so its rounding matters
  // (the level widths and u(0,0) are staged in shared memory first: the serial loop then
  // runs on shared-memory loads)
  double *dy = A2, *ur = B2;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    D[j] = D[j] / B[j];
    dy[j] = (j >= 1 && j <= nn + 1) ? (g.yv[j + dny] - g.yv[j - 1 + dny]) : 0.0;
    ur[j] = u1[(size_t)(j + dny) * nc].x;
  }
  __syncthreads();
  if (threadIdx.x == 32) {  // (a warp each: two serial sums side by side)
    double Qx0 = 0.0;
    for (int j = 1; j <= nn + 1; ++j) Qx0 = Qx0 + dy[j] * ur[j];
    gg_sh = Qx0;
  }
  double Qx1 = 0.0;
  if (threadIdx.x == 0)
    for (int j = 1; j <= nn + 1; ++j) Qx1 = Qx1 + dy[j] * D[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    const double Qx0 = gg_sh;
    const double gg = (sc->QxT - Qx0) / Qx1;
    sc->mpgx = sc->mpgx + gg;
    sc->dgx = gg;
    gg_sh = gg;
  }
  __syncthreads();
  const double gg = gg_sh;
  for (int j = threadIdx.x; j <= nn + 2; j += blockDim.x) u1[(size_t)(j + dny) * nc].x += gg * D[j];
}

// flowrateIm of u1 (0,0): Qx (meanflow_ctP, littleharsh.f90:529-545; getini)
__global__ void k_flowrate(const double2 *__restrict__ u1, Geo g, DevScalars *sc, int setQxT) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double Q = 0.0;
  for (int j = 1; j <= g.nn + 1; ++j) Q = Q + (g.yv[j + g.dny] - g.yv[j - 1 + g.dny]) * u1[(size_t)(j + g.dny) * g.ncol].x;
  sc->Qx = Q;
  if (setQxT) sc->QxT = Q;
}

// The scalar part of record_out (FOU3D.f90:3040-3070) from mode (0,0) of u1: Qx by flowrateIm,
// Umax by maxvel (littleharsh.f90:511-527: the largest Re u(j), j = 0..nn+2, not below 0) and
// the slip velocity Uslip, u(0,0) extrapolated linearly from levels 0 and 1 to y = -1.
__global__ void k_history(const double2 *__restrict__ u1, Geo g, DevScalars *sc) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int dny = g.dny, nc = g.ncol;
  double Q = 0.0, um = 0.0;
  for (int j = 1; j <= g.nn + 1; ++j) Q = Q + (g.yv[j + dny] - g.yv[j - 1 + dny]) * u1[(size_t)(j + dny) * nc].x;
  for (int j = 0; j <= g.nn + 2; ++j) um = fmax(um, u1[(size_t)(j + dny) * nc].x);
  const double u0 = u1[(size_t)dny * nc].x, u1v = u1[(size_t)(1 + dny) * nc].x;
  const double y0 = g.yu[dny], y1 = g.yu[1 + dny];
  sc->Qx = Q;
  sc->Umax = um;
  sc->Uslip = (u1v * (-1.0 - y0) + u0 * (y1 + 1.0)) / (y1 - y0);
}

__global__ void k_step_end(DevScalars *sc) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  sc->iter += 1;
  const double e = sqrt(__longlong_as_double((long long)sc->errbits));
  sc->err = e;
  if (!(e == e) || isinf(e) || !(sc->dt == sc->dt)) sc->status = LH_ENONFINITE;
}

// ============================================================================
// LU_buildP + LU_decP (tridLU_3D.f90:333-407, 477-518), once per channel: the
// pressure matrix does not depend on time. dg1 = a1 (lower), dg2 = 1/pivot,
// dg3 = upper factor; [qp][col], qp = 0..np-1 <-> p level N(4,0)+1+qp.
// ============================================================================
__global__ void __launch_bounds__(NTHR) k_build_dg(double *__restrict__ dg1, double *__restrict__ dg2,
                                                   double *__restrict__ dg3, Geo g) {
  const int vc = blockIdx.x * blockDim.x + threadIdx.x;
  const int nc = g.ncol;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int plo = g.bq[bd][4], phi = g.bq[bd][5];
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const double k2x = g.k2x[kx], k2z = g.k2z[r];
  const double dd = g.dd;
  double a3raw = 0.0, a2p = 0.0;
  for (int qp = plo; qp <= phi; ++qp) {
    const int q = qp + 1;
    const double Dt = dd * g.thu[q];
    const double Gb = -dd * g.thv[q];
    double A1, A2, A3;
    if (qp == plo) {
      A1 = 0.0;
      A2 = (Dt * Gb) + k2x + k2z;
      A3 = (Dt * (dd * g.thv[q]));
      if (c == 0 && bd == 1) {  // gauge of mode (0,0)
        const double h = g.yu[2 + g.dny] - g.yu[1 + g.dny];
        A1 = 0.0; A2 = 1.0 / (h * h); A3 = 0.0;
      }
    } else {
      const double Db = -dd * g.thu[q];
      const double Gt = dd * g.thv[q - 1];
      const double Gbm = -dd * g.thv[q - 1];
      if (qp == phi) { A2 = (Db * Gt) + k2x + k2z; A1 = (Db * Gbm); A3 = 0.0; }
      else { A2 = (Db * Gt) + (Dt * Gb) + k2x + k2z; A1 = (Db * Gbm); A3 = (Dt * (dd * g.thv[q])); }
    }
    if (qp == plo) a2p = 1.0 / A2;
    else {
      const double a3p = a3raw * a2p;
      dg3[(size_t)(qp - 1) * nc + c] = a3p;
      a2p = 1.0 / (A2 - A1 * a3p);
    }
    dg1[(size_t)qp * nc + c] = A1;
    dg2[(size_t)qp * nc + c] = a2p;
    a3raw = A3;
  }
  dg3[(size_t)phi * nc + c] = 0.0;
}

// a b + c d + t dv, the sum of both routes of the pressure step: written out, as the compiler's choice of
// the product to round need not be the same in each kernel (they agree bit for bit)
__device__ __forceinline__ double press_div(double a, double b, double c, double d, double t, double dv) {
  return __fma_rn(t, dv, __fma_rn(a, b, __dmul_rn(c, d)));
}

// ============================================================================
// Pressure: divergence, psi = dti/(a+b) div (gauge on (0,0)), LUsolP with the
// stored factors, p += psi, v_corr, and the divergence of the corrected field
// (max |div|^2 -> errbits) when need_div: the reference recomputes div after
// every v_corr but only reads it (error()) at the start of a step, so it is
// formed in the third substep. p levels qp <-> u/v index q = qp + 1;
// `psi` holds the forward-sweep values (psi itself stays in registers).
// ============================================================================
// One lane per (column, real/imaginary part): the pressure matrix is real, so the two
// parts are independent systems; the i*k couplings of the divergence and of v_corr
// exchange the other part through a shuffle within the lane pair. Two lanes per column
// double the warps in flight (the solves are latency-bound at the 384x192 wall grid).
// Scalar views: element (level, col, part) at (level*ncol + col)*2 + part.
__global__ void __launch_bounds__(NTHR, LH_PRESS_MINB) k_press2(double *__restrict__ u1, double *__restrict__ u2,
                                                 double *__restrict__ u3, double *__restrict__ p,
                                                 double *__restrict__ psi, const double *__restrict__ dg1,
                                                 const double *__restrict__ dg2, const double *__restrict__ dg3, Geo g,
                                                 DevScalars *sc, int kRK, int need_div) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const unsigned pm = 3u << ((threadIdx.x & 31) & ~1);  // the lane pair
  const int nc = g.ncol;
  unsigned long long dmax = 0ull;  // max |div|^2 as bits
  // per-level factors of this substep: dti/(a+b) dd thu (divergence -> right-hand side)
  // and dt (a+b) dd thv (v_corr), so that the lanes spend no FP64 multiply on them
  extern __shared__ double ptab[];
  {
    const double aRb0 = g.aRK[kRK - 1] + g.bRK[kRK - 1];
    const double dti0 = sc->dti / aRb0, dtk0 = sc->dt * aRb0 * g.dd;
    for (int i = threadIdx.x; i < g.nu; i += blockDim.x) ptab[i] = dti0 * g.thud[i];
    for (int i = threadIdx.x; i < g.nv; i += blockDim.x) ptab[g.nu + i] = dtk0 * g.thv[i];
    __syncthreads();
  }
  if (vc < g.nvc) {
    int c, bd;
    vcol_of(g, vc, c, bd);
    const int plo = g.bq[bd][4], phi = g.bq[bd][5];
    const int ulo = g.bq[bd][0], uhi = g.bq[bd][1], vlo = g.bq[bd][2], vhi = g.bq[bd][3];
    const int r = c / g.N1h, kx = c - r * g.N1h;
    const double kxv = g.k1x[kx], kzv = g.k1z[r];
    // i*k*z: real part -k*z.y, imaginary part k*z.x; lane `part` reads the other part
    const double sgn = part ? 1.0 : -1.0;
    const double skx = sgn * kxv, skz = sgn * kzv;  // sgn*(a+b) = sgn*a + sgn*b exactly
    const double aRb = g.aRK[kRK - 1] + g.bRK[kRK - 1];
    const double dtirk = sc->dti / aRb;
    const double dt = sc->dt;
    const size_t ls = (size_t)nc * 2;
    const size_t ci = (size_t)c * 2 + part, co = (size_t)c * 2 + (part ^ 1);
    constexpr int D = LH_PF_PRESS > 0 ? LH_PF_PRESS : 1;
    const double dskx = dtirk * skx, dskz = dtirk * skz;
#define HP_TH(q_) ptab[q_]
#define HP_TV(q_) ptab[g.nu + (q_)]
    double y = 0.0;
    double vm = u2[(size_t)plo * ls + ci];
    {  // forward sweep; the inputs of a level are loaded D levels ahead
      double fa[D], fw[D], fv[D], f1[D], f2[D], ft[D];
#define HP_FETCH(s_, qq_)                                              \
  {                                                                    \
    const int qp_ = (qq_);                                             \
    const size_t e_ = (size_t)(qp_ + 1) * ls;                          \
    fa[s_] = u1[e_ + co]; fw[s_] = u3[e_ + co]; fv[s_] = u2[e_ + ci];  \
    f1[s_] = dg1[(size_t)qp_ * nc + c]; f2[s_] = dg2[(size_t)qp_ * nc + c]; \
    ft[s_] = HP_TH(qp_ + 1);                                           \
  }
#pragma unroll
      for (int s_ = 0; s_ < D; ++s_)
        if (plo + s_ <= phi) HP_FETCH(s_, plo + s_)
      for (int qb = plo; qb <= phi; qb += D) {
#pragma unroll
        for (int s_ = 0; s_ < D; ++s_) {
          const int qp = qb + s_;
          if (qp > phi) break;
          const double ao = fa[s_], wo = fw[s_], v = fv[s_], A1 = f1[s_], a2p = f2[s_];
          const double th = ft[s_];
          if (qp + D <= phi) HP_FETCH(s_, qp + D)
          double rhs = press_div(dskx, ao, dskz, wo, th, v - vm);
          vm = v;
          if (qp == plo && c == 0 && bd == 1) rhs = 0.0;
          y = (qp == plo) ? rhs * a2p : (rhs - A1 * y) * a2p;
          psi[(size_t)qp * ls + ci] = y;
        }
      }
#undef HP_FETCH
    }
    const double dtrk = dt * aRb;
    const double kxd = dtrk * kxv, kzd = dtrk * kzv;
    double xn = y;
    double vup = 0.0, aup_o = 0.0, wup_o = 0.0;
    {  // backward sweep, v_corr and the divergence of the corrected field; loads D levels ahead
      double bs[D], b3[D], bp[D], bu[D], bw[D], bv[D], btv[D], btu[D];
#define HB_FETCH(s_, qq_)                                                   \
  {                                                                         \
    const int qp_ = (qq_);                                                  \
    const size_t e_ = (size_t)(qp_ + 1) * ls + ci;                          \
    bs[s_] = psi[(size_t)qp_ * ls + ci]; b3[s_] = dg3[(size_t)qp_ * nc + c]; \
    bp[s_] = p[(size_t)qp_ * ls + ci];                                      \
    bu[s_] = u1[e_]; bw[s_] = u3[e_]; bv[s_] = u2[e_];                      \
    btv[s_] = HP_TV(qp_ + 1); btu[s_] = g.thud[qp_ + 2];                    \
  }
#pragma unroll
      for (int s_ = 0; s_ < D; ++s_)
        if (phi - s_ >= plo) HB_FETCH(s_, phi - s_)
      for (int qb = phi; qb >= plo; qb -= D) {
#pragma unroll
        for (int s_ = 0; s_ < D; ++s_) {
          const int qp = qb - s_;
          if (qp < plo) break;
          const int q = qp + 1;
          const size_t e = (size_t)q * ls;
          const double ps = bs[s_], d3 = b3[s_], pq = bp[s_], uq = bu[s_], wq = bw[s_];
          const double thv = btv[s_], thu1 = btu[s_];
          double v = bv[s_];
          if (qp - D >= plo) HB_FETCH(s_, qp - D)
          const double x = (qp == phi) ? xn : ps - d3 * xn;
          p[(size_t)qp * ls + ci] = pq + x;
          // u -= dtrk i kx psi: the real part gains kxd*psi.y, the imaginary part loses kxd*psi.x
          const double xo = __shfl_xor_sync(pm, x, 1);
          const double a = uq - sgn * kxd * xo;
          const double w = wq - sgn * kzd * xo;
          u1[e + ci] = a;
          u3[e + ci] = w;
          if (q <= vhi - 1) {
            v = v - thv * (xn - x);
            u2[e + ci] = v;
          }
          // divergence of the corrected field at the level above (p level qp + 1)
          const double ao = __shfl_xor_sync(pm, a, 1), wo = __shfl_xor_sync(pm, w, 1);
          if (need_div && qp < phi) {
            const double th = thu1;
            const double dvp = press_div(skx, aup_o, skz, wup_o, th, vup - v);
            const double d2 = __dmul_rn(dvp, dvp);
            bits_max(dmax, __dadd_rn(d2, __shfl_xor_sync(pm, d2, 1)));
          }
          aup_o = ao; wup_o = wo; vup = v;
          xn = x;
        }
      }
#undef HB_FETCH
#undef HP_TH
#undef HP_TV
    }
    if (need_div) {
      const double th = g.thud[plo + 1];
      const double vb = u2[(size_t)plo * ls + ci];
      const double dvp = press_div(skx, aup_o, skz, wup_o, th, vup - vb);
      const double d2 = __dmul_rn(dvp, dvp);
      bits_max(dmax, __dadd_rn(d2, __shfl_xor_sync(pm, d2, 1)));
    }
    if (bd <= 1) {
      u1[(size_t)ulo * ls + ci] = g.gwbc1 * u1[(size_t)(ulo + 1) * ls + ci];
      u3[(size_t)ulo * ls + ci] = g.gwbc3 * u3[(size_t)(ulo + 1) * ls + ci];
    }
    if (bd >= 1) {
      u1[(size_t)uhi * ls + ci] = g.gwbc1 * u1[(size_t)(uhi - 1) * ls + ci];
      u3[(size_t)uhi * ls + ci] = g.gwbc3 * u3[(size_t)(uhi - 1) * ls + ci];
    }
    u2[(size_t)vlo * ls + ci] = 0.0;
    u2[(size_t)vhi * ls + ci] = 0.0;
  }
  // |div|^2 = re^2 + im^2 per level, summed over the lane pair above
  dmax = warp_max_bits(dmax);
  if ((threadIdx.x & 31) == 0) atomicMax(&sc->errbits, dmax);
}

// ============================================================================
// The pressure step of k_press2 with the y-columns staged through shared memory: every lane
// keeps a ring of D + 1 levels of its inputs, filled by cp.async copies issued D levels ahead
// of the sweep (into the slot not being read), so that D memory latencies overlap without
// holding the prefetched values in registers (the solves have few warps per SM: one lane per
// column and part). Same arithmetic as k_press2, so the same results bit for bit. Shared
// memory: the per-level factor tables (nu + nv doubles) and the ring, 6 (D + 1) doubles per
// thread.
// ============================================================================

template <int D>
__global__ void __launch_bounds__(NTHR) k_press3(double *__restrict__ u1, double *__restrict__ u2,
                                                 double *__restrict__ u3, double *__restrict__ p,
                                                 double *__restrict__ psi, const double *__restrict__ dg1,
                                                 const double *__restrict__ dg2, const double *__restrict__ dg3, Geo g,
                                                 DevScalars *sc, int kRK, int need_div) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int vc = tid >> 1, part = tid & 1;
  const unsigned pm = 3u << ((threadIdx.x & 31) & ~1);  // the lane pair
  const int nc = g.ncol;
  unsigned long long dmax = 0ull;  // max |div|^2 as bits
  extern __shared__ double ptab[];
  const int nt = blockDim.x;
  double *ring = ptab + ((g.nu + g.nv + 1) & ~1);  // [D + 1][6][nt]
  constexpr int NS = D + 1;
  {
    const double aRb0 = g.aRK[kRK - 1] + g.bRK[kRK - 1];
    const double dti0 = sc->dti / aRb0, dtk0 = sc->dt * aRb0 * g.dd;
    for (int i = threadIdx.x; i < g.nu; i += blockDim.x) ptab[i] = dti0 * g.thud[i];
    for (int i = threadIdx.x; i < g.nv; i += blockDim.x) ptab[g.nu + i] = dtk0 * g.thv[i];
    __syncthreads();
  }
#define RS(s_, f_) ring[((s_) * 6 + (f_)) * nt + threadIdx.x]
  if (vc < g.nvc) {
    int c, bd;
    vcol_of(g, vc, c, bd);
    const int plo = g.bq[bd][4], phi = g.bq[bd][5];
    const int ulo = g.bq[bd][0], uhi = g.bq[bd][1], vlo = g.bq[bd][2], vhi = g.bq[bd][3];
    const int r = c / g.N1h, kx = c - r * g.N1h;
    const double kxv = g.k1x[kx], kzv = g.k1z[r];
    const double sgn = part ? 1.0 : -1.0;
    const double skx = sgn * kxv, skz = sgn * kzv;
    const double aRb = g.aRK[kRK - 1] + g.bRK[kRK - 1];
    const double dtirk = sc->dti / aRb;
    const double dt = sc->dt;
    const size_t ls = (size_t)nc * 2;
    const size_t ci = (size_t)c * 2 + part, co = (size_t)c * 2 + (part ^ 1);
    const double dskx = dtirk * skx, dskz = dtirk * skz;
    double y = 0.0;
    double vm = u2[(size_t)plo * ls + ci];
    // forward sweep: level qp's inputs (u1, u3 of the other part, v, dg1, dg2) in ring slot qp % D
    auto fetch_f = [&](int qp) {
      const int s_ = (qp - plo) % NS;
      const size_t e_ = (size_t)(qp + 1) * ls;
      cpa8(&RS(s_, 0), u1 + e_ + co); cpa8(&RS(s_, 1), u3 + e_ + co); cpa8(&RS(s_, 2), u2 + e_ + ci);
      cpa8(&RS(s_, 3), dg1 + (size_t)qp * nc + c); cpa8(&RS(s_, 4), dg2 + (size_t)qp * nc + c);
    };
#pragma unroll
    for (int s_ = 0; s_ < D; ++s_) {
      if (plo + s_ <= phi) fetch_f(plo + s_);
      cpa_commit();
    }
    for (int qp = plo; qp <= phi; ++qp) {
      cpa_wait<D - 1>();
      const int s_ = (qp - plo) % NS;
      const double ao = RS(s_, 0), wo = RS(s_, 1), v = RS(s_, 2), A1 = RS(s_, 3), a2p = RS(s_, 4);
      const double th = ptab[qp + 1];
      if (qp + D <= phi) fetch_f(qp + D);
      cpa_commit();
      double rhs = press_div(dskx, ao, dskz, wo, th, v - vm);
      vm = v;
      if (qp == plo && c == 0 && bd == 1) rhs = 0.0;
      y = (qp == plo) ? rhs * a2p : (rhs - A1 * y) * a2p;
      psi[(size_t)qp * ls + ci] = y;
    }
    cpa_wait<0>();
    __threadfence_block();  // the backward sweep's copies read psi written above by this thread
    const double dtrk = dt * aRb;
    const double kxd = dtrk * kxv, kzd = dtrk * kzv;
    double xn = y;
    double vup = 0.0, aup_o = 0.0, wup_o = 0.0;
    // backward sweep: level qp's inputs (psi, dg3, p, u1, u3, v of this part) in slot (phi - qp) % D
    auto fetch_b = [&](int qp) {
      const int s_ = (phi - qp) % NS;
      const size_t e_ = (size_t)(qp + 1) * ls + ci;
      cpa8(&RS(s_, 0), psi + (size_t)qp * ls + ci); cpa8(&RS(s_, 1), dg3 + (size_t)qp * nc + c);
      cpa8(&RS(s_, 2), p + (size_t)qp * ls + ci);
      cpa8(&RS(s_, 3), u1 + e_); cpa8(&RS(s_, 4), u3 + e_); cpa8(&RS(s_, 5), u2 + e_);
    };
#pragma unroll
    for (int s_ = 0; s_ < D; ++s_) {
      if (phi - s_ >= plo) fetch_b(phi - s_);
      cpa_commit();
    }
    for (int qp = phi; qp >= plo; --qp) {
      cpa_wait<D - 1>();
      const int s_ = (phi - qp) % NS;
      const int q = qp + 1;
      const size_t e = (size_t)q * ls;
      const double ps = RS(s_, 0), d3 = RS(s_, 1), pq = RS(s_, 2), uq = RS(s_, 3), wq = RS(s_, 4);
      double v = RS(s_, 5);
      const double thv = ptab[g.nu + q], thu1 = g.thud[qp + 2];
      if (qp - D >= plo) fetch_b(qp - D);
      cpa_commit();
      const double x = (qp == phi) ? xn : ps - d3 * xn;
      p[(size_t)qp * ls + ci] = pq + x;
      const double xo = __shfl_xor_sync(pm, x, 1);
      const double a = uq - sgn * kxd * xo;
      const double w = wq - sgn * kzd * xo;
      u1[e + ci] = a;
      u3[e + ci] = w;
      if (q <= vhi - 1) {
        v = v - thv * (xn - x);
        u2[e + ci] = v;
      }
      const double ao = __shfl_xor_sync(pm, a, 1), wo = __shfl_xor_sync(pm, w, 1);
      if (need_div && qp < phi) {
        const double dvp = press_div(skx, aup_o, skz, wup_o, thu1, vup - v);
        const double d2 = __dmul_rn(dvp, dvp);
        bits_max(dmax, __dadd_rn(d2, __shfl_xor_sync(pm, d2, 1)));
      }
      aup_o = ao; wup_o = wo; vup = v;
      xn = x;
    }
    cpa_wait<0>();
    if (need_div) {
      const double th = g.thud[plo + 1];
      const double vb = u2[(size_t)plo * ls + ci];
      const double dvp = press_div(skx, aup_o, skz, wup_o, th, vup - vb);
      const double d2 = __dmul_rn(dvp, dvp);
      bits_max(dmax, __dadd_rn(d2, __shfl_xor_sync(pm, d2, 1)));
    }
    if (bd <= 1) {
      u1[(size_t)ulo * ls + ci] = g.gwbc1 * u1[(size_t)(ulo + 1) * ls + ci];
      u3[(size_t)ulo * ls + ci] = g.gwbc3 * u3[(size_t)(ulo + 1) * ls + ci];
    }
    if (bd >= 1) {
      u1[(size_t)uhi * ls + ci] = g.gwbc1 * u1[(size_t)(uhi - 1) * ls + ci];
      u3[(size_t)uhi * ls + ci] = g.gwbc3 * u3[(size_t)(uhi - 1) * ls + ci];
    }
    u2[(size_t)vlo * ls + ci] = 0.0;
    u2[(size_t)vhi * ls + ci] = 0.0;
  }
#undef RS
  dmax = warp_max_bits(dmax);
  if ((threadIdx.x & 31) == 0) atomicMax(&sc->errbits, dmax);
}

// ============================================================================
// The pressure step of channels below LH_PRESS_SPLIT_COLS columns in three launches. An FP64 warp
// instruction holds its scheduler's half lane a clock for 64 cycles, so k_press3's sweep, which
// also forms its right-hand side and applies its result (12 FP64 instructions a level), is a
// chain of 768 cycles a level however few columns there are. Here the right-hand side and the
// corrections are element-wise over (column, chunk of levels), and the sweep keeps the
// recurrences: two dependent operations a level up, one down. The same operations in the same
// order per element, so the same results bit for bit, and no more FP64 operations; but psi
// crosses memory three more times (3.7 instead of 2.9 GB at 256 x 256 x 301), so larger channels
// keep the fused sweep. us a launch, fused -> the three launches together: 32 x 32 x 153 (544
// columns) 143 -> 59, 128 x 96 x 201 (6240) 190 -> 127. us a step, mixed form alone / among others:
// 128 x 128 x 201 (8320) 1784 / 1330 -> 1555 / 1263, 192 x 128 x 201 (12416) 2368 / 2004 -> 2184 /
// 2003, 192 x 192 x 201 (18624) 3025 / 2936 -> 3100 / 3038.
// In a batch the columns of all its channels count: they run beside each other, so the split route's
// extra launches and traffic cost what they cost a large channel (16 uneven channels: 4233 us a step
// split, 4214 fused; 4211 before there was a choice).
// ============================================================================
#define LH_PRESS_SPLIT_COLS 16384
#define LH_PL 8  // levels of a thread of the element-wise kernels (rolling v, psi)
__host__ __forceinline__ int press_chunks(const Geo &g) { return (g.np + LH_PL - 1) / LH_PL; }
// the third substep's faces below the chunks, [chunk][segment]
__host__ __forceinline__ size_t press_faces_bytes(const Geo &g) { return sizeof(double2) * press_chunks(g) * (size_t)g.nvc; }
// psi = dti/(a+b) div: thread = (column segment, chunk), both parts; vlow (third substep): the face
// below each chunk, [chunk][segment], for the corrections' divergence. u and w of mode (0,0), whose
// factors are zero, are not read (v is, in their place): the mean-flow correction may be writing u(0,0)
// beside this kernel.
__global__ void __launch_bounds__(128) k_press_rhs(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                   const double2 *__restrict__ u3, double2 *__restrict__ psi,
                                                   double2 *__restrict__ vlow, Geo g, const DevScalars *__restrict__ sc,
                                                   int kRK) {
  const int vc = blockIdx.x * 128 + threadIdx.x;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int plo = g.bq[bd][4], phi = g.bq[bd][5];
  const int q0 = plo + blockIdx.y * LH_PL;
  if (q0 > phi) return;
  const int nc = g.ncol, r = c / g.N1h, kx = c - r * g.N1h;
  const double dtirk = sc->dti / (g.aRK[kRK - 1] + g.bRK[kRK - 1]);
  const double dkx = dtirk * g.k1x[kx], dkz = dtirk * g.k1z[r];
  const double2 *uc = c != 0 ? u1 : u2, *wc = c != 0 ? u3 : u2;
  double2 vm = u2[(size_t)q0 * nc + c];
  if (vlow) vlow[(size_t)blockIdx.y * g.nvc + vc] = vm;
#pragma unroll
  for (int i = 0; i < LH_PL; ++i) {
    const int qp = q0 + i;
    if (qp > phi) break;
    const size_t e = (size_t)(qp + 1) * nc + c;
    const double2 a = uc[e], w = wc[e], v = u2[e];
    const double th = dtirk * g.thud[qp + 1];
    double2 rhs;
    rhs.x = press_div(-dkx, a.y, -dkz, w.y, th, v.x - vm.x);
    rhs.y = press_div(dkx, a.x, dkz, w.x, th, v.y - vm.y);
    if (qp == plo && c == 0 && bd == 1) rhs = make_double2(0.0, 0.0);
    psi[e - nc] = rhs;
    vm = v;
  }
}

// LUsolP in place on psi: lane = (column segment, part), U levels a batch, two batches ahead
#define LH_PS_U 4
__host__ __device__ constexpr int press_region() { return 3 * LH_PS_U * 3 | 1; }  // doubles of a thread's ring
__global__ void __launch_bounds__(32) k_press_sweep(double *__restrict__ psi, const double *__restrict__ dg1,
                                                    const double *__restrict__ dg2, const double *__restrict__ dg3, Geo g) {
  constexpr int U = LH_PS_U, BE = 3 * U;
  __shared__ double ring_all[32 * press_region()];
  double *ring = ring_all + threadIdx.x * press_region();
  const unsigned rs = (unsigned)__cvta_generic_to_shared(ring);
  const int tid = blockIdx.x * 32 + threadIdx.x, vc = tid >> 1, part = tid & 1;
  if (vc >= g.nvc) return;
  int c, bd;
  vcol_of(g, vc, c, bd);
  const int plo = g.bq[bd][4], phi = g.bq[bd][5];
  const size_t nc = g.ncol, ls = 2 * nc, ci = 2 * (size_t)c + part;
  double y = 0.0;
  {  // forward: a level's right-hand side, dg1, dg2
    const double *fs = psi + (size_t)plo * ls + ci, *f1 = dg1 + (size_t)plo * nc + c, *f2 = dg2 + (size_t)plo * nc + c;
    double *ps = psi + (size_t)plo * ls + ci;
    int left = phi - plo + 1;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (left > i) {
          cpa8s(dst + 24 * i, fs); cpa8s(dst + 24 * i + 8, f1); cpa8s(dst + 24 * i + 16, f2);
          fs += ls; f1 += nc; f2 += nc;
        }
      }
      left -= U;
      dst = dst == rs + 8 * 2 * BE ? rs : dst + 8 * BE;
      cpa_commit();
    };
    fetch();
    fetch();
    const double *h = ring;
    bool first = true;
    for (int n = phi - plo + 1; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        const double rhs = h[3 * i], A1 = h[3 * i + 1], a2p = h[3 * i + 2];
        y = (i == 0 && first) ? __dmul_rn(rhs, a2p) : __dmul_rn(__fma_rn(-A1, y, rhs), a2p);
        *ps = y;
        ps += ls;
      }
      first = false;
      h = h == ring + 2 * BE ? ring : h + BE;
    }
  }
  cpa_wait<0>();
  __threadfence();  // the copies below read what this thread stored above
  {  // backward from the level below the top: a level's y, dg3
    const double *fs = psi + (size_t)(phi - 1) * ls + ci, *f3 = dg3 + (size_t)(phi - 1) * nc + c;
    double *ps = psi + (size_t)(phi - 1) * ls + ci;
    int left = phi - plo;
    unsigned dst = rs;
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (left > i) {
          cpa8s(dst + 24 * i, fs); cpa8s(dst + 24 * i + 8, f3);
          fs -= ls; f3 -= nc;
        }
      }
      left -= U;
      dst = dst == rs + 8 * 2 * BE ? rs : dst + 8 * BE;
      cpa_commit();
    };
    fetch();
    fetch();
    const double *h = ring;
    for (int n = phi - plo; n > 0; n -= U) {
      fetch();
      cpa_wait<2>();
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i > 0 && n <= i) break;
        y = __fma_rn(-h[3 * i + 1], y, h[3 * i]);
        *ps = y;
        ps -= ls;
      }
      h = h == ring + 2 * BE ? ring : h + BE;
    }
  }
  cpa_wait<0>();
}

// p += psi, v_corr, ghost rows, v = 0 at the segment's ends: thread = (column segment, chunk)
template <bool DIV>
__global__ void __launch_bounds__(128) k_press_corr(double2 *__restrict__ u1, double2 *__restrict__ u2,
                                                    double2 *__restrict__ u3, double2 *__restrict__ p,
                                                    const double2 *__restrict__ psi, const double2 *__restrict__ vlow, Geo g,
                                                    DevScalars *sc, int kRK) {
  const int vc = blockIdx.x * 128 + threadIdx.x;
  unsigned long long dmax = 0ull;  // max |div|^2 as bits
  int c = 0, bd = 1, plo = 0, phi = -1;
  if (vc < g.nvc) {
    vcol_of(g, vc, c, bd);
    plo = g.bq[bd][4];
    phi = g.bq[bd][5];
  }
  const int q0 = plo + blockIdx.y * LH_PL;
  if (vc < g.nvc && q0 <= phi) {
    const int nc = g.ncol, r = c / g.N1h, kx = c - r * g.N1h;
    const int ulo = g.bq[bd][0], uhi = g.bq[bd][1], vlo = g.bq[bd][2], vhi = g.bq[bd][3];
    const double kxv = g.k1x[kx], kzv = g.k1z[r], dtrk = sc->dt * (g.aRK[kRK - 1] + g.bRK[kRK - 1]);
    const double kxd = dtrk * kxv, kzd = dtrk * kzv, dtd = dtrk * g.dd;
    const int q1 = min(q0 + LH_PL, phi + 1);  // levels q0 .. q1 - 1
    double2 x = psi[(size_t)q0 * nc + c], vm = make_double2(0.0, 0.0);
    if (DIV) {  // the face below, corrected here too (another thread stores it, hence the copy)
      vm = vlow[(size_t)blockIdx.y * g.nvc + vc];
      if (q0 > plo && q0 <= vhi - 1) {
        const double2 xm = psi[(size_t)(q0 - 1) * nc + c];
        const double t = dtd * g.thv[q0];
        vm.x = __fma_rn(-t, x.x - xm.x, vm.x);
        vm.y = __fma_rn(-t, x.y - xm.y, vm.y);
      }
    }
#pragma unroll
    for (int i = 0; i < LH_PL; ++i) {
      const int qp = q0 + i, q = qp + 1;
      if (qp >= q1) break;
      const size_t e = (size_t)q * nc + c;
      double2 pq = p[e - nc], a = u1[e], w = u3[e], v = u2[e], xn = x;
      if (qp < phi) xn = psi[e];
      pq.x = pq.x + x.x; pq.y = pq.y + x.y;
      a.x = __fma_rn(kxd, x.y, a.x); a.y = __fma_rn(-kxd, x.x, a.y);
      w.x = __fma_rn(kzd, x.y, w.x); w.y = __fma_rn(-kzd, x.x, w.y);
      p[e - nc] = pq;
      u1[e] = a;
      u3[e] = w;
      if (q <= vhi - 1) {
        const double t = dtd * g.thv[q];
        v.x = __fma_rn(-t, xn.x - x.x, v.x);
        v.y = __fma_rn(-t, xn.y - x.y, v.y);
        u2[e] = v;
      }
      if (DIV) {
        const double t = g.thud[q];
        const double dx = press_div(-kxv, a.y, -kzv, w.y, t, v.x - vm.x);
        const double dy = press_div(kxv, a.x, kzv, w.x, t, v.y - vm.y);
        bits_max(dmax, __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
        vm = v;
      }
      if (qp == plo) {
        if (bd <= 1) {
          u1[(size_t)ulo * nc + c] = cscale(a, g.gwbc1);
          u3[(size_t)ulo * nc + c] = cscale(w, g.gwbc3);
        }
        u2[(size_t)vlo * nc + c] = make_double2(0.0, 0.0);
      }
      if (qp == phi) {
        if (bd >= 1) {
          u1[(size_t)uhi * nc + c] = cscale(a, g.gwbc1);
          u3[(size_t)uhi * nc + c] = cscale(w, g.gwbc3);
        }
        u2[(size_t)vhi * nc + c] = make_double2(0.0, 0.0);
      }
      x = xn;
    }
  }
  if (DIV) {
    dmax = warp_max_bits(dmax);
    if ((threadIdx.x & 31) == 0) atomicMax(&sc->errbits, dmax);
  }
}

__global__ void k_reset_err(DevScalars *sc) {
  if (threadIdx.x == 0 && blockIdx.x == 0) sc->errbits = 0ull;
}

// max |div| of the current state (getini's divergence + error())
__global__ void __launch_bounds__(NTHR) k_divmax(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                 const double2 *__restrict__ u3, Geo g, DevScalars *sc) {
  const int vc = blockIdx.x * blockDim.x + threadIdx.x;
  double dmax = 0.0;
  if (vc < g.nvc) {
    int c, bd;
    vcol_of(g, vc, c, bd);
    const int r = c / g.N1h, kx = c - r * g.N1h;
    const double kxv = g.k1x[kx], kzv = g.k1z[r];
    for (int q = g.bq[bd][4] + 1; q <= g.bq[bd][5] + 1; ++q) {
      const size_t o = (size_t)q * g.ncol + c;
      const double2 a = u1[o], w = u3[o], v = u2[o], vm = u2[o - g.ncol];
      const double th = g.dd * g.thu[q];
      double2 dv;
      dv.x = (-kxv * a.y + -kzv * w.y) + th * (v.x - vm.x);
      dv.y = (kxv * a.x + kzv * w.x) + th * (v.y - vm.y);
      dmax = nmax(dmax, dv.x * dv.x + dv.y * dv.y);
    }
  }
  dmax = warp_max(dmax);
  if ((threadIdx.x & 31) == 0) atomic_max_pos(&sc->errbits, dmax);
}

// err = max |div| (errbits holds the maximum of |div|^2)
__global__ void k_err_from_bits(DevScalars *sc) {
  if (threadIdx.x == 0 && blockIdx.x == 0) sc->err = sqrt(__longlong_as_double((long long)sc->errbits));
}

// one band's host cfield [k][l] (staged) <-> device [lev0 + l][cols[k]]; put = 1 writes the device
// ============================================================================
// The other sums of the statistics step, formed from the spectral state (FP64 in both
// forms; launched on request only, LH_STAT_THREADS threads per block).
// ============================================================================
#define LH_STAT_THREADS 256
// omega_x = -der_z_N(v) + der_yv_h_wx(w) at every v level (FOU3D.f90:300-327), and its
// plane sums over the N1 x N2 points of four_to_phys_N (stats.f90:56-63), by Parseval:
// sum f = N1 N2 Re c(0,0); sum f^2 = N1 N2 [ sum over 0 < kx < N1/2 of 2 |c|^2, plus for
// kx = 0 and N1/2 (whose Im the real transform drops) 1/2 |c(kz)|^2 + 1/2 Re c(kz) c(-kz) ].
// One block per level; the level's plane class gives N1, N2 (wall bands: nhw, n2w; the
// core band: nhc, n2c). pl: [11][nu], quantities 9 and 10.
__device__ __forceinline__ double2 wx_mode(const double2 *__restrict__ u2, const double2 *__restrict__ u3,
                                           const Geo &g, int q, int c, int fr, double fy) {
  const double2 v = u2[(size_t)q * g.ncolF + c];
  const double2 a = u3[(size_t)(q + 1) * g.ncolF + c], b = u3[(size_t)q * g.ncolF + c];
  const double kz = g.k1z[fr];
  // -(i kz v) + (a - b) fy
  return make_double2(kz * v.y + (a.x - b.x) * fy, -kz * v.x + (a.y - b.y) * fy);
}
__global__ void __launch_bounds__(LH_STAT_THREADS) k_wx_stats(const double2 *__restrict__ u2, const double2 *__restrict__ u3,
                                                     Geo g, int nhc, int n2c, double *__restrict__ pl) {
  __shared__ double red[LH_STAT_THREADS / 32][2];
  const int q = blockIdx.x;
  const int j = q - g.dny;
  const bool fine = !g.mb || j <= g.N3[1] || j > g.N3[2];
  const int nh = fine ? g.N1hF : nhc, n2 = fine ? g.N2F : n2c, n1 = 2 * (nh - 1);
  const double fy = g.thv[q] * g.dd;
  double s = 0.0, s2 = 0.0;
  for (int e = threadIdx.x; e < nh * n2; e += blockDim.x) {
    const int r = e / nh, kx = e - r * nh;
    const int fr = r < n2 / 2 ? r : r + g.N2F - n2;
    const double2 cv = wx_mode(u2, u3, g, q, fr * g.N1hF + kx, fr, fy);
    const double m2 = cv.x * cv.x + cv.y * cv.y;
    if (kx == 0 || kx == nh - 1) {
      const int rm = (n2 - r) % n2;
      const int frm = rm < n2 / 2 ? rm : rm + g.N2F - n2;
      const double2 cm = wx_mode(u2, u3, g, q, frm * g.N1hF + kx, frm, fy);
      s2 += 0.5 * m2 + 0.5 * (cv.x * cm.x - cv.y * cm.y);
      if (e == 0) s = cv.x;
    } else {
      s2 += 2.0 * m2;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5][0] = s; red[threadIdx.x >> 5][1] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < LH_STAT_THREADS / 32; ++w) { a += red[w][0]; b += red[w][1]; }
    const double nn = (double)n1 * (double)n2;
    pl[9 * (size_t)g.nu + q] += nn * a;
    pl[10 * (size_t)g.nu + q] += nn * b;
  }
}

// Pressure plane sums (stats.f90:43-50 over the physical pressure): one block per p level q
// (reference level j = q + 1 - dny). Wall-band planes (j <= N(4,1)-1, j >= N(4,2)+2, the
// pgrid plane ranges of the outer bands) hold every mode of the wall-band grid, on the
// Gf = G1 x G2 dealiased points; core planes the long columns (nhc x n2c) on Gc points.
// Parseval on the padded grid: sum p = G p(0,0); sum p^2 = G (sum over kx >= 1 of 2|p|^2,
// kx = N1/2 included, + the kx = 0 column's Hermitian part, whose row -N2/2 has no mirror).
// pp: [2][np].
__global__ void __launch_bounds__(LH_STAT_THREADS) k_p_stats(const double2 *__restrict__ p, Geo g, int nhc, int n2c,
                                                    double Gf, double Gc, double *__restrict__ pp) {
  __shared__ double red[LH_STAT_THREADS / 32][2];
  const int q = blockIdx.x;
  const int j = q + 1 - g.dny;
  const bool fine = !g.mb || j <= g.N4[1] - 1 || j >= g.N4[2] + 2;
  const int nh = fine ? g.N1hF : nhc, n2 = fine ? g.N2F : n2c;
  const double2 *P = p + (size_t)q * g.ncolF;
  double s = 0.0, s2 = 0.0;
  for (int e = threadIdx.x; e < nh * n2; e += blockDim.x) {
    const int r = e / nh, kx = e - r * nh;
    const int fr = r < n2 / 2 ? r : r + g.N2F - n2;
    const double2 a = P[fr * g.N1hF + kx];
    const double m2 = a.x * a.x + a.y * a.y;
    if (kx > 0) {
      s2 += 2.0 * m2;
    } else if (r == n2 / 2) {
      s2 += 0.5 * m2;
    } else {
      const int rm = (n2 - r) % n2;
      const int frm = rm < n2 / 2 ? rm : rm + g.N2F - n2;
      const double2 b = P[frm * g.N1hF];
      s2 += 0.5 * m2 + 0.5 * (a.x * b.x - a.y * b.y);
      if (r == 0) s = a.x;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5][0] = s; red[threadIdx.x >> 5][1] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < LH_STAT_THREADS / 32; ++w) { a += red[w][0]; b += red[w][1]; }
    const double G = fine ? Gf : Gc;
    pp[q] += G * a;
    pp[(size_t)g.np + q] += G * b;
  }
}

// Spectral planes of the tile-conditioned P and omega_x sums: plane b of the chunk is
// list[b] = (kind, level, j1): kind 0 copies p level `level`; kind 1 forms omega_x at v level
// `level` (-i kz v + (w(q+1) - w(q)) dthdyv ddthetavi, FOU3D.f90:300-327). spec: [nb][ncolF].
__global__ void __launch_bounds__(LH_STAT_THREADS) k_cond_spec(const double2 *__restrict__ u2, const double2 *__restrict__ u3,
                                                      const double2 *__restrict__ p, Geo g,
                                                      const int4 *__restrict__ list, double2 *__restrict__ spec) {
  const int4 d = list[blockIdx.y];
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= (size_t)g.ncolF) return;
  double2 *o = spec + (size_t)blockIdx.y * g.ncolF + c;
  if (d.x == 0) {
    *o = p[(size_t)d.y * g.ncolF + c];
  } else {
    *o = wx_mode(u2, u3, g, d.y, (int)c, (int)(c / g.N1hF), g.thv[d.y] * g.dd);
  }
}

// conddown1 / condup1 with xsign 1 (stats.f90:109-138, 178-210) of the chunk's physical
// planes (phys [nb][G2][G1]): one thread per tile position (i, k), summing the value and
// its square over the ntx x ntz tiles into the pair 2 kind, 2 kind + 1 of
// cd4 [4][ncl1][dnz][dnx] at level j1 (bottom and top planes of a level add into one cell).
__global__ void __launch_bounds__(LH_STAT_THREADS) k_cond_phys(const double *__restrict__ phys, const int4 *__restrict__ list,
                                                      int G1, int G2, int dnx, int dnz, int ncl1,
                                                      double *__restrict__ cd4) {
  const int4 d = list[blockIdx.y];
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= dnx * dnz) return;
  const int k = cell / dnx, i = cell - k * dnx;
  const double *f = phys + (size_t)blockIdx.y * G1 * G2;
  double s = 0.0, s2 = 0.0;
  for (int l = k; l < G2; l += dnz)
    for (int m = i; m < G1; m += dnx) {
      const double x = f[(size_t)l * G1 + m];
      s += x;
      s2 += x * x;
    }
  const size_t lv = (size_t)dnz * dnx;
  atomicAdd(&cd4[((size_t)(2 * d.x) * ncl1 + d.z) * lv + cell], s);
  atomicAdd(&cd4[((size_t)(2 * d.x + 1) * ncl1 + d.z) * lv + cell], s2);
}

// spectra (spectra.f90:1-56): band 2's levels x the long columns (cols[0..nlong)),
// sp(level, column) += |u|^2 (U, V, W, P) and Re u1 Re v + Im u1 Im v with v interpolated
// to the centres (interp_v, FOU3D.f90:427-474; band 2's end levels extrapolated with
// gridweighting_interp(2, 1:2) = gi0, gi1). sp: 5 arrays [level][nlong] at offsets off[].
__device__ __forceinline__ double2 itp_v(const double2 *__restrict__ u2, const Geo &g, int q, int c) {
  const double2 a = u2[(size_t)q * g.ncolF + c], b = u2[(size_t)(q - 1) * g.ncolF + c];
  const double w0 = g.yu[q] - g.yv[q - 1], w1 = g.yv[q] - g.yu[q], d = g.yv[q] - g.yv[q - 1];
  return make_double2((w0 * a.x + w1 * b.x) / d, (w0 * a.y + w1 * b.y) / d);
}
__global__ void __launch_bounds__(LH_STAT_THREADS) k_spectra(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                    const double2 *__restrict__ u3, const double2 *__restrict__ p,
                                                    Geo g, const int *__restrict__ cols, int nlong, double gi0,
                                                    double gi1, double *__restrict__ sp) {
  const int ulo = g.bq[1][0], uhi = g.bq[1][1], vlo = g.bq[1][2], vhi = g.bq[1][3];
  const int plo = g.bq[1][4], phi = g.bq[1][5];
  const int nlu = uhi - ulo + 1, nlv = vhi - vlo + 1, nlp = phi - plo + 1;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nlu * nlong) return;
  const int l = (int)(i / nlong), k = (int)(i - (size_t)l * nlong);
  const int c = cols[k];
  const size_t nc = g.ncolF;
  double *sU = sp, *sV = sU + (size_t)nlu * nlong, *sW = sV + (size_t)nlv * nlong, *sUV = sW + (size_t)nlu * nlong;
  double *sP = sUV + (size_t)nlu * nlong;
  const int q = ulo + l;
  const double2 a = u1[q * nc + c], w = u3[q * nc + c];
  double2 v;
  if (q > ulo && q < uhi) v = itp_v(u2, g, q, c);
  else if (q == ulo) {
    const double2 i1 = itp_v(u2, g, ulo + 1, c), b = u2[(size_t)vlo * nc + c];
    v = make_double2(gi0 * (b.x - i1.x) + i1.x, gi0 * (b.y - i1.y) + i1.y);
  } else {
    const double2 i2 = itp_v(u2, g, uhi - 1, c), b = u2[(size_t)vhi * nc + c];
    v = make_double2(gi1 * (b.x - i2.x) + i2.x, gi1 * (b.y - i2.y) + i2.y);
  }
  sU[i] = sU[i] + a.x * a.x + a.y * a.y;
  sW[i] = sW[i] + w.x * w.x + w.y * w.y;
  sUV[i] = sUV[i] + a.x * v.x + a.y * v.y;
  if (l < nlv) {
    const double2 b = u2[(size_t)(vlo + l) * nc + c];
    sV[i] = sV[i] + b.x * b.x + b.y * b.y;
  }
  if (l < nlp) {
    const double2 b = p[(size_t)(plo + l) * nc + c];
    sP[i] = sP[i] + b.x * b.x + b.y * b.y;
  }
}

// slip statistics (sl_stats2.f90:33-121, inst_sl_stats.f90:1-62) at the wall faces
// jlim(1, vgrid, 2) and jlim(2, vgrid, 2) (v array indices qb, qt), every wall-grid column:
// u1 and u3 interpolated to the face (interp_u) and (u(q+1) - u(q)) dthdyv ddthetavi,
// negated at the top. out: [2][4][ncolF]; acc: add (sl_stats) or store (inst_sl_stats).
__global__ void __launch_bounds__(LH_STAT_THREADS) k_slip(const double2 *__restrict__ u1, const double2 *__restrict__ u3, Geo g,
                                                 int qb, int qt, double2 *__restrict__ out, int acc) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.ncolF) return;
  const size_t nc = g.ncolF;
  for (int w = 0; w < 2; ++w) {
    const int q = w ? qt : qb;
    const double sg = w ? -1.0 : 1.0;
    const double fy = g.thv[q] * g.dd;
    const double ya = g.yu[q], yb = g.yu[q + 1], yv = g.yv[q];
    for (int f = 0; f < 2; ++f) {
      const double2 *u = f ? u3 : u1;
      const double2 hi = u[(size_t)(q + 1) * nc + c], lo = u[(size_t)q * nc + c];
      const double2 it = make_double2(((yv - ya) * hi.x + (yb - yv) * lo.x) / (yb - ya),
                                      ((yv - ya) * hi.y + (yb - yv) * lo.y) / (yb - ya));
      const double2 dy = make_double2(sg * ((hi.x - lo.x) * fy), sg * ((hi.y - lo.y) * fy));
      double2 *o0 = out + ((size_t)(w * 4 + 2 * f) * nc + c), *o1 = o0 + nc;
      if (acc) {
        *o0 = make_double2(o0->x + it.x, o0->y + it.y);
        *o1 = make_double2(o1->x + dy.x, o1->y + dy.y);
      } else {
        *o0 = it;
        *o1 = dy;
      }
    }
  }
}

__global__ void k_band_io(double2 *__restrict__ dev, double2 *__restrict__ stage, const int *__restrict__ cols,
                          int ncb, int nlev, int lev0, int ncol, int put) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)ncb * nlev) return;
  const int k = (int)(i / nlev), l = (int)(i - (size_t)k * nlev);
  double2 *d = dev + (size_t)(lev0 + l) * ncol + cols[k];
  if (put) *d = stage[i];
  else stage[i] = *d;
}

// host cfield [col][lev] <-> device [lev][col] (complex; real for the spectra), tiled transpose
template <typename V>
__global__ void k_transpose(const V *__restrict__ src, V *__restrict__ dst, int rows, int cols) {
  __shared__ V tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int rr = by + i, cc = bx + threadIdx.x;
    if (rr < rows && cc < cols) tile[i][threadIdx.x] = src[(size_t)rr * cols + cc];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int rr = bx + i, cc = by + threadIdx.x;  // dst is cols x rows
    if (rr < cols && cc < rows) dst[(size_t)rr * rows + cc] = tile[threadIdx.x][i];
  }
}

// ============================================================================
// Plane transforms of lh_four_to_phys_noalloc (FP64 Stockham: its scratch holds FP64 tables
// that every call makes on the device). spec [plane][N2][N1h] complex128, phys [plane][G2][G1]
// double, scratch A [plane][l][kx]. The handles' leaves run in lh_fxpass.cuh.
// ============================================================================
template <typename T, int N>
__global__ void __launch_bounds__(NTHR) k_spec_zinv(const double2 *__restrict__ spec, typename C2<T>::t *__restrict__ A,
                                                    Geo g, const typename C2<T>::t *__restrict__ twz) {
  typedef typename C2<T>::t V;
  constexpr int KB = kb_zinv<V>(N);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *b0 = reinterpret_cast<V *>(smem_raw);
  V *b1 = b0 + KB * N;
  const int pl = blockIdx.y, kx0 = blockIdx.x * KB;
  for (int i = threadIdx.x; i < KB * N; i += blockDim.x) b0[i] = czero<V>();
  __syncthreads();
  const double2 *S = spec + (size_t)pl * g.ncol;
  for (int idx = threadIdx.x; idx < g.N2 * KB; idx += blockDim.x) {
    const int r = idx / KB, kk = idx - r * KB, kx = kx0 + kk;
    if (kx >= g.N1h) continue;
    const double2 val = S[r * g.N1h + kx];
    V v; v.x = to_t<T>(val.x); v.y = to_t<T>(val.y);
    b0[prow(g, r) * KB + kk] = v;
  }
  __syncthreads();
  V *res = line_fft<true, N, KB, true>(b0, b1, twz);
  V *dst = A + (size_t)pl * N * g.N1h;
  for (int idx = threadIdx.x; idx < N * KB; idx += blockDim.x) {
    const int l = idx / KB, kk = idx - l * KB, kx = kx0 + kk;
    if (kx < g.N1h) dst[(size_t)l * g.N1h + kx] = res[l * KB + kk];
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(NTHR) k_xinv_phys(const typename C2<T>::t *__restrict__ A, double *__restrict__ phys,
                                                    Geo g, const typename C2<T>::t *__restrict__ twx) {
  typedef typename C2<T>::t V;
  constexpr int PB = 4 * pb_xpass<V>(N);
  constexpr int G1 = N, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G2 = g.G2, N1h = g.N1h;
  V *b0 = reinterpret_cast<V *>(smem_raw);
  V *b1 = b0 + PB * G1;
  const int pl = blockIdx.y, l0 = blockIdx.x * PB * 2;
  const int npairs = min(PB, (G2 - l0) / 2);
  const V *Ap = A + (size_t)pl * G2 * N1h;
  for (int idx = threadIdx.x; idx < PB * G1; idx += blockDim.x) {
    const int pb = idx / G1, m = idx - pb * G1;
    V z = czero<V>();
    if (pb < npairs) {
      const int l = l0 + 2 * pb;
      int k = m; bool cj = false;
      if (m > H) { k = G1 - m; cj = true; }
      if (k < N1h) {
        V a = Ap[(size_t)l * N1h + k], b = Ap[(size_t)(l + 1) * N1h + k];
        if (k == 0 || k == H) { a.y = 0; b.y = 0; }
        if (!cj) { z.x = a.x - b.y; z.y = a.y + b.x; } else { z.x = a.x + b.y; z.y = -a.y + b.x; }
      }
    }
    b0[idx] = z;
  }
  __syncthreads();
  V *res = line_fft<true, N, PB, false>(b0, b1, twx);
  double *P = phys + (size_t)pl * G2 * G1;
  for (int idx = threadIdx.x; idx < PB * G1; idx += blockDim.x) {
    const int pb = idx / G1, m = idx - pb * G1;
    if (pb >= npairs) continue;
    const int l = l0 + 2 * pb;
    P[(size_t)l * G1 + m] = to_d(res[idx].x);
    P[(size_t)(l + 1) * G1 + m] = to_d(res[idx].y);
  }
}

// ============================================================================
// Immersed boundaries (FOU3D.f90:806-998): assemble du at the listed levels,
// then (after the inverse transform) the forcing at the solid points.
// duib layout: [ibslot][field 0..2][col], complex128 (FP64 form) or complex64 (mixed form, whose
// values are FP32); ib levels of u (fields 0, 2) and v (1).
// ============================================================================
template <typename TN>
__global__ void __launch_bounds__(NTHR) k_ib_du(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                const double2 *__restrict__ u3, typename C2<TN>::t *__restrict__ Nu1o,
                                                typename C2<TN>::t *__restrict__ Nu2o, typename C2<TN>::t *__restrict__ Nu3o,
                                                const typename C2<TN>::t *__restrict__ N1xz, const typename C2<TN>::t *__restrict__ N2xz,
                                                const typename C2<TN>::t *__restrict__ N3xz, const typename C2<TN>::t *__restrict__ uvf,
                                                const typename C2<TN>::t *__restrict__ vvc, const typename C2<TN>::t *__restrict__ wvf,
                                                const double2 *__restrict__ p, double2 *__restrict__ duib,
                                                const int *__restrict__ iblev, int nib, Geo g,
                                                const DevScalars *__restrict__ sc, int kRK) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y;  // ib slot
  const int nc = g.ncol;
  if (c >= nc || s >= nib) return;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const double k2x = g.k2x[kx], k2z = g.k2z[r];
  const double C1 = g.aRK[kRK - 1] / g.Re, C2 = -g.cRK[kRK - 1], dR = g.dRK[kRK - 1];
  const double G = -g.gRK[kRK - 1];
  const int qu = iblev[2 * s], qv = iblev[2 * s + 1];
  if (qu > 0) {  // u and w at u-level qu
    const double *d0 = g.d2u, *d1 = g.d2u + g.nu, *d2 = g.d2u + 2 * g.nu;
    const size_t o = (size_t)qu * nc + c;
    const double a = d0[qu], dg = (k2x + k2z) + d1[qu], cc = d2[qu];
    const double2 pj = p[(size_t)(qu - 1) * nc + c];
    const double C3x = -dR * g.k1x[kx], C3z = -dR * g.k1z[r];
    const double th = g.thu[qu];
    for (int f = 0; f < 2; ++f) {
      const double2 *U = f ? u3 : u1;
      typename ::C2<TN>::t *No = f ? Nu3o : Nu1o;
      const typename ::C2<TN>::t *X = f ? N3xz : N1xz;
      const typename ::C2<TN>::t *F = f ? wvf : uvf;
      const double C3 = f ? C3z : C3x;
      const double2 um = U[o - nc], u0 = U[o], up = U[o + nc];
      double2 L;
      L.x = (a * um.x + dg * u0.x) + cc * up.x; L.y = (a * um.y + dg * u0.y) + cc * up.y;
      const double2 no = ld2(No[o]);
      double2 du;
      du.x = (C1 * L.x + C2 * no.x) + (-C3 * pj.y);
      du.y = (C1 * L.y + C2 * no.y) + (C3 * pj.x);
      if (f == 0 && c == 0) du.x += -dR * sc->mpgx;
      const double2 x = ld2(X[o]), fq = ld2(F[o]), fm = ld2(F[o - nc]);
      double2 n;
      n.x = x.x + (fq.x - fm.x) * th * g.dd; n.y = x.y + (fq.y - fm.y) * th * g.dd;
      No[o].x = n.x; No[o].y = n.y;  // N of this substep (the next substep's -cRK term)
      du.x = du.x + G * n.x; du.y = du.y + G * n.y;
      duib[((size_t)s * 3 + (f ? 2 : 0)) * nc + c] = du;
    }
  }
  if (qv > 0) {
    const double *d0 = g.d2v, *d1 = g.d2v + g.nv, *d2 = g.d2v + 2 * g.nv;
    const size_t o = (size_t)qv * nc + c;
    const double a = d0[qv], dg = (k2x + k2z) + d1[qv], cc = d2[qv];
    const double2 vm = u2[o - nc], v0 = u2[o], vp = u2[o + nc];
    double2 L;
    L.x = (a * vm.x + dg * v0.x) + cc * vp.x; L.y = (a * vm.y + dg * v0.y) + cc * vp.y;
    const double C3 = -dR * g.dd * g.thv[qv];
    const double2 pp = p[(size_t)qv * nc + c], pm = p[(size_t)(qv - 1) * nc + c];
    const double2 no = ld2(Nu2o[o]);
    double2 du;
    du.x = (C1 * L.x + C2 * no.x) + C3 * (pp.x - pm.x);
    du.y = (C1 * L.y + C2 * no.y) + C3 * (pp.y - pm.y);
    const double th = g.thv[qv];
    const double2 x = ld2(N2xz[o]), vp1 = ld2(vvc[o + nc]), vq = ld2(vvc[o]);
    double2 n;
    n.x = x.x + (vp1.x - vq.x) * th * g.dd; n.y = x.y + (vp1.y - vq.y) * th * g.dd;
    Nu2o[o].x = n.x; Nu2o[o].y = n.y;
    du.x = du.x + G * n.x; du.y = du.y + G * n.y;
    duib[((size_t)s * 3 + 1) * nc + c] = du;
  }
}

// Mixed form of k_ib_du: the same right-hand side in FP32 (FP64 neighbour
// differences for the Laplacian, integer-pipe conversions), N and du stored in FP32.
__global__ void __launch_bounds__(NTHR, LH_IBDU_MINB) k_ib_du_mx(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                   const double2 *__restrict__ u3, float2 *__restrict__ Nu1o,
                                                   float2 *__restrict__ Nu2o, float2 *__restrict__ Nu3o,
                                                   const float2 *__restrict__ N1xz, const float2 *__restrict__ N2xz,
                                                   const float2 *__restrict__ N3xz, const float2 *__restrict__ uvf,
                                                   const float2 *__restrict__ vvc, const float2 *__restrict__ wvf,
                                                   const double2 *__restrict__ p, float2 *__restrict__ duib,
                                                   const int *__restrict__ iblev, int nib, Geo g,
                                                   const DevScalars *__restrict__ sc, int kRK) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y;
  const int nc = g.ncol;
  if (c >= nc || s >= nib) return;
  const int r = c / g.N1h, kx = c - r * g.N1h;
  const float k2f = (float)(g.k2x[kx] + g.k2z[r]);
  const float C1 = (float)(g.aRK[kRK - 1] / g.Re), C2 = (float)(-g.cRK[kRK - 1]);
  const double dR = g.dRK[kRK - 1];
  const float dRf = (float)dR;
  const float G = (float)(-g.gRK[kRK - 1]);
  const float dd = (float)g.dd;
  const int qu = iblev[2 * s], qv = iblev[2 * s + 1];
  // every input of the thread is loaded before the first store, so that the latencies of the
  // u-level and v-level loads overlap (the kernel is bound by them, not by bandwidth)
  const size_t ou = (size_t)qu * nc + c, ov = (size_t)qv * nc + c;
  double2 um[2], u0[2], up[2], pj, vm, v0, vp, pp, pm;
  float2 no[2], xq[2], fq[2], fm[2], nov, xv, vp1, vq;
  double mpgx = 0.0;
  if (qu > 0) {
    pj = p[(size_t)(qu - 1) * nc + c];
    if (c == 0) mpgx = sc->mpgx;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const double2 *U = f ? u3 : u1;
      const float2 *F = f ? wvf : uvf;
      um[f] = U[ou - nc]; u0[f] = U[ou]; up[f] = U[ou + nc];
      no[f] = (f ? Nu3o : Nu1o)[ou];
      xq[f] = (f ? N3xz : N1xz)[ou];
      fq[f] = F[ou]; fm[f] = F[ou - nc];
    }
  }
  if (qv > 0) {
    vm = u2[ov - nc]; v0 = u2[ov]; vp = u2[ov + nc];
    pp = p[(size_t)qv * nc + c]; pm = p[(size_t)(qv - 1) * nc + c];
    nov = Nu2o[ov]; xv = N2xz[ov]; vp1 = vvc[ov + nc]; vq = vvc[ov];
  }
  if (qu > 0) {
    const int nu = g.nu;
    const float a = g.d2uf[qu], cc = g.d2uf[2 * nu + qu], sdg = g.sdgu[qu] + k2f;
    const float pjx = d2f_alu(pj.x), pjy = d2f_alu(pj.y);
    const float C3x = (float)(-dR * g.k1x[kx]), C3z = (float)(-dR * g.k1z[r]);
    const float th = g.thuf[qu];
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const float C3 = f ? C3z : C3x;
      float2 L;
      L.x = a * d2f_alu(um[f].x - u0[f].x) + cc * d2f_alu(up[f].x - u0[f].x) + sdg * d2f_alu(u0[f].x);
      L.y = a * d2f_alu(um[f].y - u0[f].y) + cc * d2f_alu(up[f].y - u0[f].y) + sdg * d2f_alu(u0[f].y);
      float2 du;
      du.x = (C1 * L.x + C2 * no[f].x) + (-C3 * pjy);
      du.y = (C1 * L.y + C2 * no[f].y) + (C3 * pjx);
      if (f == 0 && c == 0) du.x += (float)(-dR * mpgx);
      float2 n;
      n.x = xq[f].x + (fq[f].x - fm[f].x) * th * dd; n.y = xq[f].y + (fq[f].y - fm[f].y) * th * dd;
      (f ? Nu3o : Nu1o)[ou] = n;
      du.x += G * n.x; du.y += G * n.y;
      duib[((size_t)s * 3 + (f ? 2 : 0)) * nc + c] = du;
    }
  }
  if (qv > 0) {
    const int nv = g.nv;
    const float a = g.d2vf[qv], cc = g.d2vf[2 * nv + qv], sdg = g.sdgv[qv] + k2f;
    float2 L;
    L.x = a * d2f_alu(vm.x - v0.x) + cc * d2f_alu(vp.x - v0.x) + sdg * d2f_alu(v0.x);
    L.y = a * d2f_alu(vm.y - v0.y) + cc * d2f_alu(vp.y - v0.y) + sdg * d2f_alu(v0.y);
    const float C3 = -dRf * dd * g.thvf[qv];
    float2 du;
    du.x = (C1 * L.x + C2 * nov.x) + C3 * (d2f_alu(pp.x) - d2f_alu(pm.x));
    du.y = (C1 * L.y + C2 * nov.y) + C3 * (d2f_alu(pp.y) - d2f_alu(pm.y));
    const float th = g.thvf[qv];
    float2 n;
    n.x = xv.x + (vp1.x - vq.x) * th * dd; n.y = xv.y + (vp1.y - vq.y) * th * dd;
    Nu2o[ov] = n;
    du.x += G * n.x; du.y += G * n.y;
    duib[((size_t)s * 3 + 1) * nc + c] = du;
  }
}

// ============================================================================
// Immersed-boundary forcing in one x pass (imm_bounds_u/v, FOU3D.f90:806-998): the rows
// of du's planes (z pass done, A layout) go to physical space, the forced points of the
// rows are overwritten with Kib/dt (A u(i1,k1,j1) - u(i,k,j)) from the captured physical
// velocities, and the rows go back (B layout for the z pass). Forced points come as
// records sorted by (plane, row): rec_off[plane * G2 + row] .. rec_off[... + 1];
// cap [capslot][field][G2][G1] holds the physical u, v, w the x pass captured, in the
// transform precision (FP32 in the mixed form: the values are FP32 there). Here the mixed
// form's kernel; the FP64 form's is k_ib_xforce_fx.
// ============================================================================
struct IbRec {
  int i, k;        // 0-based point of the plane: x index, row
  long long src;   // cap offset of u at the point
  long long ref;   // cap offset of u at the reference point (i1, k1, j1)
  double A;
};
template <int N>
__global__ void __launch_bounds__(NTHR, LH_IBX_MINB) k_ib_xforce(const float2 *__restrict__ A, float2 *__restrict__ B,
                                                    Geo g, const float2 *__restrict__ twx,
                                                    const IbRec *__restrict__ rec, const int *__restrict__ rec_off,
                                                    const float *__restrict__ cap, const DevScalars *__restrict__ sc) {
  typedef float T;
  typedef float2 V;
  constexpr int PB = 4 * pb_xpass<V>(N);
  constexpr int G1 = N, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G2 = g.G2, N1h = g.N1h;
  V *b0 = reinterpret_cast<V *>(smem_raw);
  V *b1 = b0 + PB * G1;
  const int pl = blockIdx.y, l0 = blockIdx.x * PB * 2;
  const int npairs = min(PB, (G2 - l0) / 2);
  const V *Ap = A + (size_t)pl * G2 * N1h;
  // one work item per retained x-mode (N1h = G1 / 3 + 1), the dealiasing band zeroed
  constexpr int NK = G1 / 3 + 1, NZ = G1 - 2 * NK + 1;
  static_assert(NK <= H, "retained x-modes below the Nyquist index");
  for (int idx = threadIdx.x; idx < PB * NK; idx += blockDim.x) {
    const int pb = idx / NK, k = idx - pb * NK;
    V zd = czero<V>(), zc = czero<V>();
    if (pb < npairs) {
      const int l = l0 + 2 * pb;
      V a = Ap[(size_t)l * NK + k], b = Ap[(size_t)(l + 1) * NK + k];
      if (k == 0) { a.y = 0; b.y = 0; }
      zd.x = a.x - b.y; zd.y = a.y + b.x;
      zc.x = a.x + b.y; zc.y = -a.y + b.x;
    }
    b0[pb * G1 + k] = zd;
    if (k > 0) b0[pb * G1 + G1 - k] = zc;
  }
  for (int idx = threadIdx.x; idx < PB * NZ; idx += blockDim.x) {
    const int pb = idx / NZ, m = idx - pb * NZ;
    b0[pb * G1 + NK + m] = czero<V>();
  }
  __syncthreads();
  V *res = line_fft<true, N, PB, false>(b0, b1, twx);
  V *oth = (res == b0) ? b1 : b0;
  {
    const float Kibdtf = d2f_alu(g.Kib / sc->dt);
    const int r0 = rec_off[(size_t)pl * G2 + l0], r1 = rec_off[(size_t)pl * G2 + l0 + 2 * npairs];
    for (int e = r0 + threadIdx.x; e < r1; e += blockDim.x) {
      const IbRec R = rec[e];
      // one rounding of A u_ref - u (fused), one of the scaling
      const float val = Kibdtf * fmaf(d2f_alu(R.A), cap[R.ref], -cap[R.src]);
      const int rr = R.k - l0;
      V *z = res + (rr >> 1) * G1 + R.i;
      if (rr & 1) z->y = val;
      else z->x = val;
    }
  }
  __syncthreads();
  V *fres = line_fft<false, N, PB, false>(res, oth, twx);
  const T s1 = (T)1 / (T)G1;
  for (int idx = threadIdx.x; idx < PB * 2 * N1h; idx += blockDim.x) {
    const int k = idx % N1h, rest = idx / N1h;
    const int half = rest & 1, pb = rest >> 1;
    if (pb >= npairs) continue;
    const V *L = fres + pb * G1;
    const V z = L[k], zc = cconj(L[k == 0 ? 0 : G1 - k]);
    V o;
    if (!half) { o.x = (T)0.5 * (z.x + zc.x) * s1; o.y = (T)0.5 * (z.y + zc.y) * s1; }
    else { o.x = (T)0.5 * (z.y - zc.y) * s1; o.y = (T)-0.5 * (z.x - zc.x) * s1; }
    if (k == 0) o.y = 0;
    B[((size_t)pl * G2 + l0 + 2 * pb + half) * N1h + k] = o;
  }
}


