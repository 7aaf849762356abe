// lh_fx.cuh — the FP64 form's transforms in 64-bit block fixed point.
//
// GB300 issues 2 FP64 operations per clock and SM; a Stockham pass in FP64 kept that pipe
// 85 % busy with DRAM at 2-5 %. The same transform on 64-bit integers runs on the integer
// pipe: a 64-bit add measures 17x the rate of a DADD, and a rounded 64 x 64 -> high 64
// product (three mad.wide) 3.8x the rate of a DMUL. A line of doubles is converted once to
// integers x * 2^s with s from the line's largest modulus, and the transform's outputs are
// converted back with one rounding.
//
// Scaling. A stage of radix R grows a modulus by at most R, and every stage after the first
// multiplies by twiddles stored as w * 2^62 and keeps the high word of the 128-bit product,
// i.e. divides by 4. s is the largest power of two for which no stage can pass 63 bits
// (fx_headroom). The quantum of an N-point result is then N * max / 2^63 of the line or
// finer (of a line of subnormal values N * 2^-1022 / 2^63); the rounding error of a transform, measured over the line shapes of
// tests/fx_host_check.cu, is below that of the FP64 Stockham passes at every length.
// A line that holds an Inf or NaN gives NaN everywhere, as its FP64 transform does.
#pragma once
#include <math.h>

#include "lh_internal.cuh"

struct __align__(16) fx2 { long long x, y; };

// ---- scale of a line ------------------------------------------------------------------
// k0: shift base of fx_in; S: a value v of the result stands for v * 2^-S; pre: the line's
// values are below 2^-895 and are multiplied by 2^512 first (keeps subnormal inputs exact)
struct FxScale { int k0, S, pre; };
#define FX_NAN (-2147483647 - 1)  /* S of a line with an Inf or NaN (or a little above it) */

__host__ __device__ __forceinline__ int fx_ilogb(float m) {  // m > 0, normal
#ifdef __CUDA_ARCH__
  return (int)(__float_as_uint(m) >> 23) - 127;
#else
  return ilogbf(m);
#endif
}
// max(|re|, |im|) of an element, from its high words (fx_hi): a float that counts only where
// the element lies in [2^-126, 2^127); fx_scale leaves the sum aside unless the line's largest
// element is far inside that range
__host__ __device__ __forceinline__ float fx_mag(unsigned hi) {
  const unsigned u = ((hi > 0x38000000u ? hi : 0x38000000u) - 0x38000000u) << 3;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  __builtin_memcpy(&f, &u, 4);
  return f;
#endif
}
// hi: largest high word of |re|, |im| over the line; l1: sum of fx_mag over it (0: unknown);
// head: growth of the largest modulus to allow for, after the `drop` bits that the twiddle
// stages take off. No modulus of any stage is above the sum of the line's moduli either, which
// is the tighter bound where a few elements carry the line (a mean mode).
__host__ __device__ __forceinline__ FxScale fx_scale(unsigned hi, float l1, float head, int drop) {
  FxScale r;
  const int E = (int)(hi >> 20);
  if (E >= 0x7ff) { r.k0 = 4096; r.S = FX_NAN; r.pre = 0; return r; }
  // modulus below sqrt(2) (1 + (mant + 1) / 2^20) 2^(E - 1023)
  const float m = (E ? 1.0f + (float)((hi & 0xfffffu) + 1u) * 9.5367431640625e-7f : 2.0f) * head * 1.4142137f;
  int s = 62 - fx_ilogb(m) - ((E ? E : 1) - 1023) + drop;
  if (l1 > 0 && E > 1023 - 90 && E < 1023 + 100) {
    // 1.15: a stage's output before its twiddles stays below 2^62.8; 1.002: fx_mag's truncation
    const int t = 62 - fx_ilogb(l1 * (1.4142137f * 1.15f * 1.002f));
    s = t > s ? t : s;
  }
  r.pre = E < 128;
  r.k0 = 1085 - (r.pre ? s - 512 : s);
  r.S = s - drop;
  return r;
}
// x * 2^s as an integer, truncated toward zero; |x| 2^s < 2^63
__host__ __device__ __forceinline__ long long fx_in(double x, int k0) {
#ifdef __CUDA_ARCH__
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b;
  __builtin_memcpy(&b, &x, 8);
#endif
  const unsigned hi = (unsigned)(b >> 32);
  int k = k0 - (int)((hi >> 20) & 0x7ffu);
  k = k > 63 ? 63 : k;
  // the mantissa with its leading one at bit 62 (for a zero or subnormal input k = 63 here)
  const unsigned long long M = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
  const long long v = (long long)(M >> k), sg = (long long)((int)hi >> 31);
  return (v ^ sg) - sg;
}
__host__ __device__ __forceinline__ fx2 fx_in2(double2 z, const FxScale &s) {
  if (s.pre) { z.x *= 0x1p512; z.y *= 0x1p512; }
  fx2 r;
  r.x = fx_in(z.x, s.k0);
  r.y = fx_in(z.y, s.k0);
  return r;
}
// v * 2^-S rounded to nearest. The hardware conversion counts as one operation of the FP64 pipe
// (two FP64 additions on split halves measured as two); the scaling is an exponent add.
__host__ __device__ __forceinline__ double fx_out(long long v, int S) {
#ifdef __CUDA_ARCH__
  const double r = __ll2double_rn(v);
  if ((unsigned)(S + 900) <= 1900u)
    return v != 0 ? __hiloint2double(__double2hiint(r) - (S << 20), __double2loint(r)) : r;
  if (S < FX_NAN / 2) return __longlong_as_double(0x7ff8000000000000ll);
  return scalbn(r, -S);
#else
  return S < FX_NAN / 2 ? (double)NAN : ldexp((double)v, -S);
#endif
}
// high word of |re|, |im|, whichever is larger
__host__ __device__ __forceinline__ unsigned fx_hi(double2 z) {
#ifdef __CUDA_ARCH__
  const unsigned a = (unsigned)__double2hiint(z.x) & 0x7fffffffu, b = (unsigned)__double2hiint(z.y) & 0x7fffffffu;
#else
  unsigned long long p, q;
  __builtin_memcpy(&p, &z.x, 8);
  __builtin_memcpy(&q, &z.y, 8);
  const unsigned a = (unsigned)(p >> 32) & 0x7fffffffu, b = (unsigned)(q >> 32) & 0x7fffffffu;
#endif
  return a > b ? a : b;
}

// ---- products -------------------------------------------------------------------------
__host__ __device__ __forceinline__ long long fx_mad(int a, int b, long long c) { return (long long)a * b + c; }
// balanced halves: v = h * 2^32 + l with a signed 32-bit l
__host__ __device__ __forceinline__ int fx_l(long long v) { return (int)v; }
__host__ __device__ __forceinline__ int fx_h(long long v) { return (int)(v >> 32) + (int)((unsigned)v >> 31); }
// (a b) / 2^64 rounded; |a|, |b| < 2^62
__host__ __device__ __forceinline__ long long fx_mul(long long a, long long b) {
  const int al = fx_l(a), ah = fx_h(a), bl = fx_l(b), bh = fx_h(b);
  const long long t = fx_mad(ah, bl, fx_mad(al, bh, 0x80000000ll));
  return fx_mad(ah, bh, t >> 32);
}
// a * w / 4 for a twiddle w = (re h, re l, im h, im l) * 2^-62, conjugated when CONJ; |a| < 2^62.8
template <bool CONJ>
__host__ __device__ __forceinline__ fx2 fx_twiddle(fx2 a, int4 w) {
  const int rl = fx_l(a.x), rh = fx_h(a.x), il = fx_l(a.y), ih = fx_h(a.y);
  const int wih = CONJ ? -w.z : w.z, wil = CONJ ? -w.w : w.w;
  fx2 o;
  long long t = fx_mad(rl, w.x, 0x80000000ll);
  t = fx_mad(rh, w.y, t);
  t = fx_mad(il, -wih, t);
  t = fx_mad(ih, -wil, t);
  o.x = fx_mad(ih, -wih, fx_mad(rh, w.x, t >> 32));
  t = fx_mad(il, w.x, 0x80000000ll);
  t = fx_mad(ih, w.y, t);
  t = fx_mad(rl, wih, t);
  t = fx_mad(rh, wil, t);
  o.y = fx_mad(rh, wih, fx_mad(ih, w.x, t >> 32));
  return o;
}
// a c for a constant c in (1/2, 1): a - a (1 - c), q = (1 - c) 2^64 in balanced halves
template <unsigned long long Q>
__host__ __device__ __forceinline__ long long fx_cmul(long long a) {
  constexpr int ql = (int)(unsigned)Q;
  constexpr int qh = (int)(Q >> 32) + (int)((unsigned)Q >> 31);
  const int al = fx_l(a), ah = fx_h(a);
  const long long t = fx_mad(ah, -ql, fx_mad(al, -qh, 0x80000000ll));
  return fx_mad(ah, -qh, a) + (t >> 32);
}
// a / 4 and a / 2, ties of the half to even (no bias)
__host__ __device__ __forceinline__ long long fx_q4(long long a) { return (a + 2) >> 2; }
__host__ __device__ __forceinline__ long long fx_half(long long a) { return (a + ((a >> 1) & 1)) >> 1; }

#define FX_1M_SQRT1_2 0x4AFB0CCC06219B7Cull  /* (1 - sqrt(1/2)) 2^64 */
#define FX_1M_SIN60 0x224C28BD3D9AAC62ull    /* (1 - sqrt(3)/2) 2^64 */

// ---- register DFTs on integers, unscaled ----------------------------------------------
template <int R, bool INV> struct FxDft;
template <bool INV> struct FxDft<3, INV> {
  static __host__ __device__ __forceinline__ void run(fx2 *v) {
    const fx2 t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]), m = v[0];
    const long long sx = fx_cmul<FX_1M_SIN60>(t2.x), sy = fx_cmul<FX_1M_SIN60>(t2.y);
    const long long bx = m.x - fx_half(t1.x), by = m.y - fx_half(t1.y);
    v[0] = cadd(m, t1);
    if (INV) { v[1].x = bx - sy; v[1].y = by + sx; v[2].x = bx + sy; v[2].y = by - sx; }
    else { v[1].x = bx + sy; v[1].y = by - sx; v[2].x = bx - sy; v[2].y = by + sx; }
  }
};
template <bool INV> struct FxDft<4, INV> {
  static __host__ __device__ __forceinline__ void run(fx2 *v) { dftR<4, INV>(v); }
};
// 6 = 2 x 3 and 12 = 4 x 3 as prime-factor products: no twiddles inside
template <bool INV> struct FxDft<6, INV> {
  static __host__ __device__ __forceinline__ void run(fx2 *v) {
    fx2 e[3] = {cadd(v[0], v[3]), cadd(v[2], v[5]), cadd(v[4], v[1])};
    fx2 o[3] = {csub(v[0], v[3]), csub(v[2], v[5]), csub(v[4], v[1])};
    FxDft<3, INV>::run(e);
    FxDft<3, INV>::run(o);
    v[0] = e[0]; v[4] = e[1]; v[2] = e[2];
    v[3] = o[0]; v[1] = o[1]; v[5] = o[2];
  }
};
template <bool INV> struct FxDft<12, INV> {
  static __host__ __device__ __forceinline__ void run(fx2 *v) {
    fx2 c[3][4];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) c[n2][n1] = v[(3 * n1 + 4 * n2) % 12];
      dftR<4, INV>(c[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      fx2 t[3] = {c[0][k1], c[1][k1], c[2][k1]};
      FxDft<3, INV>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[(9 * k1 + 4 * k2) % 12] = t[k2];
    }
  }
};
template <bool INV> struct FxDft<8, INV> {
  static __host__ __device__ __forceinline__ void run(fx2 *v) {
    fx2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dftR<4, INV>(e);
    dftR<4, INV>(o);
    // forward W8 = (1 - i) / sqrt 2, W8^2 = -i, W8^3 = (-1 - i) / sqrt 2; backward conjugate
    const long long a = fx_cmul<FX_1M_SQRT1_2>(o[1].x), b = fx_cmul<FX_1M_SQRT1_2>(o[1].y);
    const long long c = fx_cmul<FX_1M_SQRT1_2>(o[3].x), d = fx_cmul<FX_1M_SQRT1_2>(o[3].y);
    fx2 t1, t2, t3;
    if (INV) {
      t1.x = a - b; t1.y = a + b; t2.x = -o[2].y; t2.y = o[2].x; t3.x = -(c + d); t3.y = c - d;
    } else {
      t1.x = a + b; t1.y = b - a; t2.x = o[2].y; t2.y = -o[2].x; t3.x = d - c; t3.y = -(c + d);
    }
    v[0] = cadd(e[0], o[0]); v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], t1); v[5] = csub(e[1], t1);
    v[2] = cadd(e[2], t2); v[6] = csub(e[2], t2);
    v[3] = cadd(e[3], t3); v[7] = csub(e[3], t3);
  }
};

// table entry of the twiddle c + i s (host): c, s times 2^62 in balanced halves
static inline void fx_split(long double c, int &h, int &l) {
  const long double q = c * 4611686018427387904.0L;  // 2^62
  long long v = (long long)(q < 0 ? q - 0.5L : q + 0.5L);
  if ((int)(unsigned)v == -2147483647 - 1) v += 1;  // keeps -l representable
  l = (int)(unsigned)(unsigned long long)v;
  h = (int)((v - l) / 4294967296ll);
}
static inline int4 fx_twiddle_word(long double c, long double s) {
  int4 w;
  fx_split(c, w.x, w.y);
  fx_split(s, w.z, w.w);
  return w;
}

// ---- plans ----------------------------------------------------------------------------
// At most three stages. The inverse passes run the factor that holds the 3 first: it then
// reads the zero third of a dealiased line as whole inputs and leaves them out; the forward
// passes run it last and leave the discarded third out of the outputs.
__host__ __device__ constexpr int fx_first(int n) {
  return n == 24 ? 3 : (n == 96 || n == 144 || n == 768 || n == 1152) ? 12 : 6;
}
__host__ __device__ constexpr int fx_second(int n) {
  return n == 72 || n == 144 || n == 576 || n == 1152 ? 12 : n == 192 ? 4 : n == 288 ? 6 : 8;
}
__host__ __device__ constexpr int fx_stages(int n) { return n / (fx_first(n) * fx_second(n)) > 1 ? 3 : 2; }
// radix of stage st of the inverse (INV) or forward (reversed) transform; 1 past the end
template <int N, bool INV>
__host__ __device__ constexpr int fx_radix(int st) {
  constexpr int f = fx_first(N), s = fx_second(N), l = N / (f * s), n = fx_stages(N);
  const int i = INV ? st : n - 1 - st;
  return i == 0 ? f : i == 1 ? s : i == 2 ? l : 1;
}
// largest growth of a modulus, each stage's output brought to the scale of the final one
// (a stage's output that is multiplied by twiddles next must stay below 2^62.8)
template <int N, bool INV>
__host__ __device__ constexpr float fx_headroom() {
  constexpr int n = fx_stages(N);
  double m = N;
  double p = 1;
  for (int i = 0; i + 1 < n; ++i) {
    p *= fx_radix<N, INV>(i);
    double g = p * 1.15;
    for (int j = i; j + 1 < n; ++j) g *= 4;
    m = g > m ? g : m;
  }
  return (float)(m * 1.001);
}
__host__ __device__ constexpr int fx_log2_up(double v) {
  int e = 0;
  for (double p = 1; p < v; p *= 2) ++e;
  return e;
}
template <int N> __host__ __device__ constexpr int fx_drop() { return 2 * (fx_stages(N) - 1); }
template <int N, bool INV>
__host__ __device__ __forceinline__ FxScale fx_line_scale(unsigned hi, float l1) {
  return fx_scale(hi, l1, fx_headroom<N, INV>(), fx_drop<N>());
}

// element i of the lines' shared-memory buffer between two stages: a permutation within
// aligned groups of 8 (16-byte elements, 8 per bank row), so that the strided stores of a
// stage spread over the banks
__host__ __device__ __forceinline__ int fx_swz(int i) { return i ^ ((i >> 3) & 7); }
// plain layout: line-contiguous (IL = false) or interleaved (IL = true)
template <int N, int NL, bool IL>
__host__ __device__ __forceinline__ int fx_at(int line, int e) { return IL ? e * NL + line : line * N + e; }

// One stage over NL lines. ld(line, e) gives input e of a line, st(line, e, v) takes output e,
// all(line, v, R) sees a butterfly's outputs first; nl: lines in use (IL = false). Inputs t in [Z0, Z1) are zero and not read,
// outputs t in [W0, W1) are not stored; XE (x lines: modes -N/3 .. N/3 are kept): of t = Z0 and
// t = W0 the element j = 0 is kept.
#pragma nv_exec_check_disable
template <int N, int NL, bool IL, bool INV, int ST, int Z0, int Z1, int W0, int W1, bool XE, class LD, class SF, class AL>
__host__ __device__ __forceinline__ void fx_stage(int tid, int nthr, const int4 *__restrict__ tw, LD ld, SF st, AL all,
                                                  int nl = NL) {
  constexpr int R = fx_radix<N, INV>(ST);
  constexpr int Ns = ST == 0 ? 1 : ST == 1 ? fx_radix<N, INV>(0) : fx_radix<N, INV>(0) * fx_radix<N, INV>(1);
  constexpr int nb = N / R, step = N / (Ns * R);
  for (int idx = tid; idx < nb * nl; idx += nthr) {
    int line, j;
    if (IL) { j = idx / NL; line = idx - j * NL; }
    else { line = idx / nb; j = idx - line * nb; }
    const int k = j % Ns;
    fx2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      if (t >= Z0 && t < Z1) {
        v[t].x = 0; v[t].y = 0;
        if (XE && t == Z0 && j == 0) v[t] = ld(line, t * nb);
      } else {
        v[t] = ld(line, j + t * nb);
      }
    }
    if constexpr (ST > 0) {
      v[0].x = fx_q4(v[0].x);
      v[0].y = fx_q4(v[0].y);
#pragma unroll
      for (int t = 1; t < R; ++t) v[t] = fx_twiddle<INV>(v[t], tw[k * step * t]);
    }
    FxDft<R, INV>::run(v);
    all(line, v, R);
    const int base = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int t = 0; t < R; ++t)
      if (t < W0 || t >= W1 || (XE && t == W0 && j == 0)) st(line, base + t * Ns, v[t]);
  }
}

struct FxNone { __host__ __device__ void operator()(int, const fx2 *, int) const {} };
#ifdef __CUDACC__
// The transform of NL lines: stage 0 from ld, the last stage to st, the stages between
// through b1 (after stage 0) and b0 (after stage 1). ld may read b0; st may write the
// buffer the last stage does not read: b1 (three stages) or b0 (two).
template <int N, int NL, bool IL, bool INV, int Z0, int Z1, int W0, int W1, bool XE, class LD, class SF, class AL = FxNone>
__device__ __forceinline__ void fx_fft(fx2 *b0, fx2 *b1, const int4 *__restrict__ tw, LD ld, SF st, AL all = AL(), int nl = NL) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  fx_stage<N, NL, IL, INV, 0, Z0, Z1, 0, 0, XE>(tid, nthr, tw, ld,
      [&](int line, int e, fx2 v) { b1[fx_swz(fx_at<N, NL, IL>(line, e))] = v; }, FxNone(), nl);
  __syncthreads();
  if constexpr (fx_stages(N) == 3) {
    fx_stage<N, NL, IL, INV, 1, 0, 0, 0, 0, false>(tid, nthr, tw,
        [&](int line, int e) { return b1[fx_swz(fx_at<N, NL, IL>(line, e))]; },
        [&](int line, int e, fx2 v) { b0[fx_swz(fx_at<N, NL, IL>(line, e))] = v; }, FxNone(), nl);
    __syncthreads();
    fx_stage<N, NL, IL, INV, 2, 0, 0, W0, W1, XE>(tid, nthr, tw,
        [&](int line, int e) { return b0[fx_swz(fx_at<N, NL, IL>(line, e))]; }, st, all, nl);
  } else {
    fx_stage<N, NL, IL, INV, 1, 0, 0, W0, W1, XE>(tid, nthr, tw,
        [&](int line, int e) { return b1[fx_swz(fx_at<N, NL, IL>(line, e))]; }, st, all, nl);
  }
}
#endif
