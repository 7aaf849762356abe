// lh_fxpass.cuh — the FP64 form's transform passes on the fixed-point transforms of lh_fx.cuh:
// the passes of the substep (inverse z with the stagger interpolation, x with the products,
// forward z with der_x / der_z), the leaf plane transforms, the immersed-boundary round trip
// and the statistics' inverse x transform. Memory layouts are those of lh_kernels.cuh
// (A [plane][l][kx], B [product][l/2][kx][l%2]); A and B hold doubles.
//
// Measured at 256 x 256 x 301 with posts (transforms of 384), ms per step (three launches),
// against the FP64 Stockham passes that they replaced (FP64 pipe 85 % busy, DRAM 2-5 %):
//   inverse z 18.52 -> 4.74, x 62.94 -> 15.30, forward z 19.01 -> 5.76, immersed-boundary
//   x round trip 6.58 -> 1.68, its z transforms 1.95 -> 0.49 and 2.04 -> 0.59; the whole
//   step 123.4 -> 38.7 (6.20, 16.85, 7.39 and 43.0 with two FP64 additions per converted
//   result, which kept the FP64 pipe 57-74 % busy). The x pass issues on 52 % of the cycles
//   (ALU 45 %, FP64 26 %) and waits on barriers and instruction fetch; the forward z pass
//   waits on its conversions (FP64 56 %) and on shared memory.
#pragma once
#include "lh_fx.cuh"
#include "lh_kernels.cuh"

// threads and lines per block (the same values on the host). Lines are powers of two, so that
// a thread of an interleaved pass works on one line and a warp holds every line equally often.
__host__ __device__ constexpr int fx_pow2(int v) { return v >= 16 ? 16 : v >= 8 ? 8 : v >= 4 ? 4 : v >= 2 ? 2 : 1; }
__host__ __device__ constexpr int fx_kbz(int n) { return fx_pow2(49152 / (32 * n)); }   // inverse z: columns
__host__ __device__ constexpr int fx_kbf(int n) { return lh_clamp(fx_pow2(49152 / (128 * n)), 1, 8); }  // forward z: columns of four products
__host__ __device__ constexpr int fx_pbx(int n) { return lh_clamp(fx_pow2(49152 / (128 * n)), 1, 8); }  // x: row pairs
__host__ __device__ constexpr int fx_pbl(int n) { return lh_clamp(fx_pow2(49152 / (32 * n)), 1, 16); }  // leaf x: row pairs, one line each
__host__ __device__ constexpr size_t fx_smem(int n, int lines) { return (size_t)32 * n * lines; }  // two buffers
// Threads of a block: as many as the stage with the most butterflies has, so that each stage is
// one round (a stage of 256 butterflies on 192 threads is two, the second one third full), within
// the registers of as many blocks as the SM's shared memory (233472 bytes) holds, four at most.
// ms a step against 192 threads (384 above a length of 384) everywhere, smooth channels of 385 ... 49
// levels; only the passes whose threads the rule changes:
//   length       24     48    144    192    384    576    768   1152
//   inverse z  .118          .511   .518   .820  2.093  3.371  8.946   192 / 384 threads
//              .111          .468   .492   .777  1.611  2.699  7.270   the rule
//   forward z  .074   .169   .506   .548  1.068  2.147
//              .073   .159   .460   .504   .939  2.161
//   x                       1.309                5.270
//                           1.129                5.201
// The forward z pass of 576 is the one that lost (0.7 %). 256 threads above a length of 384 give 576 forward z
// 1.883 and x 4.514, but 1152 x 28.99 (25.70) and forward z 11.97 (10.63), and inverse z less everywhere.
// The x pass keeps 192 up to a length of 384: its instruction issue gains nothing from more warps
// (384: 192 threads 2.401, 256 2.453; 192: .911, .953).
__host__ __device__ constexpr int fx_threads(int n, int lines, int most = 384) {
  const int f = fx_first(n), s = fx_second(n), l = n / (f * s);
  const int r = l > 1 && l < (f < s ? f : s) ? l : (f < s ? f : s);
  const int blocks = 233472 / (32 * n * lines), cap = lh_clamp(1024 / lh_clamp(blocks, 1, 4) / 64 * 64, 128, most);
  return lh_clamp((lines * (n / r) + 31) / 32 * 32, 128, cap);
}
__host__ __device__ constexpr int fx_zt(int n) { return fx_threads(n, fx_kbz(n)); }      // inverse z, leaf z
__host__ __device__ constexpr int fx_ft(int n) { return fx_threads(n, 4 * fx_kbf(n)); }  // forward z
__host__ __device__ constexpr int fx_xt(int n) { return fx_threads(n, 4 * fx_pbx(n), n > 384 ? 384 : 192); }  // x
__host__ __device__ constexpr int fx_lt(int n) { return fx_threads(n, fx_pbl(n)); }      // leaf x

// ---- scales of the lines of an interleaved pass -----------------------------------------
// After each thread has put its elements of line (tid % KB) through hi / l1: the line's scale.
// One barrier (which also publishes the elements in shared memory).
template <int KB>
__device__ __forceinline__ void fx_warp_line(unsigned &hi, float &l1) {
#pragma unroll
  for (int o = KB; o < 32; o *= 2) {
    const unsigned h = __shfl_xor_sync(0xffffffffu, hi, o);
    hi = h > hi ? h : hi;
    l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  }
}
// the slots (hi, l1) that the warps left for a line, combined in warp order
__device__ __forceinline__ void fx_slots(const uint2 *s, int n, int stride, unsigned &hi, float &l1) {
  hi = 0;
  l1 = 0.f;
  for (int i = 0; i < n; ++i) {
    const uint2 q = s[i * stride];
    hi = q.x > hi ? q.x : hi;
    l1 += __uint_as_float(q.y);
  }
}

// ============================================================================
// Inverse z transform of KB columns: get(r, kk) gives element r of column kk, put(l, kk, z)
// takes the result's row l. Z: N2 = 2 (N / 3), so that the zero third is left out.
// ============================================================================
template <int N, int KB, class GET, class PUT>
__device__ __forceinline__ void fx_zinv_body(unsigned char *smem, const int4 *__restrict__ tw, GET get, PUT put) {
  constexpr int NT = fx_zt(N), NW = NT / 32, N2 = 2 * (N / 3), R0 = fx_radix<N, true>(0);
  static_assert(NT % KB == 0 && 32 % KB == 0, "a thread keeps one column");
  __shared__ uint2 slot[NW * KB];
  fx2 *b0 = reinterpret_cast<fx2 *>(smem), *b1 = b0 + KB * N;
  double2 *raw = reinterpret_cast<double2 *>(smem);
  const int tid = threadIdx.x;
  unsigned hi = 0;
  float l1 = 0.f;
#pragma unroll 4
  for (int idx = tid; idx < N2 * KB; idx += NT) {
    const int r = idx / KB, kk = idx - r * KB;
    const double2 z = get(r, kk);
    raw[(r < N2 / 2 ? r : r + N - N2) * KB + kk] = z;
    const unsigned h = fx_hi(z);
    hi = h > hi ? h : hi;
    l1 += fx_mag(h);
  }
  fx_warp_line<KB>(hi, l1);
  if ((tid & 31) < KB) slot[(tid >> 5) * KB + (tid & 31)] = make_uint2(hi, __float_as_uint(l1));
  __syncthreads();
  fx_slots(slot + (tid & (KB - 1)), NW, KB, hi, l1);
  const FxScale sc = fx_line_scale<N, true>(hi, l1);
  fx_fft<N, KB, true, true, R0 / 3, 2 * R0 / 3, 0, 0, false>(
      b0, b1, tw, [&](int line, int e) { return fx_in2(raw[e * KB + line], sc); },
      [&](int line, int e, fx2 v) { put(e, line, make_double2(fx_out(v.x, sc.S), fx_out(v.y, sc.S))); });
}

// Inverse z transforms of the velocity planes with the stagger interpolation (FOU3D.f90:427-474).
// grid: x = column group, y = level slot, z = field.
template <int N>
__global__ void __launch_bounds__(fx_zt(N)) k_zinv_fx(const double2 *__restrict__ u1, const double2 *__restrict__ u2,
                                                      const double2 *__restrict__ u3, double2 *__restrict__ A, Geo g,
                                                      const int4 *__restrict__ tw) {
  constexpr int KB = fx_kbz(N);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = zinv_slot(g, blockIdx.y), f = blockIdx.z, kx0 = blockIdx.x * KB;
  const bool isU = slot < g.nuI;
  const int q = slot_level(g, slot, isU);
  const int nc = g.ncolF;
  // the level itself, or the two levels of an interpolation: v faces q, q - 1 -> centre q;
  // centres q + 1, q -> face q
  const bool own = isU ? f != 1 : f == 1;
  const double2 *s0 = (f == 1) ? u2 + (size_t)q * nc : (f == 0 ? u1 : u3) + (size_t)(isU ? q : q + 1) * nc;
  const double2 *s1 = own ? s0 : s0 - nc;
  const double a = own ? 1.0 : (isU ? g.iua[q] : g.iva[q]), b = own ? 0.0 : (isU ? g.iub[q] : g.ivb[q]);
  double2 *dst = A + (size_t)(slot * 3 + f) * N * g.N1h;
  fx_zinv_body<N, KB>(
      smem_raw, tw,
      [&](int r, int kk) {
        double2 z = make_double2(0.0, 0.0);
        const int kx = kx0 + kk;
        if (kx < g.N1h) {
          const int c = gcol(g, r, kx);
          z = s0[c];
          if (!own) {
            const double2 y = s1[c];
            z.x = a * z.x + b * y.x;
            z.y = a * z.y + b * y.y;
          }
        }
        return z;
      },
      [&](int l, int kk, double2 z) {
        if (kx0 + kk < g.N1h) dst[(size_t)l * g.N1h + kx0 + kk] = z;
      });
}

// plane transform of the leaves and of du's planes (mixed form: k_spec_zinv2)
template <int N>
__global__ void __launch_bounds__(fx_zt(N)) k_spec_zinv_fx(const double2 *__restrict__ spec, double2 *__restrict__ A,
                                                           Geo g, const int4 *__restrict__ tw) {
  constexpr int KB = fx_kbz(N);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pl = blockIdx.y, kx0 = blockIdx.x * KB;
  const double2 *S = spec + (size_t)pl * g.ncol;
  double2 *dst = A + (size_t)pl * N * g.N1h;
  fx_zinv_body<N, KB>(
      smem_raw, tw,
      [&](int r, int kk) { return kx0 + kk < g.N1h ? S[r * g.N1h + kx0 + kk] : make_double2(0.0, 0.0); },
      [&](int l, int kk, double2 z) {
        if (kx0 + kk < g.N1h) dst[(size_t)l * g.N1h + kx0 + kk] = z;
      });
}

// ============================================================================
// Forward z transforms. NP products of KB columns: lines p * KB + kk.
// ============================================================================
// Stages of the transform after the elements are in raw[l * NL + line] with each line's scale
// in sc; the kept rows go to fx2 res[l * NL + line] (the returned buffer; a barrier follows).
template <int N, int NL>
__device__ __forceinline__ const fx2 *fx_zfwd_stages(unsigned char *smem, const int4 *__restrict__ tw, const FxScale &sc) {
  constexpr int RL = fx_radix<N, false>(fx_stages(N) - 1);
  fx2 *b0 = reinterpret_cast<fx2 *>(smem), *b1 = b0 + NL * N;
  const double2 *raw = reinterpret_cast<const double2 *>(smem);
  fx2 *res = fx_stages(N) == 3 ? b1 : b0;
  fx_fft<N, NL, true, false, 0, 0, RL / 3, 2 * RL / 3, false>(
      b0, b1, tw, [&](int line, int e) { return fx_in2(raw[e * NL + line], sc); },
      [&](int line, int e, fx2 v) { res[e * NL + line] = v; });
  __syncthreads();
  return res;
}

template <int N, int NP, int KB>
__device__ __forceinline__ void fx_zfwd_body(const double2 *__restrict__ B, const Geo &g, const int4 *__restrict__ tw,
                                             int q, int pbase, int kx0, double2 *oa, double2 *ob, double2 *oc) {
  constexpr int NL = NP * KB, NT = fx_ft(N), NW = NT / 32;
  static_assert(NT % NL == 0 && 32 % (2 * KB) == 0, "a thread keeps one column in each product and one line");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[NW * NL];
  __shared__ int sS[NL];
  double2 *raw = reinterpret_cast<double2 *>(smem_raw);
  const int N1h = g.N1h, N2 = g.N2, tid = threadIdx.x;
  unsigned hi[NP];
  float l1[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) { hi[p] = 0; l1[p] = 0.f; }
  // the KB columns of a row pair are 2 KB contiguous values of B
  for (int idx = tid; idx < N * KB; idx += NT) {
    const int h = idx & 1, kk = (idx >> 1) % KB, lp = (idx >> 1) / KB, kx = kx0 + kk;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      double2 z = make_double2(0.0, 0.0);
      if (kx < N1h) z = B[(((size_t)(pbase + p) * (N / 2) + lp) * N1h + kx) * 2 + h];
      raw[(2 * lp + h) * NL + p * KB + kk] = z;
      const unsigned m = fx_hi(z);
      hi[p] = m > hi[p] ? m : hi[p];
      l1[p] += fx_mag(m);
    }
  }
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const unsigned m = __shfl_xor_sync(0xffffffffu, hi[p], 1);
    hi[p] = m > hi[p] ? m : hi[p];
    l1[p] += __shfl_xor_sync(0xffffffffu, l1[p], 1);
    fx_warp_line<2 * KB>(hi[p], l1[p]);
    if ((tid & 31) < 2 * KB && (tid & 1) == 0)
      slot[(tid >> 5) * NL + p * KB + ((tid & 31) >> 1)] = make_uint2(hi[p], __float_as_uint(l1[p]));
  }
  __syncthreads();
  unsigned H;
  float L;
  fx_slots(slot + (tid & (NL - 1)), NW, NL, H, L);
  const FxScale sc = fx_line_scale<N, false>(H, L);
  if (tid < NL) sS[tid] = sc.S;
  const fx2 *res = fx_zfwd_stages<N, NL>(smem_raw, tw, sc);
  // both transforms' normalisation; the x pass leaves its own out
  const double s2 = 1.0 / ((double)N * (double)g.G1);
  const size_t off = (size_t)q * g.ncolF;
  for (int idx = tid; idx < N2 * KB; idx += NT) {
    const int r = idx / KB, kk = idx - r * KB, kx = kx0 + kk;
    if (kx >= N1h) continue;
    const fx2 *R = res + prow(g, r) * NL + kk;
    const int c = gcol(g, r, kx);
    // der_x / der_z zero the kz = -N2/2 row
    const bool zr = (r == N2 / 2);
    const double kxv = zr ? 0.0 : g.k1x[kx] * s2, kzv = zr ? 0.0 : g.k1z[grow(g, r)] * s2;
    double2 z[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int S = sS[p * KB + kk];
      z[p] = make_double2(fx_out(R[p * KB].x, S), fx_out(R[p * KB].y, S));
    }
    if constexpr (NP == 4) {  // uu, uw, vv, ww -> N1xz, N3xz, vvc
      oa[off + c] = make_double2(-(kxv * z[0].y + kzv * z[1].y), kxv * z[0].x + kzv * z[1].x);
      ob[off + c] = make_double2(-(kxv * z[1].y + kzv * z[3].y), kxv * z[1].x + kzv * z[3].x);
      oc[off + c] = make_double2(z[2].x * s2, z[2].y * s2);
    } else {  // uv, wv -> N2xz, uvf, wvf
      oa[off + c] = make_double2(-(kxv * z[0].y + kzv * z[1].y), kxv * z[0].x + kzv * z[1].x);
      ob[off + c] = make_double2(z[0].x * s2, z[0].y * s2);
      oc[off + c] = make_double2(z[1].x * s2, z[1].y * s2);
    }
  }
}

// Forward z transforms + der_x / der_z (FOU3D.f90:476-593). grid: x = column group, y = level slot; a v
// level has two products instead of four and takes twice the columns, so that every block
// carries the same lines.
template <int N>
__global__ void __launch_bounds__(fx_ft(N)) k_zfwd_fx(const double2 *__restrict__ B, Geo g, const int4 *__restrict__ tw,
                                                      double2 *__restrict__ N1xz, double2 *__restrict__ N2xz,
                                                      double2 *__restrict__ N3xz, double2 *__restrict__ uvf,
                                                      double2 *__restrict__ vvc, double2 *__restrict__ wvf) {
  constexpr int KB = fx_kbf(N);
  const int slot = blockIdx.y;
  const bool isU = slot < g.nuI;
  const int q = slot_level(g, slot, isU);
  if (isU) {
    fx_zfwd_body<N, 4, KB>(B, g, tw, q, slot * 4, blockIdx.x * KB, N1xz, N3xz, vvc);
  } else {
    const int kx0 = blockIdx.x * 2 * KB;
    if (kx0 < g.N1h) fx_zfwd_body<N, 2, 2 * KB>(B, g, tw, q, g.nuI * 4 + (slot - g.nuI) * 2, kx0, N2xz, uvf, wvf);
  }
}

// plane transform of the leaves and of du's planes (mixed form: k_zfwd_spec2); B [plane][l][kx]. scale: the
// factor of both transforms (the x passes below leave theirs out)
template <int N>
__global__ void __launch_bounds__(fx_zt(N)) k_zfwd_spec_fx(const double2 *__restrict__ B, double2 *__restrict__ spec,
                                                           Geo g, const int4 *__restrict__ tw) {
  constexpr int KB = fx_kbz(N), NT = fx_zt(N), NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[NW * KB];
  double2 *raw = reinterpret_cast<double2 *>(smem_raw);
  const int N1h = g.N1h, N2 = g.N2, tid = threadIdx.x;
  const int pl = blockIdx.y, kx0 = blockIdx.x * KB;
  unsigned hi = 0;
  float l1 = 0.f;
#pragma unroll 4
  for (int idx = tid; idx < N * KB; idx += NT) {
    const int l = idx / KB, kk = idx - l * KB, kx = kx0 + kk;
    double2 z = make_double2(0.0, 0.0);
    if (kx < N1h) z = B[((size_t)pl * N + l) * N1h + kx];
    raw[idx] = z;
    const unsigned h = fx_hi(z);
    hi = h > hi ? h : hi;
    l1 += fx_mag(h);
  }
  fx_warp_line<KB>(hi, l1);
  if ((tid & 31) < KB) slot[(tid >> 5) * KB + (tid & 31)] = make_uint2(hi, __float_as_uint(l1));
  __syncthreads();
  fx_slots(slot + (tid & (KB - 1)), NW, KB, hi, l1);
  const FxScale sc = fx_line_scale<N, false>(hi, l1);
  const fx2 *res = fx_zfwd_stages<N, KB>(smem_raw, tw, sc);
  const double s2 = 1.0 / ((double)N * (double)g.G1);
  double2 *S = spec + (size_t)pl * g.ncol;
  for (int idx = tid; idx < N2 * KB; idx += NT) {
    const int r = idx / KB, kk = idx - r * KB, kx = kx0 + kk;  // idx % KB is the thread's line
    if (kx >= N1h) continue;
    const fx2 t = res[prow(g, r) * KB + kk];
    S[r * N1h + kx] = make_double2(fx_out(t.x, sc.S) * s2, fx_out(t.y, sc.S) * s2);
  }
}

// ============================================================================
// x lines. A line carries the row pair (l, l + 1): row l in .x, row l + 1 in .y after the
// inverse transform.
// ============================================================================
// Gather of NL Hermitian-completed lines into raw[line * N + e] (elements N/3 < e < 2N/3 are
// zero and not written) and their scales into sc[line]; rows(line, k, a, b) gives mode k of the
// two rows (false: the line is not there). Two barriers.
template <int N>
struct fx_xgather {
  static constexpr int M = N / 3;  // modes 0 .. M retained
  static constexpr int GS = M > 16 ? 32 : (M > 8 ? 16 : 8);  // lanes on one (line, chunk of modes)
  static constexpr int NCH = (M + GS - 1) / GS;
};
template <int N, int NL, class ROWS>
__device__ __forceinline__ void fx_xgather_lines(double2 *raw, FxScale *sc, uint2 *slot, ROWS rows) {
  constexpr int M = fx_xgather<N>::M, GS = fx_xgather<N>::GS, NCH = fx_xgather<N>::NCH, PW = 32 / GS;
  const int lane = threadIdx.x & 31, sub = lane % GS;
  const int nw = blockDim.x >> 5;
  for (int base = (threadIdx.x >> 5) * PW; base < NL * NCH; base += nw * PW) {
    const int it = base + lane / GS;
    const int line = it / NCH, ch = it - line * NCH;
    unsigned hi = 0;
    float l1 = 0.f;
    auto put = [&](int k) {
      double2 a, b, zd = make_double2(0.0, 0.0), zc = zd;
      if (rows(line, k, a, b)) {
        if (k == 0) { a.y = 0; b.y = 0; }
        zd = make_double2(a.x - b.y, a.y + b.x);   // a + i b
        zc = make_double2(a.x + b.y, b.x - a.y);   // conj(a) + i conj(b)
      }
      raw[line * N + k] = zd;
      const unsigned h = fx_hi(zd);
      hi = h > hi ? h : hi;
      l1 += fx_mag(h);
      if (k > 0) {
        raw[line * N + N - k] = zc;
        const unsigned hc = fx_hi(zc);
        hi = hc > hi ? hc : hi;
        l1 += fx_mag(hc);
      }
    };
    if (it < NL * NCH) {
      const int k = ch * GS + sub;
      if (k < M) put(k);
      if (ch == 0 && sub == 0) put(M);
    }
#pragma unroll
    for (int o = 1; o < GS; o *= 2) {
      const unsigned h = __shfl_xor_sync(0xffffffffu, hi, o);
      hi = h > hi ? h : hi;
      l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (sub == 0 && it < NL * NCH) slot[it] = make_uint2(hi, __float_as_uint(l1));
  }
  __syncthreads();
  if (threadIdx.x < NL) {
    unsigned hi;
    float l1;
    fx_slots(slot + threadIdx.x * NCH, NCH, 1, hi, l1);
    sc[threadIdx.x] = fx_line_scale<N, true>(hi, l1);
  }
  __syncthreads();
}

// Inverse x transform of NL lines gathered from rows(): doubles in the returned buffer,
// [line * N + m]. One barrier after the last store.
template <int N, int NL, class ROWS>
__device__ __forceinline__ double2 *fx_xinv_lines(unsigned char *smem, FxScale *sc, uint2 *slot,
                                                  const int4 *__restrict__ tw, ROWS rows) {
  constexpr int R0 = fx_radix<N, true>(0);
  fx2 *b0 = reinterpret_cast<fx2 *>(smem), *b1 = b0 + NL * N;
  double2 *raw = reinterpret_cast<double2 *>(smem);
  fx_xgather_lines<N, NL>(raw, sc, slot, rows);
  double2 *res = reinterpret_cast<double2 *>(fx_stages(N) == 3 ? b1 : b0);
  fx_fft<N, NL, false, true, R0 / 3, 2 * R0 / 3, 0, 0, true>(
      b0, b1, tw, [&](int line, int e) { return fx_in2(raw[line * N + e], sc[line]); },
      [&](int line, int e, fx2 v) {
        const int S = sc[line].S;
        res[line * N + e] = make_double2(fx_out(v.x, S), fx_out(v.y, S));
      });
  __syncthreads();
  return res;
}

// Forward x transform of NL lines of doubles in src[line * N + m] (one of the two buffers of
// smem): the retained elements as fx2 in the returned buffer, each line's exponent in sc[].S.
// The caller's values must be visible (a barrier) before the call.
template <int N, int NL>
__device__ __forceinline__ const fx2 *fx_xfwd_lines(const double2 *src, unsigned char *smem, FxScale *sc, uint2 *slot,
                                                    const int4 *__restrict__ tw) {
  constexpr int RL = fx_radix<N, false>(fx_stages(N) - 1);
  constexpr int GS = N >= 32 ? 32 : 8, NCH = (N + GS - 1) / GS, PW = 32 / GS;
  const int lane = threadIdx.x & 31, sub = lane % GS, nw = blockDim.x >> 5;
  for (int base = (threadIdx.x >> 5) * PW; base < NL * NCH; base += nw * PW) {
    const int it = base + lane / GS;
    const int line = it / NCH, m = (it - line * NCH) * GS + sub;
    unsigned hi = 0;
    float l1 = 0.f;
    if (it < NL * NCH && m < N) { hi = fx_hi(src[line * N + m]); l1 = fx_mag(hi); }
#pragma unroll
    for (int o = 1; o < GS; o *= 2) {
      const unsigned h = __shfl_xor_sync(0xffffffffu, hi, o);
      hi = h > hi ? h : hi;
      l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (sub == 0 && it < NL * NCH) slot[it] = make_uint2(hi, __float_as_uint(l1));
  }
  __syncthreads();
  if (threadIdx.x < NL) {
    unsigned hi;
    float l1;
    fx_slots(slot + threadIdx.x * NCH, NCH, 1, hi, l1);
    // twice the sums of the moduli: the row separation adds two elements
    sc[threadIdx.x] = fx_scale(hi, 2.0f * l1, 2.0f * fx_headroom<N, false>(), fx_drop<N>());
  }
  __syncthreads();
  fx2 *b0 = reinterpret_cast<fx2 *>(smem), *b1 = b0 + NL * N;
  fx2 *s0 = reinterpret_cast<const unsigned char *>(src) == smem ? b0 : b1, *s1 = s0 == b0 ? b1 : b0;
  fx2 *res = fx_stages(N) == 3 ? s1 : s0;
  fx_fft<N, NL, false, false, 0, 0, RL / 3, 2 * RL / 3, true>(
      s0, s1, tw, [&](int line, int e) { return fx_in2(src[line * N + e], sc[line]); },
      [&](int line, int e, fx2 v) { res[line * N + e] = v; });
  __syncthreads();
  return res;
}
// rows of a pair from its transformed line (elements k and N - k), not normalised: rows[h] =
// (z + conj(z')) / 2 and -i (z - conj(z')) / 2
template <int N>
__device__ __forceinline__ void fx_rows(const fx2 *L, int k, int S, double2 &o0, double2 &o1) {
  const fx2 z = L[k], c = L[k == 0 ? 0 : N - k];
  o0 = make_double2(fx_out(z.x + c.x, S + 1), fx_out(z.y - c.y, S + 1));
  o1 = make_double2(fx_out(z.y + c.y, S + 1), fx_out(c.x - z.x, S + 1));
  if (k == 0) { o0.y = 0.0; o1.y = 0.0; }
}
__host__ __device__ constexpr int fx_max(int a, int b) { return a > b ? a : b; }
// (hi, l1) slots of NL x lines (gather or forward)
template <int N, int NL> __host__ __device__ constexpr int fx_xslots() {
  return NL * fx_max(fx_xgather<N>::NCH, (N + (N >= 32 ? 31 : 7)) / (N >= 32 ? 32 : 8));
}

// ============================================================================
// x pass of the substep: inverse transform, products, CFL maxima, forward
// transform. The products are formed from the integer fields, normalised by each field's
// largest value on the line, as the forward transform's first stage reads them.
// ============================================================================
// bits of a product's operands: two of them give products that the forward transform has headroom
// for (and one bit for the row separation)
template <int N> __host__ __device__ constexpr int fx_opbits() {
  constexpr int PBITS = 62 + fx_drop<N>() - fx_log2_up(fx_headroom<N, false>() * 1.4143f);
  constexpr int TB = (64 + PBITS) / 2;
  static_assert(TB <= 62, "operands of fx_mul");
  return TB;
}
// Products uu, uw, vv, ww (u level) or uv, wv (v level) of the fields' lines f * PB + pb in res and
// their forward transforms, lines p * PB + pb in res (two stages) or oth (three). One code for
// both kinds of level: the kernel's code has to stay in the instruction cache.
template <int N, int PB>
__device__ __forceinline__ void fx_xpass_forward(bool isU, fx2 *res, fx2 *oth, const int *fl, const int *fS, int *sP,
                                                 const int4 *__restrict__ tw) {
  constexpr int RL = fx_radix<N, false>(fx_stages(N) - 1);
  constexpr int DROP = fx_drop<N>();
  auto fa = [&](int p) { return isU ? (p > 0 ? p - 1 : 0) : 2 * p; };
  auto fb = [&](int p) { return isU ? (p == 0 ? 0 : p == 2 ? 1 : 2) : 1; };
  // to 63 bits by the line's shift, then to TB bits
  auto shift = [](fx2 v, int l) {
    fx2 r;
    r.x = (long long)((unsigned long long)v.x << l) >> (63 - fx_opbits<N>());
    r.y = (long long)((unsigned long long)v.y << l) >> (63 - fx_opbits<N>());
    return r;
  };
  const int nl = (isU ? 4 : 2) * PB;
  if ((int)threadIdx.x < nl) {
    const int p = threadIdx.x / PB, pb = threadIdx.x - p * PB, a = fa(p) * PB + pb, b = fb(p) * PB + pb;
    sP[threadIdx.x] = (fS[a] == FX_NAN || fS[b] == FX_NAN) ? FX_NAN : fS[a] + fl[a] + fS[b] + fl[b] - 2 * (63 - fx_opbits<N>()) - 64 - DROP;
  }
  auto ld = [&](int line, int e) {
    const int p = line / PB, pb = line - p * PB, a = fa(p) * PB + pb, b = fb(p) * PB + pb;
    const fx2 x = shift(res[a * N + e], fl[a]), y = shift(res[b * N + e], fl[b]);
    fx2 r;
    r.x = fx_mul(x.x, y.x);
    r.y = fx_mul(x.y, y.y);
    return r;
  };
  fx2 *last = fx_stages(N) == 3 ? oth : res;
  // stage 0 reads res and writes oth, stage 1 writes res, the last stage writes `last`
  fx_fft<N, 4 * PB, false, false, 0, 0, RL / 3, 2 * RL / 3, true>(
      res, oth, tw, ld, [&](int line, int e, fx2 v) { last[line * N + e] = v; }, FxNone(), nl);
  __syncthreads();
}

template <int N>
__global__ void __launch_bounds__(fx_xt(N)) k_xpass_fx(const double2 *__restrict__ A, double2 *__restrict__ B, Geo g,
                                                       const int4 *__restrict__ tw, int doCFL, DevScalars *sc,
                                                       const int *__restrict__ capslot, double *__restrict__ cap) {
  constexpr int PB = fx_pbx(N), NL = 3 * PB, NT = fx_xt(N), NK = N / 3 + 1;
  constexpr int R0 = fx_radix<N, true>(0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[NL * fx_xgather<N>::NCH];
  __shared__ FxScale sL[NL];
  __shared__ int lm[NL], fl[NL], fS[NL], sP[4 * PB];
  fx2 *b0 = reinterpret_cast<fx2 *>(smem_raw), *b1 = b0 + 4 * PB * N;
  double2 *raw = reinterpret_cast<double2 *>(smem_raw);
  const int G2 = g.G2, N1h = g.N1h, tid = threadIdx.x;
  const int slot_i = blockIdx.y;
  const bool isU = slot_i < g.nuI;
  const int q = slot_level(g, slot_i, isU);
  const int l0 = blockIdx.x * PB * 2, npairs = min(PB, (G2 - l0) / 2);
  const size_t fstride = (size_t)G2 * N1h;
  const double2 *Af = A + (size_t)slot_i * 3 * fstride + (size_t)l0 * N1h;
  if (tid < NL) lm[tid] = 0;
  fx_xgather_lines<N, NL>(raw, sL, slot, [&](int line, int k, double2 &a, double2 &b) {
    const int f = line / PB, pb = line - f * PB;
    if (pb >= npairs) return false;
    const double2 *s = Af + f * fstride + (size_t)(2 * pb) * NK + k;
    a = s[0];
    b = s[NK];
    return true;
  });
  // the inverse transform's result stays in integers; each line's largest high word in lm
  fx2 *res = fx_stages(N) == 3 ? b1 : b0, *oth = res == b0 ? b1 : b0;
  fx_fft<N, NL, false, true, R0 / 3, 2 * R0 / 3, 0, 0, true>(
      b0, b1, tw, [&](int line, int e) { return fx_in2(raw[line * N + e], sL[line]); },
      [&](int line, int e, fx2 v) { res[line * N + e] = v; },
      [&](int line, const fx2 *v, int n) {
        int m = 0;
        for (int t = 0; t < n; ++t) {
          const int hx = (int)(v[t].x >> 32), hy = (int)(v[t].y >> 32);
          m |= (hx ^ (hx >> 31)) | (hy ^ (hy >> 31));
        }
        atomicOr(&lm[line], m);
      });
  __syncthreads();
  if (tid < NL) {
    // |v| <= 2^(64 - clz)
    fl[tid] = __clz(lm[tid]) - 1;
    fS[tid] = sL[tid].S;
  }
  __syncthreads();
  if (capslot) {
    const int cs = capslot[slot_i];
    if (cs >= 0) {
      for (int idx = tid; idx < NL * N; idx += NT) {
        const int line = idx / N, m = idx - line * N, f = line / PB, pb = line - f * PB;
        if (pb >= npairs) continue;
        double *cp = cap + ((size_t)cs * 3 + f) * (size_t)G2 * N + (size_t)(l0 + 2 * pb) * N + m;
        cp[0] = fx_out(res[idx].x, fS[line]);
        cp[N] = fx_out(res[idx].y, fS[line]);
      }
    }
  }
  if (doCFL) {  // first substep only
    double m0 = 0, m1 = 0;
    const double thv = isU ? 0.0 : g.thv[q];
    for (int idx = tid; idx < npairs * N; idx += NT) {
      const int pb = idx / N, m = idx - pb * N;
      if (isU) {
        const fx2 u = res[pb * N + m], w = res[(2 * PB + pb) * N + m];
        m0 = nmax(m0, nmax(fabs(fx_out(u.x, fS[pb])), fabs(fx_out(u.y, fS[pb]))));
        m1 = nmax(m1, nmax(fabs(fx_out(w.x, fS[2 * PB + pb])), fabs(fx_out(w.y, fS[2 * PB + pb]))));
      } else {
        const fx2 v = res[(PB + pb) * N + m];
        m0 = nmax(m0, nmax(fabs(fx_out(v.x, fS[PB + pb])), fabs(fx_out(v.y, fS[PB + pb]))) * thv);
      }
    }
    m0 = warp_max(m0);
    m1 = warp_max(m1);
    if ((tid & 31) == 0) {
      if (isU) { atomic_max_pos(&sc->u1m, m0); atomic_max_pos(&sc->u3m, m1); }
      else atomic_max_pos(&sc->u2m, m0);
    }
  }
  fx_xpass_forward<N, PB>(isU, res, oth, fl, fS, sP, tw);
  const fx2 *pres = fx_stages(N) == 3 ? oth : res;
  const int nprod = isU ? 4 : 2;
  const int pbase = isU ? slot_i * 4 : g.nuI * 4 + (slot_i - g.nuI) * 2;
  for (int idx = tid; idx < nprod * PB * NK; idx += NT) {
    const int k = idx % NK, r2 = idx / NK, pb = r2 % PB, p = r2 / PB;
    if (pb >= npairs) continue;
    double2 o0, o1;
    fx_rows<N>(pres + (p * PB + pb) * N, k, sP[p * PB + pb], o0, o1);
    double2 *dst = B + (((size_t)(pbase + p) * (G2 / 2) + (l0 >> 1) + pb) * N1h + k) * 2;
    dst[0] = o0;
    dst[1] = o1;
  }
}

// ============================================================================
// Leaf plane transforms, the immersed-boundary round trip (mixed form: k_ib_xforce) and the
// statistics' plane sums (mixed form: k_xstats) on the same lines.
// ============================================================================
template <int N>
__global__ void __launch_bounds__(fx_lt(N)) k_xinv_phys_fx(const double2 *__restrict__ A, double *__restrict__ phys, Geo g,
                                                           const int4 *__restrict__ tw) {
  constexpr int PB = fx_pbl(N), NK = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[fx_xslots<N, PB>()];
  __shared__ FxScale sc[PB];
  const int pl = blockIdx.y, l0 = blockIdx.x * PB * 2, npairs = min(PB, (g.G2 - l0) / 2);
  const double2 *Ap = A + ((size_t)pl * g.G2 + l0) * NK;
  const double2 *res = fx_xinv_lines<N, PB>(smem_raw, sc, slot, tw, [&](int pb, int k, double2 &a, double2 &b) {
    if (pb >= npairs) return false;
    a = Ap[(size_t)(2 * pb) * NK + k];
    b = Ap[(size_t)(2 * pb + 1) * NK + k];
    return true;
  });
  double *P = phys + ((size_t)pl * g.G2 + l0) * N;
  for (int idx = threadIdx.x; idx < npairs * N; idx += blockDim.x) {
    const int pb = idx / N, m = idx - pb * N;
    P[(size_t)(2 * pb) * N + m] = res[idx].x;
    P[(size_t)(2 * pb + 1) * N + m] = res[idx].y;
  }
}

// rows of NL transformed lines to B [plane][l][kx] (k_zfwd_spec_fx applies the normalisation)
template <int N, int PB>
__device__ __forceinline__ void fx_rows_out(const fx2 *L, const FxScale *sc, double2 *Bp, int npairs) {
  constexpr int NK = N / 3 + 1;
  for (int idx = threadIdx.x; idx < npairs * NK; idx += blockDim.x) {
    const int pb = idx / NK, k = idx - pb * NK;
    double2 o0, o1;
    fx_rows<N>(L + pb * N, k, sc[pb].S, o0, o1);
    Bp[(size_t)(2 * pb) * NK + k] = o0;
    Bp[(size_t)(2 * pb + 1) * NK + k] = o1;
  }
}

template <int N>
__global__ void __launch_bounds__(fx_lt(N)) k_xfwd_phys_fx(const double *__restrict__ phys, double2 *__restrict__ B, Geo g,
                                                           const int4 *__restrict__ tw) {
  constexpr int PB = fx_pbl(N), NK = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[fx_xslots<N, PB>()];
  __shared__ FxScale sc[PB];
  double2 *raw = reinterpret_cast<double2 *>(smem_raw);
  const int pl = blockIdx.y, l0 = blockIdx.x * PB * 2, npairs = min(PB, (g.G2 - l0) / 2);
  const double *P = phys + ((size_t)pl * g.G2 + l0) * N;
  for (int idx = threadIdx.x; idx < PB * N; idx += blockDim.x) {
    const int pb = idx / N, m = idx - pb * N;
    raw[idx] = pb < npairs ? make_double2(P[(size_t)(2 * pb) * N + m], P[(size_t)(2 * pb + 1) * N + m])
                           : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const fx2 *L = fx_xfwd_lines<N, PB>(raw, smem_raw, sc, slot, tw);
  fx_rows_out<N, PB>(L, sc, B + ((size_t)pl * g.G2 + l0) * NK, npairs);
}

template <int N>
__global__ void __launch_bounds__(fx_lt(N)) k_ib_xforce_fx(const double2 *__restrict__ A, double2 *__restrict__ B, Geo g,
                                                           const int4 *__restrict__ tw, const IbRec *__restrict__ rec,
                                                           const int *__restrict__ rec_off, const double *__restrict__ cap,
                                                           const DevScalars *__restrict__ dsc) {
  constexpr int PB = fx_pbl(N), NK = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[fx_xslots<N, PB>()];
  __shared__ FxScale sc[PB];
  const int pl = blockIdx.y, l0 = blockIdx.x * PB * 2, npairs = min(PB, (g.G2 - l0) / 2);
  const double2 *Ap = A + ((size_t)pl * g.G2 + l0) * NK;
  double2 *res = fx_xinv_lines<N, PB>(smem_raw, sc, slot, tw, [&](int pb, int k, double2 &a, double2 &b) {
    if (pb >= npairs) return false;
    a = Ap[(size_t)(2 * pb) * NK + k];
    b = Ap[(size_t)(2 * pb + 1) * NK + k];
    return true;
  });
  {  // the forced points of the rows
    const double Kibdt = g.Kib / dsc->dt;
    const int r0 = rec_off[(size_t)pl * g.G2 + l0], r1 = rec_off[(size_t)pl * g.G2 + l0 + 2 * npairs];
    for (int e = r0 + threadIdx.x; e < r1; e += blockDim.x) {
      const IbRec R = rec[e];
      const double val = Kibdt * (R.A * cap[R.ref] - cap[R.src]);
      const int rr = R.k - l0;
      double2 *z = res + (rr >> 1) * N + R.i;
      if (rr & 1) z->y = val;
      else z->x = val;
    }
  }
  __syncthreads();
  const fx2 *L = fx_xfwd_lines<N, PB>(res, smem_raw, sc, slot, tw);
  fx_rows_out<N, PB>(L, sc, B + ((size_t)pl * g.G2 + l0) * NK, npairs);
}

// plane and tile-conditioned sums of one plane class (k_xstats' FP64 form)
template <int N>
__global__ void __launch_bounds__(fx_xt(N)) k_xstats_fx(const double2 *__restrict__ A, Geo g, const int4 *__restrict__ tw,
                                                        double *__restrict__ pl, double *__restrict__ cd, int ncl, int dnx,
                                                        int dnz, int ntx) {
  constexpr int PB = fx_pbx(N), NL = 3 * PB, NK = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slot[fx_xslots<N, NL>()];
  __shared__ FxScale sc[NL];
  const int slot_i = blockIdx.y;
  const bool isU = slot_i < g.nuI;
  const int q = slot_level(g, slot_i, isU);
  const int l0 = blockIdx.x * PB * 2, npairs = min(PB, (g.G2 - l0) / 2);
  const size_t fstride = (size_t)g.G2 * g.N1h;
  const double2 *Af = A + (size_t)slot_i * 3 * fstride + (size_t)l0 * g.N1h;
  const double2 *res = fx_xinv_lines<N, NL>(smem_raw, sc, slot, tw, [&](int line, int k, double2 &a, double2 &b) {
    const int f = line / PB, pb = line - f * PB;
    if (pb >= npairs) return false;
    const double2 *s = Af + f * fstride + (size_t)(2 * pb) * NK + k;
    a = s[0];
    b = s[NK];
    return true;
  });
  xstats_sums<N, PB>(res, g, pl, cd, ncl, dnx, dnz, ntx, isU, q, l0, npairs);
}
