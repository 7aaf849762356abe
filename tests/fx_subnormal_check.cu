// Host check of the fixed-point transforms (lh_fx.cuh) on lines of subnormal values
// (tests/test_fx_subnormal_host.py builds and runs it): every length, both directions, against a direct
// DFT in long double, beside the FP64 Stockham plan on the same lines. Prints the largest error of a
// component of either, in units of 2^-1074, beyond 2.3e-16 of the component (results may be normal).
#include "../rnl_multiblock_nofft_gb300/csrc/lh_fx.cuh"

#include <cmath>
#include <complex>
#include <cstdio>
#include <vector>

typedef std::complex<long double> cld;
template <int R, bool INV, int N, int Ns>
static void stage64(const double2 *src, double2 *dst, const double2 *tw) {
  constexpr int nb = N / R, step = N / (Ns * R);
  for (int j = 0; j < nb; ++j) {
    const int k = j % Ns;
    double2 v[R];
    for (int t = 0; t < R; ++t) v[t] = src[j + t * nb];
    if (Ns > 1)
      for (int t = 1; t < R; ++t) {
        double2 w = tw[k * step * t];
        if (INV) w.y = -w.y;
        v[t] = cmul(v[t], w);
      }
    dftR<R, INV>(v);
    const int base = (j / Ns) * Ns * R + k;
    for (int t = 0; t < R; ++t) dst[base + t * Ns] = v[t];
  }
}
template <bool INV, int N, int Ns>
static double2 *fft64(double2 *a, double2 *b, const double2 *tw) {
  if constexpr (Ns >= N) {
    return a;
  } else {
    constexpr int rem = N / Ns;
    constexpr int R = (rem % 8 == 0) ? 8 : ((rem % 6 == 0) ? 6 : ((rem % 4 == 0) ? 4 : ((rem % 2 == 0) ? 2 : 3)));
    stage64<R, INV, N, Ns>(a, b, tw);
    return fft64<INV, N, Ns * R>(b, a, tw);
  }
}

static unsigned rs = 54321u;
static double uni() { rs = rs * 1664525u + 1013904223u; return (rs >> 8) / 16777216.0 - 0.5; }

template <int N, bool INV>
static void check() {
  const long double PI = 3.14159265358979323846264338327950288L;
  std::vector<double2> in(N), out(N);
  std::vector<int4> tw(N);
  std::vector<double2> twd(N), p(N), q(N);
  std::vector<cld> ex(N);
  for (int e = 0; e < N; ++e) {
    const long double a = -2.0L * PI * e / N;
    ex[e] = cld(cosl(a), sinl(a));
    twd[e].x = (double)cosl(a); twd[e].y = (double)sinl(a);
    tw[e] = fx_twiddle_word(cosl(a), sinl(a));
  }
  std::vector<fx2> b0(N), b1(N);
  // largest values: just below the smallest normal, 1e-310, 1e-320 (eleven bits), one smallest value, zero
  const double amp[5] = {2.2250738585072009e-308, 1e-310, 1e-320, 0, 0};
  for (int shape = 0; shape < 5; ++shape) {
    for (int e = 0; e < N; ++e) {
      in[e].x = amp[shape] * 2 * uni();
      in[e].y = amp[shape] * 2 * uni();
    }
    if (shape == 3) in[7].y = -4.9406564584124654e-324;
    unsigned hi = 0;
    float l1 = 0;
    for (int e = 0; e < N; ++e) {
      const unsigned h = fx_hi(in[e]);
      hi = h > hi ? h : hi;
      l1 += fx_mag(h);
    }
    if (hi >> 20) { printf("%d %d %d not subnormal\n", N, (int)INV, shape); continue; }
    const FxScale s = fx_line_scale<N, INV>(hi, l1);
    auto ld = [&](int, int e) { return fx_in2(in[e], s); };
    auto st1 = [&](int, int e, fx2 v) { b1[fx_swz(e)] = v; };
    auto m1 = [&](int, int e) { return b1[fx_swz(e)]; };
    auto fin = [&](int, int e, fx2 v) { out[e].x = fx_out(v.x, s.S); out[e].y = fx_out(v.y, s.S); };
    fx_stage<N, 1, false, INV, 0, 0, 0, 0, 0, false>(0, 1, tw.data(), ld, st1, FxNone());
    if constexpr (fx_stages(N) == 3) {
      fx_stage<N, 1, false, INV, 1, 0, 0, 0, 0, false>(0, 1, tw.data(), m1, [&](int, int e, fx2 v) { b0[fx_swz(e)] = v; }, FxNone());
      fx_stage<N, 1, false, INV, 2, 0, 0, 0, 0, false>(0, 1, tw.data(), [&](int, int e) { return b0[fx_swz(e)]; }, fin, FxNone());
    } else {
      fx_stage<N, 1, false, INV, 1, 0, 0, 0, 0, false>(0, 1, tw.data(), m1, fin, FxNone());
    }
    const long double up = ldexpl(1.0L, 1074);
    p = in;
    const double2 *d = fft64<INV, N, 1>(p.data(), q.data(), twd.data());
    long double worst = 0, wd = 0;
    for (int k = 0; k < N; ++k) {
      cld sum = 0;
      for (int e = 0; e < N; ++e) {
        const cld w = ex[(long)e * k % N];
        sum += cld(in[e].x * up, in[e].y * up) * (INV ? std::conj(w) : w);
      }
      worst = fmaxl(worst, fabsl(out[k].x * up - sum.real()) - 2.3e-16L * fabsl(sum.real()));
      worst = fmaxl(worst, fabsl(out[k].y * up - sum.imag()) - 2.3e-16L * fabsl(sum.imag()));
      wd = fmaxl(wd, fabsl(d[k].x * up - sum.real()) - 2.3e-16L * fabsl(sum.real()));
      wd = fmaxl(wd, fabsl(d[k].y * up - sum.imag()) - 2.3e-16L * fabsl(sum.imag()));
    }
    printf("%d %d %d %.3f %.3f\n", N, (int)INV, shape, (double)worst, (double)wd);
  }
}
template <int N> static void all() { check<N, false>(); check<N, true>(); }

int main() {
  all<24>(); all<48>(); all<72>(); all<96>(); all<144>(); all<192>(); all<288>(); all<384>();
  all<576>(); all<768>(); all<1152>();
  return 0;
}
