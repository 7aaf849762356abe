// Host check of the fixed-point transforms (lh_fx.cuh; tests/test_fft_host.py builds and runs
// it): every length, both directions, against a direct DFT in long double, beside the FP64
// Stockham plan's error on the same lines. The stages, scales and conversions are the
// library's own code; the kernels add only the threads.
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

static unsigned rs = 12345u;
static double uni() { rs = rs * 1664525u + 1013904223u; return (rs >> 8) / 16777216.0 - 0.5; }

// line shapes: 0 flat noise; 1 mean mode 1, noise 1e-3 elsewhere; 2 exponentially decaying
// spectrum (both ends); 3 constant plus 10 % noise; 4 one spike in noise of 1e-6; 5 all equal;
// 6 flat noise near the smallest normal double; 7 near the largest
template <int N>
static void fill(int shape, double2 *x) {
  for (int e = 0; e < N; ++e) {
    const double a = uni(), b = uni();
    const int k = e <= N / 2 ? e : N - e;
    const double dec = exp(-8.0 * k / N * 3);
    double2 z;
    switch (shape) {
      case 0: z.x = a; z.y = b; break;
      case 1: z.x = e == 0 ? 1.3 : 1e-3 * a; z.y = e == 0 ? 0.0 : 1e-3 * b; break;
      case 2: z.x = a * dec; z.y = b * dec; break;
      case 3: z.x = 1.7 + 0.1 * a; z.y = -0.6 + 0.1 * b; break;
      case 4: z.x = e == 5 ? 0.9 : 1e-6 * a; z.y = 1e-6 * b; break;
      case 5: z.x = 1.999999; z.y = -1.999999; break;
      case 6: z.x = a * 3e-307; z.y = b * 3e-307; break;
      default: z.x = a * 1e300; z.y = b * 1e300; break;
    }
    if (shape <= 2 && shape >= 1 && e >= N / 3 && e < 2 * N / 3) z.x = z.y = 0;  // dealiased spectrum
    x[e] = z;
  }
}

template <int N, bool INV>
static void check() {
  const long double PI = 3.14159265358979323846264338327950288L;
  std::vector<double2> tw(N), in(N), a(N), b(N), out(N);
  std::vector<int4> twf(N);
  std::vector<cld> ex(N);
  for (int e = 0; e < N; ++e) {
    const long double ang = -2.0L * PI * e / N, c = cosl(ang), s = sinl(ang);
    tw[e].x = (double)c; tw[e].y = (double)s;
    ex[e] = cld(c, s);
    twf[e] = fx_twiddle_word(c, s);
  }
  std::vector<fx2> b0(N), b1(N);
  for (int shape = 0; shape < 8; ++shape) {
    double ef = 0, ed = 0, mf = 0;
    const int reps = shape == 5 ? 1 : 4;
    for (int rep = 0; rep < reps; ++rep) {
      fill<N>(shape, in.data());
      unsigned hi = 0;
      float l1 = 0;
      for (int e = 0; e < N; ++e) {
        const unsigned h = fx_hi(in[e]);
        hi = h > hi ? h : hi;
        l1 += fx_mag(h);
      }
      const FxScale s = fx_line_scale<N, INV>(hi, l1);
      const bool z = INV && (shape == 1 || shape == 2);  // zero third left out
      auto ld = [&](int, int e) { return fx_in2(in[e], s); };
      auto st1 = [&](int, int e, fx2 v) { b1[fx_swz(e)] = v; };
      constexpr int R0 = fx_radix<N, INV>(0), Z0 = INV ? R0 / 3 : 0, Z1 = INV ? 2 * R0 / 3 : 0;
      if (z) fx_stage<N, 1, false, INV, 0, Z0, Z1, 0, 0, false>(0, 1, twf.data(), ld, st1, FxNone());
      else fx_stage<N, 1, false, INV, 0, 0, 0, 0, 0, false>(0, 1, twf.data(), ld, st1, FxNone());
      auto m1 = [&](int, int e) { return b1[fx_swz(e)]; };
      auto fin = [&](int, int e, fx2 v) { out[e].x = fx_out(v.x, s.S); out[e].y = fx_out(v.y, s.S); };
      if constexpr (fx_stages(N) == 3) {
        fx_stage<N, 1, false, INV, 1, 0, 0, 0, 0, false>(0, 1, twf.data(), m1, [&](int, int e, fx2 v) { b0[fx_swz(e)] = v; }, FxNone());
        fx_stage<N, 1, false, INV, 2, 0, 0, 0, 0, false>(0, 1, twf.data(), [&](int, int e) { return b0[fx_swz(e)]; }, fin, FxNone());
      } else {
        fx_stage<N, 1, false, INV, 1, 0, 0, 0, 0, false>(0, 1, twf.data(), m1, fin, FxNone());
      }
      a = in;
      const double2 *d = fft64<INV, N, 1>(a.data(), b.data(), tw.data());
      long double sf = 0, sd = 0, n = 0, mx = 0, me = 0;
      for (int k = 0; k < N; ++k) {
        cld sum = 0;
        for (int e = 0; e < N; ++e) {
          const cld w = ex[(long)e * k % N];
          sum += cld(in[e].x, in[e].y) * (INV ? std::conj(w) : w);
        }
        const long double f = std::abs(sum - cld(out[k].x, out[k].y));
        sf += f * f;
        sd += std::norm(sum - cld(d[k].x, d[k].y));
        n += std::norm(sum);
        me = fmaxl(me, f); mx = fmaxl(mx, std::abs(sum));
      }
      ef += (double)sqrtl(sf / n) / reps;
      ed += (double)sqrtl(sd / n) / reps;
      mf = fmax(mf, (double)(me / mx));
    }
    printf("%d %d %d %.3e %.3e %.3e\n", N, (int)INV, shape, ef, ed, mf);
  }
}
template <int N> static void all() { check<N, false>(); check<N, true>(); }

int main() {
  all<24>(); all<48>(); all<72>(); all<96>(); all<144>(); all<192>(); all<288>(); all<384>();
  all<576>(); all<768>(); all<1152>();
  return 0;
}
