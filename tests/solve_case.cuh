// A channel's worth of seeded random fields, coefficients and column segments for checks that launch
// the solve kernels of lh_kernels.cuh themselves (the results are compared, not physical).
#pragma once
#include "../rnl_multiblock_nofft_gb300/csrc/lh_kernels.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#define CKC(x)                                                                                \
  do {                                                                                        \
    cudaError_t e_ = (x);                                                                     \
    if (e_ != cudaSuccess) { fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_)); exit(2); } \
  } while (0)

template <typename T>
static T *to_device(const std::vector<T> &v) {
  T *d;
  CKC(cudaMalloc(&d, sizeof(T) * v.size()));
  CKC(cudaMemcpy(d, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return d;
}
template <typename T>
static std::vector<T> to_host(const T *d, size_t n) {
  std::vector<T> v(n);
  CKC(cudaMemcpy(v.data(), d, sizeof(T) * n, cudaMemcpyDeviceToHost));
  return v;
}

struct SolveCase {
  Geo g;
  DevScalars *sc;
  size_t nU, nV, nP;  // doubles of a u, v, p field
  std::mt19937_64 rng;

  std::vector<double> reals(size_t n, double lo, double hi) {
    std::uniform_real_distribution<double> u(lo, hi);
    std::vector<double> v(n);
    for (double &x : v) x = u(rng);
    return v;
  }
  std::vector<float> floats(size_t n, float lo, float hi) {
    std::vector<float> v(n);
    std::uniform_real_distribution<float> u(lo, hi);
    for (float &x : v) x = u(rng);
    return v;
  }
  // N1 x N2 modes, nu levels of u; mb: columns with kx > N1 / 4 live in wall bands of m + 1 levels of u
  SolveCase(int N1, int N2, int nu, bool mb, unsigned seed) : rng(seed) {
    memset(&g, 0, sizeof(g));
    g.N1 = g.N1 = N1; g.N2 = g.N2F = N2; g.N1h = g.N1hF = N1 / 2 + 1; g.ncol = g.ncolF = g.N1h * N2;
    g.nu = nu; g.nv = nu - 1; g.np = nu - 2; g.nuI = nu - 2; g.nvI = nu - 3; g.nn = nu - 2;
    nU = 2 * (size_t)g.nu * g.ncol; nV = 2 * (size_t)g.nv * g.ncol; nP = 2 * (size_t)g.np * g.ncol;
    const int m = nu / 4, t = nu - 1 - m;
    const int bq[3][6] = {{0, m, 0, m - 1, 0, m - 2}, {0, nu - 1, 0, nu - 2, 0, nu - 3}, {t, nu - 1, t, nu - 2, t, nu - 3}};
    memcpy(g.bq, bq, sizeof(bq));
    g.mb = mb;
    g.nvc = g.ncol;
    if (mb) {
      std::vector<int2> lo, hi, all;
      for (int c = 0; c < g.ncol; ++c) {
        if (c % g.N1h <= N1 / 4) all.push_back(make_int2(c, 1));
        else { lo.push_back(make_int2(c, 0)); hi.push_back(make_int2(c, 2)); }
      }
      all.insert(all.end(), lo.begin(), lo.end());
      all.insert(all.end(), hi.begin(), hi.end());
      g.nvc = (int)all.size();
      g.vcol = to_device(all);
    }
    // second differences: positive neighbours, the diagonal minus their sum
    auto d2 = [&](int n, const double *&d, const float *&f, const float *&sum) {
      std::vector<double> v = reals(3 * n, 20.0, 90.0);
      for (int q = 0; q < n; ++q) v[n + q] = -(v[q] + v[2 * n + q]);
      std::vector<float> vf(v.begin(), v.end()), s(n, 0.f);
      d = to_device(v); f = to_device(vf); sum = to_device(s);
    };
    d2(g.nu, g.d2u, g.d2uf, g.sdgu);
    d2(g.nv, g.d2v, g.d2vf, g.sdgv);
    const std::vector<double> tu = reals(g.nu, 0.5, 2.0), tv = reals(g.nv, 0.5, 2.0);
    g.thu = to_device(tu); g.thv = to_device(tv); g.thud = to_device(reals(g.nu, 2.0, 9.0));
    g.thuf = to_device(std::vector<float>(tu.begin(), tu.end()));
    g.thvf = to_device(std::vector<float>(tv.begin(), tv.end()));
    std::vector<double> kx(g.N1h), kx2(g.N1h), kz(N2), kz2(N2);
    for (int i = 0; i < g.N1h; ++i) { kx[i] = i; kx2[i] = -kx[i] * kx[i]; }
    for (int r = 0; r < N2; ++r) { kz[r] = 2.0 * (r < N2 / 2 ? r : r - N2); kz2[r] = -kz[r] * kz[r]; }
    g.k1x = to_device(kx); g.k2x = to_device(kx2); g.k1z = to_device(kz); g.k2z = to_device(kz2);
    g.Re = 3250.0; g.dd = 3.7;
    const double a[3] = {29.0 / 96, -3.0 / 40, 1.0 / 6}, b[3] = {37.0 / 160, 5.0 / 24, 1.0 / 6};
    const double c[3] = {0.0, -17.0 / 60, -5.0 / 12}, d[3] = {8.0 / 15, 2.0 / 15, 1.0 / 3}, e[3] = {8.0 / 15, 5.0 / 12, 3.0 / 4};
    memcpy(g.aRK, a, sizeof(a)); memcpy(g.bRK, b, sizeof(b)); memcpy(g.cRK, c, sizeof(c));
    memcpy(g.dRK, d, sizeof(d)); memcpy(g.gRK, e, sizeof(e));
    for (int i = 0; i < 3; ++i) { g.gw[i][0] = 0.31; g.gw[i][1] = 0.27; }
    g.gwbc1 = g.gwbc3 = -0.4;
    DevScalars h;
    memset(&h, 0, sizeof(h));
    h.dt = 0.013; h.dti = 1.0 / 0.013; h.mpgx = -0.003;
    sc = to_device(std::vector<DevScalars>(1, h));
  }
};
