// Every form of the mixed solves and of the pressure step on the same data (tests/test_gpu_variants.py):
// the fused kernels with 0 (register prefetch), 2, 4 and 8 levels staged and blocks of 64, 128 and 256
// threads, and the split launches. Prints per form and case the values that differ from the split ones'.
#include <cstring>
#include <string>

#include "solve_case.cuh"

static size_t staged(int nlev, int pf, int tb) {
  return pf == 0 ? 0 : (((size_t)6 * nlev * 4 + 15) & ~(size_t)15) + (size_t)28 * (pf + 1) * tb;
}
static size_t staged_press(const Geo &g, int pf, int tb) {
  return pf == 0 ? 8 * (size_t)(g.nu + g.nv) : 8 * (((size_t)g.nu + g.nv + 1) & ~(size_t)1) + (size_t)48 * (pf + 1) * tb;
}
// a == b in value (both zeros are one, and so are all NaN)
template <typename T>
static long differ(const std::vector<T> &a, const std::vector<T> &b) {
  long n = 0;
  for (size_t i = 0; i < a.size(); ++i) n += !(a[i] == b[i] || (a[i] != a[i] && b[i] != b[i]));
  return n;
}

// ---- pressure ----
struct Press { std::vector<double> u, v, w, p; unsigned long long err; };
static Press press(SolveCase &s, const Press &in, const double *dg1, const double *dg2, const double *dg3, int kRK, int pf, int tb) {
  const Geo &g = s.g;
  double *u = to_device(in.u), *v = to_device(in.v), *w = to_device(in.w), *p = to_device(in.p), *psi, *faces;
  CKC(cudaMalloc(&psi, sizeof(double) * s.nP));
  CKC(cudaMemset(psi, 0, sizeof(double) * s.nP));
  CKC(cudaMalloc(&faces, press_faces_bytes(g)));
  CKC(cudaMemset(&s.sc->errbits, 0, sizeof(unsigned long long)));
  const int nd = kRK == 3;
  if (pf < 0) {
    const dim3 ge((g.nvc + 127) / 128, press_chunks(g));
    double2 *U = (double2 *)u, *V = (double2 *)v, *W = (double2 *)w, *P = (double2 *)p, *S = (double2 *)psi,
            *F = nd ? (double2 *)faces : nullptr;
    k_press_rhs<<<ge, 128>>>(U, V, W, S, F, g, s.sc, kRK);
    k_press_sweep<<<(2 * g.nvc + 31) / 32, 32>>>(psi, dg1, dg2, dg3, g);
    if (nd) k_press_corr<true><<<ge, 128>>>(U, V, W, P, S, F, g, s.sc, kRK);
    else k_press_corr<false><<<ge, 128>>>(U, V, W, P, S, F, g, s.sc, kRK);
  } else {
    const int nb = (2 * g.nvc + tb - 1) / tb;
    const size_t sm = staged_press(g, pf, tb);
    switch (pf) {
      case 0: k_press2<<<nb, tb, sm>>>(u, v, w, p, psi, dg1, dg2, dg3, g, s.sc, kRK, nd); break;
      case 2: k_press3<2><<<nb, tb, sm>>>(u, v, w, p, psi, dg1, dg2, dg3, g, s.sc, kRK, nd); break;
      case 4: k_press3<4><<<nb, tb, sm>>>(u, v, w, p, psi, dg1, dg2, dg3, g, s.sc, kRK, nd); break;
      default: k_press3<8><<<nb, tb, sm>>>(u, v, w, p, psi, dg1, dg2, dg3, g, s.sc, kRK, nd);
    }
  }
  CKC(cudaGetLastError());
  CKC(cudaDeviceSynchronize());
  Press o = {to_host(u, s.nU), to_host(v, s.nV), to_host(w, s.nU), to_host(p, s.nP), to_host(&s.sc->errbits, 1)[0]};
  for (double *q : {u, v, w, p, psi, faces}) CKC(cudaFree(q));
  return o;
}

// ---- mixed Helmholtz ----
struct Helm { std::vector<double> f[3], p; std::vector<float> N[3], X[3], F[3]; };  // u, w, v
static Helm helm(SolveCase &s, const Helm &in, const int *iu, const int *iv, const float2 *duib, int kRK, int pf, int tb) {
  const Geo &g = s.g;
  double *f[3], *p = to_device(in.p);
  float *N[3], *X[3], *F[3];
  float2 *ys;
  for (int i = 0; i < 3; ++i) { f[i] = to_device(in.f[i]); N[i] = to_device(in.N[i]); X[i] = to_device(in.X[i]); F[i] = to_device(in.F[i]); }
  CKC(cudaMalloc(&ys, sizeof(float2) * 3 * s.nU));
  float2 *ysv = ys + 2 * s.nU;
  if (pf < 0) {
    HelmMxArgs a = {{f[0], f[1], f[2]}, {N[0], N[1], N[2]}, {X[0], X[1], X[2]}, {F[0], F[1], F[2]}, p,
                    {ys, ys + s.nU, ysv}, {iu, iu, iv}, duib, kRK};
    k_helm_rhs_mx<<<dim3(3 * ((2 * g.nvc + 127) / 128), (g.nu + LH_HL - 1) / LH_HL), 128>>>(a, g, s.sc);
    k_helm_sweep_mx<<<dim3((2 * g.nvc + LH_HS_T - 1) / LH_HS_T, 3), LH_HS_T, hsweep_mx_smem(g.nu)>>>(a, g, s.sc);
  } else {
    const int nb = (2 * g.nvc + tb - 1) / tb;
    const size_t su = staged(g.nu, pf, tb), sv = staged(g.nv, pf, tb);
    const double2 *P = (const double2 *)p;
    switch (pf) {
      case 0:
        k_helm_u_mx2<<<dim3(nb, 2), tb, su>>>(f[0], f[1], N[0], N[1], X[0], X[1], F[0], F[1], P, ys, g, s.sc, kRK, iu, duib);
        k_helm_v_mx2<<<nb, tb, sv>>>(f[2], N[2], X[2], F[2], p, ysv, g, s.sc, kRK, iv, duib);
        break;
      case 2:
        k_helm_u_mx3<2><<<dim3(nb, 2), tb, su>>>(f[0], f[1], N[0], N[1], X[0], X[1], F[0], F[1], P, ys, g, s.sc, kRK, iu, duib);
        k_helm_v_mx3<2><<<nb, tb, sv>>>(f[2], N[2], X[2], F[2], p, ysv, g, s.sc, kRK, iv, duib);
        break;
      case 4:
        k_helm_u_mx3<4><<<dim3(nb, 2), tb, su>>>(f[0], f[1], N[0], N[1], X[0], X[1], F[0], F[1], P, ys, g, s.sc, kRK, iu, duib);
        k_helm_v_mx3<4><<<nb, tb, sv>>>(f[2], N[2], X[2], F[2], p, ysv, g, s.sc, kRK, iv, duib);
        break;
      default:
        k_helm_u_mx3<8><<<dim3(nb, 2), tb, su>>>(f[0], f[1], N[0], N[1], X[0], X[1], F[0], F[1], P, ys, g, s.sc, kRK, iu, duib);
        k_helm_v_mx3<8><<<nb, tb, sv>>>(f[2], N[2], X[2], F[2], p, ysv, g, s.sc, kRK, iv, duib);
    }
  }
  CKC(cudaGetLastError());
  CKC(cudaDeviceSynchronize());
  Helm o;
  for (int i = 0; i < 3; ++i) { o.f[i] = to_host(f[i], in.f[i].size()); o.N[i] = to_host(N[i], in.N[i].size()); }
  for (int i = 0; i < 3; ++i) { CKC(cudaFree(f[i])); CKC(cudaFree(N[i])); CKC(cudaFree(X[i])); CKC(cudaFree(F[i])); }
  CKC(cudaFree(p));
  CKC(cudaFree(ys));
  return o;
}

int main() {
  int optin = 0;
  CKC(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0));
  const void *kern[] = {(const void *)k_press3<2>, (const void *)k_press3<4>, (const void *)k_press3<8>, (const void *)k_helm_u_mx3<2>,
                        (const void *)k_helm_u_mx3<4>, (const void *)k_helm_u_mx3<8>, (const void *)k_helm_v_mx3<2>,
                        (const void *)k_helm_v_mx3<4>, (const void *)k_helm_v_mx3<8>};
  for (const void *k : kern) CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
  const int depths[] = {0, 2, 4, 8}, blocks[] = {64, 128, 256};
  struct Shape { int N1, N2, nu; bool mb, ib; };
  // 72, 136 and 612 columns; levels of every remainder modulo the staging depths and the split's chunks
  const Shape shapes[] = {{16, 8, 11, false, false}, {16, 8, 12, false, true}, {16, 8, 29, true, false}, {32, 8, 38, false, true},
                          {32, 8, 47, true, false}, {32, 36, 64, false, false}};
  for (const Shape &z : shapes)
    for (int k = 1; k <= 3; ++k) {
      SolveCase s(z.N1, z.N2, z.nu, z.mb, 31 * z.nu + k);
      const Geo &g = s.g;
      const size_t nd = (size_t)g.np * g.ncol;
      double *dg1 = to_device(s.reals(nd, -0.4, 0.4)), *dg2 = to_device(s.reals(nd, 0.5, 1.0)), *dg3 = to_device(s.reals(nd, -0.4, 0.4));
      const Press pin = {s.reals(s.nU, -1, 1), s.reals(s.nV, -1, 1), s.reals(s.nU, -1, 1), s.reals(s.nP, -1, 1), 0};
      Helm hin;
      hin.p = s.reals(s.nP, -1, 1);
      for (int i = 0; i < 3; ++i) {
        const size_t n = i == 2 ? s.nV : s.nU;
        hin.f[i] = s.reals(n, -1, 1);
        hin.N[i] = s.floats(n, -1, 1); hin.X[i] = s.floats(n, -1, 1);
        hin.F[i] = s.floats(i == 2 ? s.nU : s.nV, -1, 1);
      }
      // immersed levels: the lowest and highest two interior ones
      std::vector<int> slu(g.nu, -1), slv(g.nv, -1);
      if (z.ib) {
        slu[1] = slv[1] = 0; slu[2] = slv[2] = 1;
        slu[g.nu - 3] = slv[g.nv - 3] = 2; slu[g.nu - 2] = slv[g.nv - 2] = 3;
      }
      int *iu = z.ib ? to_device(slu) : nullptr, *iv = z.ib ? to_device(slv) : nullptr;
      float *duib = to_device(s.floats((size_t)4 * 3 * 2 * g.ncol, -1, 1));
      const Press p0 = press(s, pin, dg1, dg2, dg3, k, -1, 0);
      const Helm h0 = helm(s, hin, iu, iv, (const float2 *)duib, k, -1, 0);
      for (int pf : depths)
        for (int tb : blocks) {
          const Press p = press(s, pin, dg1, dg2, dg3, k, pf, tb);
          const Helm h = helm(s, hin, iu, iv, (const float2 *)duib, k, pf, tb);
          const long dp = differ(p.u, p0.u) + differ(p.v, p0.v) + differ(p.w, p0.w) + differ(p.p, p0.p) + (p.err != p0.err);
          long du = 0, dv = differ(h.f[2], h0.f[2]) + differ(h.N[2], h0.N[2]);
          for (int i = 0; i < 2; ++i) du += differ(h.f[i], h0.f[i]) + differ(h.N[i], h0.N[i]);
          printf("%d %d %d %d %d %d %d %ld %ld %ld %d\n", z.N1, z.N2, z.nu, (int)z.mb, k, pf, tb, dp, du, dv, (int)(p0.err != 0));
        }
      for (double *q : {dg1, dg2, dg3}) CKC(cudaFree(q));
      CKC(cudaFree(duib));
    }
  return 0;
}
