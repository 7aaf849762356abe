// The split pressure step's right-hand side of mode (0,0) (tests/test_gpu_press_mean.py): u and w of that
// column hold NaN, as a value that another kernel is about to write may. Prints the psi values that are
// not finite, or, in the column, not thud dti / (a + b) dv (three roundings on either side: 7e-16).
#include <cstring>

#include "solve_case.cuh"

int main() {
  long bad = 0, n = 0;
  for (int mb = 0; mb < 2; ++mb)
    for (int nu : {11, 18, 43})
      for (int k = 1; k <= 3; ++k) {
        SolveCase s(16, 8, nu, mb, 100 * nu + k);
        const Geo &g = s.g;
        std::vector<double> u = s.reals(s.nU, -1, 1), v = s.reals(s.nV, -1, 1), w = s.reals(s.nU, -1, 1);
        for (int q = 0; q < nu; ++q)
          for (int t = 0; t < 2; ++t) u[2 * (size_t)q * g.ncol + t] = w[2 * (size_t)q * g.ncol + t] = NAN;
        double *d[3] = {to_device(u), to_device(v), to_device(w)}, *psi, *faces;
        CKC(cudaMalloc(&psi, sizeof(double) * s.nP));
        CKC(cudaMemset(psi, 0, sizeof(double) * s.nP));
        CKC(cudaMalloc(&faces, press_faces_bytes(g)));
        k_press_rhs<<<dim3((g.nvc + 127) / 128, press_chunks(g)), 128>>>((double2 *)d[0], (double2 *)d[1], (double2 *)d[2],
                                                                        (double2 *)psi, k == 3 ? (double2 *)faces : nullptr, g, s.sc, k);
        CKC(cudaDeviceSynchronize());
        const std::vector<double> out = to_host(psi, s.nP), th = to_host(g.thud, nu);
        const double f = (1.0 / 0.013) / (g.aRK[k - 1] + g.bRK[k - 1]);
        for (size_t i = 0; i < s.nP; ++i, ++n) {
          const size_t qp = i / (2 * g.ncol), c = i % (2 * g.ncol);
          bool ok = isfinite(out[i]);
          if (c < 2) {  // its first level is the gauge
            const double e = qp == 0 ? 0.0 : f * th[qp + 1] * (v[(qp + 1) * 2 * g.ncol + c] - v[qp * 2 * g.ncol + c]);
            ok = ok && fabs(out[i] - e) <= 1e-15 * fabs(e);
          }
          bad += !ok;
        }
        for (double *p : d) CKC(cudaFree(p));
        CKC(cudaFree(psi));
        CKC(cudaFree(faces));
      }
  printf("%ld %ld\n", n, bad);
  return 0;
}
