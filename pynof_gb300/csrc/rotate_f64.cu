// Orbital rotation C' = C expm(Y) on the device, FP64 (rotate_orbital,
// utils.py:550-565): Y is the antisymmetric matrix whose strict upper
// triangle, rows i < nbf5, holds the packed step y (row-major over (i, j > i),
// the order of numpy's triu_indices(nbf, 1) restricted to i < nbf5).
//
// expm by scaling and squaring: X = Y / 2^s with ||X||_1 <= 1/2, the degree-16
// Taylor polynomial of X (truncation < 0.5^17 / 17! ~ 2e-20 relative), then s
// squarings.  X is antisymmetric, so Z = X^2 and every polynomial in it are
// symmetric, and half of each such product is computed:
//   p(X) = E(Z) + X O(Z),  E = sum_k Z^k / (2k)!,  O = sum_k Z^k / (2k+1)!,
//   E = e0 + e1 Z + e2 Z^2 + e3 Z^3 + Z^4 (e4 + e5 Z + e6 Z^2 + e7 Z^3 + e8 Z^4),
// O alike with k <= 7.  Products: Z, Z^2, then Z^3 and Z^4 as one launch, both
// brackets times Z^4 as one launch, and X O, the only one computed whole: four
// products' work in five launches, where a Horner scheme in X^4 took six of each.
// Then s squarings and the final C U.  Bound by the FP64 pipe: at nbf=300 with three
// squarings 481 us, 586 before (the Horner scheme, nine products and C U of 62 us each).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "f64_tc.cuh"

using namespace gb;

namespace {

constexpr int TAYLOR_DEG = 16;

// Y[i][j] from the packed step: +y for i < j (i < P), -y for i > j (j < P).
__global__ void build_antisym_kernel(const double* __restrict__ y, int N, int P, double* __restrict__ Y) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)N * N) return;
  const int i = (int)(idx / N), j = (int)(idx % N);
  double v = 0.0;
  const int lo = i < j ? i : j, hi = i < j ? j : i;
  if (lo != hi && lo < P) {
    // offset of row lo in the packed upper triangle: sum_{r < lo} (N - 1 - r)
    const long long off = (long long)lo * (N - 1) - (long long)lo * (lo - 1) / 2;
    v = y[off + (hi - lo - 1)];
    if (i > j) v = -v;
  }
  Y[idx] = v;
}

// norm[0] = max_j sum_i |Y[i][j]| (bit-pattern max: non-negative doubles order as integers)
__global__ void col_abs_max_kernel(const double* __restrict__ Y, int N, unsigned long long* __restrict__ norm) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  double s = 0.0;
  for (int i = 0; i < N; ++i) s += fabs(Y[(long long)i * N + j]);
  atomicMax(norm, (unsigned long long)__double_as_longlong(s));
}

// The coefficients of E and O: 1 / (2k)! and 1 / (2k+1)!
struct Coefs {
  double e[9], o[9];
};

// HIGH: the brackets that Z^4 multiplies, dst = [E's, O's], from Z, Z^2 (z) and Z^3,
// Z^4 (q).  Otherwise the whole: dst = [E, O], from the products w, Z, Z^2 and Z^3.
template <bool HIGH>
__global__ void poly_kernel(double* __restrict__ dst, const double* __restrict__ z, const double* __restrict__ q,
                            const double* __restrict__ w, int N, const __grid_constant__ Coefs c) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x, NN = (long long)N * N;
  if (idx >= NN) return;
  const bool diag = idx / N == idx % N;
  const double z1 = z[idx], z2 = z[NN + idx], z3 = q[idx], z4 = HIGH ? q[NN + idx] : 0.0;
  constexpr int B = HIGH ? 4 : 0;
  double e = HIGH ? c.e[8] * z4 : w[idx], o = HIGH ? 0.0 : w[NN + idx];
  if (diag) {
    e += c.e[B];
    o += c.o[B];
  }
  e = fma(c.e[B + 3], z3, fma(c.e[B + 2], z2, fma(c.e[B + 1], z1, e)));
  o = fma(c.o[B + 3], z3, fma(c.o[B + 2], z2, fma(c.o[B + 1], z1, o)));
  dst[idx] = e;
  dst[NN + idx] = o;
}

__global__ void scale_kernel(const double* __restrict__ src, double* __restrict__ dst, long long n, double f) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < n) dst[idx] = src[idx] * f;
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// C = A B (+ C when accumulate), square row-major N x N; sym: the product is
// symmetric.  batch: consecutive A and C, one B.
int matmul(const double* A, const double* B, double* C, int N, bool accumulate, const TcWork& tw, cudaStream_t s,
           const char* tag, int sym = SYM_NONE, int batch = 1) {
  const long long NN = batch > 1 ? (long long)N * N : 0;
  GemmF64 g{};
  g.M = N; g.N = N; g.K = N; g.batch = batch;
  g.A = {A, NN, lin(N), lin(1)};
  g.B = {B, 0, lin(N), lin(1)};
  g.C = {C, NN, lin(N), lin(1)};
  g.alpha = 1.0; g.beta = accumulate ? 1.0 : 0.0; g.sym = sym;
  g.a_kfast = true; g.b_kfast = false;
  g.tag = tag;
  return gemm_f64_tc(g, tw, s);
}

template <class Cv>
void rotate_layout(Cv& c, int N, double** bufs, unsigned long long** norm) {
  // X, then pairs: Z Z^2, Z^3 Z^4, the brackets (then E, O), their products
  for (int k = 0; k < 5; ++k) {
    double* p = c.template take<double>((size_t)(k == 0 ? 1 : 2) * N * N);
    if (bufs) bufs[k] = p;
  }
  auto* nm = c.template take<unsigned long long>(1);
  if (norm) *norm = nm;
}

}  // namespace

extern "C" size_t gb_rotate_orbital_workspace_f64(int nbf) {
  SizeCarve c;
  rotate_layout(c, nbf, nullptr, nullptr);
  size_t tc = gemm_f64_tc_bytes(nbf, nbf, nbf, 1, true, true);
  tc = std::max(tc, gemm_f64_tc_bytes(nbf, nbf, nbf, 1, true, true, SYM_ROWCOL));
  tc = std::max(tc, gemm_f64_tc_bytes(nbf, nbf, nbf, 2, false, true, SYM_ROWCOL));
  return c.used + align256(tc);
}

extern "C" int gb_rotate_orbital_f64(const double* y, const double* C, int nbf, int nbf5, double norm1,
                                     double* Cout, void* workspace, size_t workspace_bytes, void* stream) {
  clear_error();
  const int N = nbf, P = nbf5;
  GB_REQUIRE(N > 0 && P > 0 && P <= N, GB_ERR_BAD_SHAPE, "gb_rotate_orbital_f64: need 0 < nbf5 <= nbf");
  GB_REQUIRE(y && C && Cout, GB_ERR_INVALID_ARG, "gb_rotate_orbital_f64: null pointer");
  GB_REQUIRE(C != Cout, GB_ERR_INVALID_ARG, "gb_rotate_orbital_f64: C and Cout must not alias");
  SizeCarve base;
  rotate_layout(base, N, nullptr, nullptr);
  GB_REQUIRE(workspace_bytes >= base.used, GB_ERR_WORKSPACE,
             "gb_rotate_orbital_f64: workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Carve wc(workspace, workspace_bytes);
  double* buf[5];
  unsigned long long* dnorm = nullptr;
  rotate_layout(wc, N, buf, &dnorm);
  const TcWork tw = tc_work(wc);
  double *Y = buf[0], *Z = buf[1], *Q = buf[2], *B = buf[3], *W = buf[4];
  const long long NN = (long long)N * N;

  GB_LAUNCH_CHAIN("rotate_build", s, build_antisym_kernel, dim3(cdiv(NN, 256)), dim3(256), 0, y, N, P, Y);
  double norm = norm1;
  if (!(norm1 >= 0.0)) {
    // no bound from the caller: measure ||Y||_1 on the device (one synchronisation)
    GB_TRY(cuda_status(cudaMemsetAsync(dnorm, 0, sizeof(unsigned long long), s), "cudaMemsetAsync"));
    GB_LAUNCH("rotate_norm", s, col_abs_max_kernel<<<cdiv(N, 128), 128, 0, s>>>(Y, N, dnorm));
    unsigned long long nbits = 0;
    GB_TRY(cuda_status(cudaMemcpyAsync(&nbits, dnorm, sizeof(nbits), cudaMemcpyDeviceToHost, s), "norm copy"));
    GB_TRY(cuda_status(cudaStreamSynchronize(s), "cudaStreamSynchronize"));
    memcpy(&norm, &nbits, sizeof(norm));
  }
  GB_REQUIRE(std::isfinite(norm), GB_ERR_NONFINITE, "gb_rotate_orbital_f64: step y is not finite");
  GB_REQUIRE(norm < 0x1p60, GB_ERR_INVALID_ARG, "gb_rotate_orbital_f64: step norm %g too large", norm);
  int sq = 0;
  while (norm > 0.5) {
    norm *= 0.5;
    ++sq;
  }
  // X = Y / 2^sq in place
  if (sq > 0)
    GB_LAUNCH_CHAIN("rotate_scale", s, scale_kernel, dim3(cdiv(NN, 256)), dim3(256), 0, Y, Y, NN,
                    std::ldexp(1.0, -sq));
  const double* X = Y;
  Coefs c{};
  double f = 1.0;
  for (int k = 0; k <= TAYLOR_DEG; ++k) {
    if (k > 0) f /= k;
    (k % 2 ? c.o : c.e)[k / 2] = f;
  }
  const char* tag = "gemm_f64:expm";
  GB_TRY(matmul(X, X, Z, N, false, tw, s, tag, SYM_ROWCOL));
  GB_TRY(matmul(Z, Z, Z + NN, N, false, tw, s, tag, SYM_ROWCOL));
  GB_TRY(matmul(Z, Z + NN, Q, N, false, tw, s, tag, SYM_ROWCOL, 2));
  GB_LAUNCH_CHAIN("rotate_poly", s, poly_kernel<true>, dim3(cdiv(NN, 256)), dim3(256), 0, B, Z, Q, nullptr, N, c);
  GB_TRY(matmul(B, Q + NN, W, N, false, tw, s, tag, SYM_ROWCOL, 2));
  GB_LAUNCH_CHAIN("rotate_poly", s, poly_kernel<false>, dim3(cdiv(NN, 256)), dim3(256), 0, B, Z, Q, W, N, c);
  // R = E + X O
  double* R = B;
  GB_TRY(matmul(X, B + NN, R, N, true, tw, s, tag));
  // s squarings, ping-ponging between R and a free buffer
  double* spare = W;
  for (int k = 0; k < sq; ++k) {
    GB_TRY(matmul(R, R, spare, N, false, tw, s, "gemm_f64:expm"));
    double* t = R;
    R = spare;
    spare = t;
  }
  return matmul(C, R, Cout, N, false, tw, s, "gemm_f64:rotate");
}
