// Orbital rotation C' = C expm(Y) on the device, FP64 (rotate_orbital,
// utils.py:550-565): Y is the antisymmetric matrix whose strict upper
// triangle, rows i < nbf5, holds the packed step y (row-major over (i, j > i),
// the order of numpy's triu_indices(nbf, 1) restricted to i < nbf5).
//
// expm by scaling and squaring: X = Y / 2^s with ||X||_1 <= 1/2, the degree-16
// Taylor polynomial of X (truncation < 0.5^17 / 17! ~ 2e-20 relative), then s
// squarings.  X is antisymmetric, so Z = X^2 and every polynomial in it are
// symmetric, and half of each such product is computed:
//   p(X) - I = E(Z) + X + X O(Z),  E = sum_(k>0) Z^k / (2k)!,  O = sum_(k>0) Z^k / (2k+1)!,
//   E = e1 Z + e2 Z^2 + e3 Z^3 + e4 Z^4 + (e5 Z + e6 Z^2 + e7 Z^3 + e8 Z^4) Z^4,
// O alike with k <= 7.  Products: Z, Z^2, then Z^3 and Z^4 as one launch, both
// brackets times Z^4 as one launch, and X O, the only one computed whole: four
// products' work in five launches.  Then s squarings of F = p - I, 2 F + F F, and the
// final C + C F.  Without the identity in them no operand's rows are near multiples
// of it, whose products the tensor cores would leave to FP64 arithmetic
// (f64_tc.cuh): at nbf=600 4.8 ms with it, 0.97 ms without, and an error of 2e-15
// instead of 2e-14.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "f64_tc.cuh"

using namespace gb;

namespace {

constexpr int TAYLOR_DEG = 16;

// Y[i][j] from the packed step: +y for i < j (i < P), -y for i > j (j < P),
// scaled by the power of two f.
__global__ void build_antisym_kernel(const double* __restrict__ y, int N, int P, double f, double* __restrict__ Y) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)N * N) return;
  const int i = (int)(idx / N), j = (int)(idx % N);
  double v = 0.0;
  const int lo = i < j ? i : j, hi = i < j ? j : i;
  if (lo != hi && lo < P) {
    // offset of row lo in the packed upper triangle: sum_{r < lo} (N - 1 - r)
    const long long off = (long long)lo * (N - 1) - (long long)lo * (lo - 1) / 2;
    v = f * y[off + (hi - lo - 1)];
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
  double e[9], o[8];
};

// From Z, Z^2, Z^4, Z^3 in s[0..3]: E's and O's first four terms into s[0], s[1], their
// brackets into s[3], s[4].
__global__ void poly_kernel(double* __restrict__ s, int N, const __grid_constant__ Coefs c) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x, NN = (long long)N * N;
  if (idx >= NN) return;
  double* p = s + idx;
  const double z1 = p[0], z2 = p[NN], z4 = p[2 * NN], z3 = p[3 * NN];
  auto poly = [&](const double* k) { return fma(k[0], z1, fma(k[1], z2, fma(k[2], z3, k[3] * z4))); };
  p[0] = poly(c.e + 1);
  p[NN] = poly(c.o + 1);
  p[3 * NN] = poly(c.e + 5);
  p[4 * NN] = fma(c.o[5], z1, fma(c.o[6], z2, c.o[7] * z3));
}

__global__ void add_kernel(double* __restrict__ dst, const double* __restrict__ src, long long n) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < n) dst[idx] += src[idx];
}

__global__ void scale_kernel(const double* __restrict__ src, double* __restrict__ dst, long long n, double f) {
  chain_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < n) dst[idx] = src[idx] * f;
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// C = A B + beta C0, square row-major N x N; sym: the product is symmetric (and C0).
// batch: two consecutive A, C cs apart, one B.
int matmul(const double* A, const double* B, double* C, int N, double beta, const double* C0, const TcWork& tw,
           cudaStream_t s, const char* tag, int sym = SYM_NONE, long long cs = 0) {
  GemmF64 g{};
  g.M = N; g.N = N; g.K = N; g.batch = cs ? 2 : 1;
  g.A = {A, cs ? (long long)N * N : 0, lin(N), lin(1)};
  g.B = {B, 0, lin(N), lin(1)};
  g.C = {C, cs, lin(N), lin(1)};
  g.alpha = 1.0; g.beta = beta; g.sym = sym; g.C0 = C0;
  g.a_kfast = true; g.b_kfast = false;
  g.tag = tag;
  return gemm_f64_tc(g, tw, s);
}

template <class Cv>
void rotate_layout(Cv& c, int N, double** X, double** S, unsigned long long** norm) {
  // X, and five consecutive: Z, Z^2, Z^4, Z^3 and one more (poly_kernel)
  double* x = c.template take<double>((size_t)N * N);
  double* z = c.template take<double>((size_t)5 * N * N);
  auto* nm = c.template take<unsigned long long>(1);
  if (X) *X = x;
  if (S) *S = z;
  if (norm) *norm = nm;
}

}  // namespace

extern "C" size_t gb_rotate_orbital_workspace_f64(int nbf) {
  SizeCarve c;
  rotate_layout(c, nbf, nullptr, nullptr, nullptr);
  size_t tc = gemm_f64_tc_bytes(nbf, nbf, nbf, 1, true, true);
  tc = std::max(tc, gemm_f64_tc_bytes(nbf, nbf, nbf, 1, true, true, SYM_ROWCOL));
  tc = std::max(tc, gemm_f64_tc_bytes(nbf, nbf, nbf, 2, false, true, SYM_ROWCOL));
  tc = std::max(tc, gemm_f64_tc_bytes(nbf, nbf, nbf, 2, false, true, SYM_ROWCOL, 0, true));
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
  rotate_layout(base, N, nullptr, nullptr, nullptr);
  GB_REQUIRE(workspace_bytes >= base.used, GB_ERR_WORKSPACE,
             "gb_rotate_orbital_f64: workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Carve wc(workspace, workspace_bytes);
  double *Y, *S;
  unsigned long long* dnorm = nullptr;
  rotate_layout(wc, N, &Y, &S, &dnorm);
  const TcWork tw = tc_work(wc);
  const long long NN = (long long)N * N;

  const dim3 grid(cdiv(NN, 256)), block(256);
  double norm = norm1;
  const bool measure = !(norm1 >= 0.0);
  if (measure) {
    // no bound from the caller: measure ||Y||_1 on the device (one synchronisation)
    GB_LAUNCH_CHAIN("rotate_build", s, build_antisym_kernel, grid, block, 0, y, N, P, 1.0, Y);
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
  // X = Y / 2^sq
  if (!measure)
    GB_LAUNCH_CHAIN("rotate_build", s, build_antisym_kernel, grid, block, 0, y, N, P, std::ldexp(1.0, -sq), Y);
  else if (sq > 0)
    GB_LAUNCH_CHAIN("rotate_scale", s, scale_kernel, grid, block, 0, Y, Y, NN, std::ldexp(1.0, -sq));
  const double* X = Y;
  Coefs c{};
  double f = 1.0;
  for (int k = 0; k <= TAYLOR_DEG; ++k) {
    if (k > 0) f /= k;
    (k % 2 ? c.o : c.e)[k / 2] = f;
  }
  const char* tag = "gemm_f64:expm";
  double *Z = S, *Z2 = S + NN, *Z4 = S + 2 * NN, *Z3 = S + 3 * NN;
  GB_TRY(matmul(X, X, Z, N, 0.0, nullptr, tw, s, tag, SYM_ROWCOL));
  GB_TRY(matmul(Z, Z, Z2, N, 0.0, nullptr, tw, s, tag, SYM_ROWCOL));
  GB_TRY(matmul(Z, Z2, Z3, N, 0.0, nullptr, tw, s, tag, SYM_ROWCOL, -NN));
  GB_LAUNCH_CHAIN("rotate_poly", s, poly_kernel, grid, block, 0, S, N, c);
  // E, O += their brackets (S + 3 NN and on) times Z^4
  double *E = S, *O = S + NN;
  GB_TRY(matmul(S + 3 * NN, Z4, E, N, 1.0, E, tw, s, tag, SYM_ROWCOL, NN));
  // F = (E + X) + X O
  GB_LAUNCH_CHAIN("rotate_add", s, add_kernel, grid, block, 0, E, X, NN);
  double *F = S + 3 * NN, *spare = S;
  GB_TRY(matmul(X, O, F, N, 1.0, E, tw, s, tag));
  for (int k = 0; k < sq; ++k) {
    GB_TRY(matmul(F, F, spare, N, 2.0, F, tw, s, tag));
    std::swap(F, spare);
  }
  return matmul(C, F, Cout, N, 1.0, C, tw, s, "gemm_f64:rotate");
}
