// Bandwidth-bound helper kernels of the FP64 RI path.
#include "ri_kernels.cuh"

namespace gb {
namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void contract_diag_kernel(const double* __restrict__ C, const double* __restrict__ T,
                                     double* __restrict__ d, int N, int P, int Q) {
  chain_wait();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  if (l >= Q) return;
  const double* Tq = T + (long long)q * N * Q + l;
  double acc = 0.0;
  for (int n = 0; n < N; ++n) acc = fma(__ldg(C + (long long)n * N + q), __ldg(Tq + (long long)n * Q), acc);
  d[(long long)q * Q + l] = acc;
}

// The same contraction, also recording the row exponents of T's digit
// slicing with rows (q, n) and K = l: texps[q N + n] = E with
// |T[q][n][l]| < 2^E for all l (entries preset below any E).  A warp holds 32
// consecutive l; the exponent field's maximum over them comes from one warp
// reduction per n and lands in lane n % 32, which folds it in with atomicMax
// every 32 n.
// A NaN or an infinity in T (exponent field 0x7FF) is reported in the status
// word, as the slicer does for the rows it measures.
// Two rows of T are loaded before either is used: 783 us against 869 at nbf=600
// (FP64 arithmetic alone ~790), 62 against 73 at nbf=171; with eight it was 1054
// and 57.
__global__ void contract_diag_exps_kernel(const double* __restrict__ C, const double* __restrict__ T,
                                          double* __restrict__ d, int* __restrict__ texps, int N, int P, int Q,
                                          int* status) {
  constexpr int U = 2;
  chain_wait();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  const int lane = threadIdx.x & 31;
  const bool in = l < Q;  // the whole warp stays for the reductions
  const double* Tq = T + (long long)q * N * Q + (in ? l : 0);
  int* eq = texps + (long long)q * N;
  double acc = 0.0;
  unsigned int mine = 0;  // exponent field maximum of row n0 + lane
  for (int n0 = 0; n0 < N; n0 += 32) {
    const int nn = min(32, N - n0);
    for (int j0 = 0; j0 < nn; j0 += U) {
      double t[U], c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int n = n0 + j0 + u;
        const bool ok = n < N;
        t[u] = in && ok ? __ldg(Tq + (long long)n * Q) : 0.0;
        c[u] = ok ? __ldg(C + (long long)n * N + q) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j0 + u < nn) acc = fma(c[u], t[u], acc);
        const unsigned int ex = (unsigned int)((unsigned long long)__double_as_longlong(t[u]) >> 52) & 0x7FFu;
        const unsigned int mx = __reduce_max_sync(0xffffffffu, ex);
        if (lane == j0 + u) mine = mx;
      }
    }
    if (lane < nn) {
      atomicMax(eq + n0 + lane, (int)(mine > 1u ? mine : 1u) - 1022);
      if (mine == 0x7FFu && status) atomicCAS(status, 0, GB_ERR_NONFINITE);
    }
  }
  if (in) d[(long long)q * Q + l] = acc;
}

// Exponent E of |x| < 2^E from the exponent field (or the bits) of the largest |x|.
__device__ __forceinline__ int field_exponent(unsigned int field) { return (int)(field > 1u ? field : 1u) - 1022; }
__device__ __forceinline__ unsigned int exp_field(double x) {
  return ((unsigned int)__double2hiint(x) >> 20) & 0x7FFu;
}

// A thread's l keeps its maximum over m; a warp's 32 l share one reduction per m,
// which lands in lane m % 32 and is folded in with atomicMax every 32 m.  One read
// of T, where two exponent passes read it twice.
__global__ void __launch_bounds__(128) t_exponents_kernel(const double* __restrict__ T, int* __restrict__ et,
                                                          int* __restrict__ ex, int N, int Q, int qps, int* status) {
  constexpr int U = 4;
  chain_wait();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  const int lane = threadIdx.x & 31;
  const bool in = l < Q;  // the whole warp stays for the reductions
  const double* Tq = T + (long long)q * N * Q + (in ? l : 0);
  int* e = ex + (long long)(q / qps) * N;
  unsigned int over_m = 0, mine = 0;
  for (int m0 = 0; m0 < N; m0 += 32) {
    const int nm = min(32, N - m0);
    for (int j0 = 0; j0 < nm; j0 += U) {
      double t[U];
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = in && j0 + u < nm ? __ldg(Tq + (long long)(m0 + j0 + u) * Q) : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned int f = exp_field(t[u]);
        over_m = max(over_m, f);
        const unsigned int mx = __reduce_max_sync(0xffffffffu, f);
        if (lane == j0 + u) mine = mx;
      }
    }
    if (lane < nm) atomicMax(e + m0 + lane, field_exponent(mine));
  }
  if (in) {
    et[(long long)q * Q + l] = field_exponent(over_m);
    if (over_m == 0x7FFu && status) atomicCAS(status, 0, GB_ERR_NONFINITE);
  }
}

// One warp per pair q <= b: the largest |bMO[b][q][l]|, whose scaled value bounds
// both rows' operands (the product is rounded monotonically), and the square sum.
__global__ void __launch_bounds__(256) mo_rows_kernel(const double* __restrict__ bMO, const double* __restrict__ ck12,
                                                      const double* __restrict__ w, int* __restrict__ ey,
                                                      double* __restrict__ K_MO, int P, int Q, int qps, int* status) {
  chain_wait();
  const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= (long long)P * P) return;
  const int b = (int)(r / P), q = (int)(r % P);
  if (q > b) return;
  const double* x = bMO + r * Q;
  const double* y = w + (long long)b * Q;
  double sum = 0.0;
  unsigned long long mx = 0;
  auto largest = [&](double v) {
    const unsigned long long a = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
    mx = a > mx ? a : mx;
  };
  // four loads and four sums in flight (an FP64 FMA's latency is 64 clocks here)
  double part[4] = {};
  for (int l0 = lane; l0 < Q; l0 += 128) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = l0 + 32 * u < Q ? __ldg(x + l0 + 32 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (K_MO) part[u] = fma(v[u], v[u], part[u]);
      if (q < b) largest(v[u]);
    }
  }
  sum = (part[0] + part[1]) + (part[2] + part[3]);
  if (q == b)
    for (int l = lane; l < Q; l += 32) largest(y[l]);
  if (K_MO) sum = warp_sum(sum);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx ? v : mx;
  }
  if (lane != 0) return;
  if (K_MO) {
    K_MO[r] = sum;
    K_MO[(long long)q * P + b] = sum;
  }
  auto record = [&](int row, int orb, double v) {
    const unsigned int f = exp_field(v);
    atomicMax(ey + (long long)(orb / qps) * P + row, field_exponent(f));
    if (f == 0x7FFu && status) atomicCAS(status, 0, GB_ERR_NONFINITE);
  };
  const double m = __longlong_as_double((long long)mx);
  if (q == b) {
    record(b, b, m);
  } else {
    record(b, q, ck12[(long long)b * P + q] * m);
    record(q, b, ck12[(long long)q * P + b] * m);
  }
}

__global__ void gather_diag_kernel(const double* __restrict__ src, double* __restrict__ d, int Q,
                                   long long stride_pp) {
  chain_wait();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y;
  if (l < Q) d[(long long)p * Q + l] = src[(long long)p * stride_pp + l];
}

// one warp per row
__global__ void row_sumsq_kernel(const double* __restrict__ src, double* __restrict__ out, long long rows,
                                 int Q,
                                 int sym_p) {
  chain_wait();
  const long long r = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const long long p = sym_p > 0 ? r / sym_p : 0, q = sym_p > 0 ? r % sym_p : 0;
  if (q > p) return;
  const double* s = src + r * Q;
  double acc = 0.0;
  for (int l = lane; l < Q; l += 32) {
    const double v = s[l];
    acc = fma(v, v, acc);
  }
  acc = warp_sum(acc);
  if (lane == 0) {
    out[r] = acc;
    if (sym_p > 0) out[q * sym_p + p] = acc;
  }
}

__global__ void col_dot_kernel(const double* __restrict__ C, int ldc, const double* __restrict__ X, int ldx,
                               double* __restrict__ out, int N, int P) {
  chain_wait();
  const int p = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= P) return;
  double acc = 0.0;
  for (int m = lane; m < N; m += 32) acc = fma(C[(long long)m * ldc + p], X[(long long)m * ldx + p], acc);
  acc = warp_sum(acc);
  if (lane == 0) out[p] = acc;
}

__global__ void copy_zero_diag_kernel(const double* __restrict__ src, double* __restrict__ dst, int P) {
  chain_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)P * P) return;
  const int r = (int)(i / P), c = (int)(i % P);
  dst[i] = (r == c) ? 0.0 : src[i];
}

__global__ void add_scaled_rows_kernel(double* __restrict__ w, const double* __restrict__ d,
                                       const double* __restrict__ n, int P, int Q, int nbeta, int nalpha) {
  chain_wait();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (k >= Q) return;
  if (b < nbeta || b >= nalpha) {
    const long long i = (long long)b * Q + k;
    w[i] = fma(n[b], d[i], w[i]);
  }
}

__global__ void make_ck_weighted_kernel(const double* __restrict__ bMO, const double* __restrict__ ck12,
                                        double* __restrict__ Y, int P, int Q) {
  chain_wait();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  const int b = blockIdx.z;
  if (k >= Q) return;
  const long long i = ((long long)b * P + q) * Q + k;
  const double c = (q == b) ? 0.0 : ck12[(long long)b * P + q];
  Y[i] = c * bMO[i];
}

// one warp per (a, b) with b < P; blocks past the dot range zero elag[:, P:]
__global__ void lagrange2_finish_kernel(const double* __restrict__ bMO, const double* __restrict__ w,
                                        const double* __restrict__ Hmat, const double* __restrict__ n,
                                        double* __restrict__ elag, int N, int P, int Q) {
  chain_wait();
  const long long pair = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (pair >= (long long)N * P) return;
  const int a = (int)(pair / P), b = (int)(pair % P);
  const double* x = bMO + ((long long)a * P + b) * Q;
  const double* y = w + (long long)b * Q;
  double acc = 0.0;
  for (int k = lane; k < Q; k += 32) acc = fma(x[k], y[k], acc);
  acc = warp_sum(acc);
  if (lane == 0) {
    double* e = elag + (long long)a * N + b;
    *e = *e + n[b] * Hmat[(long long)a * P + b] + acc;
  }
}

// Exchange operand of the tensor-core Lagrangian: Y[b][q][k] = ck12[b][q]
// bMO[b][q][k] for q != b and -w[b][k] on the diagonal block q == b, so that
// -sum_(q,k) bMO[a][q][k] Y[b][q][k] also carries + sum_k bMO[a][b][k] w[b][k].
// Grid-stride over (b, q) rows of Q; two elements per thread and step
// (16-byte accesses when Q is even).
__global__ void make_exchange_operand_kernel(const double* __restrict__ bMO, const double* __restrict__ ck12,
                                             const double* __restrict__ w, double* __restrict__ Y, int P, int Q) {
  chain_wait();
  const long long rows = (long long)P * P;
  const int half = Q >> 1;
  const bool even = (Q & 1) == 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const int b = (int)(row / P), q = (int)(row % P);
    const bool diag = q == b;
    const double c = diag ? -1.0 : ck12[(long long)b * P + q];
    const double* src = diag ? w + (long long)b * Q : bMO + row * Q;
    double* dst = Y + row * Q;
    if (even) {
      for (int k2 = threadIdx.x; k2 < half; k2 += blockDim.x) {
        const double2 v = __ldcs(reinterpret_cast<const double2*>(src) + k2);
        __stcs(reinterpret_cast<double2*>(dst) + k2, make_double2(c * v.x, c * v.y));
      }
    } else {
      for (int k = threadIdx.x; k < Q; k += blockDim.x) dst[k] = c * src[k];
    }
  }
}

// elag[a][b] += n[b] Hmat[a][b] for b < P; elag[a][b] = 0 for b >= P
__global__ void lagrange2_hterm_kernel(const double* __restrict__ Hmat, const double* __restrict__ n,
                                       double* __restrict__ elag, int N, int P) {
  chain_wait();
  const long long total = (long long)N * N;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(i / N), b = (int)(i % N);
    elag[i] = b < P ? elag[i] + n[b] * Hmat[(long long)a * P + b] : 0.0;
  }
}

__global__ void zero_tail_cols_kernel(double* __restrict__ elag, int N, int P) {
  chain_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int W = N - P;
  if (i >= (long long)N * W) return;
  const int a = (int)(i / W), c = P + (int)(i % W);
  elag[(long long)a * N + c] = 0.0;
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

int launch_contract_diag(const double* C, const double* T, double* d, int N, int P, int Q, cudaStream_t s,
                         int* texps) {
  if (texps) {
    GB_LAUNCH_CHAIN("contract_diag", s, contract_diag_exps_kernel, dim3(cdiv(Q, 128), P), dim3(128), 0, C, T, d, texps,
                    N, P, Q, device_status_word());
    return GB_OK;
  }
  GB_LAUNCH_CHAIN("contract_diag", s, contract_diag_kernel, dim3(dim3(cdiv(Q, 128), P)), dim3(128), 0, C, T, d, N, P,
                  Q);
  return GB_OK;
}

int launch_gather_diag(const double* src, double* d, int P, int Q, long long stride_pp, cudaStream_t s) {
  GB_LAUNCH_CHAIN("gather_diag", s, gather_diag_kernel, dim3(dim3(cdiv(Q, 128), P)), dim3(128), 0, src, d, Q,
                  stride_pp);
  return GB_OK;
}

int launch_row_sumsq(const double* src, double* out, long long rows, int Q, cudaStream_t s, int sym_p) {
  if (rows <= 0) return GB_OK;
  GB_LAUNCH_CHAIN("row_sumsq", s, row_sumsq_kernel, dim3(cdiv(rows, 8)), dim3(256), 0, src, out, rows, Q, sym_p);
  return GB_OK;
}

int launch_t_exponents(const double* T, int* et, int* ex, int N, int P, int Q, int qps, cudaStream_t s) {
  GB_LAUNCH_CHAIN("t_exponents", s, t_exponents_kernel, dim3(cdiv(Q, 128), P), dim3(128), 0, T, et, ex, N, Q, qps,
                  device_status_word());
  return GB_OK;
}

int launch_mo_rows(const double* bMO, const double* ck12, const double* w, int* ey, double* K_MO, int P, int Q, int qps,
                   cudaStream_t s) {
  GB_LAUNCH_CHAIN("mo_rows", s, mo_rows_kernel, dim3(cdiv((long long)P * P, 8)), dim3(256), 0, bMO, ck12, w, ey, K_MO, P,
                  Q, qps, device_status_word());
  return GB_OK;
}

int launch_col_dot(const double* C, int ldc, const double* X, int ldx, double* out, int N, int P,
                   cudaStream_t s) {
  GB_LAUNCH_CHAIN("col_dot", s, col_dot_kernel, dim3(cdiv(P, 8)), dim3(256), 0, C, ldc, X, ldx, out, N, P);
  return GB_OK;
}

int launch_copy_zero_diag(const double* src, double* dst, int P, cudaStream_t s) {
  GB_LAUNCH_CHAIN("copy_zero_diag", s, copy_zero_diag_kernel, dim3(cdiv((long long)P * P, 256)), dim3(256), 0, src,
                  dst, P);
  return GB_OK;
}

int launch_add_scaled_rows(double* w, const double* d, const double* n, int P, int Q, int nbeta, int nalpha,
                           cudaStream_t s) {
  GB_LAUNCH_CHAIN("add_scaled_rows", s, add_scaled_rows_kernel, dim3(dim3(cdiv(Q, 128), P)), dim3(128), 0, w, d, n, P,
                  Q, nbeta, nalpha);
  return GB_OK;
}

int launch_make_ck_weighted(const double* bMO, const double* ck12, double* Y, int P, int Q, cudaStream_t s) {
  GB_LAUNCH_CHAIN("make_ck_weighted", s, make_ck_weighted_kernel, dim3(dim3(cdiv(Q, 128), P, P)), dim3(128), 0, bMO,
                  ck12, Y, P, Q);
  return GB_OK;
}

int launch_make_exchange_operand(const double* bMO, const double* ck12, const double* w, double* Y, int P, int Q,
                                 cudaStream_t s) {
  const long long rows = (long long)P * P;
  if (rows == 0 || Q == 0) return GB_OK;
  const unsigned grid = (unsigned)(rows < 152LL * 16 ? rows : 152LL * 16);
  GB_LAUNCH_CHAIN("make_exchange_operand", s, make_exchange_operand_kernel, dim3(grid), dim3(256), 0, bMO, ck12, w, Y,
                  P, Q);
  return GB_OK;
}

int launch_lagrange2_hterm(const double* Hmat, const double* n, double* elag, int N, int P, cudaStream_t s) {
  const long long total = (long long)N * N;
  if (total == 0) return GB_OK;
  const unsigned grid = (unsigned)(cdiv(total, 256) < 152u * 8 ? cdiv(total, 256) : 152u * 8);
  GB_LAUNCH_CHAIN("lagrange2_hterm", s, lagrange2_hterm_kernel, dim3(grid), dim3(256), 0, Hmat, n, elag, N, P);
  return GB_OK;
}

int launch_lagrange2_finish(const double* bMO, const double* w, const double* Hmat, const double* n,
                            double* elag, int N, int P, int Q, cudaStream_t s) {
  GB_LAUNCH_CHAIN("lagrange2_finish", s, lagrange2_finish_kernel, dim3(cdiv((long long)N * P, 8)), dim3(256), 0, bMO,
                  w, Hmat, n, elag, N, P, Q);
  if (N > P) {
    GB_LAUNCH_CHAIN("zero_tail_cols", s, zero_tail_cols_kernel, dim3(cdiv((long long)N * (N - P), 256)), dim3(256), 0,
                    elag, N, P);
  }
  return GB_OK;
}

}  // namespace gb
