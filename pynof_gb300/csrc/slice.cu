// Digit slicing of FP64 operands (see slice.cuh for the representation).
#include "slice.cuh"

namespace gb {
namespace {

__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// |x| < 2^E for every x whose |bits| <= maxbits (order of |x| == order of its bits).
__device__ __forceinline__ int exponent_of(unsigned long long maxbits) {
  const int ex = (int)(maxbits >> 52);
  return (ex == 0 ? 1 : ex) - 1022;
}

// Balanced W-bit digits of round(x 2^(e_S - E)), pre-weighted: digit s as the
// FP32 bits of d 2^-e_s (exact in bf16, so the upper half of those bits is the
// bf16 pattern; the lower half is zero).  Half a digit's range added at every
// place makes the balanced digits plain fields of a non-negative integer, with no
// carries between them.  A field's FP32 value comes from the 1.5 * 2^23 magic
// number (the field or-ed into its low bits), its bias and weight from one exact
// fused multiply-add: three instructions a digit (with carries from digit to digit
// five; the slicer, at 87 % of the copy rate at nbf=600, takes the same time).
template <int S, int W>
__device__ __forceinline__ void make_digits(double x, int E, uint32_t* out) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  int ex = (int)((bits >> 52) & 0x7FF);
  unsigned long long m = bits & 0xFFFFFFFFFFFFFull;
  if (ex) m |= 1ull << 52; else ex = 1;
  // right shift of the 53-bit mantissa (>= 9 for e_S <= 44, a left shift of at most 9 for 62)
  const int r = 1075 + E - ex - digit_exp(W, S);
  unsigned long long mag;
  if (digit_exp(W, S) > 52 && r <= 0) mag = m << -r;
  else if (r >= 64) mag = 0;
  else mag = (m + (1ull << (r - 1))) >> r;
  // half a digit's range at every place, the leading digit's bound 2^e_1 at its own
  constexpr int E1 = digit_exp(W, 1);
  constexpr unsigned long long ONES = ((1ull << (W * S)) - 1) / ((1ull << W) - 1);
  constexpr unsigned long long BIAS =
      (ONES << (W - 1)) + (((1ull << E1) - (1ull << (W - 1))) << (W * (S - 1)));
  const unsigned long long sg = (unsigned long long)((long long)bits >> 63);
  const unsigned long long u = (mag ^ sg) + (BIAS - sg);
#pragma unroll
  for (int s = S; s >= 1; --s) {
    // the leading digit's field is 0 .. 2^(e_1 + 1)
    const uint32_t f = (uint32_t)(u >> (W * (S - s))) & ((1u << (s == 1 ? E1 + 2 : W)) - 1u);
    const float w = __int_as_float((127 - digit_exp(W, s)) << 23);
    const float zero = 12582912.0f + (float)(1 << (s == 1 ? E1 : W - 1));
    out[s - 1] = __float_as_uint(fmaf(__uint_as_float(0x4B400000u | f), w, -zero * w));
  }
}

// A NaN or an infinity has the largest magnitude bits of all; it has no digits,
// so the row that holds one is reported in the status word (the first error
// recorded there stays) and the split-product kernels refuse to start.
__device__ __forceinline__ void note_nonfinite(unsigned long long maxbits, int* status) {
  if (maxbits >= 0x7FF0000000000000ull && status) atomicCAS(status, 0, GB_ERR_NONFINITE);
}

// The warp (all 32 lanes, `row` its first row) that meets the first row of a
// 128-row block clears the block's norms for the digit kernel.
__device__ __forceinline__ void clear_norms(int* norms, long long b, long long row, int rows, int lane) {
  if (norms && row % SL_ROWS == 0 && lane < SL_NORMS)
    norms[(b * ((rows + SL_ROWS - 1) / SL_ROWS) + row / SL_ROWS) * SL_NORMS + lane] = 0;
}

// One warp per row; K is the unit-stride index.  (One launch for exponents and
// digits, a CTA reading its 32 rows twice, was slower: 1093 us against 903 for
// the nine slicings of an orbital step at nbf=300.  So were four and eight
// explicit loads in flight here and below: 430 us of 285.)
__global__ void rowexp_kfast_kernel(SliceSrc src, int rows, int K, int* __restrict__ exps, int* __restrict__ norms,
                                    int* status) {
  chain_wait();
  const long long b = blockIdx.y;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  clear_norms(norms, b, row, rows, lane);
  const double* base = src.p + b * src.sb + src.row_at(row);
  unsigned long long mx = 0;
  if (src.k.div == 0) {
    for (int k = lane; k < K; k += 32) {
      const unsigned long long v = abs_bits(base[(long long)k * src.k.s0]);
      mx = v > mx ? v : mx;
    }
  } else {
    // k runs of length div (stride s0 inside, s1 between runs): no division per element
    const long long div = src.k.div;
    for (long long k0 = 0, r = 0; k0 < K; k0 += div, ++r) {
      const double* bp = base + r * src.k.s1;
      const long long lim = K - k0 < div ? K - k0 : div;
      for (long long j = lane; j < lim; j += 32) {
        const unsigned long long v = abs_bits(bp[j * src.k.s0]);
        mx = v > mx ? v : mx;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx ? v : mx;
  }
  if (lane == 0) {
    exps[b * rows + row] = exponent_of(mx);
    note_nonfinite(mx, status);
  }
}

// The same with a row's K cut into gridDim.z ranges, for few long rows (300
// rows of 180000 took 0.6 ms on 300 warps): every warp folds its range's
// exponent in with atomicMax; exps and norms are preset below any value.
__global__ void rowexp_kfast_split_kernel(SliceSrc src, int rows, int K, int* __restrict__ exps, int* status) {
  chain_wait();
  const long long b = blockIdx.y;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int per = (K + gridDim.z - 1) / gridDim.z, k0 = blockIdx.z * per, k1 = min(K, k0 + per);
  if (k0 >= k1) return;
  const double* base = src.p + b * src.sb + src.row_at(row);
  unsigned long long mx = 0;
  for (int k = k0 + lane; k < k1; k += 32) {
    const unsigned long long v = abs_bits(base[src.k.at(k)]);
    mx = v > mx ? v : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx ? v : mx;
  }
  if (lane == 0) {
    atomicMax(exps + b * rows + row, exponent_of(mx));
    note_nonfinite(mx, status);
  }
}

// Rows are the unit-stride index: 32 consecutive rows per CTA (lane = row,
// each warp reads 256 contiguous bytes per k) and its 8 warps split K, or 32 warps
// where the grid has fewer CTAs than two per SM (a warp's loads follow each other,
// ~0.3 us each: C^T's pass at nbf=600 21 us with 8, 14 with 32); the partial maxima
// meet in shared memory.
template <int NW>
__global__ void __launch_bounds__(32 * NW) rowexp_rfast_kernel(SliceSrc src, int rows, int K, int* __restrict__ exps,
                                                               int* __restrict__ norms, int* status) {
  __shared__ unsigned long long part[NW][32];
  chain_wait();
  const long long b = blockIdx.y;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long row = (long long)blockIdx.x * 32 + lane;
  if (w == 0) clear_norms(norms, b, (long long)blockIdx.x * 32, rows, lane);
  if (b == 0)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < src.preset_n; i += gridDim.x * blockDim.x)
      src.preset[i] = META_PRESET;
  unsigned long long mx = 0;
  if (row < rows) {
    const double* base = src.p + b * src.sb + src.row_at(row);
    for (int k = w; k < K; k += NW) {
      const unsigned long long v = abs_bits(base[src.k.at(k)]);
      mx = v > mx ? v : mx;
    }
  }
  part[w][lane] = mx;
  __syncthreads();
  if (w == 0 && row < rows) {
#pragma unroll
    for (int j = 1; j < NW; ++j) mx = part[j][lane] > mx ? part[j][lane] : mx;
    exps[b * rows + row] = exponent_of(mx);
    note_nonfinite(mx, status);
  }
}

// The 8 source values of thread (row r, k group at k0) of one k block.
__device__ __forceinline__ void load_group(const SliceSrc& src, const double* base, bool rok, int k0, int K,
                                           double (&xs)[8]) {
  // k0 is a multiple of 8: with a unit k stride inside runs of a multiple of 8
  // (k.div), the 8 values are contiguous
  const double* p8 = base + src.k.at(k0);
  if (rok && src.kfast && src.k.s0 == 1 && (src.k.div == 0 || src.k.div % 8 == 0) && k0 + 8 <= K &&
      (reinterpret_cast<uintptr_t>(p8) & 15) == 0) {
    // contiguous, 16-byte aligned k run: four 16-byte loads
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(p8) + u);
      xs[2 * u] = v.x;
      xs[2 * u + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u;
      xs[u] = (rok && k < K) ? base[src.k.at(k)] : 0.0;
    }
  }
}

// The same of an exchange operand (SliceSrc::ex_scale); r: the row, b: the batch entry.
__device__ __forceinline__ void load_group_exchange(const SliceSrc& src, const double* base, bool rok, int r, int b,
                                                    int k0, int K, double (&xs)[8]) {
  const int div = (int)src.k.div;
  int q = k0 / div, l = k0 - q * div;
  q += b * src.ex_runs;
  const double* p8 = base + k0;
  if (rok && div % 8 == 0 && k0 + 8 <= K && q != r && (reinterpret_cast<uintptr_t>(p8) & 15) == 0) {
    const double c = __ldg(src.ex_scale + (long long)r * src.ex_n + q);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(p8) + u);
      xs[2 * u] = c * v.x;
      xs[2 * u + 1] = c * v.y;
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    double v = 0.0;
    if (rok && k0 + u < K) {
      if (q == r)
        v = -src.ex_diag[(long long)r * div + l];
      else
        v = src.ex_scale[(long long)r * src.ex_n + q] * p8[u];
    }
    xs[u] = v;
    if (++l == div) {
      l = 0;
      ++q;
    }
  }
}

// The size plane's value of an element whose leading digit's FP32 bits are d1.
__device__ __forceinline__ uint32_t size_bits(double x, uint32_t d1) {
  const uint32_t a = d1 & 0x7FFFFFFFu;
  return a != 0 || abs_bits(x) == 0 ? a : (127u - 30u) << 23;
}

// Digits of the 8 values, packed per slice as 8 bf16 (one 16-byte store each), and
// the size plane behind seven of them;
// nq[s] += the sum of the squares of the weighted digits of slice s < SL_NORMS
// (nine-bit digits).
template <int S, int W>
__device__ __forceinline__ void store_group(const double (&xs)[8], int e, unsigned char* out, float (&nq)[SL_NORMS]) {
  constexpr bool SIZES = S == F64_DIGITS;
  uint32_t pk[S + SIZES][4];
#pragma unroll
  for (int u = 0; u < 8; u += 2) {
    uint32_t d0[S], d1[S];
    make_digits<S, W>(xs[u], e, d0);
    make_digits<S, W>(xs[u + 1], e, d1);
    // the two bf16 patterns (upper halves) side by side
#pragma unroll
    for (int s = 0; s < S; ++s) pk[s][u >> 1] = __byte_perm(d0[s], d1[s], 0x7632);
    if constexpr (SIZES) pk[S][u >> 1] = __byte_perm(size_bits(xs[u], d0[0]), size_bits(xs[u + 1], d1[0]), 0x7632);
#pragma unroll
    for (int s = 0; s < (W != 9 ? 0 : SIZES ? SL_NORMS : 3); ++s) {
      const float a = __uint_as_float(d0[s]), b = __uint_as_float(d1[s]);
      nq[s] = fmaf(a, a, fmaf(b, b, nq[s]));
    }
  }
#pragma unroll
  for (int s = 0; s < S + SIZES; ++s)
    *reinterpret_cast<uint4*>(out + s * SL_SLICE_STEP) = make_uint4(pk[s][0], pk[s][1], pk[s][2], pk[s][3]);
}

// One CTA of G 256-thread groups per (row block, kpc consecutive k blocks, a run
// of the norms); group g takes the run's k blocks g, g + G, ..: thread -> (row r, k group
// of 8).  Lanes 0..7 take consecutive rows of one core matrix and a warp covers 32
// consecutive rows of one k group, i.e. four whole consecutive core matrices (512
// contiguous bytes) per slice, written with 16-byte stores; it reads 64
// contiguous source bytes per row and k block (K-fast sources: the run reads
// SL_KPC x 128 contiguous bytes of each row) or 256 contiguous bytes per k
// (row-fast sources).  At most 64 registers (four CTAs per SM): occupancy keeps
// more loads in flight than prefetching the next k block into registers did
// (measured: 1.62 ms against 1.87-1.93 ms for the T of one nbf=600 build, 8.64 GB).
// Where the grid has fewer CTAs than two per SM (a thread's k blocks follow each
// other, ~1 us each): a CTA per k block for K up to one run (its norms times the
// eight blocks of a run bound the run's), G = 4 for longer ones, whose chunks need
// the tighter norms (half transform at nbf=600 6.20 ms, 6.89 with the looser).
// Three slicings of an nbf=24 build: 41 us with runs of eight, 33 with G = 4, 20.
template <int S, int W, bool EX = false>
__global__ void __launch_bounds__(S == F64_DIGITS ? 256 : 1024, S == F64_DIGITS ? 3 : 1)
    digits_blocked_kernel(SliceSrc src, SlicedDesc dst, int kpc) {
  constexpr int ND = W != 9 ? 0 : S == F64_DIGITS ? SL_NORMS : 3;  // digits with norms
  constexpr int PL = S == F64_DIGITS ? F64_PLANES : S;
  __shared__ float s_nq[S == F64_DIGITS || W != 9 ? 1 : 3 * 256 * 3];
  chain_wait();
  const long long b = blockIdx.y;
  const int kbn = dst.kblocks();
  const int runs = (kbn + kpc - 1) / kpc;
  const int rb = blockIdx.x / runs, kb0 = (blockIdx.x % runs) * kpc;
  const int kb1 = min(kb0 + kpc, kbn);
  const int G = blockDim.x >> 8, grp = threadIdx.x >> 8;
  const int warp = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31;
  const int ri = lane & 7, kg = warp >> 2, rg = (warp & 3) * 4 + (lane >> 3);
  const int r = rb * SL_ROWS + rg * 8 + ri;
  const bool rok = r < dst.rows;
  const double* base = src.p + b * src.sb + (rok ? src.row_at(r) : 0);
  const int e = rok ? dst.exps[b * dst.rows + r] : 0;
  unsigned char* out0 = reinterpret_cast<unsigned char*>(dst.planes) + b * dst.batch_bytes() +
                        ((long long)rb * kbn * PL) * SL_TILE_BYTES + (kg * PL * 16 + rg) * 128 + ri * 16;
  double xa[8];
  float nq[SL_NORMS] = {};
  for (int kb = kb0 + grp; kb < kb1; kb += G) {
    if (EX)
      load_group_exchange(src, base, rok, r, (int)b, kb * SL_K + kg * 8, dst.K, xa);
    else
      load_group(src, base, rok, kb * SL_K + kg * 8, dst.K, xa);
    store_group<S, W>(xa, e, out0 + (long long)kb * PL * SL_TILE_BYTES, nq);
  }
  if (S != F64_DIGITS && ND > 0 && G > 1) {
    // the run's sums of squares over the groups
    const int t = threadIdx.x & 255;
    if (grp > 0)
#pragma unroll
      for (int s = 0; s < ND; ++s) s_nq[((grp - 1) * ND + s) * 256 + t] = nq[s];
    __syncthreads();
    if (grp > 0) return;
    for (int g = 0; g < G - 1; ++g)
#pragma unroll
      for (int s = 0; s < ND; ++s) nq[s] += s_nq[(g * ND + s) * 256 + t];
  }
  if constexpr (W == 9) {
    // non-negative floats order as their bits
    int* nb = dst.norms + (b * dst.rblocks() + rb) * SL_NORMS;
#pragma unroll
    for (int s = 0; s < ND; ++s) {
      // back to squares of the digits, for a whole run
      const float scale = __int_as_float((127 + 2 * digit_exp(W, s + 1)) << 23) * (float)(SL_KPC / kpc);
      const unsigned int mx = __reduce_max_sync(0xffffffffu, __float_as_uint(nq[s] * scale));
      if (lane == 0) atomicMax(nb + s, (int)mx);
    }
  }
}

// TF32 hi / lo of y = x 2^-E (|x| < 2^E), as FP32 bit patterns: hi = tf32(y),
// lo = tf32(y - hi), each rounded to nearest even to 11 significant bits from
// the FP64 bits with integer arithmetic (y - hi is exact); values below the
// FP32 normal range are flushed to zero.
__device__ __forceinline__ void tf32_split(double x, int E, uint32_t& hi, uint32_t& lo) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const uint32_t sign = (uint32_t)(bits >> 63);
  const int ex = (int)((bits >> 52) & 0x7FF);
  hi = 0u;
  lo = 0u;
  if (ex == 0) return;  // zero (FP64 subnormals are far below the FP32 range after scaling)
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);  // y = m 2^(ex - 1075 - E)
  int fe = ex - E - 1023 + 127;
  unsigned long long q = m >> 42;
  const unsigned long long rem = m & ((1ull << 42) - 1), half = 1ull << 41;
  if (rem > half || (rem == half && (q & 1ull))) ++q;
  const long long r = (long long)m - (long long)(q << 42);  // |r| <= 2^41
  if (q == (1ull << 11)) {
    q >>= 1;
    ++fe;
  }
  if (fe > 0) hi = (sign << 31) | ((uint32_t)fe << 23) | (((uint32_t)q & 0x3FFu) << 13);
  if (r == 0 || fe <= 0) return;
  const uint32_t rs = sign ^ (r < 0 ? 1u : 0u);
  const unsigned long long ra = (unsigned long long)(r < 0 ? -r : r);
  int top = 63 - __clzll((long long)ra);  // leading one of |r|
  unsigned long long q2;
  if (top > 10) {
    const int sh = top - 10;
    q2 = ra >> sh;
    const unsigned long long rem2 = ra & ((1ull << sh) - 1), h2 = 1ull << (sh - 1);
    if (rem2 > h2 || (rem2 == h2 && (q2 & 1ull))) ++q2;
    if (q2 == (1ull << 11)) {
      q2 >>= 1;
      ++top;
    }
  } else {
    q2 = ra << (10 - top);
  }
  const int fe2 = ex - 1075 - E + top + 127;
  if (fe2 > 0) lo = (rs << 31) | ((uint32_t)fe2 << 23) | (((uint32_t)q2 & 0x3FFu) << 13);
}

// TF32x3 planes, one CTA of 256 threads per (row block, k block of 8): thread
// -> (row r, k group of 4), 16-byte stores per plane (same thread map as the
// bf16 digits).
__global__ void __launch_bounds__(256) tf32_blocked_kernel(SliceSrc src, SlicedDesc dst) {
  chain_wait();
  const long long b = blockIdx.y;
  const int kbn = dst.kblocks();
  const int rb = blockIdx.x / kbn, kb = blockIdx.x % kbn;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ri = lane & 7, kg = warp >> 2, rg = (warp & 3) * 4 + (lane >> 3);
  const int r = rb * SL_ROWS + rg * 8 + ri;
  const int k0 = kb * (SL_K / 2) + kg * 4;
  const bool rok = r < dst.rows;
  const double* base = src.p + b * src.sb + (rok ? src.row_at(r) : 0);
  const int e = rok ? dst.exps[b * dst.rows + r] : 0;
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int k = k0 + u;
    tf32_split((rok && k < dst.K) ? base[src.k.at(k)] : 0.0, e, hi[u], lo[u]);
  }
  unsigned char* out = reinterpret_cast<unsigned char*>(dst.planes) + b * dst.batch_bytes() +
                       ((long long)blockIdx.x * 2) * SL_TILE_BYTES + (kg * 2 * 16 + rg) * 128 + ri * 16;
  *reinterpret_cast<uint4*>(out) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(out + SL_SLICE_STEP) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

int slice_operand(const SliceSrc& src, const SlicedDesc& dst, cudaStream_t s, bool exps_ready, int* status) {
  GB_REQUIRE((dst.kind == 0 && ((dst.S >= 1 && dst.S <= 5) || dst.S == F64_PLANES)) || (dst.kind == 1 && dst.S == 2), GB_ERR_INVALID_ARG,
             "slice_operand: bad split form (planes %d, kind %d)", dst.S, dst.kind);
  GB_REQUIRE(dst.batch >= 1 && dst.batch <= 65535 && dst.rows >= 0, GB_ERR_BAD_SHAPE, "slice_operand: bad batch");
  GB_REQUIRE((reinterpret_cast<uintptr_t>(dst.planes) & 15) == 0, GB_ERR_INVALID_ARG,
             "slice_operand: planes not 16-byte aligned");
  if (dst.rows == 0 || dst.K == 0) return GB_OK;
  GB_REQUIRE(!src.preset || (!src.kfast && !exps_ready), GB_ERR_INVALID_ARG,
             "slice_operand: words are preset by the exponent kernel of unit-stride rows");
  int* norms = dst.kind == 0 ? dst.norms : nullptr;
  GB_REQUIRE(dst.kind != 0 || norms, GB_ERR_INVALID_ARG, "slice_operand: no norms");
  int* st = status ? status : device_status_word();
  const long long warps = (long long)dst.rows * dst.batch;
  if (exps_ready) {
    GB_REQUIRE(dst.kind == 0, GB_ERR_INVALID_ARG, "slice_operand: recorded exponents are for digit slices");
  } else if (src.kfast && dst.kind == 0 && dst.K >= 8192 && warps <= 4096 &&
             dst.norms == dst.exps + (size_t)dst.batch * dst.rows) {
    // fewer warps than the SMs hold: ranges of K of at least 2048
    long long z = 8192 / warps + 1;
    z = z < dst.K / 2048 ? z : dst.K / 2048;
    GB_TRY(cuda_status(cudaMemsetAsync(dst.exps, 0x80, sizeof(int) * sliced_meta_ints(dst.batch, dst.rows), s),
                       "slice_operand: exponents"));
    GB_LAUNCH_CHAIN("slice_rowexp", s, rowexp_kfast_split_kernel,
                    dim3(cdiv(dst.rows, 8), dst.batch, (unsigned)z), dim3(256), 0, src, dst.rows, dst.K, dst.exps, st);
  } else if (src.kfast) {
    GB_LAUNCH_CHAIN("slice_rowexp", s, rowexp_kfast_kernel, dim3(cdiv(dst.rows, 8), dst.batch), dim3(256), 0, src,
                    dst.rows, dst.K, dst.exps, norms, st);
  } else {
    const dim3 grid(cdiv(dst.rows, 32), dst.batch);
    if ((long long)grid.x * dst.batch < 304)
      GB_LAUNCH_CHAIN("slice_rowexp", s, rowexp_rfast_kernel<32>, grid, dim3(1024), 0, src, dst.rows, dst.K, dst.exps,
                      norms, st);
    else
      GB_LAUNCH_CHAIN("slice_rowexp", s, rowexp_rfast_kernel<8>, grid, dim3(256), 0, src, dst.rows, dst.K, dst.exps,
                      norms, st);
  }
  const long long blocks = (long long)dst.rblocks() * dst.kblocks();
  GB_REQUIRE(blocks <= 2147483647LL, GB_ERR_BAD_SHAPE, "slice_operand: too many blocks");
  if (dst.kind == 1) {
    GB_LAUNCH_CHAIN("slice_tf32", s, tf32_blocked_kernel, dim3((unsigned)blocks, dst.batch), dim3(256), 0, src,
                    dst);
    return GB_OK;
  }
  const long long runs = (dst.kblocks() + SL_KPC - 1) / SL_KPC;
  const bool few = (long long)dst.rblocks() * runs * dst.batch < 304;
  const int kpc = few && runs == 1 ? 1 : SL_KPC;
  const dim3 grid((unsigned)((long long)dst.rblocks() * ((dst.kblocks() + kpc - 1) / kpc)), dst.batch);
  const dim3 block(few && runs > 1 && dst.S != F64_PLANES ? 1024 : 256);
  if (src.ex_scale) {
    GB_REQUIRE(exps_ready && src.kfast && src.k.div > 0 && dst.S == 5 && dst.W == 9, GB_ERR_INVALID_ARG,
               "slice_operand: an exchange operand takes six digits and recorded exponents");
    GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<5, 9, true>), grid, block, 0, src, dst, kpc);
    return GB_OK;
  }
  if (dst.W == 9) {
    GB_REQUIRE(dst.S == 5 || dst.S == F64_PLANES, GB_ERR_INVALID_ARG,
               "slice_operand: nine-bit digits come in five planes or eight");
    if (dst.S == 5)
      GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<5, 9>), grid, block, 0, src, dst, kpc);
    else
      GB_LAUNCH_CHAIN("slice_digits7", s, (digits_blocked_kernel<F64_DIGITS, 9>), grid, block, 0, src, dst, kpc);
    return GB_OK;
  }
  switch (dst.S) {
    case 1: GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<1, 7>), grid, block, 0, src, dst, kpc); break;
    case 2: GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<2, 7>), grid, block, 0, src, dst, kpc); break;
    case 3: GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<3, 7>), grid, block, 0, src, dst, kpc); break;
    case 4: GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<4, 7>), grid, block, 0, src, dst, kpc); break;
    default: GB_LAUNCH_CHAIN("slice_digits", s, (digits_blocked_kernel<5, 7>), grid, block, 0, src, dst, kpc); break;
  }
  return GB_OK;
}

}  // namespace gb
