// tcgen05 split-product FP64 GEMM (see ozaki_tc.cuh).
//
// CTA tile: 128 rows of A (M) x BN rows of B (N), BN in {32, 64, 128}.
// 18 warps.  warp 0 lane 0 is the producer: a ring of STAGES stages in which
// every stage holds the S slices of a 128 x 16 block of A (one contiguous
// cp.async.bulk copy -- the slicer stores the digits in the tensor-core
// core-matrix order, slice.cuh) and of a BN x 16 block of B (one copy, or two
// per slice when BN < 128).  warp 1 allocates TMEM (4 BN columns) and its
// lane 0 issues tcgen05.mma (M=128, K=16, bf16 -> f32; N=BN, or a multiple of
// it where consecutive B slices go to consecutive accumulators).  warps 2..17
// drain and finish: warp w reads TMEM lanes 32 (w % 4) .. +31 (tile rows) and
// BN/4 columns from (w - 2) / 4 * BN/4 of every accumulator.
//
// TMEM columns: [0,BN) group 2, [BN,2BN) group 3, [2BN,3BN) group 4 (exact,
// drained after every chunk, chunk_blocks), [3BN,4BN) groups 5.. (whole K, or
// per chunk with fdrain).
//
// One launch covers one GEMM (optionally batched), or -- the grouped kernel --
// a table of GEMMs of different shapes (e.g. one per molecule of a batch).
//
// Every mbarrier wait is bounded (the launch's wait_ns, 2 s unless
// gb_set_wait_limit_ns changed it); on timeout the CTA records GB_ERR_TIMEOUT
// in the device status word, stops issuing work, waits (bounded) for its own
// TMA copies and MMAs in flight, frees TMEM and exits.
#include <cuda_bf16.h>

#include <cuda.h>

#include <atomic>
#include <cstdio>
#include <mutex>
#include <vector>

#include "ozaki_tc.cuh"
#include "tc_prims.cuh"

static __device__ int g_tc_status;

namespace gb {
namespace {

constexpr int BM = 128, BK = SL_K, STAGES = 5;
constexpr int CH_TF32 = 12;  // stages per chunk of the TF32x3 form (96 k)
constexpr int CH_W7 = 12;    // and of seven-bit digits (192 k: groups 2 and 4 below 2^22 units whatever the digits are)
// Nine-bit digits: stages per chunk that are exact whatever the digits are: 48 k, where group 2
// stays below 2^16 * 48 < 2^22 - 2^16 units and groups 3 and 4 below
// 3 * 2^16 * 48 < 2^24 - 2^16 (see drain_exact for the limits).
constexpr int CH_MIN = 3;
constexpr float LIM_G2 = 4194304.0f - 65536.0f, LIM_G34 = 16777216.0f - 65536.0f;
constexpr int CH_RUNS_MAX = 32;  // runs of 128 k per chunk at most (the FP32 group's own range)
constexpr int THREADS = 32 * (2 + NUM_EPI_WARPS);
// 18 warps put 5 warps on two of the four SM sub-partitions, whose register
// files hold 16K registers each: 5 * 32 * 96 <= 16384 caps the kernel at 96.
constexpr int MAX_REGS = 96;
constexpr uint32_t TILE_BYTES = SL_TILE_BYTES;  // 4 KB per A slice tile (BM == SL_ROWS)

// KIND 0: bf16 digit slices (kind::f16), four accumulators (three exact
// groups and the FP32 group); KIND 1: TF32x3 (kind::tf32), two FP32
// accumulators used alternately by consecutive chunks (one is drained while
// the MMAs fill the other).
template <int BN, int KIND>
struct TileCfg {
  static_assert(BN == 32 || BN == 64 || BN == 128, "BN must be 32, 64 or 128");
  static constexpr uint32_t B_TILE = BN * SL_K * 2;              // bytes of one B slice tile
  static constexpr uint32_t TMEM_COLS = KIND ? 2 * BN : 4 * BN;  // power of two >= 32
  static constexpr int CW = BN / 4;                              // columns per epilogue warp
  static constexpr int KPER = KIND ? SL_K / 2 : SL_K;            // k per stage (one MMA)
  static constexpr uint32_t FMT = KIND ? 2u : 1u;                // operand format: tf32 / bf16
  // instruction descriptor: f32 accumulate, both operands K-major, M=128, N=BN
  static constexpr uint32_t IDESC = (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(BN >> 3) << 17) |
                                    ((uint32_t)(BM >> 4) << 24);
};
// bytes of the per-tile assembly tables (see cta_tile)
__host__ __device__ constexpr uint32_t epi_table_bytes(int BN) { return 20u * (uint32_t)(BM + BN); }
constexpr int FDRAIN_K = 4096;  // K above which the FP32 group is drained per chunk (OzGemm::fdrain)
constexpr int PAIR_FRAC = 9;    // fraction bits of the assembly up to FDRAIN_K (fold_pair)

// The first error recorded in the status word stays (a timeout does not
// overwrite an earlier non-finite report, nor the other way round).
__device__ __forceinline__ void signal_abort(volatile int* abort_flag) {
  *abort_flag = 1;
  atomicCAS(&g_tc_status, 0, GB_ERR_TIMEOUT);
}

// t * 2^frac rounded to nearest as a 64-bit integer, for |t| < 2^22 and
// frac <= 16: rint(t) * 2^frac + rint((t - rint(t)) * 2^frac), both parts
// through magic_int; (t - rint(t)) is exact.
__device__ __forceinline__ long long split_round(float t, int frac, float two_frac) {
  const float f1 = t + MAGIC;
  const int ti = __float_as_int(f1) - MAGIC_BITS;
  const int fi = magic_int(t - (f1 - MAGIC), two_frac);
  return (long long)((unsigned long long)(long long)ti << frac) + fi;
}

// One element's exact groups, as FP32 values x2, x3, x4 (integers u_g over the
// unit U_g): from the last group up, the nearest multiple of 2^W units is
// carried into the group above (exact in FP32 while |u_3|, |u_4| stay below
// 2^24 - 2^16).  Leaves the top group with its carry (below 2^22 units) in x2 and
// returns the remainders, an FP32 value below 2^(2 W - 1) + 2^(W - 1) units of the last
// group.
template <int W, int gE>
__device__ __forceinline__ float carry_groups(float& x2, float x3, float x4) {
  constexpr float B = (float)(1 << W);
  constexpr float U2 = (float)(1ll << group_exp(W, 2)), U3 = U2 * B, U4 = U3 * B;  // units per 1.0
  float low = 0.0f;
  if (gE >= 4) {
    const float h4 = fmaf(x4, U4 / B, MAGIC) - MAGIC;  // rint(u_4 / 2^W), in units of group 3
    low = fmaf(h4, -1.0f / U3, x4);
    x3 = fmaf(h4, 1.0f / U3, x3);
  }
  if (gE >= 3) {
    const float h3 = fmaf(x3, U3 / B, MAGIC) - MAGIC;
    const float l3 = fmaf(h3, -1.0f / U2, x3);
    low = gE >= 4 ? low + l3 : l3;
    x2 = fmaf(h3, 1.0f / U2, x2);
  }
  return low;
}

// Drain of the exact groups g = 2..gE of CW columns of this warp's TMEM lanes.
//
// Up to FDRAIN_K of K (fdrain off) an element's sum is a pair of 32-bit parts
// held in the two halves of its R: the top group's units as an integer (the
// magic number's bits are added as they are; their bias comes off in
// fold_pair) and the remainders as an FP32 number, exact below 2^24 units, i.e.
// for FDRAIN_K / 48 = 86 chunks of at most 2^17.1 units.  That is 11 single-issue
// instructions an element; 64-bit sums take about twice that, and at one
// instruction a clock and sub-partition a drain took 3.8 to 4.3 K clocks of
// which the MMAs waited for most (1.8 K now).
// With fdrain R is a 64-bit integer in units of the last group, scaled by 2^fr.
template <int BN, int W, int gE, bool PAIR, int CW>
__device__ __forceinline__ void drain_exact(uint32_t lbase, long long (&R)[CW], int fr) {
  constexpr float U2 = (float)(1ll << group_exp(W, 2)), UE = (float)(1ll << group_exp(W, gE));
#pragma unroll
  for (int h = 0; h < CW / 4; ++h) {
    uint32_t v2[4], v3[4] = {}, v4[4] = {};
    tmem_ld4_async(lbase + (uint32_t)(h * 4), v2);
    if (gE >= 3) tmem_ld4_async(lbase + (uint32_t)(BN + h * 4), v3);
    if (gE >= 4) tmem_ld4_async(lbase + (uint32_t)(2 * BN + h * 4), v4);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x2 = __uint_as_float(v2[j]);
      const float low = carry_groups<W, gE>(x2, __uint_as_float(v3[j]), __uint_as_float(v4[j]));
      long long& r = R[h * 4 + j];
      if constexpr (PAIR) {
        const uint32_t top = (uint32_t)r + __float_as_uint(fmaf(x2, U2, MAGIC));
        const float rest = __uint_as_float((uint32_t)((unsigned long long)r >> 32)) + low;
        r = (long long)(((unsigned long long)__float_as_uint(rest) << 32) | top);
      } else {
        asm volatile("" : "+l"(r));
        const long long acc = (long long)magic_int(x2, U2) * (1 << (group_exp(W, gE) - group_exp(W, 2))) +
                              (gE >= 3 ? magic_int(low, UE) : 0);
        r += (long long)((unsigned long long)acc << fr);
      }
    }
  }
}

// An element's pair (see drain_exact) after `chunks` drains with the FP32 group's
// value f (|f| < 2^21 units of the last exact group) added: the top part keeps
// its unit, the other half becomes an integer in units of the last exact
// group's 2^-PAIR_FRAC, |rest| < 2^17 + 2^21 of them.  wide_pair makes one 64-bit
// integer of the two.
template <int W, int gE, bool HAS_F>
__device__ __forceinline__ long long fold_pair(long long r, float f, uint32_t bias) {
  constexpr float U2 = (float)(1ll << group_exp(W, 2)), UE = (float)(1ll << group_exp(W, gE));
  uint32_t top = (uint32_t)r - bias, rest = 0;
  if (gE > 2) {
    const float low = __uint_as_float((uint32_t)((unsigned long long)r >> 32));
    const float h = fmaf(low, U2, MAGIC);  // carry of the summed remainders
    top += __float_as_uint(h) - (uint32_t)MAGIC_BITS;
    rest = (uint32_t)magic_int(fmaf(h - MAGIC, -1.0f / U2, low), UE) << PAIR_FRAC;
    if (HAS_F) rest += (uint32_t)__float2int_rn(f * (UE * (float)(1 << PAIR_FRAC)));
  }
  return (long long)(((unsigned long long)rest << 32) | top);
}
template <int W, int gE>
__device__ __forceinline__ long long wide_pair(long long r) {
  constexpr int A = group_exp(W, gE) - group_exp(W, 2) + PAIR_FRAC;
  return (long long)(int)(uint32_t)r * (1ll << A) + (long long)(int)(uint32_t)((unsigned long long)r >> 32);
}

// int64 fixed point z * 2^scale -> double, round to nearest even, integer ops
// only (the FP64 pipe is narrow on this part).  The leading one is moved to
// bit 63; the top 53 bits are the significand (implicit bit included, so adding
// it to (exponent - 1) << 52 forms the exponent field and a rounding carry out
// of the significand bumps the exponent), the low 11 bits decide the rounding.
__device__ __forceinline__ double fixed_to_double(long long z, int scale, int negate) {
  if (z == 0) return 0.0;
  const unsigned long long sign = (unsigned long long)((z < 0) != (negate != 0)) << 63;
  const unsigned long long u = z < 0 ? 0ull - (unsigned long long)z : (unsigned long long)z;
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << lz;
  const unsigned long long mant = m >> 11;
  const uint32_t low = (uint32_t)m & 0x7FFu;
  const unsigned long long up = (low > 0x400u || (low == 0x400u && (mant & 1ull))) ? 1ull : 0ull;
  const int ef = 63 - lz + scale + 1023;  // biased exponent of the leading one
  if (ef <= 0) return __longlong_as_double((long long)sign);  // underflow -> signed zero
  if (ef >= 2047) return __longlong_as_double((long long)(sign | 0x7FF0000000000000ull));
  return __longlong_as_double((long long)(sign | ((((unsigned long long)(ef - 1)) << 52) + mant + up)));
}

// z * 2^scale as a double, with the sign flipped where `flip` has its top bit: the
// hardware int64 -> double conversion with the scale added to the exponent
// field (shifting the leading one into place with integer instructions instead
// made a tile's stores 18 K clocks long, this way 12 K).  False for results
// outside the normal range, which are for fixed_to_double.
__device__ __forceinline__ bool scaled_to_double(long long z, int scale, uint32_t flip, double& out) {
  const double d = __ll2double_rn(z);
  const uint32_t h = (uint32_t)__double2hiint(d);
  const uint32_t e0 = ((h >> 20) & 0x7FFu) + (uint32_t)scale - 1u;
  const bool zero = h == 0;
  out = zero ? 0.0 : __hiloint2double((int)((h + ((uint32_t)scale << 20)) ^ flip), __double2loint(d));
  return zero || e0 < 2046u;
}

// Widest store (in doubles) that p's alignment allows, and a store of four.
__device__ __forceinline__ int store_width(const double* p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  return (a & 31) == 0 ? 4 : (a & 15) == 0 ? 2 : 1;
}
__device__ __forceinline__ void store4(double* p, const double (&v)[4]) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
               : "memory");
}

struct KArgs {
  OzGemm g;
  SlicedDesc A, B;
  int frac;
  unsigned long long wait_ns;  // limit of every mbarrier wait
  // Test hook: the first CTA's producer never issues global stage `withhold`
  // (-1: every stage is issued), so the MMA issuer's wait for it runs out.
  int withhold;
};

// Stages per chunk of a tile: the longest multiple of the slicer's 128-k runs
// whose exact groups' partial sums provably stay within the drain's limits, from
// the norms of the two row blocks (a run's sum of products of digits s and t is
// at most 2 sqrt(norm_s norm_t)); CH_MIN where not even one run is.  Digits of
// the path's operands (Gaussian-like rows) allow 2 to 3 runs, 256 to 384 k; the
// worst case alone would allow 48 k, and the 192-k chunks of seven-bit digits
// took 21 products instead of 15.
template <int W>
__device__ __forceinline__ int chunk_blocks(const SlicedDesc& A, const SlicedDesc& B, int bz, int m0, int n0,
                                            int nkb) {
  if (W != 9) return CH_W7;
  if (nkb <= CH_MIN) return CH_MIN;
  float a[3], b[3];
  block_norms(A, bz, m0, a);
  block_norms(B, bz, n0, b);
  const float up = 2.002f;  // the bound's 2, and room for the roundings of the norms
  const float g2 = up * a[0] * b[0], g3 = up * (a[0] * b[1] + a[1] * b[0]),
              g4 = up * (a[0] * b[2] + a[2] * b[0] + a[1] * b[1]);
  const float most = fminf(LIM_G2 / fmaxf(g2, 1.0f), LIM_G34 / fmaxf(fmaxf(g3, g4), 1.0f));
  if (!(most >= 1.0f)) return CH_MIN;
  return SL_KPC * (most < (float)CH_RUNS_MAX ? (int)most : CH_RUNS_MAX);
}

// The same with the width chosen at run time: a tile whose last columns are
// missing runs one MMA per product, only as wide as it needs, when that is
// cheaper (below ~104 columns an MMA takes 53 clocks whatever its width, a
// 128-column one 65).
template <int S, int BN, int SEL>
__device__ __forceinline__ void issue_stage(bool wide, uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc,
                                            bool restart_exact, bool restart_f) {
  constexpr int GE = 4;  // groups 2..4 are exact
  if (wide)
    issue_products<S, GE, S + 1, BN, SEL, true>(tmem, da, db, idesc, restart_exact, restart_f);
  else
    issue_products<S, GE, S + 1, BN, SEL, false>(tmem, da, db, idesc, restart_exact, restart_f);
}
template <int BN>
__device__ __forceinline__ bool wide_tile(int n_mma) {
  return BN < 128 || n_mma > 104;
}

// TF32x3 products of one stage: hi hi + hi lo + lo hi into the one accumulator.
template <int BN>
__device__ __forceinline__ void issue_tf32(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, bool& started) {
  mma_tf32(tmem, da, db, idesc, started);
  mma_tf32(tmem, da, db + (uint64_t)BN, idesc, true);
  mma_tf32(tmem, da + (uint64_t)(SL_SLICE_STEP >> 4), db, idesc, true);
  started = true;
}

// Problem of global tile u in a grouped launch: the p with starts[p] <= u <
// starts[p + 1] (always 0 for a single problem, starts == nullptr).
__device__ __forceinline__ int find_problem(const long long* starts, int nprob, unsigned int u) {
  if (starts == nullptr || nprob <= 1) return 0;
  int lo = 0, hi = nprob;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (starts[mid] <= (long long)u) lo = mid; else hi = mid;
  }
  return lo;
}

// The problem a tile belongs to: the table entry of a grouped launch, the
// launch's own argument otherwise.
template <bool GROUPED>
__device__ __forceinline__ const KArgs& prob_ref(const KArgs& a0, const KArgs* probs, int p) {
  if constexpr (GROUPED) return probs[p];
  else return a0;
}

// Local tile index -> (batch, m0, n0).  The dimension with fewer tiles runs
// fastest, so that the CTAs sharing a block of the large operand run together
// (that block is read once from HBM, then from L2).  Returns false
// for tiles a symmetric output does not need.
template <int BN>
__device__ __forceinline__ bool decode_tile(const OzGemm& g, long long t, int& bz, int& m0, int& n0) {
  const int mtiles = (g.M + BM - 1) / BM;
  const int ntiles = (g.N + BN - 1) / BN;
  const long long per_batch = (long long)mtiles * ntiles;
  bz = (int)(t / per_batch);
  const long long r = t % per_batch;
  if (mtiles <= ntiles) {
    m0 = (int)(r % mtiles) * BM;
    n0 = (int)(r / mtiles) * BN;
  } else {
    n0 = (int)(r % ntiles) * BN;
    m0 = (int)(r / ntiles) * BM;
  }
  return !(g.sym == SYM_ROWCOL && m0 > n0) && !(g.sym == SYM_BATCHCOL && n0 > bz);
}

// Columns a tile needs (from n0 on; more than BN: all).
__device__ __forceinline__ int tile_cols(const OzGemm& g, int bz, int n0) {
  return (g.sym == SYM_BATCHCOL && bz + 1 < g.N ? bz + 1 : g.N) - n0;
}

// One output tile, all roles.
template <int CODE, int BN>
__device__ __forceinline__ void cta_tile(const KArgs& a, int bz, int m0, int n0, unsigned char* smem_raw) {
  constexpr int S = form_of(CODE).S, KIND = form_of(CODE).kind, W = form_of(CODE).W;
  using T = TileCfg<BN, KIND>;
  const OzGemm& g = a.g;
  constexpr int gE = (S + 1) < 4 ? (S + 1) : 4;
  constexpr bool has_inexact = (S + 1) > 4;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t a_bytes = (uint32_t)S * TILE_BYTES, b_bytes = (uint32_t)S * T::B_TILE;
  constexpr uint32_t stage_bytes = a_bytes + b_bytes;
  // the assembly parks the tile's int64 results in the stage buffers
  constexpr uint32_t zs_bytes = BM * (BN + 1) * 8;
  constexpr uint32_t data_bytes = STAGES * stage_bytes > zs_bytes ? STAGES * stage_bytes : zs_bytes;
  // assembly tables: roff, mr [BM], coff, mc [BN] (int64), srow [BM], scol [BN] (int)
  long long* e_roff = reinterpret_cast<long long*>(smem + data_bytes);
  long long* e_mr = e_roff + BM;
  long long* e_coff = e_mr + BM;
  long long* e_mc = e_coff + BN;
  int* e_srow = reinterpret_cast<int*>(e_mc + BN);
  int* e_scol = e_srow + BM;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + data_bytes + epi_table_bytes(BN));
  // bars: full[STAGES], empty[STAGES], accfull, accempty, done, (slot, flag), accfull1, accempty1
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 5);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int st) { return bar0 + 8u * st; };
  auto empty_bar = [&](int st) { return bar0 + 8u * (STAGES + st); };
  const uint32_t accfull_bar = bar0 + 8u * (2 * STAGES), accempty_bar = bar0 + 8u * (2 * STAGES + 1),
                 done_bar = bar0 + 8u * (2 * STAGES + 2);
  // TF32x3: the second accumulator's pair (chunk c uses accumulator c & 1)
  const uint32_t accfull1_bar = bar0 + 8u * (2 * STAGES + 6), accempty1_bar = bar0 + 8u * (2 * STAGES + 7);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(accfull_bar, 1);
    mbar_init(accempty_bar, NUM_EPI_WARPS);
    mbar_init(done_bar, 1);
    mbar_init(accfull1_bar, 1);
    mbar_init(accempty1_bar, NUM_EPI_WARPS);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(const_cast<uint32_t*>(tmem_slot))),
                 "r"(T::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  const int nkb = (g.K + T::KPER - 1) / T::KPER;
  const int ch = KIND ? CH_TF32 : chunk_blocks<W>(a.A, a.B, bz, m0, n0, nkb);  // stages per chunk
  const int nchunks = (nkb + ch - 1) / ch;
  // A ragged last column tile runs its MMAs only as wide as it needs (N a
  // multiple of 16 for M = 128); the idle epilogue warps skip their columns.
  const int n_valid = min(BN, g.N - n0);
  const int n_mma = (n_valid + 15) & ~15;
  const uint32_t idesc = (T::IDESC & ~(0x3Fu << 17)) | ((uint32_t)(n_mma >> 3) << 17);

  int issued = 0;  // stages the producer handled (its lane 0)
  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      // an operand sliced once (batch 1) is shared by every batch entry
      const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
      const unsigned char* ga = reinterpret_cast<const unsigned char*>(a.A.planes) + abz * a.A.batch_bytes() +
                                (long long)(m0 / BM) * a.A.kblocks() * a_bytes;
      const int rb = n0 / SL_ROWS, r0 = n0 % SL_ROWS;
      const unsigned char* gbp = reinterpret_cast<const unsigned char*>(a.B.planes) + bbz * a.B.batch_bytes() +
                                 (long long)rb * a.B.kblocks() * (S * TILE_BYTES) + (r0 / 8) * 128;
      for (int kb = 0; kb < nkb; ++kb) {
        const int st = kb % STAGES;
        const uint32_t ph = (kb / STAGES) & 1;
        if (!mbar_wait(empty_bar(st), ph ^ 1, abort_flag, a.wait_ns)) {
          signal_abort(abort_flag);
          break;
        }
        if (kb == a.withhold && blockIdx.x == 0 && blockIdx.y == 0) {
          ++issued;  // test hook: this stage never arrives
          continue;
        }
        mbar_expect_tx(full_bar(st), stage_bytes);
        const uint32_t sa = sbase + st * stage_bytes;
        bulk_load(sa, ga + (long long)kb * a_bytes, a_bytes, full_bar(st));
        const unsigned char* gblk = gbp + (long long)kb * (S * TILE_BYTES);
        if (BN == SL_ROWS) {
          bulk_load(sa + a_bytes, gblk, b_bytes, full_bar(st));
        } else {
          // BN rows of each slice of each k group: two runs of BN * 16 bytes per slice
#pragma unroll
          for (int kg = 0; kg < 2; ++kg)
#pragma unroll
            for (int s = 0; s < S; ++s)
              bulk_load(sa + a_bytes + (kg * S + s) * (BN * 16), gblk + (kg * S + s) * SL_SLICE_STEP, BN * 16,
                        full_bar(st));
        }
        ++issued;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      bool f_started = false;
      int c = 0, kc = 0;  // chunk, stage in the chunk
      for (int kb = 0; kb < nkb; ++kb, ++kc) {
        const int st = kb % STAGES;
        if (kc == ch) {
          kc = 0;
          ++c;
        }
        if (!mbar_wait(full_bar(st), (kb / STAGES) & 1, abort_flag, a.wait_ns)) {
          signal_abort(abort_flag);
          break;
        }
        tc_fence_after();
        const uint32_t sa = sbase + st * stage_bytes;
        const uint64_t da = desc_tile(sa, S * BM), db = desc_tile(sa + a_bytes, S * BN);
        if constexpr (KIND == 1) {
          // chunk c accumulates in buffer c & 1, drained by the epilogue while
          // chunk c + 1 runs; before reusing a buffer wait for its last drain
          const int bsel = c & 1;
          if (kc == 0) {
            if (c >= 2) {
              if (!mbar_wait(bsel ? accempty1_bar : accempty_bar, ((c >> 1) - 1) & 1, abort_flag, a.wait_ns)) {
                signal_abort(abort_flag);
                break;
              }
              tc_fence_after();
            }
            f_started = false;
          }
          issue_tf32<BN>(tmem + (uint32_t)(bsel * BN), da, db, idesc, f_started);
          if (kc == ch - 1 || kb == nkb - 1) mma_commit(bsel ? accfull1_bar : accfull_bar);
          mma_commit(empty_bar(st));
          continue;
        }
        const bool wide = wide_tile<BN>(n_mma);
        if (kc != 0) {
          issue_stage<S, BN, 0>(wide, tmem, da, db, idesc, false, false);
        } else if (c == 0) {
          issue_stage<S, BN, 0>(wide, tmem, da, db, idesc, true, true);
        } else if (g.fdrain) {
          // the FP32 accumulator is drained with the exact groups: it restarts
          // every chunk, after the drain
          if (!mbar_wait(accempty_bar, (c - 1) & 1, abort_flag, a.wait_ns)) {
            signal_abort(abort_flag);
            break;
          }
          tc_fence_after();
          issue_stage<S, BN, 0>(wide, tmem, da, db, idesc, true, true);
        } else {
          // the FP32 group runs ahead while the exact groups drain
          issue_stage<S, BN, 1>(wide, tmem, da, db, idesc, false, false);
          if (!mbar_wait(accempty_bar, (c - 1) & 1, abort_flag, a.wait_ns)) {
            signal_abort(abort_flag);
            break;
          }
          tc_fence_after();
          issue_stage<S, BN, 2>(wide, tmem, da, db, idesc, true, false);
        }
        if (kc == ch - 1 || kb == nkb - 1) mma_commit(accfull_bar);
        mma_commit(empty_bar(st));
      }
      mma_commit(done_bar);
    }
  } else {
    // ---------------- epilogue: drain exact groups, assemble FP64 ----------------
    constexpr int CW = T::CW;
    const int q = warp & 3;
    const int cg = (warp - 2) >> 2;
    const int et = threadIdx.x - 64;  // 0 .. 511
    const uint32_t lbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cg * CW);
    const bool cols_live = cg * CW < n_valid;  // warp-uniform
    // Row / column tables of the tile for the assembly, filled while the MMAs
    // run: output offsets, mirror offsets (-1: none) and exponent scales.
    {
      const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
      if (et < BM) {
        const int i = m0 + et;
        const bool in = i < g.M;
        long long mr = -1;
        if (in && g.sym == SYM_ROWCOL) mr = g.c_c.at(i);
        long long ri = i;  // the pair's index for a packed-triangle row
        if (in && g.sym == SYM_TRIROW) {
          int mm, nn;
          tri_pair(i, g.pair_n, mm, nn);
          ri = (long long)mm * g.pair_n + nn;
          if (nn > mm) mr = g.c_r.at((long long)nn * g.pair_n + mm);
        }
        e_roff[et] = in ? g.c_r.at(ri) : 0;
        e_mr[et] = mr;
        e_srow[et] = in ? a.A.exps[abz * g.M + i] : 0;
      } else if (et < BM + BN) {
        const int c = et - BM, jj = n0 + c;
        const bool in = jj < g.N;
        long long mc = -1;
        if (in && g.sym == SYM_ROWCOL) mc = g.c_r.at(jj);
        long long cj = jj;
        if (in && g.sym == SYM_TRICOL) {
          int mm, nn;
          tri_pair(jj, g.pair_n, mm, nn);
          cj = (long long)mm * g.pair_n + nn;
          if (nn > mm) mc = g.c_c.at((long long)nn * g.pair_n + mm);
        }
        e_coff[c] = in ? g.c_c.at(cj) : 0;
        e_mc[c] = mc;
        e_scol[c] = in ? a.B.exps[bbz * g.N + jj] - (KIND ? 31 : group_exp(W, gE) + a.frac) : 0;
      }
    }
    long long R[CW];
#pragma unroll
    for (int j = 0; j < CW; ++j) R[j] = 0;
    const float two_frac = __int_as_float((127 + a.frac) << 23);  // 2^frac
    const float upE = __int_as_float((127 + (KIND ? 0 : group_exp(W, gE))) << 23);  // units of group gE per 1.0
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      if constexpr (KIND == 1) {
        // R (units of 2^-31) += rint(F 2^31): |F| < 2^7 per chunk of 96 k
        // (every |tf32 operand| < 1), so F 2^15 < 2^22 suits split_round
        const int bsel = c & 1;
        const bool got = mbar_wait(bsel ? accfull1_bar : accfull_bar, (c >> 1) & 1, abort_flag, a.wait_ns);
        if (!__all_sync(0xffffffffu, got)) {
          signal_abort(abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        if (cols_live) {
#pragma unroll
          for (int h = 0; h < CW / 8; ++h) {
            uint32_t v[8];
            tmem_ld8_async(lbase + (uint32_t)(bsel * BN + h * 8), v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) R[h * 8 + j] += split_round(__uint_as_float(v[j]) * 32768.0f, 16, 65536.0f);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bsel ? accempty1_bar : accempty_bar);
        continue;
      }
      const bool got = mbar_wait(accfull_bar, c & 1, abort_flag, a.wait_ns);
      if (!__all_sync(0xffffffffu, got)) {
        signal_abort(abort_flag);
        ok = false;
        break;
      }
      tc_fence_after();
      if (cols_live) {
        if (g.fdrain)
          drain_exact<BN, W, gE, false>(lbase, R, a.frac);
        else
          drain_exact<BN, W, gE, true>(lbase, R, 0);
      }
      if (has_inexact && g.fdrain && cols_live) {
#pragma unroll
        for (int h = 0; h < CW / 8; ++h) {
          uint32_t v[8];
          tmem_ld8_async(lbase + (uint32_t)(3 * BN + h * 8), v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) R[h * 8 + j] += split_round(__uint_as_float(v[j]) * upE, a.frac, two_frac);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accempty_bar);
    }
    if (ok) {
      const bool got = mbar_wait(done_bar, 0, abort_flag, a.wait_ns);
      if (!__all_sync(0xffffffffu, got)) signal_abort(abort_flag);
    }

    // CTA-uniform go / no-go for the assembly (every epilogue warp arrives here)
    if (epi_barrier_any(*abort_flag != 0)) ok = false;
    if (ok) {
      tc_fence_after();
      double* Cb = g.C + (long long)bz * g.c_sb;
      const bool mirror_rc = (g.sym == SYM_ROWCOL) && (m0 != n0);
      const bool rows_fast = g.c_c.div == 0 && g.c_c.s0 == 1 ? false : (g.c_r.div == 0 && g.c_r.s0 == 1);
      const int rlim = min(BM, g.M - m0), clim = min(BN, g.N - n0);
      // one output element: convert and store (plus its mirror)
      auto put = [&](long long z, int scale, long long ro, long long co, long long mr, long long mc) {
        double val;
        if (!scaled_to_double(z, scale, g.negate ? 0x80000000u : 0u, val)) val = fixed_to_double(z, scale, g.negate);
        Cb[ro + co] = val;
        if (mirror_rc) {
          Cb[mc + mr] = val;
        } else if (g.sym == SYM_TRICOL) {
          if (mc >= 0) Cb[ro + mc] = val;
        } else if (g.sym == SYM_TRIROW) {
          if (mr >= 0) Cb[mr + co] = val;
        }
      };
      // 1) fold the FP32 accumulator into the fixed point.  When the output's
      //    unit-stride index is the tile row (the TMEM lane), this layout
      //    already stores coalesced: convert and store here.  Otherwise park z
      //    in shared memory (the stage buffers are idle once every MMA has
      //    completed) for a transposed pass.
      const int row = q * 32 + lane;
      long long* Zs = reinterpret_cast<long long*>(smem);
      // z of this thread's row for its CW columns, handed to sink(c, z)
      auto fold = [&](auto&& sink) {
#pragma unroll
        for (int h = 0; h < CW / 8; ++h) {
          if constexpr (KIND == 1) {
            // every chunk is already in R (fixed point, 31 fraction bits)
#pragma unroll
            for (int j = 0; j < 8; ++j) sink(cg * CW + h * 8 + j, R[h * 8 + j]);
          } else {
            uint32_t v[8];
            if (has_inexact && !g.fdrain && cols_live) {
              tmem_ld8_async(lbase + (uint32_t)(3 * BN + h * 8), v);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              long long z = R[h * 8 + j];
              if (!g.fdrain)
                z = wide_pair<W, gE>(fold_pair<W, gE, has_inexact>(z, __uint_as_float(v[j]),
                                                                   (uint32_t)nchunks * (uint32_t)MAGIC_BITS));
              sink(cg * CW + h * 8 + j, z);
            }
          }
        }
      };
      // (the TMEM loads inside fold are warp-collective: no per-thread branch around it)
      if (rows_fast) {
        const bool row_live = row < rlim;
        fold([&](int c, long long z) {
          if (row_live && c < clim) put(z, e_srow[row] + e_scol[c], e_roff[row], e_coff[c], e_mr[row], e_mc[c]);
        });
      } else {
        fold([&](int c, long long z) { Zs[row * (BN + 1) + c] = z; });
      }
      // 2) rows are not the unit stride: assemble FP64 from shared memory with
      //    each thread on one column, lanes along the columns
      constexpr int U = 4;  // elements in flight per thread
      if (!rows_fast) {
        epi_barrier_any(false);
        constexpr int RSTEP = NUM_EPI_WARPS * 32 / BN;
        constexpr int NIT = BM / RSTEP;
        const int c = et % BN, r0 = et / BN;
        if (c < clim) {
          const int sc = e_scol[c];
          const long long co = e_coff[c], mc = e_mc[c];
          if (rlim == BM) {
#pragma unroll 1
            for (int it = 0; it < NIT; it += U) {
              long long zv[U], ro[U], mr[U];
              int sr[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int r = r0 + (it + u) * RSTEP;
                zv[u] = Zs[r * (BN + 1) + c];
                sr[u] = e_srow[r];
                ro[u] = e_roff[r];
                mr[u] = g.sym == SYM_NONE ? -1 : e_mr[r];
              }
#pragma unroll
              for (int u = 0; u < U; ++u) put(zv[u], sr[u] + sc, ro[u], co, mr[u], mc);
            }
          } else {
            for (int r = r0; r < rlim; r += RSTEP)
              put(Zs[r * (BN + 1) + c], e_srow[r] + sc, e_roff[r], co, e_mr[r], mc);
          }
        }
      }
    }
  }

  __syncthreads();
  // the abort flag is final here: after an abort, the copies the producer
  // issued must land before the CTA exits (a withheld stage's wait runs out)
  if (warp == 0 && lane == 0 && *abort_flag) {
    for (int kb = max(0, issued - STAGES); kb < issued; ++kb)
      mbar_wait(full_bar(kb % STAGES), (kb / STAGES) & 1, nullptr, a.wait_ns);
  }
  if (warp == 1) {
    if (*abort_flag) {
      // every MMA this CTA issued must be complete before TMEM is released
      mbar_wait(done_bar, 0, nullptr, a.wait_ns);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM_COLS) : "memory");
  }
}

// Persistent form (bf16 digits; outputs whose tile rows are the unit stride,
// so the epilogue stores straight from registers and never parks results in
// the stage buffers).  One CTA per SM; its producer takes the tiles from a
// counter in the caller's memory (so tiles start in order across the GPU, as
// with the hardware's block dispatch, and the CTAs that share a block of the
// large operand read it together) or, without one, walks t = blockIdx.x,
// + gridDim.x, ...; it hands each tile index to the MMA issuer and the
// epilogue through a small ring in shared memory.  The producer runs ahead across tile boundaries (the next
// tile's first stages load during this tile's epilogue), and the epilogue
// releases TMEM as soon as the last chunk is folded into registers, so the
// next tile's MMAs overlap the conversion and stores.  Pipeline phases
// (stages, chunks) count on across tiles.
template <int CODE, int BN, bool GROUPED, bool FD>
__device__ __forceinline__ void cta_persistent(const KArgs& a0, const KArgs* __restrict__ probs,
                                               const long long* __restrict__ starts, int nprob, int ntiles,
                                               unsigned int* counter, unsigned char* smem_raw) {
  constexpr int S = form_of(CODE).S, W = form_of(CODE).W;
  using T = TileCfg<BN, 0>;
  constexpr int gE = (S + 1) < 4 ? (S + 1) : 4;
  constexpr bool has_inexact = (S + 1) > 4;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t a_bytes = (uint32_t)S * TILE_BYTES, b_bytes = (uint32_t)S * T::B_TILE;
  constexpr uint32_t stage_bytes = a_bytes + b_bytes;
  constexpr uint32_t zs_bytes = BM * (BN + 1) * 8;  // same layout as cta_tile (smem_bytes)
  constexpr uint32_t data_bytes = STAGES * stage_bytes > zs_bytes ? STAGES * stage_bytes : zs_bytes;
  long long* e_roff = reinterpret_cast<long long*>(smem + data_bytes);
  long long* e_mr = e_roff + BM;
  long long* e_coff = e_mr + BM;
  long long* e_mc = e_coff + BN;
  int* e_srow = reinterpret_cast<int*>(e_mc + BN);
  int* e_scol = e_srow + BM;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + data_bytes + epi_table_bytes(BN));
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 5);
  // tile hand-off from the producer to the MMA issuer and the epilogue: a
  // ring of (problem, tile, stages per chunk) (tile -1 ends the walk) behind
  // full / empty barriers
  constexpr int RING = 4;
  static_assert(2 * STAGES + 6 <= 16 && 24 * 8 + 3 * RING * 4 <= 256, "barrier block of smem_bytes");
  volatile int* ring = reinterpret_cast<volatile int*>(bars + 24);
  volatile int* ringp = ring + RING;
  volatile int* ringc = ringp + RING;
  const uint32_t ringbar0 = smem_u32(bars + 16);
  auto ring_full = [&](int r) { return ringbar0 + 8u * r; };
  auto ring_empty = [&](int r) { return ringbar0 + 8u * (RING + r); };
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int st) { return bar0 + 8u * st; };
  auto empty_bar = [&](int st) { return bar0 + 8u * (STAGES + st); };
  const uint32_t accfull_bar = bar0 + 8u * (2 * STAGES), accempty_bar = bar0 + 8u * (2 * STAGES + 1),
                 done_bar = bar0 + 8u * (2 * STAGES + 2), fempty_bar = bar0 + 8u * (2 * STAGES + 3);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(empty_bar(i), 1);
    }
    mbar_init(accfull_bar, 1);
    mbar_init(accempty_bar, NUM_EPI_WARPS);
    mbar_init(done_bar, 1);
    mbar_init(fempty_bar, NUM_EPI_WARPS);
    for (int r = 0; r < RING; ++r) {
      mbar_init(ring_full(r), 1);
      mbar_init(ring_empty(r), 1 + NUM_EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(const_cast<uint32_t*>(tmem_slot))),
                 "r"(T::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  int gkb_issued = 0;  // stages the producer handled, all tiles (its lane 0)
  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      int& gkb = gkb_issued;
      bool aborted = false;
      unsigned int next = blockIdx.x;  // static walk when no tile counter is given
      for (int i = 0; !aborted; ++i) {
        const int slot = i % RING;
        if (!mbar_wait(ring_empty(slot), (uint32_t)(((i / RING) & 1) ^ 1), abort_flag, a0.wait_ns)) {
          signal_abort(abort_flag);
          break;
        }
        // next tile that has work (tiles a symmetry skips are passed over here)
        int t, p = 0, bz, m0, n0;
        for (;;) {
          unsigned int u;
          if (counter) {
            u = atomicAdd(counter, 1u) - a0.g.counter_start;
          } else {
            u = next;
            next += gridDim.x;
          }
          if (u >= (unsigned int)ntiles) {
            t = -1;
            break;
          }
          if constexpr (GROUPED) {
            p = find_problem(starts, nprob, u);
            t = (int)(u - starts[p]);
          } else {
            t = (int)u;
          }
          if (decode_tile<BN>(prob_ref<GROUPED>(a0, probs, p).g, t, bz, m0, n0)) break;
        }
        const KArgs& a = prob_ref<GROUPED>(a0, probs, p);
        const int nkb = (a.g.K + BK - 1) / BK;
        ring[slot] = t;
        ringp[slot] = p;
        if (t >= 0) ringc[slot] = chunk_blocks<W>(a.A, a.B, bz, m0, n0, nkb);
        mbar_arrive(ring_full(slot));
        if (t < 0) break;
        const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
        const unsigned char* ga = reinterpret_cast<const unsigned char*>(a.A.planes) + abz * a.A.batch_bytes() +
                                  (long long)(m0 / BM) * a.A.kblocks() * a_bytes;
        const int rb = n0 / SL_ROWS, r0 = n0 % SL_ROWS;
        const unsigned char* gbp = reinterpret_cast<const unsigned char*>(a.B.planes) + bbz * a.B.batch_bytes() +
                                   (long long)rb * a.B.kblocks() * (S * TILE_BYTES) + (r0 / 8) * 128;
        for (int kb = 0; kb < nkb; ++kb) {
          const int st = gkb % STAGES;
          const uint32_t ph = (uint32_t)((gkb / STAGES) & 1);
          if (!mbar_wait(empty_bar(st), ph ^ 1, abort_flag, a0.wait_ns)) {
            signal_abort(abort_flag);
            aborted = true;
            break;
          }
          if (gkb == a0.withhold && blockIdx.x == 0) {
            ++gkb;  // test hook: this stage never arrives
            continue;
          }
          mbar_expect_tx(full_bar(st), stage_bytes);
          const uint32_t sa = sbase + st * stage_bytes;
          bulk_load(sa, ga + (long long)kb * a_bytes, a_bytes, full_bar(st));
          const unsigned char* gblk = gbp + (long long)kb * (S * TILE_BYTES);
          if (BN == SL_ROWS) {
            bulk_load(sa + a_bytes, gblk, b_bytes, full_bar(st));
          } else {
#pragma unroll
            for (int kg = 0; kg < 2; ++kg)
#pragma unroll
              for (int s2 = 0; s2 < S; ++s2)
                bulk_load(sa + a_bytes + (kg * S + s2) * (BN * 16), gblk + (kg * S + s2) * SL_SLICE_STEP, BN * 16,
                          full_bar(st));
          }
          ++gkb;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int gkb = 0, gch = 0;
      bool aborted = false;
      for (int i = 0; !aborted; ++i) {
        const int slot = i % RING;
        if (!mbar_wait(ring_full(slot), (uint32_t)((i / RING) & 1), abort_flag, a0.wait_ns)) {
          signal_abort(abort_flag);
          break;
        }
        const int t = ring[slot], p = ringp[slot], ch = ringc[slot];  // ch: stages per chunk
        mbar_arrive(ring_empty(slot));
        if (t < 0) break;
        const OzGemm& g = prob_ref<GROUPED>(a0, probs, p).g;
        const int nkb = (g.K + BK - 1) / BK;
        int bz, m0, n0;
        decode_tile<BN>(g, t, bz, m0, n0);
        const int n_valid = min(BN, tile_cols(g, bz, n0));
        const int n_mma = (n_valid + 15) & ~15;
        const uint32_t idesc = (T::IDESC & ~(0x3Fu << 17)) | ((uint32_t)(n_mma >> 3) << 17);
        const bool wide = wide_tile<BN>(n_mma);
        // wait until the epilogue has read an accumulator
        auto drained = [&](uint32_t bar, uint32_t parity) {
          if (!mbar_wait(bar, parity, abort_flag, a0.wait_ns)) return false;
          tc_fence_after();
          return true;
        };
        int kc = 0;  // stage of the chunk
        for (int kb = 0; kb < nkb; ++kb) {
          const int st = gkb % STAGES;
          bool ok = mbar_wait(full_bar(st), (uint32_t)((gkb / STAGES) & 1), abort_flag, a0.wait_ns);
          if (ok) {
            tc_fence_after();
            const uint32_t sa = sbase + st * stage_bytes;
            const uint64_t da = desc_tile(sa, S * BM), db = desc_tile(sa + a_bytes, S * BN);
            const uint32_t last_chunk = (uint32_t)((gch - 1) & 1), last_tile = (uint32_t)((i - 1) & 1);
            if (kc > 0 || gch == 0) {
              issue_stage<S, BN, 0>(wide, tmem, da, db, idesc, kb == 0, kb == 0);
            } else if (FD || !has_inexact) {
              // a chunk's first stage: everything is drained after every chunk
              ok = drained(accempty_bar, last_chunk) && (FD || kb > 0 || drained(fempty_bar, last_tile));
              if (ok) issue_stage<S, BN, 0>(wide, tmem, da, db, idesc, true, true);
            } else if (kb == 0) {
              // a tile's first stage: the exact groups are drained before the
              // FP32 group is folded in
              ok = drained(accempty_bar, last_chunk);
              if (ok) issue_stage<S, BN, 2>(wide, tmem, da, db, idesc, true, false);
              ok = ok && drained(fempty_bar, last_tile);
              if (ok) issue_stage<S, BN, 1>(wide, tmem, da, db, idesc, false, true);
            } else {
              // a later chunk's: the FP32 group goes on while the exact groups
              // drain (one stage of it: taking several stages of one kind first
              // hides the drain but splits the merged MMAs, 8 reads of A slices a
              // stage instead of 5, and shared memory bounds the MMAs: 1592 clocks
              // a stage with four, 1541 with one)
              issue_stage<S, BN, 1>(wide, tmem, da, db, idesc, false, false);
              ok = drained(accempty_bar, last_chunk);
              if (ok) issue_stage<S, BN, 2>(wide, tmem, da, db, idesc, true, false);
            }
          }
          if (!ok) {
            signal_abort(abort_flag);
            aborted = true;
            break;
          }
          mma_commit(empty_bar(st));
          ++gkb;
          if (++kc == ch || kb == nkb - 1) {
            mma_commit(accfull_bar);
            ++gch;
            kc = 0;
          }
        }
      }
      mma_commit(done_bar);
    }
  } else {
    // ---------------- epilogue ----------------
    constexpr int CW = T::CW;
    const int q = warp & 3;
    const int cg = (warp - 2) >> 2;
    const int et = threadIdx.x - 64;
    const uint32_t lbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cg * CW);
    const float upE = __int_as_float((127 + group_exp(W, gE)) << 23);
    const int row = q * 32 + lane;
    int gch = 0;
    for (int i = 0;; ++i) {
      const int slot = i % RING;
      const bool got = mbar_wait(ring_full(slot), (uint32_t)((i / RING) & 1), abort_flag, a0.wait_ns);
      if (!got) signal_abort(abort_flag);
      const int t = got ? ring[slot] : -1;
      const int p = got ? ringp[slot] : 0, ch = got ? (int)ringc[slot] : (int)CH_MIN;
      __syncwarp();
      if (lane == 0) mbar_arrive(ring_empty(slot));
      // every epilogue warp is done with the previous tile's tables, and all
      // of them take the same branch
      if (epi_barrier_any(!got || *abort_flag != 0)) break;
      if (t < 0) break;
      const KArgs& a = prob_ref<GROUPED>(a0, probs, p);
      const OzGemm& g = a.g;
      const float two_frac = __int_as_float((127 + a.frac) << 23);  // 2^frac
      int bz, m0, n0;
      decode_tile<BN>(g, t, bz, m0, n0);
      const int nkb = (g.K + BK - 1) / BK;
      const int nchunks = (nkb + ch - 1) / ch;
      {
        const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
        if (et < BM) {
          const int i = m0 + et;
          const bool in = i < g.M;
          long long mr = -1;
          if (in && g.sym == SYM_ROWCOL) mr = g.c_c.at(i);
          long long ri = i;  // the pair's index for a packed-triangle row
          if (in && g.sym == SYM_TRIROW) {
            int mm, nn;
            tri_pair(i, g.pair_n, mm, nn);
            ri = (long long)mm * g.pair_n + nn;
            if (nn > mm) mr = g.c_r.at((long long)nn * g.pair_n + mm);
          }
          e_roff[et] = in ? g.c_r.at(ri) : 0;
          e_mr[et] = mr;
          e_srow[et] = in ? a.A.exps[abz * g.M + i] : 0;
        } else if (et < BM + BN) {
          const int c = et - BM, jj = n0 + c;
          const bool in = jj < g.N;
          long long mc = -1;
          if (in && g.sym == SYM_ROWCOL) mc = g.c_r.at(jj);
          if (in && g.sym == SYM_BATCHCOL) mc = (long long)jj * g.c_sb + g.c_c.at(bz);
          e_coff[c] = in ? g.c_c.at(jj) : 0;
          e_mc[c] = mc;
          e_scol[c] = in ? a.B.exps[bbz * g.N + jj] - group_exp(W, gE) - a.frac : 0;
        }
      }
      epi_barrier_any(false);  // tables visible
      const int n_valid = min(BN, tile_cols(g, bz, n0));
      const bool cols_live = cg * CW < n_valid;  // warp-uniform
      long long R[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) R[j] = 0;
      bool ok = true;
      for (int c = 0; c < nchunks; ++c) {
        const bool got = mbar_wait(accfull_bar, (uint32_t)(gch & 1), abort_flag, a0.wait_ns);
        if (!__all_sync(0xffffffffu, got)) {
          signal_abort(abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        if (FD && cols_live) {
          // the FP32 group is drained every chunk too
          drain_exact<BN, W, gE, false>(lbase, R, a.frac);
          if (has_inexact) {
#pragma unroll
            for (int h = 0; h < CW / 8; ++h) {
              uint32_t v[8];
              tmem_ld8_async(lbase + (uint32_t)(3 * BN + h * 8), v);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j)
                R[h * 8 + j] += split_round(__uint_as_float(v[j]) * upE, a.frac, two_frac);
            }
          }
        } else if (cols_live) {
          drain_exact<BN, W, gE, true>(lbase, R, 0);
        }
        ++gch;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty_bar);  // the exact groups (FD: all of TMEM) are free
      }
      if (!ok) continue;  // the next tile's barrier sees the abort flag in every warp
      if (!FD && cols_live) {
        // fold the FP32 group in, so that nothing is left in TMEM
        const uint32_t bias = (uint32_t)nchunks * (uint32_t)MAGIC_BITS;
#pragma unroll
        for (int h = 0; h < CW / 4; ++h) {
          uint32_t v[4] = {};
          if (has_inexact) {
            tmem_ld4_async(lbase + (uint32_t)(3 * BN + h * 4), v);
            tmem_wait_ld();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            asm volatile("" : "+l"(R[h * 4 + j]), "+r"(v[j]));  // in order: few live temporaries
            R[h * 4 + j] = fold_pair<W, gE, has_inexact>(R[h * 4 + j], __uint_as_float(v[j]), bias);
            asm volatile("" : "+l"(R[h * 4 + j]));
          }
        }
      }
      if (!FD) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(fempty_bar);  // the FP32 group is free
      }
      // convert and store from registers (rows are the output's unit stride)
      double* Cb = g.C + (long long)bz * g.c_sb;
      const int rlim = min(BM, g.M - m0), cw = min(CW, tile_cols(g, bz, n0) - cg * CW);  // this warp's columns
      if (row < rlim && cw > 0) {
        const uint32_t flip = g.negate ? 0x80000000u : 0u;
        const int c0 = cg * CW, srow = e_srow[row];
        // a mirror image: none, of an off-diagonal tile (SYM_ROWCOL; the row's
        // columns are consecutive there), of a pair (SYM_TRIROW), or the batch
        // entry of each column below the batch index (SYM_BATCHCOL)
        const bool mirror_rc = g.sym == SYM_ROWCOL && m0 != n0;
        const long long ro = e_roff[row], mr = g.sym == SYM_TRIROW || mirror_rc ? e_mr[row] : -1;
        double* mir = mirror_rc ? Cb + mr + e_mc[c0] : nullptr;
        const int vec = !mirror_rc || cw < CW ? 1 : store_width(mir);
        bool fine = true;
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          double v[4];
          const int4 sc = *reinterpret_cast<const int4*>(e_scol + c0 + j);
          const int scs[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            fine &= scaled_to_double(FD ? R[j + u] : wide_pair<W, gE>(R[j + u]), srow + scs[u], flip, v[u]) ||
                    j + u >= cw;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (j + u < cw) {
              const long long co = e_coff[c0 + j + u];
              Cb[ro + co] = v[u];
              if (mr >= 0 && !mirror_rc) Cb[mr + co] = v[u];
              if (g.sym == SYM_BATCHCOL && n0 + c0 + j + u < bz) g.C[ro + e_mc[c0 + j + u]] = v[u];
            }
          if (mirror_rc) {
            if (vec == 4) {
              store4(mir + j, v);
            } else if (vec == 2) {
              *reinterpret_cast<double2*>(mir + j) = make_double2(v[0], v[1]);
              *reinterpret_cast<double2*>(mir + j + 2) = make_double2(v[2], v[3]);
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (j + u < cw) mir[j + u] = v[u];
            }
          }
          asm volatile("" ::: "memory");  // four columns at a time: 64 of the 96 registers hold R
        }
        if (!fine) {  // a result outside the normal range: the general conversion for the row, from local memory
          long long z[CW];
#pragma unroll
          for (int j = 0; j < CW; ++j) z[j] = R[j];
#pragma unroll 1
          for (int j = 0; j < cw; ++j) {
            const double val =
                fixed_to_double(FD ? z[j] : wide_pair<W, gE>(z[j]), srow + e_scol[c0 + j], g.negate);
            const long long co = e_coff[c0 + j];
            Cb[ro + co] = val;
            if (mirror_rc) mir[j] = val;
            else if (mr >= 0) Cb[mr + co] = val;
            if (g.sym == SYM_BATCHCOL && n0 + c0 + j < bz) g.C[ro + e_mc[c0 + j]] = val;
          }
        }
      }
    }
  }

  __syncthreads();
  // after an abort, the producer's copies land before the CTA exits
  if (warp == 0 && lane == 0 && *abort_flag) {
    for (int k = gkb_issued > STAGES ? gkb_issued - STAGES : 0; k < gkb_issued; ++k)
      mbar_wait(full_bar(k % STAGES), (uint32_t)((k / STAGES) & 1), nullptr, a0.wait_ns);
  }
  if (warp == 1) {
    if (*abort_flag) mbar_wait(done_bar, 0, nullptr, a0.wait_ns);
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM_COLS) : "memory");
  }
}

template <int CODE, int BN, bool FD>
__global__ void __maxnreg__(MAX_REGS) ozaki_persistent_kernel(const __grid_constant__ KArgs a, int ntiles) {
  extern __shared__ unsigned char smem_raw[];
  chain_wait();
  if (*(volatile int*)&g_tc_status != 0) return;
  cta_persistent<CODE, BN, false, FD>(a, nullptr, nullptr, 1, ntiles, a.g.tile_counter, smem_raw);
}

// Grouped persistent launch: problem p owns the tiles [starts[p], starts[p + 1])
// of one tile space walked in order through `counter` (caller memory, zeroed
// before the launch), one CTA per SM.
template <int CODE, int BN, bool FD>
__global__ void __maxnreg__(MAX_REGS)
    ozaki_persistent_grouped_kernel(const KArgs* __restrict__ probs, const long long* __restrict__ starts, int nprob,
                                    int ntiles, unsigned int* counter) {
  extern __shared__ unsigned char smem_raw[];
  chain_wait();
  if (*(volatile int*)&g_tc_status != 0) return;
  cta_persistent<CODE, BN, true, FD>(probs[0], probs, starts, nprob, ntiles, counter, smem_raw);
}

template <int CODE, int BN>
__global__ void __maxnreg__(MAX_REGS) ozaki_kernel(const __grid_constant__ KArgs a) {
  chain_wait();
  extern __shared__ unsigned char smem_raw[];
  // a CTA of this or an earlier launch gave up: do not start (the host sees the status word)
  if (*(volatile int*)&g_tc_status != 0) return;
  int bz, m0, n0;
  if (!decode_tile<BN>(a.g, (long long)blockIdx.x + (long long)blockIdx.y * gridDim.x, bz, m0, n0)) return;
  cta_tile<CODE, BN>(a, bz, m0, n0, smem_raw);
}

// Grouped launch: problem p owns the tiles [starts[p], starts[p + 1]).
template <int CODE, int BN>
__global__ void __maxnreg__(MAX_REGS)
    ozaki_grouped_kernel(const KArgs* __restrict__ probs, const long long* __restrict__ starts, int nprob) {
  chain_wait();
  extern __shared__ unsigned char smem_raw[];
  if (*(volatile int*)&g_tc_status != 0) return;
  const long long t = (long long)blockIdx.x + (long long)blockIdx.y * gridDim.x;
  int lo = 0, hi = nprob;  // find p with starts[p] <= t < starts[p + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (starts[mid] <= t) lo = mid; else hi = mid;
  }
  if (t >= starts[nprob]) return;
  const KArgs& a = probs[lo];
  int bz, m0, n0;
  if (!decode_tile<BN>(a.g, t - starts[lo], bz, m0, n0)) return;
  cta_tile<CODE, BN>(a, bz, m0, n0, smem_raw);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// `code`: split code (1..6 digit slices or SPLIT_TF32X3)
size_t smem_bytes(int code, int BN) {
  const int S = form_of(code).S;
  const size_t stages = (size_t)STAGES * S * (TILE_BYTES + BN * SL_K * 2);
  const size_t zs = (size_t)BM * (BN + 1) * 8;
  return (stages > zs ? stages : zs) + epi_table_bytes(BN) + 256 + 1024;
}

using KernelFn = void (*)(KArgs);
using GroupedFn = void (*)(const KArgs*, const long long*, int);

template <int BN>
KernelFn single_for(int S) {
  switch (S) {
    case 1: return ozaki_kernel<1, BN>;
    case 2: return ozaki_kernel<2, BN>;
    case 3: return ozaki_kernel<3, BN>;
    case 4: return ozaki_kernel<4, BN>;
    case 5: return ozaki_kernel<5, BN>;
    case SPLIT_TF32X3: return ozaki_kernel<SPLIT_TF32X3, BN>;
    default: return ozaki_kernel<6, BN>;
  }
}

template <int BN>
GroupedFn grouped_for(int S) {
  switch (S) {
    case 1: return ozaki_grouped_kernel<1, BN>;
    case 2: return ozaki_grouped_kernel<2, BN>;
    case 3: return ozaki_grouped_kernel<3, BN>;
    case 4: return ozaki_grouped_kernel<4, BN>;
    case 5: return ozaki_grouped_kernel<5, BN>;
    case SPLIT_TF32X3: return ozaki_grouped_kernel<SPLIT_TF32X3, BN>;
    default: return ozaki_grouped_kernel<6, BN>;
  }
}

// fd: the FP32 group is drained per chunk (K > FDRAIN_K)
using PersistFn = void (*)(KArgs, int);
template <bool FD>
PersistFn persistent_of(int S) {
  switch (S) {
    case 1: return ozaki_persistent_kernel<1, 128, FD>;
    case 2: return ozaki_persistent_kernel<2, 128, FD>;
    case 3: return ozaki_persistent_kernel<3, 128, FD>;
    case 4: return ozaki_persistent_kernel<4, 128, FD>;
    case 5: return ozaki_persistent_kernel<5, 128, FD>;
    default: return ozaki_persistent_kernel<6, 128, FD>;
  }
}
PersistFn persistent_for(int S, bool fd) { return fd ? persistent_of<true>(S) : persistent_of<false>(S); }

using PersistGroupedFn = void (*)(const KArgs*, const long long*, int, int, unsigned int*);
template <bool FD>
PersistGroupedFn persistent_grouped_of(int S) {
  switch (S) {
    case 1: return ozaki_persistent_grouped_kernel<1, 128, FD>;
    case 2: return ozaki_persistent_grouped_kernel<2, 128, FD>;
    case 3: return ozaki_persistent_grouped_kernel<3, 128, FD>;
    case 4: return ozaki_persistent_grouped_kernel<4, 128, FD>;
    case 5: return ozaki_persistent_grouped_kernel<5, 128, FD>;
    default: return ozaki_persistent_grouped_kernel<6, 128, FD>;
  }
}
PersistGroupedFn persistent_grouped_for(int S, bool fd) {
  return fd ? persistent_grouped_of<true>(S) : persistent_grouped_of<false>(S);
}

KernelFn kernel_for(int S, int BN) {
  return BN == 32 ? single_for<32>(S) : BN == 64 ? single_for<64>(S) : single_for<128>(S);
}
GroupedFn grouped_kernel_for(int S, int BN) {
  return BN == 32 ? grouped_for<32>(S) : BN == 64 ? grouped_for<64>(S) : grouped_for<128>(S);
}

// Opt every instantiation in to its dynamic shared memory once per device
// context (again after a cudaDeviceReset, whose new context has a new id).
int g_num_sms[64] = {0};

int configure_device() {
  static std::mutex mu;
  static unsigned long long configured[64] = {0};  // context id configured on each device
  int dev = 0;
  GB_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
  const unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64 || (ctx != 0 && configured[dev] == ctx)) return GB_OK;
  for (int bn : {32, 64, 128})
    for (int sl : {1, 2, 3, 4, 5, 6, SPLIT_TF32X3}) {
      const int sm = (int)smem_bytes(sl, bn);
      GB_TRY(cuda_status(cudaFuncSetAttribute(kernel_for(sl, bn), cudaFuncAttributeMaxDynamicSharedMemorySize, sm),
                         "cudaFuncSetAttribute"));
      GB_TRY(cuda_status(
          cudaFuncSetAttribute(grouped_kernel_for(sl, bn), cudaFuncAttributeMaxDynamicSharedMemorySize, sm),
          "cudaFuncSetAttribute"));
    }
  for (int sl = 1; sl <= 6; ++sl)
    for (bool fd : {false, true}) {
      const int sm = (int)smem_bytes(sl, 128);
      GB_TRY(cuda_status(cudaFuncSetAttribute(persistent_for(sl, fd), cudaFuncAttributeMaxDynamicSharedMemorySize, sm),
                         "cudaFuncSetAttribute"));
      GB_TRY(cuda_status(
          cudaFuncSetAttribute(persistent_grouped_for(sl, fd), cudaFuncAttributeMaxDynamicSharedMemorySize, sm),
          "cudaFuncSetAttribute"));
    }
  GB_TRY(cuda_status(cudaDeviceGetAttribute(&g_num_sms[dev], cudaDevAttrMultiProcessorCount, dev),
                     "cudaDeviceGetAttribute"));
  configured[dev] = current_context_id();
  return GB_OK;
}

// Fraction bits of the fixed-point assembly: keep |z| < 2^62 (|z| 2^-frac is
// below 1.01 K units of 1.0, each 2^group_exp units of the last exact group).
int frac_bits(int code, int K) {
  if (code == SPLIT_TF32X3) return 0;
  if (K <= FDRAIN_K) return PAIR_FRAC;
  const SliceForm f = form_of(code);
  const int gE = f.S + 1 < 4 ? f.S + 1 : 4;
  int lg = 0;
  while (lg < 31 && (1ll << lg) < K) ++lg;
  const int rbits = lg + 1 + group_exp(f.W, gE);
  int frac = 62 - rbits;
  if (frac > 16) frac = 16;
  if (frac < 0) frac = 0;
  return frac;
}

int check_problem(const SlicedDesc& A, const SlicedDesc& B, const OzGemm& g) {
  const SliceForm f = form_of(g.S);
  GB_REQUIRE(valid_split(g.S) && A.S == f.S && B.S == f.S && A.kind == f.kind && B.kind == f.kind && A.W == f.W &&
                 B.W == f.W,
             GB_ERR_INVALID_ARG, "ozaki_gemm: split form mismatch (code %d)", g.S);
  GB_REQUIRE(g.bn == 32 || g.bn == 64 || g.bn == 128, GB_ERR_INVALID_ARG, "ozaki_gemm: N tile %d not in {32,64,128}",
             g.bn);
  GB_REQUIRE(A.rows == g.M && B.rows == g.N && A.K == g.K && B.K == g.K && (A.batch == g.batch || A.batch == 1) &&
                 (B.batch == g.batch || B.batch == 1),
             GB_ERR_BAD_SHAPE, "ozaki_gemm: operand shapes do not match the GEMM");
  GB_REQUIRE(g.sym != SYM_ROWCOL || (g.M == g.N && g.bn == BM), GB_ERR_BAD_SHAPE,
             "ozaki_gemm: SYM_ROWCOL needs M == N and 128-wide tiles");
  GB_REQUIRE(g.sym != SYM_PAIRCOL, GB_ERR_INVALID_ARG,
             "ozaki_gemm: pair symmetry runs over the packed pair triangle here (SYM_TRIROW / SYM_TRICOL)");
  GB_REQUIRE(g.sym != SYM_BATCHCOL || (g.batch == g.N && g.S <= 6 && g.bn == 128 && g.c_r.div == 0 && g.c_r.s0 == 1 &&
                                       !(g.c_c.div == 0 && g.c_c.s0 == 1)),
             GB_ERR_BAD_SHAPE, "ozaki_gemm: SYM_BATCHCOL needs batch == N and the persistent form");
  GB_REQUIRE(g.sym != SYM_TRIROW || (long long)g.pair_n * (g.pair_n + 1) / 2 == g.M, GB_ERR_BAD_SHAPE,
             "ozaki_gemm: SYM_TRIROW needs M == pair_n (pair_n + 1) / 2");
  GB_REQUIRE(g.sym != SYM_TRICOL || (long long)g.pair_n * (g.pair_n + 1) / 2 == g.N, GB_ERR_BAD_SHAPE,
             "ozaki_gemm: SYM_TRICOL needs N == pair_n (pair_n + 1) / 2");
  GB_REQUIRE(g.K > 0 && g.batch <= 65535, GB_ERR_BAD_SHAPE, "ozaki_gemm: bad K or batch");
  GB_REQUIRE((reinterpret_cast<uintptr_t>(A.planes) & 15) == 0 && (reinterpret_cast<uintptr_t>(B.planes) & 15) == 0,
             GB_ERR_INVALID_ARG, "ozaki_gemm: slice planes not 16-byte aligned");
  return GB_OK;
}

constexpr unsigned long long kDefaultWaitNs = 2000000000ull;  // 2 s per wait
std::atomic<unsigned long long> g_wait_limit_ns{kDefaultWaitNs};
std::atomic<int> g_withhold_stage{-1};

KArgs make_args(const SlicedDesc& A, const SlicedDesc& B, const OzGemm& g) {
  KArgs ka{g, A, B, frac_bits(g.S, g.K), wait_limit_ns(), withheld_stage()};
  if (g.K > FDRAIN_K && g.S != SPLIT_TF32X3) ka.g.fdrain = 1;
  return ka;
}

dim3 grid_for(long long tiles) {
  // x up to 2^31 - 1; split very large tile counts over y
  const long long gx = tiles < 2147483647LL ? tiles : 65536;
  return dim3((unsigned)gx, (unsigned)((tiles + gx - 1) / gx));
}

int launch_error(const char* tag, cudaError_t le, int S, int BN) {
  char info[512];
  ozaki_kernel_info(info, sizeof(info));
  set_error(GB_ERR_CUDA, "%s: %s (S=%d BN=%d threads %d, dynamic smem %zu; %s)", tag, cudaGetErrorString(le), S, BN,
            THREADS, smem_bytes(S, BN), info);
  return GB_ERR_CUDA;
}

}  // namespace

unsigned long long wait_limit_ns() { return g_wait_limit_ns.load(); }
int withheld_stage() { return g_withhold_stage.load(); }

long long ozaki_tiles(const OzGemm& g) {
  return ((long long)(g.M + BM - 1) / BM) * ((g.N + g.bn - 1) / g.bn) * (long long)g.batch;
}

int ozaki_gemm(const SlicedDesc& A, const SlicedDesc& B, const OzGemm& g, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return GB_OK;
  GB_TRY(check_problem(A, B, g));
  GB_TRY(configure_device());
  const KArgs ka = make_args(A, B, g);
  const long long tiles = ozaki_tiles(g);
  // outputs whose tile rows are the unit stride take the persistent kernel
  const bool rows_fast = !(g.c_c.div == 0 && g.c_c.s0 == 1) && (g.c_r.div == 0 && g.c_r.s0 == 1);
  int dev = 0;
  cudaGetDevice(&dev);
  const int nsm = (dev >= 0 && dev < 64 && g_num_sms[dev] > 0) ? g_num_sms[dev] : 0;
  if (g.S >= 1 && g.S <= 6 && g.bn == 128 && rows_fast && nsm > 0 && tiles < (1LL << 30)) {
    const long long grid = tiles < nsm ? tiles : nsm;
    KArgs kp = ka;
    if (g.tile_counter && tiles > grid) {
      if (g.counter_start == 0)
        GB_TRY(cuda_status(cudaMemsetAsync(g.tile_counter, 0, sizeof(unsigned int), stream), "tile counter"));
    } else {
      kp.g.tile_counter = nullptr;  // one tile per CTA, or the static walk
    }
    const int pi = prof_begin(g.tag, stream);
    const cudaError_t e = launch_chain(persistent_for(g.S, ka.g.fdrain), dim3((unsigned)grid), dim3(THREADS),
                                       smem_bytes(g.S, 128), stream, kp, (int)tiles);
    prof_end(pi, stream);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return launch_error(g.tag, e, g.S, g.bn);
    }
  } else {
    GB_REQUIRE(g.sym != SYM_BATCHCOL, GB_ERR_BAD_SHAPE, "%s: SYM_BATCHCOL runs on the persistent kernel alone", g.tag);
    const int pi = prof_begin(g.tag, stream);
    const cudaError_t e =
        launch_chain(kernel_for(g.S, g.bn), grid_for(tiles), dim3(THREADS), smem_bytes(g.S, g.bn), stream, ka);
    prof_end(pi, stream);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return launch_error(g.tag, e, g.S, g.bn);
    }
  }
  const cudaError_t le = cudaGetLastError();
  if (le != cudaSuccess) return launch_error(g.tag, le, g.S, g.bn);
  return GB_OK;
}

// table layout: KArgs[nprob] | starts[nprob + 1] | tile counter
size_t ozaki_group_table_bytes(int nprob) {
  return align256((size_t)nprob * sizeof(KArgs)) + align256((size_t)(nprob + 1) * sizeof(long long)) + 256;
}

int ozaki_group_upload(const OzProblem* probs, int nprob, void* table, bool* persistent, bool* group_fdrain) {
  GB_REQUIRE(nprob >= 1 && probs && table, GB_ERR_INVALID_ARG, "ozaki_group_upload: empty group");
  std::vector<KArgs> args;
  std::vector<long long> starts(1, 0);
  bool all_rows_fast = true;
  int fdrain = 0;
  for (int i = 0; i < nprob; ++i) {
    GB_TRY(check_problem(probs[i].A, probs[i].B, probs[i].g));
    GB_REQUIRE(probs[i].g.S == probs[0].g.S && probs[i].g.bn == probs[0].g.bn, GB_ERR_INVALID_ARG,
               "ozaki_group_upload: a group shares one slice count and tile width");
    args.push_back(make_args(probs[i].A, probs[i].B, probs[i].g));
    fdrain |= args.back().g.fdrain;
    starts.push_back(starts.back() + ozaki_tiles(probs[i].g));
    const OzGemm& g = probs[i].g;
    all_rows_fast = all_rows_fast && !(g.c_c.div == 0 && g.c_c.s0 == 1) && (g.c_r.div == 0 && g.c_r.s0 == 1);
  }
  for (int i = 0; i < nprob; ++i)
    GB_REQUIRE(probs[i].g.sym != SYM_BATCHCOL, GB_ERR_INVALID_ARG, "ozaki_group_upload: no SYM_BATCHCOL in a group");
  // one drain form for the group (the fraction bits suit both)
  for (KArgs& ka : args) ka.g.fdrain = fdrain;
  if (group_fdrain) *group_fdrain = fdrain != 0;
  // the persistent form stores from the epilogue's registers: every output's
  // tile rows must be its unit stride; bf16 digits and 128-wide tiles
  if (persistent)
    *persistent = all_rows_fast && probs[0].g.S >= 1 && probs[0].g.S <= 6 && probs[0].g.bn == 128 &&
                  starts.back() < (1LL << 30);
  char* t = static_cast<char*>(table);
  GB_TRY(cuda_status(cudaMemcpy(t, args.data(), nprob * sizeof(KArgs), cudaMemcpyHostToDevice), "group table"));
  GB_TRY(cuda_status(cudaMemcpy(t + align256((size_t)nprob * sizeof(KArgs)), starts.data(),
                                (nprob + 1) * sizeof(long long), cudaMemcpyHostToDevice),
                     "group table"));
  return GB_OK;
}

int ozaki_gemm_grouped(const void* table, int nprob, long long total_tiles, int S, int bn, cudaStream_t stream,
                       const char* tag, bool persistent, bool fdrain) {
  if (total_tiles <= 0) return GB_OK;
  GB_TRY(configure_device());
  const char* t = static_cast<const char*>(table);
  const KArgs* probs = reinterpret_cast<const KArgs*>(t);
  const size_t off_starts = align256((size_t)nprob * sizeof(KArgs));
  const long long* starts = reinterpret_cast<const long long*>(t + off_starts);
  int dev = 0;
  cudaGetDevice(&dev);
  const int nsm = (dev >= 0 && dev < 64 && g_num_sms[dev] > 0) ? g_num_sms[dev] : 0;
  if (persistent && S >= 1 && S <= 6 && bn == 128 && nsm > 0 && total_tiles < (1LL << 30)) {
    // one CTA per SM walking the concatenated tile space in order
    unsigned int* counter = reinterpret_cast<unsigned int*>(
        const_cast<char*>(t) + off_starts + align256((size_t)(nprob + 1) * sizeof(long long)));
    const long long grid = total_tiles < nsm ? total_tiles : nsm;
    GB_TRY(cuda_status(cudaMemsetAsync(counter, 0, sizeof(unsigned int), stream), "grouped tile counter"));
    const int pi = prof_begin(tag, stream);
    persistent_grouped_for(S, fdrain)<<<(unsigned)grid, THREADS, smem_bytes(S, 128), stream>>>(probs, starts, nprob,
                                                                                      (int)total_tiles, counter);
    prof_end(pi, stream);
    const cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return launch_error(tag, le, S, 128);
    return GB_OK;
  }
  const int pi = prof_begin(tag, stream);
  grouped_kernel_for(S, bn)<<<grid_for(total_tiles), THREADS, smem_bytes(S, bn), stream>>>(probs, starts, nprob);
  prof_end(pi, stream);
  const cudaError_t le = cudaGetLastError();
  if (le != cudaSuccess) return launch_error(tag, le, S, bn);
  return GB_OK;
}

int ozaki_status(int reset, int* out) {
  int v = 0;
  GB_TRY(cuda_status(cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int)), "read tensor-core status"));
  if (reset) {
    const int zero = 0;
    GB_TRY(cuda_status(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)), "reset tensor-core status"));
  }
  *out = v;
  return GB_OK;
}

int* device_status_word() {
  static std::mutex mu;
  static unsigned long long ctx_ids[64] = {0};
  static int* addrs[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  const unsigned long long id = current_context_id();
  std::lock_guard<std::mutex> lk(mu);
  if (addrs[dev] == nullptr || id == 0 || ctx_ids[dev] != id) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_tc_status) != cudaSuccess) return nullptr;
    addrs[dev] = static_cast<int*>(p);
    ctx_ids[dev] = current_context_id();
  }
  return addrs[dev];
}

// The two driver functions come through the runtime's entry-point query, so
// the library keeps no link-time dependency on the driver library (it loads
// on a machine without a GPU, where only its size queries are used).
unsigned long long current_context_id() {
  using GetCurrentFn = CUresult (*)(CUcontext*);
  using GetIdFn = CUresult (*)(CUcontext, unsigned long long*);
  static GetCurrentFn get_current = nullptr;
  static GetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetIdFn>(f);
  });
  if (!get_current || !get_id) return 0;
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return 0;
  unsigned long long id = 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

int ozaki_kernel_info(char* out, size_t len) {
  cudaFuncAttributes fa{};
  cudaError_t e = cudaFuncGetAttributes(&fa, kernel_for(6, 128));
  int occ = -1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel_for(6, 128), THREADS, smem_bytes(6, 128));
  int dev = 0, regs_sm = 0, smem_optin = 0, max_thr = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&max_thr, cudaDevAttrMaxThreadsPerBlock, dev);
  snprintf(out, len,
           "attr=%s regs=%d maxThreadsPerBlock=%d localBytes=%zu staticSmem=%zu maxDynSmem=%d occupancy=%d "
           "regsPerSM=%d smemOptin=%d devMaxThreads=%d",
           cudaGetErrorString(e), fa.numRegs, fa.maxThreadsPerBlock, fa.localSizeBytes, fa.sharedSizeBytes,
           fa.maxDynamicSharedSizeBytes, occ, regs_sm, smem_optin, max_thr);
  return GB_OK;
}

}  // namespace gb

extern "C" int gb_set_wait_limit_ns(unsigned long long limit_ns) {
  gb::clear_error();
  gb::g_wait_limit_ns.store(limit_ns ? limit_ns : gb::kDefaultWaitNs);
  return GB_OK;
}

extern "C" int gb_test_withhold_stage(int stage) {
  gb::clear_error();
  gb::g_withhold_stage.store(stage < 0 ? -1 : stage);
  return GB_OK;
}
