// FP64-accurate GEMM on the tensor cores: see f64_tc.cuh.
//
// One persistent CTA per SM, 18 warps as in ozaki_tc.cu: a producer (one bulk
// copy of A's planes and two per plane of B's per 16-k stage, four stages), the
// MMA issuer, and 16 epilogue warps.  CTA tile 128 x 64: five exact accumulators,
// the FP32 one and the sizes' take 448 TMEM columns (a 128-wide tile's would need
// 896), and an epilogue thread keeps 16 elements, each as a 64-bit integer and an FP64
// sum, in registers.
//
// Per 16-k stage there are 28 products of 128 x 64 and the one of the sizes, of which
// the exact ones run as MMAs up to 256 columns wide (consecutive B slices into
// consecutive accumulators); a 64-column MMA takes 53 clocks, 83 % of a 128-column one:
// ~1150 clocks of MMAs.  Measured: 2300 to 2500 clocks a stage of a long K, 3300 where a
// tile has 15 stages, no unit above 40 %.  What bounds it is the latency of one tile's
// epilogue (TMEM loads, 3.75 FP64 instructions an element at 64 clocks a warp, stores)
// with one CTA on an SM.  A Lagrangian at nbf=300 takes 91.5 ms on the FP64 units, 5.6 here.
//
// Which tiles are done: an element is held to FP64's bound by its sum of sizes P,
// about S = sum_k |a_k b_k| over the product of its two row bounds.  The dropped
// digits and digit products leave 2^-63.2 sqrt(K) of the row bounds (exact emulation of
// Gaussian, graded and decaying rows, K = 40 .. 2000; 2^-60 K with every digit at its
// largest), FP64 arithmetic up to 2^-53 K S and typically ~2^-54.5 sqrt(K) S where a
// few terms dominate.  P >= 2^-6 keeps the first an order of magnitude below the second.
// Gaussian rows, also ones that fall off by e^-0.05 per k, have P of 0.04 and more.  A
// tile with an element below (P > 0: an element whose products are all zero is exact) is
// not stored: gemm_f64's kernel, launched behind this one, computes the 64 x 64
// tiles that are not marked done.
// It also computes whatever a CTA left that gave up on a bounded wait, so these GEMMs
// always end in their result and record no error.
#include "f64_tc.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "ozaki_tc.cuh"
#include "tc_prims.cuh"

namespace gb {
namespace {

constexpr int S = F64_DIGITS, PL = F64_PLANES, GE = 6, GMAX = 8;
constexpr int BM = TC_BM, BN = 64, STAGES = 4, CW = BN / 4;
constexpr int THREADS = 32 * (2 + NUM_EPI_WARPS), MAX_REGS = 96;
constexpr uint32_t A_BYTES = PL * SL_TILE_BYTES, B_BYTES = PL * BN * SL_K * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t TABLE_BYTES = 20u * (BM + BN);
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_BYTES + TABLE_BYTES + 256 + 1024;
constexpr int SUPER = 64;   // stages (1024 k) an element's 64-bit sum covers: |sum| < 1024 * 1.01 * 2^52 < 2^63
constexpr int SMS = 152;    // GB300's, for estimates and splits (the launch asks the device)
constexpr int CH_MIN = 3;   // stages per chunk whatever the digits are: 5 * 2^16 * 48 < 2^24 - 2^16 units of group 6
constexpr float SIZE_MIN = 0x1p-6f;  // smallest sum of sizes of an element stored here
constexpr float LIM_TOP = 4194304.0f - 65536.0f, LIM = 16777216.0f - 65536.0f;

struct DArgs {
  SlicedDesc A, B;  // A: rows of the tile (M), B: columns (N)
  int M, N, K, batch;
  int m_off, n_off;  // the output indices of row / column 0 (panels)
  double* C;
  long long c_sb;
  Index2 c_r, c_c;
  int sym, pair_n;  // SYM_NONE, SYM_ROWCOL, SYM_TRIROW, SYM_TRICOL
  double alpha, beta;
  int times, plus;   // alpha is not 1, beta not 0 (FP64 comparisons cost what additions do)
  const double* C0;  // what beta multiplies (C itself where it is added in place)
  int nsplit, kbs;  // K splits and stages per split; partial sums go to part
  double* part;     // [split][batch][j][i]
  float* psize;     // the splits' sums of sizes, as part
  int* done;        // gemm_f64's tiles (GemmF64::done): splits stored, GRADED with an element too small
  int b_off, done_i, done_j;  // batch entry 0's; tiles of 64 over all rows / columns
  int swap;         // the rows are the GEMM's columns
  const int* nonfinite;
  unsigned int* counter;
  unsigned long long wait_ns;
  int withhold;  // test hook: the first CTA's producer never issues this stage (-1: every one is)
  int ntiles;
};

constexpr int GRADED = 1 << 20;

// gemm_f64's word of the 64 x 64 tile of rows from i, columns from j of batch entry b.
__device__ __forceinline__ int* done_word(const DArgs& a, int b, int i, int j) {
  const int ti = (a.m_off + i) / 64, tj = (a.n_off + j) / 64;
  const long long r = a.swap ? tj : ti, c = a.swap ? ti : tj;
  return a.done + ((a.b_off + b) * (long long)(a.swap ? a.done_j : a.done_i) + r) * (a.swap ? a.done_i : a.done_j) + c;
}

// Tile -> (split, batch, m0, n0); false for tiles a symmetric output does not
// need.  The dimension with fewer tiles runs fastest (CTAs that share a block of
// the other operand run together).
__device__ __forceinline__ bool decode(const DArgs& a, int t, int& sp, int& bz, int& m0, int& n0) {
  const int mt = (a.M + BM - 1) / BM, nt = (a.N + BN - 1) / BN;
  const int per = mt * nt;
  const int z = t / per, r = t % per;
  sp = z / a.batch;
  bz = z % a.batch;
  if (mt <= nt) {
    m0 = (r % mt) * BM;
    n0 = (r / mt) * BN;
  } else {
    n0 = (r % nt) * BN;
    m0 = (r / nt) * BM;
  }
  return !(a.sym == SYM_ROWCOL && n0 + BN - 1 < m0);
}

// Stages per chunk: see chunk_blocks in ozaki_tc.cu; here groups 2..6.
__device__ __forceinline__ int chunk_stages(const DArgs& a, int bz, int m0, int n0, int nkb) {
  if (nkb <= CH_MIN) return CH_MIN;
  float x[GE - 1], y[GE - 1];
  block_norms(a.A, bz, m0, x);
  block_norms(a.B, bz, n0, y);
  const float up = 2.002f;
  float most = LIM_TOP / fmaxf(up * x[0] * y[0], 1.0f);
#pragma unroll
  for (int g = 3; g <= GE; ++g) {
    float sum = 0.0f;
#pragma unroll
    for (int s = 1; s < g; ++s) sum = fmaf(x[s - 1], y[g - s - 1], sum);
    most = fminf(most, LIM / fmaxf(up * sum, 1.0f));
  }
  if (!(most >= 1.0f)) return CH_MIN;
  return most < (float)(SUPER / SL_KPC) ? SL_KPC * (int)most : SUPER;
}

// value * 2^scale (scale any sum of two row exponents)
__device__ __forceinline__ double scaled(double v, int scale) {
  const uint32_t h = (uint32_t)__double2hiint(v);
  const uint32_t e0 = ((h >> 20) & 0x7FFu) + (uint32_t)scale - 1u;
  if (e0 < 2046u && h != 0) return __hiloint2double((int)(h + ((uint32_t)scale << 20)), __double2loint(v));
  return v == 0.0 ? 0.0 : scalbn(v, scale);
}

// Element off of batch entry bz's finished result, with its mirror image.
__device__ __forceinline__ void put(const DArgs& a, int bz, long long off, long long moff, double v) {
  double* C = a.C + (long long)bz * a.c_sb;
  if (a.times) v *= a.alpha;
  if (a.plus) v = fma(a.beta, a.C0[(long long)bz * a.c_sb + off], v);
  C[off] = v;
  if (moff >= 0) C[moff] = v;
}

// One element's exact groups in units of group 6 (2^-52): carries of 512 units
// upwards, exact in FP32 while |u_3..6| < 2^24 - 2^16; the remainders of groups 6, 5
// and of 4, 3 are summed (below 2^18 units) and the three integers come from the
// magic number.
__device__ __forceinline__ long long exact_sum(float x2, float x3, float x4, float x5, float x6) {
  constexpr float U2 = 65536.0f, U3 = U2 * 512.0f, U4 = U3 * 512.0f, U5 = U4 * 512.0f, U6 = U5 * 512.0f;
  const float h6 = fmaf(x6, U6 / 512.0f, MAGIC) - MAGIC;
  float low = fmaf(h6, -1.0f / U5, x6);
  x5 = fmaf(h6, 1.0f / U5, x5);
  const float h5 = fmaf(x5, U5 / 512.0f, MAGIC) - MAGIC;
  low += fmaf(h5, -1.0f / U4, x5);
  x4 = fmaf(h5, 1.0f / U4, x4);
  const float h4 = fmaf(x4, U4 / 512.0f, MAGIC) - MAGIC;
  float mid = fmaf(h4, -1.0f / U3, x4);
  x3 = fmaf(h4, 1.0f / U3, x3);
  const float h3 = fmaf(x3, U3 / 512.0f, MAGIC) - MAGIC;
  mid += fmaf(h3, -1.0f / U2, x3);
  x2 = fmaf(h3, 1.0f / U2, x2);
  return (long long)magic_int(x2, U2) * (1ll << 36) + (long long)magic_int(mid, U4) * (1ll << 18) + magic_int(low, U6);
}

// R plus the FP32 group f (units of 2^-52; |f| < 2^20 of them).  Where R leaves room the
// result is in units of 2^-59, which keeps f's fraction: true then.
__device__ __forceinline__ bool add_rest(long long& R, float f) {
  const int m = magic_int(f, 0x1p52f);
  const int rest = magic_int(fmaf(f, 0x1p52f, -(float)m), 128.0f);
  R += m;
  const bool room = (unsigned long long)(R + (1ll << 55)) < (1ull << 56);
  if (room) R = R * 128 + rest;
  return room;
}

// R as a double in units of 2^-52.
__device__ __forceinline__ double from_units(long long R, bool fine) {
  const double d = __ll2double_rn(R);
  const int h = __double2hiint(d);
  return fine && h != 0 ? __hiloint2double(h - (7 << 20), __double2loint(d)) : d;
}

__global__ void __maxnreg__(MAX_REGS) f64_tc_kernel(const __grid_constant__ DArgs a) {
  chain_wait();
  extern __shared__ unsigned char smem_raw[];
  if (*a.nonfinite != 0) return;  // gemm_f64's kernel computes every tile
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  long long* e_roff = reinterpret_cast<long long*>(smem + STAGES * STAGE_BYTES);
  long long* e_mr = e_roff + BM;
  long long* e_coff = e_mr + BM;
  long long* e_mc = e_coff + BN;
  int* e_srow = reinterpret_cast<int*>(e_mc + BN);
  int* e_scol = e_srow + BM;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + TABLE_BYTES);
  // bars: full[5], empty[5], accfull, accempty, done, fempty, (slot, flag), ring full[4], ring empty[4], ring
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 15);
  constexpr int RING = 4;
  static_assert(2 * STAGES <= 10 && 24 * 8 + 2 * RING * 4 <= 256, "barrier block");
  volatile int* ring = reinterpret_cast<volatile int*>(bars + 24);
  volatile int* ringc = ring + RING;
  const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(bars);
  auto full_bar = [&](int st) { return bar0 + 8u * st; };
  auto empty_bar = [&](int st) { return bar0 + 8u * (STAGES + st); };
  const uint32_t accfull_bar = bar0 + 80, accempty_bar = bar0 + 88, done_bar = bar0 + 96, fempty_bar = bar0 + 104;
  auto ring_full = [&](int r) { return bar0 + 128u + 8u * r; };
  auto ring_empty = [&](int r) { return bar0 + 160u + 8u * r; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

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
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int nkb = (a.K + SL_K - 1) / SL_K;

  int gkb_issued = 0;
  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      int& gkb = gkb_issued;
      bool aborted = false;
      for (int i = 0; !aborted; ++i) {
        const int slot = i % RING;
        if (!mbar_wait(ring_empty(slot), (uint32_t)(((i / RING) & 1) ^ 1), abort_flag, a.wait_ns)) {
          *abort_flag = 1;
          break;
        }
        int t, sp = 0, bz = 0, m0 = 0, n0 = 0;
        for (;;) {
          const unsigned int u = atomicAdd(a.counter, 1u);
          t = u >= (unsigned int)a.ntiles ? -1 : (int)u;
          if (t < 0 || decode(a, t, sp, bz, m0, n0)) break;
        }
        const int kb0 = sp * a.kbs, kb1 = min(kb0 + a.kbs, nkb);
        ring[slot] = t;
        if (t >= 0) ringc[slot] = chunk_stages(a, bz, m0, n0, kb1 - kb0);
        mbar_arrive(ring_full(slot));
        if (t < 0) break;
        const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
        const unsigned char* ga = reinterpret_cast<const unsigned char*>(a.A.planes) + abz * a.A.batch_bytes() +
                                  (long long)(m0 / BM) * nkb * A_BYTES;
        const unsigned char* gbp = reinterpret_cast<const unsigned char*>(a.B.planes) + bbz * a.B.batch_bytes() +
                                   (long long)(n0 / SL_ROWS) * nkb * (PL * SL_TILE_BYTES) + ((n0 % SL_ROWS) / 8) * 128;
        for (int kb = kb0; kb < kb1; ++kb) {
          const int st = gkb % STAGES;
          if (!mbar_wait(empty_bar(st), (uint32_t)(((gkb / STAGES) & 1) ^ 1), abort_flag, a.wait_ns)) {
            *abort_flag = 1;
            aborted = true;
            break;
          }
          if (gkb == a.withhold && blockIdx.x == 0) {
            ++gkb;  // test hook: this stage never arrives
            continue;
          }
          mbar_expect_tx(full_bar(st), STAGE_BYTES);
          const uint32_t sa = sbase + st * STAGE_BYTES;
          bulk_load(sa, ga + (long long)kb * A_BYTES, A_BYTES, full_bar(st));
          const unsigned char* gblk = gbp + (long long)kb * (PL * SL_TILE_BYTES);
#pragma unroll
          for (int x = 0; x < 2 * PL; ++x)  // 64 rows of each plane of each k group
            bulk_load(sa + A_BYTES + x * (BN * 16), gblk + x * SL_SLICE_STEP, BN * 16, full_bar(st));
          ++gkb;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int gkb = 0, gch = 0, gsc = 0;  // stages, chunks, 64-bit sums so far
      bool aborted = false;
      for (int i = 0; !aborted; ++i) {
        const int slot = i % RING;
        if (!mbar_wait(ring_full(slot), (uint32_t)((i / RING) & 1), abort_flag, a.wait_ns)) {
          *abort_flag = 1;
          break;
        }
        const int t = ring[slot], ch = ringc[slot];
        mbar_arrive(ring_empty(slot));
        if (t < 0) break;
        int sp, bz, m0, n0;
        decode(a, t, sp, bz, m0, n0);
        const int kb0 = sp * a.kbs, kb1 = min(kb0 + a.kbs, nkb);
        auto drained = [&](uint32_t bar, int n) {
          if (!mbar_wait(bar, (uint32_t)((n - 1) & 1), abort_flag, a.wait_ns)) return false;
          tc_fence_after();
          return true;
        };
        int kc = 0, ks = 0;  // stage of the chunk, of the 64-bit sum
        for (int kb = kb0; kb < kb1; ++kb) {
          const int st = gkb % STAGES;
          bool ok = mbar_wait(full_bar(st), (uint32_t)((gkb / STAGES) & 1), abort_flag, a.wait_ns);
          if (ok) {
            tc_fence_after();
            const uint32_t sa = sbase + st * STAGE_BYTES;
            const uint64_t da = desc_tile(sa, PL * BM), db = desc_tile(sa + A_BYTES, PL * BN);
            if (kc > 0 || gch == 0) {
              issue_products<S, GE, GMAX, BN, 0, true>(tmem, da, db, 0, kc == 0, kc == 0);
            } else if (ks == 0) {
              // a sum's first stage: the exact groups are drained before the FP32 group
              ok = drained(accempty_bar, gch);
              if (ok) issue_products<S, GE, GMAX, BN, 2, true>(tmem, da, db, 0, true, false);
              ok = ok && drained(fempty_bar, gsc);
              if (ok) issue_products<S, GE, GMAX, BN, 1, true>(tmem, da, db, 0, false, true);
            } else {
              issue_products<S, GE, GMAX, BN, 1, true>(tmem, da, db, 0, false, false);
              ok = drained(accempty_bar, gch);
              if (ok) issue_products<S, GE, GMAX, BN, 2, true>(tmem, da, db, 0, true, false);
            }
            // the sizes, over the whole tile (read with its last FP32 group)
            if (ok)
              mma_bf16(tmem + GE * BN, da + (uint64_t)(S * (SL_SLICE_STEP >> 4)), db + (uint64_t)(S * BN), mma_idesc(BN),
                       kb > kb0);
          }
          if (!ok) {
            *abort_flag = 1;
            aborted = true;
            break;
          }
          mma_commit(empty_bar(st));
          ++gkb;
          ++kc;
          ++ks;
          const bool sum_end = ks == SUPER || kb == kb1 - 1;
          if (kc == ch || sum_end) {
            mma_commit(accfull_bar);
            ++gch;
            kc = 0;
          }
          if (sum_end) {
            ++gsc;
            ks = 0;
          }
        }
      }
      mma_commit(done_bar);
    }
  } else {
    // ---------------- epilogue ----------------
    const int q = warp & 3, cg = (warp - 2) >> 2, et = threadIdx.x - 64;
    const uint32_t lbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cg * CW);
    const int row = q * 32 + lane;
    int gch = 0;
    for (int i = 0;; ++i) {
      const int slot = i % RING;
      const bool got = mbar_wait(ring_full(slot), (uint32_t)((i / RING) & 1), abort_flag, a.wait_ns);
      if (!got) *abort_flag = 1;
      const int t = got ? ring[slot] : -1, ch = got ? (int)ringc[slot] : (int)CH_MIN;
      __syncwarp();
      if (lane == 0) mbar_arrive(ring_empty(slot));
      if (epi_barrier_any(!got || *abort_flag != 0)) break;
      if (t < 0) break;
      int sp, bz, m0, n0;
      decode(a, t, sp, bz, m0, n0);
      const int kb0 = sp * a.kbs, kb1 = min(kb0 + a.kbs, nkb);
      const bool parts = a.nsplit > 1;
      {
        const long long abz = a.A.batch == 1 ? 0 : bz, bbz = a.B.batch == 1 ? 0 : bz;
        if (et < BM) {
          const int li = m0 + et;
          const bool in = li < a.M;
          const long long gi = (long long)a.m_off + li;
          long long ro = li, mr = -1;
          if (in && !parts) {
            ro = a.c_r.at(gi);
            if (a.sym == SYM_ROWCOL) mr = a.c_c.at(gi);
            if (a.sym == SYM_TRIROW) {
              int mm, nn;
              tri_pair(gi, a.pair_n, mm, nn);
              ro = a.c_r.at((long long)mm * a.pair_n + nn);
              if (nn > mm) mr = a.c_r.at((long long)nn * a.pair_n + mm);
            }
          }
          e_roff[et] = ro;
          e_mr[et] = mr;
          e_srow[et] = in ? a.A.exps[abz * a.M + li] : 0;
        } else if (et < BM + BN) {
          const int c = et - BM, lj = n0 + c;
          const bool in = lj < a.N;
          const long long gj = (long long)a.n_off + lj;
          long long co = (long long)lj * a.M, mc = -1;
          if (in && !parts) {
            co = a.c_c.at(gj);
            if (a.sym == SYM_ROWCOL) mc = a.c_r.at(gj);
            if (a.sym == SYM_TRICOL) {
              int mm, nn;
              tri_pair(gj, a.pair_n, mm, nn);
              co = a.c_c.at((long long)mm * a.pair_n + nn);
              if (nn > mm) mc = a.c_c.at((long long)nn * a.pair_n + mm);
            }
          }
          e_coff[c] = co;
          e_mc[c] = mc;
          e_scol[c] = in ? a.B.exps[bbz * a.N + lj] : 0;
        }
      }
      epi_barrier_any(false);  // tables visible
      double acc[CW];
      long long R[CW];
      bool ok = true, graded = false, skip = false;
      for (int s0 = kb0; s0 < kb1 && ok; s0 += SUPER) {
        const int s1 = min(s0 + SUPER, kb1);
#pragma unroll
        for (int j = 0; j < CW; ++j) R[j] = 0;
        for (int c0 = s0; c0 < s1; c0 += ch) {
          const bool have = mbar_wait(accfull_bar, (uint32_t)(gch & 1), abort_flag, a.wait_ns);
          if (!__all_sync(0xffffffffu, have)) {
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < CW / 4; ++h) {
            uint32_t v[GE - 1][4];
#pragma unroll
            for (int g = 0; g < GE - 1; ++g) tmem_ld4_async(lbase + (uint32_t)(g * BN + h * 4), v[g]);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              R[h * 4 + j] += exact_sum(__uint_as_float(v[0][j]), __uint_as_float(v[1][j]), __uint_as_float(v[2][j]),
                                        __uint_as_float(v[3][j]), __uint_as_float(v[4][j]));
          }
          ++gch;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(accempty_bar);
        }
        if (!ok) break;
        // the FP32 group
        uint32_t fine = 0;  // elements in units of 2^-59
#pragma unroll
        for (int h = 0; h < CW / 4; ++h) {
          uint32_t f[4];
          tmem_ld4_async(lbase + (uint32_t)((GE - 1) * BN + h * 4), f);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 4; ++j) fine |= (uint32_t)add_rest(R[h * 4 + j], __uint_as_float(f[j])) << (h * 4 + j);
        }
        if (s1 == kb1) {
          // the tile's sums of sizes
          float* ps = nullptr;
          int pn = 0;  // columns to keep
          if (parts && m0 + row < a.M) {
            pn = a.N - n0 - cg * CW;
            ps = a.psize + (((long long)sp * a.batch + bz) * a.N + n0 + cg * CW) * a.M + m0 + row;
          }
#pragma unroll
          for (int h = 0; h < CW / 4; ++h) {
            uint32_t p[4];
            tmem_ld4_async(lbase + (uint32_t)(GE * BN + h * 4), p);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float v = __uint_as_float(p[j]);
              graded |= !parts && v > 0.0f && v < SIZE_MIN;
              if (h * 4 + j < pn) *ps = v;
              ps += a.M;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(fempty_bar);
        // a tile is stored by all warps or by none
        if (s1 == kb1) skip = epi_barrier_any(graded);
        // into FP64: one conversion an element (the FP64 pipe takes ~2 a clock and SM),
        // one addition more from the second 1024 k on
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const double d = from_units(R[j], (fine >> j) & 1u);
          if (s0 == kb0)
            acc[j] = d;
          else
            acc[j] += d;
        }
      }
      if (!ok) skip = epi_barrier_any(true);  // (the next tile's barrier ends the walk)
      if (skip) continue;
      if (et < 2 && m0 + 64 * et < a.M) {
        int* d = done_word(a, bz, m0 + 64 * et, n0);
        if (parts)
          atomicAdd(d, 1);
        else
          *d = 1;
      }
      const int gi = m0 + row;
      if (gi < a.M) {
        double* Cb = parts ? a.part + ((long long)sp * a.batch + bz) * (long long)a.M * a.N : nullptr;
        const long long ro = e_roff[row], mr = e_mr[row];
        const int srow = e_srow[row];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const int c = cg * CW + j, gj = n0 + c;
          if (gj < a.N) {
            const double v = scaled(acc[j], srow + e_scol[c] - 52);
            const long long co = e_coff[c];
            if (parts) {
              Cb[ro + co] = v;
            } else if (a.sym == SYM_ROWCOL) {
              if (gj >= gi) put(a, bz, ro + co, gj > gi ? mr + e_mc[c] : -1, v);
            } else if (a.sym == SYM_TRIROW) {
              put(a, bz, ro + co, mr >= 0 ? mr + co : -1, v);
            } else if (a.sym == SYM_TRICOL) {
              const long long mc = e_mc[c];
              put(a, bz, ro + co, mc >= 0 ? ro + mc : -1, v);
            } else {
              put(a, bz, ro + co, -1, v);
            }
          }
          asm volatile("" ::: "memory");
        }
      }
    }
  }

  __syncthreads();
  if (warp == 0 && lane == 0 && *abort_flag) {
    for (int k = gkb_issued > STAGES ? gkb_issued - STAGES : 0; k < gkb_issued; ++k)
      mbar_wait(full_bar(k % STAGES), (uint32_t)((k / STAGES) & 1), nullptr, a.wait_ns);
  }
  if (warp == 1) {
    if (*abort_flag) mbar_wait(done_bar, 0, nullptr, a.wait_ns);
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Partial sums of the K splits, in order, into the output, where every split has stored
// its tile.  An element whose sum of sizes is too small leaves the tile to gemm_f64's
// kernel, which writes all of it again.
__global__ void __launch_bounds__(256) sum_parts_kernel(const __grid_constant__ DArgs a) {
  chain_wait();
  const long long MN = (long long)a.M * a.N, all = MN * a.batch;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  if (idx >= all) return;
  const int bz = (int)(idx / MN);
  const long long r = idx % MN;
  const int i = (int)(r % a.M), j = (int)(r / a.M);
  if (a.sym == SYM_ROWCOL && j < i) return;
  int* done = done_word(a, bz, i, j);
  if ((*(volatile int*)done & (GRADED - 1)) != a.nsplit) return;
  double v = 0.0;
  float p = 0.0f;
  for (int s = 0; s < a.nsplit; ++s) {
    v += a.part[s * all + idx];
    p += a.psize[s * all + idx];
  }
  if (p > 0.0f && p < SIZE_MIN) atomicOr(done, GRADED);
  const long long gi = (long long)a.m_off + i, gj = (long long)a.n_off + j;
  long long off, moff = -1;
  int mm, nn;
  if (a.sym == SYM_TRIROW) {
    tri_pair(gi, a.pair_n, mm, nn);
    off = a.c_r.at((long long)mm * a.pair_n + nn) + a.c_c.at(gj);
    if (nn > mm) moff = a.c_r.at((long long)nn * a.pair_n + mm) + a.c_c.at(gj);
  } else if (a.sym == SYM_TRICOL) {
    tri_pair(gj, a.pair_n, mm, nn);
    off = a.c_r.at(gi) + a.c_c.at((long long)mm * a.pair_n + nn);
    if (nn > mm) moff = a.c_r.at(gi) + a.c_c.at((long long)nn * a.pair_n + mm);
  } else {
    off = a.c_r.at(gi) + a.c_c.at(gj);
    if (a.sym == SYM_ROWCOL && j > i) moff = a.c_r.at(gj) + a.c_c.at(gi);
  }
  put(a, bz, off, moff, v);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Slices held at a time, where an operand is cut into panels (3 GB; less by the test hook).
constexpr size_t PANEL_BYTES = (size_t)3 << 30;
std::atomic<size_t> g_panel_bytes{PANEL_BYTES};
thread_local bool t_query_minimum = false;  // this thread's queries leave the scratch out

long long up128(long long x) { return (x + 127) / 128 * 128; }
size_t slice_bytes(long long batch, long long rows, long long K) {
  return align256(sliced_plane_bytes((int)batch, (int)rows, (int)K, SPLIT_F64)) +
         align256(sliced_meta_ints((int)batch, (int)rows) * sizeof(int));
}

// How a GEMM is run: X is the operand on the tile rows, Y on its columns.
struct Plan {
  bool use = false;
  bool swap = false;         // X is B
  bool tri = false;          // the pair operand (B) is packed to its upper triangle
  long long xr = 0, yr = 0;  // rows of X and Y
  int pb = 1;                // batch entries per panel
  long long px = 0, py = 0;  // rows of X, Y per panel
  int nsplit = 1, kbs = 0;   // K splits per panel, stages each
  size_t xb = 0, yb = 0, partb = 0, doneb = 0;
  size_t bytes() const { return doneb + xb + yb + partb; }
};

// Words in front of the done tiles: [0] non-finite operand, [1] tile counter.
constexpr size_t WORDS = 2;
size_t done_words(long long M, long long N, int batch) { return (size_t)((M + 63) / 64 * ((N + 63) / 64) * batch); }

// The two kernels' estimated times, from these measured on GB300 (whole calls, each
// GEMM forced one way, us FP64 units / us tensor cores): Fock matrices of nbf5, nbf
// (two GEMMs) 20, 80 39/90; 20, 160 268/129; 40, 110 286/97; 60, 60 74/107; 60, 90
// 151/115; 150, 150 2650/368; four-index J, K of nbf 24 134/170; 30 209/183; 53 917/293;
// FP64 Lagrangian of nbf 24 151/182; 32 238/184; 60 969/244; rotation of nbf 300
// 492/773; 371 877/818; 450 1785/964.
//
// gemm_f64: 64 x 64 tiles at ~1.0 TFLOP/s in whole rounds of the SMs, or 8 x 8 blocks at
// 0.8, at least 0.115 us per k (one warp's chain); of the skipped blocks of a square grid
// half are paid for.
double time_f64(long long M, long long N, long long K, int batch, int sym) {
  auto up = [](long long x, long long to) { return (double)((x + to - 1) / to * to); };
  const double t64 = up(M, 64) / 64 * up(N, 64) / 64 * batch;
  const double half = sym == SYM_NONE ? 1.0 : 0.5;
  if (t64 >= SMS) return std::ceil(t64 * half / SMS) * SMS * 8192.0 * up(K, 16) / 1.0e12;
  const double part = sym == SYM_PAIRCOL ? 0.75 : half;
  return 4e-6 + std::max(0.115e-6 * K, 2.0 * up(M, 8) * up(N, 8) * K * batch * part / 0.8e12);
}

// The tensor cores: seven launches, 32 bytes of slicing an element, and a stage of a
// tile 1.1 (long K) to 1.5 us with ~7 us a tile, in whole rounds of the SMs.
double time_tc(double tiles, long long nkb, double el, bool in_place) {
  const double fixed = 50e-6 + el * 32.0 / 3.5e12, stage = 1.4e-6, tile = 7e-6;
  if (tiles >= SMS) return fixed + std::ceil(tiles / SMS) * (nkb * stage + tile);
  const double ctas = in_place ? tiles : std::min((double)SMS, tiles * (double)std::max(1ll, nkb / 16));
  return fixed + tiles * nkb * stage / ctas + tile + (ctas > tiles ? 5e-6 : 0.0);
}

Plan make_plan(long long M, long long N, long long K, int batch, bool a_shared, bool b_shared, int sym, int pair_n,
               bool in_place) {
  Plan p;
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return p;
  p.tri = sym == SYM_PAIRCOL;
  const long long n = p.tri ? (long long)pair_n * (pair_n + 1) / 2 : N;
  // orientation: less padding of the 128 x 64 tiles
  auto tiles = [](long long x, long long y) { return ((x + BM - 1) / BM) * ((y + BN - 1) / BN); };
  p.swap = tiles(n, M) < tiles(M, n);
  p.xr = p.swap ? n : M;
  p.yr = p.swap ? M : n;
  const bool xs = batch == 1 || (p.swap ? b_shared : a_shared), ys = batch == 1 || (p.swap ? a_shared : b_shared);
  const long long nkb = (K + SL_K - 1) / SL_K;
  if (p.xr > (1 << 30) || p.yr > (1 << 30) || K > (1 << 30)) return p;
  const double all_tiles = (double)tiles(p.xr, p.yr) * batch * (sym == SYM_ROWCOL ? 0.55 : 1.0);
  const double el = ((double)M * (a_shared ? 1 : batch) + (double)n * (b_shared ? 1 : batch)) * (double)(nkb * SL_K);
  // (0.7: graded rows pay for both)
  p.use = time_tc(all_tiles, nkb, el, in_place) < 0.7 * time_f64(M, N, K, batch, sym);
  if (!p.use) return p;
  // panels: over the batch, or over the rows of the operand with more of them
  p.px = p.xr;
  p.py = p.yr;
  p.pb = batch;
  auto size = [&]() {
    p.xb = slice_bytes(xs ? 1 : p.pb, p.px, K);
    p.yb = slice_bytes(ys ? 1 : p.pb, p.py, K);
  };
  size();
  const size_t most = g_panel_bytes.load();
  if (p.xb + p.yb > most) {
    if (batch > 1) {
      while (p.pb > 1 && p.xb + p.yb > most) {
        p.pb = (p.pb + 1) / 2;
        size();
      }
    } else {
      long long& big = p.px >= p.py ? p.px : p.py;
      while (big > 128 && p.xb + p.yb > most) {
        big = up128((big + 1) / 2);
        size();
      }
    }
  }
  // the symmetric tiles of a panel would need its offsets
  if (sym == SYM_ROWCOL && (p.px < p.xr || p.py < p.yr)) {
    p.use = false;
    return p;
  }
  // K splits of at least 16 stages, whole norm runs: the split count whose tiles
  // take the fewest stages in a row on the SMs (a tile more costs an SM its
  // epilogue, ~12 stages' time)
  const long long pt = tiles(p.px, p.py) * p.pb;
  long long kbs = nkb;
  double best = 1e300;
  // (none where the output is added to in place: no element of a tile is stored before
  // all are known to be kept, which sum_parts_kernel does not see)
  for (long long ns = 1; ns <= (in_place ? 1 : 64) && (ns == 1 || nkb / ns >= 16) && (ns == 1 || pt * ns <= SMS * 8); ++ns) {
    long long k = (nkb + ns - 1) / ns;
    if (ns > 1) k = (k + SL_KPC - 1) / SL_KPC * SL_KPC;
    const double cost = (double)((pt * ((nkb + k - 1) / k) + SMS - 1) / SMS) * (double)(k + 12);
    if (cost < best) {
      best = cost;
      kbs = k;
    }
  }
  p.kbs = (int)kbs;
  p.nsplit = (int)((nkb + kbs - 1) / kbs);
  const size_t parts = p.nsplit > 1 ? (size_t)p.nsplit * p.pb * p.px * p.py : 0;
  p.partb = align256(sizeof(double) * parts) + align256(sizeof(float) * parts);
  p.doneb = align256(sizeof(int) * (WORDS + done_words(M, n, batch)));
  return p;
}

// Once per device context; *sms: the device's SMs.
int configure(int* sms) {
  static std::mutex mu;
  static unsigned long long done[64] = {0};
  static int count[64] = {0};
  int dev = 0;
  GB_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
  const unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64) return GB_OK;
  if (ctx != 0 && done[dev] == ctx) {
    *sms = count[dev];
    return GB_OK;
  }
  GB_TRY(cuda_status(
      cudaFuncSetAttribute(f64_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES),
      "f64_tc: cudaFuncSetAttribute"));
  GB_TRY(cuda_status(cudaDeviceGetAttribute(&count[dev], cudaDevAttrMultiProcessorCount, dev),
                     "cudaDeviceGetAttribute"));
  *sms = count[dev];
  done[dev] = current_context_id();
  return GB_OK;
}

bool same_index(const Index2& a, const Index2& b) { return a.div == b.div && a.s1 == b.s1 && a.s0 == b.s0; }

}  // namespace

size_t gemm_f64_tc_bytes(long long M, long long N, long long K, int batch, bool a_shared, bool b_shared, int sym,
                         int pair_n, bool in_place) {
  if (t_query_minimum) return 0;
  const Plan p = make_plan(M, N, K, batch, a_shared, b_shared, sym, pair_n, in_place);
  return p.use ? p.bytes() : 0;
}

int gemm_f64_tc(const GemmF64& g, const TcWork& w, cudaStream_t s) {
  const bool a_shared = g.batch == 1 || g.A.sb == 0, b_shared = g.batch == 1 || g.B.sb == 0;
  const double* C0 = g.C0 ? g.C0 : g.C.p;
  const Plan p = make_plan(g.M, g.N, g.K, g.batch, a_shared, b_shared, g.sym, g.pair_n,
                           g.beta != 0.0 && C0 == g.C.p);
  if (!p.use || !w.p || w.bytes < p.bytes()) return gemm_f64(g, s);
  int sms = SMS;
  GB_TRY(configure(&sms));
  Carve cv(w.p, w.bytes);
  const long long n = p.tri ? (long long)g.pair_n * (g.pair_n + 1) / 2 : g.N;
  const size_t nwords = WORDS + done_words(g.M, n, g.batch);
  int* words = cv.take<int>(nwords);
  auto sliced = [&](long long batch, long long rows) { return take_sliced(cv, (int)batch, (int)rows, g.K, SPLIT_F64); };
  const bool xs = p.swap ? b_shared : a_shared, ys = p.swap ? a_shared : b_shared;
  // the sources: A's rows are the M index, B's the N index
  const SliceSrc sa{g.A.p, g.A.sb, g.A.r, g.A.c, g.a_kfast};
  SliceSrc sb{g.B.p, g.B.sb, g.B.c, g.B.r, g.b_kfast};
  if (p.tri) sb.tri_n = g.pair_n;
  const bool one = !p.tri && g.M == g.N && g.A.p == g.B.p && g.A.sb == g.B.sb && same_index(g.A.r, g.B.c) &&
                   same_index(g.A.c, g.B.r) && p.px == p.xr && p.py == p.yr;
  SlicedDesc X = sliced(xs ? 1 : p.pb, p.px), Y = one ? X : sliced(ys ? 1 : p.pb, p.py);
  const size_t parts = p.nsplit > 1 ? (size_t)p.nsplit * p.pb * p.px * p.py : 0;
  double* part = parts ? cv.take<double>(parts) : nullptr;
  float* psize = parts ? cv.take<float>(parts) : nullptr;
  GB_TRY(cuda_status(cudaMemsetAsync(words, 0, nwords * sizeof(int), s), "f64_tc: words"));
  bool first = true;
  for (int b0 = 0; b0 < g.batch; b0 += p.pb) {
    const int nb = std::min(p.pb, g.batch - b0);
    for (long long x0 = 0; x0 < p.xr; x0 += p.px) {
      for (long long y0 = 0; y0 < p.yr; y0 += p.py) {
        const int xn = (int)std::min(p.px, p.xr - x0), yn = (int)std::min(p.py, p.yr - y0);
        auto cut = [&](SlicedDesc d, SliceSrc src, bool shared, long long r0, int rows, SlicedDesc& out, bool fresh) -> int {
          d.rows = rows;
          d.batch = shared ? 1 : nb;
          d.norms = d.exps + (size_t)d.batch * rows;
          out = d;
          if (!fresh) return GB_OK;
          src.row0 = r0;
          if (!shared) src.p += (long long)b0 * src.sb;
          return slice_operand(src, d, s, false, words);
        };
        // an operand that this panel shares with the one before is there already
        SlicedDesc x, y;
        const bool fx = first || !xs || p.px < p.xr, fy = first || !ys || p.py < p.yr;
        GB_TRY(cut(X, p.swap ? sb : sa, xs, x0, xn, x, fx));
        if (one)
          y = x;
        else
          GB_TRY(cut(Y, p.swap ? sa : sb, ys, y0, yn, y, fy));
        if (!first) GB_TRY(cuda_status(cudaMemsetAsync(words + 1, 0, sizeof(int), s), "f64_tc: tile counter"));
        first = false;
        DArgs a{};
        a.A = x;
        a.B = y;
        a.M = xn;
        a.N = yn;
        a.K = g.K;
        a.batch = nb;
        a.m_off = (int)x0;
        a.n_off = (int)y0;
        a.C = g.C.p + (long long)b0 * g.C.sb;
        a.c_sb = g.C.sb;
        a.c_r = p.swap ? g.C.c : g.C.r;
        a.c_c = p.swap ? g.C.r : g.C.c;
        a.sym = p.tri ? (p.swap ? SYM_TRIROW : SYM_TRICOL) : g.sym;
        a.pair_n = g.pair_n;
        a.alpha = g.alpha;
        a.beta = g.beta;
        a.times = g.alpha != 1.0;
        a.plus = g.beta != 0.0;
        a.C0 = C0 + (long long)b0 * g.C.sb;
        a.nsplit = p.nsplit;
        a.kbs = p.kbs;
        a.part = part;
        a.psize = psize;
        a.done = words + WORDS;
        a.b_off = b0;
        a.done_i = (int)((p.xr + 63) / 64);
        a.done_j = (int)((p.yr + 63) / 64);
        a.swap = p.swap;
        a.nonfinite = words;
        a.counter = reinterpret_cast<unsigned int*>(words + 1);
        a.wait_ns = wait_limit_ns();
        a.withhold = withheld_stage();
        a.ntiles = (int)(((xn + BM - 1) / BM) * (long long)((yn + BN - 1) / BN) * nb * p.nsplit);
        const unsigned grid = (unsigned)std::min(a.ntiles, sms);
        GB_LAUNCH_CHAIN(g.tag, s, f64_tc_kernel, dim3(grid), dim3(THREADS), SMEM_BYTES, a);
        if (p.nsplit > 1) {
          const long long all = (long long)xn * yn * nb;
          GB_LAUNCH_CHAIN("f64_tc:sum_parts", s, sum_parts_kernel, dim3((unsigned)((all + 255) / 256)), dim3(256), 0,
                          a);
        }
      }
    }
  }
  // FP64 arithmetic for the tiles that are not done: graded rows, and every tile where
  // an operand holds a NaN or an infinity
  GemmF64 f = g;
  f.done = words + WORDS;
  f.done_value = p.nsplit;
  if (p.tri) {
    f.sym = SYM_TRICOL;
    f.N = (int)n;
  }
  return gemm_f64(f, s);
}

}  // namespace gb

extern "C" int gb_query_minimum(int on) {
  gb::clear_error();
  gb::t_query_minimum = on != 0;
  return GB_OK;
}

extern "C" int gb_test_panel_bytes(size_t bytes) {
  gb::clear_error();
  gb::g_panel_bytes.store(bytes ? bytes : gb::PANEL_BYTES);
  return GB_OK;
}
