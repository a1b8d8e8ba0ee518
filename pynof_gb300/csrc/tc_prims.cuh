// Device-side building blocks of the tcgen05 kernels: barriers with bounded
// waits, bulk copies, descriptors, MMAs, TMEM loads and the issue of one stage's
// digit products.  Included by the kernels' translation units.
#pragma once

#include <cuda_bf16.h>

#include "slice.cuh"

namespace gb {
namespace {

constexpr int NUM_EPI_WARPS = 16;
constexpr int TC_BM = 128;  // tile rows (M of every MMA)

constexpr float MAGIC = 12582912.0f;                          // 1.5 * 2^23
constexpr int MAGIC_BITS = 0x4B400000;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// A waiting thread may sleep this long per try: 17 warps that poll take issue
// slots and shared-memory cycles from the MMA warp.
constexpr uint32_t WAIT_HINT_NS = 20000;

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity), "r"(WAIT_HINT_NS)
      : "memory");
  return done != 0;
}

// Bounded wait: false after limit_ns, or (if abort_flag != nullptr) as soon
// as another role has aborted.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned long long limit_ns) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if (abort_flag && *abort_flag) return false;
    if ((it & 63) == 0 && now_ns() - t0 > limit_ns) return false;
  }
}

// Named barrier of the 16 epilogue warps with an OR reduction: every one of
// them gets the same answer, so their control flow cannot diverge.
__device__ __forceinline__ bool epi_barrier_any(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred pin, pout;\n setp.ne.u32 pin, %1, 0;\n"
      " bar.red.or.pred pout, 1, %2, pin;\n selp.u32 %0, 1, 0, pout;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)pred), "n"(NUM_EPI_WARPS * 32)
      : "memory");
  return r != 0;
}

// Contiguous global -> shared bulk copy completing on an mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// UMMA shared-memory descriptor of the first slice of a stage's operand, whose
// k groups hold `rows` rows in all (S slices one after another): K-major, no
// swizzle; core matrices (8 rows x 16 B) rows*16 B apart along K (leading byte
// offset) and 128 B apart along the rows (stride byte offset).
__device__ __forceinline__ uint64_t desc_tile(uint32_t saddr, uint32_t rows) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((rows * 16u) >> 4) << 16;  // leading byte offset
  d |= (uint64_t)(128u >> 4) << 32;          // stride byte offset
  d |= (uint64_t)1 << 46;                    // descriptor version
  return d;                                  // layout type 0: no swizzle
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 8 consecutive TMEM columns of this warp's 32 lanes; complete after tmem_wait_ld().
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4_async(uint32_t taddr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Exact integer of an FP32 value x * 2^k with |x * 2^k| < 2^22 (rounded to
// nearest even otherwise): adding 1.5 * 2^23 leaves the integer in the low
// mantissa bits.  Pure FP32/ALU work, no float->int conversion unit.
__device__ __forceinline__ int magic_int(float x, float scale) {
  return __float_as_int(fmaf(x, scale, MAGIC)) - MAGIC_BITS;
}

// Exponent of group g's unit 2^-(e_s + e_t), s + t = g.
__host__ __device__ constexpr int group_exp(int W, int g) { return W == 9 ? 9 * g - 2 : W * g; }

// bf16 MMA with an A-collector qualifier: COLL 0 none, 1 fill (read A from
// shared memory and keep it in the tensor core's collector), 2 use (take A
// from the collector), 3 lastuse (take it and release the collector).
template <int COLL>
__device__ __forceinline__ void mma_bf16_c(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  if constexpr (COLL == 0)
    mma_bf16(d_tmem, a, b, idesc, accumulate);
  else if constexpr (COLL == 1)
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
  else if constexpr (COLL == 2)
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16.collector::a::use [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// Instruction descriptor of a bf16 MMA: f32 accumulate, both operands K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t mma_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// Products of one stage (S digit slices; product (s, t) of A slice s and B
// slice t goes to group g = s + t, kept only for g <= GMAX), fully unrolled
// and ordered by A slice: the products of one A slice run back to back and
// take A from the collector after the first, so each A slice tile is read
// from shared memory once per stage (5 reads instead of 15 for five slices; B
// is read per product).  The slices' descriptors differ from the stage's first
// ones only in the start-address field.
//   SEL 0: every product; 1: the FP32 group only (g > GE); 2: the exact
//   groups only (g <= GE, accumulator columns (g - 2) BN).
//   WIDE: consecutive B slices whose groups' accumulators are consecutive (g,
//   g + 1, .. <= GE + 1) go into one MMA of up to 256 columns (11 MMAs instead of
//   15 for five slices at BN = 128); otherwise one MMA per product, as wide as idesc says.
//   restart_exact: the exact groups start from zero (their first product,
//   s = 1, overwrites); restart_f: the FP32 group (at (GE - 1) BN) starts from zero
//   (equal to restart_exact when SEL == 0).
template <int S, int GE, int GMAX, int BN, int SEL, bool WIDE>
__device__ __forceinline__ void issue_products(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc,
                                               bool restart_exact, bool restart_f) {
  bool f_first = true;
#pragma unroll
  for (int s = 1; s <= S; ++s) {
    const uint64_t das = da + (uint64_t)((s - 1) * (SL_SLICE_STEP >> 4));
    // this slice's products under SEL: t in [t0, t1]
    const int t0 = SEL == 1 ? (GE + 1 - s > 1 ? GE + 1 - s : 1) : 1;
    const int tm = GMAX - s < S ? GMAX - s : S;
    const int t1 = SEL == 2 && GE - s < tm ? GE - s : tm;
    int t = t0;
#pragma unroll
    for (int it = 0; it < S; ++it) {
      if (t > t1) break;
      const int gg = s + t;
      const bool exact = gg <= GE;
      int w = 1;  // products in this MMA
      if (WIDE && exact) {
        w = 256 / BN;
        w = w < t1 - t + 1 ? w : t1 - t + 1;
        w = w < GE + 2 - gg ? w : GE + 2 - gg;
      }
      const uint32_t d = tmem + (uint32_t)((exact ? gg - 2 : GE - 1) * BN);
      const uint64_t dbt = db + (uint64_t)((t - 1) * BN);
      const uint32_t id = WIDE ? mma_idesc(w * BN) : idesc;
      bool acc;
      if (exact) {
        acc = !(restart_exact && s == 1);
      } else {
        acc = !(restart_f && f_first);
      }
      if (gg + w - 1 > GE) f_first = false;
      const bool head = t == t0, tail = t + w > t1;
      if (head && tail)
        mma_bf16_c<0>(d, das, dbt, id, acc);
      else if (head)
        mma_bf16_c<1>(d, das, dbt, id, acc);
      else if (tail)
        mma_bf16_c<3>(d, das, dbt, id, acc);
      else
        mma_bf16_c<2>(d, das, dbt, id, acc);
      t += w;
    }
  }
}

}  // namespace
}  // namespace gb
