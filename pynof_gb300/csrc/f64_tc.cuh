// FP64 GEMMs on the tcgen05 tensor cores, as accurate as FP64 arithmetic element by
// element.
//
// The operands are cut into seven nine-bit digit planes (62 bits below each
// row's power-of-two bound, slice.cuh); the products of digits s and t with
// s + t <= 8 (28 of them) run as bf16 MMAs.  Groups s + t = 2..6 accumulate exactly,
// groups 7 and 8 in FP32, the rest is dropped.  An element's sum is carried as a
// 64-bit integer over at most 1024 k and those parts are added in FP64, so it is
// rounded K / 1024 times where FP64 arithmetic rounds K times.
//
// What is dropped is small against the product of the two row bounds, not against
// the element's own terms, which are far below it where rows are graded against one
// another (A's columns scaled by d_k, B's rows by 1 / d_k).  So one more MMA product
// sums the terms' sizes, and the 64 x 64 tiles with an element whose sum is too small
// (the rule and its figures: f64_tc.cu) are left to gemm_f64's kernel, launched behind
// the tensor cores' and skipping the tiles that are done.  The same kernel computes
// everything where an operand holds a NaN or an infinity, which digits cannot.
//
// Error over 2^-53 sum |a b| at K = 400, largest of 7500 elements: 0.2 on Gaussian
// rows (FP64 arithmetic 3.1), 0.5 on rows that fall off by e^-0.05 per k (14.9), 0.9
// by e^-0.2 per k (18.8), 1.1 on rows whose bounds come from elements that do not meet
// (6.0).
//
// GB300's FP64 pipe gives ~1.1 TFLOP/s to gemm_f64; the same GEMMs run at 30 to 40
// TFLOP/s here, less the slicing of the operands (32 bytes of traffic per
// element).
#pragma once

#include "gemm_f64.cuh"

namespace gb {

// Workspace of the slices and partial sums; null or too small: gemm_f64 runs.
struct TcWork {
  void* p = nullptr;
  size_t bytes = 0;
};

// What a workspace holds behind the buffers already carved.
inline TcWork tc_work(const Carve& c) {
  return c.used < c.cap ? TcWork{c.base + c.used, c.cap - c.used} : TcWork{};
}

// Bytes gemm_f64_tc takes for a GEMM of these sizes (0: it runs on gemm_f64).
// a_shared / b_shared: the operand's batch stride is 0; in_place: beta is not 0 and
// multiplies C itself.  sym: SYM_PAIRCOL counts the N = pair_n^2 columns.
size_t gemm_f64_tc_bytes(long long M, long long N, long long K, int batch, bool a_shared, bool b_shared,
                         int sym = SYM_NONE, int pair_n = 0, bool in_place = false);

// gemm_f64 with the tensor cores where they are faster.
int gemm_f64_tc(const GemmF64& g, const TcWork& w, cudaStream_t stream);

}  // namespace gb
