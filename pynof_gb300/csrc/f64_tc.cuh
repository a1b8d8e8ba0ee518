// FP64 GEMMs on the tcgen05 tensor cores, as accurate as FP64 arithmetic.
//
// The operands are cut into seven nine-bit digit planes (62 bits below each
// row's power-of-two bound, slice.cuh); the products of digits s and t with
// s + t <= 8 (28 of them) run as bf16 MMAs.  Groups s + t = 2..6 (down to 2^-52 of
// the leading ones) accumulate exactly, groups 7 and 8 in FP32 (below 2^-61
// relative error), the rest is below 2^-63.  An element's sum is carried as a
// 64-bit integer over at most 1024 k and those parts are added in FP64, so it is
// rounded K / 1024 times where FP64 arithmetic rounds K times.
//
// GB300's FP64 pipe gives ~1.1 TFLOP/s to gemm_f64; the same GEMMs run at 30 to 40
// TFLOP/s here, less the slicing of the operands (30 bytes of traffic per
// element).
//
// What FP64 arithmetic does and digits cannot: NaN and infinity.  The slicer
// notes them in a device word of the workspace; the tensor-core kernel then
// does nothing and gemm_f64's kernel, launched behind it, runs instead.
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
// a_shared / b_shared: the operand's batch stride is 0; same: A and B^T are one
// operand.  sym: SYM_PAIRCOL counts the N = pair_n^2 columns.
size_t gemm_f64_tc_bytes(long long M, long long N, long long K, int batch, bool a_shared, bool b_shared,
                         int sym = SYM_NONE, int pair_n = 0);

// gemm_f64 with the tensor cores where they are faster.
int gemm_f64_tc(const GemmF64& g, const TcWork& w, cudaStream_t stream);

}  // namespace gb
