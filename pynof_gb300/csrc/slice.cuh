// Digit slicing of FP64 operands for the split-product tensor-core path.
//
// A row x[0..K) of an FP64 operand is written as
//     x[k] = 2^E * sum_{s=1..S} d_s[k] 2^-e_s   (+ rounding error <= 2^(E - 1 - e_S))
// with E the row's power-of-two exponent (|x[k]| < 2^E for the whole row) and
// d_s balanced digits of W bits: W = 9, |d_s| <= 256, e_s = 9 s - 1 for the
// six-digit code, W = 7, |d_1| <= 128, |d_s| <= 64, e_s = 7 s for the codes
// below it.  Nine bits is what bf16 holds of a signed integer (every integer up
// to 256 is exact), so each digit is stored pre-weighted as the bf16 value
// d_s 2^-e_s.  Products of two slices then carry their positional weight, and a
// sum of slice products over a K-chunk is an integer multiple of 2^-(e_s + e_t),
// the same for equal s + t = g, that FP32 holds exactly while it stays within
// 2^24 units -- the property the tensor-core kernel relies on.  How long such a
// chunk of nine-bit digits may be depends on their sizes, so the slicer also
// records a bound of them per 128-row block (norms below).
//
// The digits are computed from the FP64 bit pattern with integer arithmetic
// only (GB300's FP64 ALU rate is ~1/64 of FP32).
//
// Memory layout ("blocked"): the slices are stored in exactly the order the
// tensor-core kernel's shared memory wants them, so that one pipeline stage of
// one operand is a single contiguous bulk copy.  Rows are cut into blocks of
// 128 and K into blocks of 16; block (rb, kb) holds the S slices of 128 x 16
// bf16 (4 KB each) as 8 x 8 "core matrices" (8 rows of 16 bytes), k group
// major, then slice, then row group:
//   byte(s, r, k) = (((k / 8) * S + s) * 16 + r / 8) * 128 + (r % 8) * 16 + (k % 8) * 2.
// The rows of consecutive slices thus follow each other inside a k group, and
// one MMA can take several slices of B as one wider operand.
// Blocks are ordered [batch][rb][kb].  Rows and K are zero-padded to whole
// blocks.  Exponents: exps[b][r] (int32).
//
// Norms: norms[b][rb][s - 1], s <= 3 (five digits) or 5 (seven), is the FP32 bit
// pattern of an upper bound of sum d_s^2 over one k group parity (8 of every 16 k)
// of any run of 128 k of any row of the block; a run's sum of products of two
// digits is then at most 2 sqrt(norm_a norm_b) (Cauchy-Schwarz).
//
// Size plane (the eighth plane of SPLIT_F64): |d_1| 2^-e_1, or 2^-30 where d_1 is zero
// and the element is not, 0 for a zero.  A sum of products of two size planes is zero
// only where every product of the elements is, and otherwise sum |a b| over the
// two row bounds, to the accuracy of the leading digits (below four times it).
//
// TF32x3 form (split code SPLIT_TF32X3): two planes, hi = tf32(x 2^-E) and
// lo = tf32(x 2^-E - hi) (each rounded to nearest even, 11 significant bits,
// FP32 exponent), for the classic three-product TF32 split (hi hi + hi lo +
// lo hi with FP32 accumulation).  A block is then 128 rows x 8 k of 32-bit
// elements, the same 4 KB tiles and core-matrix order with 4 elements per
// 16-byte core-matrix row:
//   byte(s, r, k) = (((k / 4) * 2 + s) * 16 + r / 8) * 128 + (r % 8) * 16 + (k % 4) * 4.
#pragma once

#include <cuda_bf16.h>

#include "gemm_f64.cuh"

namespace gb {

constexpr int SL_ROWS = 128;               // rows per block
constexpr int SL_K = 16;                   // K per block
constexpr int SL_TILE_BYTES = SL_ROWS * SL_K * 2;  // one slice of one block: 4 KB

constexpr int SL_SLICE_STEP = SL_ROWS * 16;  // from one slice of a k group to the next
constexpr int SL_KPC = 8;                  // k blocks per slicer CTA, and per run of the norms
constexpr int SL_NORMS = 5;                // digits whose norms are recorded (three of five, five of seven)

// Split codes ("nslices" in the C ABI): 1..5 seven-bit digit slices, 6 (42 bits,
// 21 products of s + t <= 7 if they were seven-bit ones) is five nine-bit slices
// (45 bits, 15 products of s + t <= 6), or the TF32x3 split.
// SPLIT_F64 (inside the library only): seven nine-bit slices, 62 bits, and the size
// plane, for products that are as accurate as FP64 arithmetic (f64_tc.cuh).
constexpr int SPLIT_TF32X3 = 32, SPLIT_F64 = 64;
constexpr int F64_DIGITS = 7, F64_PLANES = 8;
struct SliceForm {
  int S, kind, W;  // planes; 0 = bf16 digits, 1 = tf32 hi/lo; bits per digit
};
__host__ __device__ constexpr bool valid_split(int code) { return (code >= 1 && code <= 6) || code == SPLIT_TF32X3; }
__host__ __device__ constexpr SliceForm form_of(int code) {
  return code == SPLIT_TF32X3 ? SliceForm{2, 1, 0}
         : code == SPLIT_F64  ? SliceForm{F64_PLANES, 0, 9}
         : code == 6          ? SliceForm{5, 0, 9}
                              : SliceForm{code, 0, 7};
}
// e_s of W-bit digits
__host__ __device__ constexpr int digit_exp(int W, int s) { return W == 9 ? 9 * s - 1 : W * s; }

struct SliceSrc {
  const double* p;
  long long sb;  // batch stride
  Index2 r, k;   // row and K index maps
  bool kfast;    // K is the unit-stride index (else rows are)
  // > 0: the rows are the packed upper triangle of tri_n x tri_n index
  // pairs (tri_pair); row r reads r.at(m * tri_n + n)
  int tri_n = 0;
  long long row0 = 0;  // row 0 of the slices is row row0 of the source (a panel of its rows)
  // The exchange operand (six digits, recorded exponents; its k runs of k.div
  // follow each other): with ex_scale the element of row r in k run q = batch
  // ex_runs + k / k.div is ex_scale[r ex_n + q] times the source's, and
  // -ex_diag[r k.div + k % k.div] in run q == r.
  const double* ex_scale = nullptr;
  const double* ex_diag = nullptr;
  int ex_n = 0, ex_runs = 0;
  // words that the exponent kernel of unit-stride rows presets to META_PRESET for
  // the kernels after it
  unsigned int* preset = nullptr;
  int preset_n = 0;
  __host__ __device__ __forceinline__ long long row_at(long long row) const {
    if (tri_n <= 0) return r.at(row0 + row);
    int m, n;
    tri_pair(row0 + row, tri_n, m, n);
    return r.at((long long)m * tri_n + n);
  }
};

struct SlicedDesc {
  __nv_bfloat16* planes;  // blocked digit tiles (32-bit elements when kind == 1)
  int* exps;              // [batch][rows]
  int batch, rows, K, S;
  int kind = 0;  // 0: bf16 digits, 16 k per block; 1: tf32 hi/lo, 8 k per block
  int W = 7;     // bits per digit (kind 0)
  int* norms = nullptr;  // [batch][row block][SL_NORMS], directly behind exps where it is carved (kind 0)
  __host__ __device__ int kper() const { return kind ? SL_K / 2 : SL_K; }
  __host__ __device__ int code() const { return kind ? SPLIT_TF32X3 : W == 9 ? (S == F64_PLANES ? SPLIT_F64 : 6) : S; }  // the split code it was cut with
  __host__ __device__ int rblocks() const { return (rows + SL_ROWS - 1) / SL_ROWS; }
  __host__ __device__ int kblocks() const { return (K + kper() - 1) / kper(); }
  __host__ __device__ long long block_bytes() const { return (long long)S * SL_TILE_BYTES; }
  __host__ __device__ long long batch_bytes() const { return (long long)rblocks() * kblocks() * block_bytes(); }
};

// sqrt of the norms of digits 1..n of the row block that holds row r0 of batch entry b.
template <int n>
__device__ __forceinline__ void block_norms(const SlicedDesc& d, int b, int r0, float (&x)[n]) {
  const int* p = d.norms + ((long long)(d.batch == 1 ? 0 : b) * d.rblocks() + r0 / SL_ROWS) * SL_NORMS;
#pragma unroll
  for (int i = 0; i < n; ++i) x[i] = sqrtf(__int_as_float(__ldg(p + i)));
}

// `code` is a split code (1..6 or SPLIT_TF32X3).
inline size_t sliced_plane_bytes(int batch, int rows, int K, int code) {
  const SliceForm f = form_of(code);
  SlicedDesc d{nullptr, nullptr, batch, rows, K, f.S, f.kind, f.W};
  return (size_t)batch * d.batch_bytes();
}
// Exponents and, behind them, the norms (int32 each).
inline size_t sliced_meta_ints(int batch, int rows) {
  return (size_t)batch * rows + (size_t)batch * ((rows + SL_ROWS - 1) / SL_ROWS) * SL_NORMS;
}

// Carve a sliced operand (planes + exponents) out of a workspace or buffer.
template <class Cv>
SlicedDesc take_sliced(Cv& c, int batch, int rows, int K, int code) {
  auto* p = c.template take<unsigned char>(sliced_plane_bytes(batch, rows, K, code));
  auto* e = c.template take<int>(sliced_meta_ints(batch, rows));
  const SliceForm f = form_of(code);
  return SlicedDesc{reinterpret_cast<__nv_bfloat16*>(p), e, batch, rows, K, f.S, f.kind, f.W,
                    e ? e + (size_t)batch * rows : nullptr};
}

// The same with the exponents and norms in `meta`, which is moved past them: several
// operands' that one memset presets (META_PRESET below any exponent and any norm).
constexpr int META_PRESET_BYTE = 0x80;
constexpr unsigned int META_PRESET = 0x80808080u;
template <class Cv>
SlicedDesc take_planes(Cv& c, int batch, int rows, int K, int code, int*& meta) {
  auto* p = c.template take<unsigned char>(sliced_plane_bytes(batch, rows, K, code));
  int* e = meta;
  if (meta) meta += sliced_meta_ints(batch, rows);
  const SliceForm f = form_of(code);
  return SlicedDesc{reinterpret_cast<__nv_bfloat16*>(p), e, batch, rows, K, f.S, f.kind, f.W,
                    e ? e + (size_t)batch * rows : nullptr};
}

// Exponents and digits.  With exps_ready the row exponents are already in
// dst.exps (recorded by the kernel that read the source before) and only the
// digits are formed; the norms then hold a value below every float's bits
// (memset with 0x80 bytes).  A NaN or an infinity is recorded in *status, the
// device's status word when null.
int slice_operand(const SliceSrc& src, const SlicedDesc& dst, cudaStream_t s, bool exps_ready = false,
                  int* status = nullptr);

}  // namespace gb
