// FP64 contraction on the 5th-generation tensor cores (tcgen05) in integer digits.
//
// C = alpha * A B + beta * C with FP64 operands (the Ozaki scheme on signed 8-bit
// integers): every row of A (and every column of B) is scaled by a power of two so that
// its largest element is below 1 and written in balanced base-256 digits,
//     a = 2^e 2^-6 (d0 + d1 2^-8 + d2 2^-16 + ...),  -128 <= d <= 127.
// The digit products d_p d_q are summed exactly by tcgen05.mma (kind::i8, S32
// accumulation in TMEM) into one group per weight 2^-8(p+q), and the groups are
// combined in exact 64-bit integers before the one conversion to FP64.
//   digits = 4 (30 bits of each operand relative to its row / column maximum): the ten
//     products p + q < 4; the split-precision form.
//   digits = 8 (62 bits): the 36 products p + q < 8; the FP64 form.
//
// The error of a digit form is relative to the row and column maxima: with the row of A
// below 2^ea and the column of B below 2^eb it is about 2^-61 sqrt(K) 2^(ea+eb) in eight
// digits, while an FP64 accumulation is off by about 2^-54 sum_k |a_k b_k|.  Where the large
// elements of a row of A meet small ones of a column of B, that sum is far below
// K 2^(ea+eb), and a digit form loses what FP64 keeps.  So eight digits hold only where the
// sum is large enough.  The slicing pass takes a profile over k of every 64 rows of an
// operand (the least, over its groups of 8 rows, of their mean of |x| 2^-e); the product
// sum of two profiles stands for sum_k |a_k b_k| 2^-(ea+eb) of that 64 x 64 block of the
// output, and a block below 2^-9 sqrt(K), or with a non-finite element or a row maximum
// outside 2^+-400, is refused: gemm() computes it on the FP64 tensor pipe, all decided on
// the device.  Measured on 64 x 64 outputs, K = 64 .. 4096, largest error over sum |a b| in
// 2^-53 (FP64 chain, eight digits), by the product sum over sqrt(K): even Gaussian rows 0.1
// .. 0.8: 3, 0.4 .. 0.04; one element 300 times the others 1e-3 (refused) .. 7e-3: 14, 2 .. 0.5; A
// falling and B rising along k over a factor of 300 2e-3 .. 3e-3: 3, 4 .. 0.7, over 1000
// 7e-4 .. 1e-3: 3, 12 .. 2 (refused), over 1e6 1e-6: 3, 14000 .. 2000.
// (Seven digits of 34 products were at 17 on the factor of 100 that eight hold at 1.)  What
// passes was at most 1.25 times as far off as the FP64 chain.  The rule holds for 8 rows at a
// time: where a single row falls along k among even ones while B rises, its outputs are held
// to the 2^-61 sqrt(K) of the maxima only.
// In four digits, a row or column holding an Inf or NaN gives NaN in all its outputs.
#pragma once

#include <algorithm>
#include <cmath>

#include "gemm_f64.cuh"

namespace cc4s_b200 {

struct SplitScratch {
  void* p = nullptr;     // device scratch for the packed slices
  size_t bytes = 0;
  int* error = nullptr;  // device flag: non-zero if a bounded wait gave up
  GemmScratch fp64;      // split-K partials of the blocks that eight digits refuse
};

// The rule above: what the product sum of two profiles has to reach.
inline float split_profile_least(int64_t K) {
  return static_cast<float>(std::sqrt(static_cast<double>(K)) * 0x1p-9);
}
// Row maxima within these powers of two keep every scale and partial product normal.
constexpr int kSplitMaxExponent = 400;

// Ranges of k that share out the SMs when an output has few tiles (each range writes its
// own FP64 partial, added in order afterwards): the number with the least time by waves of
// 148 tiles, a k costing `per_k` microseconds and a tile 4 for its drain and store.
inline int64_t split_k_most(int64_t M, int64_t N, int64_t K) {
  return std::min<int64_t>(std::min<int64_t>(K / 1024, 40),
                           (int64_t(1) << 23) / std::max<int64_t>(M * N, 1));
}
inline int split_k_parts(int64_t tiles, int64_t M, int64_t N, int64_t K, int digits) {
  const double per_k = digits == 8 ? 0.020 : 0.012;
  const int64_t most = split_k_most(M, N, K);
  int best = 1;
  double least = 0.0;
  for (int n = 1; n <= std::max<int64_t>(most, 1); ++n) {
    const double t = double((tiles * n + 147) / 148) * (per_k * double(K) / n + 4.0) +
                     (n > 1 ? 6.0 : 0.0);
    if (n == 1 || t < least) { best = n; least = t; }
  }
  return best;
}

// True where an FP64 contraction (planar complex: one of gemm_split_complex) runs faster in
// eight digits than on the FP64 tensor pipe.
bool digits8_pays(const Contraction& c, bool cplx);

// Same contraction semantics as gemm() (two-level index maps, optional C2).
// The batch dimension must be 1.  Falls back to nothing: throws if the
// contraction cannot be expressed (the caller then uses gemm()).
void gemm_split(const Contraction& g, cudaStream_t s, SplitScratch& ws);

// Bytes of scratch gemm_split needs for this contraction.
size_t gemm_split_scratch_bytes(const Contraction& g);

// The planar complex contraction (imaginary planes at the given element offsets, conjA /
// conjB conjugate an operand) as two real ones over K' = 2 K with the planes side by side
// along k: every plane is sliced once or twice instead of twice or four times, and each
// output plane is written once.
void gemm_split_complex(const Contraction& g, int64_t a_im, int64_t b_im, int64_t c_im, bool conjA,
                        bool conjB, cudaStream_t s, SplitScratch& ws);
size_t gemm_split_complex_scratch_bytes(const Contraction& g);

// Operand B of a one-panel split contraction, sliced once and reused by several
// contractions that share B (same N, K and B view), e.g. the ladder's X panel
// for every block pair of one c range.
struct SplitPackedB {
  void* slices = nullptr;  // [digits][Np][Kp] signed bytes
  int* exps = nullptr;     // [Np] power-of-two column scales
  float* prof = nullptr;   // [Np / 64][Kp] profiles (eight digits)
  int64_t N = 0, K = 0, Np = 0, Kp = 0;
  int digits = 4;
};
// Bytes split_pack_b writes (slices, row maxima, exponents).
size_t split_packed_b_bytes(const Contraction& g);
// Scratch bytes of gemm_split_packed_b for this contraction (packed A and metadata).
size_t split_scratch_bytes_packed_b(const Contraction& g);
// True if g runs as one K panel (the condition for a pre-packed B).
bool split_single_panel(const Contraction& g);
// Slices B of g into dst (device memory of split_packed_b_bytes(g) bytes, 1 KiB aligned).
SplitPackedB split_pack_b(const Contraction& g, void* dst, cudaStream_t s);
// gemm_split with B taken from split_pack_b (A is sliced into ws as usual; ws must
// not overlap b).
void gemm_split_packed_b(const Contraction& g, const SplitPackedB& b, cudaStream_t s,
                         SplitScratch& ws);

// An operand sliced once for many contractions: R rows of K elements as digit
// planes [digits][Rp][Kp] with one power-of-two exponent per row (the scaling of every
// row over its whole K, as gemm_split slices its operands).
struct SplitOperand {
  void* slices = nullptr;
  int* exps = nullptr;   // [Rp]
  float* prof = nullptr;   // [Rp / 64][Kp] profiles (eight digits)
  int64_t R = 0, K = 0, Rp = 0, Kp = 0;
  int digits = 4;
};
// Device bytes of a sliced operand of R rows and K columns.
size_t split_operand_bytes(int64_t R, int64_t K, int digits = 4);
// Slices the rows of src into dst (device memory of split_operand_bytes bytes):
// element (r, k) at src[(r / Ri) * s_ro + (r % Ri) * s_ri + k * s_k] (Ri = 0: one level).
SplitOperand split_pack_operand(const double* src, int64_t R, int64_t Ri, int64_t s_ro,
                                int64_t s_ri, int64_t K, int64_t s_k, void* dst, cudaStream_t s,
                                int digits = 4);
// The rows of a contraction inside a sliced operand: logical index x is packed row
//   base + (x / run) * stride + x % run.
struct SplitRuns {
  int64_t base = 0, run = 0, stride = 0;
};
// C = alpha A B + beta C (g gives M, N, K, the output views, alpha, beta) with the rows
// m of A and the columns n of B taken from sliced operands (B sliced by its columns,
// i.e. its rows are n).  Tiles never straddle a run, so a run shorter than a tile
// costs a partial tile.  Nothing is refused here: see split_refused.
void gemm_split_prepacked(const Contraction& g, const SplitOperand& A, const SplitRuns& ar,
                          const SplitOperand& B, const SplitRuns& br, cudaStream_t s,
                          SplitScratch& ws);

// Whether eight digits refuse any block of the products of these two operands' rows: *word
// (8 bytes of device memory, cleared here) is non-zero if so.
void split_refused(const SplitOperand& A, const SplitOperand& B, int* word, cudaStream_t s);

uint64_t split_launch_count();
// Number of operand-slicing kernel launches issued so far (two per
// contraction whose operands are sliced in it).
uint64_t split_pack_launch_count();

}  // namespace cc4s_b200
