// fire_sliced.cuh -- contractions at (or above) the accuracy of the plain FP64 dot product and of the compensated FP32
// one, on the FP16 tensor cores.
//
// C[M, N] = A[M, K] * W[K, N].  Every row of A and every column of W is scaled by a power of two to the grid of its own
// largest magnitude and cut into NS slices of SL_BITS bits each, a = sum_i s_i 2^(-BITS i) (the error-free splitting of
// Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012).  The slices are integers of magnitude at most 2^(BITS - 1),
// exact in FP16, so a product of two of them is an integer and the tensor core's FP32 accumulator sums up to 256 of them
// exactly, whatever order and rounding it uses.  Products are grouped by their level l = i + j (their common scale is
// 2^(-bits l)); levels l < NS are computed, each in a tensor-memory accumulator of its own, and the epilogue puts them
// together.  Two formats (an operand's bits count from its row's or column's largest value, so the error is relative to the
// product of the two largest magnitudes, not to the terms: rows whose large values meet zero weights are not for this, see
// stage_orbitals for the envelopes):
//   SL_PAIR  FP32 operands, 6 slices (8 + 5 x 9 bits), 21 MMAs per product; the result is a hi + lo float pair.  The slices
//            hold 53 bits below the row's largest value.  Five slices of 9 bits (15 MMAs) left errors up to 10 times those
//            of the compensated dot product on the CUDA cores (k_gemm_comp).
//   SL_F64   FP64 operands, 8 slices of 8 bits, 36 MMAs per product; the levels are put together in integer arithmetic and
//            rounded once.  63 bits below the largest value, 10 more than an FP64 number has (7 slices left errors up to
//            twice FP64's own).  FP64 denormals count as zero.
// Sums of the first levels stay below 2^24, the range of exact integers: SL_PAIR's first slice is at most 2^7 in magnitude
// (2 x 256 x 2^7 x 2^8 for level 1), SL_F64's all are ((l + 1) 256 x 2^14 for level l <= 3).  From level 2 (3) on an
// accumulator could lose its lowest bit if every product had the same sign and nearly the largest size, at 2^-17 (2^-32)
// of the result times 2^-24.
//
// The CUDA-core FP64 contraction ran at the FP64 pipe's rate (about 1.2 TFLOP/s on GB300, 1/64 of FP32): one 128 x 128 x 256
// tile took 1.05 ms.  Here it takes ~25 us.
//
// Work split.  k_slice_rows cuts the rows of A once per contraction into the order the MMA reads (every column tile of
// the output reads it again, from L2), the weights are cut when the parameters are prepared.  k_gemm_sl is persistent,
// one CTA per SM: a loader thread streams 16-deep steps of all slices of A and W through a ring with bulk copies, one
// thread issues the MMAs, eight warps drain tensor memory.  The accumulators of one 128-row tile fill tensor memory, so
// the next tile's MMAs wait for the drain, but not for the element-wise epilogue and its stores.  Both kernels run over
// blocks of rows that give every SM a whole number of tiles and whose slices (~60 MB at K = 256) stay in L2: the slices of
// a larger launch would go through HBM twice, and need scratch in proportion.
#pragma once
#include <algorithm>

#include "fire_gemm.cuh"
#include "fire_internal.cuh"

namespace fire {

enum SlKind { SL_PAIR = 0, SL_F64 = 1 };

template <int KIND>
struct SlFmt;
template <>
struct SlFmt<SL_PAIR> {
  using T = float;
  static constexpr int NS = 6, NMAX = 80, STAGES = 4;
};
template <>
struct SlFmt<SL_F64> {
  using T = double;
  static constexpr int NS = 8, NMAX = 64, STAGES = 3;
};

constexpr int SL_KCH = 16;  // 16-deep steps per exact chunk: K is summed in chunks of 256, put together in the epilogue

// Column tiles of a K x N weight: nt tiles of nc columns (a multiple of 16, at most nmax), nkb 16-deep steps.  A tile is
// stored with nmax rows, so that the MMA's operand and accumulator strides are constants (with strides that followed nc, the
// one issuing thread needed 87 cycles per MMA of 128 x 80 x 16, which the tensor core finishes in 52).
struct SlTile {
  int nt, nc, nkb;
};
__host__ __device__ inline SlTile sl_tile(int K, int N, int nmax) {
  SlTile t;
  t.nt = (N + nmax - 1) / nmax;
  t.nc = ((N + t.nt - 1) / t.nt + 15) / 16 * 16;
  t.nkb = (K + 15) / 16;
  return t;
}
template <int KIND>
inline size_t sl_w_bytes(int K, int N) {  // slices of one weight, then its N column exponents
  const SlTile t = sl_tile(K, N, SlFmt<KIND>::NMAX);
  return (size_t)t.nt * t.nkb * SlFmt<KIND>::NS * 32 * SlFmt<KIND>::NMAX + ((size_t)N * 4 + 255) / 256 * 256;
}
template <int KIND>
inline size_t sl_w_code_offset(int K, int N) {
  const SlTile t = sl_tile(K, N, SlFmt<KIND>::NMAX);
  return (size_t)t.nt * t.nkb * SlFmt<KIND>::NS * 32 * SlFmt<KIND>::NMAX;
}
inline long sl_rows(long M) { return (M + 127) / 128 * 128; }
template <int KIND>
inline size_t sl_a_bytes(long M, int K) {  // slices of M rows (whole 128-row tiles)
  return (size_t)sl_rows(M) * ((K + 15) / 16) * 32 * SlFmt<KIND>::NS;
}
// Row tiles of one pass over all segments: one per SM, as many whole tiles as that leaves to each of the `segs` segments.
// (SL_SMS is GB300's count: the scratch is sized with it, so that another count only leaves a pass less even.)
constexpr int SL_SMS = 152;
inline long sl_pass_rows(long M, int segs) {
  return std::min<long>(sl_rows(M), 128 * std::max<long>(1, SL_SMS / segs));
}
// scratch of a contraction's A: the slices of a pass, then one exponent per row, for every segment (M: the larger segment's
// rows)
template <int KIND>
inline size_t sl_scratch_bytes(long M, int K, int segs = 1) {
  const long r = sl_pass_rows(M, segs);
  return (size_t)segs * ((sl_a_bytes<KIND>(r, K) + (size_t)r * 4 + 255) / 256 * 256);
}

// One contraction, or two that differ in their rows and weights (the spins).  Segment g multiplies its own rows
// (p[g].A, M, lda ...) by its own weight.  ns[g] > 0: row q of the segment is row (q / ns) n_el + soff + q % ns of A, of C and
// of the per-row operands; 0: row q.
template <typename T>
struct SlCall {
  int nseg;
  GemmP<T> p[2];
  const unsigned char* w[2];  // sliced weights
  int ns[2], soff[2];
  int spin[2];                // bias2 instead of bias for 1; ORB_J: the rows' spin that the segment stores
  int share_a;                // both segments read the same rows: sliced once
  const int* tile_mask;       // ORB_J: spins present in every 128-row tile
  float* C_lo;
  const float* env_lo;
  long ld_lo;
};
cudaError_t sl_prepare_pair(const float* W, int K, int N, unsigned char* out, cudaStream_t s);
cudaError_t sl_prepare_f64(const double* W, int K, int N, unsigned char* out, cudaStream_t s);
// spins present in every 128-row tile (bit 0 up, bit 1 down) of a contraction's rows
void sl_tile_mask(const GemmP<double>& p, int* mask, cudaStream_t s);
// mode: CompMode for hi + lo pairs, EpiMode for FP64.  scratch: sl_scratch_bytes over the call's segments (one if
// they share A), 256-byte aligned.  Returns the number of kernels launched, or -1 on an error.
int sl_gemm_pair(int mode, const SlCall<float>& c, unsigned char* scratch, int32_t* status, cudaStream_t s);
int sl_gemm_f64(int mode, const SlCall<double>& c, unsigned char* scratch, int32_t* status, cudaStream_t s);

}  // namespace fire
