// fire_sliced.cu -- slicing kernels and the tensor-core contraction of sliced operands (fire_sliced.cuh).
#include "fire_sliced.cuh"

#include <cstring>

#include "fire_tc.cuh"

namespace fire {

namespace {

// ----------------------------------------------------------------------------------------------- slicing
// Exponent of the largest magnitude (its bits, sign cleared) of a row or column: SL_ZERO when everything vanishes,
// SL_NAN when an infinity or a NaN is among the values (the outputs are then NaN).
constexpr int SL_ZERO = -32768, SL_NAN = 32767;
__device__ __forceinline__ unsigned long long mag_bits(double a) {
  return (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ unsigned mag_bits(float a) { return __float_as_uint(a) & 0x7fffffffu; }
__device__ __forceinline__ int sl_code(unsigned long long m) {
  const int f = (int)(m >> 52);
  return f == 0 ? SL_ZERO : (f == 0x7ff ? SL_NAN : f - 1023);  // FP64 denormals count as zero
}
__device__ __forceinline__ int sl_code(unsigned m) {
  const int f = (int)(m >> 23);
  return m == 0u ? SL_ZERO : (f == 255 ? SL_NAN : max(f - 127, -119));  // 2^(6 - e) stays a float
}
template <typename T>
struct Mag;
template <>
struct Mag<float> {
  using U = unsigned;
};
template <>
struct Mag<double> {
  using U = unsigned long long;
};

// Two values of one row -> their NS slices, packed FP16 pairs.
// FP32: x = a 2^(6 - e) in (-128, 128); slice 0 is x rounded to an integer, the next ones the remainder times 2^9 rounded
// again (every step exact); the last slice keeps its fraction (FP16's 11 bits).
__device__ __forceinline__ float rint_small(float x) {  // |x| < 2^22
  return __fsub_rn(__fadd_rn(x, 12582912.f), 12582912.f);
}
template <int NS>
__device__ __forceinline__ void slices2(float a, float b, int code, uint32_t (&w)[NS]) {
  const float inv = (code == SL_ZERO || code == SL_NAN) ? 0.f : __int_as_float((127 + 6 - code) << 23);
  float x = a * inv, y = b * inv;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const bool last = i == NS - 1;
    const float s = last ? x : rint_small(x), t = last ? y : rint_small(y);
    const __half2 h = __floats2half2_rn(s, t);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
    x = (x - s) * 512.f;
    y = (y - t) * 512.f;
  }
}
// FP64: q = a 2^(6 - e) 2^56 rounded to an integer (|q| < 2^63), cut into balanced base-256 digits from the lowest.
__device__ __forceinline__ long long fixed56(double a, int code) {
  const long long bits = __double_as_longlong(a);
  const int f = (int)((bits >> 52) & 0x7ff);
  if (f == 0 || code == SL_ZERO || code == SL_NAN) return 0;
  const unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
  const int d = code - (f - 1023) - 10;  // q = m 2^-d, d >= -10
  long long q;
  if (d <= 0) q = (long long)(m << -d);
  else q = d > 56 ? 0 : (long long)((m + (1ull << (d - 1))) >> d);
  return bits < 0 ? -q : q;
}
template <int NS>
__device__ __forceinline__ void slices2(double a, double b, int code, uint32_t (&w)[NS]) {
  long long qa = fixed56(a, code), qb = fixed56(b, code);
  const __half2 off = __halves2half2(__ushort_as_half(0x6600), __ushort_as_half(0x6600));  // 1536
#pragma unroll
  for (int i = NS - 1; i >= 0; --i) {
    const int da = i ? (int)((qa + 128) & 255) - 128 : (int)qa, db = i ? (int)((qb + 128) & 255) - 128 : (int)qb;
    qa = (qa - da) >> 8;
    qb = (qb - db) >> 8;
    // integers of magnitude <= 128 as FP16: the bits of 1536 + d, minus 1536
    const uint32_t u = (uint32_t)((0x6600 + da) & 0xffff) | ((uint32_t)((0x6600 + db) & 0xffff) << 16);
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), off);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
// Eight K-consecutive values of one row -> one 16-byte core-matrix row per slice, slices `stride` bytes apart.
template <int KIND, typename T>
__device__ __forceinline__ void store_slices(const T (&v)[8], int code, unsigned char* out, size_t stride) {
  constexpr int NS = SlFmt<KIND>::NS;
  uint32_t w[4][NS];
#pragma unroll
  for (int q = 0; q < 4; ++q) slices2(v[2 * q], v[2 * q + 1], code, w[q]);
#pragma unroll
  for (int i = 0; i < NS; ++i)
    *reinterpret_cast<uint4*>(out + i * stride) = make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
}
template <typename T>
__device__ __forceinline__ void load8(const T* p, int k, int K, bool ok, bool vec, T (&v)[8]) {
  if (ok && vec && k + 8 <= K) {
    if constexpr (sizeof(T) == 4) {
      const float4 x = *reinterpret_cast<const float4*>(p + k), y = *reinterpret_cast<const float4*>(p + k + 4);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double2 x = *reinterpret_cast<const double2*>(p + k + 2 * u);
        v[2 * u] = x.x; v[2 * u + 1] = x.y;
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (ok && k + u < K) ? p[k + u] : T(0);
  }
}

template <typename T>
struct SliceArgs {
  const T* A[2];
  long lda[2];
  int M[2];
  const int* M_dev;
  int M_scale[2];
  int row0, row1;  // this pass's rows of every segment
  int K, nkb, n_el;
  int ns[2], soff[2];  // ns > 0: row q is row (q / ns) n_el + soff + q % ns of A
  unsigned char* out[2];
  int* code[2];
};

// 32 rows per CTA (lane = row), warps over the 8-deep k-groups: every load takes a 32- or 64-byte piece of 32 rows, every
// store fills 512 consecutive bytes.  First the rows' largest magnitudes, then the slices; rows of up to 256 values stay in
// registers in between.  Bound by memory: it reads A once (twice beyond 256) and writes 2 NS bytes per value.
constexpr int SLR_WARPS = 8, SLR_KEEP = 4;
template <int KIND, typename T>
__global__ void __launch_bounds__(32 * SLR_WARPS) k_slice_rows(SliceArgs<T> a) {
  constexpr int NS = SlFmt<KIND>::NS;
  using U = typename Mag<T>::U;
  __shared__ U part[SLR_WARPS][32];
  const int g = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int rows = a.M[g];
  if (a.M_dev) rows = min(rows, a.M_scale[g] * *a.M_dev);
  rows = min(rows, a.row1) - a.row0;  // of this pass
  const int ql = blockIdx.x * 32 + lane, q = a.row0 + ql;
  if ((int)blockIdx.x * 32 >= (rows + 127) / 128 * 128) return;
  const bool ok = ql < rows;
  const long src = a.ns[g] > 0 ? (long)(q / a.ns[g]) * a.n_el + a.soff[g] + q % a.ns[g] : (long)q;
  const T* p = a.A[g] + (ok ? src : 0) * a.lda[g];
  const bool vec = (a.lda[g] * sizeof(T)) % 16 == 0 && (reinterpret_cast<uintptr_t>(a.A[g]) & 15) == 0;
  const int nkg = 2 * a.nkb;
  const bool keep = nkg <= SLR_KEEP * SLR_WARPS;
  T v[SLR_KEEP][8];
  U mx = 0;
  if (keep) {
#pragma unroll
    for (int t = 0; t < SLR_KEEP; ++t) {
      const int kg = warp + t * SLR_WARPS;
      load8(p, kg * 8, a.K, ok && kg < nkg, vec, v[t]);
    }
#pragma unroll
    for (int t = 0; t < SLR_KEEP; ++t)
#pragma unroll
      for (int u = 0; u < 8; ++u) mx = max(mx, (U)mag_bits(v[t][u]));
  } else {
#pragma unroll 4
    for (int kg = warp; kg < nkg; kg += SLR_WARPS) {
      load8(p, kg * 8, a.K, ok, vec, v[0]);
#pragma unroll
      for (int u = 0; u < 8; ++u) mx = max(mx, (U)mag_bits(v[0][u]));
    }
  }
  part[warp][lane] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < SLR_WARPS; ++w) mx = max(mx, part[w][lane]);
  const int code = sl_code(mx);
  if (warp == 0) a.code[g][ql] = code;
  // [128-row tile][16-deep step][slice][k-group][128 rows][16 bytes]
  unsigned char* out = a.out[g] + (size_t)(ql >> 7) * a.nkb * NS * 4096 + (ql & 127) * 16;
  auto put = [&](const T (&x)[8], int kg) {
    store_slices<KIND>(x, code, out + (size_t)(kg >> 1) * NS * 4096 + (kg & 1) * 2048, 4096);
  };
  if (keep) {
#pragma unroll
    for (int t = 0; t < SLR_KEEP; ++t) {
      const int kg = warp + t * SLR_WARPS;
      if (kg < nkg) put(v[t], kg);
    }
  } else {
#pragma unroll 2
    for (int kg = warp; kg < nkg; kg += SLR_WARPS) {
      load8(p, kg * 8, a.K, ok, vec, v[0]);
      put(v[0], kg);
    }
  }
}

// Weights W [K][N] (row-major) -> [column tile][16-deep step][slice][k-group][NMAX columns][16 bytes] (nc of them used),
// then N column exponents.  32 columns per CTA (lane = column), warps over k.
template <int KIND, typename T>
__global__ void __launch_bounds__(256) k_slice_w(const T* __restrict__ W, int K, int N, SlTile tl,
                                                 unsigned char* __restrict__ out, size_t code_off) {
  constexpr int NS = SlFmt<KIND>::NS;
  using U = typename Mag<T>::U;
  __shared__ U part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  const bool ok = c < N;
  U mx = 0;
#pragma unroll 8
  for (int k = warp; k < K; k += 8) mx = max(mx, ok ? (U)mag_bits(W[(size_t)k * N + c]) : (U)0);
  part[warp][lane] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) mx = max(mx, part[w][lane]);
  const int code = sl_code(mx);
  if (warp == 0 && ok) reinterpret_cast<int*>(out + code_off)[c] = code;
  if (c >= tl.nt * tl.nc) return;
  const int j = c / tl.nc, r = c % tl.nc;
  constexpr int NMAX = SlFmt<KIND>::NMAX;
  constexpr size_t step = (size_t)NS * 32 * NMAX;
  for (int kg = warp; kg < 2 * tl.nkb; kg += 8) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (ok && kg * 8 + u < K) ? W[(size_t)(kg * 8 + u) * N + c] : T(0);
    store_slices<KIND>(v, code, out + ((size_t)j * tl.nkb + (kg >> 1)) * step + (size_t)(kg & 1) * 16 * NMAX + r * 16,
                       (size_t)32 * NMAX);
  }
}

// ----------------------------------------------------------------------------------------------- contraction
template <int KIND>
struct SlSmem {
  using Fm = SlFmt<KIND>;
  static constexpr int A_STEP = Fm::NS * 4096;
  static constexpr int B_STEP = Fm::NS * 32 * Fm::NMAX;
  static constexpr int STAGE = A_STEP + B_STEP;
  // staging of one epilogue warp: 32 rows x 16 columns (17: no bank conflicts) of hi and lo floats, or of the high 64
  // and the low 32 bits of the FP64 sums
  static constexpr int STG = 32 * 17 * (KIND == SL_PAIR ? 8 : 12);
  static constexpr int TOTAL = Fm::STAGES * STAGE + 8 * STG + 256;
};
constexpr int SL_THREADS = 320;  // warps 0-7 epilogue, 8 loader, 9 MMA issuer

template <typename T>
struct SlArgs {
  int nseg;
  GemmP<T> p[2];
  const unsigned char* At[2];
  const int* ac[2];
  const unsigned char* Bt[2];
  size_t b_code;
  SlTile tl;
  int pw;  // 16-column pieces of a column tile per unit of work
  int row0, row1;  // this pass's rows of every segment
  int ns[2], soff[2], spin[2];
  const int* tile_mask;
  float* C_lo;
  const float* env_lo;
  long ld_lo;
};

template <int STAGES>
struct SlBar {
  uint64_t full[STAGES], empty[STAGES], tfull, tempty;
  uint32_t tmem;
  int abort;
};

// Three 16-column pieces of this warp's 32 lanes, in flight together.
__device__ __forceinline__ void tmem_ld16x3(uint32_t a0, uint32_t a1, uint32_t a2, float (&v)[3][16]) {
  uint32_t r[48];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%48];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, "
      "[%49];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, "
      "[%50];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]),
        "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]),
        "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
      : "r"(a0), "r"(a1), "r"(a2)
      : "memory");
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int k = 0; k < 16; ++k) v[q][k] = __uint_as_float(r[16 * q + k]);
}

// (h 2^32 + l) 2^e as a double, rounded to nearest.  Integer arithmetic: the FP64 pipe would take longer
// for the same than the tile's MMAs.
__device__ __forceinline__ double sl_assemble(long long h, uint32_t l, int e) {
  // magnitude in one's complement form: off by one unit of the lowest slices' product
  const long long neg = h >> 63;
  h ^= neg;
  uint32_t z = l ^ (uint32_t)neg;
  uint32_t x = (uint32_t)((unsigned long long)h >> 32), y = (uint32_t)h;
  int up = 0;  // words shifted out
  if (x == 0) { x = y; y = z; z = 0; up = 32; }
  if (x == 0) { x = y; y = 0; up = 64; }
  if (x == 0) return 0.0;
  const int lz = __clz(x);
  x = __funnelshift_l(y, x, lz);
  y = __funnelshift_l(z, y, lz);
  const unsigned long long m = ((unsigned long long)x << 32) | y;  // bit 63 set
  const int field = e + 32 - up - lz + 1086;  // the exponent's field; in a denormal more than 11 bits are rounded away
  const int drop = field > 0 ? 11 : 12 - field;
  unsigned long long q = 0;
  if (drop < 64) q = m >> drop;
  if (drop <= 64) q += (m >> (drop - 1)) & 1;
  if (field > 0) q += (unsigned long long)(field - 1) << 52;  // a carry to 2^53 goes into the exponent
  if (field > 2046) q = 0x7ff0000000000000ull;
  return __longlong_as_double((neg & (long long)0x8000000000000000ull) | (long long)q);
}

// 2^(e - 6), the scale of a row or column of SL_PAIR
__device__ __forceinline__ float sl_scale(int code) {
  if (code == SL_ZERO) return 0.f;
  if (code == SL_NAN) return __int_as_float(0x7fc00000);
  return __int_as_float((code - 6 + 127) << 23);  // code >= -119
}

// Element-wise epilogues of the hi + lo results (CompMode); row: row of C, q: row of the segment.
template <int MODE>
__device__ __forceinline__ void sl_store_pair(const SlArgs<float>& a, const GemmP<float>& p, int spin, int q, long row,
                                              int col, float h, float l) {
  const float* bias = spin == 1 ? p.bias2 : p.bias;
  if (bias && (MODE != COMP_PLAIN || (p.bias_period > 0 && q % p.bias_period == 0))) {
    float s, e;
    two_sum(h, bias[col], s, e);
    h = s;
    l += e;
  }
  float s, e;  // normalised pair: s = fl(h + l)
  two_sum(h, l, s, e);
  if (MODE == COMP_PLAIN) {
    p.C[row * p.ldc + col] = s;
  } else if (MODE == COMP_SILU) {
    if (p.aux0) {
      float y, d1, d2;
      silu3(s, y, d1, d2);
      p.C[row * p.ldc + col] = y;
      p.aux0[row * p.ld_aux + col] = d1;
      p.aux2[row * p.ld_aux + col] = d2;
    } else {
      p.C[row * p.ldc + col] = silu(s);
    }
  } else {  // COMP_ORB: raw orbital times envelope, hi + lo
    p.aux0[row * p.ld_aux + col] = s;
    const float eh = p.aux1[row * p.env_nv * p.ld_aux + col], el = a.env_lo[row * a.ld_lo + col];
    const float ph = s * eh;
    const float pl = fmaf(s, eh, -ph) + (s * el + e * eh);
    float oh, ol;
    two_sum(ph, pl, oh, ol);
    p.C[row * p.ldc + col] = oh;
    a.C_lo[row * a.ld_lo + col] = ol;
  }
}

// What one epilogue thread keeps of its row: up to NC pieces of 16 columns, unscaled.
template <int KIND>
struct SlAcc;
template <>
struct SlAcc<SL_PAIR> {
  static constexpr int NC = 3;
  float hi[NC][16], lo[NC][16];
};
template <>
struct SlAcc<SL_F64> {  // value = h 2^32 + l, in units of 2^-56 of slice 0's
  static constexpr int NC = 2;
  long long h[NC][16];
  uint32_t l[NC][16];
};

// Drains one chunk of K: the levels of piece ci (16 columns at tensor-memory column t of the first accumulator), put
// together and, after the first chunk, added to what the earlier chunks gave.
__device__ __forceinline__ void sl_drain(SlAcc<SL_PAIR>& s, int ci, uint32_t t, bool first) {
  constexpr int nc = SlFmt<SL_PAIR>::NMAX;
  float v[3][16];
  tmem_ld16x3(t + 3 * nc, t + 4 * nc, t + 5 * nc, v);  // levels 3, 4, 5
  float l[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) l[k] = fmaf(fmaf(v[2][k], 0x1p-9f, v[1][k]), 0x1p-9f, v[0][k]) * 0x1p-27f;
  tmem_ld16x3(t, t + nc, t + 2 * nc, v);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    float h, e, e2;
    two_sum(v[0][k], v[1][k] * 0x1p-9f, h, e);
    two_sum(h, v[2][k] * 0x1p-18f, h, e2);
    const float lo = (e + e2) + l[k];
    if (first) {
      s.hi[ci][k] = h;
      s.lo[ci][k] = lo;
    } else {
      two_sum(s.hi[ci][k], h, s.hi[ci][k], e);
      s.lo[ci][k] += e + lo;
    }
  }
}
__device__ __forceinline__ void sl_drain(SlAcc<SL_F64>& s, int ci, uint32_t t, bool first) {
  constexpr int nc = SlFmt<SL_F64>::NMAX;
  float v[3][16], w[16];
  long long low[16];
  tmem_ld16x3(t + 5 * nc, t + 6 * nc, t + 7 * nc, v);  // levels 5, 6, 7
  tmem_ld16(t + 4 * nc, w);
#pragma unroll
  for (int k = 0; k < 16; ++k)
    low[k] = ((long long)__float2int_rn(w[k]) * 256 + __float2int_rn(v[0][k])) * 65536 +
             ((long long)__float2int_rn(v[1][k]) * 256 + __float2int_rn(v[2][k]));
  tmem_ld16x3(t, t + nc, t + 2 * nc, v);
  tmem_ld16(t + 3 * nc, w);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int a = __float2int_rn(v[0][k]) * 256 + __float2int_rn(v[1][k]);  // levels 0, 1: below 2^31
    const long long top =
        (long long)a * 65536 + ((long long)__float2int_rn(v[2][k]) * 256 + __float2int_rn(w[k]));
    long long h = top + (low[k] >> 32);
    uint32_t l = (uint32_t)low[k];
    if (!first) {
      const unsigned long long ls = (unsigned long long)l + s.l[ci][k];
      h += s.h[ci][k] + (long long)(ls >> 32);
      l = (uint32_t)ls;
    }
    s.h[ci][k] = h;
    s.l[ci][k] = l;
  }
}

template <int KIND, int MODE>
__global__ void __launch_bounds__(SL_THREADS, 1) k_gemm_sl(const __grid_constant__ SlArgs<typename SlFmt<KIND>::T> a,
                                                          int32_t* status) {
  using Fm = SlFmt<KIND>;
  using T = typename Fm::T;
  using Sm = SlSmem<KIND>;
  constexpr int NS = Fm::NS, STAGES = Fm::STAGES;
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  unsigned char* stg = tc_smem + STAGES * Sm::STAGE;
  SlBar<STAGES>* bars = reinterpret_cast<SlBar<STAGES>*>(stg + 8 * Sm::STG);
  volatile int* abort = &bars->abort;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int nt = a.tl.nt, nc = a.tl.nc, nkb = a.tl.nkb;
  int rows[2] = {0, 0}, mt[2] = {0, 0};
#pragma unroll
  for (int g = 0; g < 2; ++g)
    if (g < a.nseg) {
      rows[g] = a.p[g].M;
      if (a.p[g].M_dev) rows[g] = min(rows[g], a.p[g].M_scale * *a.p[g].M_dev);
      rows[g] = max(0, min(rows[g], a.row1) - a.row0);
      mt[g] = (rows[g] + 127) / 128;
    }
  // a column tile may be split into ncp parts of pw pieces of 16 columns, each its own unit of work (few rows)
  const int np = nc / 16, pw = a.pw, ncp = (np + pw - 1) / pw, nu = nt * ncp;
  const int t0 = mt[0] * nu, total = t0 + mt[1] * nu;
  if ((int)blockIdx.x >= total) return;
  // unit t: segment, row tile, column tile and the first piece in it (column tiles of a row tile run next to each other: its
  // slices come from L2)
  auto decode = [&](int t, int& g, int& m, int& n, int& p0) -> bool {
    g = t >= t0 ? 1 : 0;
    if (g) t -= t0;
    n = t % nu;
    m = t / nu;
    p0 = n % ncp * pw;
    n /= ncp;
    return !a.tile_mask || ((a.tile_mask[a.row0 / 128 + m] >> a.spin[g]) & 1);
  };

  if (tid == 0) {
    for (int q = 0; q < STAGES; ++q) {
      mbar_init(smem_u32(&bars->full[q]), 2);  // the A and the W copy
      mbar_init(smem_u32(&bars->empty[q]), 1);
    }
    mbar_init(smem_u32(&bars->tfull), 1);
    mbar_init(smem_u32(&bars->tempty), 256);
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  proxy_fence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem, 0);
  const uint32_t s0 = smem_u32(tc_smem);
  long issued = 0;  // steps whose copies were issued (loader lane)

  if (warp == 8) {
    // ------------------------------------------------------------------ loader
    if (lane == 0) {
      for (int t = blockIdx.x; t < total && !*abort; t += gridDim.x) {
        int g, m, n, p0;
        if (!decode(t, g, m, n, p0)) continue;
        const unsigned char* as = a.At[g] + (size_t)m * nkb * Sm::A_STEP;
        const unsigned char* bs = a.Bt[g] + (size_t)n * nkb * Sm::B_STEP;
        for (int kb = 0; kb < nkb; ++kb) {
          const int q = (int)(issued % STAGES);
          const long use = issued / STAGES;
          if (use > 0 && !tc_wait(&bars->empty[q], (uint32_t)((use - 1) & 1), abort)) break;
          const uint32_t dst = s0 + q * Sm::STAGE, bar = smem_u32(&bars->full[q]);
          bulk_load(dst, as + (size_t)kb * Sm::A_STEP, Sm::A_STEP, bar);
          bulk_load(dst + Sm::A_STEP, bs + (size_t)kb * Sm::B_STEP, Sm::B_STEP, bar);
          ++issued;
        }
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform; one lane issues)
    long kc = 0, uc = 0;
    bool live = true;
    for (int t = blockIdx.x; t < total && live; t += gridDim.x) {
      int g, m, n, p0;
      if (!decode(t, g, m, n, p0)) continue;
      const uint32_t idesc = (1u << 4) | ((uint32_t)(2 * min(pw, np - p0)) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
      for (int kb = 0; kb < nkb; ++kb, ++kc) {
        const bool start = kb % SL_KCH == 0;
        if (start && uc > 0) {
          live = __all_sync(0xffffffffu, tc_wait(&bars->tempty, (uint32_t)((uc - 1) & 1), abort));
          if (!live) break;
          tc_fence_after();
        }
        const int q = (int)(kc % STAGES);
        live = __all_sync(0xffffffffu, tc_wait(&bars->full[q], (uint32_t)((kc / STAGES) & 1), abort));
        if (!live) break;
        tc_fence_after();
        const uint64_t da = tc_desc_s(s0 + q * Sm::STAGE, 2048, 128);
        const uint64_t db = tc_desc_s(s0 + q * Sm::STAGE + Sm::A_STEP + p0 * 256, 16 * Fm::NMAX, 128);  // 16 columns: 256 bytes
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
          for (int j = 0; j < NS - i; ++j)  // level i + j; i == 0 is the level's first product of the step
            tc_mma_elect(tmem + (uint32_t)((i + j) * Fm::NMAX), da + (uint64_t)(i * 256), db + (uint64_t)(j * 2 * Fm::NMAX),
                         idesc, (start && i == 0) ? 0u : 1u);
        tc_commit_elect(smem_u32(&bars->empty[q]));
        if (kb % SL_KCH == SL_KCH - 1 || kb == nkb - 1) {
          tc_commit_elect(smem_u32(&bars->tfull));
          ++uc;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 0-7)
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t tq = tmem + ((uint32_t)(quad * 32) << 16);
    long uc = 0;
    bool live = true;  // warp-uniform
    for (int t = blockIdx.x; t < total && live; t += gridDim.x) {
      int g, m, n, p0;
      if (!decode(t, g, m, n, p0)) continue;
      const GemmP<T>& p = a.p[g];
      const int M = a.row0 + rows[g], N = p.N, l0 = m * 128 + quad * 32, m0 = a.row0 + l0, n0 = n * nc + p0 * 16;
      const int nl = min(pw, np - p0);  // pieces of this unit
      const int* bc = reinterpret_cast<const int*>(a.Bt[g] + a.b_code);
      const int rc = a.ac[g][l0 + lane];
      SlAcc<KIND> acc;
      for (int k0 = 0; k0 < nkb; k0 += SL_KCH) {
        live = __all_sync(0xffffffffu, tc_wait(&bars->tfull, (uint32_t)(uc & 1), abort));
        if (!live) break;
        tc_fence_after();
#pragma unroll
        for (int ci = 0; ci < SlAcc<KIND>::NC; ++ci) {  // pieces half, half + 2, ... of the tile's columns
          const int c = half + 2 * ci;
          if (c < nl) sl_drain(acc, ci, tq + (uint32_t)(c * 16), k0 == 0);
        }
        tc_fence_before();
        tc_arrive(&bars->tempty);
        ++uc;
      }
      if (!live) break;
      // Element-wise epilogue through the warp's staging rows, so that 16 lanes take the 16 columns of one row.  This
      // lane's row of the segment: its row in C (-1: none), for FP32 its scale.
      const int cl = lane & 15, hl = lane >> 4, q0 = m0 + lane;
      int crow = q0 < M ? q0 : -1;
      if (a.ns[g] > 0 && q0 < M) crow = (q0 / a.ns[g]) * p.n_el + a.soff[g] + q0 % a.ns[g];
      if (KIND == SL_F64 && MODE == EPI_ORB_J && crow >= 0 &&
          (((gemm_node(p, crow) % p.n_el) < p.n_up) ? 0 : 1) != a.spin[g])
        crow = -1;
      [[maybe_unused]] float rs = 0.f;
      if (KIND == SL_PAIR) rs = sl_scale(rc);
#pragma unroll
      for (int ci = 0; ci < SlAcc<KIND>::NC; ++ci) {
        const int c = half + 2 * ci;
        if (c >= nl) continue;
        const int col = n0 + c * 16 + cl;
        const int cc = col < N ? bc[col] : SL_ZERO;
        if constexpr (KIND == SL_PAIR) {
          float* sh = reinterpret_cast<float*>(stg + warp * Sm::STG);
          float* sl = sh + 32 * 17;
          const float cs = sl_scale(cc);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            sh[lane * 17 + k] = acc.hi[ci][k];
            sl[lane * 17 + k] = acc.lo[ci][k];
          }
          __syncwarp();
#pragma unroll 4
          for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + hl, row = __shfl_sync(0xffffffffu, crow, r);
            const float sc = __shfl_sync(0xffffffffu, rs, r);
            if (row >= 0 && col < N)
              sl_store_pair<MODE>(a, p, a.spin[g], m0 + r, (long)row, col, sh[r * 17 + cl] * sc * cs,
                                  sl[r * 17 + cl] * sc * cs);
          }
        } else {
          long long* sh = reinterpret_cast<long long*>(stg + warp * Sm::STG);
          uint32_t* sl = reinterpret_cast<uint32_t*>(sh + 32 * 17);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            sh[lane * 17 + k] = acc.h[ci][k];
            sl[lane * 17 + k] = acc.l[ci][k];
          }
          __syncwarp();
          [[maybe_unused]] double s2 = 0.0;
          [[maybe_unused]] int cur = -1;
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + hl, row = __shfl_sync(0xffffffffu, crow, r), ra = __shfl_sync(0xffffffffu, rc, r);
            double x = 0.0;
            if (ra == SL_NAN || cc == SL_NAN) x = __longlong_as_double(0x7ff8000000000000ll);
            else if (ra != SL_ZERO && cc != SL_ZERO) x = sl_assemble(sh[r * 17 + cl], sl[r * 17 + cl], ra + cc - 68);
            if constexpr (MODE == EPI_SILU_J) {
              // per-center sums of squares: lanes 0-15 the even rows of a column, lanes 16-31 the odd ones, one atomic
              // per run of a center
              const int node = row >= 0 ? gemm_node(p, row) : -1;
              if (node != cur) {
                if (cur >= 0 && col < N) atomic_add(&p.aux2[(long)cur * p.ld_aux + col], s2);
                s2 = 0.0;
                cur = node;
              }
              s2 += x * x;
            }
            if (row >= 0 && col < N) gemm_store<double, MODE>(p, row, col, x, a.spin[g]);
          }
          if constexpr (MODE == EPI_SILU_J) {
            if (cur >= 0 && col < N) atomic_add(&p.aux2[(long)cur * p.ld_aux + col], s2);
          }
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  if (*abort && tid == 0) set_flag(status, FIRE_FLAG_TIMEOUT);
  if (*abort && warp == 8 && lane == 0) {
    // bounded drain: copies still in flight must land before the CTA's shared memory goes away
    for (long q = issued > STAGES ? issued - STAGES : 0; q < issued; ++q) {
      const uint32_t bar = smem_u32(&bars->full[q % STAGES]);
      const uint32_t par = (uint32_t)((q / STAGES) & 1);
      for (int i = 0; i < (1 << 16); ++i) {
        uint32_t d;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(d)
            : "r"(bar), "r"(par)
            : "memory");
        if (d) break;
      }
    }
  }
  if (*abort && warp == 9 && lane == 0) {
    // bounded drain: MMAs still in flight must finish before tensor memory is released
    for (int q = 0; q < STAGES; ++q) {
      const uint32_t bar = smem_u32(&bars->empty[q]);
      for (int i = 0; i < (1 << 16); ++i) {
        uint32_t d0, d1;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(d0)
            : "r"(bar)
            : "memory");
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 1;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(d1)
            : "r"(bar)
            : "memory");
        if (d0 || d1) break;
      }
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 9) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

int device_sms() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

template <int KIND, int MODE>
int sl_launch(const SlCall<typename SlFmt<KIND>::T>& c, unsigned char* scratch, int32_t* status, cudaStream_t s) {
  using T = typename SlFmt<KIND>::T;
  const GemmP<T>& p0 = c.p[0];
  if (c.nseg < 1 || c.nseg > 2 || p0.K < 1 || p0.N < 1) return -1;
  SlArgs<T> a;
  SliceArgs<T> r;
  std::memset(&a, 0, sizeof(a));
  std::memset(&r, 0, sizeof(r));
  a.nseg = c.nseg;
  a.tl = sl_tile(p0.K, p0.N, SlFmt<KIND>::NMAX);
  a.b_code = sl_w_code_offset<KIND>(p0.K, p0.N);
  a.tile_mask = c.tile_mask;
  a.C_lo = c.C_lo;
  a.env_lo = c.env_lo;
  a.ld_lo = c.ld_lo;
  r.M_dev = p0.M_dev;
  r.K = p0.K;
  r.nkb = a.tl.nkb;
  r.n_el = p0.n_el;
  const int sliced = c.share_a ? 1 : c.nseg;
  long mmax = 0;
  for (int g = 0; g < c.nseg; ++g) mmax = std::max<long>(mmax, c.p[g].M);
  if (mmax == 0) return 0;
  const long pass = sl_pass_rows(mmax, sliced);
  const size_t a_bytes = sl_a_bytes<KIND>(pass, p0.K), block = (a_bytes + (size_t)pass * 4 + 255) / 256 * 256;
  for (int g = 0; g < c.nseg; ++g) {
    const GemmP<T>& p = c.p[g];
    if (p.K != p0.K || p.N != p0.N || !c.w[g]) return -1;
    const int q = c.share_a ? 0 : g;  // whose slices
    a.p[g] = p;
    a.Bt[g] = c.w[g];
    a.ns[g] = c.ns[g];
    a.soff[g] = c.soff[g];
    a.spin[g] = c.spin[g];
    a.At[g] = scratch + (size_t)q * block;
    a.ac[g] = reinterpret_cast<const int*>(a.At[g] + a_bytes);
    r.A[g] = p.A;
    r.lda[g] = p.lda;
    r.M[g] = p.M;
    r.M_scale[g] = p.M_scale;
    r.ns[g] = c.ns[g];
    r.soff[g] = c.soff[g];
    r.out[g] = const_cast<unsigned char*>(a.At[g]);
    r.code[g] = const_cast<int*>(a.ac[g]);
  }
  constexpr int smem = SlSmem<KIND>::TOTAL;
  if (cudaFuncSetAttribute(k_gemm_sl<KIND, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1;
  const int sms = device_sms();
  int launched = 0;
  for (long r0 = 0; r0 < mmax; r0 += pass) {
    a.row0 = r.row0 = (int)r0;
    a.row1 = r.row1 = (int)std::min<long>(r0 + pass, mmax);
    long tiles = 0, rows = 0;
    for (int g = 0; g < c.nseg; ++g) {
      const long m = std::max<long>(0, std::min<long>(c.p[g].M, a.row1) - r0);
      tiles += ((m + 127) / 128) * a.tl.nt;
      rows = std::max(rows, m);
    }
    const dim3 gr((unsigned)(sl_rows(rows) / 32), (unsigned)sliced);
    k_slice_rows<KIND, T><<<gr, 32 * SLR_WARPS, 0, s>>>(r);
    // Few tiles: parts of two pieces or of one, as long as each gets an SM of its own (an MMA of 16 columns takes 36 cycles
    // where 64 take 48, and a unit's epilogue goes with its columns): 160 rows x 256 x 256 26 -> 20 us.
    const int np = a.tl.nc / 16;
    a.pw = tiles * np <= sms ? 1 : (tiles * ((np + 1) / 2) <= sms ? std::min(2, np) : np);
    const long units = tiles * ((np + a.pw - 1) / a.pw);
    k_gemm_sl<KIND, MODE><<<(unsigned)std::min<long>(units, sms), SL_THREADS, smem, s>>>(a, status);
    launched += 2;
  }
  return cudaPeekAtLastError() == cudaSuccess ? launched : -1;
}

template <int KIND>
cudaError_t sl_prepare(const typename SlFmt<KIND>::T* W, int K, int N, unsigned char* out, cudaStream_t s) {
  const SlTile t = sl_tile(K, N, SlFmt<KIND>::NMAX);
  k_slice_w<KIND><<<(unsigned)((t.nt * t.nc + 31) / 32), 256, 0, s>>>(W, K, N, t, out, sl_w_code_offset<KIND>(K, N));
  return cudaPeekAtLastError();
}

__global__ void k_sl_tile_mask(GemmP<double> p, int* mask) {
  int rows = p.M;
  if (p.M_dev) rows = min(rows, p.M_scale * *p.M_dev);
  const int row = blockIdx.x * 128 + threadIdx.x;
  int up = 0, dn = 0;
  if (row < rows) {
    if ((gemm_node(p, row) % p.n_el) < p.n_up) up = 1; else dn = 1;
  }
  up = __syncthreads_or(up);
  dn = __syncthreads_or(dn);
  if (threadIdx.x == 0) mask[blockIdx.x] = up | (dn << 1);
}

}  // namespace

cudaError_t sl_prepare_pair(const float* W, int K, int N, unsigned char* out, cudaStream_t s) {
  return sl_prepare<SL_PAIR>(W, K, N, out, s);
}
cudaError_t sl_prepare_f64(const double* W, int K, int N, unsigned char* out, cudaStream_t s) {
  return sl_prepare<SL_F64>(W, K, N, out, s);
}

void sl_tile_mask(const GemmP<double>& p, int* mask, cudaStream_t s) {
  if (p.M > 0) k_sl_tile_mask<<<(unsigned)((p.M + 127) / 128), 128, 0, s>>>(p, mask);
}

int sl_gemm_pair(int mode, const SlCall<float>& c, unsigned char* scratch, int32_t* status, cudaStream_t s) {
  switch (mode) {
    case COMP_PLAIN: return sl_launch<SL_PAIR, COMP_PLAIN>(c, scratch, status, s);
    case COMP_SILU: return sl_launch<SL_PAIR, COMP_SILU>(c, scratch, status, s);
    case COMP_ORB: return sl_launch<SL_PAIR, COMP_ORB>(c, scratch, status, s);
    default: return -1;
  }
}

int sl_gemm_f64(int mode, const SlCall<double>& c, unsigned char* scratch, int32_t* status, cudaStream_t s) {
  switch (mode) {
    case EPI_PLAIN: return sl_launch<SL_F64, EPI_PLAIN>(c, scratch, status, s);
    case EPI_SILU_X: return sl_launch<SL_F64, EPI_SILU_X>(c, scratch, status, s);
    case EPI_SILU_J: return sl_launch<SL_F64, EPI_SILU_J>(c, scratch, status, s);
    case EPI_SILU_L: return sl_launch<SL_F64, EPI_SILU_L>(c, scratch, status, s);
    case EPI_ORB_X: return sl_launch<SL_F64, EPI_ORB_X>(c, scratch, status, s);
    case EPI_ORB_J: return sl_launch<SL_F64, EPI_ORB_J>(c, scratch, status, s);
    case EPI_ORB_L: return sl_launch<SL_F64, EPI_ORB_L>(c, scratch, status, s);
    default: return -1;
  }
}

}  // namespace fire
