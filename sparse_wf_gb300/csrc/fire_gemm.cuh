// fire_gemm.cuh -- CUDA-core GEMM C = A[M,K] * B[K,N] with fused forward-Laplacian epilogues.
//
// k_gemm_f: FP32 (derivative planes of the FP32 path, plain value rows, gradients); k_gemm_d: FP64 (the refinement's values,
// narrow layers and envelopes; fire_sliced.cu has the FP64 build's wide layers); k_gemm_comp: the FP32 local energy's
// compensated value rows and every hi + lo envelope row; k_gemm_env_df: the refinement's envelope rows.  Every dense layer of
// the sparse forward Laplacian (sparse_fwd_lap.py:160-225) is applied to three "planes" of one node:
//   X plane  [nodes, K]        values            (bias added)
//   J plane  [3 * positions, K] Jacobian rows    (sorted by center)
//   L plane  [nodes, K]        Laplacians
// and the ElementWise rule (sparse_fwd_lap.py:196-206) is fused into the epilogues:
//   X:  z = acc + b;  store z and silu(z)
//   J:  out = acc * silu'(z[center]);  jsq[center] += acc^2  (segmented over the tile's rows)
//   L:  out = acc * silu'(z) + jsq * silu''(z)
// The orbital layer (orbitals.py:148-174 + multiply_with_1el_fn, sparse_fwd_lap.py:322-335) uses
// per-spin weights (rows of spin-up centers use B, spin-down centers B2) and multiplies by the
// envelope carrier in its epilogues.
#pragma once
#include "fire_common.cuh"
#include "fire_f32x2.cuh"

namespace fire {

enum EpiMode { EPI_PLAIN = 0, EPI_SILU_X, EPI_SILU_J, EPI_SILU_L, EPI_ORB_X, EPI_ORB_J, EPI_ORB_L, EPI_ENV, EPI_ACC };  // EPI_ACC: added to C

template <typename T>
struct GemmP {
  const T* A;
  long lda;
  const T* B;
  long ldb;
  const T* B2;  // spin-down weights (or nullptr)
  const T* bias;
  const T* bias2;
  int bias_period;  // bias added on rows with row % bias_period == 0 (0: no bias)
  T* C;
  long ldc;
  int M;             // row capacity
  const int* M_dev;  // optional device row count: rows = min(M, M_scale * *M_dev)
  int M_scale;
  int N, K;
  const int* node_map;  // node of a row = node_map ? node_map[row / node_div] : row / node_div
  int node_div;
  int n_el, n_up;       // spin of node g: (g % n_el) < n_up
  T* aux0;
  const T* aux1;
  T* aux2;
  const T* aux3;
  long ld_aux;
  const int* dep_map;  // ORB_J: a position is "self" when dep_map[pos] == node
  int env_ns, env_soff;  // ENV: rows are (w * env_ns + i) * env_nv + v  ->  electron w * n_el + env_soff + i
  int env_nv;            // rows per electron of the envelope carrier (5: x, jac xyz, lap; 1: value)
  int row_skip;          // tensor-core path: rows with row % row_skip == 0 are not stored (0: none)
};

template <typename T>
__device__ __forceinline__ int gemm_node(const GemmP<T>& p, int row) {
  return p.node_map ? p.node_map[row / p.node_div] : row / p.node_div;
}

template <typename T, int MODE>
__device__ __forceinline__ void gemm_store(const GemmP<T>& p, int row, int col, T acc, int pass_spin) {
  if (MODE == EPI_PLAIN) {
    T v = acc;
    if (p.bias && p.bias_period > 0 && (row % p.bias_period) == 0) v += p.bias[col];
    p.C[(long)row * p.ldc + col] = v;
  } else if (MODE == EPI_ACC) {
    p.C[(long)row * p.ldc + col] += acc;
  } else if (MODE == EPI_SILU_X) {
    // value plane; with aux0 set it also writes silu'(z) (aux0) and silu''(z) (aux2), which the
    // Jacobian and Laplacian epilogues of the same layer read instead of re-evaluating them per row
    T z = acc + (p.bias ? p.bias[col] : T(0));
    p.C[(long)row * p.ldc + col] = silu(z);
    if (p.aux0) {
      T y, d1, d2;
      silu3(z, y, d1, d2);
      p.aux0[(long)row * p.ld_aux + col] = d1;
      p.aux2[(long)row * p.ld_aux + col] = d2;
    }
  } else if (MODE == EPI_SILU_J) {  // aux1: silu' plane
    const int node = gemm_node(p, row);
    p.C[(long)row * p.ldc + col] = acc * p.aux1[(long)node * p.ld_aux + col];
  } else if (MODE == EPI_SILU_L) {  // aux1: silu', aux0: silu'', aux3: sum of squared Jacobian rows
    const long o = (long)row * p.ld_aux + col;
    p.C[(long)row * p.ldc + col] = acc * p.aux1[o] + p.aux3[o] * p.aux0[o];
  } else if (MODE == EPI_ORB_X) {
    const T* b = pass_spin == 0 ? p.bias : p.bias2;
    const T raw = acc + b[col];
    p.aux0[(long)row * p.ld_aux + col] = raw;
    p.C[(long)row * p.ldc + col] = raw * p.aux1[(long)row * p.env_nv * p.ld_aux + col];
  } else if (MODE == EPI_ORB_J) {
    const int pos = row / 3, t = row - 3 * (row / 3);
    const int node = p.node_map[pos];
    const T* env = p.aux1 + (long)node * 5 * p.ld_aux;
    const T ex = env[col];
    if (p.dep_map[pos] == node) {
      const T raw = p.aux3[(long)node * p.ld_aux + col];
      p.C[(long)row * p.ldc + col] = raw * env[(1 + t) * p.ld_aux + col] + ex * acc;
      p.aux2[((long)node * 3 + t) * p.ld_aux + col] = acc;
    } else {
      p.C[(long)row * p.ldc + col] = ex * acc;
    }
  } else if (MODE == EPI_ORB_L) {
    const T* env = p.aux1 + (long)row * 5 * p.ld_aux;
    const T* rjs = p.aux2 + (long)row * 3 * p.ld_aux;
    T v = acc * env[col] + env[4 * p.ld_aux + col] * p.aux3[(long)row * p.ld_aux + col];
    v += T(2) * (rjs[col] * env[p.ld_aux + col] + rjs[p.ld_aux + col] * env[2 * p.ld_aux + col] +
                 rjs[2 * p.ld_aux + col] * env[3 * p.ld_aux + col]);
    p.C[(long)row * p.ldc + col] = v;
  } else if (MODE == EPI_ENV) {
    const int rr = row / p.env_nv, v = row - p.env_nv * rr;
    const int g = (rr / p.env_ns) * p.n_el + p.env_soff + rr % p.env_ns;
    p.C[((long)g * p.env_nv + v) * p.ldc + col] = acc;
  }
}

__device__ __forceinline__ void cp_async_n(void* dst, const void* src, int bytes, bool ok) {  // bytes 4, 8 or 16, zero fill
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
  else if (bytes == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_left() {  // at most N groups of this thread in flight
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// FP32 contraction on the CUDA cores: 128 x 128 (256 threads, 8 x 8 outputs each), 64 x 64 (64 threads, 8 x 8) or 32 x 32 (64
// threads, 4 x 4) outputs per CTA, FGK k per stage, copied asynchronously FGS - 1 stages ahead.  Every output is one chain of fused
// multiply-adds over ascending k, whatever the tile: all tiles and the scalar kernel before them give the same bits.  Bound by
// the FMA pipes (128 and 64: 60 to 63 % busy, their latency between few warps the rest; 41 to 45 TFLOP/s), the 32 x 32 tile by
// shared-memory loads (76 % of their rate, FMA pipes 57 %) or, with few rows, by the chain of stages: a small tile then puts
// more SMs to work.
constexpr int FGS = 4;
template <int BM, bool BT = false>
struct FgCfg {
  static constexpr int BN = BM, TM = BM >= 64 ? 8 : 4, THREADS = (BM / TM) * (BN / TM);
  static constexpr int FGK = BM == 32 ? 32 : 16;
  static constexpr int FGA = FGK + 4;  // row length of the A tile (k contiguous, rows on different banks)
  static constexpr int STAGE = BM * FGA + (BT ? BN * FGA : FGK * BN);  // floats
  static constexpr int SQ = BM * (BN + 1);
  static constexpr size_t smem(bool sq) { return sizeof(float) * (sq && SQ > FGS * STAGE ? SQ : FGS * STAGE); }
  // CTAs per SM that the registers are shared out for: what 228 KB of shared memory (1 KB of each CTA's reserved) hold, and no
  // more than 6 (a bound of 7 for the 64 x 64 tile, of which 6 fit, kept it at 128 registers and made it spill)
  static constexpr int FIT = 228 * 1024 / (int)(smem(false) + 1024 + sizeof(int) * BM);
  static constexpr int CTAS = BM == 128 ? 2 : (FIT < 6 ? FIT : 6);
};

// BT: B is the transpose of p.B [N, K] (p.ldb); its tile is kept like A's, k contiguous, and a thread's columns lie TX apart
// so that their rows are read without bank conflicts.
template <int MODE, int BM, bool BT = false>
__global__ void __launch_bounds__(FgCfg<BM, BT>::THREADS, FgCfg<BM, BT>::CTAS) k_gemm_f(GemmP<float> p) {
  using Cf = FgCfg<BM, BT>;
  constexpr int BN = Cf::BN, TM = Cf::TM, NT = Cf::THREADS, H = BM / 2;  // H: rows (columns) between a thread's two halves
  constexpr int TX = BN / TM, FGK = Cf::FGK, FGA = Cf::FGA;
  extern __shared__ __align__(16) float fg_smem[];  // [stage][A: BM x FGA, B: FGK x BN]; at the end the squares of SILU_J
  __shared__ int row_node[BM];
  int rows = p.M;
  if (p.M_dev) rows = min(rows, p.M_scale * (*p.M_dev));
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (m0 >= rows) return;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  // rows and columns of the thread: groups of 4, with 8 x 8 a second group half a tile further
  auto rloc = [&](int i) { return (i & 3) + ty * 4 + (i >> 2) * H; };
  auto cloc = [&](int j) { return BT ? tx + j * TX : (j & 3) + tx * 4 + (j >> 2) * H; };

  // spin composition of the tile (per-spin weights)
  int passes = 1, first_spin = 0;
  if (p.B2) {
    int up = 0, dn = 0;
    for (int r = tid; r < BM && m0 + r < rows; r += NT) {
      const int node = gemm_node(p, m0 + r);
      if ((node % p.n_el) < p.n_up) up = 1; else dn = 1;
    }
    up = __syncthreads_or(up);
    dn = __syncthreads_or(dn);
    first_spin = up ? 0 : 1;
    passes = up + dn;
  }
  if (MODE == EPI_SILU_J) {
    for (int r = tid; r < BM; r += NT) row_node[r] = (m0 + r < rows) ? gemm_node(p, m0 + r) : -1;
  }
  const bool va = p.lda % 4 == 0 && p.K % 4 == 0 && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int spin = first_spin + pass;
    const float* Bp = spin == 0 ? p.B : p.B2;
    const bool vb = p.ldb % 4 == 0 && (BT ? p.K : p.N) % 4 == 0 && (reinterpret_cast<uintptr_t>(Bp) & 15) == 0;
    f32x2 acc[TM][TM / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TM / 2; ++j) acc[i][j] = 0ull;
    const int ks = (p.K + FGK - 1) / FGK;
    auto fetch = [&](int st) {
      if (st < ks) {
        float* As = fg_smem + (st % FGS) * Cf::STAGE;
        float* Bs = As + BM * FGA;
        const int k0 = st * FGK;
        if (va) {
#pragma unroll
          for (int u = 0; u < BM * FGK / 4 / NT; ++u) {
            const int e = tid + u * NT, r = e / (FGK / 4), k = (e % (FGK / 4)) * 4;
            const bool ok = m0 + r < rows && k0 + k < p.K;
            cp_async_n(As + r * FGA + k, ok ? p.A + (long)(m0 + r) * p.lda + k0 + k : p.A, 16, ok);
          }
        } else {
          for (int e = tid; e < BM * FGK; e += NT) {
            const int r = e / FGK, k = e % FGK;
            const bool ok = m0 + r < rows && k0 + k < p.K;
            cp_async_n(As + r * FGA + k, ok ? p.A + (long)(m0 + r) * p.lda + k0 + k : p.A, 4, ok);
          }
        }
        if (BT) {
          for (int e = tid; e < BN * FGK / (vb ? 4 : 1); e += NT) {
            const int w = vb ? 4 : 1, c = e / (FGK / w), k = e % (FGK / w) * w;
            const bool ok = n0 + c < p.N && k0 + k < p.K;
            cp_async_n(Bs + c * FGA + k, ok ? Bp + (long)(n0 + c) * p.ldb + k0 + k : Bp, 4 * w, ok);
          }
        } else if (vb) {
#pragma unroll
          for (int u = 0; u < FGK * BN / 4 / NT; ++u) {
            const int e = tid + u * NT, k = e / (BN / 4), c = (e % (BN / 4)) * 4;
            const bool ok = k0 + k < p.K && n0 + c < p.N;
            cp_async_n(Bs + k * BN + c, ok ? Bp + (long)(k0 + k) * p.ldb + n0 + c : Bp, 16, ok);
          }
        } else {
          for (int e = tid; e < FGK * BN; e += NT) {
            const int k = e / BN, c = e % BN;
            const bool ok = k0 + k < p.K && n0 + c < p.N;
            cp_async_n(Bs + k * BN + c, ok ? Bp + (long)(k0 + k) * p.ldb + n0 + c : Bp, 4, ok);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < FGS - 1; ++st) fetch(st);
    for (int st = 0; st < ks; ++st) {
      cp_async_left<FGS - 2>();
      __syncthreads();  // stage st has landed for everyone, and everyone has left stage st - 1
      fetch(st + FGS - 1);
      const float* As = fg_smem + (st % FGS) * Cf::STAGE;
      const float* Bs = As + BM * FGA;
#pragma unroll
      for (int kq = 0; kq < FGK; kq += 4) {
        float a[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float4 q = *reinterpret_cast<const float4*>(As + rloc(i) * FGA + kq);
          a[i][0] = q.x; a[i][1] = q.y; a[i][2] = q.z; a[i][3] = q.w;
        }
        float bt[BT ? TM : 1][4];
        if (BT) {
#pragma unroll
          for (int j = 0; j < TM; ++j) {
            const float4 q = *reinterpret_cast<const float4*>(Bs + cloc(j) * FGA + kq);
            bt[BT ? j : 0][0] = q.x; bt[BT ? j : 0][1] = q.y; bt[BT ? j : 0][2] = q.z; bt[BT ? j : 0][3] = q.w;
          }
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          f32x2 b[TM / 2];
          if (BT) {
#pragma unroll
            for (int j = 0; j < TM / 2; ++j) b[j] = pack2(bt[BT ? 2 * j : 0][kk], bt[BT ? 2 * j + 1 : 0][kk]);
          } else
#pragma unroll
          for (int h = 0; h < TM / 4; ++h) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Bs + (kq + kk) * BN + tx * 4 + h * H);
            b[2 * h] = q.x;
            b[2 * h + 1] = q.y;
          }
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const f32x2 aa = pack2(a[i][kk], a[i][kk]);
#pragma unroll
            for (int j = 0; j < TM / 2; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
          }
        }
      }
    }
    cp_async_left<0>();

    // ---- epilogue
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int row = m0 + rloc(i);
      if (row >= rows) continue;
      if (p.B2) {
        const int node = gemm_node(p, row);
        const int s = ((node % p.n_el) < p.n_up) ? 0 : 1;
        if (s != spin) continue;
      }
#pragma unroll
      for (int j = 0; j < TM / 2; ++j) {
        const int cx = n0 + cloc(2 * j), cy = n0 + cloc(2 * j + 1);
        float x, y;
        unpack2(acc[i][j], x, y);
        if (cx < p.N) gemm_store<float, MODE>(p, row, cx, x, spin);
        if (cy < p.N) gemm_store<float, MODE>(p, row, cy, y, spin);
      }
    }
    if (MODE == EPI_SILU_J || pass + 1 < passes) __syncthreads();  // everyone has left the tiles
    if (MODE == EPI_SILU_J) {
      // segmented sum of acc^2 over rows of the same center, one atomic per (segment, column)
      float* sq = fg_smem;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TM / 2; ++j) {
          const int c = (j & 1) * 2 + tx * 4 + (j >> 1) * H;
          float x, y;
          unpack2(acc[i][j], x, y);
          sq[rloc(i) * (BN + 1) + c] = x * x;
          sq[rloc(i) * (BN + 1) + c + 1] = y * y;
        }
      __syncthreads();
      // NT / BN row groups, one column per thread
      constexpr int RG = NT / BN > 0 ? NT / BN : 1, RL = BM / RG;
      const int lc = tid % BN, grp = tid / BN, col = n0 + lc;
      if (col < p.N) {
        int cur = -1;
        float s = 0.f;
        for (int lr = grp * RL; lr < grp * RL + RL; ++lr) {
          const int nd = row_node[lr];
          if (nd != cur) {
            if (cur >= 0) atomic_add(&p.aux2[(long)cur * p.ld_aux + col], s);
            cur = nd;
            s = 0.f;
          }
          if (nd >= 0) s += sq[lr * (BN + 1) + lc];
        }
        if (cur >= 0) atomic_add(&p.aux2[(long)cur * p.ld_aux + col], s);
      }
      if (pass + 1 < passes) __syncthreads();
    }
  }
}

template <int MODE, int BM, bool BT = false>
inline cudaError_t launch_gemm_f(const GemmP<float>& p, cudaStream_t s) {
  using Cf = FgCfg<BM, BT>;
  const dim3 grid((p.N + Cf::BN - 1) / Cf::BN, (p.M + BM - 1) / BM);
  const size_t smem = Cf::smem(MODE == EPI_SILU_J);
  const cudaError_t e = cudaFuncSetAttribute(k_gemm_f<MODE, BM, BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (grid.y == 0 || grid.x == 0) return cudaSuccess;
  k_gemm_f<MODE, BM, BT><<<grid, Cf::THREADS, smem, s>>>(p);
  return cudaPeekAtLastError();
}

// FP64 contraction on the CUDA cores (the refinement pass, the low-rank blocks, narrow layers, envelopes): every output one chain
// of fused multiply-adds over ascending k.  Bound by the FP64 pipe (97 % busy), which GB300 has at 1/64 of the FP32 rate: 128 x 128 outputs per CTA
// at K = N = 256 kept an SM for 1.05 ms while the others idled.  16 x 16 outputs per CTA, 2 x 2 per thread: small enough that
// any row count loads the SMs evenly, and two warps per CTA hide the chain.  At K = N = 256 with 160 / 600 / 2050 / 16400 rows
// 48 / 110 / 271 / 1751 us (the pipe alone: 18 / 68 / 233 / 1861 at 1.9 GHz); 32 x 32 with 2 x 2 per thread 72 / 135 / 265 /
// 1727, 16 x 16 with 4 x 4, half a warp, 150 / 246 / 645 / 3557.
constexpr int DG_BM = 16, DG_RT = 2, DG_K = 16, DG_ST = 3, DG_LA = DG_K + 2, DG_THREADS = (DG_BM / DG_RT) * (DG_BM / DG_RT);
constexpr int DG_STAGE = DG_BM * DG_LA + DG_K * DG_BM;
template <int MODE>
__global__ void __launch_bounds__(DG_THREADS) k_gemm_d(GemmP<double> p) {
  constexpr int BM = DG_BM, RT = DG_RT, NT = DG_THREADS, TX = BM / RT, LA = DG_LA, DK = DG_K, ST = DG_ST;
  __shared__ __align__(16) double sm[ST * DG_STAGE];
  int rows = p.M;
  if (p.M_dev) rows = min(rows, p.M_scale * (*p.M_dev));
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BM;
  if (m0 >= rows) return;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  int passes = 1, first_spin = 0;
  if (p.B2) {  // per-spin weights: a pass per spin present in the tile
    int up = 0, dn = 0;
    for (int r = tid; r < BM && m0 + r < rows; r += NT) {
      if ((gemm_node(p, m0 + r) % p.n_el) < p.n_up) up = 1; else dn = 1;
    }
    up = __syncthreads_or(up);
    dn = __syncthreads_or(dn);
    first_spin = up ? 0 : 1;
    passes = up + dn;
  }
  const bool va = p.lda % 2 == 0 && p.K % 2 == 0 && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int spin = first_spin + pass, ks = (p.K + DK - 1) / DK;
    const double* Bp = spin == 0 ? p.B : p.B2;
    auto fetch = [&](int st) {
      if (st < ks) {
        double* As = sm + (st % ST) * DG_STAGE;
        double* Bs = As + BM * LA;
        const int k0 = st * DK;
        if (va) {
          for (int e = tid; e < BM * DK / 2; e += NT) {
            const int r = e / (DK / 2), k = e % (DK / 2) * 2;
            const bool ok = m0 + r < rows && k0 + k < p.K;
            cp_async_n(As + r * LA + k, ok ? p.A + (long)(m0 + r) * p.lda + k0 + k : p.A, 16, ok);
          }
        } else {
          for (int e = tid; e < BM * DK; e += NT) {
            const int r = e / DK, k = e % DK;
            const bool ok = m0 + r < rows && k0 + k < p.K;
            cp_async_n(As + r * LA + k, ok ? p.A + (long)(m0 + r) * p.lda + k0 + k : p.A, 8, ok);
          }
        }
        for (int e = tid; e < DK * BM; e += NT) {
          const int k = e / BM, c = e % BM;
          const bool ok = k0 + k < p.K && n0 + c < p.N;
          cp_async_n(Bs + k * BM + c, ok ? Bp + (long)(k0 + k) * p.ldb + n0 + c : Bp, 8, ok);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[RT][RT];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < RT; ++j) acc[i][j] = 0.0;
#pragma unroll
    for (int st = 0; st < ST - 1; ++st) fetch(st);
    for (int st = 0; st < ks; ++st) {
      cp_async_left<ST - 2>();
      __syncthreads();  // stage st has landed for everyone, and everyone has left stage st - 1
      fetch(st + ST - 1);
      const double* As = sm + (st % ST) * DG_STAGE + ty * RT * LA;
      const double* Bs = sm + (st % ST) * DG_STAGE + BM * LA + tx * RT;
#pragma unroll 4
      for (int k = 0; k < DK; ++k) {
        double b[RT];
#pragma unroll
        for (int j = 0; j < RT; j += 2) {
          const double2 v = *reinterpret_cast<const double2*>(Bs + k * BM + j);
          b[j] = v.x;
          b[j + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const double a = As[i * LA + k];
#pragma unroll
          for (int j = 0; j < RT; ++j) acc[i][j] = fma(a, b[j], acc[i][j]);
        }
      }
    }
    cp_async_left<0>();
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int row = m0 + ty * RT + i;
      if (row >= rows) continue;
      if (p.B2 && (((gemm_node(p, row) % p.n_el) < p.n_up) ? 0 : 1) != spin) continue;
#pragma unroll
      for (int j = 0; j < RT; ++j) {
        const int col = n0 + tx * RT + j;
        if (col < p.N) gemm_store<double, MODE>(p, row, col, acc[i][j], spin);
      }
    }
    if (pass + 1 < passes) __syncthreads();
  }
}
template <int MODE>
inline cudaError_t launch_gemm_d(const GemmP<double>& p, cudaStream_t s) {
  const dim3 grid((p.M + DG_BM - 1) / DG_BM, (p.N + DG_BM - 1) / DG_BM);
  if (grid.y == 0 || grid.x == 0) return cudaSuccess;
  k_gemm_d<MODE><<<grid, DG_THREADS, 0, s>>>(p);
  return cudaPeekAtLastError();
}

// modes that the FP64 contraction on the CUDA cores is built for
constexpr bool gemm_d_mode(int mode) { return mode == EPI_PLAIN || mode == EPI_SILU_X || mode == EPI_ORB_X || mode == EPI_ENV; }
template <typename T, int MODE, bool BT = false>
inline cudaError_t launch_gemm(const GemmP<T>& p, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) {
    auto tiles = [&](int b) { return (long)((p.N + b - 1) / b) * ((p.M + b - 1) / b); };
    // Where the lines lie (us at K = 256, tiles of 128 / 64 / 32): 184500 x 256 588 / 657 / 733, 20992 x 1280 302 / 305 / 358,
    // 20992 x 256 90 / 79 / 78, 6400 x 256 38 / 38 / 30, 2560 x 256 38 / 27 / 16, 160 x 256 38 / 26 / 9 (the scalar 128 x 128
    // kernel before: 880, 441, 120, 42, 42, 41).  Slower: 256 x 128 outputs, 16 x 8 per thread (814 and 399 on the first two).
    if (tiles(128) >= 1200) return launch_gemm_f<MODE, 128, BT>(p, s);
    if (tiles(64) >= 1600) return launch_gemm_f<MODE, 64, BT>(p, s);
    return launch_gemm_f<MODE, 32, BT>(p, s);
  } else {
    static_assert(gemm_d_mode(MODE), "FP64 derivative rows: the sliced contraction");
    return launch_gemm_d<MODE>(p, s);
  }
}

// ----------------------------------------------------------------------------- hi + lo value rows
// FP32 and mixed paths: the value planes (one row per node) feed the orbital matrices, whose inverse amplifies
// their rounding by the condition number in the derivatives of log det.  Their contractions (k_gemm_comp below; for the dense
// layers of log|psi| alone k_gemm_sl, fire_sliced.cuh) give each dot product as a hi + lo float pair, as if summed in twice
// the working precision; the orbital-matrix values and the
// envelope values they are made of also leave as unevaluated pairs, so that the double-FP32 elimination sees them to
// ~2^-48.
//   COMP_PLAIN  C = a.b + bias (bias on rows with row % bias_period == 0)
//   COMP_SILU   C = silu(z), z = a.b + bias; with aux0 set also silu'(z) (aux0) and silu''(z) (aux2)
//   COMP_ENV    envelope value rows: hi into C, lo into C_lo [g][ld_lo]
//   COMP_ORB    orbital values (EPI_ORB_X): raw = a.b + bias (per-spin weights and bias), rawx (aux0) = raw,
//               C + C_lo = raw (env + env_lo) with env = aux1 [row * env_nv * ld_aux], env_lo [row * ld_lo]
enum CompMode { COMP_PLAIN = 0, COMP_SILU, COMP_ENV, COMP_ORB };

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

constexpr int CBM = 64, CBN = 64, CBK = 16, CTHREADS = 256;

// Grid of a column whose values are bounded by m >= 0: |b| < 2^eb (eb in [-100, 119]); sg = 3 * 2^eb, g = 2^(eb-22)
// (the spacing of the floats in [2^(eb+1), 2^(eb+2)]), sb16 = 16 bits(sg) (the offset of 16 summed products).
// A non-finite or huge bound gives NaN, which every output of the column then carries.
__device__ __forceinline__ void comp_grid_col(float m, float& sg, float& g, unsigned& sb16) {
  const int field = (__float_as_int(m) >> 23) & 0xff;
  int eb = field - 126;  // m < 2^(field - 126)
  if (eb < -100) eb = -100;
  if (field == 255 || eb > 119) {
    sg = g = __int_as_float(0x7fc00000);
    sb16 = 0u;
    return;
  }
  sg = 3.f * __int_as_float((eb + 127) << 23);
  g = __int_as_float((eb + 105) << 23);
  sb16 = 16u * (unsigned)__float_as_int(sg);
}

// Scale of a row tile whose values are bounded by m >= 0: inv = 2^-ea (|a| inv < 1), sc = 2^ea; a non-finite or
// huge bound gives NaN.
__device__ __forceinline__ void comp_grid_row(float m, float& inv, float& sc) {
  if (m == 0.f) {
    inv = sc = 1.f;
    return;
  }
  const int field = (__float_as_int(m) >> 23) & 0xff;
  int ea = field - 126;  // m < 2^ea
  if (ea < -125) ea = -125;
  if (field == 255 || ea > 126) {
    inv = sc = __int_as_float(0x7fc00000);
    return;
  }
  inv = __int_as_float((127 - ea) << 23);
  sc = __int_as_float((127 + ea) << 23);
}

// The CUDA-core form of the hi + lo value rows: all of a local energy's (Ctx::pair in fire_api.cu says why) and every
// envelope value row (stage_orbitals).  The exact part of every product is summed on a power-of-two grid instead of by a
// TwoSum per product (Ogita, Rump and Oishi's Dot2), in the spirit of Rump's error-free extraction against a fixed power of two:
//   - each column of B is bounded over the whole K by |b| < 2^eb, and each row of a staged 16-k tile of A is
//     scaled by a power of two so that |a'| < 1 (the row's scale 2^ea kept beside the tile);
//   - t = fma(a', b, 3 * 2^eb) then lies in [2^(eb+1), 2^(eb+2)], where floats are evenly spaced by G = 2^(eb-22),
//     so bits(t) - bits(3 * 2^eb) is the product rounded to that grid, counted in steps and summed exactly in a
//     32-bit integer (at most 16 * 2^22 per tile);
//   - fma(a', b, 3 * 2^eb - t) is the exact remainder below G / 2, summed in FP32;
//   - after each tile the step count leaves as xh + xl (xh its FP32 rounding, |xl| <= 2), and (xh G, xl G + rest),
//     scaled back by 2^ea, join a hi + lo pair by one TwoSum.
// The FP32 operations are packed two columns at a time (f32x2): six instructions for two products.
// 64 x 64 outputs per CTA, 4 x 4 per thread (rows 4 ty.., columns 4 tx..); A and B tiles of 16 k staged in shared
// memory (A transposed and scaled per row), the next tile prefetched into registers while the current one is
// summed.  Before the first tile every pass bounds its 64 columns of B over the whole K.
template <int MODE>
__device__ __forceinline__ void gemm_comp_tile(const GemmP<float>& p, float* __restrict__ C_lo,
                                               const float* __restrict__ env_lo, long ld_lo) {
  __shared__ __align__(16) float As[2][CBK][CBM];
  __shared__ __align__(16) float Bs[2][CBK][CBN];
  __shared__ __align__(16) float Asc[2][CBM];     // 2^ea of every row of the staged A tile
  __shared__ float Bmx[CTHREADS / 32][CBN];       // per-warp column maxima of |B|
  __shared__ __align__(16) float Csg[CBN];        // per column: 3 * 2^eb, the grid spacing 2^(eb-22), 16 bits(3 * 2^eb)
  __shared__ __align__(16) float Cg[CBN];
  __shared__ __align__(16) unsigned Cs16[CBN];
  int rows = p.M;
  if (p.M_dev) rows = min(rows, p.M_scale * (*p.M_dev));
  const int m0 = blockIdx.y * CBM, n0 = blockIdx.x * CBN;
  if (m0 >= rows) return;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  int passes = 1, first_spin = 0;
  if (p.B2) {  // per-spin weights: a pass per spin present in the tile
    int up = 0, dn = 0;
    if (tid < CBM && m0 + tid < rows) {
      if (((m0 + tid) % p.n_el) < p.n_up) up = 1; else dn = 1;
    }
    up = __syncthreads_or(up);
    dn = __syncthreads_or(dn);
    first_spin = up ? 0 : 1;
    passes = up + dn;
  }
  const int ar = tid >> 2, aq = (tid & 3) * 4;   // A: row ar, k aq..aq+3 of the tile
  const int bk = tid >> 4, bc = (tid & 15) * 4;  // B: k bk, columns bc..bc+3
  const bool va = p.lda % 4 == 0 && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int spin = first_spin + pass;
    const float* Bp = spin == 0 ? p.B : p.B2;
    const bool vb = p.ldb % 4 == 0 && (reinterpret_cast<uintptr_t>(Bp) & 15) == 0;
    // the bounds of this CTA's columns over the whole K: 16 threads per k row (4 columns each), k strided by 16
    {
      const int c4 = (tid & 15) * 4, gc = n0 + c4;
      float m[4] = {0.f, 0.f, 0.f, 0.f};
      if (vb && gc + 3 < p.N) {
#pragma unroll 4
        for (int k = tid >> 4; k < p.K; k += 16) {
          const float4 q = *reinterpret_cast<const float4*>(Bp + (long)k * p.ldb + gc);
          m[0] = fmaxf(m[0], fabsf(q.x));
          m[1] = fmaxf(m[1], fabsf(q.y));
          m[2] = fmaxf(m[2], fabsf(q.z));
          m[3] = fmaxf(m[3], fabsf(q.w));
        }
      } else {
        for (int k = tid >> 4; k < p.K; k += 16) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (gc + u < p.N) m[u] = fmaxf(m[u], fabsf(Bp[(long)k * p.ldb + gc + u]));
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        m[u] = fmaxf(m[u], __shfl_xor_sync(0xffffffffu, m[u], 16));  // the warp's two k rows
        if ((tid & 16) == 0) Bmx[tid >> 5][c4 + u] = m[u];
      }
    }
    __syncthreads();
    if (tid < CBN) {  // one column each; read after the barrier that follows the first tile's staging
      float m = 0.f;
#pragma unroll
      for (int w = 0; w < CTHREADS / 32; ++w) m = fmaxf(m, Bmx[w][tid]);
      comp_grid_col(m, Csg[tid], Cg[tid], Cs16[tid]);
    }
    float ra[4], rb[4];
    auto load = [&](int k0) {
      const int gr = m0 + ar, gk = k0 + aq;
      if (va && gr < rows && gk + 3 < p.K) {
        const float4 q = *reinterpret_cast<const float4*>(p.A + (long)gr * p.lda + gk);
        ra[0] = q.x; ra[1] = q.y; ra[2] = q.z; ra[3] = q.w;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) ra[u] = (gr < rows && gk + u < p.K) ? p.A[(long)gr * p.lda + gk + u] : 0.f;
      }
      const int gk2 = k0 + bk, gc = n0 + bc;
      if (vb && gk2 < p.K && gc + 3 < p.N) {
        const float4 q = *reinterpret_cast<const float4*>(Bp + (long)gk2 * p.ldb + gc);
        rb[0] = q.x; rb[1] = q.y; rb[2] = q.z; rb[3] = q.w;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) rb[u] = (gk2 < p.K && gc + u < p.N) ? Bp[(long)gk2 * p.ldb + gc + u] : 0.f;
      }
    };
    // A's 16 values of row ar are held by the 4 lanes tid ^ {0, 1, 2, 3}: their maximum scales the row
    auto store = [&](int buf) {
      float m = fmaxf(fmaxf(fabsf(ra[0]), fabsf(ra[1])), fmaxf(fabsf(ra[2]), fabsf(ra[3])));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      float inv, sc;
      comp_grid_row(m, inv, sc);
#pragma unroll
      for (int u = 0; u < 4; ++u) As[buf][aq + u][ar] = ra[u] * inv;
      if ((tid & 3) == 0) Asc[buf][ar] = sc;
      *reinterpret_cast<float4*>(&Bs[buf][bk][bc]) = make_float4(rb[0], rb[1], rb[2], rb[3]);
    };
    f32x2 hi[4][2], lo[4][2], rh[4][2];  // columns 2 j, 2 j + 1
    unsigned ti[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        hi[i][j >> 1] = lo[i][j >> 1] = rh[i][j >> 1] = 0ull;
        ti[i][j] = 0u;
      }
    load(0);
    store(0);
    __syncthreads();
    const ulonglong2 sg = *reinterpret_cast<const ulonglong2*>(&Csg[tx * 4]);
    const f32x2 minus1 = pack2(-1.f, -1.f);
    int buf = 0;
    for (int k0 = 0; k0 < p.K; k0 += CBK) {
      const bool more = k0 + CBK < p.K;
      if (more) load(k0 + CBK);
#pragma unroll 4
      for (int kk = 0; kk < CBK; ++kk) {
        const float4 a = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 aa = pack2(av[i], av[i]);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const f32x2 bj = j ? b.y : b.x, sj = j ? sg.y : sg.x;
            const f32x2 t = fma2(aa, bj, sj);  // the products on the grid, offset by 3 * 2^eb
            ti[i][2 * j] += (unsigned)t;
            ti[i][2 * j + 1] += (unsigned)(t >> 32);
            rh[i][j] = add2(rh[i][j], fma2(aa, bj, fma2(t, minus1, sj)));  // their exact remainders
          }
        }
      }
      // the tile's sums into the hi + lo pairs: the step count d (< 2^26) as its FP32 rounding xh plus xl (|xl| <= 2).  d is
      // converted in two exact halves (2^12 dh + dl) through the floats' own grid at 1.5 2^23: an integer-to-float
      // conversion, rounded to nearest like fma(dh, 2^12, dl), runs at a fraction of the rate.
      {
        const float4 s4 = *reinterpret_cast<const float4*>(&Asc[buf][ty * 4]);
        const ulonglong2 g4 = *reinterpret_cast<const ulonglong2*>(&Cg[tx * 4]);
        const uint4 o4 = *reinterpret_cast<const uint4*>(&Cs16[tx * 4]);
        const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
        const unsigned sb16[4] = {o4.x, o4.y, o4.z, o4.w};
        const f32x2 magic = pack2(-12582912.f, -12582912.f), k4096 = pack2(4096.f, 4096.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 sc = pack2(sv[i], sv[i]);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int d0 = (int)(ti[i][2 * j] - sb16[2 * j]), d1 = (int)(ti[i][2 * j + 1] - sb16[2 * j + 1]);
            const f32x2 dh = add2(pack2(__int_as_float(0x4b400000 + (d0 >> 12)), __int_as_float(0x4b400000 + (d1 >> 12))), magic);
            const f32x2 dl =
                add2(pack2(__int_as_float(0x4b400000 + (d0 & 4095)), __int_as_float(0x4b400000 + (d1 & 4095))), magic);
            const f32x2 gg = j ? g4.y : g4.x;
            const f32x2 xh = fma2(dh, k4096, dl);
            const f32x2 xl = add2(fma2(dh, k4096, mul2(xh, minus1)), dl);
            const f32x2 uh = mul2(mul2(xh, gg), sc);
            const f32x2 ul = mul2(fma2(xl, gg, rh[i][j]), sc);
            const f32x2 h = hi[i][j], s2 = add2(h, uh);  // two_sum(hi, uh)
            const f32x2 bb = fma2(h, minus1, s2);
            const f32x2 e = add2(fma2(fma2(bb, minus1, s2), minus1, h), fma2(bb, minus1, uh));
            hi[i][j] = s2;
            lo[i][j] = add2(lo[i][j], add2(e, ul));
            ti[i][2 * j] = ti[i][2 * j + 1] = 0u;
            rh[i][j] = 0ull;
          }
        }
      }
      if (more) {
        store(buf ^ 1);
        __syncthreads();
        buf ^= 1;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = m0 + ty * 4 + i;
      if (row >= rows) continue;
      if (p.B2 && (((row % p.n_el) < p.n_up) ? 0 : 1) != spin) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = n0 + tx * 4 + j;
        if (col >= p.N) continue;
        float h, l, other;
        if (j & 1) {
          unpack2(hi[i][j >> 1], other, h);
          unpack2(lo[i][j >> 1], other, l);
        } else {
          unpack2(hi[i][j >> 1], h, other);
          unpack2(lo[i][j >> 1], l, other);
        }
        if (MODE == COMP_PLAIN || MODE == COMP_SILU || MODE == COMP_ORB) {
          const float* bias = (MODE == COMP_ORB && spin == 1) ? p.bias2 : p.bias;
          const bool has_b = bias && (MODE != COMP_PLAIN || (p.bias_period > 0 && row % p.bias_period == 0));
          if (has_b) {
            float s2, e;
            two_sum(h, bias[col], s2, e);
            h = s2;
            l += e;
          }
        }
        float s2, e;  // normalised pair: s2 = fl(h + l)
        two_sum(h, l, s2, e);
        if (MODE == COMP_PLAIN) {
          p.C[(long)row * p.ldc + col] = s2;
        } else if (MODE == COMP_SILU) {
          p.C[(long)row * p.ldc + col] = silu(s2);
          if (p.aux0) {
            float y, d1, d2;
            silu3(s2, y, d1, d2);
            p.aux0[(long)row * p.ld_aux + col] = d1;
            p.aux2[(long)row * p.ld_aux + col] = d2;
          }
        } else if (MODE == COMP_ENV) {
          const int g = (row / p.env_ns) * p.n_el + p.env_soff + row % p.env_ns;
          p.C[(long)g * p.ldc + col] = s2;
          C_lo[(long)g * ld_lo + col] = e;
        } else {  // COMP_ORB
          p.aux0[(long)row * p.ld_aux + col] = s2;
          const float eh = p.aux1[(long)row * p.env_nv * p.ld_aux + col], el = env_lo[(long)row * ld_lo + col];
          const float ph = s2 * eh;
          const float pl = fmaf(s2, eh, -ph) + (s2 * el + e * eh);
          float oh, ol;
          two_sum(ph, pl, oh, ol);
          p.C[(long)row * p.ldc + col] = oh;
          C_lo[(long)row * ld_lo + col] = ol;
        }
      }
    }
    if (pass + 1 < passes) __syncthreads();
  }
}

template <int MODE>
__global__ void __launch_bounds__(CTHREADS, 2) k_gemm_comp(GemmP<float> p, float* __restrict__ C_lo,
                                                           const float* __restrict__ env_lo, long ld_lo) {
  gemm_comp_tile<MODE>(p, C_lo, env_lo, ld_lo);
}
// Envelope value rows (COMP_ENV) of both spins and every determinant: blockIdx.z = spin NDET + determinant, whose
// coefficients, weights and columns of C and C_lo lie a_bs[spin], b_bs and c_bs elements further on.
struct CompEnvP {
  GemmP<float> p[2];
  long a_bs[2], b_bs, c_bs;
};
template <int V = 0>  // a template so that every translation unit that includes this header may hold it
__global__ void __launch_bounds__(CTHREADS, 2) k_gemm_comp_env(CompEnvP q, float* __restrict__ C_lo, long ld_lo) {
  const int s = blockIdx.z / NDET, d = blockIdx.z % NDET;
  GemmP<float> p = s == 0 ? q.p[0] : q.p[1];
  p.A += d * (s == 0 ? q.a_bs[0] : q.a_bs[1]);
  p.B += d * q.b_bs;
  p.C += d * q.c_bs;
  gemm_comp_tile<COMP_ENV>(p, C_lo + d * q.c_bs, nullptr, ld_lo);
}

// Envelope value rows of the refinement pass (EPI_ENV's row map, env_nv = 1) on the FP32 pipes: A holds FP64
// coefficients, B weights whose values are exact in FP32 (the float32 parameter blob's), C is FP64.  Each a is split
// into a_hi + a_lo floats; a_hi b by Dot2 (as in k_gemm_comp), a_lo b by FP32 FMAs into the low accumulator, and the
// result hi + lo leaves as a double: ~2^-44 of the terms' magnitude, where the FP64 pipe (~1/64 of the FP32 rate)
// would spend most of the pass.
template <int V = 0>  // a template so that every translation unit that includes this header may hold it
__global__ void __launch_bounds__(CTHREADS) k_gemm_env_df(GemmP<double> p) {
  __shared__ __align__(16) float Ah[2][CBK][CBM];
  __shared__ __align__(16) float Al[2][CBK][CBM];
  __shared__ __align__(16) float Bs[2][CBK][CBN];
  int rows = p.M;
  if (p.M_dev) rows = min(rows, p.M_scale * (*p.M_dev));
  const int m0 = blockIdx.y * CBM, n0 = blockIdx.x * CBN;
  if (m0 >= rows) return;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int ar = tid >> 2, aq = (tid & 3) * 4;   // A: row ar, k aq..aq+3 of the tile
  const int bk = tid >> 4, bc = (tid & 15) * 4;  // B: k bk, columns bc..bc+3
  double ra[4];
  float rb[4];
  auto load = [&](int k0) {
    const int gr = m0 + ar, gk = k0 + aq;
#pragma unroll
    for (int u = 0; u < 4; ++u) ra[u] = (gr < rows && gk + u < p.K) ? p.A[(long)gr * p.lda + gk + u] : 0.0;
    const int gk2 = k0 + bk, gc = n0 + bc;
#pragma unroll
    for (int u = 0; u < 4; ++u) rb[u] = (gk2 < p.K && gc + u < p.N) ? (float)p.B[(long)gk2 * p.ldb + gc + u] : 0.f;
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float h = __double2float_rn(ra[u]);
      Ah[buf][aq + u][ar] = h;
      Al[buf][aq + u][ar] = __double2float_rn(ra[u] - (double)h);
    }
    *reinterpret_cast<float4*>(&Bs[buf][bk][bc]) = make_float4(rb[0], rb[1], rb[2], rb[3]);
  };
  float hi[4][4], lo[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) hi[i][j] = lo[i][j] = 0.f;
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < p.K; k0 += CBK) {
    const bool more = k0 + CBK < p.K;
    if (more) load(k0 + CBK);
#pragma unroll 4
    for (int kk = 0; kk < CBK; ++kk) {
      const float4 a = *reinterpret_cast<const float4*>(&Ah[buf][kk][ty * 4]);
      const float4 al = *reinterpret_cast<const float4*>(&Al[buf][kk][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, alv[4] = {al.x, al.y, al.z, al.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float pr = av[i] * bv[j];
          const float pe = fmaf(av[i], bv[j], -pr);
          float s2, e;
          two_sum(hi[i][j], pr, s2, e);
          hi[i][j] = s2;
          lo[i][j] = fmaf(alv[i], bv[j], lo[i][j] + (e + pe));
        }
    }
    if (more) {
      store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + ty * 4 + i;
    if (row >= rows) continue;
    const int g = (row / p.env_ns) * p.n_el + p.env_soff + row % p.env_ns;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = n0 + tx * 4 + j;
      if (col < p.N) p.C[(long)g * p.ldc + col] = (double)hi[i][j] + (double)lo[i][j];
    }
  }
}

inline cudaError_t launch_gemm_env_df(const GemmP<double>& p, cudaStream_t s) {
  dim3 grid((p.N + CBN - 1) / CBN, (p.M + CBM - 1) / CBM);
  if (grid.y == 0 || grid.x == 0) return cudaSuccess;
  k_gemm_env_df<0><<<grid, CTHREADS, 0, s>>>(p);
  return cudaPeekAtLastError();
}

template <int MODE>
inline cudaError_t launch_gemm_comp(const GemmP<float>& p, float* C_lo, const float* env_lo, long ld_lo,
                                    cudaStream_t s) {
  dim3 grid((p.N + CBN - 1) / CBN, (p.M + CBM - 1) / CBM);
  if (grid.y == 0 || grid.x == 0) return cudaSuccess;
  k_gemm_comp<MODE><<<grid, CTHREADS, 0, s>>>(p, C_lo, env_lo, ld_lo);
  return cudaPeekAtLastError();
}

inline cudaError_t launch_gemm_comp_env(const CompEnvP& q, float* C_lo, long ld_lo, cudaStream_t s) {
  const int M = q.p[0].M > q.p[1].M ? q.p[0].M : q.p[1].M;
  const dim3 grid((q.p[0].N + CBN - 1) / CBN, (M + CBM - 1) / CBM, 2 * NDET);
  if (grid.y == 0 || grid.x == 0) return cudaSuccess;
  k_gemm_comp_env<0><<<grid, CTHREADS, 0, s>>>(q, C_lo, ld_lo);
  return cudaPeekAtLastError();
}

}  // namespace fire
