// fire_det.cu -- orbital envelopes, slogdet/inverse of the orbital matrices and the sparse
// determinant Laplacian.
//
//  k_env_coef   forward-Laplacian coefficients of exp(-softplus(sigma) |r - R|) per electron,
//               nucleus, determinant and envelope (EfficientIsotropicEnvelopes, envelopes.py:55-82);
//               a GEMM with pi then gives the envelope carrier [x, jac(3), lap] per orbital.
//  k_gj_global  sign/log|det| and (optionally) the inverse of every orbital matrix, computed in
//               double precision (native FP64 in the FP64 build, double-FP32 "df64" with a 48-bit
//               significand in the FP32 and mixed paths, fire_df64.cuh; the value-only path's LU in
//               FP32), one CTA per matrix with the working matrix in the workspace, eliminated in
//               panels.  Partial pivoting like jax.lax.linalg.lu, sign/log|det| as slogdet_from_lu
//               (model/utils.py:153-161), inverse as get_inverse_from_lu (144-150).
//  k_detlap     sparse_slogdet_with_fwd_lap (model/sparse_fwd_lap.py:294-319) restricted to the
//               triplets: for every dependency m, B = J[(i, m) rows] @ A^-1[:, k] for i, k in {m} + N(m)
//               gives d log det / d r_m = sum_i B[(i,m)][i] and the triplet term
//               -sum_xyz sum_{i,k} B[(i,m)][k] B[(k,m)][i]; the first Laplacian term tr(lap A A^-1) is
//               accumulated row by row.
#include <type_traits>

#include "fire_df64.cuh"
#include "fire_f32x2.cuh"
#include "fire_internal.cuh"

namespace fire {

// coef layout: [det][rows = (w * n_s + i) * NV + v][N * 8]
template <typename T, int NV>
__global__ void k_env_coef(const T* __restrict__ r, const float* __restrict__ R, const T* __restrict__ sp,
                           int n, int n_s, int s_off, int N, int Wn, T* __restrict__ coef,
                           const int* __restrict__ live) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;  // over (w * n_s + i, I, k)
  const long total = (long)Wn * n_s * N * NENV_ORB;
  if (idx >= total) return;
  const int k = (int)(idx % NENV_ORB);
  const int I = (int)((idx / NENV_ORB) % N);
  const long rr = idx / ((long)NENV_ORB * N);
  const int w = (int)(rr / n_s), i = (int)(rr % n_s);
  if (live && w >= *live) return;
  const long g = (long)w * n + s_off + i;
  const T dx = r[3 * g] - (T)R[3 * I], dy = r[3 * g + 1] - (T)R[3 * I + 1], dz = r[3 * g + 2] - (T)R[3 * I + 2];
  const T rho = dsqrt(dx * dx + dy * dy + dz * dz);
  const T irho = T(1) / rho;
  const long rows = (long)Wn * n_s * NV;
  const int K8 = N * NENV_ORB;
#pragma unroll
  for (int d = 0; d < NDET; ++d) {
    const T a = sp[(I * NDET + d) * NENV_ORB + k];
    const T e = dexp(-a * rho);
    T* out = coef + (long)d * rows * K8 + (rr * NV) * K8 + I * NENV_ORB + k;
    out[0] = e;
    if (NV > 1) {
      const T gj = -a * e * irho;
      out[K8] = gj * dx;
      out[2 * K8] = gj * dy;
      out[3 * K8] = gj * dz;
      out[4 * K8] = e * (a * a - T(2) * a * irho);
    }
  }
}

// Two adjacent columns' SubDot sums against one row's factors; Y holds the columns' factors of one term, read with one
// 16-byte load (8 bytes for float) from an aligned pair.
template <typename S>
struct PairDot {
  struct Y {
    S y0, y1;
    __device__ __forceinline__ explicit Y(const S* p) : y0(p[0]), y1(p[1]) {}
  };
  SubDot<S> d0, d1;
  __device__ __forceinline__ void add(S w, const Y& y) {
    d0.add(w, y.y0);
    d1.add(w, y.y1);
  }
  __device__ __forceinline__ S finish0(S a) const { return d0.finish(a); }
  __device__ __forceinline__ S finish1(S a) const { return d1.finish(a); }
};
// double-FP32: SubDot<df64>'s operations on packed pairs, in the same order and with the same roundings.  The packed
// instructions have no operand negation, so the sums run with the opposite sign (ns = -s; rounding to nearest is symmetric)
// and differences are a - b = fma(b, -1, a).  Columns staged as (hi0, hi1, lo0, lo1).
template <>
struct PairDot<df64> {
  struct Y {
    f32x2 hi, lo;
    __device__ __forceinline__ explicit Y(const df64* p) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
      hi = v.x;
      lo = v.y;
    }
  };
  f32x2 ns, c;
  __device__ __forceinline__ PairDot() : ns(0x8000000080000000ull), c(0ull) {}
  __device__ __forceinline__ void add(df64 w, const Y& y) {
    const f32x2 m1 = pack2(-1.f, -1.f), wh = pack2(w.hi, w.hi), wl = pack2(w.lo, w.lo), nwh = pack2(-w.hi, -w.hi);
    const f32x2 np = mul2(nwh, y.hi);      // -p
    const f32x2 e = fma2(wh, y.hi, np);    // the product's exact low part
    c = fma2(wh, y.lo, c);
    c = fma2(wl, y.hi, c);
    const f32x2 ns1 = add2(ns, np);        // -(s + p)
    const f32x2 nbb = fma2(ns, m1, ns1);
    const f32x2 nq = add2(fma2(fma2(nbb, m1, ns1), m1, ns), fma2(nbb, m1, np));  // -(TwoSum error)
    c = add2(c, fma2(nq, m1, e));
    ns = ns1;
  }
  __device__ __forceinline__ df64 finish(df64 a, float nsx, float cx) const {
    const df64 r = df_two_sum(a.hi, nsx);
    return df_two_sum(r.hi, __fadd_rn(r.lo, __fsub_rn(a.lo, cx)));
  }
  __device__ __forceinline__ df64 finish0(df64 a) const {
    float n0, n1, c0, c1;
    unpack2(ns, n0, n1);
    unpack2(c, c0, c1);
    return finish(a, n0, c0);
  }
  __device__ __forceinline__ df64 finish1(df64 a) const {
    float n0, n1, c0, c1;
    unpack2(ns, n0, n1);
    unpack2(c, c0, c1);
    return finish(a, n1, c1);
  }
};

__device__ __forceinline__ uint32_t smem_u32_det(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

constexpr int GJG_BW = 16, GJG_THREADS = 512;

// Gauss-Jordan inversion / LU with partial pivoting, one matrix per CTA, the working matrix in global
// memory (the caller's workspace, row-major [n][n] in the elimination type S) instead of shared memory, so
// that every matrix of the batch is in flight at once (two CTAs per SM) and the kernel is bound by
// arithmetic, not by the latency of n dependent steps.  Columns are eliminated in panels of GJG_BW:
//  1. the panel is loaded into shared memory and factored there, recording the pivot row p_t of every
//     step and the step's transform x <- x - w_t x[k_t] of any other column x (w_t kept in the final row
//     order of the panel: later interchanges are applied to it as well);
//  2. W~ = W L^-1 with L[t][s] = w_s[k_t] (unit lower triangular), so that the whole panel acts on another
//     column as: interchange rows k_t <-> p_t, then x <- x - W~ x[k_0 .. k_{b-1}];
//  3. every other column (LU: every column right of the panel) is streamed through shared memory in chunks
//     of GJG_BW columns and updated with that rank-b product.
// A: element (i, o) of matrix (w, d) at A[((w * n + i) * NDET + d) * n + o]  (the orbital plane [G][D * n]);
// A_lo (double-FP32 elimination only, may be null): the low parts of the same elements.
// The block has 32 to 512 threads (launch_gjg): n steps with three barriers each leave a small matrix waiting, so small
// matrices take small blocks and more of them share an SM.  The double-FP32 update packs two columns (PairDot: 12 packed
// operations for two products; it is bound by their issue rate).  LU of 1024 matrices of 82: 1.53 ms with 512 threads each,
// the logarithm of every pivot inside its step and scalar arithmetic.
// Outputs: logdet[w * NDET + d], sign[...] (double); if INV the inverse, transposed and aligned for
// k_detlap: Ainv[((w * NDET + d) * n + i) * ainv_ld(n) + sh + o] = (A^-1)[o][i] with sh = (d n) mod 4 and zeros
// in the other entries of the row, written after undoing the column permutation; if INV and cond is not null,
// cond[w * NDET + d] = ||A||_F ||A^-1||_F (the Frobenius condition number, >= the 2-norm one).
template <typename S, typename TI, typename TO, bool INV>
__global__ void __launch_bounds__(GJG_THREADS, 2) k_gj_global(const TI* __restrict__ A, const TI* __restrict__ A_lo,
                                                             int n, S* __restrict__ work,
                                                             double* __restrict__ logdet, double* __restrict__ sign,
                                                             double* __restrict__ cond, TO* __restrict__ Ainv,
                                                             const int* __restrict__ live, int32_t* status) {
  extern __shared__ __align__(16) unsigned char gj_smem[];
  constexpr int BW = GJG_BW, LD = GJG_BW + 1;  // shared rows padded: column walks spread over the banks
  const int mat = blockIdx.x;
  const int w = mat / NDET, d = mat - w * NDET;
  if (live && w >= *live) return;
  // two working copies per matrix: every panel reads one and writes the other
  S* Mb[2] = {work + (size_t)mat * n * n, work + ((size_t)gridDim.x + mat) * n * n};
  S* pan = reinterpret_cast<S*>(gj_smem);  // [n][LD] the panel, then each chunk of other columns
  S* W = pan + (size_t)n * LD;             // [n][LD] panel transforms (then W~)
  S* Li = W + (size_t)n * LD;              // [BW][BW] L^-1
  S* colk = Li + BW * BW;                  // [n] pivot column before the step (interchanged order)
  S* rk = colk + n;                        // [BW] row k of the panel before the step
  S* rp = rk + BW;                         // [BW] row p
  S* rj = rp + BW;                         // [BW] row p scaled by the inverse pivot
  int* perm = reinterpret_cast<int*>(rj + BW);  // [n]
  int* piv = perm + n;                     // [BW]
  int* rowmap = piv + BW;                  // [n] source row of every row after the panel's interchanges
  static_assert(sizeof(S) == 8, "redv doubles as the double reduction buffer");
  __shared__ __align__(8) S redv[32];
  __shared__ int redi[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarp = blockDim.x >> 5;
  double sq = 0.0;  // ||A||_F^2, then ||A^-1||_F^2 (condition number output)
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int i = e / n, o = e - i * n;
    const long ia = ((long)(w * n + i) * NDET + d) * n + o;
    const TI a = A[ia];
    if constexpr (std::is_same<S, df64>::value && std::is_same<TI, float>::value)
      Mb[0][e] = A_lo ? df64(a, A_lo[ia]) : S(a);  // the compensated orbital values: a normalised hi + lo pair
    else
      Mb[0][e] = (S)a;
    sq += (double)a * (double)a;
  }
  // the block sums of the condition number go through redv (8-byte elements; no static shared memory is added,
  // so that the largest matrix still fits): thread 0 keeps ||A||_F^2
  double* redd = reinterpret_cast<double*>(redv);
  double a2 = 0.0;
  if (INV && cond) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) redd[wid] = sq;
    sq = 0.0;
  }
  __syncthreads();
  if (INV && cond && tid == 0)  // before the first panel's barrier, after which redv is written again
    for (int q = 0; q < nwarp; ++q) a2 += redd[q];
  double ld = 0.0;
  int neg = 0, sing = 0;
  // the pivots, one per thread and round of steps (n <= 2 blockDim): their logarithms are taken together at the end
  double pv_keep[2] = {1.0, 1.0};
  const int npan = (n + BW - 1) / BW;
  const int cj = tid % BW, rg = tid / BW, rn = blockDim.x / BW;  // chunk update: column, row group
  // panel update: row, and its share of the columns when the block has several threads per row
  const int nr32 = (n + 31) & ~31, ncg = max(1, (int)blockDim.x / nr32), cg = tid / nr32, prow = tid % nr32;
  for (int P = 0; P < npan; ++P) {
    const int k0 = P * BW, bw = min(BW, n - k0);
    const S* src = Mb[P & 1];
    S* dst = Mb[(P + 1) & 1];
    if (cj < bw)
      for (int i = rg; i < n; i += rn) pan[i * LD + cj] = src[(size_t)i * n + k0 + cj];
    for (int i = tid; i < n; i += blockDim.x) rowmap[i] = i;
    __syncthreads();
    // ---- factor the panel
    for (int t = 0; t < bw; ++t) {
      const int k = k0 + t;
      S best = S(-1);
      int bi = n;
      for (int i = k + tid; i < n; i += blockDim.x) {
        const S v = absv(pan[i * LD + t]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const S ov = shfl_xor_any(best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
          best = ov;
          bi = oi;
        }
      }
      if (lane == 0) {
        redv[wid] = best;
        redi[wid] = bi;
      }
      __syncthreads();
      S bv = redv[lane & (nwarp - 1)];  // nwarp is a power of two
      int p = redi[lane & (nwarp - 1)];
      for (int o = nwarp >> 1; o > 0; o >>= 1) {
        const S ov = shfl_xor_any(bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, p, o);
        if (ov > bv || (ov == bv && oi < p)) {
          bv = ov;
          p = oi;
        }
      }
      if (p >= n) p = k;
      const S pv = pan[p * LD + t];
      if (tid == k % (int)blockDim.x) pv_keep[k / (int)blockDim.x] = (double)pv;
      if (wid == 0) {  // the inverse pivot (31: beyond the warps' entries) and the scaled pivot row
        const S iv = pv != S(0) ? S(1) / pv : S(0);
        if (lane == 0) {
          redv[31] = iv;
          piv[t] = p;
          perm[k] = p;
          if (pv == S(0)) sing = 1;
          if (pv < S(0)) neg ^= 1;
          if (p != k) neg ^= 1;
        }
        if (lane < bw) {
          const S y = pan[p * LD + lane];
          rk[lane] = pan[k * LD + lane];
          rp[lane] = y;
          rj[lane] = y * iv;
        }
      }
      for (int i = (INV ? 0 : k) + tid; i < n; i += blockDim.x) colk[i] = pan[(i == k ? p : (i == p ? k : i)) * LD + t];
      if (p != k)  // earlier transforms follow the interchange
        for (int s2 = tid; s2 < t; s2 += blockDim.x) {
          const S tk = W[k * LD + s2];
          W[k * LD + s2] = W[p * LD + s2];
          W[p * LD + s2] = tk;
        }
      __syncthreads();
      const S ipv = redv[31];
      // Gauss-Jordan: every row of the panel columns not yet eliminated (the eliminated ones are rebuilt from W~ after
      // the panel).  LU: rows k.. of the panel columns right of the pivot (rows above k do not change).
      if (cg < ncg)
        for (int i = prow; i < n; i += nr32 > (int)blockDim.x ? (int)blockDim.x : nr32) {
          S* row = pan + i * LD;
          const S ci = INV || i >= k ? colk[i] : S(0);
          const S ml = INV ? ci : (i > k ? ci * ipv : S(0));
          if (INV) {
            for (int j2 = t + 1 + cg; j2 < bw; j2 += ncg)
              row[j2] = i == k ? rj[j2] : df_sub_mul(i == p ? rk[j2] : row[j2], ml, rj[j2]);
          } else if (i >= k) {
            for (int j2 = t + 1 + cg; j2 < bw; j2 += ncg) {
              const S old = i == k ? rp[j2] : (i == p ? rk[j2] : row[j2]);
              row[j2] = i > k ? df_sub_mul(old, ml, rp[j2]) : old;
            }
          }
          if (cg == 0) W[i * LD + t] = INV ? (i == k ? S(1) - ipv : ci * ipv) : ml;
        }
      __syncthreads();
    }
    // ---- L^-1 (one lane per column s: Li[t][s] = -sum_{u=s}^{t-1} L[t][u] Li[u][s]) and W~ = W L^-1
    if (tid < bw) {
      for (int t = 0; t < bw; ++t) {
        SubDot<S> acc;
        for (int u = tid; u < t; ++u) acc.add(W[(k0 + t) * LD + u], Li[u * BW + tid]);
        Li[t * BW + tid] = acc.finish(t == tid ? S(1) : S(0));
      }
    }
    if (tid == 0) {  // the panel's row interchanges as one permutation
      for (int t = 0; t < bw; ++t) {
        const int q = piv[t];
        const int tmp = rowmap[k0 + t];
        rowmap[k0 + t] = rowmap[q];
        rowmap[q] = tmp;
      }
    }
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) {
      S wr[BW];
#pragma unroll
      for (int q = 0; q < BW; ++q) wr[q] = q < bw ? W[i * LD + q] : S(0);
#pragma unroll
      for (int t = 0; t < BW; ++t) {
        if (t >= bw) break;
        SubDot<S> acc;
#pragma unroll
        for (int q = 0; q < BW; ++q)
          if (q >= t && q < bw) acc.add(wr[q], Li[q * BW + t]);
        W[i * LD + t] = acc.sum();
      }
    }
    __syncthreads();
    if (INV && cj < bw)  // the panel's final columns, e_{k0+s} - W~[:, s] (the LU never reads finished panels)
      for (int i = rg; i < n; i += rn) dst[(size_t)i * n + k0 + cj] = (i == k0 + cj ? S(1) : S(0)) - W[i * LD + cj];
    // ---- apply the panel to the other columns (LU: the columns right of the panel, rows from k0):
    // x <- x - W~ y with y the panel's pivot rows of x.  Y (the bw pivot rows of every column, interchanged
    // order, rows padded to an even length) is staged over the panel buffer, which is free now; each thread
    // owns a pair of adjacent columns and walks its rows two at a time (2 x 2 tiles: three shared loads per
    // four products), reading the interchanged rows of src and writing dst (no in-place hazard).
    // For double-FP32 a pair of columns is staged as (hi, hi, lo, lo), the operands of the packed update.
    S* Y = pan;
    const int ldy = n + (n & 1);
    for (int t = 0; t < bw; ++t) {
      const S* yr = src + (size_t)rowmap[k0 + t] * n;
      for (int c = (INV ? 0 : k0 + bw) + tid; c < n; c += blockDim.x) {
        if constexpr (std::is_same<S, df64>::value) {
          const df64 y = yr[c];
          float* q = reinterpret_cast<float*>(Y + t * ldy + (c & ~1)) + (c & 1);
          q[0] = y.hi;
          q[2] = y.lo;
        } else {
          Y[t * ldy + c] = yr[c];
        }
      }
    }
    __syncthreads();
    {
      const int cp = tid & 15, rg = tid >> 4, rn2 = blockDim.x >> 4;  // column pair, row group
      const int i0 = INV ? 0 : k0;
      for (int c = (INV ? 0 : k0 + bw) + 2 * cp; c < n; c += 32) {
        if (INV && c >= k0 && c < k0 + bw) continue;  // the panel's own columns (pairs never straddle it)
        const bool c1 = c + 1 < n;
        int i = i0 + rg;
        for (; i + rn2 < n; i += 2 * rn2) {
          const S* s0 = src + (size_t)rowmap[i] * n + c;
          const S* s1 = src + (size_t)rowmap[i + rn2] * n + c;
          const S a00 = s0[0], a10 = s1[0];
          const S a01 = c1 ? s0[1] : S(0), a11 = c1 ? s1[1] : S(0);
          const S *w0 = W + i * LD, *w1 = W + (i + rn2) * LD;
          PairDot<S> d0, d1;
          if (bw == BW) {
#pragma unroll
            for (int t = 0; t < BW; ++t) {
              const typename PairDot<S>::Y y(Y + t * ldy + c);
              d0.add(w0[t], y);
              d1.add(w1[t], y);
            }
          } else {
            for (int t = 0; t < bw; ++t) {
              const typename PairDot<S>::Y y(Y + t * ldy + c);
              d0.add(w0[t], y);
              d1.add(w1[t], y);
            }
          }
          S* o0 = dst + (size_t)i * n + c;
          S* o1 = dst + (size_t)(i + rn2) * n + c;
          o0[0] = d0.finish0(a00);
          o1[0] = d1.finish0(a10);
          if (c1) {
            o0[1] = d0.finish1(a01);
            o1[1] = d1.finish1(a11);
          }
        }
        if (i < n) {
          const S* s0 = src + (size_t)rowmap[i] * n + c;
          const S a00 = s0[0], a01 = c1 ? s0[1] : S(0);
          const S* w0 = W + i * LD;
          PairDot<S> d0;
          for (int t = 0; t < bw; ++t) d0.add(w0[t], typename PairDot<S>::Y(Y + t * ldy + c));
          S* o0 = dst + (size_t)i * n + c;
          o0[0] = d0.finish0(a00);
          if (c1) o0[1] = d0.finish1(a01);
        }
      }
    }
    __syncthreads();  // dst complete before the next panel reads it
  }
  {
    double* lg = reinterpret_cast<double*>(pan);
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (tid + q * (int)blockDim.x < n) lg[tid + q * blockDim.x] = ::log(::fabs(pv_keep[q]));
    __syncthreads();
    if (tid == 0)
      for (int k = 0; k < n; ++k) ld += lg[k];
    __syncthreads();  // the panel buffer is staged over next
  }
  if (tid == 0) {
    logdet[mat] = ld;
    sign[mat] = neg ? -1.0 : 1.0;
    if (sing) set_flag(status, FIRE_FLAG_SINGULAR);
  }
  if (INV) {
    // undo the row interchanges on the columns: final column jc holds working column src(jc)
    int* srcc = reinterpret_cast<int*>(colk);
    for (int q = tid; q < n; q += blockDim.x) srcc[q] = q;
    __syncthreads();
    if (tid == 0) {
      for (int k = n - 1; k >= 0; --k) {
        const int p = perm[k];
        if (p != k) {
          const int t = srcc[k];
          srcc[k] = srcc[p];
          srcc[p] = t;
        }
      }
    }
    __syncthreads();
    // transposed output, row i = column i of the inverse, shifted by the determinant's offset sh within the
    // orbital plane and zero-padded (see ainv_ld): 32 rows of the working matrix at a time are staged in
    // shared memory (the panel buffers are free) so that both the reads and the writes are row-contiguous
    const int nA = ainv_ld(n), sh = (d * n) & 3;
    TO* out = Ainv + (size_t)mat * n * nA;
    const S* M = Mb[npan & 1];
    S* tile = pan;  // [32][n]
    for (int o0 = 0; o0 < n; o0 += 32) {
      const int ro = min(32, n - o0);
      for (int e = tid; e < ro * n; e += blockDim.x) {
        const S v = M[(size_t)o0 * n + e];
        tile[e] = v;
        sq += (double)v * (double)v;
      }
      __syncthreads();
      for (int e = tid; e < n * 32; e += blockDim.x) {
        const int i = e >> 5, r = e & 31;
        if (r < ro) out[(size_t)i * nA + sh + o0 + r] = (TO)tile[r * n + srcc[i]];
      }
      __syncthreads();
    }
    const int npad = nA - n;
    for (int e = tid; e < n * npad; e += blockDim.x) {
      const int i = e / npad, q = e - i * npad;
      out[(size_t)i * nA + (q < sh ? q : n + q)] = TO(0);
    }
    if (cond) {  // kappa_F = ||A||_F ||A^-1||_F
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane == 0) redd[wid] = sq;
      __syncthreads();
      if (tid == 0) {
        double b2 = 0.0;
        for (int q = 0; q < nwarp; ++q) b2 += redd[q];
        cond[mat] = sqrt(a2 * b2);
      }
    }
  }
}

// Determinant Laplacian for one (walker, det, dependency m).  Jp: orbital Jacobian plane
// [3 * positions][NDET * n]; AinvT: the transposed, shifted inverse written by k_gj_global; lapA [G][NDET * n].
// Outputs: grad [W][NDET][n][3], lap [W * NDET] (double, +=).
// B = J[(i, m) rows] (3c x n) @ A^-1[:, {i}] (n x c): both operands are read along the contraction index o
// (J rows and rows of the transposed inverse), in 16-byte quads of x = o + sh where sh = (d n) mod 4 makes the
// J rows of determinant d 16-byte aligned; the inverse rows carry the same shift and zeros outside o in [0, n),
// which cancel the neighbouring columns the J quads pick up.  Chunks of DL_OC x are copied asynchronously
// (cp.async) into a ring of DL_STAGES shared-memory buffers, rows of DL_LD elements; each thread accumulates one TH x 4 tile
// whose rows (r, r + TR, r + 2 TR, ...) and columns (k, k + TC, ...) are strided, so that a warp's 16-byte
// loads hit consecutive rows, no bank conflicts.  The result tile reuses the staging memory.
// TH is the smallest height with a tile per thread at most: with 4 x 4 tiles, 25 positions made 133 tiles of 128 threads,
// so that one scheduler ran two rounds, and 10 positions 24 tiles of 256 (FP64).  The triplet sums were bound by the FP64
// pipe (two conversions and a product per element at 2 per cycle and SM): of FP32 factors they are now exact three-term
// FP32 expansions.  Before / after, 341 walkers of 82 electrons (25 positions each): 3710 -> 2970 us;
// 171 walkers of 322: 5440 -> 4270; FP64, 512 walkers of 10 electrons: 2790 -> 327.
static_assert(3 * DL_CMAX * (DL_CMAX + 1) <= dl_smem_elems(DL_CMAX), "result tile inside the staging buffers");
static_assert(3 * DL_DSPLIT * (DL_DSPLIT + 1) <= dl_smem_elems(DL_DSPLIT), "result tile inside the staging buffers");
static_assert(3 * DL_CSPLIT * (DL_CSPLIT + 1) <= dl_smem_elems(DL_CSPLIT), "result tile inside the staging buffers");
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32_det(dst)), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// four consecutive elements of a 16-byte aligned row
__device__ __forceinline__ void ld_quad(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld_quad(const double* p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
// One thread's TH x 4 tile of B over one chunk, ascending in the contracted index.
template <int TH, int QPR, typename T>
__device__ __forceinline__ void dl_chunk(const T* Jb, const T* Ac, int TR, int TC, T (&acc)[TH * 4]) {
#pragma unroll 2
  for (int qx = 0; qx < QPR; ++qx) {
    T b[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y) ld_quad(Ac + TC * y * DL_LD + 4 * qx, b[y]);
#pragma unroll
    for (int j = 0; j < TH; ++j) {
      T a[4];
      ld_quad(Jb + TR * j * DL_LD + 4 * qx, a);
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int o = 0; o < 4; ++o) acc[4 * j + y] += a[o] * b[y][o];
    }
  }
}
// Sum of products: in double, or of FP32 factors as the exact products' three-term expansion (each addition's and each
// product's rounding error is kept; what is lost is below 2^-70 of the largest partial sum, a double loses 2^-53).  An FP32
// overflow makes the sum non-finite: the caller then sums in double.
template <typename T>
struct DlSum {
  double s = 0.0;
  __device__ __forceinline__ void add(T a, T b) { s += a * b; }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct DlSum<float> {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  __device__ __forceinline__ void add(float a, float b) {
    const float p = __fmul_rn(a, b);
    const df64 h = df_two_sum(s0, p), l = df_two_sum(s1, fmaf(a, b, -p)), m = df_two_sum(l.hi, h.lo);
    s0 = h.hi;
    s1 = m.hi;
    s2 += l.lo + m.lo;
  }
  __device__ __forceinline__ double value() const { return (double)s0 + ((double)s1 + (double)s2); }
};
// NT threads; jobs with CLO < cnt <= CHI (the others are left to the other instance; cnt > DL_CMAX reports a
// pair overflow)
template <typename T, int NT, int CLO, int CHI>
__global__ void __launch_bounds__(NT) k_detlap(Nbr nb, Layout L, const T* __restrict__ Jp,
                                               const T* __restrict__ AinvT, const T* __restrict__ lapA,
                                               double* __restrict__ grad, double* __restrict__ lap, int32_t* status) {
  constexpr int JROWS = dl_jrows(CHI), STAGE = dl_stage_elems(CHI), BLD = CHI + 1;
  extern __shared__ __align__(16) unsigned char dl_smem[];
  const int n = nb.n, nA = ainv_ld(n);
  const int d = blockIdx.y, w = blockIdx.z;
  if (!walker_live(nb, w)) return;
  const int* rp = nb.rowptr + (size_t)w * (n + 1);
  if (rp[n] > nb.cap_p) return;
  T* stg = reinterpret_cast<T*>(dl_smem);  // [DL_STAGES][J rows JROWS, inverse rows CHI + 4][DL_LD]
  T* Bm = reinterpret_cast<T*>(dl_smem);   // [3 * CHI][BLD] after the main loop
  __shared__ const T* prow[4 * CHI];       // x = 0 of the R J rows, then of the cnt inverse rows
  __shared__ double rs[NT / 32];
  const int tid = threadIdx.x;
  const int off = L.pos_off[w];
  const T* Ab = AinvT + ((size_t)w * NDET + d) * n * nA;
  const long ldj = (long)NDET * n;
  const int sh = (d * n) & 3, XN = (sh + n + 3) & ~3;
  constexpr int EPC = 16 / sizeof(T), CPR = DL_OC / EPC;  // elements per 16-byte copy, copies per row and chunk
  constexpr int QPR = DL_OC / 4;                          // quads per row and chunk
  for (int m = blockIdx.x; m < n; m += gridDim.x) {
    const int cnt = rp[m + 1] - rp[m] + 1;
    if (cnt <= CLO) continue;
    if (cnt > CHI) {
      if (CHI == DL_CMAX && tid == 0) set_flag(status, FIRE_FLAG_PAIR_OVERFLOW);
      continue;
    }
    const int s0 = off + rp[m] + m, R = 3 * cnt;
    __syncthreads();  // the last job's sums have been read
    for (int k = tid; k < cnt; k += NT) {
      const int q = L.dep_pos[s0 + k];
      for (int t = 0; t < 3; ++t) prow[3 * k + t] = Jp + (3L * q + t) * ldj + (long)d * n - sh;
      prow[R + k] = Ab + (size_t)(L.pos_ctr[q] - w * n) * nA;
    }
    __syncthreads();
    // staging: CPR neighbouring lanes copy one row's chunk, so that a warp touches 4 lines (2 of doubles) per copy; a thread
    // per row touched 32 and kept the load unit's tag stage busy for a third of the time
    auto stage = [&](int buf, int x0) {
#pragma unroll 4
      for (int e = tid; e < (R + cnt) * CPR; e += NT) {
        const int row = e / CPR, c = e % CPR * EPC;
        const bool ok = x0 + c < XN;
        cp_async16(stg + (size_t)buf * STAGE + (row < R ? row : JROWS + row - R) * DL_LD + c, ok ? prow[row] + x0 + c : Ab, ok);
      }
    };
    const int TC = (cnt + 3) / 4;
    const int nch = (XN + DL_OC - 1) / DL_OC;
    // DL_STAGES - 1 chunks ahead; one commit group per chunk (empty past the end), one barrier per chunk: the
    // buffer restaged after the barrier of chunk ch held chunk ch - 1, which every thread has finished
    auto contract = [&](auto th) {
      constexpr int TH = decltype(th)::value;
      const int TR = (R + TH - 1) / TH, r0 = tid / TC, k0 = tid - r0 * TC;
      T acc[TH * 4];
#pragma unroll
      for (int q = 0; q < TH * 4; ++q) acc[q] = T(0);
#pragma unroll
      for (int c = 0; c < DL_STAGES - 1; ++c) {
        if (c < nch) stage(c, c * DL_OC);
        cp_async_commit();
      }
      for (int ch = 0; ch < nch; ++ch) {
        cp_async_wait<DL_STAGES - 2>();
        __syncthreads();
        const int nx = ch + DL_STAGES - 1;
        if (nx < nch) stage(nx % DL_STAGES, nx * DL_OC);
        cp_async_commit();
        const T* Jb = stg + (size_t)(ch % DL_STAGES) * STAGE;
        if (r0 < TR) dl_chunk<TH, QPR>(Jb + r0 * DL_LD, Jb + (JROWS + k0) * DL_LD, TR, TC, acc);
      }
      cp_async_wait<0>();
      __syncthreads();  // every chunk consumed: the result tile overwrites the staging buffers
      if (r0 < TR) {
#pragma unroll
        for (int j = 0; j < TH; ++j)
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            const int r = r0 + TR * j, k = k0 + TC * y;
            if (r < R && k < cnt) Bm[r * BLD + k] = acc[4 * j + y];
          }
      }
    };
    const int rt = NT / TC;  // tile rows that the CTA's threads hold
    if (R <= rt) contract(std::integral_constant<int, 1>());
    else if (R <= 2 * rt) contract(std::integral_constant<int, 2>());
    else if (R <= 4 * rt) contract(std::integral_constant<int, 4>());
    else if (R <= 5 * rt) contract(std::integral_constant<int, 5>());
    else if (R <= 6 * rt) contract(std::integral_constant<int, 6>());
    else if (R <= 8 * rt) contract(std::integral_constant<int, 8>());
    else contract(std::integral_constant<int, 12>());
    __syncthreads();
    // triplet term: sum_t sum_{k, k2} B[(k, t)][k2] * B[(k2, t)][k], a warp per row (k, t);  gradient: sum_k B[(k, t)][k];
    // tr(lap A A^-1) row m: sum_o lapA[m][o] Ainv[o][m]
    const int lane = tid & 31;
    const T* lrow = lapA + ((size_t)w * n + m) * ldj + (long)d * n;
    const T* irow = Ab + (size_t)m * nA + sh;
    DlSum<T> tl, tr;
    for (int rr = tid >> 5; rr < R; rr += NT / 32) {
      const int k = rr / 3, t = rr - 3 * k;
      for (int k2 = lane; k2 < cnt; k2 += 32) tl.add(Bm[rr * BLD + k2], Bm[(3 * k2 + t) * BLD + k]);
    }
    for (int o = tid; o < n; o += NT) tr.add(lrow[o], irow[o]);
    double v = tr.value() - tl.value();
    if (sizeof(T) == 4) {
      if (__syncthreads_or(!isfinite(v))) {  // factors beyond 10^19, an infinity or a NaN: in double
        DlSum<double> tl2, tr2;
        for (int rr = tid >> 5; rr < R; rr += NT / 32) {
          const int k = rr / 3, t = rr - 3 * k;
          for (int k2 = lane; k2 < cnt; k2 += 32) tl2.add((double)Bm[rr * BLD + k2], (double)Bm[(3 * k2 + t) * BLD + k]);
        }
        for (int o = tid; o < n; o += NT) tr2.add((double)lrow[o], (double)irow[o]);
        v = tr2.value() - tl2.value();
      }
    }
    v = warp_sum(v);
    if (lane == 0) rs[tid >> 5] = v;
    if (tid < 96) {  // kept in double: near a node |grad log psi|^2 is ~1e4 |E_loc|
      const int t = tid >> 5;
      double gsum = 0.0;
      for (int k = lane; k < cnt; k += 32) gsum += (double)Bm[(3 * k + t) * BLD + k];
      gsum = warp_sum(gsum);
      if (lane == 0) grad[(((size_t)w * NDET + d) * n + m) * 3 + t] = gsum;
    }
    __syncthreads();
    if (tid == 0) {
      double sum = 0.0;
      for (int q = 0; q < NT / 32; ++q) sum += rs[q];
      atomicAdd(&lap[w * NDET + d], sum);
    }
  }
}

// One thread per 4 consecutive orbital columns of one electron (DN % 4 == 0, every plane 16-byte aligned).  env: the
// envelope carrier [G][5][DN] (value, Jacobian xyz, Laplacian), raw [G][DN], rjs: the raw orbitals' self Jacobian
// rows [G][3][DN] (written by the Jacobian contraction's epilogue).
__global__ void k_orb_lap(float* __restrict__ lapA, const float* __restrict__ env, const float* __restrict__ raw,
                          const float* __restrict__ rjs, long G, int DN) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x, nq = (long)DN / 4;
  if (q >= G * nq) return;
  const long g = q / nq;
  const int c = (int)(q - g * nq) * 4;
  const float* e = env + g * 5 * DN + c;
  const float* rj = rjs + g * 3 * DN + c;
  float4* out = reinterpret_cast<float4*>(lapA + g * DN + c);
  const float4 a = *out, ex = *reinterpret_cast<const float4*>(e), el = *reinterpret_cast<const float4*>(e + 4 * DN),
               rw = *reinterpret_cast<const float4*>(raw + g * DN + c);
  float4 v = make_float4(a.x * ex.x + el.x * rw.x, a.y * ex.y + el.y * rw.y, a.z * ex.z + el.z * rw.z,
                         a.w * ex.w + el.w * rw.w);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const float4 r = *reinterpret_cast<const float4*>(rj + t * DN), ej = *reinterpret_cast<const float4*>(e + (1 + t) * DN);
    v.x += 2.f * r.x * ej.x; v.y += 2.f * r.y * ej.y; v.z += 2.f * r.z * ej.z; v.w += 2.f * r.w * ej.w;
  }
  *out = v;
}

template __global__ void k_env_coef<float, 1>(const float*, const float*, const float*, int, int, int, int, int,
                                              float*, const int*);
template __global__ void k_env_coef<float, 5>(const float*, const float*, const float*, int, int, int, int, int,
                                              float*, const int*);
template __global__ void k_env_coef<double, 1>(const double*, const float*, const double*, int, int, int, int,
                                               int, double*, const int*);
template __global__ void k_env_coef<double, 5>(const double*, const float*, const double*, int, int, int, int,
                                               int, double*, const int*);
template __global__ void k_gj_global<df64, float, float, false>(const float*, const float*, int, df64*, double*, double*, double*,
                                                                 float*, const int*, int32_t*);
template __global__ void k_gj_global<df64, float, float, true>(const float*, const float*, int, df64*, double*, double*, double*,
                                                                float*, const int*, int32_t*);
// FP64 elimination of FP64 orbital matrices with the inverse in FP32 (the refinement pass of the FP32 / mixed local
// energy, whose determinant Laplacian reads an FP32 inverse)
template __global__ void k_gj_global<double, double, float, true>(const double*, const double*, int, double*, double*, double*,
                                                                   double*, float*, const int*, int32_t*);
template __global__ void k_gj_global<double, double, double, true>(const double*, const double*, int, double*, double*, double*,
                                                                    double*, double*, const int*, int32_t*);
template __global__ void k_gj_global<double, double, double, false>(const double*, const double*, int, double*, double*, double*,
                                                                     double*, double*, const int*, int32_t*);
template __global__ void k_detlap<float, 128, 0, DL_DSPLIT>(Nbr, Layout, const float*, const float*, const float*,
                                                            double*, double*, int32_t*);
template __global__ void k_detlap<float, 128, 0, DL_CSPLIT>(Nbr, Layout, const float*, const float*, const float*,
                                                            double*, double*, int32_t*);
template __global__ void k_detlap<float, 256, DL_CSPLIT, DL_CMAX>(Nbr, Layout, const float*, const float*,
                                                                  const float*, double*, double*, int32_t*);
template __global__ void k_detlap<double, 128, 0, DL_DSPLIT>(Nbr, Layout, const double*, const double*,
                                                            const double*, double*, double*, int32_t*);
template __global__ void k_detlap<double, 256, DL_DSPLIT, DL_CMAX>(Nbr, Layout, const double*, const double*,
                                                            const double*, double*, double*, int32_t*);

}  // namespace fire
