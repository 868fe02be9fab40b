// Dense factor contraction of the operator programs (Dense @ X, cola/ops/operators.py:26-28, and the
// Kronecker factors, :216-223): Y[m, n] = alpha * sum_k A[m, k] X[k, n] + beta * Y[m, n] for more than
// a few columns, in the compute type's own arithmetic (FP32 or FP64 FMAs; BF16 / FP32 storage is
// widened as it is staged).
//
// A column n stands for the pair (p, j) = (n / q, n % q): X[k, n] lies at X + p x_p + k x_k + j and
// Y[m, n] at Y + p y_p + m y_m + j.  A plain product has q = N; a Kronecker factor with `pre` leading
// and q trailing entries is one product over N = pre * q columns (no transposed copies, A read once
// per column tile); the repeated blocks of a BlockDiag are p = 0 .. batch - 1.
//
// A warp owns 32 rows x (8 TN) columns, 8 x TN sums per thread: 8 lanes side by side in n read one
// 16-byte piece of a staged row of A by broadcast, so four k-steps cost 8 + 4 TN/4 shared loads for
// 32 TN FMAs.  Two or three k-slices are in flight as asynchronous copies while one is used: a narrow
// product reads its matrix once at few operations per byte and is bound by the bytes in flight.
// Narrow products leave few output tiles (4096 x 32: 64 of them), so the k range is divided twice:
// over WK warp groups of a CTA and over a cluster of up to eight CTAs, whose partial tiles are added
// in rank order through distributed shared memory.  No workspace, no atomics: the sum order depends
// on the shape alone.
//
// The earlier kernel (64 x 64 tile, one k range, scalar loads) took 129 us for 1500 x 1500 x 16 and
// ~330 us for 4096 x 4096 x 32, FP32.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "ops.cuh"

namespace colagb {

template <class T, class S>
struct GemmArgs {
  const S* A;
  int64_t lda, M, K;
  const T* X;
  int64_t x_p, x_k;
  T* Y;
  int64_t y_p, y_m;
  int64_t N, q;
  T alpha, beta;
  // quads of A (along k) / of X (along n, or along k when XK) may be read, of Y (along n) written as vectors
  int avec, xvec, yvec;
  int64_t mtiles;
  int split;
  const int* skip;
};

// quotient and remainder of a column or tile index; 32-bit operands (nearly always) avoid the long division
__device__ __forceinline__ void div_mod(int64_t a, int64_t b, int64_t& d, int64_t& m) {
  if ((a | b) >> 32 == 0) {
    d = (uint32_t)a / (uint32_t)b;
    m = (uint32_t)a - (uint32_t)d * (uint32_t)b;
  } else {
    d = a / b;
    m = a - d * b;
  }
}

template <class T> __device__ __forceinline__ void ld_quad(const T* p, T v[4]);
template <> __device__ __forceinline__ void ld_quad<float>(const float* p, float v[4]) {
  const float4 t = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <> __device__ __forceinline__ void ld_quad<double>(const double* p, double v[4]) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <class T, class S> __device__ __forceinline__ void ld_quad_as(const S* p, T v[4]) {
  if constexpr (std::is_same<S, __nv_bfloat16>::value) {
    const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
    v[0] = T(a.x); v[1] = T(a.y); v[2] = T(b.x); v[3] = T(b.y);
  } else {
    S t[4];
    ld_quad<S>(p, t);
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = T(t[c]);
  }
}
__device__ __forceinline__ void st_quad(float* p, const float v[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st_quad(double* p, const double v[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void lds_quad(const float* p, float v[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void lds_quad(const double* p, double v[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void lds_quad(const __nv_bfloat16* p, float v[4]) {
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool in) {  // the same, 8 bytes
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {  // zero-fills when !in
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// BM x BN output tile, WM x WN x WK warps, k-slices of BK, ST staging buffers.  XK: the quads of X run
// along k (columns of few contiguous entries, q < 4), else along n.  ASYNC: both operands are quads at their
// natural boundaries with whole quads inside K and N: ST - 1 slices are in flight as asynchronous copies (BF16
// rows beside FP32 columns stay BF16 in shared memory and are widened as they are read; through registers,
// 4096 x 4096 x 1024 took 1393 us).  Otherwise one slice is in flight through registers, widened or gathered
// element by element on the way (ST = 2).
template <class T, class S>
constexpr bool gemm_async_types = std::is_same<T, S>::value || (std::is_same<T, float>::value && std::is_same<S, __nv_bfloat16>::value);

// entries of a padded row of A's slice, of type AS (neighbouring rows in other banks), and the slice's length in T
template <class AS, int BK> constexpr int gemm_row = BK + 16 / (int)sizeof(AS);
template <class T, class AS, int BM, int BK> constexpr int gemm_slice = BM * gemm_row<AS, BK> * (int)sizeof(AS) / (int)sizeof(T);

template <class T, class S, int BM, int BN, int BK, int WM, int WN, int WK, int ST, bool XK, bool ASYNC>
__global__ void __launch_bounds__(32 * WM * WN * WK) k_gemm(const __grid_constant__ GemmArgs<T, S> g) {
  if (g.skip && *g.skip) return;
  namespace cgx = cooperative_groups;
  constexpr int NT = 32 * WM * WN * WK;
  constexpr int TM = BM / WM / 4, TN = BN / WN / 8;
  using AS = typename std::conditional<ASYNC, S, T>::type;
  constexpr int PA = gemm_row<AS, BK>;
  constexpr int PX = XK ? BN + 1 : BN;
  constexpr int AQ = BM * BK / 4, XQ = BK * BN / 4;
  constexpr int NA = (AQ + NT - 1) / NT, NX = (XQ + NT - 1) / NT;
  constexpr int KW = BK / WK;  // k-steps of one warp group per slice
  constexpr int LA = gemm_slice<T, AS, BM, BK>, LX = (BK * PX + 3) / 4 * 4;
  static_assert(KW % 4 == 0 && TM * 4 * WM == BM && TN * 8 * WN == BN && LA % 4 == 0, "tile shape");
  static_assert(!(ASYNC && XK) && (ASYNC ? gemm_async_types<T, S> : ST == 2), "staging form");
  extern __shared__ __align__(16) unsigned char gemm_smem[];
  T* const smem = reinterpret_cast<T*>(gemm_smem);  // ST buffers of (A slice, X slice); then the partial tile

  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int wk = warp / (WM * WN), wmn = warp % (WM * WN), wm = wmn % WM, wn = wmn / WM;
  const int ly = lane >> 3, lx = lane & 7;
  const int rank = (int)(blockIdx.x % (unsigned)g.split);
  const int64_t tid = blockIdx.x / (unsigned)g.split;
  int64_t tile_n, tile_m;
  div_mod(tid, g.mtiles, tile_n, tile_m);
  const int64_t m0 = tile_m * BM, n0 = tile_n * BN;
  // this CTA's k range, in whole slices
  const int64_t slices = ceil_div(g.K, (int64_t)BK), per = ceil_div(slices, (int64_t)g.split);
  const int64_t s0 = rank * per < slices ? rank * per : slices;
  const int64_t s1 = s0 + per < slices ? s0 + per : slices;

  // staging: thread t moves quads t, t + NT, ... of each operand's slice, at addresses that advance by
  // a constant from slice to slice; rows and columns beyond the edge read the last or first one (never stored), but
  // asynchronous copies of the large plain tiles leave such rows zero: every CTA copying the same line many times,
  // 16 x 16 x 100,000 took 22 instead of 12 us.  Only tiles at the edge look at the rows (in all tiles, it cost
  // 4096 x 4096 x 1024 16 %).
  const S* pa[NA];
  unsigned rows_in = 0;  // bit i: row of pa[i] exists
  constexpr bool MASK = ASYNC && WK == 1 && BM * BN > 1024;
  const bool edge = MASK && m0 + BM > g.M;
  const T* px[NX];
  int left[NX];  // columns from the quad's first one to the end of its p (a quad may run over into the next)
  bool xin[NX];
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    const int u = t + i * NT;
    const int64_t m = m0 + (u < AQ ? u / (BK / 4) : 0);
    pa[i] = g.A + (m < g.M ? m : g.M - 1) * g.lda + s0 * BK + 4 * (u % (BK / 4));
    if (MASK && m < g.M) rows_in |= 1u << i;
  }
#pragma unroll
  for (int i = 0; i < NX; ++i) {
    const int u = t + i * NT;
    const int nn = XK ? u / (BK / 4) : 4 * (u % (BN / 4)), kk = XK ? 4 * (u % (BK / 4)) : u / (BN / 4);
    xin[i] = u < XQ && n0 + nn < g.N;
    const int64_t n = xin[i] ? n0 + nn : 0;
    int64_t p, j;
    div_mod(n, g.q, p, j);
    px[i] = g.X + p * g.x_p + j + (s0 * BK + kk) * g.x_k;
    left[i] = (int)(g.q - j < 4 ? g.q - j : 4);
  }
  T ra[ASYNC ? 1 : NA][4], rx[ASYNC ? 1 : NX][4];
  auto fetch = [&](int64_t s, int b) {  // slice s: into buffer b (ASYNC) or into registers
    const int kl = (int)(g.K - s * BK < BK ? g.K - s * BK : BK);  // k entries of this slice
    AS* const as = reinterpret_cast<AS*>(smem + b * (LA + LX));
    T* const xs = smem + b * (LA + LX) + LA;
    auto copy_a = [&](int i, bool in) {  // quad i of A
      const int u = t + i * NT, k = 4 * (u % (BK / 4));
      if (AQ % NT == 0 || u < AQ) {
        if constexpr (ASYNC && sizeof(S) == 2) {
          cp_async8(as + (u / (BK / 4)) * PA + k, pa[i], in && k < kl);
        } else if constexpr (ASYNC) {
#pragma unroll
          for (int h = 0; h < (int)sizeof(T) / 4; ++h) {
            constexpr int E = 16 / (int)sizeof(T);
            cp_async16(as + (u / (BK / 4)) * PA + k + h * E, pa[i] + h * E, in && k < kl);
          }
        } else if (g.avec && k + 3 < kl) {
          ld_quad_as<T, S>(pa[i], ra[i]);
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) ra[i][c] = k + c < kl ? cvt<T>(pa[i][c]) : T(0);
        }
      }
      pa[i] += BK;
    };
    if (MASK && edge) {
#pragma unroll
      for (int i = 0; i < NA; ++i) copy_a(i, rows_in >> i & 1);
    } else {
#pragma unroll
      for (int i = 0; i < NA; ++i) copy_a(i, true);
    }
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int u = t + i * NT;
      if (XQ % NT == 0 || u < XQ) {
        if constexpr (ASYNC) {
#pragma unroll
          for (int h = 0; h < (int)sizeof(T) / 4; ++h) {
            constexpr int E = 16 / (int)sizeof(T);
            cp_async16(xs + (u / (BN / 4)) * PX + 4 * (u % (BN / 4)) + h * E, px[i] + h * E, xin[i] && u / (BN / 4) < kl);
          }
        } else if constexpr (XK) {
          const int k = 4 * (u % (BK / 4));
          if (xin[i] && g.xvec && k + 3 < kl) {
            ld_quad<T>(px[i], rx[i]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) rx[i][c] = xin[i] && k + c < kl ? px[i][c * g.x_k] : T(0);
          }
        } else {
          const int64_t n = n0 + 4 * (u % (BN / 4));
          const bool kin = u / (BN / 4) < kl;
          if (g.xvec && kin && n + 3 < g.N) {
            ld_quad<T>(px[i], rx[i]);
          } else {
            const T* p = px[i];
            int l = left[i];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              rx[i][c] = kin && n + c < g.N ? *p : T(0);
              ++p;
              if (--l == 0) {
                p += g.x_p - g.q;
                l = (int)(g.q < 4 ? g.q : 4);
              }
            }
          }
        }
      }
      px[i] += BK * g.x_k;
    }
    if constexpr (ASYNC) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto stage = [&](int b) {  // registers -> buffer b
    if constexpr (!ASYNC) {
      T* const as = smem + b * (LA + LX);
      T* const xs = as + LA;
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        const int u = t + i * NT;
        if (u < AQ) st_quad(as + (u / (BK / 4)) * PA + 4 * (u % (BK / 4)), ra[i]);
      }
#pragma unroll
      for (int i = 0; i < NX; ++i) {
        const int u = t + i * NT;
        if (u < XQ) {
          if constexpr (XK) {
            const int nn = u / (BK / 4), kk = 4 * (u % (BK / 4));
#pragma unroll
            for (int c = 0; c < 4; ++c) xs[(kk + c) * PX + nn] = rx[i][c];
          } else {
            st_quad(xs + (u / (BN / 4)) * PX + 4 * (u % (BN / 4)), rx[i]);
          }
        }
      }
    }
  };

  // The long FP32 sums of the narrow tiles (32 x 16, 32 x 8) are added up in pieces of 64 terms: one chain of K / (4 split) terms
  // left the solution of a 3900 x 6 CG 1.9 times further from the exact one than the row kernels did.
  constexpr bool PIECES = std::is_same<T, float>::value && WK > 1 && TM * TN <= 16;
  T acc[TM][TN], total[PIECES ? TM : 1][PIECES ? TN : 1];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      acc[i][j] = T(0);
      if constexpr (PIECES) total[i][j] = T(0);
    }
  // thread's rows: wm * 32 + ly + 4 i; columns: wn * 8 TN + (TN >= 4: 32 h + 4 lx + c, else TN lx + j)
  auto col_of = [&](int j) { return wn * 8 * TN + (TN >= 4 ? 32 * (j / 4) + 4 * lx + (j & 3) : TN * lx + j); };

  const int64_t ns = s1 - s0;
  if constexpr (ASYNC) {
#pragma unroll
    for (int i = 0; i < ST - 1; ++i) {
      if (i < ns) fetch(s0 + i, i);
      else asm volatile("cp.async.commit_group;" ::: "memory");  // empty groups keep the count
    }
  } else if (ns > 0) {
    fetch(s0, 0);
    stage(0);
    __syncthreads();
  }
  {
    int b = 0;
    for (int64_t i = 0; i < ns; ++i) {
      if constexpr (ASYNC) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();  // slice i has landed for all threads; all are done with the buffer refilled next
        const int bn = b == 0 ? ST - 1 : b - 1;
        if (i + ST - 1 < ns) fetch(s0 + i + ST - 1, bn);
        else asm volatile("cp.async.commit_group;" ::: "memory");
      } else if (i + 1 < ns) {
        fetch(s0 + i + 1, b ^ 1);
      }
      const AS* as = reinterpret_cast<const AS*>(smem + b * (LA + LX)) + (wm * 4 * TM + ly) * PA + wk * KW;
      const T* xs = smem + b * (LA + LX) + LA + wk * KW * PX;
      const int64_t kleft = g.K - (s0 + i) * BK - wk * KW;  // k-steps of this warp group that exist
#pragma unroll
      for (int kq = 0; kq < KW; kq += 4) {
        if (kq >= kleft) break;
        T av[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i) lds_quad(as + 4 * i * PA + kq, av[i]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          T xv[TN];
          if constexpr (TN >= 4 && !XK) {
#pragma unroll
            for (int h = 0; h < TN / 4; ++h) lds_quad(xs + (kq + c) * PX + col_of(4 * h), xv + 4 * h);
          } else {
#pragma unroll
            for (int j = 0; j < TN; ++j) xv[j] = xs[(kq + c) * PX + col_of(j)];
          }
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] += av[i][c] * xv[j];
        }
      }
      if constexpr (PIECES)
        if ((i + 1) % (64 / KW) == 0 || i + 1 == ns) {
          const bool last = i + 1 == ns;
#pragma unroll
          for (int u = 0; u < TM; ++u)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              total[u][j] += acc[u][j];
              acc[u][j] = last ? total[u][j] : T(0);
            }
        }
      if constexpr (!ASYNC) {
        if (i + 1 < ns) stage(b ^ 1);
        __syncthreads();
      }
      b = b + 1 == ST ? 0 : b + 1;
    }
  }
  if constexpr (ASYNC) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the buffers become the partial tile
  }
  if constexpr (WK == 1) {  // many tiles: no split, sums go straight to Y
    constexpr int VW = TN >= 4 ? 4 : TN;  // neighbouring columns of a thread
#pragma unroll
    for (int j0 = 0; j0 < TN; j0 += VW) {
      const int64_t n = n0 + col_of(j0);
      if (n >= g.N) continue;
      int64_t p, jj;
      div_mod(n, g.q, p, jj);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int64_t m = m0 + wm * 4 * TM + ly + 4 * i;
        if (m >= g.M) continue;
        T* const y = g.Y + p * g.y_p + jj + m * g.y_m;
        if (g.yvec) {  // q is whole quads, so the columns are in range and side by side
          alignas(VW * sizeof(T)) T v[VW];
          T o[VW];
          if (g.beta != T(0)) {
#pragma unroll
            for (int c = 0; c < VW; ++c) o[c] = y[c];
          }
#pragma unroll
          for (int c = 0; c < VW; ++c)
            v[c] = g.beta == T(0) ? g.alpha * acc[i][j0 + c] : g.alpha * acc[i][j0 + c] + g.beta * o[c];
          if constexpr (VW == 4) {
            st_quad(y, v);
          } else {
            struct alignas(VW * sizeof(T)) Piece { T v[VW]; };
            *reinterpret_cast<Piece*>(y) = *reinterpret_cast<Piece*>(v);
          }
          continue;
        }
        T* yc = y;
        int left = (int)(g.q - jj < VW ? g.q - jj : VW);
#pragma unroll
        for (int c = 0; c < VW; ++c) {
          if (n + c < g.N) *yc = g.beta == T(0) ? g.alpha * acc[i][j0 + c] : g.alpha * acc[i][j0 + c] + g.beta * (*yc);
          ++yc;
          if (--left == 0) {  // the next p
            yc += g.y_p - g.q;
            left = (int)(g.q < VW ? g.q : VW);
          }
        }
      }
    }
    return;
  } else {
  T* const tile = smem;
  // warp groups of the CTA in order, then the CTAs of the cluster in rank order
#pragma unroll
  for (int w = 0; w < WK; ++w) {
    if (wk == w)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          T* d = &tile[(wm * 4 * TM + ly + 4 * i) * BN + col_of(j)];
          *d = w == 0 ? acc[i][j] : *d + acc[i][j];
        }
    __syncthreads();
  }
  cgx::cluster_group cl = cgx::this_cluster();
  if (g.split > 1) cl.sync();
  // consecutive threads write along m when that is the contiguous direction of Y
  const bool along_m = g.y_m == 1 && g.q < 8;
  const int lo = BM * BN / g.split * rank, hi = rank + 1 == g.split ? BM * BN : lo + BM * BN / g.split;
  for (int e = lo + t; e < hi; e += NT) {
    const int mm = along_m ? e % BM : e / BN, nn = along_m ? e / BM : e % BN;
    const int64_t m = m0 + mm, n = n0 + nn;
    if (m >= g.M || n >= g.N) continue;
    T sum = T(0);
    if (g.split == 1) {
      sum = tile[mm * BN + nn];
    } else {
      for (int r = 0; r < g.split; ++r) sum += *cl.map_shared_rank(&tile[mm * BN + nn], r);
    }
    int64_t p, j;
    div_mod(n, g.q, p, j);
    T* y = g.Y + p * g.y_p + m * g.y_m + j;
    *y = g.beta == T(0) ? g.alpha * sum : g.alpha * sum + g.beta * (*y);
  }
  if (g.split > 1) cl.sync();  // no CTA leaves while a peer may still read its tile
  }
}

template <class T, class S, int BM, int BN, int BK, int WM, int WN, int WK, int ST, bool XK, bool ASYNC>
static int launch_form(GemmArgs<T, S>& g, cudaStream_t st) {
  auto* f = k_gemm<T, S, BM, BN, BK, WM, WN, WK, ST, XK, ASYNC>;
  using AS = typename std::conditional<ASYNC, S, T>::type;
  constexpr int LA = gemm_slice<T, AS, BM, BK>, LX = (BK * (XK ? BN + 1 : BN) + 3) / 4 * 4;
  constexpr size_t stage_b = sizeof(T) * ST * (LA + LX), tile_b = WK > 1 ? sizeof(T) * BM * BN : 0;
  constexpr size_t smem = stage_b > tile_b ? stage_b : tile_b;
  if (smem > 48 * 1024) COLAGB_CUDA(set_smem_limit(f, smem));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)g.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)(g.mtiles * ceil_div(g.N, (int64_t)BN) * g.split));
  cfg.blockDim = dim3(32 * WM * WN * WK);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  COLAGB_CUDA(cudaLaunchKernelEx(&cfg, f, g));
  return COLAGB_OK;
}

template <class T, class S>
static bool gemm_async(const GemmArgs<T, S>& g) { return g.avec && g.xvec && g.K % 4 == 0 && g.N % 4 == 0; }

template <class T, class S, int BM, int BN, int BK, int WM, int WN, int WK, int ST, bool MAY_ASYNC = true>
static int launch_tile(GemmArgs<T, S>& g, int split, bool xk, cudaStream_t st) {
  g.mtiles = ceil_div(g.M, (int64_t)BM);
  g.split = split;
  if (xk) return launch_form<T, S, BM, BN, BK, WM, WN, WK, 2, true, false>(g, st);
  if constexpr (gemm_async_types<T, S> && MAY_ASYNC)
    if (gemm_async(g)) return launch_form<T, S, BM, BN, BK, WM, WN, WK, ST, false, true>(g, st);
  return launch_form<T, S, BM, BN, BK, WM, WN, WK, 2, false, false>(g, st);
}

// Tile choice, FP32 sums.  Short ones (K <= 256, and K <= 1024 where the caller asks for it: Kronecker factors, whose
// products feed Lanczos recurrences) keep the plain order of k, one warp group and no split; the tiles differ in
// shape alone:
//   up to 16 columns: 128 x 16 while that gives every SM two tiles (100,000 x 16 x 16 8.5 us, 50,000 x 64 x 8 10.5;
//     64 x 128 tiles 25 and 27, 32 x 16 12.4 and 14.4), else 32 x 16;
//   1.5 tiles of 64 x 64 an SM and more: 48 or 64 rows (whichever pads M less) x 128 columns where the copies are
//     asynchronous and there are 1.8 tiles an SM (48 x 48 x 36,864 10.5 us, 64 x 64 x 36,864 14.5), else 64 x 64, in
//     slices of 16 for up to 128 terms (720 x 720 x 1440 51 us, 720 products with blocks of 2 columns 68; 48 x 128 tiles
//     took 75 and 135; 200,000 x 32 x 64 33 in slices of 16, 37 in slices of 32);
//   fewer: 32 x 32 (512 x 512 x 512 18 us, 700 x 256 x 300 12).
// Longer sums: 64 x 64 while that gives every SM a tile, else the column tile that N fills, with clusters along k
// until the grid covers 1.5 times the SMs and each CTA keeps at least two k-slices.  Measured (FP32, back-to-back
// launches, which cost 6.2 us for the smallest product): 4096 x 4096 x 32 35 us (64 x 32, split 4; 39 us for 64 x 64
// tiles), x 512 370 us = 46 TFLOP/s; 1500 x 1500 x 16 8.4 us (split 8; 10.3 us at split 4); 3000 x 3000 x 8 14.5 us.  BF16
// rows that go through registers take slices of 16 with twice the warps (3001 x 3001 x 300 267 us, 302 otherwise).
// The tiles of up to 16 sums a thread (32 x 16, 32 x 8) add them in pieces of 64 terms; 64 x 64 and 64 x 32 have chains of
// K / (WK split) terms, 256 at 4096 x 4096 x 32, where the row and tile kernels before had K / 32 and K.
template <class T, class S>
int dense_contract(const S* A, int64_t lda, int64_t M, int64_t K, const T* X, int64_t x_p, int64_t x_k, T* Y,
                   int64_t y_p, int64_t y_m, int64_t P, int64_t q, T alpha, T beta, bool plain, const int* skip,
                   cudaStream_t st) {
  GemmArgs<T, S> g;
  g.A = A; g.lda = lda; g.M = M; g.K = K;
  g.X = X; g.x_p = x_p; g.x_k = x_k;
  g.Y = Y; g.y_p = y_p; g.y_m = y_m;
  g.N = P * q; g.q = q;
  g.alpha = alpha; g.beta = beta; g.skip = skip;
  if (M == 0 || g.N == 0) return COLAGB_OK;
  const size_t aq = 4 * sizeof(S) < 16 ? 4 * sizeof(S) : 16, xq = 16, ae = aq / sizeof(S), xe = xq / sizeof(T);
  g.avec = reinterpret_cast<uintptr_t>(A) % aq == 0 && lda % (int64_t)ae == 0;
  const bool xal = reinterpret_cast<uintptr_t>(X) % xq == 0;
  const bool xk = q < 4 && x_k == 1;  // contiguous along k
  g.xvec = xk ? xal && x_p % (int64_t)xe == 0 && q == 1
              : xal && q % 4 == 0 && x_p % (int64_t)xe == 0 && x_k % (int64_t)xe == 0;
  g.yvec = reinterpret_cast<uintptr_t>(Y) % xq == 0 && q % 4 == 0 && y_p % (int64_t)xe == 0 && y_m % (int64_t)xe == 0;
  const int64_t sms = num_sms();
  auto tiles = [&](int64_t bm, int64_t bn) { return ceil_div(M, bm) * ceil_div(g.N, bn); };
  auto split_for = [&](int64_t bm, int64_t bn, int64_t bk) {
    const int64_t n = tiles(bm, bn), slices = ceil_div(K, bk);
    int s = 1;
    while (s < 8 && 2 * n * s < 3 * sms && slices >= 4 * s) s *= 2;
    return s;
  };
  if constexpr (std::is_same<T, float>::value) {
    const int64_t t64 = tiles(64, 64);
    if (K <= 256 || (plain && K <= 1024)) {
      if (g.N <= 16) {
        if (tiles(128, 16) >= 2 * sms) return launch_tile<T, S, 128, 16, 16, 4, 1, 1, 3>(g, 1, xk, st);
        return launch_tile<T, S, 32, 16, 32, 2, 1, 1, 4>(g, 1, xk, st);
      }
      if (2 * t64 < 3 * sms) return launch_tile<T, S, 32, 32, 32, 2, 2, 1, 3>(g, 1, xk, st);
      const bool b48 = ceil_div(M, 48) * 48 < ceil_div(M, 64) * 64;
      if (!xk && gemm_async(g) && g.N >= 96 && 5 * tiles(b48 ? 48 : 64, 128) >= 9 * sms)
        return b48 ? launch_tile<T, S, 48, 128, 16, 2, 2, 1, 3>(g, 1, xk, st)
                   : launch_tile<T, S, 64, 128, 16, 2, 2, 1, 3>(g, 1, xk, st);
      if (K <= 128) return launch_tile<T, S, 64, 64, 16, 2, 2, 1, 3>(g, 1, xk, st);
      return launch_tile<T, S, 64, 64, 32, 2, 2, 1, 3>(g, 1, xk, st);
    }
    if (g.N > 32 && (t64 >= sms || (g.N <= 64 && K >= 512))) {
      if constexpr (!std::is_same<T, S>::value)
        if (!gemm_async(g)) return launch_tile<T, S, 64, 64, 16, 2, 2, 2, 2, false>(g, split_for(64, 64, 16), xk, st);
      return launch_tile<T, S, 64, 64, 32, 2, 1, 2, 3>(g, split_for(64, 64, 32), xk, st);
    }
    if (g.N > 16 && K >= 512) return launch_tile<T, S, 64, 32, 64, 2, 1, 4, 3>(g, split_for(64, 32, 64), xk, st);
    if (g.N > 8) return launch_tile<T, S, 32, 16, 32, 1, 1, 4, 4>(g, split_for(32, 16, 32), xk, st);
    return launch_tile<T, S, 32, 8, 64, 1, 1, 4, 4>(g, split_for(32, 8, 64), xk, st);
  } else {
    // FP64 multiply-adds are the bound (64 cycles of a scheduler per warp instruction, on padding too):
    // the largest tile that gives every scheduler two warps, else 16 x 8
    if (g.N > 16 && tiles(32, 32) >= 2 * sms) return launch_tile<T, S, 32, 32, 16, 1, 1, 4, 4>(g, 1, xk, st);
    if (g.N > 8 && tiles(32, 16) >= 2 * sms) return launch_tile<T, S, 32, 16, 32, 1, 1, 4, 4>(g, 1, xk, st);
    return launch_tile<T, S, 16, 8, 32, 1, 1, 4, 4>(g, split_for(16, 8, 32), xk, st);
  }
}

#define COLAGB_INST(T, S)                                                                                         \
  template int dense_contract<T, S>(const S*, int64_t, int64_t, int64_t, const T*, int64_t, int64_t, T*, int64_t, \
                                    int64_t, int64_t, int64_t, T, T, bool, const int*, cudaStream_t);
COLAGB_INST(float, float)
COLAGB_INST(float, __nv_bfloat16)
COLAGB_INST(double, double)
COLAGB_INST(double, float)
COLAGB_INST(double, __nv_bfloat16)
#undef COLAGB_INST

}  // namespace colagb
