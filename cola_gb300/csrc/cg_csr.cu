// Fused CG for one CSR operator of short rows (+ c*I), one right-hand side, P = identity or Diagonal, over
// all SMs with two grid barriers per step.
//
// Same loop, stop rule and history as cg.cu (run_batched_cg, cola/linalg/inverse/cg.py:94-178).  A CTA owns
// a contiguous range of rows and keeps r, x, Ap of it, and its rows of A when they fit, in shared memory
// for the whole solve.  What the others need of it is z = M r, published before the barrier that also
// carries <r, z> and |r|^2; p is not exchanged: the CTA holds p for every column its rows touch (the window
// from their smallest to their largest column, e.g. two grid lines around the range for a 5-point stencil)
// and forms p = z + beta p there itself.  So a step is
//   window: z from L2, p = z + beta p;  rows: Ap, <p, Ap>    -> barrier ->
//   x += alpha p, r -= alpha Ap, z = M r, <r, z>, |r|^2      -> barrier.
// Where the columns spread too far for a window (graphs numbered at random) the CTA gathers z and the
// previous p (double buffered, each CTA publishes its own) from L2 and combines them on the fly.
//
// It is bound by the two barriers (1.3 us each on 152 CTAs), the L2 round trips after them and, in FP64, by
// the arithmetic itself (64 cycles of a scheduler per warp instruction: 128 threads own the rows so that
// the sums cost one warp's shuffles per scheduler).  Before, 16 CTAs of one cluster ran matrices up to
// 32 MB: 37 us a step for 256 x 256 5-point FP64 with Jacobi.
#include <algorithm>
#include <type_traits>

#include "cg_csr.cuh"
#include "common.cuh"

namespace colagb {

template <class T> struct CsOwn {
  static constexpr int threads = std::is_same<T, double>::value ? 128 : 512;
  static constexpr int warps = threads / 32;
};

template <class T>
__device__ __forceinline__ T cs_safe_div(T num, T den) {
  const T eps = std::is_same<T, float>::value ? T(1e-40f) : T(1e-40);
  return num / (fabs(den) < eps ? eps : den);
}

// Block sums of V values, every thread gets them.  buf: V * warps slots, alternated between two buffers.
template <int V, class T>
__device__ __forceinline__ void cs_sums(T (&v)[V], T* buf) {
  constexpr int W = CsOwn<T>::warps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const T x = warp_sum(v[q]);
    if (lane == 0) buf[q * W + warp] = x;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < V; ++q) {
    T a[W];
#pragma unroll
    for (int i = 0; i < W; ++i) a[i] = buf[q * W + i];
#pragma unroll
    for (int h = W / 2; h >= 1; h >>= 1)
#pragma unroll
      for (int i = 0; i < h; ++i) a[i] += a[i + h];
    v[q] = a[0];
  }
}

template <class T, class S>
__global__ void __launch_bounds__(CsOwn<T>::threads, 1) k_cg_csr(const __grid_constant__ CsrCgArgs<T, S> a) {
  constexpr int NT = CsOwn<T>::threads, RED = 2 * CsOwn<T>::warps;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  __shared__ T red[2][RED];
  __shared__ int s_bad, s_lo, s_hi;
  const int t = threadIdx.x, n = a.n, nb = gridDim.x, b = blockIdx.x;
  const int r0 = (int)((int64_t)n * b / nb), R = (int)((int64_t)n * (b + 1) / nb) - r0;
  const int Rm = (n + nb - 1) / nb;
  T* const r = reinterpret_cast<T*>(cs_smem);  // own rows
  T* const x = r + Rm;
  T* const ap = x + Rm;
  T* const po = ap + Rm;                        // p of the own rows
  T* const dv = po + Rm;                        // Jacobi diagonal
  size_t used = (size_t)5 * Rm * sizeof(T);
  int rbuf = 0;
  unsigned int epoch = 0;

  // the rows' entries: resident when they fit half of what is left
  const int32_t e0 = a.indptr[r0], e1 = a.indptr[r0 + R], ne = e1 - e0;
  used = (used + 15) / 16 * 16;
  const size_t mat = ((size_t)ne * sizeof(S) + 15) / 16 * 16 + ((size_t)ne * 4 + 15) / 16 * 16;
  const bool resident = used + mat <= (size_t)a.smem && mat <= ((size_t)a.smem - used) / 2;
  const S* vals = a.vals + e0;
  const int32_t* cols = a.indices + e0;
  if (t == 0) {
    s_bad = 0;
    s_lo = n;
    s_hi = 0;
  }
  __syncthreads();
  int lo = n, hi = 0;
  if (resident) {
    S* const sv = reinterpret_cast<S*>(cs_smem + used);
    int32_t* const sc = reinterpret_cast<int32_t*>(cs_smem + used + ((size_t)ne * sizeof(S) + 15) / 16 * 16);
    for (int e = t; e < ne; e += NT) {
      const int32_t c = cols[e];
      sv[e] = vals[e];
      sc[e] = c;
      lo = min(lo, c);
      hi = max(hi, c + 1);
    }
    vals = sv;
    cols = sc;
    used += mat;
  } else {
    for (int e = t; e < ne; e += NT) {
      const int32_t c = cols[e];
      lo = min(lo, c);
      hi = max(hi, c + 1);
    }
  }
  // the window of columns, own rows included
  atomicMin(&s_lo, min(lo, r0));
  atomicMax(&s_hi, max(hi, r0 + R));
  __syncthreads();
  const int w0 = s_lo, W = s_hi - s_lo;
  const bool window = used + (size_t)W * sizeof(T) <= (size_t)a.smem;
  T* const pw = reinterpret_cast<T*>(cs_smem + used);

  // arrive, wait for all CTAs; false when the wait gave up here or elsewhere
  auto barrier = [&]() -> bool {
    __syncthreads();
    if (t == 0) {
      const unsigned int target = ++epoch * (unsigned)nb;
      __threadfence();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.count) : "memory");
      long long spins = 0;
      unsigned int v;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.count) : "memory");
        if ((int)(v - target) >= 0) break;
        if (ld_volatile_i(a.err) != 0) { s_bad = 1; break; }
        if (++spins > a.spin_limit) {
          atomicCAS(a.err, 0, COLAGB_ERR_TIMEOUT);
          s_bad = 1;
          break;
        }
      }
    }
    __syncthreads();
    return s_bad == 0;
  };
  // grid-wide sums of V values: partials by parity, so that a CTA one barrier ahead writes the other half
  int par = 0;
  auto publish = [&](auto& v) {  // this CTA's sums; call barrier() next
    constexpr int V = sizeof(v) / sizeof(T);
    cs_sums<V, T>(v, red[rbuf]);
    rbuf ^= 1;
    if (t == 0)
#pragma unroll
      for (int q = 0; q < V; ++q) a.part[(par * 2 + q) * nb + b] = v[q];
  };
  auto totals = [&](auto& v) {
    constexpr int V = sizeof(v) / sizeof(T);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      T s = T(0);
      for (int i = t; i < nb; i += NT) s += __ldcg(a.part + (par * 2 + q) * nb + i);
      v[q] = s;
    }
    par ^= 1;
    cs_sums<V, T>(v, red[rbuf]);
    rbuf ^= 1;
  };
  // rows of A on p (window), or on z + beta * pold gathered from L2
  auto rows = [&](T beta, const T* pold) -> T {
    T dot = T(0);
    for (int i = t; i < R; i += NT) {
      int32_t e = a.indptr[r0 + i] - e0;
      const int32_t end = a.indptr[r0 + i + 1] - e0;
      const T pi = window ? pw[r0 + i - w0] : po[i];
      T acc = a.shift * pi;
      if (window) {
        for (; e < end; ++e) acc += cvt<T>(vals[e]) * pw[cols[e] - w0];
      } else {
        for (; e < end; e += 4) {  // entries in groups of four, their gathers in flight together
          T zc[4], pc[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int32_t c = e + q < end ? cols[e + q] : 0;
            zc[q] = __ldcg(a.Z + c);
            pc[q] = __ldcg(pold + c);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (e + q < end) acc += cvt<T>(vals[e + q]) * (zc[q] + beta * pc[q]);
        }
      }
      ap[i] = acc;
      if (window) po[i] = pi;
      dot += pi * acc;
    }
    return dot;
  };
  const T tiny = std::is_same<T, float>::value ? T(0) : T(1e-80);  // |r| < 1e-40 <=> |r|^2 <= tiny
  auto above = [&](T rr, T tol_eff) {  // |r| > tol_eff, without the root unless equal to rounding
    const T t2 = tol_eff * tol_eff, u = std::is_same<T, float>::value ? T(1e-6f) : T(1e-14);
    return rr > t2 + u * t2 ? true : rr < t2 - u * t2 ? false : sqrt(rr) > tol_eff;
  };

  // mult = |b| ; x0 published through Z (and the previous p = 0) for the first product
  T q1[1] = {T(0)};
  for (int i = t; i < R; i += NT) {
    const T bv = a.B[(int64_t)(r0 + i) * a.ldb], xv = a.X[(int64_t)(r0 + i) * a.ldx];
    q1[0] += bv * bv;
    x[i] = xv;
    po[i] = xv;
    dv[i] = a.dinv ? a.dinv[r0 + i] : T(1);
    a.Z[r0 + i] = xv;
    a.P0[r0 + i] = T(0);
  }
  publish(q1);
  if (!barrier()) return;
  totals(q1);
  const T mult = sqrt(q1[0]);
  if (window)
    for (int j = t; j < W; j += NT) pw[j] = __ldcg(a.Z + w0 + j);
  __syncthreads();
  rows(T(0), a.P0);
  if (!barrier()) return;  // everyone is done reading x0 out of Z
  T q2[2] = {T(0), T(0)};
  for (int i = t; i < R; i += NT) {
    const T rv = cs_safe_div(a.B[(int64_t)(r0 + i) * a.ldb], mult) - ap[i];
    const T z = dv[i] * rv;
    r[i] = rv;
    a.Z[r0 + i] = z;
    q2[0] += rv * rv;
    q2[1] += rv * z;
  }
  publish(q2);
  if (!barrier()) return;
  totals(q2);
  T rr = q2[0], gamma = q2[1], beta = T(0);
  T tol_eff;
  {
    const T rn = sqrt(rr);
    tol_eff = (T)a.tol * rn + (T)a.tol;
    if (b == 0 && t == 0 && a.hist) a.hist[0] = rn;
  }
  // p of the step before, by parity: zero before the first one
  for (int i = t; i < R; i += NT) po[i] = T(0);
  if (window)
    for (int j = t; j < W; j += NT) pw[j] = T(0);
  int it = 0;
  bool running = above(rr, tol_eff) && it < a.max_iters;
  while (running) {
    const T* const pold = (it & 1) ? a.P1 : a.P0;
    T* const pnew = (it & 1) ? a.P0 : a.P1;
    if (window) {
      for (int j0 = t; j0 < W; j0 += 8 * NT) {
        T z[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) z[q] = j0 + q * NT < W ? __ldcg(a.Z + w0 + j0 + q * NT) : T(0);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (j0 + q * NT < W) pw[j0 + q * NT] = z[q] + beta * pw[j0 + q * NT];
      }
      __syncthreads();
      for (int i = t; i < R; i += NT) pnew[r0 + i] = pw[r0 + i - w0];
    } else {
      for (int i = t; i < R; i += NT) {
        const T p = dv[i] * r[i] + beta * po[i];
        po[i] = p;
        pnew[r0 + i] = p;
      }
    }
    T qa[1];
    qa[0] = rows(beta, pold);
    publish(qa);
    if (!barrier()) return;
    totals(qa);
    const bool conv = rr <= tiny;
    const T alpha = conv ? T(0) : cs_safe_div(gamma, qa[0]);
    q2[0] = q2[1] = T(0);
    for (int i = t; i < R; i += NT) {
      x[i] += alpha * po[i];
      const T rv = r[i] - alpha * ap[i];
      const T z = dv[i] * rv;
      r[i] = rv;
      a.Z[r0 + i] = z;
      q2[0] += rv * rv;
      q2[1] += rv * z;
    }
    publish(q2);
    if (!barrier()) return;
    totals(q2);
    rr = q2[0];
    beta = conv ? T(0) : cs_safe_div(q2[1], gamma);
    gamma = q2[1];
    ++it;
    if (b == nb - 1 && t == NT - 1 && a.hist) a.hist[it] = sqrt(rr);
    running = above(rr, tol_eff) && it < a.max_iters;
  }
  for (int i = t; i < R; i += NT) a.X[(int64_t)(r0 + i) * a.ldx] = x[i] * mult;
  if (b == 0 && t == 0) *a.iters = it;
}

int cg_csr_blocks(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(num_sms(), ceil_div(n, (int64_t)32))); }

constexpr int kCsSmem = 216 * 1024;

template <class T, class S>
int cg_csr_solve(CsrCgArgs<T, S>& a, int64_t nnz, cudaStream_t st, bool* ran) {
  *ran = false;
  const int nb = cg_csr_blocks(a.n);
  const size_t own = (size_t)5 * ceil_div((int64_t)a.n, (int64_t)nb) * sizeof(T);
  // a thread takes a row: rows longer than about 32 entries on average, and vectors too long for shared
  // memory beside a window of the same order, stay with the general kernel
  if (nnz > (int64_t)32 * a.n || own > (size_t)kCsSmem * 3 / 4) return COLAGB_OK;
  auto* f = k_cg_csr<T, S>;
  a.smem = kCsSmem;
  COLAGB_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, a.smem));
  int occ = 0;
  COLAGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, CsOwn<T>::threads, a.smem));
  if (occ < 1) return COLAGB_OK;
  void* args[] = {&a};
  COLAGB_CUDA(cudaLaunchCooperativeKernel((const void*)f, dim3(nb), dim3(CsOwn<T>::threads), args, a.smem, st));
  *ran = true;
  return COLAGB_OK;
}

template int cg_csr_solve<float, float>(CsrCgArgs<float, float>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<float, __nv_bfloat16>(CsrCgArgs<float, __nv_bfloat16>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<double, double>(CsrCgArgs<double, double>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<double, __nv_bfloat16>(CsrCgArgs<double, __nv_bfloat16>&, int64_t, cudaStream_t, bool*);

}  // namespace colagb
