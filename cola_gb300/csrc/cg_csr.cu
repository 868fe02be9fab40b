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
// the arithmetic itself (64 cycles of a scheduler per warp instruction: all 512 threads take rows, so
// that their loads overlap, but 128 of them form the sums and the divisions).  Before, 16 CTAs of one cluster ran matrices up to
// 32 MB: 37 us a step for 256 x 256 5-point FP64 with Jacobi; now 11.6 (FP32 6.1; the barriers and round
// trips alone take 5.6).
#include <algorithm>
#include <type_traits>

#include "cg_csr.cuh"
#include "common.cuh"

namespace colagb {

// The threads that form sums and scalars: all for FP32, one warp per scheduler for FP64 (see above).
template <class T> struct CsOwn {
  static constexpr int threads = std::is_same<T, double>::value ? 128 : 512;
  static constexpr int warps = threads / 32;
  __device__ static void sync() { asm volatile("bar.sync 1, %0;" ::"n"(threads) : "memory"); }
};

template <class T>
__device__ __forceinline__ T cs_safe_div(T num, T den) {
  const T eps = std::is_same<T, float>::value ? T(1e-40f) : T(1e-40);
  return num / (fabs(den) < eps ? eps : den);
}

// Sums of one or two values over the owning threads, each of which gets them.  buf: V * warps slots, alternated between two
// buffers.  Two values share the warp instructions: half a warp each after the first exchange, and lane q
// adds the warps' parts of value q.
template <int V, class T>
__device__ __forceinline__ void cs_sums(T (&v)[V], T* buf) {
  constexpr int W = CsOwn<T>::warps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x;
  if constexpr (V == 2) {
    const bool up = lane & 16;
    const T keep = up ? v[1] : v[0], send = up ? v[0] : v[1];
    x = keep + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((lane & 15) == 0) buf[(lane >> 4) * W + warp] = x;
  } else {
    x = warp_sum(v[0]);
    if (lane == 0) buf[warp] = x;
  }
  CsOwn<T>::sync();
  T a[W];
  const T* src = buf + (V == 2 ? (lane & 1) * W : 0);
#pragma unroll
  for (int i = 0; i < W; ++i) a[i] = src[i];
#pragma unroll
  for (int h = W / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int i = 0; i < h; ++i) a[i] += a[i + h];
  if constexpr (V == 2) {
    v[0] = __shfl_sync(0xffffffffu, a[0], 0);
    v[1] = __shfl_sync(0xffffffffu, a[0], 1);
  } else {
    v[0] = a[0];
  }
}

template <class T, class S, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_csr(const __grid_constant__ CsrCgArgs<T, S> a) {
  constexpr int OT = CsOwn<T>::threads, RED = 2 * CsOwn<T>::warps;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  __shared__ T red[2][RED];
  __shared__ T gather[2 * (NT > OT ? NT - OT : 1)];  // the other threads' terms of a sum
  __shared__ T s_scalar;
  __shared__ int s_bad, s_lo, s_hi, s_run;
  const int t = threadIdx.x, n = a.n, nb = gridDim.x, b = blockIdx.x;
  const bool owner = t < OT;
  const int r0 = (int)((int64_t)n * b / nb), R = (int)((int64_t)n * (b + 1) / nb) - r0;
  const int Rm = (n + nb - 1) / nb;
  T* const r = reinterpret_cast<T*>(cs_smem);  // own rows
  T* const x = r + Rm;
  T* const ap = x + Rm;
  T* const po = ap + Rm;                        // p of the own rows
  T* const dv = po + Rm;                        // Jacobi diagonal
  int* const rp = reinterpret_cast<int*>(dv + Rm);  // R + 1 offsets of the rows' entries
  size_t used = (size_t)5 * Rm * sizeof(T) + (size_t)(Rm + 1) * sizeof(int);
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
  for (int i = t; i <= R; i += NT) rp[i] = a.indptr[r0 + i] - e0;
  atomicMin(&s_lo, min(lo, r0));
  atomicMax(&s_hi, max(hi, r0 + R));
  __syncthreads();
  const int w0 = s_lo, W = s_hi - s_lo;
  const bool window = used + (size_t)W * sizeof(T) <= (size_t)a.smem;
  T* const pw = reinterpret_cast<T*>(cs_smem + used);
  bool too_long = false;
  for (int i = t; i < R; i += NT) too_long |= rp[i + 1] - rp[i] > a.longest;
  too_long = __syncthreads_or(too_long);
  if (t == 0 && (too_long || !window)) atomicAdd(a.votes, too_long ? (unsigned)nb + 1 : 1u);  // gathers <= nb

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
    if constexpr (NT > OT) {
      if (!owner)
#pragma unroll
        for (int q = 0; q < V; ++q) gather[q * (NT - OT) + t - OT] = v[q];
      __syncthreads();
      if (owner)
#pragma unroll
        for (int q = 0; q < V; ++q)
#pragma unroll
          for (int l = 0; l < NT / OT - 1; ++l) v[q] += gather[q * (NT - OT) + l * OT + t];
    }
    if (owner) {
      cs_sums<V, T>(v, red[rbuf]);
      if (t == 0)
#pragma unroll
        for (int q = 0; q < V; ++q) a.part[(par * 2 + q) * nb + b] = v[q];
    }
    rbuf ^= 1;
  };
  auto totals = [&](auto& v) {  // the owning threads get the sums over all CTAs
    constexpr int V = sizeof(v) / sizeof(T);
    constexpr int L = 2;  // CTAs per thread and round: 2 * 128 >= the SMs
    if (owner) {
#pragma unroll
      for (int q = 0; q < V; ++q) v[q] = T(0);
      for (int i = t; i < nb; i += L * OT) {
        T p[V][L];
#pragma unroll
        for (int q = 0; q < V; ++q)
#pragma unroll
          for (int l = 0; l < L; ++l) p[q][l] = i + l * OT < nb ? __ldcg(a.part + (par * 2 + q) * nb + i + l * OT) : T(0);
#pragma unroll
        for (int q = 0; q < V; ++q) v[q] += p[q][0] + p[q][1];
      }
      cs_sums<V, T>(v, red[rbuf]);
    }
    par ^= 1;
    rbuf ^= 1;
  };
  auto share = [&](T x) -> T {  // thread 0's value to all
    if (t == 0) s_scalar = x;
    __syncthreads();
    return s_scalar;
  };
  // Rows of A on p (window), or on z + beta * pold gathered from L2: two rows of a thread at a time, entries
  // in groups of four, so that the loads of eight entries are in flight together.
  auto rows = [&](T beta, const T* pold) -> T {
    T dot = T(0);
    for (int i = t; i < R; i += 2 * NT) {
      int e[2], end[2];
      T pi[2], acc[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = i + h * NT;
        const bool in = k < R;
        e[h] = in ? rp[k] : 0;
        end[h] = in ? rp[k + 1] : 0;
        pi[h] = !in ? T(0) : window ? pw[r0 + k - w0] : po[k];
        acc[h] = a.shift != T(0) ? a.shift * pi[h] : T(0);
      }
      while (e[0] < end[0] || e[1] < end[1]) {
        T v[2][4], p[2][4];
        int c[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const bool in = e[h] + q < end[h];
            c[h][q] = in ? cols[e[h] + q] : -1;
            v[h][q] = in ? cvt<T>(vals[e[h] + q]) : T(0);
          }
        if (window) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) p[h][q] = c[h][q] >= 0 ? pw[c[h][q] - w0] : T(0);
        } else {
          T zc[2][4];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              zc[h][q] = c[h][q] >= 0 ? __ldcg(a.Z + c[h][q]) : T(0);
              p[h][q] = c[h][q] >= 0 ? __ldcg(pold + c[h][q]) : T(0);
            }
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) p[h][q] = zc[h][q] + beta * p[h][q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (c[h][q] >= 0) acc[h] += v[h][q] * p[h][q];
        e[0] += 4;
        e[1] += 4;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = i + h * NT;
        if (k < R) {
          ap[k] = acc[h];
          if (window) po[k] = pi[h];
          dot += pi[h] * acc[h];
        }
      }
    }
    return dot;
  };
  const T tiny = std::is_same<T, float>::value ? T(0) : T(1e-80);  // |r| < 1e-40 <=> |r|^2 <= tiny

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
  if (__ldcg(a.votes) > (unsigned)a.gathers) {  // every vote was cast before the barrier: all CTAs leave
    if (b == 0 && t == 0) *a.err = kCsrLeft;
    return;
  }
  totals(q1);
  const T mult = share(owner ? sqrt(q1[0]) : T(0));
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
  // rr, gamma, tol_eff and the decisions live in the owning threads
  T rr = q2[0], gamma = q2[1], beta = T(0), tol_eff = T(0);
  int it = 0;
  if (owner) {
    const T rn = sqrt(rr);
    tol_eff = (T)a.tol * rn + (T)a.tol;
    if (b == 0 && t == 0 && a.hist) a.hist[0] = rn;
    if (t == 0) s_run = norm_above(rr, tol_eff) && it < a.max_iters;
  }
  // p of the step before, by parity: zero before the first one
  for (int i = t; i < R; i += NT) po[i] = T(0);
  if (window)
    for (int j = t; j < W; j += NT) pw[j] = T(0);
  // z of the window, fetched as soon as the barrier that publishes it is through, beside the partial sums
  constexpr int ZQ = 8;
  T zq[ZQ];
  const bool zfits = window && W <= ZQ * NT;
  auto fetch_z = [&]() {
    if (zfits)
#pragma unroll
      for (int q = 0; q < ZQ; ++q) zq[q] = t + q * NT < W ? __ldcg(a.Z + w0 + t + q * NT) : T(0);
  };
  __syncthreads();
  if (s_run) fetch_z();
  while (s_run) {
    const T* const pold = (it & 1) ? a.P1 : a.P0;
    T* const pnew = (it & 1) ? a.P0 : a.P1;
    if (zfits) {
#pragma unroll
      for (int q = 0; q < ZQ; ++q)
        if (t + q * NT < W) pw[t + q * NT] = zq[q] + beta * pw[t + q * NT];
      __syncthreads();
      for (int i = t; i < R; i += NT) pnew[r0 + i] = pw[r0 + i - w0];
    } else if (window) {
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
    const T alpha = share(owner && !conv ? cs_safe_div(gamma, qa[0]) : T(0));
    if (a.dinv) {
      q2[0] = q2[1] = T(0);
#pragma unroll 4
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
      fetch_z();
      totals(q2);
    } else {  // z = r: one sum
      q1[0] = T(0);
#pragma unroll 4
      for (int i = t; i < R; i += NT) {
        x[i] += alpha * po[i];
        const T rv = r[i] - alpha * ap[i];
        r[i] = rv;
        a.Z[r0 + i] = rv;
        q1[0] += rv * rv;
      }
      publish(q1);
      if (!barrier()) return;
      fetch_z();
      totals(q1);
      q2[0] = q2[1] = q1[0];
    }
    ++it;
    T bnew = T(0);
    if (owner) {
      rr = q2[0];
      bnew = conv ? T(0) : cs_safe_div(q2[1], gamma);
      gamma = q2[1];
      if (t == 0) s_run = norm_above(rr, tol_eff) && it < a.max_iters;
      // off the other CTAs' path: the last owning warp of the last CTA writes the history
      if (b == nb - 1 && t == OT - 1 && a.hist) a.hist[it] = sqrt(rr);
    }
    beta = share(bnew);
  }
  for (int i = t; i < R; i += NT) a.X[(int64_t)(r0 + i) * a.ldx] = x[i] * mult;
  if (b == 0 && t == 0) *a.iters = it;
}

int cg_csr_blocks(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(num_sms(), ceil_div(n, (int64_t)32))); }

constexpr int kCsSmem = 216 * 1024;

template <class T, class S, int NT>
static int cs_launch(CsrCgArgs<T, S>& a, int nb, cudaStream_t st, bool* ran) {
  auto* f = k_cg_csr<T, S, NT>;
  a.smem = kCsSmem;
  COLAGB_CUDA(set_smem_limit(f, kCsSmem));
  int occ = 0;
  COLAGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, NT, a.smem));
  if (occ < 1) return COLAGB_OK;
  void* args[] = {&a};
  COLAGB_CUDA(cudaLaunchCooperativeKernel((const void*)f, dim3(nb), dim3(NT), args, a.smem, st));
  *ran = true;
  return COLAGB_OK;
}

template <class T, class S>
int cg_csr_solve(CsrCgArgs<T, S>& a, int64_t nnz, cudaStream_t st, bool* ran) {
  *ran = false;
  const int nb = cg_csr_blocks(a.n);
  const size_t own = (size_t)ceil_div((int64_t)a.n, (int64_t)nb) * (5 * sizeof(T) + 4);
  // a thread takes a row: rows longer than about 32 entries on average, and vectors too long for shared
  // memory beside a window of the same order, stay with the general kernel
  if (nnz > (int64_t)32 * a.n || own > (size_t)kCsSmem * 3 / 4) return COLAGB_OK;
  // So do, us a step (general kernel / here, with Jacobi):
  // short FP32 vectors, whose step is one cluster's three hardware barriers there and two software ones here:
  // 64 unknowns per side 2-D 8.4 / 9.5, 90 9.1 / 9.4, 100 11.7 / 9.3; rows of 21 entries or more 12.0 / 11.1;
  if (std::is_same<T, float>::value && a.n <= 8192 && nnz <= (int64_t)16 * a.n) return COLAGB_OK;
  // matrices above 32 MB, which that kernel too spreads over all SMs (up to 32 MB it is one cluster), when
  // their rows stream past a small L1 here: 15 random entries a row, n = 300,000 FP32 64 / 91, 21 in FP64
  // 82 / 161, 31 within 5,000 columns, n = 100,000 FP64 52 / 83; 27-point 64^3 FP32 48 / 73; but 7 random entries,
  // n = 600,000 FP32 86 / 73, 9-point 900^2 74 / 27, 15 near the diagonal, n = 600,000 FP32 64 / 57, 27-point 48^3
  // FP64 (36 MB) 51 / 44;
  const double mb = (double)nnz * (sizeof(S) + 4) / (1024 * 1024);
  if ((mb > 48 && nnz > (int64_t)18 * a.n) || (mb > 32 && nnz > (int64_t)28 * a.n)) return COLAGB_OK;
  a.gathers = mb <= 32 || nnz <= (int64_t)8 * a.n ? nb : nb / 8;  // a few: the ends of a periodic grid
  // and rows of many entries, which one thread walks in both kernels: one full row, FP32 n = 30,000
  // 2193 / 1826, 100,000 7275 / 10950; FP64 n = 50 26 / 20, 500 81 / 90, 30,000 3692 / 8360.
  a.longest = std::is_same<T, float>::value ? 32768 : 256;
  // FP64: with few rows a CTA the 128 summing threads do everything (us a step with Jacobi, 128 / 512 threads:
  // 576 unknowns 8.6 / 10.0, 16,384 8.8 / 10.2, 65,536 11.7 / 11.6, 90,000 14.5 / 12.4, 262,144 23.1 / 18.1)
  if constexpr (std::is_same<T, double>::value)
    if (ceil_div((int64_t)a.n, (int64_t)nb) <= 400) return cs_launch<T, S, 128>(a, nb, st, ran);
  return cs_launch<T, S, 512>(a, nb, st, ran);
}

template int cg_csr_solve<float, float>(CsrCgArgs<float, float>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<float, __nv_bfloat16>(CsrCgArgs<float, __nv_bfloat16>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<double, double>(CsrCgArgs<double, double>&, int64_t, cudaStream_t, bool*);
template int cg_csr_solve<double, __nv_bfloat16>(CsrCgArgs<double, __nv_bfloat16>&, int64_t, cudaStream_t, bool*);

}  // namespace colagb
