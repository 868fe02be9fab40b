// Fused CG for one Dense operator (+ c*I) and up to eight right-hand sides, P = identity or Diagonal,
// with ONE exchange per step.
//
// Same loop, stop rule and history as cg.cu (run_batched_cg, cola/linalg/inverse/cg.py:94-178).  The
// vectors of a dense solve are short beside the matrix, so every CTA keeps whole copies of p, r and Ap
// in its shared memory and owns only a range of the matrix's rows.  A step is
//   own rows of A p  ->  exchange Ap  ->  <p, Ap>, r -= alpha Ap, <r, z>, |r|^2, p = z + beta p,
// everything after the exchange done by every CTA on the same numbers in the same order, so all hold
// bit-identical scalars and nothing else has to be communicated.  x is kept for the own rows.
//
// Two exchanges: GRID spreads the rows over all SMs and passes Ap through global memory (L2) at one
// software grid barrier (1.3 us on 152 CTAs); CLUSTER keeps a small matrix on 16 CTAs, stores the sums
// straight into every peer's shared memory and ends in one hardware cluster barrier.
//
// A CTA's rows stay in its shared memory for the whole solve when they fit (2048 x 2048 FP32 over 152
// CTAs: 110 KB); otherwise they stream from L2 or HBM.  The 16 warps split a row into 128-column units
// (WC of them side by side), eight rows at a time, so one 16-byte piece of p feeds eight loads of A and
// 64 KB a CTA are in flight; the partial sums of the rows are reduced together (a transposing shuffle
// tree: 9 shuffles for 8 sums).
//
// The schedules before: 16 CTAs in one cluster for matrices up to 32 MB, which two cluster reductions, a
// third barrier and 1 MB of L2 reads per CTA held at 12.9 us a step for 2048 x 2048 FP32 and 19.5 us for
// 200 x 200 FP64; several right-hand sides read the matrix once each (111 us for 3001 x 3001 BF16 x 3).
// Now 4.6, 5.3 and 11.5 us; what is left is the barrier (1.3 us), the L2 round trips around it and the
// two block sums, in FP64 also the divisions and adds themselves (64 cycles of a scheduler each).
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "cg_dense.cuh"
#include "common.cuh"

namespace colagb {

constexpr int kDcThreads = 512, kDcWarps = kDcThreads / 32, kDcCluster = 16;

template <class T>
__device__ __forceinline__ T dc_safe_div(T num, T den) {
  const T eps = std::is_same<T, float>::value ? T(1e-40f) : T(1e-40);
  return num / (fabs(den) < eps ? eps : den);
}

// Sums of V (a power of two) values over a warp.  Lane l ends with the total of value l >> (5 - log2 V).
template <int V, class T>
__device__ __forceinline__ T warp_sum_many(T (&v)[V]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int h = V / 2; h >= 1; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const T keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  T x = v[0];
  for (; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__host__ __device__ constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v / 2); }

// The threads that work on the vectors.  An FP64 instruction of a warp occupies its scheduler's FP64 unit
// for 64 cycles on this chip, so FP64 keeps one warp per scheduler busy (128 threads) and the others out
// of the sums and divisions; FP32 uses the whole CTA.
template <class T> struct DcOwn {
  static constexpr int threads = std::is_same<T, double>::value ? 128 : kDcThreads;
  static constexpr int warps = threads / 32;
  __device__ static void sync() { asm volatile("bar.sync 1, %0;" ::"n"(threads) : "memory"); }
};

template <int N, class T>
__device__ __forceinline__ T tree_sum(const T* p) {
  T a[N];
#pragma unroll
  for (int i = 0; i < N; ++i) a[i] = p[i];
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int i = 0; i < h; ++i) a[i] += a[i + h];
  return a[0];
}

// Sums of V values over the owning threads, every one of them gets the totals.  wred: V * warps slots + V
// totals, alternated by the caller between two buffers, so one (V <= 2) or two barriers are enough.
template <int V, class T>
__device__ __forceinline__ void dc_own_sums(T (&v)[V], T* wred) {
  constexpr int W = DcOwn<T>::warps, LV = ilog2(V);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T x = warp_sum_many<V, T>(v);
  if ((lane & ((32 >> LV) - 1)) == 0) wred[(lane >> (5 - LV)) * W + warp] = x;
  DcOwn<T>::sync();
  if constexpr (V <= 2) {
#pragma unroll
    for (int q = 0; q < V; ++q) v[q] = tree_sum<W>(wred + q * W);
  } else {
    T* tot = wred + V * W;
    if (threadIdx.x < V) tot[threadIdx.x] = tree_sum<W>(wred + threadIdx.x * W);
    DcOwn<T>::sync();
#pragma unroll
    for (int q = 0; q < V; ++q) v[q] = tot[q];
  }
}

template <class T, class S> __device__ __forceinline__ void dc_quad(const S* p, T v[4], bool global) {
  if constexpr (std::is_same<S, float>::value) {
    const float4 t = global ? __ldg(reinterpret_cast<const float4*>(p)) : *reinterpret_cast<const float4*>(p);
    v[0] = T(t.x); v[1] = T(t.y); v[2] = T(t.z); v[3] = T(t.w);
  } else if constexpr (std::is_same<S, double>::value) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = global ? __ldg(q) : q[0], b = global ? __ldg(q + 1) : q[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
    const uint2 t = global ? __ldg(reinterpret_cast<const uint2*>(p)) : *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
    v[0] = T(a.x); v[1] = T(a.y); v[2] = T(b.x); v[3] = T(b.y);
  }
}

// Sums of the CTA's rows r (0 <= r < R) over this warp's column units into part[(wc * R + r) * K + c].
// FORM 0: rows in shared memory (stride np, zero-padded); 1: global rows at quad boundaries, n % 4 == 0;
// 2: global rows at any address, four single elements 32 apart.
template <class T, class S, int K, int RB, int FORM>
__device__ __forceinline__ void dc_rows(const S* A, int64_t lda, int R, int n, int np, const T* p, int WC, T* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wc = warp % WC, wr = warp / WC, WR = kDcWarps / WC;
  const int U = (np + 127) / 128;
  constexpr int V = RB * K, LV = ilog2(V);
  for (int rb = wr * RB; rb < R; rb += WR * RB) {
    // One FP32 column: a quad's four products are added to each other before they join the lane's sum, so that
    // a lane's chain has a link per quad.  (A link per product, 32 of them at n = 2048, left the solutions at
    // condition 1000 1.15 times further from the exact ones.)
    constexpr bool QUADS = std::is_same<T, float>::value && K == 1;
    T acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = T(0);
    const S* row[RB];  // rows beyond R repeat the last one; their sums are not stored
#pragma unroll
    for (int i = 0; i < RB; ++i) row[i] = A + (int64_t)(rb + i < R ? rb + i : R - 1) * lda;
#pragma unroll 2
    for (int u = wc; u < U; u += WC) {
      const int j = 128 * u + (FORM == 2 ? lane : 4 * lane);
      if (FORM != 2 && j >= np) break;
      T a[RB][4];
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        if constexpr (FORM == 2) {
#pragma unroll
          for (int e = 0; e < 4; ++e) a[i][e] = j + 32 * e < n ? cvt<T>(__ldg(row[i] + j + 32 * e)) : T(0);
        } else {
          dc_quad<T, S>(row[i] + j, a[i], FORM == 1);
        }
      }
#pragma unroll
      for (int c = 0; c < K; ++c) {
        T x[4];
        if constexpr (FORM == 2) {
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = j + 32 * e < n ? p[c * np + j + 32 * e] : T(0);
        } else {
          dc_quad<T, T>(p + c * np + j, x, false);
        }
#pragma unroll
        for (int i = 0; i < RB; ++i) {
          T sum = QUADS ? T(0) : acc[i * K + c];
#pragma unroll
          for (int e = 0; e < 4; ++e) sum += a[i][e] * x[e];
          acc[i * K + c] = QUADS ? acc[i * K + c] + sum : sum;
        }
      }
    }
    const T s = warp_sum_many<V, T>(acc);
    const int id = lane >> (5 - LV);
    if ((lane & ((32 >> LV) - 1)) == 0 && rb + id / K < R) part[((size_t)wc * R + rb) * K + id] = s;
  }
}

template <class T, int K> struct DcRows {  // rows of A at a time: many, and few (FP64 with a row or two per CTA)
  static constexpr bool f64 = std::is_same<T, double>::value;
  static constexpr int many = f64 ? (K >= 8 ? 1 : K >= 4 ? 2 : 4) : (K >= 8 ? 2 : K >= 4 ? 4 : 8);
  static constexpr int few = f64 ? 1 : many;
};

template <class T, class S, int K, bool CLUSTER>
__global__ void __launch_bounds__(kDcThreads, 1) k_cg_dense(const __grid_constant__ DenseCgArgs<T, S> a) {
  namespace cgx = cooperative_groups;
  extern __shared__ __align__(16) unsigned char dc_smem[];
  const int t = threadIdx.x, n = a.n, k = a.k, np = (n + 3) / 4 * 4, nb = gridDim.x, b = blockIdx.x;
  const int r0 = (int)((int64_t)n * b / nb), R = (int)((int64_t)n * (b + 1) / nb) - r0;
  const int maxR = (n + nb - 1) / nb;
  constexpr int NV = 2 * K;  // |r|^2 and <r, z> per column
  constexpr int OT = DcOwn<T>::threads, E = 16 / (int)sizeof(T);  // owning threads, entries per 16 bytes
  constexpr int RED = NV * (DcOwn<T>::warps + 1);
  const int vec = np * K;
  T* const p = reinterpret_cast<T*>(dc_smem);   // column c at c * np
  T* const r = p + vec;
  T* const ap0 = r + vec;                        // CLUSTER: two buffers, written by the peers in turn
  T* const part = ap0 + (CLUSTER ? 2 : 1) * vec; // 16 x maxR x K row sums
  T* const xs = part + kDcWarps * maxR * K;      // own rows of x
  T* const wred = xs + (maxR * K + 3) / 4 * 4;   // two reduction buffers (As stays on a 16-byte boundary)
  S* const As = reinterpret_cast<S*>(wred + 2 * RED);
  __shared__ int s_bad, s_run;
  __shared__ T s_rr[K];
  int rbuf = 0, par = 0;
  unsigned int epoch = 0;
  const bool owner = t < OT;
  if (t == 0) s_bad = 0;

  const S* A = a.A + (int64_t)r0 * a.lda;
  if (a.resident) {
    for (int i = 0; i < R; ++i)
      for (int j = t; j < np; j += kDcThreads) As[i * np + j] = j < n ? A[(int64_t)i * a.lda + j] : S(0.f);
  }
  // p = x0 (the start), Ap's padding 0
  for (int c = 0; c < K; ++c)
    for (int i = t; i < np; i += kDcThreads) {
      p[c * np + i] = (c < k && i < n) ? a.X[(int64_t)i * a.ldx + c] : T(0);
      ap0[c * np + i] = T(0);
      if (CLUSTER) ap0[vec + c * np + i] = T(0);
    }
  for (int u = t; u < R * K; u += OT) {
    const int i = u / K, c = u - i * K;
    if (owner) xs[u] = c < k ? a.X[(int64_t)(r0 + i) * a.ldx + c] : T(0);
  }
  // |b| per column, by every CTA from the whole right-hand side
  T mult[K];
  if (owner) {
    T q[K];
#pragma unroll
    for (int c = 0; c < K; ++c) {
      q[c] = T(0);
      if (c < k)
        for (int i = t; i < n; i += OT) {
          const T v = a.B[(int64_t)i * a.ldb + c];
          q[c] += v * v;
        }
    }
    dc_own_sums<K, T>(q, wred + rbuf * RED);
    rbuf ^= 1;
#pragma unroll
    for (int c = 0; c < K; ++c) mult[c] = sqrt(q[c]);
  }
  if constexpr (CLUSTER) cgx::this_cluster().sync();  // peers' buffers are cleared before anyone writes them
  else __syncthreads();

  // Ap of the whole vector into ap (shared; the owning threads may read it); false when a barrier gave up
  auto product = [&](T*& ap) -> bool {
    constexpr int RM = DcRows<T, K>::many, RF = DcRows<T, K>::few;
    if (RF != RM && a.few) {
      if (a.resident) dc_rows<T, S, K, RF, 0>(As, np, R, n, np, p, a.wc, part);
      else if (a.aligned) dc_rows<T, S, K, RF, 1>(A, a.lda, R, n, np, p, a.wc, part);
      else dc_rows<T, S, K, RF, 2>(A, a.lda, R, n, np, p, a.wc, part);
    } else {
      if (a.resident) dc_rows<T, S, K, RM, 0>(As, np, R, n, np, p, a.wc, part);
      else if (a.aligned) dc_rows<T, S, K, RM, 1>(A, a.lda, R, n, np, p, a.wc, part);
      else dc_rows<T, S, K, RM, 2>(A, a.lda, R, n, np, p, a.wc, part);
    }
    __syncthreads();
    auto row_sum = [&](int u) {  // u = row * K + c: the column parts in order, plus the shift
      T s = part[u];
      for (int w = 1; w < a.wc; ++w) s += part[w * R * K + u];
      return s + a.shift * p[(u % K) * np + r0 + u / K];
    };
    if constexpr (CLUSTER) {
      cgx::cluster_group cl = cgx::this_cluster();
      ap = ap0 + par * vec;
      par ^= 1;
      for (int u = t; u < R * K * kDcCluster; u += kDcThreads) {
        const int v = u / kDcCluster, peer = u % kDcCluster;
        *cl.map_shared_rank(ap + (v % K) * np + r0 + v / K, peer) = row_sum(v);
      }
      cl.sync();
      return true;
    } else {
      ap = ap0;
      T* const out = a.AP + par * (int64_t)np * k;
      par ^= 1;
      for (int u = t; u < R * K; u += kDcThreads)
        if (u % K < k) out[(u % K) * np + r0 + u / K] = row_sum(u);
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
      if (s_bad) return false;
      if (owner) {  // a thread reads back only the entries it wrote
#pragma unroll(K == 1 ? 4 : 1)
        for (int i = E * t; i < np; i += E * OT) {
          float4 v[K];
#pragma unroll
          for (int c = 0; c < K; ++c)
            if (c < k) v[c] = __ldcg(reinterpret_cast<const float4*>(out + c * np + i));
#pragma unroll
          for (int c = 0; c < K; ++c)
            if (c < k) {
              const T* w = reinterpret_cast<const T*>(&v[c]);
#pragma unroll
              for (int e = 0; e < E; ++e) ap[c * np + i + e] = i + e < n ? w[e] : T(0);
            }
        }
      }
      return true;
    }
  };
  // f(c, i) for the entries i .. i + E - 1 a thread owns (the same ones in all phases)
  auto own = [&](auto f) {
    for (int i = E * t; i < np; i += E * OT)
#pragma unroll
      for (int c = 0; c < K; ++c) f(c, i);
  };
  auto m_of = [&](int i, int e) -> T { return a.dinv ? (i + e < n ? a.dinv[i + e] : T(0)) : T(1); };
  const T tiny = std::is_same<T, float>::value ? T(0) : T(1e-80);  // |r| < 1e-40 <=> |r|^2 <= tiny
  T gamma[K], tol_eff[K], rr[K];
  auto above = [&]() {  // for any column
    bool any = false;
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (c < k) any |= norm_above(rr[c], tol_eff[c]);
    return any;
  };
  int it = 0;
  // the last warp's lane 0 of CTA 0 writes the history off the other warps' path
  auto write_hist = [&]() {
    if (b == 0 && t == kDcThreads - 1 && a.hist) {
      T mean = T(0);
      for (int c = 0; c < k; ++c) mean += sqrt(s_rr[c]);
      a.hist[it] = mean / (T)k;
    }
  };

  T* ap;
  if (!product(ap)) return;
  // r = b / |b| - A x0 ; p = z = M r ; <r, z>, |r|^2
  __syncthreads();  // every warp has read x0 out of p
  if (owner) {
    T q2[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) q2[q] = T(0);
    own([&](int c, int i) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const T rv =
            (c < k && i + e < n) ? dc_safe_div(a.B[(int64_t)(i + e) * a.ldb + c], mult[c]) - ap[c * np + i + e] : T(0);
        const T z = m_of(i, e) * rv;
        r[c * np + i + e] = rv;
        p[c * np + i + e] = z;
        q2[c] += rv * rv;
        q2[K + c] += rv * z;
      }
    });
    dc_own_sums<NV, T>(q2, wred + rbuf * RED);
    rbuf ^= 1;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      rr[c] = q2[c];
      gamma[c] = q2[K + c];
      const T rn = sqrt(rr[c]);
      tol_eff[c] = (T)a.tol * rn + (T)a.tol;
      if (t == 0) s_rr[c] = rr[c];
    }
    if (t == 0) s_run = above() && it < a.max_iters;
  }
  __syncthreads();  // p, the flag and s_rr complete
  write_hist();
  while (s_run) {
    if (!product(ap)) return;
    ++it;
    if (owner) {
      T qa[K];
#pragma unroll
      for (int c = 0; c < K; ++c) qa[c] = T(0);
      own([&](int c, int i) {
#pragma unroll
        for (int e = 0; e < E; ++e) qa[c] += p[c * np + i + e] * ap[c * np + i + e];
      });
      dc_own_sums<K, T>(qa, wred + rbuf * RED);
      rbuf ^= 1;
      T alpha[K], q2[NV];
      bool conv[K];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        conv[c] = rr[c] <= tiny;
        alpha[c] = conv[c] ? T(0) : dc_safe_div(gamma[c], qa[c]);
        q2[c] = q2[K + c] = T(0);
      }
      own([&](int c, int i) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const T rv = r[c * np + i + e] - alpha[c] * ap[c * np + i + e];
          r[c * np + i + e] = rv;
          q2[c] += rv * rv;
          if (a.dinv) q2[K + c] += rv * (m_of(i, e) * rv);
        }
      });
      for (int u = t; u < R * K; u += OT) {
        T al = alpha[0];
#pragma unroll
        for (int c = 1; c < K; ++c) al = u % K == c ? alpha[c] : al;
        xs[u] += al * p[(u % K) * np + r0 + u / K];
      }
      if (a.dinv) {
        dc_own_sums<NV, T>(q2, wred + rbuf * RED);
      } else {
        T q1[K];
#pragma unroll
        for (int c = 0; c < K; ++c) q1[c] = q2[c];
        dc_own_sums<K, T>(q1, wred + rbuf * RED);
#pragma unroll
        for (int c = 0; c < K; ++c) q2[c] = q2[K + c] = q1[c];
      }
      rbuf ^= 1;
      T beta[K];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        beta[c] = conv[c] ? T(0) : dc_safe_div(q2[K + c], gamma[c]);
        gamma[c] = q2[K + c];
        rr[c] = q2[c];
        if (t == 0) s_rr[c] = rr[c];
      }
      if (t == 0) s_run = above() && it < a.max_iters;
      own([&](int c, int i) {
#pragma unroll
        for (int e = 0; e < E; ++e)
          p[c * np + i + e] = m_of(i, e) * r[c * np + i + e] + beta[c] * p[c * np + i + e];
      });
    }
    __syncthreads();  // p, the flag and s_rr complete
    write_hist();
  }
  if (owner)
    for (int u = t; u < R * K; u += OT) {
      const int i = u / K, c = u - i * K;
      T m = mult[0];
#pragma unroll
      for (int q = 1; q < K; ++q) m = c == q ? mult[q] : m;
      if (c < k) a.X[(int64_t)(r0 + i) * a.ldx + c] = xs[u] * m;
    }
  if (b == 0 && t == 0) *a.iters = it;
  if constexpr (CLUSTER) cgx::this_cluster().sync();  // no CTA leaves while a peer may still write to it
}

// ---------------------------------------------------------------------------------------------
constexpr size_t kDcSmem = 220 * 1024;
// Where 16 CTAs with the hardware barrier beat 152 with the software one, measured in us a step (16 / 152
// CTAs): FP32 n = 64 2.6 / 3.6, 500 3.0 / 3.8, 700 3.6 / 3.9, 800 (2.6 MB) 3.9 / 3.9; FP64, whose 16 SMs run
// out of FP64 units, n = 64 4.1 / 5.1, 200 (320 KB) 5.5 / 5.3, 400 8.3 / 6.5.
template <class T> constexpr size_t kDcClusterBytes = std::is_same<T, double>::value ? 200 << 10 : 2 << 20;

// Shared memory of the vectors, sums and (separately) the resident rows for nb CTAs.
template <class T, class S>
static size_t dc_smem_bytes(int64_t n, int K, int nb, bool cluster, size_t* rows_bytes) {
  const size_t np = (size_t)(n + 3) / 4 * 4, maxR = (size_t)ceil_div(n, nb), NV = 2 * (size_t)K;
  *rows_bytes = align_up(maxR * np * sizeof(S), 16);
  return sizeof(T) * ((cluster ? 4 : 3) * np * K + kDcWarps * maxR * K + (maxR * K + 3) / 4 * 4 + 2 * NV * (DcOwn<T>::warps + 1));
}

// How the warps share a CTA's R rows: wc of them side by side in a row's 128-column units, the others on
// other rows; whether rows are taken few at a time.  Least work of the busiest warp, counted in FMAs plus
// the adds of the row sums.
template <class T, int K>
static void dc_split(int64_t n, int R, int* wc, int* few) {
  const int64_t U = ceil_div(n, (int64_t)128);
  int64_t best = -1;
  for (int f = 0; f < 2; ++f) {
    const int rb = f ? DcRows<T, K>::few : DcRows<T, K>::many;
    for (int c = 1; c <= kDcWarps && (c == 1 || c <= U); c *= 2) {
      const int wr = kDcWarps / c, V = rb * K;
      const int64_t groups = ceil_div((int64_t)R, (int64_t)wr * rb);
      const int64_t w = groups * (ceil_div(U, (int64_t)c) * 4 * V + V + 5) + c - 1;
      // warps that share a scheduler take turns: idle ones make room
      const int64_t busy = std::min<int64_t>(kDcWarps, c * ceil_div((int64_t)R, (int64_t)rb));
      const int64_t cost = w * ceil_div(busy, (int64_t)4);
      if (best < 0 || cost < best) {
        best = cost;
        *wc = c;
        *few = f;
      }
    }
  }
}

template <class T, class S, int K>
static int dc_launch(DenseCgArgs<T, S>& a, cudaStream_t st, bool* ran) {
  *ran = false;
  const int64_t n = a.n;
  size_t rows_b = 0;
  // 16 CTAs while their rows and vectors fit in shared memory and the sixteenth of the matrix is read
  // from there faster than a grid barrier takes (kDcClusterBytes)
  if constexpr (K <= 2) {
  const size_t cl_b = dc_smem_bytes<T, S>(n, K, kDcCluster, true, &rows_b);
  if (n >= kDcCluster && (size_t)n * n * sizeof(S) <= kDcClusterBytes<T> && cl_b + rows_b <= kDcSmem) {
    auto* f = k_cg_dense<T, S, K, true>;
    COLAGB_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    COLAGB_CUDA(set_smem_limit(f, kDcSmem));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kDcCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kDcCluster);
    cfg.blockDim = dim3(kDcThreads);
    cfg.dynamicSmemBytes = cl_b + rows_b;
    cfg.stream = st;
    int ncl = 0;
    if (cudaOccupancyMaxActiveClusters(&ncl, f, &cfg) == cudaSuccess && ncl >= 1) {
      a.resident = 1;
      dc_split<T, K>(n, (int)ceil_div(n, (int64_t)kDcCluster), &a.wc, &a.few);
      COLAGB_CUDA(cudaLaunchKernelEx(&cfg, f, a));
      *ran = true;
      return COLAGB_OK;
    }
    cudaGetLastError();
  }
  }
  auto* f = k_cg_dense<T, S, K, false>;
  const int nb = (int)std::min<int64_t>(num_sms(), n);
  size_t smem = dc_smem_bytes<T, S>(n, K, nb, false, &rows_b);
  if (smem > kDcSmem) return COLAGB_OK;  // vectors too long: the general kernel
  a.resident = smem + rows_b <= kDcSmem;
  if (a.resident) smem += rows_b;
  // Vectors above 195 KB leave half the L1 for the rows that stream past them (us a step at n = 16,000, 16,200 and
  // 17,000, FP32: 168, 223 and 243).  One aligned FP32 column without Jacobi is faster on the general kernel then
  // (192 and 195); with Jacobi (411 and 407 there), other types and more columns are not.
  if (std::is_same<T, float>::value && std::is_same<S, float>::value && K == 1 && a.aligned && !a.dinv && !a.resident &&
      smem > 195 * 1024)
    return COLAGB_OK;
  dc_split<T, K>(n, (int)ceil_div(n, (int64_t)nb), &a.wc, &a.few);
  // rows streamed element by element: the whole CTA sweeps a row (4001 FP32: 10.4 us a step, 13.6 otherwise)
  if (!a.resident && !a.aligned)
    for (a.wc = 1; a.wc < kDcWarps && 2 * a.wc <= ceil_div(n, (int64_t)128);) a.wc *= 2;
  COLAGB_CUDA(set_smem_limit(f, kDcSmem));
  int occ = 0;
  COLAGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, kDcThreads, smem));
  if (occ < 1) return COLAGB_OK;
  void* args[] = {&a};
  COLAGB_CUDA(cudaLaunchCooperativeKernel((const void*)f, dim3(nb), dim3(kDcThreads), args, smem, st));
  *ran = true;
  return COLAGB_OK;
}

template <class T, class S>
int cg_dense_solve(DenseCgArgs<T, S>& a, cudaStream_t st, bool* ran) {
  *ran = false;
  if (a.n < 8 || a.k < 1 || a.k > 8) return COLAGB_OK;
  if (a.k == 1) return dc_launch<T, S, 1>(a, st, ran);
  if (a.k == 2) return dc_launch<T, S, 2>(a, st, ran);
  if (a.k <= 4) return dc_launch<T, S, 4>(a, st, ran);
  return dc_launch<T, S, 8>(a, st, ran);
}

template int cg_dense_solve<float, float>(DenseCgArgs<float, float>&, cudaStream_t, bool*);
template int cg_dense_solve<float, __nv_bfloat16>(DenseCgArgs<float, __nv_bfloat16>&, cudaStream_t, bool*);
template int cg_dense_solve<double, double>(DenseCgArgs<double, double>&, cudaStream_t, bool*);

}  // namespace colagb
