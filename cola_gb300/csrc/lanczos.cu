// Lanczos with full reorthogonalisation and the tridiagonal eigensolver (FP64, or FP32 for FP32 recurrences).
//
// Reference (cola/linalg/decompositions/lanczos.py):
//   init_lanczos :275-284   V[..., 1] = rhs / |rhs|, i = 1
//   lanczos_fact :235-272   while i <= max_iters and any(subdiag[i-1] > tol*subdiag[1] or i <= 1):
//       V[i] /= |V[i]| ; w = A V[i] ; diag[i-1] = <w, V[i]>
//       w -= diag[i-1] V[i] + subdiag[i-1] V[i-1] ; w = CGS2(V, w) ; V[i+1] = w ; subdiag[i] = |w| ; i++
//   do_double_gram :287-296 two passes of w -= V (V^T w) over the basis.
// The reference's CGS passes run over all max_iters+2 slots; the unfilled ones are zero, so only
// slots 1..i are visited here (same values, fewer bytes).
//
// Basis layout: slot j is an n x bs row-major block at basis + j*n*bs (probe index fastest), so
// every pass reads contiguous, coalesced rows.  Per step: 1 operator application and 2 x (V^T w then w -= V h)
// over the filled slots, with the norm summed in the last sweep and, in FP32, one dot and the three-term
// update before; short vectors fuse a subtraction with the next projection, long ones take each as a pass.
#include <cmath>
#include <string>
#include <vector>

#include <type_traits>

#include "common.cuh"
#include "ops.cuh"

namespace colagb {

template <class T>
struct LzState {
  T* nrm;         // bs
  T* hbuf;        // (max_iters + 2) x bs projection coefficients
  T* hpart;       // nblk x (max_iters + 2) x bs partial projections
  T* npart;       // nblk x bs partial norms / dots
  int* done;
  int* step;      // current i
  unsigned int* counters;
};

__device__ __forceinline__ bool lz_last_block(unsigned int* counter) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (s_last) __threadfence();
  return s_last != 0;
}

// Per-probe column reduction over rows of an n x bs block: f(r, b) summed per b.
// Block layout: threads = (rows_per_pass x bsc), bsc = min(bs, 256).
// U: rows in flight.
template <class T, int U = 1, class F>
__device__ __forceinline__ void lz_partials(int64_t n, int64_t bs, F f, T* out, T* smem) {
  const int t = threadIdx.x;
  for (int64_t b0 = 0; b0 < bs; b0 += blockDim.x) {
    const int bc = (int)((bs - b0) < (int64_t)blockDim.x ? (bs - b0) : (int64_t)blockDim.x);
    const int rpp = blockDim.x / bc;
    const int my_b = t % bc, my_r = t / bc;
    T acc = T(0);
    if (my_r < rpp)
#pragma unroll U
      for (int64_t r = (int64_t)blockIdx.x * rpp + my_r; r < n; r += (int64_t)rpp * gridDim.x) acc += f(r, b0 + my_b);
    smem[t] = acc;
    __syncthreads();
    // tree over the rpp row slots (a serial sum by one thread per column is rpp dependent
    // shared-memory round trips)
    for (int w = rpp; w > 1;) {
      const int h = (w + 1) >> 1;
      if (my_r < w - h) smem[t] += smem[t + h * bc];
      __syncthreads();
      w = h;
    }
    if (t < bc) out[b0 + t] = smem[t];
    __syncthreads();
  }
}

// The same per-column sums of a[r][b] * c[r][b] for FP32 blocks with bs a multiple of 4 (bs <= 1024):
// thread t takes column quad t % (bs / 4) and rows t / (bs / 4), t / (bs / 4) + rpp, ... with 128-bit
// loads, four rows per round on independent accumulators (a thread per column and row with scalar
// loads waited on one load at a time: ~0.6 TB/s on 64-column blocks).  Row slots are then summed in a
// fixed tree as in lz_partials.
__device__ __forceinline__ void lz_partials4(int64_t n, int64_t bs, const float* __restrict__ a,
                                             const float* __restrict__ c, float4* out4, float4* smem4) {
  const int t = threadIdx.x;
  const int qd = (int)(bs / 4);
  const int rpp = (int)blockDim.x / qd;
  const int my_q = t % qd, my_r = t / qd;
  float4 acc[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (my_r < rpp) {
    const int64_t stride = (int64_t)rpp * gridDim.x;
    int64_t r = (int64_t)blockIdx.x * rpp + my_r;
    for (; r + 3 * stride < n; r += 4 * stride) {
      float4 x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t o = (r + u * stride) * bs + 4 * my_q;
        x[u] = __ldg(reinterpret_cast<const float4*>(a + o));
        y[u] = __ldg(reinterpret_cast<const float4*>(c + o));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc[u].x += x[u].x * y[u].x;
        acc[u].y += x[u].y * y[u].y;
        acc[u].z += x[u].z * y[u].z;
        acc[u].w += x[u].w * y[u].w;
      }
    }
    float4 x[3], y[3];  // the last one to three rows, in order
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (r + u * stride < n) {
        const int64_t o = (r + u * stride) * bs + 4 * my_q;
        x[u] = __ldg(reinterpret_cast<const float4*>(a + o));
        y[u] = __ldg(reinterpret_cast<const float4*>(c + o));
      }
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (r + u * stride < n) {
        acc[0].x = fmaf(x[u].x, y[u].x, acc[0].x);
        acc[0].y = fmaf(x[u].y, y[u].y, acc[0].y);
        acc[0].z = fmaf(x[u].z, y[u].z, acc[0].z);
        acc[0].w = fmaf(x[u].w, y[u].w, acc[0].w);
      }
  }
  float4 tot;
  tot.x = (acc[0].x + acc[1].x) + (acc[2].x + acc[3].x);
  tot.y = (acc[0].y + acc[1].y) + (acc[2].y + acc[3].y);
  tot.z = (acc[0].z + acc[1].z) + (acc[2].z + acc[3].z);
  tot.w = (acc[0].w + acc[1].w) + (acc[2].w + acc[3].w);
  smem4[t] = tot;
  __syncthreads();
  for (int w = rpp; w > 1;) {
    const int h = (w + 1) >> 1;
    if (my_r < w - h) {
      const float4 o = smem4[t + h * qd];
      smem4[t].x += o.x;
      smem4[t].y += o.y;
      smem4[t].z += o.z;
      smem4[t].w += o.w;
    }
    __syncthreads();
    w = h;
  }
  if (t < qd) out4[t] = smem4[t];
  __syncthreads();
}

// Column sums of a .* c into this CTA's partials: the 128-bit path for FP32 blocks of 4..1024 columns
// and for single FP32 columns with n % 4 == 0 (16-byte aligned), the generic one otherwise.
template <class T>
__device__ __forceinline__ void lz_colsum(int64_t n, int64_t bs, const T* a, const T* c, T* out, T* smem) {
  if constexpr (std::is_same<T, float>::value) {
    const bool al = (reinterpret_cast<uintptr_t>(a) % 16) == 0 && (reinterpret_cast<uintptr_t>(c) % 16) == 0;
    if (al && bs % 4 == 0 && bs <= 1024) {
      __shared__ float4 smem4[256];
      lz_partials4(n, bs, a, c, reinterpret_cast<float4*>(out), smem4);
      return;
    }
    if (al && bs == 1 && n % 4 == 0) {  // one column: four consecutive rows per 128-bit load
      __shared__ float4 smem4b[256];
      __shared__ float4 quad;
      lz_partials4(n / 4, 4, a, c, &quad, smem4b);
      if (threadIdx.x == 0) out[0] = (quad.x + quad.y) + (quad.z + quad.w);
      __syncthreads();
      return;
    }
  }
  lz_partials<T, 4>(n, bs, [&](int64_t r, int64_t b) { return a[r * bs + b] * c[r * bs + b]; }, out, smem);
}

// Sum over the nb per-CTA partials of column b, formed by the whole block (all threads get it).
template <class T>
__device__ __forceinline__ T lz_block_total(const T* part, int nb, int64_t bs, int64_t b, T* red) {
  T v = T(0);
  for (int q = threadIdx.x; q < nb; q += blockDim.x) v += __ldcg(part + (int64_t)q * bs + b);
  return block_sum(v, red);
}

// Totals of the first kLzStage columns into shared memory, block-parallel; lz_total reads them
// (serial sum only beyond kLzStage columns).
constexpr int kLzStage = 64;
template <class T>
__device__ __forceinline__ void lz_stage(const T* part, int nb, int64_t bs, T* tot, T* red, T* scratch) {
  const int64_t kk = bs < kLzStage ? bs : kLzStage;
  if (kk >= 8 && blockDim.x % kk == 0) {
    // all columns at once: thread (b, g) sums partials g, g + G, ... of column b (consecutive threads,
    // consecutive columns), then the G group sums of each column are added in order
    const int G = (int)(blockDim.x / kk);
    const int b = (int)(threadIdx.x % kk), g = (int)(threadIdx.x / kk);
    T acc = T(0);
    constexpr int B = 16;  // loads in flight
    for (int q = g; q < nb; q += B * G) {
      T v[B];
#pragma unroll
      for (int e = 0; e < B; ++e)
        if (q + e * G < nb) v[e] = __ldcg(part + (int64_t)(q + e * G) * bs + b);
#pragma unroll
      for (int e = 0; e < B; ++e)
        if (q + e * G < nb) acc += v[e];
    }
    scratch[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < kk) {
      T sum = T(0);
      for (int gg = 0; gg < G; ++gg) sum += scratch[gg * kk + threadIdx.x];
      tot[threadIdx.x] = sum;
    }
    __syncthreads();
    return;
  }
  for (int64_t b = 0; b < kk; ++b) {
    const T v = lz_block_total(part, nb, bs, b, red);
    if (threadIdx.x == 0) tot[b] = v;
  }
  __syncthreads();
}

template <class T>
__device__ __forceinline__ T lz_sum(const T* part, int nb, int64_t bs, int64_t b) {
  T s = T(0);
  for (int q = 0; q < nb; ++q) s += __ldcg(part + (int64_t)q * bs + b);
  return s;
}

template <class T>
__device__ __forceinline__ T lz_total(const T* part, int nb, int64_t bs, int64_t b, const T* tot) {
  return b < kLzStage ? tot[b] : lz_sum(part, nb, bs, b);
}

// V[i] /= |V[i]|   (norm pass; the division is k_lz_scale)
template <class T>
__global__ void __launch_bounds__(256) k_lz_norm(const T* v, int64_t n, int64_t bs, LzState<T> s) {
  if (*s.done) return;
  __shared__ T smem[256];
  lz_colsum<T>(n, bs, v, v, s.npart + (int64_t)blockIdx.x * bs, smem);
  if (lz_last_block(s.counters + 0)) {
    __shared__ T tot[kLzStage], red[32];
    lz_stage(s.npart, gridDim.x, bs, tot, red, smem);
    for (int64_t b = threadIdx.x; b < bs; b += blockDim.x) s.nrm[b] = sqrt(lz_total(s.npart, gridDim.x, bs, b, tot));
    if (threadIdx.x == 0) s.counters[0] = 0;
  }
}

// VEC = 4: FP32 blocks of 4, 8, ... columns or a single one with n % 4 == 0, 16-byte aligned.
template <class T, int VEC>
__global__ void k_lz_scale(T* v, int64_t n, int64_t bs, LzState<T> s) {
  if (*s.done) return;
  const int64_t units = n * bs / VEC;
  const unsigned C = VEC == 4 && bs > 1 ? (unsigned)(bs / VEC) : (unsigned)bs;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += (int64_t)gridDim.x * blockDim.x) {
    const unsigned c = bs == 1 ? 0u : units < ((int64_t)1 << 32) ? (unsigned)u % C : (unsigned)(u % C);
    if constexpr (VEC == 4) {
      float4* p = reinterpret_cast<float4*>(v) + u;
      float4 x = *p;
      if (bs == 1) {
        const float d = s.nrm[0];
        x.x /= d; x.y /= d; x.z /= d; x.w /= d;
      } else {
        const float4 d = reinterpret_cast<const float4*>(s.nrm)[c];
        x.x /= d.x; x.y /= d.y; x.z /= d.z; x.w /= d.w;
      }
      *p = x;
    } else {
      v[u] = v[u] / s.nrm[c];
    }
  }
}

// diag[b][i-1] = <w, V[i]>
__global__ void __launch_bounds__(256) k_lz_alpha(const float* w, const float* vi, int64_t n, int64_t bs, float* diag,
                                                  int max_iters, LzState<float> s) {
  if (*s.done) return;
  __shared__ float smem[256];
  lz_colsum<float>(n, bs, w, vi, s.npart + (int64_t)blockIdx.x * bs, smem);
  if (lz_last_block(s.counters + 1)) {
    __shared__ float tot[kLzStage], red[32];
    lz_stage(s.npart, gridDim.x, bs, tot, red, smem);
    const int i = *s.step;
    for (int64_t b = threadIdx.x; b < bs; b += blockDim.x)
      diag[b * max_iters + (i - 1)] = lz_total(s.npart, gridDim.x, bs, b, tot);
    if (threadIdx.x == 0) s.counters[1] = 0;
  }
}

// ---------------------------------------------------------------------------------------------
// FP32 step after w = A V[i] (bs probes):
//   k_lz_alpha      diag[i-1] = <w, V[i]>
//   TERMS_PROJ      w -= diag[i-1] V[i] + subdiag[i-1] V[i-1] as the run is staged, then h1 = V^T w
//   SUB_PROJ        w -= V h1, then h2 = V^T w on the same run: the second read of a run's slots follows
//                   the first at once and hits L1 / L2
//   k_lz_fin        w -= V h2 with |w| per column summed on the way; the last CTA does the bookkeeping
// and a reduction of the CTAs' partial projections after each projection.  A single FP32 vector's sums
// decide the last bits of the quadrature, so every sum keeps one fixed order: the partition into runs,
// the lane and slot-team orders below and the plain order of j for each element of w.  Before, the
// three-term update, the two subtractions and a second norm of the same vector were sweeps and launches
// of their own (12 a step beside the operator; now 7), and the reduction read its partials 4 bytes per
// sector (7.2 us for 40 x 16 sums of 608 partials).
enum { LZ_TERMS_PROJ = 0, LZ_SUB_PROJ = 1 };

struct LzStep {
  const float* basis;
  float* w;                // slot i + 1
  const float *vi, *vim1;  // slots i, i - 1
  const float *diag, *subdiag;
  int64_t n, bs, chunk;    // chunk: rows of a CTA's run
  int64_t slots;
  int max_iters;
  LzState<float> s;
};

__device__ __forceinline__ float lz_term(float w, float d, float vi, float sb, float vim1) {
  return w - fmaf(d, vi, sb * vim1);
}

// (fmaf is written out where an addition is predicated: the compiler may otherwise select the product and
// add it, rounding twice.)
// sum over j = 1..i, in that order, of V[j] h[j] at one / two / four entries (offset o, column(s) of h).  The
// loads of a batch of slots are issued together, the last batch predicated: a remainder loop would wait
// for one load at a time (74 us instead of 30 for 20 slots of 1.8M entries).
__device__ __forceinline__ float lz_comb1(const float* basis, int64_t N, int64_t o, const float* h, int64_t bs, int i) {
  constexpr int B = 16;
  float acc = 0.f;
  const float* v = basis + N + o;
  for (int j = 1; j <= i; j += B, v += B * N) {
    float x[B], c[B];
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (j + q <= i) {
        x[q] = __ldg(v + q * N);
        c[q] = __ldg(h + (int64_t)(j + q) * bs);
      }
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (j + q <= i) acc = fmaf(x[q], c[q], acc);
  }
  return acc;
}
__device__ __forceinline__ float2 lz_comb2(const float* basis, int64_t N, int64_t o, const float* h, int i) {
  constexpr int B = 16;
  float2 acc = make_float2(0.f, 0.f);
  const float* v = basis + N + o;
  for (int j = 1; j <= i; j += B, v += B * N) {
    float2 x[B];
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (j + q <= i) x[q] = __ldg(reinterpret_cast<const float2*>(v + q * N));
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (j + q <= i) {
        const float c = h[j + q];
        acc.x = fmaf(x[q].x, c, acc.x);
        acc.y = fmaf(x[q].y, c, acc.y);
      }
  }
  return acc;
}
template <bool ONE, int B>
__device__ __forceinline__ float4 lz_comb4(const float* basis, int64_t N, int64_t o, const float* h, int64_t bs, int i) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* v = basis + N + o;
  for (int j = 1; j <= i; j += B, v += B * N) {
    float4 x[B];
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (j + q <= i) x[q] = __ldg(reinterpret_cast<const float4*>(v + q * N));
    if constexpr (ONE) {
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (j + q <= i) {
          const float c = __ldg(h + j + q);
          acc.x = fmaf(x[q].x, c, acc.x);
          acc.y = fmaf(x[q].y, c, acc.y);
          acc.z = fmaf(x[q].z, c, acc.z);
          acc.w = fmaf(x[q].w, c, acc.w);
        }
    } else {
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (j + q <= i) {
          const float4 c = __ldg(reinterpret_cast<const float4*>(h + (int64_t)(j + q) * bs));
          acc.x = fmaf(x[q].x, c.x, acc.x);
          acc.y = fmaf(x[q].y, c.y, acc.y);
          acc.z = fmaf(x[q].z, c.z, acc.z);
          acc.w = fmaf(x[q].w, c.w, acc.w);
        }
    }
  }
  return acc;
}

// Single vector (bs == 1, n % 4 == 0): a CTA's run is `chunk` rows (a multiple of 128); a warp takes whole
// slots, its lanes stream the run with 128-bit loads against w from shared memory.
template <int MODE>
__global__ void __launch_bounds__(512, 2) k_lz_proj1(const __grid_constant__ LzStep a) {
  const LzState<float>& s = a.s;
  if (*s.done) return;
  constexpr int B = 8;
  extern __shared__ float4 wsm[];
  const int i = *s.step;
  const int64_t n = a.n, r0 = (int64_t)blockIdx.x * a.chunk;
  const int64_t r1 = r0 + a.chunk < n ? r0 + a.chunk : n;
  const int n2 = (int)((r1 - r0) / 2), n4 = n2 / 2;
  float2* w2 = reinterpret_cast<float2*>(a.w + r0);
  const float d = MODE == LZ_TERMS_PROJ ? a.diag[i - 1] : 0.f, sb = MODE == LZ_TERMS_PROJ ? a.subdiag[i - 1] : 0.f;
  float* const hs = reinterpret_cast<float*>(wsm) + a.chunk;  // the coefficients, behind the run
  if (MODE == LZ_SUB_PROJ) {
    for (int j = threadIdx.x; j <= i; j += blockDim.x) hs[j] = s.hbuf[j];
    __syncthreads();
  }
  for (int u = threadIdx.x; u < n2; u += blockDim.x) {
    float2 x = w2[u];
    if (MODE == LZ_TERMS_PROJ) {
      const float2 p = reinterpret_cast<const float2*>(a.vi + r0)[u], q = reinterpret_cast<const float2*>(a.vim1 + r0)[u];
      x.x = lz_term(x.x, d, p.x, sb, q.x);
      x.y = lz_term(x.y, d, p.y, sb, q.y);
    } else {
      const float2 c = lz_comb2(a.basis, n, r0 + 2 * u, hs, i);
      x.x -= c.x;
      x.y -= c.y;
    }
    w2[u] = x;
    reinterpret_cast<float2*>(wsm)[u] = x;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* out = s.hpart + (int64_t)blockIdx.x * a.slots;
  for (int j = 1 + warp; j <= i; j += nw) {
    const float4* v4 = reinterpret_cast<const float4*>(a.basis + (int64_t)j * n + r0);
    float acc0 = 0.f, acc1 = 0.f;  // even and odd 32-quad pieces
    for (int u = lane; u < n4; u += 32 * B) {
      float4 v[B];
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (u + 32 * q < n4) v[q] = __ldg(v4 + u + 32 * q);
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (u + 32 * q < n4) {
          const float4 p = v[q], x = wsm[u + 32 * q];
          const float d4 = fmaf(p.w, x.w, fmaf(p.z, x.z, fmaf(p.x, x.x, p.y * x.y)));
          if (q % 2 == 0) acc0 += d4;
          else acc1 += d4;
        }
    }
    const float t = warp_sum(acc0 + acc1);
    if (lane == 0) out[j] = t;
  }
}

// Block form (bs in {4, 8, ..., 128}): a run is chunk * bs contiguous floats per slot, a whole number of
// 128-float warp steps, so lane l always holds column quad l % (bs / 4).
template <int MODE>
__global__ void __launch_bounds__(512, 2) k_lz_projq(const __grid_constant__ LzStep a) {
  const LzState<float>& s = a.s;
  if (*s.done) return;
  constexpr int B = 8;
  extern __shared__ float4 wsm[];
  const int i = *s.step;
  const int64_t n = a.n, bs = a.bs, N = n * bs, r0 = (int64_t)blockIdx.x * a.chunk;
  const int64_t r1 = r0 + a.chunk < n ? r0 + a.chunk : n;
  const int n4 = (int)((r1 - r0) * bs / 4), qd = (int)(bs / 4);  // qd: a power of two in [1, 32]
  float4* w4 = reinterpret_cast<float4*>(a.w + r0 * bs);
  for (int u = threadIdx.x; u < n4; u += blockDim.x) {
    float4 x = w4[u];
    const int b = 4 * (u & (qd - 1));
    if (MODE == LZ_TERMS_PROJ) {
      const float4 p = reinterpret_cast<const float4*>(a.vi + r0 * bs)[u], q = reinterpret_cast<const float4*>(a.vim1 + r0 * bs)[u];
      const float* dg = a.diag + (int64_t)b * a.max_iters + (i - 1);
      const float* sb = a.subdiag + (int64_t)b * (a.max_iters + 1) + (i - 1);
      const int64_t m = a.max_iters;
      x.x = lz_term(x.x, __ldg(dg), p.x, __ldg(sb), q.x);
      x.y = lz_term(x.y, __ldg(dg + m), p.y, __ldg(sb + (m + 1)), q.y);
      x.z = lz_term(x.z, __ldg(dg + 2 * m), p.z, __ldg(sb + 2 * (m + 1)), q.z);
      x.w = lz_term(x.w, __ldg(dg + 3 * m), p.w, __ldg(sb + 3 * (m + 1)), q.w);
    } else {
      const float4 c = lz_comb4<false, 8>(a.basis, N, r0 * bs + 4 * u, s.hbuf + b, bs, i);
      x.x -= c.x;
      x.y -= c.y;
      x.z -= c.z;
      x.w -= c.w;
    }
    w4[u] = x;
    wsm[u] = x;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* out = s.hpart + (int64_t)blockIdx.x * a.slots * bs;
  for (int j = 1 + warp; j <= i; j += nw) {
    const float4* v4 = reinterpret_cast<const float4*>(a.basis + (int64_t)j * N + r0 * bs);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), acc2 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int u = lane; u < n4; u += 32 * B) {  // even 32-quad pieces into acc, odd ones into acc2
      float4 v[B];
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (u + 32 * q < n4) v[q] = __ldg(v4 + u + 32 * q);
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (u + 32 * q < n4) {
          const float4 p = v[q], x = wsm[u + 32 * q];
          float4& d = q % 2 == 0 ? acc : acc2;
          d.x = fmaf(p.x, x.x, d.x); d.y = fmaf(p.y, x.y, d.y); d.z = fmaf(p.z, x.z, d.z); d.w = fmaf(p.w, x.w, d.w);
        }
    }
    acc.x += acc2.x; acc.y += acc2.y; acc.z += acc2.z; acc.w += acc2.w;
    for (int o = 16; o >= qd; o >>= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
      acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
      acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
    }
    if (lane < qd) reinterpret_cast<float4*>(out + (int64_t)j * bs)[lane] = acc;
  }
}

// Partial projections of rows [r0, r1) on slots j0 .. j0 + 3 for j0 = first, first + stride, ... <= i, by 256 threads
// (t of them, sync() their barrier, smem 4 x 256): threads are rows x columns, w is read once for four slots
// and the four sums share one tree over the rows.
constexpr int kLzTeam = 256, kLzSlots = 4;
template <class T, int U, class Sync>
__device__ __forceinline__ void lz_project_rows(const T* basis, const T* w, int64_t N, int64_t bs, int64_t r0, int64_t r1,
                                                int first, int stride, int i, T* out, T* smem, int t, Sync sync) {
  constexpr int JB = kLzSlots, TT = kLzTeam;
  for (int64_t b0 = 0; b0 < bs; b0 += TT) {
    const int bc = (int)((bs - b0) < TT ? (bs - b0) : TT);
    const int rpp = TT / bc;
    const int my_b = t % bc, my_r = t / bc;
    for (int j0 = first; j0 <= i; j0 += stride) {
      const int nj = (i - j0 + 1) < JB ? (i - j0 + 1) : JB;
      T acc[JB] = {T(0), T(0), T(0), T(0)};
      if (my_r < rpp) {
        const T* v0 = basis + (int64_t)j0 * N + b0 + my_b;
        // U rows' loads in flight together, the terms added in row order
        for (int64_t r = r0 + my_r; r < r1; r += U * rpp) {
          T wv[U], v[U][JB];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int64_t o = (r + u * rpp) * bs;
            const bool in = r + u * rpp < r1;
            wv[u] = in ? w[o + b0 + my_b] : T(0);
#pragma unroll
            for (int q = 0; q < JB; ++q) v[u][q] = in && q < nj ? v0[(int64_t)q * N + o] : T(0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (r + u * rpp < r1) {
#pragma unroll
              for (int q = 0; q < JB; ++q) acc[q] = fma(v[u][q], wv[u], acc[q]);
            }
        }
      }
#pragma unroll
      for (int q = 0; q < JB; ++q) smem[q * TT + t] = acc[q];
      sync();
      for (int wd = rpp; wd > 1;) {  // tree over the row slots, all JB sums at once
        const int h = (wd + 1) >> 1;
        if (my_r < wd - h) {
#pragma unroll
          for (int q = 0; q < JB; ++q) smem[q * TT + t] += smem[q * TT + t + h * bc];
        }
        sync();
        wd = h;
      }
      if (t < bc) {
        for (int q = 0; q < nj; ++q) out[(int64_t)(j0 + q) * bs + b0 + t] = smem[q * TT + t];
      }
      sync();
    }
  }
}

// Any bs, short vectors: a run is `chunk` rows; teams of 256 threads take four slots at a time (team q the
// groups q, q + 4, ...).
constexpr int kLzTeams = 4;
template <int MODE>
__global__ void __launch_bounds__(256 * kLzTeams) k_lz_projx(const __grid_constant__ LzStep a) {
  const LzState<float>& s = a.s;
  if (*s.done) return;
  __shared__ float smem_all[kLzTeams * kLzSlots * kLzTeam];
  const int i = *s.step;
  const int64_t n = a.n, bs = a.bs, N = n * bs;
  const int64_t r0 = (int64_t)blockIdx.x * a.chunk < n ? (int64_t)blockIdx.x * a.chunk : n;
  const int64_t r1 = r0 + a.chunk < n ? r0 + a.chunk : n;
  float* const w = a.w;
  for (int64_t u = r0 * bs + threadIdx.x; u < r1 * bs; u += blockDim.x) {
    const int64_t b = u % bs;
    if (MODE == LZ_TERMS_PROJ)
      w[u] = lz_term(w[u], a.diag[b * a.max_iters + (i - 1)], a.vi[u], a.subdiag[b * (a.max_iters + 1) + (i - 1)], a.vim1[u]);
    else
      w[u] -= lz_comb1(a.basis, N, u, s.hbuf + b, bs, i);
  }
  __syncthreads();
  const int team = threadIdx.x / kLzTeam;
  lz_project_rows<float, 1>(a.basis, w, N, bs, r0, r1, 1 + kLzSlots * team, kLzSlots * kLzTeams, i,
                         s.hpart + (int64_t)blockIdx.x * a.slots * bs, smem_all + team * kLzSlots * kLzTeam,
                         threadIdx.x % kLzTeam, [&]() { asm volatile("bar.sync %0, 256;" ::"r"(team + 1) : "memory"); });
}

// The same sums and updates as passes of their own, for long vectors: every pass then streams with all the
// loads an SM can hold, where the fused kernels wait for one run at a time.  One CTA's run of rows is the
// projx kernel's, so the sums are the same to the bit.
template <class T>
__global__ void __launch_bounds__(kLzTeam, 4) k_lz_project(const T* basis, const T* w, int64_t n, int64_t bs, int64_t slots,
                                                        LzState<T> s) {
  if (*s.done) return;
  __shared__ T smem[kLzSlots * kLzTeam];
  const int64_t chunk = ceil_div(n, (int64_t)gridDim.x);
  const int64_t r0 = (int64_t)blockIdx.x * chunk < n ? (int64_t)blockIdx.x * chunk : n;
  const int64_t r1 = r0 + chunk < n ? r0 + chunk : n;
  // two rows at a time (one, at the compiler's choice: 2.4 instead of 0.95 ms for 64 columns of 1,000,000 FP32
  // rows and 12 slots), within the 64 registers of four CTAs an SM
  lz_project_rows<T, 2>(basis, w, n * bs, bs, r0, r1, 1, kLzSlots, *s.step, s.hpart + (int64_t)blockIdx.x * slots * bs, smem,
                     threadIdx.x, []() { __syncthreads(); });
}

// w -= diag[i-1] V[i] + subdiag[i-1] V[i-1]
__global__ void k_lz_terms(const __grid_constant__ LzStep a) {
  if (*a.s.done) return;
  const int i = *a.s.step;
  const int64_t N = a.n * a.bs, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < N; u += step) {
    const int64_t b = u % a.bs;
    a.w[u] = lz_term(a.w[u], a.diag[b * a.max_iters + (i - 1)], a.vi[u], a.subdiag[b * (a.max_iters + 1) + (i - 1)], a.vim1[u]);
  }
}

// w -= sum_j V[j] h[j], j = 1..i in order.  FORM 0: any bs; 1: float4 of blocks with bs % 4 == 0; 2: float4 of
// one column.  The grid is eight CTAs an SM for the quads and four for single entries, of which a thread takes
// four at a time; fewer loads in flight, or registers for fewer CTAs, were slower by up to two times.
template <class T, int FORM>
__global__ void __launch_bounds__(256, FORM == 1 ? 8 : FORM == 2 ? 5 : 4) k_lz_subtract(const T* basis, T* w, int64_t n, int64_t bs, LzState<T> s) {
  if (*s.done) return;
  const int i = *s.step;
  const int64_t N = n * bs, step = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = FORM ? 1 : 4;
  const bool narrow = N < ((int64_t)1 << 32);  // 32-bit remainders
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < (FORM ? N / 4 : N); u += U * step) {
    if constexpr (FORM != 0) {
      const int64_t b = FORM == 2 ? 0 : 4 * u % bs;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int j = 1; j <= i; ++j) {
        const float4 v = reinterpret_cast<const float4*>(basis + (int64_t)j * N)[u];
        const float* h = s.hbuf + (int64_t)j * bs + b;
        acc.x += v.x * h[0];
        acc.y += v.y * h[FORM == 2 ? 0 : 1];
        acc.z += v.z * h[FORM == 2 ? 0 : 2];
        acc.w += v.w * h[FORM == 2 ? 0 : 3];
      }
      float4 x = reinterpret_cast<const float4*>(w)[u];
      x.x -= acc.x;
      x.y -= acc.y;
      x.z -= acc.z;
      x.w -= acc.w;
      reinterpret_cast<float4*>(w)[u] = x;
    } else {
      T acc[U];
      const T *v[U], *h[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int64_t o = u + q * step < N ? u + q * step : u;  // past the end: the first one again, not stored
        acc[q] = T(0);
        v[q] = basis + o;
        h[q] = s.hbuf + (narrow ? (int64_t)((uint32_t)o % (uint32_t)bs) : o % bs);
      }
#pragma unroll 2
      for (int j = 1; j <= i; ++j)
#pragma unroll
        for (int q = 0; q < U; ++q) acc[q] = fma(__ldg(v[q] + (int64_t)j * N), __ldg(h[q] + (int64_t)j * bs), acc[q]);
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (u + q * step < N) w[u + q * step] -= acc[q];
    }
  }
}

static unsigned lz_sweep_blocks(int64_t units, int per_sm = 8) {
  return (unsigned)std::min<int64_t>(std::max<int64_t>(ceil_div(units, (int64_t)256), 1), (int64_t)num_sms() * per_sm);
}

// h[j][b] = sum over the CTAs of hpart: 32 interleaved sums, then a tree over them.  32 neighbouring (j, b)
// per CTA so that the partials are read by whole sectors.
__global__ void __launch_bounds__(1024) k_lz_reduce32(int nblk, int64_t bs, int64_t slots, LzState<float> s) {
  if (*s.done) return;
  __shared__ float part[32][33];
  const int i = *s.step;
  const int64_t total = (int64_t)(i + 1) * bs;
  const int l = threadIdx.x & 31, q0 = threadIdx.x >> 5;
  for (int64_t u0 = (int64_t)blockIdx.x * 32; u0 < total; u0 += (int64_t)gridDim.x * 32) {
    float acc = 0.f;
    const int64_t u = u0 + l;
    if (u < total && u >= bs) {  // slot 0 is the zero vector
      constexpr int B = 10;      // loads in flight
      for (int q = q0; q < nblk; q += 32 * B) {
        float v[B];
#pragma unroll
        for (int e = 0; e < B; ++e)
          if (q + 32 * e < nblk) v[e] = __ldg(s.hpart + (int64_t)(q + 32 * e) * slots * bs + u);
#pragma unroll
        for (int e = 0; e < B; ++e)
          if (q + 32 * e < nblk) acc += v[e];
      }
    }
    part[q0][l] = acc;
    __syncthreads();
    const float h = warp_sum(part[l][q0]);
    if (l == 0 && u0 + q0 < total) s.hbuf[u0 + q0] = h;
    __syncthreads();
  }
}

// The end of a Lanczos step, by the last CTA: subdiag[b][i] = |w| from the CTAs' sums of squares, i += 1 and
// the stop test of lanczos_fact.cond_fun.  Without subdiag (Arnoldi) only the norms are left in nrm.
template <class T>
__device__ __forceinline__ void lz_step_end(const LzState<T>& s, int64_t bs, int i, T* subdiag, int max_iters, double tol,
                                            T* scratch) {
  __shared__ int s_any;
  __shared__ T tot[kLzStage], red[32];
  lz_stage(s.npart, gridDim.x, bs, tot, red, scratch);
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  for (int64_t b = threadIdx.x; b < bs; b += blockDim.x) {
    const T nv = sqrt(lz_total(s.npart, gridDim.x, bs, b, tot));
    s.nrm[b] = nv;  // what V[i + 1] is divided by
    if (subdiag) {
      subdiag[b * (max_iters + 1) + i] = nv;
      const T first = subdiag[b * (max_iters + 1) + 1];
      if (nv > (T)tol * first) atomicOr(&s_any, 1);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (subdiag) {
      const int ni = i + 1;
      *s.step = ni;
      *s.done = !(ni <= max_iters && (s_any || ni <= 1));
    }
    s.counters[2] = 0;
  }
}

// |w| per column and the end of the step, w complete.
template <class T>
__global__ void __launch_bounds__(256) k_lz_finish(const T* w, int64_t n, int64_t bs, T* subdiag, int max_iters,
                                                   double tol, LzState<T> s) {
  if (*s.done) return;
  __shared__ T smem[256];
  lz_colsum<T>(n, bs, w, w, s.npart + (int64_t)blockIdx.x * bs, smem);
  if (lz_last_block(s.counters + 2)) lz_step_end<T>(s, bs, *s.step, subdiag, max_iters, tol, smem);
}

// The last subtraction with the sums of squares of lz_colsum on the way (the same rows per thread), then
// subdiag[b][i] = |w|, i += 1 and the stop test of lanczos_fact.cond_fun in the last CTA.
// FORM 0: any bs; 1: float4 of blocks with bs % 4 == 0; 2: float4 of one column.
template <int FORM>
__global__ void __launch_bounds__(256, FORM == 1 ? 4 : 2) k_lz_fin(const __grid_constant__ LzStep a, float* subdiag, double tol) {
  const LzState<float>& s = a.s;
  if (*s.done) return;
  __shared__ float4 smem4[256];
  float* const smem = reinterpret_cast<float*>(smem4);
  const int i = *s.step, t = threadIdx.x;
  const int64_t n = a.n, bs = a.bs, N = n * bs;
  float* const out = s.npart + (int64_t)blockIdx.x * bs;
  constexpr bool one = FORM == 2;
  if constexpr (FORM != 0) {
    const int64_t rows = one ? n / 4 : n;  // a single column: rows of four entries
    const int qd = one ? 1 : (int)(bs / 4), rpp = 256 / qd;
    const int my_q = t % qd, my_r = t / qd;
    float4 acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (my_r < rpp) {
      // rounds of four rows on four accumulators, the last one to three rows all on the first
      const int64_t stride = (int64_t)rpp * gridDim.x;
      for (int64_t r = (int64_t)blockIdx.x * rpp + my_r; r < rows; r += 4 * stride) {
        const bool full = r + 3 * stride < rows;
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
          const int64_t ru = r + u * stride;
          if (ru >= rows) break;
          const int64_t o = (ru * qd + my_q) * 4;
          float4 x = *reinterpret_cast<const float4*>(a.w + o);
          const float4 c = lz_comb4<one, one ? 16 : 6>(a.basis, N, o, s.hbuf + (one ? 0 : 4 * my_q), bs, i);
          x.x -= c.x;
          x.y -= c.y;
          x.z -= c.z;
          x.w -= c.w;
          *reinterpret_cast<float4*>(a.w + o) = x;
          const int to = full ? u : 0;
#pragma unroll
          for (int d = 0; d < 4; ++d)
            if (to == d) {
              acc[d].x = fmaf(x.x, x.x, acc[d].x);
              acc[d].y = fmaf(x.y, x.y, acc[d].y);
              acc[d].z = fmaf(x.z, x.z, acc[d].z);
              acc[d].w = fmaf(x.w, x.w, acc[d].w);
            }
        }
      }
    }
    float4 tot;
    tot.x = (acc[0].x + acc[1].x) + (acc[2].x + acc[3].x);
    tot.y = (acc[0].y + acc[1].y) + (acc[2].y + acc[3].y);
    tot.z = (acc[0].z + acc[1].z) + (acc[2].z + acc[3].z);
    tot.w = (acc[0].w + acc[1].w) + (acc[2].w + acc[3].w);
    smem4[t] = tot;
    __syncthreads();
    for (int w = rpp; w > 1;) {
      const int h = (w + 1) >> 1;
      if (my_r < w - h) {
        const float4 o = smem4[t + h * qd];
        smem4[t].x += o.x;
        smem4[t].y += o.y;
        smem4[t].z += o.z;
        smem4[t].w += o.w;
      }
      __syncthreads();
      w = h;
    }
    if (one) {
      if (t == 0) out[0] = (smem4[0].x + smem4[0].y) + (smem4[0].z + smem4[0].w);
    } else if (t < qd) {
      reinterpret_cast<float4*>(out)[t] = smem4[t];
    }
    __syncthreads();
  } else {
    lz_partials<float>(n, bs,
                       [&](int64_t r, int64_t b) {
                         const int64_t o = r * bs + b;
                         const float x = a.w[o] - lz_comb1(a.basis, N, o, s.hbuf + b, bs, i);
                         a.w[o] = x;
                         return x * x;
                       },
                       out, smem);
  }
  if (lz_last_block(s.counters + 2)) lz_step_end<float>(s, bs, i, subdiag, a.max_iters, tol, smem);
}

// Which projection form a run of the FP32 method uses, and its launch shape (nb: the partials' capacity).
struct LzForm {
  int form = 2;  // 0: k_lz_proj1, 1: k_lz_projq, 2: k_lz_projx, 3: passes of their own
  int blocks = 1;
  int64_t chunk = 0;
  size_t smem = 0;
};
// Blocks of more entries than this that have no staged form take their passes one by one.  ms for 24 steps of an
// FP32 block, staged in teams / pass by pass: 50,000 x 3 1.60 / 1.87, 100,000 x 3 2.08 / 2.11, 50,000 x 7 2.70 / 2.55,
// 100,000 x 10 4.28 / 3.59, 1,000,000 x 7 24.7 / 13.2.
constexpr int64_t kLzSplit = 320 * 1024;
constexpr size_t kLzRunSmem = 160 * 1024, kLzProj1Smem = 220 * 1024;
static int lz_form(const float* basis, int64_t n, int64_t bs, int nb, int64_t slots, LzForm& f) {
  const bool al = (uintptr_t)basis % 16 == 0;
  f.blocks = nb;
  f.chunk = ceil_div(n, (int64_t)nb);
  if (n * bs > kLzSplit) f.form = 3;
  int64_t step = 0;
  if (bs == 1 && n % 4 == 0 && al) step = 128;
  else if (bs >= 4 && bs <= 128 && (bs & (bs - 1)) == 0 && al) step = 128 / bs;
  if (step == 0) return COLAGB_OK;
  const int64_t chunk = ceil_div(f.chunk, step) * step;  // a whole number of 128-float warp steps
  size_t smem = (size_t)(chunk * bs) * sizeof(float);
  if (smem > kLzRunSmem) return COLAGB_OK;
  if (bs == 1) {  // the single-vector form keeps the coefficients in shared memory, too
    smem += (size_t)slots * sizeof(float);
    if (smem > kLzProj1Smem) return COLAGB_OK;
  }
  f.form = bs == 1 ? 0 : 1;
  f.chunk = chunk;
  f.blocks = (int)ceil_div(n, chunk);
  f.smem = smem;
  if (f.form == 0) {
    COLAGB_CUDA(set_smem_limit(k_lz_proj1<0>, kLzProj1Smem));
    COLAGB_CUDA(set_smem_limit(k_lz_proj1<1>, kLzProj1Smem));
  } else {
    COLAGB_CUDA(set_smem_limit(k_lz_projq<0>, kLzRunSmem));
    COLAGB_CUDA(set_smem_limit(k_lz_projq<1>, kLzRunSmem));
  }
  return COLAGB_OK;
}

// A warp takes whole slots: as many warps (8 to 16) as share i slots evenly.
template <int MODE>
static void lz_project(const LzForm& f, const LzStep& a, int i, cudaStream_t st) {
  const int rounds = (i + 15) / 16, warps = std::max(8, (i + rounds - 1) / rounds);
  if (f.form == 0) k_lz_proj1<MODE><<<f.blocks, 32 * warps, f.smem, st>>>(a);
  else if (f.form == 1) k_lz_projq<MODE><<<f.blocks, 32 * warps, f.smem, st>>>(a);
  else k_lz_projx<MODE><<<f.blocks, 256 * kLzTeams, 0, st>>>(a);
}

// Everything of a step after the operator's product, w = slot i + 1 holding A V[i].
static int lz_step_f32(const LzForm& f, const LzStep& a, int i, int nb, float* diag, float* subdiag, double tol,
                       cudaStream_t st) {
  const unsigned rb = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div((int64_t)(i + 1) * a.bs, 32), 4096));
  // the 128-bit form where lz_colsum takes it: blocks of 4, 8, ... columns and single ones with n % 4 == 0
  const bool quads = (uintptr_t)a.basis % 16 == 0 && (uintptr_t)a.w % 16 == 0 &&
                     ((a.bs == 1 && a.n % 4 == 0) || (a.bs % 4 == 0 && a.bs <= 1024));
  auto subtract = [&]() {
    const int64_t N = a.n * a.bs;
    if (!quads) k_lz_subtract<float, 0><<<lz_sweep_blocks(N, 4), 256, 0, st>>>(a.basis, a.w, a.n, a.bs, a.s);
    else if (a.bs == 1) k_lz_subtract<float, 2><<<lz_sweep_blocks(N / 4), 256, 0, st>>>(a.basis, a.w, a.n, a.bs, a.s);
    else k_lz_subtract<float, 1><<<lz_sweep_blocks(N / 4), 256, 0, st>>>(a.basis, a.w, a.n, a.bs, a.s);
  };
  k_lz_alpha<<<nb, 256, 0, st>>>(a.w, a.vi, a.n, a.bs, diag, a.max_iters, a.s);
  if (f.form == 3) {
    k_lz_terms<<<lz_sweep_blocks(a.n * a.bs), 256, 0, st>>>(a);
    k_lz_project<float><<<nb, kLzTeam, 0, st>>>(a.basis, a.w, a.n, a.bs, a.slots, a.s);
    k_lz_reduce32<<<rb, 1024, 0, st>>>(nb, a.bs, a.slots, a.s);
    subtract();
    k_lz_project<float><<<nb, kLzTeam, 0, st>>>(a.basis, a.w, a.n, a.bs, a.slots, a.s);
    k_lz_reduce32<<<rb, 1024, 0, st>>>(nb, a.bs, a.slots, a.s);
    if (!quads) {
      subtract();
      k_lz_finish<float><<<nb, 256, 0, st>>>(a.w, a.n, a.bs, subdiag, a.max_iters, tol, a.s);
      return COLAGB_OK;
    }
  } else {
    lz_project<LZ_TERMS_PROJ>(f, a, i, st);
    k_lz_reduce32<<<rb, 1024, 0, st>>>(f.blocks, a.bs, a.slots, a.s);
    lz_project<LZ_SUB_PROJ>(f, a, i, st);
    k_lz_reduce32<<<rb, 1024, 0, st>>>(f.blocks, a.bs, a.slots, a.s);
  }
  if (!quads) k_lz_fin<0><<<nb, 256, 0, st>>>(a, subdiag, tol);
  else if (a.bs == 1) k_lz_fin<2><<<nb, 256, 0, st>>>(a, subdiag, tol);
  else k_lz_fin<1><<<nb, 256, 0, st>>>(a, subdiag, tol);
  return COLAGB_OK;
}

// ---------------------------------------------------------------------------------------------
// FP64 and Arnoldi: one step's orthogonalisation.  w = A V[i] is projected on slots 1..i and the projections removed,
// twice ("twice is enough"): h = V^T w, w -= V h.  The first pass's h_i is diag[i-1] = <w, V[i]>, and
// since the pass removes it together with the component on V[i-1], the reference's separate
// three-term update (lanczos.py:262-266) needs no sweep of its own.
//
// Three launches over the filled slots (k_lz_gs), a small reduction after the first two:
//   PROJECT    h1 = V^T w                        every slot read once
//   SUB_PROJ   w -= V h1, then h2 = V^T w        each CTA on its own run of rows: the second read of a
//                                                run's slots follows the first at once and hits L1 / L2
//   SUB_NORM   w -= V h2, |w| per column, and in the last CTA the step's bookkeeping
// A CTA owns contiguous runs of whole rows; w's run is staged in shared memory.  Subtracting, a thread
// owns one 16-byte unit (or several threads share it, each with every G-th slot, when the run has fewer
// units than the CTA has threads); projecting, a warp owns a slot and its lanes keep fixed columns.  The
// unit is a float4 for FP32 with bs = 1 or a multiple of 4 on 16-byte boundaries, else one entry.
//
// It replaced norm, dot, three-term update and four sweeps, 12 launches a step beside the operator, with one
// dependent load per slot and thread.  Long vectors take the same two passes through k_lz_project and
// k_lz_subtract (gs_plan says from where on): a run's second read misses the caches then, and 512 threads with a
// run of w in shared memory keep fewer loads in flight than plain sweeps.
enum { GS_PROJECT = 0, GS_SUB_PROJ = 1, GS_SUB_NORM = 2 };
constexpr int kGsThreads = 512;

template <class T>
struct GsArgs {
  const T* basis;
  T* w;
  int64_t N, bs;       // n * bs entries per slot
  int run;             // entries of a run: whole rows, whole units
  int64_t slots;
  T* subdiag;          // SUB_NORM of Lanczos (null for Arnoldi, which only needs |w|)
  int max_iters;
  double tol;
  LzState<T> s;
};

template <class T, int VEC> struct GsUnit { T v[VEC]; };
template <class T, int VEC> __device__ __forceinline__ GsUnit<T, VEC> gs_ld(const T* p) {
  GsUnit<T, VEC> u;
  if constexpr (VEC == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    u.v[0] = q.x; u.v[1] = q.y; u.v[2] = q.z; u.v[3] = q.w;
  } else {
    u.v[0] = *p;
  }
  return u;
}
template <class T, int VEC> __device__ __forceinline__ GsUnit<T, VEC> gs_ldg(const T* p) {
  GsUnit<T, VEC> u;
  if constexpr (VEC == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    u.v[0] = q.x; u.v[1] = q.y; u.v[2] = q.z; u.v[3] = q.w;
  } else {
    u.v[0] = __ldg(p);
  }
  return u;
}
template <class T, int VEC> __device__ __forceinline__ void gs_st(T* p, const GsUnit<T, VEC>& u) {
  if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(u.v[0], u.v[1], u.v[2], u.v[3]);
  else *p = u.v[0];
}

// Sum over the lanes l, l + C, l + 2C, ... < La of a warp (C columns side by side), result in lanes < C.
template <class T>
__device__ __forceinline__ T gs_lane_sum(T x, int C, int La) {
  if ((C & (C - 1)) == 0) {
    for (int o = 16; o >= C; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  }
  T r = x;
  for (int o = C; o < La; o += C) r += __shfl_sync(0xffffffffu, x, (threadIdx.x & 31) + o);
  return r;
}

// STAGED = false: rows too long for shared memory (tens of thousands of columns); w is read back instead.
template <class T, int VEC, int MODE, bool STAGED>
__global__ void __launch_bounds__(kGsThreads) k_lz_gs(const __grid_constant__ GsArgs<T> g) {
  const LzState<T>& s = g.s;
  if (*s.done) return;
  extern __shared__ __align__(16) unsigned char gs_smem[];
  T* const red = reinterpret_cast<T*>(gs_smem);  // kGsThreads * VEC
  T* const stage = red + kGsThreads * VEC;       // the run of w
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int NW = kGsThreads / 32;
  const int i = *s.step;
  const int bs = (int)g.bs;
  const bool one = VEC == 4 && bs == 1;         // four rows of a single column per unit
  const int C = one ? 1 : bs / VEC;             // units of a row
  const int Cw = C < 32 ? C : 32, La = 32 / Cw * Cw;
  const int64_t nruns = ceil_div(g.N, (int64_t)g.run);
  T* const hp = s.hpart + (int64_t)blockIdx.x * g.slots * bs;
  if (MODE == GS_SUB_NORM) {
    for (int b = t; b < bs; b += kGsThreads) s.npart[(int64_t)blockIdx.x * bs + b] = T(0);
  }
  for (int64_t r = blockIdx.x; r < nruns; r += gridDim.x) {
    const int64_t e0 = r * g.run;
    const int len = (int)(g.N - e0 < g.run ? g.N - e0 : g.run), nu = len / VEC;
    T* const w = g.w + e0;
    const T* const v = g.basis + e0;
    T* const ws = STAGED ? stage : w;
    if (r != blockIdx.x) __syncthreads();  // the previous run's readers are done with ws
    if (MODE == GS_PROJECT) {
      if (STAGED)
        for (int u = t; u < nu; u += kGsThreads) gs_st<T, VEC>(ws + u * VEC, gs_ld<T, VEC>(w + u * VEC));
    } else {
      auto sums = [&](int u, int j0, int dj) {  // sum_j V[j] h[j] of unit u over j = j0, j0 + dj, ...
        GsUnit<T, VEC> acc;
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc.v[c] = T(0);
        const T* vp = v + (int64_t)j0 * g.N + u * VEC;
        const T* h = s.hbuf + (int64_t)j0 * bs + (one ? 0 : (u % C) * VEC);
#pragma unroll 8
        for (int j = j0; j <= i; j += dj, vp += dj * g.N, h += (int64_t)dj * bs) {
          const GsUnit<T, VEC> x = gs_ldg<T, VEC>(vp);
          if (one) {
            const T hh = __ldg(h);
#pragma unroll
            for (int c = 0; c < VEC; ++c) acc.v[c] += x.v[c] * hh;
          } else {
            const GsUnit<T, VEC> hh = gs_ldg<T, VEC>(h);
#pragma unroll
            for (int c = 0; c < VEC; ++c) acc.v[c] += x.v[c] * hh.v[c];
          }
        }
        return acc;
      };
      auto finish = [&](int u, const GsUnit<T, VEC>& acc) {
        GsUnit<T, VEC> x = gs_ld<T, VEC>(w + u * VEC);
#pragma unroll
        for (int c = 0; c < VEC; ++c) x.v[c] -= acc.v[c];
        gs_st<T, VEC>(w + u * VEC, x);
        if (STAGED) gs_st<T, VEC>(ws + u * VEC, x);
      };
      const int G = kGsThreads / nu < i ? kGsThreads / nu : i;
      if (G >= 2) {
        const int u = t % nu, gr = t / nu;
        GsUnit<T, VEC> acc;
        if (gr < G) {
          acc = sums(u, 1 + gr, G);
          if (gr > 0) gs_st<T, VEC>(red + (gr * nu + u) * VEC, acc);
        }
        __syncthreads();
        if (gr == 0) {
          for (int q = 1; q < G; ++q) {
            const GsUnit<T, VEC> o = gs_ld<T, VEC>(red + (q * nu + u) * VEC);
#pragma unroll
            for (int c = 0; c < VEC; ++c) acc.v[c] += o.v[c];
          }
          finish(u, acc);
        }
      } else {
        for (int u = t; u < nu; u += kGsThreads) finish(u, sums(u, 1, 1));
      }
    }
    __syncthreads();  // ws complete
    // per-column sums of a slot's run against w's: warp per slot (MODE 0 / 1), or of w's squares with
    // the warps sharing the run (SUB_NORM)
    const int j_first = MODE == GS_SUB_NORM ? 0 : 1 + warp, j_last = MODE == GS_SUB_NORM ? 0 : i;
    for (int j = j_first; j <= j_last; j += NW) {
      const T* const vj = MODE == GS_SUB_NORM ? ws : v + (int64_t)j * g.N;
      for (int c0 = 0; c0 < C; c0 += Cw) {  // C > 32: 32 columns of units at a time
        const int cw = C - c0 < Cw ? C - c0 : Cw;
        const int step = C <= 32 ? La : C;
        GsUnit<T, VEC> acc, acc2;
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc.v[c] = acc2.v[c] = T(0);
        if (C <= 32 ? lane < La : lane < cw) {
          const int first = c0 + lane + (MODE == GS_SUB_NORM ? warp * step : 0);
          const int stride = MODE == GS_SUB_NORM ? NW * step : step;
          auto term = [&](int u, GsUnit<T, VEC>& a2) {
            const GsUnit<T, VEC> x = gs_ld<T, VEC>(ws + u * VEC);
            GsUnit<T, VEC> y;
            if (MODE == GS_SUB_NORM) y = x;
            else y = gs_ldg<T, VEC>(vj + u * VEC);
#pragma unroll
            for (int c = 0; c < VEC; ++c) a2.v[c] += x.v[c] * y.v[c];
          };
          int u = first;
#pragma unroll 4
          for (; u + stride < nu; u += 2 * stride) {
            term(u, acc);
            term(u + stride, acc2);
          }
          if (u < nu) term(u, acc);
        }
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc.v[c] += acc2.v[c];
        if (one) {
          acc.v[0] = (acc.v[0] + acc.v[VEC > 1 ? 1 : 0]) + (acc.v[VEC > 2 ? 2 : 0] + acc.v[VEC > 3 ? 3 : 0]);
        }
        const int nc = one ? 1 : VEC;
#pragma unroll
        for (int c = 0; c < VEC; ++c)
          if (c < nc) acc.v[c] = gs_lane_sum<T>(acc.v[c], C <= 32 ? C : 32, C <= 32 ? La : 32);
        if (lane < cw) {
#pragma unroll
          for (int c = 0; c < VEC; ++c)
            if (c < nc) {
              const int b = (c0 + lane) * nc + c;
              if (MODE == GS_SUB_NORM) {
                red[(warp * Cw + lane) * VEC + c] = acc.v[c];
              } else {
                T* o = hp + (int64_t)j * bs + b;
                *o = r == blockIdx.x ? acc.v[c] : *o + acc.v[c];
              }
            }
        }
        if (MODE == GS_SUB_NORM) {
          __syncthreads();
          for (int q = t; q < cw * nc; q += kGsThreads) {
            const int l = q / nc, c = q % nc;
            T sum = T(0);
            for (int ww = 0; ww < NW; ++ww) sum += red[(ww * Cw + l) * VEC + c];
            s.npart[(int64_t)blockIdx.x * bs + (c0 + l) * nc + c] += sum;
          }
          __syncthreads();
        }
      }
    }
  }
  if (MODE == GS_SUB_NORM)
    if (lz_last_block(s.counters + 2)) lz_step_end<T>(s, g.bs, i, g.subdiag, g.max_iters, g.tol, red);
}

// h[j][b] = sum over the CTAs of hpart, 32 neighbouring sums per block and eight threads each.  What
// becomes of them: diag[b][i-1] = h[i][b] after the first pass of Lanczos, column i - 1 of Arnoldi's H
// (bs, max_iters + 1, max_iters) collects both passes.
template <class T>
__global__ void __launch_bounds__(256) k_lz_reduce_h(int nblk, int64_t bs, int64_t slots, T* diag, T* H, int first,
                                                     int max_iters, LzState<T> s) {
  if (*s.done) return;
  __shared__ T part[8][32];
  const int i = *s.step;
  const int64_t total = (int64_t)(i + 1) * bs;
  const int l = threadIdx.x & 31, q0 = threadIdx.x >> 5;
  for (int64_t u0 = (int64_t)blockIdx.x * 32; u0 < total; u0 += (int64_t)gridDim.x * 32) {
    const int64_t u = u0 + l;
    T acc = T(0);
    if (u < total && u >= bs) {  // slot 0 is the zero vector
#pragma unroll 8
      for (int q = q0; q < nblk; q += 8) acc += __ldg(s.hpart + (int64_t)q * slots * bs + u);
    }
    part[q0][l] = acc;
    __syncthreads();
    if (q0 == 0 && u < total) {
      const T h = ((part[0][l] + part[1][l]) + (part[2][l] + part[3][l])) +
                  ((part[4][l] + part[5][l]) + (part[6][l] + part[7][l]));
      s.hbuf[u] = h;
      const int64_t j = u / bs, b = u - j * bs;
      if (diag && j == i) diag[b * max_iters + (i - 1)] = h;
      if (H && j >= 1) {
        T* o = H + (b * (max_iters + 1) + (j - 1)) * max_iters + (i - 1);
        *o = first ? h : *o + h;
      }
    }
    __syncthreads();
  }
}

constexpr size_t kGsSmem = 200 * 1024;

// Launch plan of k_lz_gs for one run of the method.
struct GsPlan {
  int vec = 1, run = 0, blocks = 1;
  bool staged = true, split = false;  // split: passes of their own on `blocks` CTAs
  size_t smem = 0;
};

template <class T>
static GsPlan gs_plan(const T* basis, int64_t n, int64_t bs, int max_blocks) {
  GsPlan p;
  const int64_t N = n * bs;
  if (std::is_same<T, float>::value && (uintptr_t)basis % 16 == 0 && (bs % 4 == 0 || (bs == 1 && n % 4 == 0))) p.vec = 4;
  const int64_t target = std::min<int64_t>(max_blocks, 2 * (int64_t)num_sms());
  const int64_t unit = bs == 1 ? 32 * p.vec : bs;  // whole rows; a single column: whole warp loads
  // at most 48 KB of w per run: two CTAs per SM keep their runs' slots in flight together
  const int64_t most = std::max<int64_t>(1, (48 * 1024 / (int64_t)sizeof(T)) / unit);
  const int64_t units = std::min(most, std::max<int64_t>(1, ceil_div(ceil_div(N, target), unit)));
  p.run = (int)(units * unit);
  p.blocks = (int)std::min<int64_t>(target, ceil_div(N, (int64_t)p.run));
  p.smem = (size_t)p.run * sizeof(T) + (size_t)kGsThreads * p.vec * sizeof(T);
  if (p.smem > kGsSmem) {
    p.staged = false;
    p.vec = 1;
    p.smem = (size_t)kGsThreads * sizeof(T);
  }
  // Long vectors: pass by pass, unless the columns leave a quarter of a team idle there.  ms for 24 steps, FP64
  // Lanczos, k_lz_gs / pass by pass: 100,000 x 10 5.85 / 6.3, 400,000 x 3 6.7 / 6.2, 50,000 x 33 11.6 / 9.2, 100,000 x 20
  // 18.9 / 10.2, 1,000,000 x 33 194 / 108; FP32 Arnoldi, 100,000 x 10 2.8 / 3.0, 50,000 x 33 6.6 / 4.7, 400,000 x 10
  // 19.4 / 7.6.
  if (N > 1100000 && (bs >= kLzTeam || kLzTeam / bs * bs >= kLzTeam * 3 / 4)) {
    p.split = true;
    p.blocks = max_blocks;
  }
  return p;
}

template <class T, int VEC, int MODE, bool STAGED>
static int launch_gs_form(const GsPlan& p, const GsArgs<T>& a, cudaStream_t st) {
  auto* f = k_lz_gs<T, VEC, MODE, STAGED>;
  if (p.smem > 48 * 1024) COLAGB_CUDA(set_smem_limit(f, kGsSmem));
  f<<<p.blocks, kGsThreads, p.smem, st>>>(a);
  return COLAGB_OK;
}

template <class T, int MODE>
static int launch_gs(const GsPlan& p, const GsArgs<T>& a, cudaStream_t st) {
  if (!p.staged) return launch_gs_form<T, 1, MODE, false>(p, a, st);
  if constexpr (std::is_same<T, float>::value)
    if (p.vec == 4) return launch_gs_form<T, 4, MODE, true>(p, a, st);
  return launch_gs_form<T, 1, MODE, true>(p, a, st);
}

// The two passes on w (slots 1..i filled): Lanczos with diag / subdiag, Arnoldi with H.
template <class T>
static int gs_step(const GsPlan& p, const T* basis, T* w, int64_t n, int64_t bs, int i, T* diag, T* subdiag, T* H,
                   int max_iters, double tol, const LzState<T>& s, cudaStream_t st) {
  GsArgs<T> a{basis, w, n * bs, bs, p.run, (int64_t)max_iters + 2, subdiag, max_iters, tol, s};
  const unsigned rb = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div((int64_t)(i + 1) * bs, 32), 4096));
  if (p.split) {
    const unsigned sweep = lz_sweep_blocks(n * bs, 4);
    for (int pass = 0; pass < 2; ++pass) {
      k_lz_project<T><<<p.blocks, kLzTeam, 0, st>>>(basis, w, n, bs, a.slots, s);
      k_lz_reduce_h<T><<<rb, 256, 0, st>>>(p.blocks, bs, a.slots, pass ? (T*)nullptr : diag, H, !pass, max_iters, s);
      k_lz_subtract<T, 0><<<sweep, 256, 0, st>>>(basis, w, n, bs, s);
    }
    k_lz_finish<T><<<p.blocks, 256, 0, st>>>(w, n, bs, subdiag, max_iters, tol, s);
    return COLAGB_OK;
  }
  COLAGB_TRY((launch_gs<T, GS_PROJECT>(p, a, st)));
  k_lz_reduce_h<T><<<rb, 256, 0, st>>>(p.blocks, bs, a.slots, diag, H, 1, max_iters, s);
  COLAGB_TRY((launch_gs<T, GS_SUB_PROJ>(p, a, st)));
  k_lz_reduce_h<T><<<rb, 256, 0, st>>>(p.blocks, bs, a.slots, (T*)nullptr, H, 0, max_iters, s);
  return launch_gs<T, GS_SUB_NORM>(p, a, st);
}

// V[1] = V0 / |V0| (init_lanczos) -- norm partials then scale
template <class T>
__global__ void k_lz_init_copy(const T* v0, int64_t ldv0, T* v1, int64_t n, int64_t bs) {
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n * bs; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = u / bs, b = u % bs;
    v1[u] = v0[r * ldv0 + b];
  }
}

template <class T>
__global__ void k_lz_set_state(LzState<T> s, int max_iters) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    *s.step = 1;
    *s.done = !(1 <= max_iters);
  }
}

// out[r][b] = sum_{j<m} basis[j+1][r][b] * coef[b * ldc + j]
template <class T>
__global__ void k_basis_combine(const T* basis, int64_t n, int64_t bs, int m, const T* coef, int64_t ldc, T* out) {
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n * bs; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = u % bs;
    T acc = T(0);
    for (int j = 0; j < m; ++j) acc += basis[(int64_t)(j + 1) * n * bs + u] * coef[b * ldc + j];
    out[u] = acc;
  }
}

// ---------------------------------------------------------------------------------------------
// Symmetric tridiagonal eigensolver (batched): implicit QL with Wilkinson shifts, one CTA per
// matrix, in R = double or float.  The matrix is first scaled by a power of two (exact) so that its
// largest entry lies in [0.5, 1): the sweep below forms squares without overflow checks in either
// precision.  One thread runs the scalar recurrence; each QL sweep's Givens rotations go through shared
// memory to the other warps, which apply them to the rows of the eigenvector matrix (rows are
// independent under column rotations) or record them, and track row 0 (Gauss weights), while the next
// sweep runs.  The sweep's chain of dependent operations on one thread bounds it; with the recording, row 0 and the
// search for a split on that thread too, a 96-step FP32 tridiagonal took 1388 us, now 574 us, to the same bits.
// `rec` (optional, with evecs == nullptr): every Givens rotation (c, s) on columns (i, i+1) is
// appended in generation order to rec[sys * cap ...] / rec_i, the count to rec_n[sys] (-1 when cap
// was exceeded), and the sorting permutation to rec_perm[sys * m ...]; k_tridiag_apply replays them.
template <class R> struct TriTraits;
template <> struct TriTraits<double> {
  using R2 = double2;
  static constexpr double eps = 2.220446049250313e-16;
  __device__ static double rsq(double x) { return rsqrt(x); }
  __device__ static double hyp(double a, double b) { return hypot(a, b); }
  __device__ static double2 pack(double c, double s) { return make_double2(c, s); }
  __device__ static double ab(double x) { return fabs(x); }
  __device__ static double mx(double x, double y) { return fmax(x, y); }
  __device__ static double fm(double x, double y, double z) { return fma(x, y, z); }
  __device__ static double fr(double x, int* ex) { return frexp(x, ex); }
  __device__ static double ld(double x, int ex) { return ldexp(x, ex); }
};
template <> struct TriTraits<float> {
  using R2 = float2;
  static constexpr float eps = 1.1920928955078125e-7f;
  __device__ static float rsq(float x) { return rsqrtf(x); }
  __device__ static float hyp(float a, float b) { return hypotf(a, b); }
  __device__ static float2 pack(float c, float s) { return make_float2(c, s); }
  __device__ static float ab(float x) { return fabsf(x); }
  __device__ static float mx(float x, float y) { return fmaxf(x, y); }
  __device__ static float fm(float x, float y, float z) { return fmaf(x, y, z); }
  __device__ static float fr(float x, int* ex) { return frexpf(x, ex); }
  __device__ static float ld(float x, int ex) { return ldexpf(x, ex); }
};

// Strict total order for the eigenvalue sort: ascending, NaN last, ties by index.
template <class R>
__device__ inline bool tri_before(R x, int64_t i, R y, int64_t j) {
  const bool nx = isnan(x), ny = isnan(y);
  if (nx != ny) return ny;
  if (!nx && x != y) return x < y;
  return i < j;
}

template <class R>
__global__ void k_tridiag_ql(const R* A, const R* Bv, int64_t m, int two, R* evals, R* first_row, R* evecs,
                             int32_t* status, typename TriTraits<R>::R2* rec = nullptr, int32_t* rec_i = nullptr,
                             int32_t* rec_n = nullptr, int32_t* rec_perm = nullptr, int64_t cap = 0) {
  using TT = TriTraits<R>;
  extern __shared__ __align__(16) unsigned char tri_smem[];
  R* d = reinterpret_cast<R*>(tri_smem);  // m
  R* e = d + m;                           // m
  R* z0 = e + m;                          // m (row 0 of Z)
  R* rc = z0 + m;                         // m cosines and m sines of a sweep (of two if `two`)
  int* perm = reinterpret_cast<int*>(rc + (two ? 4 : 2) * m);  // m
  __shared__ int s_cmd[2], s_lo[2], s_hi[2], s_fail;
  __shared__ R s_amax[32];
  const int64_t sys = blockIdx.x;
  const R* a = A + sys * m;
  const R* b = Bv + sys * m;
  R* Z = evecs ? evecs + sys * m * m : nullptr;
  R amax = R(0);
  for (int64_t i = threadIdx.x; i < m; i += blockDim.x) {
    const R ai = a[i], bi = (i + 1 < m) ? b[i] : R(0);
    amax = TT::mx(amax, TT::mx(TT::ab(ai), TT::ab(bi)));
  }
  for (int o = 16; o > 0; o >>= 1) amax = TT::mx(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) s_amax[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x == 0) {
    R t = R(0);
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = TT::mx(t, s_amax[w]);
    s_amax[0] = t;
    s_fail = 0;
  }
  __syncthreads();
  // 2^-e with amax = f * 2^e, f in [0.5, 1): exact scaling, undone on the eigenvalues
  int ex = 0;
  const R amx = s_amax[0];
  if (amx > R(0) && isfinite(amx)) TT::fr(amx, &ex);
  const R scale = TT::ld(R(1), -ex), unscale = TT::ld(R(1), ex);
  for (int64_t i = threadIdx.x; i < m; i += blockDim.x) {
    d[i] = a[i] * scale;
    e[i] = (i + 1 < m) ? b[i] * scale : R(0);
    z0[i] = (i == 0) ? R(1) : R(0);
  }
  if (Z)
    for (int64_t u = threadIdx.x; u < m * m; u += blockDim.x) Z[u] = (u / m == u % m) ? R(1) : R(0);
  __syncthreads();
  // Sweep by sweep: warp 0 finds the block to work on (32 entries at a time), its lane 0 runs the sweep -- one
  // dependent chain, kept free of everything else -- and leaves the rotations in shared memory; the other
  // warps meanwhile finish the sweep before it (two buffers): record its rotations or apply them to Z's
  // rows, and carry row 0 of Z along.
  int l = 0, iter = 0;
  int64_t nrec = 0;
  typename TT::R2* my_rec = rec ? rec + sys * cap : nullptr;
  int32_t* my_rec_i = rec ? rec_i + sys * cap : nullptr;
  const int lane = threadIdx.x & 31;
  // what the warps from the second on do with the rotations of sweep pb, generated for i = hi - 1 down to lo
  auto finish = [&](int pb) {
    const int lo = s_lo[pb & 1], hi = s_hi[pb & 1];
    const R* const pc = rc + (pb & two) * 2 * m;
    const R* const ps = pc + m;
    const int w = threadIdx.x - 32, nw = blockDim.x - 32;
    if (w == nw - 1) {  // row 0 of Z
      R zi1 = hi > lo ? z0[hi] : R(0);
      for (int i = hi - 1; i >= lo; --i) {
        const R c = pc[i], s = ps[i], zi = z0[i];
        z0[i + 1] = s * zi + c * zi1;
        zi1 = c * zi - s * zi1;
        z0[i] = zi1;
      }
    }
    if (my_rec)
      for (int i = hi - 1 - w; i >= lo; i -= nw) {
        const int64_t at = nrec + (hi - 1 - i);
        if (at < cap) {
          my_rec[at] = TT::pack(pc[i], ps[i]);
          my_rec_i[at] = i;
        }
      }
    nrec += hi - lo;
    if (Z)
      for (int64_t row = w; row < m; row += nw) {
        R* zr = Z + row * m;
        for (int i = hi - 1; i >= lo; --i) {
          const R c = pc[i], s = ps[i];
          const R f = zr[i + 1];
          zr[i + 1] = s * zr[i] + c * f;
          zr[i] = c * zr[i] - s * f;
        }
      }
  };
  for (int turn = 0;; ++turn) {
    R* const rcb = rc + (turn & two) * 2 * m;  // this sweep's cosines; sines m entries on
    R* const rsb = rcb + m;
    if (threadIdx.x < 32) {
      int cmd = 2, lo = 0, hi = 0;  // 1 = rotations [lo, hi) were generated, 2 = finished
      while (l < m) {
        int mm = (int)m - 1;  // first mm >= l with a negligible off-diagonal entry
        for (int b0 = l; b0 < (int)m - 1; b0 += 32) {
          const int j = b0 + lane;
          bool small = false;
          if (j < (int)m - 1) {
            const R dd = TT::ab(d[j]) + TT::ab(d[j + 1]);
            small = TT::ab(e[j]) <= TT::eps * dd;
          }
          const unsigned hit = __ballot_sync(0xffffffffu, small);
          if (hit) {
            mm = b0 + __ffs(hit) - 1;
            break;
          }
        }
        if (mm == l) { ++l; iter = 0; continue; }
        if (iter++ >= 60) {
          if (lane == 0) s_fail = 1;
          ++l;
          iter = 0;
          continue;
        }
        if (lane == 0) {
          R g = (d[l + 1] - d[l]) / (R(2) * e[l]);
          R r = TT::hyp(g, R(1));
          g = d[mm] - d[l] + e[l] / (g + (g >= R(0) ? TT::ab(r) : -TT::ab(r)));
          R s = R(1), c = R(1), p = R(0);
          int i = mm - 1;
          bool underflow = false;
          // The operands of step i - 1 (e[i-1], d[i-1]), which step i does not modify, are loaded ahead,
          // d[i] is carried in a register, and each rotation takes one reciprocal square root instead of
          // a hypot and two divisions (|f|, |g| are bounded by a small multiple of the scaled matrix's norm).
          R ei = e[i], di1 = d[i + 1], di = d[i];
          for (; i >= l; --i) {
            const R e_nx = i > l ? e[i - 1] : R(0);
            const R d_nx = i > l ? d[i - 1] : R(0);
            const R f = s * ei, bb = c * ei;
            const R q = TT::fm(f, f, g * g);
            if (q == R(0)) {
              e[i + 1] = R(0);
              d[i + 1] = di1 - p;
              e[mm] = R(0);
              underflow = true;
              break;
            }
            const R ri = TT::rsq(q);
            e[i + 1] = q * ri;
            s = f * ri;
            c = g * ri;
            g = di1 - p;
            r = (di - g) * s + R(2) * c * bb;
            p = s * r;
            d[i + 1] = g + p;
            g = c * r - bb;
            rcb[i] = c;
            rsb[i] = s;
            ei = e_nx;
            di1 = di;
            di = d_nx;
          }
          hi = mm;
          lo = underflow ? i + 1 : l;
          if (!underflow) {
            d[l] -= p;
            e[l] = g;
            e[mm] = R(0);
          }
        }
        cmd = 1;
        break;
      }
      __syncwarp();
      if (lane == 0) {
        s_cmd[turn & 1] = cmd;
        s_lo[turn & 1] = lo;
        s_hi[turn & 1] = hi;
      }
    } else if (two && turn > 0) {
      finish(turn - 1);
    }
    __syncthreads();
    if (s_cmd[turn & 1] == 2) break;
    if (!two) {
      if (threadIdx.x >= 32) finish(turn);
      __syncthreads();
    }
  }
  // ascending order by rank (ties by index): every thread ranks its own entries, O(m) each
  for (int64_t j = threadIdx.x; j < m; j += blockDim.x) {
    const R dj = d[j];
    int rank = 0;
    for (int64_t i = 0; i < m; ++i) rank += tri_before(d[i], i, dj, j);
    perm[rank] = (int)j;
  }
  __syncthreads();
  for (int64_t j = threadIdx.x; j < m; j += blockDim.x) {
    evals[sys * m + j] = d[perm[j]] * unscale;
    if (first_row) first_row[sys * m + j] = Z ? Z[perm[j]] : z0[perm[j]];
    if (rec_perm) rec_perm[sys * m + j] = perm[j];
  }
  if (rec && threadIdx.x == blockDim.x - 1) rec_n[sys] = nrec <= cap ? (int32_t)nrec : -1;
  __syncthreads();
  if (Z) {
    R* tmp = rc;  // reuse as a row buffer
    for (int64_t row = 0; row < m; ++row) {
      for (int64_t j = threadIdx.x; j < m; j += blockDim.x) tmp[j] = Z[row * m + perm[j]];
      __syncthreads();
      for (int64_t j = threadIdx.x; j < m; j += blockDim.x) Z[row * m + j] = tmp[j];
      __syncthreads();
    }
  }
  if (threadIdx.x == 0 && status) status[sys] = s_fail;
}

// Replays the recorded rotations on the eigenvector matrix: Z starts as the identity, each thread
// owns one row (rows are independent), held in shared memory as zs[col][lane] (conflict-free);
// every rotation acts on columns (i, i+1).  Output columns follow the sorted eigenvalues.
constexpr int kRotRows = 32;
template <class R>
__global__ void __launch_bounds__(kRotRows) k_tridiag_apply(const typename TriTraits<R>::R2* rec,
                                                            const int32_t* rec_i, const int32_t* rec_n,
                                                            const int32_t* rec_perm, int64_t m, int64_t cap,
                                                            R* evecs) {
  extern __shared__ __align__(16) unsigned char rot_smem[];
  R* zs = reinterpret_cast<R*>(rot_smem);  // m x kRotRows
  const int64_t sys = blockIdx.y;
  const int t = threadIdx.x;
  const int64_t row = (int64_t)blockIdx.x * kRotRows + t;
  const int32_t nr = rec_n[sys];
  if (nr < 0) return;  // the recording overflowed: the in-kernel path produced Z
  for (int64_t i = 0; i < m; ++i) zs[i * kRotRows + t] = (row == i) ? R(1) : R(0);
  const typename TriTraits<R>::R2* r = rec + sys * cap;
  const int32_t* ri = rec_i + sys * cap;
  for (int32_t q = 0; q < nr; ++q) {
    const auto cs = r[q];
    const int i = ri[q];
    const R zi = zs[i * kRotRows + t], f = zs[(i + 1) * kRotRows + t];
    zs[(i + 1) * kRotRows + t] = cs.y * zi + cs.x * f;
    zs[i * kRotRows + t] = cs.x * zi - cs.y * f;
  }
  if (row < m) {
    R* out = evecs + sys * m * m + row * m;
    const int32_t* perm = rec_perm + sys * m;
    for (int64_t j = 0; j < m; ++j) out[j] = zs[perm[j] * kRotRows + t];
  }
}

// ---------------------------------------------------------------------------------------------
// host

static int lz_blocks(int64_t n, int64_t bs) {
  const int64_t want = ceil_div(n * bs, 1024);
  const int64_t cap = (int64_t)num_sms() * 4;
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}

template <class T>
static LzState<T> lz_carve(Bump& ws, int64_t bs, int32_t max_iters, int nb) {
  LzState<T> s;
  const int64_t slots = (int64_t)max_iters + 2;
  s.nrm = ws.take<T>(bs);
  s.hbuf = ws.take<T>(slots * bs);
  s.hpart = ws.take<T>((size_t)nb * slots * bs);
  s.npart = ws.take<T>((size_t)nb * bs);
  s.done = ws.take<int>(4);
  s.step = ws.take<int>(4);
  s.counters = ws.take<unsigned int>(8);
  return s;
}

// The slots past `last` read as zero, like slot 0: the steps write slots 1..last only.
template <class T>
static int clear_unfilled(T* basis, size_t blk, int last, int m, cudaStream_t st) {
  if (last < m + 1)
    COLAGB_CUDA(cudaMemsetAsync(basis + (size_t)(last + 1) * blk, 0, sizeof(T) * blk * (size_t)(m + 1 - last), st));
  return COLAGB_OK;
}

template <class T>
static int lanczos_t(const colagb_op* A, const T* V0, int64_t ldv0, int64_t bs, const colagb_lanczos_params& prm,
                     T* basis, T* diag, T* subdiag, int32_t* steps, void* workspace, size_t ws_bytes,
                     cudaStream_t st) {
  const int64_t n = A->nodes[A->root].rows;
  const int m = prm.max_iters;
  const int nb = lz_blocks(n, bs);
  Bump ws(workspace, ws_bytes);
  LzState<T> s = lz_carve<T>(ws, bs, m, nb);
  size_t opb = 0;
  COLAGB_TRY(colagb_matmat_workspace_bytes(A, bs, &opb));
  void* opws = ws.take<char>(opb > 0 ? opb : 1);
  if (workspace == nullptr || ws.overflow())
    return fail(COLAGB_ERR_WORKSPACE, "colagb_lanczos: workspace too small (need " + std::to_string(ws.peak) + ")");
  const int eg = (int)std::min<int64_t>(std::max<int64_t>(ceil_div(n * bs, 256), 1), (int64_t)num_sms() * 8);
  const size_t blk = (size_t)n * bs;
  const GsPlan plan = gs_plan<T>(basis, n, bs, nb);
  LzForm form;
  if constexpr (std::is_same<T, float>::value) COLAGB_TRY(lz_form(basis, n, bs, nb, (int64_t)m + 2, form));
  auto scale = [&](T* v) {
    if constexpr (std::is_same<T, float>::value)
      if (plan.vec == 4) {
        k_lz_scale<T, 4><<<(unsigned)std::min<int64_t>(ceil_div((int64_t)blk, 1024), eg), 256, 0, st>>>(v, n, bs, s);
        return;
      }
    k_lz_scale<T, 1><<<eg, 256, 0, st>>>(v, n, bs, s);
  };
  COLAGB_CUDA(cudaMemsetAsync(basis, 0, sizeof(T) * blk, st));  // slot 0: V[0] = 0
  COLAGB_CUDA(cudaMemsetAsync(diag, 0, sizeof(T) * bs * m, st));
  COLAGB_CUDA(cudaMemsetAsync(subdiag, 0, sizeof(T) * bs * (m + 1), st));
  COLAGB_CUDA(cudaMemsetAsync(s.counters, 0, 8 * sizeof(unsigned int), st));
  k_lz_set_state<T><<<1, 32, 0, st>>>(s, m);
  // V[1] = V0 / |V0|
  T* v1 = basis + blk;
  k_lz_init_copy<T><<<eg, 256, 0, st>>>(V0, ldv0, v1, n, bs);
  k_lz_norm<T><<<nb, 256, 0, st>>>(v1, n, bs, s);
  scale(v1);
  k_lz_norm<T><<<nb, 256, 0, st>>>(v1, n, bs, s);  // the loop divides V[1] by its norm again
  COLAGB_CUDA(cudaGetLastError());
  const int every = prm.check_every > 0 ? prm.check_every : 8;
  int host_step = 1;  // the step index the next launch group starts at (upper bound)
  int hstate[5] = {0, 0, 0, 0, 1};  // done, ..., step
  while (true) {
    for (int q = 0; q < every && host_step <= m; ++q, ++host_step) {
      const int i = host_step;  // kernels read the device step; host_step picks the basis slots
      T* vi = basis + (size_t)i * blk;
      T* w = basis + (size_t)(i + 1) * blk;
      scale(vi);  // V[i] /= |V[i]|, the norm left by the step before
      Bump ow(opws, opb > 0 ? opb : 1);
      COLAGB_TRY(op_apply<T>(A, A->root, vi, bs, 0, w, bs, 0, bs, 1, T(1), T(0), ow, s.done, st));
      if constexpr (std::is_same<T, float>::value) {
        const LzStep a{basis, w, vi, vi - blk, diag, subdiag, n, bs, form.chunk, (int64_t)m + 2, m, s};
        COLAGB_TRY(lz_step_f32(form, a, i, nb, diag, subdiag, prm.tol, st));
      } else {
        COLAGB_TRY(gs_step<T>(plan, basis, w, n, bs, i, diag, subdiag, nullptr, m, prm.tol, s, st));
      }
      COLAGB_CUDA(cudaGetLastError());
    }
    COLAGB_CUDA(cudaMemcpyAsync(&hstate[0], s.done, sizeof(int), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaMemcpyAsync(&hstate[4], s.step, sizeof(int), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaStreamSynchronize(st));
    if (hstate[0] || host_step > m) break;
  }
  COLAGB_TRY(clear_unfilled<T>(basis, blk, hstate[4], m, st));
  *steps = hstate[4];
  return COLAGB_OK;
}


// ---- Arnoldi (arnoldi.py:303-334) on the same basis slots: Q[j] lives in slot j + 1 ----------
// w /= max(|w|, tol / 2)  (the new basis vector; |w| from the second pass)
template <class T>
__global__ void k_ar_scale_clip(T* w, int64_t n, int64_t bs, double tol, LzState<T> s) {
  if (*s.done) return;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n * bs; u += (int64_t)gridDim.x * blockDim.x) {
    const T nv = s.nrm[u % bs];
    w[u] = w[u] / (nv > (T)(tol / 2) ? nv : (T)(tol / 2));
  }
}

// H[b][idx + 1][idx] = |w| ; idx += 1 ; stop test of arnoldi_fact.cond_fun:
// continue while idx < max_iters and (any |w| > tol * H[b][1][0] or idx <= 0)
template <class T>
__global__ void k_ar_finish(T* H, int64_t bs, int max_iters, double tol, LzState<T> s) {
  if (*s.done) return;
  __shared__ int s_any;
  const int i = *s.step;
  const int idx = i - 1;
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  for (int64_t b = threadIdx.x; b < bs; b += blockDim.x) {
    const T nv = s.nrm[b];
    H[(b * (max_iters + 1) + idx + 1) * max_iters + idx] = nv;
    const T h10 = H[(b * (max_iters + 1) + 1) * max_iters + 0];
    if (nv > (T)tol * h10) atomicOr(&s_any, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nidx = idx + 1;
    *s.step = nidx + 1;
    *s.done = !(nidx < max_iters && (s_any || nidx <= 0));
  }
}

template <class T>
static int arnoldi_t(const colagb_op* A, const T* V0, int64_t ldv0, int64_t bs, const colagb_lanczos_params& prm,
                     T* basis, T* H, int32_t* steps, void* workspace, size_t ws_bytes, cudaStream_t st) {
  const int64_t n = A->nodes[A->root].rows;
  const int m = prm.max_iters;
  const int nb = lz_blocks(n, bs);
  Bump ws(workspace, ws_bytes);
  LzState<T> s = lz_carve<T>(ws, bs, m, nb);
  size_t opb = 0;
  COLAGB_TRY(colagb_matmat_workspace_bytes(A, bs, &opb));
  void* opws = ws.take<char>(opb > 0 ? opb : 1);
  if (workspace == nullptr || ws.overflow())
    return fail(COLAGB_ERR_WORKSPACE, "colagb_arnoldi: workspace too small (need " + std::to_string(ws.peak) + ")");
  const int eg = (int)std::min<int64_t>(std::max<int64_t>(ceil_div(n * bs, 256), 1), (int64_t)num_sms() * 8);
  const size_t blk = (size_t)n * bs;
  const GsPlan plan = gs_plan<T>(basis, n, bs, nb);
  COLAGB_CUDA(cudaMemsetAsync(basis, 0, sizeof(T) * blk, st));  // slot 0
  COLAGB_CUDA(cudaMemsetAsync(H, 0, sizeof(T) * bs * (m + 1) * (m > 0 ? m : 1), st));
  COLAGB_CUDA(cudaMemsetAsync(s.counters, 0, 8 * sizeof(unsigned int), st));
  k_lz_set_state<T><<<1, 32, 0, st>>>(s, m);
  T* q0 = basis + blk;  // Q[0] = V0 / |V0|
  k_lz_init_copy<T><<<eg, 256, 0, st>>>(V0, ldv0, q0, n, bs);
  k_lz_norm<T><<<nb, 256, 0, st>>>(q0, n, bs, s);
  k_lz_scale<T, 1><<<eg, 256, 0, st>>>(q0, n, bs, s);
  COLAGB_CUDA(cudaGetLastError());
  const int every = prm.check_every > 0 ? prm.check_every : 8;
  int host_step = 1;  // slot of Q[idx] for the next step (idx = host_step - 1)
  int hdone = 0;
  while (true) {
    for (int q = 0; q < every && host_step <= m; ++q, ++host_step) {
      const int i = host_step;
      T* qi = basis + (size_t)i * blk;
      T* w = basis + (size_t)(i + 1) * blk;
      Bump ow(opws, opb > 0 ? opb : 1);
      COLAGB_TRY(op_apply<T>(A, A->root, qi, bs, 0, w, bs, 0, bs, 1, T(1), T(0), ow, s.done, st));
      COLAGB_TRY(gs_step<T>(plan, basis, w, n, bs, i, nullptr, nullptr, H, m, prm.tol, s, st));
      k_ar_scale_clip<T><<<eg, 256, 0, st>>>(w, n, bs, prm.tol, s);
      k_ar_finish<T><<<1, 256, 0, st>>>(H, bs, m, prm.tol, s);
      COLAGB_CUDA(cudaGetLastError());
    }
    COLAGB_CUDA(cudaMemcpyAsync(&hdone, s.done, sizeof(int), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaStreamSynchronize(st));
    if (hdone || host_step > m) break;
  }
  int dstep = 0;
  COLAGB_CUDA(cudaMemcpyAsync(&dstep, s.step, sizeof(int), cudaMemcpyDeviceToHost, st));
  COLAGB_CUDA(cudaStreamSynchronize(st));
  COLAGB_TRY(clear_unfilled<T>(basis, blk, dstep, m, st));
  *steps = dstep - 1;  // Arnoldi steps taken (idx)
  return COLAGB_OK;
}
}  // namespace colagb

using namespace colagb;

extern "C" int colagb_lanczos_workspace_bytes(const colagb_op* A, int64_t bs, int32_t max_iters, size_t* bytes) {
  if (!A || !bytes || bs < 1 || max_iters < 0) return fail(COLAGB_ERR_INVALID, "colagb_lanczos_workspace_bytes: bad arguments");
  const int64_t n = A->nodes[A->root].rows;
  Bump ws = Bump::measuring();
  if (A->compute_dtype == COLAGB_F64) lz_carve<double>(ws, bs, max_iters, lz_blocks(n, bs));
  else lz_carve<float>(ws, bs, max_iters, lz_blocks(n, bs));
  size_t opb = 0;
  COLAGB_TRY(colagb_matmat_workspace_bytes(A, bs, &opb));
  ws.take<char>(opb > 0 ? opb : 1);
  *bytes = ws.peak;
  return COLAGB_OK;
}

extern "C" int colagb_lanczos(const colagb_op* A, const void* V0, int64_t ldv0, int64_t bs,
                              const colagb_lanczos_params* params, void* basis, void* diag, void* subdiag,
                              int32_t* steps, void* workspace, size_t workspace_bytes, void* stream) {
  if (!A || !params || !V0 || !basis || !diag || !subdiag || !steps)
    return fail(COLAGB_ERR_INVALID, "colagb_lanczos: null argument");
  const colagb_op_node& r = A->nodes[A->root];
  if (r.rows != r.cols) return fail(COLAGB_ERR_INVALID, "colagb_lanczos: operator must be square");
  if (bs < 1 || ldv0 < bs || params->max_iters < 0)
    return fail(COLAGB_ERR_INVALID, "colagb_lanczos: bad bs / ldv0 / max_iters");
  cudaStream_t st = as_stream(stream);
  if (A->compute_dtype == COLAGB_F64)
    return lanczos_t<double>(A, static_cast<const double*>(V0), ldv0, bs, *params, static_cast<double*>(basis),
                             static_cast<double*>(diag), static_cast<double*>(subdiag), steps, workspace,
                             workspace_bytes, st);
  return lanczos_t<float>(A, static_cast<const float*>(V0), ldv0, bs, *params, static_cast<float*>(basis),
                          static_cast<float*>(diag), static_cast<float*>(subdiag), steps, workspace, workspace_bytes,
                          st);
}

extern "C" int colagb_basis_combine(const void* basis, int64_t n, int64_t bs, int32_t m, const void* coef,
                                    int64_t ldc, void* out, int32_t dtype, void* stream) {
  if (!basis || !coef || !out || n < 0 || bs < 1 || m < 0 || ldc < m)
    return fail(COLAGB_ERR_INVALID, "colagb_basis_combine: bad arguments");
  cudaStream_t st = as_stream(stream);
  const int eg = (int)std::min<int64_t>(std::max<int64_t>(ceil_div(n * bs, 256), 1), (int64_t)num_sms() * 8);
  if (n * bs == 0) return COLAGB_OK;
  if (dtype == COLAGB_F64)
    k_basis_combine<double><<<eg, 256, 0, st>>>(static_cast<const double*>(basis), n, bs, m,
                                                 static_cast<const double*>(coef), ldc, static_cast<double*>(out));
  else if (dtype == COLAGB_F32)
    k_basis_combine<float><<<eg, 256, 0, st>>>(static_cast<const float*>(basis), n, bs, m,
                                                static_cast<const float*>(coef), ldc, static_cast<float*>(out));
  else
    return fail(COLAGB_ERR_UNSUPPORTED, "colagb_basis_combine: dtype must be F32 or F64");
  COLAGB_CUDA(cudaGetLastError());
  return COLAGB_OK;
}

// Rayleigh quotients of the computed eigenvectors in FP64: evals[j] = s_j^T T s_j / s_j^T s_j.  After an
// FP32 QL the eigenvalues carry the sweeps' accumulated rounding (a few FP32 ulps of |T|); the quotient
// of the FP32 eigenvector is off by the square of the vector's error, so this returns each eigenvalue
// to within FP32 rounding.  One thread per eigenvector; consecutive threads read consecutive columns.
template <class R>
__global__ void k_tridiag_rq(const R* A, const R* Bv, int64_t m, const R* evecs, R* evals) {
  const int64_t sys = blockIdx.y;
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const R* a = A + sys * m;
  const R* b = Bv + sys * m;
  const R* Z = evecs + sys * m * m;
  double num = 0.0, den = 0.0, sp = 0.0, si = (double)Z[j];
  for (int64_t i = 0; i < m; ++i) {
    const double sn = i + 1 < m ? (double)Z[(i + 1) * m + j] : 0.0;
    double t = (double)a[i] * si + (i > 0 ? (double)b[i - 1] * sp : 0.0);
    if (i + 1 < m) t += (double)b[i] * sn;
    num += si * t;
    den += si * si;
    sp = si;
    si = sn;
  }
  if (den > 0.0) evals[sys * m + j] = (R)(num / den);
}

constexpr size_t kTriSmem = 200 * 1024;
template <class R>
static int tridiag_eig(const R* a, const R* b, int64_t m, int64_t batch, R* evals, R* first_row, R* evecs,
                       int32_t* status, cudaStream_t st, const char* name) {
  using R2 = typename TriTraits<R>::R2;
  if (m < 0 || batch < 0 || (m * batch > 0 && (!a || !b || !evals))) return fail(COLAGB_ERR_INVALID, name);
  if (m * batch == 0) return COLAGB_OK;
  // two sweeps' rotations while they fit, else one's: the warps then wait for the sweep they finish
  const size_t smem1 = (size_t)m * (5 * sizeof(R) + sizeof(int)), smem2 = smem1 + (size_t)m * 2 * sizeof(R);
  const int two = smem2 <= kTriSmem;
  const size_t smem = two ? smem2 : smem1;
  if (smem > kTriSmem) return fail(COLAGB_ERR_INVALID, "tridiagonal eigensolver: m too large");
  if (smem > 48 * 1024) COLAGB_CUDA(set_smem_limit(k_tridiag_ql<R>, kTriSmem));
  const size_t smem_rot = (size_t)m * kRotRows * sizeof(R);
  if (evecs && smem_rot <= kTriSmem) {
    // eigenvectors: QL records its rotations (one thread generates them serially), then many CTAs
    // replay them on the rows of Z in shared memory; applying them to Z in global memory from the
    // same CTA, row per thread, cost ~95 % of the solve
    const int64_t cap = 6 * m * m + 64;
    void* buf = nullptr;
    const size_t bytes = (size_t)batch * cap * (sizeof(R2) + sizeof(int32_t)) +
                         (size_t)batch * (m + 1) * sizeof(int32_t);
    COLAGB_CUDA(cudaMallocAsync(&buf, bytes, st));
    R2* rec = static_cast<R2*>(buf);
    int32_t* rec_i = reinterpret_cast<int32_t*>(rec + batch * cap);
    int32_t* rec_n = rec_i + batch * cap;
    int32_t* rec_perm = rec_n + batch;
    k_tridiag_ql<R><<<(unsigned)batch, 128, smem, st>>>(a, b, m, two, evals, first_row, nullptr, status, rec, rec_i,
                                                        rec_n, rec_perm, cap);
    COLAGB_CUDA(cudaGetLastError());
    if (smem_rot > 48 * 1024) COLAGB_CUDA(set_smem_limit(k_tridiag_apply<R>, kTriSmem));
    k_tridiag_apply<R><<<dim3((unsigned)ceil_div(m, (int64_t)kRotRows), (unsigned)batch), kRotRows, smem_rot, st>>>(
        rec, rec_i, rec_n, rec_perm, m, cap, evecs);
    COLAGB_CUDA(cudaGetLastError());
    std::vector<int32_t> hn(batch);
    COLAGB_CUDA(cudaMemcpyAsync(hn.data(), rec_n, batch * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaStreamSynchronize(st));
    bool overflow = false;
    for (int64_t q = 0; q < batch; ++q) overflow |= hn[q] < 0;
    COLAGB_CUDA(cudaFreeAsync(buf, st));
    if (!overflow) {
      if (std::is_same<R, float>::value) {
        k_tridiag_rq<R><<<dim3((unsigned)ceil_div(m, (int64_t)128), (unsigned)batch), 128, 0, st>>>(a, b, m, evecs, evals);
        COLAGB_CUDA(cudaGetLastError());
      }
      return COLAGB_OK;
    }
    // rare: more rotations than recorded -- recompute with Z updated inside the QL kernel
  }
  k_tridiag_ql<R><<<(unsigned)batch, 128, smem, st>>>(a, b, m, two, evals, first_row, evecs, status);
  COLAGB_CUDA(cudaGetLastError());
  if (evecs && std::is_same<R, float>::value) {
    k_tridiag_rq<R><<<dim3((unsigned)ceil_div(m, (int64_t)128), (unsigned)batch), 128, 0, st>>>(a, b, m, evecs, evals);
    COLAGB_CUDA(cudaGetLastError());
  }
  return COLAGB_OK;
}

extern "C" int colagb_tridiag_eig_f64(const double* a, const double* b, int64_t m, int64_t batch, double* evals,
                                      double* first_row, double* evecs, int32_t* status, void* stream) {
  return tridiag_eig<double>(a, b, m, batch, evals, first_row, evecs, status, as_stream(stream),
                             "colagb_tridiag_eig_f64: bad arguments");
}

extern "C" int colagb_tridiag_eig_f32(const float* a, const float* b, int64_t m, int64_t batch, float* evals,
                                      float* first_row, float* evecs, int32_t* status, void* stream) {
  return tridiag_eig<float>(a, b, m, batch, evals, first_row, evecs, status, as_stream(stream),
                            "colagb_tridiag_eig_f32: bad arguments");
}

extern "C" int colagb_arnoldi_workspace_bytes(const colagb_op* A, int64_t bs, int32_t max_iters, size_t* bytes) {
  return colagb_lanczos_workspace_bytes(A, bs, max_iters, bytes);
}

extern "C" int colagb_arnoldi(const colagb_op* A, const void* V0, int64_t ldv0, int64_t bs,
                              const colagb_lanczos_params* params, void* basis, void* H, int32_t* steps, void* workspace,
                              size_t workspace_bytes, void* stream) {
  if (!A || !params || !V0 || !basis || !H || !steps) return fail(COLAGB_ERR_INVALID, "colagb_arnoldi: null argument");
  const colagb_op_node& r = A->nodes[A->root];
  if (r.rows != r.cols) return fail(COLAGB_ERR_INVALID, "colagb_arnoldi: operator must be square");
  if (bs < 1 || ldv0 < bs || params->max_iters < 1)
    return fail(COLAGB_ERR_INVALID, "colagb_arnoldi: bad bs / ldv0 / max_iters");
  cudaStream_t st = as_stream(stream);
  if (A->compute_dtype == COLAGB_F64)
    return arnoldi_t<double>(A, static_cast<const double*>(V0), ldv0, bs, *params, static_cast<double*>(basis),
                             static_cast<double*>(H), steps, workspace, workspace_bytes, st);
  return arnoldi_t<float>(A, static_cast<const float*>(V0), ldv0, bs, *params, static_cast<float*>(basis),
                          static_cast<float*>(H), steps, workspace, workspace_bytes, st);
}
