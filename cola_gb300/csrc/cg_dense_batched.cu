// Many independent dense SPD systems of uneven sizes, solved by plain FP32 CG in one persistent launch.
//
// Each system follows the reference's run_batched_cg exactly as a separate
// cola.linalg.solve(PSD(Dense(A_s)), b_s, CG(tol, max_iters)) call would (cg.py:94-154):
//   b <- b/|b|, r0 = b, p0 = r0, gamma0 = <r0, r0>, tol_eff = tol*|r0| + tol,
//   steps while |r| > tol_eff and k < max_iters, alpha/beta zeroed once |r| < 1e-40,
//   solution scaled back by |b|.
// Systems converge independently (per-system masks); the rows of the still-active systems are
// re-partitioned over all warps whenever one finishes, so warps stay busy: the matvec's rows in chunks
// of about equal cost (n_s per row) claimed from a counter, the vector phases' rows in units of 32
// spread over the SMs.  Three grid barriers a step.
//
// Small batches live from what a step costs beside the stream of A: with 608 CTAs, four barriers, the
// active list rebuilt three times a step by one thread, an FP64 multiply-add per matrix row and an FP64
// warp sum per eight rows (64 cycles of a scheduler for each such instruction on this chip), 24 systems of
// 300 .. 3000 rows took 108 us a step, 30 of them for the 200 MB of A a step reads on average; now 53 (and 256
// systems of 500 .. 8000 rows 3.58 ms for 23.7 GB, 0.98 of the measured copy bandwidth, after 3.85).
//
// Layout: A_s row-major at vals + a_off[s]; vectors of system s at v_off[s] in concatenated buffers.
// The search direction p of system s is kept in four copies, copy h shifted right by h elements
// (copy h holds p[i] at index i + h, each copy 16-byte aligned).  A row whose first element sits h
// floats past a 16-byte boundary is read as aligned 128-bit quads from its first boundary on, and
// copy h then lines the matching p quads up on 16-byte boundaries as well, so the matvec issues only
// 128-bit loads whatever n_s and the offsets are (the up to 3 + 3 elements before the first and
// after the last whole quad are scalar).  The shifted copies cost 3 extra n_s-float writes a step
// against the n_s^2 floats of A the step reads.
#include <algorithm>
#include <string>

#include "common.cuh"

namespace colagb {

constexpr int kDBThreads = 1024;  // one CTA per SM
constexpr int kDBMaxSystems = 1024;
// Matvec work claimed at a time: ~64 KB of A in a large batch, in a small one a third of a warp's share, but
// at least 8 KB.  (With 64 KB throughout, 330 MB of matrices are 5,000 chunks for 4,864 warps, and the few
// warps with a second one finish 25 us after the rest.)
constexpr long long kDBChunk = 16384, kDBChunkMin = 2048;

struct DenseBatchArgs {
  int S;
  const int32_t* sizes;
  const int64_t* a_off;
  const int64_t* v_off;
  const float* vals;
  const float* B;
  float* X;
  float *r, *p4, *ap;  // p4: the four shifted copies of p, system s at copy_base(s)
  double* acc;  // [3][S]: <p, Ap>, |r|^2, |b|^2
  unsigned long long* claim;  // the matvec's chunk counter (zero at every phase start)
  int* out_iters;
  int* out_status;
  double tol;
  int max_iters;
  GridBarrier gb;
};

struct DState {
  unsigned char* base;
  int S;
  __device__ __forceinline__ double* f64(int k) const { return reinterpret_cast<double*>(base) + (size_t)k * S; }
  __device__ __forceinline__ float* f32(int k) const { return reinterpret_cast<float*>(base + (size_t)2 * 8 * S) + (size_t)k * S; }
  __device__ __forceinline__ int* i32(int k) const {
    return reinterpret_cast<int*>(base + (size_t)2 * 8 * S) + (size_t)(6 + k) * S;
  }
  __device__ __forceinline__ long long* prefix() const {  // S + 1 cost prefix sums of the active list
    return reinterpret_cast<long long*>(base + (size_t)2 * 8 * S + (size_t)(6 + 4) * 4 * S + 16);
  }
  __device__ __forceinline__ long long* pbase() const { return prefix() + S + 1; }  // S offsets into p4
  __device__ __forceinline__ int* units() const { return reinterpret_cast<int*>(pbase() + S); }  // S + 1 unit prefixes
  __device__ __forceinline__ int* size() const { return units() + S + 1; }                       // S row counts
  __device__ __forceinline__ double& gamma(int s) const { return f64(0)[s]; }
  __device__ __forceinline__ double& mult(int s) const { return f64(1)[s]; }
  __device__ __forceinline__ float& alpha(int s) const { return f32(0)[s]; }
  __device__ __forceinline__ float& beta(int s) const { return f32(1)[s]; }
  __device__ __forceinline__ float& rn(int s) const { return f32(2)[s]; }
  __device__ __forceinline__ float& tol_eff(int s) const { return f32(3)[s]; }
  __device__ __forceinline__ float& conv(int s) const { return f32(4)[s]; }
  __device__ __forceinline__ int& it(int s) const { return i32(0)[s]; }
  __device__ __forceinline__ int& active(int s) const { return i32(1)[s]; }
  __device__ __forceinline__ int* act() const { return i32(2); }
};

static size_t dense_batch_smem(int S) {
  return (size_t)2 * 8 * S + (size_t)10 * 4 * S + 16 + (size_t)8 * (S + 1) + (size_t)8 * S + (size_t)4 * (2 * S + 1) + 64;
}

// Length of one shifted copy of an n-vector: room for index n - 1 + 3, rounded to whole quads.
__host__ __device__ __forceinline__ int64_t pcopy_len(int64_t n) { return ((n + 3) & ~int64_t(3)) + 4; }

// Write element i of p (value v) into all four shifted copies.
__device__ __forceinline__ void put_p(float* P0, int64_t cs, int i, float v) {
  P0[i] = v;
  P0[cs + i + 1] = v;
  P0[2 * cs + i + 2] = v;
  P0[3 * cs + i + 3] = v;
}

__device__ __forceinline__ float4 ld_a4(const float* q) {  // read-only A: no L1 allocation
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(q));
  return v;
}

__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
  s = fmaf(a.x, b.x, s);
  s = fmaf(a.y, b.y, s);
  s = fmaf(a.z, b.z, s);
  return fmaf(a.w, b.w, s);
}

// Up to N quads of a lane, 32 apart, `left` counting from the first one's position: four or more start with one
// on each accumulator, all others go to the first.
template <int N>
__device__ __forceinline__ void d_tail(const float4 (&a)[N], const float* P, int left, float& s0, float& s1, float& s2,
                                       float& s3) {
  auto p = [&](int u) { return *reinterpret_cast<const float4*>(P + 128 * u); };
  s0 = dot4(a[0], p(0), s0);
  if (left > 96) {
    s1 = dot4(a[1], p(1), s1);
    s2 = dot4(a[2], p(2), s2);
    s3 = dot4(a[3], p(3), s3);
#pragma unroll
    for (int u = 4; u < N; ++u)
      if (left > 32 * u) s0 = dot4(a[u], p(u), s0);
  } else {
    if (left > 32) s0 = dot4(a[1], p(1), s0);
    if (left > 64) s0 = dot4(a[2], p(2), s0);
  }
}

// <A row, p> over one warp; the result is in every lane.  Ar: the row (ns floats); P0: copy 0 of p,
// cs: the copy length.  Each lane keeps eight independent 128-bit loads of A in flight (4 KB per
// warp, 32 warps per SM): the matvec streams HBM and is bound by how many bytes are in
// flight, not by instructions (with 256-thread CTAs: four quads per lane and 3 blocks reached 0.46 of the copy bandwidth,
// four quads and 4 blocks 0.64, eight quads and 4 blocks 0.78; an L2 prefetch ahead of the loads
// lowered each).
__device__ __forceinline__ float row_dot(const float* __restrict__ Ar, const float* P0, int64_t cs, int ns,
                                         int lane) {
  const int h = (int)((reinterpret_cast<uintptr_t>(Ar) >> 2) & 3);  // floats past the last 16-byte boundary
  int j0 = (4 - h) & 3;                                              // first element of the first whole quad
  if (j0 > ns) j0 = ns;
  const int nq = (ns - j0) >> 2;
  const int jt = j0 + 4 * nq;
  const float* Aq = Ar + j0;              // 16-byte aligned
  const float* Pq = P0 + h * cs + j0 + h;  // copy h: p[j] at index j + h; j0 + h is 0 or 4
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  int q = lane;
  for (; q + 224 < nq; q += 256) {
    const float4 a0 = ld_a4(Aq + 4 * q), a1 = ld_a4(Aq + 4 * (q + 32));
    const float4 a2 = ld_a4(Aq + 4 * (q + 64)), a3 = ld_a4(Aq + 4 * (q + 96));
    const float4 a4 = ld_a4(Aq + 4 * (q + 128)), a5 = ld_a4(Aq + 4 * (q + 160));
    const float4 a6 = ld_a4(Aq + 4 * (q + 192)), a7 = ld_a4(Aq + 4 * (q + 224));
    s0 = dot4(a4, *reinterpret_cast<const float4*>(Pq + 4 * (q + 128)), s0);
    s1 = dot4(a5, *reinterpret_cast<const float4*>(Pq + 4 * (q + 160)), s1);
    s2 = dot4(a6, *reinterpret_cast<const float4*>(Pq + 4 * (q + 192)), s2);
    s3 = dot4(a7, *reinterpret_cast<const float4*>(Pq + 4 * (q + 224)), s3);
    const float4 p0 = *reinterpret_cast<const float4*>(Pq + 4 * q);
    const float4 p1 = *reinterpret_cast<const float4*>(Pq + 4 * (q + 32));
    const float4 p2 = *reinterpret_cast<const float4*>(Pq + 4 * (q + 64));
    const float4 p3 = *reinterpret_cast<const float4*>(Pq + 4 * (q + 96));
    s0 = dot4(a0, p0, s0);
    s1 = dot4(a1, p1, s1);
    s2 = dot4(a2, p2, s2);
    s3 = dot4(a3, p3, s3);
  }
  if (q < nq) {  // the last batch (at most seven quads), or a short row, in one round of predicated loads
    float4 a[7];
#pragma unroll
    for (int u = 0; u < 7; ++u) a[u] = q + 32 * u < nq ? ld_a4(Aq + 4 * (q + 32 * u)) : zero;
    d_tail<7>(a, Pq + 4 * q, nq - q, s0, s1, s2, s3);
  }
  if (lane < j0) s1 = fmaf(Ar[lane], P0[lane], s1);
  if (lane < ns - jt) s2 = fmaf(Ar[jt + lane], P0[jt + lane], s2);
  return warp_sum((s0 + s1) + (s2 + s3));
}

// Two short rows of one system (at most 128 whole quads each) in one round of loads; lanes 0..15 end with the
// first row's <A row, p>, lanes 16..31 with the second's.
__device__ __forceinline__ float row_dot_pair(const float* __restrict__ A0, const float* __restrict__ A1,
                                              const float* P0, int64_t cs, int ns, int lane) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* Ar[2] = {A0, A1};
  const float *Aq[2], *Pq[2];
  int j0[2], nq[2];
  float4 a[2][4];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int h = (int)((reinterpret_cast<uintptr_t>(Ar[r]) >> 2) & 3);
    j0[r] = (4 - h) & 3;
    if (j0[r] > ns) j0[r] = ns;
    nq[r] = (ns - j0[r]) >> 2;
    Aq[r] = Ar[r] + j0[r];
    Pq[r] = P0 + h * cs + j0[r] + h;
#pragma unroll
    for (int u = 0; u < 4; ++u) a[r][u] = lane + 32 * u < nq[r] ? ld_a4(Aq[r] + 4 * (lane + 32 * u)) : zero;
  }
  float s[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    if (lane < nq[r]) d_tail<4>(a[r], Pq[r] + 4 * lane, nq[r] - lane, t[0], t[1], t[2], t[3]);
    const int jt = j0[r] + 4 * nq[r];
    if (lane < j0[r]) t[1] = fmaf(Ar[r][lane], P0[lane], t[1]);
    if (lane < ns - jt) t[2] = fmaf(Ar[r][jt + lane], P0[jt + lane], t[2]);
    s[r] = (t[0] + t[1]) + (t[2] + t[3]);
  }
  const bool up = lane & 16;
  const float keep = up ? s[1] : s[0], send = up ? s[0] : s[1];
  float x = keep + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// The active list with its prefix sums of matvec cost (n_s^2) and of 32-row units, by one warp.
__device__ __forceinline__ int d_build(const DState& m) {
  __shared__ int s_n;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int c = 0, unit = 0;
    long long cost = 0;
    for (int s0 = 0; s0 < m.S; s0 += 32) {
      const int s = s0 + lane;
      const bool on = s < m.S && m.active(s);
      const long long ns = on ? m.size()[s] : 0;
      long long cs = ns * ns;
      int us = (int)((ns + 31) / 32);
      const long long c1 = cs;
      const int u1 = us;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long x = __shfl_up_sync(0xffffffffu, cs, o);
        const int y = __shfl_up_sync(0xffffffffu, us, o);
        if (lane >= o) {
          cs += x;
          us += y;
        }
      }
      const unsigned mask = __ballot_sync(0xffffffffu, on);
      if (on) {
        const int k = c + __popc(mask & ((1u << lane) - 1));
        m.act()[k] = s;
        m.prefix()[k] = cost + cs - c1;
        m.units()[k] = unit + us - u1;
      }
      c += __popc(mask);
      cost += __shfl_sync(0xffffffffu, cs, 31);
      unit += __shfl_sync(0xffffffffu, us, 31);
    }
    if (lane == 0) {
      m.prefix()[c] = cost;
      m.units()[c] = unit;
      s_n = c;
    }
  }
  __syncthreads();
  return s_n;
}

// (list position, row) of the first row whose cost start is >= c
__device__ __forceinline__ void d_locate(const DState& m, int nact, long long c, int& k, int& row) {
  const long long* P = m.prefix();
  int lo = 0, hi = nact;  // largest k with P[k] <= c
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (P[mid] <= c) lo = mid;
    else hi = mid;
  }
  k = lo;
  const unsigned ns = (unsigned)m.size()[m.act()[k]];
  // the offset within a system is below n_s^2 + kDBChunk < 2^63; most fit 32 bits
  const long long d = c - P[k] + ns - 1;
  const long long rr = d < (1ll << 32) ? (long long)((unsigned)d / ns) : d / ns;
  if (rr >= (long long)ns) {
    k += 1;
    row = 0;
  } else {
    row = (int)rr;
  }
}

// The active systems' rows in units of 32 of one system, unit u to warp u of the grid with neighbouring
// units on different SMs: f(s, i, in) with lane's row i, in = whether it exists.
template <class F>
__device__ __forceinline__ void d_units(const DState& m, int nact, F f) {
  if (nact == 0) return;
  const int lane = threadIdx.x & 31;
  const int* Q = m.units();
  const int W = gridDim.x * (kDBThreads / 32);
  for (int u = blockIdx.x + gridDim.x * (threadIdx.x >> 5); u < Q[nact]; u += W) {
    int lo = 0, hi = nact;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (Q[mid] <= u) lo = mid;
      else hi = mid;
    }
    const int s = m.act()[lo], i = 32 * (u - Q[lo]) + lane;
    f(s, i, i < m.size()[s]);
  }
}

// The matvec's rows in chunks of about equal cost, claimed from a counter in order, so
// that warps whose loads return sooner (SMs nearer the data, less contended) take more chunks and all
// finish together at the grid barrier.  A chunk holds the rows whose cost starts fall inside it.
// Each warp claims its next chunk before working on the current one, hiding the atomic's latency.
// f(s, r0, r1) per (system, row range); flush(s) when the warp moves on to another system and at the
// end.
template <class RowFn, class Flush>
__device__ __forceinline__ void d_claim_rows(const DenseBatchArgs& a, const DState& m, int nact, RowFn f,
                                             Flush flush) {
  if (nact == 0) return;
  const int lane = threadIdx.x & 31;
  const long long T = m.prefix()[nact];
  const long long W = (long long)gridDim.x * (kDBThreads / 32);
  long long chunk = T / (3 * W);
  chunk = chunk < kDBChunkMin ? kDBChunkMin : chunk > kDBChunk ? kDBChunk : chunk;
  const long long nch = (T + chunk - 1) / chunk;
  // the first chunk by position, the others from the counter
  unsigned long long c = blockIdx.x + gridDim.x * (unsigned long long)(threadIdx.x >> 5);
  int last = -1;
  while ((long long)c < nch) {
    unsigned long long next = 0;
    if (lane == 0) next = W + atomicAdd(a.claim, 1ull);
    int k0, r0, k1, r1;
    d_locate(m, nact, (long long)c * chunk, k0, r0);
    const long long e = ((long long)c + 1) * chunk;
    d_locate(m, nact, e < T ? e : T, k1, r1);
    int k = k0, row = r0;
    while (k < k1 || (k == k1 && row < r1)) {
      if (k >= nact) break;
      const int s = m.act()[k];
      const int end = (k == k1) ? r1 : m.size()[s];
      if (s != last && last >= 0) flush(last);
      last = s;
      f(s, row, end);
      k += 1;
      row = 0;
    }
    c = __shfl_sync(0xffffffffu, next, 0);
  }
  if (last >= 0) flush(last);
}

__global__ void __launch_bounds__(kDBThreads, 1) k_dense_batched_cg(const __grid_constant__ DenseBatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DState m{smem_raw, a.S};
  const int lane = threadIdx.x & 31;
  const int S = a.S;
  double* acc_pap = a.acc;
  double* acc_rr = a.acc + S;
  double* acc_bb = a.acc + 2 * S;
  auto add = [&](double* to, double v) {  // the warp's sum of v
    v = warp_sum(v);
    if (lane == 0 && v != 0.0) atomicAdd(to, v);
  };

  for (int s = threadIdx.x; s < S; s += blockDim.x) {
    m.size()[s] = a.sizes[s];
    m.active(s) = a.sizes[s] > 0;
    m.it(s) = 0;
    m.rn(s) = 0.f;
    m.tol_eff(s) = 0.f;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long off = 0;
    for (int s = 0; s < S; ++s) {
      m.pbase()[s] = off;
      off += 4 * pcopy_len(m.size()[s]);
    }
  }
  // |b|^2
  int nact = d_build(m);
  d_units(m, nact, [&](int s, int i, bool in) {
    const double b = in ? (double)a.B[a.v_off[s] + i] : 0.0;
    add(acc_bb + s, b * b);
  });
  if (!grid_sync(a.gb)) return;
  for (int s = threadIdx.x; s < S; s += blockDim.x) m.mult(s) = sqrt(__ldcg(acc_bb + s));
  __syncthreads();
  // r = b / |b| (x0 = 0), p = r, x = 0, |r|^2
  d_units(m, nact, [&](int s, int i, bool in) {
    double rr = 0.0;
    if (in) {
      const int64_t o = a.v_off[s] + i;
      const double mu = m.mult(s);
      const float rv = (mu < 1e-40) ? a.B[o] / 1e-40f : (float)(a.B[o] / mu);
      a.r[o] = rv;
      put_p(a.p4 + m.pbase()[s], pcopy_len(m.size()[s]), i, rv);
      a.X[o] = 0.f;
      rr = (double)rv * rv;
    }
    add(acc_rr + s, rr);
  });
  if (!grid_sync(a.gb)) return;
  for (int s = threadIdx.x; s < S; s += blockDim.x) {
    if (!m.active(s)) continue;
    const double rr = __ldcg(acc_rr + s);
    m.gamma(s) = rr;
    const float rn = (float)sqrt(rr);
    m.rn(s) = rn;
    m.tol_eff(s) = (float)a.tol * rn + (float)a.tol;
    m.active(s) = (rn > m.tol_eff(s)) && a.max_iters > 0;
  }
  nact = d_build(m);
  if (!grid_sync(a.gb)) return;  // everyone has read acc_rr

  while (nact > 0) {
    // acc_rr was read before the last barrier and is next added to after the next one
    if (blockIdx.x == 0)
      for (int s = threadIdx.x; s < S; s += blockDim.x) acc_rr[s] = 0.0;
    // A: Ap = A p (warp per row), <p, Ap>
    {
      double part = 0.0;  // lanes keep the terms of different rows
      d_claim_rows(a, m, nact,
                   [&](int s, int r0, int r1) {
                     const int ns = m.size()[s];
                     const float* A = a.vals + a.a_off[s];
                     const float* P0 = a.p4 + m.pbase()[s];
                     const int64_t cs = pcopy_len(ns);
                     for (int rb = r0; rb < r1; rb += 32) {
                       float keep = 0.f;
                       const int re = rb + 32 < r1 ? rb + 32 : r1;
                       int row = rb;
                       if (ns <= 512)
                         for (; row + 1 < re; row += 2) {
                           const float* A0 = A + (int64_t)row * ns;
                           const float v = row_dot_pair(A0, A0 + ns, P0, cs, ns, lane);
                           const float v0 = __shfl_sync(0xffffffffu, v, 0), v1 = __shfl_sync(0xffffffffu, v, 16);
                           if (lane == row - rb) keep = v0;
                           if (lane == row + 1 - rb) keep = v1;
                         }
                       for (; row < re; ++row) {
                         const float v = row_dot(A + (int64_t)row * ns, P0, cs, ns, lane);
                         if (lane == row - rb) keep = v;
                       }
                       if (rb + lane < re) {
                         a.ap[a.v_off[s] + rb + lane] = keep;
                         part += (double)P0[rb + lane] * keep;
                       }
                     }
                   },
                   [&](int s) {
                     add(acc_pap + s, part);
                     part = 0.0;
                   });
    }
    if (!grid_sync(a.gb)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.claim = 0ull;  // next used after two more grid barriers
    for (int j = threadIdx.x; j < nact; j += blockDim.x) {
      const int s = m.act()[j];
      const double pap = __ldcg(acc_pap + s);
      const double den = fabs(pap) < 1e-40 ? 1e-40 : pap;
      const bool conv = m.rn(s) < 1e-40f;
      m.conv(s) = conv ? 1.f : 0.f;
      m.alpha(s) = conv ? 0.f : (float)(m.gamma(s) / den);
    }
    __syncthreads();
    // B: x += alpha p, r -= alpha Ap, |r|^2
    d_units(m, nact, [&](int s, int i, bool in) {
      double rr = 0.0;
      if (in) {
        const int64_t o = a.v_off[s] + i;
        const float al = m.alpha(s);
        const float* P0 = a.p4 + m.pbase()[s];
        a.X[o] += al * P0[i];
        const float rv = a.r[o] - al * a.ap[o];
        a.r[o] = rv;
        rr = (double)rv * rv;
      }
      add(acc_rr + s, rr);
    });
    if (!grid_sync(a.gb)) return;
    if (blockIdx.x == 0)
      for (int s = threadIdx.x; s < S; s += blockDim.x) acc_pap[s] = 0.0;
    int changed = 0;
    for (int j = threadIdx.x; j < nact; j += blockDim.x) {
      const int s = m.act()[j];
      const double g1 = __ldcg(acc_rr + s);
      const double den = fabs(m.gamma(s)) < 1e-40 ? 1e-40 : m.gamma(s);
      m.beta(s) = m.conv(s) != 0.f ? 0.f : (float)(g1 / den);
      m.gamma(s) = g1;
      const float rn = (float)sqrt(g1);
      m.rn(s) = rn;
      m.it(s) += 1;
      const int on = (rn > m.tol_eff(s)) && (m.it(s) < a.max_iters);
      m.active(s) = on;
      changed |= !on;
    }
    if (__syncthreads_or(changed)) nact = d_build(m);
    // C: p = r + beta p (systems that go on)
    d_units(m, nact, [&](int s, int i, bool in) {
      if (in) {
        float* P0 = a.p4 + m.pbase()[s];
        put_p(P0, pcopy_len(m.size()[s]), i, a.r[a.v_off[s] + i] + m.beta(s) * P0[i]);
      }
    });
    if (!grid_sync(a.gb)) return;
  }
  // x *= |b|
  __syncthreads();
  for (int s = threadIdx.x; s < S; s += blockDim.x) m.active(s) = m.size()[s] > 0;
  nact = d_build(m);
  d_units(m, nact, [&](int s, int i, bool in) {
    if (in) a.X[a.v_off[s] + i] *= (float)m.mult(s);
  });
  if (blockIdx.x == 0)
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
      if (a.out_iters) a.out_iters[s] = m.it(s);
      if (a.out_status) a.out_status[s] = (m.rn(s) > m.tol_eff(s)) ? COLAGB_SYS_MAX_ITERS : COLAGB_SYS_CONVERGED;
    }
}

}  // namespace colagb

using namespace colagb;

extern "C" int colagb_cg_dense_batched_workspace_bytes(int64_t num_systems, int64_t total_rows, size_t* bytes) {
  if (!bytes || num_systems < 0 || total_rows < 0) return fail(COLAGB_ERR_INVALID, "dense batched CG: bad arguments");
  Bump ws = Bump::measuring();
  ws.take<float>(total_rows);
  ws.take<float>(4 * (total_rows + 8 * num_systems));  // >= 4 * sum of pcopy_len(n_s)
  ws.take<float>(total_rows);
  ws.take<double>(3 * (num_systems > 0 ? num_systems : 1));
  ws.take<unsigned int>(8);
  ws.take<unsigned long long>(1);
  *bytes = ws.peak;
  return COLAGB_OK;
}

extern "C" int colagb_cg_dense_batched_solve(int64_t num_systems, const int32_t* sizes, const int64_t* a_offsets,
                                             const int64_t* v_offsets, int64_t total_rows, const float* values,
                                             const float* B, float* X, double tol, int32_t max_iters,
                                             int32_t* per_system_iters, int32_t* per_system_status, void* workspace,
                                             size_t workspace_bytes, void* stream) {
  if (num_systems < 0 || num_systems > kDBMaxSystems || total_rows < 0 || max_iters < 0)
    return fail(COLAGB_ERR_INVALID, "dense batched CG: need 0 <= num_systems <= 1024, max_iters >= 0");
  if (num_systems == 0 || total_rows == 0) return COLAGB_OK;
  if (!sizes || !a_offsets || !v_offsets || !values || !B || !X)
    return fail(COLAGB_ERR_INVALID, "dense batched CG: null argument");
  size_t need = 0;
  COLAGB_TRY(colagb_cg_dense_batched_workspace_bytes(num_systems, total_rows, &need));
  if (!workspace || workspace_bytes < need) return fail(COLAGB_ERR_WORKSPACE, "dense batched CG: workspace too small");
  Bump ws(workspace, workspace_bytes);
  DenseBatchArgs a;
  a.S = (int)num_systems;
  a.sizes = sizes;
  a.a_off = a_offsets;
  a.v_off = v_offsets;
  a.vals = values;
  a.B = B;
  a.X = X;
  a.r = ws.take<float>(total_rows);
  a.p4 = ws.take<float>(4 * (total_rows + 8 * num_systems));
  a.ap = ws.take<float>(total_rows);
  a.acc = ws.take<double>(3 * num_systems);
  unsigned int* bar = ws.take<unsigned int>(8);
  a.claim = ws.take<unsigned long long>(1);
  a.out_iters = per_system_iters;
  a.out_status = per_system_status;
  a.tol = tol;
  a.max_iters = max_iters;
  a.gb.arrivals = reinterpret_cast<unsigned long long*>(bar);
  a.gb.err = reinterpret_cast<int*>(bar + 2);
  a.gb.spin_limit = kDefaultSpinLimit;
  cudaStream_t st = as_stream(stream);
  const size_t smem = dense_batch_smem(a.S);
  if (smem > 48 * 1024) COLAGB_CUDA(set_smem_limit(k_dense_batched_cg, dense_batch_smem(kDBMaxSystems)));
  int occ = 0;
  COLAGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_dense_batched_cg, kDBThreads, smem));
  if (occ < 1) return fail(COLAGB_ERR_UNSUPPORTED, "dense batched CG kernel cannot be resident");
  const int nb = num_sms();
  a.gb.nblocks = (unsigned)nb;
  COLAGB_CUDA(cudaMemsetAsync(bar, 0, 8 * sizeof(unsigned int), st));
  COLAGB_CUDA(cudaMemsetAsync(a.claim, 0, sizeof(unsigned long long), st));
  COLAGB_CUDA(cudaMemsetAsync(a.acc, 0, 3 * num_systems * sizeof(double), st));
  void* args[] = {&a};
  COLAGB_CUDA(cudaLaunchCooperativeKernel((const void*)k_dense_batched_cg, dim3(nb), dim3(kDBThreads), args, smem, st));
  unsigned int herr = 0;
  COLAGB_CUDA(cudaMemcpyAsync(&herr, bar + 2, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
  COLAGB_CUDA(cudaStreamSynchronize(st));
  if (herr != 0) return fail(COLAGB_ERR_TIMEOUT, "dense batched CG: a grid barrier timed out");
  return COLAGB_OK;
}

// ---------------------------------------------------------------------------------------------
// FP64 residual of the uneven dense batch, for iterative refinement on top of the FP32 CG above:
// R = B - A X in FP64 (A's FP32 values, FP64 products and sums), one warp per row, plus |r_s|^2 per
// system.  The system of a row comes from a binary search of v_offsets.

namespace colagb {

__global__ void __launch_bounds__(256) k_dense_residual64(int S, const int32_t* __restrict__ sizes,
                                                          const int64_t* __restrict__ a_off,
                                                          const int64_t* __restrict__ v_off, int64_t total_rows,
                                                          const float* __restrict__ vals,
                                                          const double* __restrict__ B, const double* __restrict__ X,
                                                          double* __restrict__ R, double* __restrict__ rr) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < total_rows; g += nwarps) {
    int lo = 0, hi = S - 1;  // last system whose v_off <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (v_off[mid] <= g) lo = mid;
      else hi = mid - 1;
    }
    const int s = lo;
    const int64_t n = sizes[s];
    const int64_t i = g - v_off[s];
    const float* row = vals + a_off[s] + i * n;
    const double* x = X + v_off[s];
    double acc = 0.0;
    for (int64_t j = lane; j < n; j += 32) acc += (double)row[j] * x[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const double r = B[g] - acc;
      R[g] = r;
      atomicAdd(rr + s, r * r);
    }
  }
}

}  // namespace colagb

extern "C" int colagb_dense_batched_residual64(int64_t num_systems, const int32_t* sizes, const int64_t* a_offsets,
                                               const int64_t* v_offsets, int64_t total_rows, const float* values,
                                               const double* B, const double* X, double* R, double* rr,
                                               void* stream) {
  if (num_systems < 1 || num_systems > kDBMaxSystems || total_rows < 0 || !sizes || !a_offsets || !v_offsets ||
      !values || !B || !X || !R || !rr)
    return fail(COLAGB_ERR_INVALID, "colagb_dense_batched_residual64: bad arguments");
  cudaStream_t st = as_stream(stream);
  COLAGB_CUDA(cudaMemsetAsync(rr, 0, num_systems * sizeof(double), st));
  if (total_rows == 0) return COLAGB_OK;
  const int64_t want = ceil_div(total_rows * 32, 256);
  const int blocks = (int)std::min<int64_t>(want, (int64_t)num_sms() * 16);
  k_dense_residual64<<<blocks, 256, 0, st>>>((int)num_systems, sizes, a_offsets, v_offsets, total_rows, values, B, X,
                                             R, rr);
  COLAGB_CUDA(cudaGetLastError());
  return COLAGB_OK;
}
