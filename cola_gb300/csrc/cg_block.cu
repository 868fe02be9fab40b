// Block schedule of the batched solver: many right-hand sides of ONE matrix advancing in lockstep.
//
// The reference's CG already runs a block of right-hand sides together: run_batched_cg keeps x, r, p
// as (n, k) arrays and per-column alpha / beta (cola/linalg/inverse/cg.py:94-154), so every step reads
// the matrix once for all k columns.  This kernel does the same on the GPU for a shared-values family
// (colagb_batched_csr.shared_values), with the batched solver's arithmetic: FP32 preconditioned CG
// (none / Jacobi), FP64 solution, FP64 residual replacement (reliable updates) and the FP64 true
// residual as the only convergence test, per column.
//
// Layout: the Krylov vectors are column-interleaved (n, kp) FP32 (kp = k padded to 4, 8, 16, 32, 64
// or 128), so one CSR entry multiplies a contiguous row of kp values of p: the kp / 4 threads of a row
// each take one 128-bit column quad.  The FP64 solution and the normalised right-hand side are
// (n, kp) FP64.  One persistent cooperative grid, rows split into contiguous ranges per CTA; per-column
// partial sums reduce in a fixed order (every CTA derives bit-identical scalars); three bounded grid
// barriers per step, two more per residual replacement.  A replacement happens for all columns at
// once, whenever one column's FP32 residual has dropped by inner_tol since the last one.
#include <algorithm>
#include <string>

#include "common.cuh"

namespace colagb {

constexpr int kBT = 1024;       // threads per CTA, one CTA per SM
constexpr int kBMaxK = 128;     // columns per launch (the host splits wider blocks)

struct BlockArgs {
  int64_t n;
  int kp, q, S;                 // padded columns, column quads, real columns
  const int32_t* __restrict__ indptr;
  const int32_t* __restrict__ indices;
  const float* __restrict__ vals;
  const double* B;              // (S, n) right-hand sides
  double* X;                    // (S, n) solutions
  double* Bn;                   // (n, kp) B / |B|, per column
  double* X64;                  // (n, kp)
  float *R, *P, *AP, *D, *dinv; // (n, kp) x4, n
  float* pf;                    // [nb][3][kp]
  double* pd;                   // [nb][2][kp]
  int32_t* out_status;
  int32_t* out_iters;
  double* out_relres;
  int32_t* out_nrep;            // (1,) replacement count
  double tol, inner_tol;
  int max_inner, max_sweeps, jacobi;
  int r_resident;               // r of the CTA's rows is kept in shared memory
  GridBarrier gb;
};

// Per-thread float4 partials of column quad (threadIdx % q, q a power of two <= 32), NV of them -> dst[v][0..4q)
// as fixed-order sums: a shuffle tree over the lanes of a warp that share the quad, then warp j adds the
// warps' sums of quad j.
template <int NV>
__device__ __forceinline__ void block_quad_partials(float4 (&v)[NV], int q, float* const (&dst)[NV], float4* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = kBT / 32;
  auto add = [](float4& x, int o) {
    x.x += __shfl_xor_sync(0xffffffffu, x.x, o);
    x.y += __shfl_xor_sync(0xffffffffu, x.y, o);
    x.z += __shfl_xor_sync(0xffffffffu, x.z, o);
    x.w += __shfl_xor_sync(0xffffffffu, x.w, o);
  };
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    for (int o = 16; o >= q; o >>= 1) add(v[k], o);
    if (lane < q) red[k * kBT + lane * NW + warp] = v[k];  // lane l < q holds the warp's sum for quad l
  }
  __syncthreads();
  if (warp < q) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      float4 t = red[k * kBT + warp * NW + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) add(t, o);
      if (lane == 0) reinterpret_cast<float4*>(dst[k])[warp] = t;
    }
  }
  __syncthreads();
}

// Column totals over all CTAs (partials of CTA b at p + b * stride; ncols a power of two >= 4), fixed order,
// into smem out[0..ncols): neighbouring threads take neighbouring columns, the groups of threads every
// G-th CTA with their loads in flight together, then a tree over the groups.  (One load at a time over
// 608 CTAs' partials was the larger part of a step.)
template <class T>
__device__ __forceinline__ void grid_totals(const T* p, int nb, int64_t stride, int ncols, T* out, T* tmp) {
  const int w = ncols < 32 ? ncols : 32, c = threadIdx.x % w, g = threadIdx.x / w, G = kBT / w;
  for (int cb = 0; cb < ncols; cb += w) {
    constexpr int B = 8;
    T acc = T(0);
    for (int b = g; b < nb; b += B * G) {
      T v[B];
#pragma unroll
      for (int e = 0; e < B; ++e) v[e] = b + e * G < nb ? __ldcg(p + (int64_t)(b + e * G) * stride + cb + c) : T(0);
#pragma unroll
      for (int e = 0; e < B; ++e) acc += v[e];
    }
    tmp[g * w + c] = acc;
    __syncthreads();
    for (int h = G / 2; h >= 1; h >>= 1) {
      if (g < h) tmp[g * w + c] += tmp[(g + h) * w + c];
      __syncthreads();
    }
    if (g == 0) out[cb + c] = tmp[c];
    __syncthreads();
  }
}

// One CTA of 1024 threads per SM (64 registers): the SpMM phase is latency-bound on index -> p-row gathers
// and wants full warp slots, the barriers and column totals want few CTAs; r of the CTA's rows stays in
// shared memory where it takes at most half of it (the rest caches the gathers of p).  us a step for 64^3
// unknowns x 16 columns, FP32: 57 with 256-thread CTAs, four per SM, and totals read one partial after
// another; 43 in this shape; 41 with two units of the vector phases in flight; 40 with eight entries' indices
// ahead of their gathers; 37 with r resident.  Rows of the matrix resident as well took the L1 from the
// gathers (60).
__global__ void __launch_bounds__(kBT, 1) k_block_ir(const BlockArgs a) {
  extern __shared__ float4 red[];  // 2 * kBT
  double* const tmpd = reinterpret_cast<double*>(red);  // kBT, between the reductions
  float* const tmpf = reinterpret_cast<float*>(red + kBT);
  __shared__ float alpha[kBMaxK], beta[kBMaxK], gam[kBMaxK], rmax[kBMaxK], pap[kBMaxK];
  __shared__ float rg[2 * kBMaxK];  // |r|^2, then |r|; <r, z>
  __shared__ double bnorm[kBMaxK], relres[kBMaxK], tot64[2 * kBMaxK];
  __shared__ int frozen[kBMaxK], its[kBMaxK], status[kBMaxK];

  const int64_t n = a.n;
  const int kp = a.kp, q = a.q;
  const int nb = gridDim.x;
  const int64_t rows = ceil_div(n, nb);
  const int64_t r0 = (int64_t)blockIdx.x * rows < n ? (int64_t)blockIdx.x * rows : n;
  const int64_t r1 = r0 + rows < n ? r0 + rows : n;
  const int nu = (int)((r1 - r0) * q);   // (row, quad) units of this CTA
  int qs = 0;                            // log2 q
  while ((1 << qs) < q) ++qs;
  const int cq = (int)threadIdx.x % q;
  float* const rn = rg;
  float* const gnew = rg + kp;
  float* pf = a.pf + (int64_t)blockIdx.x * 3 * kp;
  double* pd = a.pd + (int64_t)blockIdx.x * 2 * kp;
  const float4* P4 = reinterpret_cast<const float4*>(a.P);
  float4* const R4 = a.r_resident ? red + 2 * kBT : reinterpret_cast<float4*>(a.R) + r0 * q;  // the CTA's units
  float* const Rf = reinterpret_cast<float*>(R4);
  float4* Pw4 = reinterpret_cast<float4*>(a.P);
  float4* AP4 = reinterpret_cast<float4*>(a.AP);
  float4* D4 = reinterpret_cast<float4*>(a.D);

  // ---- setup: Bn = B (transposed), |B|^2 per column, X64 = D = 0, Jacobi diagonal ----
  for (int64_t u = threadIdx.x; u < (r1 - r0) * kp; u += kBT) {
    const int64_t i = r0 + u / kp;
    const int c = (int)(u % kp);
    a.Bn[i * kp + c] = c < a.S ? a.B[(int64_t)c * n + i] : 0.0;
    a.X64[i * kp + c] = 0.0;
    a.D[i * kp + c] = 0.f;
  }
  __syncthreads();
  if ((int)threadIdx.x < kp) {  // fixed-order per-column sum over this CTA's rows
    double acc = 0.0;
    for (int64_t i = r0; i < r1; ++i) {
      const double bv = a.Bn[i * kp + threadIdx.x];
      acc += bv * bv;
    }
    pd[threadIdx.x] = acc;
  }
  if (a.dinv)
    for (int64_t i = r0 + threadIdx.x; i < r1; i += kBT) {
      float dg = 0.f;
      for (int32_t j = a.indptr[i]; j < a.indptr[i + 1]; ++j)
        if (a.indices[j] == i) dg += a.vals[j];
      a.dinv[i] = dg != 0.f ? 1.f / dg : 1.f;
    }
  if (!grid_sync(a.gb)) return;
  grid_totals<double>(a.pd, nb, 2 * kp, kp, tot64, tmpd);
  for (int c = threadIdx.x; c < kp; c += kBT) {
    const double bb = sqrt(tot64[c]);
    bnorm[c] = bb;
    its[c] = 0;
    frozen[c] = !(bb > 0.0);
    status[c] = bb > 0.0 ? COLAGB_SYS_RUNNING : (bb == 0.0 ? COLAGB_SYS_CONVERGED : COLAGB_SYS_NAN);
    relres[c] = bb > 0.0 ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int64_t u = threadIdx.x; u < (r1 - r0) * kp; u += kBT) {
    const int c = (int)(u % kp);
    const int64_t e = (r0 + u / kp) * kp + c;
    a.Bn[e] = bnorm[c] > 0.0 ? a.Bn[e] / bnorm[c] : 0.0;
  }

  // FP64 residual replacement of every running column: X64 += D + alpha P (the step's correction,
  // which phase C would otherwise add to D), D = 0, R = Bn - A X64 (FP64), then |r64|^2 and <r, z>;
  // afterwards relres, gamma and rmax are set and converged columns frozen.
  auto replace = [&](bool first) -> bool {
    if (!first) {
      for (int64_t u = threadIdx.x; u < (r1 - r0) * kp; u += kBT) {
        const int64_t e = r0 * kp + u;
        const int c = (int)(u % kp);
        a.X64[e] += (double)(a.D[e] + alpha[c] * a.P[e]);
        a.D[e] = 0.f;
      }
      if (!grid_sync(a.gb)) return false;
    }
    double acc_rr = 0.0;
    float acc_rz = 0.f;
    const int col = (int)threadIdx.x % kp;  // kp divides kBT: thread t always takes column t % kp
    for (int64_t u = threadIdx.x; u < (r1 - r0) * kp; u += kBT) {
      const int64_t i = r0 + u / kp;
      double ax = 0.0;
      if (!first)
        for (int32_t j = a.indptr[i]; j < a.indptr[i + 1]; ++j)
          ax += (double)a.vals[j] * a.X64[(int64_t)a.indices[j] * kp + col];
      const double rv = frozen[col] ? 0.0 : a.Bn[i * kp + col] - ax;
      const float rf = (float)rv;
      Rf[u] = rf;
      acc_rr += rv * rv;
      acc_rz += rf * (a.jacobi ? a.dinv[i] : 1.f) * rf;
    }
    // fixed-order per-column block sums (thread t accumulated column t % kp)
    tmpd[threadIdx.x] = acc_rr;
    tmpf[threadIdx.x] = acc_rz;
    __syncthreads();
    if ((int)threadIdx.x < kp) {
      double s1 = 0.0;
      float s2 = 0.f;
      for (int t = threadIdx.x; t < kBT; t += kp) {
        s1 += tmpd[t];
        s2 += tmpf[t];
      }
      pd[kp + threadIdx.x] = s1;
      pf[2 * kp + threadIdx.x] = s2;
    }
    __syncthreads();
    if (!grid_sync(a.gb)) return false;
    grid_totals<double>(a.pd + kp, nb, 2 * kp, kp, tot64, tmpd);
    grid_totals<float>(a.pf + 2 * kp, nb, 3 * kp, kp, gnew, tmpf);
    for (int c = threadIdx.x; c < kp; c += kBT) {
      if (frozen[c]) continue;
      const double rr = sqrt(tot64[c]);
      relres[c] = rr;
      rmax[c] = (float)rr;
      rn[c] = (float)rr;
      if (!(rr == rr)) {
        status[c] = COLAGB_SYS_NAN;
        frozen[c] = 1;
      } else if (rr <= a.tol) {
        status[c] = COLAGB_SYS_CONVERGED;
        frozen[c] = 1;
      }
    }
    __syncthreads();
    return true;
  };

  if (!replace(true)) return;
  for (int c = threadIdx.x; c < kp; c += kBT) gam[c] = gnew[c];
  __syncthreads();
  // p = z
  for (int u = threadIdx.x; u < nu; u += kBT) {
    const int64_t i = r0 + (u >> qs);
    const float4 r = R4[u];
    const float d = a.jacobi ? a.dinv[i] : 1.f;
    Pw4[i * q + cq] = make_float4(d * r.x, d * r.y, d * r.z, d * r.w);
  }
  if (!grid_sync(a.gb)) return;

  int it = 0, nrep = 1;
  while (true) {
    if (!__syncthreads_or((int)threadIdx.x < kp && !frozen[threadIdx.x])) break;
    // ---- A: AP = A P, <p, Ap> ----
    float4 parts[1] = {make_float4(0.f, 0.f, 0.f, 0.f)};
    float4& part = parts[0];
    for (int u = threadIdx.x; u < nu; u += kBT) {
      const int64_t i = r0 + (u >> qs);
      const int32_t b = __ldg(a.indptr + i), e = __ldg(a.indptr + i + 1);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      // eight entries' indices and values at a time, then their p-row gathers four by four, so that the
      // loads of a group are in flight together; the products are added in entry order
      for (int32_t j0 = b; j0 < e; j0 += 8) {
        int32_t col[8];
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const bool ok = j0 + t < e;
          col[t] = ok ? __ldg(a.indices + j0 + t) : 0;
          v[t] = ok ? __ldg(a.vals + j0 + t) : 0.f;
        }
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          float4 x[4];
#pragma unroll
          for (int t = 0; t < 4; ++t)
            x[t] = j0 + h + t < e ? P4[(int64_t)col[h + t] * q + cq] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (j0 + h + t < e) {
              acc.x += v[h + t] * x[t].x; acc.y += v[h + t] * x[t].y; acc.z += v[h + t] * x[t].z; acc.w += v[h + t] * x[t].w;
            }
          }
        }
      }
      AP4[i * q + cq] = acc;
      const float4 p = P4[i * q + cq];
      part.x += p.x * acc.x; part.y += p.y * acc.y; part.z += p.z * acc.z; part.w += p.w * acc.w;
    }
    float* const to_a[1] = {pf};
    block_quad_partials<1>(parts, q, to_a, red);
    if (!grid_sync(a.gb)) return;
    grid_totals<float>(a.pf, nb, 3 * kp, kp, pap, tmpf);
    for (int c = threadIdx.x; c < kp; c += kBT) {
      if (frozen[c]) { alpha[c] = 0.f; continue; }
      if (!(pap[c] > 0.f)) {
        status[c] = pap[c] == pap[c] ? COLAGB_SYS_BREAKDOWN : COLAGB_SYS_NAN;
        frozen[c] = 1;
        alpha[c] = 0.f;
      } else {
        alpha[c] = gam[c] / pap[c];
      }
    }
    __syncthreads();
    // ---- B: r -= alpha Ap, |r|^2, <r, z> (d += alpha p waits for phase C, which reads p anyway) ----
    float4 sums[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    float4 &prr = sums[0], &prz = sums[1];
    const float4 al = make_float4(alpha[4 * cq], alpha[4 * cq + 1], alpha[4 * cq + 2], alpha[4 * cq + 3]);
    // unit u is element r0 * q + u: two units in flight, the second one's terms zero past the end
    for (int u = threadIdx.x; u < nu; u += 2 * kBT) {
      const int64_t e0 = r0 * q + u, e1 = u + kBT < nu ? e0 + kBT : e0;
      const float4 ap0 = AP4[e0], ap1 = AP4[e1];
      float4 x0 = R4[u], x1 = R4[u + (int)(e1 - e0)];
      const float d0 = a.jacobi ? a.dinv[e0 >> qs] : 1.f, d1 = a.jacobi ? a.dinv[e1 >> qs] : 1.f;
      x0.x -= al.x * ap0.x; x0.y -= al.y * ap0.y; x0.z -= al.z * ap0.z; x0.w -= al.w * ap0.w;
      R4[u] = x0;
      prr.x += x0.x * x0.x; prr.y += x0.y * x0.y; prr.z += x0.z * x0.z; prr.w += x0.w * x0.w;
      prz.x += x0.x * d0 * x0.x; prz.y += x0.y * d0 * x0.y; prz.z += x0.z * d0 * x0.z; prz.w += x0.w * d0 * x0.w;
      if (e1 != e0) {
        x1.x -= al.x * ap1.x; x1.y -= al.y * ap1.y; x1.z -= al.z * ap1.z; x1.w -= al.w * ap1.w;
        R4[u + kBT] = x1;
        prr.x += x1.x * x1.x; prr.y += x1.y * x1.y; prr.z += x1.z * x1.z; prr.w += x1.w * x1.w;
        prz.x += x1.x * d1 * x1.x; prz.y += x1.y * d1 * x1.y; prz.z += x1.z * d1 * x1.z; prz.w += x1.w * d1 * x1.w;
      }
    }
    float* const to_b[2] = {pf + kp, pf + 2 * kp};
    block_quad_partials<2>(sums, q, to_b, red);
    if (!grid_sync(a.gb)) return;
    grid_totals<float>(a.pf + kp, nb, 3 * kp, 2 * kp, rg, tmpf);  // rn and gnew
    ++it;
    int trig = it >= a.max_inner;
    if ((int)threadIdx.x < kp && !frozen[threadIdx.x]) {
      const int c = threadIdx.x;
      its[c] = it;
      const float r = sqrtf(rn[c]);
      rn[c] = r;
      if (!(r == r)) {
        status[c] = COLAGB_SYS_NAN;
        frozen[c] = 1;
      } else if (r <= (float)a.inner_tol * rmax[c] || r <= (float)a.tol) {
        trig = 1;
      }
    }
    trig = __syncthreads_or(trig);
    const bool dpend = !trig;  // a replacement has already added this step's alpha p to x
    if (trig) {
      if (!replace(false)) return;
      ++nrep;
      if (it >= a.max_inner || nrep > a.max_sweeps) break;
    }
    // ---- C: beta, p = z + beta p ----
    for (int c = threadIdx.x; c < kp; c += kBT) {
      beta[c] = frozen[c] || gam[c] == 0.f ? 0.f : gnew[c] / gam[c];
      gam[c] = gnew[c];
    }
    __syncthreads();
    const float4 be = make_float4(beta[4 * cq], beta[4 * cq + 1], beta[4 * cq + 2], beta[4 * cq + 3]);
    for (int u = threadIdx.x; u < nu; u += 2 * kBT) {
      const int64_t e0 = r0 * q + u, e1 = u + kBT < nu ? e0 + kBT : e0;
      const float4 x0 = R4[u], x1 = R4[u + (int)(e1 - e0)], p0 = P4[e0], p1 = P4[e1];
      const float d0 = a.jacobi ? a.dinv[e0 >> qs] : 1.f, d1 = a.jacobi ? a.dinv[e1 >> qs] : 1.f;
      if (dpend) {
        float4 y0 = D4[e0], y1 = D4[e1];
        y0.x += al.x * p0.x; y0.y += al.y * p0.y; y0.z += al.z * p0.z; y0.w += al.w * p0.w;
        D4[e0] = y0;
        y1.x += al.x * p1.x; y1.y += al.y * p1.y; y1.z += al.z * p1.z; y1.w += al.w * p1.w;
        if (e1 != e0) D4[e1] = y1;
      }
      Pw4[e0] = make_float4(d0 * x0.x + be.x * p0.x, d0 * x0.y + be.y * p0.y, d0 * x0.z + be.z * p0.z, d0 * x0.w + be.w * p0.w);
      if (e1 != e0)
        Pw4[e1] = make_float4(d1 * x1.x + be.x * p1.x, d1 * x1.y + be.y * p1.y, d1 * x1.z + be.z * p1.z, d1 * x1.w + be.w * p1.w);
    }
    if (!grid_sync(a.gb)) return;
  }
  // ---- finish: x = (X64 + D) |b| into the (S, n) output ----
  for (int64_t u = threadIdx.x; u < (r1 - r0) * kp; u += kBT) {
    const int64_t i = r0 + u / kp;
    const int c = (int)(u % kp);
    if (c < a.S) a.X[(int64_t)c * n + i] = (a.X64[i * kp + c] + (double)a.D[i * kp + c]) * bnorm[c];
  }
  if (blockIdx.x == 0) {
    for (int c = threadIdx.x; c < a.S; c += kBT) {
      int st = status[c] == COLAGB_SYS_RUNNING ? COLAGB_SYS_MAX_ITERS : status[c];
      if (a.out_status) a.out_status[c] = st;
      if (a.out_iters) a.out_iters[c] = its[c];
      if (a.out_relres) a.out_relres[c] = relres[c];
    }
    if (threadIdx.x == 0 && a.out_nrep) *a.out_nrep = nrep;
  }
}

constexpr size_t kBlockRed = 2 * kBT * sizeof(float4), kBlockRows = 120 * 1024;

int block_padded_width(int64_t k) {
  int kp = 4;
  while (kp < k) kp *= 2;
  return kp;
}

size_t block_workspace_bytes(int64_t n, int64_t S, int nb_max) {
  const int64_t k = S < kBMaxK ? S : kBMaxK;
  const int kp = block_padded_width(k);
  Bump ws = Bump::measuring();
  ws.take<double>((size_t)(n * kp));      // Bn
  ws.take<double>((size_t)(n * kp));      // X64
  for (int v = 0; v < 4; ++v) ws.take<float>((size_t)(n * kp));
  ws.take<float>((size_t)n);               // dinv
  ws.take<float>((size_t)nb_max * 3 * kp);
  ws.take<double>((size_t)nb_max * 2 * kp);
  ws.take<unsigned int>(8);
  ws.take<int>(4);
  return ws.peak;
}

int block_grid_blocks() {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_block_ir, kBT, kBlockRed) != cudaSuccess || occ < 1) {
    cudaGetLastError();
    return 0;
  }
  return num_sms();
}

// One shared-matrix block of up to kBMaxK right-hand sides (B, X: (S, n) FP64).
int block_pcg_solve(const colagb_batched_csr* A, const double* B, double* X, const colagb_ir_params* prm,
                    int32_t* iters, int32_t* status, double* relres, void* ws_ptr, size_t ws_bytes, int* max_rep,
                    cudaStream_t st) {
  const int64_t n = A->n;
  for (int64_t s0 = 0; s0 < A->num_systems; s0 += kBMaxK) {
    const int S = (int)std::min<int64_t>(kBMaxK, A->num_systems - s0);
    const int kp = block_padded_width(S);
    const int nb = block_grid_blocks();
    if (nb < 1) return fail(COLAGB_ERR_UNSUPPORTED, "block schedule: kernel cannot be resident");
    Bump ws(ws_ptr, ws_bytes);
    BlockArgs a;
    a.n = n;
    a.kp = kp;
    a.q = kp / 4;
    a.S = S;
    a.indptr = A->indptr;
    a.indices = A->indices;
    a.vals = A->values;
    a.B = B + s0 * n;
    a.X = X + s0 * n;
    a.Bn = ws.take<double>((size_t)(n * kp));
    a.X64 = ws.take<double>((size_t)(n * kp));
    a.R = ws.take<float>((size_t)(n * kp));
    a.P = ws.take<float>((size_t)(n * kp));
    a.AP = ws.take<float>((size_t)(n * kp));
    a.D = ws.take<float>((size_t)(n * kp));
    float* dinv = ws.take<float>((size_t)n);
    a.pf = ws.take<float>((size_t)nb * 3 * kp);
    a.pd = ws.take<double>((size_t)nb * 2 * kp);
    unsigned int* bar = ws.take<unsigned int>(8);
    int* nrep = ws.take<int>(4);
    if (ws.overflow()) return fail(COLAGB_ERR_WORKSPACE, "block schedule: workspace too small");
    a.jacobi = prm->preconditioner == COLAGB_PREC_JACOBI ? 1 : 0;
    a.dinv = a.jacobi ? dinv : nullptr;
    a.out_status = status ? status + s0 : nullptr;
    a.out_iters = iters ? iters + s0 : nullptr;
    a.out_relres = relres ? relres + s0 : nullptr;
    a.out_nrep = nrep;
    a.tol = prm->tol;
    a.inner_tol = prm->inner_tol;
    a.max_inner = prm->max_inner_iters;
    a.max_sweeps = prm->max_sweeps;
    // r in shared memory where the rows' share is at most half of it: three of a step's vector streams less
    const size_t r_bytes = (size_t)ceil_div(n, (int64_t)nb) * kp * sizeof(float);
    a.r_resident = r_bytes <= kBlockRows;
    const size_t smem = kBlockRed + (a.r_resident ? r_bytes : 0);
    COLAGB_CUDA(set_smem_limit(k_block_ir, kBlockRed + kBlockRows));
    a.gb.arrivals = reinterpret_cast<unsigned long long*>(bar);
    a.gb.err = reinterpret_cast<int*>(bar + 2);
    a.gb.nblocks = (unsigned)nb;
    a.gb.spin_limit = prm->spin_limit > 0 ? prm->spin_limit : kDefaultSpinLimit;
    COLAGB_CUDA(cudaMemsetAsync(bar, 0, 8 * sizeof(unsigned int), st));
    void* args[] = {&a};
    COLAGB_CUDA(cudaLaunchCooperativeKernel((const void*)k_block_ir, dim3(nb), dim3(kBT), args, smem, st));
    int h[2] = {0, 0};
    COLAGB_CUDA(cudaMemcpyAsync(&h[0], bar + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaMemcpyAsync(&h[1], nrep, sizeof(int), cudaMemcpyDeviceToHost, st));
    COLAGB_CUDA(cudaStreamSynchronize(st));
    if (h[0] != 0) return fail(COLAGB_ERR_TIMEOUT, "block schedule: a grid barrier timed out");
    if (h[1] > *max_rep) *max_rep = h[1];
  }
  return COLAGB_OK;
}

}  // namespace colagb
