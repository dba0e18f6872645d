// h1free.cuh -- products with the first-order operator H1 and its transpose
// formed from the states instead of read from stored blocks.
//
// H1 is the linearised first-order Roe flux (roejac6.f on every edge,
// Edge.C:4503-4523) plus boundary-face blocks and I/dt.  With n the outward
// normal of an edge of row r, unit normal e, A(V, e) the Euler flux Jacobian
// and |A| the Roe dissipation at the average of the two states, the row is
//   (H1 p)_r = 1/vol_r sum_s |n|/2 [A(V_r, e) p_r + A(V_s, e) p_s + |A| (p_r - p_s)]
//              + (face blocks p_r) / vol_r + p_r / dt_r,
// the sum of A(V_r, e)|n|/2 over the row being A(V_r, m_r), m_r = sum n / 2
// (zero up to round-off where the dual cell is closed).  Both matrices act
// through two vectors: with u, H, c, un = u.e, a = e.q_m - un q_0, b =
// (gam - 1)(u^2/2 q_0 - u.q_m + q_4), R1 = (1, u, H), R2 = (0, e, un),
//   A q   = un q + a R1 + b R2,
//   |A| q = |un| q + (S1 b/c^2 + S2 a/c) R1 + (S1 a + S2 b/c) R2,
// S1 = (|un+c| + |un-c|)/2 - |un|, S2 = (|un+c| - |un-c|)/2 (the projection
// form of Liu and Vinokur, "Nonequilibrium flow computations", 1989).  So a
// block-vector product takes ~90 operations on 20 bytes per neighbour (unit
// normal, half length, local slot) plus the staged node records, against 25
// multiplications on a 100-byte FP32 (200-byte FP64) block: the stored
// product is bound by HBM at ~92 % of the copy rate, this one by latency and
// issue.  Twenty FP32 iterations of 81^3 take 3.45 ms, 4.93 with the stored
// blocks, and the Newton and linearised solves assemble the diagonal blocks
// only.
//
// With FP32 storage a neighbour's block-vector product is formed in FP32 from
// FP32 states, where the stored form multiplies FP32 blocks in FP64; both sum
// a row in FP64.  The stored blocks carry the rounding of their own formation
// in FP32, so this is no less accurate: over 72 systems (9^3 to 31^3, CFL 10
// to 1e4, both preconditioners and orientations) the solutions after twenty
// iterations are 9.8e-8 from the FP64 solver's in the mean against 11.2e-8
// with the stored blocks (0.63 to 1.03 times), and the step of 81^3 is 1.4e-7
// from the 64-bit one.
//
// CTA per Morton block of the blocked residual: the records (sqrt rho, u, H)
// and the vector p of the block's nodes and of all their neighbours are
// staged in shared memory (48-byte FP32 or 80-byte FP64 records: odd
// multiples of 16 bytes, conflict-free vector loads); L lanes per node take
// its neighbours r, r + L, ..., the row sum is FP64 (fixed xor tree).  The
// per-neighbour data is stored warp by warp, coalesced per step, and copied
// to shared memory four steps ahead, before the wait for the packed vector:
// requested one step ahead into registers, its latency was most of the kernel.
// Four steps and four CTAs per SM (64 registers): 41 us at 61^3, 28 warps
// active, an instruction issued in 56 % of the cycles, 4.4 of 12.6 warps
// waiting for global loads per issue.
#pragma once

#include "common.cuh"
#include "physics.cuh"

namespace aerof {

// widths (elements) of a node's record, global and staged, and the steps of
// neighbour data in flight per lane of the product kernel
template <class S> struct H1Rec;
template <> struct H1Rec<float> { static constexpr int W = 8, SM = 12, D = 4; };
template <> struct H1Rec<double> { static constexpr int W = 6, SM = 10, D = 4; };

// (sqrt rho, u, v, w, H) of every node, blocked numbering, from the caller's
// primitive records; and 1/dt (0 without time steps)
template <class S>
__global__ void k_h1_records(int N, Gas g, const int* __restrict__ n2o, const double* __restrict__ P,
                             const double* __restrict__ dt, S* __restrict__ rec, double* __restrict__ idt) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const size_t o = (size_t)n2o[n];
  double v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = P[8 * o + k];
  S* r = rec + (size_t)H1Rec<S>::W * n;
  r[0] = (S)sqrt(v[0]);
  r[1] = (S)v[1];
  r[2] = (S)v[2];
  r[3] = (S)v[3];
  r[4] = (S)(g.gam * g.invgam1 * v[4] / v[0] + 0.5 * (v[1] * v[1] + v[2] * v[2] + v[3] * v[3]));
#pragma unroll
  for (int k = 5; k < H1Rec<S>::W; ++k) r[k] = S(0);
  idt[n] = dt ? 1.0 / dt[o] : 0.0;
}

// Per-neighbour data of every node, in the order the product kernel reads
// it (warp w's step k, lane l at (wptr[w] + k) 32 + l): outward unit normal
// and half length, four values, and the neighbour's staged slot; entries
// past a node's list have zero length and its first neighbour's slot (with its
// own, the average at a node without pressure would be no number, and no
// length cancels that).  mrow[n]: (sum of n/2, 1/vol).  Thread per lane of the
// product kernel.
template <class S>
__global__ void k_h1_geometry(int N, int NB, int E, const int* __restrict__ n2o, const int* __restrict__ o2n,
                              const int* __restrict__ nbr_ptr, const int* __restrict__ nbr_node,
                              const int* __restrict__ nbr_edge, const double* __restrict__ en,
                              const int* __restrict__ hptr, const int* __restrict__ hnode,
                              const double* __restrict__ vol, const int* __restrict__ wptr, S* __restrict__ nrm,
                              int* __restrict__ slot, double* __restrict__ mrow) {
  const int blk = blockIdx.x, L = blockDim.x / NB;
  const int t = threadIdx.x / L, r = threadIdx.x % L;
  const int n0 = blk * NB, nn = min(NB, N - n0);
  const int gw = blk * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int w0 = wptr[gw], steps = wptr[gw + 1] - w0;
  const bool act = t < nn;
  const int o = act ? n2o[n0 + t] : 0;
  const int p0 = act ? nbr_ptr[o] : 0, deg = act ? nbr_ptr[o + 1] - p0 : 0;
  auto staged = [&](int e) {   // slot of neighbour e
    const int j = o2n[nbr_node[p0 + e]];
    if (j >= n0 && j < n0 + nn) return j - n0;
    int lo = hptr[blk], hi = hptr[blk + 1] - 1;   // ascending halo ids
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (hnode[mid] < j) lo = mid + 1;
      else hi = mid;
    }
    return nn + lo - hptr[blk];
  };
  for (int k = 0; k < steps; ++k) {
    const size_t at = ((size_t)w0 + k) * 32 + lane;
    const int e = r + k * L;
    double u[4] = {0.0, 0.0, 0.0, 0.0};
    const int sl = deg ? staged(e < deg ? e : 0) : (act ? t : 0);
    if (e < deg) {
      const int er = nbr_edge[p0 + e];
      const size_t l = (size_t)(er & 0x7fffffff);
      const double sg = er < 0 ? -1.0 : 1.0;
      const double a = sg * en[l], b = sg * en[(size_t)E + l], c = sg * en[2 * (size_t)E + l];
      const double len = sqrt(a * a + b * b + c * c);
      if (len >= 1e-18) {
        u[0] = a / len; u[1] = b / len; u[2] = c / len; u[3] = 0.5 * len;
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) nrm[4 * at + a] = (S)u[a];
    slot[at] = sl;
  }
  if (!act || r != 0) return;
  double m[3] = {0.0, 0.0, 0.0};
  for (int p = p0; p < p0 + deg; ++p) {
    const int er = nbr_edge[p];
    const size_t l = (size_t)(er & 0x7fffffff);
    const double sg = er < 0 ? -0.5 : 0.5;
#pragma unroll
    for (int a = 0; a < 3; ++a) m[a] += sg * en[(size_t)a * E + l];
  }
  double* mr = mrow + 4 * (size_t)(n0 + t);
  mr[0] = m[0]; mr[1] = m[1]; mr[2] = m[2]; mr[3] = 1.0 / vol[o];
}

// row o of a vector (caller numbering) into row o2n[o] of the packed blocked
// vector, scaled by 1/vol for the transposed product
template <class S>
__device__ __forceinline__ void h1_put(S* __restrict__ z, int n, double sc, const double* v) {
  S* r = z + (size_t)H1Rec<S>::W * n;
  if constexpr (sizeof(S) == 4) {
    float4* q = reinterpret_cast<float4*>(r);
    q[0] = make_float4((float)(sc * v[0]), (float)(sc * v[1]), (float)(sc * v[2]), (float)(sc * v[3]));
    q[1] = make_float4((float)(sc * v[4]), 0.f, 0.f, 0.f);
  } else {
    double2* q = reinterpret_cast<double2*>(r);
    q[0] = make_double2(sc * v[0], sc * v[1]);
    q[1] = make_double2(sc * v[2], sc * v[3]);
    q[2] = make_double2(sc * v[4], 0.0);
  }
}
// vectors x (system q: X.p[q], or X0 + q xs) packed without a preconditioner
template <class S, class TI>
__global__ void k_h1_pack(int N, const int* __restrict__ o2n, const double* __restrict__ vol, int tr,
                          const TI* x, size_t xs, S* z, size_t zs, const int* skip) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  pdl_trigger();
  pdl_wait();
  if (o >= N || (skip && skip[8 * q])) return;
  double v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = (double)x[(size_t)q * xs + 5 * (size_t)o + k];
  h1_put<S>(z + (size_t)q * zs, o2n[o], tr ? 1.0 / vol[o] : 1.0, v);
}

__device__ __forceinline__ float h1_rcp(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double h1_rcp(double x) { return rcp_(x); }
__device__ __forceinline__ float h1_rsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double h1_rsqrt(double x) { return rsqrt_(x); }
__device__ __forceinline__ float h1_abs(float x) { return fabsf(x); }
__device__ __forceinline__ double h1_abs(double x) { return fabs(x); }

// y = H1 z (TR: H1^T with z packed as p/vol), system blockIdx.y; y in the
// caller's numbering.  skip: flags, one per 8 ints.
template <class S, bool TR>
__global__ void __launch_bounds__(256, sizeof(S) == 4 ? 4 : 2)
    k_h1_apply(int N, int NB, Gas g, const int* __restrict__ n2o, const int* __restrict__ hptr,
               const int* __restrict__ hnode, const int* __restrict__ wptr, const S* __restrict__ nrm,
               const int* __restrict__ slot, const double* __restrict__ mrow,
               const S* __restrict__ rec, const double* __restrict__ idt, const int* __restrict__ brow,
               const double* __restrict__ fsum, const S* z, size_t zs, S* __restrict__ y, size_t ys, const int* skip) {
  extern __shared__ __align__(16) char raw[];
  const int q = blockIdx.y;
  pdl_trigger();
  constexpr int W = H1Rec<S>::W, SM = H1Rec<S>::SM, D = H1Rec<S>::D;
  // a ring of D steps of neighbour data per lane, then the staged nodes
  S* rn = reinterpret_cast<S*>(raw) + 4 * threadIdx.x;                         // step d: + 4 d blockDim.x
  int* rs = reinterpret_cast<int*>(raw + (size_t)4 * sizeof(S) * D * blockDim.x) + threadIdx.x;
  S* sm = reinterpret_cast<S*>(raw + (size_t)(4 * sizeof(S) + sizeof(int)) * D * blockDim.x);
  const int blk = blockIdx.x, L = blockDim.x / NB;
  const int n0 = blk * NB, nn = min(NB, N - n0);
  const int h0 = hptr[blk], ns = nn + hptr[blk + 1] - h0;
  const S* zq = z + (size_t)q * zs;
  const int t = threadIdx.x / L, r = threadIdx.x % L;
  const bool act = t < nn;
  const int gw = blk * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int w0 = wptr[gw], steps = wptr[gw + 1] - w0;
  const size_t at = (size_t)w0 * 32 + (threadIdx.x & 31);
  auto issue = [&](int k) {
    const int d = k % D * blockDim.x;
    cp_async16(rn + 4 * d, nrm + 4 * (at + 32 * (size_t)k));
    if constexpr (sizeof(S) == 8) cp_async16(rn + 4 * d + 2, nrm + 4 * (at + 32 * (size_t)k) + 2);
    cp_async4(rs + d, slot + at + 32 * (size_t)k);
  };
  // the neighbour data and the node records do not depend on the kernel
  // before (the one that packs z)
  for (int k = 0; k < min(D, steps); ++k) issue(k);
  for (int k = threadIdx.x; k < ns; k += blockDim.x) {
    const size_t j = (size_t)W * (k < nn ? n0 + k : hnode[h0 + k - nn]);
    S* d = sm + SM * k;
    cp_async16(d, rec + j);
    if constexpr (sizeof(S) == 4) {
      // state 0-3 | vector 0-3 | H, vector 4
      cp_async4(d + 8, rec + j + 4);
    } else {
      // state 0-3 | H, vector 4 | vector 0-3
      cp_async16(d + 2, rec + j + 2);
      cp_async8(d + 4, rec + j + 4);
    }
  }
  auto load = [&](int s, S* st, S* p) {
    const S* d = sm + SM * s;
    if constexpr (sizeof(S) == 4) {
      const float4* f = reinterpret_cast<const float4*>(d);
      const float4 a = f[0], b = f[1];
      const float2 c = reinterpret_cast<const float2*>(d + 8)[0];
      st[0] = a.x; st[1] = a.y; st[2] = a.z; st[3] = a.w; st[4] = c.x;
      p[0] = b.x; p[1] = b.y; p[2] = b.z; p[3] = b.w; p[4] = c.y;
    } else {
      const double2* f = reinterpret_cast<const double2*>(d);
      const double2 a = f[0], b = f[1], c = f[2], e = f[3], h = f[4];
      st[0] = a.x; st[1] = a.y; st[2] = b.x; st[3] = b.y; st[4] = c.x;
      p[0] = e.x; p[1] = e.y; p[2] = h.x; p[3] = h.y; p[4] = c.y;
    }
  };
  pdl_wait();
  if (skip && skip[8 * q]) {
    cp_async_wait_all();
    return;
  }
  for (int k = threadIdx.x; k < ns; k += blockDim.x) {
    const size_t j = (size_t)W * (k < nn ? n0 + k : hnode[h0 + k - nn]);
    S* d = sm + SM * k;
    if constexpr (sizeof(S) == 4) {
      cp_async16(d + 4, zq + j);
      cp_async4(d + 9, zq + j + 4);
    } else {
      cp_async8(d + 5, zq + j + 4);
      cp_async16(d + 6, zq + j);
      cp_async16(d + 8, zq + j + 2);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  const S gam1 = (S)g.gam1, half = (S)0.5;
  S sr[5], pr[5];
  load(act ? t : 0, sr, pr);
  const S qr = half * (sr[1] * sr[1] + sr[2] * sr[2] + sr[3] * sr[3]);
  double acc[5] = {0, 0, 0, 0, 0};
#pragma unroll 1
  for (int k = 0; k < steps; ++k) {
    // (a slot of the ring is refilled an iteration after it was read)
    if (steps > D && k > 0) {
      if (k - 1 + D < steps) issue(k - 1 + D);
      cp_async_commit();
      if (k >= D) cp_async_wait_group<D - 1>();
    }
    const int d = k % D * blockDim.x;
    const S* e = rn + 4 * d;
    S x0, x1, x2, hk;
    if constexpr (sizeof(S) == 4) {
      const float4 f = *reinterpret_cast<const float4*>(e);
      x0 = f.x; x1 = f.y; x2 = f.z; hk = f.w;
    } else {
      const double2 f = reinterpret_cast<const double2*>(e)[0], h = reinterpret_cast<const double2*>(e)[1];
      x0 = f.x; x1 = f.y; x2 = h.x; hk = h.y;
    }
    const int s = rs[d];
    S ss[5], ps[5];
    load(s, ss, ps);
    // Roe average
    const S rw = h1_rcp(sr[0] + ss[0]), ws = ss[0] * rw, wr = sr[0] * rw;
    const S u0 = wr * sr[1] + ws * ss[1], u1 = wr * sr[2] + ws * ss[2], u2 = wr * sr[3] + ws * ss[3];
    const S H = wr * sr[4] + ws * ss[4];
    const S qq = half * (u0 * u0 + u1 * u1 + u2 * u2);
    const S c2 = gam1 * (H - qq), ic = h1_rsqrt(c2), c = c2 * ic;
    const S un = u0 * x0 + u1 * x1 + u2 * x2;
    const S f1 = h1_abs(un), fp = h1_abs(un + c), fm = h1_abs(un - c);
    const S S1 = half * (fp + fm) - f1, S2 = half * (fp - fm);
    const S d0 = pr[0] - ps[0], d1 = pr[1] - ps[1], d2 = pr[2] - ps[2], d3 = pr[3] - ps[3], d4 = pr[4] - ps[4];
    S v0, v1, v2, v3, v4;
    if (!TR) {
      const S al = x0 * d1 + x1 * d2 + x2 * d3 - un * d0;
      const S be = gam1 * (qq * d0 - u0 * d1 - u1 * d2 - u2 * d3 + d4) * ic;   // b / c
      const S k1 = (S1 * be + S2 * al) * ic, k2 = S1 * al + S2 * be;
      // A(V_s, e) p_s
      const S us = ss[1] * x0 + ss[2] * x1 + ss[3] * x2;
      const S qs = half * (ss[1] * ss[1] + ss[2] * ss[2] + ss[3] * ss[3]);
      const S as = x0 * ps[1] + x1 * ps[2] + x2 * ps[3] - us * ps[0];
      const S bs = gam1 * (qs * ps[0] - ss[1] * ps[1] - ss[2] * ps[2] - ss[3] * ps[3] + ps[4]);
      const S kb = k2 + bs;
      v0 = f1 * d0 + k1 + us * ps[0] + as;
      v1 = f1 * d1 + k1 * u0 + kb * x0 + us * ps[1] + as * ss[1];
      v2 = f1 * d2 + k1 * u1 + kb * x1 + us * ps[2] + as * ss[2];
      v3 = f1 * d3 + k1 * u2 + kb * x2 + us * ps[3] + as * ss[3];
      v4 = f1 * d4 + k1 * H + k2 * un + us * ps[4] + as * ss[4] + bs * us;
    } else {
      // d = q_r - q_s: |A|^T d + A(V_r, e)^T d
      const S r1 = (d0 + u0 * d1 + u1 * d2 + u2 * d3 + H * d4) * ic;            // R1.d / c
      const S r2 = x0 * d1 + x1 * d2 + x2 * d3 + un * d4;
      const S ka = S1 * r2 + S2 * r1, kb = gam1 * (S1 * r1 + S2 * r2) * ic;
      const S ur = sr[1] * x0 + sr[2] * x1 + sr[3] * x2;
      const S ra = d0 + sr[1] * d1 + sr[2] * d2 + sr[3] * d3 + sr[4] * d4;
      const S rb = gam1 * (x0 * d1 + x1 * d2 + x2 * d3 + ur * d4);
      const S fu = f1 + ur, kr = ka + ra;
      v0 = fu * d0 - un * ka - ur * ra + kb * qq + rb * qr;
      v1 = fu * d1 + kr * x0 - kb * u0 - rb * sr[1];
      v2 = fu * d2 + kr * x1 - kb * u1 - rb * sr[2];
      v3 = fu * d3 + kr * x2 - kb * u2 - rb * sr[3];
      v4 = fu * d4 + kb + rb;
    }
    const double hd = (double)hk;
    acc[0] += hd * (double)v0;
    acc[1] += hd * (double)v1;
    acc[2] += hd * (double)v2;
    acc[3] += hd * (double)v3;
    acc[4] += hd * (double)v4;
  }
  for (int o = 1; o < L; o <<= 1) {
#pragma unroll
    for (int k = 0; k < 5; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  }
  if (!act || r != 0) return;
  const int n = n0 + t;
  const size_t o = (size_t)n2o[n];
  const double2* mr = reinterpret_cast<const double2*>(mrow + 4 * (size_t)n);
  const double2 ma = mr[0], mb = mr[1];
  const double p0 = pr[0], p1 = pr[1], p2 = pr[2], p3 = pr[3], p4 = pr[4];
  const int br = brow[o];
  if (!TR) {
    // the row's own A(V_r, m) p_r
    const double a = sr[1], b = sr[2], cc = sr[3];
    const double um = a * ma.x + b * ma.y + cc * mb.x;
    const double am = ma.x * p1 + ma.y * p2 + mb.x * p3 - um * p0;
    const double bm = g.gam1 * (0.5 * (a * a + b * b + cc * cc) * p0 - a * p1 - b * p2 - cc * p3 + p4);
    acc[0] += um * p0 + am;
    acc[1] += um * p1 + am * a + bm * ma.x;
    acc[2] += um * p2 + am * b + bm * ma.y;
    acc[3] += um * p3 + am * cc + bm * mb.x;
    acc[4] += um * p4 + am * (double)sr[4] + bm * um;
  }
  if (br >= 0) {
    const double* f = fsum + 25 * (size_t)br;
    const double pv[5] = {p0, p1, p2, p3, p4};
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) acc[a] += f[TR ? 5 * b + a : 5 * a + b] * pv[b];
  }
  const double it = idt[n];
  S* yo = y + (size_t)q * ys + 5 * o;
  // the transposed product's vector is p/vol
  const double sc = TR ? 1.0 : mb.y, si = TR ? it / mb.y : it;
  yo[0] = (S)(acc[0] * sc + si * p0);
  yo[1] = (S)(acc[1] * sc + si * p1);
  yo[2] = (S)(acc[2] * sc + si * p2);
  yo[3] = (S)(acc[3] * sc + si * p3);
  yo[4] = (S)(acc[4] * sc + si * p4);
}

__device__ __forceinline__ void load5(const double* __restrict__ P, int j, double* v) {
  const double2* q = reinterpret_cast<const double2*>(P + 8 * (size_t)j);
  const double2 a = q[0], b = q[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  v[4] = P[8 * (size_t)j + 4];
}

// Diagonal entries that cancelled to exactly zero, of contributions whose
// identity parts add up to size: round-off of that size instead.  The
// reference's eigenvector products leave some there (the first entry of |A| on
// supersonic edges), and block-Jacobi leaves a block with a zero on its
// diagonal uninverted (DiagMatrix.C:44-80); a fluid at rest has no such
// contributions and keeps its zero.  T: stride of the block's elements.
template <int T>
__device__ __forceinline__ void keep_nonzero(double* a, double size) {
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if (a[T * 6 * k] == 0.0 && size > 0.0) a[T * 6 * k] = 0x1p-54 * size;
}

// Diagonal blocks of H1 alone (what block-Jacobi needs), in FP64 from the
// caller's records: thread per row, sum over its edges of |A||n|/2 (the two
// rank-one terms and |un| I), A(V_r, m_r), the face blocks, 1/vol, I/dt.
template <class S, bool TR>
__global__ void __launch_bounds__(128) k_h1_diag(int N, int E, Gas g, const int* __restrict__ nbr_ptr,
                                                 const int* __restrict__ nbr_node, const int* __restrict__ nbr_edge,
                                                 const double* __restrict__ en, const double* __restrict__ P,
                                                 const double* __restrict__ vol, const int* __restrict__ brow,
                                                 const double* __restrict__ fsum, const double* __restrict__ dt,
                                                 S* __restrict__ diag) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  double Vr[5], a[25], m[3] = {0.0, 0.0, 0.0};
  load5(P, r, Vr);
#pragma unroll
  for (int k = 0; k < 25; ++k) a[k] = 0.0;
  // + w I + R1 (x) p + R2 (x) t with R1 = (1, u, H), R2 = (0, n, un)
  double size = 0.0;   // sum of |w|, see keep_nonzero
  auto rank = [&](double w, const double* u, double H, const double* n, double un, const double* p, const double* t) {
    size += fabs(w);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      a[c] += p[c];
#pragma unroll
      for (int k = 0; k < 3; ++k) a[5 * (k + 1) + c] += u[k] * p[c] + n[k] * t[c];
      a[20 + c] += H * p[c] + un * t[c];
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) a[6 * c] += w;
  };
  const double sr = sqrt(Vr[0]);
  const double Hr = g.gam * g.invgam1 * Vr[4] / Vr[0] + 0.5 * (Vr[1] * Vr[1] + Vr[2] * Vr[2] + Vr[3] * Vr[3]);
  for (int p = nbr_ptr[r]; p < nbr_ptr[r + 1]; ++p) {
    const int er = nbr_edge[p];
    const size_t e = (size_t)(er & 0x7fffffff);
    const double sg = er < 0 ? -1.0 : 1.0;
    const double n0 = sg * en[e], n1 = sg * en[(size_t)E + e], n2 = sg * en[2 * (size_t)E + e];
    double Vs[5];
    load5(P, nbr_node[p], Vs);
    m[0] += 0.5 * n0; m[1] += 0.5 * n1; m[2] += 0.5 * n2;
    const double l2 = n0 * n0 + n1 * n1 + n2 * n2;
    if (l2 < 1e-36) continue;
    const double il = rsqrt_(l2), h = 0.5 * (l2 * il);
    const double n[3] = {n0 * il, n1 * il, n2 * il};
    const double is = rsqrt_(Vs[0]), ss = Vs[0] * is;
    const double Hs = g.gam * g.invgam1 * Vs[4] * (is * is) + 0.5 * (Vs[1] * Vs[1] + Vs[2] * Vs[2] + Vs[3] * Vs[3]);
    const double rw = rcp_(sr + ss), wr = sr * rw, ws = ss * rw;
    const double u[3] = {wr * Vr[1] + ws * Vs[1], wr * Vr[2] + ws * Vs[2], wr * Vr[3] + ws * Vs[3]};
    const double H = wr * Hr + ws * Hs;
    const double q = 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    const double c2 = g.gam1 * (H - q), ic = rsqrt_(c2), c = c2 * ic;
    const double un = u[0] * n[0] + u[1] * n[1] + u[2] * n[2];
    const double f1 = fabs(un), fp = fabs(un + c), fm = fabs(un - c);
    const double S1 = h * (0.5 * (fp + fm) - f1), S2 = h * (0.5 * (fp - fm)) * ic;
    const double kb = g.gam1 * S1 * (ic * ic), tb = g.gam1 * S2;
    const double al[5] = {-un, n[0], n[1], n[2], 0.0}, be[5] = {q, -u[0], -u[1], -u[2], 1.0};
    double pv[5], tv[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      pv[k] = kb * be[k] + S2 * al[k];
      tv[k] = S1 * al[k] + tb * be[k];
    }
    rank(h * f1, u, H, n, un, pv, tv);
  }
  {
    const double u[3] = {Vr[1], Vr[2], Vr[3]};
    const double um = u[0] * m[0] + u[1] * m[1] + u[2] * m[2];
    const double q = 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    const double al[5] = {-um, m[0], m[1], m[2], 0.0};
    const double be[5] = {g.gam1 * q, -g.gam1 * u[0], -g.gam1 * u[1], -g.gam1 * u[2], g.gam1};
    rank(um, u, Hr, m, um, al, be);
  }
  const int br = brow[r];
  if (br >= 0) {
#pragma unroll
    for (int k = 0; k < 25; ++k) a[k] += fsum[25 * (size_t)br + k];
  }
  const double iv = 1.0 / vol[r], it = dt ? 1.0 / dt[r] : 0.0;
  keep_nonzero<1>(a, size);
#pragma unroll
  for (int k = 0; k < 25; ++k) a[k] = a[k] * iv + (k % 6 == 0 ? it : 0.0);
  store_diag<S, TR>(diag, r, a);
}

}  // namespace aerof
