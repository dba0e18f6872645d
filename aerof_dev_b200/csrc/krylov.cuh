// krylov.cuh -- Gram-Schmidt kernels of the device-driven GMRES
// (GmresSolver::solve, KspSolver.C:396-449, with applyPreviousRotations /
// applyNewRotation / backwardSolve, KspSolver.C:917-982) for R systems that
// run together (grid.y = system).
//
// The coefficients of modified Gram-Schmidt, h_0 = v_0.w, h_1 = v_1.(w -
// h_0 v_0), ..., satisfy (I + L) h = V^T w with L the strictly lower part of
// V^T V: one sweep over the basis gives every v_i.w and the new row v_j.v_k
// of L, a triangular solve gives h, and a second sweep forms w - V h
// (Swirydowicz, Langou, Ananthan, Yang, Thomas, "Low synchronization
// Gram-Schmidt and GMRES algorithms", 2021: the same projector as MGS).
// Two reads of the basis per iteration and two launches, instead of two
// reads of the basis, j reads and writes of w and j + 1 grid-wide sums
// (bound: HBM; figures at gs_iteration).
//
// The first basis vector of a cycle is stored normalised, so that the vectors
// do not depend on the scale of the right-hand side.  The others are stored
// as they come out of the projection, of the size of the preconditioned
// operator, with the factor sig_i = 1/norm beside them (v_i = sig_i *
// stored), so no pass normalises them.  The flexible method hands its vectors
// to inner solves and does normalise them (k_gs_unit, sig_i = 1).  Dots, norms
// and the Hessenberg system are FP64 for either storage type; a vector is
// rounded to it once.
// Reductions run over a fixed grid in a fixed order (no atomics on values):
// every block of the second sweep forms the coefficients from the first
// sweep's partial sums, and its block that finishes last does the Givens
// update.  The launches of an iteration overlap (launch_pdl).
#pragma once

#include "common.cuh"

namespace aerof {

constexpr int kGsT = 512;        // threads of the sweeps
constexpr int kGsL = 4000;       // doubles of L kept in shared memory by the triangular solve
constexpr int kGsMax = 7199;     // longest restart whose coefficients fit in shared memory (200 KB)
constexpr int kMaxSys = 64;      // systems per launch

// what the host reads while the cycle runs (page-locked, mapped)
struct GsPub {
  int seq;                       // iterations finished in this cycle
  int done, iter, pad;
  double l2res;
};

// Device state of the systems: system q's block of doubles at d + q sd,
// its integers at i + 8 q: [0] iterations, [1] done, [2] last column,
// [3] active in this cycle, [4] maxits, [5] breakdown, [6] [7] tickets.
struct GsDev {
  double* d;
  size_t sd;
  int* i;
  double* part;                  // [R][2 (m + 1)][G] partial sums of the dot products
  double* norm_part;             // [R][G] of the norm
  GsPub* pub;
  double* scratch;               // m > kGsMax: [R][G][3 (m + 1)] for the coefficients, else null
  int m, G;
  bool unit;                     // every basis vector is stored normalised (k_gs_unit)
  __host__ __device__ size_t oL() const { return (size_t)(m + 1) * m; }
  __host__ __device__ size_t oCs() const { return oL() + (size_t)m * m; }
  __host__ __device__ size_t oG() const { return oCs() + 2 * (size_t)m; }
  __host__ __device__ size_t oY() const { return oG() + m + 1; }
  __host__ __device__ size_t oSig() const { return oY() + m; }
  // l2res, target, 1/norm of the vector to be normalised
  __host__ __device__ size_t oScal() const { return oSig() + m + 1; }
  __host__ __device__ size_t size() const { return oScal() + 3; }
};

struct VecIn { const double* p[kMaxSys]; };
struct VecOut { double* p[kMaxSys]; };

template <class TV> struct Vec16;
template <> struct Vec16<float> { using T = float4; static constexpr int W = 4; };
template <> struct Vec16<double> { using T = double2; static constexpr int W = 2; };

// sum of C values over the block's warps (xor tree, then the warps in
// order): result v of the block at out[v * stride] by thread v
template <int C>
__device__ __forceinline__ void block_sums(const double* v, int nv, double* red, double* out, size_t stride) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if (c >= nv) break;
    double t = v[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) red[warp * C + c] = t;
  }
  __syncthreads();
  if ((int)threadIdx.x < nv) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[w * C + threadIdx.x];
    out[threadIdx.x * stride] = t;
  }
}

// true in every thread of the block that arrives last; the partial sums of
// the others are then visible (the ticket re-arms itself)
__device__ __forceinline__ bool last_block(int* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    if (last) *ticket = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// vals[v] = sum of part[v][0, G) for v < nv, LG lanes per value with eight
// loads in flight each (G is at most a few hundred): a warp for one or two
// values, eight lanes for the dot products, so that up to 64 of them are
// summed side by side
template <int LG>
__device__ __forceinline__ void sum_partials(const double* part, int G, int nv, double* vals) {
  const int lane = threadIdx.x % LG, ng = blockDim.x / LG;
  for (int v0 = 0; v0 < nv; v0 += ng) {   // the same trips in every thread
    const int v = v0 + (int)threadIdx.x / LG;
    const double* p = part + (size_t)v * G;
    double t = 0.0;
    if (v < nv) {
      for (int k0 = lane; k0 < G; k0 += 8 * LG) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = k0 + LG * u < G ? __ldcg(p + k0 + LG * u) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) t += x[u];
      }
    }
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0 && v < nv) vals[v] = t;
  }
  __syncthreads();
}

// The sums of 16 values over a warp's lanes: the lanes exchange halves, so
// that 16 shuffles do what a tree per value does in 80; lane l returns the
// total of value l / 2.
__device__ __forceinline__ double warp_sums16(const double* s) {
  const int lane = threadIdx.x & 31;
  double a[8], b[4], c[2];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double keep = lane & 16 ? s[8 + k] : s[k], give = lane & 16 ? s[k] : s[8 + k];
    a[k] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double keep = lane & 8 ? a[4 + k] : a[k], give = lane & 8 ? a[k] : a[4 + k];
    b[k] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double keep = lane & 4 ? b[2 + k] : b[k], give = lane & 4 ? b[k] : b[2 + k];
    c[k] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
  }
  const double keep = lane & 2 ? c[1] : c[0], give = lane & 2 ? c[0] : c[1];
  double d = keep + __shfl_xor_sync(0xffffffffu, give, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  return d;
}

__device__ __forceinline__ void publish(GsPub* pub, int seq, int done, int iter, double l2res) {
  volatile GsPub* p = pub;
  p->done = done;
  p->iter = iter;
  p->l2res = l2res;
  __threadfence_system();
  p->seq = seq;
}

// Start of a cycle: the norm of b (FIRST, which also zeroes x) or of b - w,
// b's for the target, and the cycle's state.  The vector itself is left to
// k_gs_first: rounded to TV before it is normalised, a right-hand side far
// from 1 would lose its range.
template <class TV, bool FIRST>
__global__ void __launch_bounds__(kGsT) k_gs_start(size_t n, VecIn B, VecOut X, const TV* __restrict__ Wv, size_t ws,
                                                   GsDev st, double eps, int maxits) {
  __shared__ double red[kGsT / 32];
  __shared__ double vals[1];
  const int q = blockIdx.y;
  int* ist = st.i + 8 * q;
  if (!FIRST && ist[1]) {
    // done in an earlier cycle: its words stand
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ist[3] = 0;
      publish(st.pub + q, 0, 1, ist[0], st.d[(size_t)q * st.sd + st.oScal()]);
    }
    return;
  }
  const double* __restrict__ b = B.p[q];
  const TV* __restrict__ w = Wv + (size_t)q * ws;
  double s = 0.0;
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const double r = FIRST ? b[p] : b[p] - (double)w[p];
    if (FIRST) X.p[q][p] = 0.0;
    s += r * r;
  }
  double* part = st.part + (size_t)q * 2 * (st.m + 1) * st.G;
  block_sums<1>(&s, 1, red, part + blockIdx.x, st.G);
  if (!last_block(ist + 6)) return;
  sum_partials<32>(part, st.G, 1, vals);
  if (threadIdx.x == 0) {
    double* d = st.d + (size_t)q * st.sd;
    const double beta = sqrt(vals[0]);
    if (FIRST) {
      ist[0] = 0;
      ist[4] = maxits;
      d[st.oScal()] = 0.0;
      d[st.oScal() + 1] = eps * beta;
    }
    const int done = beta == 0.0;
    if (done) d[st.oScal()] = 0.0;
    ist[1] = done;
    ist[2] = -1;
    ist[3] = 1;
    ist[5] = 0;
    d[st.oG()] = beta;
    d[st.oSig()] = 1.0;
    d[st.oScal() + 2] = done ? 0.0 : 1.0 / beta;
    if (done) publish(st.pub + q, 0, 1, ist[0], 0.0);
  }
}
// v_0 = (b or b - w) / its norm, rounded once
template <class TV, bool FIRST>
__global__ void __launch_bounds__(256) k_gs_first(size_t n, VecIn B, const TV* __restrict__ Wv, size_t ws,
                                                  TV* __restrict__ V, size_t vs, GsDev st) {
  const int q = blockIdx.y;
  if (st.i[8 * q + 1]) return;
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double b = B.p[q][p], r = FIRST ? b : b - (double)Wv[(size_t)q * ws + p];
  // (a norm beyond FP64 has the reciprocal 0: FP32 vectors are then not a
  // number, as the right-hand side is infinite in FP32, and so is the result)
  const double sc = st.d[(size_t)q * st.sd + st.oScal() + 2];
  V[(size_t)q * vs + p] = sc != 0.0 ? (TV)(sc * r) : (TV)r * TV(0);
}
// basis vector v of the running systems normalised (flexible method)
template <class TV>
__global__ void __launch_bounds__(256) k_gs_unit(size_t n, TV* __restrict__ v, size_t vs, GsDev st) {
  const int q = blockIdx.y;
  if (st.i[8 * q + 1]) return;
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) v[(size_t)q * vs + p] *= (TV)st.d[(size_t)q * st.sd + st.oScal() + 2];
}

// Sweep 1 of iteration j: partial sums of v_i.w and v_i.v_j for every i <= j
// (eight basis vectors per pass over w and v_j, so that a thread has ten
// 16-byte loads in flight).  Their totals and the coefficients are formed by
// every block of sweep 2: a last block that did it here put its fences, its
// reads and the solve in series between the sweeps (~10 us per iteration).
template <class TV>
__global__ void __launch_bounds__(kGsT, 1) k_gs_dots(size_t n, int j, const TV* V, size_t vs, size_t ld,
                                                     const TV* W, size_t ws, GsDev st) {
  constexpr int PB = 8;            // passes whose warp sums wait for one addition over the warps
  __shared__ double red[kGsT / 32][16 * PB];
  const int q = blockIdx.y;
  pdl_trigger();
  pdl_wait();
  if (st.i[8 * q + 1]) return;
  using VT = typename Vec16<TV>::T;
  constexpr int E = Vec16<TV>::W, U = 8;
  const TV* Vq = V + (size_t)q * vs;
  const TV* w = W + (size_t)q * ws;
  const TV* vj = Vq + (size_t)j * ld;
  double* part = st.part + (size_t)q * 2 * (st.m + 1) * st.G;
  const size_t nv = n / E, t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (int i0 = 0; i0 <= j; i0 += U) {
    const int c = min(U, j + 1 - i0);
    const TV* Vi = Vq + (size_t)i0 * ld;
    double s[2 * U];
#pragma unroll
    for (int u = 0; u < 2 * U; ++u) s[u] = 0.0;
    for (size_t p = t0; p < nv; p += stride) {
      const VT wv = reinterpret_cast<const VT*>(w)[p], jv = reinterpret_cast<const VT*>(vj)[p];
      VT x[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < c) x[u] = reinterpret_cast<const VT*>(Vi + (size_t)u * ld)[p];
      const TV* wp = reinterpret_cast<const TV*>(&wv);
      const TV* jp = reinterpret_cast<const TV*>(&jv);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < c) {
          const TV* xp = reinterpret_cast<const TV*>(&x[u]);
#pragma unroll
          for (int k = 0; k < E; ++k) {
            s[2 * u] += (double)wp[k] * (double)xp[k];
            s[2 * u + 1] += (double)jp[k] * (double)xp[k];
          }
        }
    }
    for (size_t p = nv * E + t0; p < n; p += stride) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < c) {
          const double x = (double)Vi[(size_t)u * ld + p];
          s[2 * u] += (double)w[p] * x;
          s[2 * u + 1] += (double)vj[p] * x;
        }
    }
    const int at = 2 * (i0 % (U * PB));
    const double t = warp_sums16(s);
    if (!(threadIdx.x & 1)) red[threadIdx.x >> 5][at + ((threadIdx.x & 31) >> 1)] = t;
    if (i0 + U > j || at + 2 * U == 16 * PB) {
      __syncthreads();
      const int first = 2 * i0 - at;   // value of the buffer's first column
      for (int v = threadIdx.x; v < at + 2 * c; v += blockDim.x) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < kGsT / 32; ++w) x += red[w][v];
        part[(size_t)(first + v) * st.G + blockIdx.x] = x;
      }
      __syncthreads();
    }
  }
}

// The coefficients of iteration j in a[0..j] (shared memory), from the
// partial sums: the block computes them whole, so every block has the same
// ones without a grid-wide step.  Block 0 keeps row j of L.  vals
// [3 (m + 1)]: the sums, then the coefficients; sL: L (packed rows 1..j while
// they fit).
__device__ __forceinline__ double* gs_coefficients(const GsDev& st, int q, int j, double* vals, double* sL) {
  double* a = vals + 2 * (st.m + 1);
  double* d = st.d + (size_t)q * st.sd;
  double* L = d + st.oL();
  const double* sig = d + st.oSig();
  const bool cached = j * (j + 1) / 2 <= kGsL;
  const double sj = sig[j];
  if (cached)
    for (int i = 1 + (int)(threadIdx.x >> 5); i < j; i += blockDim.x >> 5)
      for (int k = threadIdx.x & 31; k < i; k += 32) sL[i * (i - 1) / 2 + k] = L[(size_t)i * st.m + k];
  sum_partials<8>(st.part + (size_t)q * 2 * (st.m + 1) * st.G, st.G, 2 * (j + 1), vals);
  for (int k = threadIdx.x; k <= j; k += blockDim.x) {
    const double sk = sig[k];
    a[k] = sj * sk * vals[2 * k];
    if (k < j) {
      const double l = sj * sk * vals[2 * k + 1];
      vals[2 * k + 1] = l;
      if (blockIdx.x == 0) L[(size_t)j * st.m + k] = l;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    for (int k = 0; k < j; ++k) {
      const double hk = a[k];
      for (int i = k + 1 + (int)threadIdx.x; i <= j; i += 32)
        a[i] -= (i == j ? vals[2 * k + 1] : (cached ? sL[i * (i - 1) / 2 + k] : L[(size_t)i * st.m + k])) * hk;
      __syncwarp();
    }
  }
  __syncthreads();
  return a;
}

// Sweep 2 of iteration j: v_{j+1} = w - sum_i h_i v_i (FP64 per element,
// rounded once) and its norm; then the Givens update of the Hessenberg
// column, written with explicitly rounded operations (the host loop's
// arithmetic), and the step's result for the host.
// BIG: the coefficients in global memory (m > kGsMax).  A kernel of its own:
// chosen at run time, the pointer made the inner loop's coefficient loads
// generic ones, 1.8 us per iteration of 61^3.
template <class TV, bool BIG>
__global__ void __launch_bounds__(kGsT, 1) k_gs_update(size_t n, int j, TV* V, size_t vs, size_t ld,
                                                       const TV* W, size_t ws, GsDev st) {
  extern __shared__ double smem[];   // see gs_coefficients
  __shared__ double red[kGsT / 32];
  __shared__ double nrm[1];
  const int q = blockIdx.y;
  int* ist = st.i + 8 * q;
  pdl_trigger();
  pdl_wait();
  if (ist[1]) return;
  using VT = typename Vec16<TV>::T;
  constexpr int E = Vec16<TV>::W, U = 8;
  double* d = st.d + (size_t)q * st.sd;
  const double* sig = d + st.oSig();
  const double sj = sig[j];
  const size_t len = 3 * ((size_t)st.m + 1);
  double* sh = BIG ? st.scratch + ((size_t)q * gridDim.x + blockIdx.x) * len : smem;
  const double* hcol = gs_coefficients(st, q, j, sh, BIG ? smem : smem + len);
  double* cf = sh;                 // h_i sig_i, over the finished sums
  for (int k = threadIdx.x; k <= j; k += blockDim.x) cf[k] = hcol[k] * sig[k];
  __syncthreads();
  const TV* Vq = V + (size_t)q * vs;
  const TV* w = W + (size_t)q * ws;
  TV* vn = V + (size_t)q * vs + (size_t)(j + 1) * ld;
  const size_t nv = n / E, t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  double s = 0.0;
  for (size_t p = t0; p < nv; p += stride) {
    VT wv = reinterpret_cast<const VT*>(w)[p];
    TV* wp = reinterpret_cast<TV*>(&wv);
    double acc[E];
#pragma unroll
    for (int k = 0; k < E; ++k) acc[k] = sj * (double)wp[k];
    for (int i0 = 0; i0 <= j; i0 += U) {
      const int c = min(U, j + 1 - i0);
      const TV* Vi = Vq + (size_t)i0 * ld;
      VT x[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < c) x[u] = reinterpret_cast<const VT*>(Vi + (size_t)u * ld)[p];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < c) {
          const TV* xp = reinterpret_cast<const TV*>(&x[u]);
          const double h = cf[i0 + u];
#pragma unroll
          for (int k = 0; k < E; ++k) acc[k] -= h * (double)xp[k];
        }
    }
#pragma unroll
    for (int k = 0; k < E; ++k) {
      wp[k] = (TV)acc[k];
      s += (double)wp[k] * (double)wp[k];
    }
    reinterpret_cast<VT*>(vn)[p] = wv;
  }
  for (size_t p = nv * E + t0; p < n; p += stride) {
    double acc = sj * (double)w[p];
    for (int i = 0; i <= j; ++i) acc -= cf[i] * (double)Vq[(size_t)i * ld + p];
    const TV r = (TV)acc;
    vn[p] = r;
    s += (double)r * (double)r;
  }
  // (not over the dot products' partials, which other blocks may still read)
  double* part = st.norm_part + (size_t)q * st.G;
  block_sums<1>(&s, 1, red, part + blockIdx.x, st.G);
  if (!last_block(ist + 7)) return;
  sum_partials<32>(part, st.G, 1, nrm);
  // the rotations and the state in shared memory before the serial part
  double* cs = d + st.oCs();
  double* g = d + st.oG();
  double* H = d;
  const int m = st.m;
  double* scs = sh;                // [2 j], over the coefficients
  double* col = const_cast<double*>(hcol);
  for (int k = threadIdx.x; k < 2 * j; k += blockDim.x) scs[k] = cs[k];
  __shared__ double sg[3];
  __shared__ int si[2];
  if (threadIdx.x == 0) {
    sg[0] = g[j];
    sg[1] = d[st.oScal()];
    sg[2] = d[st.oScal() + 1];
    si[0] = ist[0];
    si[1] = ist[4];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double hj1 = __dsqrt_rn(nrm[0]);
    const bool breakdown = hj1 == 0.0;
    double cur = col[0];
    for (int i = 0; i < j; ++i) {
      const double c0 = scs[2 * i], c1 = scs[2 * i + 1];
      const double a = cur, bb = col[i + 1];
      col[i] = __dadd_rn(__dmul_rn(c1, a), __dmul_rn(c0, bb));
      cur = __dadd_rn(__dmul_rn(-c0, a), __dmul_rn(c1, bb));
    }
    double c0, c1;
    if (__dmul_rn(cur, cur) == 0.0) {
      c1 = 0.0;
      c0 = 1.0;
    } else {
      const double coef = __ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__dmul_rn(cur, cur), __dmul_rn(hj1, hj1))));
      c1 = __dmul_rn(__dsqrt_rn(__dmul_rn(cur, cur)), coef);
      c0 = __ddiv_rn(__dmul_rn(c1, hj1), cur);
    }
    col[j] = __dadd_rn(__dmul_rn(c1, cur), __dmul_rn(c0, hj1));
    H[(size_t)(j + 1) * m + j] = 0.0;
    const double gj = sg[0], gj1 = __dmul_rn(-c0, gj);
    g[j + 1] = gj1;
    g[j] = __dmul_rn(c1, gj);
    cs[2 * j] = c0;
    cs[2 * j + 1] = c1;
    const double inv = breakdown ? 0.0 : 1.0 / hj1;
    d[st.oSig() + j + 1] = st.unit ? 1.0 : inv;
    d[st.oScal() + 2] = inv;
    const int iter = si[0] + 1;
    double l2res = sg[1];
    bool done = breakdown;
    if (!breakdown) {
      l2res = fabs(gj1);
      done = l2res <= sg[2] || iter >= si[1];
    }
    d[st.oScal()] = l2res;
    ist[0] = iter;
    ist[2] = j;
    ist[5] = breakdown;
    ist[1] = done;
    publish(st.pub + q, j + 1, done, iter, l2res);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= j; i += blockDim.x) H[(size_t)i * m + j] = col[i];
}

// back substitution (KspSolver.C:966-982) of the cycle, one block per
// system: y from the rotated Hessenberg matrix (staged, row by row of the
// upper triangle) and g; lane i subtracts column k's product as y_k is known
template <bool BIG>
__global__ void __launch_bounds__(256) k_gs_backsolve(GsDev st) {
  extern __shared__ double sh[];   // g [m] (BIG: in y itself), H (packed columns while they fit)
  const int q = blockIdx.x;
  const int* ist = st.i + 8 * q;
  if (!ist[3]) return;
  double* d = st.d + (size_t)q * st.sd;
  const double *H = d, *g = d + st.oG();
  double* y = d + st.oY();
  const int j = ist[2], n = j + 1;
  double *sy = BIG ? y : sh, *sH = BIG ? sh : sh + st.m;
  const bool cached = n * (n + 1) / 2 <= kGsL;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sy[i] = g[i];
  if (cached)
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, k = e - n * i;
      if (i <= k) sH[k * (k + 1) / 2 + i] = H[(size_t)i * st.m + k];
    }
  __syncthreads();
  if (threadIdx.x < 32) {
    auto h = [&](int i, int k) { return cached ? sH[k * (k + 1) / 2 + i] : H[(size_t)i * st.m + k]; };
    for (int k = j; k >= 0; --k) {
      if (threadIdx.x == 0) sy[k] = __ddiv_rn(sy[k], h(k, k));
      __syncwarp();
      const double yk = sy[k];
      for (int i = (int)threadIdx.x; i < k; i += 32) sy[i] = __dsub_rn(sy[i], __dmul_rn(h(i, k), yk));
      __syncwarp();
    }
  }
  __syncthreads();
  if (!BIG)
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = sy[i];
}

constexpr int kGsChunk = 512;    // coefficients staged at a time
// out = sum_i y_i sig_i Z_i over the cycle's columns: stored as TV (ADD
// false), or added to x (the flexible method's corrections)
template <class TV, bool ADD>
__global__ void __launch_bounds__(256) k_gs_combine(size_t n, const TV* __restrict__ Z, size_t zs, size_t ld, GsDev st,
                                                    TV* __restrict__ out, size_t os, VecOut X) {
  __shared__ double c[kGsChunk];
  const int q = blockIdx.y;
  const int* ist = st.i + 8 * q;
  if (!ist[3]) return;
  const double* d = st.d + (size_t)q * st.sd;
  const int k = ist[2] + 1;
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  for (int i0 = 0; i0 < k; i0 += kGsChunk) {
    const int nc = min(kGsChunk, k - i0);
    __syncthreads();
    for (int i = threadIdx.x; i < nc; i += blockDim.x) c[i] = d[st.oY() + i0 + i] * d[st.oSig() + i0 + i];
    __syncthreads();
    if (p < n) {
#pragma unroll 8
      for (int i = 0; i < nc; ++i) s += c[i] * (double)Z[(size_t)q * zs + (size_t)(i0 + i) * ld + p];
    }
  }
  if (p >= n) return;
  if (ADD) X.p[q][p] += s;
  else out[(size_t)q * os + p] = (TV)s;
}
// x += r of the systems active in the cycle
template <class TV>
__global__ void k_gs_add(size_t n, const TV* __restrict__ r, size_t rs, GsDev st, VecOut X) {
  const int q = blockIdx.y;
  if (!st.i[8 * q + 3]) return;
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) X.p[q][p] += (double)r[(size_t)q * rs + p];
}

}  // namespace aerof
