// fg_solver.cu -- SELL-C-sigma SpMV and the preconditioned CG, on the device.
//
// FP64 path (the drop-in): the operation sequence of cg_solve_body
// (Sources/Lib/LinearAlgebra/IterativeLinearSolver/cg.f90:101-238) and its stopping
// criteria (:279-407), with Jacobi z = D^-1 r (jacobi_preconditioner.f90:356-412):
//   r = b - A x0; z = M r; r_z = <r,z>; p = z
//   loop: Ap = A p; alpha = r_z/<Ap,p>; x += alpha p; r -= alpha Ap; test;
//         z = M r; beta = (1/r_z) * <r,z>; r_z = <r,z>; p = z + beta p
// One cooperative launch runs many iterations (k_pcg64): SpMV with <Ap,p>, the x/r update
// with the norms and the convergence test, and the p update, a grid barrier after each.
// Scalars stay on the device; the host polls after each launch.
//
// Mixed path: CG on an FP32 copy of the matrix with FP32 vectors, with "reliable updates"
// in FP64: whenever the recursive FP32 residual has dropped by a factor delta (default 0.1)
// since the last update, or the estimate of the true residual reaches the tolerance, the
// FP32 correction is folded into the FP64 solution, the true residual r = b - A x is
// recomputed with the FP64 matrix, the FP32 residual is replaced by it (rescaled) and the
// search direction is kept (rescaled).  The solve stops on the FP64 true residual.  Keeping
// the direction keeps the iteration count close to the FP64 CG's, where restarting an inner
// solve per refinement step would lose the Krylov space each time.  With Jacobi the FP32
// segments run CG on D^-1/2 A D^-1/2 (the same iterates in exact arithmetic, no diagonal
// read per iteration) in two steps per iteration (see k_pcg32).
//
// Inner products.  GB300 runs FP64 FMA and FP32<->FP64 conversion at about 0.5 Tera-op/s,
// some 70x below FP32.  FP64-path dots accumulate in FP64.  FP32-path dots form each
// product exactly as an FP32 pair (p = a*b, e = fma(a,b,-p)) and accumulate it with a
// compensated (double-float) sum; blocks add their threads' pairs in three FP32 words (more than FP64
// holds) and the grid total is formed in FP64.  Reductions are deterministic: fixed grid, fixed per-thread index
// sets, block partials summed in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "fg_arith.h"
#include "fg_internal.h"

namespace fg {

static constexpr int RB = 256;  // threads per block of the vector / SpMV kernels

enum { S_RZ = 0, S_ALPHA, S_BETA, S_ERR, S_TOL, S_APP, S_RNRMM, S_BNRM, S_SIGMA, S_RMAX, S_DELTA, S_RRH, S_COUNT = 16 };
// I_PEND: a segment end decided by the last x/r/p update, taken at the next iteration;
// I_SKIPP: this iteration's update keeps p (the segment ends after it)
// I_ABORT: a grid barrier of the CG kernels ran out of time
enum { I_ITER = 0, I_DONE, I_CONV, I_MAXIT, I_FLAG, I_PEND, I_SKIPP, I_ABORT, I_COUNT = 8 };
// FLAG_BREAK: the FP32 recurrence broke down (non-finite or non-positive r_z, residual grown
// 1e4-fold): the segment's correction is dropped and the solve finishes in FP64
enum { FLAG_NONE = 0, FLAG_UPDATE = 1, FLAG_CHECK = 2, FLAG_MAXIT = 3, FLAG_BREAK = 4 };

struct RedBuf {
  double* part;  // [4][nblocks]
  unsigned* ticket;
  int nblocks;
};

// per-thread dot accumulators
template <typename VT>
struct Acc;
template <>
struct Acc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double a, double b) { s = fma(a, b, s); }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<float> {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float a, float b) {
    const float p = __fmul_rn(a, b);
    const float pe = fmaf(a, b, -p);  // exact: a*b = p + pe
    const float s = __fadd_rn(hi, p);
    const float bb = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));  // TwoSum error
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(e, pe));
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// plain FP32 per-thread sum (products rounded): for sums whose terms are all positive
struct AccPlain {
  float s = 0.f;
  __device__ __forceinline__ void add(float a, float b) { s = fmaf(a, b, s); }
  __device__ __forceinline__ double value() const { return (double)s; }
};

// (<q,q> of the mixed iteration, all terms positive: a thread's 107 at 128^3 Q2 go to two plain sums in turn,
// the block's sum and the grid's lose less than FP64.  Compensated sums per thread, with 71 terms in a
// thread, took 1106 iterations there against 1097, and 0.863 ms each against 0.853.)

// the mixed update sums the unscaled residual norm (the stop estimate) every
// FG_MIXED_EXACT_EVERY iterations; 8 vs 4: -2 us per iteration at 128^3 Q2
#ifndef FG_MIXED_EXACT_EVERY
#define FG_MIXED_EXACT_EVERY 8
#endif

template <int NV>
__device__ __forceinline__ bool block_reduce_last(double (&v)[NV], const RedBuf& rb, double (&tot)[NV]) {
  __shared__ double sw[NV][RB / 32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sw[k][w] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = 0.0;
      for (int i = 0; i < RB / 32; ++i) s += sw[k][i];
      rb.part[k * rb.nblocks + blockIdx.x] = s;
    }
    __threadfence();
    unsigned t = atomicAdd(rb.ticket, 1u);
    s_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double s = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += RB) s += __ldcg(rb.part + k * rb.nblocks + i);
    v[k] = s;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
  }
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sw[k][w] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = 0.0;
      for (int i = 0; i < RB / 32; ++i) s += sw[k][i];
      tot[k] = s;
    }
    *rb.ticket = 0u;
  }
  return true;
}

__device__ __forceinline__ double fmaT(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaT(float a, float b, float c) { return fmaf(a, b, c); }

// 4 consecutive matrix entries of one lane: one 128-bit (FP32) or 256-bit (FP64) streaming load
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 t = __ldcs(reinterpret_cast<const float4*>(p));
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
  asm("ld.global.cs.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// ---------------------------------------------------------------------------
// Mixed path, FP32 segments on the scaled system A^ = S A S, S = D^-1/2 (D = diag A): Jacobi
// PCG on A is CG on A^ with x = S x^ and r = S^-1 r^, so no diagonal is streamed per
// iteration (k_pcg32).  Around a segment: fold the correction, refresh the residual.

// x64 += sigma * s x^32; x^32 = 0 (s = D^-1/2 per slot; null: 1)
__global__ void k_fold_scaled(int64_t n, double sigma, const double* __restrict__ sd, float* __restrict__ x32,
                              double* __restrict__ x64) {
  for (int64_t i = blockIdx.x * (int64_t)RB + threadIdx.x; i < n; i += (int64_t)gridDim.x * RB) {
    const double si = sd ? sd[i] : 1.0;
    x64[i] = fma(sigma * si, (double)x32[i], x64[i]);
    x32[i] = 0.f;
  }
}

// r^32 = s r64 / sigma_new; |r^|^2; beta for keeping the direction (first: p = r^).
__global__ void __launch_bounds__(RB)
    k_refresh_scaled(int64_t n, const double* __restrict__ r64, const double* __restrict__ sd, float* __restrict__ r32,
                     int first, RedBuf rb, double* S, int* I) {
  const double inv = 1.0 / S[S_ERR];  // S_ERR = ||b - A x64|| from the FP64 residual SpMV
  Acc<float> rr;
  for (int64_t i = blockIdx.x * (int64_t)RB + threadIdx.x; i < n; i += (int64_t)gridDim.x * RB) {
    const float ri = (float)(r64[i] * inv * (sd ? sd[i] : 1.0));
    r32[i] = ri;
    rr.add(ri, ri);
  }
  double v[1] = {rr.value()}, tot[1];
  if (block_reduce_last<1>(v, rb, tot) && threadIdx.x == 0) {
    const double sig_old = S[S_SIGMA], sig_new = S[S_ERR];
    if (first) {
      S[S_BETA] = 0.0;
    } else {
      // old |r^|^2 and direction in the new scale: rr*(s_old/s_new)^2, p*(s_old/s_new)
      const double q = sig_old / sig_new;
      S[S_BETA] = tot[0] / (S[S_RRH] * q * q) * q;
    }
    S[S_RRH] = tot[0];
    S[S_SIGMA] = sig_new;
    S[S_RMAX] = sqrt(tot[0]);
    I[I_DONE] = 0;
    I[I_FLAG] = FLAG_NONE;
    I[I_PEND] = FLAG_NONE;
    I[I_SKIPP] = 0;
  }
}

// s = sqrt(1/d) per solver slot (0 where 1/d is 0: slots that are not free dofs)
__global__ void k_sqrt_idiag(int64_t n, const double* __restrict__ idiag, double* __restrict__ sd) {
  for (int64_t i = blockIdx.x * (int64_t)RB + threadIdx.x; i < n; i += (int64_t)gridDim.x * RB) {
    const double v = idiag[i];
    sd[i] = v > 0.0 ? sqrt(v) : 0.0;
  }
}

// FP32 copy of A^ = S A S in the lattice-implicit layout, from the FP64 values
__global__ void __launch_bounds__(RB)
    k_scale_stencil32(int64_t nslices, const uint8_t* __restrict__ scls, const int64_t* __restrict__ voff,
                      const StencilClass* __restrict__ cls,
                      const int32_t* __restrict__ soff, const int32_t* __restrict__ st_row,
                      const double* __restrict__ tval, const double* __restrict__ sd, int ncomp, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  for (int64_t s = warp; s < nslices; s += nwarps) {
    const int k = scls[s];
    const int Bp = cls[k].Bp, offbase = cls[k].offbase;
    int32_t st = st_row[s * 32 + lane];
    if (st < 0) st = ~st;  // padding lane: the slice's first row (its values are 0)
    const int32_t base = ncomp == 1 ? st : st - st % ncomp;
    const double srow = sd[st + cls[k].ownoff];
    const int64_t v0 = voff[s] + 4 * lane;
    for (int j = 0; j < (Bp >> 2); ++j) {
      const int4 o = __ldg(reinterpret_cast<const int4*>(soff + offbase) + j);
      const int64_t e = v0 + (int64_t)j * 128;
      // s_i s_j is one product for (i, j) and (j, i): the FP32 copy of an exactly symmetric
      // matrix stays exactly symmetric
      out[e + 0] = (float)(tval[e + 0] * (srow * sd[base + o.x]));
      out[e + 1] = (float)(tval[e + 1] * (srow * sd[base + o.y]));
      out[e + 2] = (float)(tval[e + 2] * (srow * sd[base + o.z]));
      out[e + 3] = (float)(tval[e + 3] * (srow * sd[base + o.w]));
    }
  }
}

// the same in the explicit-column SELL layout
__global__ void __launch_bounds__(RB)
    k_scale_sell32(int64_t nslices, int64_t n, const int64_t* __restrict__ sptr, const int32_t* __restrict__ scol,
                   const double* __restrict__ sval, const double* __restrict__ sd, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  for (int64_t s = warp; s < nslices; s += nwarps) {
    const int64_t base = sptr[s];
    const int w4 = (int)((sptr[s + 1] - base) >> 7);
    const int64_t slot = s * 32 + lane;
    const double srow = slot < n ? sd[slot] : 0.0;
    for (int j = 0; j < w4; ++j) {
      const int64_t e = base + 4 * lane + (int64_t)j * 128;
#pragma unroll
      for (int t = 0; t < 4; ++t) out[e + t] = (float)(sval[e + t] * (srow * sd[scol[e + t]]));
    }
  }
}

// ---------------------------------------------------------------------------
// SELL SpMV, warp per slice, lane per row, slices strided over a fixed grid.
// MODE 0: y = A x.  MODE 2: y = b - A x (b FP64), <y,y> reduced into S_ERR as a norm.
template <typename T, int MODE>
__global__ void __launch_bounds__(RB)
    k_sell_spmv(int64_t nslices, int64_t n, const int64_t* __restrict__ sptr, const int32_t* __restrict__ scol,
                const T* __restrict__ sval, const T* __restrict__ x, T* __restrict__ y, const double* __restrict__ b,
                RedBuf rb, double* S) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  Acc<T> dot;
  for (int64_t s = warp; s < nslices; s += nwarps) {
    const int64_t base = sptr[s];
    const int w4 = (int)((sptr[s + 1] - base) >> 7);  // groups of 4 entries per lane
    const T* vp = sval + base + 4 * lane;
    const int32_t* cp = scol + base + 4 * lane;
    T acc = 0;
#pragma unroll 2
    for (int j = 0; j < w4; ++j) {
      T v[4];
      ld4(vp, v);
      const int4 c = __ldcs(reinterpret_cast<const int4*>(cp));
      const T x0 = __ldg(x + c.x), x1 = __ldg(x + c.y), x2 = __ldg(x + c.z), x3 = __ldg(x + c.w);
      acc = fmaT(v[0], x0, acc);
      acc = fmaT(v[1], x1, acc);
      acc = fmaT(v[2], x2, acc);
      acc = fmaT(v[3], x3, acc);
      vp += 128;
      cp += 128;
    }
    const int64_t slot = s * 32 + lane;
    if (slot < n) {
      if (MODE == 2) {
        const T rr = (T)(b[slot] - (double)acc);
        y[slot] = rr;
        dot.add(rr, rr);
      } else {
        y[slot] = acc;
      }
    }
  }
  if (MODE == 0) return;
  double v[1] = {dot.value()}, tot[1];
  if (block_reduce_last<1>(v, rb, tot) && threadIdx.x == 0) S[S_ERR] = sqrt(tot[0]);
}

// FP64 path start: r = b - r (r holds A x0) or r = b; z = M r; p = z; <r,r>, <r,z>, <b,b>, <b,Mb>.
__global__ void __launch_bounds__(RB)
    k_init64(int64_t n, const double* __restrict__ b, int have_x0, double* __restrict__ r, double* __restrict__ p,
             const double* __restrict__ idiag, int precond, int criterion, double rtol, double atol, int maxit,
             RedBuf rb, double* S, int* I) {
  Acc<double> rr, rz, bb, bmb;
  for (int64_t i = blockIdx.x * (int64_t)RB + threadIdx.x; i < n; i += (int64_t)gridDim.x * RB) {
    const double bi = b[i];
    const double ri = have_x0 ? bi - r[i] : bi;
    const double zi = precond ? idiag[i] * ri : ri;
    r[i] = ri;
    p[i] = zi;
    rr.add(ri, ri);
    rz.add(ri, zi);
    bb.add(bi, bi);
    bmb.add(bi, precond ? idiag[i] * bi : bi);
  }
  double v[4] = {rr.value(), rz.value(), bb.value(), bmb.value()}, tot[4];
  if (block_reduce_last<4>(v, rb, tot) && threadIdx.x == 0) {
    S[S_RZ] = tot[1];
    S[S_RNRMM] = sqrt(tot[1]);
    const double rn = sqrt(tot[0]), bn = sqrt(tot[2]), bnm = sqrt(tot[3]);
    S[S_BNRM] = bn;
    double tol = 0.0;
    switch (criterion) {
      case FG_RES_RHS: case FG_DELTA_RHS: tol = rtol * bn + atol; break;
      case FG_RES_RES: tol = rtol * rn + atol; break;
      case FG_RES_NRMGIVEN_RHS_NRMGIVEN: tol = rtol * bnm + atol; break;
      case FG_RES_NRMGIVEN_RES_NRMGIVEN: tol = rtol * S[S_RNRMM] + atol; break;
      default: break;
    }
    S[S_TOL] = tol;
    S[S_ERR] = rn;
    I[I_ITER] = 0;
    I[I_DONE] = 0;
    I[I_CONV] = 0;
    I[I_MAXIT] = maxit;
    I[I_FLAG] = FLAG_NONE;
  }
}

// p = r + beta p, four entries per thread and load (the vectors are 16-byte aligned)
__global__ void __launch_bounds__(RB)
    k_pupdate(int64_t n, float* __restrict__ p, const float* __restrict__ r, const double* S) {
  const float b = (float)S[S_BETA];
  const int64_t t0 = blockIdx.x * (int64_t)RB + threadIdx.x, stride = (int64_t)gridDim.x * RB;
  const int64_t n4 = n >> 2;
  float4* p4 = reinterpret_cast<float4*>(p);
  const float4* r4 = reinterpret_cast<const float4*>(r);
  for (int64_t i = t0; i < n4; i += stride) {
    const float4 ri = r4[i];
    float4 pi = p4[i];
    pi.x = fmaf(b, pi.x, ri.x);
    pi.y = fmaf(b, pi.y, ri.y);
    pi.z = fmaf(b, pi.z, ri.z);
    pi.w = fmaf(b, pi.w, ri.w);
    p4[i] = pi;
  }
  for (int64_t i = (n4 << 2) + t0; i < n; i += stride) p[i] = fmaf(b, p[i], r[i]);
}

// ---------------------------------------------------------------------------
// Lattice-implicit SELL SpMV: warp per slice, lane per row, 4 values per lane per load;
// the column of box position k is the row's node plus the class offset k.
// L2 prefetch distance of the FP32 SpMV's value stream, in groups of 4 entries per lane.
// Swept on GB300 at 128^3 Q2 (unroll 2): 2-4 groups 0.731-0.735 ms per launch, 6 0.747,
// 8 0.757, 16 0.810.
#ifndef FG_SPMV_PREFETCH
#define FG_SPMV_PREFETCH 3
#endif
#ifndef FG_SPMV_UNROLL
#define FG_SPMV_UNROLL 2
#endif
static constexpr int kPrefetch = FG_SPMV_PREFETCH;  // value groups (of 4 entries per lane) prefetched ahead
static constexpr int kUnroll = FG_SPMV_UNROLL;      // value groups per unrolled step
template <typename T, int MODE>
__global__ void __launch_bounds__(RB)
    k_stencil_spmv(int64_t nslices, const uint8_t* __restrict__ scls, const int64_t* __restrict__ voff,
                   const StencilClass* __restrict__ cls, const int32_t* __restrict__ soff,
                   const int32_t* __restrict__ st_row, const T* __restrict__ tval,
                   int ncomp, const T* __restrict__ x, T* __restrict__ y, const double* __restrict__ b, RedBuf rb,
                   double* S) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  Acc<T> dot;
  for (int64_t s = warp; s < nslices; s += nwarps) {
    const int k = scls[s];
    const int64_t vb = voff[s];
    const int Bp = cls[k].Bp, offbase = cls[k].offbase;
    // st = node index in the class sub-lattice * ncomp + component; the row's own entry is
    // in the class's sub-lattice, its box columns are base + table offsets.  Padding lanes
    // hold the complement of the slice's first row (valid addresses, values 0, no store).
    int32_t st = st_row[s * 32 + lane];
    const bool valid = st >= 0;
    if (!valid) st = ~st;
    const int32_t base = ncomp == 1 ? st : st - st % ncomp;
    const int64_t vec = st + cls[k].ownoff;
    const T* vp = tval + vb + 4 * lane;
    const int4* op = reinterpret_cast<const int4*>(soff + offbase);
    const T* xb = x + base;
    T acc = 0;
    const int w4 = Bp >> 2;
#pragma unroll kUnroll
    for (int j = 0; j < w4; ++j) {
      // FP32: keep the value stream ahead of the gathers by asking L2 for this lane's values
      // kPrefetch groups ahead (no registers held; a hint only, kept inside the slice).  The
      // FP64 variant is bound by the FP64 pipe and runs slower with it.
      if (sizeof(T) == 4 && j + kPrefetch < w4) asm volatile("prefetch.global.L2 [%0];" ::"l"(vp + kPrefetch * 128));
      T v[4];
      ld4(vp, v);
      const int4 o = __ldg(op + j);
      const T x0 = __ldg(xb + o.x), x1 = __ldg(xb + o.y), x2 = __ldg(xb + o.z), x3 = __ldg(xb + o.w);
      acc = fmaT(v[0], x0, acc);
      acc = fmaT(v[1], x1, acc);
      acc = fmaT(v[2], x2, acc);
      acc = fmaT(v[3], x3, acc);
      vp += 128;
    }
    if (valid) {
      if (MODE == 2) {
        const T rr = (T)(b[vec] - (double)acc);
        y[vec] = rr;
        dot.add(rr, rr);
      } else {
        y[vec] = acc;
      }
    }
  }
  if (MODE == 0) return;
  double v[1] = {dot.value()}, tot[1];
  if (block_reduce_last<1>(v, rb, tot) && threadIdx.x == 0) S[S_ERR] = sqrt(tot[0]);
}

// ---------------------------------------------------------------------------
// The CG loop as one cooperative launch.  A launch runs up to max_launch iterations; its
// blocks are co-resident and meet at grid barriers (one per inner product, and one before
// the next SpMV gathers the new p; ~1.4 us each), so an iteration costs two or three barriers
// instead of two or three kernels of a CUDA graph, whose reductions cost 12-18 us each whatever the
// size (32^3 Q1 FP64 solve 3.54 -> 1.28 ms, 24^3 Q2 mixed 10.9 -> 4.4, 96^3 Q2 mixed 374 -> 358).  Bound by
// barriers and FP64 latency where the matrix is small, by the SpMV (FP64 pipe; HBM in FP32) where it is
// large.
//
// Rows: warp w of the solve's block b (nb of them) owns the slices w nb + b + k (warps nb), k = 0.. (an SM then
// holds slices of every width).  R > 0: a lane keeps its R rows' x, r, p and 1/d in registers
// (small and medium systems: at most R slices per warp); only p goes through memory.  R = 0:
// any size, vectors streamed.

struct GridSync {
  double* part;     // [2 buffers][3 values][blocks] partial sums
  unsigned* count;  // arrivals of this launch (zero at launch)
  int* abort;       // set by a wait that ran out
  unsigned long long limit_ns;  // a wait gives up after this long
  int drop;         // test switch (FG_PCG_TEST_DROP_ARRIVAL): block 0 skips its first arrival
};

template <typename T>
struct MatArgs {
  int64_t nslices, n;  // slices; rows (SELL: the vector length)
  const T* val;
  // lattice-implicit
  const uint8_t* scls;
  const int64_t* voff;
  const StencilClass* cls;
  const int32_t* soff;
  const int32_t* st_row;
  int ncomp;
  int noff;            // entries of soff
  // explicit columns
  const int64_t* sptr;
  const int32_t* scol;
  // cell blocks (dG)
  const int32_t* blk;
  int nn;
};

// matrix layout of a kernel: lattice-implicit, explicit columns, cell blocks
enum { ML_STENCIL = 0, ML_SELL = 1, ML_DG = 2 };

// One arrival of the calling block (its other threads have met at a block barrier) and the
// bounded wait for all blocks; called by one thread.  False: the wait ran out or another
// block's did.
__device__ __forceinline__ bool grid_wait(const GridSync& g, unsigned target) {
  __threadfence();
  if (!(g.drop && blockIdx.x == 0 && target == gridDim.x)) atomicAdd(g.count, 1u);
  unsigned spins = 0;
  unsigned long long t0 = 0;
  for (;;) {
    unsigned c;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(g.count) : "memory");
    if (c >= target) break;
    if ((++spins & 255u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (*(volatile int*)g.abort || t - t0 > g.limit_ns) {
        *(volatile int*)g.abort = 1;
        __threadfence();
        return false;
      }
    }
  }
  __threadfence();  // what the other blocks wrote before arriving is visible to this block
  return true;
}

// Block and grid sums of NV accumulators, then f(totals) on thread 0 (the step's scalars, in
// shared memory); every thread returns after f.  Threads leave their sums in shared memory and
// the first four warps add them: an FP64 warp instruction holds the pipe of its SM quarter 64
// cycles, so a warp alone pays that for each of its ~NT/32 + 5 dependent additions per value; the
// four sit in different quarters and take a quarter of the sums each.  The grid's partial sums go
// to one warp per value.  FP32 accumulators (pairs) are added in three FP32 words, which lose less
// than FP64 additions (Sum3), and become FP64 once per block.  Sums in fixed order: deterministic.
// False: the grid barrier gave up.
// (Solve with one warp adding and the scalar steps' square roots and reciprocals on their path, and so:
// 8^3 Q1 FP64, one block, 0.236 -> 0.201 ms; 384^2 Q2 FP64 57.9 -> 55.3 us per iteration.)
template <typename T>
struct RedShared;
template <>
struct RedShared<double> {
  double v[3][1024], w[4][3], tot[3];
};
template <>
struct RedShared<float> {
  float2 v[2][1024];
  Sum3 w[4][3];
  double tot[3];
};

// sums over the warp (lane 0), two FP64 values in one butterfly
template <int NV>
__device__ __forceinline__ void warp_sums(double (&s)[NV], int lane) {
  constexpr int N1 = NV >= 2 ? 2 : 0;  // values summed together
  if (NV >= 2) {
    const bool up = lane >= 16;
    double x = (up ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, up ? s[0] : s[1], 16);
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    s[0] = x;
    s[1] = __shfl_sync(0xffffffffu, x, 16);
  }
#pragma unroll
  for (int k = N1; k < NV; ++k)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
}

// sums of the values V: FP64, or pairs in three words
template <typename V>
struct SumOf;
template <>
struct SumOf<double> { using type = double; };
template <>
struct SumOf<float2> { using type = Sum3; };
__device__ __forceinline__ void sum_in(double& s, double v) { s += v; }
__device__ __forceinline__ void sum_in(Sum3& s, float2 v) { s.add(v.x, v.y, 0.f); }
__device__ __forceinline__ void sum_in(Sum3& s, const Sum3& v) { s.add(v.h, v.m, v.l); }
__device__ __forceinline__ double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ Sum3 shfl_xor(const Sum3& v, int m) {
  Sum3 o;
  o.h = __shfl_xor_sync(0xffffffffu, v.h, m);
  o.m = __shfl_xor_sync(0xffffffffu, v.m, m);
  o.l = __shfl_xor_sync(0xffffffffu, v.l, m);
  return o;
}
__device__ __forceinline__ double to_f64(double v) { return v; }
__device__ __forceinline__ double to_f64(const Sum3& v) { return v.value(); }
template <int NV>
__device__ __forceinline__ void warp_sums(Sum3 (&s)[NV], int) {
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum_in(s[k], shfl_xor(s[k], off));
}

// barrier of the first nt threads
__device__ __forceinline__ void adders_meet(int nt) {
  if (nt > 32) asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
  else __syncwarp();
}

// the block's sums as place blk of nblk in part (or, alone, the totals); the values wait in sh.v until the
// first four warps have added them
template <int NV, typename T, typename V>
__device__ __forceinline__ void block_part(RedShared<T>& sh, const V (&v)[NV], double* part, int blk, int nblk) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) sh.v[k][t] = v[k];
  __syncthreads();
  const int nt = blockDim.x < 128 ? blockDim.x : 128;  // the adding threads
  if (t >= nt) return;
  using A = typename SumOf<V>::type;
  A s[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    s[k] = A{};
    for (int i = t; i < (int)blockDim.x; i += nt) sum_in(s[k], sh.v[k][i]);
  }
  warp_sums(s, lane);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh.w[warp][k] = s[k];
  adders_meet(nt);
  if (warp == 0) {
    // lane 4 k + w: value k of warp w
    A y = lane < 4 * NV && (lane & 3) < (nt >> 5) ? sh.w[lane & 3][lane >> 2] : A{};
    sum_in(y, shfl_xor(y, 1));
    sum_in(y, shfl_xor(y, 2));
    if (lane < 4 * NV && (lane & 3) == 0) {
      const double d = to_f64(y);
      if (nblk > 1) part[(lane >> 2) * nblk + blk] = d;
      else sh.tot[lane >> 2] = d;
    }
    __syncwarp();
  }
}

// body(b, values): the values of block b of the solve's gridDim.x x vb blocks, which a block of the
// launch does one after another (PcgShape)
template <int NV, typename V, typename T, typename B, typename F>
__device__ __forceinline__ bool grid_reduce(RedShared<T>& sh, const GridSync& g, int buf, unsigned& target, int* s_ok,
                                            int vb, B&& body, F&& f) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int nblk = (int)gridDim.x * vb;
  double* part = g.part + (size_t)buf * 3 * nblk;
  for (int v = 0; v < vb; ++v) {
    V val[NV];
    const int blk = blockIdx.x + v * gridDim.x;
    body(blk, val);
    if (v > 0) __syncthreads();  // the last one's values have been added
    block_part<NV>(sh, val, part, blk, nblk);
  }
  target += gridDim.x;
  const int nt = blockDim.x < 128 ? blockDim.x : 128;
  if (t < nt) {
    if (t == 0) *s_ok = nblk == 1 || grid_wait(g, target) ? 1 : 0;
    __syncwarp();
    if (nblk > 1) {
      adders_meet(nt);
      for (int k = warp; k < NV; k += nt >> 5) {
        double z[1] = {0.0};
#pragma unroll 4
        for (int i = lane; i < nblk; i += 32) z[0] += __ldcg(part + (size_t)k * nblk + i);
        warp_sums(z, lane);
        if (lane == 0) sh.tot[k] = z[0];
      }
      adders_meet(nt);
    }
    if (t == 0 && *s_ok) {
      double tot[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) tot[k] = sh.tot[k];
      f(tot);
    }
  }
  __syncthreads();
  return *s_ok != 0;
}

// barrier without a sum
__device__ __forceinline__ bool grid_barrier(const GridSync& g, unsigned& target, int* s_ok) {
  __syncthreads();
  target += gridDim.x;
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) *s_ok = grid_wait(g, target) ? 1 : 0;
  __syncthreads();
  return *s_ok != 0;
}

// matrix values of one group: kept in L2 (R > 0: the matrix of such a system mostly stays there
// from one iteration to the next; not in L1, which is the gathered vector's) or streamed
template <bool KEEP>
__device__ __forceinline__ void ld4k(const float* p, float (&v)[4]) {
  if (!KEEP) { ld4(p, v); return; }
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}
template <bool KEEP>
__device__ __forceinline__ void ld4k(const double* p, double (&v)[4]) {
  if (!KEEP) { ld4(p, v); return; }
  asm("ld.global.nc.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// One slice of the matrix as one lane sees it.
template <typename T, int ML>
struct SliceRef {
  static constexpr bool STENCIL = ML == ML_STENCIL;
  const T* vp;         // the lane's first value
  const int32_t* cp;   // lattice-implicit: offsets of the class; explicit: the lane's first column;
                       // cell blocks: first columns of the row's 7 blocks
  int w4;              // groups of 4 entries (cell blocks: of one block)
  int32_t base, vec;   // gather base (cell blocks: columns per block); the row's vector index (-1: no row)
  const float4* sv;    // the lane's values in shared memory (keep), or null

  // 16-byte pieces of a lane's group of 4 entries, and groups of the slice
  static constexpr int PC = sizeof(T) / 4;
  __device__ __forceinline__ int groups() const { return ML == ML_DG ? 7 * w4 : w4; }
  // Copies the slice into shared memory at `dst` (32 PC pieces per group, piece by piece: the warp's
  // accesses are contiguous).  A lane reads back only what it wrote.
  __device__ __forceinline__ void keep(float4* dst, int lane) {
    dst += lane;
    sv = dst;
    const float4* src = reinterpret_cast<const float4*>(vp);
    const int n = groups();
#pragma unroll 4
    for (int j = 0; j < n; ++j)
#pragma unroll
      for (int q = 0; q < PC; ++q) dst[(j * PC + q) * 32] = __ldcs(src + (size_t)j * 32 * PC + q);
  }
  static __device__ __forceinline__ void lds4(const float4* s, float (&v)[4]) {
    const float4 a = s[0];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
  static __device__ __forceinline__ void lds4(const float4* s, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(s), b = *reinterpret_cast<const double2*>(s + 32);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
  // dot with the values in shared memory: the gathers of four groups are in flight together
  __device__ __forceinline__ T dot_kept(const T* x) const {
    T acc = 0;
    const float4* v0 = sv;
    if (ML == ML_DG) {
#pragma unroll 1
      for (int k = 0; k < 7; ++k) {
        const T* xb = x + cp[k];
#pragma unroll 4
        for (int j = 0; j < w4; ++j, v0 += 32 * PC) {
          const T x0 = xb[4 * j], x1 = xb[4 * j + 1], x2 = xb[4 * j + 2], x3 = xb[min(4 * j + 3, base - 1)];
          T v[4];
          lds4(v0, v);
          acc = fmaT(v[0], x0, acc);
          acc = fmaT(v[1], x1, acc);
          acc = fmaT(v[2], x2, acc);
          acc = fmaT(v[3], x3, acc);
        }
      }
      return acc;
    }
    const T* xb = x + base;
    const int32_t* c0 = cp;
#pragma unroll 4
    for (int j = 0; j < w4; ++j, v0 += 32 * PC) {
      int4 o;
      if (STENCIL) o = reinterpret_cast<const int4*>(c0)[j];
      else o = __ldg(reinterpret_cast<const int4*>(c0 + j * 128));
      const T x0 = xb[o.x], x1 = xb[o.y], x2 = xb[o.z], x3 = xb[o.w];
      T v[4];
      lds4(v0, v);
      acc = fmaT(v[0], x0, acc);
      acc = fmaT(v[1], x1, acc);
      acc = fmaT(v[2], x2, acc);
      acc = fmaT(v[3], x3, acc);
    }
    return acc;
  }
  // a warp's place without a slice (fewer slices than warps): no groups, no row.  The products still
  // run over it, so every pointer is a valid one (cell blocks read their first columns before the
  // loop over the groups)
  __device__ __forceinline__ void none(const MatArgs<T>& m, const int32_t* s_off) {
    vp = m.val;
    cp = STENCIL ? s_off : ML == ML_DG ? m.blk : m.scol;
    w4 = 0;
    base = ML == ML_DG ? m.nn : 0;
    vec = -1;
    sv = nullptr;
  }
  __device__ __forceinline__ void load(const MatArgs<T>& m, int64_t s, int lane, const int32_t* s_off) {
    if (STENCIL) {
      const int k = m.scls[s];
      const StencilClass& C = m.cls[k];
      int32_t st = m.st_row[s * 32 + lane];
      const bool valid = st >= 0;
      if (!valid) st = ~st;
      base = m.ncomp == 1 ? st : st - st % m.ncomp;
      vec = valid ? (int32_t)(st + C.ownoff) : -1;
      w4 = C.Bp >> 2;
      vp = m.val + m.voff[s] + 4 * lane;
      cp = s_off + C.offbase;
    } else if (ML == ML_DG) {
      const int64_t slot = s * 32 + lane;
      w4 = (m.nn + 3) >> 2;
      vp = m.val + s * (32 * 7 * 4) * w4 + 4 * lane;
      cp = m.blk + 8 * ((slot < m.n ? slot : m.n - 1) / m.nn);
      base = m.nn;
      vec = slot < m.n ? (int32_t)slot : -1;
    } else {
      const int64_t b = m.sptr[s];
      w4 = (int)((m.sptr[s + 1] - b) >> 7);
      vp = m.val + b + 4 * lane;
      cp = m.scol + b + 4 * lane;
      const int64_t slot = s * 32 + lane;
      base = 0;
      vec = slot < m.n ? (int32_t)slot : -1;
    }
  }
  // the row's products with x; x changes during the launch, so it is read with plain loads
  // (coherent after a grid barrier), never through the read-only path
  template <bool KEEP, int UNROLL>
  __device__ __forceinline__ T dot(const T* x) const {
    T acc = 0;
    const T* v0 = vp;
    const int32_t* c0 = cp;
    if (ML == ML_DG) {
      // the rows of a cell read the same x: a warp's gather is one or two addresses
#pragma unroll 1
      for (int k = 0; k < 7; ++k) {
        const T* xb = x + cp[k];
#pragma unroll UNROLL
        for (int j = 0; j < w4; ++j) {
          if (!KEEP && sizeof(T) == 4 && k * w4 + j + kPrefetch < 7 * w4)  // inside the slice
            asm volatile("prefetch.global.L2 [%0];" ::"l"(v0 + kPrefetch * 128));
          T v[4];
          ld4k<KEEP>(v0, v);
          const T x0 = xb[4 * j], x1 = xb[4 * j + 1], x2 = xb[4 * j + 2], x3 = xb[min(4 * j + 3, base - 1)];
          acc = fmaT(v[0], x0, acc);
          acc = fmaT(v[1], x1, acc);
          acc = fmaT(v[2], x2, acc);
          acc = fmaT(v[3], x3, acc);
          v0 += 128;
        }
      }
      return acc;
    }
    const T* xb = x + base;
#pragma unroll UNROLL
    for (int j = 0; j < w4; ++j) {
      // FP32 streams, and FP64 matrices of a few hundred MB (R > 0: 22 warps with two groups in
      // flight hold too few bytes; 23 x 17 x 21 Q3 70.8 -> 64.2 us per iteration)
      if (STENCIL && KEEP == (sizeof(T) == 8) && j + kPrefetch < w4)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(v0 + kPrefetch * 128));
      // explicit columns: both streams, the gathers wait for the columns
      if (ML == ML_SELL && sizeof(T) == 4 && j + kPrefetch < w4) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(v0 + kPrefetch * 128));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(c0 + kPrefetch * 128));
      }
      T v[4];
      ld4k<KEEP>(v0, v);
      int4 o;
      if (STENCIL) o = reinterpret_cast<const int4*>(c0)[j];
      else if (KEEP) o = __ldg(reinterpret_cast<const int4*>(c0));
      else o = __ldcs(reinterpret_cast<const int4*>(c0));
      const T x0 = xb[o.x], x1 = xb[o.y], x2 = xb[o.z], x3 = xb[o.w];
      acc = fmaT(v[0], x0, acc);
      acc = fmaT(v[1], x1, acc);
      acc = fmaT(v[2], x2, acc);
      acc = fmaT(v[3], x3, acc);
      v0 += 128;
      if (!STENCIL) c0 += 128;
    }
    return acc;
  }
};

// the class offsets in shared memory (lattice-implicit layout)
template <typename T, int ML>
__device__ __forceinline__ const int32_t* stage_offsets(const MatArgs<T>& m, int32_t* s_off) {
  if (ML != ML_STENCIL) return nullptr;
  for (int i = threadIdx.x; i < m.noff; i += blockDim.x) s_off[i] = m.soff[i];
  __syncthreads();
  return s_off;
}

// Keeps as many of the block's slices in shared memory as fit `cap` groups (KBs of matrix that no
// iteration reads again from L2).  s_cnt: RR x 32 ints of shared memory.
template <typename T, int ML, int RR>
__device__ __forceinline__ void keep_slices(SliceRef<T, ML> (&ref)[RR], float4* buf, int cap, int* s_cnt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < RR; ++k) s_cnt[k * 32 + warp] = ref[k].groups();
  __syncthreads();
  int before = 0;  // groups of the slices before mine (k by k, warp by warp)
#pragma unroll
  for (int k = 0; k < RR; ++k) {
    const int mine = lane < nw ? s_cnt[k * 32 + lane] : 0;
    const int upto = before + (int)__reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
    ref[k].sv = nullptr;
    if (ref[k].groups() > 0 && upto + ref[k].groups() <= cap)
      ref[k].keep(buf + (size_t)upto * 32 * SliceRef<T, ML>::PC, lane);
    before += (int)__reduce_add_sync(0xffffffffu, mine);
  }
}

// Threads per block.  Streaming kernels: 2 x 16 warps of 64 registers, i.e. more of a slice in flight
// per warp, rather than 2 x 24 of 40 (96^3 Q2 mixed 370 -> 360 us per iteration, 32^3 Q2 dG mixed 130 ->
// 124, 384^2 Q2 FP64 55.3 -> 52; 2 x 12 of 80: 377, 130, 57).  FP32 with explicit columns waits for its
// gathers, each behind a column: 2 x 32 warps (unstructured Q2 40^3 90 -> 69, 48^3 119 -> 110, 64^3
// 256 -> 234 against 2 x 16, with both streams prefetched).  FP64 with explicit columns from HBM
// (R = PCG_WIDE): 2 x 24, two groups in flight (quadrilaterals 1024^2 0.289 -> 0.282 ms, 2048^2 1.113 ->
// 1.056, unstructured 88^3 1.062 -> 0.994; 384^2, whose 127 MB stay in L2, 52.2 -> 55.2 us; 700^2, 420 MB,
// the same either way).
static constexpr int PCG_WIDE = -1;
static constexpr int pcg_threads(int R, int ML, bool fp32) {
  return R > 0 || (fp32 && ML == ML_SELL) ? 1024 : R == PCG_WIDE ? 768 : 512;
}
static constexpr int pcg_blocks(int R) { return R > 0 ? 1 : 2; }

// the polling chunk that iteration `it` lies in ends before the iteration limit
__host__ __device__ __forceinline__ bool chunk_ends_before(int it, int chunk, int maxit) {
  return ((int64_t)it + chunk - 1) / chunk * chunk < maxit;
}

// FP64 CG, the sequence and stopping tests of the reference (cg.f90:101-238, 279-407).
// idiag null: no preconditioner.  chunk: the polling interval the caller asked for (a
// non-finite iteration is reported at its end, if the iteration limit lies beyond it).
template <int ML, int R>
__global__ void __launch_bounds__(pcg_threads(R, ML, false), pcg_blocks(R))
    k_pcg64(MatArgs<double> m, int64_t nvec, double* x, double* r, double* p, double* Ap,
            const double* __restrict__ idiag, int criterion, double rtol, double atol, int max_launch, int chunk,
            int keep, int vblocks, GridSync g, double* S, int* I) {
  extern __shared__ __align__(16) int32_t s_off_buf[];
  __shared__ RedShared<double> sh;
  __shared__ double sc[9];  // alpha, beta, rz, err, tol, rnrmm, <r,r>, its bound, 1/rz
  __shared__ int si[4];     // stop (1 done, 2 non-finite), converged, ok
  if (I[I_DONE]) return;
  constexpr int RR = R > 0 ? R : 1;
  const int lane = threadIdx.x & 31;
  const int vb = R > 0 ? 1 : vblocks, nblk = (int)gridDim.x * vb;
  const int64_t nwarps = (int64_t)(blockDim.x >> 5) * nblk;
  auto warp_of = [&](int blk) { return (int64_t)(threadIdx.x >> 5) * nblk + blk; };
  const bool need_pp = criterion == FG_DELTA_RHS || criterion == FG_DELTA_DELTA;
  const bool res = criterion == FG_RES_RES || criterion == FG_RES_RHS;
  const int32_t* s_off = stage_offsets<double, ML>(m, s_off_buf);
  const int it0 = I[I_ITER], maxit = I[I_MAXIT];
  if (threadIdx.x == 0) {
    sc[2] = S[S_RZ];
    sc[3] = S[S_ERR];
    sc[4] = S[S_TOL];
    sc[5] = S[S_RNRMM];
    // <r,r> above this cannot have a root within the tolerance: no square root then
    const double t2 = sc[4] * sc[4] * (1.0 + 1e-12);
    sc[7] = t2 > 1e-290 ? t2 : INFINITY;
    si[0] = si[1] = 0;
  }
  SliceRef<double, ML> ref[RR];
  double rx[RR], rr_[RR], rp[RR], rd[RR], ra[RR];
  if (R > 0) {
#pragma unroll
    for (int k = 0; k < RR; ++k) {
      const int64_t s = warp_of(blockIdx.x) + k * nwarps;
      rx[k] = rr_[k] = rp[k] = rd[k] = 0.0;
      if (s >= m.nslices) {
        ref[k].none(m, s_off);
      } else {
        ref[k].load(m, s, lane, s_off);
        const int32_t v = ref[k].vec;
        if (v >= 0) {
          rx[k] = x[v];
          rr_[k] = r[v];
          rp[k] = p[v];
          rd[k] = idiag ? idiag[v] : 1.0;
        }
      }
    }
  }
  if (R > 0) {
    __shared__ int s_cnt[32 * RR];
    keep_slices(ref, reinterpret_cast<float4*>(s_off_buf + ((m.noff + 3) & ~3)), keep, s_cnt);
  }
  const int64_t stride = (int64_t)nblk * blockDim.x;
  auto thread_of = [&](int blk) { return (int64_t)blk * blockDim.x + threadIdx.x; };
  unsigned target = 0;
  __syncthreads();  // the scalars
  int it = it0;
  for (int n = 0; n < max_launch; ++n) {
    // beside the product: 1/rz for beta (a division on thread 0 between two barriers is 0.4 us)
    if (threadIdx.x == blockDim.x - 32) sc[8] = 1.0 / sc[2];
    // Ap = A p, <Ap,p>
    auto product = [&](int blk, double (&v)[1]) {
      Acc<double> dot;
      if (R > 0) {
#pragma unroll
        for (int k = 0; k < RR; ++k) {
          ra[k] = ref[k].sv ? ref[k].dot_kept(p) : ref[k].template dot<true, 2>(p);
          if (ref[k].vec >= 0) dot.add(ra[k], rp[k]);
        }
      } else {
        for (int64_t s = warp_of(blk); s < m.nslices; s += nwarps) {
          SliceRef<double, ML> q;
          q.load(m, s, lane, s_off);
          const double a = q.template dot<false, ML == ML_SELL && R == 0 ? 4 : kUnroll>(p);
          if (q.vec >= 0) {
            Ap[q.vec] = a;
            dot.add(a, p[q.vec]);
          }
        }
      }
      v[0] = dot.value();
    };
    if (!grid_reduce<1, double>(sh, g, 0, target, &si[2], vb, product,
                                [&](double (&t)[1]) { sc[0] = t[0] != 0.0 ? sc[2] / t[0] : 0.0; }))
      return;
    // x += alpha p; r -= alpha Ap; the convergence test; beta
    const double a = sc[0];
    auto update = [&](int blk, Acc<double>& rr, Acc<double>& rz, Acc<double>& pp) {
      if (R > 0) {
#pragma unroll
        for (int k = 0; k < RR; ++k) {
          rx[k] = fma(a, rp[k], rx[k]);
          if (ref[k].vec >= 0) rr_[k] = fma(-a, ra[k], rr_[k]);
          rr.add(rr_[k], rr_[k]);
          if (idiag) rz.add(rr_[k], rd[k] * rr_[k]);
          if (need_pp) pp.add(rp[k], rp[k]);
        }
      } else {
        for (int64_t i = thread_of(blk); i < nvec; i += stride) {
          const double pi = p[i];
          x[i] = fma(a, pi, x[i]);
          const double ri = fma(-a, Ap[i], r[i]);
          r[i] = ri;
          rr.add(ri, ri);
          if (idiag) rz.add(ri, idiag[i] * ri);
          if (need_pp) pp.add(pi, pi);
        }
      }
    };
    ++it;
    auto test = [&](double trr, double trz, double tpp) {
      bool conv = false;
      if (res) {
        sc[6] = trr;
        if (trr <= sc[7]) conv = sqrt(trr) <= sc[4];
      } else {
        double err = sc[5];
        if (need_pp) {
          err = a * sqrt(tpp);
          if (it == 1 && criterion == FG_DELTA_DELTA) sc[4] = rtol * err + atol;
        }
        sc[3] = err;
        conv = err <= sc[4];
      }
      if (conv || it >= maxit) {
        si[0] = 1;
        si[1] = conv ? 1 : 0;
        return;
      }
      sc[2] = trz;
      sc[1] = sc[8] * trz;
      if (!res && !need_pp) sc[5] = sqrt(trz);  // the next iteration's estimate
      if (!(isfinite(a) && isfinite(trz)) && chunk_ends_before(it, chunk, maxit)) si[0] = 2;
    };
    bool ok;
    if (need_pp) {
      ok = grid_reduce<3, double>(
          sh, g, 1, target, &si[2], vb,
          [&](int blk, double (&v)[3]) {
            Acc<double> rr, rz, pp;
            update(blk, rr, rz, pp);
            v[0] = rr.value();
            v[1] = idiag ? rz.value() : rr.value();
            v[2] = pp.value();
          },
          [&](double (&t)[3]) { test(t[0], t[1], t[2]); });
    } else if (idiag) {
      ok = grid_reduce<2, double>(
          sh, g, 1, target, &si[2], vb,
          [&](int blk, double (&v)[2]) {
            Acc<double> rr, rz, pp;
            update(blk, rr, rz, pp);
            v[0] = rr.value();
            v[1] = rz.value();
          },
          [&](double (&t)[2]) { test(t[0], t[1], 0.0); });
    } else {
      ok = grid_reduce<1, double>(
          sh, g, 1, target, &si[2], vb,
          [&](int blk, double (&v)[1]) {
            Acc<double> rr, rz, pp;
            update(blk, rr, rz, pp);
            v[0] = rr.value();
          },
          [&](double (&t)[1]) { test(t[0], t[0], 0.0); });
    }
    if (!ok) return;
    if (si[0]) break;
    // p = z + beta p
    const double beta = sc[1];
    if (R > 0) {
#pragma unroll
      for (int k = 0; k < RR; ++k) {
        rp[k] = fma(beta, rp[k], rd[k] * rr_[k]);
        if (ref[k].vec >= 0) p[ref[k].vec] = rp[k];
      }
    } else {
      for (int v = 0; v < vb; ++v)
        for (int64_t i = thread_of(blockIdx.x + v * gridDim.x); i < nvec; i += stride) {
          const double ri = r[i];
          p[i] = fma(beta, p[i], idiag ? idiag[i] * ri : ri);
        }
    }
    if (n + 1 < max_launch && !grid_barrier(g, target, &si[2])) return;
  }
  if (R > 0) {
#pragma unroll
    for (int k = 0; k < RR; ++k)
      if (ref[k].vec >= 0) {
        x[ref[k].vec] = rx[k];
        r[ref[k].vec] = rr_[k];
      }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S[S_ALPHA] = sc[0];
    S[S_BETA] = sc[1];
    S[S_RZ] = sc[2];
    S[S_ERR] = res ? sqrt(sc[6]) : sc[3];
    S[S_TOL] = sc[4];
    S[S_RNRMM] = sc[5];
    I[I_ITER] = it;
    I[I_DONE] = si[0] == 1;
    I[I_CONV] = si[1];
  }
}

// FP32 segment of the mixed path on A^ = S A S (or A): two grid barriers per iteration.
//   q = A^ p, <p,q>, <q,q>; then alpha = |r|^2/<p,q> and, by the recurrence
//   |r - alpha q|^2 = alpha^2 |q|^2 - |r|^2 (as <r,q> = <p,q> in CG), beta = |r_new|^2/|r|^2;
//   x += alpha p; r -= alpha q; p = r + beta p; the exact |r_new|^2 for the next alpha, and on
//   every FG_MIXED_EXACT_EVERY-th iteration of the segment (phase: those before this launch) sum r^2 D
//   (the unscaled residual, for the stop estimate), with the caller's polling interval also on its last.
// A segment end (reliable update, stop check, breakdown, iteration limit) found by an update
// is taken one iteration later: that iteration's update keeps p, so the host can fold x and
// restart the recursion from the true residual with the direction kept.
template <int ML, int R>
__global__ void __launch_bounds__(pcg_threads(R, ML, true), pcg_blocks(R))
    k_pcg32(MatArgs<float> m, int64_t nvec, float* x, float* r, float* p, float* q, const float* __restrict__ idiag,
            int max_launch, int phase, int last_exact, int keep, int vblocks, GridSync g, double* S, int* I) {
  extern __shared__ __align__(16) int32_t s_off_buf[];
  __shared__ RedShared<float> sh;
  __shared__ double sd[8];  // rr, rmax^2, delta^2, (tol/sigma)^2, 1/rr, app, alpha, beta
  __shared__ float sf[2];   // alpha, beta
  __shared__ int si[8];     // pend, skip, done flag, ok
  if (I[I_DONE]) return;
  constexpr int RR = R > 0 ? R : 1;
  const int lane = threadIdx.x & 31;
  const int vb = R > 0 ? 1 : vblocks, nblk = (int)gridDim.x * vb;
  const int64_t nwarps = (int64_t)(blockDim.x >> 5) * nblk;
  auto warp_of = [&](int blk) { return (int64_t)(threadIdx.x >> 5) * nblk + blk; };
  const int32_t* s_off = stage_offsets<float, ML>(m, s_off_buf);
  const int maxit = I[I_MAXIT];
  int it = I[I_ITER];
  if (threadIdx.x == 0) {
    sd[0] = S[S_RRH];
    const double rmax = S[S_RMAX], delta = S[S_DELTA], lim = S[S_TOL] / S[S_SIGMA];
    sd[1] = rmax * rmax;
    sd[2] = delta * delta;
    sd[3] = lim * lim;
    sd[5] = S[S_APP];
    si[0] = I[I_PEND];
    si[1] = I[I_SKIPP];
    si[2] = FLAG_NONE;
  }
  SliceRef<float, ML> ref[RR];
  float rx[RR], rr_[RR], rp[RR], rq[RR];
  if (R > 0) {
#pragma unroll
    for (int k = 0; k < RR; ++k) {
      const int64_t s = warp_of(blockIdx.x) + k * nwarps;
      rx[k] = rr_[k] = rp[k] = 0.f;
      if (s >= m.nslices) {
        ref[k].none(m, s_off);
      } else {
        ref[k].load(m, s, lane, s_off);
        const int32_t v = ref[k].vec;
        if (v >= 0) {
          rx[k] = x[v];
          rr_[k] = r[v];
          rp[k] = p[v];
        }
      }
    }
  }
  if (R > 0) {
    __shared__ int s_cnt[32 * RR];
    keep_slices(ref, reinterpret_cast<float4*>(s_off_buf + ((m.noff + 3) & ~3)), keep, s_cnt);
  }
  const int64_t stride = (int64_t)nblk * blockDim.x;
  auto thread_of = [&](int blk) { return (int64_t)blk * blockDim.x + threadIdx.x; };
  unsigned target = 0;
  __syncthreads();  // the scalars
  for (int n = 0; n < max_launch; ++n) {
    // beside the product: 1/rr for beta (see k_pcg64)
    if (threadIdx.x == blockDim.x - 32) sd[4] = 1.0 / sd[0];
    auto product = [&](int blk, float2 (&v)[2]) {
      Acc<float> pq;
      AccPlain qq, qq1;  // <q,q>: the slices' rows alternate between two sums
      if (R > 0) {
#pragma unroll
        for (int k = 0; k < RR; ++k) {
          rq[k] = ref[k].sv ? ref[k].dot_kept(p) : ref[k].template dot<true, R == 1 ? 4 : 2>(p);
          if (ref[k].vec >= 0) {
            pq.add(rq[k], rp[k]);
            qq.add(rq[k], rq[k]);
          }
        }
      } else {
        for (int64_t s = warp_of(blk); s < m.nslices; s += nwarps) {
          SliceRef<float, ML> w;
          w.load(m, s, lane, s_off);
          const float a = w.template dot<false, ML == ML_SELL ? 4 : kUnroll>(p);
          if (w.vec >= 0) {
            q[w.vec] = a;
            pq.add(a, p[w.vec]);
            qq.add(a, a);
          }
          const float t = qq.s;
          qq.s = qq1.s;
          qq1.s = t;
        }
      }
      v[0] = make_float2(pq.hi, pq.lo);
      v[1] = make_float2(qq.s, 0.f);
      if (R <= 0) two_sum(qq.s, qq1.s, v[1].x, v[1].y);
    };
    if (!grid_reduce<2, float2>(sh, g, 0, target, &si[3], vb, product, [&](double (&t)[2]) {
          const double pap = t[0], nq = t[1], rr = sd[0];
          int skip = si[0] != FLAG_NONE;
          double a = 0.0, b = 0.0;
          if (!(pap > 0.0 && pap <= 1e300) || !(nq <= 1e300)) {
            si[0] = FLAG_BREAK;  // alpha = 0: the update leaves x and r as they are
            skip = 1;
          } else {
            a = rr / pap;
            const double rrn = a * a * nq - rr;
            b = rrn * sd[4];
            if (!(rrn > 0.0)) {  // the recurrence lost its digits: end the segment here
              skip = 1;
              if (si[0] == FLAG_NONE) si[0] = FLAG_UPDATE;
            }
          }
          sf[0] = (float)a;
          sf[1] = (float)b;
          sd[6] = a;
          sd[7] = b;
          si[1] = skip;
        }))
      return;
    const float a = sf[0], b = sf[1];
    const bool keep_p = si[1] != 0;
    const bool exact = (n + phase) % FG_MIXED_EXACT_EVERY == FG_MIXED_EXACT_EVERY - 1 || (last_exact && n == max_launch - 1);
    // unscaled residual entry r^ sqrt(d): r^2 d = r^2 / (1/d); slots that are not free dofs hold
    // r = 0 and 1/d = 0: skipped
    auto unscaled = [](Acc<float>& rt, float ri, float di) { rt.add(ri, di != 0.f ? ri / di : 0.f); };
    auto update = [&](int blk, Acc<float>& rr, Acc<float>& rt) {
      if (R > 0) {
#pragma unroll
        for (int k = 0; k < RR; ++k) {
          if (ref[k].vec < 0) continue;
          rx[k] = fmaf(a, rp[k], rx[k]);
          rr_[k] = fmaf(-a, rq[k], rr_[k]);
          if (!keep_p) {
            rp[k] = fmaf(b, rp[k], rr_[k]);
            p[ref[k].vec] = rp[k];
          }
          rr.add(rr_[k], rr_[k]);
          if (exact) unscaled(rt, rr_[k], idiag ? idiag[ref[k].vec] : 1.f);
        }
      } else {
        const int64_t n4 = nvec >> 2;
        float4* x4 = reinterpret_cast<float4*>(x);
        float4* r4 = reinterpret_cast<float4*>(r);
        float4* p4 = reinterpret_cast<float4*>(p);
        const float4* q4 = reinterpret_cast<const float4*>(q);
        const float4* d4 = reinterpret_cast<const float4*>(idiag);
        for (int64_t i = thread_of(blk); i < n4; i += stride) {
          float4 xi = x4[i], ri = r4[i], pi = p4[i];
          const float4 qi = q4[i];
          xi.x = fmaf(a, pi.x, xi.x);
          xi.y = fmaf(a, pi.y, xi.y);
          xi.z = fmaf(a, pi.z, xi.z);
          xi.w = fmaf(a, pi.w, xi.w);
          ri.x = fmaf(-a, qi.x, ri.x);
          ri.y = fmaf(-a, qi.y, ri.y);
          ri.z = fmaf(-a, qi.z, ri.z);
          ri.w = fmaf(-a, qi.w, ri.w);
          x4[i] = xi;
          r4[i] = ri;
          if (!keep_p) {
            pi.x = fmaf(b, pi.x, ri.x);
            pi.y = fmaf(b, pi.y, ri.y);
            pi.z = fmaf(b, pi.z, ri.z);
            pi.w = fmaf(b, pi.w, ri.w);
            p4[i] = pi;
          }
          rr.add(ri.x, ri.x);
          rr.add(ri.y, ri.y);
          rr.add(ri.z, ri.z);
          rr.add(ri.w, ri.w);
          if (exact) {
            const float4 di = idiag ? d4[i] : make_float4(1.f, 1.f, 1.f, 1.f);
            unscaled(rt, ri.x, di.x);
            unscaled(rt, ri.y, di.y);
            unscaled(rt, ri.z, di.z);
            unscaled(rt, ri.w, di.w);
          }
        }
        for (int64_t i = (n4 << 2) + thread_of(blk); i < nvec; i += stride) {
          x[i] = fmaf(a, p[i], x[i]);
          const float ri = fmaf(-a, q[i], r[i]);
          r[i] = ri;
          if (!keep_p) p[i] = fmaf(b, p[i], ri);
          rr.add(ri, ri);
          if (exact) unscaled(rt, ri, idiag ? idiag[i] : 1.f);
        }
      }
    };
    ++it;
    auto decide = [&](double trr, double trt) {
      if (keep_p) {
        // the segment ends: |r|^2 of the new residual for the record; the old one stays in
        // S_RRH for the direction the host keeps
        sd[5] = trr;
        si[2] = si[0] != FLAG_NONE ? si[0] : FLAG_UPDATE;
        return;
      }
      sd[0] = trr;
      // norms compared as squares (no square root on the path)
      int pend = FLAG_NONE;
      if (!(trr <= 1e8 * sd[1])) pend = FLAG_BREAK;  // NaN fails too
      else if (exact && trt <= sd[3]) pend = FLAG_CHECK;
      else if (trr < sd[2] * sd[1]) pend = FLAG_UPDATE;
      else if (it + 1 >= maxit) pend = FLAG_MAXIT;
      if (trr > sd[1]) sd[1] = trr;
      si[0] = pend;
    };
    bool ok;
    if (exact) {
      ok = grid_reduce<2, float2>(
          sh, g, 1, target, &si[3], vb,
          [&](int blk, float2 (&v)[2]) {
            Acc<float> rr, rt;
            update(blk, rr, rt);
            v[0] = make_float2(rr.hi, rr.lo);
            v[1] = make_float2(rt.hi, rt.lo);
          },
          [&](double (&t)[2]) { decide(t[0], t[1]); });
    } else {
      ok = grid_reduce<1, float2>(
          sh, g, 1, target, &si[3], vb,
          [&](int blk, float2 (&v)[1]) {
            Acc<float> rr, rt;
            update(blk, rr, rt);
            v[0] = make_float2(rr.hi, rr.lo);
          },
          [&](double (&t)[1]) { decide(t[0], 0.0); });
    }
    if (!ok) return;
    if (si[2] != FLAG_NONE) break;
  }
  if (R > 0) {
#pragma unroll
    for (int k = 0; k < RR; ++k)
      if (ref[k].vec >= 0) {
        x[ref[k].vec] = rx[k];
        r[ref[k].vec] = rr_[k];
      }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S[S_ALPHA] = sd[6];
    S[S_BETA] = sd[7];
    S[S_RRH] = sd[0];
    S[S_RMAX] = sqrt(sd[1]);
    S[S_APP] = sd[5];
    I[I_ITER] = it;
    I[I_PEND] = si[0];
    I[I_SKIPP] = si[1];
    if (si[2] != FLAG_NONE) {
      I[I_FLAG] = si[2];
      I[I_DONE] = 1;
    }
  }
}

// y = A x (MODE 0) or y = b - A x with its norm (MODE 2) in the cell-block layout
template <typename T, int MODE>
__global__ void __launch_bounds__(RB)
    k_dg_spmv(MatArgs<T> m, const T* x, T* __restrict__ y, const double* __restrict__ b, RedBuf rb, double* S) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  Acc<T> dot;
  for (int64_t s = warp; s < m.nslices; s += nwarps) {
    SliceRef<T, ML_DG> r;
    r.load(m, s, lane, nullptr);
    const T a = r.template dot<false, kUnroll>(x);
    if (r.vec < 0) continue;
    if (MODE == 2) {
      const T rr = (T)(b[r.vec] - (double)a);
      y[r.vec] = rr;
      dot.add(rr, rr);
    } else {
      y[r.vec] = a;
    }
  }
  if (MODE == 0) return;
  double v[1] = {dot.value()}, tot[1];
  if (block_reduce_last<1>(v, rb, tot) && threadIdx.x == 0) S[S_ERR] = sqrt(tot[0]);
}

// FP32 copy of S A S in the cell-block layout (padding stays 0)
__global__ void __launch_bounds__(RB) k_scale_dg32(MatArgs<double> m, const double* __restrict__ sd, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * RB + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * RB) >> 5;
  for (int64_t s = warp; s < m.nslices; s += nwarps) {
    SliceRef<double, ML_DG> r;
    r.load(m, s, lane, nullptr);
    const double srow = r.vec >= 0 ? sd[r.vec] : 0.0;
    const double* v0 = r.vp;
    for (int k = 0; k < 7; ++k) {
      const double* sb = sd + r.cp[k];
      for (int j = 0; j < r.w4; ++j, v0 += 128) {
        double v[4];
        ld4(v0, v);
        float4 f;
        f.x = (float)(v[0] * (srow * sb[4 * j]));
        f.y = (float)(v[1] * (srow * sb[4 * j + 1]));
        f.z = (float)(v[2] * (srow * sb[4 * j + 2]));
        f.w = (float)(v[3] * (srow * sb[min(4 * j + 3, m.nn - 1)]));
        *reinterpret_cast<float4*>(out + (v0 - m.val)) = f;
      }
    }
  }
}

// inverse diagonal in the solver layout (extract_diagonal by binary search,
// csr_sparse_matrix.f90:4231-4256); entries of non-free vector slots stay 0
__global__ void k_inv_diag(int64_t n, const int64_t* rp, const int32_t* ci, const double* av, const int32_t* row2vec,
                           double* d64, float* d32) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  int64_t lo = rp[r], hi = rp[r + 1];
  while (lo < hi) {
    int64_t m = (lo + hi) >> 1;
    if (ci[m] < r) lo = m + 1;
    else hi = m;
  }
  const double d = (lo < rp[r + 1] && ci[lo] == r) ? av[lo] : 0.0;
  const double inv = 1.0 / d;
  const int32_t v = row2vec[r];
  d64[v] = inv;
  d32[v] = (float)inv;
}

// row order <-> solver layout
template <typename TS, typename TD>
__global__ void k_rows_to_vec(int64_t n, const int32_t* __restrict__ row2vec, const TS* __restrict__ src,
                              TD* __restrict__ dst) {
  int64_t r = blockIdx.x * (int64_t)RB + threadIdx.x;
  if (r < n) dst[row2vec[r]] = (TD)src[r];
}
template <typename TS, typename TD>
__global__ void k_vec_to_rows(int64_t n, const int32_t* __restrict__ row2vec, const TS* __restrict__ src,
                              TD* __restrict__ dst) {
  int64_t r = blockIdx.x * (int64_t)RB + threadIdx.x;
  if (r < n) dst[r] = (TD)src[row2vec[r]];
}
template <typename T>
__global__ void k_fill(int64_t n, T* a, T v) {
  int64_t i = blockIdx.x * (int64_t)RB + threadIdx.x;
  if (i < n) a[i] = v;
}
__global__ void k_set_scalar(double* S, int slot, double v) { S[slot] = v; }

static inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

struct Work {
  double *x, *r, *p, *Ap, *b, *t;  // FP64, solver layout
  float *x32, *r32, *p32, *Ap32;
  double* S;
  int* I;
  RedBuf rb;
  int sms;
};

// Grid of a grid-stride kernel: exactly the blocks that are co-resident (one wave), from
// the occupancy of that kernel.  Every block does the same share of the work, so a
// second wave would double the kernel's time; the grid is fixed per kernel, which keeps
// the block-partial reductions deterministic.
static unsigned grid_for(const void* k, int sms) {
  static std::mutex mu;
  static std::map<const void*, unsigned> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(k);
  if (it != cache.end()) return it->second;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, RB, 0) != cudaSuccess) { cudaGetLastError(); nb = 1; }
  if (nb < 1) nb = 1;
  if (nb > 8) nb = 8;
  const unsigned g = (unsigned)(nb * sms);
  cache[k] = g;
  return g;
}

template <typename... KA, typename... A>
static inline void launch_k(void (*k)(KA...), const Work& w, cudaStream_t st, A... args) {
  k<<<grid_for((const void*)k, w.sms), RB, 0, st>>>(args...);
}
// the same for `threads` threads of work: no more blocks than they fill (a reducing kernel's
// blocks each take a ticket, 15 us of them at 1216 blocks)
template <typename... KA, typename... A>
static inline void launch_kn(void (*k)(KA...), const Work& w, cudaStream_t st, int64_t threads, A... args) {
  const unsigned need = (unsigned)std::max<int64_t>(1, (threads + RB - 1) / RB);
  k<<<std::min(grid_for((const void*)k, w.sms), need), RB, 0, st>>>(args...);
}

static fg_status ensure_work(fg_system* sys, Work& w) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  // vector stride a multiple of 4 entries: every FP32 vector starts on a 16-byte boundary
  // (the FP32 update kernels load float4)
  const int64_t n = ((sp->nvec > 0 ? sp->nvec : 1) + 3) & ~(int64_t)3;
  if (!sys->d_work) {
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_work, sizeof(double) * 6 * n));
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_work32, sizeof(float) * 4 * n));
    // entries of non-free vector slots must read zero for the whole life of the buffers
    FG_CUDA_TRY(cudaMemsetAsync(sys->d_work, 0, sizeof(double) * 6 * n, ctx->stream));
    FG_CUDA_TRY(cudaMemsetAsync(sys->d_work32, 0, sizeof(float) * 4 * n, ctx->stream));
    sys->red_blocks = ctx->sm_count * 8;
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_red, sizeof(double) * (4 * sys->red_blocks + S_COUNT) + sizeof(int) * I_COUNT));
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_ticket, sizeof(unsigned) * 4));
    FG_CUDA_TRY(cudaMemsetAsync(sys->d_ticket, 0, sizeof(unsigned) * 4, ctx->stream));
  }
  w.x = sys->d_work; w.r = w.x + n; w.p = w.r + n; w.Ap = w.p + n; w.b = w.Ap + n; w.t = w.b + n;
  w.x32 = sys->d_work32; w.r32 = w.x32 + n; w.p32 = w.r32 + n; w.Ap32 = w.p32 + n;
  w.S = sys->d_red + 4 * sys->red_blocks;
  w.I = (int*)(w.S + S_COUNT);
  w.rb.part = sys->d_red;
  w.rb.ticket = sys->d_ticket;
  w.rb.nblocks = sys->red_blocks;
  w.sms = ctx->sm_count;
  return FG_OK;
}

fg_status system_prepare_diag(fg_system* sys) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  const int64_t n = sp->nfree, nv = sp->nvec > 0 ? sp->nvec : 1;
  if (!sys->d_idiag) {
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_idiag, sizeof(double) * nv));
    FG_TRY(dev_alloc(ctx, (void**)&sys->d_idiag32, sizeof(float) * nv));
    FG_CUDA_TRY(cudaMemsetAsync(sys->d_idiag, 0, sizeof(double) * nv, ctx->stream));
    FG_CUDA_TRY(cudaMemsetAsync(sys->d_idiag32, 0, sizeof(float) * nv, ctx->stream));
  }
  if (sp->layout == FG_LAYOUT_STENCIL && sys->d_tval) return system_inv_diag_stencil(sys);
  if (n > 0) {
    ctx->launches += 1;
    k_inv_diag<<<nblk(n, 256), 256, 0, ctx->stream>>>(n, sp->d_rowptr, sp->d_col, sys->d_val, sp->d_row2vec,
                                                       sys->d_idiag, sys->d_idiag32);
    FG_CUDA_TRY(cudaGetLastError());
  }
  return FG_OK;
}

static int mat_layout(const fg_space* sp) {
  return sp->layout == FG_LAYOUT_STENCIL ? ML_STENCIL : (sp->d_dgblk ? ML_DG : ML_SELL);
}

// matrix arguments of the CG kernels
template <typename T>
static MatArgs<T> mat_args(const fg_space* sp, const T* vals) {
  MatArgs<T> m;
  const bool stencil = sp->layout == FG_LAYOUT_STENCIL;
  m.nslices = stencil ? sp->st_nslices : sp->nslices;
  m.n = sp->nfree;
  m.val = vals;
  m.scls = sp->d_st_scls;
  m.voff = sp->d_st_voff;
  m.cls = sp->d_st_cls;
  m.soff = sp->d_st_off;
  m.st_row = sp->d_st_row;
  m.ncomp = sp->ncomp;
  m.noff = 0;
  if (stencil)
    for (const StencilClass& C : sp->h_st_cls) m.noff += C.Bp;
  m.sptr = sp->d_sptr;
  m.scol = sp->d_scol;
  m.blk = sp->d_dgblk;
  m.nn = sp->tab.nn;
  return m;
}

// SpMV of the active solver layout on solver-layout vectors
template <typename T, int MODE>
static void spmv_k(fg_system* sys, const Work& w, const T* x, T* y, const double* b, cudaStream_t st);

#define FG_SPMV_IMPL(T, MODE, VALS, TVALS)                                                                          \
  template <>                                                                                                       \
  void spmv_k<T, MODE>(fg_system * sys, const Work& w, const T* x, T* y, const double* b, cudaStream_t st) {       \
    fg_space* sp = sys->space;                                                                                      \
    if (sp->layout == FG_LAYOUT_STENCIL)                                                                            \
      launch_kn(k_stencil_spmv<T, MODE>, w, st, sp->st_nslices * 32, sp->st_nslices, (const uint8_t*)sp->d_st_scls,                       \
               (const int64_t*)sp->d_st_voff, (const StencilClass*)sp->d_st_cls, (const int32_t*)sp->d_st_off, (const int32_t*)sp->d_st_row,       \
               (const T*)sys->TVALS, sp->ncomp, x, y, b, w.rb, w.S);                                                \
    else if (sp->d_dgblk)                                                                                           \
      launch_kn(k_dg_spmv<T, MODE>, w, st, sp->nslices * 32, mat_args<T>(sp, sys->VALS), x, y, b, w.rb, w.S);       \
    else                                                                                                            \
      launch_kn(k_sell_spmv<T, MODE>, w, st, sp->nslices * 32, sp->nslices, sp->nfree, (const int64_t*)sp->d_sptr,                     \
               (const int32_t*)sp->d_scol, (const T*)sys->VALS, x, y, b, w.rb, w.S);                               \
    sp->mesh->ctx->launches += 1;                                                                                   \
  }
FG_SPMV_IMPL(double, 0, d_sval, d_tval)
FG_SPMV_IMPL(double, 2, d_sval, d_tval)
FG_SPMV_IMPL(float, 0, d_sval32, d_tval32)
#undef FG_SPMV_IMPL

// D^-1/2 and the FP32 copy of D^-1/2 A D^-1/2 (once per numeric assembly)
static fg_status ensure_scaled(fg_system* sys, const Work& w) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  if (sys->scaled_valid) return FG_OK;
  const bool stencil = sp->layout == FG_LAYOUT_STENCIL;
  const int64_t nvals = stencil ? sp->st_nvals : sp->sell_nnz;
  const double* v64 = stencil ? sys->d_tval : sys->d_sval;
  if (!v64) { set_error("the FP64 solver-layout values are not available"); return FG_ERR_UNSUPPORTED; }
  const int64_t nv = sp->nvec > 0 ? sp->nvec : 1;
  if (!sys->d_sdiag) FG_TRY(dev_alloc(ctx, (void**)&sys->d_sdiag, sizeof(double) * nv));
  if (!sys->d_val32s) FG_TRY(dev_alloc(ctx, (void**)&sys->d_val32s, sizeof(float) * (nvals > 0 ? nvals : 1)));
  cudaStream_t st = ctx->stream;
  launch_k(k_sqrt_idiag, w, st, nv, (const double*)sys->d_idiag, sys->d_sdiag);
  if (stencil)
    launch_k(k_scale_stencil32, w, st, sp->st_nslices, (const uint8_t*)sp->d_st_scls, (const int64_t*)sp->d_st_voff,
             (const StencilClass*)sp->d_st_cls,
             (const int32_t*)sp->d_st_off, (const int32_t*)sp->d_st_row, v64, (const double*)sys->d_sdiag, sp->ncomp,
             sys->d_val32s);
  else if (sp->d_dgblk)
    launch_k(k_scale_dg32, w, st, mat_args<double>(sp, v64), (const double*)sys->d_sdiag, sys->d_val32s);
  else
    launch_k(k_scale_sell32, w, st, sp->nslices, sp->nfree, (const int64_t*)sp->d_sptr, (const int32_t*)sp->d_scol, v64,
             (const double*)sys->d_sdiag, sys->d_val32s);
  ctx->launches += 2;
  FG_CUDA_TRY(cudaGetLastError());
  sys->scaled_valid = true;
  return FG_OK;
}

// y = A x in row order (device pointers): into the solver layout, SpMV, back.
fg_status system_spmv(fg_system* sys, int precision, const void* x, void* y, cudaStream_t st) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  Work w;
  FG_TRY(ensure_work(sys, w));
  const int64_t n = sp->nfree;
  if (n == 0) return FG_OK;
  if (precision == FG_MIXED) {
    k_rows_to_vec<float, float><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, (const float*)x, w.p32);
    spmv_k<float, 0>(sys, w, w.p32, w.Ap32, nullptr, st);
    k_vec_to_rows<float, float><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, w.Ap32, (float*)y);
  } else {
    k_rows_to_vec<double, double><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, (const double*)x, w.p);
    spmv_k<double, 0>(sys, w, w.p, w.Ap, nullptr, st);
    k_vec_to_rows<double, double><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, w.Ap, (double*)y);
  }
  ctx->launches += 2;
  FG_CUDA_TRY(cudaGetLastError());
  return FG_OK;
}

// reps launches of the solver-layout SpMV alone on solver-layout vectors (timing)
fg_status system_spmv_slot(fg_system* sys, int precision, const void* x, void* y, int reps, cudaStream_t st) {
  Work w;
  FG_TRY(ensure_work(sys, w));
  if (sys->space->nfree == 0) return FG_OK;
  for (int k = 0; k < reps; ++k) {
    if (precision == FG_MIXED) spmv_k<float, 0>(sys, w, (const float*)x, (float*)y, nullptr, st);
    else spmv_k<double, 0>(sys, w, (const double*)x, (double*)y, nullptr, st);
  }
  FG_CUDA_TRY(cudaGetLastError());
  return FG_OK;
}

int64_t system_vec_len(fg_system* sys) { return sys->space->nvec; }

// One SpMV of the active solver layout on caller-provided solver-layout vectors, without
// touching the system's work buffers (no allocation).  The MODE 0 kernels take no
// reduction buffers.
fg_status system_spmv_layout_noalloc(fg_system* sys, int precision, const void* xvec, void* yvec, cudaStream_t st) {
  Work w;
  std::memset(&w, 0, sizeof(w));
  w.sms = sys->space->mesh->ctx->sm_count;
  if (sys->space->nfree == 0) return FG_OK;
  if (precision == FG_MIXED) spmv_k<float, 0>(sys, w, (const float*)xvec, (float*)yvec, nullptr, st);
  else spmv_k<double, 0>(sys, w, (const double*)xvec, (double*)yvec, nullptr, st);
  FG_CUDA_TRY(cudaGetLastError());
  return FG_OK;
}

// Launch shape of the CG kernels.  One block per SM, a slice per warp while the warps suffice
// (32 per SM): its lanes' vector entries stay in registers.  Up to 16 slices fit one block,
// whose barriers are block barriers (8^3 Q1: 8.7 us per iteration, 11.4 with 4 blocks, 12.9
// with 11).  Twice the slices take two per warp (23 x 17 x 21 Q3 in FP64: 85 us per iteration
// against 103 streaming; four per warp 120).  Beyond that two blocks per SM stream the vectors:
// four slices per warp were slower there too (unstructured 40^3 Q2, 15.4 k slices: 136-144 us
// against 92).
struct PcgShape {
  int R;
  unsigned blocks, threads;
};
static PcgShape pcg_shape(int64_t nslices, int64_t value_bytes, bool fp32, int ml, int sms) {
  const int64_t cap = (int64_t)sms * 32;
  // FP32 with two slices per warp only while the matrix stays in L2: streaming it wants the 48
  // warps and the prefetch (dG 20^3 Q2, 169 MB: 38 us per iteration against 64; 19^3 Q3, 150 MB: 45
  // against 48; 34^3 Q2, 80 MB: 36 against 29).  FP64 is bound by its pipe there (103 against 90).
  const bool streams = fp32 && nslices > cap && value_bytes > (int64_t)112 << 20;
  if (nslices > 2 * cap || streams) {
    const int R = !fp32 && ml == ML_SELL && value_bytes > (int64_t)170 << 20 ? PCG_WIDE : 0;  // 1.5 x that with columns
    return PcgShape{R, (unsigned)(2 * sms), (unsigned)pcg_threads(R, ml, fp32)};
  }
  const int R = nslices <= cap ? 1 : 2;
  const int64_t warps = std::max<int64_t>(1, (nslices + R - 1) / R);
  const int64_t blocks = warps <= 16 ? 1 : std::min<int64_t>(sms, warps);
  return PcgShape{R, (unsigned)blocks, (unsigned)(32 * ((warps + blocks - 1) / blocks))};
}

// keep: groups of 4 x 32 matrix entries (of `bytes` each) that a block holds in shared memory for the
// launch: its share of the matrix, or what fits beside the class offsets and the kernel's own
// (24^3 Q2 mixed 16.1 -> 15.5 us per iteration, 23 x 17 x 21 Q3 FP64 81 -> 73, the widest slices').
// Not where the vectors are streamed: the gathers want the L1 (unstructured 40^3 Q2 89 -> 112).
template <typename... KA>
static fg_status pcg_keep(void (*k)(KA...), const PcgShape& sh, int noff, int64_t entries, int bytes, int* keep,
                          size_t* smem) {
  *smem = sizeof(int32_t) * (size_t)((noff + 3) & ~3);
  cudaFuncAttributes fa;
  FG_CUDA_TRY(cudaFuncGetAttributes(&fa, (const void*)k));
  int dev = 0, most = 0;
  FG_CUDA_TRY(cudaGetDevice(&dev));
  FG_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const int64_t limit = (int64_t)most - (int64_t)fa.sharedSizeBytes;
  // the same limit on every call: contexts on other threads launch this kernel with other sizes
  FG_CUDA_TRY(cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  *keep = 0;
  if (sh.R > 0) {
    // slices are dealt out block by block; a block may have one more of each kind than another
    const int64_t share = entries / 128 / sh.blocks * 5 / 4 + 64;
    *keep = (int)std::max<int64_t>(0, std::min((limit - (int64_t)*smem) / (128 * bytes), share));
    *smem += (size_t)*keep * 128 * bytes;
  }
  return FG_OK;
}

template <typename... KA>
static fg_status launch_pcg(void (*k)(KA...), const PcgShape& sh, int vblocks, const Work& w, size_t smem, cudaStream_t st,
                            void** args) {
  FG_CUDA_TRY(cudaMemsetAsync(w.rb.ticket + 1, 0, sizeof(unsigned), st));
  FG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k, dim3(sh.blocks / vblocks), dim3(sh.threads), args, smem, st));
  return FG_OK;
}

// Blocks of a solve per block of the launch.  A streaming solve's 2 x SMs blocks fill the SMs, so those of
// several contexts would take turns; while another context of the device solves, a launch is half as wide
// and its blocks do two of the solve's each, so that two solves share the SMs and fill one another's waits.
// The sums are the same blocks' in the same order: the same bits.  Alone, half the warps cost 15-25 %
// (96^3 Q2 mixed 361 -> 480 us per iteration); two contexts at once solve 24^3 Q2 elasticity 11.9 times a
// second against 10.0 in turn, 64^3 Q2 Poisson 18.1 against 17.5, 48^3 in FP64 22.5 against 21.5.
// FG_PCG_TEST_SHARE=1: always (tests).
static int pcg_vblocks(const fg_ctx* ctx, const PcgShape& sh) {
  if (sh.R > 0) return 1;
  const char* e = getenv("FG_PCG_TEST_SHARE");
  if (e && e[0] == '1') return 2;
  return ctx->load->solving.load(std::memory_order_relaxed) > 1 ? 2 : 1;
}

// Iterations of one launch: the caller's polling interval; or about 5 ms, at least 16 iterations while they
// stay under 15 ms (a launch costs ~20 us of host time: 0.3 % of a 128^3 Q2 step in launches of 5 ms); or about 1 ms
// while another thread is in a call on the device, as a launch holds the SMs and every kernel and host
// synchronisation of a small solve beside it waits for its end.  (Launches of at least 16 iterations, 50 ms at
// 96^3 Q2 elasticity, gave a server's mix a median latency of 237 ms; kernels in a graph 161; this 97-113.)  The
// iterates do not depend on it.
static int pcg_iters(const fg_ctx* ctx, const fg_solver_params* prm, int64_t entries, int64_t nvec, int width) {
  if (prm->check_every > 0) return prm->check_every;
  if (const char* e = getenv("FG_PCG_TEST_LAUNCH_ITERS")) return std::max(1, atoi(e));  // tests
  const double us = 8.0 + ((double)entries + 10.0 * (double)nvec) * width / 5.5e6;
  const bool beside = ctx->load->running.load(std::memory_order_relaxed) > 1;
  const double n = beside ? 1000.0 / us : std::max(5000.0 / us, std::min(16.0, 15000.0 / us));
  return (int)std::min(1024.0, std::max(1.0, n));
}

// scalars and flags of the solve, copied to the host in one piece
struct SolveState {
  double S[S_COUNT];
  int I[I_COUNT];
};
static fg_status read_state(const Work& w, SolveState& h, cudaStream_t st) {
  static_assert(sizeof(SolveState) == sizeof(double) * S_COUNT + sizeof(int) * I_COUNT, "the device keeps I after S");
  FG_CUDA_TRY(cudaMemcpyAsync(&h, w.S, sizeof(h), cudaMemcpyDeviceToHost, st));
  FG_CUDA_TRY(cudaStreamSynchronize(st));
  if (h.I[I_ABORT]) {
    set_error("the CG kernel's grid barrier ran out of time");
    return FG_ERR_TIMEOUT;
  }
  return FG_OK;
}

// grid barriers of the CG kernels: bounded at 10 s, or FG_PCG_BARRIER_TIMEOUT_MS (read per solve; a value
// that is not a positive number of milliseconds changes nothing)
static GridSync grid_sync(const Work& w) {
  unsigned long long ms = 10000;
  if (const char* e = getenv("FG_PCG_BARRIER_TIMEOUT_MS")) {
    char* end = nullptr;
    const long long v = strtoll(e, &end, 10);
    if (end != e && *end == 0 && v > 0) ms = (unsigned long long)std::min<long long>(v, 86400000);
  }
  const char* drop = getenv("FG_PCG_TEST_DROP_ARRIVAL");
  return GridSync{w.rb.part, w.rb.ticket + 1, w.I + I_ABORT, ms * 1000000ull, drop ? atoi(drop) : 0};
}

static int64_t solver_entries(const fg_space* sp) {
  return sp->layout == FG_LAYOUT_STENCIL ? sp->st_nvals : sp->sell_nnz;
}

// FP64 CG from the state k_init64 left, until it is done.
static fg_status run_pcg64(fg_system* sys, const Work& w, const fg_solver_params* prm, int criterion, double rtol,
                           double atol, int chunk, SolveState& h, cudaStream_t st) {
  fg_space* sp = sys->space;
  const int ml = mat_layout(sp);
  MatArgs<double> m = mat_args<double>(sp, ml == ML_STENCIL ? sys->d_tval : sys->d_sval);
  const PcgShape sh = pcg_shape(m.nslices, 8 * solver_entries(sp), false, ml, w.sms);
  int64_t nvec = sp->nvec;
  double *x = w.x, *r = w.r, *p = w.p, *Ap = w.Ap;
  const double* idiag = prm->precond == FG_PREC_JACOBI ? sys->d_idiag : nullptr;
  int iters = 0;
  GridSync g = grid_sync(w);
  double* S = w.S;
  int* I = w.I;
  int keep = 0;
  size_t smem = 0;
  int vb = 1;
  void* args[] = {&m, &nvec, &x, &r, &p, &Ap, &idiag, &criterion, &rtol, &atol, &iters, &chunk, &keep, &vb, &g, &S, &I};
#define FG_PCG64(L) (sh.R == 1 ? k_pcg64<L, 1> : sh.R == 2 ? k_pcg64<L, 2> : k_pcg64<L, 0>)
  auto k = ml == ML_STENCIL ? FG_PCG64(ML_STENCIL) : ml == ML_DG ? FG_PCG64(ML_DG) : sh.R == PCG_WIDE ? k_pcg64<ML_SELL, PCG_WIDE> : FG_PCG64(ML_SELL);
#undef FG_PCG64
  FG_TRY(pcg_keep(k, sh, m.noff, solver_entries(sp), 8, &keep, &smem));
  for (;;) {
    vb = pcg_vblocks(sp->mesh->ctx, sh);
    iters = pcg_iters(sp->mesh->ctx, prm, solver_entries(sp), nvec, 8);
    FG_TRY(launch_pcg(k, sh, vb, w, smem, st, args));
    sp->mesh->ctx->launches += 1;
    FG_TRY(read_state(w, h, st));
    if (h.I[I_DONE]) return FG_OK;
    // (a launch may end inside a chunk)
    if ((!std::isfinite(h.S[S_ALPHA]) || !std::isfinite(h.S[S_RZ])) &&
        chunk_ends_before(h.I[I_ITER], chunk, h.I[I_MAXIT])) {
      set_error("non-finite CG scalars");
      return FG_ERR_NUMERIC;
    }
  }
}

// FP32 iterations of the mixed path until the segment ends.
static fg_status run_pcg32(fg_system* sys, const Work& w, const fg_solver_params* prm, const float* vals,
                           const float* idiag, SolveState& h, cudaStream_t st) {
  fg_space* sp = sys->space;
  const int ml = mat_layout(sp);
  MatArgs<float> m = mat_args<float>(sp, vals);
  const PcgShape sh = pcg_shape(m.nslices, 4 * solver_entries(sp), true, ml, w.sms);
  int64_t nvec = sp->nvec;
  float *x = w.x32, *r = w.r32, *p = w.p32, *q = w.Ap32;
  // (the first segment of a solve starts with no state on the host)
  int iters = 0, phase = 0, last_exact = prm->check_every > 0 ? 1 : 0;
  const int it0 = h.I[I_ITER];
  GridSync g = grid_sync(w);
  double* S = w.S;
  int* I = w.I;
  int keep = 0;
  size_t smem = 0;
  int vb = 1;
  void* args[] = {&m, &nvec, &x, &r, &p, &q, &idiag, &iters, &phase, &last_exact, &keep, &vb, &g, &S, &I};
#define FG_PCG32(L) (sh.R == 1 ? k_pcg32<L, 1> : sh.R == 2 ? k_pcg32<L, 2> : k_pcg32<L, 0>)
  auto k = ml == ML_STENCIL ? FG_PCG32(ML_STENCIL) : ml == ML_DG ? FG_PCG32(ML_DG) : FG_PCG32(ML_SELL);
#undef FG_PCG32
  FG_TRY(pcg_keep(k, sh, m.noff, solver_entries(sp), 4, &keep, &smem));
  do {
    vb = pcg_vblocks(sp->mesh->ctx, sh);
    iters = pcg_iters(sp->mesh->ctx, prm, solver_entries(sp), nvec, 4);
    FG_TRY(launch_pcg(k, sh, vb, w, smem, st, args));
    sp->mesh->ctx->launches += 1;
    FG_TRY(read_state(w, h, st));
    if (!last_exact) phase = (h.I[I_ITER] - it0) % FG_MIXED_EXACT_EVERY;
  } while (!h.I[I_DONE]);
  return FG_OK;
}

fg_status system_solve(fg_system* sys, const fg_solver_params* prm, const double* d_b, const double* d_x0,
                       double* d_x, fg_solve_info* info) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  const SolveScope solving(ctx->load);
  cudaStream_t st = ctx->stream;
  const int64_t n = sp->nfree, nv = sp->nvec;
  fg_solve_info out;
  std::memset(&out, 0, sizeof(out));
  if (n == 0) {
    out.converged = 1;
    if (info) *info = out;
    return FG_OK;
  }
  Work w;
  FG_TRY(ensure_work(sys, w));
  if (!sys->d_idiag) FG_TRY(system_prepare_diag(sys));
  const double* b_row = d_b ? d_b : sys->d_rhs;
  const int precond = prm->precond == FG_PREC_JACOBI ? 1 : 0;
  const int chunk = prm->check_every > 0 ? prm->check_every : (n < 200000 ? 64 : 16);
  SolveState h;
  std::memset(&h, 0, sizeof(h));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, st);
  const int64_t launches0 = ctx->launches;
  fg_status status = FG_OK;
  // right-hand side and initial guess into the solver layout (other entries are zero)
  k_rows_to_vec<double, double><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, b_row, w.b);
  if (d_x0) k_rows_to_vec<double, double><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, d_x0, w.x);
  else k_fill<double><<<nblk(nv, RB), RB, 0, st>>>(nv, w.x, 0.0);
  ctx->launches += 2;
  FG_CUDA_TRY(cudaGetLastError());
  FG_CUDA_TRY(cudaMemsetAsync(w.I, 0, sizeof(int) * I_COUNT, st));
  if (prm->precision == FG_FP64) {
    if (d_x0) spmv_k<double, 0>(sys, w, w.x, w.r, nullptr, st);
    launch_kn(k_init64, w, st, nv, nv, (const double*)w.b, d_x0 ? 1 : 0, w.r, w.p, (const double*)sys->d_idiag, precond,
              prm->criterion, prm->rtol, prm->atol, prm->max_iters, w.rb, w.S, w.I);
    ctx->launches += 1;
    FG_CUDA_TRY(cudaGetLastError());
    status = run_pcg64(sys, w, prm, prm->criterion, prm->rtol, prm->atol, chunk, h, st);
    out.iterations = h.I[I_ITER];
    out.converged = h.I[I_CONV];
    out.error_estimate = h.S[S_ERR];
    out.tolerance = h.S[S_TOL];
  } else {
    const double delta = prm->inner_rtol > 0 ? prm->inner_rtol : 0.1;
    // true residual of the initial guess and the tolerance
    spmv_k<double, 2>(sys, w, w.x, w.r, w.b, st);
    FG_TRY(read_state(w, h, st));
    double rn = h.S[S_ERR];
    double tol;
    if (prm->criterion == FG_RES_RHS) {
      launch_kn(k_init64, w, st, nv, nv, (const double*)w.b, 0, w.t, w.Ap, (const double*)sys->d_idiag, 0,
                (int)FG_RES_RHS, prm->rtol, prm->atol, 1, w.rb, w.S, w.I);
      ctx->launches += 1;
      FG_TRY(read_state(w, h, st));
      tol = prm->rtol * h.S[S_BNRM] + prm->atol;
      spmv_k<double, 2>(sys, w, w.x, w.r, w.b, st);
    } else {
      tol = prm->rtol * rn + prm->atol;
    }
    int outer = 0, stalls = 0, polish_its = 0;
    bool polish = false;
    double rn_prev = rn;
    if (!std::isfinite(rn)) {
      status = FG_ERR_NUMERIC;
      set_error("non-finite initial residual");
    } else if (rn <= tol) {
      out.converged = 1;
    } else {
      k_set_scalar<<<1, 1, 0, st>>>(w.S, S_TOL, tol);
      k_set_scalar<<<1, 1, 0, st>>>(w.S, S_DELTA, delta);
      k_set_scalar<<<1, 1, 0, st>>>(w.S, S_SIGMA, rn);
      k_fill<float><<<nblk(nv, RB), RB, 0, st>>>(nv, w.x32, 0.0f);
      k_fill<float><<<nblk(nv, RB), RB, 0, st>>>(nv, w.p32, 0.0f);
      ctx->launches += 5;
      int hI0[I_COUNT] = {0};
      hI0[I_MAXIT] = prm->max_iters;
      FG_CUDA_TRY(cudaMemcpyAsync(w.I, hI0, sizeof(hI0), cudaMemcpyHostToDevice, st));
      // FP32 segments on D^-1/2 A D^-1/2 (Jacobi) or A (no preconditioner)
      const double* sd = nullptr;
      const float* vals32 = sp->layout == FG_LAYOUT_STENCIL ? sys->d_tval32 : sys->d_sval32;
      const float* id32 = nullptr;
      if (precond) {
        FG_TRY(ensure_scaled(sys, w));
        sd = sys->d_sdiag;
        vals32 = sys->d_val32s;
        id32 = sys->d_idiag32;
      }
      auto refresh = [&](int first) {
        launch_kn(k_refresh_scaled, w, st, nv, nv, (const double*)w.r, sd, w.r32, first, w.rb, w.S, w.I);
        launch_kn(k_pupdate, w, st, (nv + 3) / 4, nv, w.p32, (const float*)w.r32, (const double*)w.S);
        ctx->launches += 2;
      };
      refresh(1);
      FG_CUDA_TRY(cudaGetLastError());
      // FP32 segments; reliable updates on the host's cue
      for (;;) {
        status = run_pcg32(sys, w, prm, vals32, id32, h, st);
        if (status != FG_OK) break;
        // reliable update: fold the FP32 correction into x64 and recompute the true residual
        // (after a breakdown the segment's correction is dropped instead)
        const bool broke = h.I[I_FLAG] == FLAG_BREAK;
        if (broke) k_fill<float><<<nblk(nv, RB), RB, 0, st>>>(nv, w.x32, 0.0f);
        else launch_kn(k_fold_scaled, w, st, nv, nv, h.S[S_SIGMA], sd, w.x32, w.x);
        ctx->launches += 1;
        spmv_k<double, 2>(sys, w, w.x, w.r, w.b, st);
        ++outer;
        FG_TRY(read_state(w, h, st));
        rn = h.S[S_ERR];
        if (!std::isfinite(rn)) { status = FG_ERR_NUMERIC; set_error("non-finite residual"); break; }
        if (rn <= tol) { out.converged = 1; break; }
        if (h.I[I_ITER] >= prm->max_iters) break;
        // FP32 segments aim at a 10x reduction of the true residual; a breakdown, or two
        // segments in a row that gain less than 2x (FP32 rounding of an ill-conditioned
        // matrix near a tight tolerance), hand the rest of the solve to the FP64 PCG
        stalls = rn > 0.5 * rn_prev ? stalls + 1 : 0;
        rn_prev = rn;
        if (broke || stalls >= 2) { polish = true; break; }
        refresh(0);
        FG_CUDA_TRY(cudaGetLastError());
      }
      if (polish && status == FG_OK) {
        // FP64 PCG from x64 to the same absolute tolerance, with the iterations left
        const int mixed_its = h.I[I_ITER];
        spmv_k<double, 0>(sys, w, w.x, w.r, nullptr, st);
        launch_kn(k_init64, w, st, nv, nv, (const double*)w.b, 1, w.r, w.p, (const double*)sys->d_idiag, precond,
                  (int)FG_RES_RES, 0.0, tol, std::max(prm->max_iters - mixed_its, 1), w.rb, w.S, w.I);
        ctx->launches += 1;
        FG_CUDA_TRY(cudaGetLastError());
        status = run_pcg64(sys, w, prm, (int)FG_RES_RES, 0.0, tol, chunk, h, st);
        polish_its = h.I[I_ITER];
        out.converged = h.I[I_CONV];
        rn = h.S[S_ERR];
        h.I[I_ITER] = mixed_its;
      }
    }
    out.iterations = h.I[I_ITER] + polish_its;
    out.outer_iterations = outer;
    out.error_estimate = rn;
    out.tolerance = tol;
  }
  // solution back to row order
  k_vec_to_rows<double, double><<<nblk(n, RB), RB, 0, st>>>(n, sp->d_row2vec, w.x, d_x);
  ctx->launches += 1;
  FG_CUDA_TRY(cudaGetLastError());
  cudaEventRecord(e1, st);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  out.solve_ms = ms;
  out.kernel_launches = ctx->launches - launches0;
  if (info) *info = out;
  if (status == FG_OK && !out.converged) status = FG_ERR_NOT_CONVERGED;
  return status;
}

}  // namespace fg
