// fg_batch.cu -- many independent Poisson problems assembled and solved in one persistent launch.
//
// Each problem: -div(k grad u) = f on the unit cube, n^3 uniform hexahedra, Lagrangian Q_p
// (p = 1..3), constant k, f given at the Gauss points, u = 0 on the whole boundary; Jacobi-PCG
// to ||b - A x|| <= rtol ||b||.  Per problem this is the reference's tutorial / test_poisson
// path (integration of the tutorial integrand, strong Dirichlet, CG with the Jacobi
// preconditioner: Sources/Lib/LinearAlgebra/IterativeLinearSolver/cg.f90:101-238,
// Sources/Lib/LinearAlgebra/Preconditioner/jacobi_preconditioner.f90:356-412); FEMPAR runs
// one problem per program, the batch form has no counterpart there.
//
// Design (GB300):
//  * Matrix-free operator.  On a uniform mesh with one coefficient the cell matrix is
//    (h/2) k (s x m x m + m x s x m + m x m x s) for the 1D Gauss-integrated mass m and
//    stiffness s of the reference element (the reference's structured-mesh path reuses the
//    first cell's Jacobian the same way, sbm_cell_map.i90:272-320), so the assembled
//    operator is Sx My Mz + Mx Sy Mz + Mx My Sz in the 1D assembled matrices (rows per node class
//    I mod p), applied one direction after the other: nothing is stored per nonzero.
//  * Right-hand side assembled in the kernel: each cell's load vector by sum factorisation
//    in FP64, gathered per node over its cells in increasing cell order.
//  * Mixed precision without the FP64 pipe in the loop: the inner CG runs in FP32; the
//    solution, the right-hand side and the true residual b - A x are kept in float-float
//    (pairs of FP32, ~2^-48 relative), the operator applied with error-free FP32 products.
//    Every time the FP32 recursive residual has dropped 10x the float-float true residual
//    replaces it (reliable update, the direction is kept).
//  * One persistent cooperative launch.  A host planner orders the problems by estimated
//    work and gives each a team of co-resident CTAs (one CTA for most problems); team
//    members synchronise through a counter in global memory with a bounded spin; one warp sums
//    the per-CTA partials in a fixed order (deterministic for a given plan) and one thread does
//    the scalar step (96 problems, n 8-24: 155 -> 99 ms).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "fg_internal.h"

namespace fg {

static constexpr int kBatchMaxP = 3;
static constexpr int kMaxCls = 27;
static constexpr int kApplySmem = 32768;  // bytes for the partly summed rows of an operator chunk

struct BatchProb {
  int n, p, L, F;        // cells per direction, order, lattice nodes, interior nodes per direction
  float kh_hi, kh_lo;    // stencil scale k h / 2 (times the line tables') as float-float
  double h3;             // (h/2)^3, load-vector scale
  const double* f;       // Gauss-point source, n^3 (p+1)^3
  double* x;             // output, F^3 interior nodes
  int64_t voff;          // 8 float vectors of L^3 in the float pool
  int64_t eoff;          // load vectors, n^3 (p+1)^3 doubles
  int64_t roff;          // partials: 3 slots x team x 4 doubles
  int team;              // CTAs in the team
};

struct BatchJob {
  int prob, rank;
};

// 1D assembled rows of mass and stiffness per node class c = I mod p, as float-float: column t is
// the neighbour I - p + t for class 0 (2p + 1 of them) and I - c + t for the others (p + 1).  The entries
// are rational with a common denominator per order and table, so the tables hold small integers (times a
// power of two), exact in FP32, and kScale goes into each problem's stencil scale.  Rounded entries
// (1/3, 7/3, ..) made the FP32 operator's <v, A v> for smooth v off by 4e-7 (Q1, 32 nodes in a direction) to
// 7e-6 (Q3); so it is off by 3e-9 to 1e-7, and the assembled stencil's was by 5e-7 to 9e-6.
struct LineTables {
  float m[kBatchMaxP][2 * kBatchMaxP + 1][2], s[kBatchMaxP][2 * kBatchMaxP + 1][2];
};

// mass and stiffness entries times kMass and kStiff are integers (in the tables times 2^-kMassExp and
// 2^-kStiffExp); index p - 1
static constexpr double kMass[kBatchMaxP] = {3, 15, 840}, kStiff[kBatchMaxP] = {2, 6, 80};
static constexpr int kMassExp[kBatchMaxP] = {0, 4, 10}, kStiffExp[kBatchMaxP] = {0, 3, 6};
// the tables' operator times this is the unit operator
static double line_scale(int p) {
  return std::ldexp(1.0, 2 * kMassExp[p - 1] + kStiffExp[p - 1]) / (kMass[p - 1] * kMass[p - 1] * kStiff[p - 1]);
}

struct OrderTables {
  int ncls;
  float dg[kMaxCls];     // centre coefficient (unit) per class
  double mw[(kBatchMaxP + 1) * (kBatchMaxP + 1)];  // w_q phi_a(xi_q), [a][q]
};

struct BatchArgs {
  const BatchProb* probs;
  const int* job_ptr;     // per CTA: first job
  const BatchJob* jobs;
  const OrderTables* tabs;  // index p-1
  LineTables line[kBatchMaxP];
  float* vpool;
  double* epool;
  double* rpool;
  unsigned* bar;          // per problem barrier counter
  int* status;            // per problem
  int* iters;
  int* refines;
  double* relres;
  double rtol, atol;
  int max_iters;
  float delta;            // reliable-update factor
  unsigned long long timeout_ns;  // a team wait gives up after this long (globaltimer)
  int* abort_all;         // set by the first wait that gives up: every CTA stops
  int drop_arrival;       // test of the bounded wait: rank 1 of a team skips its first arrival
};

// ---- float-float helpers (error-free transformations; no reassociation in this file)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void quick_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  e = b - (s - a);
}
// (sh, sl) += (ch, cl) * (xh, xl)
__device__ __forceinline__ void ff_fma_acc(float ch, float cl, float xh, float xl, float& sh, float& sl) {
  float p = ch * xh;
  float e = fmaf(ch, xh, -p);
  e = fmaf(ch, xl, fmaf(cl, xh, e));
  float s, t;
  two_sum(sh, p, s, t);
  sh = s;
  sl += t + e;
}
__device__ __forceinline__ void ff_mul(float ah, float al, float bh, float bl, float& h, float& l) {
  float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, fmaf(al, bh, e));
  quick_two_sum(p, e, h, l);
}
__device__ __forceinline__ void ff_add(float ah, float al, float bh, float bl, float& h, float& l) {
  float s, e;
  two_sum(ah, bh, s, e);
  e += al + bl;
  quick_two_sum(s, e, h, l);
}

// Kahan-compensated FP32 accumulator
struct Kf {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double val() const { return (double)s - (double)c; }
};

struct BatchSmem {
  __align__(16) unsigned char rows[kApplySmem];
  float2 zc[kBatchMaxP][2 * kBatchMaxP + 1][2];  // (mass, stiffness) per class and neighbour: hi, lo
  float dinv[kMaxCls];
  double mw[(kBatchMaxP + 1) * (kBatchMaxP + 1)];
  double red[16][2];
  float alpha, beta;
  int flag;
  int abort_flag;
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Arrive at the team's barrier and wait for the others (one thread).  False if the wait gave up
// (status set).
__device__ bool team_arrive_wait(const BatchArgs& a, const BatchProb& P, int prob, int rank, int phase) {
  __threadfence();
  if (!(a.drop_arrival && rank == 1 && phase == 0)) atomicAdd(a.bar + prob, 1u);
  const unsigned target = (unsigned)(phase + 1) * (unsigned)P.team;
  const unsigned long long t0 = global_ns();
  while (ld_acquire(a.bar + prob) < target) {
    if (*(volatile int*)a.abort_all || global_ns() - t0 > a.timeout_ns) {
      atomicExch(a.status + prob, (int)FG_ERR_TIMEOUT);
      atomicExch(a.abort_all, 1);
      return false;
    }
    __nanosleep(20);
  }
  __threadfence();
  return true;
}

// Team reduction of NV (1 or 2) values, then post(totals) on thread 0, whose results in shared
// memory every thread sees after the call.  Returns false if the barrier gave up.
// FP64 is scarce here (a warp's FP64 instruction holds the SM's pipe 16 cycles), so nothing is
// summed or divided by more than one warp: two values share a butterfly (lanes 0-15 go on with the
// first, 16-31 with the second), warp 0 alone adds the warps' sums, writes the CTA's partial,
// waits, adds the team's partials (16 lanes per value) and thread 0 does the scalar step.  With
// every thread adding the partials of all ranks, a team of 89 spent ~25 us per reduction.
template <int NV, class Post>
__device__ bool team_sum(const BatchArgs& a, const BatchProb& P, int prob, int rank, int& phase, const double* v,
                         BatchSmem& sm, Post post) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int k = lane >> 4;  // value of this half warp (NV = 2)
  double x;
  if (NV == 2) {
    const double give = k ? v[0] : v[1], keep = k ? v[1] : v[0];
    x = keep + __shfl_xor_sync(0xffffffffu, give, 16);
  } else {
    x = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
  }
  auto half_sum = [](double y) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y;
  };
  x = half_sum(x);
  if ((lane & 15) == 0 && k < NV) sm.red[warp][k] = x;
  __syncthreads();
  if (warp == 0) {
    x = half_sum((lane & 15) < nw && k < NV ? sm.red[lane & 15][k] : 0.0);
    bool ok = true;
    if (P.team > 1) {
      double* slot = a.rpool + P.roff + (int64_t)(phase % 3) * P.team * 4;
      if ((lane & 15) == 0 && k < NV) slot[rank * 4 + k] = x;
      __syncwarp();
      if (lane == 0) ok = team_arrive_wait(a, P, prob, rank, phase);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      __syncwarp();  // lane 0 acquired the other CTAs' partials (a shuffle orders no memory)
      x = 0.0;
      if (ok && k < NV)
#pragma unroll 4
        for (int r = lane & 15; r < P.team; r += 16) x += ((volatile double*)slot)[r * 4 + k];
      x = half_sum(x);
    }
    const double y = __shfl_sync(0xffffffffu, x, 16);
    if (lane == 0) {
      sm.abort_flag = ok ? 0 : 1;
      if (ok) post(x, y);
    }
  }
  __syncthreads();
  ++phase;
  return !sm.abort_flag;
}

// Barrier without values (phases shared with team_sum).
__device__ bool team_sync(const BatchArgs& a, const BatchProb& P, int prob, int rank, int& phase, BatchSmem& sm) {
  __syncthreads();
  if (P.team > 1) {
    if (threadIdx.x == 0) sm.abort_flag = team_arrive_wait(a, P, prob, rank, phase) ? 0 : 1;
    __syncthreads();
  } else if (threadIdx.x == 0) {
    sm.abort_flag = 0;
  }
  ++phase;
  return P.team == 1 || !sm.abort_flag;
}

// Cell load vectors E_c[a] = (h/2)^3 sum_q w_q f_q phi_a(q) by sum factorisation, FP64, cells [c0, c1).
// Interior nodes u = u0 + threadIdx.x + k blockDim.x of the F^3 block (x fastest), with the
// lattice coordinates advanced incrementally: no integer division inside the loops.
struct NodeWalk {
  int u, u1, I, J, K, g, dI, dJ, dK, F, L, step;
  __device__ __forceinline__ NodeWalk(int u0_, int u1_, int F_, int L_) : u1(u1_), F(F_), L(L_) {
    step = blockDim.x;
    u = u0_ + threadIdx.x;
    if (F > 0) {
      I = 1 + u % F;
      J = 1 + (u / F) % F;
      K = 1 + u / (F * F);
      dI = step % F;
      dJ = (step / F) % F;
      dK = step / (F * F);
    } else {
      I = J = K = 1;
      dI = dJ = dK = 0;
    }
    g = I + L * (J + L * K);
  }
  __device__ __forceinline__ bool ok() const { return u < u1; }
  __device__ __forceinline__ void next() {
    u += step;
    I += dI;
    int c = I > F ? 1 : 0;
    I -= c * F;
    J += dJ + c;
    c = J > F ? 1 : 0;
    J -= c * F;
    K += dK + c;
    g = I + L * (J + L * K);
  }
};

// Scalars of the operator: FP32, and float-float with error-free products.  Acc is a running sum.
struct S32 {
  using V = float;
  using P2 = float2;  // two values in shared memory
  static __device__ __forceinline__ V zero() { return 0.f; }
  static __device__ __forceinline__ V load(const float* h, const float*, int64_t g) { return h[g]; }
  static __device__ __forceinline__ void fma(const float (&c)[2], V x, V& s) { s = fmaf(c[0], x, s); }
  static __device__ __forceinline__ void fma(float ch, float, V x, V& s) { s = fmaf(ch, x, s); }
  static __device__ __forceinline__ void norm(V&) {}
  static __device__ __forceinline__ P2 pack(V a, V b) { return make_float2(a, b); }
  static __device__ __forceinline__ V first(P2 p) { return p.x; }
  static __device__ __forceinline__ V second(P2 p) { return p.y; }
};
struct Sff {
  struct V { float h, l; };
  using P2 = float4;
  static __device__ __forceinline__ V zero() { return {0.f, 0.f}; }
  static __device__ __forceinline__ V load(const float* h, const float* l, int64_t g) { return {h[g], l[g]}; }
  static __device__ __forceinline__ void fma(const float (&c)[2], V x, V& s) { ff_fma_acc(c[0], c[1], x.h, x.l, s.h, s.l); }
  static __device__ __forceinline__ void fma(float ch, float cl, V x, V& s) { ff_fma_acc(ch, cl, x.h, x.l, s.h, s.l); }
  static __device__ __forceinline__ void norm(V& s) { quick_two_sum(s.h, s.l, s.h, s.l); }
  static __device__ __forceinline__ P2 pack(V a, V b) { return make_float4(a.h, a.l, b.h, b.l); }
  static __device__ __forceinline__ V first(P2 p) { return {p.x, p.y}; }
  static __device__ __forceinline__ V second(P2 p) { return {p.z, p.w}; }
};

// The unit operator Sx My Mz + Mx Sy Mz + Mx My Sz applied direction by direction, to a row block at
// a time: NR = p YB rows in y (YB periods: 4, 2, 1 for p = 1, 2, 3) of one plane.
//   1. thread per x (consecutive lanes read consecutive nodes): the z sums t = Mz v, u = Sz v of the
//      rows' y window, then a = My t and b = Sy t + My u for the NR rows, into shared memory;
//   2. thread per x period of a row: Sx a + Mx b for its p nodes, handed to out(node, I, J, K, value).
// About 50 multiply-adds per node at p = 3 where the assembled stencil has 125 (and read one
// coefficient from shared memory for each, and its window with stride p).
// A rank's row blocks [w0, w1) go in chunks of G row blocks (or pieces of one, for rows that do not
// fit kApplySmem) that fill the block's threads.
// What bounds it: instruction issue and the latency of phase 1's loads (everything is in L2); the next
// plane's loads run beside a plane's products.  One CTA of 512 threads alone on an SM, 314 k nodes at
// p = 3: 5.7 ns per node and CG iteration, everything included; 96 problems, n 8-24: 99 -> 66 ms with
// this operator, 55 ms with the loads ahead (here and in the vector updates).
template <int PO>
struct ApplyShape {
  static constexpr int YB = PO == 1 ? 4 : (PO == 2 ? 2 : 1);
  static constexpr int NR = PO * YB;            // rows of a block: J0 + 1 .. J0 + NR
  static constexpr int NY = PO * (YB + 1) + 1;  // their y window: J0 .. J0 + NY - 1
};
template <int PO, class S, class Out>
__device__ __forceinline__ void apply_rows(const LineTables& T, BatchSmem& sm, const float* vh, const float* vl, int n,
                                           int F, int L, int w0, int w1, Out out) {
  using V = typename S::V;
  using P2 = typename S::P2;
  constexpr int NR = ApplyShape<PO>::NR, NY = ApplyShape<PO>::NY, YB = ApplyShape<PO>::YB;
  constexpr int CAP = kApplySmem / (int)sizeof(P2) / NR;  // nodes of x
  constexpr bool kDiff = PO == 1 && std::is_same<S, S32>::value;
  P2* rows = reinterpret_cast<P2*>(sm.rows);
  const int nyb = (n + YB - 1) / YB;
  // pieces of a row block: SP periods each, nodes PO m0 .. PO (m0 + SP) + PO
  const int SP = PO * (n + 1) + 1 <= CAP ? n : (CAP - 1) / PO - 1;
  const int nseg = (n + SP - 1) / SP, W = PO * (SP + 1) + 1;
  const int G = max(1, CAP / W);
  const int q1 = w1 * nseg;
  for (int q0 = w0 * nseg; q0 < q1; q0 += G) {
    const int ng = min(G, q1 - q0);
    for (int t = threadIdx.x; t < ng * W; t += blockDim.x) {
      const int gi = t / W, i = t - gi * W;
      const int q = q0 + gi, blk = q / nseg, m0 = (q - blk * nseg) * SP;
      const int K = 1 + blk / nyb, J0 = (blk - (K - 1) * nyb) * NR, I = PO * m0 + i;
      V a[NR], b[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) a[r] = b[r] = S::zero();
      if (I >= 1 && I <= F && kDiff) {
        // Q1, FP32: the tables are (-1, 2, -1) and (1, 4, 1), i.e. S w = (w_0 - w_-) + (w_0 - w_+) and M w =
        // 6 w_0 - S w: differences of close values cost no digits, and a sum is rounded once
        const int ny = min(NY, F + 1 - J0), L2 = L * L;
        const int g = I + L * J0 + L2 * K;
        float v0[NY], vm[NY], vp[NY], tz[NY], uz[NY];
#pragma unroll
        for (int y = 0; y < NY; ++y) {
          v0[y] = y < ny ? vh[g + y * L] : 0.f;
          vm[y] = y < ny ? vh[g + y * L - L2] : 0.f;
          vp[y] = y < ny ? vh[g + y * L + L2] : 0.f;
        }
#pragma unroll
        for (int y = 0; y < NY; ++y) {
          uz[y] = (v0[y] - vm[y]) + (v0[y] - vp[y]);
          tz[y] = fmaf(6.f, v0[y], -uz[y]);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const float st = (tz[r + 1] - tz[r]) + (tz[r + 1] - tz[r + 2]);
          const float su = (uz[r + 1] - uz[r]) + (uz[r + 1] - uz[r + 2]);
          reinterpret_cast<float*>(a)[r] = fmaf(6.f, tz[r + 1], -st);
          reinterpret_cast<float*>(b)[r] = fmaf(6.f, uz[r + 1], -su) + st;
        }
      } else if (I >= 1 && I <= F) {
        V tz[NY], uz[NY];
#pragma unroll
        for (int y = 0; y < NY; ++y) tz[y] = uz[y] = S::zero();
        const int cz = K % PO, kz = cz ? cz : PO, nz = cz ? PO + 1 : 2 * PO + 1;
        const int ny = min(NY, F + 1 - J0);  // rows from the boundary on are zero
        const int L2 = L * L;
        int g = I + L * J0 + L2 * (K - kz);
        V v[NY];
#pragma unroll
        for (int y = 0; y < NY; ++y) v[y] = y < ny ? S::load(vh, vl, g + y * L) : S::zero();
        for (int z = 0; z < nz; ++z) {
          V nxt[NY];  // the next plane's loads run beside this one's products
          if (z + 1 < nz) {
            g += L2;
#pragma unroll
            for (int y = 0; y < NY; ++y) nxt[y] = y < ny ? S::load(vh, vl, g + y * L) : S::zero();
          }
          const float2 ch = sm.zc[cz][z][0], cl = sm.zc[cz][z][1];
#pragma unroll
          for (int y = 0; y < NY; ++y) {
            S::fma(ch.x, cl.x, v[y], tz[y]);
            S::fma(ch.y, cl.y, v[y], uz[y]);
          }
#pragma unroll
          for (int y = 0; y < NY; ++y) v[y] = nxt[y];
        }
#pragma unroll
        for (int y = 0; y < NY; ++y) {
          S::norm(tz[y]);
          S::norm(uz[y]);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          // row J0 + 1 + r: class (r + 1) mod p, first neighbour at window row y0
          constexpr int P = PO;
          const int c = (r + 1) % P, y0 = c ? r + 1 - c : r + 1 - P, nn = c ? P + 1 : 2 * P + 1;
#pragma unroll
          for (int t2 = 0; t2 < 2 * P + 1; ++t2)
            if (t2 < nn) {
              S::fma(T.m[c][t2], tz[y0 + t2], a[r]);
              S::fma(T.s[c][t2], tz[y0 + t2], b[r]);
              S::fma(T.m[c][t2], uz[y0 + t2], b[r]);
            }
          S::norm(a[r]);
          S::norm(b[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) rows[(gi * NR + r) * W + i] = S::pack(a[r], b[r]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ng * NR * SP; t += blockDim.x) {
      const int row = t / SP, m = t - row * SP, gi = row / NR;
      const int q = q0 + gi, blk = q / nseg, m0 = (q - blk * nseg) * SP;
      const int K = 1 + blk / nyb, J = (blk - (K - 1) * nyb) * NR + 1 + (row - gi * NR);
      if (J > F || m0 + m >= n) continue;
      const P2* w = rows + row * W + PO * m;
      V o[PO];  // o[0]: the class-0 node at the period's end
#pragma unroll
      for (int k = 0; k < PO; ++k) o[k] = S::zero();
      if (kDiff) {
        const float2* wf = reinterpret_cast<const float2*>(w);
        const float2 m = wf[0], c = wf[1], n1 = wf[2];
        const float sa = (c.x - m.x) + (c.x - n1.x), sb = (c.y - m.y) + (c.y - n1.y);
        reinterpret_cast<float*>(o)[0] = fmaf(6.f, c.y, sa) - sb;
      } else
#pragma unroll
      for (int t2 = 0; t2 < 2 * PO + 1; ++t2) {
        const P2 ab = w[t2];
#pragma unroll
        for (int k = 0; k < PO; ++k)
          if (k == 0 || t2 <= PO) {
            S::fma(T.s[k][t2], S::first(ab), o[k]);
            S::fma(T.m[k][t2], S::second(ab), o[k]);
          }
      }
      const int I0 = PO * (m0 + m), g0 = I0 + L * (J + L * K);
#pragma unroll
      for (int k = 1; k <= PO; ++k)
        if (I0 + k <= F) out(g0 + k, I0 + k, J, K, o[k % PO]);
    }
    __syncthreads();
  }
}

template <int PO>
__device__ __noinline__ void load_vectors(const BatchProb& P, double* E, int64_t c0, int64_t c1, const BatchSmem& sm) {
  constexpr int NP1 = PO + 1, NQ = NP1 * NP1 * NP1;
  for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
    const double* f = P.f + c * NQ;
    double t1[NQ], t2[NQ];
#pragma unroll
    for (int qz = 0; qz < NP1; ++qz)
#pragma unroll
      for (int qy = 0; qy < NP1; ++qy)
#pragma unroll
        for (int ax = 0; ax < NP1; ++ax) {
          double s = 0.0;
#pragma unroll
          for (int qx = 0; qx < NP1; ++qx) s += sm.mw[ax * NP1 + qx] * f[qx + NP1 * (qy + NP1 * qz)];
          t1[ax + NP1 * (qy + NP1 * qz)] = s;
        }
#pragma unroll
    for (int qz = 0; qz < NP1; ++qz)
#pragma unroll
      for (int ay = 0; ay < NP1; ++ay)
#pragma unroll
        for (int ax = 0; ax < NP1; ++ax) {
          double s = 0.0;
#pragma unroll
          for (int qy = 0; qy < NP1; ++qy) s += sm.mw[ay * NP1 + qy] * t1[ax + NP1 * (qy + NP1 * qz)];
          t2[ax + NP1 * (ay + NP1 * qz)] = s;
        }
#pragma unroll
    for (int az = 0; az < NP1; ++az)
#pragma unroll
      for (int ay = 0; ay < NP1; ++ay)
#pragma unroll
        for (int ax = 0; ax < NP1; ++ax) {
          double s = 0.0;
#pragma unroll
          for (int qz = 0; qz < NP1; ++qz) s += sm.mw[az * NP1 + qz] * t2[ax + NP1 * (ay + NP1 * qz)];
          E[c * NQ + ax + NP1 * (ay + NP1 * az)] = s * P.h3;
        }
  }
}

template <int PO>
__device__ void solve_problem(const BatchArgs& a, int prob, int rank, BatchSmem& sm) {
  const BatchProb P = a.probs[prob];
  const OrderTables& T = a.tabs[PO - 1];
  constexpr int NP1 = PO + 1, NQ = NP1 * NP1 * NP1;
  const int L = P.L, F = P.F, n = P.n;
  const int64_t L2 = (int64_t)L * L;
  const LineTables& line = a.line[PO - 1];
  for (int c = threadIdx.x; c < T.ncls; c += blockDim.x) sm.dinv[c] = 1.0f / (T.dg[c] * P.kh_hi);
  for (int t = threadIdx.x; t < PO * (2 * PO + 1) * 2; t += blockDim.x) {
    const int part = t & 1, z = (t >> 1) % (2 * PO + 1), c = (t >> 1) / (2 * PO + 1);
    sm.zc[c][z][part] = make_float2(line.m[c][z][part], line.s[c][z][part]);
  }
  for (int t = threadIdx.x; t < NP1 * NP1; t += blockDim.x) sm.mw[t] = T.mw[t];
  __syncthreads();
  float* bh = a.vpool + P.voff;
  float* bl = bh + L * L2;
  float* xh = bl + L * L2;
  float* xl = xh + L * L2;
  float* xc = xl + L * L2;
  float* r = xc + L * L2;
  float* pp = r + L * L2;
  float* q = pp + L * L2;
  double* E = a.epool + P.eoff;
  int phase = 0;
  // team ranges: cells and interior nodes
  const int64_t ncells = (int64_t)n * n * n, nint = (int64_t)F * F * F;
  const int64_t c0 = ncells * rank / P.team, c1 = ncells * (rank + 1) / P.team;
  const int64_t u0 = nint * rank / P.team, u1 = nint * (rank + 1) / P.team;
  // row blocks of the operator
  const int64_t nblk = (int64_t)((n + ApplyShape<PO>::YB - 1) / ApplyShape<PO>::YB) * F;
  const int w0 = (int)(nblk * rank / P.team), w1 = (int)(nblk * (rank + 1) / P.team);
  // 1. load vectors by sum factorisation (FP64)
  load_vectors<PO>(P, E, c0, c1, sm);
  if (!team_sync(a, P, prob, rank, phase, sm)) return;
  // 2. gather b per node (cells in increasing order), initial state
  double loc[4] = {0.0, 0.0, 0.0, 0.0};
  {
    Kf rz;
    double bb = 0.0;
    for (NodeWalk w((int)u0, (int)u1, F, L); w.ok(); w.next()) {
      const int I = w.I, J = w.J, K = w.K;
      int cx[2], lx[2], nx = 0, cy[2], ly[2], ny = 0, cz[2], lz[2], nz = 0;
      if (I % PO == 0) { cx[0] = I / PO - 1; lx[0] = PO; cx[1] = I / PO; lx[1] = 0; nx = 2; }
      else { cx[0] = I / PO; lx[0] = I % PO; nx = 1; }
      if (J % PO == 0) { cy[0] = J / PO - 1; ly[0] = PO; cy[1] = J / PO; ly[1] = 0; ny = 2; }
      else { cy[0] = J / PO; ly[0] = J % PO; ny = 1; }
      if (K % PO == 0) { cz[0] = K / PO - 1; lz[0] = PO; cz[1] = K / PO; lz[1] = 0; nz = 2; }
      else { cz[0] = K / PO; lz[0] = K % PO; nz = 1; }
      double b = 0.0;
      for (int kz = 0; kz < nz; ++kz)
        for (int ky = 0; ky < ny; ++ky)
          for (int kx = 0; kx < nx; ++kx) {
            int64_t c = cx[kx] + (int64_t)n * (cy[ky] + (int64_t)n * cz[kz]);
            b += E[c * NQ + lx[kx] + NP1 * (ly[ky] + NP1 * lz[kz])];
          }
      const int64_t g = w.g;
      float h = (float)b;
      float l = (float)(b - (double)h);
      bh[g] = h;
      bl[g] = l;
      xh[g] = 0.f;
      xl[g] = 0.f;
      xc[g] = 0.f;
      r[g] = h;
      const int cls = (I % PO) + PO * ((J % PO) + PO * (K % PO));
      float z = sm.dinv[cls] * h;
      pp[g] = z;
      rz.add(h * z);
      bb = fma(b, b, bb);
    }
    loc[0] = bb;
    loc[1] = rz.val();
  }
  // the scalars of the iteration live on thread 0; alpha, beta and what to do next go through
  // shared memory
  enum { STEP = 0, REFINE = 1, BREAKDOWN = 2, CONVERGED = 3 };
  double bnorm = 0.0, rzv = 0.0, rtrue2 = 0.0, tol = 0.0, relres = 1.0;
  if (!team_sum<2>(a, P, prob, rank, phase, loc, sm, [&](double t0, double t1) {
        bnorm = sqrt(t0);
        rzv = t1;
        rtrue2 = t0;
        tol = a.rtol * bnorm + a.atol;
        sm.flag = bnorm <= a.atol ? CONVERGED : STEP;
      }))
    return;
  int it = 0, nref = 0, conv = sm.flag == CONVERGED ? 1 : 0;
  const float khf = P.kh_hi;
  while (!conv && it < a.max_iters) {
    ++it;
    // q = A p (FP32), <p, q>
    {
      Kf pq;
      apply_rows<PO, S32>(line, sm, pp, nullptr, n, F, L, w0, w1, [&](int g, int, int, int, float o) {
        const float y = o * khf;
        q[g] = y;
        pq.add(y * pp[g]);
      });
      loc[0] = pq.val();
    }
    if (!team_sum<1>(a, P, prob, rank, phase, loc, sm, [&](double pq, double) {
          sm.flag = pq > 0.0 ? STEP : BREAKDOWN;
          if (pq > 0.0) sm.alpha = (float)(rzv / pq);
        }))
      return;
    if (sm.flag == BREAKDOWN) {
      if (threadIdx.x == 0 && rank == 0) atomicExch(a.status + prob, (int)FG_ERR_NUMERIC);
      break;
    }
    const float alpha = sm.alpha;
    {
      Kf rr, rzn;
      for (NodeWalk w((int)u0, (int)u1, F, L); w.ok();) {
        // four nodes' loads before the first store
        int g[4];
        float di[4], pv[4], qv[4], xv[4], rv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k, w.next()) {
          g[k] = w.ok() ? w.g : -1;
          if (g[k] < 0) continue;
          di[k] = sm.dinv[(w.I % PO) + PO * ((w.J % PO) + PO * (w.K % PO))];
          pv[k] = pp[g[k]];
          qv[k] = q[g[k]];
          xv[k] = xc[g[k]];
          rv[k] = r[g[k]];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (g[k] < 0) continue;
          xc[g[k]] = fmaf(alpha, pv[k], xv[k]);
          const float ri = fmaf(-alpha, qv[k], rv[k]);
          r[g[k]] = ri;
          rr.add(ri * ri);
          rzn.add(ri * (di[k] * ri));
        }
      }
      loc[0] = rr.val();
      loc[1] = rzn.val();
    }
    if (!team_sum<2>(a, P, prob, rank, phase, loc, sm, [&](double rr, double rzn) {
          const bool near = rr <= 0.25 * tol * tol;
          if (rr <= (double)a.delta * (double)a.delta * rtrue2 || near || it >= a.max_iters) {
            sm.flag = REFINE;
          } else {
            sm.flag = STEP;
            sm.beta = (float)(rzn / rzv);
            rzv = rzn;
          }
        }))
      return;
    if (sm.flag == REFINE) {
      // reliable update: x += xc (float-float), then r = b - A x in float-float
      for (NodeWalk w((int)u0, (int)u1, F, L); w.ok(); w.next()) {
        const int64_t g = w.g;
        float h, l;
        ff_add(xh[g], xl[g], xc[g], 0.f, h, l);
        xh[g] = h;
        xl[g] = l;
        xc[g] = 0.f;
      }
      if (!team_sync(a, P, prob, rank, phase, sm)) return;
      Kf rr2, rz2;
      apply_rows<PO, Sff>(line, sm, xh, xl, n, F, L, w0, w1, [&](int g, int I, int J, int K, Sff::V o) {
        float h, l, ah, al;
        quick_two_sum(o.h, o.l, h, l);
        ff_mul(P.kh_hi, P.kh_lo, h, l, ah, al);
        float rh, rl;
        ff_add(bh[g], bl[g], -ah, -al, rh, rl);
        const float ri = rh + rl;
        r[g] = ri;
        rr2.add(ri * ri);
        rz2.add(ri * (sm.dinv[(I % PO) + PO * ((J % PO) + PO * (K % PO))] * ri));
      });
      loc[0] = rr2.val();
      loc[1] = rz2.val();
      ++nref;
      if (!team_sum<2>(a, P, prob, rank, phase, loc, sm, [&](double rr, double rzn) {
            rtrue2 = rr;
            relres = bnorm > 0.0 ? sqrt(rtrue2) / bnorm : 0.0;
            sm.flag = sqrt(rtrue2) <= tol ? CONVERGED : STEP;
            sm.beta = (float)(rzn / rzv);
            rzv = rzn;
          }))
        return;
      if (sm.flag == CONVERGED) {
        conv = 1;
        break;
      }
    }
    const float beta = sm.beta;
    for (NodeWalk w((int)u0, (int)u1, F, L); w.ok();) {
      int g[4];
      float pv[4], zv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k, w.next()) {
        g[k] = w.ok() ? w.g : -1;
        if (g[k] < 0) continue;
        pv[k] = pp[g[k]];
        zv[k] = sm.dinv[(w.I % PO) + PO * ((w.J % PO) + PO * (w.K % PO))] * r[g[k]];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (g[k] >= 0) pp[g[k]] = fmaf(beta, pv[k], zv[k]);
    }
    if (!team_sync(a, P, prob, rank, phase, sm)) return;
  }
  // solution: x = xh + xl at the interior nodes, x fastest
  for (NodeWalk w((int)u0, (int)u1, F, L); w.ok(); w.next()) {
    const int64_t g = w.g;
    P.x[w.u] = (double)xh[g] + (double)xl[g];
  }
  if (rank == 0 && threadIdx.x == 0) {
    a.iters[prob] = it;
    a.refines[prob] = nref;
    a.relres[prob] = relres;
    if (!conv) atomicCAS(a.status + prob, 0, (int)FG_ERR_NOT_CONVERGED);
  }
}

__global__ void __launch_bounds__(512, 2) k_batch_solve(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  BatchSmem& sm = *reinterpret_cast<BatchSmem*>(smraw);
  for (int j = a.job_ptr[blockIdx.x]; j < a.job_ptr[blockIdx.x + 1]; ++j) {
    if (threadIdx.x == 0) sm.abort_flag = *(volatile int*)a.abort_all;
    __syncthreads();
    const int stop = sm.abort_flag;  // one value for the whole CTA
    __syncthreads();
    if (stop) {
      // the problems this CTA leads and has not started are reported, not silently skipped
      if (threadIdx.x == 0)
        for (int k = j; k < a.job_ptr[blockIdx.x + 1]; ++k)
          if (a.jobs[k].rank == 0) atomicCAS(a.status + a.jobs[k].prob, 0, (int)FG_ERR_TIMEOUT);
      break;
    }
    const BatchJob J = a.jobs[j];
    const int p = a.probs[J.prob].p;
    if (p == 1) solve_problem<1>(a, J.prob, J.rank, sm);
    else if (p == 2) solve_problem<2>(a, J.prob, J.rank, sm);
    else solve_problem<3>(a, J.prob, J.rank, sm);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// Host

static void build_order_tables(int p, OrderTables& T, LineTables& line) {
  std::memset(&T, 0, sizeof(T));
  std::memset(&line, 0, sizeof(line));
  const int np1 = p + 1;
  double xq[kBatchMaxP + 1], wq[kBatchMaxP + 1];
  gl_rule(np1, xq, wq);
  double phi[kBatchMaxP + 1][kBatchMaxP + 1], dphi[kBatchMaxP + 1][kBatchMaxP + 1];
  for (int a = 0; a < np1; ++a)
    for (int q = 0; q < np1; ++q) lagrange_1d(p, a, xq[q], phi[a][q], dphi[a][q]);
  double m[kBatchMaxP + 1][kBatchMaxP + 1], s[kBatchMaxP + 1][kBatchMaxP + 1];
  for (int a = 0; a < np1; ++a)
    for (int b = 0; b < np1; ++b) {
      double sm = 0.0, ss = 0.0;
      for (int q = 0; q < np1; ++q) {
        sm += wq[q] * phi[a][q] * phi[b][q];
        ss += wq[q] * dphi[a][q] * dphi[b][q];
      }
      m[a][b] = sm;
      s[a][b] = ss;
    }
  for (int a = 0; a < np1; ++a)
    for (int q = 0; q < np1; ++q) T.mw[a * np1 + q] = wq[q] * phi[a][q];
  // 1D assembled rows per class: offsets [lo, lo + w)
  int lo1[kBatchMaxP], w1[kBatchMaxP];
  double M1[kBatchMaxP][2 * kBatchMaxP + 1], S1[kBatchMaxP][2 * kBatchMaxP + 1];
  for (int c = 0; c < p; ++c) {
    if (c == 0) {
      lo1[c] = -p;
      w1[c] = 2 * p + 1;
      for (int o = -p; o <= p; ++o) {
        double mm = 0.0, ss = 0.0;
        if (o <= 0) { mm += m[p][p + o]; ss += s[p][p + o]; }
        if (o >= 0) { mm += m[0][o]; ss += s[0][o]; }
        M1[c][o + p] = mm;
        S1[c][o + p] = ss;
      }
    } else {
      lo1[c] = -c;
      w1[c] = p + 1;
      for (int o = -c; o <= p - c; ++o) {
        M1[c][o + c] = m[c][c + o];
        S1[c][o + c] = s[c][c + o];
      }
    }
  }
  T.ncls = p * p * p;
  // exact entries: the quadrature's rounding goes, the scale moves to the stencil scale
  for (int c = 0; c < p; ++c)
    for (int t = 0; t < w1[c]; ++t) {
      M1[c][t] = std::ldexp(std::round(M1[c][t] * kMass[p - 1]), -kMassExp[p - 1]);
      S1[c][t] = std::ldexp(std::round(S1[c][t] * kStiff[p - 1]), -kStiffExp[p - 1]);
    }
  auto split = [](double v, float (&f)[2]) {
    f[0] = (float)v;
    f[1] = (float)(v - (double)f[0]);
  };
  for (int c = 0; c < p; ++c)
    for (int t = 0; t < w1[c]; ++t) {
      split(M1[c][t], line.m[c][t]);
      split(S1[c][t], line.s[c][t]);
    }
  for (int cz = 0; cz < p; ++cz)
    for (int cy = 0; cy < p; ++cy)
      for (int cx = 0; cx < p; ++cx) {
        const double mx = M1[cx][-lo1[cx]], my = M1[cy][-lo1[cy]], mz = M1[cz][-lo1[cz]];
        const double sx = S1[cx][-lo1[cx]], sy = S1[cy][-lo1[cy]], sz = S1[cz][-lo1[cz]];
        T.dg[cx + p * (cy + p * cz)] = (float)(sx * my * mz + mx * sy * mz + mx * my * sz);
      }
}

static double avg_nnz(int p) {
  double w = (2.0 * p + 1.0 + (p - 1) * (p + 1.0)) / p;
  return w * w * w;
}

}  // namespace fg

struct fg_batch {
  fg_ctx* ctx = nullptr;
  int nprob = 0, flags = 0;
  fg_solver_params prm;
  std::vector<fg::BatchProb> probs;       // device-facing descriptors
  std::vector<const double*> user_f;      // caller's source pointers
  std::vector<double*> user_x;            // caller's output pointers
  fg::LineTables line[fg::kBatchMaxP];
  std::vector<int64_t> nf, nx;            // source / output lengths
  int threads = 0, ctas = 0, max_team = 0, teams_gt1 = 0;
  // team sizing: a problem gets about ceil(work / (team_share * per-CTA share)) CTAs
  // (0.5, or FG_BATCH_TEAM_SHARE when set > 0)
  double team_share = 0.5;
  double predicted_balance = 0.0, autotune_ms = 0.0, run_ms = 0.0;
  int64_t total_dofs = 0;
  fg::BatchProb* d_probs = nullptr;
  int* d_job_ptr = nullptr;
  fg::BatchJob* d_jobs = nullptr;
  fg::OrderTables* d_tabs = nullptr;
  float* vpool = nullptr;
  double* epool = nullptr;
  double* rpool = nullptr;
  unsigned* bar = nullptr;
  int* abort_all = nullptr;
  int* status = nullptr;
  int* iters = nullptr;
  int* refines = nullptr;
  double* relres = nullptr;
  double* fstage = nullptr;  // host-input mode: staged sources and outputs
  double* xstage = nullptr;
  int64_t nrp = 0;
  std::vector<void*> owned;
  cudaGraphExec_t graph = nullptr;
  bool use_graph = false;
};

namespace fg {

static fg_status ba(fg_batch* B, void** p, size_t bytes) {
  FG_TRY(dev_alloc(B->ctx, p, bytes));
  B->owned.push_back(*p);
  return FG_OK;
}

static size_t batch_smem() { return sizeof(BatchSmem); }

// Team sizes and the per-CTA job lists (greedy list scheduling, problems by decreasing work).
// A problem with t CTAs takes its iterations (measured: 3, 8, 20 per cell in a direction at
// orders 1-3) times its share of the nodes plus what an iteration's reductions and barriers cost:
// on GB300 12 us with one CTA of 512 threads, ~30 us in a large team, against 7.9 ns per node, i.e. 3
// and 8 nodes per thread.  A problem's team is about ceil(work / (team_share x a CTA's share));
// all teams are scaled together and the schedule that ends first by this model is taken (96
// problems, n 8-24: 66 ms unscaled, 44 ms; 200 problems, n 6-30: 130 ms with four scales and 5
// nodes per thread, 118 ms so).
static void batch_schedule(fg_batch* B, int G, std::vector<int>& job_ptr, std::vector<BatchJob>& jobs) {
  const int np = B->nprob;
  std::vector<double> nodes(np), its(np), w(np);
  double W = 0.0;
  for (int i = 0; i < np; ++i) {
    const BatchProb& P = B->probs[i];
    nodes[i] = std::max(1.0, (double)P.F * P.F * P.F);
    its[i] = P.n * (P.p == 1 ? 3.0 : (P.p == 2 ? 8.0 : 20.0));
    w[i] = its[i] * (nodes[i] + 3.0 * B->threads);
    W += w[i];
  }
  std::vector<int> order(np);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return w[x] > w[y]; });
  const double target = W / G;
  double best = -1.0;
  std::vector<int> team(np), best_team(np);
  std::vector<std::vector<BatchJob>> per(G), best_per(G);
  std::vector<double> avail(G);
  std::vector<int> idx(G);
  // (a schedule of thousands of problems takes the host tens of ms, and its teams are few)
  const std::vector<double> scales = np <= 1024 ? std::vector<double>{0.7, 0.85, 1.0, 1.2, 1.4, 1.7, 2.0, 2.4, 2.8, 3.4}
                                                : std::vector<double>{1.0, 1.4, 2.0, 2.8};
  for (double scale : scales) {
    std::fill(avail.begin(), avail.end(), 0.0);
    for (auto& v : per) v.clear();
    for (int i : order) {
      const BatchProb& P = B->probs[i];
      const int64_t F3 = (int64_t)P.F * P.F * P.F;
      int t = (int)std::ceil(w[i] / (scale * B->team_share * target));
      t = std::max(1, std::min(t, G));
      t = (int)std::min<int64_t>(t, std::max<int64_t>(1, F3 / (4 * B->threads)));
      team[i] = t;
      std::iota(idx.begin(), idx.end(), 0);
      std::partial_sort(idx.begin(), idx.begin() + t, idx.end(),
                        [&](int x, int y) { return avail[x] < avail[y] || (avail[x] == avail[y] && x < y); });
      std::sort(idx.begin(), idx.begin() + t);
      double start = 0.0;
      for (int k = 0; k < t; ++k) start = std::max(start, avail[idx[k]]);
      const double end = start + its[i] * (nodes[i] / t + (t > 1 ? 8.0 : 3.0) * B->threads);
      for (int k = 0; k < t; ++k) {
        avail[idx[k]] = end;
        per[idx[k]].push_back({i, k});
      }
    }
    const double mk = *std::max_element(avail.begin(), avail.end());
    if (best < 0.0 || mk < best) {
      best = mk;
      best_team = team;
      best_per.swap(per);
    }
  }
  B->max_team = 1;
  B->teams_gt1 = 0;
  for (int i = 0; i < np; ++i) {
    B->probs[i].team = best_team[i];
    B->max_team = std::max(B->max_team, best_team[i]);
    if (best_team[i] > 1) B->teams_gt1++;
  }
  B->predicted_balance = best > 0 ? std::min(1.0, (W / G) / best) : 1.0;
  job_ptr.assign(G + 1, 0);
  jobs.clear();
  for (int g = 0; g < G; ++g) {
    job_ptr[g] = (int)jobs.size();
    for (auto& j : best_per[g]) jobs.push_back(j);
  }
  job_ptr[G] = (int)jobs.size();
}

static fg_status batch_launch(fg_batch* B, cudaStream_t st) {
  BatchArgs a;
  a.probs = B->d_probs;
  a.job_ptr = B->d_job_ptr;
  a.jobs = B->d_jobs;
  a.tabs = B->d_tabs;
  std::memcpy(a.line, B->line, sizeof(a.line));
  a.vpool = B->vpool;
  a.epool = B->epool;
  a.rpool = B->rpool;
  a.bar = B->bar;
  a.status = B->status;
  a.iters = B->iters;
  a.refines = B->refines;
  a.relres = B->relres;
  a.rtol = B->prm.rtol;
  a.atol = B->prm.atol;
  a.max_iters = B->prm.max_iters;
  a.delta = B->prm.inner_rtol > 0.0 ? (float)B->prm.inner_rtol : 0.1f;
  // team waits give up after 60 s (FG_BATCH_BARRIER_TIMEOUT_MS overrides); the test switch
  // FG_BATCH_TEST_DROP_ARRIVAL=1 makes one team member skip an arrival so that the wait runs out
  a.timeout_ns = 60ull * 1000000000ull;
  if (const char* e = std::getenv("FG_BATCH_BARRIER_TIMEOUT_MS")) {
    const long long ms = std::atoll(e);
    if (ms > 0) a.timeout_ns = (unsigned long long)ms * 1000000ull;
  }
  {
    const char* e = std::getenv("FG_BATCH_TEST_DROP_ARRIVAL");
    a.drop_arrival = (e && e[0] == '1') ? 1 : 0;
  }
  a.abort_all = B->abort_all;
  FG_CUDA_TRY(cudaMemsetAsync(B->bar, 0, sizeof(unsigned) * B->nprob, st));
  FG_CUDA_TRY(cudaMemsetAsync(B->abort_all, 0, sizeof(int), st));
  FG_CUDA_TRY(cudaMemsetAsync(B->status, 0, sizeof(int) * B->nprob, st));
  void* args[] = {&a};
  FG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_batch_solve, dim3(B->ctas), dim3(B->threads), args,
                                          batch_smem(), st));
  B->ctx->launches += 1;
  return FG_OK;
}

// Co-resident CTAs for a block size, the schedule and its device copy.
static fg_status batch_plan(fg_batch* B, int threads) {
  fg_ctx* ctx = B->ctx;
  B->threads = threads;
  int per_sm = 0;
  FG_CUDA_TRY(cudaFuncSetAttribute((const void*)k_batch_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)batch_smem()));
  FG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_batch_solve, threads,
                                                            batch_smem()));
  if (per_sm < 1) {
    set_error("batch kernel does not fit an SM with %d threads", threads);
    return FG_ERR_UNSUPPORTED;
  }
  B->ctas = per_sm * ctx->sm_count;
  std::vector<int> job_ptr;
  std::vector<BatchJob> jobs;
  batch_schedule(B, B->ctas, job_ptr, jobs);
  // partial slots per problem: 3 x team x 4 doubles
  int64_t roff = 0;
  for (auto& P : B->probs) {
    P.roff = roff;
    roff += 3 * (int64_t)P.team * 4;
  }
  if (roff > B->nrp) {
    if (B->rpool) {
      dev_free(ctx, B->rpool);
      B->owned.erase(std::find(B->owned.begin(), B->owned.end(), (void*)B->rpool));
    }
    FG_TRY(ba(B, (void**)&B->rpool, sizeof(double) * roff));
    B->nrp = roff;
  }
  if (B->d_job_ptr) {
    dev_free(ctx, B->d_job_ptr);
    B->owned.erase(std::find(B->owned.begin(), B->owned.end(), (void*)B->d_job_ptr));
  }
  if (B->d_jobs) {
    dev_free(ctx, B->d_jobs);
    B->owned.erase(std::find(B->owned.begin(), B->owned.end(), (void*)B->d_jobs));
  }
  FG_TRY(ba(B, (void**)&B->d_job_ptr, sizeof(int) * job_ptr.size()));
  FG_TRY(ba(B, (void**)&B->d_jobs, sizeof(BatchJob) * std::max<size_t>(1, jobs.size())));
  FG_CUDA_TRY(cudaMemcpyAsync(B->d_job_ptr, job_ptr.data(), sizeof(int) * job_ptr.size(), cudaMemcpyHostToDevice,
                              ctx->stream));
  if (!jobs.empty())
    FG_CUDA_TRY(cudaMemcpyAsync(B->d_jobs, jobs.data(), sizeof(BatchJob) * jobs.size(), cudaMemcpyHostToDevice,
                                ctx->stream));
  FG_CUDA_TRY(cudaMemcpyAsync(B->d_probs, B->probs.data(), sizeof(BatchProb) * B->nprob, cudaMemcpyHostToDevice,
                              ctx->stream));
  FG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return FG_OK;
}

static fg_status batch_time(fg_batch* B, float* ms) {
  cudaStream_t st = B->ctx->stream;
  cudaEvent_t e0, e1;
  FG_CUDA_TRY(cudaEventCreate(&e0));
  FG_CUDA_TRY(cudaEventCreate(&e1));
  FG_CUDA_TRY(cudaEventRecord(e0, st));
  fg_status s = batch_launch(B, st);
  FG_CUDA_TRY(cudaEventRecord(e1, st));
  FG_CUDA_TRY(cudaEventSynchronize(e1));
  cudaEventElapsedTime(ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return s;
}

static void batch_free(fg_batch* B) {
  if (!B) return;
  cudaSetDevice(B->ctx->device);
  cudaStreamSynchronize(B->ctx->stream);
  if (B->graph) cudaGraphExecDestroy(B->graph);
  for (void* p : B->owned) dev_free(B->ctx, p);
  delete B;
}

}  // namespace fg

using namespace fg;

extern "C" {

fg_status fg_batch_create(fg_ctx* ctx, int32_t nprob, const fg_batch_problem* probs, int32_t flags,
                          const fg_solver_params* params, int32_t threads, fg_batch** out) {
  if (!ctx || !probs || !params || !out || nprob < 1) {
    set_error("bad argument: ctx/probs/params/out/nprob");
    return FG_ERR_BADARG;
  }
  *out = nullptr;
  if (threads != 0 && threads != 128 && threads != 256 && threads != 512) {
    set_error("bad argument: threads must be 0 (autotune), 128, 256 or 512");
    return FG_ERR_BADARG;
  }
  if (!(params->rtol >= 0.0) || !(params->atol >= 0.0) || params->max_iters < 1) {
    set_error("bad argument: rtol/atol/max_iters");
    return FG_ERR_BADARG;
  }
  FG_CUDA_TRY(cudaSetDevice(ctx->device));
  const CallScope call(ctx->load);
  fg_batch* B = new fg_batch();
  B->ctx = ctx;
  if (const char* env = std::getenv("FG_BATCH_TEAM_SHARE"))
    if (std::atof(env) > 0.0) B->team_share = std::atof(env);
  B->nprob = nprob;
  B->flags = flags;
  B->prm = *params;
  const bool dev = (flags & FG_INPUTS_ON_DEVICE) != 0;
  int64_t voff = 0, eoff = 0, fstage = 0, xstage = 0;
  for (int i = 0; i < nprob; ++i) {
    const fg_batch_problem& q = probs[i];
    const bool no_interior = q.order * q.n - 1 <= 0;
    if (q.n < 1 || q.order < 1 || q.order > kBatchMaxP || !(q.coef > 0.0) || !q.qp_source || (!q.x && !no_interior)) {
      delete B;
      set_error("bad argument: problem %d (n >= 1, order 1..3, coef > 0, qp_source and x required)", i);
      return FG_ERR_BADARG;
    }
    if ((int64_t)(q.order * q.n + 1) * (q.order * q.n + 1) * (q.order * q.n + 1) >= (1ll << 31)) {
      delete B;
      set_error("problem %d: (order n + 1)^3 lattice nodes exceed the 32-bit index range", i);
      return FG_ERR_UNSUPPORTED;
    }
    BatchProb P;
    std::memset(&P, 0, sizeof(P));
    P.n = q.n;
    P.p = q.order;
    P.L = q.order * q.n + 1;
    P.F = q.order * q.n - 1;
    const double kh = q.coef * (0.5 / q.n) * line_scale(q.order);
    P.kh_hi = (float)kh;
    P.kh_lo = (float)(kh - (double)P.kh_hi);
    const double hh = 0.5 / q.n;
    P.h3 = hh * hh * hh;
    P.voff = voff;
    voff += 8 * (int64_t)P.L * P.L * P.L;
    const int64_t nq = (int64_t)(q.order + 1) * (q.order + 1) * (q.order + 1);
    const int64_t ncells = (int64_t)q.n * q.n * q.n;
    P.eoff = eoff;
    eoff += ncells * nq;
    B->nf.push_back(ncells * nq);
    const int64_t F3 = P.F > 0 ? (int64_t)P.F * P.F * P.F : 0;
    B->nx.push_back(F3);
    B->total_dofs += F3;
    B->user_f.push_back(q.qp_source);
    B->user_x.push_back(q.x);
    P.f = dev ? q.qp_source : nullptr;
    P.x = dev ? q.x : nullptr;
    fstage += ncells * nq;
    xstage += F3;
    B->probs.push_back(P);
  }
  fg_status s = FG_OK;
  auto A = [&](void** p, size_t b) { if (s == FG_OK) s = ba(B, p, b); };
  A((void**)&B->vpool, sizeof(float) * std::max<int64_t>(1, voff));
  A((void**)&B->epool, sizeof(double) * std::max<int64_t>(1, eoff));
  A((void**)&B->d_probs, sizeof(BatchProb) * nprob);
  A((void**)&B->d_tabs, sizeof(OrderTables) * kBatchMaxP);
  A((void**)&B->bar, sizeof(unsigned) * nprob);
  A((void**)&B->abort_all, sizeof(int));
  A((void**)&B->status, sizeof(int) * nprob);
  A((void**)&B->iters, sizeof(int) * nprob);
  A((void**)&B->refines, sizeof(int) * nprob);
  A((void**)&B->relres, sizeof(double) * nprob);
  if (!dev) {
    A((void**)&B->fstage, sizeof(double) * std::max<int64_t>(1, fstage));
    A((void**)&B->xstage, sizeof(double) * std::max<int64_t>(1, xstage));
  }
  if (s != FG_OK) {
    batch_free(B);
    return s;
  }
  if (!dev) {
    int64_t fo = 0, xo = 0;
    for (int i = 0; i < nprob; ++i) {
      B->probs[i].f = B->fstage + fo;
      B->probs[i].x = B->xstage + xo;
      fo += B->nf[i];
      xo += B->nx[i];
    }
  }
  // vectors: boundary nodes stay zero for the life of the plan
  cudaError_t e = cudaMemsetAsync(B->vpool, 0, sizeof(float) * std::max<int64_t>(1, voff), ctx->stream);
  OrderTables tabs[kBatchMaxP];
  for (int p = 1; p <= kBatchMaxP; ++p) build_order_tables(p, tabs[p - 1], B->line[p - 1]);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(B->d_tabs, tabs, sizeof(tabs), cudaMemcpyHostToDevice, ctx->stream);
  if (e != cudaSuccess) {
    set_error("batch setup: %s", cudaGetErrorString(e));
    batch_free(B);
    return FG_ERR_CUDA;
  }
  // block size: given, or the fastest of 128/256/512 on this batch (inputs must be valid);
  // large batches are timed on a stratified sample of at most 256 problems.  Team sizing is
  // not timed (a sample run with the full plan's team sizes lasts as long as its largest
  // problem, about half a full run): 0.5, or FG_BATCH_TEAM_SHARE
  if (threads == 0 && nprob > 256) {
    std::vector<int> order(nprob);
    std::iota(order.begin(), order.end(), 0);
    std::vector<double> w(nprob);
    for (int i = 0; i < nprob; ++i) w[i] = (double)B->nx[i] * avg_nnz(probs[i].order);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return w[x] > w[y]; });
    std::vector<fg_batch_problem> sub;
    const int stride = (nprob + 255) / 256;
    for (int k = 0; k < nprob; k += stride) sub.push_back(probs[order[k]]);
    auto t0 = std::chrono::steady_clock::now();
    fg_batch* S = nullptr;
    s = fg_batch_create(ctx, (int32_t)sub.size(), sub.data(), flags, params, 0, &S);
    if (s != FG_OK) {
      batch_free(B);
      return s;
    }
    threads = S->threads;
    batch_free(S);
    B->autotune_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  }
  if (threads == 0) {
    auto t0 = std::chrono::steady_clock::now();
    if (!dev) {
      for (int i = 0; i < nprob; ++i) {
        e = cudaMemcpyAsync((void*)B->probs[i].f, B->user_f[i], sizeof(double) * B->nf[i], cudaMemcpyHostToDevice,
                            ctx->stream);
        if (e != cudaSuccess) break;
      }
    }
    float best = 0.f;
    int best_t = 256;
    for (int t : {128, 256, 512}) {
      s = batch_plan(B, t);
      if (s != FG_OK) break;
      float ms = 0.f;
      s = batch_time(B, &ms);
      if (s != FG_OK) break;
      if (best == 0.f || ms < best) {
        best = ms;
        best_t = t;
      }
    }
    B->autotune_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    threads = best_t;
    if (s != FG_OK) {
      batch_free(B);
      return s;
    }
  }
  s = batch_plan(B, threads);
  if (s != FG_OK) {
    batch_free(B);
    return s;
  }
  // capture the launch (counter resets + the cooperative kernel) in a CUDA graph
  {
    cudaGraph_t g = nullptr;
    cudaStream_t st = ctx->stream;
    if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      fg_status ls = batch_launch(B, st);
      cudaError_t ce = cudaStreamEndCapture(st, &g);
      if (ls == FG_OK && ce == cudaSuccess && g && cudaGraphInstantiate(&B->graph, g, 0) == cudaSuccess)
        B->use_graph = true;
      if (g) cudaGraphDestroy(g);
      ctx->launches -= 1;  // the captured launch did not run
    }
    cudaGetLastError();
  }
  *out = B;
  return FG_OK;
}

fg_status fg_batch_run(fg_batch* B, fg_batch_result* results) {
  if (!B) {
    set_error("bad argument: batch");
    return FG_ERR_BADARG;
  }
  fg_ctx* ctx = B->ctx;
  FG_CUDA_TRY(cudaSetDevice(ctx->device));
  const CallScope call(ctx->load);
  cudaStream_t st = ctx->stream;
  const bool dev = (B->flags & FG_INPUTS_ON_DEVICE) != 0;
  cudaEvent_t e0, e1;
  FG_CUDA_TRY(cudaEventCreate(&e0));
  FG_CUDA_TRY(cudaEventCreate(&e1));
  FG_CUDA_TRY(cudaEventRecord(e0, st));
  if (!dev)
    for (int i = 0; i < B->nprob; ++i)
      FG_CUDA_TRY(cudaMemcpyAsync((void*)B->probs[i].f, B->user_f[i], sizeof(double) * B->nf[i],
                                  cudaMemcpyHostToDevice, st));
  if (B->use_graph) {
    FG_CUDA_TRY(cudaGraphLaunch(B->graph, st));
    ctx->launches += 1;
  } else {
    FG_TRY(batch_launch(B, st));
  }
  if (!dev)
    for (int i = 0; i < B->nprob; ++i)
      FG_CUDA_TRY(cudaMemcpyAsync(B->user_x[i], B->probs[i].x, sizeof(double) * B->nx[i], cudaMemcpyDeviceToHost, st));
  FG_CUDA_TRY(cudaEventRecord(e1, st));
  FG_CUDA_TRY(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  B->run_ms = ms;
  std::vector<int> stt(B->nprob), it(B->nprob), rf(B->nprob);
  std::vector<double> rr(B->nprob);
  FG_CUDA_TRY(cudaMemcpy(stt.data(), B->status, sizeof(int) * B->nprob, cudaMemcpyDeviceToHost));
  FG_CUDA_TRY(cudaMemcpy(it.data(), B->iters, sizeof(int) * B->nprob, cudaMemcpyDeviceToHost));
  FG_CUDA_TRY(cudaMemcpy(rf.data(), B->refines, sizeof(int) * B->nprob, cudaMemcpyDeviceToHost));
  FG_CUDA_TRY(cudaMemcpy(rr.data(), B->relres, sizeof(double) * B->nprob, cudaMemcpyDeviceToHost));
  fg_status worst = FG_OK;
  for (int i = 0; i < B->nprob; ++i) {
    if (results) {
      results[i].status = stt[i];
      results[i].iterations = it[i];
      results[i].refinements = rf[i];
      results[i].team = B->probs[i].team;
      results[i].rel_residual = rr[i];
    }
    if (stt[i] != 0 && (worst == FG_OK || stt[i] == FG_ERR_TIMEOUT)) worst = stt[i];
  }
  if (worst == FG_ERR_TIMEOUT) set_error("batch: a team barrier gave up");
  else if (worst == FG_ERR_NOT_CONVERGED) set_error("batch: some problems did not converge");
  return worst;
}

fg_status fg_batch_get_info(fg_batch* B, fg_batch_info* info) {
  if (!B || !info) {
    set_error("bad argument: batch/info");
    return FG_ERR_BADARG;
  }
  info->threads = B->threads;
  info->ctas = B->ctas;
  info->max_team = B->max_team;
  info->teams_gt1 = B->teams_gt1;
  info->graph = B->use_graph ? 1 : 0;
  info->total_dofs = B->total_dofs;
  info->predicted_balance = B->predicted_balance;
  info->run_ms = B->run_ms;
  info->autotune_ms = B->autotune_ms;
  info->team_share = B->team_share;
  return FG_OK;
}

fg_status fg_batch_destroy(fg_batch* B) {
  batch_free(B);
  return FG_OK;
}

}  // extern "C"
