// fg_ozaki.cu -- FP64 matrix products on the bf16 tensor cores (tcgen05) by digit slicing.
//
// GB300 runs FP64 at ~1 TFLOP/s (DFMA and the FP64 MMA alike) and bf16 MMAs at ~1.9
// PFLOP/s.  The dense FP64 products of the BDDC set-up are moved onto the tensor cores with
// the Ozaki scheme (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and its
// applications", Numer. Algorithms 59, 2012), in its fixed-point digit form (H. Ootomo,
// K. Ozaki, R. Yokota, "DGEMM on integer matrix multiplication unit", IJHPCA 2024), with
// bf16 digits instead of int8 ones because this part's int8 MMA rate is low:
//
//   * every row i of an operand gets a power of two 2^e_i with |x_il| 2^-e_i < 1/4 and is cut
//     into S = 7 signed digits, x_il = 2^e_i sum_s d_s 2^(-8(s+1)) (+ a tail below
//     2^(e_i-56)), |d_0| <= 64, |d_s| <= 128, so every digit is an exact bf16.  The cut is
//     integer arithmetic on the FP64 bit pattern (56 fraction bits, 54 of them below the row
//     maximum, digits rounded to nearest);
//   * the digit matrices are multiplied by tcgen05.mma kind::f16 (bf16 x bf16 -> FP32).  A
//     digit product is at most 2^14 (2^13 with a leading digit), and an accumulator sums at
//     most the equivalent of 6 full pairs (class 6: two leading-digit pairs and five others;
//     class 7: six others) over at most 170 K values: every FP32 partial sum is an integer
//     below 6 2^14 170 < 2^24, i.e. exact.  K up to 170 is one exact chunk (the Poisson
//     element matrices' K = 162 among them), longer K is cut into chunks of 160;
//   * the products of weight 2^(-8k), k = s + t = 0..7 (34 digit pairs), go to 8 FP32
//     accumulators in tensor memory (8 x 64 columns: all 512); pairs with s + t >= 8 are
//     dropped (|error| <~ K 2^-57 max_l |x_il| max_l |y_jl|).  The cut keeps 54 bits below
//     the row maximum, so a value far below it loses its low bits: overall the product is
//     within ~K 2^-52 max|x_i.| max|y_j.| of the exact one (about the FP64 dot-product bound);
//   * with S = 8 digits (the elasticity element matrices) the cut keeps 62 bits below the row
//     maximum and the error left is that of the dropped pairs, ~50 times smaller than the cut's
//     at S = 7 (36 pairs instead of 34; a class 7 sum could pass 2^24 by 11 % if every digit were
//     extreme, and would then round in its last bit, below what the dropped pairs leave out);
//   * the epilogue converts the 8 class sums to integers and adds them, over all chunks of K,
//     into one exact 96-bit integer per output element; that becomes FP64 with one rounding, and
//     the power of two 2^(e_i + f_j - 16) goes into the exponent field, all in integer arithmetic:
//     one FP64 operation per output element where C is updated, none where it is written.
//
// Digit layout in HBM: per operand, blocks of 128 rows x 16 columns (one MMA K step) per
// digit, 4 KB each, ordered [row tile][K step][digit]; inside a block the rows are in the
// canonical K-major, non-swizzled UMMA layout: core matrices of 8 rows x 16 bytes, the two
// 8-column halves 128 B apart (LBO), row groups 256 B apart (SBO).  An operand B tile of 64
// rows is half a block (2 KB).  A CTA computes 128 x 64 output tiles: warp 17's lane 0 streams
// the digit blocks into shared memory with cp.async.bulk (5 stages, mbarrier transaction
// counts), warp 0 issues the MMAs, warps 1-16 read the accumulators (tcgen05.ld, four warps per
// TMEM lane quarter, 16 columns each) and write C.  CTAs are persistent (one per SM, tiles
// round robin).  Every wait is bounded: after ~1 s the CTA records FG_ERR_TIMEOUT, stops, waits
// (bounded) for its copies and MMAs in flight, frees its tensor memory and returns.
//
// What bounds it: at 4096^3 the MMAs (34 digit pairs, 4.7 PFLOP of bf16 in 2.9 ms beside 0.2 ms
// of cutting: 1.6 PFLOP/s, 85 % of the measured bf16 rate; without any epilogue work the kernel
// takes as long).  At K = 128 (8192 x 8192: 0.44 ms) the MMAs run 56 % of the time and the epilogue's
// ~120 instructions per element, a C tile every 8 K steps, are as long.  From 13.7 to 44 TFLOP/s at 4096^3 (13 to
// 33 at K = 128): accumulators released before they are converted, MMAs issued from warp-uniform code,
// an A digit against four B digits per MMA, chunks of K added as integers, the classes in two halves with barriers
// of their own, a conversion without branches.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstdint>

#include "fg_internal.h"

namespace fg {

namespace {

constexpr int OZ_S = 7;                       // digits per value (8 where asked for)
constexpr int OZ_NACC = 8;                    // accumulators: digit weights k = s + t = 0..7
constexpr int OZ_BM = 128, OZ_BK = 16;
constexpr int OZ_KEXACT = 170;                // K values one exact accumulation may sum
constexpr int OZ_CHUNK_STEPS = 10;            // K steps of a chunk when K > OZ_KEXACT (160 values)
constexpr uint32_t OZ_BLOCK = OZ_BM * OZ_BK * 2;           // one digit block: 4096 B
constexpr uint32_t oz_a_bytes(int S) { return S * OZ_BLOCK; }  // a row tile's digits per K step
constexpr uint32_t OZ_TMEM_COLS = 512;                     // all of it
constexpr long long OZ_WAIT_CYCLES = 1ll << 31;            // ~1 s at 2 GHz
constexpr int OZ_EPI_WARPS = 16;                           // epilogue warps: 4 per TMEM lane quarter
constexpr int OZ_NONFINITE = 1 << 28;                      // row exponent of a row with a NaN or an infinity
constexpr int OZ_THREADS = (OZ_EPI_WARPS + 2) * 32;        // with the MMA warp (0) and the copy warp (17)

// Output tiles of 128 x BN: the 8 accumulators of BN = 64 columns fill the tensor memory.
constexpr int OZ_BN = 64;
template <int BN, int S>
struct OzT {
  static_assert(OZ_NACC * BN == (int)OZ_TMEM_COLS, "the accumulators fill the tensor memory");
  static constexpr int EPI = BN * 4 / OZ_EPI_WARPS;           // columns per epilogue thread
  static constexpr int QB = OZ_BM / BN;                       // B tiles per 128-row digit block
  static constexpr uint32_t B_DIGIT = BN * OZ_BK * 2;         // one digit of a B tile per K step
  static constexpr uint32_t A_BYTES = oz_a_bytes(S);
  static constexpr uint32_t STAGE = A_BYTES + S * B_DIGIT;
  static constexpr int NBUF = S == 7 ? 5 : 4;                 // stages: 215040 or 196608 B
  static constexpr uint32_t SMEM = NBUF * STAGE;
  // kind::f16: FP32 accumulator, bf16 A and B, both K-major, N = nd digits of BN, M = 128
  static constexpr uint32_t idesc(int nd) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nd * BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
  }
};
constexpr int OZ_MAXBUF = 5;

// ---- PTX wrappers -------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
// global -> own shared memory, completion counted in bytes on the mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
// one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, 128 x N x 16, bf16 -> FP32
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// arrive on the mbarrier once every tcgen05 operation issued so far by this thread is done
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, no swizzle; LBO = 128 B (the two 8-column
// halves of a 16-column step), SBO = 256 B (consecutive 8-row groups); version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(256u >> 4) << 32) |
         (1ull << 46);
}

// bounded wait; false (and the CTA's abort flag and the error status set) when it runs out
// after an abort: wait (bounded, ignoring the abort flag) for the copies or MMAs still in
// flight, so that nothing writes this CTA's shared or tensor memory once it is released
__device__ __forceinline__ void mbar_drain(uint32_t a, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try(a, parity)) {
    __nanosleep(64);
    if (clock64() - t0 > OZ_WAIT_CYCLES) return;
  }
}

__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, volatile int* abort_flag, int* err) {
  const long long t0 = clock64();
  int spins = 0;
  while (!mbar_try(a, parity)) {
    if (*abort_flag) return false;
    if (++spins > 64) __nanosleep(64);
    if (clock64() - t0 > OZ_WAIT_CYCLES) {
      *abort_flag = 1;
      atomicExch(err, (int)FG_ERR_TIMEOUT);
      return false;
    }
  }
  return true;
}

}  // namespace

// ---- operands: one or more row blocks cut into digits ------------------------------------
// A split item: rows x k values, element (r, l) at x[r*rs + l*cs], cut into the digit row
// tiles rtile0 .. rtile0 + ceil(rows/128) - 1 of the workspace (exponents at 128 rtile + r).
struct OzSplit {
  const double* x;
  int64_t rs, cs;
  int rows, k;
  int rtile0;
};
struct OzSplitArgs {
  const OzSplit* items;  // device array, or nullptr: one[0 .. none-1]
  int nitems;
  OzSplit one[2];
  int none;
  int ksteps;
  int32_t* ex;
  uint4* dig;
};

__device__ __forceinline__ OzSplit split_of(const OzSplitArgs& a, int rtile) {
  if (!a.items) return (a.none > 1 && rtile >= a.one[1].rtile0) ? a.one[1] : a.one[0];
  int lo = 0, hi = a.nitems - 1;  // last item with rtile0 <= rtile
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.items[mid].rtile0 <= rtile) lo = mid;
    else hi = mid - 1;
  }
  return a.items[lo];
}

// Row exponents: e_r with max_l |x_rl| < 2^(e_r - 2), from the largest biased exponent of
// the row (an all-zero or padding row gets 0).  Blocks (digit row tile, part of 32).  Rows
// with consecutive elements (cs == 1): a warp per row, lanes along it, part p taking rows
// 4p .. 4p + 3.  Otherwise part p < 4 takes rows 32p .. 32p + 31 (consecutive rows are
// consecutive in memory), a warp per quarter of the columns: one thread per row walking the
// 128 columns of a Cholesky panel alone took 56 us of load latency.
__global__ void __launch_bounds__(OZ_BM) k_oz_rowexp(OzSplitArgs a) {
  __shared__ unsigned long long s_mx[OZ_BM / 32][32];
  const int rtile = blockIdx.x;
  const OzSplit it = split_of(a, rtile);
  if (it.cs != 1 && blockIdx.y >= OZ_BM / 32) return;
  const int64_t r0 = (int64_t)(rtile - it.rtile0) * OZ_BM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto finish = [&](int local, unsigned long long mx) {
    const int E = (int)(mx >> 52);  // biased exponent of the largest |x| (0: zero/subnormal)
    // a NaN or an infinity in the row: no digits, the epilogue makes its results NaN
    a.ex[(int64_t)rtile * OZ_BM + local] = E == 0x7FF ? OZ_NONFINITE : mx == 0 ? 0 : (E == 0 ? 1 : E) - 1020;
  };
  auto bits = [&](int64_t r, int64_t l) {
    return (unsigned long long)__double_as_longlong(it.x[r * it.rs + l * it.cs]) & 0x7FFFFFFFFFFFFFFFull;
  };
  unsigned long long mx = 0;
  if (it.cs == 1) {
    const int local = blockIdx.y * (OZ_BM / 32) + warp;
    const int64_t r = r0 + local;
    if (r < it.rows)
      for (int64_t l = lane; l < it.k; l += 32) mx = max(mx, bits(r, l));
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) finish(local, mx);
  } else {
    const int local = blockIdx.y * 32 + lane;
    const int64_t r = r0 + local;
    if (r < it.rows) {
      const int64_t q = (it.k + 3) / 4, l1 = min((int64_t)it.k, q * (warp + 1));
#pragma unroll 8
      for (int64_t l = q * warp; l < l1; ++l) mx = max(mx, bits(r, l));
    }
    s_mx[warp][lane] = mx;
    __syncthreads();
    if (warp == 0) finish(local, max(max(mx, s_mx[1][lane]), max(s_mx[2][lane], s_mx[3][lane])));
  }
}

// Digits: block (digit row tile, K step), thread per row; 16 values, S digits each, written as
// the S digit blocks' 32-byte rows.  Rows past the item and columns >= k are zero.
template <int S>
__global__ void __launch_bounds__(OZ_BM) k_oz_split(OzSplitArgs a) {
  const int tid = threadIdx.x;
  const int rtile = blockIdx.x, ks = blockIdx.y;
  const OzSplit it = split_of(a, rtile);
  const int64_t r = (int64_t)(rtile - it.rtile0) * OZ_BM + tid;
  const int er = a.ex[(int64_t)rtile * OZ_BM + tid];
  uint32_t w[S][8];
#pragma unroll
  for (int c = 0; c < OZ_BK; c += 2) {
    int32_t d[2][S];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t l = (int64_t)ks * OZ_BK + c + h;
      const double v = (r < it.rows && l < it.k) ? it.x[r * it.rs + l * it.cs] : 0.0;
      const unsigned long long b = (unsigned long long)__double_as_longlong(v);
      const int E = (int)((b >> 52) & 0x7FF);
      const long long mant = (long long)(b & 0xFFFFFFFFFFFFFull) | (E ? (1ll << 52) : 0ll);
      // F = |v| 2^(8 S - e_r) as an integer: v = mant 2^(max(E,1) - 1075)
      const int sh = (E ? E : 1) - 1075 + 8 * S - er;  // F < 2^(8 S - 2) by the choice of e_r
      long long F = sh >= 0 ? (mant << sh) : (sh > -64 ? (mant >> -sh) : 0ll);
      if (b >> 63) F = -F;
#pragma unroll
      for (int s = 0; s < S - 1; ++s) {
        const int q = 8 * (S - 1 - s);
        const long long dg = (F + (1ll << (q - 1))) >> q;  // nearest digit, in [-128, 128] ([-64, 64] for s = 0)
        F -= dg << q;
        d[h][s] = (int32_t)dg;
      }
      d[h][S - 1] = (int32_t)F;  // |F| <= 128 after the others
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      // small integers are exact in bf16: the upper half of their FP32 pattern
      const uint32_t lo = __float_as_uint((float)d[0][s]) >> 16;
      const uint32_t hi = __float_as_uint((float)d[1][s]) >> 16;
      w[s][c / 2] = lo | (hi << 16);
    }
  }
  const size_t blk = ((size_t)rtile * a.ksteps + ks) * S;
  const int g = tid >> 3, r8 = tid & 7;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    uint4* p = a.dig + (blk + s) * (OZ_BLOCK / 16);
    p[g * 16 + r8] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);      // columns 0-7
    p[g * 16 + 8 + r8] = make_uint4(w[s][4], w[s][5], w[s][6], w[s][7]);  // columns 8-15
  }
}

// ---- products --------------------------------------------------------------------------
// One product of a launch: C (m x n; (i, j) at c[i*c_rs + j*c_cs]) from the digit row tiles
// arow0.. (A) and brow0.. (B); its output tiles are tile0 .. tile0 + ceil(m/128) tiles_n - 1.
struct OzItem {
  double* c;
  int64_t c_rs, c_cs;
  int m, n;
  int arow0, brow0;
  int tiles_n;
  int tile0;
  int tiles_m;  // > 0: tiles numbered down the columns (tiles_m row tiles each); -1: along the
                // rows, only the tiles that reach the lower triangle (row tile r has 2 r + 2 of
                // them, at most tiles_n).  With the others numbered too and skipped, a round robin
                // gave one CTA 50 and another 25 tiles of 9492 x 9492 (now 38 and 37: the coarse
                // updates of 24^3 BDDC 525 -> 405 us)
  __host__ __device__ int64_t lower_full() const { return (int64_t)(tiles_n / 2) * (tiles_n / 2 + 1); }
  __device__ __forceinline__ void locate(int t, int& rt, int& ct) const {
    const int lt = t - tile0;
    if (tiles_m > 0) {
      ct = lt / tiles_m;
      rt = lt - ct * tiles_m;
    } else if (tiles_m == 0) {
      rt = lt / tiles_n;
      ct = lt - rt * tiles_n;
    } else if (lt < lower_full()) {
      // tiles before row r: r (r + 1)
      rt = (int)((sqrtf(4.0f * (float)lt + 1.0f) - 1.0f) * 0.5f);
      while ((int64_t)rt * (rt + 1) > lt) --rt;
      while ((int64_t)(rt + 1) * (rt + 2) <= lt) ++rt;
      ct = lt - rt * (rt + 1);
    } else {
      const int r = (int)(lt - lower_full());
      rt = tiles_n / 2 + r / tiles_n;
      ct = r % tiles_n;
    }
  }
};
// output tiles of an m x n product, all or those of the lower triangle
static int64_t lower_tiles(int64_t tiles_m, int64_t tiles_n) {
  const int64_t r = std::min(tiles_m, tiles_n / 2);
  return r * (r + 1) + (tiles_m - r) * tiles_n;
}

struct OzGemmArgs {
  const uint8_t* dig;    // digit blocks [row tile][K step][digit]
  const int32_t* ex;     // row exponents [row tile][128]
  const OzItem* items;   // device array, or nullptr: `one`
  int nitems;
  OzItem one;
  int ntiles;            // output tiles of all items
  int ksteps;
  int chunk;             // K steps per exact accumulation
  double alpha, beta;
  int lower;             // write only i >= j
  int drop_stage;        // test switch (FG_OZ_TEST_DROP_STAGE): CTA 0 never issues this stage's copies
  int* err;
};

__device__ __forceinline__ OzItem item_of(const OzGemmArgs& g, int t) {
  if (!g.items) return g.one;
  int lo = 0, hi = g.nitems - 1;  // last item with tile0 <= t
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (g.items[mid].tile0 <= t) lo = mid;
    else hi = mid - 1;
  }
  return g.items[lo];
}

// (h 2^32 + l) 2^(off - 72) as FP64, rounded to nearest (ties to even), the sign flipped by flip =
// 2^31, by integer operations and without a branch (the columns' chains then overlap).  slow: the
// result is not a normal FP64 number; sum_slow does it.
__device__ __forceinline__ double sum_f64(long long h, uint32_t l, int off, uint32_t flip, bool& slow) {
  const uint32_t sgn = (uint32_t)(h >> 63);  // 0 or all ones: |x| = (x ^ sgn) - sgn
  const unsigned long long lo = (unsigned long long)(l ^ sgn) + (sgn & 1u);
  const unsigned long long a = ((unsigned long long)h ^ (unsigned long long)(h >> 63)) + (lo >> 32);
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, al2 = (uint32_t)lo;
  // the upper word with the leading bit (a2), and the two after it
  const uint32_t b2 = al ? al : al2, b1 = al ? al2 : 0u;
  const uint32_t a2 = ah ? ah : b2, a1 = ah ? al : b1, a0 = ah ? al2 : 0u;
  const int lz = __clz((int)a2);  // 32: the sum is zero
  const uint32_t n2 = __funnelshift_l(a1, a2, lz), n1 = __funnelshift_l(a0, a1, lz), n0 = a0 << (lz & 31);
  const int e = off + (1023 + 95 - 72) - (ah ? 0 : (al ? 32 : 64)) - lz;  // biased exponent of the leading bit
  slow = a2 != 0 && (unsigned)(e - 1) > 2044u;                            // 2046 could round up to infinity
  const unsigned long long m = ((unsigned long long)n2 << 21) | (n1 >> 11);  // 53 bits, the leading one included
  // half an ulp is 0x400 of the 11 bits left; the bits below them and an odd m break the tie
  const uint32_t up = ((n1 & 0x7FFu) * 2 + (n0 != 0 ? 1u : 0u) + ((uint32_t)m & 1u)) > 0x800u ? 1u : 0u;
  const uint32_t top = a2 != 0 ? ((uint32_t)(e - 1) << 20) + ((sgn ^ flip) & 0x80000000u) : 0u;
  return __longlong_as_double((long long)(m + up + ((unsigned long long)top << 32)));
}

// the same for any sum (kept out of line: it costs FP64 operations)
__device__ __noinline__ double sum_slow(long long h, uint32_t l, int off, uint32_t flip) {
  if (off >= OZ_NONFINITE / 2) return __longlong_as_double(0x7FF8000000000000ll);
  bool slow;
  return ldexp(sum_f64(h, l, 0, flip, slow), off);
}

// Persistent: CTA b takes the output tiles b, b + gridDim.x, ... of all items (lower: those that reach
// the triangle).  The accumulators are released as soon as the epilogue
// has read them, so the next tile's MMAs run while the epilogue writes C.
template <int BN, int S>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_oz_gemm(OzGemmArgs g) {
  using T = OzT<BN, S>;
  constexpr int OZ_NBUF = T::NBUF;
  extern __shared__ __align__(1024) uint8_t oz_smem[];
  __shared__ __align__(8) uint64_t bar_full[OZ_MAXBUF], bar_empty[OZ_MAXBUF], bar_acc_full[2], bar_acc_empty[2], bar_stop;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntiles = g.ntiles;
  auto next_tile = [&](int t) { return t + (int)gridDim.x; };
  const int first = blockIdx.x;
  if (first >= ntiles) return;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(OZ_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    if (lane == 0) {
      for (int i = 0; i < OZ_NBUF; ++i) {
        mbar_init(smem_u32(&bar_full[i]), 1);
        mbar_init(smem_u32(&bar_empty[i]), 1);
      }
      for (int z = 0; z < 2; ++z) {
        mbar_init(smem_u32(&bar_acc_full[z]), 1);
        mbar_init(smem_u32(&bar_acc_empty[z]), OZ_EPI_WARPS);
      }
      mbar_init(smem_u32(&bar_stop), 1);
      abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int KS = g.ksteps;
  const int nchunks = (KS + g.chunk - 1) / g.chunk;

  const uint32_t sbase = smem_u32(oz_smem);
  if (warp == 0) {
    // MMA warp.  The whole warp runs the loop and one elected lane issues: the descriptors then
    // stay in uniform registers.  (Issued from a branch on lane == 0, an MMA cost ~80 cycles
    // of moves to the uniform registers, more than the 32 it runs.)
    //
    // An MMA takes an A digit against up to four B digits: digits t, t + 1, .. of the stage are
    // consecutive rows of one operand and their classes s + t, .. consecutive accumulators.
    // The K steps of a chunk go in groups of NBUF stages, per group first the classes 0-3 (lo) of
    // every stage, then the classes 4-7 (hi), each half with its own pair of barriers: the
    // epilogue takes the lo sums out while the last group's hi MMAs run, and the hi sums while
    // the next chunk's lo MMAs do.
    bool ok = true;
    int gs = 0, gc = 0;
    const uint64_t d0 = smem_desc(sbase);
    for (int t = first; t < ntiles && ok; t = next_tile(t)) {
      for (int c0 = 0; c0 < KS && ok; c0 += g.chunk, ++gc) {
        const int c1 = min(KS, c0 + g.chunk);
        for (int g0 = c0; g0 < c1 && ok; g0 += OZ_NBUF) {
          const int ng = min(OZ_NBUF, c1 - g0);
          const bool last = g0 + ng == c1;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (g0 == c0 && gc > 0 && ok)
              ok = mbar_wait(smem_u32(&bar_acc_empty[half]), (gc - 1) & 1, &abort_flag, g.err);
            for (int q = 0; q < ng; ++q) {
              const int buf = (gs + q) % OZ_NBUF;
              if (half == 0) ok = ok && mbar_wait(smem_u32(&bar_full[buf]), ((gs + q) / OZ_NBUF) & 1, &abort_flag, g.err);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok) break;
              tc_fence_after();
              if (elect_one()) {
                const uint64_t da = d0 + (uint64_t)((uint32_t)buf * (T::STAGE >> 4)), db = da + (T::A_BYTES >> 4);
                // the first pair of a class starts the chunk's sum: s = 0, and s = 1 for class 7
                // of S = 7 (t = 6), which then goes by itself
                const uint32_t cont = g0 + q > c0 ? 1u : 0u;
                auto mma = [&](int s, int t0, int nd, uint32_t acc) {
                  tc_mma(tmem + (s + t0) * BN, da + (uint64_t)(s * (OZ_BLOCK >> 4)),
                         db + (uint64_t)(t0 * (T::B_DIGIT >> 4)), T::idesc(nd), acc);
                };
                if (half == 0) {
#pragma unroll
                  for (int s = 0; s < 4; ++s) mma(s, 0, 4 - s, s == 0 ? cont : 1u);
                } else {
#pragma unroll
                  for (int s = 0; s < S; ++s) {
                    const int t0 = s < 4 ? 4 - s : 0, t1 = 7 - s < S - 1 ? 7 - s : S - 1;
                    if (S == 7 && s == 1 && cont == 0) {
                      mma(s, t0, t1 - t0, 1u);
                      mma(s, t1, 1, 0u);
                    } else {
                      mma(s, t0, t1 - t0 + 1, s == 0 ? cont : 1u);
                    }
                  }
                  tc_commit(smem_u32(&bar_empty[buf]));
                }
                if (last && q == ng - 1) tc_commit(smem_u32(&bar_acc_full[half]));
              }
              __syncwarp();
            }
          }
          gs += ng;
        }
      }
    }
    // after an abort: every MMA issued
    if (!ok) {
      if (elect_one()) tc_commit(smem_u32(&bar_stop));
      __syncwarp();
      mbar_drain(smem_u32(&bar_stop), 0);
    }
    __syncwarp();
  } else if (warp == OZ_EPI_WARPS + 1) {
    // copy warp: lane 0 streams the stages
    if (lane == 0) {
      bool ok = true;
      int gs = 0;
      for (int t = first; t < ntiles && ok; t = next_tile(t)) {
        const OzItem it = item_of(g, t);
        int rt, ct;
        it.locate(t, rt, ct);
        const uint8_t* pa = g.dig + (size_t)(it.arow0 + rt) * KS * T::A_BYTES;
        const uint8_t* pb =
            g.dig + (size_t)(it.brow0 + ct / T::QB) * KS * T::A_BYTES + (size_t)(ct % T::QB) * T::B_DIGIT;
        for (int ks = 0; ks < KS; ++ks, ++gs) {
          const int buf = gs % OZ_NBUF;
          if (gs >= OZ_NBUF && !mbar_wait(smem_u32(&bar_empty[buf]), ((gs / OZ_NBUF) - 1) & 1, &abort_flag, g.err)) {
            ok = false;
            break;
          }
          const uint32_t full = smem_u32(&bar_full[buf]);
          const uint32_t dst = sbase + buf * T::STAGE;
          mbar_expect_tx(full, T::STAGE);
          if (blockIdx.x == 0 && gs == g.drop_stage) continue;
          bulk_g2s(dst, pa + (size_t)ks * T::A_BYTES, T::A_BYTES, full);
          for (int d = 0; d < S; ++d)
            bulk_g2s(dst + T::A_BYTES + d * T::B_DIGIT, pb + ((size_t)ks * S + d) * OZ_BLOCK, T::B_DIGIT, full);
        }
      }
      // nothing may land in this CTA's shared memory after it is gone (an abort elsewhere leaves
      // copies nobody waits for): wait for the last one into each stage
      for (int q = gs > OZ_NBUF ? gs - OZ_NBUF : 0; q < gs; ++q)
        mbar_drain(smem_u32(&bar_full[q % OZ_NBUF]), (q / OZ_NBUF) & 1);
    }
    __syncwarp();
  } else {
    // epilogue: warps 1-16; warp w reads TMEM lanes 32 (w % 4) .. +31 (tile rows), columns
    // EPI h .. EPI h + EPI - 1 with h = (w - 1) / 4.  The next tile's MMAs need the
    // accumulators, so a warp first takes all its class sums as integers (hi, lo per column)
    // and releases them; the conversion to FP64 and the update of C run beside those MMAs.
    constexpr int OZ_EPI_COLS = T::EPI;
    const int quarter = warp & 3, part4 = (warp - 1) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t trow0 = tmem + ((uint32_t)(quarter * 32) << 16) + part4 * OZ_EPI_COLS;
    // alpha, beta cases as integers, decided once (an FP64 compare per element would cost as
    // much as the element's arithmetic)
    const int amode = g.alpha == -1.0 ? 0 : (g.alpha == 1.0 ? 1 : 2);
    const int bmode = g.beta == 0.0 ? 0 : (g.beta == 1.0 ? 1 : 2);
    const uint32_t flip = amode == 0 ? 0x80000000u : 0u;
    int gc = 0;
    for (int t = first; t < ntiles; t = next_tile(t)) {
      if (bmode != 0) {
        // C is needed after the sums: ask L2 for this thread's elements while the MMAs run
        const OzItem it = item_of(g, t);
        int rt, ct;
        it.locate(t, rt, ct);
        const int i = rt * OZ_BM + row, c0 = ct * BN + part4 * OZ_EPI_COLS;
        const int nv = i < it.m ? min(it.n - c0, g.lower ? i - c0 + 1 : OZ_EPI_COLS) : 0;
        const double* p = it.c + (int64_t)i * it.c_rs + (int64_t)c0 * it.c_cs;
#pragma unroll
        for (int j = 0; j < OZ_EPI_COLS; ++j)
          if (j < nv) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (int64_t)j * it.c_cs));
      }
      // per column: the product / 2^(e_i + f_j - 16) as an exact integer H 2^-24 + L 2^-56 over
      // all K chunks (|H| < 2^44 per chunk, at most 2^16 K steps), three registers
      long long H[OZ_EPI_COLS];
      uint32_t L[OZ_EPI_COLS];
#pragma unroll
      for (int j = 0; j < OZ_EPI_COLS; ++j) {
        H[j] = 0;
        L[j] = 0;
      }
      bool ok = true;
      for (int chunk = 0; chunk < nchunks; ++chunk, ++gc) {
        // sum_k v_k 2^(-8k), every v_k an integer below 2^24 held in FP32
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          ok = ok && mbar_wait(smem_u32(&bar_acc_full[half]), gc & 1, &abort_flag, g.err);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int cb = 0; cb < OZ_EPI_COLS / 8; ++cb) {
            uint32_t v[OZ_NACC / 2][8];
#pragma unroll
            for (int q = 0; q < OZ_NACC / 2; ++q) tc_ld8(trow0 + (half * 4 + q) * BN + cb * 8, v[q]);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              int a[OZ_NACC / 2];
#pragma unroll
              for (int q = 0; q < OZ_NACC / 2; ++q) a[q] = __float2int_rn(__uint_as_float(v[q][j]));
              // as multiply-adds into 64 bits (|a0| < 2^19.5, |a1| < 2^21.5, |a2| < 2^22.5,
              // |a3| < 2^23: those two pairs fit 32 bits)
              long long& h = H[cb * 8 + j];
              if (half == 0) {
                h += (long long)(a[0] * 256 + a[1]) * 65536;
                h += a[2] * 256 + a[3];
              } else {
                long long x = (long long)a[0] * 16777216 + (long long)(unsigned long long)L[cb * 8 + j];
                x += (long long)a[1] * 65536;
                x += (long long)a[2] * 256;
                x += a[3];
                h += x >> 32;
                L[cb * 8 + j] = (uint32_t)x;
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          // accumulators free: the next MMAs on them may start
          if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[half]));
        }
        if (!ok) break;
      }
#pragma unroll
      for (int j = 0; j < OZ_EPI_COLS; ++j)
        // keeps the update of C below the release (volatile statements stay in order)
        asm volatile("" : "+l"(H[j]), "+r"(L[j]));
      if (!ok) break;
      const OzItem it = item_of(g, t);
      int rt, ct;
      it.locate(t, rt, ct);
      const int i = rt * OZ_BM + row;
      const int c0 = ct * BN + part4 * OZ_EPI_COLS;
      const int ei = g.ex[(int64_t)(it.arow0 + rt) * OZ_BM + row];
      // lane j < EPI holds the exponent of column c0 + j (padding rows of the exponents are 0)
      const int ecol = g.ex[(int64_t)(it.brow0 + ct / T::QB) * OZ_BM + (ct % T::QB) * BN + part4 * OZ_EPI_COLS +
                            (lane < OZ_EPI_COLS ? lane : 0)];
      // a row of A or B in this warp's part holds a NaN or an infinity
      const bool nonfinite = __any_sync(0xffffffffu, max(ei, ecol) == OZ_NONFINITE);
      const int nv = i < it.m ? min(it.n - c0, g.lower ? i - c0 + 1 : OZ_EPI_COLS) : 0;  // columns to write
      double* crow = it.c + (int64_t)i * it.c_rs + (int64_t)c0 * it.c_cs;
#pragma unroll
      for (int j0 = 0; j0 < OZ_EPI_COLS; j0 += 8) {
        // eight columns at a time: their C values are loaded before any store
        double cv[8], xs[8];
        bool any = nonfinite;
#pragma unroll
        for (int j = 0; j < 8; ++j) cv[j] = (j0 + j < nv && bmode != 0) ? crow[(int64_t)(j0 + j) * it.c_cs] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          bool slow;  // x = (-)(H 2^(off - 40) + L 2^(off - 72))
          xs[j] = sum_f64(H[j0 + j], L[j0 + j], ei + __shfl_sync(0xffffffffu, ecol, j0 + j), flip, slow);
          any |= slow;
        }
        if (__any_sync(0xffffffffu, any))
#pragma unroll
          for (int j = 0; j < 8; ++j)
            xs[j] = sum_slow(H[j0 + j], L[j0 + j], ei + __shfl_sync(0xffffffffu, ecol, j0 + j), flip);
        if (amode != 2 && bmode != 2) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j0 + j < nv) crow[(int64_t)(j0 + j) * it.c_cs] = bmode == 0 ? xs[j] : cv[j] + xs[j];
        } else {
          const double alpha = amode == 0 ? 1.0 : g.alpha;  // -1: in the sign already
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j0 + j < nv)
              crow[(int64_t)(j0 + j) * it.c_cs] = bmode == 0 ? alpha * xs[j] : fma(alpha, xs[j], bmode == 1 ? cv[j] : g.beta * cv[j]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS) : "memory");
  }
}

// k = 0: C = beta C (the product is empty).
__global__ void k_oz_scale(int64_t m, int64_t n, double beta, double* c, int64_t c_rs, int64_t c_cs, int lower) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= m * n) return;
  const int64_t i = idx % m, j = idx / m;
  if (lower && j > i) return;
  double* cp = c + i * c_rs + j * c_cs;
  *cp = beta == 0.0 ? 0.0 : beta * *cp;
}

static int64_t rtiles_of(int64_t rows) { return (rows + OZ_BM - 1) / OZ_BM; }

size_t ozaki_workspace_bytes(int64_t m, int64_t n, int64_t k, bool same, int digits) {
  const int64_t rt = rtiles_of(m) + (same ? 0 : rtiles_of(n));
  const int64_t ks = std::max<int64_t>(1, (k + OZ_BK - 1) / OZ_BK);
  return (size_t)rt * ks * oz_a_bytes(digits) + (size_t)rt * OZ_BM * sizeof(int32_t) + 256;
}

template <int BN, int S>
static fg_status oz_gemm_launch(fg_ctx* ctx, cudaStream_t st, OzGemmArgs& g, int64_t ntiles) {
  FG_CUDA_TRY(cudaFuncSetAttribute((const void*)k_oz_gemm<BN, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)OzT<BN, S>::SMEM));
  // persistent: one CTA per SM (the shared memory allows no second), at most one per tile
  k_oz_gemm<BN, S><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ntiles, ctx->sm_count)), OZ_THREADS,
                  OzT<BN, S>::SMEM, st>>>(g);
  return FG_OK;
}

template <int S>
static fg_status oz_launch(fg_ctx* ctx, cudaStream_t st, OzSplitArgs& sa, int64_t rtiles, OzGemmArgs& g,
                           int64_t ntiles) {
  // test switch for the failure-detection test: a stage whose copies never arrive makes the
  // bounded wait run out (FG_ERR_TIMEOUT) without a fault
  const char* drop = std::getenv("FG_OZ_TEST_DROP_STAGE");
  g.drop_stage = drop ? std::atoi(drop) : -1;
  k_oz_rowexp<<<dim3((unsigned)rtiles, 32), OZ_BM, 0, st>>>(sa);
  k_oz_split<S><<<dim3((unsigned)rtiles, (unsigned)sa.ksteps), OZ_BM, 0, st>>>(sa);
  FG_TRY((oz_gemm_launch<OZ_BN, S>(ctx, st, g, ntiles)));
  ctx->launches += 3;
  FG_CUDA_TRY(cudaGetLastError());
  return FG_OK;
}

// C = alpha A B^T + beta C (lower: only i >= j).  B == nullptr: B = A (same strides).
fg_status ozaki_gemm_nt(fg_ctx* ctx, cudaStream_t st, int64_t m, int64_t n, int64_t k, double alpha,
                        const double* A, int64_t a_rs, int64_t a_cs, const double* B, int64_t b_rs, int64_t b_cs,
                        double beta, double* C, int64_t c_rs, int64_t c_cs, bool lower, void* work, int* d_err,
                        int digits) {
  if (m <= 0 || n <= 0) return FG_OK;
  if (k <= 0) {
    if (beta != 1.0) {
      k_oz_scale<<<(unsigned)((m * n + 255) / 256), 256, 0, st>>>(m, n, beta, C, c_rs, c_cs, lower ? 1 : 0);
      ctx->launches += 1;
      FG_CUDA_TRY(cudaGetLastError());
    }
    return FG_OK;
  }
  const bool same = B == nullptr;
  // The epilogue's lanes are consecutive rows of a tile: a row-major C is computed as its
  // transpose B A^T, so that a warp's store is 256 contiguous bytes instead of 32 sectors (the
  // digit sums are exact integers: the same results bit for bit).
  if (c_cs == 1 && c_rs != 1 && !lower) {
    if (!same) {
      std::swap(A, B);
      std::swap(a_rs, b_rs);
      std::swap(a_cs, b_cs);
    }
    std::swap(m, n);
    std::swap(c_rs, c_cs);
  }
  const int64_t ksteps = (k + OZ_BK - 1) / OZ_BK;
  const int64_t rta = rtiles_of(m), rtb = same ? 0 : rtiles_of(n);
  const int64_t tiles_n = (n + OZ_BN - 1) / OZ_BN;
  if (rta * tiles_n > (1ll << 31) - 1 || rta + rtb > (1ll << 31) - 1 || ksteps > 65535) {
    set_error("ozaki_gemm_nt: %lld x %lld x %lld is too large", (long long)m, (long long)n, (long long)k);
    return FG_ERR_UNSUPPORTED;
  }
  OzSplitArgs sa;
  sa.items = nullptr;
  sa.nitems = 0;
  sa.one[0] = OzSplit{A, a_rs, a_cs, (int)m, (int)k, 0};
  sa.one[1] = OzSplit{B, b_rs, b_cs, (int)n, (int)k, (int)rta};
  sa.none = same ? 1 : 2;
  sa.ksteps = (int)ksteps;
  sa.dig = (uint4*)work;
  sa.ex = (int32_t*)((uint8_t*)work + (size_t)(rta + rtb) * ksteps * oz_a_bytes(digits));
  OzGemmArgs g;
  g.dig = (const uint8_t*)work;
  g.ex = sa.ex;
  g.items = nullptr;
  g.nitems = 1;
  // consecutive CTAs walk the shorter side of the tile grid: the longer operand's digits are
  // read from HBM once and shared through L2
  g.one = OzItem{C, c_rs, c_cs, (int)m, (int)n, 0, same ? 0 : (int)rta, (int)tiles_n, 0,
                 lower ? -1 : (rta < tiles_n ? (int)rta : 0)};
  const int64_t ntiles = lower ? lower_tiles(rta, tiles_n) : rta * tiles_n;
  g.ntiles = (int)ntiles;
  g.ksteps = (int)ksteps;
  g.chunk = k <= OZ_KEXACT ? (int)ksteps : OZ_CHUNK_STEPS;
  g.alpha = alpha;
  g.beta = beta;
  g.lower = lower ? 1 : 0;
  g.err = d_err;
  return digits == 8 ? oz_launch<8>(ctx, st, sa, rta + rtb, g, ntiles)
                     : oz_launch<OZ_S>(ctx, st, sa, rta + rtb, g, ntiles);
}

// Batch of lower updates C_b -= P_b P_b^T, P_b m_b x k_b (k_b <= 128), all column-major; the first
// n_b columns of C_b.  All items take the K steps of the longest.
static int syrk_ksteps(const std::vector<OzSyrk>& b) {
  int k = 1;
  for (const auto& x : b) k = std::max(k, x.k);
  return (k + OZ_BK - 1) / OZ_BK;
}
size_t ozaki_syrk_batch_bytes(const std::vector<OzSyrk>& b, int digits) {
  int64_t rt = 0;
  for (const auto& x : b) rt += rtiles_of(x.m);
  return (size_t)rt * syrk_ksteps(b) * oz_a_bytes(digits) + (size_t)rt * OZ_BM * sizeof(int32_t) +
         b.size() * (sizeof(OzSplit) + sizeof(OzItem)) + 512;
}

fg_status ozaki_syrk_batch(fg_ctx* ctx, cudaStream_t st, const std::vector<OzSyrk>& b, void* work, size_t bytes,
                           int* d_err, int digits) {
  std::vector<OzSplit> hs;
  std::vector<OzItem> hi;
  int64_t rt = 0, tiles = 0;
  for (const auto& x : b) {
    if (x.m <= 0 || x.k <= 0) continue;
    if (x.k > 128) {
      set_error("ozaki_syrk_batch: k = %d > 128", x.k);
      return FG_ERR_UNSUPPORTED;
    }
    const int64_t tn = (x.n + OZ_BN - 1) / OZ_BN;
    hs.push_back(OzSplit{x.p, 1, x.ld, x.m, x.k, (int)rt});
    hi.push_back(OzItem{x.c, 1, x.ld, x.m, x.n, (int)rt, (int)rt, (int)tn, (int)tiles, -1});
    rt += rtiles_of(x.m);
    tiles += lower_tiles(rtiles_of(x.m), tn);
  }
  if (hs.empty()) return FG_OK;
  if (tiles > (1ll << 31) - 1 || ozaki_syrk_batch_bytes(b, digits) > bytes) {
    set_error("ozaki_syrk_batch: workspace too small or too many tiles");
    return FG_ERR_UNSUPPORTED;
  }
  const int ksteps = syrk_ksteps(b);
  uint8_t* w = (uint8_t*)work;
  const size_t dig_bytes = (size_t)rt * ksteps * oz_a_bytes(digits);
  int32_t* ex = (int32_t*)(w + dig_bytes);
  uint8_t* tail = (uint8_t*)ex + (size_t)rt * OZ_BM * sizeof(int32_t);
  tail = (uint8_t*)(((uintptr_t)tail + 255) & ~(uintptr_t)255);
  OzSplit* ds = (OzSplit*)tail;
  OzItem* di = (OzItem*)(tail + ((hs.size() * sizeof(OzSplit) + 255) / 256) * 256);
  FG_CUDA_TRY(cudaMemcpyAsync(ds, hs.data(), hs.size() * sizeof(OzSplit), cudaMemcpyHostToDevice, st));
  FG_CUDA_TRY(cudaMemcpyAsync(di, hi.data(), hi.size() * sizeof(OzItem), cudaMemcpyHostToDevice, st));
  OzSplitArgs sa;
  sa.items = ds;
  sa.nitems = (int)hs.size();
  sa.none = 0;
  sa.ksteps = ksteps;
  sa.dig = (uint4*)w;
  sa.ex = ex;
  OzGemmArgs g;
  g.dig = w;
  g.ex = ex;
  g.items = di;
  g.nitems = (int)hi.size();
  g.ntiles = (int)tiles;
  g.ksteps = ksteps;
  g.chunk = ksteps;  // k <= 128 <= OZ_KEXACT
  g.alpha = -1.0;
  g.beta = 1.0;
  g.lower = 1;
  g.err = d_err;
  return digits == 8 ? oz_launch<8>(ctx, st, sa, rt, g, tiles) : oz_launch<OZ_S>(ctx, st, sa, rt, g, tiles);
}

}  // namespace fg

using namespace fg;

extern "C" {

fg_status fg_dense_gemm_nt(fg_ctx* ctx, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                           int64_t a_rs, int64_t a_cs, const double* B, int64_t b_rs, int64_t b_cs, double beta,
                           double* C, int64_t c_rs, int64_t c_cs, int32_t flags) {
  if (!ctx || (!A && k > 0) || !C || m < 0 || n < 0 || k < 0 || (flags & ~FG_DENSE_LOWER) ||
      (!B && n != m && k > 0)) {
    set_error("bad argument: ctx/A/C/m/n/k/flags (B = NULL needs n = m)");
    return FG_ERR_BADARG;
  }
  if (m > (1ll << 31) - 1 || n > (1ll << 31) - 1) {
    set_error("bad argument: m, n < 2^31");
    return FG_ERR_BADARG;
  }
  FG_CUDA_TRY(cudaSetDevice(ctx->device));
  const CallScope call(ctx->load);
  if (m == 0 || n == 0) return FG_OK;
  void* work = nullptr;
  FG_TRY(dev_alloc(ctx, &work, ozaki_workspace_bytes(m, n, k, B == nullptr) + 16));
  int* d_err = (int*)((uint8_t*)work + ozaki_workspace_bytes(m, n, k, B == nullptr));
  fg_status s = FG_OK;
  int h_err = 0;
  cudaError_t e = cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream);
  if (e == cudaSuccess) {
    s = ozaki_gemm_nt(ctx, ctx->stream, m, n, k, alpha, A, a_rs, a_cs, B, b_rs, b_cs, beta, C, c_rs, c_cs,
                      (flags & FG_DENSE_LOWER) != 0, work, d_err);
    if (s == FG_OK) e = cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (s == FG_OK && e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  }
  dev_free(ctx, work);
  if (s != FG_OK) return s;
  if (e != cudaSuccess) {
    set_error("fg_dense_gemm_nt: %s", cudaGetErrorString(e));
    return FG_ERR_CUDA;
  }
  if (h_err) {
    set_error("fg_dense_gemm_nt: a bounded tensor-core wait ran out");
    return (fg_status)h_err;
  }
  return FG_OK;
}

}  // extern "C"
