// BSOF as one persistent kernel.
//
// Reference: lapackXbsof, src/bsofi_cpu.c:86-118: for k = 0..L-3, dgeqrf of
// the stacked 2n x n panel [R~_k; B_k] at A_BLK(k,k), dormqr('L','T') of
// A_BLK(k,k+1) and A_BLK(k,L-1); then dgeqrf of the final 2n x 2n block.
//
// Work decomposition.  Every block column is cut into tiles of 16 columns, 8
// above n = 256 (the last one may be narrower).  A "leaf" is the Householder QR of one tile
// inside its panel; leaves are numbered s = 0..S-1 in the reference's order
// (panel k, left to right; the final panel has the tiles of block columns L-2
// and L-1).  Leaf s updates a set of target tiles with its block reflector
// (I - V T V^T)^T: the rest of its panel, the next diagonal block column
// (A_BLK(k,k+1)) and the last block column (A_BLK(k,L-1)).
//
// For a physical tile x the leaves that update it form one contiguous range
// [lo(x), hi(x)) of leaf numbers, and hi(x) is the leaf that factors it.  A
// counter cnt[x] holds how many of those updates are done, so leaf s may
// update x once cnt[x] == s - lo(x), and may factor x once cnt[x] == hi - lo.
//
// CTA 0 runs the critical chain: factor leaf s, then immediately apply it to
// the tile of leaf s+1 (target 0).  The other CTAs claim the remaining
// (leaf, target) updates from an ordered task counter.  Every wait depends
// only on tasks earlier in that order and all CTAs are co-resident
// (cooperative launch), so the schedule cannot deadlock; every spin is
// bounded and sets an error word instead of hanging.
//
// The chain is a serial sequence of N Householder columns, so its time is the
// latency of one column step.  The leaf stays in registers from one leaf to
// the next, laid out as the accumulators of mma.m16n8k8.f64 hold C^T: lane
// 4 g + t of a warp owns two columns (one of an 8-wide leaf) and rows 2t, 2t+1 of each of its 8-row
// blocks.  That layout makes a column step cheap in every part: the pivot
// column reaches the lanes of a row block by one shuffle per row, a column's
// dot products end in a sum over four lanes (a DMMA with ones), and there is
// one barrier per column, after which every warp sums the warps' partials and
// forms the reflector's scalars for itself (a second barrier, with one warp
// forming them for all, measured the same at n = 256 and slower below; two
// columns per barrier, the second one's products corrected for the first
// reflector, measured slower everywhere: one warp's scalar code then takes
// longer than the barrier it saves).  The pivot rows of a leaf belong to
// one warp of their own (the top warp), so the row warps need no row masks; T
// is built one column behind by another.  The same registers are the B operand
// of W^T = C^T V and the accumulators of C^T -= (W T)^T V^T, so the update of
// the next tile reads V from shared memory once and leaves the tile where the
// next factorization wants it.
//
// Measured (chain of one inversion, ms; before: two barriers a column, a
// five-level shuffle sum of 16 values a thread, the tile through L2 and shared
// memory between leaves, 8-wide leaves above n = 256): n = 64, p = 16 1.03 ->
// 0.55; n = 100, p = 64 6.87 -> 4.63; n = 256, p = 32 10.6 -> 7.1; n = 400,
// p = 64 41.2 -> 28, n = 576, p = 12 16.0 -> 9.7 (8-wide).  Per 16-column leaf at n = 256: 9.5 us of column steps
// (about 1160 cycles each, half of them FP64 issue: DFMA takes 3 cycles a warp
// instruction per scheduler), 1.2 us for each half of the next tile's update
// (64 cycles per m16n8k8, two row warps per scheduler).
#include <climits>
#include <type_traits>
#include "bsof_sched.cuh"
#include "bsofi_kernels.h"
#include "tcgen05.cuh"

namespace bsofi {

// FW row warps of NI 8-row blocks each, one top warp, helper warps (which
// stage the next tile in shared memory beside V while the leaf is factored).
// NIW: 8-row blocks per warp of a worker (all FW + 1 warps take rows there).
// CN: columns per lane; leaves and tiles are LW = 8 CN wide.
template <int FW_, int NI_, int NIW_, int CN_ = 2>
struct ChainCfg {
  static constexpr int FW = FW_, NI = NI_, NIW = NIW_, CN = CN_, LW = 8 * CN;
  static constexpr int MW = FW + 1, MT = 32 * MW;
  static constexpr int HW = 4;  // helper warps: one builds T, the others load and store
  static constexpr int THREADS = MT + 32 * HW;
  static constexpr int CT = MT + 32;  // column barrier: with the T warp, the last helper
  // Largest panel height 2n: rows owned by the chain's warps and a worker's.
  static constexpr int ROWS_CHAIN = 8 * (CN + FW * NI), ROWS_WORK = 8 * MW * NIW;
  static constexpr int MAX_ROWS = ROWS_CHAIN < ROWS_WORK ? ROWS_CHAIN : ROWS_WORK;
  // Row slots are taken in groups of GS, skipped when every row is finished.
  static constexpr int GS = 3, NG = (NI + GS - 1) / GS;
  // Tiles move between global and shared memory by bulk copies, which keep the
  // load/store pipe free for the computing warps, or (short panels, where the
  // chain waits for the workers' answer and latency counts) by cp.async and
  // by stores of the warps that hold the reflectors.
  static constexpr bool BULK = NI > 5;
  // Loads a lane and column in flight where unaligned columns are copied by plain loads
  // (16-wide forms: their chain does not wait for them; the 8-wide ones use spans).
  static constexpr int LOADS = ROWS_WORK <= 128 ? 4 : (ROWS_WORK <= 256 ? 8 : 16);
  // EARLY: a leaf is published when V is in shared memory, not when the next tile
  // is, so that the workers' answer may take a chain step longer.  Where the chain
  // waits for them, an inversion at n = 576, p = 12 went from 19.6 to 17.6 ms and at
  // n = 529 from 20.3 to 18.0 (it still waits there, 2 of 11 us a leaf at n = 576); 16-wide
  // leaves do not wait, and the extra barrier costs (n = 256, p = 32 11.65 -> 11.82).
  static constexpr bool EARLY = CN == 1;
  // With 12 warps a thread gets 168 registers at launch; the helper warpgroup
  // gives most of its own to the two that compute
  // (2 x 128 x 224 + 128 x 56 = 384 x 168).
  static constexpr bool REGS = THREADS == 384;
  static_assert(MW == 4 || MW == 8, "partial sums are read as 4 or 8 per column");
};

// Leaf s as the chain CTA sees it.  Rows are counted from the top of the
// panel, except in the second half of the final panel when n is not a
// multiple of the leaf width: there from its row n on, so that a leaf's first
// row is always a multiple of it.
struct ChainStep {
  Leaf f;
  int base, ab, rows, nb;  // first row counted, the leaf's first row, panel rows, 8-row blocks
  int m2, t2, lo2, w2;     // the tile of leaf s+1
  bool next, fresh, trans;
  double *P, *C;           // row 0, column 0 of the leaf's tile and of the next one
  long long ldp, ldc;
};

BSOFI_DEVINL int leaf_base(const BsofGeom& g, const Leaf& f) {
  return (f.k == g.L - 2 && f.l >= g.nl && g.n % g.NB != 0) ? g.n : 0;
}

BSOFI_DEVINL ChainStep chain_step(const BsofGeom& g, const BsofState& st, int s) {
  ChainStep c;
  c.f = leaf_of(g, s);
  c.base = leaf_base(g, c.f);
  c.ab = c.f.j0 - c.base;
  c.rows = 2 * g.n - c.base;
  c.nb = (c.rows + 7) / 8;
  c.next = ntargets(g, c.f) > 0;
  c.m2 = c.t2 = c.lo2 = 0;
  c.C = nullptr;
  c.ldc = 2;
  if (c.next) {
    int hi2;
    target_of(g, c.f, 0, c.m2, c.t2);
    tile_range(g, c.m2, c.t2, c.lo2, hi2);
    c.C = tile_ptr(g, st, c.f.k, c.base, c.m2, c.t2, c.ldc);
  }
  c.P = mat_ptr(g, st, (long long)c.f.k * g.n + c.base, c.f.m, c.f.t * g.NB, c.ldp);
  c.w2 = min(g.NB, g.n - c.t2 * g.NB);
  // Panel change (rows shift by n, n fresh rows come in), and the shift by n
  // inside the final panel when n is not a multiple of the leaf width.
  c.fresh = c.next && c.f.l == g.nl - 1 && c.f.k <= g.L - 3;
  c.trans = c.fresh || (c.next && c.f.l == g.nl - 1 && g.n % g.NB != 0);
  return c;
}

template <int MW>
struct ChainSmem {
  // Two buffers, of even and odd columns; columns in the lane groups' order
  // (g, then 8 + g).
  double red[2][16 * MW];  // per column: one partial dot product per warp
  double prow[2][16];      // pivot row
  double sc[16];           // 1/(alpha - beta) of the finished columns
  double vtv[2][17];       // v_j^T v_I of the finished columns j < I, and tau_I
  alignas(16) double top[16 * 16];     // pivot rows of the next leaf on their way to the top warp
  // T, and (once every warp has used it) W^T T in the same place.
  union {
    double T[16][17];
    alignas(16) double W[256];
  };
  ChainStep step[2];       // of leaves s, s+1
  uint64_t bar;            // bulk loads
  int ok[2];               // the next tile of an even / odd leaf arrived
  int flag;
  int task;
};

// Tiles in shared memory are plain column-major, so that one bulk copy moves
// a column.  The column stride is 2 mod 16 doubles and the lane group g owns
// columns col_of(g) and col_of(g) + 8 (not g and g + 8): then both fragment
// patterns, 16-byte row pairs of two groups' columns and single rows of every
// second column, touch every bank once.
BSOFI_DEVINL int col_of(int g) { return (g >> 1) + 4 * (g & 1); }
BSOFI_DEVINL int group_of(int c) { return 2 * (c & 3) + ((c >> 2) & 1); }  // c = 0..7
BSOFI_DEVINL int sidx(int r, int c, int S) { return c * S + r; }
// Column stride of a panel's tile (2n rows, rounded up to 16).
__host__ __device__ __forceinline__ int tile_stride(int n) { return ((2 * n + 15) & ~15) + 2; }

// Bulk copies of one column between global and shared memory (16-byte
// aligned, a multiple of 16 bytes), off the load/store pipe that the
// computing warps need.
BSOFI_DEVINL void bulk_load(double* dst, const double* src, int rows, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          tc::smem_u32(dst)),
      "l"(src), "r"(rows * 8), "r"(tc::smem_u32(bar))
      : "memory");
}
BSOFI_DEVINL void bulk_store(double* dst, const double* src, int rows) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(tc::smem_u32(src)), "r"(rows * 8)
               : "memory");
}
BSOFI_DEVINL void bulk_store_wait() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Between this thread's generic accesses (and those it has synchronised with)
// and asynchronous copies of the same memory.
BSOFI_DEVINL void fence_proxy() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Bounded wait for the bulk loads of one phase; reports through the error word.
BSOFI_DEVINL bool bulk_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (int i = 0; i < (1 << 22); i++)
    if (tc::mbar_try_wait(bar, parity)) return true;
  atomicExch(err, 1);
  return false;
}

template <int COUNT>
BSOFI_DEVINL void bar_main() {
  asm volatile("bar.sync 1, %0;" ::"n"(COUNT) : "memory");
}
// Column step barrier: the factoring warps and the T warp.
template <int COUNT>
BSOFI_DEVINL void bar_col() {
  asm volatile("bar.sync 4, %0;" ::"n"(COUNT) : "memory");
}
// Per leaf: V, T and the next tile are in shared memory (the T warp only
// arrives); the leaf is done.
template <int COUNT>
BSOFI_DEVINL void bar_ready() {
  asm volatile("bar.sync 3, %0;" ::"n"(COUNT) : "memory");
}
template <int COUNT>
BSOFI_DEVINL void bar_ready_arrive() {
  asm volatile("bar.arrive 3, %0;" ::"n"(COUNT) : "memory");
}
template <int COUNT>
BSOFI_DEVINL void bar_done() {
  asm volatile("bar.sync 6, %0;" ::"n"(COUNT) : "memory");
}
// V is in shared memory: the factoring warps arrive, the T warp waits.
template <int COUNT>
BSOFI_DEVINL void bar_v() {
  asm volatile("bar.sync 5, %0;" ::"n"(COUNT) : "memory");
}
template <int COUNT>
BSOFI_DEVINL void bar_v_arrive() {
  asm volatile("bar.arrive 5, %0;" ::"n"(COUNT) : "memory");
}
template <int COUNT>
BSOFI_DEVINL void bar_help() {
  asm volatile("bar.sync 2, %0;" ::"n"(COUNT) : "memory");
}

BSOFI_DEVINL double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
BSOFI_DEVINL double shfl_x(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// One thread's bounded wait until *p >= target; false when it gave up.
BSOFI_DEVINL bool wait_geq(const BsofState& st, const int* p, int target) {
  long long it = 0;
  while (ld_acquire(p) < target) {
    if (ld_acquire(st.err) != 0) return false;
    if (++it > st.spin_limit) {
      atomicExch(st.err, 1);
      return false;
    }
    __nanosleep(32);
  }
  return true;
}

// Rows r, r+1 of one column in global memory (through L2: the tile may have
// been written by another SM).  vec: the pair is 16-byte aligned.
BSOFI_DEVINL double2 ld_pair(const double* col, int r, int rows, bool ok, bool vec) {
  double2 v = make_double2(0.0, 0.0);
  if (ok) {
    if (vec && r + 1 < rows) {
      v = __ldcg(reinterpret_cast<const double2*>(col + r));
    } else {
      if (r < rows) v.x = __ldcg(col + r);
      if (r + 1 < rows) v.y = __ldcg(col + r + 1);
    }
  }
  return v;
}
BSOFI_DEVINL void st_pair(double* col, int r, int rows, bool ok, bool vec, double x, double y) {
  if (!ok) return;
  if (vec && r + 1 < rows) {
    __stcg(reinterpret_cast<double2*>(col + r), make_double2(x, y));
  } else {
    if (r < rows) __stcg(col + r, x);
    if (r + 1 < rows) __stcg(col + r + 1, y);
  }
}
// Rows [r0, r1) of NC columns (c, c + step, .., those below c1) of a tile that
// breaks 16-byte alignment, from src (leading dimension ld) to dst (column
// stride S) by one warp, U loads a lane and column in flight (through L2:
// cp.async of 8 bytes would leave lines in this SM's L1 that other SMs still
// write).
template <int NC, int U>
BSOFI_DEVINL void copy_cols(double* dst, int S, const double* src, long long ld, int c, int step,
                            int c1, int r0, int r1, int lane) {
  for (int r = r0 + lane; r < r1; r += 32 * U) {
    double v[NC][U];
#pragma unroll
    for (int j = 0; j < NC; j++) {
      const double* p = src + cm(r, c + j * step, ld);
#pragma unroll
      for (int u = 0; u < U; u++)
        v[j][u] = c + j * step < c1 && r + 32 * u < r1 ? __ldcg(p + 32 * u) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < NC; j++) {
      double* q = dst + (c + j * step) * S + r;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (c + j * step < c1 && r + 32 * u < r1) q[32 * u] = v[j][u];
    }
  }
}
BSOFI_DEVINL bool pair_aligned(const double* p, long long ld) {
  return ((reinterpret_cast<uintptr_t>(p) & 15) == 0) && ((ld & 1) == 0);
}

// cnt elements of one column from src (8-byte aligned) to dst (16-byte aligned)
// with bulk copies, which need 16 bytes on both sides: from an odd address the
// copy starts at the second element and lands one element late (never beyond
// dst[cnt - 1]); once it has arrived a warp moves it down and fetches the edges.
BSOFI_DEVINL int span_late(const double* src) {
  return (int)(reinterpret_cast<uintptr_t>(src) >> 3) & 1;
}
BSOFI_DEVINL int span_bulk(const double* src, int cnt) {
  return max(0, cnt - 2 * span_late(src)) & ~1;
}
BSOFI_DEVINL void span_issue(double* dst, const double* src, int cnt, uint64_t* bar) {
  const int late = span_late(src), m = span_bulk(src, cnt);
  if (m > 0) bulk_load(dst + 2 * late, src + late, m, bar);
}
BSOFI_DEVINL void span_finish(double* dst, const double* src, int cnt, int lane) {
  const int late = span_late(src), m = span_bulk(src, cnt);
  const int edge = late && lane == 0 ? 0 : m + lane;  // the first element, and those past the copy
  const bool mine = lane < 3 && edge < cnt;
  const double v = mine ? __ldcg(src + edge) : 0.0;
  if (late) {
    constexpr int U = 8;
#pragma unroll 1
    for (int r = 1 + lane; r - lane <= m; r += 32 * U) {
      double x[U];
#pragma unroll
      for (int u = 0; u < U; u++) x[u] = r + 32 * u <= m ? dst[r + 32 * u + 1] : 0.0;
      __syncwarp();
#pragma unroll
      for (int u = 0; u < U; u++)
        if (r + 32 * u <= m) dst[r + 32 * u] = x[u];
      __syncwarp();
    }
  }
  if (mine) dst[edge] = v;
}

// One thread's start of all w columns (vec: none of them needs span_finish).
BSOFI_DEVINL void issue_columns(double* dst, int S, const double* src, long long ld, int w, int cnt,
                                bool vec, uint64_t* bar) {
  int total = w * cnt;
  if (!vec) {
    total = 0;
    for (int c = 0; c < w; c++) total += span_bulk(src + cm(0, c, ld), cnt);
  }
  fence_proxy();
  tc::mbar_arrive_expect_tx(bar, 8 * total);
  for (int c = 0; c < w; c++) {
    if (vec) bulk_load(dst + c * S, src + cm(0, c, ld), cnt, bar);
    else span_issue(dst + c * S, src + cm(0, c, ld), cnt, bar);
  }
}

// ------------------------------------------------------------ column steps
struct Refl {
  double tau, scale, beta, q;  // q = tau * scale = -1 / beta
};
// LAPACK dlarfg: beta = -sign(alpha) ||(alpha, x)||, tau = (beta - alpha)/beta
// = 1 + |alpha|/||.||, scale = 1/(alpha - beta).  The square root, its
// reciprocal and 1/(|alpha| + ||.||) are the longest dependent chain of a
// column step, so they share one: Goldschmidt's coupled iteration (Markstein,
// "Software division and square root using Goldschmidt's algorithms", 2004)
// from the hardware's approximation gives the norm and half its reciprocal
// together, and a Newton step on the residual finishes each.  The last reciprocal
// starts from the first norm estimate meanwhile and takes one step of
// Chebyshev's third-order iteration (Traub, "Iterative Methods for the Solution
// of Equations", 1964): with d = 1 - x z the reciprocal is z / (1 - d), of
// whose series z (1 + d + d^2) keeps the terms that count at d of 2^-20.
// Error bounds, counting a rounding as at most 2^-53: beta 1.5 units of it (half
// of the sum's, one of the last step), q 2.5, tau 2.25, scale 3.5 and d^3.  The
// self-test below samples them against long double.  Outside the range
// where the approximations are normal numbers rsqrt() and a division are used.
BSOFI_DEVINL Refl reflector(double xnorm2, double alpha) {
  Refl r;
  const double s2 = fma(alpha, alpha, xnorm2), aa = fabs(alpha);
  // Every lane holds the same values: one vote keeps the branch uniform.
  const unsigned hi = __double2hiint(s2);  // [2^-930, 2^930) or not
  const bool rare = xnorm2 == 0.0 || hi - 0x05d00000u >= 0x74400000u;
  const unsigned any = __any_sync(0xffffffffu, rare);
  double y, z;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s2));
  double nrm = s2 * y, h = 0.5 * y;
  const double est = aa + nrm;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(est));
  const double e = fma(-nrm, h, 0.5);
  nrm = fma(nrm, e, nrm);
  h = fma(h, e, h);
  nrm = fma(fma(-nrm, nrm, s2), h, nrm);
  double rn = h + h;
  rn = fma(rn, fma(-nrm, rn, 1.0), rn);
  const double d = fma(-(aa + nrm), z, 1.0);
  z = fma(z, fma(d, d, d), z);
  r.beta = -copysign(nrm, alpha);
  r.tau = fma(aa, rn, 1.0);
  r.scale = copysign(z, alpha);
  r.q = copysign(rn, alpha);
  if (any) {
    if (xnorm2 == 0.0) {
      r.tau = 0.0;
      r.beta = alpha;
      r.scale = 1.0;
      r.q = 0.0;
    } else {
      const double rs = rsqrt(s2);
      r.beta = -copysign(s2 * rs, alpha);
      r.tau = fma(aa, rs, 1.0);
      r.scale = 1.0 / (alpha - r.beta);
      r.q = copysign(rs, alpha);
    }
  }
  return r;
}

// Self-test: a warp per pair, whose lanes hold the same values as in a column
// step; beta, tau, scale, q, and the first three by rsqrt() and a division.
__global__ void __launch_bounds__(256) reflector_kernel(int count, const double* xnorm2,
                                                        const double* alpha, double* out) {
  const int i = (int)((blockIdx.x * 256ll + threadIdx.x) >> 5);
  if (i >= count) return;
  const double x2 = xnorm2[i], a = alpha[i];
  const Refl r = reflector(x2, a);
  if ((threadIdx.x & 31) != 0) return;
  const double rs = rsqrt(fma(a, a, x2)), beta = -copysign(fma(a, a, x2) * rs, a);
  double* o = out + 7ll * i;
  o[0] = r.beta;
  o[1] = r.tau;
  o[2] = r.scale;
  o[3] = r.q;
  o[4] = beta;
  o[5] = fma(fabs(a), rs, 1.0);
  o[6] = 1.0 / (a - beta);
}

// Sum over the four lanes t of a column's group (lane 4 g + t), to all four:
// one DMMA with a matrix of ones (27 cycles against about 70 for two shuffle
// and add levels).
BSOFI_DEVINL double quad_sum(double v) {
  double d[2] = {0.0, 0.0};
  dmma_8x8x4(d, v, 1.0);
  return d[0];
}

// Sum over the warps' partials of a column (c in the lane groups' order).
template <int MW>
BSOFI_DEVINL double col_total(const double* red, int c, int t) {
  if constexpr (MW == 8) {
    const double2 a = *reinterpret_cast<const double2*>(red + c * 8 + 2 * t);
    return quad_sum(a.x + a.y);
  } else {
    return quad_sum(red[c * 4 + t]);
  }
}

// Warp sums of the lane's columns' partial dot products into red[column][warp]:
// again DMMAs with ones, whose results lane 4 g + t holds for columns 2t, 2t+1.
template <class K>
BSOFI_DEVINL void put_partials(double* red, const double (&d)[K::CN], int g, int t, int warp) {
  double e[K::CN][2];
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) {
    e[cs][0] = e[cs][1] = 0.0;
    dmma_8x8x4(e[cs], 1.0, d[cs]);
  }
  if (g < K::CN) {
    double* dst = red + (8 * g + 2 * t) * K::MW + warp;
    dst[0] = g == 0 ? e[0][0] : e[K::CN - 1][0];
    dst[K::MW] = g == 0 ? e[0][1] : e[K::CN - 1][1];
  }
}

// One pass of a row warp over its rows: the update by the finished pivot
// column (f: factors of the lane's columns, zero where a column is finished;
// column sets below CSU are all finished) and the dot products with the next
// pivot column (set CSD, lane srcd).  ab8: first 8-row block of the leaf; nb:
// row blocks of the panel.
template <class K, int CSU, int CSD>
BSOFI_DEVINL void row_pass(double (&a)[K::NI][K::CN][2], double (&x)[K::NI][2],
                           const double (&f)[K::CN], int srcd, int ab8, int nb, int warp,
                           double (&d)[K::CN]) {
  double s[K::CN][2] = {};
#pragma unroll
  for (int q = 0; q < K::NG; q++) {
    constexpr int GS = K::GS;
    const int ia = q * GS, ie = (ia + GS < K::NI ? ia + GS : K::NI);
    if ((ie - 1) * K::FW + warp < ab8 || K::CN + ia * K::FW + warp >= nb) continue;
#pragma unroll
    for (int i = ia; i < ie; i++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const double xo = x[i][h];
#pragma unroll
        for (int cs = CSU; cs < K::CN; cs++) a[i][cs][h] = fma(-xo, f[cs], a[i][cs][h]);
        const double xn = shfl_d(a[i][CSD][h], srcd);
        x[i][h] = xn;
#pragma unroll
        for (int cs = 0; cs < K::CN; cs++) s[cs][h] = fma(xn, a[i][cs][h], s[cs][h]);
      }
    }
  }
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) d[cs] = s[cs][0] + s[cs][1];
}

// The dot products with column 0, before the first column step.
template <class K>
BSOFI_DEVINL void row_first(double (&a)[K::NI][K::CN][2], double (&x)[K::NI][2], int t,
                            double (&d)[K::CN]) {
  double s[K::CN][2] = {};
#pragma unroll
  for (int i = 0; i < K::NI; i++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double xn = shfl_d(a[i][0][h], t);
      x[i][h] = xn;
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++) s[cs][h] = fma(xn, a[i][cs][h], s[cs][h]);
    }
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) d[cs] = s[cs][0] + s[cs][1];
}

// Sums, reflector and v_I^T a_c of this lane's columns at column step I.
template <class K>
struct ColStep {
  Refl rf;
  double w[K::CN];
};
template <class K>
BSOFI_DEVINL ColStep<K> col_step(const ChainSmem<K::MW>& sm, int I, int g, int t) {
  const int buf = I & 1, ri = group_of(I & 7) + (I & 8);
  ColStep<K> c;
  double pr[K::CN], s[K::CN];
  const double alpha = sm.prow[buf][ri];
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) pr[cs] = sm.prow[buf][g + 8 * cs];
  const double sp = col_total<K::MW>(sm.red[buf], ri, t);
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) s[cs] = col_total<K::MW>(sm.red[buf], g + 8 * cs, t);
  c.rf = reflector(sp, alpha);
  // v_I^T a_c = a_Ic + scale d_c.
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) c.w[cs] = fma(c.rf.scale, s[cs], pr[cs]);
  return c;
}

// The column loop of a row warp.
template <class K>
BSOFI_DEVINL void factor_rows(double (&a)[K::NI][K::CN][2], ChainSmem<K::MW>& sm, int w, int ab8,
                              int nb, int g, int t, int warp) {
  const int c0 = col_of(g);
  double x[K::NI][2], d[K::CN];
  row_first<K>(a, x, t, d);
  put_partials<K>(sm.red[0], d, g, t, warp);
  int I = 0;
  auto step = [&](auto csu, auto csd) {
    bar_col<K::CT>();
    const ColStep<K> c = col_step<K>(sm, I, g, t);
    double f[K::CN];
#pragma unroll
    for (int cs = 0; cs < K::CN; cs++) f[cs] = c0 + 8 * cs > I ? c.rf.q * c.w[cs] : 0.0;
    const int sd = group_of((I + 1) & 7) * 4 + t;
    row_pass<K, csu.value, csd.value>(a, x, f, sd, ab8, nb, warp, d);
    put_partials<K>(sm.red[(I + 1) & 1], d, g, t, warp);
  };
  using Z = std::integral_constant<int, 0>;
  using O = std::integral_constant<int, 1>;
  const int last = w - 1;
#pragma unroll 1
  for (; I < min(last, 7); I++) step(Z{}, Z{});
  if constexpr (K::CN == 2) {
    if (I < last) {  // I = 7
      step(O{}, O{});
      I++;
#pragma unroll 1
      for (; I < last; I++) step(O{}, O{});
    }
  }
  bar_col<K::CT>();  // the last column's sums are there
  bar_col<K::CT>();  // and its scale
}

// The top warp's LW pivot rows (blocks 0.. in a[0]..): update by pivot column I
// (set CSU; rows below I; row I by v_I = 1, its pivot entry becomes beta).
template <class K, int CSU>
BSOFI_DEVINL void top_update(double (&a)[K::NI][K::CN][2], const double (&x)[K::CN][2],
                             const Refl& rf, const double (&F)[K::CN], int I, int g, int t) {
#pragma unroll
  for (int b = CSU; b < K::CN; b++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int row = 8 * b + 2 * t + h;
      const double v = row == I ? 1.0 : x[b][h] * rf.scale;
#pragma unroll
      for (int cs = CSU; cs < K::CN; cs++) a[b][cs][h] = fma(-v, F[cs], a[b][cs][h]);
      if (b == CSU && row == I && g == group_of(I & 7)) a[b][CSU][h] = rf.beta;
    }
}

// Dot products with column J (set CSD) over rows below J, and row J to prow.
template <class K, int CSD>
BSOFI_DEVINL void top_dots(const double (&a)[K::NI][K::CN][2], double (&x)[K::CN][2], int J, int g,
                           int t, double* prow, double (&d)[K::CN]) {
  const int src = group_of(J & 7) * 4 + t;
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) d[cs] = 0.0;
#pragma unroll
  for (int b = CSD; b < K::CN; b++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int row = 8 * b + 2 * t + h;
      const double xs = shfl_d(a[b][CSD][h], src);
      x[b][h] = row > J ? xs : 0.0;
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++) d[cs] = fma(x[b][h], a[b][cs][h], d[cs]);
      if (b == CSD && row == J) {
#pragma unroll
        for (int cs = 0; cs < K::CN; cs++) prow[g + 8 * cs] = a[b][cs][h];
      }
    }
}

// The column loop of the top warp.
template <class K>
BSOFI_DEVINL void factor_top(double (&a)[K::NI][K::CN][2], ChainSmem<K::MW>& sm, int w, int g,
                             int t, double* tau) {
  const int c0 = col_of(g);
  double x[K::CN][2], d[K::CN], sc[K::CN];
#pragma unroll
  for (int cs = 0; cs < K::CN; cs++) sc[cs] = 0.0;
  top_dots<K, 0>(a, x, 0, g, t, sm.prow[0], d);
  put_partials<K>(sm.red[0], d, g, t, K::FW);
  int I = 0;
  auto step = [&](auto csu, auto csd, auto dot) {
    bar_col<K::CT>();
    const ColStep<K> c = col_step<K>(sm, I, g, t);
    double F[K::CN];
#pragma unroll
    for (int cs = 0; cs < K::CN; cs++) F[cs] = c0 + 8 * cs > I ? c.rf.tau * c.w[cs] : 0.0;
    top_update<K, csu.value>(a, x, c.rf, F, I, g, t);
    if (dot.value) {
      top_dots<K, csd.value>(a, x, I + 1, g, t, sm.prow[(I + 1) & 1], d);
      put_partials<K>(sm.red[(I + 1) & 1], d, g, t, K::FW);
    }
    // v_j^T v_I of the finished columns j < I (both unscaled in registers,
    // row I of v_I is 1) for the T warp.
    if (t == 0) {
      double* v = sm.vtv[I & 1];
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++)
        v[c0 + 8 * cs] = c0 + 8 * cs < I ? sc[cs] * c.w[cs] : 0.0;
      if (g == 0) {
        v[16] = c.rf.tau;
        tau[I] = c.rf.tau;
        sm.sc[I] = c.rf.scale;
      }
    }
#pragma unroll
    for (int cs = 0; cs < K::CN; cs++)
      if (I == c0 + 8 * cs) sc[cs] = c.rf.scale;
  };
  using Z = std::integral_constant<int, 0>;
  using O = std::integral_constant<int, 1>;
  const int last = w - 1;
#pragma unroll 1
  for (; I < min(last, 7); I++) step(Z{}, Z{}, O{});
  if constexpr (K::CN == 2) {
    if (I < last) {  // I = 7
      step(Z{}, O{}, O{});
      I++;
#pragma unroll 1
      for (; I < last; I++) step(O{}, O{}, O{});
    }
    if (I < 8) step(Z{}, Z{}, Z{});
    else step(O{}, O{}, Z{});
  } else {
    step(Z{}, Z{}, Z{});
  }
  bar_col<K::CT>();
}

// The T warp: column I of T one barrier behind the factorization (LAPACK
// dlarft): T(0:I,I) = -tau_I T(0:I,0:I) V(:,0:I)^T v_I.  Lane 4 g + t holds
// rows g (and g+8) of columns t, t+4, ..
template <int CN>
BSOFI_DEVINL void t_column(double (&T)[CN][2 * CN], const double* vtv, int I, int g, int t) {
  double r[CN];
#pragma unroll
  for (int cs = 0; cs < CN; cs++) {
    r[cs] = 0.0;
#pragma unroll
    for (int q = 0; q < 2 * CN; q++) r[cs] = fma(T[cs][q], vtv[t + 4 * q], r[cs]);
  }
  const double tau = vtv[16];
#pragma unroll
  for (int cs = 0; cs < CN; cs++) {
    const double s = quad_sum(r[cs]);
    const double v = g + 8 * cs == I ? tau : (g + 8 * cs < I ? -tau * s : 0.0);
#pragma unroll
    for (int q = 0; q < 2 * CN; q++)
      if (I == t + 4 * q) T[cs][q] = v;
  }
}

// ------------------------------------------------------------ block update
// Element (c, j) of a 16 x 16 matrix kept row by row with the halves exchanged
// in rows c = 4..7, 12..15: row pairs (c, c+4) of a quarter-warp access meet
// different banks.
BSOFI_DEVINL int widx(int c, int j) { return c * 16 + (j ^ ((c & 4) << 1)); }

// From this warp's W^T = C^T V over its own rows to the A fragments of
// -(W^T T) summed over all MW warps.  acc[jt] holds rows c = col_of(g),
// col_of(g) + 8 and (its B operand having V's columns in the lane groups'
// order) columns 8 jt + t, 8 jt + t + 4.  The fragments' K index t stands for
// j = 8 kk + 2t and t + 4 for 8 kk + 2t + 1.  Two barriers among the MW warps.
//
// With 8-wide leaves the same with one tile, m8n8k4 and its K index t for j = t
// and t + 4, or 2t and 2t + 1 in the fragments.
template <int CN>
BSOFI_DEVINL void mma_w(double (&acc)[2 * CN], const double (&c)[CN][2], double v0, double v1) {
  if constexpr (CN == 2) {
    dmma_16x8x8(acc, c[0][0], c[1][0], c[0][1], c[1][1], v0, v1);
  } else {
    dmma_8x8x4(acc, c[0][0], v0);
    dmma_8x8x4(acc, c[0][1], v1);
  }
}

template <int MW, int CN>
BSOFI_DEVINL void reduce_w(double (&acc)[CN][2 * CN], double (&fr)[CN][2 * CN], double* part,
                           ChainSmem<MW>& sm, int g, int t, int warp) {
  constexpr int E = 64 * CN * CN;  // elements of W
  double* mine = part + warp * E;
  const int c0 = col_of(g);
  if constexpr (CN == 2) {
    // (W^T T): T is upper triangular, so columns 0..7 need only rows 0..7.
    double o[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
    dmma_16x8x8(o[0], acc[0][0], acc[0][2], acc[0][1], acc[0][3], sm.T[t][g], sm.T[t + 4][g]);
    dmma_16x8x8(o[1], acc[0][0], acc[0][2], acc[0][1], acc[0][3], sm.T[t][g + 8],
                sm.T[t + 4][g + 8]);
    dmma_16x8x8(o[1], acc[1][0], acc[1][2], acc[1][1], acc[1][3], sm.T[8 + t][g + 8],
                sm.T[12 + t][g + 8]);
#pragma unroll
    for (int jt = 0; jt < 2; jt++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        *reinterpret_cast<double2*>(mine + widx(c0 + 8 * h, 8 * jt + 2 * t)) =
            make_double2(o[jt][2 * h], o[jt][2 * h + 1]);
  } else {
    double o[2] = {0.0, 0.0};
    dmma_8x8x4(o, acc[0][0], sm.T[t][g]);
    dmma_8x8x4(o, acc[0][1], sm.T[t + 4][g]);
    *reinterpret_cast<double2*>(mine + c0 * 8 + 2 * t) = make_double2(o[0], o[1]);
  }
  bar_main<32 * MW>();
#pragma unroll
  for (int e = threadIdx.x; e < E; e += 32 * MW) {
    double s[MW];
#pragma unroll
    for (int k = 0; k < MW; k++) s[k] = part[k * E + e];
#pragma unroll
    for (int m = MW / 2; m > 0; m /= 2)
#pragma unroll
      for (int k = 0; k < m; k++) s[k] += s[k + m];
    sm.W[e] = -s[0];
  }
  bar_main<32 * MW>();
  if constexpr (CN == 2) {
#pragma unroll
    for (int kk = 0; kk < 2; kk++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const double2 v =
            *reinterpret_cast<const double2*>(sm.W + widx(c0 + 8 * h, 8 * kk + 2 * t));
        fr[kk][h] = v.x;
        fr[kk][2 + h] = v.y;
      }
  } else {
    const double2 v = *reinterpret_cast<const double2*>(sm.W + c0 * 8 + 2 * t);
    fr[0][0] = v.x;
    fr[0][1] = v.y;
  }
}

// C^T += fr V^T for the 8-row block at row r0 of V in shared memory.
template <int CN>
BSOFI_DEVINL void update_block(double (&c)[CN][2], const double (&fr)[CN][2 * CN],
                               const double* sV, int SV, int r0, int g, int t) {
  if constexpr (CN == 2) {
    double d[4] = {c[0][0], c[0][1], c[1][0], c[1][1]};
#pragma unroll
    for (int kk = 0; kk < 2; kk++)
      dmma_16x8x8(d, fr[kk][0], fr[kk][1], fr[kk][2], fr[kk][3],
                  sV[sidx(r0 + g, 8 * kk + 2 * t, SV)], sV[sidx(r0 + g, 8 * kk + 2 * t + 1, SV)]);
    c[0][0] = d[0];
    c[0][1] = d[1];
    c[1][0] = d[2];
    c[1][1] = d[3];
  } else {
    dmma_8x8x4(c[0], fr[0][0], sV[sidx(r0 + g, 2 * t, SV)]);
    dmma_8x8x4(c[0], fr[0][1], sV[sidx(r0 + g, 2 * t + 1, SV)]);
  }
}

// ------------------------------------------------------------ the chain CTA
// The reflectors below the pivot rows to global memory, by W warps of which this
// is warp w (the pivot rows and, in short panels, all of V are stored by the
// warps that hold them).
template <class K, int W>
BSOFI_DEVINL void store_leaf(const ChainStep& z, const double* sV, int SV, int lane, int w) {
  if constexpr (K::BULK) {
    const int r0 = z.ab + K::LW, cnt = max(0, z.rows - r0), even = cnt & ~1;
    if (pair_aligned(z.P, z.ldp) && even == cnt) {
      if (w == 0 && lane == 0 && cnt > 0) {
        for (int c = 0; c < z.f.w; c++)
          bulk_store(z.P + cm(r0, c, z.ldp), sV + sidx(r0, c, SV), cnt);
        bulk_store_wait();
        fence_proxy();
      }
      return;
    }
    // EARLY: aligned columns (every second one with an odd leading dimension) still by
    // bulk copies, as one warp stores them: n = 451, p = 9 10.27 -> 9.94 ms.
    auto bulk = [&](int c) { return K::EARLY && span_late(z.P + cm(r0, c, z.ldp)) == 0; };
    if (w == 0 && lane == 0 && even > 0)
      for (int c = 0; c < z.f.w; c++)
        if (bulk(c)) bulk_store(z.P + cm(r0, c, z.ldp), sV + sidx(r0, c, SV), even);
#pragma unroll 1
    for (int c = w; c < z.f.w; c += W) {
      double* col = z.P + cm(r0, c, z.ldp);
      const double* v = sV + sidx(r0, c, SV);
      if (bulk(c)) {
        if (lane == 0 && even < cnt) __stcg(col + even, v[even]);
        continue;
      }
#pragma unroll 4
      for (int r = lane; r < cnt; r += 32) __stcg(col + r, v[r]);
    }
    if (K::EARLY && lane == 0) {
      bulk_store_wait();
      fence_proxy();
    }
  }
}

// The helper warps: wait for the next tile and stage it while the leaf is being
// factored; the last one (the T warp) builds T.  One side or the other stores
// and publishes the leaf.
template <class K>
BSOFI_DEVINL void chain_helper(const BsofGeom& g, const BsofState& st, const double* sV, double* sC,
                               int SV, ChainSmem<K::MW>& sm) {
  const int ht = threadIdx.x - K::MT, lane = threadIdx.x & 31, hw = ht >> 5;
  const int n = g.n, SC = SV + 16, capc = SC - 2;
  uint32_t phase = 0;
  constexpr int LD = K::HW - 1;  // loading warps; the last one builds T
  if (hw == LD) {
    const int gq = lane >> 2, t = lane & 3;
    for (int s = st.s_begin; s < st.s_end; s++) {
      const Leaf f = sm.step[s & 1].f;
      double T[K::CN][2 * K::CN] = {};
      for (int I = 0; I <= f.w; I++) {
        bar_col<K::CT>();
        if (I > 0) t_column<K::CN>(T, sm.vtv[(I - 1) & 1], I - 1, gq, t);
      }
      // (Stamps by this warp where they can be: the chain does not wait for it.  The
      // third one by a warp that stores the leaf took n = 255, p = 12 from 4.69 to 4.82 ms.)
      const unsigned long long factored = gtimer();
      double* Tout = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
#pragma unroll
      for (int r = 0; r < K::CN; r++)
#pragma unroll
        for (int q = 0; q < 2 * K::CN; q++) {
          const int i = gq + 8 * r, j = t + 4 * q;
          sm.T[i][j] = T[r][q];
          Tout[i + 16 * j] = T[r][q];
        }
      if (lane == 0) st.timeline[4 * s + 1] = factored;
      if constexpr (K::EARLY) {
        bar_ready_arrive<K::THREADS>();
        bar_v<K::CT>();
        store_leaf<K, 1>(sm.step[s & 1], sV, SV, lane, 0);
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          red_release_add(st.factored + s, 1);
        }
      } else {
        bar_ready<K::THREADS>();
        // (Behind a value read after the barrier, or the compiler takes the timer before it;
        // not by the lane that works out the next step: n = 16, p = 40 0.468 -> 0.466 ms.)
        if (lane == 16 && sm.ok[s & 1]) st.timeline[4 * s + 3] = gtimer();
      }
      if (lane == 0 && s + 1 < st.s_end) sm.step[(s + 1) & 1] = chain_step(g, st, s + 1);
      bar_done<K::THREADS>();
      if (!sm.ok[s & 1]) return;
    }
    return;
  }
  for (int s = st.s_begin; s < st.s_end; s++) {
    const ChainStep& z = sm.step[s & 1];
    int& ok = sm.ok[s & 1];
    if (ht == 0) ok = !z.next || wait_geq(st, st.cnt + tile_id(g, z.m2, z.t2), s - z.lo2) ? 1 : 0;
    {
      bar_help<32 * LD>();
      if (z.next && ok) {
        // Rows [ab, rows) of the tile, then (fresh) the n rows below the panel
        // at shared rows 8 nb, 8 nb + 1, .. (mod capc; the tile's own rows
        // above ab leave room).
        const int f0 = 8 * z.nb, q0 = min(n, capc - f0);
        const double* F = z.C + 2 * n;
        const bool vec = pair_aligned(z.C, z.ldc) &&
                         (K::EARLY ? ((z.rows | (z.fresh ? n : 0)) & 1) == 0 : (n & 1) == 0);
        if (K::BULK && (vec || K::EARLY)) {
          // The spans of column c: f(dst, src, elements).
          auto spans = [&](int c, auto f) {
            const long long at = cm(0, c, z.ldc);
            f(sC + sidx(z.ab, c, SC), z.C + at + z.ab, z.rows - z.ab);
            if (z.fresh) {
              f(sC + sidx(f0, c, SC), F + at, q0);
              if (n > q0) f(sC + sidx(0, c, SC), F + at + q0, n - q0);
            }
          };
          if (ht == 0) {
            int total = z.w2 * (z.rows - z.ab + (z.fresh ? n : 0));
            if (K::EARLY && !vec) {
              total = 0;
              for (int c = 0; c < z.w2; c++)
                spans(c, [&](double*, const double* src, int cnt) { total += span_bulk(src, cnt); });
            }
            fence_proxy();
            tc::mbar_arrive_expect_tx(&sm.bar, 8 * total);
            for (int c = 0; c < z.w2; c++)
              spans(c, [&](double* dst, const double* src, int cnt) {
                if (!K::EARLY || vec) bulk_load(dst, src, cnt, &sm.bar);
                else span_issue(dst, src, cnt, &sm.bar);
              });
          }
        }
        if constexpr (K::EARLY) {
          if (!vec) {
            if (ht == 0 && !bulk_wait(&sm.bar, phase, st.err)) ok = 0;
            bar_help<32 * LD>();
#pragma unroll 1
            for (int c = hw; c < z.w2; c += LD) {
              const long long at = cm(0, c, z.ldc);
              span_finish(sC + sidx(z.ab, c, SC), z.C + at + z.ab, z.rows - z.ab, lane);
              if (z.fresh) {
                span_finish(sC + sidx(f0, c, SC), F + at, q0, lane);
                if (n > q0) span_finish(sC + sidx(0, c, SC), F + at + q0, n - q0, lane);
              }
            }
          }
        } else if (!vec) {
          constexpr int NC = 16 / K::LOADS;
#pragma unroll 1
          for (int c = hw; c < z.w2; c += NC * LD) {
            copy_cols<NC, K::LOADS>(sC, SC, z.C, z.ldc, c, LD, z.w2, z.ab, z.rows, lane);
            if (z.fresh) {
              copy_cols<NC, K::LOADS>(sC + f0, SC, F, z.ldc, c, LD, z.w2, 0, q0, lane);
              copy_cols<NC, K::LOADS>(sC - q0, SC, F, z.ldc, c, LD, z.w2, q0, n, lane);
            }
          }
        }
#pragma unroll 1
        for (int c = hw; c < K::LW; c += LD) {
          const double* col = z.C + cm(0, c, z.ldc);
          if (c >= z.w2) {
            for (int r = z.ab + lane; r < 8 * z.nb; r += 32) sC[sidx(r, c, SC)] = 0.0;
            continue;
          }
          if (vec && !K::BULK) {
#pragma unroll 1
            for (int r = z.ab + 2 * lane; r < z.rows; r += 64)
              cp_async16(sC + sidx(r, c, SC), col + r, 16);
            if (z.fresh) {
#pragma unroll 1
              for (int q = 2 * lane; q < n; q += 64)
                cp_async16(sC + sidx(q < q0 ? f0 + q : q - q0, c, SC), col + 2 * n + q, 16);
            }
          }
          // Zero rows up to a full block.
          if (z.rows + lane < 8 * z.nb)
            sC[sidx(z.rows + lane, c, SC)] = 0.0;
        }
        if (!K::BULK) {
          cp_async_commit();
          cp_async_wait<0>();
        } else if (vec || K::EARLY) {
          if (vec && ht == 0 && !bulk_wait(&sm.bar, phase, st.err)) ok = 0;
          phase ^= 1;
        }
      }
    }
    bar_ready<K::THREADS>();
    const bool go = ok != 0;
    if (K::EARLY && ht == 0 && go) st.timeline[4 * s + 3] = gtimer();
    if constexpr (!K::EARLY) {
      if (go) {
        store_leaf<K, LD>(z, sV, SV, lane, hw);
        if constexpr (K::BULK) bar_help<32 * LD>();
        if (ht == 0) {
          __threadfence();
          red_release_add(st.factored + s, 1);
        }
      }
    }
    bar_done<K::THREADS>();
    if (!go) return;
  }
}

template <class K>
BSOFI_DEVINL void chain_main(const BsofGeom& g, const BsofState& st, double* sV, double* part,
                             double* sC, int SV, ChainSmem<K::MW>& sm) {
  constexpr int FW = K::FW, NI = K::NI, MW = K::MW, MT = K::MT, CN = K::CN;
  static_assert(NI * CN <= 23, "V and C in registers");
  // (The shuffle tells the compiler that the warp index is uniform.)
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int gq = lane >> 2, t = lane & 3, gc = col_of(gq);
  const bool top = warp == FW;
  const int n = g.n, SC = SV + 16, capc = SC - 2;
  // Slot i of this warp is 8-row block bb + i bs of the panel.
  double a[NI][CN][2];
#pragma unroll
  for (int i = 0; i < NI; i++)
#pragma unroll
    for (int cs = 0; cs < CN; cs++) a[i][cs][0] = a[i][cs][1] = 0.0;
  {
    const Leaf f = leaf_of(g, st.s_begin);
    const int base = leaf_base(g, f), ab8 = (f.j0 - base) / 8, rows = 2 * n - base;
    long long ld;
    const double* P = mat_ptr(g, st, (long long)f.k * n + base, f.m, f.t * g.NB, ld);
    const bool vec = pair_aligned(P, ld);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int b = top ? ab8 + i : CN + i * FW + warp;
      if (top ? i >= CN : b < ab8 + CN) continue;
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++) {
        const int c = gc + 8 * cs;
        const double2 v = ld_pair(P + cm(0, c, ld), 8 * b + 2 * t, rows, c < f.w, vec);
        a[i][cs][0] = v.x;
        a[i][cs][1] = v.y;
      }
    }
  }
  for (int s = st.s_begin; s < st.s_end; s++) {
    const ChainStep& z = sm.step[s & 1];  // (written before this loop, then by the T warp)
    const int w = z.f.w, ab = z.ab, ab8 = ab / 8, rows = z.rows, nb = z.nb, w2 = z.w2;
    const bool next = z.next, fresh = z.fresh, trans = z.trans;
    double* C = z.C;
    const long long ldc = z.ldc;
    const int blo = top ? ab8 : ab8 + CN, bhi = top ? min(nb, ab8 + CN) : nb;
    const int bb = top ? ab8 : CN + warp, bs = top ? 1 : FW;
    {
      // ---- factor the leaf
      if (top) {
        // (The second store, which the T warp's follows, only keeps an order of
        // instructions that measured faster: n = 144, p = 20 3.51 ms against 3.54.)
        if (lane == 0) {
          const unsigned long long now = gtimer();
          st.timeline[4 * s + 0] = now;
          st.timeline[4 * s + 1] = now;
        }
        factor_top<K>(a, sm, w, gq, t, st.tau + (long long)z.f.k * n + z.f.j0);
      } else {
        factor_rows<K>(a, sm, w, ab8, nb, gq, t, warp);
      }
      // ---- V to shared memory, the pivot rows (R and V) to global memory
      // (columns beyond the leaf's width are zero whatever their scale).
      double sc[CN];
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++) sc[cs] = gc + 8 * cs < w ? sm.sc[gc + 8 * cs] : 0.0;
      const bool vecp = pair_aligned(z.P, z.ldp);
      if (top) {
#pragma unroll
        for (int i = 0; i < CN; i++) {
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) {
            const int c = gc + 8 * cs, r = ab + 8 * i + 2 * t;
            double o[2], v[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const double e = a[i][cs][h];
              const int d = 8 * i + 2 * t + h - c;  // row minus column of the leaf
              o[h] = d > 0 ? e * sc[cs] : e;
              v[h] = d > 0 ? o[h] : ((d == 0 && c < w) ? 1.0 : 0.0);
              a[i][cs][h] = v[h];
            }
            st_pair(z.P + cm(0, c, z.ldp), r, rows, c < w, vecp, o[0], o[1]);
            if (ab8 + i < nb)
              *reinterpret_cast<double2*>(sV + sidx(r, c, SV)) = make_double2(v[0], v[1]);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) {
            const int c = gc + 8 * cs, r = 8 * b + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; h++) a[i][cs][h] *= sc[cs];
            if constexpr (!K::BULK)
              st_pair(z.P + cm(0, c, z.ldp), r, rows, c < w, vecp, a[i][cs][0], a[i][cs][1]);
            *reinterpret_cast<double2*>(sV + sidx(r, c, SV)) =
                make_double2(a[i][cs][0], a[i][cs][1]);
          }
        }
      }
      if constexpr (K::BULK) tc::fence_proxy_async_smem();  // V is stored to global memory by bulk copies
      if constexpr (K::EARLY) bar_v_arrive<K::CT>();
    }
    bar_ready<K::THREADS>();
    if (!sm.ok[s & 1]) {
      bar_done<K::THREADS>();
      return;
    }
    if (next) {
      // ---- leaf s on the tile of leaf s+1, V from the registers that factored
      // it.  That is the tile's last update and only this CTA reads the tile
      // next, so it stays in registers; its rows above the next leaf are final
      // and go to global memory.
      double c[NI][CN][2];
      double acc[CN][2 * CN] = {};
      const bool vec = pair_aligned(C, ldc);
      constexpr int GS = K::GS;
#pragma unroll
      for (int q = 0; q < K::NG; q++) {
        const int ia = q * GS, ie = (ia + GS < NI ? ia + GS : NI);
        const bool any = bb + (ie - 1) * bs >= blo && bb + ia * bs < bhi;
#pragma unroll
        for (int i = ia; i < ie; i++)
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) c[i][cs][0] = c[i][cs][1] = 0.0;
        if (!any) continue;
#pragma unroll
        for (int i = ia; i < ie; i++) {
          const int b = bb + i * bs, r = 8 * b + 2 * t;
          const bool live = b >= blo && b < bhi;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) {
            const int cc = gc + 8 * cs;
            double2 v = make_double2(0.0, 0.0);
            if (live) v = *reinterpret_cast<const double2*>(sC + sidx(r, cc, SC));
            c[i][cs][0] = v.x;
            c[i][cs][1] = v.y;
          }
        }
#pragma unroll
        for (int i = ia; i < ie; i++)
#pragma unroll
          for (int jt = 0; jt < CN; jt++) mma_w<CN>(acc[jt], c[i], a[i][jt][0], a[i][jt][1]);
      }
      double fr[CN][2 * CN];
      reduce_w<MW, CN>(acc, fr, part, sm, gq, t, warp);
      const bool keep_all = s + 1 == st.s_end;
#pragma unroll
      for (int q = 0; q < K::NG; q++) {
        const int ia = q * GS, ie = (ia + GS < NI ? ia + GS : NI);
        if (bb + (ie - 1) * bs < blo || bb + ia * bs >= bhi) continue;
        // (Slots of the group that are not live compute values nobody uses.)
#pragma unroll
        for (int i = ia; i < ie; i++)
          update_block<CN>(c[i], fr, sV, SV, 8 * min(bb + i * bs, nb - 1), gq, t);
      }
      if (top || keep_all) {
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs, r = 8 * b + 2 * t;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++)
            st_pair(C + cm(0, gc + 8 * cs, ldc), r, rows, gc + 8 * cs < w2, vec, c[i][cs][0],
                    c[i][cs][1]);
        }
      }
      if (!trans) {
        // Blocks ab8 + CN .. ab8 + 2 CN - 1 become the next leaf's pivot rows.
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int d = bb + i * bs - (ab8 + CN);
          const bool live = !top && d >= 0 && bb + i * bs < bhi;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) {
            if (live && d < CN)
              *reinterpret_cast<double2*>(sm.top + (gc + 8 * cs) * 16 + 8 * d + 2 * t) =
                  make_double2(c[i][cs][0], c[i][cs][1]);
#pragma unroll
            for (int h = 0; h < 2; h++) a[i][cs][h] = live && d >= CN ? c[i][cs][h] : 0.0;
          }
        }
      } else {
        // Through shared memory, over the tile just read.
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++)
            *reinterpret_cast<double2*>(sC + sidx(8 * b + 2 * t, gc + 8 * cs, SC)) =
                make_double2(c[i][cs][0], c[i][cs][1]);
        }
        bar_main<MT>();
        const int rows2 = fresh ? 2 * n : n;
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = top ? i : CN + i * FW + warp;
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int r = 8 * b + 2 * t + h, cc = gc + 8 * cs;
              double v = 0.0;
              if ((!top || i < CN) && r < rows2 && cc < w2) {
                if (r < n) {
                  v = sC[sidx(n + r, cc, SC)];
                } else {
                  int rr = 8 * nb + r - n;
                  if (rr >= capc) rr -= capc;
                  v = sC[sidx(rr, cc, SC)];
                }
              }
              a[i][cs][h] = v;
            }
        }
      }
    }
    bar_done<K::THREADS>();
    if (top) {
      if (next && !trans) {
#pragma unroll
        for (int i = 0; i < CN; i++)
#pragma unroll
          for (int cs = 0; cs < K::CN; cs++) {
            double2 v = make_double2(0.0, 0.0);
            if (ab8 + CN + i < nb)
              v = *reinterpret_cast<const double2*>(sm.top + (gc + 8 * cs) * 16 + 8 * i + 2 * t);
            a[i][cs][0] = v.x;
            a[i][cs][1] = v.y;
          }
      }
      if (lane == 0) st.timeline[4 * s + 2] = gtimer();
    }
  }
}

// ------------------------------------------------------------ workers
template <class K>
BSOFI_DEVINL void worker(const BsofGeom& g, const BsofState& st, double* sV, double* part, int SV,
                         ChainSmem<K::MW>& sm) {
  constexpr int MW = K::MW, MT = K::MT, NIW = K::NIW, CN = K::CN, LW = K::LW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, t = lane & 3, gc = col_of(gq);
  uint32_t phase = 0;
  const long long first_task = tasks_before(g, st.s_begin);
  const long long total_tasks = tasks_before(g, st.s_end);
  for (;;) {
    if (tid == 0) sm.task = atomicAdd(st.next_task, 1);
    bar_main<MT>();
    const long long task = first_task + sm.task;
    if (task >= total_tasks) return;
    // Leaf of this task: largest s with tasks_before(s) <= task.
    int lo_s = 0, hi_s = g.S - 1;
    while (lo_s < hi_s) {
      const int mid = (lo_s + hi_s + 1) / 2;
      if (tasks_before(g, mid) <= task) lo_s = mid;
      else hi_s = mid - 1;
    }
    const int s = lo_s;
    const int q = 1 + (int)(task - tasks_before(g, s));
    const Leaf f = leaf_of(g, s);
    int m2, t2, lo2, hi2;
    target_of(g, f, q, m2, t2);
    tile_range(g, m2, t2, lo2, hi2);
    const int x2 = tile_id(g, m2, t2);
    const int rows = 2 * g.n - f.j0, nb = (rows + 7) / 8;
    long long ldp, ldc;
    const double* P = mat_ptr(g, st, (long long)f.k * g.n + f.j0, f.m, f.t * g.NB, ldp);
    double* C = tile_ptr(g, st, f.k, f.j0, m2, t2, ldc);
    const int w2 = min(g.NB, g.n - t2 * g.NB);
    // The tile is loaded while the leaf is still being factored.
    if (tid == 0) sm.flag = wait_geq(st, st.cnt + x2, s - lo2) ? 1 : 0;
    bar_main<MT>();
    if (!sm.flag) return;
    double c[NIW][CN][2];
    const bool vecc = pair_aligned(C, ldc);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
#pragma unroll
      for (int cs = 0; cs < K::CN; cs++) {
        const int cc = gc + 8 * cs;
        const double2 v = ld_pair(C + cm(0, cc, ldc), 8 * b + 2 * t, rows, b < nb && cc < w2, vecc);
        c[i][cs][0] = v.x;
        c[i][cs][1] = v.y;
      }
    }
    bar_main<MT>();  // everyone has read sm.flag
    if (tid == 0) sm.flag = wait_geq(st, st.factored + s, 1) ? 1 : 0;
    bar_main<MT>();
    if (!sm.flag) return;
    // V (unit lower trapezoidal) and T to shared memory.
    {
      const bool vec = pair_aligned(P, ldp) && (rows & 1) == 0;
      if (K::BULK && vec && tid == 0 && rows > LW) {
        fence_proxy();
        tc::mbar_arrive_expect_tx(&sm.bar, 8 * f.w * (rows - LW));
        for (int cc = 0; cc < f.w; cc++)
          bulk_load(sV + sidx(LW, cc, SV), P + cm(LW, cc, ldp), rows - LW, &sm.bar);
      }
      if (!vec) {
#pragma unroll
        for (int cc = warp; cc < LW; cc += 2 * MW)
          copy_cols<2, K::LOADS>(sV, SV, P, ldp, cc, MW, f.w, LW, rows, lane);
      }
      for (int cc = warp; cc < LW; cc += MW) {
        const double* col = P + cm(0, cc, ldp);
        if (cc >= f.w) {
          for (int r = LW + lane; r < 8 * nb; r += 32) sV[sidx(r, cc, SV)] = 0.0;
        } else if (vec) {
          if (!K::BULK) {
#pragma unroll 1
            for (int r = LW + 2 * lane; r < rows; r += 64)
              cp_async16(sV + sidx(r, cc, SV), col + r, 16);
          }
          if (lane < 8 && max(rows, LW) + lane < 8 * nb) sV[sidx(max(rows, LW) + lane, cc, SV)] = 0.0;
        } else if (lane < 8 && max(rows, LW) + lane < 8 * nb) {
          sV[sidx(max(rows, LW) + lane, cc, SV)] = 0.0;
        }
      }
      const double* T = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
      for (int e = tid; e < LW * LW; e += MT) {
        const int r = e % LW, cc = e / LW;
        double v = 0.0;
        if (cc < f.w && r < rows) v = r == cc ? 1.0 : (r > cc ? __ldcg(P + cm(r, cc, ldp)) : 0.0);
        sV[sidx(r, cc, SV)] = v;
        sm.T[r][cc] = __ldcg(T + r + 16 * cc);
      }
      if (!K::BULK) {
        cp_async_commit();
        cp_async_wait<0>();
      } else if (vec && rows > LW) {
        if (tid == 0 && !bulk_wait(&sm.bar, phase, st.err)) sm.flag = 0;
        phase ^= 1;
      }
    }
    bar_main<MT>();
    if (!sm.flag) return;
    double acc[CN][2 * CN] = {};
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (b < nb) {
#pragma unroll
        for (int jt = 0; jt < CN; jt++) {
          const double2 v =
              *reinterpret_cast<const double2*>(sV + sidx(8 * b + 2 * t, gc + 8 * jt, SV));
          mma_w<CN>(acc[jt], c[i], v.x, v.y);
        }
      }
    }
    double fr[CN][2 * CN];
    reduce_w<MW, CN>(acc, fr, part, sm, gq, t, warp);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (b < nb) {
        update_block<CN>(c[i], fr, sV, SV, 8 * b, gq, t);
#pragma unroll
        for (int cs = 0; cs < K::CN; cs++)
          st_pair(C + cm(0, gc + 8 * cs, ldc), 8 * b + 2 * t, rows, gc + 8 * cs < w2, vecc,
                  c[i][cs][0], c[i][cs][1]);
      }
    }
    bar_main<MT>();
    if (tid == 0) {
      __threadfence();
      red_release_add(st.cnt + x2, 1);
    }
  }
}

// Workers of the 8-wide forms.  A claimed task is a tile or a pair of neighbouring
// tiles (16 columns) for a whole stage: its rows stay in registers while the
// stage's leaves are applied one after another, so that a leaf costs the load of V
// and the two products, and the tiles move twice a stage instead of twice a leaf.
// Stage j is panel j's leaves; the final panel is two stages, the second one
// (j = L-1) with its rows counted from row n of the panel.  Tiles of the stage
// itself (block column j) need the leaves up to two before their own (the chain
// applies the one before), the others all.  Tasks are claimed in order, a stage's
// own tiles first and from the left: a task waits for leaves that depend on earlier
// tasks only, so any number of workers ends.
//
// What bounds them: the round trip from a published leaf to the tile of the leaf
// after next (store of V, its load, the products, store and load of the tile), which
// has one chain step and a half before the chain waits.  So a stage's own tiles, which
// the chain needs next, are taken one by one (m8n8k4, half the time for the products)
// and the others, whose time is the load of V, in pairs.  An inversion at n = 576,
// p = 12 took 21.5 ms with one task per leaf and tile as in worker(), 18.7 with held
// pairs, 17.4 with early publication, 17.1 with single own tiles (at n = 400,
// p = 64 93.1 -> 91.2).
template <class K>
BSOFI_DEVINL void holder(const BsofGeom& g, const BsofState& st, double* sV, double* part, int SV,
                         ChainSmem<K::MW>& sm) {
  constexpr int MW = K::MW, MT = K::MT, NIW = K::NIW, LW = K::LW;
  static_assert(LW == 8, "a pair of 8-wide tiles is one 16-row operand");
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int gq = lane >> 2, t = lane & 3, gc = col_of(gq);
  const int n = g.n, L = g.L, nl = g.nl;
  uint32_t phase = 0;
  // Pairs per stage: its own tiles 1.., a block column, the halves of G.
  const int own = nl - 1, half = (nl + 1) / 2, gp = g.form_g ? 2 * half : 0;
  const int per = own + 2 * half + gp, regular = (L - 2) * per;
  const int total = regular + (own + half + gp) + (own + gp);
  for (;;) {
    if (tid == 0) sm.task = atomicAdd(st.next_task, 1);
    bar_main<MT>();
    int q = sm.task;
    if (q >= total) return;
    int j = L - 2;
    if (q < regular) {
      j = q / per;
      q -= j * per;
    } else {
      q -= regular;
      if (q >= own + half + gp) {
        q -= own + half + gp;
        j = L - 1;
      }
    }
    // Tiles t0, t0 + 1 of block column m, and how many of the stage's leaves each gets.
    int m, t0, e0, e1;
    if (q < own) {
      m = j;
      t0 = 1 + q;
      e0 = t0 - 1;
      e1 = 0;
    } else {
      q -= own;
      const int part_of = q / half, nmat = j <= L - 3 ? 2 : (j == L - 2 ? 1 : 0);
      t0 = 2 * (q % half);
      m = part_of >= nmat ? L + 2 * min(j, L - 2) + part_of - nmat : (part_of == 0 ? j + 1 : L - 1);
      // The chain applies a leaf to its first target: the stage's last leaf to tile 0 of block
      // column j+1, and after the last one of all to the first tile of G.
      const bool first = m == j + 1 || (j == L - 1 && m == L + 2 * (L - 2));
      e0 = first && t0 == 0 ? nl - 1 : nl;
      e1 = nl;
    }
    if (t0 + 1 >= nl) e1 = 0;
    const bool pair = e1 > 0;
    int lo, hi;
    tile_range(g, m, t0, lo, hi);
    int* cnt = st.cnt + tile_id(g, m, t0);
    if (tid == 0)
      sm.flag = (e0 == 0 || wait_geq(st, cnt, j * nl - lo)) &&
                        (e1 == 0 || wait_geq(st, cnt + 1, j * nl - lo))
                    ? 1
                    : 0;
    bar_main<MT>();
    if (!sm.flag) return;
    const int k = min(j, L - 2), base = j == L - 1 ? n : 0;
    const int rows = 2 * n - base, nb = (rows + 7) / 8, w2 = min(2 * LW, n - t0 * LW);
    long long ldc;
    double* C = tile_ptr(g, st, k, base, m, t0, ldc);
    const bool vecc = pair_aligned(C, ldc);
    double c[NIW][2][2];
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
#pragma unroll
      for (int cs = 0; cs < 2; cs++) {
        const double2 v = ld_pair(C + cm(0, gc + 8 * cs, ldc), 8 * b + 2 * t, rows,
                                  b < nb && gc + 8 * cs < w2 && (cs == 0 ? e0 : e1) > 0, vecc);
        c[i][cs][0] = v.x;
        c[i][cs][1] = v.y;
      }
    }
#pragma unroll 1
    for (int l = 0; l < max(e0, e1); l++) {
      const int s = j * nl + l, ab = LW * l;
      bar_main<MT>();  // everyone has read sm.flag and V
      if (tid == 0) sm.flag = wait_geq(st, st.factored + s, 1) ? 1 : 0;
      bar_main<MT>();
      if (!sm.flag) return;
      // V (unit lower trapezoidal) and T to shared memory.
      {
        const Leaf f = leaf_of(g, s);
        long long ldp;
        const double* P = mat_ptr(g, st, (long long)k * n + f.j0, f.m, f.t * LW, ldp);
        const int left = rows - ab;  // rows from the leaf's first on
        const bool vec = pair_aligned(P, ldp) && (left & 1) == 0;
        double* V = sV + ab;
        if (tid == 0 && left > LW) {
          issue_columns(V + LW, SV, P + LW, ldp, f.w, left - LW, vec, &sm.bar);
        }
        static_assert(MW == LW, "a warp per column");
        if (warp >= f.w) {
          for (int r = LW + lane; r < 8 * nb - ab; r += 32) V[sidx(r, warp, SV)] = 0.0;
        } else {
          if (max(left, LW) + lane < 8 * nb - ab) V[sidx(max(left, LW) + lane, warp, SV)] = 0.0;
        }
        const double* T = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
        if (tid < LW * LW) {
          const int r = tid % LW, cc = tid / LW;
          double v = 0.0;
          if (cc < f.w && r < left) v = r == cc ? 1.0 : (r > cc ? __ldcg(P + cm(r, cc, ldp)) : 0.0);
          V[sidx(r, cc, SV)] = v;
        } else if (tid < 2 * LW * LW) {
          const int r = tid % LW, cc = (tid - LW * LW) / LW;
          sm.T[r][cc] = __ldcg(T + r + 16 * cc);
        }
        if (left > LW) {
          if (tid == 0 && !bulk_wait(&sm.bar, phase, st.err)) sm.flag = 0;
          phase ^= 1;
          if (!vec) {
            bar_main<MT>();
            if (warp < f.w)
              span_finish(V + sidx(LW, warp, SV), P + cm(LW, warp, ldp), left - LW, lane);
          }
        }
      }
      bar_main<MT>();
      if (!sm.flag) return;
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      if (pair) {
#pragma unroll
        for (int i = 0; i < NIW; i++) {
          const int b = warp + i * MW;
          if (b < l || b >= nb) continue;
          const double2 v = *reinterpret_cast<const double2*>(sV + sidx(8 * b + 2 * t, gc, SV));
          dmma_16x8x8(acc, c[i][0][0], c[i][1][0], c[i][0][1], c[i][1][1], v.x, v.y);
        }
      } else {
        double a2[2] = {0.0, 0.0};
#pragma unroll
        for (int i = 0; i < NIW; i++) {
          const int b = warp + i * MW;
          if (b < l || b >= nb) continue;
          const double2 v = *reinterpret_cast<const double2*>(sV + sidx(8 * b + 2 * t, gc, SV));
          dmma_8x8x4(a2, c[i][0][0], v.x);
          dmma_8x8x4(a2, c[i][0][1], v.y);
        }
        acc[0] = a2[0];
        acc[1] = a2[1];
      }
      // -(W^T T) summed over the warps, as in reduce_w.
      double fr[4];
      {
        double o[4] = {0.0, 0.0, 0.0, 0.0};
        dmma_16x8x8(o, acc[0], acc[2], acc[1], acc[3], sm.T[t][gq], sm.T[t + 4][gq]);
#pragma unroll
        for (int h = 0; h < 2; h++)
          *reinterpret_cast<double2*>(part + warp * 128 + (gc + 8 * h) * 8 + 2 * t) =
              make_double2(o[2 * h], o[2 * h + 1]);
        bar_main<MT>();
        if (tid < 128) {
          double sum[MW];
#pragma unroll
          for (int u = 0; u < MW; u++) sum[u] = part[u * 128 + tid];
#pragma unroll
          for (int d = MW / 2; d > 0; d /= 2)
#pragma unroll
            for (int u = 0; u < d; u++) sum[u] += sum[u + d];
          sm.W[tid] = -sum[0];
        }
        bar_main<MT>();
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const double2 v = *reinterpret_cast<const double2*>(sm.W + (gc + 8 * h) * 8 + 2 * t);
          fr[h] = v.x;
          fr[2 + h] = v.y;
        }
      }
      if (pair) {
#pragma unroll
        for (int i = 0; i < NIW; i++) {
          const int b = warp + i * MW;
          if (b < l || b >= nb) continue;
          double d[4] = {c[i][0][0], c[i][0][1], c[i][1][0], c[i][1][1]};
          dmma_16x8x8(d, fr[0], fr[1], fr[2], fr[3], sV[sidx(8 * b + gq, 2 * t, SV)],
                      sV[sidx(8 * b + gq, 2 * t + 1, SV)]);
          c[i][0][0] = d[0];
          c[i][0][1] = d[1];
          c[i][1][0] = d[2];
          c[i][1][1] = d[3];
        }
      } else {
#pragma unroll
        for (int i = 0; i < NIW; i++) {
          const int b = warp + i * MW;
          if (b < l || b >= nb) continue;
          dmma_8x8x4(c[i][0], fr[0], sV[sidx(8 * b + gq, 2 * t, SV)]);
          dmma_8x8x4(c[i][0], fr[2], sV[sidx(8 * b + gq, 2 * t + 1, SV)]);
        }
      }
      const bool out0 = l + 1 == e0, out1 = l + 1 == e1;
      if (out0 || out1) {
#pragma unroll
        for (int i = 0; i < NIW; i++) {
          const int b = warp + i * MW;
          if (b >= nb) continue;
#pragma unroll
          for (int cs = 0; cs < 2; cs++)
            st_pair(C + cm(0, gc + 8 * cs, ldc), 8 * b + 2 * t, rows,
                    gc + 8 * cs < w2 && (cs == 0 ? out0 : out1), vecc, c[i][cs][0], c[i][cs][1]);
        }
        bar_main<MT>();
        if (tid == 0) {
          __threadfence();
          if (out0) red_release_add(cnt, e0);
          if (out1) red_release_add(cnt + 1, e1);
        }
      }
    }
  }
}

template <class K>
__global__ void __launch_bounds__(K::THREADS, 1) bsof_persistent_kernel(BsofGeom g, BsofState st) {
  extern __shared__ __align__(16) double dyn_bsof[];
  __shared__ __align__(16) ChainSmem<K::MW> sm;
  const int SV = tile_stride(g.n);
  double* sV = dyn_bsof;
  double* part = sV + K::LW * SV;
  double* sC = part + K::MW * 16 * K::LW;
  if (threadIdx.x == 0) {
    tc::mbar_init(&sm.bar, 1);
    tc::fence_barrier_init();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    sm.step[st.s_begin & 1] = chain_step(g, st, st.s_begin);
  __syncthreads();
  if (threadIdx.x >= K::MT) {
    if constexpr (K::REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (blockIdx.x == 0) chain_helper<K>(g, st, sV, sC, SV, sm);
  } else {
    if constexpr (K::REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    if (blockIdx.x == 0) chain_main<K>(g, st, sV, part, sC, SV, sm);
    else if constexpr (K::CN == 1) holder<K>(g, st, sV, part, SV, sm);
    else worker<K>(g, st, sV, part, SV, sm);
  }
}

// ------------------------------------------------------------------ Q_k^T
// G_k = Q_k^T of every panel from the stored reflectors and the leaves' T, for
// callers whose BSOI comes with a state of its own (reference: the dormqr of
// lapackXbsoi_ormqr, src/bsofi_cpu.c:234-245).  A CTA owns 16 columns of one
// G_k: they stay in its registers, from the identity on, while the panel's
// leaves pass through shared memory, so G is written once and read never.
// What bounds it: the FP64 tensor pipe (four m16n8k8 per 8 rows and leaf) and
// the barriers around W; two or more CTAs an SM overlap them.  Before, one
// launch per leaf read and wrote all of G: 653 us at n = 144, p = 20 and 445 us
// at n = 100, p = 64 (a few tens of them products at the tensor rate); now 59 and
// 64 us.
struct FormQArgs {
  const double* A;
  long long ld;
  int n, L;
  const double* T;  // 256 doubles per leaf: (k * maxleaves + l) * 256
  int maxleaves, nbw;
  double* G;
};

template <class K, int PER>
__global__ void __launch_bounds__(K::MT, PER) form_q_kernel(FormQArgs s) {
  extern __shared__ __align__(16) double dyn_bsof[];
  __shared__ __align__(16) ChainSmem<K::MW> sm;
  constexpr int MW = K::MW, MT = K::MT, NIW = K::NIW;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int gq = lane >> 2, t = lane & 3, gc = col_of(gq);
  const int n = s.n, n2 = 2 * n, SV = tile_stride(n), nb = (n2 + 7) / 8;
  double* sV = dyn_bsof;
  double* part = sV + 16 * SV;
  // The last panel has twice the leaves: first.
  const int k = s.L - 2 - blockIdx.y, x0 = blockIdx.x * 16;
  const int refl = k == s.L - 2 ? n2 : n;
  double c[NIW][2][2];
#pragma unroll
  for (int i = 0; i < NIW; i++)
#pragma unroll
    for (int cs = 0; cs < 2; cs++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        c[i][cs][h] = 8 * (warp + i * MW) + 2 * t + h == x0 + gc + 8 * cs ? 1.0 : 0.0;
  for (int j0 = 0, l = 0; j0 < refl; j0 += s.nbw, l++) {
    const int w = min(s.nbw, refl - j0);
    const double* P = s.A + cm((long long)k * n, (long long)k * n + j0, s.ld);  // row 0
    const bool vec = pair_aligned(P, s.ld);
    const double* T = s.T + ((long long)k * s.maxleaves + l) * 256;
    // Rows from j0 + 16 on as stored, the 16 above masked to unit lower
    // trapezoidal; zero up to a full block and in columns beyond the leaf.
    for (int cc = warp; cc < 16; cc += MW) {
      const double* col = P + cm(0, cc, s.ld);
      if (cc < w && vec) {
        for (int r = j0 + 16 + 2 * lane; r < 8 * nb; r += 64)
          cp_async16(sV + sidx(r, cc, SV), r < n2 ? col + r : col, r + 1 < n2 ? 16 : (r < n2 ? 8 : 0));
      } else {
        for (int r = j0 + 16 + lane; r < 8 * nb; r += 32)
          sV[sidx(r, cc, SV)] = cc < w && r < n2 ? col[r] : 0.0;
      }
    }
    cp_async_commit();
    for (int e = tid; e < 256; e += MT) {
      const int r = e & 15, cc = e >> 4;
      double v = 0.0;
      if (cc < w && j0 + r < n2) v = r == cc ? 1.0 : (r > cc ? P[cm(j0 + r, cc, s.ld)] : 0.0);
      if (j0 + r < 8 * nb) sV[sidx(j0 + r, cc, SV)] = v;
      sm.T[r][cc] = T[e];
    }
    cp_async_wait<0>();
    bar_main<MT>();
    double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (8 * b + 7 >= j0 && b < nb) {
#pragma unroll
        for (int jt = 0; jt < 2; jt++) {
          const double2 v =
              *reinterpret_cast<const double2*>(sV + sidx(8 * b + 2 * t, gc + 8 * jt, SV));
          dmma_16x8x8(acc[jt], c[i][0][0], c[i][1][0], c[i][0][1], c[i][1][1], v.x, v.y);
        }
      }
    }
    double fr[2][4];
    reduce_w<MW, 2>(acc, fr, part, sm, gq, t, warp);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (8 * b + 7 >= j0 && b < nb) update_block<2>(c[i], fr, sV, SV, 8 * b, gq, t);
    }
    bar_main<MT>();  // V, T and W are no longer read
  }
  double* C = s.G + (long long)k * n2 * n2 + cm(0, x0, n2);
  const bool vecc = pair_aligned(C, n2);  // (as the caller's workspace is)
#pragma unroll
  for (int i = 0; i < NIW; i++) {
    const int b = warp + i * MW;
#pragma unroll
    for (int cs = 0; cs < 2; cs++)
      st_pair(C + cm(0, gc + 8 * cs, n2), 8 * b + 2 * t, n2, b < nb && x0 + gc + 8 * cs < n2, vecc,
              c[i][cs][0], c[i][cs][1]);
  }
}

// ------------------------------------------------------------------ launcher
using Chain64 = ChainCfg<3, 5, 4>;
using Chain128 = ChainCfg<7, 5, 4>;
using Chain256 = ChainCfg<7, 9, 8>;
using Chain416 = ChainCfg<7, 15, 13, 1>;
// (The next two spill 260 and 340 bytes a thread: the leaf takes 84 and 92 registers, the
// pivot column or the next tile beside it as many again.)
using Chain592 = ChainCfg<7, 21, 19, 1>;
using Chain640 = ChainCfg<7, 23, 20, 1>;
using FormQ400 = ChainCfg<7, 14, 13>;
using FormQ640 = ChainCfg<7, 23, 20>;

// Leaf width.  Wide leaves halve the publications and updates, but a column step's
// two column sets and an update's 16 columns cost the chain more than twice the
// narrow ones' time once a warp has many row blocks: inversion in ms, 16-wide ->
// 8-wide with held tiles: n = 300, p = 20 11.7 -> 10.3; 361, 20 17.1 -> 16.2; 400, 64
// 95.6 -> 91.2.  Up to n = 256 the 16-wide leaves' chain does not wait for its
// workers, and their fine tasks suit the few workers of a batch's instances.
int bsof_leaf_width(int n) { return n <= Chain256::MAX_ROWS / 2 ? 16 : 8; }

int bsof_tiles(int n) { return (n + bsof_leaf_width(n) - 1) / bsof_leaf_width(n); }

template <class K>
static size_t dyn_smem(int n) {
  const size_t SV = tile_stride(n);
  return sizeof(double) * (K::LW * SV + 16 * K::LW * K::MW + K::LW * (SV + 16));
}

template <class K>
static cudaError_t launch_cfg(const BsofGeom& g, const BsofState& st, int workers, cudaStream_t s) {
  static PerDevice once;
  static int sms[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int count = dev < kMaxDevices ? sms[dev] : 0;
  if (once.pending() >= 0 || count == 0) {
    if ((e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
      return e;
    e = cudaFuncSetAttribute(bsof_persistent_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dyn_smem<K>(K::MAX_ROWS / 2));
    if (e != cudaSuccess) return e;
    if (dev < kMaxDevices) sms[dev] = count;
    once.mark(dev);
  }
  // At least one CTA of any size fits each SM.
  const int grid = min(1 + workers, count);
  void* args[] = {(void*)&g, (void*)&st};
  return cudaLaunchCooperativeKernel((const void*)bsof_persistent_kernel<K>, dim3(grid),
                                     dim3(K::THREADS), args, dyn_smem<K>(g.n), s);
}

cudaError_t launch_bsof_persistent(double* A, long long ld, int n, int L, double* tau, double* T,
                                   double* G, int maxleaves, int* cnt, int* factored,
                                   int* next_task, int* err, unsigned long long* timeline,
                                   int workers, cudaStream_t st, int s_begin, int s_end,
                                   double* Al, long long ldl) {
  BsofGeom g;
  g.form_g = G != nullptr;
  g.n = n;
  g.L = L;
  g.NB = bsof_leaf_width(n);
  g.nl = bsof_tiles(n);
  g.S = (L - 2) * g.nl + 2 * g.nl;
  BsofState s;
  s.A = A;
  s.ld = ld;
  s.Al = Al ? Al : A + cm(0, (long long)(L - 1) * n, ld);
  s.ldl = Al ? ldl : ld;
  s.G = G;
  s.tau = tau;
  s.T = T;
  s.maxleaves = maxleaves;
  s.cnt = cnt;
  s.factored = factored;
  s.next_task = next_task;
  s.err = err;
  s.timeline = timeline;
  s.spin_limit = 1ll << 22;  // polls of ~0.5 us each: a few seconds at most
  s.s_begin = s_begin > 0 ? s_begin : 0;
  s.s_end = (s_end < 0 || s_end > g.S) ? g.S : s_end;
  if (s.s_begin >= s.s_end) return cudaSuccess;
  if (2 * n <= Chain64::MAX_ROWS) return launch_cfg<Chain64>(g, s, workers, st);
  if (2 * n <= Chain128::MAX_ROWS) return launch_cfg<Chain128>(g, s, workers, st);
  if (2 * n <= Chain256::MAX_ROWS) return launch_cfg<Chain256>(g, s, workers, st);
  if (s.s_begin > 0 || s.s_end < g.S) return cudaErrorInvalidValue;  // stages are not split
  if (2 * n <= Chain416::MAX_ROWS) return launch_cfg<Chain416>(g, s, workers, st);
  if (2 * n <= Chain592::MAX_ROWS) return launch_cfg<Chain592>(g, s, workers, st);
  if (2 * n <= Chain640::MAX_ROWS) return launch_cfg<Chain640>(g, s, workers, st);
  return launch_bsof_tall(g, s, workers, st);
}

template <class K, int PER>
static cudaError_t launch_form_q_cfg(const FormQArgs& a, cudaStream_t st) {
  static PerDevice once;
  const int dev = once.pending();
  if (dev >= 0) {
    const size_t most =
        sizeof(double) * (16 * (size_t)tile_stride(K::MAX_ROWS / 2) + 256 * K::MW);
    cudaError_t e = cudaFuncSetAttribute(form_q_kernel<K, PER>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return e;
    once.mark(dev);
  }
  form_q_kernel<K, PER><<<dim3((2 * a.n + 15) / 16, a.L - 1), K::MT,
                          sizeof(double) * (16 * (size_t)tile_stride(a.n) + 256 * K::MW), st>>>(a);
  return cudaGetLastError();
}

bool form_q_fits(int n) { return 2 * n <= FormQ640::MAX_ROWS; }

cudaError_t launch_form_q(const double* A, long long ld, int n, int L, const double* T,
                          int maxleaves, int nbw, double* G, cudaStream_t st) {
  const FormQArgs a = {A, ld, n, L, T, maxleaves, nbw, G};
  if (2 * n <= Chain64::MAX_ROWS) return launch_form_q_cfg<Chain64, 4>(a, st);
  if (2 * n <= Chain128::MAX_ROWS) return launch_form_q_cfg<Chain128, 2>(a, st);
  if (2 * n <= Chain256::MAX_ROWS) return launch_form_q_cfg<Chain256, 2>(a, st);
  if (2 * n <= FormQ400::MAX_ROWS) return launch_form_q_cfg<FormQ400, 1>(a, st);
  if (2 * n <= FormQ640::MAX_ROWS) return launch_form_q_cfg<FormQ640, 1>(a, st);
  return cudaErrorInvalidValue;
}

cudaError_t launch_reflector(int count, const double* xnorm2, const double* alpha, double* out,
                             cudaStream_t st) {
  reflector_kernel<<<(unsigned)((count + 7ll) / 8), 256, 0, st>>>(count, xnorm2, alpha, out);
  return cudaGetLastError();
}

cudaError_t preload_bsof(size_t* local) {
  cudaError_t e;
  if ((e = preload_one(bsof_persistent_kernel<Chain64>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain128>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain256>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain416>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain64, 4>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain128, 2>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain256, 2>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<FormQ400, 1>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<FormQ640, 1>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain592>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain640>, local)) != cudaSuccess) return e;
  return preload_bsof_tall(local);
}

}  // namespace bsofi
