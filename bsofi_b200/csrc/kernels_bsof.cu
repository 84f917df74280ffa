// BSOF as one persistent kernel.
//
// Reference: lapackXbsof, src/bsofi_cpu.c:86-118: for k = 0..L-3, dgeqrf of
// the stacked 2n x n panel [R~_k; B_k] at A_BLK(k,k), dormqr('L','T') of
// A_BLK(k,k+1) and A_BLK(k,L-1); then dgeqrf of the final 2n x 2n block.
//
// Work decomposition.  Every block column is cut into tiles of 16 columns
// (the last one may be narrower).  A "leaf" is the Householder QR of one tile
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
// 4 g + t of a warp owns two columns and rows 2t, 2t+1 of each of its 8-row
// blocks.  That layout makes a column step cheap in every part: the pivot
// column reaches the lanes of a row block by one shuffle per row, a column's
// dot products end in a sum over four lanes (a DMMA with ones), and there is
// one barrier per column, after which every warp sums the warps' partials and
// forms the reflector's scalars for itself (a second barrier, with one warp
// forming them for all, measured the same at n = 256 and slower below; two
// columns per barrier, the second one's products corrected for the first
// reflector, measured slower everywhere: one warp's scalar code then takes
// longer than the barrier it saves).  The 16 pivot rows of a leaf belong to
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
// p = 64 41.2 -> 32.  Per 16-column leaf at n = 256: 9.5 us of column steps
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
template <int FW_, int NI_, int NIW_>
struct ChainCfg {
  static constexpr int FW = FW_, NI = NI_, NIW = NIW_;
  static constexpr int MW = FW + 1, MT = 32 * MW;
  static constexpr int HW = 4;  // helper warps: one builds T, the others load and store
  static constexpr int THREADS = MT + 32 * HW;
  static constexpr int CT = MT + 32;  // column barrier: with the T warp, the last helper
  // Largest panel height 2n: rows owned by the chain's warps and a worker's.
  static constexpr int ROWS_CHAIN = 8 * (2 + FW * NI), ROWS_WORK = 8 * MW * NIW;
  static constexpr int MAX_ROWS = ROWS_CHAIN < ROWS_WORK ? ROWS_CHAIN : ROWS_WORK;
  // Row slots are taken in groups of GS, skipped when every row is finished.
  static constexpr int GS = 3, NG = (NI + GS - 1) / GS;
  // Tiles move between global and shared memory by bulk copies, which keep the
  // load/store pipe free for the computing warps, or (short panels, where the
  // chain waits for the workers' answer and latency counts) by cp.async and
  // by stores of the warps that hold the reflectors.
  static constexpr bool BULK = NI > 5;
  // Loads a lane and column in flight where columns are copied by plain loads.
  static constexpr int LOADS = ROWS_WORK <= 128 ? 4 : (ROWS_WORK <= 256 ? 8 : 16);
  // V as the operand of W = V^T C comes from the registers that factored it,
  // or, where V and C do not fit in registers together, from shared memory.
  static constexpr bool VREG = NI <= 9;
  // With 12 warps a thread gets 168 registers at launch; the helper warpgroup
  // gives most of its own to the two that compute
  // (2 x 128 x 224 + 128 x 56 = 384 x 168).
  static constexpr bool REGS = THREADS == 384;
  static_assert(MW == 4 || MW == 8, "partial sums are read as 4 or 8 per column");
};

// Leaf s as the chain CTA sees it.  Rows are counted from the top of the
// panel, except in the second half of the final panel when n is not a
// multiple of 16: there from its row n on, so that a leaf's first row is
// always a multiple of 16.
struct ChainStep {
  Leaf f;
  int base, ab, rows, nb;  // first row counted, the leaf's first row, panel rows, 8-row blocks
  int m2, t2, lo2, w2;     // the tile of leaf s+1
  bool next, fresh, trans;
  double *P, *C;           // row 0, column 0 of the leaf's tile and of the next one
  long long ldp, ldc;
};

BSOFI_DEVINL int leaf_base(const BsofGeom& g, const Leaf& f) {
  return (f.k == g.L - 2 && f.l >= g.nl && (g.n & 15) != 0) ? g.n : 0;
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
  c.P = mat_ptr(g, st, (long long)c.f.k * g.n + c.base, c.f.m, c.f.t * 16, c.ldp);
  c.w2 = min(16, g.n - c.t2 * 16);
  // Panel change (rows shift by n, n fresh rows come in), and the shift by n
  // inside the final panel when n is not a multiple of 16.
  c.fresh = c.next && c.f.l == g.nl - 1 && c.f.k <= g.L - 3;
  c.trans = c.fresh || (c.next && c.f.l == g.nl - 1 && (g.n & 15) != 0);
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
template <int COUNT>
BSOFI_DEVINL void bar_all() {
  asm volatile("bar.sync 3, %0;" ::"n"(COUNT) : "memory");
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

// ------------------------------------------------------------ column steps
struct Refl {
  double tau, scale, beta, q;  // q = tau * scale = -1 / beta
};
// LAPACK dlarfg: beta = -sign(alpha) ||(alpha, x)||, tau = (beta - alpha)/beta
// = 1 + |alpha|/||.||, scale = 1/(alpha - beta).  The square root, its
// reciprocal and 1/(|alpha| + ||.||) are the longest dependent chain of a
// column step, so they share one: Goldschmidt's coupled iteration (Markstein,
// "Software division and square root using Goldschmidt's algorithms", 2004)
// from the hardware's approximation gives norm and half its reciprocal
// together, Newton's residual step finishes each, and the last reciprocal
// starts from the first norm estimate meanwhile.  Against long double on 10^6
// random pairs the largest errors are, in units of 2^-53, beta 1.48, tau 1.40, scale
// 2.62 (with rsqrt() and a division: beta 1.92, scale 3.04).  Outside the range
// where the approximations are normal numbers those functions are called.
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

// Warp sums of the two columns' partial dot products into red[column][warp]:
// again DMMAs with ones, whose results lane 4 g + t holds for columns 2t, 2t+1.
template <int MW>
BSOFI_DEVINL void put_partials(double* red, double d0, double d1, int g, int t, int warp) {
  double e0[2] = {0.0, 0.0}, e1[2] = {0.0, 0.0};
  dmma_8x8x4(e0, 1.0, d0);
  dmma_8x8x4(e1, 1.0, d1);
  if (g < 2) {
    double* dst = red + (8 * g + 2 * t) * MW + warp;
    dst[0] = g == 0 ? e0[0] : e1[0];
    dst[MW] = g == 0 ? e0[1] : e1[1];
  }
}

// One pass of a row warp over its rows: the update by the finished pivot
// column I (half CSU; factors f0, f1 for columns g, g+8, zero where a column
// is finished; UPD0: some of columns g are pending) and the dot products with
// the next pivot column J = I+1 (half CSD).  ab8: first 8-row block of the
// leaf; nb: row blocks of the panel.
template <class K, bool UPD0, int CSU, int CSD>
BSOFI_DEVINL void row_pass(double (&a)[K::NI][2][2], double (&x)[K::NI][2],
                           double f0, double f1, int srcd, int ab8, int nb, int warp,
                           double& d0, double& d1) {
  double s0[2] = {0.0, 0.0}, s1[2] = {0.0, 0.0};
#pragma unroll
  for (int q = 0; q < K::NG; q++) {
    constexpr int GS = K::GS;
    const int ia = q * GS, ie = (ia + GS < K::NI ? ia + GS : K::NI);
    if ((ie - 1) * K::FW + warp < ab8 || 2 + ia * K::FW + warp >= nb) continue;
#pragma unroll
    for (int i = ia; i < ie; i++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const double xo = x[i][h];
        if (UPD0) a[i][0][h] = fma(-xo, f0, a[i][0][h]);
        a[i][1][h] = fma(-xo, f1, a[i][1][h]);
        const double xn = shfl_d(a[i][CSD][h], srcd);
        x[i][h] = xn;
        s0[h] = fma(xn, a[i][0][h], s0[h]);
        s1[h] = fma(xn, a[i][1][h], s1[h]);
      }
    }
  }
  d0 = s0[0] + s0[1];
  d1 = s1[0] + s1[1];
}

// The dot products with column 0, before the first column step.
template <class K>
BSOFI_DEVINL void row_first(double (&a)[K::NI][2][2], double (&x)[K::NI][2], int t,
                            double& d0, double& d1) {
  double s0[2] = {0.0, 0.0}, s1[2] = {0.0, 0.0};
#pragma unroll
  for (int i = 0; i < K::NI; i++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double xn = shfl_d(a[i][0][h], t);
      x[i][h] = xn;
      s0[h] = fma(xn, a[i][0][h], s0[h]);
      s1[h] = fma(xn, a[i][1][h], s1[h]);
    }
  d0 = s0[0] + s0[1];
  d1 = s1[0] + s1[1];
}

// Sums, reflector and v_I^T a_c of this lane's columns at column step I.
struct ColStep {
  Refl rf;
  double w0, w1;
};
template <int MW>
BSOFI_DEVINL ColStep col_step(const ChainSmem<MW>& sm, int I, int g, int t) {
  const int buf = I & 1, ri = group_of(I & 7) + (I & 8);
  ColStep c;
  const double alpha = sm.prow[buf][ri], pr0 = sm.prow[buf][g], pr1 = sm.prow[buf][g + 8];
  const double sp = col_total<MW>(sm.red[buf], ri, t);
  const double s0 = col_total<MW>(sm.red[buf], g, t);
  const double s1 = col_total<MW>(sm.red[buf], g + 8, t);
  c.rf = reflector(sp, alpha);
  // v_I^T a_c = a_Ic + scale d_c.
  c.w0 = fma(c.rf.scale, s0, pr0);
  c.w1 = fma(c.rf.scale, s1, pr1);
  return c;
}

// The column loop of a row warp.
template <class K>
BSOFI_DEVINL void factor_rows(double (&a)[K::NI][2][2], ChainSmem<K::MW>& sm, int w, int ab8,
                              int nb, int g, int t, int warp) {
  constexpr int MW = K::MW;
  const int c0 = col_of(g), c1 = c0 + 8;
  double x[K::NI][2];
  double d0, d1;
  row_first<K>(a, x, t, d0, d1);
  put_partials<MW>(sm.red[0], d0, d1, g, t, warp);
  int I = 0;
  auto step = [&](auto upd0, auto csu, auto csd) {
    bar_col<K::CT>();
    const ColStep c = col_step<MW>(sm, I, g, t);
    const double f0 = c0 > I ? c.rf.q * c.w0 : 0.0, f1 = c1 > I ? c.rf.q * c.w1 : 0.0;
    const int sd = group_of((I + 1) & 7) * 4 + t;
    row_pass<K, upd0.value != 0, csu.value, csd.value>(a, x, f0, f1, sd, ab8, nb, warp, d0, d1);
    put_partials<MW>(sm.red[(I + 1) & 1], d0, d1, g, t, warp);
  };
  using Z = std::integral_constant<int, 0>;
  using O = std::integral_constant<int, 1>;
  const int last = w - 1;
#pragma unroll 1
  for (; I < min(last, 7); I++) step(O{}, Z{}, Z{});
  if (I < last) {  // I = 7
    step(Z{}, Z{}, O{});
    I++;
#pragma unroll 1
    for (; I < last; I++) step(Z{}, O{}, O{});
  }
  bar_col<K::CT>();  // the last column's sums are there
  bar_col<K::CT>();  // and its scale
}

// The top warp's 16 pivot rows (blocks 0, 1 in a[0], a[1]): update by pivot
// column I (half CSU; rows below I; row I by v_I = 1, its pivot entry becomes
// beta).
template <class K, int CSU>
BSOFI_DEVINL void top_update(double (&a)[K::NI][2][2], const double (&x)[2][2], const Refl& rf,
                             double F0, double F1, int I, int g, int t) {
#pragma unroll
  for (int b = CSU; b < 2; b++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int row = 8 * b + 2 * t + h;
      const double v = row == I ? 1.0 : x[b][h] * rf.scale;
      if (CSU == 0) a[b][0][h] = fma(-v, F0, a[b][0][h]);
      a[b][1][h] = fma(-v, F1, a[b][1][h]);
      if (b == CSU && row == I && g == group_of(I & 7)) a[b][CSU][h] = rf.beta;
    }
}

// Dot products with column J (half CSD) over rows below J, and row J to prow.
template <class K, int CSD>
BSOFI_DEVINL void top_dots(const double (&a)[K::NI][2][2], double (&x)[2][2], int J, int g, int t,
                           double* prow, double& d0, double& d1) {
  const int src = group_of(J & 7) * 4 + t;
  d0 = d1 = 0.0;
#pragma unroll
  for (int b = CSD; b < 2; b++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int row = 8 * b + 2 * t + h;
      const double xs = shfl_d(a[b][CSD][h], src);
      x[b][h] = row > J ? xs : 0.0;
      d0 = fma(x[b][h], a[b][0][h], d0);
      d1 = fma(x[b][h], a[b][1][h], d1);
      if (b == CSD && row == J) {
        prow[g] = a[b][0][h];
        prow[g + 8] = a[b][1][h];
      }
    }
}

// The column loop of the top warp.
template <class K>
BSOFI_DEVINL void factor_top(double (&a)[K::NI][2][2], ChainSmem<K::MW>& sm, int w, int g, int t,
                             double* tau) {
  constexpr int MW = K::MW;
  const int c0 = col_of(g), c1 = c0 + 8;
  double x[2][2], d0, d1, sc0 = 0.0, sc1 = 0.0;
  top_dots<K, 0>(a, x, 0, g, t, sm.prow[0], d0, d1);
  put_partials<MW>(sm.red[0], d0, d1, g, t, K::FW);
  int I = 0;
  auto step = [&](auto csu, auto csd, auto dot) {
    bar_col<K::CT>();
    const ColStep c = col_step<MW>(sm, I, g, t);
    const double F0 = c0 > I ? c.rf.tau * c.w0 : 0.0, F1 = c1 > I ? c.rf.tau * c.w1 : 0.0;
    top_update<K, csu.value>(a, x, c.rf, F0, F1, I, g, t);
    if (dot.value) {
      top_dots<K, csd.value>(a, x, I + 1, g, t, sm.prow[(I + 1) & 1], d0, d1);
      put_partials<MW>(sm.red[(I + 1) & 1], d0, d1, g, t, K::FW);
    }
    // v_j^T v_I of the finished columns j < I (both unscaled in registers,
    // row I of v_I is 1) for the T warp.
    if (t == 0) {
      double* v = sm.vtv[I & 1];
      v[c0] = c0 < I ? sc0 * c.w0 : 0.0;
      v[c1] = c1 < I ? sc1 * c.w1 : 0.0;
      if (g == 0) {
        v[16] = c.rf.tau;
        tau[I] = c.rf.tau;
        sm.sc[I] = c.rf.scale;
      }
    }
    if (I == c0) sc0 = c.rf.scale;
    if (I == c1) sc1 = c.rf.scale;
  };
  using Z = std::integral_constant<int, 0>;
  using O = std::integral_constant<int, 1>;
  const int last = w - 1;
#pragma unroll 1
  for (; I < min(last, 7); I++) step(Z{}, Z{}, O{});
  if (I < last) {  // I = 7
    step(Z{}, O{}, O{});
    I++;
#pragma unroll 1
    for (; I < last; I++) step(O{}, O{}, O{});
  }
  if (I < 8) step(Z{}, Z{}, Z{});
  else step(O{}, O{}, Z{});
  bar_col<K::CT>();
}

// The T warp: column I of T one barrier behind the factorization (LAPACK
// dlarft): T(0:I,I) = -tau_I T(0:I,0:I) V(:,0:I)^T v_I.  Lane 4 g + t holds
// rows g and g+8 of columns t, t+4, t+8, t+12.
BSOFI_DEVINL void t_column(double (&T)[2][4], const double* vtv, int I, int g, int t) {
  double r0 = 0.0, r1 = 0.0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const double gb = vtv[t + 4 * q];
    r0 = fma(T[0][q], gb, r0);
    r1 = fma(T[1][q], gb, r1);
  }
  const double tau = vtv[16];
  r0 = quad_sum(r0);
  r1 = quad_sum(r1);
  const double v0 = g == I ? tau : (g < I ? -tau * r0 : 0.0);
  const double v1 = g + 8 == I ? tau : (g + 8 < I ? -tau * r1 : 0.0);
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (I == t + 4 * q) {
      T[0][q] = v0;
      T[1][q] = v1;
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
template <int MW>
BSOFI_DEVINL void reduce_w(double (&acc)[2][4], double (&fr)[2][4], double* part, ChainSmem<MW>& sm,
                           int g, int t, int warp) {
  // (W^T T): T is upper triangular, so columns 0..7 need only rows 0..7.
  double o[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
  dmma_16x8x8(o[0], acc[0][0], acc[0][2], acc[0][1], acc[0][3], sm.T[t][g], sm.T[t + 4][g]);
  dmma_16x8x8(o[1], acc[0][0], acc[0][2], acc[0][1], acc[0][3], sm.T[t][g + 8],
              sm.T[t + 4][g + 8]);
  dmma_16x8x8(o[1], acc[1][0], acc[1][2], acc[1][1], acc[1][3], sm.T[8 + t][g + 8],
              sm.T[12 + t][g + 8]);
  double* mine = part + warp * 256;
  const int c0 = col_of(g);
#pragma unroll
  for (int jt = 0; jt < 2; jt++)
#pragma unroll
    for (int h = 0; h < 2; h++)
      *reinterpret_cast<double2*>(mine + widx(c0 + 8 * h, 8 * jt + 2 * t)) =
          make_double2(o[jt][2 * h], o[jt][2 * h + 1]);
  bar_main<32 * MW>();
#pragma unroll
  for (int e = threadIdx.x; e < 256; e += 32 * MW) {
    double s[MW];
#pragma unroll
    for (int k = 0; k < MW; k++) s[k] = part[k * 256 + e];
#pragma unroll
    for (int m = MW / 2; m > 0; m /= 2)
#pragma unroll
      for (int k = 0; k < m; k++) s[k] += s[k + m];
    sm.W[e] = -s[0];
  }
  bar_main<32 * MW>();
#pragma unroll
  for (int kk = 0; kk < 2; kk++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double2 v =
          *reinterpret_cast<const double2*>(sm.W + widx(c0 + 8 * h, 8 * kk + 2 * t));
      fr[kk][h] = v.x;
      fr[kk][2 + h] = v.y;
    }
}

// C^T += fr V^T for the 8-row block at row r0 of V in shared memory.
BSOFI_DEVINL void update_block(double (&c)[2][2], const double (&fr)[2][4], const double* sV, int SV,
                               int r0, int g, int t) {
  double d[4] = {c[0][0], c[0][1], c[1][0], c[1][1]};
#pragma unroll
  for (int kk = 0; kk < 2; kk++)
    dmma_16x8x8(d, fr[kk][0], fr[kk][1], fr[kk][2], fr[kk][3],
                sV[sidx(r0 + g, 8 * kk + 2 * t, SV)], sV[sidx(r0 + g, 8 * kk + 2 * t + 1, SV)]);
  c[0][0] = d[0];
  c[0][1] = d[1];
  c[1][0] = d[2];
  c[1][1] = d[3];
}

// ------------------------------------------------------------ the chain CTA
// The helper warps: wait for the next tile and stage it while the leaf
// is being factored, build T; store and publish the leaf while the next tile
// is being updated.
template <class K>
BSOFI_DEVINL void chain_helper(const BsofGeom& g, const BsofState& st, const double* sV, double* sC,
                               int SV, ChainSmem<K::MW>& sm) {
  const int ht = threadIdx.x - K::MT, lane = threadIdx.x & 31, hw = ht >> 5;
  const int n = g.n, SC = SV + 16, capc = SC - 2;
  uint32_t phase = 0;
  constexpr int LW = K::HW - 1;  // loading warps; the last one builds T
  if (hw == LW) {
    const int gq = lane >> 2, t = lane & 3;
    for (int s = st.s_begin; s < st.s_end; s++) {
      const Leaf f = sm.step[s & 1].f;
      double T[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
      for (int I = 0; I <= f.w; I++) {
        bar_col<K::CT>();
        if (I > 0) t_column(T, sm.vtv[(I - 1) & 1], I - 1, gq, t);
      }
      double* Tout = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
#pragma unroll
      for (int r = 0; r < 2; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int i = gq + 8 * r, j = t + 4 * q;
          sm.T[i][j] = T[r][q];
          Tout[i + 16 * j] = T[r][q];
        }
      bar_all<K::THREADS>();
      if (!sm.flag) return;
      if (lane == 0 && s + 1 < st.s_end) sm.step[(s + 1) & 1] = chain_step(g, st, s + 1);
      bar_all<K::THREADS>();
    }
    return;
  }
  for (int s = st.s_begin; s < st.s_end; s++) {
    const ChainStep& z = sm.step[s & 1];
    if (ht == 0)
      sm.flag = !z.next || wait_geq(st, st.cnt + tile_id(g, z.m2, z.t2), s - z.lo2) ? 1 : 0;
    {
      bar_help<32 * LW>();
      if (z.next && sm.flag) {
        // Rows [ab, rows) of the tile, then (fresh) the n rows below the panel
        // at shared rows 8 nb, 8 nb + 1, .. (mod capc; the tile's own rows
        // above ab leave room).
        const bool vec = pair_aligned(z.C, z.ldc) && (n & 1) == 0;
        const int f0 = 8 * z.nb, q0 = min(n, capc - f0);
        if (vec && K::BULK) {
          if (ht == 0) {
            fence_proxy();
            tc::mbar_arrive_expect_tx(&sm.bar, 8 * z.w2 * (z.rows - z.ab + (z.fresh ? n : 0)));
            for (int c = 0; c < z.w2; c++) {
              const double* col = z.C + cm(0, c, z.ldc);
              bulk_load(sC + sidx(z.ab, c, SC), col + z.ab, z.rows - z.ab, &sm.bar);
              if (z.fresh) {
                bulk_load(sC + sidx(f0, c, SC), col + 2 * n, q0, &sm.bar);
                if (n > q0) bulk_load(sC + sidx(0, c, SC), col + 2 * n + q0, n - q0, &sm.bar);
              }
            }
          }
        }
        if (!vec) {
          constexpr int NC = 16 / K::LOADS;
#pragma unroll 1
          for (int c = hw; c < z.w2; c += NC * LW) {
            copy_cols<NC, K::LOADS>(sC, SC, z.C, z.ldc, c, LW, z.w2, z.ab, z.rows, lane);
            if (z.fresh) {
              const double* F = z.C + 2 * n;
              copy_cols<NC, K::LOADS>(sC + f0, SC, F, z.ldc, c, LW, z.w2, 0, q0, lane);
              copy_cols<NC, K::LOADS>(sC - q0, SC, F, z.ldc, c, LW, z.w2, q0, n, lane);
            }
          }
        }
#pragma unroll 1
        for (int c = hw; c < 16; c += LW) {
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
        } else if (vec && ht == 0) {
          if (!bulk_wait(&sm.bar, phase, st.err)) sm.flag = 0;
          phase ^= 1;
        }
      }
    }
    bar_all<K::THREADS>();
    if (!sm.flag) return;
    // The reflectors below the pivot rows to global memory.
    if (ht == 0) st.timeline[4 * s + 3] = gtimer();
    if constexpr (K::BULK) {
      const bool vec = pair_aligned(z.P, z.ldp);
      const int r0 = z.ab + 16;
      if (vec && ((z.rows - r0) & 1) == 0) {
        if (ht == 0 && z.rows > r0) {
          for (int c = 0; c < z.f.w; c++)
            bulk_store(z.P + cm(r0, c, z.ldp), sV + sidx(r0, c, SV), z.rows - r0);
          bulk_store_wait();
          fence_proxy();
        }
      } else {
#pragma unroll 1
        for (int c = hw; c < z.f.w; c += LW) {
          double* col = z.P + cm(0, c, z.ldp);
#pragma unroll 4
          for (int r = r0 + lane; r < z.rows; r += 32) __stcg(col + r, sV[sidx(r, c, SV)]);
        }
      }
    }
    if constexpr (K::BULK) bar_help<32 * LW>();
    if (ht == 0) {
      __threadfence();
      red_release_add(st.factored + s, 1);
    }
    bar_all<K::THREADS>();
  }
}

template <class K>
BSOFI_DEVINL void chain_main(const BsofGeom& g, const BsofState& st, double* sV, double* part,
                             double* sC, int SV, ChainSmem<K::MW>& sm) {
  constexpr int FW = K::FW, NI = K::NI, MW = K::MW, MT = K::MT;
  // (The shuffle tells the compiler that the warp index is uniform.)
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int gq = lane >> 2, t = lane & 3, gc = col_of(gq);
  const bool top = warp == FW;
  const int n = g.n, SC = SV + 16, capc = SC - 2;
  // Slot i of this warp is 8-row block bb + i bs of the panel.
  double a[NI][2][2];
#pragma unroll
  for (int i = 0; i < NI; i++) a[i][0][0] = a[i][0][1] = a[i][1][0] = a[i][1][1] = 0.0;
  {
    const Leaf f = leaf_of(g, st.s_begin);
    const int base = leaf_base(g, f), ab8 = (f.j0 - base) / 8, rows = 2 * n - base;
    long long ld;
    const double* P = mat_ptr(g, st, (long long)f.k * n + base, f.m, f.t * 16, ld);
    const bool vec = pair_aligned(P, ld);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int b = top ? ab8 + i : 2 + i * FW + warp;
      if (top ? i >= 2 : b < ab8 + 2) continue;
#pragma unroll
      for (int cs = 0; cs < 2; cs++) {
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
    const int blo = top ? ab8 : ab8 + 2, bhi = top ? min(nb, ab8 + 2) : nb;
    const int bb = top ? ab8 : 2 + warp, bs = top ? 1 : FW;
    {
      // ---- factor the leaf
      if (top) {
        if (lane == 0) {
          st.timeline[4 * s + 0] = gtimer();
          st.timeline[4 * s + 1] = st.timeline[4 * s + 0];
        }
        factor_top<K>(a, sm, w, gq, t, st.tau + (long long)z.f.k * n + z.f.j0);
      } else {
        factor_rows<K>(a, sm, w, ab8, nb, gq, t, warp);
      }
      // ---- V to shared memory, the pivot rows (R and V) to global memory
      // (columns beyond the leaf's width are zero whatever their scale).
      const double sc0 = gc < w ? sm.sc[gc] : 0.0, sc1 = gc + 8 < w ? sm.sc[gc + 8] : 0.0;
      const bool vecp = pair_aligned(z.P, z.ldp);
      if (top) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
#pragma unroll
          for (int cs = 0; cs < 2; cs++) {
            const int c = gc + 8 * cs, r = ab + 8 * i + 2 * t;
            double o[2], v[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const double e = a[i][cs][h];
              const int d = 8 * i + 2 * t + h - c;  // row minus column of the leaf
              o[h] = d > 0 ? e * (cs == 0 ? sc0 : sc1) : e;
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
          for (int cs = 0; cs < 2; cs++) {
            const int c = gc + 8 * cs, r = 8 * b + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; h++) a[i][cs][h] *= cs == 0 ? sc0 : sc1;
            if constexpr (!K::BULK)
              st_pair(z.P + cm(0, c, z.ldp), r, rows, c < w, vecp, a[i][cs][0], a[i][cs][1]);
            *reinterpret_cast<double2*>(sV + sidx(r, c, SV)) =
                make_double2(a[i][cs][0], a[i][cs][1]);
          }
        }
      }
      if constexpr (K::BULK) tc::fence_proxy_async_smem();  // V is stored to global memory by bulk copies
    }
    bar_all<K::THREADS>();
    if (!sm.flag) return;
    if (next) {
      // ---- leaf s on the tile of leaf s+1.  That is the tile's last update
      // and only this CTA reads the tile next, so it stays in registers; its
      // rows above the next leaf are final and go to global memory.
      double c[NI][2][2];
      double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
      const bool vec = pair_aligned(C, ldc);
      constexpr int GS = K::GS;
#pragma unroll
      for (int q = 0; q < K::NG; q++) {
        const int ia = q * GS, ie = (ia + GS < NI ? ia + GS : NI);
        const bool any = bb + (ie - 1) * bs >= blo && bb + ia * bs < bhi;
#pragma unroll
        for (int i = ia; i < ie; i++) c[i][0][0] = c[i][0][1] = c[i][1][0] = c[i][1][1] = 0.0;
        if (!any) continue;
#pragma unroll
        for (int i = ia; i < ie; i++) {
          const int b = bb + i * bs, r = 8 * b + 2 * t;
          const bool live = b >= blo && b < bhi;
#pragma unroll
          for (int cs = 0; cs < 2; cs++) {
            const int cc = gc + 8 * cs;
            double2 v = make_double2(0.0, 0.0);
            if (live) v = *reinterpret_cast<const double2*>(sC + sidx(r, cc, SC));
            c[i][cs][0] = v.x;
            c[i][cs][1] = v.y;
          }
        }
        if constexpr (K::VREG) {
#pragma unroll
          for (int i = ia; i < ie; i++)
#pragma unroll
            for (int jt = 0; jt < 2; jt++)
              dmma_16x8x8(acc[jt], c[i][0][0], c[i][1][0], c[i][0][1], c[i][1][1], a[i][jt][0],
                          a[i][jt][1]);
        }
      }
      if constexpr (!K::VREG) {
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs, r = 8 * b + 2 * t;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int jt = 0; jt < 2; jt++) {
            const double2 v = *reinterpret_cast<const double2*>(sV + sidx(r, gc + 8 * jt, SV));
            dmma_16x8x8(acc[jt], c[i][0][0], c[i][1][0], c[i][0][1], c[i][1][1], v.x, v.y);
          }
        }
      }
      double fr[2][4];
      reduce_w<MW>(acc, fr, part, sm, gq, t, warp);
      const bool keep_all = s + 1 == st.s_end;
#pragma unroll
      for (int q = 0; q < K::NG; q++) {
        const int ia = q * GS, ie = (ia + GS < NI ? ia + GS : NI);
        if (bb + (ie - 1) * bs < blo || bb + ia * bs >= bhi) continue;
        // (Slots of the group that are not live compute values nobody uses.)
#pragma unroll
        for (int i = ia; i < ie; i++)
          update_block(c[i], fr, sV, SV, 8 * min(bb + i * bs, nb - 1), gq, t);
      }
      if (top || keep_all) {
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs, r = 8 * b + 2 * t;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int cs = 0; cs < 2; cs++)
            st_pair(C + cm(0, gc + 8 * cs, ldc), r, rows, gc + 8 * cs < w2, vec, c[i][cs][0],
                    c[i][cs][1]);
        }
      }
      if (!trans) {
        // Blocks ab8 + 2 and ab8 + 3 become the next leaf's pivot rows.
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int d = bb + i * bs - (ab8 + 2);
          const bool live = !top && d >= 0 && bb + i * bs < bhi;
#pragma unroll
          for (int cs = 0; cs < 2; cs++) {
            if (live && d < 2)
              *reinterpret_cast<double2*>(sm.top + (gc + 8 * cs) * 16 + 8 * d + 2 * t) =
                  make_double2(c[i][cs][0], c[i][cs][1]);
#pragma unroll
            for (int h = 0; h < 2; h++) a[i][cs][h] = live && d >= 2 ? c[i][cs][h] : 0.0;
          }
        }
      } else {
        // Through shared memory, over the tile just read.
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = bb + i * bs;
          if (b < blo || b >= bhi) continue;
#pragma unroll
          for (int cs = 0; cs < 2; cs++)
            *reinterpret_cast<double2*>(sC + sidx(8 * b + 2 * t, gc + 8 * cs, SC)) =
                make_double2(c[i][cs][0], c[i][cs][1]);
        }
        bar_main<MT>();
        const int rows2 = fresh ? 2 * n : n;
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int b = top ? i : 2 + i * FW + warp;
#pragma unroll
          for (int cs = 0; cs < 2; cs++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int r = 8 * b + 2 * t + h, cc = gc + 8 * cs;
              double v = 0.0;
              if ((!top || i < 2) && r < rows2 && cc < w2) {
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
    bar_all<K::THREADS>();
    if (top) {
      if (next && !trans) {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int cs = 0; cs < 2; cs++) {
            double2 v = make_double2(0.0, 0.0);
            if (ab8 + 2 + i < nb)
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
  constexpr int MW = K::MW, MT = K::MT, NIW = K::NIW;
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
    const double* P = mat_ptr(g, st, (long long)f.k * g.n + f.j0, f.m, f.t * 16, ldp);
    double* C = tile_ptr(g, st, f.k, f.j0, m2, t2, ldc);
    const int w2 = min(16, g.n - t2 * 16);
    // The tile is loaded while the leaf is still being factored.
    if (tid == 0) sm.flag = wait_geq(st, st.cnt + x2, s - lo2) ? 1 : 0;
    bar_main<MT>();
    if (!sm.flag) return;
    double c[NIW][2][2];
    const bool vecc = pair_aligned(C, ldc);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
#pragma unroll
      for (int cs = 0; cs < 2; cs++) {
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
      if (K::BULK && vec && tid == 0 && rows > 16) {
        fence_proxy();
        tc::mbar_arrive_expect_tx(&sm.bar, 8 * f.w * (rows - 16));
        for (int cc = 0; cc < f.w; cc++)
          bulk_load(sV + sidx(16, cc, SV), P + cm(16, cc, ldp), rows - 16, &sm.bar);
      }
      if (!vec) {
#pragma unroll
        for (int cc = warp; cc < 16; cc += 2 * MW)
          copy_cols<2, K::LOADS>(sV, SV, P, ldp, cc, MW, f.w, 16, rows, lane);
      }
      for (int cc = warp; cc < 16; cc += MW) {
        const double* col = P + cm(0, cc, ldp);
        if (cc >= f.w) {
          for (int r = 16 + lane; r < 8 * nb; r += 32) sV[sidx(r, cc, SV)] = 0.0;
        } else if (vec) {
          if (!K::BULK) {
#pragma unroll 1
            for (int r = 16 + 2 * lane; r < rows; r += 64)
              cp_async16(sV + sidx(r, cc, SV), col + r, 16);
          }
          if (lane < 8 && max(rows, 16) + lane < 8 * nb) sV[sidx(max(rows, 16) + lane, cc, SV)] = 0.0;
        } else if (lane < 8 && max(rows, 16) + lane < 8 * nb) {
          sV[sidx(max(rows, 16) + lane, cc, SV)] = 0.0;
        }
      }
      const double* T = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
      for (int e = tid; e < 256; e += MT) {
        const int r = e & 15, cc = e >> 4;
        double v = 0.0;
        if (cc < f.w && r < rows) v = r == cc ? 1.0 : (r > cc ? __ldcg(P + cm(r, cc, ldp)) : 0.0);
        sV[sidx(r, cc, SV)] = v;
        sm.T[r][cc] = __ldcg(T + e);
      }
      if (!K::BULK) {
        cp_async_wait<0>();
      } else if (vec && rows > 16) {
        if (tid == 0 && !bulk_wait(&sm.bar, phase, st.err)) sm.flag = 0;
        phase ^= 1;
      }
    }
    bar_main<MT>();
    if (!sm.flag) return;
    double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (b < nb) {
#pragma unroll
        for (int jt = 0; jt < 2; jt++) {
          const double2 v =
              *reinterpret_cast<const double2*>(sV + sidx(8 * b + 2 * t, gc + 8 * jt, SV));
          dmma_16x8x8(acc[jt], c[i][0][0], c[i][1][0], c[i][0][1], c[i][1][1], v.x, v.y);
        }
      }
    }
    double fr[2][4];
    reduce_w<MW>(acc, fr, part, sm, gq, t, warp);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (b < nb) {
        update_block(c[i], fr, sV, SV, 8 * b, gq, t);
#pragma unroll
        for (int cs = 0; cs < 2; cs++)
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

template <class K>
__global__ void __launch_bounds__(K::THREADS, 1) bsof_persistent_kernel(BsofGeom g, BsofState st) {
  extern __shared__ __align__(16) double dyn_bsof[];
  __shared__ __align__(16) ChainSmem<K::MW> sm;
  const int SV = tile_stride(g.n);
  double* sV = dyn_bsof;
  double* part = sV + 16 * SV;
  double* sC = part + K::MW * 256;
  if (threadIdx.x == 0) {
    tc::mbar_init(&sm.bar, 1);
    tc::fence_barrier_init();
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) sm.step[st.s_begin & 1] = chain_step(g, st, st.s_begin);
      }
  __syncthreads();
  if (threadIdx.x >= K::MT) {
    if constexpr (K::REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (blockIdx.x == 0) chain_helper<K>(g, st, sV, sC, SV, sm);
  } else {
    if constexpr (K::REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    if (blockIdx.x == 0) chain_main<K>(g, st, sV, part, sC, SV, sm);
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
    reduce_w<MW>(acc, fr, part, sm, gq, t, warp);
#pragma unroll
    for (int i = 0; i < NIW; i++) {
      const int b = warp + i * MW;
      if (8 * b + 7 >= j0 && b < nb) update_block(c[i], fr, sV, SV, 8 * b, gq, t);
    }
    bar_main<MT>();  // V, T and W are no longer read
  }
  double* C = s.G + (long long)k * n2 * n2 + cm(0, x0, n2);
#pragma unroll
  for (int i = 0; i < NIW; i++) {
    const int b = warp + i * MW;
#pragma unroll
    for (int cs = 0; cs < 2; cs++)
      st_pair(C + cm(0, gc + 8 * cs, n2), 8 * b + 2 * t, n2, b < nb && x0 + gc + 8 * cs < n2, true,
              c[i][cs][0], c[i][cs][1]);
  }
}

// ------------------------------------------------------------------ launcher
using Chain64 = ChainCfg<3, 5, 4>;
using Chain128 = ChainCfg<7, 5, 4>;
using Chain256 = ChainCfg<7, 9, 8>;
using Chain400 = ChainCfg<7, 14, 13>;
using Chain640 = ChainCfg<7, 23, 20>;  // (its worker shape only: form_q_kernel)

// 16-wide leaves up to n = 400, where the next tile still fits in shared
// memory beside V; the tall kernel's 8-wide ones above.
int bsof_leaf_width(int n) { return n <= Chain400::MAX_ROWS / 2 ? 16 : 8; }

int bsof_tiles(int n) { return (n + bsof_leaf_width(n) - 1) / bsof_leaf_width(n); }

template <class K>
static size_t dyn_smem(int n) {
  const size_t SV = tile_stride(n);
  return sizeof(double) * (16 * SV + 256 * K::MW + 16 * (SV + 16));
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
  if (2 * n <= Chain400::MAX_ROWS) return launch_cfg<Chain400>(g, s, workers, st);
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

bool form_q_fits(int n) { return 2 * n <= Chain640::MAX_ROWS; }

cudaError_t launch_form_q(const double* A, long long ld, int n, int L, const double* T,
                          int maxleaves, int nbw, double* G, cudaStream_t st) {
  const FormQArgs a = {A, ld, n, L, T, maxleaves, nbw, G};
  if (2 * n <= Chain64::MAX_ROWS) return launch_form_q_cfg<Chain64, 4>(a, st);
  if (2 * n <= Chain128::MAX_ROWS) return launch_form_q_cfg<Chain128, 2>(a, st);
  if (2 * n <= Chain256::MAX_ROWS) return launch_form_q_cfg<Chain256, 2>(a, st);
  if (2 * n <= Chain400::MAX_ROWS) return launch_form_q_cfg<Chain400, 1>(a, st);
  if (2 * n <= Chain640::MAX_ROWS) return launch_form_q_cfg<Chain640, 1>(a, st);
  return cudaErrorInvalidValue;
}

cudaError_t preload_bsof(size_t* local) {
  cudaError_t e;
  if ((e = preload_one(bsof_persistent_kernel<Chain64>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain128>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain256>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bsof_persistent_kernel<Chain400>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain64, 4>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain128, 2>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain256, 2>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain400, 1>, local)) != cudaSuccess) return e;
  if ((e = preload_one(form_q_kernel<Chain640, 1>, local)) != cudaSuccess) return e;
  return preload_bsof_tall(local);
}

}  // namespace bsofi
