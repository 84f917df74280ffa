// BSOF for the tallest panels (n = 641..768): the schedule of kernels_bsof.cu
// with 8-wide leaves and one task per leaf and tile, 1536 rows in the registers
// of one CTA (six rows of eight columns a thread).  The layout of kernels_bsof.cu
// needs the pivot column beside the leaf in registers, which ends at n = 640.
#include <climits>
#include "bsof_sched.cuh"
#include "bsofi_kernels.h"

namespace bsofi {
namespace {

constexpr int BT = 256;  // threads per CTA
constexpr int BW = BT / 32;
constexpr int NB = 8;   // leaf width
constexpr int ROWS_PER = 6;  // rows a thread

// Sum NB values per lane over a warp (transpose reduction): lane l ends with
// the warp sum of value (l >> 2) & 7.
BSOFI_DEVINL double wsum_t(double (&v)[NB], int lane) {
  constexpr int LOG = 3;
#pragma unroll
  for (int lev = 0; lev < LOG; lev++) {
    const int off = 16 >> lev, half = NB >> (lev + 1);
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < half; j++) {
      double send = up ? v[j] : v[j + half];
      double keep = up ? v[j + half] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  double s = v[0];
#pragma unroll
  for (int off = 16 >> LOG; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

struct Smem {
  double red[2][BW][NB];
  double coef[2][NB + 4];   // tau*w_c (c < NB), tau, scale, beta
  double prow[2][NB];
  double gsh[2][NB];
  double T[NB][NB + 1];
  double redW[BW][NB][NB + 1];
  double W[NB][NB + 1];
  int flag;
  int task;
};

// T(0:I, I) = -tau_I T(0:I,0:I) g_I (LAPACK dlarft), run by one warp one
// column behind the factorization; T and g are zero outside their ranges.
BSOFI_DEVINL void t_column(Smem& sm, int I, int lane) {
  const int buf = I & 1;
  const double taui = sm.coef[buf][NB];
  if (lane < I) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int b = 0; b < NB; b += 2) {
      s0 = fma(sm.T[lane][b], sm.gsh[buf][b], s0);
      s1 = fma(sm.T[lane][b + 1], sm.gsh[buf][b + 1], s1);
    }
    sm.T[lane][I] = -taui * (s0 + s1);
  }
  if (lane == I) sm.T[I][I] = taui;
  __syncwarp();
}

// Householder QR of one leaf held in registers (thread t owns rows t + BT*i).
// The column loop is a runtime loop over a rotating layout: at step I
// position 0 holds column I, positions 1..NB-1-I the columns not yet
// factored, and positions NB-I..NB-1 the finished reflectors 0..I-1; the
// array rotates left by one position after each step, so every register index
// is a compile-time constant while the loop body exists once (a fully
// unrolled column loop overflows the instruction cache).
//
// One block reduction per column carries, per position, either the dot
// product d_c = sum_{r>I} a_rI a_rc with a pending column (position 0 gives
// ||x||^2) or e_j = sum_{r>I} v_j[r] a_rI with a finished reflector, which
// builds the dlarft factor T(0:I,I) = -tau_I T(0:I,0:I) V^T v_I.
template <int TR>
BSOFI_DEVINL void factor_leaf(double (&a)[TR][NB], Smem& sm, int m, int w, double* tau_out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int SH = 2;
#pragma unroll 1
  for (int I = 0; I < w; I++) {
    const int buf = I & 1;
    const int ndone0 = NB - I;  // first position holding a finished reflector
    if (tid == I) {
#pragma unroll
      for (int p = 0; p < NB; p++) sm.prow[buf][p] = a[0][p];
    }
    double part[NB];
#pragma unroll
    for (int p = 0; p < NB; p++) part[p] = 0.0;
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const int r = tid + BT * i;
      const double x = (r > I) ? a[i][0] : 0.0;  // rows >= m hold zeros
#pragma unroll
      for (int p = 0; p < NB; p++) part[p] = fma(x, a[i][p], part[p]);
    }
    {
      double sum = wsum_t(part, lane);
      if ((lane & ((1 << SH) - 1)) == 0) sm.red[buf][warp][(lane >> SH) & (NB - 1)] = sum;
    }
    __syncthreads();
    if (warp == 0) {
      const int slot = lane % NB;
      double tot = 0.0;
#pragma unroll
      for (int k = lane / NB; k < BW; k += 32 / NB) tot += sm.red[buf][k][slot];
#pragma unroll
      for (int off = NB; off < 32; off <<= 1) tot += __shfl_xor_sync(0xffffffffu, tot, off);
      const double xnorm2 = __shfl_sync(0xffffffffu, tot, 0);
      const double alpha = sm.prow[buf][0];
      double beta, taui, scale;
      if (xnorm2 == 0.0) {
        taui = 0.0;
        beta = alpha;
        scale = 1.0;
      } else {
        // beta = -sign(alpha) ||(alpha, x)||, tau = (beta - alpha)/beta = 1 + |alpha|/||.||,
        // scale = 1/(alpha - beta): one reciprocal square root and one division.
        const double s2 = fma(alpha, alpha, xnorm2);
        const double rn = rsqrt(s2);
        beta = -copysign(s2 * rn, alpha);
        taui = fma(fabs(alpha), rn, 1.0);
        scale = 1.0 / (alpha - beta);
      }
      const double val = fma(scale, tot, sm.prow[buf][slot]);
      if (lane < NB) {
        // tau*w_c at pending positions 1..NB-1-I, zero elsewhere, so the row
        // update below needs no predicates.
        sm.coef[buf][slot] = (slot >= 1 && slot < ndone0) ? taui * val : 0.0;
        // g_j = v_j^T v_I for j < I, zero for j >= I.
        // lane slot writes g at index (slot - ndone0) mod NB: indices < I get
        // the reflector dot products, the others zero.
        const int j = (slot + I) & (NB - 1);
        sm.gsh[buf][j] = (slot >= ndone0) ? val : 0.0;
      }
      if (lane == 0) {
        sm.coef[buf][NB] = taui;
        sm.coef[buf][NB + 1] = scale;
        sm.coef[buf][NB + 2] = beta;
        tau_out[I] = taui;
      }
    }
    if (warp == 1 && I > 0) t_column(sm, I - 1, lane);
    __syncthreads();
    const double scale = sm.coef[buf][NB + 1],
                 beta = sm.coef[buf][NB + 2];
    double cf[NB];
#pragma unroll
    for (int p = 1; p < NB; p++) cf[p] = sm.coef[buf][p];
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const int r = tid + BT * i;
      const double sv = a[i][0] * scale;
      const double v = (r > I) ? sv : ((r == I) ? 1.0 : 0.0);
      a[i][0] = (r > I) ? sv : ((r == I) ? beta : a[i][0]);
#pragma unroll
      for (int p = 1; p < NB; p++) a[i][p] = fma(-v, cf[p], a[i][p]);
    }
    // Rotate left: the finished column moves to the last position.
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const double t0 = a[i][0];
#pragma unroll
      for (int p = 0; p < NB - 1; p++) a[i][p] = a[i][p + 1];
      a[i][NB - 1] = t0;
    }
  }
  __syncthreads();
  if (warp == 1) t_column(sm, w - 1, lane);
  __syncthreads();
  // A leaf narrower than NB needs NB - w more rotations to restore column order.
#pragma unroll 1
  for (int k = w; k < NB; k++) {
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const double t0 = a[i][0];
#pragma unroll
      for (int p = 0; p < NB - 1; p++) a[i][p] = a[i][p + 1];
      a[i][NB - 1] = t0;
    }
  }
}

// 8-wide block reflector with DMMA m8n8k4 (f64), all rows in one pass:
//   W = V^T C (8 x 8; K = the leaf's rows, split over the 8 warps),
//   W <- -T^T W,  C <- C + V W  (rows split over the warps).
// V and C are staged column-major with column stride S8 = TR*BT + 4 (4 mod 16
// doubles): the staging writes (one row per thread) and the fragment loads of
// both products are free of bank conflicts.  VREG: V comes from the factoring
// CTA's registers (thread t owns rows t + BT*i), else from the stored leaf.
// wv: width of the leaf, w: width of the target tile.
template <int TR>
struct Stage8 {
  static constexpr int S8 = TR * BT + 4;
};

template <int TR, bool VREG>
BSOFI_DEVINL void apply_qt_mma8(double* sV, double* sC, const double (&a)[TR][8],
                                const double* P, long long ldp, int wv, double* C, long long ld,
                                int m, int w, Smem& sm) {
  constexpr int S8 = Stage8<TR>::S8, KW = TR * BT / BW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < TR; i++) {
    const int r = tid + BT * i;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      double v = 0.0;
      if (r < m && c < wv) {
        if (r == c) v = 1.0;
        else if (r > c) v = VREG ? a[i][c] : __ldcg(P + cm(r, c, ldp));
      }
      sV[c * S8 + r] = v;
      sC[c * S8 + r] = (r < m && c < w) ? __ldcg(C + cm(r, c, ld)) : 0.0;
    }
  }
  __syncthreads();
  {
    // Four independent accumulators over interleaved 4-deep K steps, so the
    // DMMAs of a warp do not wait on each other's results.
    static_assert(KW % 16 == 0, "8-wide W split");
    double acc[4][2] = {};
    const int k1 = warp * KW;
#pragma unroll
    for (int k0 = k1; k0 < k1 + KW; k0 += 16)
#pragma unroll
      for (int q = 0; q < 4; q++)
        dmma_8x8x4(acc[q], sV[g * S8 + k0 + 4 * q + t], sC[g * S8 + k0 + 4 * q + t]);
    sm.redW[warp][g][2 * t] = (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
    sm.redW[warp][g][2 * t + 1] = (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]);
  }
  __syncthreads();
  if (tid < 64) {
    const int ai = tid & 7, cc = tid >> 3;
    double s2 = 0.0;
#pragma unroll
    for (int k = 0; k < BW; k++) s2 += sm.redW[k][ai][cc];
    sm.W[ai][cc] = s2;
  }
  __syncthreads();
  if (tid < 64) {  // -(T^T W); T is zero below its diagonal
    const int ai = tid & 7, cc = tid >> 3;
    double s2 = 0.0;
#pragma unroll
    for (int b = 0; b < 8; b++) s2 = fma(sm.T[b][ai], sm.W[b][cc], s2);
    sm.redW[0][ai][cc] = -s2;
  }
  __syncthreads();
#pragma unroll 4
  for (int m0 = warp * KW; m0 < (warp + 1) * KW; m0 += 8) {
    double d[2] = {sC[(2 * t) * S8 + m0 + g], sC[(2 * t + 1) * S8 + m0 + g]};
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += 4)
      dmma_8x8x4(d, sV[(k0 + t) * S8 + m0 + g], sm.redW[0][k0 + t][g]);
    const int rr = m0 + g;
    if (rr < m) {
      if (2 * t < w) __stcg(C + cm(rr, 2 * t, ld), d[0]);
      if (2 * t + 1 < w) __stcg(C + cm(rr, 2 * t + 1, ld), d[1]);
    }
  }
  __syncthreads();
}

template <int TR>
__global__ void __launch_bounds__(BT, 1) bsof_tall_kernel(BsofGeom g, BsofState st) {
  constexpr int S8 = Stage8<TR>::S8;
  __shared__ Smem sm;
  extern __shared__ __align__(16) double sC[];  // V and C tiles, 8 columns of S8 each
  const int tid = threadIdx.x;
  const long long first_task = tasks_before(g, st.s_begin);
  const long long total_tasks = tasks_before(g, st.s_end);

  if (blockIdx.x == 0) {
    // ---------------------------------------------------------- panel chain
    // The first leaf's tile has no update to wait for, and this CTA makes the last
    // one of every other leaf's (shared barriers order its own global writes).
    for (int s = st.s_begin; s < st.s_end; s++) {
      const Leaf f = leaf_of(g, s);
      if (tid == 0) st.timeline[4 * s + 0] = gtimer();
      const int mrows = 2 * g.n - f.j0;
      long long ldp;
      double* P = mat_ptr(g, st, (long long)f.k * g.n + f.j0, f.m, f.t * g.NB, ldp);
      // Target 0 of leaf s: the tile of leaf s+1.
      const bool next = ntargets(g, f) > 0;
      int m2 = 0, t2 = 0, lo2 = 0, hi2 = 0;
      if (next) {
        target_of(g, f, 0, m2, t2);
        tile_range(g, m2, t2, lo2, hi2);
      }
      const int x2 = tile_id(g, m2, t2);
      long long ldc = st.ld;
      double* C = next ? tile_ptr(g, st, f.k, f.j0, m2, t2, ldc) : nullptr;
      const int w2 = min(g.NB, g.n - t2 * g.NB);
      for (int e = tid; e < NB * (NB + 1); e += BT) (&sm.T[0][0])[e] = 0.0;
      if (tid < 2 * NB) (&sm.gsh[0][0])[tid] = 0.0;
      __syncthreads();
      double a[TR][NB];
#pragma unroll
      for (int i = 0; i < TR; i++) {
        const int r = tid + BT * i;
#pragma unroll
        for (int c = 0; c < NB; c++)
          a[i][c] = (r < mrows && c < f.w) ? __ldcg(P + cm(r, c, ldp)) : 0.0;
      }
      factor_leaf<TR>(a, sm, mrows, f.w, st.tau + (long long)f.k * g.n + f.j0);
#pragma unroll
      for (int i = 0; i < TR; i++) {
        const int r = tid + BT * i;
        if (r < mrows) {
#pragma unroll
          for (int c = 0; c < NB; c++)
            if (c < f.w) __stcg(P + cm(r, c, ldp), a[i][c]);
        }
      }
      double* Tout = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
      for (int e = tid; e < 256; e += BT) {
        const int rr = e % 16, cc = e / 16;
        Tout[e] = (rr < f.w && cc < f.w) ? sm.T[rr][cc] : 0.0;
      }
      __syncthreads();
      if (tid == 0) st.timeline[4 * s + 1] = gtimer();
      // Apply leaf s to the tile of leaf s+1.  That is the tile's last update
      // and only this CTA reads the tile next, so it is not published; the
      // leaf itself (reflectors and T) is published after the update, with one
      // fence for both.
      if (next) {
        if (!block_wait_geq(st, st.cnt + x2, s - lo2, &sm.flag)) return;
        if (tid == 0) st.timeline[4 * s + 3] = gtimer();
        apply_qt_mma8<TR, true>(sC, sC + 8 * S8, a, P, ldp, f.w, C, ldc, mrows, w2, sm);
      }
      if (tid == 0) {
        __threadfence();
        red_release_add(st.factored + s, 1);
        st.timeline[4 * s + 2] = gtimer();
      }
    }
    return;
  }

  // ------------------------------------------------------------ workers
  for (;;) {
    if (tid == 0) sm.task = first_task + atomicAdd(st.next_task, 1);
    __syncthreads();
    const long long task = sm.task;
    __syncthreads();
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
    int m2, t2;
    target_of(g, f, q, m2, t2);
    int lo2, hi2;
    tile_range(g, m2, t2, lo2, hi2);
    const int x2 = tile_id(g, m2, t2);
    if (!block_wait_geq(st, st.factored + s, 1, &sm.flag)) return;
    const int mrows = 2 * g.n - f.j0;
    const double* T = st.T + ((long long)f.k * st.maxleaves + f.l) * 256;
    for (int e = tid; e < NB * NB; e += BT) sm.T[e % NB][e / NB] = __ldcg(T + (e % NB) + 16 * (e / NB));
    long long ldp, ldc;
    const double* P = mat_ptr(g, st, (long long)f.k * g.n + f.j0, f.m, f.t * g.NB, ldp);
    double* C = tile_ptr(g, st, f.k, f.j0, m2, t2, ldc);
    const int w2 = min(g.NB, g.n - t2 * g.NB);
    if (!block_wait_geq(st, st.cnt + x2, s - lo2, &sm.flag)) return;
    double none[TR][8];
    apply_qt_mma8<TR, false>(sC, sC + 8 * S8, none, P, ldp, f.w, C, ldc, mrows, w2, sm);
    if (tid == 0) {
      __threadfence();
      red_release_add(st.cnt + x2, 1);
    }
  }
}

template <int TR>
cudaError_t launch_tr(const BsofGeom& g, const BsofState& st, int workers, cudaStream_t s) {
  constexpr size_t smem = sizeof(double) * 2 * 8 * (size_t)Stage8<TR>::S8;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(bsof_tall_kernel<TR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&g, (void*)&st};
  return cudaLaunchCooperativeKernel((const void*)bsof_tall_kernel<TR>,
                                     dim3(min(1 + workers, sms)), dim3(BT), args, smem, s);
}
}  // namespace

cudaError_t launch_bsof_tall(const BsofGeom& g, const BsofState& st, int workers, cudaStream_t s) {
  if (2 * g.n <= ROWS_PER * BT) return launch_tr<ROWS_PER>(g, st, workers, s);
  return cudaErrorInvalidValue;
}

cudaError_t preload_bsof_tall(size_t* local) {
  return preload_one(bsof_tall_kernel<ROWS_PER>, local);
}

}  // namespace bsofi
