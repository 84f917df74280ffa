// BSTRI's row recurrence of small blocks: one CTA per band of columns.
//
// Reference: lapackXbstri, src/bsofi_cpu.c:159-172.  With the diagonal blocks
// inverted and W_i = -X_ii R_{i,i+1}, Z_i = -X_ii R_{i,L-1} X_{L-1,L-1} formed
// (Z in block column L-1), X_{i,c} = W_i X_{i+1,c} (+ Z_i for c = L-1), read by
// columns: a column of X depends on no other.  So a CTA that owns a band of
// columns of block column c runs its steps from the diagonal block up, the
// block it just made staying in shared memory as the next step's right
// operand, and the W_i streaming in from L2.
//
// What bounds it: the latency of a step (n x n x band on one SM) times the
// L - 2 steps of the longest columns; the row recurrence in launches or tiles
// waits L - 2 times for a launch or a dependent tile of a larger product.
// Bands of 8 columns have the shortest step; bands of 16 halve the W_i traffic
// where there are enough columns to fill the GPU (N > 2048).  Measured (the
// recurrence alone, us; before: blocked row recurrence, in-group products
// included): n = 16, p = 8 30 -> 5; n = 64, p = 16 126 -> 24; n = 100, p = 64
// 900 -> 517.
#include "bsofi_common.cuh"
#include "bsofi_kernels.h"

namespace bsofi {

namespace {

constexpr int kThreads = 128, kWarps = 4;
// A chunk of W_i is consumed in a few hundred cycles, so several must be on
// their way (3 stages: 280 us at n = 100, p = 32).
constexpr int KC = 16, STAGES = 6;

struct RecBandArgs {
  double* A;
  long long ld;
  const double* W;  // (L-2) x n^2
  int n, L, bands;  // bands of one block column
  bool vec;         // W: 16-byte aligned and n even
};

// Row stride of a stage of W_i (columns of rows) and of the right operand for
// blocks of at most 64 mtw: 4 mod 16 doubles (free of bank conflicts), and a
// constant, so that every shared address is one register and an immediate (the
// kernel is bound by instruction issue where a step's products are short).
__host__ __device__ constexpr int rec_stride(int mtw) { return 64 * mtw + 4; }
__host__ __device__ constexpr int rec_smem_doubles(int mtw, int C) { return (STAGES * KC + C) * rec_stride(mtw); }

// Columns [k0, k0 + KC) of the n x n matrix M into one stage [k][row]; columns
// beyond n are zero.  Warp w loads columns w, w + 4, ..
template <int MTW>
BSOFI_DEVINL void load_m(double* dst, const double* M, int n, int k0, bool vec, int lane,
                         int warp) {
  constexpr int S = rec_stride(MTW);
  const double* src = M + (long long)(k0 + warp) * n;
  dst += warp * S;
  if (vec) {
    const bool in0 = 2 * lane < n, in1 = MTW > 1 && 64 + 2 * lane < n;
    src += 2 * lane;
    dst += 2 * lane;
#pragma unroll
    for (int kk = 0; kk < KC; kk += kWarps) {
      const int bytes = k0 + warp + kk < n ? 16 : 0;
      const double* p = bytes ? src + (long long)kk * n : M;
      if (in0) cp_async16(dst + kk * S, p, bytes);
      if (in1) cp_async16(dst + kk * S + 64, bytes ? p + 64 : M, bytes);
    }
  } else {
#pragma unroll
    for (int kk = 0; kk < KC; kk += kWarps) {
      const int bytes = k0 + warp + kk < n ? 8 : 0;
#pragma unroll
      for (int r = 0; r < 64 * MTW; r += 32)
        if (r + lane < n)
          cp_async8(dst + kk * S + r + lane, bytes ? src + (long long)kk * n + r + lane : M, bytes);
    }
  }
}

// C columns per band; MTW: 16-row tiles of the block per warp (tile w + 4 i).
template <int C, int MTW>
__global__ void __launch_bounds__(kThreads) bstri_band_kernel(RecBandArgs s) {
  extern __shared__ __align__(16) double smem_rec[];
  constexpr int S = rec_stride(MTW);
  const int n = s.n, L = s.L, tiles = (n + 15) / 16, nc = (n + KC - 1) / KC;
  // The longest chains first.
  const int cb = L - 1 - blockIdx.x / s.bands, j0 = (blockIdx.x % s.bands) * C;
  const int w = min(C, n - j0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  double* sM = smem_rec;                 // [STAGES][KC][S]
  double* sCur = sM + STAGES * KC * S;   // [C][S]: X_{i+1}, columns of the band
  const bool last = cb == L - 1;
  // First right operand: the diagonal block's columns (upper triangle), in the
  // last block column Z_{L-2} = X_{L-2,L-1}.  Rows beyond n of the stages and
  // of the operand stay zero.
  const int first = last ? L - 2 : cb;
  for (int e = threadIdx.x; e < rec_smem_doubles(MTW, C); e += kThreads) smem_rec[e] = 0.0;
  __syncthreads();
  {
    const double* D = s.A + cm((long long)first * n, (long long)cb * n + j0, s.ld);
    for (int e = threadIdx.x; e < w * n; e += kThreads) {
      const int c = e / n, r = e % n;
      if (last || r <= j0 + c) sCur[c * S + r] = D[cm(r, c, s.ld)];
    }
  }
  int pi = first - 1, pc = 0, slot_in = 0;  // next chunk to load
  auto issue = [&]() {
    if (pi >= 0) {
      load_m<MTW>(sM + slot_in * KC * S, s.W + (long long)pi * n * n, n, pc * KC, s.vec, lane, warp);
      if (++pc == nc) {
        pc = 0;
        pi--;
      }
    }
    cp_async_commit();
    slot_in = slot_in + 1 == STAGES ? 0 : slot_in + 1;
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; i++) issue();
  constexpr int NT = C / 8;
  int slot = 0;
#pragma unroll 1
  for (int i = first - 1; i >= 0; i--) {
    double* out = s.A + cm((long long)i * n, (long long)cb * n + j0, s.ld);
    // (acc2: the odd 8-deep products of a single tile, a second chain.)
    double acc[MTW][NT][4], acc2[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < MTW; a++) {
      const int mt = warp + kWarps * a;
#pragma unroll
      for (int b = 0; b < NT; b++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const int r = mt * 16 + 8 * h + g, c = b * 8 + 2 * t + q;
            acc[a][b][2 * h + q] = last && r < n && c < w ? out[cm(r, c, s.ld)] : 0.0;
          }
    }
#pragma unroll 1
    for (int c = 0; c < nc; c++) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      issue();
      const double* tM = sM + slot * KC * S + g;
      const double* op = sCur + c * KC + t;
      auto product = [&](int k8) {
        double bf[NT][2];
#pragma unroll
        for (int b = 0; b < NT; b++) {
          bf[b][0] = op[(b * 8 + g) * S + k8 * 8];
          bf[b][1] = op[(b * 8 + g) * S + k8 * 8 + 4];
        }
#pragma unroll
        for (int a = 0; a < MTW; a++) {
          const int mt = warp + kWarps * a;
          const double* q0 = tM + (k8 * 8 + t) * S + mt * 16;
          const double* q1 = q0 + 4 * S;
          const double a0 = q0[0], a1 = q0[8], a2 = q1[0], a3 = q1[8];
          if (mt < tiles) {
#pragma unroll
            for (int b = 0; b < NT; b++)
              dmma_16x8x8(MTW * NT == 1 && (k8 & 1) ? acc2 : acc[a][b], a0, a1, a2, a3, bf[b][0],
                          bf[b][1]);
          }
        }
      };
      if (c * KC + KC - 8 < n) {
#pragma unroll
        for (int k8 = 0; k8 < KC / 8; k8++) product(k8);
      } else {
        product(0);
      }
      slot = slot + 1 == STAGES ? 0 : slot + 1;
    }
    if (MTW * NT == 1) {
#pragma unroll
      for (int q = 0; q < 4; q++) acc[0][0][q] += acc2[q];
    }
    __syncthreads();  // sCur is no longer read
#pragma unroll
    for (int a = 0; a < MTW; a++) {
      const int mt = warp + kWarps * a;
#pragma unroll
      for (int b = 0; b < NT; b++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const int r = mt * 16 + 8 * h + g, c = b * 8 + 2 * t + q;
            if (r < n && c < w) {
              sCur[c * S + r] = acc[a][b][2 * h + q];
              out[cm(r, c, s.ld)] = acc[a][b][2 * h + q];
            }
          }
    }
    // (The next chunk's barrier comes before sCur is read.)
  }
  cp_async_wait<0>();
}

template <int C, int MTW>
cudaError_t launch_c(const RecBandArgs& a, cudaStream_t st) {
  static PerDevice once;
  const int dev = once.pending();
  if (dev >= 0) {
    cudaError_t e = cudaFuncSetAttribute(bstri_band_kernel<C, MTW>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(rec_smem_doubles(MTW, C) * sizeof(double)));
    if (e != cudaSuccess) return e;
    once.mark(dev);
  }
  bstri_band_kernel<C, MTW><<<(a.L - 1) * a.bands, kThreads,
                              rec_smem_doubles(MTW, C) * sizeof(double), st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_bstri_band(double* A, long long ld, const double* W, int n, int L,
                              cudaStream_t st) {
  if (n > 128) return cudaErrorInvalidValue;
  if (L < 3) return cudaSuccess;
  RecBandArgs a;
  a.A = A;
  a.ld = ld;
  a.W = W;
  a.n = n;
  a.L = L;
  a.vec = ((uintptr_t)W & 15) == 0 && (n & 1) == 0;
  const bool wide = n * L > 2048;
  a.bands = (n + (wide ? 15 : 7)) / (wide ? 16 : 8);
  if (wide) return n <= 64 ? launch_c<16, 1>(a, st) : launch_c<16, 2>(a, st);
  return n <= 64 ? launch_c<8, 1>(a, st) : launch_c<8, 2>(a, st);
}

cudaError_t preload_bstri_band(size_t* local) {
  cudaError_t e;
  if ((e = preload_one(bstri_band_kernel<8, 1>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bstri_band_kernel<8, 2>, local)) != cudaSuccess) return e;
  if ((e = preload_one(bstri_band_kernel<16, 1>, local)) != cudaSuccess) return e;
  return preload_one(bstri_band_kernel<16, 2>, local);
}

}  // namespace bsofi
