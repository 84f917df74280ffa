// BSOI of small blocks: one CTA per band of rows, all p-1 steps in one launch.
//
// Reference: lapackXbsoi_ormqr / _orgqr, src/bsofi_cpu.c:211-333 (applied
// from k = L-2 down to 0): step k is [X(:,k) | carry] (N x 2n) * Q_k^T
// (2n x 2n) -> [carry' | X(:,k+1) final].  Rows never mix, so a CTA that owns
// a band of rows runs every step without waiting for any other: the carry
// stays in its shared memory, X(:,k) is read once, X(:,k+1) written once, and
// the Q_k^T stream through shared memory from L2, where all CTAs read them.
//
// What bounds it: the FP64 tensor pipe of one SM for the tall bands (64 cycles
// per m16n8k8, plus about a quarter of output tiles that do not divide by
// eight warps at n = 100), instruction issue and the barrier of every chunk
// for the 8-row bands of small problems.  Measured (BSOI alone, us; before:
// one launch of 64 x 64 tiles per step, or one persistent launch of them):
// n = 16, p = 8 75 -> 18; n = 64, p = 16 254 -> 61; n = 64, p = 100 1472 ->
// 870; n = 100, p = 32 837 -> 451; n = 100, p = 64 1565 -> 1456; n = 128,
// p = 20 564 -> 342; n = 128, p = 40 1027 -> 977.  Above n = 112 the carry and the
// stages leave room for 48 rows only, and n = 128, p = 55 takes longer than before
// (1690 -> 1948): pipeline.cu ends the bands before that.  Above n = 128 there is no
// room for tall bands at all.
//
// Bands are cut on the host: rows of X below the diagonal block are zero in
// segment X(:,k), so a row near the bottom costs half of one at the top.
#include <climits>
#include "bsofi_common.cuh"
#include "bsofi_kernels.h"

namespace bsofi {

namespace {

constexpr int kBandThreads = 256, kBandWarps = 8;
constexpr int kMaxBands = 160;

// Depth and number of the Q_k^T stages for NTW output tiles a warp: a chunk
// takes the few rows of a small problem's bands a few hundred cycles, so
// chunks are deeper and more of them on their way (16 deep and three: 87 us at
// n = 64, p = 16); taller bands of larger blocks need the room for their rows.
__host__ __device__ constexpr int kc_of(int ntw) { return ntw <= 2 ? 32 : 16; }
__host__ __device__ constexpr int stages_of(int ntw) { return ntw <= 2 ? 4 : 3; }
__host__ __device__ constexpr int ntw_of(int n) { return n <= 64 ? 2 : 4; }

struct BandArgs {
  double* A;
  long long ld;
  const double* G;  // (L-1) x (2n)^2, G_k = Q_k^T
  int n, L, N;
  int* info;        // {info, BSOF error, BSOI error, BSTRI error}
  bool vec_a, vec_g;
  unsigned short start[kMaxBands + 1];  // first row of each band, in units of 8
};

// Columns of the two segments, a whole number of chunks each.
__host__ __device__ __forceinline__ int band_npad(int n, int ntw) {
  return (n + kc_of(ntw) - 1) / kc_of(ntw) * kc_of(ntw);
}

// Doubles of shared memory for bands of `rows` rows.  (A stage's column stride
// is 4 mod 16 doubles, as is a segment's row stride: no bank conflicts.)
__host__ __device__ __forceinline__ int band_smem_doubles(int n, int rows) {
  const int ntw = ntw_of(n), n2p = (2 * n + 7) & ~7;
  return 2 * band_npad(n, ntw) * (rows + 4) + stages_of(ntw) * n2p * (kc_of(ntw) + 4);
}

// Rows [r0, r0 + ROWS) of block column m (upper triangular: element (r, c) is
// zero for r > m n + c), into sA[c][row].
template <int ROWS>
BSOFI_DEVINL void load_x(double* sA, const BandArgs& s, int r0, int m) {
  constexpr int SA = ROWS + 4;
  const double* X = s.A + cm(0, (long long)m * s.n, s.ld);
  if (s.vec_a) {
    for (int e = threadIdx.x; e < s.n * (ROWS / 2); e += kBandThreads) {
      const int c = e / (ROWS / 2), rl = (e % (ROWS / 2)) * 2, r = r0 + rl;
      const int nv = min(max(min(s.N, m * s.n + c + 1) - r, 0), 2);
      cp_async16(sA + c * SA + rl, nv ? X + cm(r, c, s.ld) : X, nv * 8);
    }
  } else {
    for (int e = threadIdx.x; e < s.n * ROWS; e += kBandThreads) {
      const int c = e / ROWS, rl = e % ROWS, r = r0 + rl;
      const bool ok = r < min(s.N, m * s.n + c + 1);
      cp_async8(sA + c * SA + rl, ok ? X + cm(r, c, s.ld) : X, ok ? 8 : 0);
    }
  }
}

// Rows [k0, k0 + KC) of the half `h` of Q_k^T (every column) into one stage;
// rows beyond the half are zero (columns beyond 2n hold anything: they only
// meet output columns that are not stored).
template <int KC>
BSOFI_DEVINL void load_g(double* sB, const BandArgs& s, int k, int h, int k0) {
  constexpr int SB = KC + 4;
  const int n2 = 2 * s.n, valid = s.n - k0;
  const double* G = s.G + (long long)k * n2 * n2 + h * s.n + k0;
  if (s.vec_g && (h == 0 || (s.n & 1) == 0)) {
    const int kk = (threadIdx.x % (KC / 2)) * 2;
    int j = threadIdx.x / (KC / 2);
    const int bytes = 8 * min(max(valid - kk, 0), 2);
    const double* src = G + (bytes ? cm(kk, j, n2) : 0);
    const long long step = bytes ? (long long)(2 * kBandThreads / KC) * n2 : 0;
    double* dst = sB + j * SB + kk;
#pragma unroll 4
    for (; j < n2; j += 2 * kBandThreads / KC) {
      cp_async16(dst, src, bytes);
      src += step;
      dst += 2 * kBandThreads / KC * SB;
    }
  } else {
    const int kk = threadIdx.x % KC;
    const bool ok = kk < valid;
#pragma unroll 4
    for (int j = threadIdx.x / KC; j < n2; j += kBandThreads / KC)
      cp_async8(sB + j * SB + kk, ok ? G + cm(kk, j, n2) : s.G, ok ? 8 : 0);
  }
}

// NTW: 8-column tiles of the output per warp (tile w + 8 i for warp w).
template <int ROWS, int NTW>
BSOFI_DEVINL void band(const BandArgs& s, int r0, double* smem) {
  // 16-row tiles, and an 8-row one at the end of an odd multiple of 8.
  constexpr int SA = ROWS + 4, MT = ROWS / 16, TAIL = (ROWS % 16) / 8;
  constexpr int BSTAGES = stages_of(NTW), KC = kc_of(NTW), SB = KC + 4;
  const int n = s.n, n2 = 2 * n, npad = band_npad(n, NTW), nc = npad / KC;
  const int n2p = (n2 + 7) & ~7, tiles = n2p / 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  double* sX = smem;                // [npad][SA]
  double* sCar = smem + npad * SA;  // [npad][SA]
  double* sB = smem + 2 * npad * SA;
  const int bstage = n2p * SB;
  // Columns n..npad-1 of both segments stay zero, and nothing in the stages'
  // columns beyond 2n is left undefined.
  for (int e = threadIdx.x; e < BSTAGES * bstage; e += kBandThreads) sB[e] = 0.0;
  for (int e = threadIdx.x; e < (npad - n) * SA; e += kBandThreads)
    sX[n * SA + e] = sCar[n * SA + e] = 0.0;
  __syncthreads();
  load_x<ROWS>(sCar, s, r0, s.L - 1);
  // Chunks in order: per step the carry's half (rows n.. of Q_k^T), then X's
  // while the band reaches above the end of block row k.
  int pk = s.L - 2, pc = 0, slot_in = 0;  // the next chunk to load
  auto chunks = [&](int k) { return r0 < (k + 1) * n ? 2 * nc : nc; };
  auto issue = [&]() {
    if (pk >= 0) {
      const bool xh = pc >= nc;
      load_g<KC>(sB + slot_in * bstage, s, pk, xh ? 0 : 1, (xh ? pc - nc : pc) * KC);
      if (++pc == chunks(pk)) {
        pc = 0;
        pk--;
      }
    }
    cp_async_commit();
    slot_in = slot_in + 1 == BSTAGES ? 0 : slot_in + 1;
  };
  if (chunks(s.L - 2) > nc) load_x<ROWS>(sX, s, r0, s.L - 2);
#pragma unroll
  for (int i = 0; i < BSTAGES - 1; i++) issue();
  int slot = 0;
#pragma unroll 1
  for (int k = s.L - 2; k >= 0; k--) {
    double acc[MT + TAIL][NTW][4];
#pragma unroll
    for (int i = 0; i < MT + TAIL; i++)
#pragma unroll
      for (int j = 0; j < NTW; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0;
    const int cnt = chunks(k);
#pragma unroll 1
    for (int c = 0; c < cnt; c++) {
      // The first chunk of X's half also waits for X(:,k), loaded with the
      // chunk issued at the start of the step.
      if (c == nc && nc < BSTAGES) cp_async_wait<0>();
      else cp_async_wait<BSTAGES - 2>();
      __syncthreads();
      issue();
      const double* tA = (c < nc ? sCar + c * KC * SA : sX + (c - nc) * KC * SA) + g;
      const double* tB = sB + slot * bstage + t;
      auto product = [&](int k8) {
        double af[MT + TAIL][4], bf[NTW][2];
#pragma unroll
        for (int i = 0; i < MT + TAIL; i++) {
          af[i][0] = tA[(k8 * 8 + t) * SA + i * 16];
          af[i][2] = tA[(k8 * 8 + t + 4) * SA + i * 16];
          if (i < MT) {
            af[i][1] = tA[(k8 * 8 + t) * SA + i * 16 + 8];
            af[i][3] = tA[(k8 * 8 + t + 4) * SA + i * 16 + 8];
          }
        }
#pragma unroll
        for (int j = 0; j < NTW; j++) {
          const int nt = min(warp + kBandWarps * j, tiles - 1);
          bf[j][0] = tB[(nt * 8 + g) * SB + k8 * 8];
          bf[j][1] = tB[(nt * 8 + g) * SB + k8 * 8 + 4];
        }
#pragma unroll
        for (int j = 0; j < NTW; j++) {
          if (warp + kBandWarps * j < tiles) {
#pragma unroll
            for (int i = 0; i < MT; i++)
              dmma_16x8x8(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bf[j][0], bf[j][1]);
            if constexpr (TAIL != 0) {
              double d[2] = {acc[MT][j][0], acc[MT][j][1]};
              dmma_8x8x4(d, af[MT][0], bf[j][0]);
              dmma_8x8x4(d, af[MT][2], bf[j][1]);
              acc[MT][j][0] = d[0];
              acc[MT][j][1] = d[1];
            }
          }
        }
      };
      const int k8n = (n - (c < nc ? c : c - nc) * KC + 7) / 8;
      if (k8n >= KC / 8) {
#pragma unroll
        for (int k8 = 0; k8 < KC / 8; k8++) product(k8);
      } else {
#pragma unroll 1
        for (int k8 = 0; k8 < k8n; k8++) product(k8);
      }
      slot = slot + 1 == BSTAGES ? 0 : slot + 1;
    }
    __syncthreads();  // the segments are no longer read
    if (k > 0 && chunks(k - 1) > nc) load_x<ROWS>(sX, s, r0, k - 1);
#pragma unroll
    for (int j = 0; j < NTW; j++) {
      const int nt = warp + kBandWarps * j;
      if (nt >= tiles) continue;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int col = nt * 8 + 2 * t + q;
        if (col >= n2) continue;
        // The new carry, at the last step X(:,0); X(:,k+1).
        const bool car = col < n && k > 0;
        double* out = s.A + cm(r0, col < n ? col : (long long)(k + 1) * n + col - n, s.ld);
#pragma unroll
        for (int i = 0; i < MT + TAIL; i++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (i == MT && h == 1) continue;
            const int rl = i * 16 + 8 * h + g;
            const double v = acc[i][j][2 * h + q];
            if (car) sCar[col * SA + rl] = v;
            else if (r0 + rl < s.N) out[rl] = v;
          }
      }
    }
  }
  cp_async_wait<0>();
}

template <int NTW>
__global__ void __launch_bounds__(kBandThreads, 1) bsoi_band_kernel(const __grid_constant__ BandArgs s) {
  extern __shared__ __align__(16) double smem_band[];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // This launch has no waits of its own; a bounded wait that gave up in an
    // earlier kernel turns the info word into an error.
    s.info[2] = 0;
    if ((s.info[1] | s.info[3]) != 0) s.info[0] = kInfoWaitFailed;
  }
  const int r0 = 8 * s.start[blockIdx.x];
  switch (s.start[blockIdx.x + 1] - s.start[blockIdx.x]) {
    case 1: band<8, NTW>(s, r0, smem_band); break;
    case 2: band<16, NTW>(s, r0, smem_band); break;
    case 3: band<24, NTW>(s, r0, smem_band); break;
    case 4: band<32, NTW>(s, r0, smem_band); break;
    case 5: band<40, NTW>(s, r0, smem_band); break;
    case 6: band<48, NTW>(s, r0, smem_band); break;
    case 7: band<56, NTW>(s, r0, smem_band); break;
    default: band<64, NTW>(s, r0, smem_band); break;
  }
}

// Steps of a row: one per k for the carry's half, one more while X(:,k)
// reaches the row.
long long row_cost(int n, int L, int r) { return (L - 1) + max(L - 1 - r / n, 0); }

// Bands whose cost (height times the top row's) stays within T, or 0 if there
// are more than `most`.
int cut_bands(int n, int L, int N, int hmax, long long T, int most, unsigned short* start) {
  int r = 0, nb = 0;
  while (r < N) {
    if (nb == most) return 0;
    int h = 8;
    while (h + 8 <= hmax && (h + 8) * row_cost(n, L, r) <= T && r + h < N) h += 8;
    start[nb++] = (unsigned short)(r / 8);
    r += h;
  }
  start[nb] = (unsigned short)(r / 8);
  return nb;
}

int band_sms() {
  static int sms[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  if (sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  return min(sms[dev], kMaxBands);
}

// The bands of (n, L), tallest in *rows; 0 when they do not fit one per SM.
int plan_bands(int n, int L, int sms, unsigned short* start, int* rows) {
  const int N = n * L;
  if (n > 128 || sms <= 0 || N > 64 * sms) return 0;
  int hmax = 64;
  while (hmax > 8 && band_smem_doubles(n, hmax) * sizeof(double) > 232448) hmax -= 8;
  long long lo = 0, hi = hmax * row_cost(n, L, 0);  // the cost that is enough
  unsigned short tmp[kMaxBands + 1];
  if (cut_bands(n, L, N, hmax, hi, sms, tmp) == 0) return 0;
  while (hi - lo > 1) {
    const long long mid = (lo + hi) / 2;
    if (cut_bands(n, L, N, hmax, mid, sms, tmp)) hi = mid;
    else lo = mid;
  }
  const int nb = cut_bands(n, L, N, hmax, hi, sms, start);
  *rows = 0;
  for (int i = 0; i < nb; i++) *rows = max(*rows, 8 * (start[i + 1] - start[i]));
  return nb;
}

template <int NTW>
cudaError_t launch_ntw(const BandArgs& a, int nb, int rows, cudaStream_t st) {
  static PerDevice once;
  const int dev = once.pending();
  if (dev >= 0) {
    cudaError_t e = cudaFuncSetAttribute(bsoi_band_kernel<NTW>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return e;
    once.mark(dev);
  }
  bsoi_band_kernel<NTW><<<nb, kBandThreads, band_smem_doubles(a.n, rows) * sizeof(double), st>>>(a);
  return cudaGetLastError();
}

}  // namespace

bool bsoi_band_fits(int n, int L) {
  unsigned short start[kMaxBands + 1];
  int rows;
  return plan_bands(n, L, band_sms(), start, &rows) > 0;
}

cudaError_t launch_bsoi_band(double* A, long long ld, const double* G, int n, int L, int* info,
                             cudaStream_t st) {
  BandArgs a;
  int rows = 0;
  const int nb = plan_bands(n, L, band_sms(), a.start, &rows);
  if (nb == 0) return cudaErrorInvalidValue;
  a.A = A;
  a.ld = ld;
  a.G = G;
  a.n = n;
  a.L = L;
  a.N = n * L;
  a.info = info;
  a.vec_a = ((uintptr_t)A & 15) == 0 && (ld & 1) == 0;
  a.vec_g = ((uintptr_t)G & 15) == 0;
  return ntw_of(n) == 2 ? launch_ntw<2>(a, nb, rows, st) : launch_ntw<4>(a, nb, rows, st);
}

cudaError_t preload_bsoi_band(size_t* local) {
  cudaError_t e;
  if ((e = preload_one(bsoi_band_kernel<2>, local)) != cudaSuccess) return e;
  return preload_one(bsoi_band_kernel<4>, local);
}

}  // namespace bsofi
