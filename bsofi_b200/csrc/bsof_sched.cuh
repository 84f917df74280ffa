// Schedule of the persistent BSOF kernels: leaves, tiles, targets and the
// counters that order them (see kernels_bsof.cu for the decomposition).
#pragma once
#include "bsofi_common.cuh"

namespace bsofi {

struct BsofGeom {
  int n, L, NB, nl, S;
  int form_g;  // 1: leaves also update G_k = Q_k^T (identity-initialised by the caller)
};

// Leaf s -> panel k, leaf index l in the panel, tile (m, t), panel column j0.
struct Leaf {
  int k, l, m, t, j0, w;
};

BSOFI_DEVINL Leaf leaf_of(const BsofGeom& g, int s) {
  Leaf f;
  const int reg = (g.L - 2) * g.nl;
  if (s < reg) {
    f.k = s / g.nl;
    f.l = s % g.nl;
    f.m = f.k;
    f.t = f.l;
    f.j0 = f.t * g.NB;
  } else {
    f.k = g.L - 2;
    f.l = s - reg;
    if (f.l < g.nl) {
      f.m = g.L - 2;
      f.t = f.l;
      f.j0 = f.t * g.NB;
    } else {
      f.m = g.L - 1;
      f.t = f.l - g.nl;
      f.j0 = g.n + f.t * g.NB;
    }
  }
  f.w = min(g.NB, g.n - f.t * g.NB);
  return f;
}

BSOFI_DEVINL int tile_id(const BsofGeom& g, int m, int t) { return m * g.nl + t; }

BSOFI_DEVINL void tile_range(const BsofGeom& g, int m, int t, int& lo, int& hi) {
  if (m >= g.L) {  // G_k tile: every leaf of panel k, in order
    const int k = (m - g.L) / 2;
    lo = k * g.nl;
    hi = lo + (k <= g.L - 3 ? g.nl : 2 * g.nl);
    return;
  }
  if (m <= g.L - 2) {
    lo = max(0, (m - 1) * g.nl);
    hi = m * g.nl + t;
  } else {
    lo = 0;
    hi = (g.L - 1) * g.nl + t;
  }
}

// Number of targets of leaf s; target q (0 = tile of leaf s+1).  With
// form_g the 2*nl column tiles of G_k follow the matrix targets; they are
// reported as block columns m = L + 2k + h (h = 0, 1) of a virtual matrix.
BSOFI_DEVINL int ntargets(const BsofGeom& g, const Leaf& f) {
  const int gt = g.form_g ? 2 * g.nl : 0;
  if (f.k <= g.L - 3) return (g.nl - 1 - f.l) + 2 * g.nl + gt;
  return 2 * g.nl - 1 - f.l + gt;
}

BSOFI_DEVINL void target_of(const BsofGeom& g, const Leaf& f, int q, int& m, int& t) {
  const int nmat = (f.k <= g.L - 3) ? (g.nl - 1 - f.l) + 2 * g.nl : 2 * g.nl - 1 - f.l;
  if (q >= nmat) {
    const int u = q - nmat;
    m = g.L + 2 * f.k + u / g.nl;
    t = u % g.nl;
    return;
  }
  if (f.k <= g.L - 3) {
    const int np = g.nl - 1 - f.l;
    if (q < np) {
      m = f.k;
      t = f.l + 1 + q;
    } else if (q < np + g.nl) {
      m = f.k + 1;
      t = q - np;
    } else {
      m = g.L - 1;
      t = q - np - g.nl;
    }
  } else {
    int u = f.l + 1 + q;
    if (u < g.nl) {
      m = g.L - 2;
      t = u;
    } else {
      m = g.L - 1;
      t = u - g.nl;
    }
  }
}

// Worker tasks before leaf s (each leaf contributes ntargets - 1 tasks).
BSOFI_DEVINL long long tasks_before(const BsofGeom& g, int s) {
  const int reg = (g.L - 2) * g.nl;
  const long long nl = g.nl, gt = g.form_g ? 2 * nl : 0;
  const long long per_reg_leaf0 = 3 * nl - 2 + gt;  // tasks of regular leaf l: 3nl - 2 - l + gt
  const long long per_panel = nl * per_reg_leaf0 - nl * (nl - 1) / 2;
  if (s <= reg) {
    long long k = s / g.nl, l = s % g.nl;
    return k * per_panel + l * per_reg_leaf0 - l * (l - 1) / 2;
  }
  long long base = (long long)(g.L - 2) * per_panel;
  long long l = s - reg;  // final leaf l has max(2nl - 2 - l + gt, 0) tasks
  if (gt > 0) return base + l * (2 * nl - 2 + gt) - l * (l - 1) / 2;
  long long full = min(l, 2 * nl - 1);
  return base + full * (2 * nl - 2) - full * (full - 1) / 2;
}

struct BsofState {
  // Block columns 0..L-2 of the matrix at A (leading dimension ld), the last
  // block column at Al (ldl).  The ordinary layout has Al = A + (L-1) n ld;
  // the compact one stores block columns 0..L-2 with ld = 3n (every access
  // of block column m stays in block rows m-1..m+1, so those windows never
  // overlap) and the last block column as its own N x n array.
  double* A;
  long long ld;
  double* Al;
  long long ldl;
  double* G;  // (L-1) x (2n)^2, used when form_g
  double* tau;
  double* T;  // 256 doubles per leaf: (k * maxleaves + l) * 256
  int maxleaves;
  int* cnt;       // per tile
  int* factored;  // per leaf
  int* next_task;
  int* err;       // 0 ok; 1 timeout
  long long spin_limit;
  unsigned long long* timeline;  // 4 stamps per leaf from the panel CTA (diagnostics)
  // This launch factors leaves [s_begin, s_end) and runs their worker tasks;
  // the per-tile and per-leaf counters carry over from an earlier launch of
  // the leaves before s_begin, whose updates are then all done.
  int s_begin, s_end;
};

// Element (row, column col of block column m) of the matrix, and the leading
// dimension there.
BSOFI_DEVINL double* mat_ptr(const BsofGeom& g, const BsofState& st, long long row, int m,
                             int col, long long& ldm) {
  if (m == g.L - 1) {
    ldm = st.ldl;
    return st.Al + cm(row, col, st.ldl);
  }
  ldm = st.ld;
  return st.A + cm(row, (long long)m * g.n + col, st.ld);
}

// Column tile (m, t) of the matrix, or of G_k for m >= L: base pointer at the
// leaf's first row j0 of its panel, and leading dimension.
BSOFI_DEVINL double* tile_ptr(const BsofGeom& g, const BsofState& st, int k, int j0, int m, int t,
                              long long& ldt) {
  if (m >= g.L) {
    const int kk = (m - g.L) / 2, h = (m - g.L) % 2;
    const long long n2 = 2ll * g.n;
    ldt = n2;
    return st.G + (long long)kk * n2 * n2 + cm(j0, (long long)h * g.n + t * g.NB, n2);
  }
  return mat_ptr(g, st, (long long)k * g.n + j0, m, t * g.NB, ldt);
}

BSOFI_DEVINL unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

BSOFI_DEVINL int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

BSOFI_DEVINL void red_release_add(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Thread 0 waits until *p >= target (bounded); the result is broadcast.
// Returns false when the wait timed out or another CTA reported an error.
BSOFI_DEVINL bool block_wait_geq(const BsofState& st, const int* p, int target, int* sflag) {
  if (threadIdx.x == 0) {
    int ok = 1;
    long long it = 0;
    while (ld_acquire(p) < target) {
      if (ld_acquire(st.err) != 0) {
        ok = 0;
        break;
      }
      if (++it > st.spin_limit) {
        atomicExch(st.err, 1);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    *sflag = ok;
  }
  __syncthreads();
  bool ok = *sflag != 0;
  __syncthreads();
  return ok;
}

// n above kernels_bsof.cu's limit (kernels_bsof_tall.cu).
cudaError_t launch_bsof_tall(const BsofGeom& g, const BsofState& st, int workers, cudaStream_t s);
cudaError_t preload_bsof_tall(size_t* local);

}  // namespace bsofi
