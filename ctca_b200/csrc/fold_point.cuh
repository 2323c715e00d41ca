// fold_point.cuh -- the guard folds of fold_ops.h in closed form: the value a
// node has after the whole list of slab operations, from the array before
// them.
//
// Every operation acts along one axis, so per axis an index has a few source
// indices and a factor:
//
//   rho (kind 0)   core 0..n.  Periodic: 0 and n are the sum of 0 and n; the
//                  guards -1 and n+1 hold copies of n and 0.  Face: 0 and n
//                  are doubled.
//   J (kind 1)     core -1..n+1.  Periodic: i <= 1 adds i + n, i >= n - 1 adds
//                  i - n; the guards -4..-2 and n+2..n+4 hold copies of
//                  n-1..n+1 and -1..1.  Face (nfbnd 1), tangential component:
//                  0 and n are doubled, n+1 copies n-1; normal component: -1,
//                  n and n+1 are minus 0, n-1 and n-2.
//   eb (kind 2)    copies only: -1, n, n+1 of a periodic axis from n-1, 0, 1.
//
// and the value is the sum over the sources of the three axes.  The ranges of
// the operations' other axes say where an axis' rule holds: the folds run z,
// y, x over the core of the axes folded after (z everywhere, y where k is in
// the core, x where j and k are); the guard copies run x, y, z over the core
// (eb: the cells 0..n-1) of the later axes, or their guards' sources.  Sums
// are formed in the operations' order (own value first, z innermost) and the
// factors are 2 and -1, so FP64 and int64 values come out bit for bit as from
// the operations one after the other, without their 6 to 12 launches over thin
// slabs.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "fold_ops.h"

namespace emsesg {

struct FoldGeo {
  int kind;    // 0 rho, 1 J (3 components a species), 2 eb
  int n[3];
  int bnd[3];  // nfbnd
};

inline FoldGeo fold_geo(const emsesg_config& c, int kind) {
  return FoldGeo{kind, {c.nx, c.ny, c.nz}, {c.nfbnd[0], c.nfbnd[1], c.nfbnd[2]}};
}

// Sources of one axis' index: count of them (at most 3: both ends of a
// two-cell axis) and the factor.
struct FoldAxis {
  int src[3];
  int count;
  int factor;
};

// copied / folded: whether the guard copy and the fold of this axis reach the
// element.
__host__ __device__ __forceinline__ FoldAxis fold_axis(int kind, int bnd, bool normal, int n, int i, bool copied,
                                                       bool folded) {
  FoldAxis a{{i, 0, 0}, 1, 1};
  if (bnd == 0) {
    if (kind == 0) {
      if (i < 0 || i > n) {
        if (copied) a.src[0] = i < 0 ? n : 0;
      } else if (folded && (i == 0 || i == n)) {
        a.src[a.count++] = n - i;
      }
    } else if (kind == 1) {
      if (i < -1 || i > n + 1) {
        if (copied) a.src[0] = i < -1 ? i + n + 3 : i - n - 3;
      } else if (folded) {
        if (i <= 1) a.src[a.count++] = i + n;
        if (i >= n - 1) a.src[a.count++] = i - n;
      }
    } else if (copied && (i < 0 || i >= n)) {
      a.src[0] = i < 0 ? i + n : i - n;
    }
  } else if (kind == 0) {
    if (folded && (i == 0 || i == n)) a.factor = 2;
  } else if (kind == 1 && bnd == 1 && folded) {
    if (normal) {
      if (i == -1 || i == n || i == n + 1) {
        a.factor = -1;
        a.src[0] = i == -1 ? 0 : i == n ? n - 1 : n - 2;
      }
    } else if (i == 0 || i == n) {
      a.factor = 2;
    } else if (i == n + 1) {
      a.src[0] = n - 1;
    }
  }
  return a;
}

// Nodes no fold or copy writes.
__host__ __device__ __forceinline__ bool fold_inner(const FoldGeo& g, int i, int j, int k) {
  return i > 1 && j > 1 && k > 1 && i < g.n[0] - 1 && j < g.n[1] - 1 && k < g.n[2] - 1;
}

template <typename T>
__host__ __device__ __forceinline__ T fold_point(const T* a, const FieldDesc& f, const FoldGeo& g, int c, int i, int j,
                                                 int k) {
  const int m = g.kind == 1 ? 1 : 0, lo = -m;  // core: -m .. n + m
  const bool cy = j >= lo && j <= g.n[1] + m, cz = k >= lo && k <= g.n[2] + m;
  // in the range of the earlier axes' copies: the core (eb: the cells), or a
  // guard that is itself a copy
  const int e = g.kind == 2 ? 1 : 0;
  const bool oy = g.bnd[1] == 0 || (cy && j <= g.n[1] + m - e), oz = g.bnd[2] == 0 || (cz && k <= g.n[2] + m - e);
  const int d = g.kind == 1 ? c % 3 : -1;
  const FoldAxis X = fold_axis(g.kind, g.bnd[0], d == 0, g.n[0], i, oy && oz, cy && cz);
  const FoldAxis Y = fold_axis(g.kind, g.bnd[1], d == 1, g.n[1], j, oz, cz);
  const FoldAxis Z = fold_axis(g.kind, g.bnd[2], d == 2, g.n[2], k, true, true);
  T sx = (T)0;
  for (int p = 0; p < X.count; p++) {
    const int ii = p == 0 ? X.src[0] : p == 1 ? X.src[1] : X.src[2];
    T sy = (T)0;
    for (int q = 0; q < Y.count; q++) {
      const int jj = q == 0 ? Y.src[0] : q == 1 ? Y.src[1] : Y.src[2];
      T sz = a[f.at(c, ii, jj, Z.src[0])];
      if (Z.count > 1) sz = sz + a[f.at(c, ii, jj, Z.src[1])];
      if (Z.count > 2) sz = sz + a[f.at(c, ii, jj, Z.src[2])];
      sy = q == 0 ? sz : sy + sz;
    }
    sx = p == 0 ? sy : sx + sy;
  }
  return sx * (T)(X.factor * Y.factor * Z.factor);
}

// Elements of an array that a fold or copy can write: the `edge` planes at
// each end of the z axis, then of y between them, then of x.
struct FoldShell {
  int lo, e0, e1;               // first index, planes at the lower and upper end
  int nx, ny, nz;               // extents
  int64_t nzs, nys, nxs;        // nodes of the three parts
};
inline FoldShell fold_shell(const FieldDesc& f) {
  FoldShell s;
  s.lo = f.lo;
  s.e0 = 2 - f.lo;              // lo .. 1
  s.nx = f.ex; s.ny = f.ey; s.nz = f.ez;
  s.e1 = f.lo == -4 ? 6 : 3;    // J: n-1..n+4, rho and eb: n-1..n+1
  const int64_t e = s.e0 + s.e1;
  const int64_t ny = std::max(0, s.ny - (int)e), nz = std::max(0, s.nz - (int)e);
  s.nzs = std::min<int64_t>(e, s.nz) * s.nx * s.ny;
  s.nys = nz * std::min<int64_t>(e, s.ny) * s.nx;
  s.nxs = nz * ny * std::min<int64_t>(e, s.nx);
  return s;
}
// Index of shell node t (relative to lo).
__host__ __device__ __forceinline__ void shell_node(const FoldShell& s, int64_t t, int (&x)[3]) {
  const int e = s.e0 + s.e1;
  auto end = [&](int v, int ext) { return v < s.e0 || ext <= e ? v : ext - e + v; };  // the v-th of the end planes
  if (t < s.nzs) {
    x[0] = (int)(t % s.nx);
    x[1] = (int)((t / s.nx) % s.ny);
    x[2] = end((int)(t / ((int64_t)s.nx * s.ny)), s.nz);
    return;
  }
  t -= s.nzs;
  if (t < s.nys) {
    const int ey = min(e, s.ny);
    x[0] = (int)(t % s.nx);
    x[1] = end((int)((t / s.nx) % ey), s.ny);
    x[2] = s.e0 + (int)(t / ((int64_t)s.nx * ey));
    return;
  }
  t -= s.nys;
  const int ex = min(e, s.nx), my = s.ny - e;
  x[0] = end((int)(t % ex), s.nx);
  x[1] = s.e0 + (int)((t / ex) % my);
  x[2] = s.e0 + (int)(t / ((int64_t)ex * my));
}

// The folds of an array in place in two launches: the shell's final values
// into scratch (part 0), scratch into the array (part 1).
template <typename T, int PART>
__global__ void k_fold_shell(T* __restrict__ a, T* __restrict__ scratch, FieldDesc f, FoldGeo g, FoldShell s) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (s.nzs + s.nys + s.nxs) * f.nc) return;
  int x[3];
  shell_node(s, t / f.nc, x);
  const int c = (int)(t % f.nc);
  const int i = x[0] + s.lo, j = x[1] + s.lo, k = x[2] + s.lo;
  if (PART == 0) scratch[t] = fold_point(a, f, g, c, i, j, k);
  else a[f.at(c, i, j, k)] = scratch[t];
}

template <typename T>
int run_fold(emsesg_ctx* ctx, T* a, const FieldDesc& f, int kind, const char* name) {
  const FoldGeo g = fold_geo(ctx->cfg, kind);
  const FoldShell s = fold_shell(f);
  const int64_t n = (s.nzs + s.nys + s.nxs) * f.nc;
  T* scratch = nullptr;
  int rc = fold_scratch(ctx, n * (int64_t)sizeof(T), (void**)&scratch);
  if (rc) return rc;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  EMSESG_LAUNCH(ctx, name, (k_fold_shell<T, 0>), blocks, 256, 0, a, scratch, f, g, s);
  EMSESG_LAUNCH(ctx, name, (k_fold_shell<T, 1>), blocks, 256, 0, a, scratch, f, g, s);
  return EMSESG_OK;
}

}  // namespace emsesg
