// fx_diag.cuh -- the FP64 checks of the FP32 / fixed-point form and the
// absorbed (background) charge (included by fx.cu inside its private
// namespace, after fx_push.cuh).
//
// * Kinetic energy (energy.F90:29-47): FP64 sums of vx^2, vy^2, vz^2 over
//   the live particles of a species region.  A v of FP32 squared is exact in
//   FP64; the sums run in a fixed order (per-block partials of a fixed grid,
//   then one block over the partials), so the result is reproducible bit for
//   bit.
// * Charge continuity (rhoupd.F90:41-49): when a step converts its folded
//   int64 rho into the FP64 rho field, the field still holds the rho of the
//   step before; k_fix_to_rho takes, over the nodes 0..n of every axis, the
//   FP64 residual |rho_new - rho_old + 2 (div J)| of the step (J already
//   converted) and keeps its largest value and that of |rho_new|.
// * Background charge (charge.F90:414-449 with rhobk(...,3) += rhobk(...,1)
//   of emses.F90:249-251): the exact int64 counts per surface cell of the
//   box bodies (absorbed minus emitted particles since the start) become the
//   node field rhobk: a surface cell's charge q * count goes in equal
//   quarters to the four nodes of its face cell.  The counts of the faces
//   that meet at a node are summed in int64 per species, then scaled once in
//   FP64, so the field is exact up to that one rounding.

constexpr int DIAG_BLOCK = 256;
constexpr int DIAG_GRID = 4 * 148;

// Per-block FP64 sums of v^2 per component over slots [0, ntile) of the
// tile regions (ntile read on the device: the last tile_pad entry) and the
// tail zone [tail0, tail0 + ntail) of one species region; dead and empty
// slots hold the DEAD cell.  part[blockIdx.x][3].
__global__ void __launch_bounds__(DIAG_BLOCK) k_fx_energy_part(const float4* __restrict__ pos,
                                                               const float* __restrict__ vx,
                                                               const float* __restrict__ vy,
                                                               const float* __restrict__ vz,
                                                               const int64_t* __restrict__ tile_end, int64_t tail0,
                                                               int64_t ntail, double* __restrict__ part) {
  __shared__ double s[3][DIAG_BLOCK / 32];
  const int64_t ntile = *tile_end;
  const int64_t n = ntile + ntail;
  double t[3] = {0.0, 0.0, 0.0};
  for (int64_t m = (int64_t)blockIdx.x * DIAG_BLOCK + threadIdx.x; m < n; m += (int64_t)gridDim.x * DIAG_BLOCK) {
    const int64_t slot = m < ntile ? m : tail0 + (m - ntile);
    if ((uint32_t)__float_as_int(pos[slot].w) == DEAD) continue;
    const double a = vx[slot], b = vy[slot], c = vz[slot];
    t[0] += a * a;
    t[1] += b * b;
    t[2] += c * c;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double v = t[d];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) s[d][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = 0.0;
    for (int w = 0; w < DIAG_BLOCK / 32; w++) v += s[threadIdx.x][w];
    part[blockIdx.x * 3 + threadIdx.x] = v;
  }
}

// out[3] = the sums of the nparts partials, in order.
__global__ void k_fx_energy_sum(const double* __restrict__ part, int nparts, double* __restrict__ out) {
  if (threadIdx.x < 3) {
    double v = 0.0;
    for (int b = 0; b < nparts; b++) v += part[b * 3 + threadIdx.x];
    out[threadIdx.x] = v;
  }
}

// Largest of non-negative doubles, as their bit patterns (which order them).
__device__ __forceinline__ void max_nonneg(unsigned long long* p, double v) {
  atomicMax(p, (unsigned long long)__double_as_longlong(v));
}

// The fields of a step from the raw int64 accumulators (scale 2^-40): J, then
// rho, each with its guard folds (fold_point: the accumulators stay as the push
// left them) in the pass that converts it to FP64.  Reading and writing the
// arrays once bounds it; as in-place slabs and two conversions it was 8
// launches (13 with faces): 136 us a step at 128^3 and 54 us at 32^3 under
// per-launch events, 116 and 19 us this way.
constexpr int FIELD_BLOCK = 256;
constexpr int FIELD_VEC = 4;
struct FieldsArgs {
  const long long* acc;
  double* out;
  FieldDesc f, fj;
  const double* aj;             // rho: the step's J, null without the current
  FoldGeo g;
  bool fold;                    // false: the accumulators are folded already (slab mode)
  unsigned blocks;              // J: blocks of its inner elements
  FoldShell shell;
  unsigned long long* res;
};
// J: the first blocks convert the elements that no fold writes, FIELD_VEC of
// a row a thread, the others the shell.  I: the type that holds an index.
template <class I>
__global__ void __launch_bounds__(FIELD_BLOCK) k_fx_j(FieldsArgs a) {
  const FieldDesc& f = a.f;
  if (blockIdx.x < a.blocks) {
    const I size = (I)f.size();
    const I e0 = ((I)blockIdx.x * FIELD_BLOCK + (I)threadIdx.x) * FIELD_VEC;
    if (e0 >= size) return;
    long long v[FIELD_VEC];
#pragma unroll
    for (int q = 0; q < FIELD_VEC; q++) v[q] = e0 + q < size ? a.acc[e0 + q] : 0;
    const I row = (I)(f.nc * f.ex);
    const I r = e0 / row;
    int x = (int)(e0 - r * row);  // element in its row
    int k = (int)(r / (I)f.ey), j = (int)(r - (I)k * (I)f.ey);
    const int xlo = f.nc * (2 - f.lo), xhi = f.nc * (a.g.n[0] - 1 - f.lo);
#pragma unroll
    for (int q = 0; q < FIELD_VEC; q++) {
      const bool inner = x >= xlo && x < xhi && j > 1 - f.lo && j < a.g.n[1] - 1 - f.lo && k > 1 - f.lo &&
                         k < a.g.n[2] - 1 - f.lo;
      if (e0 + q < size && (inner || !a.fold)) a.out[e0 + q] = (double)v[q] * FIX_INV;
      if (++x == (int)row) {
        x = 0;
        if (++j == f.ey) {
          j = 0;
          k++;
        }
      }
    }
    return;
  }
  const int64_t t = (int64_t)(blockIdx.x - a.blocks) * FIELD_BLOCK + threadIdx.x;
  if (t >= (a.shell.nzs + a.shell.nys + a.shell.nxs) * f.nc) return;
  int x[3];
  shell_node(a.shell, t / f.nc, x);
  const int c = (int)(t % f.nc), i = x[0] + f.lo, j = x[1] + f.lo, k = x[2] + f.lo;
  a.out[f.at(c, i, j, k)] = (double)fold_point(a.acc, f, a.g, c, i, j, k) * FIX_INV;
}

// rho, a node a thread, and over the nodes 0..n the continuity residual of
// the step: res[0] = max |rho_new - rho_old + 2 (div J)|, res[1] = max
// |rho_new| (rhoupd.F90:41-49 gives rho_old - 2 div J as the prediction of
// rho_new; the rho field still holds rho_old).  The maxima are taken per block
// (warp shuffles, then the block's warps) and go to memory only where they
// exceed what is there.
template <class I>
__global__ void __launch_bounds__(FIELD_BLOCK) k_fx_rho(FieldsArgs a) {
  __shared__ double wmax[2][FIELD_BLOCK / 32];
  const FieldDesc& f = a.f;
  const FieldDesc& fj = a.fj;
  const I e = (I)blockIdx.x * FIELD_BLOCK + (I)threadIdx.x;
  double r = 0.0, m = 0.0;
  if (e < (I)f.size()) {
    const I row = e / (I)f.ex, plane = row / (I)f.ey;
    const int i = (int)(e - row * (I)f.ex) + f.lo, j = (int)(row - plane * (I)f.ey) + f.lo, k = (int)plane + f.lo;
    const long long raw = a.fold && !fold_inner(a.g, i, j, k) ? fold_point(a.acc, f, a.g, 0, i, j, k) : a.acc[e];
    const double v = (double)raw * FIX_INV;
    if (i >= 0 && j >= 0 && k >= 0 && i <= a.g.n[0] && j <= a.g.n[1] && k <= a.g.n[2]) {
      if (a.aj) {  // without the step's current (the electrostatic step) no residual
        const int64_t x = fj.at(0, i, j, k), sx = fj.nc, sy = sx * fj.ex, sz = sy * fj.ey;
        const double div = (a.aj[x] - a.aj[x - sx]) + (a.aj[x + 1] - a.aj[x + 1 - sy]) + (a.aj[x + 2] - a.aj[x + 2 - sz]);
        r = fabs(v - (a.out[e] - div * 2.0));
      }
      m = fabs(v);
    }
    a.out[e] = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    r = fmax(r, __shfl_down_sync(0xffffffffu, r, o));
    m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    wmax[0][warp] = r;
    wmax[1][warp] = m;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = 0.0;
    for (int w = 0; w < FIELD_BLOCK / 32; w++) v = fmax(v, wmax[threadIdx.x][w]);
    if (v > __longlong_as_double(*(volatile long long*)&a.res[threadIdx.x])) max_nonneg(&a.res[threadIdx.x], v);
  }
}

// One body's background charge: for every node of its bounding box (one
// thread each) the counts of the surface cells of species `is` whose face
// cell has the node as a corner, summed in int64, then rhobk(node) +=
// q * 0.25 * sum.  Faces as in Bodies: -x,+x,-y,+y,-z,+z, first tangential
// axis fastest.
__global__ void k_fx_background(const unsigned long long* __restrict__ surf, Bodies bd, int q, double qs,
                                double* __restrict__ rhobk, FieldDesc fr) {
  const int lo0 = bd.lo[q][0], lo1 = bd.lo[q][1], lo2 = bd.lo[q][2];
  const int w0 = bd.hi[q][0] - lo0 + 1, w1 = bd.hi[q][1] - lo1 + 1, w2 = bd.hi[q][2] - lo2 + 1;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)w0 * w1 * w2) return;
  const int n3[3] = {lo0 + (int)(t % w0), lo1 + (int)((t / w0) % w1), lo2 + (int)(t / ((int64_t)w0 * w1))};
  long long sum = 0;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int d = f >> 1, e1 = d == 0 ? 1 : 0, e2 = d == 2 ? 1 : 2;
    if (n3[d] != ((f & 1) ? bd.hi[q][d] : bd.lo[q][d])) continue;
    const int ext1 = bd.hi[q][e1] - bd.lo[q][e1], ext2 = bd.hi[q][e2] - bd.lo[q][e2];
    const int a = n3[e1] - bd.lo[q][e1], b = n3[e2] - bd.lo[q][e2];  // node (a, b) of the face
    for (int v = b - 1; v <= b; v++)
      for (int u = a - 1; u <= a; u++)
        if (u >= 0 && v >= 0 && u < ext1 && v < ext2)
          sum += (long long)surf[bd.off[q][f] + u + (int64_t)ext1 * v];
  }
  if (sum != 0) {
    const int64_t x = fr.at(0, n3[0], n3[1], n3[2]);
    rhobk[x] = rhobk[x] + qs * 0.25 * (double)sum;
  }
}

// rho(0:n) += rhobk(0:n), or = rhobk(0:n) (charge.F90:440-448).
__global__ void k_add_background(double* __restrict__ rho, const double* __restrict__ rhobk, FieldDesc fr, int nx,
                                 int ny, int nz, int replace) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= fr.size()) return;
  const int64_t ex = fr.ex, ey = fr.ey;
  const int i = (int)(e % ex) + fr.lo, j = (int)((e / ex) % ey) + fr.lo, k = (int)(e / (ex * ey)) + fr.lo;
  if (i < 0 || j < 0 || k < 0 || i > nx || j > ny || k > nz) return;
  rho[e] = replace ? rhobk[e] : rho[e] + rhobk[e];
}
