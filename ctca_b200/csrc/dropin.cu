// dropin.cu -- the plain FP64 GPU drop-in: one kernel per reference routine,
// keeping the 64-byte oh_particle records and the Fortran operation order.
//
// This file is compiled with --fmad=false so that no multiply-add is fused:
// positions, velocities, cell indices and counters of grdcrt / psolve1 /
// psolve2 are then bit-identical to an IEEE FP64 evaluation of the Fortran
// statements.  rho and J are summed with FP64 atomics, so their summation
// order (not their terms) differs from the reference's particle order.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "fold_point.cuh"

namespace emsesg {

namespace {

constexpr int EX = 0, EY = 1, EZ = 2, BX = 3, BY = 4, BZ = 5;
constexpr int JX = 0, JY = 1, JZ = 2;

struct W8 { double v1, v2, v3, v4, v5, v6, v7, v8; };

// Trilinear weights, psolve2.F90:166-183 / charge.F90:173-192.
__device__ __forceinline__ W8 weights(double x1, double y1, double z1) {
  W8 w;
  double xy1 = x1 * y1, xz1 = x1 * z1, yz1 = y1 * z1;
  double z2 = 1.0 - z1;
  double xz2 = x1 * z2, yz2 = y1 * z2;
  w.v3 = xy1 * z1;
  w.v2 = xz1 - w.v3;
  w.v4 = yz1 - w.v3;
  w.v1 = z1 - xz1 - w.v4;
  w.v7 = xy1 * z2;
  w.v6 = xz2 - w.v7;
  w.v8 = yz2 - w.v7;
  w.v5 = z2 - xz2 - w.v8;
  return w;
}

// 64-byte particle records (64-byte aligned: cudaMalloc'd regions of whole
// records) as two 256-bit halves {x, y, z, vx}, {vy, vz, pid | preside, nid |
// spec}.  The struct itself is 8-byte aligned, so plain copies of it become
// ten loads of 8 and 4 bytes, each of which touches 16 lines a warp: at
// 64^3 x 64 ppc (16.8 M records) psolve1 took 1.34 ms with those and 1.03 ms
// with these, and positn goes from 2.0 to 3.5 TB/s.
struct __align__(32) Half { unsigned long long w[4]; };
static_assert(sizeof(emsesg_particle) == 2 * sizeof(Half), "a record is two halves");
__device__ __forceinline__ Half load_half(const emsesg_particle* p, int h) {
  Half r;
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(r.w[0]), "=l"(r.w[1]), "=l"(r.w[2]), "=l"(r.w[3])
               : "l"(reinterpret_cast<const Half*>(p) + h)
               : "memory");
  return r;
}
__device__ __forceinline__ void store_half(emsesg_particle* p, int h, const Half& r) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(reinterpret_cast<Half*>(p) + h), "l"(r.w[0]),
               "l"(r.w[1]), "l"(r.w[2]), "l"(r.w[3])
               : "memory");
}
__device__ __forceinline__ double word(unsigned long long w) { return __longlong_as_double((long long)w); }
__device__ __forceinline__ int32_t lo32(unsigned long long w) { return (int32_t)(uint32_t)w; }
__device__ __forceinline__ int32_t hi32(unsigned long long w) { return (int32_t)(uint32_t)(w >> 32); }
__device__ __forceinline__ emsesg_particle load_record(const emsesg_particle* p) {
  const Half a = load_half(p, 0), b = load_half(p, 1);
  emsesg_particle r;
  r.x = word(a.w[0]); r.y = word(a.w[1]); r.z = word(a.w[2]); r.vx = word(a.w[3]);
  r.vy = word(b.w[0]); r.vz = word(b.w[1]);
  r.pid = lo32(b.w[2]); r.preside = hi32(b.w[2]);
  r.nid = lo32(b.w[3]); r.spec = hi32(b.w[3]);
  return r;
}
__device__ __forceinline__ unsigned long long bits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ unsigned long long bits(int32_t lo, int32_t hi) {
  return (unsigned long long)(uint32_t)lo | ((unsigned long long)(uint32_t)hi << 32);
}
__device__ __forceinline__ void store_record(emsesg_particle* p, const emsesg_particle& r) {
  store_half(p, 0, Half{{bits(r.x), bits(r.y), bits(r.z), bits(r.vx)}});
  store_half(p, 1, Half{{bits(r.vy), bits(r.vz), bits(r.pid, r.preside), bits(r.nid, r.spec)}});
}

struct PushArgs {
  emsesg_particle* p;
  int64_t n;
  const int64_t* count;   // device count of this species
  int is;
  int64_t packed_base;    // index of the first particle in the packed pbuf
  const double* node;     // 8 doubles per node over (nx+1)(ny+1)(nz+1)
  const emsesg_config* cfg;
  int ustep;
  uint64_t seed, stream;
  const double* randoms;
  int64_t nrand;
  const int64_t* rand_pos;
  const uint32_t* ordinal;
  emsesg_counter* gc;
  int* status;
  long long* diag;
  double* tj;             // psolve1: per-species zigzag scratch (aj layout)
  FieldDesc fa;
};

// The drop-in node field covers nodes 0..n+1 per axis; grdcrt fills 0..n
// (grdcrt.F90:158-160) and node n+1 stays 0.  A particle that a periodic
// wrap leaves exactly on x = slx (x - slx + slx rounding) has i = n and gathers
// node n+1 with weight 0, as the reference reads wrk(n+1) with weight 0.
__device__ __forceinline__ int64_t node_index(const emsesg_config* c, int i, int j, int k) {
  return (int64_t)i + (int64_t)(c->nx + 2) * ((int64_t)j + (int64_t)(c->ny + 2) * k);
}

__device__ __forceinline__ bool cell_ok(const emsesg_config* c, int i, int j, int k) {
  return i >= 0 && j >= 0 && k >= 0 && i <= c->nx && j <= c->ny && k <= c->nz;
}

// The six field values of one node record (64 bytes, 64-byte aligned).
struct Node { double v[6]; };
__device__ __forceinline__ Node load_node(const double* __restrict__ p) {
  Node n;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(n.v[0]), "=d"(n.v[1]), "=d"(n.v[2]), "=d"(n.v[3])
      : "l"(p));
  asm("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(n.v[4]), "=d"(n.v[5]) : "l"(p + 4));
  return n;
}

// Gather + Buneman-Boris + move, psolve2.F90:185-318 (psolve1.F90:201-333).
__device__ __forceinline__ void gather_boris_move(const double* __restrict__ node, const emsesg_config* c,
                                                  emsesg_particle& p, int i, int j, int k, const W8& w,
                                                  double qmp, double gustep) {
  int64_t n1 = node_index(c, i, j, k + 1), n5 = node_index(c, i, j, k);
  int64_t sx = 1, sy = c->nx + 2;
  // one 256-bit and one 128-bit load a node (64-byte records): 16 loads a
  // particle instead of 48 of 8 bytes
  const Node c1 = load_node(node + 8 * n1);             // (i,  j,  k1)
  const Node c2 = load_node(node + 8 * (n1 + sx));      // (i1, j,  k1)
  const Node c3 = load_node(node + 8 * (n1 + sx + sy)); // (i1, j1, k1)
  const Node c4 = load_node(node + 8 * (n1 + sy));      // (i,  j1, k1)
  const Node c5 = load_node(node + 8 * n5);             // (i,  j,  k)
  const Node c6 = load_node(node + 8 * (n5 + sx));
  const Node c7 = load_node(node + 8 * (n5 + sx + sy));
  const Node c8 = load_node(node + 8 * (n5 + sy));
  double eex = c1.v[EX] * w.v1 + c2.v[EX] * w.v2 + c3.v[EX] * w.v3 + c4.v[EX] * w.v4 + c5.v[EX] * w.v5 +
               c6.v[EX] * w.v6 + c7.v[EX] * w.v7 + c8.v[EX] * w.v8;
  double eey = c1.v[EY] * w.v1 + c2.v[EY] * w.v2 + c3.v[EY] * w.v3 + c4.v[EY] * w.v4 + c5.v[EY] * w.v5 +
               c6.v[EY] * w.v6 + c7.v[EY] * w.v7 + c8.v[EY] * w.v8;
  double eez = c1.v[EZ] * w.v1 + c2.v[EZ] * w.v2 + c3.v[EZ] * w.v3 + c4.v[EZ] * w.v4 + c5.v[EZ] * w.v5 +
               c6.v[EZ] * w.v6 + c7.v[EZ] * w.v7 + c8.v[EZ] * w.v8;
  double bbx = c1.v[BX] * w.v1 + c2.v[BX] * w.v2 + c3.v[BX] * w.v3 + c4.v[BX] * w.v4 + c5.v[BX] * w.v5 +
               c6.v[BX] * w.v6 + c7.v[BX] * w.v7 + c8.v[BX] * w.v8;
  double bby = c1.v[BY] * w.v1 + c2.v[BY] * w.v2 + c3.v[BY] * w.v3 + c4.v[BY] * w.v4 + c5.v[BY] * w.v5 +
               c6.v[BY] * w.v6 + c7.v[BY] * w.v7 + c8.v[BY] * w.v8;
  double bbz = c1.v[BZ] * w.v1 + c2.v[BZ] * w.v2 + c3.v[BZ] * w.v3 + c4.v[BZ] * w.v4 + c5.v[BZ] * w.v5 +
               c6.v[BZ] * w.v6 + c7.v[BZ] * w.v7 + c8.v[BZ] * w.v8;
  const double ewx = 0.0, ewy = 0.0;
  eex = (eex + ewx) * qmp;
  eey = (eey + ewy) * qmp;
  eez = eez * qmp;
  bbx = bbx * qmp;
  bby = bby * qmp;
  bbz = bbz * qmp;
  double boris = 2.0 / (1.0 + bbx * bbx + bby * bby + bbz * bbz);
  p.vx = p.vx + eex;
  p.vy = p.vy + eey;
  p.vz = p.vz + eez;
  double vxt = p.vx + p.vy * bbz - p.vz * bby;
  double vyt = p.vy + p.vz * bbx - p.vx * bbz;
  double vzt = p.vz + p.vx * bby - p.vy * bbx;
  p.vx = p.vx + boris * (vyt * bbz - vzt * bby);
  p.vy = p.vy + boris * (vzt * bbx - vxt * bbz);
  p.vz = p.vz + boris * (vxt * bby - vyt * bbx);
  p.vx = p.vx + eex;
  p.vy = p.vy + eey;
  p.vz = p.vz + eez;
  double xmove = p.vx * gustep, ymove = p.vy * gustep, zmove = p.vz * gustep;
  p.x = p.x + xmove;
  p.y = p.y + ymove;
  p.z = p.z + zmove;
}

// Single-rank nborps: -1 as soon as a crossed axis is neither periodic (0)
// nor reflecting (1), else the rank itself (0).  src/etc/nborps.F90:29-…
__device__ __forceinline__ int nborps_single(const int32_t* nb, bool cx, bool cy, bool cz) {
  if (cx && !(nb[0] == 0 || nb[0] == 1)) return -1;
  if (cy && !(nb[1] == 0 || nb[1] == 1)) return -1;
  if (cz && !(nb[2] == 0 || nb[2] == 1)) return -1;
  return 0;
}

__device__ __forceinline__ void absorb(emsesg_counter* gc, int is, int ipc, int pid) {
  atomicAdd(&gc->influx[is][ipc], 1);
  if (pid >= 0 && pid <= EMSESG_INPC) atomicAdd(&gc->infhist[is][ipc][pid], 1);
}

// Injected-particle random number (psolve2.F90:142-146).
__device__ __forceinline__ bool draw(const PushArgs& a, int64_t m, double& u) {
  if (a.cfg->rng_mode == 1) {
    int64_t k = *a.rand_pos + a.ordinal[m];
    if (k >= a.nrand) return false;
    u = a.randoms[k];
    return true;
  }
  u = hash_u01(a.seed, a.stream, (uint64_t)(a.packed_base + m));
  return true;
}

// Status handling at the top of the particle loop (psolve2.F90:138-152).
// Returns false when the particle is skipped.
__device__ __forceinline__ bool push_status(const PushArgs& a, int64_t m, emsesg_particle& p, double& gustep,
                                            double& qmp) {
  double qm = a.cfg->qm[a.is];
  gustep = 0.0;
  qmp = 0.0;
  if (p.preside < 0) {
    p.nid = -1;
    p.preside = 0;
  } else if (p.preside == EMSESG_PCL_INJECTED) {
    double u;
    if (!draw(a, m, u)) {
      atomicOr(a.status, ST_RANDOMS);
      u = 0.0;
    }
    gustep = (double)a.ustep * u;
    qmp = qm * gustep * 0.5;
    p.preside = 0;
  } else {
    gustep = (double)a.ustep;
    qmp = qm * gustep * 0.5;
  }
  return p.nid != -1;
}

// psolve2, src/pcl2field/psolve2.F90:137-533, one thread per particle.
__global__ void k_psolve2(PushArgs a) {
  int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.n || m >= *a.count) return;
  const emsesg_config* c = a.cfg;
  emsesg_particle p = load_record(a.p + m);
  double gustep, qmp;
  if (!push_status(a, m, p, gustep, qmp)) { store_record(a.p + m, p); return; }
  const double dxl = 0.0, dyl = 0.0, dzl = 0.0;
  const double dxu = c->nx, dyu = c->ny, dzu = c->nz;
  const double slx = c->nx, sly = c->ny, slz = c->nz;
  const double tslx = 2.0 * slx, tsly = 2.0 * sly, tslz = 2.0 * slz;
  double xlocal = p.x - dxl, ylocal = p.y - dyl, zlocal = p.z - dzl;
  int i = (int)xlocal, j = (int)ylocal, k = (int)zlocal;
  if (!cell_ok(c, i, j, k) || !(xlocal >= 0.0 && ylocal >= 0.0 && zlocal >= 0.0)) {
    report_bad(a.status, a.diag, SITE_PSOLVE2, a.packed_base + m, i + 100000LL * j + 10000000000LL * k);
    return;
  }
  W8 w = weights(xlocal - i, ylocal - j, zlocal - k);
  gather_boris_move(a.node, c, p, i, j, k, w, qmp, gustep);

  int nud = 14;
  if (p.x < dxl) nud -= 1; else if (p.x >= dxu) nud += 1;
  if (p.y < dyl) nud -= 3; else if (p.y >= dyu) nud += 3;
  if (p.z < dzl) nud -= 9; else if (p.z >= dzu) nud += 9;
  if (nud != 14) {
    const int32_t* nb = c->npbnd[a.is];
    p.nid = nborps_single(nb, p.x < dxl || p.x >= dxu, p.y < dyl || p.y >= dyu, p.z < dzl || p.z >= dzu);
    if (p.x < 0.0) {
      if (nb[0] == 0) p.x = p.x + slx;
      else if (nb[0] == 1) { p.x = -p.x; p.vx = -p.vx; }
    } else if (p.x >= slx) {
      if (nb[0] == 0) p.x = p.x - slx;
      else if (nb[0] == 1) { p.x = tslx - p.x; p.vx = -p.vx; }
    }
    if (p.y < 0.0) {
      if (nb[1] == 0) p.y = p.y + sly;
      else if (nb[1] == 1) { p.y = -p.y; p.vy = -p.vy; }
    } else if (p.y >= sly) {
      if (nb[1] == 0) p.y = p.y - sly;
      else if (nb[1] == 1) { p.y = tsly - p.y; p.vy = -p.vy; }
    }
    if (p.z < 0.0) {
      if (nb[2] == 0) p.z = p.z + slz;
      else if (nb[2] == 1) { p.z = -p.z; p.vz = -p.vz; }
    } else if (p.z >= slz) {
      if (nb[2] == 0) p.z = p.z - slz;
      else if (nb[2] == 1) { p.z = tslz - p.z; p.vz = -p.vz; }
    }
    if (p.nid == -1) atomicAdd(&a.gc->nesc[a.is], 1);
  }
  // Internal boundary treatment 1, psolve2.F90:465-531.
  if (c->line_mode != 1) {
    for (int ipc = 0; ipc < c->npc; ipc++) {
      if (p.nid == -1) continue;
      const emsesg_body& b = c->body[ipc];
      bool kill = false;
      if ((b.geotype == 0 || b.geotype == 1) &&
          (p.x >= b.xlpc && p.x <= b.xupc && p.y >= b.ylpc && p.y <= b.yupc && p.z >= b.zlpc && p.z <= b.zupc)) {
        kill = true;
      } else if (b.geotype == 2) {
        double d1, d2, ax;
        if (b.cyl_align == 1) { d1 = p.y - b.cyl_axis[0]; d2 = p.z - b.cyl_axis[1]; ax = p.x; }
        else if (b.cyl_align == 2) { d1 = p.z - b.cyl_axis[0]; d2 = p.x - b.cyl_axis[1]; ax = p.y; }
        else if (b.cyl_align == 3) { d1 = p.x - b.cyl_axis[0]; d2 = p.y - b.cyl_axis[1]; ax = p.z; }
        else continue;
        if (ax >= b.cyl_edge[0] && ax <= b.cyl_edge[1] && d1 * d1 + d2 * d2 < b.radius * b.radius) kill = true;
      } else if (b.geotype == 3) {
        double d1 = p.x - b.sph_center[0], d2 = p.y - b.sph_center[1], d3 = p.z - b.sph_center[2];
        if (d1 * d1 + d2 * d2 + d3 * d3 < b.radius * b.radius) kill = true;
      }
      if (kill) {
        p.nid = -1;
        absorb(a.gc, a.is, ipc, p.pid);
      }
    }
  }
  store_record(a.p + m, p);
}

// positn, src/pcl/positn.F90:50-355: position-only advance (x += v*ustep;
// injected particles still draw, :97-101), outer boundary with nesc counted
// per escaping axis (:228-268), body test with the box bounds as the
// cylinder's axial extent (:283-316).  One thread per particle.
__global__ void k_positn(PushArgs a) {
  int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.n || m >= *a.count) return;
  const emsesg_config* c = a.cfg;
  emsesg_particle p = load_record(a.p + m);
  double gustep, qmp;
  if (!push_status(a, m, p, gustep, qmp)) { store_record(a.p + m, p); return; }
  const double dxl = 0.0, dyl = 0.0, dzl = 0.0;
  const double dxu = c->nx, dyu = c->ny, dzu = c->nz;
  const double slx = c->nx, sly = c->ny, slz = c->nz;
  const double tslx = 2.0 * slx, tsly = 2.0 * sly, tslz = 2.0 * slz;
  const double us = (double)a.ustep;
  double xmove = p.vx * us, ymove = p.vy * us, zmove = p.vz * us;
  p.x = p.x + xmove;
  p.y = p.y + ymove;
  p.z = p.z + zmove;
  int nud = 14;
  if (p.x < dxl) nud -= 1; else if (p.x >= dxu) nud += 1;
  if (p.y < dyl) nud -= 3; else if (p.y >= dyu) nud += 3;
  if (p.z < dzl) nud -= 9; else if (p.z >= dzu) nud += 9;
  if (nud != 14) {
    const int32_t* nb = c->npbnd[a.is];
    p.nid = nborps_single(nb, p.x < dxl || p.x >= dxu, p.y < dyl || p.y >= dyu, p.z < dzl || p.z >= dzu);
    int esc = 0;
    if (p.x < 0.0) {
      if (nb[0] == 0) p.x = p.x + slx;
      else if (nb[0] == 1) { p.x = -p.x; p.vx = -p.vx; }
      else esc++;
    } else if (p.x >= slx) {
      if (nb[0] == 0) p.x = p.x - slx;
      else if (nb[0] == 1) { p.x = tslx - p.x; p.vx = -p.vx; }
      else esc++;
    }
    if (p.y < 0.0) {
      if (nb[1] == 0) p.y = p.y + sly;
      else if (nb[1] == 1) { p.y = -p.y; p.vy = -p.vy; }
      else esc++;
    } else if (p.y >= sly) {
      if (nb[1] == 0) p.y = p.y - sly;
      else if (nb[1] == 1) { p.y = tsly - p.y; p.vy = -p.vy; }
      else esc++;
    }
    if (p.z < 0.0) {
      if (nb[2] == 0) p.z = p.z + slz;
      else if (nb[2] == 1) { p.z = -p.z; p.vz = -p.vz; }
      else esc++;
    } else if (p.z >= slz) {
      if (nb[2] == 0) p.z = p.z - slz;
      else if (nb[2] == 1) { p.z = tslz - p.z; p.vz = -p.vz; }
      else esc++;
    }
    if (esc) atomicAdd(&a.gc->nesc[a.is], esc);
  }
  if (c->line_mode != 1) {
    for (int ipc = 0; ipc < c->npc; ipc++) {
      if (p.nid == -1) continue;
      const emsesg_body& b = c->body[ipc];
      bool kill = false;
      if ((b.geotype == 0 || b.geotype == 1) &&
          (p.x >= b.xlpc && p.x <= b.xupc && p.y >= b.ylpc && p.y <= b.yupc && p.z >= b.zlpc && p.z <= b.zupc)) {
        kill = true;
      } else if (b.geotype == 2) {
        double d1, d2, ax, lo, hi;
        if (b.cyl_align == 1) { d1 = p.y - b.cyl_axis[0]; d2 = p.z - b.cyl_axis[1]; ax = p.x; lo = b.xlpc; hi = b.xupc; }
        else if (b.cyl_align == 2) { d1 = p.z - b.cyl_axis[0]; d2 = p.x - b.cyl_axis[1]; ax = p.y; lo = b.ylpc; hi = b.yupc; }
        else if (b.cyl_align == 3) { d1 = p.x - b.cyl_axis[0]; d2 = p.y - b.cyl_axis[1]; ax = p.z; lo = b.zlpc; hi = b.zupc; }
        else continue;
        if (ax >= lo && ax <= hi && d1 * d1 + d2 * d2 < b.radius * b.radius) kill = true;
      } else if (b.geotype == 3) {
        double d1 = p.x - b.sph_center[0], d2 = p.y - b.sph_center[1], d3 = p.z - b.sph_center[2];
        if (d1 * d1 + d2 * d2 + d3 * d3 < b.radius * b.radius) kill = true;
      }
      if (kill) {
        p.nid = -1;
        absorb(a.gc, a.is, ipc, p.pid);
      }
    }
  }
  store_record(a.p + m, p);
}

// Deposit of a warp's particles, combined per cell.  Lane values v[NV] go to
// elements base + off(s) of an FP64 array; lanes of the same base (particles
// of one cell: neighbours in a cell-sorted buffer) are summed in shared
// memory and leave one atomic per node, lanes that share a cell with fewer
// than DEP_GROUP others add their own (fewer lanes than that do not pay for
// the pass over shared memory).  FP64 atomics to few addresses bound
// the deposit: with 24 of them a particle psolve1 took 6.07 ms per 16.8 M
// sorted particles (64^3 x 64 ppc), with about 2 it took 1.34 ms; charge
// (8 before) went from 2.38 to 0.32 ms.  Works for any order (unsorted
// buffers take the single-lane path).  `sm`: NV * DEP_STRIDE doubles of this
// warp.  All 32 lanes call it.
constexpr int DEP_GROUP = 4;
constexpr int DEP_STRIDE = 33;  // odd: lanes and values fall on different banks
constexpr int DEP_THREADS = 128;
template <int NV, class Off, class Add>
__device__ __forceinline__ void warp_deposit(double* sm, bool dep, int64_t base, const double (&v)[NV], Off off,
                                             Add add) {
  const int lane = threadIdx.x & 31;
  const unsigned long long key = dep ? (unsigned long long)base : ~(unsigned long long)lane;
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  const bool group = dep && __popc(peers) >= DEP_GROUP;
  if (dep && !group) {
#pragma unroll
    for (int s = 0; s < NV; s++) add(base + off(s), v[s]);
  }
  unsigned todo = __ballot_sync(0xffffffffu, group);
  if (!todo) return;
  if (group) {
#pragma unroll
    for (int s = 0; s < NV; s++) sm[s * DEP_STRIDE + lane] = v[s];
  }
  __syncwarp();
  // lane -> value s of the part of the warp [part * W, part * W + W)
  constexpr int P = 32 / NV, W = 32 / P;
  static_assert(P * W == 32, "the parts cover the warp");
  const int s = lane % NV, part = lane / NV;
  const double* row = sm + s * DEP_STRIDE + part * W;
  const int64_t mine = off(s);
  while (todo) {
    const int leader = __ffs(todo) - 1;
    const unsigned mask = __shfl_sync(0xffffffffu, peers, leader);
    const int64_t b = __shfl_sync(0xffffffffu, base, leader);
    todo &= ~mask;
    double t0 = 0.0, t1 = 0.0;
    if (part < P) {
      const unsigned m = mask >> (part * W);
#pragma unroll
      for (int j = 0; j < W; j += 2) {
        if (m >> j & 1u) t0 += row[j];
        if (m >> (j + 1) & 1u) t1 += row[j + 1];
      }
    }
    t0 += t1;
#pragma unroll
    for (int q = 1; q < P; q *= 2) t0 += __shfl_down_sync(0xffffffffu, t0, q * NV);
    if (lane < NV) add(b + mine, t0);
  }
  __syncwarp();
}

// psolve1, src/pcl2field/psolve1.F90:146-789: push with floor() indices and
// the zigzag current into the per-species scratch tj (wrk(TJX:TJZ)).
// The push of one live particle; its current leaves as the 12 node values J
// of cell (ib, jb, kb) when both segments lie in it (returns true), else
// straight to the scratch.
__device__ __forceinline__ bool psolve1_one(const PushArgs& a, int64_t m, emsesg_particle& p, double gustep,
                                            double qmp, int& ib, int& jb, int& kb, double (&J)[12]) {
  const emsesg_config* c = a.cfg;
  const double dxl = 0.0, dyl = 0.0, dzl = 0.0;
  const double dxu = c->nx, dyu = c->ny, dzu = c->nz;
  const double slx = c->nx, sly = c->ny, slz = c->nz;
  const double tslx = 2.0 * slx, tsly = 2.0 * sly, tslz = 2.0 * slz;
  const int ngx = c->nx, ngy = c->ny, ngz = c->nz;
  const double dngx = ngx, dngy = ngy, dngz = ngz;
  const double rustep = 1.0 / a.ustep;

  double xlocalb = p.x - dxl, ylocalb = p.y - dyl, zlocalb = p.z - dzl;
  ib = (int)floor(xlocalb);
  jb = (int)floor(ylocalb);
  kb = (int)floor(zlocalb);
  if (!cell_ok(c, ib, jb, kb)) {
    report_bad(a.status, a.diag, SITE_PSOLVE1, a.packed_base + m, ib + 100000LL * jb + 10000000000LL * kb);
    return false;
  }
  double xb = ib, yb = jb, zb = kb;
  int i1b = ib + 1, j1b = jb + 1, k1b = kb + 1;
  W8 w = weights(xlocalb - xb, ylocalb - yb, zlocalb - zb);
  gather_boris_move(a.node, c, p, ib, jb, kb, w, qmp, gustep);

  double xlocala, ylocala, zlocala, xa, ya, za, xr, yr, zr;
  int ia, ja, ka, i1a, j1a, k1a;
  int nud = 14;
  if (p.x < dxl) nud -= 1; else if (p.x >= dxu) nud += 1;
  if (p.y < dyl) nud -= 3; else if (p.y >= dyu) nud += 3;
  if (p.z < dzl) nud -= 9; else if (p.z >= dzu) nud += 9;
  if (nud == 14) {
    xlocala = p.x - dxl; ylocala = p.y - dyl; zlocala = p.z - dzl;
    ia = (int)floor(xlocala); ja = (int)floor(ylocala); ka = (int)floor(zlocala);
    xa = ia; ya = ja; za = ka;
    i1a = ia + 1; j1a = ja + 1; k1a = ka + 1;
    xr = (ib == ia) ? (xlocalb + xlocala) * 0.5 : fmax(xb, xa);
    yr = (jb == ja) ? (ylocalb + ylocala) * 0.5 : fmax(yb, ya);
    zr = (kb == ka) ? (zlocalb + zlocala) * 0.5 : fmax(zb, za);
  } else {
    const int32_t* nb = c->npbnd[a.is];
    p.nid = nborps_single(nb, p.x < dxl || p.x >= dxu, p.y < dyl || p.y >= dyu, p.z < dzl || p.z >= dzu);
    if (p.x < 0.0) {
      if (nb[0] == 0) { xlocala = p.x; p.x = p.x + slx; ia = -1; xa = -1.0; i1a = 0; xr = 0.0; }
      else if (nb[0] == 1) { p.x = -p.x; p.vx = -p.vx; xlocala = p.x; ia = 0; xa = 0.0; i1a = 1; xr = 0.0; }
      else { xlocala = -1.0; ia = -1; xa = -1.0; i1a = 0; xr = 0.0; }
    } else if (p.x >= slx) {
      if (nb[0] == 0) { xlocala = p.x - dxl; p.x = p.x - slx; ia = ngx; xa = dngx; i1a = ngx + 1; xr = dngx; }
      else if (nb[0] == 1) { p.x = tslx - p.x; p.vx = -p.vx; xlocala = p.x - dxl; ia = ngx - 1; xa = dngx - 1.0; i1a = ngx; xr = dngx; }
      else { xlocala = dngx + 1.0; ia = ngx; xa = dngx; i1a = ngx + 1; xr = dngx; }
    } else {
      xlocala = p.x - dxl; ia = (int)floor(xlocala); xa = ia; i1a = ia + 1;
      xr = (ib == ia) ? (xlocalb + xlocala) * 0.5 : fmax(xb, xa);
    }
    if (p.y < 0.0) {
      if (nb[1] == 0) { ylocala = p.y; p.y = p.y + sly; ja = -1; ya = -1.0; j1a = 0; yr = 0.0; }
      else if (nb[1] == 1) { p.y = -p.y; p.vy = -p.vy; ylocala = p.y; ja = 0; ya = 0.0; j1a = 1; yr = 0.0; }
      else { ylocala = -1.0; ja = -1; ya = -1.0; j1a = 0; yr = 0.0; }
    } else if (p.y >= sly) {
      if (nb[1] == 0) { ylocala = p.y - dyl; p.y = p.y - sly; ja = ngy; ya = dngy; j1a = ngy + 1; yr = dngy; }
      else if (nb[1] == 1) { p.y = tsly - p.y; p.vy = -p.vy; ylocala = p.y - dyl; ja = ngy - 1; ya = dngy - 1.0; j1a = ngy; yr = dngy; }
      else { ylocala = dngy + 1.0; ja = ngy; ya = dngy; j1a = ngy + 1; yr = dngy; }
    } else {
      ylocala = p.y - dyl; ja = (int)floor(ylocala); ya = ja; j1a = ja + 1;
      yr = (jb == ja) ? (ylocalb + ylocala) * 0.5 : fmax(yb, ya);
    }
    if (p.z < 0.0) {
      if (nb[2] == 0) { zlocala = p.z; p.z = p.z + slz; ka = -1; za = -1.0; k1a = 0; zr = 0.0; }
      else if (nb[2] == 1) { p.z = -p.z; p.vz = -p.vz; zlocala = p.z; ka = 0; za = 0.0; k1a = 1; zr = 0.0; }
      else { zlocala = -1.0; ka = -1; za = -1.0; k1a = 0; zr = 0.0; }
    } else if (p.z >= slz) {
      if (nb[2] == 0) { zlocala = p.z - dzl; p.z = p.z - slz; ka = ngz; za = dngz; k1a = ngz + 1; zr = dngz; }
      else if (nb[2] == 1) { p.z = tslz - p.z; p.vz = -p.vz; zlocala = p.z - dzl; ka = ngz - 1; za = dngz - 1.0; k1a = ngz; zr = dngz; }
      else { zlocala = dngz + 1.0; ka = ngz; za = dngz; k1a = ngz + 1; zr = dngz; }
    } else {
      zlocala = p.z - dzl; ka = (int)floor(zlocala); za = ka; k1a = ka + 1;
      zr = (kb == ka) ? (zlocalb + zlocala) * 0.5 : fmax(zb, za);
    }
    if (p.nid == -1) atomicAdd(&a.gc->nesc[a.is], 1);
  }

  // Internal boundary treatment 1, psolve1.F90:639-715.
  if (c->line_mode != 1) {
    for (int ipc = 0; ipc < c->npc; ipc++) {
      if (p.nid == -1) continue;
      const emsesg_body& b = c->body[ipc];
      if (b.geotype == 0 || b.geotype == 1) {
        double xlc = b.xlpc - dxl, xuc = b.xupc - dxl, ylc = b.ylpc - dyl, yuc = b.yupc - dyl;
        double zlc = b.zlpc - dzl, zuc = b.zupc - dzl;
        if (xlocalb >= xlc && xlocalb <= xuc && ylocalb >= ylc && ylocalb <= yuc && zlocalb >= zlc && zlocalb <= zuc) {
          xlocalb = xr; ylocalb = yr; zlocalb = zr;
        }
        if (xlocala >= xlc && xlocala <= xuc && ylocala >= ylc && ylocala <= yuc && zlocala >= zlc && zlocala <= zuc) {
          p.nid = -1;
          absorb(a.gc, a.is, ipc, p.pid);
          xlocala = xr; ylocala = yr; zlocala = zr;
        }
      } else if (b.geotype == 2) {
        double d1, d2, ax;
        if (b.cyl_align == 1) { d1 = p.y - b.cyl_axis[0]; d2 = p.z - b.cyl_axis[1]; ax = p.x; }
        else if (b.cyl_align == 2) { d1 = p.z - b.cyl_axis[0]; d2 = p.x - b.cyl_axis[1]; ax = p.y; }
        else if (b.cyl_align == 3) { d1 = p.x - b.cyl_axis[0]; d2 = p.y - b.cyl_axis[1]; ax = p.z; }
        else continue;
        if (ax >= b.cyl_edge[0] && ax <= b.cyl_edge[1] && d1 * d1 + d2 * d2 < b.radius * b.radius) {
          p.nid = -1;
          absorb(a.gc, a.is, ipc, p.pid);
        }
      } else if (b.geotype == 3) {
        double d1 = p.x - b.sph_center[0], d2 = p.y - b.sph_center[1], d3 = p.z - b.sph_center[2];
        if (d1 * d1 + d2 * d2 + d3 * d3 < b.radius * b.radius) {
          p.nid = -1;
          absorb(a.gc, a.is, ipc, p.pid);
        }
      }
    }
  }

  // Zigzag weights, psolve1.F90:717-757.
  double xd1 = (xr + xlocalb) * 0.5 - xb, yd1 = (yr + ylocalb) * 0.5 - yb, zd1 = (zr + zlocalb) * 0.5 - zb;
  double vvx1 = (xr - xlocalb) * rustep, vvy1 = (yr - ylocalb) * rustep, vvz1 = (zr - zlocalb) * rustep;
  double vx1w4 = yd1 * zd1, vx1w2 = yd1 - vx1w4, vx1w3 = zd1 - vx1w4, vx1w1 = 1.0 - yd1 - vx1w3;
  double vy1w4 = xd1 * zd1, vy1w2 = xd1 - vy1w4, vy1w3 = zd1 - vy1w4, vy1w1 = 1.0 - xd1 - vy1w3;
  double vz1w4 = xd1 * yd1, vz1w2 = xd1 - vz1w4, vz1w3 = yd1 - vz1w4, vz1w1 = 1.0 - xd1 - vz1w3;
  double xd2 = (xlocala + xr) * 0.5 - xa, yd2 = (ylocala + yr) * 0.5 - ya, zd2 = (zlocala + zr) * 0.5 - za;
  double vvx2 = (xlocala - xr) * rustep, vvy2 = (ylocala - yr) * rustep, vvz2 = (zlocala - zr) * rustep;
  double vx2w4 = yd2 * zd2, vx2w2 = yd2 - vx2w4, vx2w3 = zd2 - vx2w4, vx2w1 = 1.0 - yd2 - vx2w3;
  double vy2w4 = xd2 * zd2, vy2w2 = xd2 - vy2w4, vy2w3 = zd2 - vy2w4, vy2w1 = 1.0 - xd2 - vy2w3;
  double vz2w4 = xd2 * yd2, vz2w2 = xd2 - vz2w4, vz2w3 = yd2 - vz2w4, vz2w1 = 1.0 - xd2 - vz2w3;

  store_record(a.p + m, p);
  if (ia == ib && ja == jb && ka == kb) {
    J[0] = vvx1 * vx1w1 + vvx2 * vx2w1; J[1] = vvx1 * vx1w2 + vvx2 * vx2w2;
    J[2] = vvx1 * vx1w3 + vvx2 * vx2w3; J[3] = vvx1 * vx1w4 + vvx2 * vx2w4;
    J[4] = vvy1 * vy1w1 + vvy2 * vy2w1; J[5] = vvy1 * vy1w2 + vvy2 * vy2w2;
    J[6] = vvy1 * vy1w3 + vvy2 * vy2w3; J[7] = vvy1 * vy1w4 + vvy2 * vy2w4;
    J[8] = vvz1 * vz1w1 + vvz2 * vz2w1; J[9] = vvz1 * vz1w2 + vvz2 * vz2w2;
    J[10] = vvz1 * vz1w3 + vvz2 * vz2w3; J[11] = vvz1 * vz1w4 + vvz2 * vz2w4;
    return true;
  }
  const FieldDesc& f = a.fa;
  double* t = a.tj;
  // The 24 scatter-adds of psolve1.F90:759-789; all indices lie in -1..n+1.
  atomicAdd(&t[f.at(JX, ib, jb, kb)], vvx1 * vx1w1);
  atomicAdd(&t[f.at(JY, ib, jb, kb)], vvy1 * vy1w1);
  atomicAdd(&t[f.at(JZ, ib, jb, kb)], vvz1 * vz1w1);
  atomicAdd(&t[f.at(JX, ib, j1b, kb)], vvx1 * vx1w2);
  atomicAdd(&t[f.at(JY, i1b, jb, kb)], vvy1 * vy1w2);
  atomicAdd(&t[f.at(JZ, i1b, jb, kb)], vvz1 * vz1w2);
  atomicAdd(&t[f.at(JX, ib, jb, k1b)], vvx1 * vx1w3);
  atomicAdd(&t[f.at(JY, ib, jb, k1b)], vvy1 * vy1w3);
  atomicAdd(&t[f.at(JZ, ib, j1b, kb)], vvz1 * vz1w3);
  atomicAdd(&t[f.at(JX, ib, j1b, k1b)], vvx1 * vx1w4);
  atomicAdd(&t[f.at(JY, i1b, jb, k1b)], vvy1 * vy1w4);
  atomicAdd(&t[f.at(JZ, i1b, j1b, kb)], vvz1 * vz1w4);
  atomicAdd(&t[f.at(JX, ia, ja, ka)], vvx2 * vx2w1);
  atomicAdd(&t[f.at(JY, ia, ja, ka)], vvy2 * vy2w1);
  atomicAdd(&t[f.at(JZ, ia, ja, ka)], vvz2 * vz2w1);
  atomicAdd(&t[f.at(JX, ia, j1a, ka)], vvx2 * vx2w2);
  atomicAdd(&t[f.at(JY, i1a, ja, ka)], vvy2 * vy2w2);
  atomicAdd(&t[f.at(JZ, i1a, ja, ka)], vvz2 * vz2w2);
  atomicAdd(&t[f.at(JX, ia, ja, k1a)], vvx2 * vx2w3);
  atomicAdd(&t[f.at(JY, ia, ja, k1a)], vvy2 * vy2w3);
  atomicAdd(&t[f.at(JZ, ia, j1a, ka)], vvz2 * vz2w3);
  atomicAdd(&t[f.at(JX, ia, j1a, k1a)], vvx2 * vx2w4);
  atomicAdd(&t[f.at(JY, i1a, ja, k1a)], vvy2 * vy2w4);
  atomicAdd(&t[f.at(JZ, i1a, j1a, ka)], vvz2 * vz2w4);
  return false;
}

// One thread per particle, the deposits combined per warp and cell.
__global__ void __launch_bounds__(DEP_THREADS) k_psolve1(PushArgs a) {
  __shared__ double sm[DEP_THREADS / 32][12 * DEP_STRIDE];
  const int64_t m = (int64_t)blockIdx.x * DEP_THREADS + threadIdx.x;
  int ib = 0, jb = 0, kb = 0;
  double J[12];
  bool dep = false;
  if (m < a.n && m < *a.count) {
    emsesg_particle p = load_record(a.p + m);
    double gustep, qmp;
    if (push_status(a, m, p, gustep, qmp)) dep = psolve1_one(a, m, p, gustep, qmp, ib, jb, kb, J);
    else store_record(a.p + m, p);
  }
  const FieldDesc& f = a.fa;
  // value s: component s / 4 on the node (0,u,v), (u,0,v) or (u,v,0) of the cell
  warp_deposit<12>(
      sm[threadIdx.x >> 5], dep, f.at(0, ib, jb, kb), J,
      [&](int s) {
        const int d = s >> 2, u = s & 1, v = (s >> 1) & 1;
        return f.at(d, f.lo + (d == 0 ? 0 : u), f.lo + (d == 0 ? u : d == 1 ? 0 : v), f.lo + (d == 2 ? 0 : v));
      },
      [&](int64_t e, double x) { atomicAdd(&a.tj[e], x); });
}

// aj += wrk(TJ)*q (and ajdg), psolve1.F90:793-817, over -1..n+1.
__global__ void k_flush_tj(const double* __restrict__ tj, double* aj, double* ajdg, FieldDesc fa, FieldDesc fj,
                           int nx, int ny, int nz, double qs, int iss, int do_dg) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t ex = nx + 3, ey = ny + 3, ez = nz + 3;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i - 1, j = at.j - 1, k = at.k - 1;
  for (int d = 0; d < 3; d++) {
    double v = tj[fa.at(d, i, j, k)];
    aj[fa.at(d, i, j, k)] = aj[fa.at(d, i, j, k)] + v * qs;
    if (do_dg) ajdg[fj.at(iss + d, i, j, k)] = ajdg[fj.at(iss + d, i, j, k)] + v * qs;
  }
}

// chgacm update after the species loop, psolve2.F90:537-543.
__global__ void k_chgacm(const emsesg_config* c, emsesg_counter* gc) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  for (int is = 0; is < c->nspec; is++)
    for (int ipc = 0; ipc < c->npc; ipc++)
      if (c->body[ipc].ncond > 0) {
        double add = (double)gc->influx[is][ipc] * c->q[is] * c->body[ipc].sqdscaled;
        gc->chgacm[ipc][0] = gc->chgacm[ipc][0] + add;
        gc->chgacm[ipc][1] = gc->chgacm[ipc][1] + add;
      }
}

// grdcrt, src/field/grdcrt.F90:156-169 and :214-230, one thread per node.
__global__ void k_grdcrt(const double* __restrict__ eb, double* __restrict__ node, FieldDesc fe, int nx, int ny,
                         int nz, double e0x, double e0y, double e0z, double b0x, double b0y, double b0z) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t ex = nx + 1, ey = ny + 1, ez = nz + 1;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i, j = at.j, k = at.k;
  double* o = node + 8 * ((int64_t)i + (ex + 1) * ((int64_t)j + (ey + 1) * k));
  o[EX] = 0.5 * (eb[fe.at(EX, i, j, k)] + eb[fe.at(EX, i - 1, j, k)]) + e0x;
  o[EY] = 0.5 * (eb[fe.at(EY, i, j, k)] + eb[fe.at(EY, i, j - 1, k)]) + e0y;
  o[EZ] = 0.5 * (eb[fe.at(EZ, i, j, k)] + eb[fe.at(EZ, i, j, k - 1)]) + e0z;
  o[BX] = 0.25 * (eb[fe.at(BX, i, j, k)] + eb[fe.at(BX, i, j - 1, k)] + eb[fe.at(BX, i, j, k - 1)] +
                   eb[fe.at(BX, i, j - 1, k - 1)]) + b0x;
  o[BY] = 0.25 * (eb[fe.at(BY, i, j, k)] + eb[fe.at(BY, i - 1, j, k)] + eb[fe.at(BY, i, j, k - 1)] +
                   eb[fe.at(BY, i - 1, j, k - 1)]) + b0y;
  o[BZ] = 0.25 * (eb[fe.at(BZ, i, j, k)] + eb[fe.at(BZ, i - 1, j, k)] + eb[fe.at(BZ, i, j - 1, k)] +
                   eb[fe.at(BZ, i - 1, j - 1, k)]) + b0z;
  o[6] = 0.0;
  o[7] = 0.0;
}

// Writes the node field into the reference wrk layout (EX..BZ at 0..n).
__global__ void k_node_to_wrk(const double* __restrict__ node, double* wrk, FieldDesc fw, int nx, int ny, int nz) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t ex = nx + 1, ey = ny + 1, ez = nz + 1;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i, j = at.j, k = at.k;
  int64_t nd = (int64_t)i + (ex + 1) * ((int64_t)j + (ey + 1) * k);
  for (int cc = 0; cc < 6; cc++) wrk[fw.at(cc, i, j, k)] = node[8 * nd + cc];
}

struct ChargeArgs {
  emsesg_particle* p;
  int64_t n;
  const int64_t* count;
  int is, nspec, func;
  double q;
  double *rho, *rhodg, *rhobk, *rhobksp;
  FieldDesc fr, fd;
  const emsesg_config* cfg;
  int* status;
  long long* diag;
};

__device__ __forceinline__ void distribute(double* rh, const FieldDesc& f, int cc, int i, int j, int k, double qc,
                                           const W8& w) {
  atomicAdd(&rh[f.at(cc, i, j, k + 1)], w.v1 * qc);
  atomicAdd(&rh[f.at(cc, i + 1, j, k + 1)], w.v2 * qc);
  atomicAdd(&rh[f.at(cc, i + 1, j + 1, k + 1)], w.v3 * qc);
  atomicAdd(&rh[f.at(cc, i, j + 1, k + 1)], w.v4 * qc);
  atomicAdd(&rh[f.at(cc, i, j, k)], w.v5 * qc);
  atomicAdd(&rh[f.at(cc, i + 1, j, k)], w.v6 * qc);
  atomicAdd(&rh[f.at(cc, i + 1, j + 1, k)], w.v7 * qc);
  atomicAdd(&rh[f.at(cc, i, j + 1, k)], w.v8 * qc);
}

// Charge of one particle record (charge.F90:53-146): the CIC weights v times
// the charge of an ordinary particle (returns true: left to the caller);
// absorbed particles and anti-particles to be accumulated go straight to
// their arrays.
__device__ __forceinline__ bool charge_one(const ChargeArgs& a, int64_t m, int& i, int& j, int& k, double (&v)[8]) {
  const emsesg_particle p = load_record(a.p + m);
  if (p.nid == -1) return false;
  double xlocal = p.x, ylocal = p.y, zlocal = p.z;
  i = (int)xlocal;
  j = (int)ylocal;
  k = (int)zlocal;
  const emsesg_config* c = a.cfg;
  if (i < -1 || j < -1 || k < -1 || i > c->nx || j > c->ny || k > c->nz) {
    report_bad(a.status, a.diag, SITE_CHARGE, m, i + 100000LL * j + 10000000000LL * k);
    return false;
  }
  W8 w = weights(xlocal - i, ylocal - j, zlocal - k);
  int func = a.func;
  if (p.preside >= 0) {
    v[0] = w.v5 * a.q; v[1] = w.v6 * a.q; v[2] = w.v8 * a.q; v[3] = w.v7 * a.q;
    v[4] = w.v1 * a.q; v[5] = w.v2 * a.q; v[6] = w.v4 * a.q; v[7] = w.v3 * a.q;
    return true;
  }
  if (p.preside == EMSESG_PCL_TO_BE_ACCUMULATED || p.preside == EMSESG_PCL_TO_BE_ACCUMULATED_AS_ANTIPCL) {
    double qq = p.preside == EMSESG_PCL_TO_BE_ACCUMULATED ? a.q : -a.q;
    distribute(a.rhobk, a.fr, 0, i, j, k, qq, w);
    distribute(a.rhobksp + (int64_t)a.is * a.fr.size(), a.fr, 0, i, j, k, qq, w);
    if (func == 1 || func == 2) {
      if (func == 2 && p.preside == EMSESG_PCL_TO_BE_ACCUMULATED_AS_ANTIPCL) distribute(a.rhodg, a.fd, a.is, i, j, k, qq, w);
      distribute(a.rhodg, a.fd, a.nspec + a.is, i, j, k, qq, w);
    }
    a.p[m].nid = -1;
    a.p[m].preside = 0;
  }
  return false;
}

// One thread per particle, the deposits combined per warp and cell.  rhodg
// has the extents of rho, so one node index e serves both (rhodg: e * nc + is).
__global__ void __launch_bounds__(DEP_THREADS) k_charge(ChargeArgs a) {
  __shared__ double sm[DEP_THREADS / 32][8 * DEP_STRIDE];
  const int64_t m = (int64_t)blockIdx.x * DEP_THREADS + threadIdx.x;
  int i = 0, j = 0, k = 0;
  double v[8];
  const bool dep = m < a.n && m < *a.count && charge_one(a, m, i, j, k, v);
  const FieldDesc& f = a.fr;
  // value s: the corner (s & 1, s >> 1 & 1, s >> 2)
  warp_deposit<8>(
      sm[threadIdx.x >> 5], dep, f.at(0, i, j, k), v,
      [&](int s) { return f.at(0, f.lo + (s & 1), f.lo + ((s >> 1) & 1), f.lo + (s >> 2)); },
      [&](int64_t e, double x) {
        if (a.func == 0 || a.func == 2) atomicAdd(&a.rho[e], x);
        if (a.func == 1 || a.func == 2) atomicAdd(&a.rhodg[e * a.fd.nc + a.is], x);
      });
}

// rhoupd, src/field/rhoupd.F90:40-49.
__global__ void k_rhoupd(double* rho, const double* __restrict__ aj, FieldDesc fr, FieldDesc fa, int nx, int ny,
                         int nz) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t ex = nx + 1, ey = ny + 1, ez = nz + 1;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i, j = at.j, k = at.k;
  rho[fr.at(0, i, j, k)] = rho[fr.at(0, i, j, k)] -
      (aj[fa.at(JX, i, j, k)] - aj[fa.at(JX, i - 1, j, k)] + aj[fa.at(JY, i, j, k)] - aj[fa.at(JY, i, j - 1, k)] +
       aj[fa.at(JZ, i, j, k)] - aj[fa.at(JZ, i, j, k - 1)]) * 2.0;
}

// bfield, src/field/bfield.F90:37-53: B(i,j,k) for i,j,k in -1..n, from E
// (the reference's statement order; B written, E read only).
__global__ void k_bfield(double* eb, FieldDesc f, int nx, int ny, int nz) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t ex = nx + 2, ey = ny + 2, ez = nz + 2;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i - 1, j = at.j - 1, k = at.k - 1;
  eb[f.at(BX, i, j, k)] = eb[f.at(BX, i, j, k)] + eb[f.at(EY, i, j, k + 1)] - eb[f.at(EY, i, j, k)] -
                          eb[f.at(EZ, i, j + 1, k)] + eb[f.at(EZ, i, j, k)];
  eb[f.at(BY, i, j, k)] = eb[f.at(BY, i, j, k)] + eb[f.at(EZ, i + 1, j, k)] - eb[f.at(EZ, i, j, k)] -
                          eb[f.at(EX, i, j, k + 1)] + eb[f.at(EX, i, j, k)];
  eb[f.at(BZ, i, j, k)] = eb[f.at(BZ, i, j, k)] + eb[f.at(EX, i, j + 1, k)] - eb[f.at(EX, i, j, k)] -
                          eb[f.at(EY, i + 1, j, k)] + eb[f.at(EY, i, j, k)];
}

// efield, src/field/efield.F90:54-70 (no lumped elements): E(i,j,k) for
// i,j,k in 0..n, from B and J (E written, B and J read only).
__global__ void k_efield(double* eb, const double* __restrict__ aj, FieldDesc f, FieldDesc fa, int nx, int ny,
                         int nz, double tcs, double dlt) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t ex = nx + 1, ey = ny + 1, ez = nz + 1;
  if (t >= ex * ey * ez) return;
  const Node3 at = node3(t, ex, ey);
  const int i = at.i, j = at.j, k = at.k;
  eb[f.at(EX, i, j, k)] = eb[f.at(EX, i, j, k)] +
                          tcs * (eb[f.at(BZ, i, j, k)] - eb[f.at(BZ, i, j - 1, k)] - eb[f.at(BY, i, j, k)] +
                                 eb[f.at(BY, i, j, k - 1)]) -
                          dlt * aj[fa.at(JX, i, j, k)];
  eb[f.at(EY, i, j, k)] = eb[f.at(EY, i, j, k)] +
                          tcs * (eb[f.at(BX, i, j, k)] - eb[f.at(BX, i, j, k - 1)] - eb[f.at(BZ, i, j, k)] +
                                 eb[f.at(BZ, i - 1, j, k)]) -
                          dlt * aj[fa.at(JY, i, j, k)];
  eb[f.at(EZ, i, j, k)] = eb[f.at(EZ, i, j, k)] +
                          tcs * (eb[f.at(BY, i, j, k)] - eb[f.at(BY, i - 1, j, k)] - eb[f.at(BX, i, j, k)] +
                                 eb[f.at(BX, i, j - 1, k)]) -
                          dlt * aj[fa.at(JZ, i, j, k)];
}

// Sum of v_d^2 of live particles (energy.F90:38-43); FP64 block partials.
__global__ void k_energy(const emsesg_particle* __restrict__ p, int64_t n, const int64_t* count, double* out) {
  __shared__ double s[3][256];
  double t[3] = {0, 0, 0};
  int64_t nn = min(n, *count);
  for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < nn; m += (int64_t)gridDim.x * blockDim.x) {
    const emsesg_particle q = load_record(p + m);
    if (q.nid == -1) continue;
    t[0] += q.vx * q.vx;
    t[1] += q.vy * q.vy;
    t[2] += q.vz * q.vz;
  }
  for (int d = 0; d < 3; d++) s[d][threadIdx.x] = t[d];
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int d = 0; d < 3; d++) s[d][threadIdx.x] += s[d][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int d = 0; d < 3; d++) atomicAdd(&out[d], s[d][0]);
}

// Canonical sort key: tile-major cell key of int() of the position, clamped.
__device__ __forceinline__ uint32_t sort_key(const emsesg_config* c, double x, double y, double z, const int* t,
                                             const int* nt) {
  int ci[3];
  double pos[3] = {x, y, z};
  int n[3] = {c->nx, c->ny, c->nz};
  for (int d = 0; d < 3; d++) {
    int v = pos[d] < 0.0 ? 0 : (int)fmin(pos[d], (double)(n[d] - 1));
    ci[d] = min(max(v, 0), n[d] - 1);
  }
  uint32_t tile = (uint32_t)(ci[0] / t[0]) + (uint32_t)nt[0] * ((uint32_t)(ci[1] / t[1]) + (uint32_t)nt[1] * (uint32_t)(ci[2] / t[2]));
  uint32_t in = (uint32_t)(ci[0] % t[0]) + (uint32_t)t[0] * ((uint32_t)(ci[1] % t[1]) + (uint32_t)t[1] * (uint32_t)(ci[2] % t[2]));
  return tile * (uint32_t)(t[0] * t[1] * t[2]) + in;
}

struct KeyArgs { int t[3], nt[3]; };

__global__ void k_make_keys(const emsesg_particle* __restrict__ p, int64_t n, const emsesg_config* c, KeyArgs ka,
                            uint32_t* keys, uint32_t* vals) {
  int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const Half h = load_half(p + m, 0);
  keys[m] = sort_key(c, word(h.w[0]), word(h.w[1]), word(h.w[2]), ka.t, ka.nt);
  vals[m] = (uint32_t)m;
}

// dst[m] = src[idx[m]]: two threads a record, one half each, so that a warp
// writes 16 whole records in a row (one thread a record, in pieces of 8
// bytes: 0.64 ms per 16.8 M records; 0.33 ms this way, 6.5 TB/s).
__global__ void k_gather_particles(const emsesg_particle* __restrict__ src, emsesg_particle* __restrict__ dst,
                                   const uint32_t* __restrict__ idx, int64_t n) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t m = t >> 1;
  if (m >= n) return;
  const int h = (int)(t & 1);
  store_half(dst + m, h, load_half(src + idx[m], h));
}

__global__ void k_live_flags(const emsesg_particle* __restrict__ p, int64_t n, uint32_t* flags) {
  int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  flags[m] = p[m].nid != -1 ? 1u : 0u;
}

// Live records to their places, two threads a record (one half each).
__global__ void k_compact_scatter(const emsesg_particle* __restrict__ src, emsesg_particle* __restrict__ dst,
                                  const uint32_t* __restrict__ pos, int64_t n) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t m = t >> 1;
  const int h = (int)(t & 1);
  Half r{};
  if (m < n) r = load_half(src + m, h);
  // nid sits in the second half, held by the odd lane of the pair
  const int32_t nid = __shfl_sync(0xffffffffu, lo32(r.w[3]), (threadIdx.x & 31) | 1);
  if (m < n && nid != -1) store_half(dst + pos[m], h, r);
}

__global__ void k_injected_flags(const emsesg_particle* __restrict__ p, int64_t n, const int64_t* count,
                                 uint32_t* flags) {
  int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  flags[m] = (m < *count && p[m].preside == EMSESG_PCL_INJECTED) ? 1u : 0u;
}

__global__ void k_advance(int64_t* pos, const uint32_t* total) { *pos += *total; }

__global__ void k_set_count(int64_t* count, const uint32_t* total) { *count = *total; }

// Synthetic plasma, same streams as orc_load_plasma (oracle/emses_oracle.cpp).
// Particles m0 .. m0+n-1 of species `is` into p[0 .. n).
__global__ void k_load_plasma(emsesg_particle* p, int64_t m0, int64_t n, int ppc, int nx, int ny, int is,
                              uint64_t seed, double vth, double vdx, double vdy, double vdz) {
  const int64_t loc = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (loc >= n) return;
  const int64_t m = m0 + loc;
  int64_t cell = m / ppc;
  int i = (int)(cell % nx), j = (int)((cell / nx) % ny), k = (int)(cell / ((int64_t)nx * ny));
  uint64_t st = 1000 + is;
  double u[8];
  for (int s = 0; s < 7; s++) u[s] = hash_u01(seed, st, (uint64_t)m * 8 + s);
  const double twopi = 6.283185307179586;
  emsesg_particle q;
  q.x = i + u[0];
  q.y = j + u[1];
  q.z = k + u[2];
  double r1 = sqrt(-2.0 * log(1.0 - u[3]));
  double r2 = sqrt(-2.0 * log(1.0 - u[5]));
  q.vx = vth * r1 * cos(twopi * u[4]) + vdx;
  q.vy = vth * r1 * sin(twopi * u[4]) + vdy;
  q.vz = vth * r2 * cos(twopi * u[6]) + vdz;
  q.pid = 0;
  q.preside = 0;
  q.nid = 0;
  q.spec = is + 1;
  p[loc] = q;
}

inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

}  // namespace

int download_wrk(emsesg_ctx* ctx, double* host) {
  FieldDesc fw = field_desc(ctx->cfg, EMSESG_FIELD_WRK);
  EMSESG_CUDA(ctx, cudaMemsetAsync(ctx->field[EMSESG_FIELD_WRK], 0, fw.size() * sizeof(double), ctx->stream));
  int64_t nn = (int64_t)(ctx->cfg.nx + 1) * (ctx->cfg.ny + 1) * (ctx->cfg.nz + 1);
  EMSESG_LAUNCH(ctx, "node_to_wrk", k_node_to_wrk, nblk(nn), 256, 0, ctx->node64, ctx->field[EMSESG_FIELD_WRK], fw,
                ctx->cfg.nx, ctx->cfg.ny, ctx->cfg.nz);
  EMSESG_CUDA(ctx, cudaMemcpyAsync(host, ctx->field[EMSESG_FIELD_WRK], fw.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  EMSESG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMSESG_OK;
}

}  // namespace emsesg

using namespace emsesg;


namespace {

int check_ps(emsesg_ctx* ctx, int ps) {
  if (!ctx) return EMSESG_ERR_ARG;
  if (ps == 2) return set_error(ctx, EMSESG_ERR_UNSUPPORTED, "ps=2 (helper subdomain) is not supported on one rank");
  if (ps != 1) return set_error(ctx, EMSESG_ERR_ARG, "ps must be 1");
  return EMSESG_OK;
}

int64_t max_count(emsesg_ctx* ctx) {
  int64_t m = 0;
  for (int is = 0; is < ctx->cfg.nspec; is++) m = std::max(m, ctx->seg.capacity[is]);
  return m;
}

// Ordinals of injected particles for the pre-drawn random stream.
int prepare_ordinals(emsesg_ctx* ctx, int is, const uint32_t** ord) {
  *ord = nullptr;
  if (ctx->cfg.rng_mode != 1) return EMSESG_OK;
  int rc = ensure_sort_scratch(ctx, max_count(ctx));
  if (rc) return rc;
  int64_t n = ctx->totalp[is];
  uint32_t* flags = ctx->sort.keys[1];
  EMSESG_LAUNCH(ctx, "injected_flags", k_injected_flags, nblk(n), 256, 0, ctx->pbuf + ctx->seg.base[is], n,
                ctx->d_count + is, flags);
  rc = exclusive_scan_u32(ctx, flags, n);
  if (rc) return rc;
  *ord = flags;
  return EMSESG_OK;
}

int advance_randoms(emsesg_ctx* ctx, int is) {
  if (ctx->cfg.rng_mode != 1) return EMSESG_OK;
  // total injected = scan total, left by exclusive_scan_u32 in scan_tmp[0]
  EMSESG_LAUNCH(ctx, "advance_randoms", k_advance, 1, 1, 0, ctx->d_rand_pos, ctx->sort.scan_tmp);
  return EMSESG_OK;
}

PushArgs push_args(emsesg_ctx* ctx, int is, int ustep) {
  PushArgs a{};
  a.p = ctx->pbuf + ctx->seg.base[is];
  a.n = ctx->totalp[is];
  a.count = ctx->d_count + is;
  a.is = is;
  int64_t pb = 0;
  for (int s = 0; s < is; s++) pb += ctx->totalp[s];
  a.packed_base = pb;
  a.node = ctx->node64;
  a.cfg = ctx->d_cfg;
  a.ustep = ustep;
  a.seed = ctx->cfg.rng_seed;
  a.stream = ctx->rng_stream;
  a.randoms = ctx->d_randoms;
  a.nrand = ctx->n_randoms;
  a.rand_pos = ctx->d_rand_pos;
  a.gc = ctx->d_counter;
  a.status = ctx->d_status;
  a.diag = ctx->d_diag;
  a.tj = ctx->tj;
  a.fa = field_desc(ctx->cfg, EMSESG_FIELD_AJ);
  return a;
}

}  // namespace

extern "C" int emsesg_grdcrt(emsesg_ctx* ctx, int ps) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if ((rc = apply_pending_eb(ctx))) return rc;
  const emsesg_config& c = ctx->cfg;
  int64_t nn = (int64_t)(c.nx + 1) * (c.ny + 1) * (c.nz + 1);
  EMSESG_LAUNCH(ctx, "grdcrt", k_grdcrt, nblk(nn), 256, 0, ctx->field[EMSESG_FIELD_EB], ctx->node64,
                field_desc(c, EMSESG_FIELD_EB), c.nx, c.ny, c.nz, c.e0[0], c.e0[1], c.e0[2], c.b0[0], c.b0[1],
                c.b0[2]);
  return EMSESG_OK;
}

static int finish_push(emsesg_ctx* ctx, emsesg_counter* gcount) {
  EMSESG_LAUNCH(ctx, "chgacm", k_chgacm, 1, 32, 0, ctx->d_cfg, ctx->d_counter);
  ctx->rng_stream++;
  if (gcount) {
    int rc = emsesg_get_counters(ctx, gcount);
    if (rc) return rc;
    return emsesg_synchronize(ctx);
  }
  return EMSESG_OK;
}

extern "C" int emsesg_psolve2(emsesg_ctx* ctx, int ps, int ustep, emsesg_counter* gcount) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if (ustep < 1) return set_error(ctx, EMSESG_ERR_ARG, "ustep must be >= 1");
  if (gcount && (rc = emsesg_set_counters(ctx, gcount))) return rc;
  for (int is = 0; is < ctx->cfg.nspec; is++) {
    if (ctx->totalp[is] == 0) continue;
    const uint32_t* ord;
    if ((rc = prepare_ordinals(ctx, is, &ord))) return rc;
    PushArgs a = push_args(ctx, is, ustep);
    a.ordinal = ord;
    EMSESG_LAUNCH(ctx, "psolve2", k_psolve2, nblk(a.n), 256, 0, a);
    if ((rc = advance_randoms(ctx, is))) return rc;
  }
  return finish_push(ctx, gcount);
}

extern "C" int emsesg_positn(emsesg_ctx* ctx, int ps, int ustep, emsesg_counter* gcount) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if (ustep < 1) return set_error(ctx, EMSESG_ERR_ARG, "ustep must be >= 1");
  if (gcount && (rc = emsesg_set_counters(ctx, gcount))) return rc;
  for (int is = 0; is < ctx->cfg.nspec; is++) {
    if (ctx->totalp[is] == 0) continue;
    const uint32_t* ord;
    if ((rc = prepare_ordinals(ctx, is, &ord))) return rc;
    PushArgs a = push_args(ctx, is, ustep);
    a.ordinal = ord;
    EMSESG_LAUNCH(ctx, "positn", k_positn, nblk(a.n), 256, 0, a);
    if ((rc = advance_randoms(ctx, is))) return rc;
  }
  ctx->rng_stream++;
  if (gcount) {
    if ((rc = emsesg_get_counters(ctx, gcount))) return rc;
    return emsesg_synchronize(ctx);
  }
  return EMSESG_OK;
}

extern "C" int emsesg_psolve1(emsesg_ctx* ctx, int ps, int ustep, int func, emsesg_counter* gcount) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if (ustep < 1) return set_error(ctx, EMSESG_ERR_ARG, "ustep must be >= 1");
  if (gcount && (rc = emsesg_set_counters(ctx, gcount))) return rc;
  const emsesg_config& c = ctx->cfg;
  FieldDesc fa = field_desc(c, EMSESG_FIELD_AJ), fj = field_desc(c, EMSESG_FIELD_AJDG);
  int64_t ng = (int64_t)(c.nx + 3) * (c.ny + 3) * (c.nz + 3);
  for (int is = 0; is < c.nspec; is++) {
    // wrk(TJX:TJZ, :, :, :) = 0, psolve1.F90:143
    EMSESG_CUDA(ctx, cudaMemsetAsync(ctx->tj, 0, fa.size() * sizeof(double), ctx->stream));
    if (ctx->totalp[is] > 0) {
      const uint32_t* ord;
      if ((rc = prepare_ordinals(ctx, is, &ord))) return rc;
      PushArgs a = push_args(ctx, is, ustep);
      a.ordinal = ord;
      EMSESG_LAUNCH(ctx, "psolve1", k_psolve1, nblk(a.n, DEP_THREADS), DEP_THREADS, 0, a);
      if ((rc = advance_randoms(ctx, is))) return rc;
    }
    EMSESG_LAUNCH(ctx, "flush_tj", k_flush_tj, nblk(ng), 256, 0, ctx->tj, ctx->field[EMSESG_FIELD_AJ],
                  ctx->field[EMSESG_FIELD_AJDG], fa, fj, c.nx, c.ny, c.nz, c.q[is], is * 3, func == 1 ? 1 : 0);
  }
  return finish_push(ctx, gcount);
}

extern "C" int emsesg_charge(emsesg_ctx* ctx, int ps, int func) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if (func < 0 || func > 2) return set_error(ctx, EMSESG_ERR_ARG, "func must be 0, 1 or 2");
  const emsesg_config& c = ctx->cfg;
  if (func == 0 || func == 2) EMSESG_CUDA(ctx, cudaMemsetAsync(ctx->field[EMSESG_FIELD_RHO], 0,
                                                               field_desc(c, EMSESG_FIELD_RHO).size() * sizeof(double), ctx->stream));
  if (func == 1 || func == 2) EMSESG_CUDA(ctx, cudaMemsetAsync(ctx->field[EMSESG_FIELD_RHODG], 0,
                                                               field_desc(c, EMSESG_FIELD_RHODG).size() * sizeof(double), ctx->stream));
  for (int is = 0; is < c.nspec; is++) {
    if (ctx->totalp[is] == 0) continue;
    ChargeArgs a{};
    a.p = ctx->pbuf + ctx->seg.base[is];
    a.n = ctx->totalp[is];
    a.count = ctx->d_count + is;
    a.is = is;
    a.nspec = c.nspec;
    a.func = func;
    a.q = c.q[is];
    a.rho = ctx->field[EMSESG_FIELD_RHO];
    a.rhodg = ctx->field[EMSESG_FIELD_RHODG];
    a.rhobk = ctx->field[EMSESG_FIELD_RHOBK];
    a.rhobksp = ctx->field[EMSESG_FIELD_RHOBKSP];
    a.fr = field_desc(c, EMSESG_FIELD_RHO);
    a.fd = field_desc(c, EMSESG_FIELD_RHODG);
    a.cfg = ctx->d_cfg;
    a.status = ctx->d_status;
    a.diag = ctx->d_diag;
    EMSESG_LAUNCH(ctx, "charge", k_charge, nblk(a.n, DEP_THREADS), DEP_THREADS, 0, a);
  }
  return EMSESG_OK;
}

extern "C" int emsesg_reduce_rho(emsesg_ctx* ctx, int field) {
  if (!ctx) return EMSESG_ERR_ARG;
  if (field != EMSESG_FIELD_RHO && field != EMSESG_FIELD_RHODG && field != EMSESG_FIELD_RHOBK &&
      field != EMSESG_FIELD_RHOBKSP)
    return set_error(ctx, EMSESG_ERR_ARG, "reduce_rho takes a rho-type field");
  FieldDesc f = field_desc(ctx->cfg, field);
  int narr = field == EMSESG_FIELD_RHOBKSP ? ctx->cfg.nspec : 1;
  for (int a = 0; a < narr; a++) {
    int rc = run_fold(ctx, ctx->field[field] + (int64_t)a * f.size(), f, 0, "reduce_rho");
    if (rc) return rc;
  }
  return EMSESG_OK;
}

extern "C" int emsesg_reduce_aj(emsesg_ctx* ctx) {
  if (!ctx) return EMSESG_ERR_ARG;
  return run_fold(ctx, ctx->field[EMSESG_FIELD_AJ], field_desc(ctx->cfg, EMSESG_FIELD_AJ), 1, "reduce_aj");
}

extern "C" int emsesg_reduce_ajdg(emsesg_ctx* ctx) {
  if (!ctx) return EMSESG_ERR_ARG;
  return run_fold(ctx, ctx->field[EMSESG_FIELD_AJDG], field_desc(ctx->cfg, EMSESG_FIELD_AJDG), 1, "reduce_ajdg");
}

extern "C" int emsesg_rhoupd(emsesg_ctx* ctx, int ps) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  const emsesg_config& c = ctx->cfg;
  int64_t nn = (int64_t)(c.nx + 1) * (c.ny + 1) * (c.nz + 1);
  EMSESG_LAUNCH(ctx, "rhoupd", k_rhoupd, nblk(nn), 256, 0, ctx->field[EMSESG_FIELD_RHO],
                ctx->field[EMSESG_FIELD_AJ], field_desc(c, EMSESG_FIELD_RHO), field_desc(c, EMSESG_FIELD_AJ), c.nx,
                c.ny, c.nz);
  return EMSESG_OK;
}

extern "C" int emsesg_bfield(emsesg_ctx* ctx, int ps) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if ((rc = apply_pending_eb(ctx))) return rc;
  const emsesg_config& c = ctx->cfg;
  const int64_t nn = (int64_t)(c.nx + 2) * (c.ny + 2) * (c.nz + 2);
  EMSESG_LAUNCH(ctx, "bfield", k_bfield, nblk(nn), 256, 0, ctx->field[EMSESG_FIELD_EB],
                field_desc(c, EMSESG_FIELD_EB), c.nx, c.ny, c.nz);
  return EMSESG_OK;
}

extern "C" int emsesg_efield(emsesg_ctx* ctx, int ps, double tcs, double dlt) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if ((rc = apply_pending_eb(ctx))) return rc;
  const emsesg_config& c = ctx->cfg;
  const int64_t nn = (int64_t)(c.nx + 1) * (c.ny + 1) * (c.nz + 1);
  EMSESG_LAUNCH(ctx, "efield", k_efield, nblk(nn), 256, 0, ctx->field[EMSESG_FIELD_EB], ctx->field[EMSESG_FIELD_AJ],
                field_desc(c, EMSESG_FIELD_EB), field_desc(c, EMSESG_FIELD_AJ), c.nx, c.ny, c.nz, tcs, dlt);
  return EMSESG_OK;
}

extern "C" int emsesg_exchange_eb(emsesg_ctx* ctx) {
  if (!ctx) return EMSESG_ERR_ARG;
  int rc = apply_pending_eb(ctx);
  if (rc) return rc;
  const FieldDesc f = field_desc(ctx->cfg, EMSESG_FIELD_EB);
  return run_fold(ctx, ctx->field[EMSESG_FIELD_EB], f, 2, "exchange_eb");
}

extern "C" int emsesg_energy(emsesg_ctx* ctx, double* engk) {
  if (!ctx || !engk) return EMSESG_ERR_ARG;
  const emsesg_config& c = ctx->cfg;
  EMSESG_CUDA(ctx, cudaMemsetAsync(ctx->d_sum, 0, 3 * EMSESG_ISPEC * sizeof(double), ctx->stream));
  for (int is = 0; is < c.nspec; is++) {
    int64_t n = ctx->totalp[is];
    if (n == 0) continue;
    unsigned blocks = (unsigned)std::min<int64_t>(nblk(n), 148 * 8);
    EMSESG_LAUNCH(ctx, "energy", k_energy, blocks, 256, 0, ctx->pbuf + ctx->seg.base[is], n, ctx->d_count + is,
                  ctx->d_sum + 3 * is);
  }
  double s[3 * EMSESG_ISPEC];
  EMSESG_CUDA(ctx, cudaMemcpyAsync(s, ctx->d_sum, sizeof s, cudaMemcpyDeviceToHost, ctx->stream));
  EMSESG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double vol = (double)c.nx * (double)c.ny * (double)c.nz;
  for (int is = 0; is < c.nspec; is++)
    for (int d = 0; d < 3; d++) engk[is * 3 + d] = 0.5 * c.rm[is] * s[3 * is + d] / vol;
  return emsesg_synchronize(ctx);
}

namespace {
KeyArgs key_args(const emsesg_config& c) {
  KeyArgs ka;
  int n[3] = {c.nx, c.ny, c.nz};
  for (int d = 0; d < 3; d++) {
    ka.t[d] = c.sort_tile[d] > 0 ? std::min(c.sort_tile[d], n[d]) : n[d];
    ka.nt[d] = (n[d] + ka.t[d] - 1) / ka.t[d];
  }
  return ka;
}
int key_bits_for(uint64_t maxkey) {
  int b = 1;
  while (b < 32 && (1ULL << b) <= maxkey) b++;
  return b;
}
int ensure_pbuf2(emsesg_ctx* ctx) {
  if (ctx->pbuf2) return EMSESG_OK;
  int64_t cap = 0;
  for (int is = 0; is < ctx->cfg.nspec; is++) cap += ctx->seg.capacity[is];
  EMSESG_CUDA(ctx, cudaMalloc(&ctx->pbuf2, std::max<int64_t>(cap, 1) * sizeof(emsesg_particle)));
  return EMSESG_OK;
}
}  // namespace

// spsort, src/etc/spsort.F90:29-35: every species segment sorted by the
// canonical key (stable), replacing particle_sort_ (psort-struct.c:7-9).
extern "C" int emsesg_spsort(emsesg_ctx* ctx, int ps) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if ((rc = ensure_sort_scratch(ctx, max_count(ctx)))) return rc;
  if ((rc = ensure_pbuf2(ctx))) return rc;
  KeyArgs ka = key_args(ctx->cfg);
  uint64_t maxkey = (uint64_t)ka.nt[0] * ka.nt[1] * ka.nt[2] * ka.t[0] * ka.t[1] * ka.t[2];
  int bits = key_bits_for(maxkey);
  for (int is = 0; is < ctx->cfg.nspec; is++) {
    int64_t n = ctx->totalp[is];
    if (n == 0) continue;
    emsesg_particle* p = ctx->pbuf + ctx->seg.base[is];
    EMSESG_LAUNCH(ctx, "sort_keys", k_make_keys, nblk(n), 256, 0, p, n, ctx->d_cfg, ka, ctx->sort.keys[0],
                  ctx->sort.vals[0]);
    uint32_t *ko, *vo;
    if ((rc = sort_pairs(ctx, ctx->sort.keys[0], ctx->sort.vals[0], n, bits, &ko, &vo))) return rc;
    emsesg_particle* q = ctx->pbuf2 + ctx->seg.base[is];
    EMSESG_LAUNCH(ctx, "sort_gather", k_gather_particles, nblk(2 * n), 256, 0, p, q, vo, n);
  }
  // the sorted buffer becomes pbuf
  std::swap(ctx->pbuf, ctx->pbuf2);
  return EMSESG_OK;
}

// Single-rank compaction (the part of oh3_transbound that one rank needs):
// drop nid == -1, keep order, update counts.
extern "C" int emsesg_compact(emsesg_ctx* ctx, int ps, int64_t* totalp) {
  int rc = check_ps(ctx, ps);
  if (rc) return rc;
  if ((rc = ensure_sort_scratch(ctx, max_count(ctx)))) return rc;
  if ((rc = ensure_pbuf2(ctx))) return rc;
  for (int is = 0; is < ctx->cfg.nspec; is++) {
    int64_t n = ctx->totalp[is];
    if (n == 0) continue;
    emsesg_particle* p = ctx->pbuf + ctx->seg.base[is];
    emsesg_particle* q = ctx->pbuf2 + ctx->seg.base[is];
    uint32_t* flags = ctx->sort.keys[0];
    EMSESG_LAUNCH(ctx, "live_flags", k_live_flags, nblk(n), 256, 0, p, n, flags);
    if ((rc = exclusive_scan_u32(ctx, flags, n))) return rc;
    EMSESG_LAUNCH(ctx, "compact_scatter", k_compact_scatter, nblk(2 * n), 256, 0, p, q, flags, n);
    EMSESG_LAUNCH(ctx, "set_count", k_set_count, 1, 1, 0, ctx->d_count + is, ctx->sort.scan_tmp);
  }
  // the compacted buffer becomes pbuf; one wait for the counts of all species
  std::swap(ctx->pbuf, ctx->pbuf2);
  int64_t kept[EMSESG_ISPEC];
  EMSESG_CUDA(ctx, cudaMemcpyAsync(kept, ctx->d_count, sizeof kept, cudaMemcpyDeviceToHost, ctx->stream));
  EMSESG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int is = 0; is < ctx->cfg.nspec; is++)
    if (ctx->totalp[is] > 0) ctx->totalp[is] = kept[is];
  if (totalp)
    for (int is = 0; is < ctx->cfg.nspec; is++) totalp[is] = ctx->totalp[is];
  return emsesg_synchronize(ctx);
}

int emsesg::plasma_records(emsesg_ctx* ctx, emsesg_particle* dst, int is, int64_t m0, int64_t n,
                           const emsesg_plasma* pl) {
  const emsesg_config& c = ctx->cfg;
  EMSESG_LAUNCH(ctx, "load_plasma", k_load_plasma, nblk(n), 256, 0, dst, m0, n, pl->ppc[is], c.nx, c.ny, is,
                pl->seed, pl->vth[is], pl->vdrift[is][0], pl->vdrift[is][1], pl->vdrift[is][2]);
  return EMSESG_OK;
}

extern "C" int emsesg_load_plasma(emsesg_ctx* ctx, const emsesg_plasma* pl) {
  if (!ctx || !pl) return EMSESG_ERR_ARG;
  if (ctx->cfg.flags & EMSESG_FLAG_FP32_ONLY)
    return set_error(ctx, EMSESG_ERR_STATE, "FP32-only context: use emsesg_fx_load_plasma");
  const emsesg_config& c = ctx->cfg;
  int64_t ncell = (int64_t)c.nx * c.ny * c.nz;
  for (int is = 0; is < c.nspec; is++) {
    int64_t n = ncell * pl->ppc[is];
    if (pl->ppc[is] < 0 || n > ctx->seg.capacity[is])
      return set_error(ctx, EMSESG_ERR_OVERFLOW, "species %d: %lld particles exceed capacity", is + 1, (long long)n);
  }
  for (int is = 0; is < c.nspec; is++) {
    int64_t n = ncell * pl->ppc[is];
    ctx->totalp[is] = n;
    if (n == 0) continue;
    int rc = plasma_records(ctx, ctx->pbuf + ctx->seg.base[is], is, 0, n, pl);
    if (rc) return rc;
  }
  EMSESG_CUDA(ctx, cudaMemcpyAsync(ctx->d_count, ctx->totalp, EMSESG_ISPEC * sizeof(int64_t), cudaMemcpyHostToDevice,
                                   ctx->stream));
  EMSESG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->fx.loaded = false;
  return EMSESG_OK;
}
