// fx_push.cuh -- the fused push + zigzag current + CIC charge kernel of the
// FP32 / fixed-point form (included by fx.cu inside its private namespace).
//
// Layout.  The sort leaves every (species, cell tile) in a padded region of
// L rows x PUSH_THREADS slots, thread-major: the particle of sorted rank q in
// the tile sits in row q % L, column q / L.  Column t of the region is thus
// thread t's contiguous run of the cell-sorted order, and row r is one
// coalesced stretch of PUSH_THREADS records.  Empty slots hold DEAD cells.
//
// One CTA of 736 threads pushes one row chunk of a region.  Each warp copies
// its own 32 columns of the rows ahead (cp.async, a ring of three rows a warp),
// so the warps share no barrier inside the rows.  The tile's FP32 E/B nodes
// (tile + 1-cell guard) sit in shared memory.
//
// Per particle: trilinear gather, Buneman-Boris, move.  A particle in its
// thread's current cell (the "run", the common case) that stays in it adds its
// two zigzag segments and its CIC charge to 20 FP32 registers; when the run
// ends the 20 sums go through a per-warp queue and are added, converted to
// int64 fixed point, into the CTA's tile accumulator by all lanes together.
// A particle out of place in the thread's run (it changed cell since the
// sort) goes on a per-warp list, and so does one that leaves its cell; a full
// batch of a list is taken by the whole warp, a particle a lane: out-of-place
// ones are kicked, moved and added with shared-memory atomics, crossing ones
// take the general path (per-axis boundary rules, relay point, two segments in
// different cells, charge at the new cell).  So the divergent work of the few
// runs with all lanes busy.
//
// What bounds it: issue slots (60 % of them) and shared-memory passes (65 %),
// with the latency of 23 warps a SM between them; DRAM is at 36 %.  At 128^3 x
// 2 x 64 ppc a push took 7.45 ms with scalar FP32, out-of-place particles in
// the run queue and rows by bulk copies on shared mbarriers (539 warp
// instructions a row of 32); 6.81 ms with packed FP32 (f32x2), the
// interpolation by lerps and the out-of-place list (455); 6.47 ms with rows
// per warp, 32-bit slot indices and the field rows padded against bank
// conflicts (433); 6.29 ms with the chunk table in place of a binary search (2.39
// TB/s at 56 B a particle).  Not kept, at the same size: rows prefetched in
// registers (spills, 6.61 ms), the lists out of line (12 ms: generic addresses
// and an array argument in local memory), all lists at the end of the chunk
// (7.23 ms: their load latency then meets no other work), a persistent CTA that
// fetches the next tile during the flush (6.46 ms, and 12 % slower where the
// push runs in parts).
//
// Determinism: a run's FP32 partial sums follow the thread's fixed order;
// every conversion to fixed point is of one value; integer atomics commute.
// Two runs on the same input give the same bits.

// 23 warps, 6 on each SM sub-partition, at 80 registers a thread (408 bytes spill with the current, five local loads
// and three stores a warp row, none without it): with 480-slot rows (16 warps, 128 registers) an
// earlier form of the kernel took 8.16 ms, with 608 (20 warps, 96) 7.53, with
// 736 7.20.
constexpr int PUSH_THREADS = 736;           // pushing threads = slots per row
constexpr int PUSH_WARPS = PUSH_THREADS / 32;
constexpr int PG = 1;           // guard cells around the tile
constexpr int NJ = 12;          // zigzag node values of one cell
constexpr int NR = 8;           // CIC node values of one cell
// run-queue entry: the sums of a run (20, charge only 8), the box index of
// its cell, one word of padding (the sums are stored in 8-byte pairs)
__host__ __device__ constexpr int run_words(bool jd) { return (jd ? NJ + NR : NR) + 2; }
constexpr int RQ_DRAIN = 8;     // drain the run queue at this many entries
constexpr int RQ_ROUND = 16;    // lanes that put their run in the queue at a time
constexpr int RQCAP = RQ_DRAIN + RQ_ROUND;
constexpr int XQW = 8;          // general-path entry: slot, cell, 3 offsets, 3 velocities
constexpr int XLCAP = 96;       // per-warp list of cross slots (emptied when nearly full)
constexpr int OLCAP = 64;       // per-warp list of out-of-place slots (a full batch is taken past 32)
constexpr int RING = 3;         // rows of a warp's ring
constexpr int ROW32 = 32 * (16 + 3 * 4);  // bytes of a row's 32 particles
constexpr uint32_t NORUN = 0xFFFFFFFEu;  // no run open (cells have at most 31 bits)
static_assert(PUSH_THREADS == EMSESG_FX_ROW_SLOTS, "row width of the thread-major layout");

// Bodies of the FP32 form, in the order of cfg.body.  Box bodies (geotype
// 0/1 with integer bounds): the absorption test and the per-surface-cell
// counts; faces -x,+x,-y,+y,-z,+z, a face's cells with its first tangential
// axis fastest (x faces: y then z; y faces: x then z; z faces: x then y).
// Cylinders (geotype 2) and spheres (3): the absorption test of the end
// point (psolve1.F90:684-712) and the body's influx; lo / hi are then the
// cells their bounding box touches, and they have no surface cells.
struct Bodies {
  int n;                        // bodies
  int ipc[EMSESG_INPC];         // their index in cfg.body
  int kind[EMSESG_INPC];        // 0 box, 2 cylinder, 3 sphere
  int lo[EMSESG_INPC][3], hi[EMSESG_INPC][3];
  int64_t off[EMSESG_INPC][6];  // first surface cell of each face (boxes)
  int64_t nsurf;                // surface cells of all box bodies
  int ncurved;                  // cylinders and spheres
  int cax[EMSESG_INPC];         // cylinder axis 0..2; its transverse axes are cax+1, cax+2 (mod 3)
  float cen[EMSESG_INPC][3];    // sphere centre; cylinder: cyl_axis(1:2) in [cax+1], [cax+2]
  float edge[EMSESG_INPC][2];   // cylinder extent along its axis (inclusive)
  float r2[EMSESG_INPC];        // radius squared (strict inside)
};

// Whether the point (cell ac, offset af per axis) lies inside curved body q
// (psolve1.F90:684-712: d1^2 + d2^2 < r^2 with the axial coordinate within
// the cylinder's edges, inclusive; |x - c|^2 < r^2 for a sphere).  Each
// difference is taken from the integer cell first, so it keeps the offset's
// precision.
__device__ __forceinline__ bool in_curved(const Bodies& bd, int q, const int (&ac)[3], const float (&af)[3]) {
  if (bd.kind[q] == 3) {
    float s = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float x = ((float)ac[d] - bd.cen[q][d]) + af[d];
      s = fmaf(x, x, s);
    }
    return s < bd.r2[q];
  }
  const int c0 = bd.cax[q], c1 = c0 == 2 ? 0 : c0 + 1, c2 = c0 == 0 ? 2 : c0 - 1;
  const float xl = ((float)ac[c0] - bd.edge[q][0]) + af[c0];
  const float xu = ((float)ac[c0] - bd.edge[q][1]) + af[c0];
  if (!(xl >= 0.f && xu <= 0.f)) return false;
  const float d1 = ((float)ac[c1] - bd.cen[q][c1]) + af[c1];
  const float d2 = ((float)ac[c2] - bd.cen[q][c2]) + af[c2];
  return fmaf(d1, d1, d2 * d2) < bd.r2[q];
}

// Slab mode (the grid is one z slab of a larger grid, periodic in z, cut
// into slabs of equal thickness): particles that leave through a z face go
// to the neighbouring slab's rank.  Their records, in that rank's frame (the
// periodic wrap of this slab), per species and direction: region
// (2 is + dir) of cap records, dir 0 through z = 0, 1 through z = nz.  pid
// holds the particle's slot here (the order of the records is then made
// independent of the atomics).
struct Outbox {
  emsesg_particle* rec;         // null: not in slab mode
  unsigned long long* count;    // [2 nspec]
  int64_t cap;
};

struct FxPushArgs {
  float4* pos;                  // all species regions (the step's result)
  float* vx;
  float* vy;
  float* vz;
  const float4* rpos;           // the state read (the same arrays, or for a
  const float* rvx;             // move-only step, those of a kept copy)
  const float* rvy;
  const float* rvz;
  const int64_t* chunk_start;   // [nspec][ntiles+1] first CTA (row chunk) of each tile
  const int4* chunks;           // [nspec][nchunk_max] the row chunks: tile, rows, first slot in the region
  int64_t nchunk_max;
  int64_t off[EMSESG_ISPEC];    // region base per species
  int npbnd[EMSESG_ISPEC][3];
  float qmp[EMSESG_ISPEC], qfix[EMSESG_ISPEC];
  float gustep, rustep;
  const float4* __restrict__ f0;
  const float4* __restrict__ f1;
  unsigned long long* acc_rho;  // rho layout (1, -1:n+1)
  unsigned long long* acc_j;    // aj layout (3, -4:n+4)
  FieldDesc fr, fj;
  Geo g;
  int64_t ntiles;
  int* nesc;                    // counter nesc(is), one int per species
  emsesg_counter* gc;           // influx / infhist of the body absorption
  unsigned long long* surf;     // [nspec][nsurf] absorbed - emitted counts
  Bodies bd;
  Outbox ob;
  int* status;
  long long* diag;
  // the tiles of this launch: t_lo .. t_lo + t_n - 1 (t_n = 0: every tile;
  // a step whose eb arrives in z chunks pushes its tile layers in parts)
  int64_t t_lo, t_n;
  // a part (PARTS) holds the node planes 0..zready; it marks here (one bit
  // per slot) a particle that would gather from a higher plane, which
  // k_fx_deferred pushes after the last part
  int zready;
  uint32_t* defer;
};

// ---------------------------------------------------------------- PTX
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// 16-byte copies global -> shared (both addresses 16-byte aligned), in groups.
template <bool CA>
__device__ __forceinline__ void cpa16(void* dst, const void* src) {
  if (CA)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- packed FP32
// Two FP32 values in a 64-bit register pair: sm_100a's f32x2 instructions do
// both in one issue slot, each rounded as the scalar instruction rounds it.
// The pushing loop is bound by issue slots.  All arithmetic of the kick, the
// move and the in-cell deposit is written with explicit roundings (these and
// the __f*_rn intrinsics), so that every kernel that holds it gives the same
// bits, however the compiler would fuse multiplies with adds.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 dup(float v) { return pk(v, v); }
__device__ __forceinline__ void upk(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 lerp2(f2 a, f2 b, f2 t) { return fma2(sub2(b, a), t, a); }

// ---------------------------------------------------------------- moves
// Per-axis move and outer boundary of psolve1.F90:366-606 on (cell, offset)
// pairs.  In: cell ib, offset ob, displacement d.  Out: the "after" point
// xlocala = (ac, af), its cell ia, the relay point xr = (rc, rf), the stored
// new position (nc, nf), and flags.
struct Axis {
  int ac, ia, rc, nc;
  float af, rf, nf;
  bool dead, flip, crossed;
};

constexpr float BELOW_ONE = 0.99999994f;  // the largest offset

// The outer boundary rules for an "after" cell ac outside 0..n-1.  A
// reflection that ends exactly on the upper face, x = n, stays in the last
// cell, as a record loaded there does.  The rules wrap or reflect once: a
// displacement longer than the axis can leave nc outside 0..n-1.
__device__ __forceinline__ Axis axis_boundary(int ib, float ob, int ac, float af, int n, int npbnd) {
  Axis o;
  o.dead = false;
  o.flip = false;
  o.crossed = true;
  if (ac < 0) {  // p%x < 0
    if (npbnd == 0) {
      o.ac = ac; o.af = af; o.ia = -1; o.rc = 0; o.rf = 0.f;
      o.nc = ac + n; o.nf = af;
    } else if (npbnd == 1) {
      int rc_ = af > 0.f ? -ac - 1 : -ac;
      float rf_ = af > 0.f ? 1.0f - af : 0.0f;
      if (rf_ >= 1.0f) { rf_ = 0.f; rc_ += 1; }
      if (rc_ == n && rf_ == 0.f) { rf_ = BELOW_ONE; rc_ -= 1; }
      o.ac = rc_; o.af = rf_; o.ia = 0; o.rc = 0; o.rf = 0.f;
      o.nc = rc_; o.nf = rf_; o.flip = true;
    } else {
      o.ac = -1; o.af = 0.f; o.ia = -1; o.rc = 0; o.rf = 0.f;
      o.nc = 0; o.nf = 0.f; o.dead = true;
    }
  } else {  // p%x >= slx
    if (npbnd == 0) {
      o.ac = ac; o.af = af; o.ia = n; o.rc = n; o.rf = 0.f;
      o.nc = ac - n; o.nf = af;
    } else if (npbnd == 1) {
      int rc_ = af > 0.f ? 2 * n - ac - 1 : 2 * n - ac;
      float rf_ = af > 0.f ? 1.0f - af : 0.0f;
      if (rf_ >= 1.0f) { rf_ = 0.f; rc_ += 1; }
      if (rc_ == n && rf_ == 0.f) { rf_ = BELOW_ONE; rc_ -= 1; }
      o.ac = rc_; o.af = rf_; o.ia = n - 1; o.rc = n; o.rf = 0.f;
      o.nc = rc_; o.nf = rf_; o.flip = true;
    } else {
      o.ac = n + 1; o.af = 0.f; o.ia = n; o.rc = n; o.rf = 0.f;
      o.nc = 0; o.nf = 0.f; o.dead = true;
    }
  }
  return o;
}

__device__ __forceinline__ Axis axis_move(int ib, float ob, float d, int n, int npbnd) {
  const float s = ob + d;
  const float fl = floorf(s);
  int ac = ib + (int)fl;
  float af = s - fl;
  if (af >= 1.0f) { af = 0.0f; ac += 1; }
  if ((unsigned)ac >= (unsigned)n) return axis_boundary(ib, ob, ac, af, n, npbnd);
  Axis o;
  o.dead = false;
  o.flip = false;
  o.crossed = false;
  o.ac = ac; o.af = af; o.ia = ac; o.nc = ac; o.nf = af;
  const bool same = ac == ib;
  o.rc = same ? ib : max(ib, ac);
  o.rf = same ? (ob + af) * 0.5f : 0.f;
  return o;
}

// Node offsets of the 12 zigzag values of a cell: 0-3 JX at (0,a,b), 4-7 JY
// at (a,0,b), 8-11 JZ at (a,b,0) with (a,b) = (s&1, s>>1&1), in the order of
// the scatter-adds of psolve1.F90:759-789 (w1, w2, w3, w4 per component).
__host__ __device__ constexpr int jcomp(int s) { return 1 + (s >> 2); }
__host__ __device__ constexpr int jdi(int s) { return s < 4 ? 0 : (s & 1); }
__host__ __device__ constexpr int jdj(int s) { return s < 4 ? (s & 1) : (s < 8 ? 0 : ((s >> 1) & 1)); }
__host__ __device__ constexpr int jdk(int s) { return s < 8 ? ((s >> 1) & 1) : 0; }
// CIC corners v1..v8 (charge.F90:202-209): (0,0,1) (1,0,1) (1,1,1) (0,1,1)
// (0,0,0) (1,0,0) (1,1,0) (0,1,0).
__host__ __device__ constexpr int rdi(int r) { return ((r & 3) == 1 || (r & 3) == 2) ? 1 : 0; }
__host__ __device__ constexpr int rdj(int r) { return (r & 3) >= 2 ? 1 : 0; }
__host__ __device__ constexpr int rdk(int r) { return r < 4 ? 1 : 0; }

// The tile's {Ex,Ey,Ez,Bx} nodes in shared memory have rows of 16 nodes for
// the 11 of an 8-cell tile: neighbouring lanes hold neighbouring cells, and
// with the next y row 16 nodes on, the 8 lanes of a 128-bit access that run
// over a row's end (cells 0..7) fall on the 8 different 16-byte banks groups
// again.  With rows of 11 a quarter of the gather's shared-memory passes were
// bank conflicts.  {By,Bz} (64-bit accesses) keeps rows of 11.
template <int B>
struct FieldT {
  static constexpr int W = B > 8 ? 16 : 8;  // row stride
  static constexpr int N = W * B * B;
};

template <int B>
struct BoxT {
  static constexpr int B2 = B * B;
  static constexpr int B3 = B * B * B;
  __host__ __device__ static constexpr int joff(int s) { return jcomp(s) * B3 + jdk(s) * B2 + jdj(s) * B + jdi(s); }
  __host__ __device__ static constexpr int roff(int r) { return rdk(r) * B2 + rdj(r) * B + rdi(r); }
};

__device__ __forceinline__ long long to_fix(float v, float scale) { return __float2ll_rn(v * scale); }

// Adds v to a 64-bit accumulator in shared memory with 32-bit atomics (a
// 64-bit shared-memory atomic add is much slower): the low word first, its
// carry out then goes with the high word.  The carries counted by all
// additions add up to the wraps of the low word, so the final value is the
// 64-bit sum in any order; only the final value is read.
__device__ __forceinline__ void box_add(unsigned long long* p, unsigned long long v) {
  unsigned int* w = reinterpret_cast<unsigned int*>(p);  // little-endian: low word first
  const unsigned int lo = (unsigned int)v, hi = (unsigned int)(v >> 32);
  const unsigned int old = atomicAdd(w, lo);
  const unsigned int h = hi + (old + lo < old ? 1u : 0u);
  if (h) atomicAdd(w + 1, h);
}

// Global arrays for deposits whose cell lies outside the tile box.
struct Sink {
  unsigned long long* acc_rho;
  unsigned long long* acc_j;
  FieldDesc fr, fj;
  int nx, ny, nz;
  int* status;
  long long* diag;
};

// Box index of cell (i,j,k) when its 2x2x2 node block lies inside the box,
// else -1.
template <int B>
__device__ __forceinline__ int box_base(const int (&o)[3], int i, int j, int k) {
  int li = i - o[0], lj = j - o[1], lk = k - o[2];
  bool ok = (unsigned)li < (unsigned)(B - 1) && (unsigned)lj < (unsigned)(B - 1) && (unsigned)lk < (unsigned)(B - 1);
  return ok ? (lk * B + lj) * B + li : -1;
}

// The same with the cell's index in the tile's {Ex,Ey,Ez,Bx} nodes.
template <int B>
__device__ __forceinline__ int box_base(const int (&o)[3], int i, int j, int k, int& fb) {
  const int li = i - o[0], lj = j - o[1], lk = k - o[2];
  const bool ok = (unsigned)li < (unsigned)(B - 1) && (unsigned)lj < (unsigned)(B - 1) && (unsigned)lk < (unsigned)(B - 1);
  fb = (lk * B + lj) * FieldT<B>::W + li;
  return ok ? (lk * B + lj) * B + li : -1;
}

struct V12 { float v[NJ]; };
struct V8 { float v[NR]; };

// Node sets whose cell lies outside the box: global int64 atomics with
// bounds checks (rare; the values come by value so that the callers'
// register arrays keep no address).
__device__ __forceinline__ void put_j_global(Sink s, int i, int j, int k, V12 v, float qfix) {
  for (int q = 0; q < NJ; q++) {
    const long long f = to_fix(v.v[q], qfix);
    if (f == 0) continue;
    const int ii = i + jdi(q), jj = j + jdj(q), kk = k + jdk(q);
    if (ii < -4 || jj < -4 || kk < -4 || ii > s.nx + 4 || jj > s.ny + 4 || kk > s.nz + 4) {
      report_bad(s.status, s.diag, SITE_FX_DEPOSIT, -2, ii + 100000LL * jj + 10000000000LL * kk);
      continue;
    }
    atomicAdd(&s.acc_j[s.fj.at(jcomp(q) - 1, ii, jj, kk)], (unsigned long long)f);
  }
}

__device__ __forceinline__ void put_r_global(Sink s, int i, int j, int k, V8 v, float qfix) {
  for (int r = 0; r < NR; r++) {
    const long long f = to_fix(v.v[r], qfix);
    const int ii = i + rdi(r), jj = j + rdj(r), kk = k + rdk(r);
    if (ii < -1 || jj < -1 || kk < -1 || ii > s.nx + 1 || jj > s.ny + 1 || kk > s.nz + 1) {
      report_bad(s.status, s.diag, SITE_FX_DEPOSIT, -1, ii + 100000LL * jj + 10000000000LL * kk);
      continue;
    }
    if (f != 0) atomicAdd(&s.acc_rho[s.fr.at(0, ii, jj, kk)], (unsigned long long)f);
  }
}

// One zigzag node set (12 values) of cell (i,j,k): into the box, or into the
// global arrays when the cell lies outside the box.
template <int B>
__device__ __forceinline__ void put_j(unsigned long long* box, const int (&o)[3], const Sink& s, int i, int j, int k,
                                      const float (&v)[NJ], float qfix) {
  const int base = box_base<B>(o, i, j, k);
  if (base >= 0) {
#pragma unroll
    for (int q = 0; q < NJ; q++) box_add(&box[base + BoxT<B>::joff(q)], (unsigned long long)to_fix(v[q], qfix));
  } else {
    V12 w;
#pragma unroll
    for (int q = 0; q < NJ; q++) w.v[q] = v[q];
    put_j_global(s, i, j, k, w, qfix);
  }
}

template <int B>
__device__ __forceinline__ void put_r(unsigned long long* box, const int (&o)[3], const Sink& s, int i, int j, int k,
                                      const float (&v)[NR], float qfix) {
  const int base = box_base<B>(o, i, j, k);
  if (base >= 0) {
#pragma unroll
    for (int r = 0; r < NR; r++) box_add(&box[base + BoxT<B>::roff(r)], (unsigned long long)to_fix(v[r], qfix));
  } else {
    V8 w;
#pragma unroll
    for (int r = 0; r < NR; r++) w.v[r] = v[r];
    put_r_global(s, i, j, k, w, qfix);
  }
}

// E and B from the global node field, corner weights times values.
__device__ __forceinline__ void gather8(const float4* f0, const float4* f1, int64_t n5, int64_t sy, int64_t sz,
                                        const float (&w)[8], float (&e)[3], float (&b)[3]) {
  const int64_t idx[8] = {n5 + sz, n5 + sz + 1, n5 + sz + 1 + sy, n5 + sz + sy, n5, n5 + 1, n5 + 1 + sy, n5 + sy};
  float ex = 0.f, ey = 0.f, ez = 0.f, bx = 0.f, by = 0.f, bz = 0.f;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const float4 p = __ldg(&f0[idx[c]]), q = __ldg(&f1[idx[c]]);
    ex += p.x * w[c];
    ey += p.y * w[c];
    ez += p.z * w[c];
    bx += p.w * w[c];
    by += q.x * w[c];
    bz += q.y * w[c];
  }
  e[0] = ex; e[1] = ey; e[2] = ez;
  b[0] = bx; b[1] = by; b[2] = bz;
}

// E and B of a cell at the offsets (x, y, z): linear interpolations along x,
// then y, then z, the six components in three pairs (Ex,Ey) (Ez,Bx) (By,Bz):
// 42 packed operations (corner weights times values: 48 plus the weights).
// n0(c) / n1(c): the node c (0..7: bit 0 x, bit 1 y, bit 2 z).
struct EB { f2 exy, ezbx, byz; };
template <class N0, class N1>
__device__ __forceinline__ EB interp(float x, float y, float z, N0 n0, N1 n1) {
  const f2 X = dup(x), Y = dup(y), Z = dup(z);
  EB plane[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    EB row[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const ulonglong2 a0 = n0(4 * k + 2 * j), b0 = n0(4 * k + 2 * j + 1);
      const f2 a1 = n1(4 * k + 2 * j), b1 = n1(4 * k + 2 * j + 1);
      row[j] = EB{lerp2(a0.x, b0.x, X), lerp2(a0.y, b0.y, X), lerp2(a1, b1, X)};
    }
    plane[k] = EB{lerp2(row[0].exy, row[1].exy, Y), lerp2(row[0].ezbx, row[1].ezbx, Y),
                  lerp2(row[0].byz, row[1].byz, Y)};
  }
  return EB{lerp2(plane[0].exy, plane[1].exy, Z), lerp2(plane[0].ezbx, plane[1].ezbx, Z),
            lerp2(plane[0].byz, plane[1].byz, Z)};
}

// Trilinear gather of E and B at the particle (from the tile's shared nodes
// when its cell lies in the box, gb >= 0, else from the global node field)
// and the Buneman-Boris velocity update (psolve1.F90:186-272).  The shared
// nodes hold the fields already multiplied by the species' qmp; the global
// ones are multiplied here.  fb: the cell's index in the {Ex,Ey,Ez,Bx} nodes
// (FieldT).  BOX: the cell is known to lie in the box.
template <int B, bool BOX = false>
__device__ __forceinline__ void kick(const FxPushArgs& a, const ulonglong2* sf0, const f2* sf1, int gb, int fb, int ib,
                                     int jb, int kb, float x, float y, float z, float qmp, float& vx, float& vy,
                                     float& vz) {
  EB f;
  if (BOX || gb >= 0) {
    f = interp(
        x, y, z,
        [&](int c) { return sf0[fb + (c & 1) + ((c >> 1) & 1) * FieldT<B>::W + (c >> 2) * FieldT<B>::W * B]; },
        [&](int c) { return sf1[gb + (c & 1) + ((c >> 1) & 1) * B + (c >> 2) * B * B]; });
  } else {
    const int64_t sy = a.g.nx + 1, sz = (int64_t)(a.g.nx + 1) * (a.g.ny + 1), n = ib + sy * jb + sz * kb;
    f = interp(
        x, y, z,
        [&](int c) {
          return __ldg(reinterpret_cast<const ulonglong2*>(a.f0) + n + (c & 1) + ((c >> 1) & 1) * sy + (c >> 2) * sz);
        },
        [&](int c) {
          return __ldg(reinterpret_cast<const ulonglong2*>(a.f1) + n + (c & 1) + ((c >> 1) & 1) * sy + (c >> 2) * sz).x;
        });
    const f2 q = dup(qmp);
    f.exy = mul2(f.exy, q);
    f.ezbx = mul2(f.ezbx, q);
    f.byz = mul2(f.byz, q);
  }
  float ex, ey, ez, bx, by, bz;
  upk(f.exy, ex, ey);
  upk(f.ezbx, ez, bx);
  upk(f.byz, by, bz);
  const float boris = __fdividef(2.0f, __fmaf_rn(bx, bx, __fmaf_rn(by, by, __fmaf_rn(bz, bz, 1.0f))));
  vx = __fadd_rn(vx, ex);
  vy = __fadd_rn(vy, ey);
  vz = __fadd_rn(vz, ez);
  const float vxt = __fmaf_rn(vy, bz, __fmaf_rn(-vz, by, vx));
  const float vyt = __fmaf_rn(vz, bx, __fmaf_rn(-vx, bz, vy));
  const float vzt = __fmaf_rn(vx, by, __fmaf_rn(-vy, bx, vz));
  vx = __fmaf_rn(boris, __fmaf_rn(vyt, bz, -__fmul_rn(vzt, by)), vx);
  vy = __fmaf_rn(boris, __fmaf_rn(vzt, bx, -__fmul_rn(vxt, bz)), vy);
  vz = __fmaf_rn(boris, __fmaf_rn(vxt, by, -__fmul_rn(vyt, bx)), vz);
  vx = __fadd_rn(vx, ex);
  vy = __fadd_rn(vy, ey);
  vz = __fadd_rn(vz, ez);
}

// The sums of a particle that stays in its cell, in pairs: with the current,
// per component c of J the pairs 2c = (node value 1, 2) and 2c + 1 = (0, 3)
// of jcomp's four, then the CIC values (r, r + 4) for r = 0..3.  Both zigzag
// segments lie in the cell: relay point at the midpoint, equal segment
// fluxes h = (a-b)/2/ustep, mid-points m -+ (a-b)/4; the sum of the two
// bilinear weight sets is written with S = a+b, D = a-b.
template <bool JD>
__device__ __forceinline__ void cell_sums(float x, float y, float z, float sx, float sy, float sz, float hr,
                                          f2 (&cv)[JD ? (NJ + NR) / 2 : NR / 2]) {
  constexpr int RP = JD ? NJ / 2 : 0;  // first rho pair
  if (JD) {
    const f2 p = pk(x, y), s = pk(sx, sy);
    const f2 Sxy = add2(s, p), Dxy = sub2(s, p);
    const float Sz = __fadd_rn(sz, z), Dz = __fsub_rn(sz, z);
    float Sx, Sy, Dx, Dy, hx, hy, Px, Py;
    upk(Sxy, Sx, Sy);
    upk(Dxy, Dx, Dy);
    upk(mul2(Dxy, dup(hr)), hx, hy);
    const float hz = __fmul_rn(Dz, hr);
    upk(fma2(Dxy, dup(__fmul_rn(0.125f, Dz)), mul2(Sxy, dup(__fmul_rn(0.5f, Sz)))), Py, Px);
    const float Pz = __fmaf_rn(__fmul_rn(0.125f, Dx), Dy, __fmul_rn(__fmul_rn(0.5f, Sx), Sy));
    const float h3[3] = {hx, hy, hz}, P3[3] = {Px, Py, Pz};
    const f2 ab[3] = {pk(Sy, Sz), pk(Sx, Sz), Sxy};  // S of the two other axes
    const float ra[3] = {__fsub_rn(2.0f, Sy), __fsub_rn(2.0f, Sx), __fsub_rn(2.0f, Sx)};
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const f2 T = sub2(ab[c], dup(P3[c]));
      float ta, tb;
      upk(T, ta, tb);
      cv[2 * c] = mul2(dup(h3[c]), T);
      cv[2 * c + 1] = mul2(dup(h3[c]), pk(__fsub_rn(ra[c], tb), P3[c]));
    }
  }
  // CIC charge at the new position (charge.F90:152-210)
  const f2 zz = pk(sz, __fsub_rn(1.0f, sz));
  const f2 r2 = mul2(dup(__fmul_rn(sx, sy)), zz), XZ = mul2(dup(sx), zz);
  const f2 r3 = sub2(mul2(dup(sy), zz), r2);
  cv[RP + 2] = r2;
  cv[RP + 1] = sub2(XZ, r2);
  cv[RP + 3] = r3;
  cv[RP + 0] = sub2(sub2(zz, XZ), r3);
}

// Box offset of sum i of that order.
template <int B, bool JD>
__host__ __device__ constexpr int sum_off(int i) {
  constexpr int RO = JD ? NJ : 0;
  if (JD && i < NJ) {
    const int q = i & 3;
    return BoxT<B>::joff((i & ~3) + (q == 0 ? 1 : q == 1 ? 2 : q == 2 ? 0 : 3));
  }
  return BoxT<B>::roff((i - RO) / 2 + ((i - RO) & 1) * 4);
}

// Empties a warp's run queue.  The queue's (entry, slot) items are dealt
// out to the lanes in order, item m to lane m mod 32, so every pass keeps all
// 32 lanes busy however few entries are queued; the items of one entry go
// to 20 different nodes.  An entry holds its 20 sums and the box index of
// its cell (only cells inside the box are queued).
template <int NC>
__device__ __forceinline__ void drain_runs(unsigned long long* box, const int* slot_off, const float* q, int qn,
                                           float qfix, int lane) {
  static_assert(NC > 0 && NC <= 32, "an entry's sums fit one pass");
  constexpr int QW = NC + 2;
  __syncwarp();
  const int items = qn * NC;
  int e = lane / NC, sl = lane % NC;
  for (int m = lane; m < items; m += 32) {
    const float* en = q + e * QW;
    const int base = __float_as_int(en[NC]);
    const long long f = to_fix(en[sl], qfix);
    if (f) box_add(&box[base + slot_off[sl]], (unsigned long long)f);
    // m += 32: 32 = (32 / NC) * NC + 32 % NC
    sl += 32 % NC;
    e += 32 / NC;
    if (sl >= NC) {
      sl -= NC;
      e += 1;
    }
  }
  __syncwarp();
}

// The runs of the lanes in mk into the warp's queue, at most RQ_ROUND at a
// time, emptied whenever RQ_DRAIN entries wait.
template <int NC>
__device__ __forceinline__ void queue_runs(unsigned long long* box, const int* slot_off, float* rq, int& rqn,
                                           unsigned mk, bool mine, const f2 (&acc)[NC / 2], int base, float qfix,
                                           int lane) {
  constexpr int QW = NC + 2;
  const unsigned lt = (1u << lane) - 1u;
  int before = __popc(mk & lt);  // lanes to go before this one
  int left = __popc(mk);
  while (left > 0) {
    if (mine && before >= 0 && before < RQ_ROUND) {
      float* en = rq + (rqn + before) * QW;
      f2* e2 = reinterpret_cast<f2*>(en);
#pragma unroll
      for (int q = 0; q < NC / 2; q++) e2[q] = acc[q];
      en[NC] = __int_as_float(base);
    }
    rqn += min(left, RQ_ROUND);
    before -= RQ_ROUND;
    left -= RQ_ROUND;
    if (rqn >= RQ_DRAIN) {
      drain_runs<NC>(box, slot_off, rq, rqn, qfix, lane);
      rqn = 0;
    }
  }
}

struct CrossCtx {
  float4* gpos;                 // the tile region's first slot
  float* gvx;
  float* gvy;
  float* gvz;
  float gustep, rustep, qfix;
  int nb[3];
  const Bodies* bd;
  emsesg_counter* gc;
  unsigned long long* surf;     // this species' surface counts
  int is;
  int64_t slot_base;            // slot of gpos[0] in the particle arrays
  const Outbox* ob;
  int* status;
};

// Absorption of the end point by the bodies in their order, the first that
// holds it taking it (psolve1.F90:639-715).  A box tests a = (ac, af) per
// axis (:644-662, inclusive bounds) and counts influx, infhist and the
// surface cell of the face crossed last on the way from b = (ib, ob) (the
// rule of the oracle's orc_surface_cell); a cylinder or sphere tests the
// stored position (nc, nf) and counts influx and infhist.  Returns 0 (not
// absorbed), ABS_BOX (the particle stops at the relay point: no second
// zigzag segment, :660-662) or ABS_CURVED (both segments deposited).
constexpr int ABS_BOX = 1, ABS_CURVED = 2;
template <bool CURV>
__device__ __forceinline__ int body_absorb(const CrossCtx& c, const int (&ib)[3], const float (&ob)[3],
                                           const Axis* a3) {
  const Bodies& bd = *c.bd;
  for (int q = 0; q < bd.n; q++) {
    if (CURV && bd.kind[q] != 0) {
      const int nc3[3] = {a3[0].nc, a3[1].nc, a3[2].nc};
      const float nf3[3] = {a3[0].nf, a3[1].nf, a3[2].nf};
      if (!in_curved(bd, q, nc3, nf3)) continue;
      atomicAdd(&c.gc->influx[c.is][bd.ipc[q]], 1);
      atomicAdd(&c.gc->infhist[c.is][bd.ipc[q]][0], 1);
      return ABS_CURVED;
    }
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int ac = a3[d].ac;
      in = in && ac >= bd.lo[q][d] && (ac < bd.hi[q][d] || (ac == bd.hi[q][d] && a3[d].af == 0.0f));
    }
    if (!in) continue;
    const int ipc = bd.ipc[q];
    atomicAdd(&c.gc->influx[c.is][ipc], 1);
    atomicAdd(&c.gc->infhist[c.is][ipc][0], 1);
    // face crossed last: the largest entry time along b -> a
    int best = -1, side = 0;
    float tb = -1.0f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int lo = bd.lo[q][d], hi = bd.hi[q][d];
      const float den = (float)(a3[d].ac - ib[d]) + (a3[d].af - ob[d]);
      float t = -1.0f;
      int sd = 0;
      if (ib[d] < lo) { t = ((float)(lo - ib[d]) - ob[d]) / den; sd = 0; }
      else if (ib[d] > hi || (ib[d] == hi && ob[d] > 0.0f)) { t = ((float)(hi - ib[d]) - ob[d]) / den; sd = 1; }
      if (t > tb) { tb = t; best = d; side = sd; }
    }
    if (best < 0) {  // start point inside: the nearest face of the end point
      float dm = 3.0e38f;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const float x = (float)a3[d].ac + a3[d].af;
        if (x - (float)bd.lo[q][d] < dm) { dm = x - (float)bd.lo[q][d]; best = d; side = 0; }
        if ((float)bd.hi[q][d] - x < dm) { dm = (float)bd.hi[q][d] - x; best = d; side = 1; }
      }
    }
    const int e1 = best == 0 ? 1 : 0, e2 = best == 2 ? 1 : 2;
    const int c1 = best == 0 ? a3[1].ac : a3[0].ac;  // selects keep a3 in registers
    const int c2 = best == 2 ? a3[1].ac : a3[2].ac;
    const int u = min(max(c1, bd.lo[q][e1]), bd.hi[q][e1] - 1) - bd.lo[q][e1];
    const int v = min(max(c2, bd.lo[q][e2]), bd.hi[q][e2] - 1) - bd.lo[q][e2];
    const int64_t cellx = bd.off[q][2 * best + side] + u + (int64_t)(bd.hi[q][e1] - bd.lo[q][e1]) * v;
    atomicAdd(&c.surf[cellx], 1ull);
    return ABS_BOX;
  }
  return 0;
}

// General path for one particle that left its cell (or whose cell lies
// outside the box): boundary rules, zigzag with relay point, charge at the
// stored cell; the final record is written here.  A particle that ends in no
// cell of the grid is reported and dropped.  CURV = false: no
// cylinder or sphere to test.  JD = false: charge only (no zigzag current).
template <int B, bool DEP = true, bool CURV = true, bool JD = true>
__device__ __forceinline__ int cross_one(const Geo& g, unsigned long long* box, const int (&o)[3], const Sink& sk,
                                         const CrossCtx& c, const float* en) {
  const uint32_t loc = (uint32_t)__float_as_int(en[0]);
  const uint32_t cell = (uint32_t)__float_as_int(en[1]);
  const float bx = en[2], by = en[3], bz = en[4];
  float vx = en[5], vy = en[6], vz = en[7];
  int ib, jb, kb;
  unpack(g, cell, ib, jb, kb);
  Axis ax = axis_move(ib, bx, vx * c.gustep, g.nx, c.nb[0]);
  Axis ay = axis_move(jb, by, vy * c.gustep, g.ny, c.nb[1]);
  Axis az = axis_move(kb, bz, vz * c.gustep, g.nz, c.nb[2]);
  if (ax.flip) vx = -vx;
  if (ay.flip) vy = -vy;
  if (az.flip) vz = -vz;
  const bool escaped = ax.dead || ay.dead || az.dead;
  int absorbed = 0;
  if (!escaped && c.bd->n > 0) {
    const int ib3[3] = {ib, jb, kb};
    const float ob3[3] = {bx, by, bz};
    const Axis a3[3] = {ax, ay, az};
    absorbed = body_absorb<CURV>(c, ib3, ob3, a3);
  }
  const bool stop = absorbed == ABS_BOX;
  // slab mode: a particle leaving through a z face moves to the neighbouring
  // slab (its stored position, the slab's periodic wrap, is its position
  // there); its current stays here, in the guard planes that the ranks
  // exchange and fold, and its charge is deposited by the receiver
  const bool migrant = c.ob != nullptr && az.crossed && !escaped && !absorbed;
  if (migrant) {
    const int dir = az.ac < 0 ? 0 : 1;
    const unsigned long long q = atomicAdd(&c.ob->count[2 * c.is + dir], 1ull);
    if (q < (unsigned long long)c.ob->cap) {
      emsesg_particle r;
      r.x = (double)ax.nc + (double)ax.nf;
      r.y = (double)ay.nc + (double)ay.nf;
      r.z = (double)az.nc + (double)az.nf;
      r.vx = vx; r.vy = vy; r.vz = vz;
      r.pid = (int32_t)(c.slot_base + loc);
      r.preside = 0; r.nid = 0; r.spec = c.is + 1;
      c.ob->rec[(int64_t)(2 * c.is + dir) * c.ob->cap + (int64_t)q] = r;
    } else {
      atomicOr(c.status, ST_OVERFLOW);
    }
  }
  const bool dead = escaped || absorbed || migrant;
  // After a displacement longer than an axis the stored cell may be none of
  // the grid; packed it would be another particle's cell or an index past every
  // per-cell table.  Such a particle is dropped.
  const bool off =
      (unsigned)ax.nc >= (unsigned)g.nx || (unsigned)ay.nc >= (unsigned)g.ny || (unsigned)az.nc >= (unsigned)g.nz;
  const uint32_t nc = dead || off ? DEAD : pack(g, ax.nc, ay.nc, az.nc);
  c.gpos[loc] = make_float4(ax.nf, ay.nf, az.nf, __int_as_float((int)nc));
  c.gvx[loc] = vx;
  c.gvy[loc] = vy;
  c.gvz[loc] = vz;
  if (!DEP) return escaped ? 1 : 0;
  if (JD) {
  // zigzag (psolve1.F90:717-757), integer parts first
  float J[NJ];
  {
    float xd = ((float)(ax.rc - ib) + ax.rf + bx) * 0.5f;
    float yd = ((float)(ay.rc - jb) + ay.rf + by) * 0.5f;
    float zd = ((float)(az.rc - kb) + az.rf + bz) * 0.5f;
    float vvx = ((float)(ax.rc - ib) + (ax.rf - bx)) * c.rustep;
    float vvy = ((float)(ay.rc - jb) + (ay.rf - by)) * c.rustep;
    float vvz = ((float)(az.rc - kb) + (az.rf - bz)) * c.rustep;
    float w;
    w = yd * zd; J[3] = vvx * w; J[1] = vvx * (yd - w); J[2] = vvx * (zd - w); J[0] = vvx * (1.0f - yd - (zd - w));
    w = xd * zd; J[7] = vvy * w; J[5] = vvy * (xd - w); J[6] = vvy * (zd - w); J[4] = vvy * (1.0f - xd - (zd - w));
    w = xd * yd; J[11] = vvz * w; J[9] = vvz * (xd - w); J[10] = vvz * (yd - w); J[8] = vvz * (1.0f - xd - (yd - w));
  }
  // a start point inside a box body moves to the relay point
  // (psolve1.F90:648-651): no first segment
  if (CURV && !escaped) {
    const Bodies& bd = *c.bd;
    const int ib3[3] = {ib, jb, kb};
    const float ob3[3] = {bx, by, bz};
    bool start_in = false;
    for (int q = 0; q < bd.n && !start_in; q++) {
      if (bd.kind[q] != 0) continue;
      bool in = true;
#pragma unroll
      for (int d = 0; d < 3; d++)
        in = in && ib3[d] >= bd.lo[q][d] && (ib3[d] < bd.hi[q][d] || (ib3[d] == bd.hi[q][d] && ob3[d] == 0.0f));
      start_in = in;
    }
    if (start_in) {
#pragma unroll
      for (int q = 0; q < NJ; q++) J[q] = 0.f;
    }
  }
  // both segments in the cell of the start point (a particle that did not
  // change cell): one set of node values.  A particle absorbed by a box
  // stops at the relay point (psolve1.F90:660-662): no second segment.
  const bool one = !stop && ax.ia == ib && ay.ia == jb && az.ia == kb;
  if (!one) put_j<B>(box, o, sk, ib, jb, kb, J, c.qfix);
  if (!stop) {
    float J2[NJ];
    float xd = ((float)(ax.ac - ax.ia) + ax.af + (float)(ax.rc - ax.ia) + ax.rf) * 0.5f;
    float yd = ((float)(ay.ac - ay.ia) + ay.af + (float)(ay.rc - ay.ia) + ay.rf) * 0.5f;
    float zd = ((float)(az.ac - az.ia) + az.af + (float)(az.rc - az.ia) + az.rf) * 0.5f;
    float vvx = ((float)(ax.ac - ax.rc) + (ax.af - ax.rf)) * c.rustep;
    float vvy = ((float)(ay.ac - ay.rc) + (ay.af - ay.rf)) * c.rustep;
    float vvz = ((float)(az.ac - az.rc) + (az.af - az.rf)) * c.rustep;
    float w;
    w = yd * zd; J2[3] = vvx * w; J2[1] = vvx * (yd - w); J2[2] = vvx * (zd - w); J2[0] = vvx * (1.0f - yd - (zd - w));
    w = xd * zd; J2[7] = vvy * w; J2[5] = vvy * (xd - w); J2[6] = vvy * (zd - w); J2[4] = vvy * (1.0f - xd - (zd - w));
    w = xd * yd; J2[11] = vvz * w; J2[9] = vvz * (xd - w); J2[10] = vvz * (yd - w); J2[8] = vvz * (1.0f - xd - (yd - w));
    if (one) {
#pragma unroll
      for (int q = 0; q < NJ; q++) J2[q] += J[q];
    }
    put_j<B>(box, o, sk, ax.ia, ay.ia, az.ia, J2, c.qfix);
  }
  }  // JD
  if (!dead) {
    // charge.F90:152-210 at the stored (wrapped / reflected) position
    float X = ax.nf, Y = ay.nf, Z = az.nf;
    float XY = X * Y, XZ = X * Z, YZ = Y * Z, Z2 = 1.0f - Z, XZ2 = X * Z2, YZ2 = Y * Z2;
    float R[NR];
    R[2] = XY * Z; R[1] = XZ - R[2]; R[3] = YZ - R[2]; R[0] = Z - XZ - R[3];
    R[6] = XY * Z2; R[5] = XZ2 - R[6]; R[7] = YZ2 - R[6]; R[4] = Z2 - XZ2 - R[7];
    // The cell comes from the packed one (fewer registers than the axes'), so
    // that of a particle dropped as off the grid unpacks to a z index of no
    // array, and the bounds check of the global deposit reports it.  (A report
    // of its own here or above cost the push 4 to 16 % where many particles
    // cross; this way 0 %, and 1.2 % without the current.)
    int ci, cj, ck;
    unpack(g, nc, ci, cj, ck);
    put_r<B>(box, o, sk, ci, cj, ck, R, c.qfix);
  }
  return escaped ? 1 : 0;
}

// The particles of a warp's cross list (slots in the tile region, still
// holding their position before this step and the velocity the row loop
// gave them): each lane takes one and runs the general path.  Returns the
// number of this lane's particles that escaped.
template <int B, bool DEP, bool CURV, bool JD>
__device__ __forceinline__ int cross_list(const FxPushArgs& a, int is, unsigned long long* box,
                                          const int (&o)[3], const uint32_t* xl, int xn, int lane) {
  __syncwarp();
  // the context comes from the kernel parameters here, so that the pushing
  // loop keeps none of it in registers
  const Geo& g = a.g;
  const Sink sk{a.acc_rho, a.acc_j, a.fr, a.fj, g.nx, g.ny, g.nz, a.status, a.diag};
  const CrossCtx c{a.pos, a.vx, a.vy, a.vz, a.gustep, a.rustep, a.qfix[is],
                   {a.npbnd[is][0], a.npbnd[is][1], a.npbnd[is][2]}, &a.bd, a.gc,
                   a.surf + (int64_t)is * a.bd.nsurf, is, 0, a.ob.rec ? &a.ob : nullptr, a.status};
  int dead = 0;
  for (int e = lane; e < xn; e += 32) {
    const uint32_t m = xl[e];
    const float4 ps = a.rpos[m];  // the position before the step
    const float vx = c.gvx[m], vy = c.gvy[m], vz = c.gvz[m];
    const float en[XQW] = {__int_as_float((int)m), ps.w, ps.x, ps.y, ps.z, vx, vy, vz};
    dead += cross_one<B, DEP, CURV, JD>(g, box, o, sk, c, en);
  }
  __syncwarp();
  return dead;
}

// An end point strictly inside its cell (a region next to a curved body
// raises flo so that none is); one exactly on a face takes the general path
// (it may lie on a body face: inclusive bounds).
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ bool in_cell(float sx, float sy, float sz, float flo) {
  return min3(sx, sy, sz) > flo && max3(sx, sy, sz) < 1.0f;
}

// Out-of-place particles (in another cell than their column's run: they
// changed cell since the sort, or lie outside the tile's box): each lane
// takes one of the list's slots, e of en: kick and move; one that stays in
// its cell adds its sums to the tile accumulator, the others join the warp's
// cross list.  Taken 32 at a time: in the row loop a single such lane would
// cost its warp the 20 sums' stores and most of a queue pass.
template <int B, bool JD, bool PARTS>
__device__ __forceinline__ int oop_list(const FxPushArgs& a, int is, unsigned long long* box,
                                         const ulonglong2* sf0, const f2* sf1, const int (&o)[3], float flo,
                                         const uint32_t* ol, int en, uint32_t* xl, int xqn, int lane) {
  constexpr int NP = (JD ? NJ + NR : NR) / 2;
  __syncwarp();
  const Geo& g = a.g;
  bool cross = false;
  uint32_t m = 0;
  if (lane < en) {
    m = ol[lane];
    const float4 ps = a.rpos[m];
    float vx = a.rvx[m], vy = a.rvy[m], vz = a.rvz[m];
    const uint32_t cell = (uint32_t)__float_as_int(ps.w);
    int ib, jb, kb;
    unpack(g, cell, ib, jb, kb);
    int fb;
    const int gb = box_base<B>(o, ib, jb, kb, fb);
    if (PARTS && gb < 0 && kb + 1 > a.zready) {
      // a part of a step whose eb arrives in z chunks: the node planes of this
      // cell are not converted yet; left as it is for k_fx_deferred
      atomicOr(a.defer + (m >> 5), 1u << (m & 31));
    } else {
      kick<B>(a, sf0, sf1, gb, fb, ib, jb, kb, ps.x, ps.y, ps.z, a.qmp[is], vx, vy, vz);
      a.vx[m] = vx;
      a.vy[m] = vy;
      a.vz[m] = vz;
      const float sx = __fmaf_rn(vx, a.gustep, ps.x), sy = __fmaf_rn(vy, a.gustep, ps.y),
                  sz = __fmaf_rn(vz, a.gustep, ps.z);
      if (gb >= 0 && in_cell(sx, sy, sz, flo)) {
        a.pos[m] = make_float4(sx, sy, sz, ps.w);
        f2 cv[NP];
        cell_sums<JD>(ps.x, ps.y, ps.z, sx, sy, sz, 0.5f * a.rustep, cv);
        const float qfix = a.qfix[is];
#pragma unroll
        for (int q = 0; q < NP; q++) {
          float lo, hi;
          upk(cv[q], lo, hi);
          box_add(&box[gb + sum_off<B, JD>(2 * q)], (unsigned long long)to_fix(lo, qfix));
          box_add(&box[gb + sum_off<B, JD>(2 * q + 1)], (unsigned long long)to_fix(hi, qfix));
        }
      } else {
        cross = true;
      }
    }
  }
  const unsigned xm = __ballot_sync(0xffffffffu, cross);
  if (cross) xl[xqn + __popc(xm & ((1u << lane) - 1u))] = m;
  __syncwarp();
  return xqn + __popc(xm);
}

// DEP = false: the move only (positions, velocities, boundary rules; no
// current, no charge), for recomputing particle states.  CURV = true: a
// particle may end inside a body without leaving its cell (cylinders or
// spheres; boxes after a load of particles that start inside one): tile
// regions next to a body push every particle on the general path; without
// that the in-cell test keeps its constant bound.
// JD = false (the electrostatic step, psolve2 + charge):
// the charge only -- runs of 8 CIC sums, an accumulator of rho alone, no
// zigzag current.
template <int T, bool DEP = true, bool CURV = false, bool JD = true, bool PARTS = false>
__global__ void __launch_bounds__(PUSH_THREADS, 1) k_fx_push(const __grid_constant__ FxPushArgs a) {
  constexpr int B = T + 2 * PG + 1;  // box and field tile edge (nodes)
  constexpr int NC = JD ? NJ + NR : NR;  // sums of a run: zigzag J and CIC rho, or rho alone
  constexpr int NP = NC / 2;             // in pairs
  constexpr int QW = run_words(JD);      // run-queue entry
  constexpr int NACC = (JD ? 4 : 1) * B * B * B;  // accumulator entries (rho, then Jx, Jy, Jz)
  constexpr int NBOX = (NACC + 1) & ~1;  // their 8-byte words, padded: the field nodes after them are float4
  constexpr int NF = B * B * B;
  static_assert((NBOX * 8) % 16 == 0, "the field tile starts on a 16-byte boundary");
  extern __shared__ __align__(128) unsigned long long smem[];
  __shared__ int slot_off[NC];
  const Geo& g = a.g;
  const int is = blockIdx.y;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;

  // this CTA's row chunk (a tile of more than chunk_rows rows is pushed by
  // several CTAs, which add their sums into the same global arrays), from the
  // table the sort leaves: one load instead of a binary search over the tiles'
  // first chunks, a chain of dependent loads in front of everything else
  const int64_t* cs = a.chunk_start + (int64_t)is * (a.ntiles + 1);
  const int64_t b = (a.t_lo > 0 ? cs[a.t_lo] : 0) + blockIdx.x;
  const int4 chunk = b < a.nchunk_max ? __ldg(a.chunks + (int64_t)is * a.nchunk_max + b) : make_int4(0, 0, 0, 0);
  if (b >= cs[a.t_n > 0 ? a.t_lo + a.t_n : a.ntiles]) return;
  const int t = chunk.x, L = chunk.y;
  const int64_t slot0 = a.off[is] + (uint32_t)chunk.z;

  int tx = t % g.nt[0], ty = (t / g.nt[0]) % g.nt[1], tz = t / (g.nt[0] * g.nt[1]);
  const int o[3] = {tx * g.t[0] - PG, ty * g.t[1] - PG, tz * g.t[2] - PG};
  unsigned long long* box = smem;
  float4* sf0 = reinterpret_cast<float4*>(smem + NBOX);
  float2* sf1 = reinterpret_cast<float2*>(sf0 + FieldT<B>::N);
  float* rq = reinterpret_cast<float*>(sf1 + (NF + 1) / 2 * 2) + warp * RQCAP * QW;
  uint32_t* xl = reinterpret_cast<uint32_t*>(reinterpret_cast<float*>(sf1 + (NF + 1) / 2 * 2) + PUSH_WARPS * RQCAP * QW) +
                 warp * (XLCAP + OLCAP);
  uint32_t* ol = xl + XLCAP;
  constexpr int ring_off = NBOX * 8 + FieldT<B>::N * 16 + (NF + 1) / 2 * 16 +
                           PUSH_WARPS * (RQCAP * QW * 4 + (XLCAP + OLCAP) * 4);
  static_assert(ring_off % 16 == 0 && ROW32 % 16 == 0, "16-byte copies");

  // slots are addressed by 32-bit indices from the arrays in the kernel's
  // parameters: eight 64-bit bases would take 16 of the 80 registers
  const uint32_t sl0 = (uint32_t)slot0 + tid;

  char* const ring = reinterpret_cast<char*>(smem) + ring_off + warp * (RING * ROW32);
  // lane 8 q + c of the first 24 copies the c-th 16 bytes of the q-th velocity
  const float* vsrc = (lane < 8 ? a.rvx : lane < 16 ? a.rvy : a.rvz) + (sl0 - lane + 4 * (lane & 7));
  auto fetch = [&](int row, uint32_t slot, char* to) {
    if (row < L) {
      cpa16<false>(to + lane * 16, a.rpos + slot);
      if (lane < 24) cpa16<false>(to + 512 + lane * 16, vsrc);
    }
    vsrc += PUSH_THREADS;
    cpa_commit();
  };
  fetch(0, sl0, ring);
  fetch(1, sl0 + PUSH_THREADS, ring + ROW32);

  if (tid < NC) slot_off[tid] = sum_off<B, JD>(tid);
  if (DEP)
    for (int e = tid; e < NBOX; e += PUSH_THREADS) box[e] = 0ull;
  const int64_t sy = g.nx + 1, sz = (int64_t)(g.nx + 1) * (g.ny + 1);
  const float sq = a.qmp[is];  // the tile's fields times the species' qmp
  for (int e = tid; e < NF; e += PUSH_THREADS) {
    int li = e % B, lj = (e / B) % B, lk = e / (B * B);
    int gi = o[0] + li, gj = o[1] + lj, gk = o[2] + lk;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
    if (gi >= 0 && gj >= 0 && gk >= 0 && gi <= g.nx && gj <= g.ny && gk <= g.nz) {
      int64_t gn = gi + sy * gj + sz * gk;
      p = __ldg(&a.f0[gn]);
      q = __ldg(&a.f1[gn]);
    }
    sf0[(lk * B + lj) * FieldT<B>::W + li] = make_float4(p.x * sq, p.y * sq, p.z * sq, p.w * sq);
    sf1[e] = make_float2(q.x * sq, q.y * sq);
  }
  __syncthreads();

  const float qfix = a.qfix[is];
  const float gustep = a.gustep, hr = 0.5f * a.rustep;
  const ulonglong2* f0s = reinterpret_cast<const ulonglong2*>(sf0);
  const f2* f1s = reinterpret_cast<const f2*>(sf1);
  // A particle can end inside a body without leaving its cell (entering a
  // cylinder or a sphere, or starting inside any body, where the reference's
  // end-point test absorbs it): in a tile region whose box touches a body's
  // cells (a box's lo..hi, its faces included; a curved body's bounding
  // cells), every particle takes the general path, whose absorption test is
  // the reference's (the in-cell test below then fails for all).
  float flo = 0.f;
  if (CURV)
    for (int q = 0; q < a.bd.n; q++) {
      bool hit = true;
#pragma unroll
      for (int d = 0; d < 3; d++) hit = hit && o[d] + B - 2 >= a.bd.lo[q][d] && o[d] <= a.bd.hi[q][d];
      if (hit) flo = 2.0f;
    }

  f2 acc[NP];
#pragma unroll
  for (int s = 0; s < NP; s++) acc[s] = 0ull;
  uint32_t runcell = NORUN;
  int runbase = -1, runfb = 0;
  int nesc = 0;
  int rqn = 0, xqn = 0, oqn = 0;  // warp-uniform queue lengths

  // Row r is read while row r + 1 is in shared memory and r + 2 under way
  // (cp.async into the warp's own ring: the warps share no barrier and no
  // registers hold rows in flight).  The cell of the thread's next particle
  // decides whether a change of cell starts a new run or is a single particle
  // out of place (one that changed cell since the sort: the next one is back in
  // the run's cell), which goes on the out-of-place list and leaves the run
  // intact.
  uint32_t sl = sl0;  // this thread's slot of row r
  int at = 0, at2 = 2 * ROW32;  // the stages of rows r and r + 2
  int r = 0;
  while (r < L) {
  for (; r < L; r++) {
    __syncwarp();  // every lane is through with the row that leaves the ring
    fetch(r + 2, sl + 2 * PUSH_THREADS, ring + at2);
    cpa_wait<1>();
    __syncwarp();
    const char* row = ring + at;
    const float4 ps = *reinterpret_cast<const float4*>(row + lane * 16);
    const float* rv = reinterpret_cast<const float*>(row + 512) + lane;
    float vx = rv[0], vy = rv[32], vz = rv[64];
    at2 = at;  // row r + 3 takes this stage
    at = at + ROW32 == RING * ROW32 ? 0 : at + ROW32;
    uint32_t nextcell = DEAD;
    if (r + 1 < L) nextcell = *reinterpret_cast<const uint32_t*>(ring + at + lane * 16 + 12);
    const uint32_t cell = (uint32_t)__float_as_int(ps.w);
    bool cross = false;
    if (DEP) {
      // ---- a particle in another cell than the thread's run: it ends the
      // run (whose sums go to the run queue) and starts its own, or it is out
      // of place
      bool in = cell == runcell, newrun = false, oop = false;
      int base = runbase, fb = runfb;
      if (!in && cell != DEAD) {
        int ib, jb, kb;
        unpack(g, cell, ib, jb, kb);
        if (ib < g.nx && jb < g.ny && kb < g.nz) {
          base = box_base<B>(o, ib, jb, kb, fb);
          newrun = base >= 0 && (runcell == NORUN || nextcell != runcell);
          oop = !newrun;
        } else {
          report_bad(a.status, a.diag, SITE_FX_PUSH, (int64_t)sl, (long long)cell);
        }
      }
      const bool evict = newrun && runcell != NORUN;
      const unsigned mk = __ballot_sync(0xffffffffu, evict);
      if (mk) queue_runs<NC>(box, slot_off, rq, rqn, mk, evict, acc, runbase, qfix, lane);
      const unsigned om = __ballot_sync(0xffffffffu, oop);
      if (oop) ol[oqn + __popc(om & lt)] = sl;
      oqn += __popc(om);
      // a new run starts from zero: folded into this particle's accumulate
      const f2 keep = dup(newrun ? 0.f : 1.f);
      if (newrun) {
        runcell = cell;
        runbase = base;
        runfb = fb;
        in = true;
      }
      // ---- gather + Buneman-Boris (psolve1.F90:186-272), the move and, in
      // the cell, the sums
      if (in) {
        kick<B, true>(a, f0s, f1s, runbase, runfb, 0, 0, 0, ps.x, ps.y, ps.z, 0.f, vx, vy, vz);
        const float sx = __fmaf_rn(vx, gustep, ps.x), sy = __fmaf_rn(vy, gustep, ps.y),
                    sz = __fmaf_rn(vz, gustep, ps.z);
        // the new velocity of every particle (a cell-crossing one keeps its
        // old position until the general path writes the whole record)
        a.vx[sl] = vx;
        a.vy[sl] = vy;
        a.vz[sl] = vz;
        if (in_cell(sx, sy, sz, flo)) {
          a.pos[sl] = make_float4(sx, sy, sz, ps.w);
          f2 cv[NP];
          cell_sums<JD>(ps.x, ps.y, ps.z, sx, sy, sz, hr, cv);
#pragma unroll
          for (int q = 0; q < NP; q++) acc[q] = fma2(acc[q], keep, cv[q]);
        } else {
          cross = true;
          if (newrun) runcell = NORUN;
        }
      }
    } else if (cell != DEAD) {
      // a move-only step
      int ib, jb, kb;
      unpack(g, cell, ib, jb, kb);
      if (ib < g.nx && jb < g.ny && kb < g.nz) {
        int fb;
        const int gb = box_base<B>(o, ib, jb, kb, fb);
        kick<B>(a, f0s, f1s, gb, fb, ib, jb, kb, ps.x, ps.y, ps.z, a.qmp[is], vx, vy, vz);
        const float sx = __fmaf_rn(vx, gustep, ps.x), sy = __fmaf_rn(vy, gustep, ps.y),
                    sz = __fmaf_rn(vz, gustep, ps.z);
        cross = !in_cell(sx, sy, sz, flo);
        if (!cross) a.pos[sl] = make_float4(sx, sy, sz, ps.w);
      } else {
        report_bad(a.status, a.diag, SITE_FX_PUSH, (int64_t)sl, (long long)cell);
        a.pos[sl] = ps;
      }
      a.vx[sl] = vx;
      a.vy[sl] = vy;
      a.vz[sl] = vz;
    } else {
      // it may write into other arrays than it reads: empty and dead slots
      // are carried over
      a.pos[sl] = ps;
      a.vx[sl] = vx;
      a.vy[sl] = vy;
      a.vz[sl] = vz;
    }
    // ---- cell-crossing particles: the warp's cross list (their positions
    // stay as they were; the general path after the row loop moves them)
    const unsigned xm = __ballot_sync(0xffffffffu, cross);
    if (cross) xl[xqn + __popc(xm & lt)] = sl;
    xqn += __popc(xm);
    sl += PUSH_THREADS;
    if (xqn > XLCAP - 32 || oqn > OLCAP - 32) {  // take full batches, then go on with the next row
      r++;
      break;
    }
  }
  // the lists: whole batches of 32 while rows are left, everything at the end
  const bool last = r >= L;
  if (DEP) {
    while (oqn >= 32 || (last && oqn > 0)) {
      const int k = min(oqn, 32);
      oqn -= k;
      if (xqn > XLCAP - 32) {
        xqn -= 32;
        nesc += cross_list<B, DEP, CURV, JD>(a, is, box, o, xl + xqn, 32, lane);
      }
      xqn = oop_list<B, JD, PARTS>(a, is, box, f0s, f1s, o, flo, ol + oqn, k, xl, xqn, lane);
    }
  }
  while (xqn > XLCAP - 32 || (last && xqn > 0)) {
    const int k = min(xqn, 32);
    xqn -= k;
    nesc += cross_list<B, DEP, CURV, JD>(a, is, box, o, xl + xqn, k, lane);
  }
  }
  // the last run of every thread, and what is left in the queue
  if (DEP) {
    const bool has = runcell != NORUN;
    const unsigned mk = __ballot_sync(0xffffffffu, has);
    if (mk) queue_runs<NC>(box, slot_off, rq, rqn, mk, has, acc, runbase, qfix, lane);
    if (rqn) drain_runs<NC>(box, slot_off, rq, rqn, qfix, lane);
  }
  if (nesc) atomicAdd(&a.nesc[is], nesc);
  __syncthreads();
  // add the tile accumulator into the global int64 arrays
  if (DEP) {
    for (int e = tid; e < NACC; e += PUSH_THREADS) {
      unsigned long long v = box[e];
      if (v == 0ull) continue;
      int li = e % B, lj = (e / B) % B, lk = (e / (B * B)) % B, comp = e / (B * B * B);
      int i = o[0] + li, j = o[1] + lj, k = o[2] + lk;
      if (comp == 0) {
        if (i < -1 || j < -1 || k < -1 || i > g.nx + 1 || j > g.ny + 1 || k > g.nz + 1) {
          report_bad(a.status, a.diag, SITE_FX_FLUSH, t, i + 100000LL * j + 10000000000LL * k);
          continue;
        }
        atomicAdd(&a.acc_rho[a.fr.at(0, i, j, k)], v);
      } else {
        if (i < -4 || j < -4 || k < -4 || i > g.nx + 4 || j > g.ny + 4 || k > g.nz + 4) {
          report_bad(a.status, a.diag, SITE_FX_FLUSH, t, i + 100000LL * j + 10000000000LL * k);
          continue;
        }
        atomicAdd(&a.acc_j[a.fj.at(comp - 1, i, j, k)], v);
      }
    }
  }
}

// The entries of tile t's row chunks (FxPushArgs::chunks) from its first one.
__device__ __forceinline__ void put_chunks(int4* out, int64_t first, int64_t t, int64_t rows, int64_t slot,
                                           int chunk_rows) {
  for (int64_t r = 0; r < rows; r += chunk_rows)
    out[first++] = make_int4((int)t, (int)min((int64_t)chunk_rows, rows - r), (int)(uint32_t)(slot + r * PUSH_THREADS), 0);
}

// The row chunks of every tile region: cs[t] = first chunk of tile t,
// cs[ntiles] = the number of chunks (one block of 1024 threads per species),
// and their entries.
__global__ void __launch_bounds__(1024) k_push_chunks(const int64_t* __restrict__ tile_start,
                                                      const int64_t* __restrict__ tile_pad, int64_t ntiles,
                                                      int64_t* chunk_start, int4* chunks, int64_t nchunk_max,
                                                      int chunk_rows) {
  __shared__ int64_t pa[1024];
  const int64_t* ts = tile_start + (int64_t)blockIdx.x * (ntiles + 1);
  const int64_t* tp = tile_pad + (int64_t)blockIdx.x * (ntiles + 1);
  int64_t* cs = chunk_start + (int64_t)blockIdx.x * (ntiles + 1);
  const int tid = threadIdx.x;
  const int64_t per = (ntiles + 1023) / 1024;
  const int64_t t0 = tid * per, t1 = min(ntiles, t0 + per);
  auto rows = [&](int64_t t) { return (ts[t + 1] - ts[t] + PUSH_THREADS - 1) / PUSH_THREADS; };
  int64_t sa = 0;
  for (int64_t t = t0; t < t1; t++) sa += (rows(t) + chunk_rows - 1) / chunk_rows;
  pa[tid] = sa;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int64_t v = tid >= d ? pa[tid - d] : 0;
    __syncthreads();
    pa[tid] += v;
    __syncthreads();
  }
  int64_t ra = pa[tid] - sa;
  for (int64_t t = t0; t < t1; t++) {
    cs[t] = ra;
    const int64_t r = rows(t);
    put_chunks(chunks + (int64_t)blockIdx.x * nchunk_max, ra, t, r, tp[t], chunk_rows);
    ra += (r + chunk_rows - 1) / chunk_rows;
  }
  if (tid == 1023) cs[ntiles] = pa[1023];
}

// Injected particles of the tail zone of species `is`, one thread each: the
// random fraction of the step for a particle injected since the last push
// (psolve1.F90:150-156: gustep = ustep * U), gather from the global node
// field, Buneman-Boris, and the general path with global deposits.
template <bool JD>
__global__ void k_fx_tail(FxPushArgs a, int is, int64_t tail0, int64_t ntail, int32_t* ord, int ustep,
                          const double* randoms, int64_t nrand, const int64_t* rand_pos, int64_t ord_base,
                          uint64_t seed, uint64_t stream, int* nesc_out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ntail) return;
  const Geo& g = a.g;
  const int64_t base = a.off[is];
  const int64_t slot = tail0 + k;
  const float4 ps = a.pos[base + slot];
  const uint32_t cell = (uint32_t)__float_as_int(ps.w);
  if (cell == DEAD) return;
  int ib, jb, kb;
  unpack(g, cell, ib, jb, kb);
  if (ib >= g.nx || jb >= g.ny || kb >= g.nz) {
    report_bad(a.status, a.diag, SITE_FX_PUSH, base + slot, (long long)cell);
    return;
  }
  float gus = (float)ustep;
  const int32_t o1 = ord[k];
  if (o1 > 0) {
    double u;
    const int64_t j = ord_base + o1 - 1;
    if (randoms) {
      const int64_t r = *rand_pos + j;
      if (r >= nrand) {
        atomicOr(a.status, ST_RANDOMS);
        u = 0.0;
      } else {
        u = randoms[r];
      }
    } else {
      u = hash_u01(seed, stream, (uint64_t)j);
    }
    gus = (float)((double)ustep * u);
    ord[k] = 0;
  }
  const float qmp = (float)((double)a.qmp[is] / (double)a.gustep * (double)gus);
  float vx = a.vx[base + slot], vy = a.vy[base + slot], vz = a.vz[base + slot];
  const float x1 = ps.x, y1 = ps.y, z1 = ps.z;
  const float xy1 = x1 * y1, xz1 = x1 * z1, yz1 = y1 * z1, z2 = 1.0f - z1;
  const float xz2 = x1 * z2, yz2 = y1 * z2;
  float wv[8];
  wv[2] = xy1 * z1; wv[1] = xz1 - wv[2]; wv[3] = yz1 - wv[2]; wv[0] = z1 - xz1 - wv[3];
  wv[6] = xy1 * z2; wv[5] = xz2 - wv[6]; wv[7] = yz2 - wv[6]; wv[4] = z2 - xz2 - wv[7];
  float fe[3], fb[3];
  const int64_t sy = g.nx + 1, sz = (int64_t)(g.nx + 1) * (g.ny + 1);
  gather8(a.f0, a.f1, ib + sy * jb + sz * kb, sy, sz, wv, fe, fb);
  const float eex = fe[0] * qmp, eey = fe[1] * qmp, eez = fe[2] * qmp;
  const float bbx = fb[0] * qmp, bby = fb[1] * qmp, bbz = fb[2] * qmp;
  const float boris = 2.0f / (1.0f + bbx * bbx + bby * bby + bbz * bbz);
  vx += eex; vy += eey; vz += eez;
  const float vxt = vx + vy * bbz - vz * bby;
  const float vyt = vy + vz * bbx - vx * bbz;
  const float vzt = vz + vx * bby - vy * bbx;
  vx += boris * (vyt * bbz - vzt * bby);
  vy += boris * (vzt * bbx - vxt * bbz);
  vz += boris * (vxt * bby - vyt * bbx);
  vx += eex; vy += eey; vz += eez;
  const Sink sk{a.acc_rho, a.acc_j, a.fr, a.fj, g.nx, g.ny, g.nz, a.status, a.diag};
  const CrossCtx c{a.pos + base, a.vx + base, a.vy + base, a.vz + base, gus, a.rustep, a.qfix[is],
                   {a.npbnd[is][0], a.npbnd[is][1], a.npbnd[is][2]}, &a.bd, a.gc,
                   a.surf + (int64_t)is * a.bd.nsurf, is, base, a.ob.rec ? &a.ob : nullptr, a.status};
  const float en[XQW] = {__int_as_float((int)slot), ps.w, ps.x, ps.y, ps.z, vx, vy, vz};
  const int far[3] = {-(1 << 28), -(1 << 28), -(1 << 28)};  // no box: global deposits
  const int esc = cross_one<11, true, true, JD>(g, nullptr, far, sk, c, en);
  if (esc) atomicAdd(nesc_out, esc);
}

// The particles the parts of a step left for later (FxPushArgs::defer: a
// gather from node planes converted after their part ran), once every plane
// is converted: what the row loop and the general path do for a particle
// whose cell lies outside its tile's box -- the global gather and the kick,
// then the general path with global deposits (a deposit takes the same
// int64 value per node as through a tile's box).  The same bits as from the
// step pushed in one launch.  One thread per 32-slot word of the bitmap, which
// it clears.
template <int T, bool CURV, bool JD>
__global__ void k_fx_deferred(FxPushArgs a, uint32_t* __restrict__ bits, int64_t nwords, int nspec) {
  constexpr int B = T + 2 * PG + 1;
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  uint32_t m = bits[w];
  if (m == 0u) return;
  bits[w] = 0u;
  const Geo& g = a.g;
  const Sink sk{a.acc_rho, a.acc_j, a.fr, a.fj, g.nx, g.ny, g.nz, a.status, a.diag};
  const int far[3] = {-(1 << 28), -(1 << 28), -(1 << 28)};  // no box: global deposits
  while (m) {
    const int64_t slot = w * 32 + (__ffs(m) - 1);
    m &= m - 1u;
    int is = 0;
    for (int s = 1; s < nspec; s++)
      if (slot >= a.off[s]) is = s;
    const int64_t base = a.off[is];
    const float4 ps = a.pos[slot];
    const uint32_t cell = (uint32_t)__float_as_int(ps.w);
    int ib, jb, kb;
    unpack(g, cell, ib, jb, kb);
    if (cell == DEAD || ib >= g.nx || jb >= g.ny || kb >= g.nz) {
      report_bad(a.status, a.diag, SITE_FX_PUSH, slot, (long long)cell);
      continue;
    }
    float vx = a.vx[slot], vy = a.vy[slot], vz = a.vz[slot];
    kick<B>(a, nullptr, nullptr, -1, 0, ib, jb, kb, ps.x, ps.y, ps.z, a.qmp[is], vx, vy, vz);
    a.vx[slot] = vx;
    a.vy[slot] = vy;
    a.vz[slot] = vz;
    const CrossCtx c{a.pos + base, a.vx + base, a.vy + base, a.vz + base, a.gustep, a.rustep, a.qfix[is],
                     {a.npbnd[is][0], a.npbnd[is][1], a.npbnd[is][2]}, &a.bd, a.gc,
                     a.surf + (int64_t)is * a.bd.nsurf, is, base, a.ob.rec ? &a.ob : nullptr, a.status};
    const float en[XQW] = {__int_as_float((int)(slot - base)), ps.w, ps.x, ps.y, ps.z, vx, vy, vz};
    const int esc = cross_one<B, true, CURV, JD>(g, nullptr, far, sk, c, en);
    if (esc) atomicAdd(&a.nesc[is], esc);
  }
}

// The compiled box edge for the largest tile edge tmax (<= 8).
inline int fx_box_tile(int tmax) { return tmax <= 4 ? 4 : 8; }

// Dynamic shared memory of the push: int64 accumulator (4 components, or
// rho alone without the current), field tile, run queues and lists.
template <int B>
constexpr int fx_push_smem_t(bool jd) {
  const int nf = B * B * B, nbox = ((jd ? 4 : 1) * nf + 1) & ~1;  // as NBOX in k_fx_push
  return nbox * (int)sizeof(unsigned long long) + FieldT<B>::N * (int)sizeof(float4) + (nf + 1) / 2 * 16 +
         PUSH_WARPS * (RQCAP * run_words(jd) * (int)sizeof(float) + (XLCAP + OLCAP) * (int)sizeof(int) + RING * ROW32);
}
inline int fx_push_smem(int tmax, bool jd = true) {
  return fx_box_tile(tmax) == 4 ? fx_push_smem_t<4 + 2 * PG + 1>(jd) : fx_push_smem_t<8 + 2 * PG + 1>(jd);
}

// The pushing kernel (DEP = true) for a compiled box tile (4 or 8), runs
// with cylinders or spheres, and with (jd) or without the current.
using PushKernel = void (*)(FxPushArgs);
using DeferredKernel = void (*)(FxPushArgs, uint32_t*, int64_t, int);
inline DeferredKernel deferred_kernel(int box, bool curved, bool jd) {
  if (box == 4) {
    if (curved) return jd ? k_fx_deferred<4, true, true> : k_fx_deferred<4, true, false>;
    return jd ? k_fx_deferred<4, false, true> : k_fx_deferred<4, false, false>;
  }
  if (curved) return jd ? k_fx_deferred<8, true, true> : k_fx_deferred<8, true, false>;
  return jd ? k_fx_deferred<8, false, true> : k_fx_deferred<8, false, false>;
}

template <bool PARTS>
inline PushKernel push_kernel_t(int box, bool curved, bool jd) {
  if (box == 4) {
    if (curved) return jd ? k_fx_push<4, true, true, true, PARTS> : k_fx_push<4, true, true, false, PARTS>;
    return jd ? k_fx_push<4, true, false, true, PARTS> : k_fx_push<4, true, false, false, PARTS>;
  }
  if (curved) return jd ? k_fx_push<8, true, true, true, PARTS> : k_fx_push<8, true, true, false, PARTS>;
  return jd ? k_fx_push<8, true, false, true, PARTS> : k_fx_push<8, true, false, false, PARTS>;
}
inline PushKernel push_kernel(int box, bool curved, bool jd, bool parts = false) {
  return parts ? push_kernel_t<true>(box, curved, jd) : push_kernel_t<false>(box, curved, jd);
}
