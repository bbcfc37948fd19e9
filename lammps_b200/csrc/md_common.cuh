// md_common.cuh -- shared device definitions of the B200 MD engine.
//
// Device-resident layout of one box (all arrays in cell-sorted order):
//   x4[i]      double4 (x, y, z, type)       -- FP64 positions, gathered per pair
//   v[3][n]    double SoA                     -- velocities
//   f[3][n]    double SoA                     -- forces (owner-summed; no ghosts)
//   xq[i]      int4 (x, y, z as 32-bit fixed-point fractions of the box edge,
//              type) -- mixed precision only (md_xq)
//   cell[i]    packed cell coordinates cx | cy<<10 | cz<<20 of the last build
//   nlist      neighbor list in int4 slabs (md_slab): bits 6..31 = neighbor
//              atom index, bits 0..5 = offset of the neighbor's cell from the
//              atom's cell, two bits per dimension (d+1 for d = -1,0,1).
// Periodic images are never stored: a neighbor in a wrapped cell is the owner
// atom plus the box shift implied by the offset code, so the reference's
// ghost atoms, forward_comm and reverse_comm disappear.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define MD_MAXTYPES 8
#define MD_ADJ_MAXTYPES 4  // types of the force-matching adjoint (16 type pairs)
#define MD_JBITS 26
#define MD_JMASK ((1u << MD_JBITS) - 1u)
#define MD_MAX_ATOMS ((int)MD_JMASK)
#define MD_CELLBITS 10
#define MD_MAX_CELLS_DIM (1 << MD_CELLBITS)

// status words in device memory (read by the host after a step or a run)
enum {
  // the first four are cleared together before a build (rebuild_sync)
  ST_MAXNEIGH = 0,   // largest per-atom full-list count seen at the last build
  ST_OVERFLOW = 1,   // a build exceeded the list capacity (sticky)
  ST_MAXSTAGE = 2,   // most shared memory (16-byte units) one builder tile needed
  ST_UNSTAGED = 3,   // atoms of builder tiles that no capacity could stage
  ST_MOVED = 12,     // some atom moved more than half the skin (check yes)
  ST_AGO = 4,        // steps since the last build (Neighbor::ago)
  ST_NCALLS = 5,     // builds since setup (Neighbor::ncalls)
  ST_NDANGER = 6,    // dangerous builds (Neighbor::ndanger)
  ST_LOST = 7,       // a coordinate was non-finite or beyond one box image
  ST_ROW = 8,        // thermo rows written by the device in this run
  ST_STEP_LO = 9,    // current timestep (low/high 32 bits)
  ST_STEP_HI = 10,
  ST_FORCE_BUILD = 11,  // rebuild on the next step regardless of the schedule
  ST_HALO_BAD = 13,     // a halo pack/unpack index was outside [0, n)
  ST_BADTYPE = 14,      // 1 + index of an uploaded atom with a type outside [1, ntypes]
  ST_BARRIER = 15,      // a grid barrier of a multi-step launch gave up
  ST_REBUILD = 16,      // decision of the current step
  ST_COUNT = 17
};

struct BoxGeom {
  double lo[3], hi[3], prd[3];
  double cinv[3];    // cells per unit length: ncell/prd
  double cs[3];      // cell edge prd/ncell
  double qinv[3];    // fixed-point units per unit length: 2^32/prd (md_xq)
  // length of one fixed-point unit, prd/2^32, as an FP32 pair hi + lo (a
  // single FP32 value would scale every separation by the same rounding
  // error); and 1/unit^2 the same way, for one unit in every dimension
  float qs[3], qs_lo[3];
  float q2inv, q2inv_lo;
  int qiso;          // the three edges are equal (one fixed-point unit)
  int ncell[3];
};

// Replica tables of a batched context: several independent periodic boxes
// advanced together in one set of device arrays.  The atoms of replica r
// always occupy the sorted indices [atom_start[r], atom_start[r+1]) (a
// rebuild only permutes atoms within their replica), and its cells the
// global cell indices [cell_base[r], cell_base[r] + ncells(r)).
struct Reps {
  const BoxGeom *box;      // per replica
  const int *rep_of_atom;  // per sorted atom index (fixed)
  const int *cell_base;    // per replica
  const int *tile_rep;     // per neighbor-builder tile
  const int *tile_base;    // per replica: its first builder tile
};

struct LJParamsDev {
  // (ntypes+1)^2 tables, row-major, as LAMMPS's 1-based arrays
  double cutsq[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  double lj1[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  double lj2[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  double lj3[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  double lj4[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  double offset[(MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
};

__host__ __device__ inline int md_cell_pack(int cx, int cy, int cz) {
  return cx | (cy << MD_CELLBITS) | (cz << (2 * MD_CELLBITS));
}
__host__ __device__ inline void md_cell_unpack(int c, int &cx, int &cy, int &cz) {
  cx = c & (MD_MAX_CELLS_DIM - 1);
  cy = (c >> MD_CELLBITS) & (MD_MAX_CELLS_DIM - 1);
  cz = c >> (2 * MD_CELLBITS);
}

// neighbor-cell offset code of a list entry: (dx+1) | (dy+1)<<2 | (dz+1)<<4
__host__ __device__ inline int md_code(int dx, int dy, int dz) {
  return (dx + 1) | ((dy + 1) << 2) | ((dz + 1) << 4);
}
#define MD_CODE_SELF 21  // md_code(0, 0, 0)
// Filler of the unused tail of an atom's last slab: the atom itself at a
// cell offset of +2 in every dimension (code bits 3), at least
// sqrt(3) * cell edge > rc + skin away, so a kernel that reads whole slabs
// rejects it by the cutoff test without checking the count.
#define MD_CODE_PAD 63
__host__ __device__ inline int md_pad_entry(int i) { return (int)(((unsigned)i << 6) | 63u); }
// list entry of neighbor j in the cell at offset code `code`
__host__ __device__ inline int md_make_entry(int j, int code) {
  return (int)(((unsigned)j << 6) | (unsigned)code);
}
__host__ __device__ inline int md_entry_j(unsigned e) { return (int)(e >> 6); }

// Periodic shift of a neighbour in the cell at offset d (-1, 0, +1) from
// cell c along one dimension: -prd / +prd when that cell wraps, else 0
struct Shift3 {
  double m, p;
};
__device__ __forceinline__ Shift3 shifts(int c, int nc, double prd) {
  Shift3 s;
  s.m = (c - 1 < 0) ? -prd : 0.0;
  s.p = (c + 1 >= nc) ? prd : 0.0;
  return s;
}
__device__ __forceinline__ double pick(const Shift3 &s, int d) {
  return d < 0 ? s.m : (d > 0 ? s.p : 0.0);
}

// Coordinates of the mixed form.  Each coordinate is a 32-bit fixed-point
// fraction of its periodic box edge: 2^32 units per edge, taken modulo 2^32.
// The difference of two such coordinates in 32-bit two's-complement
// arithmetic is the separation along that edge reduced to the minimum image
// (exact, with no periodic shift to decode), and one conversion turns it into
// an FP32 number of units.  A listed pair is at its minimum image whenever
// the box edge exceeds twice the list cutoff, which the mixed form requires.
// The quantisation step is prd / 2^32 (3.9e-8 sigma on the 168-sigma edge of
// a 4M-atom LJ box), below the FP32 rounding of a separation of one sigma.
__device__ __forceinline__ int md_fix(double x, double lo, double qinv) {
  return (int)(unsigned int)(unsigned long long)__double2ll_rn(__dmul_rn(x - lo, qinv));
}
__device__ __forceinline__ int4 md_xq(const double4 &p, const BoxGeom &b) {
  return make_int4(md_fix(p.x, b.lo[0], b.qinv[0]), md_fix(p.y, b.lo[1], b.qinv[1]),
                   md_fix(p.z, b.lo[2], b.qinv[2]), (int)p.w);
}
// separation a - b along one edge in fixed-point units, as an FP32 number
__device__ __forceinline__ float md_qdiff(int a, int b) {
  return (float)(int)((unsigned int)a - (unsigned int)b);
}
// u units in length units: u * (hi + lo) rounded once (the small product
// u * lo first, then one fused multiply-add; rounding u * hi first and adding
// the correction after would leave a bias of a fraction of an ulp)
__device__ __forceinline__ float md_qlen(float u, float hi, float lo) {
  return fmaf(u, hi, u * lo);
}

__host__ __device__ inline void md_entry(unsigned int e, int &j, int &dx, int &dy, int &dz) {
  j = (int)(e >> 6);
  dx = (int)(e & 3u) - 1;
  dy = (int)((e >> 2) & 3u) - 1;
  dz = (int)((e >> 4) & 3u) - 1;
}

// Slab layout of the neighbor list: entry k of atom i is at
//   nlist[((k >> 2) * stride + i) * 4 + (k & 3)]
// so that one int4 load returns four consecutive entries of an atom and the
// 32 atoms of a warp read 512 contiguous bytes per slab.
__host__ __device__ inline size_t md_slab(int k, int i, int stride) {
  return ((size_t)(k >> 2) * stride + i) * 4 + (k & 3);
}

// image flags packed as LAMMPS imageint: 10 bits per dimension, offset 512
// (src/lmptype.h IMGMAX/IMGBITS)
#define MD_IMGMAX 512
#define MD_IMGMASK 1023
__host__ __device__ inline int md_img_pack(int ix, int iy, int iz) {
  return ((iz + MD_IMGMAX) & MD_IMGMASK) << 20 | ((iy + MD_IMGMAX) & MD_IMGMASK) << 10 |
         ((ix + MD_IMGMAX) & MD_IMGMASK);
}

// 1/x in FP64: Newton's method on f(y) = 1/y - x, i.e. the iteration
// y <- y + y (1 - x y), started from the hardware reciprocal approximation
// (rcp.approx.ftz.f64) and applied twice.  For the normal, positive x used
// here the result is within two ulp of the correctly rounded quotient; the
// FP64 parity tests bound its effect on forces.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// 1/x in FP32 from the hardware reciprocal approximation alone (one
// instruction, relative error below 2^-22); the mixed-precision kernels use it
// where the pair term's FP32 error budget is far larger.
__device__ __forceinline__ float rcp_approx_f32(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Position loads of the pair loops.  A kernel that runs several steps reads
// positions that other blocks wrote earlier in the same launch: COH makes
// them plain loads (ordered by the grid barrier) instead of read-only ones.
template <bool COH>
__device__ __forceinline__ int4 ld_pos(const int4 *p) {
  if (!COH) return __ldg(p);
  int4 v;
  asm volatile("ld.global.v4.s32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
template <bool COH>
__device__ __forceinline__ double4 ld_pos(const double4 *p) {
  // one 32-byte load: a gather of 32-byte records by two 16-byte loads takes
  // a fifth more passes through the L1 data banks
  double4 v;
  if (COH)
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  else
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// A rejected pair's separation in the branch-free FP64 pair loops: zero, so
// that the pair adds nothing even where its neighbour's coordinates are not
// finite (a zero factor alone would make them NaN forces on every atom whose
// list names that neighbour; PairLJCut::compute and PairEAM::compute skip the
// pair).  Selecting the separations, not the sums, measured least: lj/cut at
// 495,709 atoms 8.69 ms a run against 8.70 with the factor alone and 8.88 with
// predicated sums.
__device__ __forceinline__ void drop_unless(bool in, double &dx, double &dy, double &dz) {
  dx = in ? dx : 0.0;
  dy = in ? dy : 0.0;
  dz = in ? dz : 0.0;
}

// FP64 helpers that keep a*b+c rounded twice, as the reference's x86-64
// build computes them; used wherever a comparison must be bit-exact.
__device__ __forceinline__ double dsq3(double a, double b, double c) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
}

// The entries that one lane of an atom takes from the atom's list, G at a
// time, with the next G already loading (streaming loads).  The list holds
// each atom's entries in slabs of four: slab c of atom i is int4 number
// c * stride + i.  Several lanes per atom (TPA > 1): the atom's lanes take
// consecutive entries (lane s: entries s, s + TPA, s + 2 TPA, ...), so that
// at each gather the lanes of one atom read neighbours that sit next to each
// other in the cell-sorted order and share cache lines.  The lane's G
// offsets from its row pointer are fixed, and the pointer advances by
// TPA * G / 4 slab rows per step.  Entries past the atom's last slab read as
// `pad`.  (One lane per atom reads whole slabs and does not use this.)
template <int TPA, int G>
struct ListWalk {
  static_assert(TPA > 1 && (TPA * G) % 4 == 0, "whole slab rows per step");
  const int *p;       // row pointer of the current step
  long long off[G];   // offsets (in ints) of the lane's G entries from p
  long long adv;      // ints between steps
  int e0, ne;         // first entry of the current step; 4 x the slab count
  unsigned pad;
  unsigned cur[G], nxt[G];
  __device__ __forceinline__ ListWalk(const int *nl, int stride, int i, int nslab, int lane,
                                      unsigned pad_)
      : p(nl + (size_t)i * 4), adv((long long)(TPA * G / 4) * stride * 4), e0(lane),
        ne(nslab * 4), pad(pad_) {
#pragma unroll
    for (int u = 0; u < G; u++) {
      const int e = lane + TPA * u;
      off[u] = (long long)(e >> 2) * stride * 4 + (e & 3);
    }
    load(cur, p, e0);
  }
  __device__ __forceinline__ void load(unsigned (&v)[G], const int *q, int first) const {
#pragma unroll
    for (int u = 0; u < G; u++)
      v[u] = first + TPA * u < ne ? (unsigned)__ldcs(q + off[u]) : pad;
  }
  __device__ __forceinline__ bool more() const { return e0 < ne; }
  // start loading the next step's entries; cur holds this step's
  __device__ __forceinline__ void prefetch() { load(nxt, p + adv, e0 + TPA * G); }
  // how many of this step's entries lie before `num` (the rest are pads)
  __device__ __forceinline__ int valid(int num) const {
    return e0 >= num ? 0 : min(G, (num - e0 + TPA - 1) / TPA);
  }
  __device__ __forceinline__ void advance() {
#pragma unroll
    for (int u = 0; u < G; u++) cur[u] = nxt[u];
    p += adv;
    e0 += TPA * G;
  }
};

// Calls f(ee, m) for each group of four entries that this lane takes from
// atom i's list: ee the entries, m how many of them lie before the atom's
// count num (the rest are pads).  One lane per atom: the slabs in order, the
// next slab loading (streaming) while this one is used.  Several lanes per
// atom: ListWalk's consecutive entries.
template <int TPA, class F>
__device__ __forceinline__ void walk_list(const int *nl, int stride, int i, int num, int lane,
                                          F &&f) {
  const int nslab = (num + 3) >> 2;
  if constexpr (TPA == 1) {
    const int4 *nl4 = reinterpret_cast<const int4 *>(nl);
    int4 en = make_int4(0, 0, 0, 0);
    if (nslab > 0) en = __ldcs(&nl4[i]);
    for (int c4 = 0; c4 < nslab; c4++) {
      const int4 e4 = en;
      if (c4 + 1 < nslab) en = __ldcs(&nl4[(size_t)(c4 + 1) * stride + i]);
      const unsigned ee[4] = {(unsigned)e4.x, (unsigned)e4.y, (unsigned)e4.z, (unsigned)e4.w};
      f(ee, min(4, num - 4 * c4));
    }
  } else {
    ListWalk<TPA, 4> w(nl, stride, i, nslab, lane, (unsigned)md_pad_entry(i));
    while (w.more()) {
      w.prefetch();
      f(w.cur, w.valid(num));
      w.advance();
    }
  }
}

template <int TPA>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = TPA / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int TPA>
__device__ __forceinline__ float lane_sumf(float v) {
#pragma unroll
  for (int o = TPA / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum NV doubles over the block; result valid in thread 0.  smem must hold
// NV * (blockDim.x/32) doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *smem) {
#pragma unroll
  for (int k = 0; k < NV; k++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) smem[k * nw + warp] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double s = 0.0;
      for (int w = 0; w < nw; w++) s += smem[k * nw + w];
      v[k] = s;
    }
  }
}

// Deterministic two-level reduction: each block writes NV partial sums, the
// last block to finish adds all partials in block order into out[0..NV-1]
// (overwrite or accumulate) and resets the counter for the next launch.
template <int NV>
__device__ __forceinline__ void block_partials_finish(double (&v)[NV], double *smem,
                                                      double *partial, unsigned int *counter,
                                                      double *out, bool accumulate) {
  block_sum<NV>(v, smem);
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) partial[(size_t)blockIdx.x * NV + k] = v[k];
    __threadfence();
    unsigned int done = atomicAdd(counter, 1u);
    last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    // every thread of the last block sums a fixed strided subset of the
    // block partials, then the block tree-reduces them: a fixed order, so
    // the result is reproducible run to run
    double s[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) s[k] = 0.0;
    for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
      for (int k = 0; k < NV; k++) s[k] += __ldcg(&partial[(size_t)b * NV + k]);
    __syncthreads();
    block_sum<NV>(s, smem);
    if (threadIdx.x == 0) {
#pragma unroll
      for (int k = 0; k < NV; k++) out[k] = accumulate ? out[k] + s[k] : s[k];
      *counter = 0u;
    }
  }
}

// ---- step logic shared by the fused half-step kernel (integrate.cu) and the
// one-launch replica step (pair_lj.cu) ---------------------------------------

// Neighbor::decide (src/neighbor.cpp:1294-1309) on the device: the host
// mirrors the same schedule and reads ST_REBUILD only when the distance
// criterion decides.
__device__ __forceinline__ void md_decide_dev(int *status, int every, int delay, int check,
                                           int *dcount, volatile int *mail) {
  const int ago = status[ST_AGO] + 1;
  status[ST_AGO] = ago;
  int rebuild = 0;
  const bool candidate = ago >= delay && ago % every == 0;
  if (candidate) {
    if (!check) rebuild = 1;
    else {
      rebuild = status[ST_MOVED] != 0;
      if (rebuild && ago == (every > delay ? every : delay)) status[ST_NDANGER] += 1;
    }
  }
  bool forced = false;
  if (status[ST_FORCE_BUILD]) {  // replay after a list overflow: lists are stale
    rebuild = 1;
    forced = true;
    status[ST_FORCE_BUILD] = 0;
  }
  status[ST_MOVED] = 0;
  status[ST_REBUILD] = rebuild;
  unsigned int lo = (unsigned int)status[ST_STEP_LO] + 1u;
  if (lo == 0u) status[ST_STEP_HI] += 1;
  status[ST_STEP_LO] = (int)lo;
  if (check && candidate && !forced) {
    // a decision the host waits for (the distance criterion): the flag
    // first, then, after a system-wide fence, the new decision count
    const int k = *dcount + 1;
    *dcount = k;
    mail[0] = rebuild;
    __threadfence_system();
    mail[1] = k;
  }
}

__device__ __forceinline__ void md_record_row_dev(int *status, const double *ev, double *rows,
                                               int cap) {
  const int r = status[ST_ROW];
  if (r < cap) {
    double *row = rows + 9 * (size_t)r;
    const long long step = ((long long)(unsigned int)status[ST_STEP_HI] << 32) |
                           (long long)(unsigned int)status[ST_STEP_LO];
    row[0] = (double)step;
    row[1] = ev[7];
    row[2] = ev[0];
    for (int k = 0; k < 6; k++) row[3 + k] = ev[1 + k];
  }
  status[ST_ROW] = r + 1;
}

// FixNVE::final_integrate of this step for sorted atom i with its force
// (fx, fy, fz), the kinetic-energy term of the thermo output (KE, into ke),
// then FixNVE::initial_integrate of the next step (src/fix_nve.cpp:65-142):
// every product and sum rounded separately as in the reference.  The new
// position goes to x4_out (x4_in itself for an update in place) and, in the
// mixed form, its fixed-point copy to xq_out.  Returns whether the atom moved
// more than half the skin since the last build (xhold, check yes).
template <bool KE>
__device__ __forceinline__ bool md_nve_step_atom(int i, int stride, double dtv, double dtf,
                                                 const double *__restrict__ mass,
                                                 const double4 *x4_in, double4 *x4_out,
                                                 double *__restrict__ v, double fx, double fy,
                                                 double fz, int4 *__restrict__ xq_out,
                                                 const BoxGeom &box,
                                                 const double4 *__restrict__ xhold,
                                                 double triggersq, double &ke) {
  double4 p = x4_in[i];
  const double m = mass[(int)p.w];
  const double dtfm = dtf / m;
  double vx = __dadd_rn(v[i], __dmul_rn(dtfm, fx));
  double vy = __dadd_rn(v[stride + i], __dmul_rn(dtfm, fy));
  double vz = __dadd_rn(v[2 * stride + i], __dmul_rn(dtfm, fz));
  // ComputeTemp::compute_scalar term of this step (src/compute_temp.cpp:84-86)
  if (KE) ke = (vx * vx + vy * vy + vz * vz) * m;
  vx = __dadd_rn(vx, __dmul_rn(dtfm, fx));
  vy = __dadd_rn(vy, __dmul_rn(dtfm, fy));
  vz = __dadd_rn(vz, __dmul_rn(dtfm, fz));
  p.x = __dadd_rn(p.x, __dmul_rn(dtv, vx));
  p.y = __dadd_rn(p.y, __dmul_rn(dtv, vy));
  p.z = __dadd_rn(p.z, __dmul_rn(dtv, vz));
  v[i] = vx;
  v[stride + i] = vy;
  v[2 * stride + i] = vz;
  x4_out[i] = p;
  if (xq_out) xq_out[i] = md_xq(p, box);
  if (xhold) {
    const double4 h = xhold[i];
    const double rsq = dsq3(__dsub_rn(p.x, h.x), __dsub_rn(p.y, h.y), __dsub_rn(p.z, h.z));
    return rsq > triggersq;
  }
  return false;
}

// The same step for atom i with its force read from f and its position
// updated in place (k_nve_fused, the replica step).
template <bool KE>
__device__ __forceinline__ bool md_nve_fused_atom(int i, int stride, double dtv, double dtf,
                                                  const double *__restrict__ mass,
                                                  double4 *__restrict__ x4, double *__restrict__ v,
                                                  const double *__restrict__ f,
                                                  int4 *__restrict__ xq, const BoxGeom &box,
                                                  const double4 *__restrict__ xhold,
                                                  double triggersq, double &ke) {
  return md_nve_step_atom<KE>(i, stride, dtv, dtf, mass, x4, x4, v, f[i], f[stride + i],
                              f[2 * stride + i], xq, box, xhold, triggersq, ke);
}

// ---- several MD steps in one launch (k_lj_multi, k_eam_multi) ---------------

// Barrier of all co-resident blocks of a cooperative launch, with the OR of
// `flag` over their threads.  `slot` is a zeroed word used once: arrivals in
// the low half, blocks with the flag in the high half, so the word that
// completes the barrier also carries the result.  wait = false: arrive only.
// After kBarrierPolls (a few seconds) it gives up and returns -1, which ends
// the block; so do the others at this barrier or the next.  The host finds
// ST_BARRIER set; sorts and list builds that are already queued return at once.
// A word with kBarrierExpired in it gives up at the first poll.
constexpr unsigned kBarrierPolls = 1u << 22;
constexpr unsigned kBarrierExpired = 0x8000u;  // above any number of blocks
__device__ __forceinline__ int md_grid_barrier(unsigned *slot, bool flag, bool wait, int *status) {
  __shared__ int s_or;
  const int any = __syncthreads_or(flag ? 1 : 0);
  if (threadIdx.x == 0) {
    const unsigned add = any ? 0x10001u : 1u;
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(slot), "r"(add) : "memory");
    int r = any;
    if (wait) {
      unsigned v = 0, polls = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(slot) : "memory");
      } while ((v & 0xffffu) < gridDim.x && ++polls < kBarrierPolls);
      r = (v >> 16) != 0u;
      if ((v & 0xffffu) != gridDim.x) {
        atomicExch(&status[ST_BARRIER], 1);
        r = -1;
      }
    }
    s_or = r;
  }
  __syncthreads();
  return s_or;
}

// What a launch of several steps needs beside StepArgs.  Host and device
// agree on `ago` (steps since the last build, at the launch).
struct MultiArgs {
  int nsteps;      // steps to run unless the distance criterion wants a rebuild before
  int ago;
  unsigned *bar;   // barrier words of this launch, zeroed
  unsigned *bar_next;  // words of the next launch, zeroed by this one
  int bar_words;
  int slots;           // list entries per thread kept in shared memory
};
// words of one launch: two barriers a step, at most a run chunk's steps
#define MD_BAR_WORDS 512

// The schedule after step j of the launch (0-based): Neighbor::decide for the
// step that follows (src/neighbor.cpp:1294-1309).
__device__ __forceinline__ bool md_candidate(int every, int delay, int ago) {
  return ago >= delay && ago % every == 0;
}

// The end of a launch of `done` steps, by one thread: the counters that
// md_decide_dev would have advanced step by step, and with the distance
// criterion the mailbox post (flag, steps since the build, count).
__device__ __forceinline__ void md_multi_end(int *status, int done, int ago, bool rebuild,
                                             int every, int delay, int check, int *dcount,
                                             volatile int *mail) {
  status[ST_AGO] = ago;
  status[ST_MOVED] = 0;
  status[ST_REBUILD] = rebuild ? 1 : 0;
  const unsigned lo = (unsigned)status[ST_STEP_LO], now = lo + (unsigned)done;
  if (now < lo) status[ST_STEP_HI] += 1;
  status[ST_STEP_LO] = (int)now;
  if (check) {
    if (rebuild && ago == (every > delay ? every : delay)) status[ST_NDANGER] += 1;
    const int k = *dcount + 1;
    *dcount = k;
    mail[0] = rebuild ? 1 : 0;
    mail[2] = ago;
    __threadfence_system();
    mail[1] = k;
  }
}

// ---- one-launch MD steps (k_lj_step, k_eam_force with STEP) ---------------
// A force kernel that also advances the atoms: after its pair loop each
// atom's first lane applies this step's final half-step and the next step's
// initial half-step.  The neighbour gathers read the positions in `cur`; the
// new positions go to `nxt`, a second buffer, so no update can reach a gather
// of the same launch; the host swaps the two buffers after the launch.  Mixed
// form: cur/nxt are the fixed-point coordinates and the FP64 positions x4
// are updated in place (the mixed gathers never read them); FP64 form:
// cur/nxt are the FP64 positions.
struct StepArgs {
  double dtv, dtf, triggersq;
  const double *mass;
  double4 *x4;      // mixed form: FP64 positions, updated in place
  const void *cur;  // positions the gathers read: int4 (mixed) or double4
  void *nxt;        // positions after the next initial half-step
  double *v;
  const double4 *xhold;
  int *status, *dcount, *mail;
  double *rows;
  int rows_cap, every, delay, check;
};

// The atom's half-steps, by its first lane, with its summed force.  The
// forces stay in registers on an ordinary step: within a run chunk nothing
// reads them (a chunk's last step is the two-kernel form, which stores them
// for the next chunk's first half-step and for downloads); an output step
// stores them all the same.
template <bool OUT, bool MIXED>
__device__ __forceinline__ bool md_step_atom(const StepArgs &s, int i, int stride, double *f,
                                             double fx, double fy, double fz,
                                             const BoxGeom &box, double &ke) {
  if (OUT) {
    f[i] = fx;
    f[stride + i] = fy;
    f[2 * stride + i] = fz;
  }
  if (MIXED)
    return md_nve_step_atom<OUT>(i, stride, s.dtv, s.dtf, s.mass, s.x4, s.x4, s.v, fx, fy, fz,
                                 static_cast<int4 *>(s.nxt), box, s.xhold, s.triggersq, ke);
  return md_nve_step_atom<OUT>(i, stride, s.dtv, s.dtf, s.mass,
                               static_cast<const double4 *>(s.cur),
                               static_cast<double4 *>(s.nxt), s.v, fx, fy, fz, nullptr, box,
                               s.xhold, s.triggersq, ke);
}

// The end of a one-launch step (every thread of the block).  The
// displacement flag goes to the status word.  On an output step the last
// block to finish adds the energy and virial (ev[0..6]: written, or added to
// what an earlier pass of the step left there) and the kinetic energy
// (ev[7]) in block order, records the thermo row and makes the next step's
// rebuild decision, as k_nve_fused does.  Other steps end with no
// block-completion count: one returning atomic per block lengthens every
// block's life (with that count on every step the 4M-atom LJ step ran at
// 5,020 Matom-steps/s, without it at 5,723), so their decision is a
// one-thread kernel launched after the step kernel.  red: 8 x (warps per
// block) doubles of shared memory.
template <bool OUT>
__device__ __forceinline__ void md_step_tail(const StepArgs &s, bool moved, const double (&acc)[7],
                                             double ke, double *red, double *partial,
                                             unsigned int *counter, double *ev,
                                             bool accumulate) {
  if (s.xhold && __any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) {
    atomicOr(&s.status[ST_MOVED], 1);
    if (OUT) __threadfence();  // the flag is visible before this block counts itself done
  }
  if (!OUT) return;
  __shared__ bool last;
  double v8[8];
#pragma unroll
  for (int k = 0; k < 7; k++) v8[k] = acc[k];
  v8[7] = ke;
  block_sum<8>(v8, red);
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < 8; k++) partial[(size_t)blockIdx.x * 8 + k] = v8[k];
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // block partials added in a fixed order: reproducible run to run
  double sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < 8; k++) sum[k] += __ldcg(&partial[(size_t)b * 8 + k]);
  __syncthreads();
  block_sum<8>(sum, red);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < 7; k++) ev[k] = accumulate ? ev[k] + sum[k] : sum[k];
    ev[7] = sum[7];
    md_record_row_dev(s.status, ev, s.rows, s.rows_cap);
    md_decide_dev(s.status, s.every, s.delay, s.check, s.dcount, s.mail);
    *counter = 0u;
  }
}

// ---- pieces of the multi-step kernels ---------------------------------------

constexpr int kMultiThreads = 256;  // threads of a block, at most
// doubles of an atom's state: x, y, z, v, dtf / mass, x, y, z at the last build
constexpr int kMultiState = 10;
inline size_t md_multi_smem(int tpa, int slots) {
  return (size_t)kMultiState * (kMultiThreads / tpa) * sizeof(double) +
         (size_t)slots * kMultiThreads * sizeof(int);
}

// a value of the atom's first lane to all its lanes
template <int TPA, class T>
__device__ __forceinline__ T from_first(T v) {
  return TPA == 1 ? v : __shfl_sync(0xffffffffu, v, 0, TPA);
}

// loads of data that other blocks wrote earlier in the launch
__device__ __forceinline__ double ld_plain(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_plain(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// Periodic shifts of an atom's neighbours in the FP64 form.  With two or more
// cells per edge a cell has at most one wrapping neighbour per dimension, so
// an entry's cell-offset code reduces to one bit per dimension (shifted or
// not), made once when the entry is fetched.
struct MultiShift {
  double v[3];
  int code[3];
  bool any;
  __device__ __forceinline__ MultiShift(int cell, const BoxGeom &box) {
    int c[3];
    md_cell_unpack(cell, c[0], c[1], c[2]);
    any = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const bool lo = c[d] == 0, hi = c[d] + 1 >= box.ncell[d];
      v[d] = lo ? -box.prd[d] : hi ? box.prd[d] : 0.0;
      code[d] = lo ? 0 : hi ? 2 : 3;  // 3: no entry
      any |= lo || hi;
    }
  }
  // bits 0..2: shifted in x, y, z; bits 6.. the neighbour
  __device__ __forceinline__ int encode(int e) const {
    return (e & ~63) | ((e & 3) == code[0] ? 1 : 0) | (((e >> 2) & 3) == code[1] ? 2 : 0) |
           (((e >> 4) & 3) == code[2] ? 4 : 0);
  }
  // x_i - (x_j + shift): x_j + 0.0 is x_j exactly
  template <bool WRAP>
  __device__ __forceinline__ void sep(unsigned e, const double4 &xi, const double4 &xj,
                                      double &dx, double &dy, double &dz) const {
    if (WRAP) {
      dx = __dsub_rn(xi.x, __dadd_rn(xj.x, (e & 1u) ? v[0] : 0.0));
      dy = __dsub_rn(xi.y, __dadd_rn(xj.y, (e & 2u) ? v[1] : 0.0));
      dz = __dsub_rn(xi.z, __dadd_rn(xj.z, (e & 4u) ? v[2] : 0.0));
    } else {
      dx = __dsub_rn(xi.x, xj.x);
      dy = __dsub_rn(xi.y, xj.y);
      dz = __dsub_rn(xi.z, xj.z);
    }
  }
};

// This lane's entries (lane, lane + TPA, ... of the atom's list), the first
// `slots` of them in shared memory; ENCODE: with MultiShift's bits.
template <int TPA, bool ENCODE>
struct MultiList {
  const MultiShift *shift;
  const int *nlist;
  int *mine;
  int stride, i, lane, slots, cnt;
  __device__ __forceinline__ MultiList(const int *nl, int stride_, int i_, int num, int lane_,
                                       int slots_, int *s_list, const MultiShift *shift_)
      : shift(shift_), nlist(nl), mine(s_list + threadIdx.x), stride(stride_), i(i_), lane(lane_), slots(slots_),
        cnt(num > lane_ ? (num - lane_ + TPA - 1) / TPA : 0) {
    for (int k = 0; k < cnt && k < slots; k++) mine[k * kMultiThreads] = fetch(k);
  }
  __device__ __forceinline__ int fetch(int k) const {
    const int e = nlist[md_slab(lane + TPA * k, i, stride)];
    return ENCODE ? shift->encode(e) : e;
  }
  __device__ __forceinline__ unsigned entry(int k) const {
    return (unsigned)(k < slots ? mine[k * kMultiThreads] : fetch(k));
  }
};

// The atom's state in shared memory (field k at p[k * AB]), used by its first
// lane.
template <int TPA>
struct MultiState {
  static constexpr int AB = kMultiThreads / TPA;
  double *p;
  __device__ __forceinline__ explicit MultiState(double *s_state)
      : p(s_state + threadIdx.x / TPA) {}
  __device__ __forceinline__ void load(const StepArgs &s, int i, int stride, const double4 &x) {
    p[0] = x.x;
    p[AB] = x.y;
    p[2 * AB] = x.z;
    p[3 * AB] = s.v[i];
    p[4 * AB] = s.v[stride + i];
    p[5 * AB] = s.v[2 * stride + i];
    p[6 * AB] = s.dtf / s.mass[(int)x.w];
    if (s.xhold) {
      const double4 h = s.xhold[i];
      p[7 * AB] = h.x;
      p[8 * AB] = h.y;
      p[9 * AB] = h.z;
    }
  }
  // final half-step of this step, initial half-step of the next (the rounded
  // operations of md_nve_step_atom); the new position, with type w
  __device__ __forceinline__ double4 step(const StepArgs &s, double fx, double fy, double fz,
                                          double w, bool &moved) {
    const double dtfm = p[6 * AB];
    double vx = __dadd_rn(p[3 * AB], __dmul_rn(dtfm, fx));
    double vy = __dadd_rn(p[4 * AB], __dmul_rn(dtfm, fy));
    double vz = __dadd_rn(p[5 * AB], __dmul_rn(dtfm, fz));
    vx = __dadd_rn(vx, __dmul_rn(dtfm, fx));
    vy = __dadd_rn(vy, __dmul_rn(dtfm, fy));
    vz = __dadd_rn(vz, __dmul_rn(dtfm, fz));
    const double4 x = make_double4(__dadd_rn(p[0], __dmul_rn(s.dtv, vx)),
                                   __dadd_rn(p[AB], __dmul_rn(s.dtv, vy)),
                                   __dadd_rn(p[2 * AB], __dmul_rn(s.dtv, vz)), w);
    p[0] = x.x;
    p[AB] = x.y;
    p[2 * AB] = x.z;
    p[3 * AB] = vx;
    p[4 * AB] = vy;
    p[5 * AB] = vz;
    moved = s.xhold && dsq3(__dsub_rn(x.x, p[7 * AB]), __dsub_rn(x.y, p[8 * AB]),
                            __dsub_rn(x.z, p[9 * AB])) > s.triggersq;
    return x;
  }
  // back to memory; the FP64 positions only in the mixed form (the FP64 form
  // wrote them to the position buffers)
  __device__ __forceinline__ void store(const StepArgs &s, int i, int stride, bool mixed,
                                        double w) const {
    if (mixed) s.x4[i] = make_double4(p[0], p[AB], p[2 * AB], w);
    s.v[i] = p[3 * AB];
    s.v[stride + i] = p[4 * AB];
    s.v[2 * stride + i] = p[5 * AB];
  }
};

// After step j of a launch (every thread of the block): advances `ago`, waits
// for the other blocks' positions and returns 1 to go on, 0 at the end of the
// launch (block 0 has posted it), -1 when the barrier gave up.
__device__ __forceinline__ int md_multi_next(const StepArgs &s, const MultiArgs &m, int j, int word,
                                             int &ago, bool moved) {
  ago++;
  const bool last = j + 1 == m.nsteps;
  const bool cand = md_candidate(s.every, s.delay, ago);
  bool rebuild = !s.check && cand;
  if (!last || (s.check && cand)) {
    // after the last step only the block that posts the decision waits
    const int r = md_grid_barrier(m.bar + word, moved, !last || blockIdx.x == 0, s.status);
    if (r < 0) return -1;
    if (s.check && cand) rebuild = r != 0;
  }
  if (!last && !rebuild) return 1;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    md_multi_end(s.status, j + 1, ago, rebuild, s.every, s.delay, s.check, s.dcount, s.mail);
  return 0;
}
