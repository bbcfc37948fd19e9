// neigh.cu -- device rebuild of the cell-sorted atom order and the full
// neighbor list, plus export of the reference's half list.
//
// Rebuild (every `every` steps, or when an atom moved more than half the
// skin) replaces Domain::pbc (src/domain.cpp:478-560), Atom::sort
// (src/atom.cpp:1575-1700), CommBrick::borders (src/comm_brick.cpp:696-864)
// and Neighbor::build -> half_bin_newton (src/neigh_half_bin.cpp:285-419):
//   1 k_wrap_bin    wrap into the box (image flags), count atoms per cell
//   2 k_scan_*      exclusive scan of the counts -> cell_start
//   3 k_scatter     counting-sort scatter of atom indices; zeroes the counts
//   4 k_sort_cells  order each cell by caller index (deterministic order)
//   5 k_gather      permute x, v, ids; fixed-point copy (mixed); xhold
//   6 k_copyback    permuted arrays back into the primary buffers, the
//                   caller-index -> slot map; ago = 0
//     (1 to 6 are one cooperative launch, k_sort_all, when every atom is
//     resident at once)
//   7 k_neigh_tiles full list over the 27 neighbor cells (cell >= rc+skin),
//                   neighbor-cell tiles staged in shared memory, distance
//                   tests on the tensor cores
// The pair test is the reference's, bit for bit: the periodic image is
// formed as x_j + s*L in FP64 and rsq = dx*dx + dy*dy + dz*dz is rounded
// after every operation, then compared with `<=` to (rc+skin)^2
// (src/neigh_half_bin.cpp:355-360, src/atom_vec_atomic.cpp:297-299).
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>

#include "md_state.h"

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ bool rebuild_on(const int *flag) { return flag == nullptr || *flag != 0; }

// Domain::pbc of one atom (position, image flags) and its cell; returns
// whether a coordinate is not finite or beyond one box image
__device__ __forceinline__ bool wrap_atom(double4 &p, int &img, int (&cc)[3], const BoxGeom &box) {
  double xs[3] = {p.x, p.y, p.z};
  int im[3] = {(img & MD_IMGMASK) - MD_IMGMAX, ((img >> 10) & MD_IMGMASK) - MD_IMGMAX,
               ((img >> 20) & MD_IMGMASK) - MD_IMGMAX};
  bool bad = false;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double x = xs[d];
    if (!isfinite(x)) {
      bad = true;
      x = box.lo[d];
    }
    // Domain::pbc: x < lo -> x += prd; x >= hi -> x -= prd, x = max(x, lo)
    if (x < box.lo[d]) {
      x = __dadd_rn(x, box.prd[d]);
      im[d]--;
    }
    if (x >= box.hi[d]) {
      x = __dsub_rn(x, box.prd[d]);
      x = fmax(x, box.lo[d]);
      im[d]++;
    }
    if (x < box.lo[d] || x >= box.hi[d]) bad = true;
    xs[d] = x;
    const int c = (int)((x - box.lo[d]) * box.cinv[d]);
    cc[d] = c < 0 ? 0 : (c >= box.ncell[d] ? box.ncell[d] - 1 : c);
  }
  p = make_double4(xs[0], xs[1], xs[2], p.w);
  img = md_img_pack(im[0], im[1], im[2]);
  return bad;
}

template <bool BATCH>
__global__ void k_wrap_bin(int n, BoxGeom box1, Reps reps, double4 *__restrict__ x4,
                           int *__restrict__ image, int *__restrict__ cell_count,
                           int *__restrict__ slot, int *__restrict__ cell_tmp,
                           int *__restrict__ status, const int *flag) {
  if (!rebuild_on(flag)) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int rep = BATCH ? reps.rep_of_atom[i] : 0;
  const BoxGeom &box = BATCH ? reps.box[rep] : box1;
  double4 p = x4[i];
  int img = image[i], cc[3];
  if (wrap_atom(p, img, cc, box)) atomicExch(&status[ST_LOST], 1);
  x4[i] = p;
  image[i] = img;
  int c = cc[0] + box.ncell[0] * (cc[1] + box.ncell[1] * cc[2]);
  if (BATCH) c += reps.cell_base[rep];
  slot[i] = atomicAdd(&cell_count[c], 1);
  cell_tmp[i] = c;
}

// block-wide exclusive scan of kScanTile ints; block sums to `sums`
__global__ void k_scan_tiles(int m, const int *__restrict__ in, int *__restrict__ out,
                             int *__restrict__ sums, const int *flag) {
  if (!rebuild_on(flag)) return;
  __shared__ int warp_tot[kScanThreads / 32];
  int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int run = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    int idx = base + k;
    int a = idx < m ? in[idx] : 0;
    v[k] = run;
    run += a;
  }
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int t = warp_tot[lane];
    int s = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    warp_tot[lane] = s - t;  // exclusive prefix of warp totals
    if (lane == 31 && sums) sums[blockIdx.x] = s;
  }
  __syncthreads();
  int excl = incl - run + warp_tot[warp];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    int idx = base + k;
    if (idx < m) out[idx] = v[k] + excl;
  }
}

__global__ void k_scan_add(int m, int *__restrict__ out, const int *__restrict__ sums,
                           const int *flag) {
  if (!rebuild_on(flag)) return;
  int b = blockIdx.x;
  if (b == 0) return;
  int add = sums[b];
  int base = b * kScanTile;
  for (int k = threadIdx.x; k < kScanTile; k += blockDim.x) {
    int idx = base + k;
    if (idx < m) out[idx] += add;
  }
}

// Scatter each atom to its slot in the cell-sorted order.  The scan has
// consumed the m cell counts by now, so this kernel also zeroes them for the
// next build (the counts start at zero when they are allocated).
__global__ void k_scatter(int n, const int *__restrict__ cell_tmp, const int *__restrict__ slot,
                          const int *__restrict__ cell_start, int *__restrict__ perm, int m,
                          int *__restrict__ cell_count, const int *flag) {
  if (!rebuild_on(flag)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = i; k < m; k += gridDim.x * blockDim.x) cell_count[k] = 0;
  if (i >= n) return;
  perm[cell_start[cell_tmp[i]] + slot[i]] = i;
}

// One warp per cell: rank the cell's atoms by caller index so that the
// sorted order (and with it every summation order) is reproducible.
constexpr int kSortWarps = 8;
constexpr int kSortSmall = 64;

__global__ void k_sort_cells(int ncells, const int *__restrict__ cell_start, int *__restrict__ perm,
                             int *__restrict__ tmp, const int *__restrict__ orig, const int *flag) {
  if (!rebuild_on(flag)) return;
  __shared__ int skey[kSortWarps][kSortSmall];
  __shared__ int sval[kSortWarps][kSortSmall];
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int c = blockIdx.x * kSortWarps + w;
  if (c >= ncells) return;
  int s = cell_start[c], e = cell_start[c + 1], cnt = e - s;
  if (cnt <= 1) return;
  if (cnt <= kSortSmall) {
    for (int k = lane; k < cnt; k += 32) {
      int val = perm[s + k];
      sval[w][k] = val;
      skey[w][k] = orig[val];
    }
    __syncwarp();
    for (int k = lane; k < cnt; k += 32) {
      int key = skey[w][k], r = 0;
      for (int m = 0; m < cnt; m++) r += skey[w][m] < key;
      perm[s + r] = sval[w][k];
    }
  } else {
    for (int k = lane; k < cnt; k += 32) tmp[s + k] = perm[s + k];
    __threadfence_block();
    __syncwarp();
    for (int k = lane; k < cnt; k += 32) {
      int val = tmp[s + k], key = orig[val], r = 0;
      for (int m = 0; m < cnt; m++) r += orig[tmp[s + m]] < key;
      perm[s + r] = val;
    }
  }
}

template <bool BATCH>
__global__ void k_gather(int n, int stride, BoxGeom box1, Reps reps, const int *__restrict__ perm,
                         const double4 *__restrict__ x4, double4 *__restrict__ x4b,
                         const double *__restrict__ v, double *__restrict__ vb,
                         const int *__restrict__ orig, int *__restrict__ origb,
                         const int *__restrict__ image, int *__restrict__ imageb,
                         const int *__restrict__ cell_tmp, int *__restrict__ cell,
                         int4 *__restrict__ xq, double4 *__restrict__ xhold, const int *flag) {
  if (!rebuild_on(flag)) return;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int old = perm[k];
  double4 p = x4[old];
  x4b[k] = p;
  vb[k] = v[old];
  vb[stride + k] = v[stride + old];
  vb[2 * stride + k] = v[2 * stride + old];
  origb[k] = orig[old];
  imageb[k] = image[old];
  int c = cell_tmp[old];
  const int rep = BATCH ? reps.rep_of_atom[k] : 0;
  const BoxGeom &box = BATCH ? reps.box[rep] : box1;
  if (BATCH) c -= reps.cell_base[rep];
  int cx = c % box.ncell[0];
  int cy = (c / box.ncell[0]) % box.ncell[1];
  int cz = c / (box.ncell[0] * box.ncell[1]);
  cell[k] = md_cell_pack(cx, cy, cz);
  if (xhold) xhold[k] = p;
  if (xq) xq[k] = md_xq(p, box);
}

__global__ void k_copyback(int n, int stride, const double4 *__restrict__ x4b,
                           double4 *__restrict__ x4, const double *__restrict__ vb,
                           double *__restrict__ v, const int *__restrict__ origb,
                           int *__restrict__ orig, const int *__restrict__ imageb,
                           int *__restrict__ image, int *__restrict__ where,
                           int *__restrict__ status, const int *flag) {
  if (!rebuild_on(flag)) return;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) {
    // Neighbor::build bookkeeping: ago = 0, ncalls++ (src/neighbor.cpp:1384-1386)
    status[ST_AGO] = 0;
    status[ST_NCALLS] += 1;
  }
  if (k >= n) return;
  x4[k] = x4b[k];
  v[k] = vb[k];
  v[stride + k] = vb[stride + k];
  v[2 * stride + k] = vb[2 * stride + k];
  const int o = origb[k];
  orig[k] = o;
  where[o] = k;  // caller index -> sorted slot, for the halo pack / unpack
  image[k] = imageb[k];
}

// The whole sort of a box whose atoms are all resident at once, in one
// cooperative launch instead of six or more: a thread holds one atom's data in
// registers from the wrap to its place in the new order, so nothing is copied
// through the second buffers.  Same order as the kernels above.  At these
// sizes the six kernels are 3 to 6 us each of launch and latency: runs with
// six builds went from 1,481 to 1,420 us (32,000 atoms, mixed) and from 927 to
// 902 (864), one frame of 109,059 atoms from 361 to 345.
//   1 wrap, cell, slot in the cell (atomic)            | grid barrier
//   2 block 0: exclusive scan of the cell counts       | grid barrier
//   3 caller index into the cell's slot; counts to 0   | grid barrier
//   4 rank by caller index in the cell; the atom's data to its new place
constexpr int kSortThreads = 256;
constexpr int kSortCells = 16384;  // most cells that one block scans

struct SortArgs {
  int n, stride, m;  // m: cells + 1
  BoxGeom box;
  Reps reps;
  double4 *x4;
  double *v;
  int *orig, *image, *cell, *where;
  int *cell_count, *cell_start, *key;
  int4 *xq;
  double4 *xhold;
  int *status;
  const int *flag;
  // three barrier words; 0 and 1 are zero between launches, 2 is zeroed after
  // the first barrier.  The two sets of the multi-step launches lie before them.
  unsigned *bar;
};

template <bool BATCH>
__global__ void __launch_bounds__(kSortThreads, 4) k_sort_all(SortArgs A) {
  if (!rebuild_on(A.flag)) return;
  const int i = blockIdx.x * kSortThreads + threadIdx.x;
  const bool act = i < A.n;
  const int gave_up = A.status[ST_BARRIER];  // an earlier launch's barrier
  double4 p = make_double4(0, 0, 0, 1);
  double v0 = 0, v1 = 0, v2 = 0;
  int o = 0, img = 0, c = 0, slot = 0, cc[3] = {0, 0, 0};
  const int rep = BATCH && act ? A.reps.rep_of_atom[i] : 0;
  const BoxGeom &box = BATCH ? A.reps.box[rep] : A.box;
  if (act) {
    p = A.x4[i];
    v0 = A.v[i];
    v1 = A.v[A.stride + i];
    v2 = A.v[2 * A.stride + i];
    o = A.orig[i];
    img = A.image[i];
    if (wrap_atom(p, img, cc, box)) atomicExch(&A.status[ST_LOST], 1);
    c = cc[0] + box.ncell[0] * (cc[1] + box.ncell[1] * cc[2]);
    if (BATCH) c += A.reps.cell_base[rep];
  }
  // Looked at before the first change of the cell counts: a launch that gives
  // up leaves them as they are, and counting on top of them would place atoms
  // past the arrays.
  if (gave_up) {
    // the launches of several steps that are queued behind this rebuild give up
    // at once instead of waiting again
    if (i < 2) A.bar[(i - 2) * MD_BAR_WORDS] = kBarrierExpired;
    return;
  }
  if (act) slot = atomicAdd(&A.cell_count[c], 1);
  if (md_grid_barrier(A.bar, false, true, A.status) < 0) return;
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) A.bar[2] = 0u;
    // each thread scans a run of cells, the block the runs' totals
    __shared__ int warp_tot[kSortThreads / 32];
    const int per = (A.m + kSortThreads - 1) / kSortThreads;
    const int b0 = threadIdx.x * per, b1 = min(A.m, b0 + per);
    int sum = 0;
    for (int k = b0; k < b1; k++) sum += __ldcg(&A.cell_count[k]);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int w = 0; w < warp; w++) run += warp_tot[w];
    for (int k = b0; k < b1; k++) {
      A.cell_start[k] = run;
      run += __ldcg(&A.cell_count[k]);
    }
  }
  if (md_grid_barrier(A.bar + 1, false, true, A.status) < 0) return;
  int s0 = 0, s1 = 0;
  if (act) {
    s0 = __ldcg(&A.cell_start[c]);
    s1 = __ldcg(&A.cell_start[c + 1]);
    A.key[s0 + slot] = o;
  }
  for (int k = i; k < A.m; k += gridDim.x * kSortThreads) A.cell_count[k] = 0;
  if (md_grid_barrier(A.bar + 2, false, true, A.status) < 0) return;
  if (i == 0) {
    A.bar[0] = A.bar[1] = 0u;
    // Neighbor::build bookkeeping: ago = 0, ncalls++ (src/neighbor.cpp:1384-1386)
    A.status[ST_AGO] = 0;
    A.status[ST_NCALLS] += 1;
  }
  if (!act) return;
  int k = s0;
  for (int q = s0; q < s1; q++) k += __ldcg(&A.key[q]) < o;
  A.x4[k] = p;
  A.v[k] = v0;
  A.v[A.stride + k] = v1;
  A.v[2 * A.stride + k] = v2;
  A.orig[k] = o;
  A.where[o] = k;
  A.image[k] = img;
  A.cell[k] = md_cell_pack(cc[0], cc[1], cc[2]);
  if (A.xhold) A.xhold[k] = p;
  if (A.xq) A.xq[k] = md_xq(p, box);
}

// Full neighbor list from staged neighbor-cell tiles.
// A CTA owns TC consecutive cells along x (their atoms are contiguous in the
// cell-sorted order) and stages the 3 x 3 x (TC+2) block of cells around
// them in shared memory, periodic images applied.  Three phases:
//   test    r^2 - cut^2 of every (candidate, owned atom) pair.  It is a
//           contraction, |a|^2 + (|b|^2 - cut^2) - 2 a.b, so the tensor cores
//           do it: coordinates relative to the tile centre are split into
//           FP16 hi + lo halves, whose products are exact in the FP32
//           accumulator, and one mma.m16n8k16 evaluates 128 pairs (all four
//           half products of three dimensions, the candidate's norm, and the
//           owned atom's norm less the cutoff fill K = 16).  The sign bit is the decision; a
//           funnel shift collects it, one instruction per value.  Pairs
//           within `eps` of the cutoff are decided by the reference's FP64
//           arithmetic on the FP64 positions, so the list is bit-identical
//           to the FP64 criterion.
//   order   eight atoms x four 32-candidate chunks a warp: the acceptance
//           bits are brought into candidate order (two 2-bit index fields
//           swap) and empty words dropped.
//   append  one thread per owned atom walks its words; with no empty words
//           the threads of a warp are at the same entry, so the slabs they
//           store are contiguous.
// Bound by instruction issue: one FP32 distance test per pair and lane, with a
// ballot per owned atom, took 788 warp instructions per atom (0.82 us per
// 1,000 atoms at 4,000,000); this form takes about 330 (0.5 us).  With the
// wider grid of small tiles a 32,000-atom build went from 69 us to 25 us and
// an 864-atom one from 89 us to 20 us.
// (mma.sync rather than tcgen05: the operands are a few cells, 56 x 19
// values, and the result is wanted as bits per lane, not as a tile in TMEM.)
//
// Error bound behind eps.  Let rb bound the owned atoms' distance from the
// tile centre and ra = rb + cutoff that of a candidate near an owned atom's
// cutoff.  Relative to 2^-20: a coordinate's FP32 rounding (2^-24, both sides
// of the separation) moves r^2 by at most 0.25 ra^2, the FP16 hi + lo split
// (2^-22, in the product only) by ra^2, the FP32 norms and their splits by
// 1.2 ra^2, and 16 accumulations, each truncated at 2^-23 of a sum below
// (ra + rb)^2, by 2 (ra + rb)^2.  eps = 1.25 x 2^-19 ((ra + rb)^2 + 2 ra^2) is
// above 1.25 x their sum.  How the tensor core rounds its additions is not
// documented, so the last term is an assumption: on 3.5 million pairs within
// 2 % of cutoffs in [2, 4), tiles of one and two cells, owned atoms at the
// corners among them, the largest error was 0.04 eps, and the tests put
// thousands of pairs within 1e-9 to 1e-4 of the cutoff.  (A pair further apart
// has a larger error, but its value grows 2 x cutoff per unit length, far
// faster than the bound.)
constexpr int kNeighThreads = 128;
constexpr int kMaxCols = 384;  // owned atoms of a tile, padded to eight per cell, at most
// 32-candidate chunks of one cell's nine rows, at most
constexpr int max_chunks(int tc) { return 192 / tc; }
// most dynamic shared memory a tile may take (opt-in), in 16-byte units: what
// the kernel's tables (2.8 KB) leave of an SM's 227 KB
constexpr int kStageUnitsMax = 222 * 1024 / 16;

struct NeighArgs {
  int n, stride, capacity, units, ntp1, pass, units1;
  BoxGeom box;
  Reps reps;
  double scale;   // power of two that brings the largest list cutoff into [2, 4)
  float cmax;     // largest list cutoff, scaled, squared
  float dmax;     // largest difference of a type pair's from it, scaled, squared
  const double *cutneighsq;
  const double4 *x4;
  const int *cell_start;
  int *nlist, *numneigh, *status;
  const int *flag;
};

// exact reference criterion for one candidate (FP64, no contraction)
__device__ __forceinline__ bool exact_pair(const double4 &xi, const double4 &xj, double shx,
                                           double shy, double shz, double cutsq) {
  const double delx = __dsub_rn(xi.x, __dadd_rn(xj.x, shx));
  const double dely = __dsub_rn(xi.y, __dadd_rn(xj.y, shy));
  const double delz = __dsub_rn(xi.z, __dadd_rn(xj.z, shz));
  return dsq3(delx, dely, delz) <= cutsq;
}

// staged word: (atom index << 6) + the staged cell's row code (dy+1)<<2 |
// (dz+1)<<4 + its column sx (0 .. TC+1); less the owned cell's column (0 ..
// TC-1) it is the list entry
__device__ __forceinline__ int row_code(int row) { return ((row % 3) << 2) + ((row / 3) << 4); }

// FP16 hi + lo of three coordinates and of their squared norm plus `add`,
// one word each (hi in the low half)
__device__ __forceinline__ uint4 record(float x, float y, float z, float add) {
  const float n = fmaf(x, x, fmaf(y, y, fmaf(z, z, add)));
  const __half2 hxy = __floats2half2_rn(x, y), hzn = __floats2half2_rn(z, n);
  const __half2 lxy = __floats2half2_rn(x - __low2float(hxy), y - __high2float(hxy));
  const __half2 lzn = __floats2half2_rn(z - __low2float(hzn), n - __high2float(hzn));
  const unsigned h0 = *reinterpret_cast<const unsigned *>(&hxy),
                 h1 = *reinterpret_cast<const unsigned *>(&hzn),
                 l0 = *reinterpret_cast<const unsigned *>(&lxy),
                 l1 = *reinterpret_cast<const unsigned *>(&lzn);
  return make_uint4(__byte_perm(h0, l0, 0x5410), __byte_perm(h0, l0, 0x7632),
                    __byte_perm(h1, l1, 0x5410), __byte_perm(h1, l1, 0x7632));
}
__device__ __forceinline__ float join16(unsigned w) {
  return __half2float(__ushort_as_half((unsigned short)w)) +
         __half2float(__ushort_as_half((unsigned short)(w >> 16)));
}

__device__ __forceinline__ void mma16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2,
                                      unsigned a3, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma8(float (&d)[4], unsigned a0, unsigned a1, unsigned b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// least magnitude of a lane's eight values and `m`
__device__ __forceinline__ float least(float m, const float (&d)[4], const float (&e)[4]) {
  asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(d[0]), "f"(d[1]));
  asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(d[2]), "f"(d[3]));
  asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(e[0]), "f"(e[1]));
  asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(e[2]), "f"(e[3]));
  return m;
}

// acceptance byte of one lane: the sign bits of its eight values, the even
// owned atom's four (candidates g, g+8, g+16, g+24) in the low nibble
__device__ __forceinline__ unsigned sign_byte(const float (&d)[4], const float (&e)[4]) {
  unsigned r = 0;
  r = __funnelshift_l(__float_as_uint(e[3]), r, 1);
  r = __funnelshift_l(__float_as_uint(e[1]), r, 1);
  r = __funnelshift_l(__float_as_uint(d[3]), r, 1);
  r = __funnelshift_l(__float_as_uint(d[1]), r, 1);
  r = __funnelshift_l(__float_as_uint(e[2]), r, 1);
  r = __funnelshift_l(__float_as_uint(e[0]), r, 1);
  r = __funnelshift_l(__float_as_uint(d[2]), r, 1);
  return __funnelshift_l(__float_as_uint(d[0]), r, 1);
}

// bit 8 (g & 3) + 4 (g >> 2) + m of a lane-order word is candidate g + 8 m:
// exchange the index fields (bits 4,3) and (bits 1,0)
__device__ __forceinline__ unsigned candidate_order(unsigned x) {
  unsigned t = ((x >> 14) ^ x) & 0x0000CCCCu;
  x = x ^ t ^ (t << 14);
  t = ((x >> 7) ^ x) & 0x00AA00AAu;
  return x ^ t ^ (t << 7);
}

// 16-byte units of shared memory of a tile: staged records (16 B), words
// (4 B) and, with several types, types (1 B) with 32 spare slots, and the
// acceptance words (4 B) with their first slots (2 B)
__host__ __device__ inline int tile_units(int nstage, int chunks, int cols, bool single) {
  const long long m = (long long)nstage + 32, c = (long long)chunks * cols;
  const long long u =
      m + (m + 3) / 4 + (single ? 0 : (m + 15) / 16) + (c + 3) / 4 + (c + 7) / 8;
  return u < (1 << 30) ? (int)u : 1 << 30;  // (a collapsed cell: 1e5 atoms)
}
// the units of a tile of tc cells at a mean of `per_cell` atoms per cell
inline int tile_units_of(double per_cell, int tc, bool single) {
  const int stage = (int)(1.15 * 9 * (tc + 2) * per_cell) + 32;
  const int chunks = 9 * ((int)(3.0 * per_cell / 32.0) + 1) + 3;
  const int cols = tc * (((int)(per_cell + 2.0) + 7) & ~7) + 8;
  return tile_units(stage, chunks, cols, single);
}

template <int TC, bool SINGLE, bool BATCH>
__global__ void __launch_bounds__(kNeighThreads, 8) k_neigh_tiles(NeighArgs A) {
  if (!rebuild_on(A.flag)) return;
  const int gave_up = A.status[ST_BARRIER];  // the sort's barrier
  constexpr int NSX = TC + 2, NST = 9 * NSX;
  constexpr int WPC = kNeighThreads / 32 / TC;  // warps per owned cell
  // batched: this tile's replica, its box and its cells' slice of cell_start
  const int rep = BATCH ? A.reps.tile_rep[blockIdx.x] : 0;
  const int tile = BATCH ? blockIdx.x - A.reps.tile_base[rep] : blockIdx.x;
  const BoxGeom &box = BATCH ? A.reps.box[rep] : A.box;
  const int *__restrict__ cell_start = BATCH ? A.cell_start + A.reps.cell_base[rep] : A.cell_start;
  const double4 *__restrict__ x4 = A.x4;
  extern __shared__ uint4 s_rec[];
  __shared__ int s_start[NST + 1];
  __shared__ int s_src[NST];               // first atom of the staged cell
  __shared__ signed char s_img[NST][4];    // periodic image of the staged cell
  __shared__ int s_chunk[TC][max_chunks(TC)];  // first slot | row << 16 | candidates << 20
  __shared__ int s_nchunk[TC];
  __shared__ unsigned short s_count[kMaxCols];  // neighbors of each owned atom
  __shared__ double cns[SINGLE ? 1 : (MD_MAXTYPES + 1) * (MD_MAXTYPES + 1)];
  __shared__ __align__(4) __half s_delta[SINGLE ? 1 : MD_MAXTYPES * MD_MAXTYPES];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncx = box.ncell[0], ncy = box.ncell[1], ncz = box.ncell[2];
  const int tiles_x = (ncx + TC - 1) / TC;
  const int bx = tile % tiles_x;
  const int cy = (tile / tiles_x) % ncy;
  const int cz = tile / (tiles_x * ncy);
  const int cx0 = bx * TC;
  const int ow = min(TC, ncx - cx0);  // owned cells in this tile
  if (!SINGLE) {
    const int nt = A.ntp1 - 1;
    for (int k = tid; k < A.ntp1 * A.ntp1; k += kNeighThreads) cns[k] = A.cutneighsq[k];
    for (int k = tid; k < MD_MAXTYPES * MD_MAXTYPES; k += kNeighThreads) {
      const int a = k / MD_MAXTYPES, b = k % MD_MAXTYPES;
      float d = 0.f;
      if (a < nt && b < nt)
        d = A.cmax - (float)(A.cutneighsq[(a + 1) * A.ntp1 + b + 1] * A.scale * A.scale);
      s_delta[k] = __float2half_rn(d);
    }
  }
  // staged cells: id = sx + NSX*(sy + 3*sz) is global cell
  // (cx0-1+sx, cy-1+sy, cz-1+sz), wrapped
  if (tid < NST) {
    const int id = tid;
    const int sx = id % NSX, sy = (id / NSX) % 3, sz = id / (3 * NSX);
    int s0 = 0, ix = 0, iy = 0, iz = 0, cnt = 0;
    if (sx <= ow + 1) {  // columns past the box edge are not neighbours of any owned cell
      int gx = cx0 - 1 + sx, gy = cy - 1 + sy, gz = cz - 1 + sz;
      if (gx < 0) { gx += ncx; ix = -1; } else if (gx >= ncx) { gx -= ncx; ix = 1; }
      if (gy < 0) { gy += ncy; iy = -1; } else if (gy >= ncy) { gy -= ncy; iy = 1; }
      if (gz < 0) { gz += ncz; iz = -1; } else if (gz >= ncz) { gz -= ncz; iz = 1; }
      const int g = gx + ncx * (gy + ncy * gz);
      s0 = cell_start[g];
      cnt = cell_start[g + 1] - s0;
    }
    s_src[id] = s0;
    s_img[id][0] = (signed char)ix;
    s_img[id][1] = (signed char)iy;
    s_img[id][2] = (signed char)iz;
    s_start[id + 1] = cnt;
  }
  if (gave_up) return;  // cell_start may never have been written
  __syncthreads();
  if (warp == 0) {  // prefix sum of the counts, two per lane
    const int i0 = 2 * lane, i1 = 2 * lane + 1;
    const int c0 = i0 < NST ? s_start[i0 + 1] : 0, c1 = i1 < NST ? s_start[i1 + 1] : 0;
    int incl = c0 + c1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (i0 < NST) s_start[i0 + 1] = incl - c1;
    if (i1 < NST) s_start[i1 + 1] = incl;
    if (lane == 0) s_start[0] = 0;
  }
  __syncthreads();
  // chunk table: the nine candidate rows (three cells along x) of each owned
  // cell in chunks of 32
  if (tid < 9 * TC) {
    const int c = tid / 9, r = tid % 9;
    int off = 0;
    if (c < ow) {
      for (int q = 0; q < r; q++)
        off += (s_start[c + 3 + NSX * q] - s_start[c + NSX * q] + 31) >> 5;
      const int r0 = s_start[c + NSX * r], r1 = s_start[c + 3 + NSX * r];
      for (int b = r0; b < r1; b += 32, off++)
        if (off < max_chunks(TC))
          s_chunk[c][off] = (b & 0xffff) | (r << 16) | (min(32, r1 - b) << 20);
    }
    if (r == 8) s_nchunk[c] = off;
  }
  __syncthreads();
  const int nstage = s_start[NST];
  // owned atoms: contiguous; acceptance columns padded to eight per cell
  const int own0 = 1 + NSX * 4;  // staged id of the first owned cell
  int maxw = 0, cols = 0;
#pragma unroll
  for (int c = 0; c < TC; c++) {
    maxw = max(maxw, s_nchunk[c]);
    if (c < ow) cols += (s_start[own0 + c + 1] - s_start[own0 + c] + 7) & ~7;
  }
  const int need = tile_units(nstage, maxw, cols, SINGLE);
  // pass 0: every tile (staged, or the global-memory path when it does not
  // fit); pass 1: the tiles that fit `units`; pass 2: only the tiles that
  // pass 1 left (more than units1), with more shared memory
  if ((A.pass == 1 && need > A.units) || (A.pass == 2 && need <= A.units1)) return;
  // rb: extent of the owned atoms from the tile centre; a candidate near the
  // cutoff of one lies within ra
  const float fscale = (float)A.scale;
  const float ux = 0.5f * (float)ow * (float)box.cs[0] * fscale;
  const float uy = 0.5f * (float)box.cs[1] * fscale, uz = 0.5f * (float)box.cs[2] * fscale;
  const float rb = sqrtf(ux * ux + uy * uy + uz * uz), ra = rb + sqrtf(A.cmax);
  const float eps = ((ra + rb) * (ra + rb) + 2.0f * ra * ra) * (1.25f / 524288.0f) +
                    (SINGLE ? 0.f : A.dmax * (1.0f / 2048.0f));
  // cells far wider than the cutoff would overflow FP16 or put every pair
  // inside the band
  const bool stageable = need <= kStageUnitsMax && maxw <= max_chunks(TC) && nstage < 65504 &&
                         cols <= kMaxCols && ra < 32.f;
  const bool staged = stageable && need <= A.units;
  // for the next build's capacity, and for the tiles' width
  if (tid == 0) {
    if (stageable) atomicMax(&A.status[ST_MAXSTAGE], need);
    else atomicAdd(&A.status[ST_UNSTAGED], s_start[own0 + ow] - s_start[own0]);
  }
  const int a0 = s_src[own0];
  const int nown = s_start[own0 + ow] - s_start[own0];

  if (staged) {
    unsigned *recw = reinterpret_cast<unsigned *>(s_rec);
    int *word = reinterpret_cast<int *>(s_rec + nstage + 32);
    unsigned char *type = reinterpret_cast<unsigned char *>(s_rec + nstage + 32 +
                                                            (nstage + 32 + 3) / 4);
    unsigned char *mask = SINGLE ? type : type + ((nstage + 32 + 15) & ~15);
    // first slots of the words that the order phase keeps
    unsigned short *slot = reinterpret_cast<unsigned short *>(mask + ((maxw * cols + 3) & ~3) * 4);
    const double rx = box.lo[0] + (cx0 + 0.5 * ow) * box.cs[0];
    const double ry = box.lo[1] + (cy + 0.5) * box.cs[1];
    const double rz = box.lo[2] + (cz + 0.5) * box.cs[2];
    // stage: a group of eight lanes per cell
    for (int id = tid >> 3; id < NST; id += kNeighThreads / 8) {
      const int o0 = s_start[id], cnt = s_start[id + 1] - o0, g0 = s_src[id];
      const int code = row_code(id / NSX) + id % NSX;
      const double shx = (s_img[id][0] * box.prd[0] - rx) * A.scale,
                   shy = (s_img[id][1] * box.prd[1] - ry) * A.scale,
                   shz = (s_img[id][2] * box.prd[2] - rz) * A.scale;
      for (int t = tid & 7; t < cnt; t += 8) {
        const double4 p = x4[g0 + t];
        const float x = (float)fma(p.x, A.scale, shx), y = (float)fma(p.y, A.scale, shy),
                    z = (float)fma(p.z, A.scale, shz);
        s_rec[o0 + t] = record(x, y, z, 0.f);
        word[o0 + t] = (int)((unsigned)(g0 + t) << 6) + code;
        if (!SINGLE) type[o0 + t] = (unsigned char)((int)p.w - 1);
      }
    }
    // the spare slots after the last staged row: far away, type 1
    if (tid < 32) {
      s_rec[nstage + tid] = record(64.f, 64.f, 64.f, 0.f);
      word[nstage + tid] = 0;
      if (!SINGLE) type[nstage + tid] = 0;
    }
    __syncthreads();
    // test: warps WPC*c .. WPC*c + WPC-1 take owned cell c, chunk by chunk
    const int c = warp / WPC, sub = warp % WPC;
    const int g = lane >> 2, t = lane & 3;
    if (c < ow) {
      const int o0 = s_start[own0 + c], cnt = s_start[own0 + c + 1] - o0;
      const int nch = s_nchunk[c];
      int colb = 0;
#pragma unroll
      for (int q = 0; q < TC; q++)
        if (q < c) colb += (s_start[own0 + q + 1] - s_start[own0 + q] + 7) & ~7;
      for (int ab = 0; ab < cnt; ab += 32) {
        const int na = min(32, cnt - ab), nt = (na + 7) >> 3;
        // owned atoms as the B operand: -2 b in both halves of each dimension
        unsigned b0[4], b1[4], bt[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int ia = o0 + ab + min(8 * q + g, na - 1);
          const unsigned w = recw[ia * 4 + t];
          const __half2 m2 = __floats2half2_rn(-2.f, -2.f);
          const __half2 h2 = __half2half2(__ushort_as_half((unsigned short)w));
          const __half2 l2 = __half2half2(__ushort_as_half((unsigned short)(w >> 16)));
          const __half2 ph = __hmul2(h2, m2), pl = __hmul2(l2, m2);
          b0[q] = *reinterpret_cast<const unsigned *>(&ph);
          b1[q] = *reinterpret_cast<const unsigned *>(&pl);
          if (t == 3) {  // candidate norm x 1; 1 x (norm - cutoff)
            const float v = join16(w) - A.cmax;
            const __half vh = __float2half_rn(v);
            const __half2 v2 = __halves2half2(vh, __float2half_rn(v - __half2float(vh)));
            b0[q] = 0x3C003C00u;
            b1[q] = *reinterpret_cast<const unsigned *>(&v2);
          }
          bt[q] = 0;
          if (!SINGLE)
            bt[q] = *reinterpret_cast<const unsigned *>(
                &s_delta[type[ia] * MD_MAXTYPES + 2 * t]);
        }
        for (int w = sub; w < nch; w += WPC) {
          const int info = s_chunk[c][w];
          const int cb = info & 0xffff;
          const unsigned *ap = recw + (cb + g) * 4 + t;
          const unsigned a00 = ap[0], a01 = ap[32], a10 = ap[64], a11 = ap[96];
          // the second half of K: the same coordinates against the lo halves;
          // ones against the owned side's norm
          const unsigned one = 0x3C003C00u;
          const unsigned a02 = t == 3 ? one : a00, a03 = t == 3 ? one : a01,
                         a12 = t == 3 ? one : a10, a13 = t == 3 ? one : a11;
          unsigned y00 = 0, y01 = 0, y10 = 0, y11 = 0;  // one-hot types
          if (!SINGLE) {
            auto hot = [&](int s) {
              const int ty = type[s];
              return (ty >> 1) == t ? ((ty & 1) ? 0x3C000000u : 0x00003C00u) : 0u;
            };
            y00 = hot(cb + g), y01 = hot(cb + g + 8), y10 = hot(cb + g + 16),
            y11 = hot(cb + g + 24);
          }
          unsigned char *mw = mask + (w * cols + colb + ab) * 4 + t * 8 + g;
          float near = 1.0e30f;
          float d[4], e[4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (q < nt) {
              mma16(d, a00, a01, a02, a03, b0[q], b1[q]);
              mma16(e, a10, a11, a12, a13, b0[q], b1[q]);
              if (!SINGLE) {
                mma8(d, y00, y01, bt[q]);
                mma8(e, y10, y11, bt[q]);
              }
              near = least(near, d, e);
              mw[q * 32] = (unsigned char)sign_byte(d, e);
            }
          }
          if (__any_sync(0xffffffffu, near <= eps)) {
            // some pair lies in the band: the reference's FP64 test for those
            const int row = (info >> 16) & 15, nc = info >> 20;
#pragma unroll 1
            for (int q = 0; q < nt; q++) {
              // (b0[q] etc. by selects: the loop is rolled)
              const unsigned p0 = q == 0 ? b0[0] : q == 1 ? b0[1] : q == 2 ? b0[2] : b0[3];
              const unsigned p1 = q == 0 ? b1[0] : q == 1 ? b1[1] : q == 2 ? b1[2] : b1[3];
              mma16(d, a00, a01, a02, a03, p0, p1);
              mma16(e, a10, a11, a12, a13, p0, p1);
              if (!SINGLE) {
                const unsigned pt = q == 0 ? bt[0] : q == 1 ? bt[1] : q == 2 ? bt[2] : bt[3];
                mma8(d, y00, y01, pt);
                mma8(e, y10, y11, pt);
              }
              unsigned r = sign_byte(d, e), band = 0;
              const float val[8] = {d[0], d[2], e[0], e[2], d[1], d[3], e[1], e[3]};
#pragma unroll
              for (int k = 0; k < 8; k++) band |= fabsf(val[k]) <= eps ? 1u << k : 0u;
              while (band) {
                const int k = __ffs(band) - 1;
                band &= band - 1u;
                const int ci = g + 8 * (k & 3), ai = 8 * q + 2 * t + (k >> 2);
                if (ci >= nc || ai >= na) continue;
                const int cw = word[cb + ci];
                const int id = (cw & 63) - row_code(row) + NSX * row;
                const int i = a0 + (o0 - s_start[own0]) + ab + ai;
                const double cut =
                    SINGLE ? A.cutneighsq[A.ntp1 + 1]
                           : cns[(type[o0 + ab + ai] + 1) * A.ntp1 + type[cb + ci] + 1];
                const bool in = exact_pair(x4[i], x4[(unsigned)cw >> 6], s_img[id][0] * box.prd[0],
                                           s_img[id][1] * box.prd[1], s_img[id][2] * box.prd[2],
                                           cut);
                r = in ? r | (1u << k) : r & ~(1u << k);
              }
              mw[q * 32] = (unsigned char)r;
            }
          }
        }
      }
    }
    __syncthreads();
    // order: groups of eight owned atoms of a cell, lane = (atom, one of four
    // chunks); candidates past the row end and the atom itself are cleared,
    // empty words dropped.  Candidate k is bit 31 - k: the next candidate is
    // then the leading one.
    {
      const int a = lane & 7, ws = lane >> 3;
      int grp = 0, colb = 0;
      for (int ca = 0; ca < ow; ca++) {
        const int o0 = s_start[own0 + ca], cnt = s_start[own0 + ca + 1] - o0;
        const int nch = s_nchunk[ca];
        for (int ab = 0; ab < cnt; ab += 8, colb += 8, grp++) {
          if (grp % (kNeighThreads / 32) != warp) continue;
          unsigned *mp = reinterpret_cast<unsigned *>(mask) + colb + a;
          unsigned short *sp = slot + colb + a;
          const int self = o0 + ab + a, sh = 4 * (a & 1);
          const bool act = ab + a < cnt;
          int tot = 0, kept = 0;  // kept: cols x the words kept so far
          const unsigned below = 0x01010101u & ((1u << (8 * ws)) - 1u);
          const uint2 *rp = reinterpret_cast<const uint2 *>(mp - (a & 1) + ws * cols);
          for (int w = ws; w < nch + ws; w += 4, rp += 2 * cols) {
            unsigned x = 0;
            int info = 0;
            if (w < nch) {
              info = s_chunk[ca][w];
              const uint2 raw = *rp;
              x = __brev(candidate_order(((raw.x >> sh) & 0x0F0F0F0Fu) |
                                         (((raw.y >> sh) << 4) & 0xF0F0F0F0u)));
              x &= 0xffffffffu << (32 - (info >> 20));
              const unsigned me = (unsigned)(self - (info & 0xffff));
              if (me < 32u && (info & 0xF0000) == 0x40000) x &= ~(0x80000000u >> me);
              if (!act) x = 0;
            }
            // words kept of this atom, these four chunks: bits 0, 8, 16, 24
            const unsigned full = (__ballot_sync(0xffffffffu, x != 0u) >> a) & 0x01010101u;
            if (x) {
              const int k = kept + cols * __popc(full & below);
              mp[k] = x;
              sp[k] = (unsigned short)info;
            }
            kept += cols * __popc(full);
            tot += __popc(x);
            __syncwarp();
          }
          tot += __shfl_xor_sync(0xffffffffu, tot, 8);
          tot += __shfl_xor_sync(0xffffffffu, tot, 16);
          if (ws == 0) s_count[colb + a] = (unsigned short)tot;
          const int most = __reduce_max_sync(0xffffffffu, tot);
          if (lane == 0) {
            atomicMax(&A.status[ST_MAXNEIGH], most);
            if (most > A.capacity) atomicExch(&A.status[ST_OVERFLOW], 1);
          }
        }
      }
    }
    __syncthreads();
    // append
    for (int la = tid; la < nown; la += kNeighThreads) {
      const int i = a0 + la;
      int ca = 0, col = la;
#pragma unroll
      for (int q = 0; q < TC - 1; q++)
        if (q + 1 < ow && la >= s_start[own0 + q + 1] - s_start[own0]) {
          ca = q + 1;
          // padding of the cells before this one
          const int cq = s_start[own0 + q + 1] - s_start[own0 + q];
          col += ((cq + 7) & ~7) - cq;
        }
      const int tot = s_count[col];
      // the stored count never exceeds the capacity, so readers stay in
      // bounds; an overflow is reported through the status word
      const int num = min(tot, A.capacity);
      A.numneigh[i] = num;
      const unsigned *mp = reinterpret_cast<const unsigned *>(mask) + col;
      const unsigned short *sp = slot + col;
      unsigned x = 0;
      const int *cw = word;
      auto next = [&]() -> int {
        if (x == 0u) {
          x = *mp;
          cw = word + *sp + 31;
          mp += cols;
          sp += cols;
        }
        const int b = 31 - __clz(x);
        x ^= 1u << b;
        return cw[-b] - ca;
      };
      int4 *out = reinterpret_cast<int4 *>(A.nlist) + i;
      for (int s = num >> 2; s > 0; s--, out += A.stride) {
        int4 e;
        e.x = next();
        e.y = next();
        e.z = next();
        e.w = next();
        *out = e;
      }
      if (num & 3) {
        // the last, partly filled slab ends in pad entries
        const int pad = md_pad_entry(i);
        int4 e = make_int4(pad, pad, pad, pad);
        e.x = next();
        if ((num & 3) > 1) e.y = next();
        if ((num & 3) > 2) e.z = next();
        *out = e;
      }
    }
    return;
  }
  // fallback (a tile too crowded for shared memory, or cells far wider than
  // the cutoff): one thread per owned atom, candidates read from global
  // memory, FP64 test
  for (int la = tid; la < nown; la += kNeighThreads) {
    const int i = a0 + la;
    int ca = 0;
#pragma unroll
    for (int q = 0; q < TC - 1; q++)
      if (q + 1 < ow && la >= s_start[own0 + q + 1] - s_start[own0]) ca = q + 1;
    const double4 xi = x4[i];
    const int ti = (int)xi.w;
    const int pad = md_pad_entry(i);
    int count = 0;
    int4 buf = make_int4(pad, pad, pad, pad);
    int4 *out = reinterpret_cast<int4 *>(A.nlist) + i;
    const int slabs = A.capacity >> 2;
    for (int r = 0; r < 9; r++)
      for (int dx = 0; dx < 3; dx++) {
        const int id = ca + dx + NSX * r;
        const int code = dx + row_code(r);
        const double shx = s_img[id][0] * box.prd[0], shy = s_img[id][1] * box.prd[1],
                     shz = s_img[id][2] * box.prd[2];
        const int j0 = s_src[id], j1 = j0 + s_start[id + 1] - s_start[id];
        for (int j = j0; j < j1; j++) {
          if (code == MD_CODE_SELF && j == i) continue;
          const double4 xj = x4[j];
          const double cut = SINGLE ? A.cutneighsq[A.ntp1 + 1] : cns[ti * A.ntp1 + (int)xj.w];
          if (!exact_pair(xi, xj, shx, shy, shz, cut)) continue;
          const int e = md_make_entry(j, code), k = count & 3;
          if (k == 0) buf = make_int4(e, pad, pad, pad);
          else if (k == 1) buf.y = e;
          else if (k == 2) buf.z = e;
          else buf.w = e;
          count++;
          if (k == 3 && (count >> 2) <= slabs) out[(size_t)((count >> 2) - 1) * A.stride] = buf;
        }
      }
    if ((count & 3) && (count >> 2) < slabs) out[(size_t)(count >> 2) * A.stride] = buf;
    A.numneigh[i] = count < A.capacity ? count : A.capacity;
    atomicMax(&A.status[ST_MAXNEIGH], count);
    if (count > A.capacity) atomicExch(&A.status[ST_OVERFLOW], 1);
  }
}

// ---------------------------------------------------------------------------
// Export of Neighbor::half_bin_newton's half list from the full list.
struct HalfBins {
  double lo[3], hi[3], bininv[3], binsize[3];
  int nbin[3], mbinlo[3];
  int sx, sy, sz;
  double cutneighmaxsq;
};

__device__ __forceinline__ int coord2bin_dim(double x, double lo, double hi, double inv, int nbin) {
  // Neighbor::coord2bin for one dimension (src/neighbor.cpp:1918-1947)
  int ix;
  if (x >= hi) ix = (int)((x - hi) * inv) + nbin;
  else if (x >= lo) {
    ix = (int)((x - lo) * inv);
    ix = ix < nbin - 1 ? ix : nbin - 1;
  } else ix = (int)((x - lo) * inv) - 1;
  return ix;
}

__device__ __forceinline__ double bin_distance(const HalfBins &b, int i, int j, int k) {
  double dx = i > 0 ? (i - 1) * b.binsize[0] : (i == 0 ? 0.0 : (i + 1) * b.binsize[0]);
  double dy = j > 0 ? (j - 1) * b.binsize[1] : (j == 0 ? 0.0 : (j + 1) * b.binsize[1]);
  double dz = k > 0 ? (k - 1) * b.binsize[2] : (k == 0 ? 0.0 : (k + 1) * b.binsize[2]);
  return dx * dx + dy * dy + dz * dz;
}

template <bool WRITE>
__global__ void k_half(int n, int stride, BoxGeom box, HalfBins hb, const double4 *__restrict__ x4,
                       const int *__restrict__ cell, const int *__restrict__ orig,
                       const int *__restrict__ nlist, const int *__restrict__ numneigh,
                       int *__restrict__ count_out, const long long *__restrict__ offset,
                       int *__restrict__ jowner, int *__restrict__ jimage, long long cap) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 xi = x4[i];
  int bi[3] = {coord2bin_dim(xi.x, hb.lo[0], hb.hi[0], hb.bininv[0], hb.nbin[0]),
               coord2bin_dim(xi.y, hb.lo[1], hb.hi[1], hb.bininv[1], hb.nbin[1]),
               coord2bin_dim(xi.z, hb.lo[2], hb.hi[2], hb.bininv[2], hb.nbin[2])};
  int cx, cy, cz;
  md_cell_unpack(cell[i], cx, cy, cz);
  int ci[3] = {cx, cy, cz};
  int oi = orig[i];
  int num = numneigh[i];
  long long out = WRITE ? offset[oi] : 0;
  int cnt = 0;
  for (int k = 0; k < num; k++) {
    unsigned int e = (unsigned int)nlist[md_slab(k, i, stride)];
    int j, dc[3];
    md_entry(e, j, dc[0], dc[1], dc[2]);
    int s[3];
    double g[3];
    double4 xj = x4[j];
    double xjv[3] = {xj.x, xj.y, xj.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      int c = ci[d] + dc[d];
      s[d] = c < 0 ? -1 : (c >= box.ncell[d] ? 1 : 0);
      g[d] = __dadd_rn(xjv[d], s[d] * box.prd[d]);
    }
    int bj[3] = {coord2bin_dim(g[0], hb.lo[0], hb.hi[0], hb.bininv[0], hb.nbin[0]),
                 coord2bin_dim(g[1], hb.lo[1], hb.hi[1], hb.bininv[1], hb.nbin[1]),
                 coord2bin_dim(g[2], hb.lo[2], hb.hi[2], hb.bininv[2], hb.nbin[2])};
    int ox = bj[0] - bi[0], oy = bj[1] - bi[1], oz = bj[2] - bi[2];
    bool ghost = (s[0] | s[1] | s[2]) != 0;
    bool own;
    if (ox == 0 && oy == 0 && oz == 0) {
      if (!ghost) own = orig[j] > oi;  // j beyond i in the bin's linked list
      else {                            // ghost "above and to the right"
        own = !(g[2] < xi.z) &&
              !(g[2] == xi.z && (g[1] < xi.y || (g[1] == xi.y && g[0] < xi.x)));
      }
    } else {
      own = (oz > 0 || oy > 0 || (oy == 0 && ox > 0)) && oz >= 0 && oz <= hb.sz &&
            ox >= -hb.sx && ox <= hb.sx && oy >= -hb.sy && oy <= hb.sy &&
            bin_distance(hb, ox, oy, oz) < hb.cutneighmaxsq;
    }
    if (own) {
      if (WRITE && out + cnt < cap) {
        jowner[out + cnt] = orig[j];
        jimage[out + cnt] = (s[0] + 1) + 3 * (s[1] + 1) + 9 * (s[2] + 1);
      }
      cnt++;
    }
  }
  if (!WRITE) count_out[oi] = cnt;
}

__global__ void k_prefix_ll(int n, const int *__restrict__ cnt, long long *__restrict__ off,
                            long long *__restrict__ total) {
  // single-thread prefix over atoms (export path only, not per step)
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  long long s = 0;
  for (int i = 0; i < n; i++) {
    off[i] = s;
    s += cnt[i];
  }
  *total = s;
}

}  // namespace

// Whether a tile of the mean density can be staged (what some atoms more or
// less then need, the capacity below and its feedback cover).
static bool mean_tile_fits(const b200_ctx *c, int tc) {
  const double per_cell = c->ncells > 0 ? (double)c->n / c->ncells : 0.0;
  const int chunks = 9 * ((int)(3.0 * per_cell / 32.0) + 1), cols = tc * (((int)per_cell + 7) & ~7);
  return chunks <= max_chunks(tc) && cols <= kMaxCols &&
         tile_units((int)(9 * (tc + 2) * per_cell), chunks, cols, c->ntypes == 1) <= kStageUnitsMax;
}

// Cells along x per builder tile.  A tile of two stages 18 cells per owned
// cell instead of 27, but gives half the CTAs and takes more shared memory.
// One build (sort included), one cell against two per tile:
//   19 atoms per cell: 1,000 cells 51 and 52 us, 1,331 56 and 52, 5,832 112 and
//     100, 13,824 226 and 192
//   27: 1,000 cells 58 and 63 us, 1,331 69 and 65; 32: 8,000 cells 279 and 278
//   44: 5,832 cells 347 and 331 us; 62: 4,096 cells 444 and 508; 93: 2,744
//     cells 1,122 and 1,104; from 108 on, where a tile of two no longer fits
//     (mean_tile_fits), 891 and 7,744
// so two from seven tiles per SM and up to 50 atoms per cell on the mean, unless
// the atoms are so uneven that many two-cell tiles cannot be staged (a slab in
// vacuum; md_stage_feedback).  Four cells took
// 41.5 ms where two take 41.1 (a run of 4,000,000 atoms).  Replica boxes are a
// few cells wide, so half of their two-cell tiles would own one cell (11.78
// against 11.66 ms).
int md_tile_cells(const b200_ctx *c) {
  return !c->nrep && !c->narrow && c->ncells >= 7 * md_sms(c) && (double)c->n <= 50.0 * c->ncells
             ? 2
             : 1;
}

// Shared memory of the builder tiles, in 16-byte units: what a tile of the
// mean density takes, with some room, raised when a build reports a larger
// tile.  For a batch the mean is the batch's (the common case, at full
// occupancy); the densest replicas' tiles are built in a second pass with
// md_stage_cap2.  A box whose mean tile is too crowded to be staged takes the
// global-memory path everywhere, and none of the memory, which would leave one
// CTA per SM.
int md_stage_cap(const b200_ctx *c) {
  if (!c->nrep && !mean_tile_fits(c, c->tile_cells)) return 0;
  const double per_cell = c->ncells > 0 ? (double)c->n / c->ncells : 0.0;
  int cap = tile_units_of(per_cell, c->tile_cells, c->ntypes == 1);
  if (!c->nrep && c->stage_need > cap) cap = c->stage_need;
  return std::min((cap + 31) & ~31, kStageUnitsMax);
}

// second-pass capacity of a batch: the densest replica's tiles (0 when the
// first pass holds every tile)
int md_stage_cap2(const b200_ctx *c) {
  if (!c->nrep) return 0;
  double per_cell = 0.0;
  for (int r = 0; r < c->nrep; r++) {
    const BoxGeom &b = c->rep_box[r];
    const double d = (double)c->rep_natoms[r] / ((double)b.ncell[0] * b.ncell[1] * b.ncell[2]);
    per_cell = d > per_cell ? d : per_cell;
  }
  int cap = tile_units_of(per_cell, c->tile_cells, c->ntypes == 1);
  if (c->stage_need > cap) cap = c->stage_need;
  cap = std::min((cap + 31) & ~31, kStageUnitsMax);
  return cap > md_stage_cap(c) ? cap : 0;
}

// After a build: raise the capacity when some tile needed more than the
// current one holds and, with `lower` (staged_max is of a single build of the
// current atoms), bring it down when no tile needs that much any more: it
// would cost every later system resident blocks.  Such a build also narrows the
// tiles to one cell when more than a fiftieth of the atoms (`unstaged`) lie in
// two-cell tiles that no capacity can stage: a slab of 219,488 atoms, 127 per
// cell, in a box three times as long, 12.4 ms a build with two, 1.2 with one.
// Returns true when the launch changed (the caller re-captures its graphs).
bool md_stage_feedback(b200_ctx *c, int staged_max, int unstaged, bool lower) {
  if (lower && c->tile_cells == 2 && unstaged > c->n / 50) {
    c->narrow = true;
    c->narrow_n = c->n;
    c->narrow_cells = c->ncells;
    c->tile_cells = 1;
    c->stage_need = 0;
    return true;
  }
  auto cap_now = [&] {
    const int cap2 = md_stage_cap2(c);
    return cap2 > 0 ? cap2 : md_stage_cap(c);
  };
  const int cap = cap_now();
  if (cap == 0) return false;
  const bool raise = staged_max > cap && cap < kStageUnitsMax;
  if (!raise && !(lower && staged_max + staged_max / 4 < c->stage_need)) return false;
  c->stage_need = staged_max + staged_max / 10;
  return cap_now() != cap;
}

static cudaError_t launch_scan(b200_ctx *c, int m, const int *in, int *out, const int *flag) {
  int tiles = (m + kScanTile - 1) / kScanTile;
  if (tiles > kScanTile) return cudaErrorInvalidValue;
  int *sums = c->scan_tmp;
  k_scan_tiles<<<tiles, kScanThreads, 0, c->stream>>>(m, in, out, sums, flag);
  c->launches++;
  if (tiles > 1) {
    k_scan_tiles<<<1, kScanThreads, 0, c->stream>>>(tiles, sums, sums, nullptr, flag);
    k_scan_add<<<tiles, 256, 0, c->stream>>>(m, out, sums, flag);
    c->launches += 2;
  }
  return cudaGetLastError();
}

template <int TC>
static cudaError_t launch_tiles(b200_ctx *c, const NeighArgs &A, int tiles, cudaStream_t st) {
  // the shared-memory opt-in, once per device this process uses
  static std::atomic<unsigned long long> opt_in{0ull};
  const unsigned long long dev_bit = 1ull << (c->device & 63);
  if (!(opt_in.load() & dev_bit)) {
    const int most = kStageUnitsMax * 16;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_neigh_tiles<TC, true, false>, attr, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_neigh_tiles<TC, false, false>, attr, most);
    if constexpr (TC == 1) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_neigh_tiles<1, true, true>, attr, most);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_neigh_tiles<1, false, true>, attr, most);
    }
    if (e != cudaSuccess) return e;
    opt_in.fetch_or(dev_bit);
  }
  const size_t smem = (size_t)A.units * 16;
  if constexpr (TC == 1) {  // a batch's tiles own one cell (md_tile_cells)
    if (c->nrep) {
      if (c->ntypes == 1) k_neigh_tiles<1, true, true><<<tiles, kNeighThreads, smem, st>>>(A);
      else k_neigh_tiles<1, false, true><<<tiles, kNeighThreads, smem, st>>>(A);
      c->launches++;
      return cudaGetLastError();
    }
  }
  if (c->ntypes == 1) k_neigh_tiles<TC, true, false><<<tiles, kNeighThreads, smem, st>>>(A);
  else k_neigh_tiles<TC, false, false><<<tiles, kNeighThreads, smem, st>>>(A);
  c->launches++;
  return cudaGetLastError();
}

static cudaError_t launch_list(b200_ctx *c, const int *d_flag) {
  const int tc = c->tile_cells;
  const int tiles = c->nrep ? c->ntiles
                            : ((c->box.ncell[0] + tc - 1) / tc) * c->box.ncell[1] * c->box.ncell[2];
  NeighArgs A;
  A.n = c->n;
  A.stride = c->stride;
  A.capacity = c->capacity;
  A.ntp1 = c->ntypes + 1;
  A.box = c->box;
  A.reps = c->reps();
  A.scale = std::exp2(1.0 - std::floor(std::log2(c->cutneighmax)));
  double cmax = 0.0, cmin = 1.0e300;
  for (int i = 1; i <= c->ntypes; i++)
    for (int j = 1; j <= c->ntypes; j++) {
      cmax = std::max(cmax, c->cutneighsq[i * A.ntp1 + j]);
      cmin = std::min(cmin, c->cutneighsq[i * A.ntp1 + j]);
    }
  A.cmax = (float)(cmax * A.scale * A.scale);
  A.dmax = (float)((cmax - cmin) * A.scale * A.scale);
  A.cutneighsq = c->cutneighsq_dev;
  A.x4 = c->x4;
  A.cell_start = c->cell_start;
  A.nlist = c->nlist;
  A.numneigh = c->numneigh;
  A.status = c->status;
  A.flag = d_flag;
  const int cap = md_stage_cap(c);
  const int cap2 = md_stage_cap2(c);  // a batch's densest tiles, or 0
  A.units1 = cap;
  auto launch = [&](int units, int pass, cudaStream_t st) {
    A.units = units;
    A.pass = pass;
    return tc == 2 ? launch_tiles<2>(c, A, tiles, st) : launch_tiles<1>(c, A, tiles, st);
  };
  if (cap2 == 0) return launch(cap, 0, c->stream);
  // The two passes build disjoint tiles, so the second (the densest tiles,
  // large staging, few blocks per SM) runs on the side stream beside the
  // first instead of after it; the join makes the main stream wait for both.
  // Inside a graph capture the fork and join become graph dependencies.
  cudaError_t e = cudaEventRecord(c->ev_fork, c->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->s_aux, c->ev_fork, 0);
  if (e == cudaSuccess) e = launch(cap, 1, c->stream);
  if (e == cudaSuccess) e = launch(cap2, 2, c->s_aux);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev_join, c->s_aux);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_join, 0);
  return e;
}

// the one-launch sort, for a box that fits it
static bool sort_all_fits(const b200_ctx *c) {
  return c->ncells < kSortCells && md_blocks(c->n, kSortThreads) <= 4 * md_sms(c);
}

static cudaError_t launch_sort_all(b200_ctx *c, const int *d_flag) {
  SortArgs A;
  A.n = c->n;
  A.stride = c->stride;
  A.m = c->ncells + 1;
  A.box = c->box;
  A.reps = c->reps();
  A.x4 = c->x4;
  A.v = c->v;
  A.orig = c->orig;
  A.image = c->image;
  A.cell = c->cell;
  A.where = c->where;
  A.cell_count = c->cell_count;
  A.cell_start = c->cell_start;
  A.key = c->perm;
  A.xq = c->prec == B200_PREC_MIXED ? c->xq : nullptr;
  A.xhold = c->check ? c->xhold : nullptr;
  A.status = c->status;
  A.flag = d_flag;
  A.bar = c->bar + 2 * MD_BAR_WORDS;
  void *args[1] = {&A};
  if (c->expire_waits) {
    const cudaError_t e = cudaMemsetAsync(A.bar, kExpireByte, sizeof(unsigned), c->stream);
    if (e != cudaSuccess) return e;
  }
  c->launches++;
  return cudaLaunchCooperativeKernel(
      c->nrep ? (const void *)k_sort_all<true> : (const void *)k_sort_all<false>,
      dim3(md_blocks(c->n, kSortThreads)), dim3(kSortThreads), args, 0, c->stream);
}

cudaError_t md_rebuild(b200_ctx *c, const int *d_flag) {
  if (sort_all_fits(c)) {
    const cudaError_t e = launch_sort_all(c, d_flag);
    return e != cudaSuccess ? e : launch_list(c, d_flag);
  }
  const int n = c->n, B = 256;
  const int m = c->ncells + 1;
  const Reps R = c->reps();
  if (c->nrep)
    k_wrap_bin<true><<<md_blocks(n, B), B, 0, c->stream>>>(n, c->box, R, c->x4, c->image,
                                                           c->cell_count, c->slot, c->cell_tmp,
                                                           c->status, d_flag);
  else
    k_wrap_bin<false><<<md_blocks(n, B), B, 0, c->stream>>>(n, c->box, R, c->x4, c->image,
                                                            c->cell_count, c->slot, c->cell_tmp,
                                                            c->status, d_flag);
  c->launches += 1;
  cudaError_t e = launch_scan(c, m, c->cell_count, c->cell_start, d_flag);
  if (e != cudaSuccess) return e;
  k_scatter<<<md_blocks(n, B), B, 0, c->stream>>>(n, c->cell_tmp, c->slot, c->cell_start, c->perm,
                                                  m, c->cell_count, d_flag);
  k_sort_cells<<<md_blocks(c->ncells, kSortWarps), kSortWarps * 32, 0, c->stream>>>(
      c->ncells, c->cell_start, c->perm, c->slot, c->orig, d_flag);
  if (c->nrep)
    k_gather<true><<<md_blocks(n, B), B, 0, c->stream>>>(
        n, c->stride, c->box, R, c->perm, c->x4, c->x4b, c->v, c->vb, c->orig, c->origb, c->image,
        c->imageb, c->cell_tmp, c->cell, c->prec == 1 ? c->xq : nullptr,
        c->check ? c->xhold : nullptr, d_flag);
  else
    k_gather<false><<<md_blocks(n, B), B, 0, c->stream>>>(
        n, c->stride, c->box, R, c->perm, c->x4, c->x4b, c->v, c->vb, c->orig, c->origb, c->image,
        c->imageb, c->cell_tmp, c->cell, c->prec == 1 ? c->xq : nullptr,
        c->check ? c->xhold : nullptr, d_flag);
  k_copyback<<<md_blocks(n, B), B, 0, c->stream>>>(n, c->stride, c->x4b, c->x4, c->vb, c->v,
                                                   c->origb, c->orig, c->imageb, c->image,
                                                   c->where, c->status, d_flag);
  e = launch_list(c, d_flag);
  if (e != cudaSuccess) return e;
  c->launches += 3;
  return cudaGetLastError();
}

// LAMMPS bins of Neighbor::setup_bins (src/neighbor.cpp:1538-1702) for a
// single periodic process: binsize = cutneighmax/2, bounding box extended by
// the ghost cutoff, half stencil extents sx, sy, sz.
static HalfBins half_bins(const b200_ctx *c) {
  HalfBins hb{};
  const double SMALL = 1.0e-6;
  double cutghost = c->cutneighmax;
  double binsize_optimal = 0.5 * c->cutneighmax;
  double bbox[3];
  for (int d = 0; d < 3; d++) bbox[d] = c->box.hi[d] - c->box.lo[d];
  if (binsize_optimal == 0.0) binsize_optimal = bbox[0];
  double binsizeinv = 1.0 / binsize_optimal;
  for (int d = 0; d < 3; d++) {
    hb.lo[d] = c->box.lo[d];
    hb.hi[d] = c->box.hi[d];
    int nb = (int)(bbox[d] * binsizeinv);
    if (nb == 0) nb = 1;
    hb.nbin[d] = nb;
    hb.binsize[d] = bbox[d] / nb;
    hb.bininv[d] = 1.0 / hb.binsize[d];
    double coord = (c->box.lo[d] - cutghost) - SMALL * bbox[d];
    int lo = (int)((coord - c->box.lo[d]) * hb.bininv[d]);
    if (coord < c->box.lo[d]) lo = lo - 1;
    hb.mbinlo[d] = lo - 1;
  }
  int s[3];
  for (int d = 0; d < 3; d++) {
    s[d] = (int)(c->cutneighmax * hb.bininv[d]);
    if (s[d] * hb.binsize[d] < c->cutneighmax) s[d]++;
  }
  hb.sx = s[0];
  hb.sy = s[1];
  hb.sz = s[2];
  hb.cutneighmaxsq = c->cutneighmax * c->cutneighmax;
  return hb;
}

cudaError_t md_half_list(b200_ctx *c, int *d_num, int *d_jowner, int *d_jimage, long long cap,
                         long long *total) {
  const int n = c->n, B = 128;
  HalfBins hb = half_bins(c);
  long long *d_off = nullptr, *d_total = nullptr;
  cudaError_t e = cudaMallocAsync((void **)&d_off, sizeof(long long) * (size_t)(n + 1), c->stream);
  if (e != cudaSuccess) return e;
  e = cudaMallocAsync((void **)&d_total, sizeof(long long), c->stream);
  if (e != cudaSuccess) return e;
  k_half<false><<<md_blocks(n, B), B, 0, c->stream>>>(n, c->stride, c->box, hb, c->x4, c->cell,
                                                      c->orig, c->nlist, c->numneigh, d_num,
                                                      nullptr, nullptr, nullptr, 0);
  k_prefix_ll<<<1, 1, 0, c->stream>>>(n, d_num, d_off, d_total);
  if (d_jowner && cap > 0)
    k_half<true><<<md_blocks(n, B), B, 0, c->stream>>>(n, c->stride, c->box, hb, c->x4, c->cell,
                                                       c->orig, c->nlist, c->numneigh, nullptr,
                                                       d_off, d_jowner, d_jimage, cap);
  c->launches += d_jowner && cap > 0 ? 3 : 2;
  e = cudaMemcpyAsync(total, d_total, sizeof(long long), cudaMemcpyDeviceToHost, c->stream);
  if (e != cudaSuccess) return e;
  cudaFreeAsync(d_off, c->stream);
  cudaFreeAsync(d_total, c->stream);
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}
