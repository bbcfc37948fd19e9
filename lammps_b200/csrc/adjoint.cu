// adjoint.cu -- forces and their adjoint for differentiable force matching
// with pair_style lj/cut (any number of types up to MD_ADJ_MAXTYPES).
//
// Forward:  F_i = sum_j phi_ij d_ij,  d_ij = x_i - x_j (periodic image),
//           phi = (lj1 r^-6 - lj2) r^-6 r^-2  for r^2 < cutsq[ti][tj]
//           -- the pair force of PairLJCut::compute (src/pair_lj_cut.cpp:100-113)
//           with lj1 = 48 eps sigma^12, lj2 = 24 eps sigma^6
//           (PairLJCut::init_one, src/pair_lj_cut.cpp:560-563).
// Backward, given G = dL/dF (per atom):
//   dL/dlj1[ti][tj] = sum over directed pairs (G_i . d_ij) r^-14
//   dL/dlj2[ti][tj] = -sum over directed pairs (G_i . d_ij) r^-8
//   dL/dx_i = sum_j H_ij (G_i - G_j),  H_ij = phi I + 2 phi' d d^T,
//             phi' = dphi/d(r^2) = (4 lj2 - 7 lj1 r^-6) r^-6 r^-4
// (the Hessian-vector product of the loss through the forces).  With the
// engine's full neighbor list every atom sums its own terms, so neither pass
// needs atomics; per-type-pair parameter gradients are reduced per block and
// then in a fixed order, so results are reproducible.  The cutoff itself is
// not differentiated: a pair that crosses r = rc under a parameter change
// contributes a jump that finite differences see and this gradient does not.
//
// MIXED: FP32 pair arithmetic on separations formed from the fixed-point
// coordinates (md_xq, as the mixed force kernels), FP64 accumulation of
// forces, gradients and sums.
#include "md_state.h"

namespace {

constexpr int kAdjThreads = 128;
constexpr int kAdjNP = MD_ADJ_MAXTYPES * MD_ADJ_MAXTYPES;  // type pairs

struct AdjTables {
  int ntypes;
  double lj1[kAdjNP], lj2[kAdjNP], cutsq[kAdjNP];  // [(ti-1)*ntypes + (tj-1)]
};

struct AdjArgs {
  int n, stride;
  AdjTables T;
  BoxGeom box;
  const double4 *x4;
  const int4 *xq;
  const int *cell, *nlist, *numneigh, *orig;
  const double4 *gs;  // backward: G in the sorted order
  double *out;        // forces, or dL/dx, in the caller's order
  double *partial, *gtab;
  unsigned int *counter;
};

// The type-pair tables in shared memory: a lane looks its pair up by an index
// of its own, which the parameter (constant) bank would serve one by one.
struct AdjShared {
  double lj1[kAdjNP], lj2[kAdjNP], cutsq[kAdjNP];
  float lj1f[kAdjNP], lj2f[kAdjNP];
};
__device__ __forceinline__ void load_tables(AdjShared &S, const AdjTables &T) {
  if (threadIdx.x < kAdjNP) {
    const int k = threadIdx.x;
    S.lj1[k] = T.lj1[k];
    S.lj2[k] = T.lj2[k];
    S.cutsq[k] = T.cutsq[k];
    S.lj1f[k] = (float)T.lj1[k];
    S.lj2f[k] = (float)T.lj2[k];
  }
  __syncthreads();
}

// Atom i's side of its pairs: position, type row and periodic shifts (FP64),
// or fixed-point position and unit lengths (mixed).
template <bool MIXED>
struct AdjAtom {
  double4 p;
  int4 q;
  int row;  // (ti - 1) * ntypes
  Shift3 sx, sy, sz;
  float qh[3], ql[3];
  __device__ __forceinline__ AdjAtom(const AdjArgs &a, int i) {
    if (MIXED) {
      q = a.xq[i];
      row = (q.w - 1) * a.T.ntypes;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        qh[d] = a.box.qs[d];
        ql[d] = a.box.qs_lo[d];
      }
    } else {
      p = a.x4[i];
      row = ((int)p.w - 1) * a.T.ntypes;
      int cx, cy, cz;
      md_cell_unpack(a.cell[i], cx, cy, cz);
      sx = shifts(cx, a.box.ncell[0], a.box.prd[0]);
      sy = shifts(cy, a.box.ncell[1], a.box.prd[1]);
      sz = shifts(cz, a.box.ncell[2], a.box.prd[2]);
    }
  }
  // separation, squared length and neighbour type (0-based) of entry e
  __device__ __forceinline__ void geom(unsigned e, const double4 &xj, const int4 &qj, double &dx,
                                       double &dy, double &dz, double &rsq, int &tj) const {
    if (MIXED) {
      // minimum-image separation from the fixed-point coordinates
      const float fx = md_qlen(md_qdiff(q.x, qj.x), qh[0], ql[0]);
      const float fy = md_qlen(md_qdiff(q.y, qj.y), qh[1], ql[1]);
      const float fz = md_qlen(md_qdiff(q.z, qj.z), qh[2], ql[2]);
      dx = fx;
      dy = fy;
      dz = fz;
      rsq = (double)(fx * fx + fy * fy + fz * fz);
      tj = qj.w - 1;
    } else {
      int j, ex, ey, ez;
      md_entry(e, j, ex, ey, ez);
      dx = p.x - (xj.x + pick(sx, ex));
      dy = p.y - (xj.y + pick(sy, ey));
      dz = p.z - (xj.z + pick(sz, ez));
      rsq = dx * dx + dy * dy + dz * dz;
      tj = (int)xj.w - 1;
    }
  }
};

// Forces in the caller's order.  TPA threads per atom take consecutive list
// entries (walk_list) and issue four gathers at a time.
template <bool MIXED, int TPA>
__global__ void __launch_bounds__(kAdjThreads) k_adj_forward(AdjArgs a) {
  __shared__ AdjShared S;
  load_tables(S, a.T);
  const int t = blockIdx.x * kAdjThreads + threadIdx.x;
  const int i = t / TPA, lane = t % TPA;
  const bool active = i < a.n;
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (active) {
    const AdjAtom<MIXED> me(a, i);
    auto four = [&](const unsigned (&ee)[4], int m) {
      double4 xj[4];
      int4 qj[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int j = u < m ? md_entry_j(ee[u]) : i;
        if (MIXED) qj[u] = __ldg(&a.xq[j]);
        else xj[u] = a.x4[j];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (u >= m) break;
        double dx, dy, dz, rsq;
        int tj;
        me.geom(ee[u], xj[u], qj[u], dx, dy, dz, rsq, tj);
        const int tt = me.row + tj;
        if (rsq < S.cutsq[tt]) {
          double phi;
          if (MIXED) {
            const float r2i = 1.0f / (float)rsq, r6i = r2i * r2i * r2i;
            phi = (double)((S.lj1f[tt] * r6i - S.lj2f[tt]) * r6i * r2i);
          } else {
            const double r2i = 1.0 / rsq, r6i = r2i * r2i * r2i;
            phi = (S.lj1[tt] * r6i - S.lj2[tt]) * r6i * r2i;
          }
          fx += phi * dx;
          fy += phi * dy;
          fz += phi * dz;
        }
      }
    };
    walk_list<TPA>(a.nlist, a.stride, i, a.numneigh[i], lane, four);
  }
  fx = lane_sum<TPA>(fx);
  fy = lane_sum<TPA>(fy);
  fz = lane_sum<TPA>(fz);
  if (active && lane == 0) {
    const int o = a.orig[i];
    a.out[3 * o] = fx;
    a.out[3 * o + 1] = fy;
    a.out[3 * o + 2] = fz;
  }
}

// G in the caller's order -> G in the sorted order, one 32-byte record per
// atom (a pair's gather is then one sector)
__global__ void k_adj_gather(int n, const int *__restrict__ orig, const double *__restrict__ g,
                             double4 *__restrict__ gs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = orig[i];
  gs[i] = make_double4(g[3 * o], g[3 * o + 1], g[3 * o + 2], 0.0);
}

// dL/dx in the caller's order, and dL/dlj1, dL/dlj2 per type pair.  An atom's
// type is the row of all its pairs, so a thread keeps sums for its row's NT
// columns only (2 NT accumulators; one per type pair of the whole table, 32
// of them, made the table update the largest part of the pair loop: 138 us at
// 8,000 atoms, mixed, and 182 us at 54,647, FP64).  A block
// adds its threads' sums by row in shared memory in a fixed order, the last
// block the blocks' sums.
template <bool MIXED, int NT, int TPA>
__global__ void __launch_bounds__(kAdjThreads) k_adj_backward(AdjArgs a) {
  constexpr int NV = 2 * NT * NT;
  __shared__ AdjShared S;
  __shared__ double s_acc[2 * NT][kAdjThreads];
  __shared__ int s_row[kAdjThreads];
  __shared__ bool last;
  load_tables(S, a.T);
  const int t = blockIdx.x * kAdjThreads + threadIdx.x;
  const int i = t / TPA, lane = t % TPA;
  const bool active = i < a.n;
  double acc[2 * NT];
#pragma unroll
  for (int k = 0; k < 2 * NT; k++) acc[k] = 0.0;
  double hx = 0.0, hy = 0.0, hz = 0.0;
  int myrow = -1;
  if (active) {
    const AdjAtom<MIXED> me(a, i);
    myrow = me.row / a.T.ntypes;
    const double4 gi = a.gs[i];
    auto four = [&](const unsigned (&ee)[4], int m) {
      double4 xj[4], gj[4];
      int4 qj[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int j = u < m ? md_entry_j(ee[u]) : i;
        if (MIXED) qj[u] = __ldg(&a.xq[j]);
        else xj[u] = a.x4[j];
        gj[u] = a.gs[j];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (u >= m) break;
        double dx, dy, dz, rsq;
        int tj;
        me.geom(ee[u], xj[u], qj[u], dx, dy, dz, rsq, tj);
        const int tt = me.row + tj;
        if (rsq < S.cutsq[tt]) {
          const double wx = gi.x - gj[u].x, wy = gi.y - gj[u].y, wz = gi.z - gj[u].z;
          double phi, phis, r14, r8;
          if (MIXED) {
            const float r2i = 1.0f / (float)rsq, r6i = r2i * r2i * r2i;
            const float l1 = S.lj1f[tt], l2 = S.lj2f[tt];
            phi = (double)((l1 * r6i - l2) * r6i * r2i);
            phis = (double)((4.0f * l2 - 7.0f * l1 * r6i) * r6i * r2i * r2i);
            r14 = (double)(r6i * r6i * r2i);
            r8 = (double)(r6i * r2i);
          } else {
            const double r2i = 1.0 / rsq, r6i = r2i * r2i * r2i;
            const double l1 = S.lj1[tt], l2 = S.lj2[tt];
            phi = (l1 * r6i - l2) * r6i * r2i;
            phis = (4.0 * l2 - 7.0 * l1 * r6i) * r6i * r2i * r2i;
            r14 = r6i * r6i * r2i;
            r8 = r6i * r2i;
          }
          const double dw = dx * wx + dy * wy + dz * wz;
          const double s = 2.0 * phis * dw;
          hx += phi * wx + s * dx;
          hy += phi * wy + s * dy;
          hz += phi * wz + s * dz;
          const double gd = gi.x * dx + gi.y * dy + gi.z * dz;
#pragma unroll
          for (int p = 0; p < NT; p++)
            if (NT == 1 || p == tj) {
              acc[2 * p] += gd * r14;
              acc[2 * p + 1] -= gd * r8;
            }
        }
      }
    };
    walk_list<TPA>(a.nlist, a.stride, i, a.numneigh[i], lane, four);
  }
  hx = lane_sum<TPA>(hx);
  hy = lane_sum<TPA>(hy);
  hz = lane_sum<TPA>(hz);
  if (active && lane == 0) {
    const int o = a.orig[i];
    a.out[3 * o] = hx;
    a.out[3 * o + 1] = hy;
    a.out[3 * o + 2] = hz;
  }
  // parameter gradients: value k = 2 (ti NT + tj) + q of the block
#pragma unroll
  for (int k = 0; k < 2 * NT; k++) s_acc[k][threadIdx.x] = acc[k];
  s_row[threadIdx.x] = myrow;
  __syncthreads();
  const int warp = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int k = warp; k < NV; k += kAdjThreads / 32) {
    const int ti = (k >> 1) / NT, col = 2 * ((k >> 1) % NT) + (k & 1);
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kAdjThreads / 32; q++)
      v += s_row[l + 32 * q] == ti ? s_acc[col][l + 32 * q] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) a.partial[(size_t)blockIdx.x * NV + k] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = warp; k < NV; k += kAdjThreads / 32) {
    double v = 0.0;
    for (unsigned b = l; b < gridDim.x; b += 32) v += __ldcg(&a.partial[(size_t)b * NV + k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    // the table is (ntypes x ntypes)
    const int ti = (k >> 1) / NT, tj = (k >> 1) % NT, nt = a.T.ntypes;
    if (l == 0 && ti < nt && tj < nt) a.gtab[2 * (ti * nt + tj) + (k & 1)] = v;
  }
  if (threadIdx.x == 0) *a.counter = 0u;
}

AdjTables make_tables(const b200_ctx *c, const double *lj1, const double *lj2,
                      const double *cutsq) {
  AdjTables T{};
  T.ntypes = c->ntypes;
  const int w = c->ntypes + 1;
  for (int a = 1; a <= c->ntypes; a++)
    for (int b = 1; b <= c->ntypes; b++) {
      const int p = (a - 1) * c->ntypes + (b - 1);
      T.lj1[p] = lj1[a * w + b];
      T.lj2[p] = lj2[a * w + b];
      T.cutsq[p] = cutsq[a * w + b];
    }
  return T;
}

}  // namespace

// Threads per atom of both passes: as many as the chip has room for.  Forward
// and backward call, two types, us with 1, 2, 4 and 8 (mixed | FP64):
//    8,000   112  92  78  74 | 125  91  83  76
//   10,976   112  87  80  70 | 125  96  83  80
//   13,500   112  86  79  78 | 125  96  82  82
//   23,328   107  90  81  84 | 126 103  99  98
//   28,880   108 108 104 103 | 129 108 108 115
//   42,592   118 101 101 111 | 141 134 132 135
//   55,296   120 120 116 127 | 140 153 141 152
// (one type alike; with four, fewer threads win a little earlier)
static int adj_tpa(int n) {
  return n >= 45000 ? 1 : n >= 26000 ? 2 : n >= 12000 ? 4 : 8;
}

static AdjArgs adj_args(b200_ctx *c, const double *lj1, const double *lj2, const double *cutsq) {
  AdjArgs a{};
  a.n = c->n;
  a.stride = c->stride;
  a.T = make_tables(c, lj1, lj2, cutsq);
  a.box = c->box;
  a.x4 = c->x4;
  a.xq = c->xq;
  a.cell = c->cell;
  a.nlist = c->nlist;
  a.numneigh = c->numneigh;
  a.orig = c->orig;
  a.partial = c->partial;
  a.counter = c->counter;
  return a;
}

template <bool MIXED>
static void launch_forward(b200_ctx *c, const AdjArgs &a, int tpa) {
  const int grid = md_blocks((long long)a.n * tpa, kAdjThreads);
  if (tpa == 1) k_adj_forward<MIXED, 1><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else if (tpa == 2) k_adj_forward<MIXED, 2><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else if (tpa == 4) k_adj_forward<MIXED, 4><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else k_adj_forward<MIXED, 8><<<grid, kAdjThreads, 0, c->stream>>>(a);
}

template <bool MIXED, int NT>
static void launch_backward(b200_ctx *c, const AdjArgs &a, int tpa) {
  const int grid = md_blocks((long long)a.n * tpa, kAdjThreads);
  if (tpa == 1) k_adj_backward<MIXED, NT, 1><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else if (tpa == 2) k_adj_backward<MIXED, NT, 2><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else if (tpa == 4) k_adj_backward<MIXED, NT, 4><<<grid, kAdjThreads, 0, c->stream>>>(a);
  else k_adj_backward<MIXED, NT, 8><<<grid, kAdjThreads, 0, c->stream>>>(a);
}

cudaError_t md_adj_forward(b200_ctx *c, const double *lj1, const double *lj2, const double *cutsq,
                           double *f) {
  AdjArgs a = adj_args(c, lj1, lj2, cutsq);
  a.out = f;
  const int tpa = adj_tpa(c->n);
  if (c->prec == B200_PREC_MIXED) launch_forward<true>(c, a, tpa);
  else launch_forward<false>(c, a, tpa);
  c->launches++;
  return cudaGetLastError();
}

cudaError_t md_adj_backward(b200_ctx *c, const double *lj1, const double *lj2,
                            const double *cutsq, const double *g, double *gx, double *gs,
                            double *gtab) {
  AdjArgs a = adj_args(c, lj1, lj2, cutsq);
  double4 *gs4 = reinterpret_cast<double4 *>(gs);
  a.gs = gs4;
  a.out = gx;
  a.gtab = gtab;
  const int tpa = adj_tpa(c->n), nt = c->ntypes;
  k_adj_gather<<<md_blocks(c->n, 256), 256, 0, c->stream>>>(c->n, c->orig, g, gs4);
  if (c->prec == B200_PREC_MIXED) {
    if (nt == 1) launch_backward<true, 1>(c, a, tpa);
    else if (nt == 2) launch_backward<true, 2>(c, a, tpa);
    else launch_backward<true, 4>(c, a, tpa);
  } else {
    if (nt == 1) launch_backward<false, 1>(c, a, tpa);
    else if (nt == 2) launch_backward<false, 2>(c, a, tpa);
    else launch_backward<false, 4>(c, a, tpa);
  }
  c->launches += 2;
  return cudaGetLastError();
}

// caller-order device positions -> the context's sorted FP64 positions
// (types kept, image flags restarted); the next build wraps and re-sorts.
// hxy (if given) and hz keep them as they came (b200_ctx::adj_held).
__global__ void k_adj_positions(int n, const int *__restrict__ orig, const double *__restrict__ x,
                                double4 *__restrict__ x4, int *__restrict__ image,
                                double2 *__restrict__ hxy, double *__restrict__ hz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = orig[i];
  const double4 p = x4[i];
  const double xo = x[3 * o], yo = x[3 * o + 1], zo = x[3 * o + 2];
  x4[i] = make_double4(xo, yo, zo, p.w);
  if (hxy) {
    hxy[o] = make_double2(xo, yo);
    hz[o] = zo;
  }
  image[i] = md_img_pack(0, 0, 0);
}

cudaError_t md_adj_positions(b200_ctx *c, const double *x) {
  k_adj_positions<<<md_blocks(c->n, 256), 256, 0, c->stream>>>(
      c->n, c->orig, x, c->x4, c->image,
      c->pstyle == B200_PAIR_LJ_CUT ? reinterpret_cast<double2 *>(c->xqb) : nullptr, c->rho);
  c->launches++;
  return cudaGetLastError();
}

// *diff = 1 when a bit of the n positions differs
__global__ void k_adj_compare(int n, const unsigned long long *__restrict__ x,
                              const ulonglong2 *__restrict__ hxy,
                              const unsigned long long *__restrict__ hz, int *diff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool ne = false;
  if (i < n) {
    const ulonglong2 h = hxy[i];
    ne = x[3 * i] != h.x || x[3 * i + 1] != h.y || x[3 * i + 2] != hz[i];
  }
  if (__any_sync(0xffffffffu, ne) && (threadIdx.x & 31) == 0) atomicExch(diff, 1);
}

cudaError_t md_adj_compare(b200_ctx *c, const double *x, int *diff) {
  k_adj_compare<<<md_blocks(c->n, 256), 256, 0, c->stream>>>(
      c->n, reinterpret_cast<const unsigned long long *>(x),
      reinterpret_cast<const ulonglong2 *>(c->xqb),
      reinterpret_cast<const unsigned long long *>(c->rho), diff);
  c->launches++;
  return cudaGetLastError();
}
