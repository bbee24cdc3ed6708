// nb_list.cu -- link-cell binning and Verlet-list build on the GPU.
//
// Replaces get_ngbr (energy/control/ngbr_list.c:297-581), ngbr_list
// (ngbr_list.c:35-101), get_ngbr_e (energy/control/elec_ngbr.c:220-358),
// ngbr_liste (ngbr_list.c:103-143) and the link-cell helpers get_lnklist /
// get_lnklist_e (energy/control/set_link.c:203-300).
//
// Pair membership comes out as CM3D decides it.  exact_entry takes the
// displacement in FP64, folds it with CM3D's period() arithmetic
// (md_period.new.c:39-52, CM3D's anint and operation order, no FMA contraction
// -- this file is compiled with -fmad=false as well) and compares with the
// per-interaction radius rmaxl_skin2[map[ti][tj]] / rmaxs_skin2 (LJ, after the
// map == -1 and exclusion tests) or rmaxl_skin2_e / rmaxs_skin2_e (charged
// atoms, after the charge-exclusion test).  A pair whose FP32 distance is
// further from every radius than a margin of some ten times its error, and
// whose image FP32 can tell, is decided by that distance (list_flags, fold);
// all others go through exact_entry.  The resulting pair sets are bit-identical
// to CM3D's.  The cell grid itself is our own: cells at least one list radius
// wide, atoms counting-sorted by cell (inside a cell by atom type, then atom
// index), and a stencil of unique neighbour cells, so every pair within range
// is seen exactly once per direction whatever CM3D's ncell_div is.
//
// A context may hold several independent systems (SysP, nb_common.cuh): each
// has its own box, cell grid and parameters, its cells and atoms occupy
// contiguous ranges, and a system is rebuilt only when its own displacement
// test asked for it (lreb[s]) unless the build covers every system (`all`).
//
// Outputs
//   lst[0..3]  CM3D's four half lists t, s, te, se as (i, j) with i < j
//   nbr        (mixed mode) a full list per atom in cell-sorted order; each
//              32-bit entry holds j's sorted index, the code of the cell shift
//              that turns cell-relative coordinates into the minimum-image
//              displacement, and whether the pair is in the t/s/te/se lists
//   xq, styp   cell-relative FP32 coordinates + charge and type, sorted order
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "nb_common.cuh"

namespace cm3d {

__device__ __forceinline__ bool sys_skip(int s, const int *__restrict__ sreb, int all) {
  return !all && sreb[s] == 0;
}

// ----------------------------------------------------------------- binning
// zero the cell counters of the systems being rebuilt
__global__ void k_cell_zero(int ncells, const int *__restrict__ cell_sys, const int *__restrict__ sreb, int all,
                            int *__restrict__ cell_count, const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells || sys_skip(cell_sys[c], sreb, all)) return;
  cell_count[c] = 0;
}

// the cell of atom i (and its image, in cimg)
__device__ __forceinline__ int place_in_cell(const SysP &P, int n, int i, const double *__restrict__ pos,
                                             int4 *__restrict__ cimg) {
  double x = pos[i], y = pos[n + i], z = pos[2 * n + i];
  double sv[3];
  for (int d = 0; d < 3; d++)
    sv[d] = __dadd_rn(__dadd_rn(__dmul_rn(x, P.hi[3 * d]), __dmul_rn(y, P.hi[3 * d + 1])),
                      __dmul_rn(z, P.hi[3 * d + 2]));
  int img[3], cc[3];
  for (int d = 0; d < 3; d++) {
    const int ncd = P.nc[d];
    double fl = floor(sv[d]);
    double fr = sv[d] - fl;                      // [0, 1]
    int c = (int)(fr * ncd);
    c = c < 0 ? 0 : (c >= ncd ? ncd - 1 : c);
    img[d] = (int)fl;
    cc[d] = c;
  }
  cimg[i] = make_int4(cc[0] | (cc[1] << 10) | (cc[2] << 20), img[0], img[1], img[2]);
  return P.c0 + (cc[0] * P.nc[1] + cc[1]) * P.nc[2] + cc[2];
}

__global__ void k_cell_assign(int n, const double *__restrict__ pos, const SysP *__restrict__ sp,
                              const int *__restrict__ sys_of, const int *__restrict__ sreb, int all,
                              int *__restrict__ cell_of, int *__restrict__ cell_count, int4 *__restrict__ cimg,
                              const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = sys_of[i];
  if (sys_skip(s, sreb, all)) return;
  const int cell = place_in_cell(sp[s], n, i, pos, cimg);
  cell_of[i] = cell;
  atomicAdd(cell_count + cell, 1);
}

// one block per system: cell_start[c0 ..] = a0 + exclusive scan of the
// system's cell counts; the counters are then reset for the fill
__global__ void __launch_bounds__(256) k_cell_scan(const SysP *__restrict__ sp, const int *__restrict__ sreb,
                                                   int all, int *__restrict__ cell_count,
                                                   int *__restrict__ cell_start, const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  const int s = blockIdx.x;
  if (sys_skip(s, sreb, all)) return;
  const int c0 = sp[s].c0, m = sp[s].ncells, a0 = sp[s].a0;
  __shared__ int part[256];
  const int t = threadIdx.x, nt = blockDim.x;
  const int chunk = (m + nt - 1) / nt;
  const int lo = t * chunk, hi = min(m, lo + chunk);
  int sum = 0;
  for (int k = lo; k < hi; k++) sum += cell_count[c0 + k];
  part[t] = sum;
  __syncthreads();
  for (int d = 1; d < nt; d <<= 1) {
    int v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int run = a0 + (t > 0 ? part[t - 1] : 0);
  for (int k = lo; k < hi; k++) {
    const int cnt = cell_count[c0 + k];
    cell_start[c0 + k] = run;
    cell_count[c0 + k] = 0;
    run += cnt;
  }
  if (t == nt - 1) cell_start[c0 + m] = a0 + part[nt - 1];
}

// exclusive scan of `m` ints in one block; `nseg` independent segments laid
// out back to back, one per blockIdx.y; segment totals go to tot[blockIdx.y]
template <typename TI, typename TO>
__global__ void k_scan(const TI *__restrict__ in, TO *__restrict__ out, long long *__restrict__ tot,
                       int m, const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  const TI *a = in + (size_t)blockIdx.y * m;
  TO *o = out + (size_t)blockIdx.y * (m + 1);
  __shared__ TO part[1024];
  int t = threadIdx.x, nt = blockDim.x;
  int chunk = (m + nt - 1) / nt;
  int lo = t * chunk, hi = min(m, lo + chunk);
  TO s = 0;
  for (int k = lo; k < hi; k++) s += (TO)a[k];
  part[t] = s;
  __syncthreads();
  for (int d = 1; d < nt; d <<= 1) {
    TO v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  TO run = t > 0 ? part[t - 1] : 0;
  for (int k = lo; k < hi; k++) {
    o[k] = run;
    run += (TO)a[k];
  }
  if (t == nt - 1) {
    o[m] = part[nt - 1];
    if (tot) tot[blockIdx.y] = (long long)part[nt - 1];
  }
}

__global__ void k_cell_fill(int n, const int *__restrict__ sys_of, const int *__restrict__ sreb, int all,
                            const int *__restrict__ cell_of, const int *__restrict__ cell_start,
                            int *__restrict__ cursor, int *__restrict__ cell_atoms, const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || sys_skip(sys_of[i], sreb, all)) return;
  int c = cell_of[i];
  int slot = atomicAdd(cursor + c, 1);
  cell_atoms[cell_start[c] + slot] = i;
}

// order every cell's atoms by (atom type, atom index): deterministic lists,
// and the atoms of one type are neighbours in sorted order, so the lane
// groups of a warp in the pair kernels mostly hold atoms of one type and
// walk lists of the same make-up.  One block per cell ranks each atom among
// its cell's atoms (keys are distinct).
__device__ __forceinline__ long long sort_key(const int *__restrict__ itype, int i) {
  return ((long long)itype[i] << 32) | (unsigned)i;
}

constexpr int SORT_CELLS = 8;      // most cells per block of k_cell_sort
constexpr int SORT_THREADS = 128;

__global__ void __launch_bounds__(SORT_THREADS) k_cell_sort(int ncells, int per_block, const int *__restrict__ cell_sys,
                                                             const int *__restrict__ sreb, int all,
                                                             const int *__restrict__ cell_start,
                                                             const int *__restrict__ itype,
                                                             int *__restrict__ cell_atoms,
                                                             const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  __shared__ long long s[1024];
  // per_block consecutive cells per block: up to SORT_CELLS where a batch has
  // tens of thousands of cells of a few atoms each, one where a grid of few,
  // crowded cells would otherwise leave most SMs idle
  const int c_end = min(ncells, (blockIdx.x + 1) * per_block);
  for (int c = blockIdx.x * per_block; c < c_end; c++) {
    if (sys_skip(cell_sys[c], sreb, all)) continue;     // whole blocks
    const int lo = cell_start[c], hi = cell_start[c + 1], m = hi - lo;
    if (m <= 1) continue;
    __syncthreads();                                     // the previous cell's keys are no longer read
    if (m <= 1024) {
      for (int k = threadIdx.x; k < m; k += blockDim.x) s[k] = sort_key(itype, cell_atoms[lo + k]);
      __syncthreads();
      for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const long long v = s[k];
        int r = 0;
        for (int u = 0; u < m; u++) r += s[u] < v;
        cell_atoms[lo + r] = (int)(v & 0xffffffffLL);
      }
      continue;
    }
    // a cell with more than 1024 atoms: odd-even transposition sort in place
    for (int pass = 0; pass < m; pass++) {
      for (int k = lo + (pass & 1) + 2 * threadIdx.x; k + 1 < hi; k += 2 * blockDim.x) {
        int a0 = cell_atoms[k], a1 = cell_atoms[k + 1];
        if (sort_key(itype, a0) > sort_key(itype, a1)) {
          cell_atoms[k] = a1;
          cell_atoms[k + 1] = a0;
        }
      }
      __syncthreads();
    }
  }
}

// What the sorted order holds of each atom: rank, type, the FP64 corner of the
// atom's cell (held fixed until the next rebuild) and FP32 cell-relative
// coordinates + charge.
struct Sorted {
  const int *itype;
  const double *pos, *q;
  int *rank, *styp;
  int2 *smeta;
  double *corner;
  float4 *xq;
};

// atom i, whose cell and image are ci, at sorted place t
__device__ __forceinline__ void sorted_place(const SysP &P, const Sorted &S, int n, int t, int i, int4 ci) {
  const double *h = P.h;
  double o0 = (double)ci.y + (double)(ci.x & 1023) / P.nc[0];
  double o1 = (double)ci.z + (double)((ci.x >> 10) & 1023) / P.nc[1];
  double o2 = (double)ci.w + (double)((ci.x >> 20) & 1023) / P.nc[2];
  double c0 = h[0] * o0 + h[1] * o1 + h[2] * o2;
  double c1 = h[3] * o0 + h[4] * o1 + h[5] * o2;
  double c2 = h[6] * o0 + h[7] * o1 + h[8] * o2;
  S.corner[t] = c0;
  S.corner[n + t] = c1;
  S.corner[2 * n + t] = c2;
  const double q = S.q[i];
  S.xq[t] = make_float4((float)(S.pos[i] - c0), (float)(S.pos[n + i] - c1), (float)(S.pos[2 * n + i] - c2), (float)q);
  S.rank[i] = t;
  S.styp[t] = S.itype[i];
  S.smeta[t] = make_int2(i, S.itype[i] * 2 + (q != 0.0 ? 1 : 0));
}

__global__ void k_sorted_init(int n, const SysP *__restrict__ sp, const int *__restrict__ sys_of,
                              const int *__restrict__ sreb, int all, const int *__restrict__ cell_atoms,
                              const int4 *__restrict__ cimg, const __grid_constant__ Sorted S,
                              const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int s = sys_of[t];
  if (sys_skip(s, sreb, all)) return;
  const int i = cell_atoms[t];
  sorted_place(sp[s], S, n, t, i, cimg[i]);
}

// The six binning kernels (k_cell_zero .. k_sorted_init) in one, a cluster of
// `nb` blocks per system with its barriers between the stages: same cells, same
// order.  For systems of up to BIN_ATOMS atoms, where the six are launches and
// little else -- on the steps that build nothing, too: they are replayed every
// step and each costs some 2 us to find that out (us per step, six kernels and
// one: 648 water atoms 70, 65; 2048 argon 72, 66; 2048 charged 86, 82; 37 boxes
// 183, 176; 12,288 water atoms 132, 128; 32,000 argon 89, 85; 8 boxes of 32,000
// 558, 550; 100 of 3000 water atoms 2991, 2931; 31,944 water atoms 411, 411.
// The FP64 engine, whose builds are as frequent as CM3D's: 32,000 argon atoms
// 89, 84; 1536 water atoms 157, 155; 5184, 283, 281; but 12,288, 496, 500;
// 24,000, 875, 885).
//
// A stage reads what other blocks wrote before the barrier; nothing read
// earlier in the kernel is read again after another block's write, except the
// counters, which go through L2.
constexpr int BIN_THREADS = 1024, BIN_CLUSTER = 8, BIN_ATOMS = 4 * BIN_CLUSTER * BIN_THREADS;
constexpr double BIN_PLAIN_PAIRS = 1e6;     // FP64 engine: most atoms x atoms per cell
__global__ void __launch_bounds__(BIN_THREADS, 1) k_bin(
    int n, int nb, const SysP *__restrict__ sp, const int *__restrict__ sreb, int all, const __grid_constant__ Sorted S,
    int4 *cimg, int *cell_of, int *count, int *cell_start, long long *keys, int *cell_atoms,
    const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  const int s = blockIdx.x / nb, rank = blockIdx.x - s * nb;
  if (sys_skip(s, sreb, all)) return;                     // whole clusters
  const SysP &P = sp[s];
  const int m = P.ncells, c0 = P.c0, a0 = P.a0, a1 = P.a0 + P.n;
  const int t0 = rank * BIN_THREADS + threadIdx.x, nt = nb * BIN_THREADS;
  for (int k = t0; k < m; k += nt) count[c0 + k] = 0;
  cluster_sync(nb);
  for (int i = a0 + t0; i < a1; i += nt) {
    const int cell = place_in_cell(P, n, i, S.pos, cimg);
    cell_of[i] = cell;
    atomicAdd(count + cell, 1);
  }
  cluster_sync(nb);
  if (rank == 0) {
    // cell_start: exclusive scan of the counts, `chunk` cells per thread
    __shared__ int part[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int chunk = (m + BIN_THREADS - 1) / BIN_THREADS;
    const int lo = min(m, t * chunk), hi = min(m, lo + chunk);
    int sum = 0;
    for (int k = lo; k < hi; k++) sum += __ldcg(count + c0 + k);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) part[w] = incl;
    __syncthreads();
    if (w == 0) {
      int v = part[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      part[lane] = v;
    }
    __syncthreads();
    int run = a0 + incl - sum + (w > 0 ? part[w - 1] : 0);
    for (int k = lo; k < hi; k++) {
      const int cnt = __ldcg(count + c0 + k);
      cell_start[c0 + k] = run;
      count[c0 + k] = 0;
      run += cnt;
    }
    if (t == BIN_THREADS - 1) cell_start[c0 + m] = a1;
  }
  cluster_sync(nb);
  for (int i = a0 + t0; i < a1; i += nt) {
    const int cell = cell_of[i];                          // this thread's own
    keys[cell_start[cell] + atomicAdd(count + cell, 1)] = sort_key(S.itype, i);
  }
  cluster_sync(nb);
  // k_cell_sort's order: each atom's place is the number of smaller keys in
  // its cell (neighbouring threads share the cell and read the same key)
  for (int u = a0 + t0; u < a1; u += nt) {
    const long long key = keys[u];
    const int i = (int)(key & 0xffffffffLL);
    const int cell = __ldcg(cell_of + i);
    const int lo = cell_start[cell], hi = cell_start[cell + 1];
    int r = 0;
#pragma unroll 4
    for (int v = lo; v < hi; v++) r += keys[v] < key;
    cell_atoms[lo + r] = i;
    sorted_place(P, S, n, lo + r, i, __ldcg(cimg + i));
  }
}

// What the list kernels read: atoms, cells, parameters and exclusions.
struct ListK {
  int n;
  const int *cell_atoms, *cell_start, *cell_of;
  const float4 *xq;
  const double *pos;
  const int *itype, *map;
  const double *rad, *q;               // list radii^2 of the lists being built, {s, l} per interaction
  int own;                             // the engine's own lists (otherwise CM3D's half lists)
  const int *excl_off, *excl_idx, *cexcl_off, *cexcl_idx;
  const int4 *cimg;
  const int2 *smeta, *xspan;
};

// Exact membership test of one candidate pair, in CM3D's FP64 operation
// order.  Returns the pair's full-list entry without j: its list flags
// (ENT_LJ t, ENT_LJS s, ENT_EL te, ENT_ELS se), near-image bit and cell-shift
// code, and EXACT_BAD where the code does not exist; 0 for a pair in no list.
constexpr uint32_t EXACT_BAD = 1u;
constexpr uint32_t ENT_FLAGS = ENT_LJ | ENT_EL | ENT_LJS | ENT_ELS;
__device__ __forceinline__ uint32_t exact_test(const SysP &P, const ListK &K, int i, int j) {
  const int n = K.n;
  const double *__restrict__ pos = K.pos;
  const int ti = K.itype[i];
  const int4 ci = K.cimg[i];
  const bool qi = K.q[i] != 0.0;
  const double xi = pos[i], yi = pos[n + i], zi = pos[2 * n + i];
  const double rl_e = K.own ? P.rmaxl_list2_e : P.rmaxl_skin2_e, rs_e = K.own ? P.rmaxs_list2_e : P.rmaxs_skin2_e;
  const int intr = K.map[P.map0 + ti * P.ntypes + K.itype[j]];
  const bool lj_ok = intr >= 0;
  const bool el_ok = qi && K.q[j] != 0.0;
  if (!lj_ok && !el_ok) return 0;
  double dx = xi - pos[j], dy = yi - pos[n + j], dz = zi - pos[2 * n + j];
  double sx = __dadd_rn(__dadd_rn(__dmul_rn(dx, P.hi[0]), __dmul_rn(dy, P.hi[1])), __dmul_rn(dz, P.hi[2]));
  double sy = __dadd_rn(__dadd_rn(__dmul_rn(dx, P.hi[3]), __dmul_rn(dy, P.hi[4])), __dmul_rn(dz, P.hi[5]));
  double sz = __dadd_rn(__dadd_rn(__dmul_rn(dx, P.hi[6]), __dmul_rn(dy, P.hi[7])), __dmul_rn(dz, P.hi[8]));
  const double mx = anint_ref(sx), my = anint_ref(sy), mz = anint_ref(sz);
  sx = __dsub_rn(sx, mx);
  sy = __dsub_rn(sy, my);
  sz = __dsub_rn(sz, mz);
  const double ex = __dadd_rn(__dadd_rn(__dmul_rn(sx, P.h[0]), __dmul_rn(sy, P.h[1])), __dmul_rn(sz, P.h[2]));
  const double ey = __dadd_rn(__dadd_rn(__dmul_rn(sx, P.h[3]), __dmul_rn(sy, P.h[4])), __dmul_rn(sz, P.h[5]));
  const double ez = __dadd_rn(__dadd_rn(__dmul_rn(sx, P.h[6]), __dmul_rn(sy, P.h[7])), __dmul_rn(sz, P.h[8]));
  const double r2 = r2_ref(ex, ey, ez);
  uint32_t en = 0;
  if (lj_ok && r2 < K.rad[2 * intr + 1] && !(P.excl && excluded(i, j, K.excl_off, K.excl_idx))) {
    en |= ENT_LJ;
    if (r2 < K.rad[2 * intr]) en |= ENT_LJS;
  }
  if (el_ok && r2 < rl_e && !(P.cexcl && excluded(i, j, K.cexcl_off, K.cexcl_idx))) {
    en |= ENT_EL;
    if (r2 < rs_e) en |= ENT_ELS;
  }
  if (!en) return 0;
  // small boxes: the atoms may move skin/2 each before the next rebuild, so a
  // pair whose fractional displacement is within skin / plane spacing of 1/2
  // may change its nearest image; the pair kernel checks those pairs
  if (P.smallbox && (fabs(sx) > P.near_s[0] || fabs(sy) > P.near_s[1] || fabs(sz) > P.near_s[2])) en |= ENT_NEAR;
  // shift code: k = (n_i - n_j - m) nc + (c_i - c_j) per dimension; |k| <= 1
  // whenever r < rlist <= cell width.  Anything else means the geometry
  // assumption broke: flag it and use the zero shift rather than index past
  // the shift table.
  const int4 cj = K.cimg[j];
  const int kx = (ci.y - cj.y - (int)mx) * P.nc[0] + ((ci.x & 1023) - (cj.x & 1023));
  const int ky = (ci.z - cj.z - (int)my) * P.nc[1] + (((ci.x >> 10) & 1023) - ((cj.x >> 10) & 1023));
  const int kz = (ci.w - cj.w - (int)mz) * P.nc[2] + (((ci.x >> 20) & 1023) - ((cj.x >> 20) & 1023));
  if (kx < -1 || kx > 1 || ky < -1 || ky > 1 || kz < -1 || kz > 1) return en | 13u << ENT_CODE_SHIFT | EXACT_BAD;
  return en | (uint32_t)((kx + 1) * 9 + (ky + 1) * 3 + (kz + 1)) << ENT_CODE_SHIFT;
}
// Not inlined in the full-list kernels: the few pairs that FP32 cannot decide
// would otherwise cost them their registers.
__device__ __noinline__ uint32_t exact_entry(const SysP &P, const ListK &K, int i, int j) {
  return exact_test(P, K, i, j);
}

// The candidate walk shared by both list kernels.  One warp owns the
// cell-sorted atom t; its lanes walk the stencil cells 32 candidates at a
// time (consecutive sorted atoms: coalesced FP32 loads) and drop those
// clearly beyond the largest list radius with an FP32 distance from
// cell-relative coordinates (margin 1e-3 A, far above FP32 rounding).  The
// survivors -- typically a few of every 32 -- are queued in shared memory in
// candidate order, and whenever 32 are waiting the whole warp runs the exact
// FP64 test on them at once (`decide(first, m)`: lane l < m takes queue entry
// first + l), so the expensive test runs on full warps.
//
// The queue keeps each survivor's FP32 squared distance (qr) beside its index
// and the code of its cell shift (bits ENT_CODE_SHIFT and up), for the
// FP32-first flags (list_flags).  In a grid of 3 or more cells per axis
// (G_STENCIL) the stencil image is the only image in range and its code the
// pair's; with `prune` (such a grid in an orthorhombic box, cells cw wide)
// stencil cells wholly beyond lim2 from the atom, by the gaps to their faces
// less 1e-3 A, are skipped -- none of their atoms would pass the prefilter, so
// the lists are the same.  In a coarser grid (G_IMAGE) the minimum image is
// taken in FP32 (fold), which also gives the code; a pair whose fractional
// displacement lies so close to 1/2 (or to a small box's near-image bound)
// that FP32 may choose another image than CM3D's FP64 arithmetic carries
// CODE_EXACT instead, and is decided in FP64.  G_EXACT takes no FP32 decision.
constexpr int LQ = 64;                     // queue entries per warp (> 2 * 32 - 1)
constexpr int CODE_EXACT = 31;             // queue code: the FP64 test decides
constexpr int QUEUE_NEAR = (int)ENT_NEAR;  // queue bit: ENT_NEAR of a small box
enum { G_EXACT = 0, G_STENCIL = 1, G_IMAGE = 2 };

__host__ __device__ __forceinline__ int grid_kind(const SysP &P) {
  if (P.nc[0] >= 3 && P.nc[1] >= 3 && P.nc[2] >= 3) return P.smallbox ? G_EXACT : G_STENCIL;
  return P.image_ok ? G_IMAGE : G_EXACT;
}

// Minimum image of the FP32 displacement (dx, dy, dz) to an atom of the
// stencil cell of shift code `code`: period()'s fold in FP32.  Returns the
// squared distance and leaves the image's shift code (CODE_EXACT where FP32
// cannot tell, see above) and near-image bit in `code`.  The displacement is
// a difference of coordinates no larger than a box of at most 8 list radii
// per axis, so s carries an error of about 1e-7; 1e-5 is the margin.  In a
// sheared box the two images of a pair half a box apart are not equally long,
// and the other one may be within a list radius where this one is not: such a
// pair returns 0 and so gets to its FP64 test.
__device__ __forceinline__ float fold(const SysP &P, float dx, float dy, float dz, int &code) {
  const float sx = P.hiF[0] * dx + P.hiF[1] * dy + P.hiF[2] * dz;
  const float sy = P.hiF[3] * dx + P.hiF[4] * dy + P.hiF[5] * dz;
  const float sz = P.hiF[6] * dx + P.hiF[7] * dy + P.hiF[8] * dz;
  const float mx = rintf(sx), my = rintf(sy), mz = rintf(sz);
  dx -= P.hF[0] * mx + P.hF[1] * my + P.hF[2] * mz;
  dy -= P.hF[3] * mx + P.hF[4] * my + P.hF[5] * mz;
  dz -= P.hF[6] * mx + P.hF[7] * my + P.hF[8] * mz;
  const float ax = fabsf(sx - mx), ay = fabsf(sy - my), az = fabsf(sz - mz);
  constexpr float EPS = 1e-5f;
  const bool half = ax > 0.5f - EPS || ay > 0.5f - EPS || az > 0.5f - EPS;
  bool exact = half;
  int near = 0;
  if (P.smallbox) {
    const float nx = (float)P.near_s[0], ny = (float)P.near_s[1], nz = (float)P.near_s[2];
    exact |= fabsf(ax - nx) < EPS || fabsf(ay - ny) < EPS || fabsf(az - nz) < EPS;
    if (ax > nx || ay > ny || az > nz) near = QUEUE_NEAR;
  }
  const int kx = code / 9 - 1 - (int)mx * P.nc[0], ky = (code / 3) % 3 - 1 - (int)my * P.nc[1],
            kz = code % 3 - 1 - (int)mz * P.nc[2];
  exact |= kx < -1 || kx > 1 || ky < -1 || ky > 1 || kz < -1 || kz > 1;
  code = exact ? CODE_EXACT << ENT_CODE_SHIFT : ((kx + 1) * 9 + (ky + 1) * 3 + (kz + 1)) << ENT_CODE_SHIFT | near;
  return half && P.sheared ? 0.f : fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

template <class Decide>
__device__ __forceinline__ void walk_candidates(const SysP &P, const ListK &K, int i, bool half_only, int *qbuf,
                                                float *qr, Decide &decide, int kind, bool prune, float3 cw, int t) {
  const int *__restrict__ cell_start = K.cell_start;
  const float4 *__restrict__ xq = K.xq;
  const int4 ci = K.cimg[i];
  const float4 xi4 = xq[t];
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int cx = ci.x & 1023, cy = (ci.x >> 10) & 1023, cz = (ci.x >> 20) & 1023;
  const float lim2 = kind == G_IMAGE ? P.lim2_image : P.lim2;
  // the stencil cells in walk order (x offsets outermost), one per lane:
  // their sorted-atom ranges (empty where pruned) and shift codes, loaded
  // together up front
  const int nw = P.nsx * P.nsy * P.nsz;
  int my_lo = 0, my_hi = 0, my_code = 13;
  if (lane < nw) {
    const int ox = P.sx[lane / (P.nsy * P.nsz)], oy = P.sy[(lane / P.nsz) % P.nsy], oz = P.sz[lane % P.nsz];
    bool vis = true;
    if (prune) {
      const float gx = fmaxf((ox > 0 ? cw.x - xi4.x : ox < 0 ? xi4.x : 0.f) - 1e-3f, 0.f);
      const float gy = fmaxf((oy > 0 ? cw.y - xi4.y : oy < 0 ? xi4.y : 0.f) - 1e-3f, 0.f);
      const float gz = fmaxf((oz > 0 ? cw.z - xi4.z : oz < 0 ? xi4.z : 0.f) - 1e-3f, 0.f);
      vis = gx * gx + gy * gy + gz * gz < lim2;
    }
    int jx = cx + ox, jy = cy + oy, jz = cz + oz;
    jx = jx < 0 ? jx + P.nc[0] : (jx >= P.nc[0] ? jx - P.nc[0] : jx);
    jy = jy < 0 ? jy + P.nc[1] : (jy >= P.nc[1] ? jy - P.nc[1] : jy);
    jz = jz < 0 ? jz + P.nc[2] : (jz >= P.nc[2] ? jz - P.nc[2] : jz);
    const int cell = P.c0 + (jx * P.nc[1] + jy) * P.nc[2] + jz;
    // cell-corner shift of this stencil offset (k = -offset)
    my_code = (1 - ox) * 9 + (1 - oy) * 3 + (1 - oz);
    if (vis) {
      my_lo = cell_start[cell];
      my_hi = cell_start[cell + 1];
    }
  }
  unsigned left = __ballot_sync(0xffffffffu, my_hi > my_lo);
  // the chunks of 32 candidates in walk order; the next chunk's positions
  // are loaded while the current one is tested
  int w = left ? __ffs(left) - 1 : -1;
  int u0 = 0, hi = 0, code = 13;
  float4 S = make_float4(0.f, 0.f, 0.f, 0.f), xn = S;
  if (w >= 0) {
    u0 = __shfl_sync(0xffffffffu, my_lo, w);
    hi = __shfl_sync(0xffffffffu, my_hi, w);
    code = __shfl_sync(0xffffffffu, my_code, w);
    S = P.shift[code];
    if (u0 + lane < hi) xn = xq[u0 + lane];
  }
  int head = 0, tail = 0;
  while (w >= 0) {
    const int u = u0 + lane, hcur = hi, ccur = code;
    const float4 Sc = S, xj = xn;
    u0 += 32;
    if (u0 >= hi) {
      left &= ~(1u << w);
      w = left ? __ffs(left) - 1 : -1;
      if (w >= 0) {
        u0 = __shfl_sync(0xffffffffu, my_lo, w);
        hi = __shfl_sync(0xffffffffu, my_hi, w);
        code = __shfl_sync(0xffffffffu, my_code, w);
        S = P.shift[code];
      }
    }
    if (w >= 0 && u0 + lane < hi) xn = xq[u0 + lane];
    bool keep = false;
    float r2f = 0.f;
    int qc = ccur << ENT_CODE_SHIFT;
    if (u < hcur) {
      const float dx = (xi4.x - xj.x) + Sc.x, dy = (xi4.y - xj.y) + Sc.y, dz = (xi4.z - xj.z) + Sc.z;
      if (kind == G_IMAGE) {
        qc = ccur;
        r2f = fold(P, dx, dy, dz, qc);
      } else {
        r2f = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        if (kind == G_EXACT) qc = CODE_EXACT << ENT_CODE_SHIFT;
      }
      // the atom itself; half lists: j > i
      keep = r2f < lim2 && (half_only ? K.cell_atoms[u] > i : u != t);
    }
    const unsigned bk = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int slot = (tail + __popc(bk & lt_mask)) & (LQ - 1);
      // half lists need no code, only whether FP32 may decide (the plain
      // engine's sorted indices can need more than ENT_JBITS bits)
      qbuf[slot] = half_only ? u : u | qc;
      qr[slot] = half_only && ((qc >> ENT_CODE_SHIFT) & 31) == CODE_EXACT ? -1.f : r2f;
    }
    tail += __popc(bk);
    __syncwarp();
    if (tail - head >= 32) {
      decide(head, 32);
      head += 32;
      __syncwarp();
    }
  }
  while (tail > head) {
    const int m = tail - head < 32 ? tail - head : 32;
    decide(head, m);
    head += m;
  }
}

// What an atom's list flags need of the atom itself, loaded once per warp:
// its types' list radii (lane tj: the LJ radii of the interaction with type
// tj, FP32, -1 for none; read by shuffle -- no table load per pair), its
// charge's, and the span of the atom indices excluded from it (a pair outside
// it needs no look-up of the exclusion lists).
struct ListAtom {
  int ti;
  bool rows;                               // the types fit the lanes
  float rl, rs;                            // lane tj: LJ list radii^2 (t, s)
  float el, es;                            // electrostatic list radii^2 (te, se), -1 without charge
  float near;                              // FP32 decides beyond this distance from every radius^2
  int xlo;
  unsigned xw;                             // excluded from it: atoms among xlo .. xlo + xw
};

__device__ __forceinline__ ListAtom list_atom(const SysP &P, const ListK &K, int2 meta) {
  const int lane = threadIdx.x & 31;
  ListAtom A;
  A.ti = meta.y >> 1;
  A.rows = P.ntypes <= 32;
  A.rl = A.rs = A.el = A.es = -1.f;
  if (A.rows && lane < P.ntypes) {
    const int intr = K.map[P.map0 + A.ti * P.ntypes + lane];
    if (intr >= 0) {
      A.rl = (float)K.rad[2 * intr + 1];
      A.rs = (float)K.rad[2 * intr];
    }
  }
  if (meta.y & 1) {
    A.el = (float)(K.own ? P.rmaxl_list2_e : P.rmaxl_skin2_e);
    A.es = (float)(K.own ? P.rmaxs_list2_e : P.rmaxs_skin2_e);
  }
  A.near = fmaf(4e-5f, P.lim2_image, 2e-3f);
  const int2 x = K.xspan[meta.x];
  A.xlo = x.x;
  A.xw = (unsigned)x.y;
  return A;
}

// r2f against the LJ and electrostatic list radii^2 (-1: no such list);
// *near: within `margin` of one of them
__device__ __forceinline__ uint32_t radii_flags(float r2f, float rl, float rs, float el, float es, float margin,
                                                bool *near) {
  *near = fminf(fminf(fabsf(r2f - rl), fabsf(r2f - rs)), fminf(fabsf(r2f - el), fabsf(r2f - es))) < margin;
  uint32_t fl = r2f < rl ? (r2f < rs ? ENT_LJ | ENT_LJS : ENT_LJ) : 0u;
  if (r2f < el) fl |= r2f < es ? ENT_EL | ENT_ELS : ENT_EL;
  return fl;
}

__device__ __forceinline__ uint32_t strike_excluded(const SysP &P, const ListK &K, uint32_t fl, int i, int j) {
  if (P.excl && excluded(i, j, K.excl_off, K.excl_idx)) fl &= ~(ENT_LJ | ENT_LJS);
  if (P.cexcl && excluded(i, j, K.cexcl_off, K.cexcl_idx)) fl &= ~(ENT_EL | ENT_ELS);
  return fl;
}

// List flags (ENT_*) of a pair from its FP32 squared distance: the tests of
// exact_entry.  Each comparison with a list radius R^2 matches CM3D's FP64 one
// unless the FP32 value lies within 4e-5 R^2 + 2e-3 A^2 of R^2 -- a margin ten
// times the FP32 error of a squared distance formed from cell-relative
// coordinates (cells are narrower than two list radii); the largest R^2 of
// the system gives the margin for all of them -- and then *exact is set and
// the caller decides in FP64 (exact_entry).  Called by the whole warp (the
// radii come by shuffle); `on`: this lane has a pair.
__device__ __forceinline__ uint32_t list_flags(const SysP &P, const ListK &K, const ListAtom &A, bool on, int i,
                                               int2 mj, float r2f, bool *exact) {
  const int j = mj.x, tj = mj.y >> 1;
  float rl, rs;
  if (A.rows) {
    rl = __shfl_sync(0xffffffffu, A.rl, tj & 31);
    rs = __shfl_sync(0xffffffffu, A.rs, tj & 31);
  } else {
    rl = rs = -1.f;
    const int intr = on ? K.map[P.map0 + A.ti * P.ntypes + tj] : -1;
    if (intr >= 0) {
      rl = (float)K.rad[2 * intr + 1];
      rs = (float)K.rad[2 * intr];
    }
  }
  const bool qj = (mj.y & 1) != 0;
  bool near;
  uint32_t fl = radii_flags(r2f, rl, rs, qj ? A.el : -1.f, qj ? A.es : -1.f, A.near, &near);
  *exact = on && near;
  if (!on) fl = 0u;
  if (fl && (unsigned)(j - A.xlo) <= A.xw) fl = strike_excluded(P, K, fl, i, j);
  return fl;
}

// Appends a warp's entries to an atom's slot (na, nb: its segments so far):
// the pairs in an LJ list from the front, the electrostatics-only ones from
// the back.  Every write lands inside the slot; once the two segments meet (an
// overflow) the slot's contents no longer matter: the lengths are set to zero
// at the end and the list is built again with wider slots.
__device__ __forceinline__ void append(uint32_t *__restrict__ out, int stride, uint32_t en, int &na, int &nb) {
  const unsigned lt_mask = (1u << (threadIdx.x & 31)) - 1u;
  const bool fa = (en & (ENT_LJ | ENT_LJS)) != 0, any = (en & ENT_FLAGS) != 0;
  const unsigned ba = __ballot_sync(0xffffffffu, fa), bb = __ballot_sync(0xffffffffu, any && !fa);
  const int at = fa ? na + __popc(ba & lt_mask) : stride - 1 - (nb + __popc(bb & lt_mask));
  if (any && (fa ? at < stride - nb : at >= na)) out[at] = en;
  na += __popc(ba);
  nb += __popc(bb);
}

__host__ __device__ __forceinline__ bool ortho(const SysP &P) {
  return P.h[1] == 0. && P.h[2] == 0. && P.h[3] == 0. && P.h[5] == 0. && P.h[6] == 0. && P.h[7] == 0.;
}
// edges of an orthorhombic box's cells
__device__ __forceinline__ float3 cell_width(const SysP &P) {
  return make_float3(P.hF[0] / (float)P.nc[0], P.hF[4] / (float)P.nc[1], P.hF[8] / (float)P.nc[2]);
}

struct ListCaps {
  long long cap[4];
};

// CM3D's four half lists (i < j): FILL = false counts the pairs of every
// list per atom, FILL = true writes them at the scanned offsets, compacted
// with warp ballots in candidate order (deterministic).  Always built for
// every system (host-driven builds and the single-system plain engine).
// Bound by the latency of the candidates' loads, hence by the warps that the
// registers leave.  STENCIL, every system's grid of three and more cells per
// axis: the FP64 test is in line and three blocks fit an SM, where a call of it
// takes 98 registers and leaves two; stencil cells wholly out of reach are
// skipped.  (us per FP64 step of 5184, 12,288 and 24,000 water atoms: called
// 354, 671, 1274; in line 314, 577, 1057; and with the cells skipped 275, 484,
// 848.)  In coarser grids, whose few atoms do not fill the SMs, the registers
// are worth more than the warps (1536 atoms 152; bounded to three blocks, 156).
template <bool FILL, bool STENCIL>
__global__ void __launch_bounds__(256, STENCIL ? 3 : 2) k_list_half(
    const __grid_constant__ ListK K, const SysP *__restrict__ sp, const int *__restrict__ sys_of, ListCaps C,
    int *__restrict__ cnt, const long long *__restrict__ off,
    const long long *__restrict__ tot, int2 *__restrict__ l0, int2 *__restrict__ l1, int2 *__restrict__ l2,
    int2 *__restrict__ l3, long long *__restrict__ stat, int *__restrict__ halt, const int *__restrict__ gate) {
  if (block_gated_off(gate, 1)) return;
  __shared__ int qs[256 / 32][LQ];
  __shared__ float qrs[256 / 32][LQ];
  const int n = K.n;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= n) return;                                     // whole warps
  const unsigned lt_mask = (1u << lane) - 1u;
  long long p[4] = {0, 0, 0, 0};
  if (FILL) {
    bool fits = true;
    for (int k = 0; k < 4; k++) {
      fits = fits && tot[k] <= C.cap[k];
      p[k] = off[(size_t)k * (n + 1) + t];
    }
    if (!fits) {
      // a list outgrew its buffer: write nothing, halt the step (the host
      // grows the buffers and finishes it, see run_step)
      if (t == 0 && lane == 0) {
        atomicAdd((unsigned long long *)(stat + ST_OVERFLOW), 1ull);
        if (halt) *halt = 1;
      }
      return;
    }
  }
  int *qbuf = qs[threadIdx.x >> 5];
  float *qr = qrs[threadIdx.x >> 5];
  const SysP &P = sp[sys_of[t]];
  const int2 mi = K.smeta[t];
  const int i = mi.x;
  const ListAtom A = list_atom(P, K, mi);
  int c[4] = {0, 0, 0, 0};
  unsigned bad = 0;
  auto decide = [&](int first, int m) {
    const bool on = lane < m;
    const int slot = (first + lane) & (LQ - 1);
    const int2 mj = on ? K.smeta[qbuf[slot]] : make_int2(-1, 0);
    const float r2f = qr[slot];
    const int j = mj.x;
    const bool exact = !STENCIL && r2f < 0.f;
    bool near;
    uint32_t fl = list_flags(P, K, A, on && !exact, i, mj, r2f, &near);
    if (on && (exact || near)) fl = STENCIL ? exact_test(P, K, i, j) : exact_entry(P, K, i, j);
    bad |= fl & EXACT_BAD;
    const unsigned b0 = __ballot_sync(0xffffffffu, fl & ENT_LJ), b1 = __ballot_sync(0xffffffffu, fl & ENT_LJS);
    const unsigned b2 = __ballot_sync(0xffffffffu, fl & ENT_EL), b3 = __ballot_sync(0xffffffffu, fl & ENT_ELS);
    if (!FILL) {
      c[0] += __popc(b0); c[1] += __popc(b1); c[2] += __popc(b2); c[3] += __popc(b3);
    } else {
      const int2 pr = make_int2(i, j);
      if (fl & ENT_LJ) l0[p[0] + __popc(b0 & lt_mask)] = pr;
      if (fl & ENT_LJS) l1[p[1] + __popc(b1 & lt_mask)] = pr;
      if (fl & ENT_EL) l2[p[2] + __popc(b2 & lt_mask)] = pr;
      if (fl & ENT_ELS) l3[p[3] + __popc(b3 & lt_mask)] = pr;
      p[0] += __popc(b0); p[1] += __popc(b1); p[2] += __popc(b2); p[3] += __popc(b3);
    }
  };
  walk_candidates(P, K, i, true, qbuf, qr, decide, STENCIL ? G_STENCIL : grid_kind(P), STENCIL && ortho(P),
                  cell_width(P), t);
  if (FILL) {
    if (bad && lane == 0) atomicAdd((unsigned long long *)(stat + ST_BADSHIFT), 1ull);
  } else if (lane == 0) {
    for (int k = 0; k < 4; k++) cnt[(size_t)k * n + t] = c[k];
  }
}

// Candidates from a staged neighbourhood (k_list_win): `cnt` atoms with FP32
// positions moved by their cell's shift into the frame of atom t's cell
// (s_x) and their sorted indices (s_u, low ENT_JBITS bits), walked 32 at a
// time with the same prefilter and in the same order as walk_candidates.  The
// queue holds the staged index and the code, qr the FP32 squared distance.
//
// With `prune` (an orthorhombic cell grid of three or more cells per axis,
// cells cw wide), the lanes first bound atom t's distance from each stencil
// cell (the gaps to the cell's faces, each shortened by 1e-3 A) and the walk
// skips the cells that lie wholly beyond lim2: none of their atoms would pass
// the prefilter, and the others keep their order, so the lists are the same.
// s_off holds the stencil cells' first staged index, s_code their shift code.
template <class Decide>
__device__ __forceinline__ void walk_staged(const SysP &P, int t, float4 xi4, const float4 *s_x, const int *s_u,
                                            int cnt, int *qbuf, float *qr, Decide &decide, const int *s_off,
                                            const int *s_code, int nw, int kind, bool prune, float3 cw) {
  const int lane = threadIdx.x & 31;
  const float lim2 = kind == G_IMAGE ? P.lim2_image : P.lim2;
  const unsigned lt_mask = (1u << lane) - 1u;
  unsigned vis = nw >= 32 ? 0xffffffffu : (1u << nw) - 1u;
  if (prune) {
    bool v = false;
    if (lane < nw) {
      const int code = s_code[lane];
      const int ox = 1 - code / 9, oy = 1 - (code / 3) % 3, oz = 1 - code % 3;
      const float gx = fmaxf((ox > 0 ? cw.x - xi4.x : ox < 0 ? xi4.x : 0.f) - 1e-3f, 0.f);
      const float gy = fmaxf((oy > 0 ? cw.y - xi4.y : oy < 0 ? xi4.y : 0.f) - 1e-3f, 0.f);
      const float gz = fmaxf((oz > 0 ? cw.z - xi4.z : oz < 0 ? xi4.z : 0.f) - 1e-3f, 0.f);
      v = gx * gx + gy * gy + gz * gz < lim2;
    }
    vis = __ballot_sync(0xffffffffu, v);
  }
  int head = 0, tail = 0;
  for (int w = 0; w < nw;) {
    if (!((vis >> w) & 1u)) {
      w++;
      continue;
    }
    // a run of visited stencil cells is one contiguous span of staged atoms
    int e = w;
    while (e + 1 < nw && ((vis >> (e + 1)) & 1u)) e++;
    const int a = s_off[w], b = e + 1 < nw ? s_off[e + 1] : cnt;
    w = e + 1;
  for (int k0 = a; k0 < b; k0 += 32) {
    const int k = k0 + lane;
    bool keep = false;
    float r2f = 0.f;
    int qc = 0;
    if (k < b) {
      const float4 xs = s_x[k];
      const unsigned uc = (unsigned)s_u[k];
      const int u = (int)(uc & ENT_JMASK);
      const float dx = xi4.x - xs.x, dy = xi4.y - xs.y, dz = xi4.z - xs.z;
      if (kind == G_IMAGE) {
        qc = (int)(uc >> ENT_CODE_SHIFT);
        r2f = fold(P, dx, dy, dz, qc);
      } else {
        r2f = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        qc = kind == G_EXACT ? CODE_EXACT << ENT_CODE_SHIFT : (int)(uc & ~ENT_JMASK);
      }
      keep = u != t && r2f < lim2;
    }
    const unsigned bk = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int slot = (tail + __popc(bk & lt_mask)) & (LQ - 1);
      qbuf[slot] = k | qc;
      qr[slot] = r2f;
    }
    tail += __popc(bk);
    __syncwarp();
    if (tail - head >= 32) {
      decide(head, 32);
      head += 32;
      __syncwarp();
    }
  }
  }
  while (tail > head) {
    const int m = tail - head < 32 ? tail - head : 32;
    decide(head, m);
    head += m;
  }
}

// The full list of sorted atom t (mixed mode; one warp): both directions,
// every pair in CM3D's t or te list, written straight into its fixed slot
// nbr[t * stride ...] in two segments, each in candidate order: the pairs in
// an LJ list (t or s) from the front of the slot, their count in nlen[t], and
// the electrostatics-only pairs from the back (the last one at the slot's
// end), their count in nlen[n + t].  A pair kernel then runs the LJ arithmetic
// only over the front segment.  An atom with more than `stride` pairs writes
// none past its slot, records the length it needed (ST_NEED_STRIDE) and halts
// a captured step; the host then widens the slots and builds again.
// STAGED: candidates from the block's staged neighbourhood (s_x, s_u, scnt),
// otherwise from global memory through the stencil walk.
template <bool STAGED>
__device__ __forceinline__ void full_list_atom(
    const SysP &P, const ListK &K, int t, int stride, uint32_t *__restrict__ nbr, int *__restrict__ nlen,
    long long *__restrict__ stat, int *__restrict__ halt,
    int *qbuf, float *qr, int kind, bool prune, float3 cw, const float4 *s_x = nullptr, const int *s_u = nullptr,
    const int *s_j = nullptr, int scnt = 0, const int *s_off = nullptr, const int *s_code = nullptr, int nw = 0) {
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int n = K.n;
  const int2 mi = K.smeta[t];
  const int i = mi.x;
  const ListAtom A = list_atom(P, K, mi);
  uint32_t *out = nbr + (size_t)t * stride;
  int na = 0, nb = 0;
  unsigned bad = 0;
  auto decide = [&](int first, int m) {
    const bool on = lane < m;
    const int slot = (first + lane) & (LQ - 1);
    const int e = on ? qbuf[slot] : CODE_EXACT << ENT_CODE_SHIFT;
    int u = e & (int)ENT_JMASK;
    const int code = (e >> ENT_CODE_SHIFT) & 31;
    int2 mj = make_int2(-1, 0);
    if (on) {
      if (STAGED) {
        mj = make_int2(s_j[u], __float_as_int(s_x[u].w));
        u = s_u[u] & (int)ENT_JMASK;
      } else {
        mj = K.smeta[u];
      }
    }
    bool near;
    uint32_t en = list_flags(P, K, A, on && code != CODE_EXACT, i, mj, qr[slot], &near);
    if (en) en |= (uint32_t)code << ENT_CODE_SHIFT | (uint32_t)(e & QUEUE_NEAR);
    if (on && (near || code == CODE_EXACT)) en = exact_entry(P, K, i, mj.x);
    bad |= en & EXACT_BAD;
    append(out, stride, (en & ~EXACT_BAD) | (uint32_t)u, na, nb);
  };
  if (STAGED) walk_staged(P, t, K.xq[t], s_x, s_u, scnt, qbuf, qr, decide, s_off, s_code, nw, kind, prune, cw);
  else walk_candidates(P, K, i, false, qbuf, qr, decide, kind, prune, cw, t);
  const int count = na + nb;
  if (lane == 0) {
    if (count <= stride) {
      nlen[t] = na;
      nlen[n + t] = nb;
    } else {
      nlen[t] = 0;
      nlen[n + t] = 0;
    }
    if (count > stride) {
      atomicMax((unsigned long long *)(stat + ST_NEED_STRIDE), (unsigned long long)count);
      if (halt) {
        atomicAdd((unsigned long long *)(stat + ST_OVERFLOW), 1ull);
        *halt = 1;
      }
    }
    if (bad) atomicAdd((unsigned long long *)(stat + ST_BADSHIFT), 1ull);
  }
}

// Mixed mode, warp per atom over every atom, the candidates walked in global
// memory: small and ragged contexts and coarse grids, whose neighbourhoods are
// neither staged (k_list_win) nor tiled (k_list_tile).
__global__ void __launch_bounds__(256, 3) k_list_full(
    const __grid_constant__ ListK K, const SysP *__restrict__ sp, const int *__restrict__ sys_of,
    const int *__restrict__ sreb, int all, int stride, uint32_t *__restrict__ nbr, int *__restrict__ nlen,
    long long *__restrict__ stat, int *__restrict__ halt, const int *__restrict__ gate) {
  if (block_gated_off(gate, 1)) return;
  __shared__ int qs[256 / 32][LQ];
  __shared__ float qrs[256 / 32][LQ];
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= K.n) return;                                   // whole warps
  const int s = sys_of[t];
  if (sys_skip(s, sreb, all)) return;                     // whole warps
  const SysP &P = sp[s];
  const int kind = grid_kind(P);
  full_list_atom<false>(P, K, t, stride, nbr, nlen, stat, halt, qs[threadIdx.x >> 5], qrs[threadIdx.x >> 5], kind,
                        kind == G_STENCIL && ortho(P), cell_width(P));
}

// Mixed mode, grids of 3 or more cells per axis whose neighbourhoods hold
// thousands of atoms.  A block takes up to 32 (`group`) atoms of one cell, one per lane,
// and its warps share the chunks of 32 candidates of the cell's stencil.  A
// candidate, staged as (x, y, z, |x|^2) in the cell's frame, is read by all
// lanes at once and tested against all 32 atoms by three FMAs and a
// comparison (|xj|^2 - 2 xi.xj against lim2 - |xi|^2); a lane that keeps it
// appends one byte to its atom's row of survivors.  After LT_C chunks the
// warps take the atoms in turn, 32 survivors at a time: FP32 distance, list
// flags (list_flags' tests), the master list entry and, for a system on the
// compact pair path (CW), its 16-bit window entry, which needs no conversion
// pass.  Candidate order is that of the other list kernels, so are the lists.
//
// Bound by instruction issue (8 instructions per candidate and 32 atoms, some
// 150 per 32 survivors).  41,472 water atoms (485 neighbours each): both lists
// in 0.35 ms; one atom per warp (k_list_full) and the conversion pass took
// 0.53 + 0.37 ms.
constexpr int LT_C = 32;                   // chunks between decisions
constexpr int LT_WARPS = 4;
constexpr int LT_WC = LT_C / LT_WARPS;     // chunks per warp (their candidates fit a byte)
constexpr int LT_TYPES = 8;                // types whose radii are held in shared memory

struct TileSmem {
  unsigned char kept[LT_WARPS][32][LT_WC * 32 + 4];   // per warp and atom: survivors, chunk of the warp << 5 | place
  float4 cand[LT_WARPS][2][32];            // candidates being tested
  int count[LT_WARPS][32];                 // survivors
  uint2 chunk[LT_C];                       // {first candidate | shift code << ENT_CODE_SHIFT, its window index}
  unsigned char valid[LT_C];               // candidates of the chunk
  float4 shift[27];
  int lo[27], cells[27], first[28], woff[27];   // stencil cells in walk order: first atom, count, first chunk, window offset
  float4 xi[32];
  int4 atom[32];                           // {atom, 2 type + charged, lowest excluded, span}
  int na[32], nb[32];                      // segment lengths so far
  float2 radii[LT_TYPES * LT_TYPES];       // LJ list radii^2 (t, s), -1: none
};

// appends byte `v` at shared address `at` where d < limit: two predicated
// instructions (a branch per candidate cost three times the test itself)
__device__ __forceinline__ void keep_if(float d, float limit, unsigned &at, unsigned v) {
  asm volatile("{\n .reg .pred p;\n setp.lt.f32 p, %1, %2;\n @p st.shared.u8 [%0], %3;\n @p add.u32 %0, %0, 1;\n}"
               : "+r"(at)
               : "f"(d), "f"(limit), "r"(v)
               : "memory");
}

template <bool CW>
__global__ void __launch_bounds__(LT_WARPS * 32, 5) k_list_tile(
    const __grid_constant__ ListK K, int group, int parts, const SysP *__restrict__ sp,
    const int *__restrict__ cell_sys, const int *__restrict__ sreb, int all, int stride, uint32_t *__restrict__ nbr,
    int *__restrict__ nlen, const __grid_constant__ CompactOut W, long long *__restrict__ stat,
    int *__restrict__ halt, const int *__restrict__ gate) {
  if (block_gated_off(gate, 1)) return;
  __shared__ TileSmem M;
  const int cell = blockIdx.x / parts, part = blockIdx.x - cell * parts;
  const int sy = cell_sys[cell];
  if (sys_skip(sy, sreb, all)) return;
  const SysP &P = sp[sy];
  const int hi = K.cell_start[cell + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = K.n;
  const unsigned lt_mask = (1u << lane) - 1u;
  const float4 *__restrict__ xq = K.xq;
  const int first_atom = K.cell_start[cell];
  if (first_atom + part * group >= hi) return;
  const int ntypes = P.ntypes;
  const bool rows = ntypes <= LT_TYPES;
  if (warp == 0) {
    // the stencil in walk_candidates' order (x offsets outermost): shift
    // codes 26 down to 0; the compact window holds the cells in code order
    const int lc = cell - P.c0;
    const int cz = lc % P.nc[2], cy = (lc / P.nc[2]) % P.nc[1], cx = lc / (P.nc[2] * P.nc[1]);
    int lo = 0, cnt = 0;
    if (lane < 27) {
      int jx = cx + lane / 9 - 1, jy = cy + (lane / 3) % 3 - 1, jz = cz + lane % 3 - 1;
      jx = jx < 0 ? jx + P.nc[0] : (jx >= P.nc[0] ? jx - P.nc[0] : jx);
      jy = jy < 0 ? jy + P.nc[1] : (jy >= P.nc[1] ? jy - P.nc[1] : jy);
      jz = jz < 0 ? jz + P.nc[2] : (jz >= P.nc[2] ? jz - P.nc[2] : jz);
      const int jc = P.c0 + (jx * P.nc[1] + jy) * P.nc[2] + jz;
      lo = K.cell_start[jc];
      cnt = K.cell_start[jc + 1] - lo;
      M.shift[lane] = P.shift[lane];
      M.lo[lane] = lo;
      M.cells[lane] = cnt;
    }
    int chunks = (cnt + 31) >> 5, atoms = cnt;
    const int mine = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, chunks, o), u = __shfl_up_sync(0xffffffffu, atoms, o);
      if (lane >= o) {
        chunks += v;
        atoms += u;
      }
    }
    const int tot = __shfl_sync(0xffffffffu, atoms, 31);
    if (lane < 27) {
      M.first[lane] = chunks - mine;
      M.woff[lane] = tot - atoms;                          // the atoms of the cells after it
    }
    if (lane == 26) M.first[27] = chunks;
  }
  if (rows)
    for (int k = threadIdx.x; k < ntypes * ntypes; k += LT_WARPS * 32) {
      const int intr = K.map[P.map0 + k];
      M.radii[k] = intr >= 0 ? make_float2((float)K.rad[2 * intr + 1], (float)K.rad[2 * intr])
                             : make_float2(-1.f, -1.f);
    }
  __syncthreads();
  const int nchunks = M.first[27], window = M.woff[0] + M.cells[0];
  const bool fits = !CW || window <= W.cap;
  if (CW && !fits && part == 0 && threadIdx.x == 0) {
    atomicAdd((unsigned long long *)(stat + ST_CWIN), 1ull);
    if (halt) *halt = 1;
  }
  const float near_r = fmaf(4e-5f, P.lim2_image, 2e-3f);
  const float el_r = (float)P.rmaxl_list2_e, es_r = (float)P.rmaxs_list2_e;
  // the threshold's room for the rounding of the larger terms (coordinates of
  // up to two cells); the survivors' distances are formed anew
  float lim;
  {
    float ext = 0.f;
#pragma unroll
    for (int k = 0; k < 9; k++) ext += fabsf(P.hF[k]) / (float)P.nc[k % 3];
    lim = fmaf(2e-5f * ext, ext, P.lim2);
  }
  unsigned bad = 0;
  for (int t0 = first_atom + part * group; t0 < hi; t0 += parts * group) {
    const int nseg = min(group, hi - t0);
    __syncthreads();                                       // the previous atoms' arrays are no longer read
    const float4 x = xq[t0 + min(lane, nseg - 1)];
    const float X = -2.f * x.x, Y = -2.f * x.y, Z = -2.f * x.z;
    const float T = lane < nseg ? lim - fmaf(x.z, x.z, fmaf(x.y, x.y, x.x * x.x)) : -3.0e38f;
    if (threadIdx.x < nseg) {
      const int2 mi = K.smeta[t0 + threadIdx.x];
      const int2 xs = K.xspan[mi.x];
      M.atom[threadIdx.x] = make_int4(mi.x, mi.y, xs.x, xs.y);
      M.xi[threadIdx.x] = x;
      M.na[threadIdx.x] = M.nb[threadIdx.x] = 0;
    }
    for (int c0 = 0; c0 < nchunks; c0 += LT_C) {
      const int nc = min(LT_C, nchunks - c0);
      __syncthreads();                                     // the last decisions are made
      if (threadIdx.x < nc) {
        const int c = c0 + threadIdx.x;
        int wa = 0, wb = 27;                               // the last cell with first <= c
        while (wb - wa > 1) {
          const int mid = (wa + wb) >> 1;
          if (M.first[mid] <= c) wa = mid;
          else wb = mid;
        }
        const int k = (c - M.first[wa]) * 32;
        M.chunk[threadIdx.x] = make_uint2((unsigned)(M.lo[wa] + k) | (unsigned)(26 - wa) << ENT_CODE_SHIFT,
                                          (unsigned)(M.woff[wa] + k));
        M.valid[threadIdx.x] = (unsigned char)min(32, M.cells[wa] - k);
      }
      __syncthreads();
      // test: this warp's chunks
      {
        const unsigned kept0 = (unsigned)__cvta_generic_to_shared(M.kept[warp][lane]);
        unsigned kept = kept0;
        const int ca = warp * LT_WC, cb = min(nc, ca + LT_WC);
        float4 xn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ca < cb && lane < M.valid[ca]) xn = xq[(M.chunk[ca].x & ENT_JMASK) + lane];
        for (int c = ca; c < cb; c++) {
          const float4 S = M.shift[M.chunk[c].x >> ENT_CODE_SHIFT];
          const float px = xn.x - S.x, py = xn.y - S.y, pz = xn.z - S.z;
          const int nv = M.valid[c];
          float4 *cand = M.cand[warp][c & 1];
          cand[lane] = make_float4(px, py, pz, lane < nv ? fmaf(pz, pz, fmaf(py, py, px * px)) : 3.0e38f);
          __syncwarp();
          if (c + 1 < cb && lane < M.valid[c + 1]) xn = xq[(M.chunk[c + 1].x & ENT_JMASK) + lane];
          const unsigned base = (unsigned)(c - ca) << 5;
#pragma unroll 8
          for (int k = 0; k < 32; k++) {
            const float4 p = cand[k];
            keep_if(fmaf(X, p.x, fmaf(Y, p.y, fmaf(Z, p.z, p.w))), T, kept, base + k);
          }
        }
        M.count[warp][lane] = (int)(kept - kept0);
      }
      __syncthreads();
      // decide: this warp's atoms
      for (int a = warp; a < nseg; a += LT_WARPS) {
        const int n0 = M.count[0][a], n1 = n0 + M.count[1][a], n2 = n1 + M.count[2][a], total = n2 + M.count[3][a];
        const int t = t0 + a;
        const float4 xi = M.xi[a];
        const int4 at = M.atom[a];
        uint32_t *out = nbr + (size_t)t * stride;
        unsigned short *cout = CW ? reinterpret_cast<unsigned short *>(W.list + (size_t)t * W.words) : nullptr;
        int na = M.na[a], nb = M.nb[a];
        const bool qi = (at.y & 1) != 0;
        const float2 *row = M.radii + (at.y >> 1) * ntypes;
        for (int h = 0; h < total; h += 32) {
          const int k = h + lane;
          const int p = (k >= n0) + (k >= n1) + (k >= n2);
          const int k0 = p == 0 ? 0 : (p == 1 ? n0 : (p == 2 ? n1 : n2));
          const bool in = k < total;
          const int e = in ? M.kept[p][a][k - k0] : 0;
          const uint2 cu = M.chunk[in ? p * LT_WC + (e >> 5) : 0];
          const int u = (int)(cu.x & ENT_JMASK) + (e & 31);
          const unsigned code = cu.x >> ENT_CODE_SHIFT;
          const bool on = in && u != t;
          float r2f = 3.0e38f;
          int2 mj = make_int2(-1, 0);
          if (on) {
            const float4 xj = xq[u], Sc = M.shift[code];
            mj = K.smeta[u];
            const float dx = (xi.x - xj.x) + Sc.x, dy = (xi.y - xj.y) + Sc.y, dz = (xi.z - xj.z) + Sc.z;
            r2f = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
          }
          float rl = -1.f, rs = -1.f;
          if (rows) {
            const float2 r = row[mj.y >> 1];
            rl = r.x;
            rs = r.y;
          } else if (on) {
            const int intr = K.map[P.map0 + (at.y >> 1) * ntypes + (mj.y >> 1)];
            if (intr >= 0) {
              rl = (float)K.rad[2 * intr + 1];
              rs = (float)K.rad[2 * intr];
            }
          }
          const bool qq = qi && (mj.y & 1);
          bool near;
          uint32_t en = radii_flags(r2f, rl, rs, qq ? el_r : -1.f, qq ? es_r : -1.f, near_r, &near);
          if (en && (unsigned)(mj.x - at.z) <= (unsigned)at.w) en = strike_excluded(P, K, en, at.x, mj.x);
          en |= code << ENT_CODE_SHIFT;
          if (on && near) en = exact_entry(P, K, at.x, mj.x);
          bad |= en & EXACT_BAD;
          // append (see append()), to both lists
          const bool fa = (en & (ENT_LJ | ENT_LJS)) != 0, any = (en & ENT_FLAGS) != 0;
          const unsigned ba = __ballot_sync(0xffffffffu, fa), bb = __ballot_sync(0xffffffffu, any && !fa);
          const int place = fa ? na + __popc(ba & lt_mask) : nb + __popc(bb & lt_mask);
          if (any && place < stride - (fa ? nb : na)) {
            out[fa ? place : stride - 1 - place] = (en & ~EXACT_BAD) | (uint32_t)u;
            if (CW && fits) {
              // (a code other than the candidate's own names no window slot:
              // bad geometry, reported by ST_BADSHIFT)
              const unsigned o = cu.y + (unsigned)(e & 31);
              cout[compact_place(place, fa, W.blocks)] = (unsigned short)(fa && (en & ENT_EL) ? o | COMPACT_EL : o);
            }
          }
          na += __popc(ba);
          nb += __popc(bb);
        }
        if (lane == 0) {
          M.na[a] = na;
          M.nb[a] = nb;
        }
      }
    }
    __syncthreads();
    for (int a = warp; a < nseg; a += LT_WARPS) {
      const int t = t0 + a;
      int na = M.na[a], nb = M.nb[a];
      if (na + nb > stride) {
        if (lane == 0) {
          atomicMax((unsigned long long *)(stat + ST_NEED_STRIDE), (unsigned long long)(na + nb));
          if (halt) {
            atomicAdd((unsigned long long *)(stat + ST_OVERFLOW), 1ull);
            *halt = 1;
          }
        }
        na = nb = 0;
      }
      if (lane == 0) {
        nlen[t] = na;
        nlen[n + t] = nb;
      }
      if (CW) {
        if (!fits) na = nb = 0;
        // the unused places of each segment's last block name the dummy slot
        unsigned short *cout = reinterpret_cast<unsigned short *>(W.list + (size_t)t * W.words);
        const int ea = (na + COMPACT_BLOCK - 1) / COMPACT_BLOCK * COMPACT_BLOCK,
                  eb = (nb + COMPACT_BLOCK - 1) / COMPACT_BLOCK * COMPACT_BLOCK;
        for (int k = na + lane; k < ea; k += 32) cout[compact_place(k, true, W.blocks)] = (unsigned short)W.cap;
        for (int k = nb + lane; k < eb; k += 32) cout[compact_place(k, false, W.blocks)] = (unsigned short)W.cap;
        if (lane == 0) W.len[t] = make_int2(na, nb);
      }
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicAdd((unsigned long long *)(stat + ST_BADSHIFT), 1ull);
}

// The cells of the systems being rebuilt, as one index range: rb_scan[s] is
// the number of such cells in systems before s, rb_scan[nsys] their total.
// A batch rebuilds a few of its systems on most steps; the list kernel then
// walks those cells only instead of skipping every other system's.
__global__ void k_rebuild_cells(int nsys, const SysP *__restrict__ sp, const int *__restrict__ sreb, int all,
                                int *__restrict__ rb_scan, const int *__restrict__ gate) {
  if (gated_off(gate, 1)) return;
  __shared__ int warp_tot[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < nsys; base += blockDim.x) {
    const int sy = base + threadIdx.x;
    const int v = sy < nsys && (all || sreb[sy] != 0) ? sp[sy].ncells : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
      int t = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += u;
      }
      warp_tot[lane] = t;                              // inclusive over warps
    }
    __syncthreads();
    const int before = carry + (w > 0 ? warp_tot[w - 1] : 0);
    if (sy < nsys) rb_scan[sy] = before + incl - v;
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_tot[(blockDim.x >> 5) - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) rb_scan[nsys] = carry;
}

// Mixed mode, block per cell: the block stages the cell's stencil
// neighbourhood (every candidate of every atom of the cell: FP32 positions
// moved by their cell's shift, sorted index + the cell's shift code, atom
// index, type and charge flag) in shared memory once, then its warps build
// the cell's atoms' lists from it: the prefilter reads shared memory, and in
// the list flags come from the FP32 distance (list_flags; in a grid of fewer
// than 3 cells per axis that of the minimum image) except within a margin of a
// list radius, where the FP64 test decides -- the same lists as the FP64 test
// of every candidate.
// Blocks walk the cells of the systems being rebuilt; a cell whose
// neighbourhood holds more than `cap` atoms is walked in global memory
// instead (same decisions).
constexpr int LW_THREADS = 256;
constexpr size_t LW_BYTES_PER_ATOM = sizeof(float4) + 2 * sizeof(int);   // s_x (w: type, charge), s_u, s_j
constexpr int LW_MIN_ATOMS = 1024;          // atoms per SM from which neighbourhoods are staged,
constexpr int LW_MIN_EVEN = 400;            //   and where the largest is at most LW_EVEN times the mean
constexpr double LW_EVEN = 1.5;
constexpr long long LW_MAX_CAP = 2944;     // largest staged neighbourhood (69 KB: 3 blocks per SM)

__global__ void __launch_bounds__(LW_THREADS, 3) k_list_win(
    const __grid_constant__ ListK K, int nsys, const int *__restrict__ rb_scan, const SysP *__restrict__ sp,
    int stride, int cap, uint32_t *__restrict__ nbr, int *__restrict__ nlen,
    long long *__restrict__ stat, int *__restrict__ halt, const int *__restrict__ gate) {
  if (block_gated_off(gate, 1)) return;
  extern __shared__ float4 s_x[];                        // cap
  int *s_u = reinterpret_cast<int *>(s_x + cap);         // cap: sorted index | shift code << ENT_CODE_SHIFT
  int *s_j = s_u + cap;                                  // cap: atom index
  __shared__ int qs[LW_THREADS / 32][LQ];
  __shared__ float qrs[LW_THREADS / 32][LQ];
  __shared__ int s_cs[27], s_off[27], s_code[27], s_tot, s_nw;
  __shared__ float4 s_sh[27];
  const int warp = threadIdx.x >> 5;
  const int total = rb_scan[nsys];
  for (int v = blockIdx.x; v < total; v += gridDim.x) {
    // the system of rebuilt cell v: the last s with rb_scan[s] <= v (systems
    // without rebuilt cells share their successor's value and are passed)
    int sa = 0, sb = nsys;
    while (sb - sa > 1) {
      const int mid = (sa + sb) >> 1;
      if (rb_scan[mid] <= v) sa = mid;
      else sb = mid;
    }
    const int s = sa;
    const SysP &P = sp[s];
    const int c = P.c0 + (v - rb_scan[s]);
    __syncthreads();                                     // the previous neighbourhood is no longer read
    if (threadIdx.x < 32) {
      // the system's stencil around cell c, one stencil cell per lane, in
      // walk_candidates' order (x offsets outermost), and the prefix of
      // their atom counts
      const int w = threadIdx.x;
      const int nw = P.nsx * P.nsy * P.nsz;
      int cn = 0;
      if (w < nw) {
        const int lc = c - P.c0;
        const int cz = lc % P.nc[2], cy = (lc / P.nc[2]) % P.nc[1], cx = lc / (P.nc[2] * P.nc[1]);
        const int ox = P.sx[w / (P.nsy * P.nsz)], oy = P.sy[(w / P.nsz) % P.nsy], oz = P.sz[w % P.nsz];
        int jx = cx + ox, jy = cy + oy, jz = cz + oz;
        jx = jx < 0 ? jx + P.nc[0] : (jx >= P.nc[0] ? jx - P.nc[0] : jx);
        jy = jy < 0 ? jy + P.nc[1] : (jy >= P.nc[1] ? jy - P.nc[1] : jy);
        jz = jz < 0 ? jz + P.nc[2] : (jz >= P.nc[2] ? jz - P.nc[2] : jz);
        const int cell = P.c0 + (jx * P.nc[1] + jy) * P.nc[2] + jz;
        const int cs = K.cell_start[cell];
        cn = K.cell_start[cell + 1] - cs;
        s_cs[w] = cs;
        s_code[w] = (1 - ox) * 9 + (1 - oy) * 3 + (1 - oz);
        s_sh[w] = P.shift[s_code[w]];
      }
      int incl = cn;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (w >= o) incl += v;
      }
      if (w < nw) s_off[w] = incl - cn;
      if (w == 31) {
        s_nw = nw;
        s_tot = incl;
      }
    }
    __syncthreads();
    const int tot = s_tot, nw = s_nw;
    const bool staged = tot <= cap;
    if (staged) {
      // one pass over the whole neighbourhood, so that every thread's loads
      // are in flight at once: staged atom g lies in the last stencil cell w
      // with s_off[w] <= g (empty cells share their successor's offset)
      for (int g = threadIdx.x; g < tot; g += blockDim.x) {
        int wa = 0, wb = nw;
        while (wb - wa > 1) {
          const int mid = (wa + wb) >> 1;
          if (s_off[mid] <= g) wa = mid;
          else wb = mid;
        }
        const int u = s_cs[wa] + (g - s_off[wa]);
        const float4 x = K.xq[u];
        const int2 mj = K.smeta[u];
        const float4 sh = s_sh[wa];
        s_x[g] = make_float4(x.x - sh.x, x.y - sh.y, x.z - sh.z, __int_as_float(mj.y));
        s_u[g] = u | (s_code[wa] << ENT_CODE_SHIFT);
        s_j[g] = mj.x;
      }
    }
    __syncthreads();
    const int lo = K.cell_start[c], hi = K.cell_start[c + 1];
    const int kind = grid_kind(P);
    const bool prune = kind == G_STENCIL && ortho(P);
    const float3 cw = cell_width(P);
    for (int t = lo + warp; t < hi; t += LW_THREADS / 32) {
      if (staged)
        full_list_atom<true>(P, K, t, stride, nbr, nlen, stat, halt, qs[warp], qrs[warp], kind, prune && nw == 27, cw,
                             s_x, s_u, s_j, tot, s_off, s_code, nw);
      else
        full_list_atom<false>(P, K, t, stride, nbr, nlen, stat, halt, qs[warp], qrs[warp], kind, prune, cw);
    }
  }
}

static Sorted sorted_arrays(const Ctx *c) {
  return {c->itype, c->pos, c->q, c->rank, c->styp, c->smeta, c->corner, c->xq};
}

// The cell corners (and FP32 cell-relative positions) under a new box: every
// atom keeps its cell and image, its corner moves with H (mixed mode; the
// pair kernels' shifts, also H-derived, are updated beside this).
int refresh_corners(Ctx *c) {
  if (c->mode != CM3D_NB_MIXED || !c->lists_built) return CM3D_NB_OK;
  k_sorted_init<<<grid_for(c->n, 256), 256, 0, c->st>>>(c->n, c->sp, c->sys_of, c->sreb, 1, c->cell_atoms, c->cimg,
                                                        sorted_arrays(c), nullptr);
  c->launches++;
  CKL(c);
  return CM3D_NB_OK;
}

// The positions rebuilds refer to.  nrefsh's rebuilds (sreb): dxn = pos
// (ngbr_list.c:577-580), isteplast = istep (md_finter.c:98); event = 0 leaves
// them alone.  The engine's own lists (lreb; dxi null: they follow nrefsh's
// rebuilds): dxi = pos.
__global__ void k_snapshot(int n, const SysP *__restrict__ sp, const int *__restrict__ sys_of,
                           const int *__restrict__ sreb, const int *__restrict__ lreb, int all, int event, int lists,
                           const double *__restrict__ pos, double *__restrict__ dxn, double *__restrict__ dxi,
                           int *__restrict__ slast, long long *__restrict__ sstat,
                           const int *__restrict__ gate, const int *__restrict__ istate,
                           long long *__restrict__ stat) {
  if (gate && (gate[IS_HALT] != 0 || (gate[IS_REBUILD] == 0 && gate[IS_LREBUILD] == 0))) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && event && (!gate || gate[IS_REBUILD] != 0)) atomicAdd((unsigned long long *)(stat + ST_REBUILDS), 1ull);
  if (i >= n) return;
  const int s = sys_of[i];
  const double x = pos[i], y = pos[n + i], z = pos[2 * n + i];
  if (dxi && lists && (all || lreb[s] != 0)) {
    dxi[i] = x;
    dxi[n + i] = y;
    dxi[2 * n + i] = z;
  }
  if (!event || sys_skip(s, sreb, all)) return;
  dxn[i] = x;
  dxn[n + i] = y;
  dxn[2 * n + i] = z;
  if (i == sp[s].a0) {
    slast[s] = istate[IS_ISTEP];
    sstat[(size_t)s * SS_COUNT + SS_REBUILDS] += 1;
  }
}

// nrefsh's snapshot (unless no_snapshot; in a host-driven pass if the flag it
// read back asks for it) and, with `lists`, that of the lists just built
int take_snapshot(Ctx *c, bool device_flag, bool all, bool lists) {
  const bool event = !c->no_snapshot && (all || device_flag || c->h_istate[IS_REBUILD] != 0);
  k_snapshot<<<grid_for(c->n, 256), 256, 0, c->st>>>(c->n, c->sp, c->sys_of, c->sreb, c->lreb, all ? 1 : 0,
                                                      event ? 1 : 0, lists ? 1 : 0, c->pos, c->dxn, c->dxi,
                                                      c->slast, c->sstat, device_flag ? c->istate : nullptr, c->istate,
                                                      c->stat);
  c->launches++;
  CKL(c);
  return CM3D_NB_OK;
}

// --------------------------------------------------------------- host side
static void stencil(int nc, int *s, int *ns) {
  if (nc >= 3) {
    s[0] = -1; s[1] = 0; s[2] = 1; *ns = 3;
  } else if (nc == 2) {
    s[0] = 0; s[1] = 1; *ns = 2;
  } else {
    s[0] = 0; *ns = 1;
  }
}

// width of the box along each direction (1 / |row d of H^-1|)
double box_width(const SysH &H, int d) {
  return 1.0 / sqrt(H.hmati[3 * d] * H.hmati[3 * d] + H.hmati[3 * d + 1] * H.hmati[3 * d + 1] +
                    H.hmati[3 * d + 2] * H.hmati[3 * d + 2]);
}

// cells along direction d for lists of radius rlist
int cells_along(const SysH &H, int d, double rlist, double cell_scale) {
  const int m = rlist > 0 ? (int)floor(box_width(H, d) / (rlist * cell_scale)) : 1;
  return m < 1 ? 1 : (m > 1000 ? 1000 : m);
}

// the 27 neighbour-cell displacements of a system's grid (one cell step
// along each box vector), as FP32 hi + lo parts
void cell_shifts(SysP &P, const SysH &H) {
  for (int a = -1; a <= 1; a++)
    for (int b = -1; b <= 1; b++)
      for (int d = -1; d <= 1; d++) {
        double f0 = (double)a / P.nc[0], f1 = (double)b / P.nc[1], f2 = (double)d / P.nc[2];
        const double *h = H.hmat;
        const double v0 = h[0] * f0 + h[1] * f1 + h[2] * f2, v1 = h[3] * f0 + h[4] * f1 + h[5] * f2,
                     v2 = h[6] * f0 + h[7] * f1 + h[8] * f2;
        const int k = (a + 1) * 9 + (b + 1) * 3 + (d + 1);
        P.shift[k] = make_float4((float)v0, (float)v1, (float)v2, 0.f);
        P.shift_lo[k] = make_float4((float)(v0 - (double)(float)v0), (float)(v1 - (double)(float)v1),
                                    (float)(v2 - (double)(float)v2), 0.f);
      }
  // FP32 minimum images in the list tests of a coarse grid: candidates lie
  // within two cells, so cells of at most 4 list radii bound the displacement
  P.image_ok = 1;
  P.sheared = ortho(P) ? 0 : 1;
  for (int d = 0; d < 3; d++)
    if (!(box_width(H, d) / P.nc[d] <= 4.0 * H.rlist)) P.image_ok = 0;
}

// Cell grids of every system (cells at least one list radius wide in every
// fractional direction: plane spacing 1 / |row d of hmati|), their stencils,
// the 27 cell-corner shifts and the FP32 prefilter radius, in the cell fields
// of c->h_sp, and the list kernel for such cells.  At set-up, and again where a
// moving box takes the list radius back.
int grid_setup(Ctx *c) {
  int c0 = 0;
  for (int s = 0; s < c->nsys; s++) {
    SysP &P = c->h_sp[s];
    SysH &H = c->hs[s];
    int tot = 1;
    for (int d = 0; d < 3; d++) {
      P.nc[d] = cells_along(H, d, H.rlist, c->cell_scale);
      H.nc_cm[d] = cells_along(H, d, H.rlist_cm, c->cell_scale);
      tot *= P.nc[d];
    }
    P.c0 = c0;
    P.ncells = tot;
    c0 += tot;
    stencil(P.nc[0], P.sx, &P.nsx);
    stencil(P.nc[1], P.sy, &P.nsy);
    stencil(P.nc[2], P.sz, &P.nsz);
    // with three or more cells per direction the stencil neighbour's image
    // is the minimum image of every pair in range, so the FP32 prefilter is
    // exact up to rounding; with fewer cells the minimum image is taken first
    // (lim2_image), or every candidate goes to the FP64 test
    const bool pre = P.nc[0] >= 3 && P.nc[1] >= 3 && P.nc[2] >= 3;
    const double rl = H.rlist + 1e-3;
    P.lim2 = pre ? (float)(rl * rl) : INFINITY;
    P.lim2_image = (float)(rl * rl);
    cell_shifts(P, H);
  }
  c->ncells = c0;
  c->nc[0] = c->h_sp[0].nc[0];
  c->nc[1] = c->h_sp[0].nc[1];
  c->nc[2] = c->h_sp[0].nc[2];
  // system 0's shifts (the single-system pair kernel keeps them in shared memory)
  CK(cudaMemcpy(c->shift, c->h_sp[0].shift, sizeof(float4) * 27, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(c->shift + 27, c->h_sp[0].shift_lo, sizeof(float4) * 27, cudaMemcpyHostToDevice));
  if (c->mode == CM3D_NB_MIXED) {
    // staged list build: room for 1.6x the largest mean stencil neighbourhood
    // (+64), within the shared memory a block may opt into
    double nb_max = 0, nb_sum = 0;
    c->lw_atoms = 1;
    for (int sy = 0; sy < c->nsys; sy++) {
      const SysP &S = c->h_sp[sy];
      const double per_cell = (double)S.n / (double)(S.ncells > 0 ? S.ncells : 1);
      const double nb = per_cell * S.nsx * S.nsy * S.nsz;
      nb_max = std::max(nb_max, nb);
      nb_sum += nb * S.n;
      c->lw_atoms = std::max(c->lw_atoms, (int)(1.25 * per_cell) + 1);
    }
    c->lw_smem_max = c->smem_optin > 8192 ? c->smem_optin - 8192 : 0;
    long long cap = (long long)(1.6 * nb_max) + 64;
    const long long cap_max = (long long)(c->lw_smem_max / LW_BYTES_PER_ATOM);
    c->lw_cap = (int)std::min(cap, cap_max);
    // a neighbourhood of thousands of atoms leaves one block per SM: the
    // warp-per-atom walk through global memory keeps more warps in flight
    if (c->lw_cap < 64 || cap > LW_MAX_CAP) c->lw_cap = 0;
    // with a few cells per block the staging of the largest neighbourhood is
    // what the kernel waits for, and a warp per atom fills the GPU sooner: in
    // ragged batches up to 1024 atoms per SM, in even ones, whose blocks finish
    // together, up to 400.  (us per step, walked and staged.  Ragged, the
    // largest neighbourhood 2.3 times the mean: 27,000 atoms 99, 131; 71,000,
    // 181, 210; 131,000, 284, 300; 216,000, 429, 428.  Even: 24,600 atoms 57,
    // 57; 49,000 charged 151, 155; 64,000, 86, 78; 64,000 charged 204, 189;
    // 108,000 in one box 140, 131; 150,000, 163, 149.  1.47 times: 85,000,
    // 119, 112.)
    const bool even = nb_max * c->n <= LW_EVEN * nb_sum;
    if (c->n < (even ? LW_MIN_EVEN : LW_MIN_ATOMS) * c->num_sms) c->lw_cap = 0;
    const char *lk = getenv("CM3D_NB_LIST_KERNEL");
    if (lk && strcmp(lk, "walk") == 0) c->lw_cap = 0;
    c->list_tile = cap > LW_MAX_CAP ? 1 : 0;
    for (int sy = 0; sy < c->nsys; sy++)
      for (int d = 0; d < 3; d++)
        if (c->h_sp[sy].nc[d] < 3) c->list_tile = 0;
    if (lk && strcmp(lk, "walk") == 0) c->list_tile = 0;
  }
  return CM3D_NB_OK;
}

// The grids, and the binning and list arrays.
int list_setup(Ctx *c) {
  CK(cudaMalloc(&c->shift, sizeof(float4) * 54));
  int rc = grid_setup(c);
  if (rc) return rc;
  // (one system: room for the grid of CM3D's radii as well, which set_box takes up)
  const int ncells = std::max(c->ncells, c->nsys == 1 ? cells_cm(c->hs[0]) : 0);
  std::vector<int> cell_sys((size_t)ncells, 0);
  for (int s = 0; s < c->nsys; s++)
    for (int k = 0; k < c->h_sp[s].ncells; k++) cell_sys[(size_t)c->h_sp[s].c0 + k] = s;
  CK(cudaMalloc(&c->cell_sys, sizeof(int) * (size_t)ncells));
  CK(cudaMemcpy(c->cell_sys, cell_sys.data(), sizeof(int) * (size_t)ncells, cudaMemcpyHostToDevice));
  CK(cudaMalloc(&c->cell_start, sizeof(int) * ((size_t)ncells + 1)));
  CK(cudaMalloc(&c->cell_cursor, sizeof(int) * ((size_t)ncells + 1)));
  CK(cudaMemset(c->cell_cursor, 0, sizeof(int) * ((size_t)ncells + 1)));
  double est_max = 32.0;
  for (const SysH &H : c->hs) {
    // first guess of the full-list slot: 1.3 x the mean number of atoms in
    // a list sphere, plus 64
    double vol = fabs(H.hmat[0] * (H.hmat[4] * H.hmat[8] - H.hmat[5] * H.hmat[7]) +
                      H.hmat[1] * (H.hmat[5] * H.hmat[6] - H.hmat[3] * H.hmat[8]) +
                      H.hmat[2] * (H.hmat[3] * H.hmat[7] - H.hmat[4] * H.hmat[6]));
    double r = H.rlist;
    double est = 1.3 * (double)H.n / vol * (4.0 / 3.0) * M_PI * r * r * r + 64.0;
    if (est > (double)H.n + 31.0) est = (double)H.n + 31.0;
    if (est > est_max) est_max = est;
  }
  CK(cudaMalloc(&c->cell_of, sizeof(int) * (size_t)c->n));
  CK(cudaMalloc(&c->cell_atoms, sizeof(int) * (size_t)c->n));
  CK(cudaMalloc(&c->rank, sizeof(int) * (size_t)c->n));
  int n_max = 0;
  for (int s = 0; s < c->nsys; s++) n_max = std::max(n_max, c->h_sp[s].n);
  // (the FP64 engine, which builds its lists at CM3D's frequency: not where
  // each atom is ordered among hundreds in its cell, by eight SMs)
  const bool crowded = c->mode == CM3D_NB_PLAIN_FP64 && (double)n_max * n_max > BIN_PLAIN_PAIRS * c->ncells;
  if (n_max <= BIN_ATOMS && !crowded) {
    // an atom per thread, while the clusters of a batch fit the GPU side by side
    c->bin_cluster = 1;
    while (c->bin_cluster < BIN_CLUSTER && c->bin_cluster * BIN_THREADS < n_max &&
           2 * c->bin_cluster * c->nsys <= c->num_sms)
      c->bin_cluster *= 2;
    CK(cudaMalloc(&c->bin_keys, sizeof(long long) * (size_t)c->n));
  }
  CK(cudaMalloc(&c->cnt, sizeof(int) * 4 * (size_t)c->n));
  CK(cudaMalloc(&c->off, sizeof(long long) * 4 * ((size_t)c->n + 1)));
  CK(cudaMalloc(&c->ltot, sizeof(long long) * LT_COUNT));
  CK(cudaMallocHost(&c->h_ltot, sizeof(long long) * LT_COUNT));
  CK(cudaMalloc(&c->styp, sizeof(int) * (size_t)c->n));
  CK(cudaMalloc(&c->smeta, sizeof(int2) * (size_t)c->n));
  CK(cudaMalloc(&c->corner, sizeof(double) * 3 * (size_t)c->n));
  CK(cudaMalloc(&c->xq, sizeof(float4) * (size_t)c->n));
  CK(cudaMalloc(&c->cimg, sizeof(int4) * (size_t)c->n));
  if (c->mode == CM3D_NB_MIXED) {
    CK(cudaMalloc(&c->rb_scan, sizeof(int) * ((size_t)c->nsys + 1)));
    CK(cudaMalloc(&c->nlen, sizeof(int) * 2 * (size_t)c->n));
    CK(cudaMemset(c->nlen, 0, sizeof(int) * 2 * (size_t)c->n));
    long long s = ((long long)est_max + 31) / 32 * 32;
    if (s < 32) s = 32;
    c->nbr_stride = (int)s;
    CK(cudaMalloc(&c->nbr, sizeof(uint32_t) * (size_t)c->n * (size_t)s));
    c->lcap[LT_FULL] = (long long)c->n * s;
  }
  return CM3D_NB_OK;
}

// one warp per atom: its front segment (nlen[t] entries) and back segment
// (nlen[n + t]) from a slot of `old_s` entries into one of `new_s`
__global__ void k_regrow_copy(int n, int old_s, int new_s, const int *__restrict__ nlen,
                              const uint32_t *__restrict__ src, uint32_t *__restrict__ dst) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= n) return;
  const int na = min(nlen[t], old_s), nb = min(nlen[n + t], old_s - na);
  const uint32_t *a = src + (size_t)t * old_s;
  uint32_t *b = dst + (size_t)t * new_s;
  for (int k = lane; k < na; k += 32) b[k] = a[k];
  for (int k = lane; k < nb; k += 32) b[new_s - nb + k] = a[old_s - nb + k];
}

// grow list buffers to hold at least `need` entries (with 50% headroom)
static int grow(Ctx *c, int which, long long need) {
  if (need <= c->lcap[which]) return CM3D_NB_OK;
  DevLock lock(device_mutex());
  long long cap = need + need / 2 + 4096;
  if (c->graph) {
    // a captured step holds the old buffer addresses
    cudaGraphExecDestroy(c->graph);
    c->graph = nullptr;
  }
  if (c->lst[which]) cudaFree(c->lst[which]);
  c->lst[which] = nullptr;
  cudaError_t e = cudaMalloc(&c->lst[which], sizeof(int2) * (size_t)cap);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(list)");
  c->lcap[which] = cap;
  return CM3D_NB_OK;
}

// widen the full-list slots to hold `need` entries (+1/8 and 32 spare)
static int grow_full(Ctx *c, long long need) {
  DevLock lock(device_mutex());
  long long s = (need + need / 8 + 32 + 31) / 32 * 32;
  if (s <= c->nbr_stride) s = c->nbr_stride + 32;
  if (c->graph) {
    cudaGraphExecDestroy(c->graph);
    c->graph = nullptr;
  }
  CK(cudaStreamSynchronize(c->st));
  uint32_t *wider = nullptr;
  cudaError_t e = cudaMalloc(&wider, sizeof(uint32_t) * (size_t)c->n * (size_t)s);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(full list)");
  // the lists of the systems not being rebuilt stay valid: both segments of
  // every slot move into the wider slots (a rebuilt system's are rewritten)
  if (c->nbr)
    k_regrow_copy<<<grid_for((long long)c->n * 32, 256), 256, 0, c->st>>>(c->n, c->nbr_stride, (int)s, c->nlen,
                                                                           c->nbr, wider);
  CK(cudaStreamSynchronize(c->st));
  if (c->nbr) cudaFree(c->nbr);
  c->nbr = wider;
  c->nbr_stride = (int)s;
  c->lcap[LT_FULL] = (long long)c->n * s;
  return CM3D_NB_OK;
}

static ListCaps caps(Ctx *c) {
  ListCaps C;
  for (int k = 0; k < 4; k++) C.cap[k] = c->lcap[k];
  return C;
}

// Build the lists from the current positions.  `all`: every system (set-up,
// get_ngbr, export); otherwise only the systems whose displacement test
// asked for it (lreb).  With device_flag the kernels are also gated on the
// device rebuild flag (graph replay) and the capacities are not re-checked on
// the host.  The plain engine always builds CM3D's half lists (its pair
// kernels walk them); the mixed engine builds its full list and the half
// lists only when asked (export / parity checks).
int build_lists(Ctx *c, bool device_flag, bool all) {
  const int n = c->n;
  const int B = 256;
  const int *gate = device_flag ? c->istate : nullptr;
  const int al = all ? 1 : 0;
  const bool want_half = c->mode == CM3D_NB_PLAIN_FP64 || c->want_half;
  cudaEvent_t e0;
  tbegin(c, 2, &e0);
  int4 *cimg = c->cimg;
  if (c->bin_cluster > 0) {
    CK(cluster_launch(k_bin, c->nsys * c->bin_cluster, c->bin_cluster, BIN_THREADS, c->st, n, c->bin_cluster,
                      (const SysP *)c->sp, (const int *)c->lreb, al, sorted_arrays(c), cimg, c->cell_of,
                      c->cell_cursor, c->cell_start, c->bin_keys, c->cell_atoms, gate));
    c->launches++;
  } else {
    k_cell_zero<<<grid_for(c->ncells, B), B, 0, c->st>>>(c->ncells, c->cell_sys, c->lreb, al, c->cell_cursor, gate);
    k_cell_assign<<<grid_for(n, B), B, 0, c->st>>>(n, c->pos, c->sp, c->sys_of, c->lreb, al, c->cell_of,
                                                    c->cell_cursor, cimg, gate);
    k_cell_scan<<<c->nsys, 256, 0, c->st>>>(c->sp, c->lreb, al, c->cell_cursor, c->cell_start, gate);
    k_cell_fill<<<grid_for(n, B), B, 0, c->st>>>(n, c->sys_of, c->lreb, al, c->cell_of, c->cell_start,
                                                  c->cell_cursor, c->cell_atoms, gate);
    // enough blocks for four per SM where the grid allows it
    const int per_block = std::max(1, std::min(SORT_CELLS, c->ncells / std::max(1, 4 * c->num_sms)));
    k_cell_sort<<<(c->ncells + per_block - 1) / per_block, SORT_THREADS, 0, c->st>>>(
        c->ncells, per_block, c->cell_sys, c->lreb, al, c->cell_start, c->itype, c->cell_atoms, gate);
    k_sorted_init<<<grid_for(n, B), B, 0, c->st>>>(n, c->sp, c->sys_of, c->lreb, al, c->cell_atoms, cimg,
                                                    sorted_arrays(c), gate);
    c->launches += 6;
  }
  const long long warps_threads = 32LL * n;
  int *halt = device_flag ? c->istate + IS_HALT : nullptr;
  ListK K = {n, c->cell_atoms, c->cell_start, c->cell_of, c->xq, c->pos, c->itype, c->map, c->rad, c->q, 1,
                   c->excl_off, c->excl_idx, c->cexcl_off, c->cexcl_idx, cimg, c->smeta, c->xspan};
  bool direct = false;                       // the list kernel wrote the compact lists as well
  if (c->mode == CM3D_NB_MIXED) {
    for (;;) {
      CompactOut W = {nullptr, nullptr, 0, 0, 0};
      if (c->lw_cap > 0) {
        // block per cell over the cells of the systems being rebuilt, the
        // stencil neighbourhood staged in shared memory
        const size_t smem = (size_t)c->lw_cap * LW_BYTES_PER_ATOM;
        static unsigned long long attr_devs = 0;
        if (c->dev < 64 && !(attr_devs & (1ull << c->dev))) {
          cudaFuncSetAttribute(k_list_win, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c->lw_smem_max);
          attr_devs |= 1ull << c->dev;
        }
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_list_win, LW_THREADS, smem);
        long long grid = (long long)c->num_sms * (per_sm > 0 ? per_sm : 1);
        if (grid > c->ncells) grid = c->ncells;
        k_rebuild_cells<<<1, 1024, 0, c->st>>>(c->nsys, c->sp, c->lreb, al, c->rb_scan, gate);
        k_list_win<<<(int)grid, LW_THREADS, smem, c->st>>>(K, c->nsys, c->rb_scan, c->sp, c->nbr_stride, c->lw_cap,
                                                           c->nbr, c->nlen, c->stat, halt, gate);
        c->launches++;
      } else if (c->list_tile) {
        int rc = CM3D_NB_OK;
        const bool compact = cw_direct(c, device_flag, &W, &rc);
        if (rc) return rc;
        // fewer atoms per block where blocks of 32 would leave SMs idle: the
        // tests then run on fewer lanes, but a block's decisions, one atom
        // after another, are what a small system waits for (3993 atoms: 169 us
        // with 32 atoms per block, 102 with 8; 12,288: 212 with 32, 277 with 16)
        int group = 32;
        while (group > 8 && (long long)n / group < 2LL * c->num_sms) group /= 2;
        const int parts = (c->lw_atoms + group - 1) / group;
        const auto kern = compact ? k_list_tile<true> : k_list_tile<false>;
        kern<<<c->ncells * parts, LT_WARPS * 32, 0, c->st>>>(K, group, parts, c->sp, c->cell_sys, c->lreb, al,
                                                             c->nbr_stride, c->nbr, c->nlen, W, c->stat, halt, gate);
        direct = compact;
      } else {
        k_list_full<<<grid_for(warps_threads, 256), 256, 0, c->st>>>(K, c->sp, c->sys_of, c->lreb, al, c->nbr_stride,
                                                                     c->nbr, c->nlen, c->stat, halt, gate);
      }
      c->launches++;
      CKL(c);
      if (device_flag) break;
      // host-driven build: widen the slots and build again if a list did not fit
      CK(cudaMemcpyAsync(c->h_stat, c->stat, sizeof(long long) * ST_COUNT, cudaMemcpyDeviceToHost, c->st));
      CK(cudaStreamSynchronize(c->st));
      if (c->h_stat[ST_NEED_STRIDE] <= c->nbr_stride) break;
      int rc = grow_full(c, c->h_stat[ST_NEED_STRIDE]);
      if (rc) return rc;
    }
  }
  if (c->mode == CM3D_NB_MIXED) {
    int rc = direct ? cw_check(c, device_flag) : cw_convert(c, device_flag, all);
    if (rc) return rc;
  }
  if (want_half) {
    // CM3D's lists, by CM3D's radii
    const bool stencil = std::all_of(c->h_sp.begin(), c->h_sp.end(), [](const SysP &S) { return grid_kind(S) == G_STENCIL; });
    const auto half_count = stencil ? k_list_half<false, true> : k_list_half<false, false>;
    const auto half_fill = stencil ? k_list_half<true, true> : k_list_half<true, false>;
    K.rad = c->rad_cm;
    K.own = 0;
    half_count<<<grid_for(warps_threads, 256), 256, 0, c->st>>>(
        K, c->sp, c->sys_of, caps(c), c->cnt, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, c->stat, nullptr,
        gate);
    k_scan<int, long long><<<dim3(1, 4), 1024, 0, c->st>>>(c->cnt, c->off, c->ltot, n, gate);
    c->launches += 2;
    CKL(c);
    if (!device_flag) {
      CK(cudaMemcpyAsync(c->h_ltot, c->ltot, sizeof(long long) * 4, cudaMemcpyDeviceToHost, c->st));
      CK(cudaStreamSynchronize(c->st));
      for (int k = 0; k < 4; k++) {
        int rc = grow(c, k, c->h_ltot[k] > 0 ? c->h_ltot[k] : 1);
        if (rc) return rc;
        c->hcount[k] = c->h_ltot[k];
      }
    }
    half_fill<<<grid_for(warps_threads, 256), 256, 0, c->st>>>(
        K, c->sp, c->sys_of, caps(c), c->cnt, c->off, c->ltot, c->lst[0], c->lst[1], c->lst[2], c->lst[3], c->stat,
        halt, gate);
    c->launches++;
  }
  if (!c->no_snapshot || c->dxi) {
    const int rc = take_snapshot(c, device_flag, all, true);
    if (rc) return rc;
  }
  CKL(c);
  tend(c, 2, e0);
  if (!device_flag) {
    c->lists_built = true;
    c->rebuilds_host++;
  }
  return CM3D_NB_OK;
}

}  // namespace cm3d
