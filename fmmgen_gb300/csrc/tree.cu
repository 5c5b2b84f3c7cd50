// tree.cu -- device octree build and interaction lists.
//
// Reproduces build_tree (example/tree.cpp:130-233) and interact_dehnen_lazy
// (example/calculate.cpp:81-133) bit-exactly, without the sequential insertion:
//  * build_tree's final partition does not depend on insertion order: a cell
//    is split iff it holds >= ncrit particles, a child exists iff a particle
//    falls in its octant, and each particle's octant path is fixed by FP64
//    comparisons against centres that depend only on the path.  So every
//    particle gets a 63-bit key of its 21 octant digits, computed with exactly
//    the reference's FP64 centre arithmetic (example/tree.cpp:94-98, 193), the
//    keys are radix-sorted, and the cells are cut level by level from the
//    sorted keys with the count rule.
//  * the dual-tree walk is run breadth-first over a frontier of cell pairs;
//    each pair's decision (MAC, P2P, split A, split B) depends only on the
//    pair, so the visited pairs -- and the M2L/P2P lists as multisets -- are
//    those of the recursive walk.
// All FP64 arithmetic that decides structure uses __d*_rn intrinsics so that no
// FMA contraction changes a rounding relative to the reference source.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <cooperative_groups.h>
#include "internal.h"
#include "prims.cuh"
#include "deriv.cuh"

// ---------------------------------------------------------------------------
// root box (example/tree.cpp:139-187)
// ---------------------------------------------------------------------------
// The three sequential sums come from fmm_seqsum3 (seqsum.cu), bit-identical to
// the reference's loop; the maxima are order-independent.
long fmm_seqsum_chunks(long n);
size_t fmm_seqsum_scratch_tables(long chunks);
int fmm_seqsum3_systems(const double *pos, const long *sys_off, const int *chunk_off, int nsys, long chunks,
                        double *out, void *scratch, cudaStream_t st);
int fmm_seqsum3(const double *pos, long N, double *out, void *scratch, bool tables, cudaStream_t st);

__global__ void k_root_absmax(const double *__restrict__ pos, long N, const double *sums,
                              unsigned long long *mx) {
  double inv_n = (double)N;
  double ax = __ddiv_rn(sums[0], inv_n), ay = __ddiv_rn(sums[1], inv_n), az = __ddiv_rn(sums[2], inv_n);
  double mxx = 0, mxy = 0, mxz = 0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < N; i += (long)gridDim.x * blockDim.x) {
    mxx = fmax(mxx, fabs(__dsub_rn(pos[3 * i], ax)));
    mxy = fmax(mxy, fabs(__dsub_rn(pos[3 * i + 1], ay)));
    mxz = fmax(mxz, fabs(__dsub_rn(pos[3 * i + 2], az)));
  }
  for (int d = 16; d; d >>= 1) {
    mxx = fmax(mxx, __shfl_xor_sync(0xffffffffu, mxx, d));
    mxy = fmax(mxy, __shfl_xor_sync(0xffffffffu, mxy, d));
    mxz = fmax(mxz, __shfl_xor_sync(0xffffffffu, mxz, d));
  }
  if ((threadIdx.x & 31) == 0) {
    // non-negative doubles order like their bit patterns
    atomicMax(&mx[0], (unsigned long long)__double_as_longlong(mxx));
    atomicMax(&mx[1], (unsigned long long)__double_as_longlong(mxy));
    atomicMax(&mx[2], (unsigned long long)__double_as_longlong(mxz));
  }
}

// root[0..3] = centre, r; lev[2l] = r_l, lev[2l+1] = rmax_l = sqrt(3*r_l*r_l).  A lane
// per level, which halves r for itself (the halvings are exact, so as r / 2.0 one
// after the other); on one thread the chain of divisions and roots took 14 us.
__global__ void k_root_final(const double *sums, const unsigned long long *mx, long N, double *root,
                             double *lev, float2 *levf) {
  const int l = threadIdx.x;
  const double n = (double)N;
  const double xm = __longlong_as_double((long long)mx[0]);
  const double ym = __longlong_as_double((long long)mx[1]);
  const double zm = __longlong_as_double((long long)mx[2]);
  const double r = __dmul_rn((xm > ym ? (xm > zm ? xm : zm) : (ym > zm ? ym : zm)), 1.001);
  if (l < 3) root[l] = __ddiv_rn(sums[l], n);
  if (l == 3) root[3] = r;
  if (l > FMM_MAXLEVEL) return;
  double rl = r;
  for (int k = 0; k < l; k++) rl = __dmul_rn(rl, 0.5);
  lev[2 * l] = rl;
  lev[2 * l + 1] = __dsqrt_rn(__dmul_rn(__dmul_rn(3.0, rl), rl));  // example/tree.cpp:15
  const float hi = (float)rl;
  levf[l] = make_float2(hi, (float)(rl - (double)hi));
}

// ---------------------------------------------------------------------------
// per-particle octant keys (example/tree.cpp:94-98, 189-204)
// ---------------------------------------------------------------------------
// The digits of levels 1..nlev (the rest of the key is zero): the cells are cut
// from them, and the build asks for all FMM_MAXLEVEL levels only when a cell at
// level nlev still has to be split.
// The digits compare with centres that the reference adds up level by level in
// FP64, each with its rounding.  Up to ten levels they follow from the particle's
// place on the grid of the finest one, which FP32 gives to a few 1e-4 of a cell:
// only a particle that close to a boundary, or in a root cube so far from the
// origin that the centres' own rounding matters, takes the comparisons.  Bound by
// the FP64 pipe: 10^6 particles 155 -> 41 us, 9.4M of 512 systems 1.26 -> 0.28 ms.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // bit b of ten to bit 3 b
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  return (v | (v << 2)) & 0x09249249u;
}
__device__ __forceinline__ bool grid_key(double x, double y, double z, double cx, double cy, double cz, double r,
                                         int nlev, uint64_t &key) {
  if (nlev > 10) return false;
  auto ex = [](double v) { return (__double2hiint(v) >> 20) & 0x7ff; };
  if (max(ex(cx), max(ex(cy), ex(cz))) > ex(r) + 24) return false;  // the centres' rounding: below 1e-4 of a cell
  // of a cell: d, 1 / r and the product are each rounded to 2^-24, ten levels deep 2.4e-4
  const float cells = (float)(1 << nlev), scale = 0.5f * cells / (float)r, tol = 5e-4f;
  const float u = (float)(x - (cx - r)) * scale, v = (float)(y - (cy - r)) * scale, w = (float)(z - (cz - r)) * scale;
  const float fu = floorf(u), fv = floorf(v), fw = floorf(w);
  const float lo = fminf(u - fu, fminf(v - fv, w - fw)), hi = fmaxf(u - fu, fmaxf(v - fv, w - fw));
  const float least = fminf(fu, fminf(fv, fw)), most = fmaxf(fu, fmaxf(fv, fw));
  // the sum catches a NaN, which the minima and maxima pass over
  if (!(lo > tol && hi < 1.f - tol && least >= 0.f && most < cells && u + v + w < 4.f * cells)) return false;
  key = spread3((uint32_t)fu) | spread3((uint32_t)fv) << 1 | (uint64_t)spread3((uint32_t)fw) << 2;
  return true;
}
__global__ void k_keys(const double *__restrict__ pos, long N, const double *roots, const int *psys,
                       int nlev, uint64_t *keys, uint32_t *idx) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double *root = roots + 4 * (psys ? psys[i] : 0);  // the particle's system's root cube
  double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  double cx = root[0], cy = root[1], cz = root[2], r = root[3];
  uint64_t key = 0;
  if (!grid_key(x, y, z, cx, cy, cz, r, nlev, key))
#pragma unroll 3
  for (int l = 0; l < nlev; l++) {
    int oct = (x > cx) + ((y > cy) << 1) + ((z > cz) << 2);
    key = (key << 3) | (uint64_t)oct;
    // r / 2.0 and r * (+-1) are exact: halving and a sign select round identically
    r = __dmul_rn(r, 0.5);
    cx = __dadd_rn(cx, (oct & 1) ? r : -r);
    cy = __dadd_rn(cy, (oct & 2) ? r : -r);
    cz = __dadd_rn(cz, (oct & 4) ? r : -r);
  }
  keys[i] = key << (3 * (FMM_MAXLEVEL - nlev));
  idx[i] = (uint32_t)i;
}

// rank[i] += the keys below keys[i] among the block's share (blockIdx.y) of them
constexpr int RANK_BS = 256;
__global__ void __launch_bounds__(RANK_BS) k_rank(const uint64_t *keys, int n, int share, uint32_t *rank) {
  __shared__ ulonglong2 sk[RANK_BS / 2];
  const int i = blockIdx.x * RANK_BS + threadIdx.x;
  const uint64_t k = i < n ? keys[i] : 0;
  const int j1 = min(n, ((int)blockIdx.y + 1) * share);
  uint32_t below = 0;
  for (int j0 = blockIdx.y * share; j0 < j1; j0 += RANK_BS) {
    __syncthreads();
    ((uint64_t *)sk)[threadIdx.x] = j0 + (int)threadIdx.x < j1 ? keys[j0 + threadIdx.x] : ~0ull;
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < RANK_BS / 2; j++) below += (sk[j].x < k) + (sk[j].y < k);
  }
  if (i < n && below) atomicAdd(&rank[i], below);
}
// (rank starts at zero; blocks to fill the SMs, eight each)
static int rank_keys(const uint64_t *keys, int n, uint32_t *rank, cudaStream_t st) {
  const unsigned nb = fmm_blocks(std::max(n, 1), RANK_BS), shares = std::max(1u, std::min(nb, 1216u / nb));
  const int share = (int)((nb + shares - 1) / shares) * RANK_BS;
  fmm_note_launch(), k_rank<<<dim3(nb, (nb * RANK_BS + share - 1) / share), RANK_BS, 0, st>>>(keys, n, share, rank);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

// The particles of a small system in key order.  Up to KEY_RANK_MAX of them are
// ranked by counting, their index in the key's free low bits breaking the ties: one
// launch of n^2 comparisons where the radix sort's twelve launches, with few blocks,
// wait for one another (10^4 particles: 100 -> 24 us; at the limit the comparisons take
// some 30 us).
constexpr long KEY_RANK_MAX = 16384;
static_assert(3 * (FMM_MAXLEVEL - FMM_KEYLEVELS) >= 14, "free bits for the index");
__global__ void k_key_index(long N, uint64_t *keys, uint32_t *rank) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  keys[i] |= (uint64_t)i;
  rank[i] = 0;
}
__global__ void k_place(const double *__restrict__ pos, const uint64_t *keys, const uint32_t *rank, long N,
                        uint64_t *kout, uint32_t *perm, double *px, double *py, double *pz) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const uint32_t r = rank[i];
  kout[r] = keys[i] & ~(uint64_t)(KEY_RANK_MAX - 1);
  perm[r] = (uint32_t)i;
  px[r] = pos[3 * i];
  py[r] = pos[3 * i + 1];
  pz[r] = pos[3 * i + 2];
}

__global__ void k_gather_pos(const double *__restrict__ pos, const uint32_t *perm, long N, double *px,
                             double *py, double *pz) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  uint32_t j = perm[i];
  px[i] = pos[3 * (size_t)j];
  py[i] = pos[3 * (size_t)j + 1];
  pz[i] = pos[3 * (size_t)j + 2];
}

// ---------------------------------------------------------------------------
// level-by-level cell construction
// ---------------------------------------------------------------------------
__device__ __forceinline__ int digit_at(uint64_t key, int level /*1..21*/) {
  return (int)((key >> (3 * (FMM_MAXLEVEL - level))) & 7u);
}
// first index in [lo, hi) whose level-`level` digit is >= d (digits are sorted there)
__device__ __forceinline__ int lower_digit(const uint64_t *keys, int lo, int hi, int level, int d) {
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (digit_at(keys[mid], level) < d) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// half-width r of a cell, its rmax = sqrt(3 r r) as the reference computes it
// (example/tree.cpp:15), and r as an FP32 (hi, lo) pair
__device__ __forceinline__ void set_radius(int c, double r, double *cr, double *crmax, float2 *crf) {
  cr[c] = r;
  crmax[c] = __dsqrt_rn(__dmul_rn(__dmul_rn(3.0, r), r));
  const float hi = (float)r;
  crf[c] = make_float2(hi, (float)(r - (double)hi));
}

// Level 0: one root cell per system; in sorted order system s holds the
// particles [sys_off[s], sys_off[s + 1]).
__global__ void k_init_roots(int nsys, const double *roots, const long *sys_off, double *cx, double *cy,
                             double *cz, uint64_t *cid, int *ix, int *iy, int *iz, int *pstart, int *pcount,
                             int *parent, int *child_first, unsigned char *child_mask, unsigned char *clevel,
                             double *cr, double *crmax, float2 *crf, int *csys) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const double *rt = roots + 4 * s;
  cx[s] = rt[0]; cy[s] = rt[1]; cz[s] = rt[2];
  cid[s] = 1; ix[s] = iy[s] = iz[s] = 0;
  pstart[s] = (int)sys_off[s]; pcount[s] = (int)(sys_off[s + 1] - sys_off[s]);
  parent[s] = -1; child_first[s] = -1; child_mask[s] = 0; clevel[s] = 0;
  set_radius(s, rt[3], cr, crmax, crf);
  csys[s] = s;
}

// ---------------------------------------------------------------------------
// forests: per-system root cubes (example/tree.cpp:139-187 for each system)
// ---------------------------------------------------------------------------
__global__ void k_fill_psys(const long *sys_off, int *psys) {
  const int s = blockIdx.x;
  for (long i = sys_off[s] + threadIdx.x; i < sys_off[s + 1]; i += blockDim.x) psys[i] = s;
}
// max |x - mean| per system and axis (order-independent), one block per system
__global__ void k_seg_absmax(const double *pos, const long *sys_off, const double *sums, unsigned long long *mx) {
  const int s = blockIdx.x;
  const long b = sys_off[s], e = sys_off[s + 1];
  const double n = (double)(e - b);
  const double ax = __ddiv_rn(sums[3 * s], n), ay = __ddiv_rn(sums[3 * s + 1], n), az = __ddiv_rn(sums[3 * s + 2], n);
  double m0 = 0, m1 = 0, m2 = 0;
  for (long i = b + threadIdx.x; i < e; i += blockDim.x) {
    m0 = fmax(m0, fabs(__dsub_rn(pos[3 * i], ax)));
    m1 = fmax(m1, fabs(__dsub_rn(pos[3 * i + 1], ay)));
    m2 = fmax(m2, fabs(__dsub_rn(pos[3 * i + 2], az)));
  }
  for (int d = 16; d; d >>= 1) {
    m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, d));
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, d));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, d));
  }
  if ((threadIdx.x & 31) == 0) {
    // non-negative doubles order like their bit patterns
    atomicMax(&mx[3 * s], (unsigned long long)__double_as_longlong(m0));
    atomicMax(&mx[3 * s + 1], (unsigned long long)__double_as_longlong(m1));
    atomicMax(&mx[3 * s + 2], (unsigned long long)__double_as_longlong(m2));
  }
}
__global__ void k_seg_root_final(int nsys, const long *sys_off, const double *sums, const unsigned long long *mx,
                                 double *roots) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const double n = (double)(sys_off[s + 1] - sys_off[s]);
  const double ax = __ddiv_rn(sums[3 * s], n), ay = __ddiv_rn(sums[3 * s + 1], n), az = __ddiv_rn(sums[3 * s + 2], n);
  const double xm = __longlong_as_double((long long)mx[3 * s]);
  const double ym = __longlong_as_double((long long)mx[3 * s + 1]);
  const double zm = __longlong_as_double((long long)mx[3 * s + 2]);
  roots[4 * s] = ax; roots[4 * s + 1] = ay; roots[4 * s + 2] = az;
  roots[4 * s + 3] = __dmul_rn((xm > ym ? (xm > zm ? xm : zm) : (ym > zm ? ym : zm)), 1.001);
}
// sorted position -> system, for the stable sort by system after the key sort
__global__ void k_sorted_sys(const uint32_t *perm, const int *psys, long N, uint32_t *ks, uint32_t *idx) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  ks[i] = (uint32_t)psys[perm[i]];
  idx[i] = (uint32_t)i;
}
__global__ void k_apply_order(const uint32_t *idx, long N, const uint64_t *kin, const uint32_t *pin, uint64_t *kout,
                              uint32_t *pout) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  kout[i] = kin[idx[i]];
  pout[i] = pin[idx[i]];
}

// The walk's margin of a cell, for pairs in which it is the finer cell: FP32
// evaluation error plus a bound on how far FP64 centre rounding can move R relative
// to the cell half-width s (rt: its system's root cube)
__device__ __forceinline__ float cell_margin(const double *rt, double s, double theta) {
  const double cmax = fmax(fmax(fabs(rt[0]), fabs(rt[1])), fabs(rt[2])) + rt[3];
  const double m = 1e-5 + 64.0 * ldexp(1.0, -52) * cmax / s * fmax(1.0, theta);
  return s > 0 && m < 0.01 ? (float)m : 1e30f;  // 1e30: always decide in FP64
}

// All levels of cells, then the leaves, in one cooperative launch: a grid-wide
// barrier stands between the steps of a level, so the host waits once for the
// whole tree instead of once a level.  A block takes a contiguous range of a
// level's cells, eight lanes a cell:
// - lane o (1..7) finds where digit o starts in the cell's sorted keys, so the
//   eight child ranges come from seven searches side by side;
// - after the barrier, the children's places are the counts of the blocks before,
//   added up by every block, and a scan within the block, which keeps the cells of
//   a level in parent order; lane o writes child o.
// When a level does not fit the arrays the kernel stops there; the host grows them
// and starts again at that level.  At the end: the leaves in cell order, the near
// field's units (each leaf's targets in chunks of 32: cell, first target, targets,
// leaf) and the walk's records of the cells.
// With the waits, two kernels and a scan a level, from the roots to the leaves: 10^4
// charges, 4 levels: 155 -> 50 us; 10^6, 5 levels: 245 -> 85 us.
struct CellArrays {
  double *cx, *cy, *cz;
  uint64_t *cid;
  int *ix, *iy, *iz, *pstart, *pcount, *parent, *child_first;
  unsigned char *mask, *clevel;
  double *cr, *crmax;
  float2 *crf;
  int *csys, *leaf_cells, *cell_leaf;
  int4 *walk;  // the walk's record, [2]
  int4 *units;
  int *bnd;  // [8] per cell of a level: first particle of each child
  size_t cap;
};
struct CellState {
  double root[4];                     // system 0's
  int lo, hi, level;                  // the last level's cells
  int full;                           // cells that the next level would have needed
  uint32_t nleaves, nunits, eflags, pad;
  int off[FMM_MAXLEVEL + 3];          // first cell of each level reached in this launch
};
constexpr int CELL_BS = 1024, CELL_GROUPS = CELL_BS / 8;

// sum over the block; over the blocks before this one, and over all
__device__ __forceinline__ uint64_t block_sum(uint64_t v) {
  uint64_t tot;
  block_exclusive<uint64_t>(v, &tot);
  return tot;
}
__device__ __forceinline__ uint64_t blocks_before(const uint64_t *gsum, uint64_t *total) {
  uint64_t pre = 0, all = 0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
    const uint64_t v = __ldcg(&gsum[i]);
    all += v;
    if (i < blockIdx.x) pre += v;
  }
  *total = block_sum(all);
  return block_sum(pre);
}

__global__ void __launch_bounds__(CELL_BS) k_build_cells(CellArrays C, CellState *S, int lo, int hi, int level,
                                                         int nlev, long ncrit, const uint64_t *keys,
                                                         const double *roots, double theta, uint64_t *gsum,
                                                         uint32_t *eflags) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const int g = threadIdx.x >> 3, o = threadIdx.x & 7;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  int full = 0;
  for (;;) {
    const int n = hi - lo, chunk = (n + (int)gridDim.x - 1) / (int)gridDim.x;
    const int c0 = lo + (int)min((long)n, (long)blockIdx.x * chunk), c1 = min(hi, c0 + chunk);
    uint64_t mine = 0;
    for (int cb = c0; cb < c1; cb += CELL_GROUPS) {
      const int c = cb + g;
      int b = 0, e = 0;
      bool split = false;
      if (c < c1) {
        const int cnt = C.pcount[c];
        b = C.pstart[c];
        e = b + cnt;
        split = cnt >= ncrit && level < nlev;
        if (o == 0 && cnt >= ncrit && level >= nlev)  // no digits below: give up, or ask for all levels
          atomicOr(eflags, nlev >= FMM_MAXLEVEL ? FMM_EFLAG_DEPTH : FMM_EFLAG_KEYS);
        if (split && o) b = lower_digit(keys, b, e, level + 1, o);
        C.bnd[8 * (size_t)(c - lo) + o] = b;
      }
      int nb = __shfl_down_sync(0xffffffffu, b, 1, 8);  // child o holds [b, nb)
      if (o == 7) nb = e;
      const unsigned m = (__ballot_sync(0xffffffffu, split && nb > b) >> (threadIdx.x & 24)) & 0xffu;
      if (c < c1 && o == 0) {
        C.mask[c] = (unsigned char)m;
        mine += __popc(m);
      }
    }
    mine = block_sum(mine);
    if (threadIdx.x == 0) gsum[blockIdx.x] = mine;
    grid.sync();
    uint64_t total;
    int run = hi + (int)blocks_before(gsum, &total);
    if (total == 0) break;
    if ((size_t)hi + total > C.cap) {
      full = hi + (int)total;
      break;
    }
    for (int cb = c0; cb < c1; cb += CELL_GROUPS) {
      const int c = cb + g;
      const unsigned m = c < c1 ? C.mask[c] : 0u;
      uint32_t tot;
      uint32_t at = block_exclusive<uint32_t>(o == 0 ? __popc(m) : 0, &tot);
      if (o) at -= __popc(m);
      if (c < c1 && o == 0) C.child_first[c] = m ? run + (int)at : -1;
      if ((m >> o) & 1u) {
        const int j = run + (int)at + __popc(m & ((1u << o) - 1u));
        const double r = __ddiv_rn(C.cr[c], 2.0);  // child half-width = parent r / 2.0 (example/tree.cpp:95)
        const int b = C.bnd[8 * (size_t)(c - lo) + o];
        const int nb = o < 7 ? C.bnd[8 * (size_t)(c - lo) + o + 1] : C.pstart[c] + C.pcount[c];
        // add_child (example/tree.cpp:95-98)
        C.cx[j] = __dadd_rn(C.cx[c], (o & 1) ? r : -r);
        C.cy[j] = __dadd_rn(C.cy[c], (o & 2) ? r : -r);
        C.cz[j] = __dadd_rn(C.cz[c], (o & 4) ? r : -r);
        C.cid[j] = (C.cid[c] << 3) | (uint64_t)o;
        C.ix[j] = 2 * C.ix[c] + (o & 1);
        C.iy[j] = 2 * C.iy[c] + ((o >> 1) & 1);
        C.iz[j] = 2 * C.iz[c] + (o >> 2);
        C.pstart[j] = b;
        C.pcount[j] = nb - b;
        C.parent[j] = c;
        C.child_first[j] = -1;
        C.mask[j] = 0;
        C.clevel[j] = (unsigned char)(level + 1);
        set_radius(j, r, C.cr, C.crmax, C.crf);
        C.csys[j] = C.csys[c];
      }
      run += (int)tot;
    }
    lo = hi;
    hi += (int)total;
    level++;
    if (first) S->off[level + 1] = hi;
    grid.sync();
  }
  if (first) {
    for (int k = 0; k < 4; k++) S->root[k] = roots[k];
    S->lo = lo;
    S->hi = hi;
    S->level = level;
    S->full = full;
    S->eflags = __ldcg(eflags);  // every block's cells are counted
  }
  if (full) return;
  // leaves and units: counted together, the units in the high half
  const int chunk = (hi + (int)gridDim.x - 1) / (int)gridDim.x;
  const int c0 = (int)min((long)hi, (long)blockIdx.x * chunk), c1 = min(hi, c0 + chunk);
  uint64_t mine = 0;
  for (int c = c0 + (int)threadIdx.x; c < c1; c += CELL_BS) {
    const int cnt = C.pcount[c];
    if (cnt < ncrit) mine += 1ull | (uint64_t)((cnt + 31) >> 5) << 32;
  }
  mine = block_sum(mine);
  if (threadIdx.x == 0) gsum[gridDim.x + blockIdx.x] = mine;
  grid.sync();
  uint64_t total;
  uint64_t run = blocks_before(gsum + gridDim.x, &total);
  if (first) {
    S->nleaves = (uint32_t)total;
    S->nunits = (uint32_t)(total >> 32);
  }
  for (int cb = c0; cb < c1; cb += CELL_BS) {
    const int c = cb + (int)threadIdx.x, cnt = c < c1 ? C.pcount[c] : 0;
    const bool leaf = c < c1 && cnt < ncrit;
    uint64_t tot;
    const uint64_t at = run + block_exclusive<uint64_t>(leaf ? 1ull | (uint64_t)((cnt + 31) >> 5) << 32 : 0ull, &tot);
    run += tot;
    if (c >= c1) continue;
    const int ord = leaf ? (int)(uint32_t)at : -1;
    C.cell_leaf[c] = ord;
    const float margin = cell_margin(roots + 4 * (size_t)C.csys[c], C.cr[c], theta);
    C.walk[2 * c] = make_int4(C.ix[c], C.iy[c], C.iz[c], C.clevel[c] | (int)C.mask[c] << 8);
    C.walk[2 * c + 1] = make_int4(C.child_first[c], __float_as_int(margin), 0, 0);
    if (!leaf) continue;
    C.leaf_cells[ord] = c;
    for (int k = 0; 32 * k < cnt; k++) C.units[(at >> 32) + k] = make_int4(c, 32 * k, min(32, cnt - 32 * k), ord);
  }
}

// ---------------------------------------------------------------------------
// dual-tree walk (example/calculate.cpp:81-133), breadth-first
// ---------------------------------------------------------------------------
#define WALK_BS 256
struct WalkCells {
  const int4 *cell;  // per cell, one 32-byte sector: (ix, iy, iz, level + 256 children's mask), (first child, margin)
  const double *cx, *cy, *cz, *crmax;
  float theta2;
};

// The MAC  R*theta > rmax_A + rmax_B  (example/calculate.cpp:93) is first
// evaluated on the exact integer geometry of the two cells (centres on the
// level grid, rmax = sqrt(3)*r_level):  R^2 theta^2 / (rmax_A + rmax_B)^2 =
// |g_A - g_B|^2 theta^2 / (3 (2^(L-lA) + 2^(L-lB))^2)  with g the doubled
// integer coordinates at the finer level L.  Only when that ratio lies within
// `margin` of 1 -- where the rounding of the FP64 centres can matter -- is the
// reference's own FP64 expression evaluated, with the same roundings.
// Returns 0 = M2L, 1 = P2P, 2 = split A, 3 = split B.
__device__ __forceinline__ int walk_decide(const WalkCells &W, int A, int B, const int4 &a, const int4 &b, double theta) {
  const int la = a.w & 255, lb = b.w & 255, L = max(la, lb);
  const int sa = L - la, sb = L - lb;
  // (coordinates below 2^23 are exact in FP32, and the margin holds the rounding of the rest)
  const float gx = (float)(((2 * a.x + 1) << sa) - ((2 * b.x + 1) << sb));
  const float gy = (float)(((2 * a.y + 1) << sa) - ((2 * b.y + 1) << sb));
  const float gz = (float)(((2 * a.z + 1) << sa) - ((2 * b.z + 1) << sb));
  const float base = (float)((1 << sa) + (1 << sb));
  const float rho = (gx * gx + gy * gy + gz * gz) * W.theta2 / (3.f * base * base);
  // the finer cell's band around the boundary
  const float m = __int_as_float(W.cell[2 * (la >= lb ? A : B) + 1].y);
  bool mac;
  if (rho > 1.f + m) mac = true;
  else if (rho < 1.f - m) mac = false;
  else {
    double dx = __dsub_rn(W.cx[A], W.cx[B]);
    double dy = __dsub_rn(W.cy[A], W.cy[B]);
    double dz = __dsub_rn(W.cz[A], W.cz[B]);
    double R = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    double ra = W.crmax[A], rb = W.crmax[B];
    mac = __dmul_rn(R, theta) > __dadd_rn(ra, rb);
  }
  if (mac) return 0;
  const bool leafa = (a.w >> 8) == 0, leafb = (b.w >> 8) == 0;
  if (leafa && leafb) return 1;  // the nleaf >= ncrit leaf-leaf branch is unreachable
  if (leafb || (la <= lb && !leafa)) return 2;  // rmax_A >= rmax_B  <=>  lA <= lB
  return 3;
}

// One level of the walk per launch: every frontier pair gives an M2L pair, a P2P
// pair, or the split cell's children as pairs of the next frontier.  A block
// counts the outputs of WALK_TILE pairs, takes their places with one atomic of each
// kind and writes them, so the order within the lists and the frontier is that in
// which the blocks arrive; what is built from them does not depend on it (the P2P
// lists are sorted, the M2L lists ranked by class).  The sizes stay on the device,
// so WALK_BATCH levels are launched before the host looks at them.  A level whose
// outputs exceed a buffer writes only what fits and the levels after it do
// nothing; the host then grows the buffer and starts again with that level, whose
// frontier is still there.  A level's time is its blocks' chain of loads, barriers
// and atomics (2 or 4 pairs a thread: the same).  Counting, scanning and writing in
// three kernels, with the host waiting at every level, against this: a step of 10^4
// charges 924 -> 803 us, of 10^6 7.94 -> 7.82 ms, of 2x10^6 Plummer dipoles (19 levels)
// 23.2 -> 22.75 ms, of 512 systems 44.8 -> 44.3 ms.
constexpr int WALK_BATCH = 8, WALK_IPT = 2, WALK_TILE = WALK_BS * WALK_IPT;
struct WalkState {
  uint32_t nf[WALK_BATCH + 1];                // frontier pairs of each level of the batch
  uint32_t m2l[WALK_BATCH], p2p[WALK_BATCH];  // its outputs
};
struct WalkOut {
  int *m2l_src, *m2l_tgt, *p2p_tgt, *p2p_src;
  size_t cap_m2l, cap_p2p, cap_f[2];          // cap_f: the frontier written by the batch's even and odd levels
  size_t m2l, p2p;                            // pairs written before this batch
};
// the batch's first frontier; of the whole walk: each system's (root, root) pair
__global__ void k_walk_begin(WalkState *S, uint32_t nf, bool first, int *fa, int *fb) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (first && s < nf) fa[s] = fb[s] = (int)s;
  if (s <= WALK_BATCH) S->nf[s] = s == 0 ? nf : 0;
  if (s < WALK_BATCH) S->m2l[s] = S->p2p[s] = 0;
}
__global__ void __launch_bounds__(WALK_BS) k_walk(WalkCells W, double theta, int lev, WalkState *S, WalkOut O,
                                                  const int *fa, const int *fb, int *na, int *nb) {
  __shared__ uint32_t s_at[3];
  __shared__ uint64_t s_w[WALK_BS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t nf = S->nf[lev];
  size_t m0 = O.m2l, p0 = O.p2p;
  bool over = false;
  for (int j = 0; j < lev; j++) {
    m0 += S->m2l[j];
    p0 += S->p2p[j];
    over |= S->nf[j + 1] > ((j & 1) ? O.cap_f[1] : O.cap_f[0]);
  }
  if (over || m0 > O.cap_m2l || p0 > O.cap_p2p) return;
  const size_t capz = (lev & 1) ? O.cap_f[1] : O.cap_f[0];
  for (size_t t0 = (size_t)blockIdx.x * WALK_TILE; t0 < nf; t0 += (size_t)gridDim.x * WALK_TILE) {
    int A[WALK_IPT], B[WALK_IPT], d[WALK_IPT], nch[WALK_IPT];
    uint64_t c = 0;  // outputs of the three kinds, 21 bits each
#pragma unroll
    for (int q = 0; q < WALK_IPT; q++) {
      const size_t i = t0 + q * WALK_BS + threadIdx.x;
      d[q] = -1;
      if (i < nf) {
        A[q] = fa[i];
        B[q] = fb[i];
        const int4 a = W.cell[2 * A[q]], b = W.cell[2 * B[q]];
        d[q] = walk_decide(W, A[q], B[q], a, b, theta);
        nch[q] = __popc((unsigned)(d[q] == 2 ? a.w : b.w) >> 8);
        c += d[q] == 0 ? 1ull : d[q] == 1 ? 1ull << 21 : (uint64_t)nch[q] << 42;
      }
    }
    uint64_t e = c;  // exclusive over the block
#pragma unroll
    for (int sh = 1; sh < 32; sh <<= 1) {
      const uint64_t v = __shfl_up_sync(0xffffffffu, e, sh);
      if (lane >= sh) e += v;
    }
    if (lane == 31) s_w[w] = e;
    __syncthreads();
    e -= c;
    uint64_t tot = 0;
#pragma unroll
    for (int k = 0; k < WALK_BS / 32; k++) {
      const uint64_t v = s_w[k];
      tot += v;
      if (k < w) e += v;
    }
    if (threadIdx.x < 3) {
      const uint32_t n = (uint32_t)(tot >> (21 * threadIdx.x)) & 0x1fffffu;
      uint32_t *at = threadIdx.x == 0 ? &S->m2l[lev] : threadIdx.x == 1 ? &S->p2p[lev] : &S->nf[lev + 1];
      s_at[threadIdx.x] = n ? atomicAdd(at, n) : 0;
    }
    __syncthreads();
    size_t x = m0 + s_at[0] + ((uint32_t)e & 0x1fffffu), y = p0 + s_at[1] + ((uint32_t)(e >> 21) & 0x1fffffu);
    size_t z = (size_t)s_at[2] + (uint32_t)(e >> 42);
#pragma unroll
    for (int q = 0; q < WALK_IPT; q++) {
      if (d[q] < 0) continue;
      if (d[q] == 0) {
        if (x < O.cap_m2l) {
          O.m2l_src[x] = B[q];
          O.m2l_tgt[x] = A[q];
        }
        x++;
      } else if (d[q] == 1) {
        if (y < O.cap_p2p) {
          O.p2p_tgt[y] = A[q];
          O.p2p_src[y] = B[q];
        }
        y++;
      } else {
        const int ch = W.cell[2 * (d[q] == 2 ? A[q] : B[q]) + 1].x;
        for (int k = 0; k < nch[q]; k++, z++)
          if (z < capz) {
            na[z] = d[q] == 2 ? ch + k : A[q];
            nb[z] = d[q] == 2 ? B[q] : ch + k;
          }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// grouping pairs by target cell
// ---------------------------------------------------------------------------
// sort key of a pair: target in the high bits, then (optionally) its class
template <typename K>
__global__ void k_pair_keys(const int *tgt, const int *cls, long n, int cbits, K *keys) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  K k = (K)(uint32_t)tgt[i] << cbits;
  if (cls) k |= (K)(uint32_t)cls[i];
  keys[i] = k;
}
// CSR offsets of pairs sorted by target (off[c] = first pair of target c,
// off[nc] = n), and the class of each sorted pair from the key's low bits.
template <typename K>
__global__ void k_csr_from_sorted(const K *keys, long n, int cbits, int nc, int *off, int *cls) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i > n) return;
  const int cur = i < n ? (int)(keys[i] >> cbits) : nc;
  const int prev = i > 0 ? (int)(keys[i - 1] >> cbits) : -1;
  for (int c = prev + 1; c <= cur; c++) off[c] = (int)i;
  if (cls && i < n) cls[i] = (int)(keys[i] & (((K)1 << cbits) - 1));
}

// ---------------------------------------------------------------------------
// M2L translation classes
// ---------------------------------------------------------------------------
// A pair (B -> A) with levels lA, lB is, up to the scale of A, fixed by
// (dlev = lB - lA, integer offset of the centres in half-widths of the finer
// level).  Classes are shared across levels.  The class key packs
// (dlev + 64, dx + 2^18, dy + 2^18, dz + 2^18) into 7 + 3 x 19 bits, so keys
// order lexicographically by (dlev, dx, dy, dz); class ids are the ranks of
// the distinct keys in that order.
#define CLS_EMPTY 0xffffffffffffffffull
#define CLS_LIM (1LL << 18)
__device__ __forceinline__ uint64_t pair_key(const int4 a, const int4 b) {  // the walk's records of A and B
  const int la = a.w & 255, lb = b.w & 255;
  const int L = la > lb ? la : lb;
  const int sa = L - la, sb = L - lb;
  const long long dx = ((2LL * a.x + 1) << sa) - ((2LL * b.x + 1) << sb);
  const long long dy = ((2LL * a.y + 1) << sa) - ((2LL * b.y + 1) << sb);
  const long long dz = ((2LL * a.z + 1) << sa) - ((2LL * b.z + 1) << sb);
  if (llabs(dx) >= CLS_LIM || llabs(dy) >= CLS_LIM || llabs(dz) >= CLS_LIM) return CLS_EMPTY;
  return ((uint64_t)(lb - la + 64) << 57) | ((uint64_t)(dx + CLS_LIM) << 38) | ((uint64_t)(dy + CLS_LIM) << 19) |
         (uint64_t)(dz + CLS_LIM);
}
__device__ __forceinline__ void key_decode(uint64_t k, int *key4) {
  key4[0] = (int)(k >> 57) - 64;
  key4[1] = (int)((long long)((k >> 38) & 0x7FFFF) - CLS_LIM);
  key4[2] = (int)((long long)((k >> 19) & 0x7FFFF) - CLS_LIM);
  key4[3] = (int)((long long)(k & 0x7FFFF) - CLS_LIM);
}
// slot sequence of a key in the open-addressing table (splitmix64 finalizer)
__device__ __forceinline__ uint32_t key_hash(uint64_t k) {
  k ^= k >> 30;
  k *= 0xBF58476D1CE4E5B9ull;
  k ^= k >> 27;
  k *= 0x94D049BB133111EBull;
  k ^= k >> 31;
  return (uint32_t)k;
}
__device__ __forceinline__ long key_find(const uint64_t *tab, uint32_t mask, uint64_t k) {
  uint32_t h = key_hash(k) & mask;
  for (uint32_t probe = 0; probe <= mask; probe++) {
    const uint64_t cur = tab[h];
    if (cur == k) return h;
    if (cur == CLS_EMPTY) return -1;
    h = (h + 1) & mask;
  }
  return -1;
}

// Class key of every pair, inserted into the table; stat[0] counts distinct
// keys, stat[1] flags a table that filled up.
__global__ void k_class_keys(const int *src, const int *tgt, long n, const int4 *cell, uint64_t *keys, uint64_t *tab,
                             uint32_t mask, uint32_t *stat, uint32_t *eflags) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = pair_key(cell[2 * tgt[i]], cell[2 * src[i]]);
  keys[i] = k;
  if (k == CLS_EMPTY) {
    atomicOr(eflags, FMM_EFLAG_RANGE);
    return;
  }
  uint32_t h = key_hash(k) & mask;
  for (uint32_t probe = 0; probe <= mask; probe++) {
    uint64_t cur = tab[h];
    if (cur == CLS_EMPTY) {
      cur = atomicCAS((unsigned long long *)&tab[h], CLS_EMPTY, (unsigned long long)k);
      if (cur == CLS_EMPTY) {
        atomicAdd(&stat[0], 1u);
        return;
      }
    }
    if (cur == k) return;
    h = (h + 1) & mask;
  }
  atomicOr(&stat[1], 1u);
}

__global__ void k_class_collect(const uint64_t *tab, uint32_t nslots, uint64_t *uniq, uint32_t *slot,
                                uint32_t *rank, uint32_t *counter) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nslots || tab[s] == CLS_EMPTY) return;
  const uint32_t r = atomicAdd(counter, 1u);
  uniq[r] = tab[s];
  slot[r] = s;
  rank[r] = 0;
}

constexpr uint32_t RANK_MAX = 32768;

// ids by rank (none: the keys are sorted); the class table entry of each key; *same cleared unless the sorted
// keys are the previous build's, which they replace
__global__ void k_class_rank(const uint64_t *uniq, int nu, const uint32_t *slot, const uint32_t *rank, int *tabval,
                             int *key4, uint64_t *prev, uint32_t *same, int wide, uint32_t *eflags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nu) return;
  const uint32_t r = rank ? rank[i] : (uint32_t)i;
  tabval[slot[i]] = (int)r;
  int *k4 = key4 + 4 * (size_t)r;
  key_decode(uniq[i], k4);
  if (abs(k4[0]) > wide) atomicOr(eflags, FMM_EFLAG_WIDE);
  if (prev[r] != uniq[i]) {
    *same = 0;
    prev[r] = uniq[i];
  }
}

__global__ void k_class_lookup(const uint64_t *keys, long n, const uint64_t *tab, uint32_t mask, const int *tabval,
                               int *cls) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long s = keys[i] == CLS_EMPTY ? -1 : key_find(tab, mask, keys[i]);
  cls[i] = s >= 0 ? tabval[s] : 0;  // out-of-range pairs were flagged when their keys were made
}

// Key per cell for the M2L processing order: (level, octant within the
// parent, parent index).  A cell's interaction list depends on which octant of
// its parent it is (the children of the parent's neighbours that pass the MAC),
// so grouping the cells of one level by octant, with parents in Morton order
// (cell indices are Morton order within a level), puts cells with
// near-identical class lists side by side: the 128-cell tiles of the tensor-core
// M2L then visit ~1.4x the classes of one list instead of ~3.5x in plain Morton
// order, and the warps of the CUDA-core M2L read the same operator rows.
// Cells are stored level by level in parent order, so a stable sort on
// (level, octant) alone keeps the parents in Morton order.
// grouping 1 keeps plain Morton order within a level (the key is the level alone).
__global__ void k_order_keys(int nc, const uint64_t *cid, const unsigned char *clevel, int grouping, uint32_t *key,
                             uint32_t *idx) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  key[c] = (uint32_t)clevel[c] << 3 | (grouping == 0 ? (uint32_t)(cid[c] & 7u) : 0u);  // 8 bits: one pass
  idx[c] = (uint32_t)c;
}

// Operator vector of a class: D_k(d / s_A), |k| <= p, in FP64 (one warp per class).
// (skipped when `same` is set: the vectors of the previous build still hold)
__global__ void k_class_derivs(const int *key4, int ncls, int p, double *D64, float *D32, const uint32_t *same) {
  __shared__ double sD[FMM_WARPS][FMM_NTMAX], sT[FMM_WARPS][FMM_NTMAX], sB[FMM_WARPS][FMM_PMAX + 1];
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int c = blockIdx.x * FMM_WARPS + w;
  if (c >= ncls || *same) return;
  int dl = key4[4 * c];
  double sc = dl > 0 ? ldexp(1.0, -dl) : 1.0;  // finer-level half-widths -> half-widths of A
  double x = key4[4 * c + 1] * sc, y = key4[4 * c + 2] * sc, z = key4[4 * c + 3] * sc;
  warp_derivs<double>(x, y, z, p, sD[w], sT[w], sB[w]);
  int nt = fmm_nterms(p);
  for (int i = lane; i < nt; i += 32) {
    D64[(size_t)c * nt + i] = sD[w][i];
    D32[(size_t)c * fmm_stride4(nt) + i] = (float)sD[w][i];
  }
}

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
template <typename T> static int grow_keep(DevBuf<T> &b, size_t need, size_t used, cudaStream_t st) {
  if (need <= b.cap && b.p) return FMM_OK;
  size_t want = need + need / 2 + 64;
  T *p = nullptr;
  FMM_CUDA_TRY(cudaMalloc((void **)&p, want * sizeof(T)));
  if (b.p && used) FMM_CUDA_TRY(cudaMemcpyAsync(p, b.p, used * sizeof(T), cudaMemcpyDeviceToDevice, st));
  if (b.p) {
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    cudaFree(b.p);
  }
  b.p = p;
  b.cap = want;
  return FMM_OK;
}

static int tmp_reserve(DevTree *t, size_t bytes) { return fmm_reserve(t->tmp, bytes); }
static int bits_for(long n);

#define TRY(x) do { int _rc = (x); if (_rc) return _rc; } while (0)

static int rec(DevTree *t, int i, cudaStream_t st) {
  if (!t->ev_ready) return FMM_OK;
  FMM_CUDA_TRY(cudaEventRecord(t->ev[i], st));
  return FMM_OK;
}

static int build_cells(DevTree *t, cudaStream_t st, int nlev, bool *deeper);
static int build_lists(DevTree *t, cudaStream_t st);
static int build_classes(DevTree *t, cudaStream_t st);

int fmm_tree_build(DevTree *t, const double *pos, long N, long ncrit, int order, double theta, int so,
                   cudaStream_t st, const long *sys_off, int nsys, bool defer_classes,
                   int (*after_cells)(DevTree *, void *), void *arg) {
  if (N < 1 || N >= (1L << 31) - 1 || ncrit < 1 || order < so + 1 || order > FMM_PMAX || so < 0 || so > 2 ||
      !(theta > 0) || !pos || nsys < 1 || (nsys > 1 && !sys_off))
    return FMM_ERR_ARG;
  if (sys_off) {
    if (sys_off[0] != 0 || sys_off[nsys] != N) return FMM_ERR_ARG;
    for (int k = 0; k < nsys; k++)
      if (sys_off[k + 1] <= sys_off[k]) return FMM_ERR_ARG;  // every system holds particles
  }
  t->N = N; t->ncrit = ncrit; t->order = order; t->so = so; t->theta = theta;
  t->nsys = nsys;
  if (sys_off) t->sys_off_h.assign(sys_off, sys_off + nsys + 1);
  else t->sys_off_h = {0, N};
  FMM_CUDA_TRY(cudaGetDevice(&t->dev));
  if (!t->ev_ready) {
    for (int i = 0; i < 16; i++) FMM_CUDA_TRY(cudaEventCreate(&t->ev[i]));
    for (int i = 0; i < 4; i++) FMM_CUDA_TRY(cudaEventCreate(&t->ev_mk[i]));
    t->ev_ready = true;
  }
  if (!t->h_pinned) {
    FMM_CUDA_TRY(cudaMallocHost((void **)&t->h_pinned, 4 * FMM_PINNED_WORDS));
    memset(t->h_pinned, 0, 4 * FMM_PINNED_WORDS);
  }
  t->build_serial++;
  TRY(rec(t, 0, st));
  TRY(fmm_reserve(t->d_eflags, 4));
  FMM_CUDA_TRY(cudaMemsetAsync(t->d_eflags.p, 0, sizeof(uint32_t), st));
  TRY(fmm_reserve(t->sys_off, (size_t)nsys + 1));
  FMM_CUDA_TRY(cudaMemcpyAsync(t->sys_off.p, t->sys_off_h.data(), sizeof(long) * (nsys + 1),
                               cudaMemcpyHostToDevice, st));
  TRY(fmm_reserve(t->roots, 4 * (size_t)nsys));
  // d_root: [0..2] sums, [3..5] maxima (u64 bits), [6..9] root box, [16..] level r/rmax
  TRY(fmm_reserve(t->d_root, 16 + 2 * (FMM_MAXLEVEL + 1)));
  double *dr = t->d_root.p;
  if (nsys == 1) {
    // one system: the exact sequential mean through fmm_seqsum3 (parallel)
    FMM_CUDA_TRY(cudaMemsetAsync(dr, 0, sizeof(double) * 16, st));
    TRY(tmp_reserve(t, fmm_seqsum_scratch_tables(fmm_seqsum_chunks(N))));
    TRY(fmm_seqsum3(pos, N, dr, t->tmp.p, true, st));
    unsigned nbm = std::min<unsigned>(fmm_blocks(N, 256), 152 * 8);
    fmm_note_launch(), k_root_absmax<<<nbm, 256, 0, st>>>(pos, N, dr, (unsigned long long *)(dr + 3));
    TRY(fmm_reserve(t->levf, FMM_MAXLEVEL + 1));
    fmm_note_launch(), k_root_final<<<1, 32, 0, st>>>(dr, (const unsigned long long *)(dr + 3), N, t->roots.p,
                                                     dr + 16, t->levf.p);
  } else {
    // a forest: each system's exact sequential means, side by side
    TRY(fmm_reserve(t->psys, N));
    fmm_note_launch(), k_fill_psys<<<nsys, 256, 0, st>>>(t->sys_off.p, t->psys.p);
    std::vector<int> co(nsys + 1, 0);
    for (int k = 0; k < nsys; k++) co[k + 1] = co[k] + (int)fmm_seqsum_chunks(sys_off[k + 1] - sys_off[k]);
    const size_t head = (sizeof(double) * 6 * (size_t)nsys + sizeof(int) * (nsys + 1) + 255) & ~(size_t)255;
    TRY(tmp_reserve(t, head + fmm_seqsum_scratch_tables(co[nsys])));
    double *sums = (double *)t->tmp.p;
    int *chunk_off = (int *)(sums + 6 * (size_t)nsys);
    FMM_CUDA_TRY(cudaMemcpyAsync(chunk_off, co.data(), sizeof(int) * (nsys + 1), cudaMemcpyHostToDevice, st));
    unsigned long long *mx = (unsigned long long *)(sums + 3 * (size_t)nsys);
    FMM_CUDA_TRY(cudaMemsetAsync(mx, 0, sizeof(unsigned long long) * 3 * nsys, st));
    TRY(fmm_seqsum3_systems(pos, t->sys_off.p, chunk_off, nsys, co[nsys], sums, t->tmp.p + head, st));
    fmm_note_launch(), k_seg_absmax<<<nsys, 256, 0, st>>>(pos, t->sys_off.p, sums, mx);
    fmm_note_launch(), k_seg_root_final<<<fmm_blocks(nsys, 128), 128, 0, st>>>(nsys, t->sys_off.p, sums, mx,
                                                                                t->roots.p);
  }
  FMM_CUDA_TRY(cudaGetLastError());
  TRY(rec(t, 1, st));

  // keys + stable sort, then the cells; the keys hold the digits of the first
  // FMM_KEYLEVELS levels unless a tree that deep needs more (then all of them)
  TRY(fmm_reserve(t->keys, N)); TRY(fmm_reserve(t->keys2, N));
  TRY(fmm_reserve(t->perm, N)); TRY(fmm_reserve(t->perm2, N));
  for (int nlev = FMM_KEYLEVELS;; nlev = FMM_MAXLEVEL) {
    fmm_note_launch(), k_keys<<<fmm_blocks(N, 256), 256, 0, st>>>(pos, N, t->roots.p, nsys > 1 ? t->psys.p : nullptr,
                                                                   nlev, t->keys.p, t->perm.p);
    FMM_CUDA_TRY(cudaGetLastError());
    TRY(fmm_reserve(t->px, N)); TRY(fmm_reserve(t->py, N)); TRY(fmm_reserve(t->pz, N));
    if (nsys == 1 && N <= KEY_RANK_MAX && nlev == FMM_KEYLEVELS) {
      fmm_note_launch(), k_key_index<<<fmm_blocks(N, 256), 256, 0, st>>>(N, t->keys.p, t->perm2.p);
      TRY(rank_keys(t->keys.p, (int)N, t->perm2.p, st));
      fmm_note_launch(), k_place<<<fmm_blocks(N, 256), 256, 0, st>>>(pos, t->keys.p, t->perm2.p, N, t->keys2.p,
                                                                     t->perm.p, t->px.p, t->py.p, t->pz.p);
      FMM_CUDA_TRY(cudaGetLastError());
      std::swap(t->keys, t->keys2);
    } else {
      size_t nbh = fmm_rs_nblocks(N);
      size_t hist_n = 256 * nbh;
      const size_t sort_bytes = hist_n * 4 + fmm_scan_tmp_elems<uint32_t>(hist_n) * 4 + 1024;
      TRY(tmp_reserve(t, sort_bytes + (nsys > 1 ? 16 * (size_t)N : 0)));
      uint32_t *hist = (uint32_t *)t->tmp.p;
      uint32_t *scantmp = hist + hist_n;
      TRY(fmm_radix_sort(t->keys.p, t->perm.p, t->keys2.p, t->perm2.p, N, 3 * (FMM_MAXLEVEL - nlev),
                         3 * FMM_MAXLEVEL, hist, scantmp, st));
      if (nsys > 1) {
        // stable sort by system: (system, key) order, each system's particles contiguous
        uint32_t *ks = (uint32_t *)(t->tmp.p + sort_bytes);
        uint32_t *idx = ks + N, *ks2 = idx + N, *idx2 = ks2 + N;
        fmm_note_launch(), k_sorted_sys<<<fmm_blocks(N, 256), 256, 0, st>>>(t->perm.p, t->psys.p, N, ks, idx);
        TRY(fmm_radix_sort<uint32_t>(ks, idx, ks2, idx2, N, 0, bits_for(nsys), hist, scantmp, st));
        fmm_note_launch(), k_apply_order<<<fmm_blocks(N, 256), 256, 0, st>>>(idx, N, t->keys.p, t->perm.p,
                                                                             t->keys2.p, t->perm2.p);
        FMM_CUDA_TRY(cudaGetLastError());
        std::swap(t->keys, t->keys2);
        std::swap(t->perm, t->perm2);
      }
      fmm_note_launch(), k_gather_pos<<<fmm_blocks(N, 256), 256, 0, st>>>(pos, t->perm.p, N, t->px.p, t->py.p,
                                                                           t->pz.p);
      FMM_CUDA_TRY(cudaGetLastError());
    }
    TRY(rec(t, 2, st));
    bool deeper = false;
    TRY(build_cells(t, st, nlev, &deeper));
    if (!deeper) break;
  }
  TRY(rec(t, 3, st));
  if (after_cells) TRY(after_cells(t, arg));  // work that needs the cells only, beside the walk
  TRY(build_lists(t, st));
  TRY(rec(t, 4, st));
  return defer_classes ? FMM_OK : fmm_tree_finish_build(t, st);
}

// The M2L translation classes and the end of the build (fmm_tree_build with
// defer_classes leaves them to this call).
int fmm_tree_finish_build(DevTree *t, cudaStream_t st) {
  TRY(build_classes(t, st));
  if (!(t->eflags & FMM_EFLAG_DEPTH)) TRY(fmm_p2p_prepare(t, st));
  TRY(rec(t, 5, st));
  FMM_CUDA_TRY(cudaMemcpyAsync(&t->eflags, t->d_eflags.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  FMM_CUDA_TRY(cudaStreamSynchronize(st));
  if (t->ev_ready) {
    float ms;
    for (int i = 0; i < 5; i++) {
      cudaEventElapsedTime(&ms, t->ev[i], t->ev[i + 1]);
      t->build_ms[i] = ms;
    }
    cudaEventElapsedTime(&ms, t->ev[0], t->ev[5]);
    t->build_ms[5] = ms;
  }
  if (t->eflags & FMM_EFLAG_DEPTH) return FMM_ERR_DEPTH;
  if (t->eflags & FMM_EFLAG_RANGE) return FMM_ERR_RANGE;
  return FMM_OK;
}

// Cells level by level from keys holding nlev levels of digits; *deeper is set
// (and the error flag cleared) when a cell at level nlev would need the next.
static int build_cells(DevTree *t, cudaStream_t st, int nlev, bool *deeper) {
  long N = t->N;
  const int nsys = t->nsys;
  size_t cap = (size_t)(4 * N / std::max<long>(t->ncrit, 1)) + 1024 + nsys;
  TRY(fmm_reserve(t->cx, cap)); TRY(fmm_reserve(t->cy, cap)); TRY(fmm_reserve(t->cz, cap));
  TRY(fmm_reserve(t->cid, cap)); TRY(fmm_reserve(t->ix, cap)); TRY(fmm_reserve(t->iy, cap));
  TRY(fmm_reserve(t->iz, cap)); TRY(fmm_reserve(t->pstart, cap)); TRY(fmm_reserve(t->pcount, cap));
  TRY(fmm_reserve(t->parent, cap)); TRY(fmm_reserve(t->child_first, cap));
  TRY(fmm_reserve(t->child_mask, cap)); TRY(fmm_reserve(t->clevel, cap));
  TRY(fmm_reserve(t->cr, cap)); TRY(fmm_reserve(t->crmax, cap)); TRY(fmm_reserve(t->crf, cap));
  TRY(fmm_reserve(t->csys, cap));
  fmm_note_launch(), k_init_roots<<<fmm_blocks(nsys, 128), 128, 0, st>>>(
      nsys, t->roots.p, t->sys_off.p, t->cx.p, t->cy.p, t->cz.p, t->cid.p, t->ix.p, t->iy.p, t->iz.p, t->pstart.p,
      t->pcount.p, t->parent.p, t->child_first.p, t->child_mask.p, t->clevel.p, t->cr.p, t->crmax.p, t->crf.p,
      t->csys.p);
  FMM_CUDA_TRY(cudaGetLastError());
  int sms = 0, level = 0, lo = 0, hi = nsys;
  FMM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t->dev));
  // 16 cells a block at least: a grid of all SMs has the slower barrier
  const unsigned nblk = (unsigned)std::min<size_t>(sms, (cap - 1024) / 16 + 1);
  const size_t head = ((sizeof(CellState) + 255) & ~(size_t)255) + 16 * (size_t)nblk;
  CellState *H = (CellState *)(t->h_pinned + FMM_PINNED_WALK);
  static_assert(sizeof(CellState) <= 4 * (FMM_PINNED_WORDS - FMM_PINNED_WALK), "pinned words");
  t->level_off.assign(1, 0);
  t->level_off.push_back(nsys);
  for (;;) {
    size_t room = std::min({t->cx.cap, t->cy.cap, t->cz.cap, t->cid.cap, t->ix.cap, t->iy.cap, t->iz.cap, t->pstart.cap,
                            t->pcount.cap, t->parent.cap, t->child_first.cap, t->child_mask.cap, t->clevel.cap,
                            t->cr.cap, t->crmax.cap, t->crf.cap, t->csys.cap});
    TRY(fmm_reserve(t->leaf_cells, room)); TRY(fmm_reserve(t->cell_leaf, room)); TRY(fmm_reserve(t->wcell, 2 * room));
    TRY(fmm_reserve(t->p2p_units, room + (size_t)(N / 32) + 1));
    TRY(tmp_reserve(t, head + 32 * room));
    CellState *S = (CellState *)t->tmp.p;
    uint64_t *gsum = (uint64_t *)(t->tmp.p + head) - 2 * (size_t)nblk;
    CellArrays C = {t->cx.p, t->cy.p, t->cz.p, t->cid.p, t->ix.p, t->iy.p, t->iz.p, t->pstart.p, t->pcount.p,
                    t->parent.p, t->child_first.p, t->child_mask.p, t->clevel.p, t->cr.p, t->crmax.p, t->crf.p,
                    t->csys.p, t->leaf_cells.p, t->cell_leaf.p, t->wcell.p, t->p2p_units.p, (int *)(t->tmp.p + head),
                    room};
    const uint64_t *keys = t->keys.p;
    const double *roots = t->roots.p;
    uint32_t *eflags = t->d_eflags.p;
    void *args[] = {&C, &S, &lo, &hi, &level, &nlev, &t->ncrit, &keys, &roots, &t->theta, &gsum, &eflags};
    fmm_note_launch();
    FMM_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_build_cells, dim3(nblk), dim3(CELL_BS), args, 0, st));
    FMM_CUDA_TRY(cudaMemcpyAsync(H, S, sizeof(CellState), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    for (int l = level + 1; l <= H->level; l++) t->level_off.push_back(H->off[l + 1]);
    lo = H->lo;
    hi = H->hi;
    level = H->level;
    if (!H->full) break;
    const size_t need = H->full, used = hi;
    TRY(grow_keep(t->cx, need, used, st)); TRY(grow_keep(t->cy, need, used, st)); TRY(grow_keep(t->cz, need, used, st));
    TRY(grow_keep(t->cid, need, used, st)); TRY(grow_keep(t->ix, need, used, st)); TRY(grow_keep(t->iy, need, used, st));
    TRY(grow_keep(t->iz, need, used, st)); TRY(grow_keep(t->pstart, need, used, st));
    TRY(grow_keep(t->pcount, need, used, st)); TRY(grow_keep(t->parent, need, used, st));
    TRY(grow_keep(t->child_first, need, used, st)); TRY(grow_keep(t->child_mask, need, used, st));
    TRY(grow_keep(t->clevel, need, used, st)); TRY(grow_keep(t->cr, need, used, st));
    TRY(grow_keep(t->crmax, need, used, st)); TRY(grow_keep(t->crf, need, used, st));
    TRY(grow_keep(t->csys, need, used, st));
  }
  memcpy(&t->root, H->root, sizeof(t->root));
  t->ncells = hi;
  t->nlevels = level + 1;
  t->nleaves = (int)H->nleaves;
  t->np2p_units = (int)H->nunits;
  t->eflags = H->eflags;
  if (H->eflags & FMM_EFLAG_KEYS) {
    *deeper = true;
    FMM_CUDA_TRY(cudaMemsetAsync(t->d_eflags.p, 0, sizeof(uint32_t), st));
  }
  return FMM_OK;
}

static int bits_for(long n) {  // bits that hold the values 0..n-1
  int b = 0;
  while ((1L << b) < n) b++;
  return b;
}

template <typename K>
static int sort_pairs(DevTree *t, const int *tgt, const int *cls, int cbits, int end_bit, DevBuf<int> &src_raw,
                      long n, DevBuf<int> &off, int *cls_out, cudaStream_t st) {
  size_t nbh = fmm_rs_nblocks(n);
  size_t hist_n = 256 * nbh;
  size_t bytes = (size_t)n * (2 * sizeof(K) + 4) + hist_n * 4 + fmm_scan_tmp_elems<uint32_t>(hist_n) * 4 + 256;
  TRY(tmp_reserve(t, bytes));
  char *p = t->tmp.p;
  K *k1 = (K *)p; p += (size_t)n * sizeof(K);
  K *k2 = (K *)p; p += (size_t)n * sizeof(K);
  uint32_t *v2 = (uint32_t *)p; p += (size_t)n * 4;
  uint32_t *hist = (uint32_t *)p; p += hist_n * 4;
  uint32_t *stmp = (uint32_t *)p;
  fmm_note_launch(), k_pair_keys<K><<<fmm_blocks(n, 256), 256, 0, st>>>(tgt, cls, n, cbits, k1);
  FMM_CUDA_TRY(cudaGetLastError());
  TRY(fmm_radix_sort<K>(k1, (uint32_t *)src_raw.p, k2, v2, n, 0, end_bit, hist, stmp, st));
  fmm_note_launch(), k_csr_from_sorted<K><<<fmm_blocks(n + 1, 256), 256, 0, st>>>(k1, n, cbits, t->ncells, off.p,
                                                                                 cls_out);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

__global__ void k_csr_count(const int *tgt, long n, int *cnt);

// The near-field lists: pairs counted per target, put into their target's range
// in any order (one atomic per run of equal targets in a warp), and each list
// sorted by source, which makes it the same in every build whatever the order of
// the walk's output; k_p2p_sort also sums up the interaction count, a statistic
// that is read when asked for (fmm_p2p_interactions).
__global__ void k_p2p_scatter(const int *tgt, const int *src, long n, int *cur, int *list) {
  const long i = blockIdx.x * 256l + threadIdx.x;
  const int t = i < n ? tgt[i] : -1, lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xffffffffu, t);
  const int lead = __ffs(same) - 1;
  int base = 0;
  if (t >= 0 && lead == lane) base = atomicAdd(&cur[t], __popc(same));
  base = __shfl_sync(0xffffffffu, base, lead);
  if (t >= 0) list[base + __popc(same & ((1u << lane) - 1u))] = src[i];
}

// Ascending bitonic sort of a[0..n) by one warp, any n: each merge begins with
// the mirrored comparison, so that the places past n, as if infinite, never move.
__device__ __forceinline__ void warp_sort(int *a, int n) {
  const int lane = threadIdx.x & 31;
  int lp = 0;
  while ((1 << lp) < n) lp++;
  const int half = lp ? 1 << (lp - 1) : 0;  // comparisons of a step
  for (int lk = 1; lk <= lp; lk++)
    for (int ld = lk - 1; ld >= 0; ld--) {
      for (int q = lane; q < half; q += 32) {
        const int off = q & ((1 << ld) - 1), blk = (q >> ld) << (ld + 1);
        const int i = blk + off, j = ld == lk - 1 ? blk + (1 << lk) - 1 - off : i + (1 << ld);
        if (j < n) {
          const int x = a[i], y = a[j];
          if (x > y) {
            a[i] = y;
            a[j] = x;
          }
        }
      }
      __syncwarp();
    }
}
// The same network on 32 R values in registers (value 32 r + lane in v[r]).
template <int R> __device__ __forceinline__ void warp_sort_regs(int (&v)[R]) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  auto cross = [&](int x, int m, bool low) {
    const int y = __shfl_xor_sync(FULL, x, m);
    return low ? min(x, y) : max(x, y);
  };
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = cross(v[r], k - 1, !(lane & (k >> 1)));
#pragma unroll
    for (int d = k >> 2; d; d >>= 1)
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = cross(v[r], d, !(lane & d));
  }
#pragma unroll
  for (int k = 2; k <= R; k <<= 1) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int q = r ^ (k - 1);
      if (q > r) {
        const int x = __shfl_xor_sync(FULL, v[r], 31), y = __shfl_xor_sync(FULL, v[q], 31);
        v[r] = min(v[r], y);
        v[q] = max(v[q], x);
      }
    }
#pragma unroll
    for (int d = k >> 2; d; d >>= 1)
#pragma unroll
      for (int r = 0; r < R; r++)
        if (!(r & d)) {
          const int x = v[r];
          v[r] = min(x, v[r ^ d]);
          v[r ^ d] = max(x, v[r ^ d]);
        }
#pragma unroll
    for (int d = 16; d; d >>= 1)
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = cross(v[r], d, !(lane & d));
  }
}
// One target's list of n <= 32 R sources; the sum of their particles.
template <int R> __device__ __forceinline__ unsigned long long p2p_sort_regs(int *list, int n, const int *pcount) {
  const int lane = threadIdx.x & 31;
  int v[R];
  unsigned long long s = 0;
#pragma unroll
  for (int r = 0; r < R; r++) {
    v[r] = 32 * r + lane < n ? list[32 * r + lane] : 0x7fffffff;
    s += 32 * r + lane < n ? pcount[v[r]] : 0;
  }
  warp_sort_regs<R>(v);
#pragma unroll
  for (int r = 0; r < R; r++)
    if (32 * r + lane < n) list[32 * r + lane] = v[r];
  return s;
}
// Up to 256 sources in registers, up to PSORT_SMEM in shared memory, more in
// place.  5.1M pairs in lists of 156 (10^6 charges): 35 us, and 47 for the count and
// the scatter; the radix sort of (target, source) pairs, stable in the walk's
// order, took 170.  66M pairs in lists of 125 (512 systems): 1.42 ms in shared
// memory, a step 0.8 ms less in registers.
constexpr int PSORT_WARPS = 4, PSORT_SMEM = 1024;
__global__ void __launch_bounds__(32 * PSORT_WARPS) k_p2p_sort(const int *off, int nc, const int *pcount, int *list,
                                                               unsigned long long *interactions) {
  __shared__ int sm[PSORT_WARPS][PSORT_SMEM];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * PSORT_WARPS + w;
  if (c >= nc) return;
  const int k0 = off[c], n = off[c + 1] - k0;
  if (n == 0) return;
  unsigned long long s = 0;
  if (n <= 128) {
    s = p2p_sort_regs<4>(list + k0, n, pcount);
  } else if (n <= 256) {
    s = p2p_sort_regs<8>(list + k0, n, pcount);
  } else {
    const bool here = n <= PSORT_SMEM;
    int *a = here ? sm[w] : list + k0;
    for (int k = lane; k < n; k += 32) {
      const int b = list[k0 + k];
      if (here) a[k] = b;
      s += pcount[b];
    }
    __syncwarp();
    warp_sort(a, n);
    if (here)
      for (int k = lane; k < n; k += 32) list[k0 + k] = a[k];
  }
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  // a leaf's list holds itself, without the particles' own pairs
  if (lane == 0) atomicAdd(interactions, (unsigned long long)pcount[c] * (s - 1));
}

static int p2p_lists(DevTree *t, cudaStream_t st) {
  const int nc = t->ncells;
  const long n = t->np2p;
  TRY(fmm_reserve(t->p2p_off, (size_t)nc + 1));
  TRY(fmm_reserve(t->p2p_src, std::max(n, 1L)));
  TRY(fmm_reserve(t->d_p2pcount, 1));
  FMM_CUDA_TRY(cudaMemsetAsync(t->d_p2pcount.p, 0, sizeof(unsigned long long), st));
  t->p2p_count_serial = t->build_serial;
  if (n == 0) {
    FMM_CUDA_TRY(cudaMemsetAsync(t->p2p_off.p, 0, sizeof(int) * ((size_t)nc + 1), st));
    return FMM_OK;
  }
  TRY(tmp_reserve(t, sizeof(int) * ((size_t)nc + fmm_scan_tmp_elems<int>(nc))));
  int *cur = (int *)t->tmp.p, *stmp = cur + nc;
  FMM_CUDA_TRY(cudaMemsetAsync(cur, 0, sizeof(int) * nc, st));
  fmm_note_launch(), k_csr_count<<<fmm_blocks(n, 256), 256, 0, st>>>(t->p2p_tgt_raw.p, n, cur);
  TRY(fmm_scan<int>(cur, t->p2p_off.p, nc, t->p2p_off.p + nc, stmp, st));
  FMM_CUDA_TRY(cudaMemcpyAsync(cur, t->p2p_off.p, sizeof(int) * nc, cudaMemcpyDeviceToDevice, st));
  fmm_note_launch(), k_p2p_scatter<<<fmm_blocks(n, 256), 256, 0, st>>>(t->p2p_tgt_raw.p, t->p2p_src_raw.p, n, cur,
                                                                       t->p2p_src.p);
  fmm_note_launch(), k_p2p_sort<<<fmm_blocks(nc, PSORT_WARPS), 32 * PSORT_WARPS, 0, st>>>(
      t->p2p_off.p, nc, t->pcount.p, t->p2p_src.p, t->d_p2pcount.p);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

// blocks that fill the SMs, eight of 256 threads each
constexpr size_t WALK_GRID = 152 * 8;
static int build_lists(DevTree *t, cudaStream_t st) {
  const int nc = t->ncells;
  const WalkCells W{t->wcell.p, t->cx.p, t->cy.p, t->cz.p, t->crmax.p, (float)(t->theta * t->theta)};
  // raw lists in the walk's order; the buffers keep their capacity between
  // builds, so a rebuild of a similar tree allocates nothing.  At first what lists
  // are about: up to 480 M2L and 160 P2P sources a cell for theta <= 0.5 (10^6 uniform
  // charges 419 and 136), shorter with the cube of it, in systems of few cells at
  // most four times their number, and no more than an eighth of the free memory;
  // else 64.  A level that does not fit is walked again with room for it.  (64 for
  // every tree: first builds of 10^6 charges 3.4 -> 4.2 ms, of 512 systems 11.0 -> 16.4.)
  DevBuf<int> &m2l_src_raw = t->m2l_src_raw, &m2l_tgt_raw = t->m2l_tgt_raw;
  DevBuf<int> &p2p_tgt_raw = t->p2p_tgt_raw, &p2p_src_raw = t->p2p_src_raw;
  // the frontiers: in the lists that are made from the walk's output afterwards
  DevBuf<int> *fr[2][2] = {{&t->m2l_src, &t->m2l_cls}, {&t->m2l_cls_raw, &t->front}};
  TRY(fmm_reserve(t->d_walk, sizeof(WalkState)));
  WalkState *S = (WalkState *)t->d_walk.p, *H = (WalkState *)(t->h_pinned + FMM_PINNED_WALK);
  const double shorter = std::min(1.0, 0.125 / (t->theta * t->theta * t->theta)), few = 4.0 * nc / t->nsys;
  auto about = [&](double a_cell) { return (size_t)(std::min(std::max(64.0, a_cell * shorter), few) * nc) + 1024 + t->nsys; };
  auto room = [&](size_t m2l, size_t p2p, size_t f) {
    for (auto &b : fr)
      for (DevBuf<int> *q : b)
        if (fmm_reserve(*q, f)) return FMM_ERR_CUDA;
    return fmm_reserve(m2l_src_raw, m2l) || fmm_reserve(m2l_tgt_raw, m2l) || fmm_reserve(p2p_tgt_raw, p2p) ||
                   fmm_reserve(p2p_src_raw, p2p)
               ? FMM_ERR_CUDA
               : FMM_OK;
  };
  const size_t m0 = about(480), p0 = about(160), f0 = about(320);
  size_t avail = ~(size_t)0, total = 0;
  if (m2l_src_raw.cap < m0 && cudaMemGetInfo(&avail, &total) != cudaSuccess) avail = 0;
  if (avail / 8 < sizeof(int) * (2 * m0 + 2 * p0 + 4 * f0) || room(m0, p0, f0)) {
    cudaGetLastError();
    TRY(room(about(0), about(0), about(0)));
  }
  size_t nm2l = 0, np2p = 0;
  uint32_t nf = (uint32_t)t->nsys;
  int cur = 0;  // the frontier to read
  for (bool first = true; nf > 0; first = false) {
    fmm_note_launch(), k_walk_begin<<<fmm_blocks(first ? std::max(nf, 32u) : 32, 256), 256, 0, st>>>(
        S, nf, first, fr[cur][0]->p, fr[cur][1]->p);
    auto cap2 = [](const DevBuf<int> &a, const DevBuf<int> &b) { return std::min(a.cap, b.cap); };
    const WalkOut O = {m2l_src_raw.p, m2l_tgt_raw.p, p2p_tgt_raw.p, p2p_src_raw.p, cap2(m2l_src_raw, m2l_tgt_raw),
                       cap2(p2p_tgt_raw, p2p_src_raw),
                       {cap2(*fr[cur ^ 1][0], *fr[cur ^ 1][1]), cap2(*fr[cur][0], *fr[cur][1])}, nm2l, np2p};
    size_t most = nf;  // pairs the level can have
    for (int l = 0; l < WALK_BATCH; l++) {
      const int rd = cur ^ (l & 1);
      const size_t nb = std::min<size_t>((most + WALK_TILE - 1) / WALK_TILE, WALK_GRID);
      fmm_note_launch(), k_walk<<<(unsigned)nb, WALK_BS, 0, st>>>(W, t->theta, l, S, O, fr[rd][0]->p, fr[rd][1]->p,
                                                                  fr[rd ^ 1][0]->p, fr[rd ^ 1][1]->p);
      most = std::min(8 * most, (size_t)1 << 32);
    }
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaMemcpyAsync(H, S, sizeof(WalkState), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    int l = 0;
    for (; l < WALK_BATCH && H->nf[l] > 0; l++) {
      const size_t m1 = nm2l + H->m2l[l], p1 = np2p + H->p2p[l];
      const size_t f1 = H->nf[l + 1];
      if (m1 > O.cap_m2l || p1 > O.cap_p2p || f1 > O.cap_f[l & 1]) {  // grow, and again from this level
        TRY(grow_keep(m2l_src_raw, m1, nm2l, st)); TRY(grow_keep(m2l_tgt_raw, m1, nm2l, st));
        TRY(grow_keep(p2p_tgt_raw, p1, np2p, st)); TRY(grow_keep(p2p_src_raw, p1, np2p, st));
        for (DevBuf<int> *b : fr[cur ^ 1 ^ (l & 1)]) TRY(fmm_reserve(*b, f1 + f1 / 2));
        break;
      }
      nm2l = m1;
      np2p = p1;
    }
    nf = H->nf[l];
    cur ^= l & 1;
  }
  // the M2L pairs stay in walk order here: build_classes groups them by
  // (target, class) once the classes are known
  t->nm2l = (long)nm2l;
  t->np2p = (long)np2p;
  return p2p_lists(t, st);
}

long long fmm_p2p_interactions(DevTree *t) {
  if (t->p2p_count_serial == t->build_serial) {
    unsigned long long v = 0;
    // the count kernel ran on the build's stream, which may not block with the default one
    if (cudaDeviceSynchronize() == cudaSuccess &&
        cudaMemcpy(&v, t->d_p2pcount.p, sizeof(v), cudaMemcpyDeviceToHost) == cudaSuccess) {
      t->p2p_interactions = (long long)v;
      t->p2p_count_serial = ~0ull;
    }
  }
  return t->p2p_interactions;
}

static int build_classes(DevTree *t, cudaStream_t st) {
  long n = t->nm2l;
  int p = t->order;
  t->csr_serial = ~0ull;  // the target lists of this build are made on demand (fmm_m2l_csr)
  TRY(fmm_reserve(t->m2l_cls_raw, n > 0 ? n : 1));
  if (n == 0) {
    t->nclasses = 0;
    return fmm_m2l_cell_order(t, t->tune.grouping, st);
  }
  // classes of the raw (walk-order) pairs: the distinct keys through an
  // open-addressing table, ids by rank of the sorted distinct keys
  const int *tgt = t->m2l_tgt_raw.p, *src = t->m2l_src_raw.p;
  uint32_t hsize = 1u << 16;
  while ((long)hsize < std::min<long>(n, 1L << 20) / 4) hsize <<= 1;
  uint64_t *keys = nullptr, *U1 = nullptr, *U2 = nullptr;
  uint32_t *stat = nullptr, *I1 = nullptr, *I2 = nullptr, *uhist = nullptr, *uscan = nullptr;
  uint32_t ncls = 0;
  for (int attempt = 0;; attempt++) {
    const size_t umax = hsize / 2;
    const size_t histu = 256 * fmm_rs_nblocks(umax);
    TRY(tmp_reserve(t, (size_t)n * 8 + 64 + umax * 24 + histu * 4 + fmm_scan_tmp_elems<uint32_t>(histu) * 4 + 256));
    char *q = t->tmp.p;
    keys = (uint64_t *)q; q += (size_t)n * 8;
    stat = (uint32_t *)q; q += 64;
    U1 = (uint64_t *)q; q += umax * 8;
    U2 = (uint64_t *)q; q += umax * 8;
    I1 = (uint32_t *)q; q += umax * 4;
    I2 = (uint32_t *)q; q += umax * 4;
    uhist = (uint32_t *)q; q += histu * 4;
    uscan = (uint32_t *)q;
    TRY(fmm_reserve(t->cls_hkeys, hsize));
    FMM_CUDA_TRY(cudaMemsetAsync(t->cls_hkeys.p, 0xff, sizeof(uint64_t) * hsize, st));  // all CLS_EMPTY
    FMM_CUDA_TRY(cudaMemsetAsync(stat, 0, 4 * sizeof(uint32_t), st));
    fmm_note_launch(), k_class_keys<<<fmm_blocks(n, 256), 256, 0, st>>>(src, tgt, n, t->wcell.p, keys,
                                                                        t->cls_hkeys.p, hsize - 1, stat, t->d_eflags.p);
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaMemcpyAsync(t->h_pinned, stat, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    ncls = t->h_pinned[0];
    if (!t->h_pinned[1] && ncls <= umax) break;
    if (hsize >= (1u << 28) || attempt >= 4) {
      fmm_set_error_text("M2L translation classes: the class table could not hold the distinct offsets");
      return FMM_ERR_RANGE;
    }
    hsize <<= 4;
  }
  t->nclasses = (int)ncls;
  TRY(fmm_reserve(t->cls_key4, 4 * (size_t)(ncls > 0 ? ncls : 1)));
  TRY(fmm_reserve(t->cls_table, hsize));
  // Ranks by counting: a comparison for each pair of keys, in one launch, up to
  // RANK_MAX keys; the radix sort of the 64-bit keys is 24 launches of a few
  // microseconds whatever their number, 140 us.  With the cells' order in one 8-bit
  // pass instead of two: a step of 10^4 charges (1,556 classes) 1,119 -> 976 us.
  fmm_note_launch(), k_class_collect<<<fmm_blocks(hsize, 256), 256, 0, st>>>(t->cls_hkeys.p, hsize, U1, I1, I2,
                                                                              stat + 2);
  const bool counted = ncls <= RANK_MAX;
  if (counted) {
    TRY(rank_keys(U1, (int)ncls, I2, st));
  } else {
    TRY(fmm_radix_sort<uint64_t>(U1, I1, U2, I2, ncls, 0, 64, uhist, uscan, st));
  }
  // same classes as the previous build (same ids): the per-class operator
  // data of that build still holds and its kernels skip their work
  TRY(fmm_reserve(t->d_cls_same, 1));
  const uint64_t *old = t->cls_prev.p;
  TRY(fmm_reserve(t->cls_prev, ncls > 0 ? ncls : 1));
  const bool may = (int)ncls == t->ncls_prev && p == t->order_prev && t->cls_prev.p == old;
  FMM_CUDA_TRY(cudaMemsetAsync(t->d_cls_same.p, may ? 0xff : 0, sizeof(uint32_t), st));
  t->ncls_prev = (int)ncls;
  t->order_prev = p;
  fmm_note_launch(), k_class_rank<<<fmm_blocks(std::max(ncls, 1u), 256), 256, 0, st>>>(
      U1, (int)ncls, I1, counted ? I2 : nullptr, t->cls_table.p, t->cls_key4.p, t->cls_prev.p, t->d_cls_same.p,
      fmm_wide_levels(p), t->d_eflags.p);
  // the class of each walk-order pair
  fmm_note_launch(), k_class_lookup<<<fmm_blocks(n, 256), 256, 0, st>>>(keys, n, t->cls_hkeys.p, hsize - 1,
                                                                         t->cls_table.p, t->m2l_cls_raw.p);
  FMM_CUDA_TRY(cudaGetLastError());
  int nt = fmm_nterms(p);
  if (t->cls_D.cap < (size_t)ncls * nt || t->cls_Df.cap < (size_t)ncls * fmm_stride4(nt))  // contents lost
    FMM_CUDA_TRY(cudaMemsetAsync(t->d_cls_same.p, 0, sizeof(uint32_t), st));
  TRY(fmm_reserve(t->cls_D, (size_t)ncls * nt));
  TRY(fmm_reserve(t->cls_Df, (size_t)ncls * fmm_stride4(nt)));
  fmm_note_launch(), k_class_derivs<<<fmm_blocks(ncls, FMM_WARPS), 32 * FMM_WARPS, 0, st>>>(t->cls_key4.p, (int)ncls, p, t->cls_D.p,
                                                                         t->cls_Df.p, t->d_cls_same.p);
  FMM_CUDA_TRY(cudaGetLastError());
  return fmm_m2l_cell_order(t, t->tune.grouping, st);
}

// The M2L pairs grouped by target, sorted by class within a target: a target
// has at most one source per class, so the order within a list is fully
// determined.  The walk-order pairs stay as they are (the sort runs on a copy).

// The M2L pairs by target and class.  A target has at most one pair of a class
// (the class fixes the source cell), so a pair's place in its target's list is
// the number of lower classes there: the pairs go to their target's range in
// any order (atomics), and a warp per target ranks them with a bitmap of the
// classes.  Three passes over the pairs; the radix sort of (target, class) keys
// took four with a histogram, a scan and a scatter each.  It stays for more
// classes than a bitmap in shared memory holds.  15.7M pairs (10^6 charges, with the
// targets' order): 0.67 ms with an atomic per pair, 0.31 with one per run of a
// target's; a step of 10^6 charges 8.81 -> 8.55 ms, of 512 forests 52.6 -> 49.7.
constexpr int CSR_SMEM = 65536, CSR_MAX_CLASSES = CSR_SMEM / 8 * 32;
// one atomic for a warp's pairs of one target (the walk emits a target's pairs in runs)
__global__ void k_csr_count(const int *tgt, long n, int *cnt) {
  const long i = blockIdx.x * 256l + threadIdx.x;
  const int t = i < n ? tgt[i] : -1;
  const unsigned same = __match_any_sync(0xffffffffu, t);
  if (t >= 0 && __ffs(same) - 1 == (int)(threadIdx.x & 31)) atomicAdd(&cnt[t], __popc(same));
}
__global__ void k_csr_scatter(const int *tgt, const int *src, const int *cls, long n, int *cur, uint64_t *list) {
  const long i = blockIdx.x * 256l + threadIdx.x;
  const int t = i < n ? tgt[i] : -1, lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xffffffffu, t);
  const int lead = __ffs(same) - 1;
  int base = 0;
  if (t >= 0 && lead == lane) base = atomicAdd(&cur[t], __popc(same));
  base = __shfl_sync(0xffffffffu, base, lead);
  if (t >= 0)
    list[base + __popc(same & ((1u << lane) - 1u))] = ((uint64_t)(uint32_t)cls[i] << 32) | (uint32_t)src[i];
}
__global__ void k_csr_place(const int *off, int nc, int nw, const uint64_t *list, int *src, int *cls) {
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ unsigned csr_smem[];  // per warp: the bitmap, then the number of classes below each word
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int t = blockIdx.x * (blockDim.x >> 5) + w;
  if (t >= nc) return;
  const int k0 = off[t], k1 = off[t + 1];
  if (k0 == k1) return;
  unsigned *bits = csr_smem + (size_t)2 * nw * w, *below = bits + nw;
  for (int i = lane; i < nw; i += 32) bits[i] = 0;
  __syncwarp();
  for (int k = k0 + lane; k < k1; k += 32) {
    const unsigned c = (unsigned)(list[k] >> 32);
    atomicOr(&bits[c >> 5], 1u << (c & 31));
  }
  __syncwarp();
  int run = 0;
  for (int i0 = 0; i0 < nw; i0 += 32) {
    const int i = i0 + lane, n = i < nw ? __popc(bits[i]) : 0;
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += v;
    }
    if (i < nw) below[i] = run + incl - n;
    run += __shfl_sync(FULL, incl, 31);
  }
  __syncwarp();
  for (int k = k0 + lane; k < k1; k += 32) {
    const uint64_t v = list[k];
    const unsigned c = (unsigned)(v >> 32);
    const int at = k0 + (int)below[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u));
    src[at] = (int)(uint32_t)v;
    cls[at] = (int)c;
  }
}

int fmm_m2l_csr(DevTree *t, cudaStream_t st) {
  if (t->csr_serial == t->build_serial) return FMM_OK;
  const long n = t->nm2l;
  const int nc = t->ncells;
  TRY(fmm_reserve(t->m2l_off, (size_t)nc + 1));
  TRY(fmm_reserve(t->m2l_src, n > 0 ? n : 1));
  TRY(fmm_reserve(t->m2l_cls, n > 0 ? n : 1));
  if (n == 0) {
    FMM_CUDA_TRY(cudaMemsetAsync(t->m2l_off.p, 0, sizeof(int) * ((size_t)nc + 1), st));
  } else if (t->nclasses <= CSR_MAX_CLASSES) {
    const size_t pairs = (sizeof(int) * ((size_t)nc + fmm_scan_tmp_elems<int>(nc)) + 15) & ~(size_t)15;
    TRY(tmp_reserve(t, pairs + sizeof(uint64_t) * (size_t)n));
    int *cur = (int *)t->tmp.p, *stmp = cur + nc;
    uint64_t *list = (uint64_t *)(t->tmp.p + pairs);
    FMM_CUDA_TRY(cudaMemsetAsync(cur, 0, sizeof(int) * nc, st));
    fmm_note_launch(), k_csr_count<<<fmm_blocks(n, 256), 256, 0, st>>>(t->m2l_tgt_raw.p, n, cur);
    TRY(fmm_scan<int>(cur, t->m2l_off.p, nc, t->m2l_off.p + nc, stmp, st));
    FMM_CUDA_TRY(cudaMemcpyAsync(cur, t->m2l_off.p, sizeof(int) * nc, cudaMemcpyDeviceToDevice, st));
    fmm_note_launch(), k_csr_scatter<<<fmm_blocks(n, 256), 256, 0, st>>>(t->m2l_tgt_raw.p, t->m2l_src_raw.p,
                                                                         t->m2l_cls_raw.p, n, cur, list);
    const int nw = (t->nclasses + 31) / 32, warps = std::max(1, std::min(8, CSR_SMEM / (8 * nw)));
    const size_t smem = (size_t)8 * nw * warps;
    // the most it ever takes: the limit holds for the process, and another thread may be about to launch with more
    FMM_CUDA_TRY(cudaFuncSetAttribute(k_csr_place, cudaFuncAttributeMaxDynamicSharedMemorySize, CSR_SMEM));
    fmm_note_launch(), k_csr_place<<<fmm_blocks(nc, warps), 32 * warps, smem, st>>>(t->m2l_off.p, nc, nw, list,
                                                                                    t->m2l_src.p, t->m2l_cls.p);
    FMM_CUDA_TRY(cudaGetLastError());
  } else {
    FMM_CUDA_TRY(cudaMemcpyAsync(t->m2l_src.p, t->m2l_src_raw.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, st));
    const int cbits = bits_for(t->nclasses), kbits = bits_for(nc) + cbits;
    if (kbits <= 32)
      TRY(sort_pairs<uint32_t>(t, t->m2l_tgt_raw.p, t->m2l_cls_raw.p, cbits, kbits, t->m2l_src, n, t->m2l_off,
                               t->m2l_cls.p, st));
    else
      TRY(sort_pairs<uint64_t>(t, t->m2l_tgt_raw.p, t->m2l_cls_raw.p, cbits, kbits, t->m2l_src, n, t->m2l_off,
                               t->m2l_cls.p, st));
  }
  t->csr_serial = t->build_serial;
  return FMM_OK;
}

// The M2L processing order of the cells (t->m2l_order): level, then by octant
// within the parent (grouping 0) or Morton order (grouping 1).
int fmm_m2l_cell_order(DevTree *t, int grouping, cudaStream_t st) {
  const int nc = t->ncells;
  size_t nbh = fmm_rs_nblocks(nc);
  size_t hist_n = 256 * nbh;
  TRY(tmp_reserve(t, (size_t)nc * 12 + hist_n * 4 + fmm_scan_tmp_elems<uint32_t>(hist_n) * 4 + 256));
  char *q = t->tmp.p;
  uint32_t *k1 = (uint32_t *)q; q += (size_t)nc * 4;
  uint32_t *k2 = (uint32_t *)q; q += (size_t)nc * 4;
  uint32_t *v2 = (uint32_t *)q; q += (size_t)nc * 4;
  uint32_t *hist = (uint32_t *)q; q += hist_n * 4;
  uint32_t *stmp2 = (uint32_t *)q;
  TRY(fmm_reserve(t->m2l_order, nc));
  fmm_note_launch(), k_order_keys<<<fmm_blocks(nc, 256), 256, 0, st>>>(nc, t->cid.p, t->clevel.p, grouping, k1,
                                                                        (uint32_t *)t->m2l_order.p);
  FMM_CUDA_TRY(cudaGetLastError());
  TRY(fmm_radix_sort<uint32_t>(k1, (uint32_t *)t->m2l_order.p, k2, v2, nc, 0, 8, hist, stmp2, st));
  t->grouping_built = grouping;
  t->order_version++;
  return FMM_OK;
}

void fmm_tree_destroy(DevTree *t) {
  if (!t) return;
  fmm_graph_release(t);
  fmm_tcg_release(t);
  for (cudaEvent_t *e : {&t->ev_fork, &t->ev_join, &t->ev_m, &t->ev_c, &t->ev_p, &t->ev_s, &t->ev_l}) {
    if (*e) cudaEventDestroy(*e);
    *e = nullptr;
  }
  if (t->s_hi) cudaStreamDestroy(t->s_hi);
  if (t->s_near) cudaStreamDestroy(t->s_near);
  t->s_hi = t->s_near = nullptr;
  if (t->gstream) cudaStreamDestroy(t->gstream);
  t->gstream = nullptr;
  fmm_release(t->keys); fmm_release(t->keys2); fmm_release(t->perm); fmm_release(t->perm2);
  fmm_release(t->px); fmm_release(t->py); fmm_release(t->pz);
  fmm_release(t->phi4); fmm_release(t->plo4); fmm_release(t->sdip); fmm_release(t->lpad); fmm_release(t->p2p_units);
  fmm_release(t->sym_own); fmm_release(t->sym_get); fmm_release(t->sym_place); fmm_release(t->sym_shares);
  fmm_release(t->sym_units); fmm_release(t->sym_totals);
  fmm_release(t->levf);
  fmm_release(t->cx); fmm_release(t->cy); fmm_release(t->cz); fmm_release(t->cid);
  fmm_release(t->ix); fmm_release(t->iy); fmm_release(t->iz);
  fmm_release(t->pstart); fmm_release(t->pcount); fmm_release(t->parent); fmm_release(t->child_first);
  fmm_release(t->child_mask); fmm_release(t->clevel); fmm_release(t->leaf_cells); fmm_release(t->cell_leaf);
  fmm_release(t->m2l_off); fmm_release(t->m2l_src); fmm_release(t->m2l_cls); fmm_release(t->m2l_order);
  fmm_release(t->m2l_cls_raw);
  for (int k = 0; k < 2; k++) {
    fmm_release(t->hM[k]); fmm_release(t->hL[k]); fmm_release(t->hD[k]);
  }
  fmm_release(t->bhM); fmm_release(t->bhW);
  t->csr_serial = ~0ull;
  fmm_release(t->p2p_off); fmm_release(t->p2p_src);
  fmm_release(t->cls_key4); fmm_release(t->cls_D); fmm_release(t->cls_Df); fmm_release(t->cls_table);
  fmm_release(t->cls_hkeys); fmm_release(t->cls_prev); fmm_release(t->d_cls_same);
  t->ncls_prev = t->order_prev = -1;
  fmm_release(t->M); fmm_release(t->L); fmm_release(t->Mf); fmm_release(t->Lf);
  fmm_release(t->Fnear); fmm_release(t->Ffar);
  fmm_release(t->front);
  fmm_release(t->m2l_tgt_raw); fmm_release(t->m2l_src_raw);
  fmm_release(t->p2p_tgt_raw); fmm_release(t->p2p_src_raw);
  fmm_release(t->tc_T);
  fmm_release(t->d_tcerr);
  fmm_release(t->tc_sched_off); fmm_release(t->tc_sched_cls); fmm_release(t->tc_bitmap); fmm_release(t->tc_rank);
  fmm_release(t->tc_stab); fmm_release(t->tc_pos); fmm_release(t->cm_otab);
  fmm_release(t->cm_woff); fmm_release(t->cm_wstep); fmm_release(t->tp_perm); fmm_release(t->tp_tgt);
  t->cm_wserial = ~0ull;
  t->sched_serial = ~0ull;
  t->tc_serial = ~0ull;
  fmm_release(t->d_walk);
  fmm_release(t->d_p2pcount);
  fmm_release(t->m2l_ord); fmm_release(t->mnorm); fmm_release(t->feat); fmm_release(t->tscale); fmm_release(t->tpart);
  fmm_release(t->sys_pairs);
  fmm_release(t->ltgt);
  fmm_release(t->cr); fmm_release(t->crmax); fmm_release(t->crf); fmm_release(t->wcell); fmm_release(t->csys);
  fmm_release(t->sys_off); fmm_release(t->psys); fmm_release(t->roots);
  fmm_release(t->tmp); fmm_release(t->d_eflags); fmm_release(t->d_root);
  if (t->h_pinned) cudaFreeHost(t->h_pinned);
  t->h_pinned = nullptr;
  if (t->ev_ready)
    for (int i = 0; i < 16; i++) cudaEventDestroy(t->ev[i]);
  if (t->ev_ready)
    for (int i = 0; i < 4; i++) cudaEventDestroy(t->ev_mk[i]);
  t->ev_ready = false;
}
