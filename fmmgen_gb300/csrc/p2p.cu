// p2p.cu -- near-field particle-particle interactions (P2P) over the P2P list
// (P2P_Cells / evaluate_P2P_lazy, example/calculate.cpp:24-40, 208-216), in FP64
// and in the mixed-precision form, plus the per-evaluate FP32 staging.
#include <algorithm>
#include <cooperative_groups.h>
#include "internal.h"

// ---------------------------------------------------------------------------
// P2P in FP64 (example/calculate.cpp:24-40, 208-216)
// ---------------------------------------------------------------------------
// Bound by the FP64 pipe: two operations per clock and SM (FP32: 128), so a
// warp's FP64 instruction takes 16 clocks of its SM and
// everything else -- shared-memory reads, index arithmetic, shuffles, staging
// the sources again -- hides behind it.  What counts is that no lane idles.
// A leaf's targets are therefore cut into groups that fill the warp: chunks of
// 32, then 16 and 8 targets with 2 and 4 lanes each, then the last m <= 7 with
// floor(32 / m) lanes each; the f lanes of a target take every f-th source of
// the stream and their sums are added at the end.  One warp per group, from the
// build's units of up to 32 targets: the groups of a leaf are independent warps,
// so leaves of several chunks do not make a tail of long warps, and the grid
// grows with the particles, not with the largest leaf there could be.  With one
// lane per target and chunks of 32 a leaf of 14 left 56 % of the lanes idle and one
// of 40 took two full passes.  The sources of the leaf's list are one stream (the
// leaves' particle ranges one after the other), staged 64 at a time.
// For quadrupoles, and for charges and dipoles where each pair once does not pay
// or has no room (below).  Measured (one GB300), a warp per leaf before and now: 10^6
// uniform charges, 30 per leaf, 4.79e9 interactions: 229 and 158 ms; 86,400 dipoles, 11
// per leaf: 25.8 and 10.2 ms; one leaf of 10,000 charges: 2,000 and 6.9 ms.
#define P2P_WARPS 4
#define P64_CHUNK 64
// components staged per source
__host__ __device__ constexpr int p64_nq(int so) { return so == 0 ? 1 : so == 1 ? 3 : 6; }

// One source on one target.  SELF: the chunk may hold the target itself.
template <int SO, bool SELF, bool POT>
__device__ __forceinline__ void p64_one(double dx, double dy, double dz, const double (*q)[P64_CHUNK], int jj,
                                        bool self, double &phi, double &ex, double &ey, double &ez) {
  if (SO == 2) {
    if (SELF && self) return;
    const double s[6] = {q[0][jj], q[1][jj], q[2][jj], q[3][jj], q[4][jj], q[5][jj]};
    quadrupole_p2p<double>(dx, dy, dz, s, phi, ex, ey, ez);
    return;
  }
  const double r2 = dx * dx + dy * dy + dz * dz;
  double rinv = rsqrt(r2);
  if (SELF) rinv = self ? 0.0 : rinv;  // l2 != l1
  const double rr = rinv * rinv;
  if (SO == 0) {
    const double qr = q[0][jj] * rinv;
    if (POT) phi += qr;
    const double qr3 = qr * rr;
    ex += qr3 * dx;
    ey += qr3 * dy;
    ez += qr3 * dz;
  } else {
    const double sx = q[0][jj], sy = q[1][jj], sz = q[2][jj];
    const double r3 = rr * rinv;
    const double u = (sx * dx + sy * dy + sz * dz) * r3;
    if (POT) phi -= u;
    const double r5 = (3.0 * rr) * u;
    ex += sx * r3 - r5 * dx;
    ey += sy * r3 - r5 * dy;
    ez += sz * r3 - r5 * dz;
  }
}

template <int SO, bool POT>
__global__ void __launch_bounds__(32 * P2P_WARPS) k_p2p64(const int4 *units, int nunits, int nub, const int *pstart,
                                                          const int *pcount, const int *off_, const int *src,
                                                          const double *px, const double *py, const double *pz,
                                                          const uint32_t *perm, const double *S, double *Fnear) {
  constexpr int NQ = p64_nq(SO);
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ double sp[P2P_WARPS][3][P64_CHUNK], sq[P2P_WARPS][NQ][P64_CHUNK];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int y = blockIdx.x / nub;  // blocks by group: every unit's 32 or 16 targets, then the groups of 8, then the rest
  const int u = (blockIdx.x - y * nub) * P2P_WARPS + w;
  if (u >= nunits) return;
  const int4 unit = units[u];
  const int A = unit.x, rest = unit.z & 31;  // rest: of a leaf's last unit, where that is not full
  const int a0 = pstart[A], na = pcount[A];
  // this warp's group of targets: [tb, tb + m)
  const int tb = unit.y + (y == 0 ? 0 : y == 1 ? rest & 16 : rest & 24);
  const int m = y == 0 ? (rest ? rest & 16 : 32) : y == 1 ? rest & 8 : rest & 7;
  if (m == 0) return;
  const int f = 32 / m;  // lanes per target
  const int tl = lane / f, slice = lane - tl * f;
  const bool ok = tl < m;
  const int i = a0 + tb + (ok ? tl : 0);
  const double xi = px[i], yi = py[i], zi = pz[i];
  double phi = 0, ex = 0, ey = 0, ez = 0;
  const int k0 = off_[A], k1 = off_[A + 1];
  for (int kb = k0; kb < k1; kb += 32) {
    // up to 32 source leaves: lane q holds leaf kb + q's particle range and the
    // exclusive prefix of the counts (its offset in the stream)
    const int nbat = min(32, k1 - kb);
    int B = -1, start = 0, cnt = 0;
    if (lane < nbat) {
      B = src[kb + lane];
      start = pstart[B];
      cnt = pcount[B];
    }
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += v;
    }
    const int excl = incl - cnt;
    const int total = __shfl_sync(FULL, incl, 31);
    const unsigned selfq = __ballot_sync(FULL, B == A);
    const int self_lo = selfq ? __shfl_sync(FULL, excl, __ffs(selfq) - 1) : -1;
    for (int cb = 0; cb < total; cb += P64_CHUNK) {
      const int n = min(P64_CHUNK, total - cb);
      __syncwarp();
#pragma unroll
      for (int u = 0; u < P64_CHUNK / 32; u++) {
        // the lane's source: the last leaf q whose stream offset is <= s
        const int s = cb + 32 * u + lane;
        int q = 0;
#pragma unroll
        for (int stp = 16; stp; stp >>= 1) {
          const int cand = q + stp;
          const int v = __shfl_sync(FULL, excl, cand & 31);
          if (cand < nbat && v <= s) q = cand;
        }
        const int jb = __shfl_sync(FULL, start, q), je = __shfl_sync(FULL, excl, q);
        if (s < total) {
          const int j = jb + (s - je);
          const size_t o = perm[j];
          sp[w][0][32 * u + lane] = px[j];
          sp[w][1][32 * u + lane] = py[j];
          sp[w][2][32 * u + lane] = pz[j];
#pragma unroll
          for (int k = 0; k < NQ; k++) sq[w][k][32 * u + lane] = S[NQ * o + k];
        }
      }
      __syncwarp();
      if (!ok) continue;  // the spare lanes of a group of 3, 5, 6 or 7
      const int me = self_lo + tb + tl - cb;  // the target's own place in the chunk
      if (self_lo >= 0 && self_lo < cb + n && self_lo + na > cb) {
        for (int jj = slice; jj < n; jj += f)
          p64_one<SO, true, POT>(xi - sp[w][0][jj], yi - sp[w][1][jj], zi - sp[w][2][jj], sq[w], jj, jj == me, phi, ex,
                                 ey, ez);
      } else {
#pragma unroll 2
        for (int jj = slice; jj < n; jj += f)
          p64_one<SO, false, POT>(xi - sp[w][0][jj], yi - sp[w][1][jj], zi - sp[w][2][jj], sq[w], jj, false, phi, ex,
                                  ey, ez);
      }
    }
  }
  // the f partial sums of each target
  __syncwarp();
  for (int o = 16; o; o >>= 1) {
    if (o >= f) continue;
    const double v0 = __shfl_down_sync(FULL, phi, o), v1 = __shfl_down_sync(FULL, ex, o);
    const double v2 = __shfl_down_sync(FULL, ey, o), v3 = __shfl_down_sync(FULL, ez, o);
    if (slice < o && slice + o < f) {
      phi += v0;
      ex += v1;
      ey += v2;
      ez += v3;
    }
  }
  if (ok && slice == 0) {
    Fnear[4 * (size_t)i] = phi;
    Fnear[4 * (size_t)i + 1] = ex;
    Fnear[4 * (size_t)i + 2] = ey;
    Fnear[4 * (size_t)i + 3] = ez;
  }
}

// ---------------------------------------------------------------------------
// P2P in FP64, each pair of particles once (charges and dipoles)
// ---------------------------------------------------------------------------
// Two leaves that list each other need the displacement, the distance and its
// reciprocal powers of a pair of particles only once: 22.6 FP64 operations for
// both directions instead of 2 x 17.6 (dipoles 37.6 instead of 2 x 25.6).  One
// leaf of every such pair owns it (which one alternates with the cells'
// parities, so that each leaf owns about half of its list): the sources' side is
// added up in shared memory and left in a buffer, 32 bytes per particle of the
// other leaf.  A unit of work is 32 entries of a leaf's list and one warp (a warp
// per leaf made a tail of the densest ones: a single warp gets a quarter of its
// SM's FP64 rate at most); it leaves its targets' sums in the buffer too, and
// k_p2p64_gather adds a leaf's shares up in list order, so that every pass gives
// the same bits, wherever in the buffer the shares lie.  In a step, the 32 lanes
// are at 32 different staged sources, so that each adds to its own; a warp
// barrier orders the steps.
// An entry whose reverse is not listed (the walk gives symmetric lists; nothing
// here relies on it) and the leaf itself go one way.  The buffer is at most
// P64_SHARES; systems that would need more, or whose leaves are few and large
// (p64_pays), take k_p2p64, which adds in another order: the choice is the tree's alone, not that of the memory that happens to be
// free (but for a device that has none left for the buffer).
// Measured (one GB300): 10^6 charges: 158 -> 114 ms, the 86,400 dipoles 10.2 -> 8.8 ms.
constexpr size_t P64_SHARES = (size_t)4 << 30;

__device__ __forceinline__ bool p64_owns(int A, int B) { return ((A ^ B) & 1) ? A < B : A > B; }

// Places in the buffer (in particles): for each leaf the sums of its units, one
// after the other, then what its owned entries leave for their sources, place[k];
// and the units (cell, leaf, batch of 32 entries).  totals: units, places, then for
// p64_pays, in interactions: the largest unit, all of them one way, and the most
// that a warp of k_p2p64 takes (32 targets, or a smaller leaf's, on all its sources).
__global__ void k_sym_places(const int *leaf_cells, int nleaves, const int *pcount, const int *off, const int *src,
                             uint32_t *place, uint32_t *leaf_place, int4 *units, unsigned long long *totals) {
  constexpr unsigned FULL = 0xffffffffu;
  const int leaf = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (leaf >= nleaves) return;
  const int A = leaf_cells[leaf], k0 = off[A], k1 = off[A + 1], nb = (k1 - k0 + 31) >> 5, na = pcount[A];
  unsigned sum = 0, all = 0;
  for (int k = k0 + lane; k < k1; k += 32) {
    const int B = src[k];
    const unsigned n = (unsigned)pcount[B];
    all += n;
    if (A != B && p64_owns(A, B)) sum += n;
  }
  for (int d = 16; d; d >>= 1) {
    sum += __shfl_xor_sync(FULL, sum, d);
    all += __shfl_xor_sync(FULL, all, d);
  }
  unsigned long long at = 0, ub = 0;
  if (lane == 0) {
    at = atomicAdd(&totals[1], (unsigned long long)sum + (unsigned long long)na * nb);
    ub = atomicAdd(&totals[0], (unsigned long long)nb);
    leaf_place[leaf] = (uint32_t)at;
    atomicAdd(&totals[3], (unsigned long long)na * all);
    atomicMax(&totals[4], (unsigned long long)min(na, 32) * all);
  }
  uint32_t run = __shfl_sync(FULL, (uint32_t)at, 0) + (uint32_t)(na * nb);
  ub = __shfl_sync(FULL, ub, 0);
  for (int b = lane; b < nb; b += 32) units[ub + b] = make_int4(A, leaf, b, 0);
  unsigned most = 0;  // sources of the unit that has most
  for (int kb = k0; kb < k1; kb += 32) {
    const int k = kb + lane, B = k < k1 ? src[k] : A;
    const int n = A != B && p64_owns(A, B) ? pcount[B] : 0;
    const bool self = __any_sync(FULL, k < k1 && A == B);
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += v;
    }
    if (k < k1) place[k] = run + (uint32_t)(incl - n);
    const unsigned both = (unsigned)__shfl_sync(FULL, incl, 31);
    run += both;
    most = max(most, both + (self ? (unsigned)na : 0u));
  }
  if (lane == 0) atomicMax(&totals[2], (unsigned long long)na * most);
}
// own[k]: place of the shares entry k's target leaves for its source, -1: one way,
// -2: the source owns the pair, and leaves the target's shares at get[k] (else -1).
// One warp per unit.
__global__ void k_sym_pairs(const int4 *units, const unsigned long long *totals, const int *off, const int *src,
                            const uint32_t *place, int *own, int *get) {
  const unsigned long long u = blockIdx.x * 8ull + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (u >= totals[0]) return;
  const int A = units[u].x, k = off[A] + 32 * units[u].z + lane;
  const bool in = k < off[A + 1];
  const int B = in ? src[k] : A;
  int o = -1, g = -1;
  const bool mine = A != B && p64_owns(A, B), seek = A != B && !mine;
  if (mine) o = (int)place[k];
  if (seek) {  // A's place in B's list, which is sorted
    const int end = off[B + 1];
    int lo = off[B], hi = end;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (src[mid] < A) lo = mid + 1;
      else hi = mid;
    }
    if (lo < end && src[lo] == A) {
      o = -2;
      g = (int)place[lo];
    }
  }
  if (in) {
    own[k] = o;
    get[k] = g;
  }
}

// A pair of particles both ways: source jj (components sq[.][jj]) on the target
// (si), and the target on the source, into acc[.][aj].  (dx, dy, dz) = target - source.
template <int SO, bool POT, int STRIDE>
__device__ __forceinline__ void p64_both(double dx, double dy, double dz, const double (*sq)[P64_CHUNK], int jj,
                                         const double *si, double &phi, double &ex, double &ey, double &ez,
                                         double (*acc)[STRIDE], int aj) {
  constexpr int LAST = p64_nq(SO) - 1;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double rinv = rsqrt(r2), rr = rinv * rinv, r3 = rr * rinv;
  if (SO == 0) {
    const double qj = sq[0][jj], bj = qj * r3, bi = si[0] * r3;
    if (POT) phi += qj * rinv;
    ex += bj * dx;
    ey += bj * dy;
    ez += bj * dz;
    if (POT) acc[0][aj] += si[0] * rinv;
    acc[1][aj] -= bi * dx;
    acc[2][aj] -= bi * dy;
    acc[3][aj] -= bi * dz;
  } else {
    const double mx = sq[0][jj], my = sq[LAST > 1 ? 1 : 0][jj], mz = sq[LAST][jj], t3 = 3.0 * rr;
    const double uj = (mx * dx + my * dy + mz * dz) * r3, wj = t3 * uj;
    const double sx = si[0], sy = si[LAST > 1 ? 1 : 0], sz = si[LAST];
    const double ui = (sx * dx + sy * dy + sz * dz) * r3, wi = t3 * ui;
    if (POT) phi -= uj;
    ex += mx * r3 - wj * dx;
    ey += my * r3 - wj * dy;
    ez += mz * r3 - wj * dz;
    if (POT) acc[0][aj] += ui;  // seen from the source the displacement is -d
    acc[1][aj] += sx * r3 - wi * dx;
    acc[2][aj] += sy * r3 - wi * dy;
    acc[3][aj] += sz * r3 - wi * dz;
  }
}

struct P64Args {
  const int4 *units;
  const int *leaf_cells, *pstart, *pcount, *off, *src;
  const double *px, *py, *pz;
  const uint32_t *perm;
  const double *S;
  const int *own, *get;
  const uint32_t *leaf_place;
  double *shares;  // [places][4]
  double *Fnear;
};

template <int SO, bool POT>
__global__ void __launch_bounds__(32) k_p2p64_sym(const P64Args P) {
  constexpr int NQ = p64_nq(SO);
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ double sp[3][P64_CHUNK], sq[NQ][P64_CHUNK], acc[4][32];
  const int lane = threadIdx.x;
  const int4 unit = P.units[blockIdx.x];
  const int A = unit.x, a0 = P.pstart[A], na = P.pcount[A];
  double *const mine_out = P.shares + 4 * ((size_t)P.leaf_place[unit.y] + (size_t)na * unit.z);
  // up to 32 source leaves: lane q holds entry q's particle range and owner
  const int k0 = P.off[A] + 32 * unit.z, nbat = min(32, P.off[A + 1] - k0);
  int B = -1, start = 0, cnt = 0, own = -2;
  if (lane < nbat) {
    B = P.src[k0 + lane];
    start = P.pstart[B];
    cnt = P.pcount[B];
    own = P.own[k0 + lane];
  }
  for (int tb = 0; tb < na;) {
    // the next group of targets: 32 with a lane each, 16 with two, 8 with four, ...
    // (25 to 31, or 13 to 15, idle a few lanes rather than go over the sources again)
    const int rem = na - tb, lf = rem > 24 ? 0 : rem > 12 ? 1 : rem > 4 ? 2 : rem > 2 ? 3 : 4;
    const int m = min(rem, 32 >> lf);
    const int f = 1 << lf, steps = 32 >> lf;
    const int tl = lane >> lf, slice = lane & (f - 1);
    const bool ok = tl < m;
    const int i = a0 + tb + (ok ? tl : 0);
    const double xi = P.px[i], yi = P.py[i], zi = P.pz[i];
    double si[NQ];
#pragma unroll
    for (int k = 0; k < NQ; k++) si[k] = P.S[NQ * (size_t)P.perm[i] + k];
    double phi = 0, ex = 0, ey = 0, ez = 0;
#pragma unroll 1
    for (int both = 1; both >= 0; both--) {  // the owned leaves' particles, then those that go one way
      const int mine = (both ? own >= 0 : own == -1) ? cnt : 0;
      int incl = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += v;
      }
      const int excl = incl - mine;
      const int total = __shfl_sync(FULL, incl, 31);
      const unsigned selfq = both ? 0u : __ballot_sync(FULL, B == A);
      const int self_lo = selfq ? __shfl_sync(FULL, excl, __ffs(selfq) - 1) : -1;
      for (int cb = 0; cb < total; cb += 32) {
        const int n = min(32, total - cb), s = cb + lane;
        int q = 0;
#pragma unroll
        for (int stp = 16; stp; stp >>= 1) {
          const int v = __shfl_sync(FULL, excl, q + stp);
          if (v <= s) q += stp;
        }
        const int at = s - __shfl_sync(FULL, excl, q);  // the source's place in its leaf
        const int j = __shfl_sync(FULL, start, q) + at, base = __shfl_sync(FULL, own, q);
        double *share = P.shares + 4 * ((size_t)(both ? base : 0) + at);
        __syncwarp();
        if (s < total) {
          const size_t o = P.perm[j];
          sp[0][lane] = P.px[j];
          sp[1][lane] = P.py[j];
          sp[2][lane] = P.pz[j];
#pragma unroll
          for (int k = 0; k < NQ; k++) sq[k][lane] = P.S[NQ * o + k];
          if (both)  // this leaf's earlier groups have left their part
#pragma unroll
            for (int c = 0; c < 4; c++) acc[c][lane] = tb > 0 ? share[c] : 0.0;
        }
        __syncwarp();
        if (!both) {
          const int me = self_lo >= 0 ? self_lo + tb + tl - cb : -1;
          if (ok)
            for (int jj = slice; jj < n; jj += f)
              p64_one<SO, true, POT>(xi - sp[0][jj], yi - sp[1][jj], zi - sp[2][jj], sq, jj, jj == me, phi, ex, ey, ez);
          continue;
        }
        for (int st = 0; st < steps; st++) {
          const int jj = (slice * steps + st + tl) & 31;
          if (ok && jj < n) {
            const double dx = xi - sp[0][jj], dy = yi - sp[1][jj], dz = zi - sp[2][jj];
            p64_both<SO, POT, 32>(dx, dy, dz, sq, jj, si, phi, ex, ey, ez, acc, jj);
          }
          __syncwarp();
        }
        if (s < total)
#pragma unroll
          for (int c = POT ? 0 : 1; c < 4; c++) share[c] = acc[c][lane];
      }
    }
    __syncwarp();
    for (int o = 1; o < f; o <<= 1) {
      phi += __shfl_xor_sync(FULL, phi, o);
      ex += __shfl_xor_sync(FULL, ex, o);
      ey += __shfl_xor_sync(FULL, ey, o);
      ez += __shfl_xor_sync(FULL, ez, o);
    }
    if (ok && slice == 0) {
      double *v = mine_out + 4 * (size_t)(tb + tl);
      v[0] = phi;
      v[1] = ex;
      v[2] = ey;
      v[3] = ez;
    }
    tb += m;
  }
}

// A leaf's sums: each of its units' and, after it, the shares that the owners of
// the unit's other pairs left, in list order.
template <bool POT>
__global__ void __launch_bounds__(128) k_p2p64_gather(const P64Args P, int nleaves) {
  const int leaf = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (leaf >= nleaves) return;
  const int A = P.leaf_cells[leaf];
  const int a0 = P.pstart[A], na = P.pcount[A], k0 = P.off[A], k1 = P.off[A + 1];
  const double *own = P.shares + 4 * (size_t)P.leaf_place[leaf];
  for (int tb = 0; tb < na; tb += 32) {
    const int at = tb + lane;
    double v[4] = {0, 0, 0, 0};
    for (int kb = k0; kb < k1; kb += 32) {
      if (at < na)
#pragma unroll
        for (int c = 0; c < 4; c++) v[c] += own[4 * ((size_t)na * ((kb - k0) >> 5) + at) + c];
      const int g = kb + lane < k1 ? P.get[kb + lane] : -1;
      unsigned has = __ballot_sync(0xffffffffu, g >= 0);
      while (has) {
        const int base = __shfl_sync(0xffffffffu, g, __ffs(has) - 1);
        has &= has - 1;
        if (at < na)
#pragma unroll
          for (int c = POT ? 0 : 1; c < 4; c++) v[c] += P.shares[4 * ((size_t)base + at) + c];
      }
    }
    if (at < na)
#pragma unroll
      for (int c = 0; c < 4; c++) P.Fnear[4 * (size_t)(a0 + at) + c] = v[c];
  }
}

// Whether each pair once is the faster way.  A unit is one warp, all targets of its
// leaf on up to 32 leaves, so in trees of few large leaves the largest unit decides:
// a warp does 3.3e7 of its pairs a second (dipoles 2e7).  One way a warp does 4.7e7
// (3e7) interactions, and the chip 2.4e10 (1.5e10), of which uneven leaves reach two
// thirds.  Charges, ms each pair once / one way: one leaf of 300 1.87 / 0.21, of 10^4
// 2,047 / 6.9; 10^4 uniform in 64 leaves 14.8 / 6.9, in 512 0.76 / 2.1; 3x10^4 in 64 leaves
// 129 / 36, in 512 5.5 / 11.2; 10^5 in 64 leaves 1,357 / 321, in 512 57.8 / 91.7; 3,000 in 64
// leaves 1.65 / 1.96, in 8 19.5 / 2.1; 3x10^4 clustered in 800 leaves 10.4 / 15.9, in 190 98 /
// 35; 10^5 clustered in 954 99 / 73.
static bool p64_pays(const unsigned long long *totals) {
  const double unit = (double)totals[2], all = (double)totals[3], warp = (double)totals[4];
  return unit <= std::max(all / 730.0, 0.69 * warp);
}

// The owners and places of this build's pairs and room for the shares: once per
// build, with a wait for the totals.  No room on the device leaves the build without
// them, for all its passes.
static int p64_layout(DevTree *t, cudaStream_t st) {
  if (t->sym_serial == t->build_serial) return FMM_OK;
  const int nl = t->nleaves;
  const size_t n = (size_t)std::max(t->np2p, 1L), nu = (size_t)nl + n / 32;
  t->sym_serial = t->build_serial;
  t->sym_places = -1;
  if (fmm_reserve(t->sym_own, n) || fmm_reserve(t->sym_get, n) || fmm_reserve(t->sym_place, n + (size_t)nl) ||
      fmm_reserve(t->sym_units, nu) || fmm_reserve(t->sym_totals, 5)) {
    cudaGetLastError();
    return FMM_OK;
  }
  FMM_CUDA_TRY(cudaMemsetAsync(t->sym_totals.p, 0, 5 * sizeof(unsigned long long), st));
  fmm_note_launch(), k_sym_places<<<fmm_blocks(nl, 8), 256, 0, st>>>(
      t->leaf_cells.p, nl, t->pcount.p, t->p2p_off.p, t->p2p_src.p, t->sym_place.p, t->sym_place.p + n, t->sym_units.p,
      t->sym_totals.p);
  FMM_CUDA_TRY(cudaGetLastError());
  unsigned long long v[5] = {};
  FMM_CUDA_TRY(cudaMemcpyAsync(v, t->sym_totals.p, sizeof(v), cudaMemcpyDeviceToHost, st));
  FMM_CUDA_TRY(cudaStreamSynchronize(st));
  const size_t room = 4 * std::max((size_t)v[1], (size_t)1);
  if (room * sizeof(double) > P64_SHARES || !p64_pays(v)) return FMM_OK;
  if (fmm_reserve(t->sym_shares, room)) {
    cudaGetLastError();
    return FMM_OK;
  }
  fmm_note_launch(), k_sym_pairs<<<fmm_blocks(nu, 8), 256, 0, st>>>(t->sym_units.p, t->sym_totals.p, t->p2p_off.p,
                                                                    t->p2p_src.p, t->sym_place.p, t->sym_own.p,
                                                                    t->sym_get.p);
  FMM_CUDA_TRY(cudaGetLastError());
  t->sym_nunits = (long)v[0];
  t->sym_places = (long)v[1];
  return FMM_OK;
}

// At the end of a build of a tree last evaluated in FP64: the next pass may be captured.
int fmm_p2p_prepare(DevTree *t, cudaStream_t st) {
  return t->so <= 1 && t->p64_last ? p64_layout(t, st) : FMM_OK;
}

// ---------------------------------------------------------------------------

// Per evaluate: positions as two-float offsets from the particle's system root
// centre (hi in .xyz, the charge in .w; lo in .xyz, the particle's own index
// in .w for the self test); dipole moments in FP32; per leaf a coordinate outside
// the root cube, for sources that fill a chunk up.
// A thread per particle, and per leaf (psys: the particles' systems, of a forest);
// bound by memory.  A block of 128 per leaf of 30: 10^6 particles 60 -> 32 us,
// 512 systems of 17.7 a leaf 0.79 -> 0.25 ms.
__global__ void k_stage_particles(long N, const int *leaf_cells, int nleaves, const int *csys, const int *psys,
                                  const double *roots, const double *px, const double *py, const double *pz,
                                  const uint32_t *perm, const double *S, int so, float4 *phi4, float4 *plo4,
                                  float4 *sdip, float *lpad) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < nleaves) {
    const double r = roots[4 * (size_t)csys[leaf_cells[i]] + 3];
    lpad[i] = r > 0 ? 3.f * (float)r : 1.f;
  }
  if (i >= N) return;
  const uint32_t o = perm[i];
  const double *root = roots + 4 * (size_t)(psys ? psys[o] : 0);
  const double dx = px[i] - root[0], dy = py[i] - root[1], dz = pz[i] - root[2];
  const float hx = (float)dx, hy = (float)dy, hz = (float)dz;
  phi4[i] = make_float4(hx, hy, hz, so == 0 ? (float)S[o] : 0.f);
  plo4[i] = make_float4((float)(dx - (double)hx), (float)(dy - (double)hy), (float)(dz - (double)hz),
                        __int_as_float((int)i));
  if (so) sdip[i] = make_float4((float)S[3 * (size_t)o], (float)S[3 * (size_t)o + 1], (float)S[3 * (size_t)o + 2], 0.f);
}

// ---------------------------------------------------------------------------
// P2P in FP32 with compensated accumulation (mixed precision)
// ---------------------------------------------------------------------------
// Bound by the FP32 pipe: an add, multiply or FMA on two packed sources takes
// it two clocks, so what counts is operations per interaction and full lanes.
//
// One warp (a block) takes a chunk of 32 targets of a leaf, or its last m < 32.
// A lane holds two targets, so that a staged source read from shared memory
// serves both; two lanes share them when m > 16, four when m > 8, else eight,
// each taking its share of the sources.  The source particles of the leaf's P2P
// list are one stream -- the leaves' particle ranges one after the other, up to
// 32 leaves at a time -- staged in chunks of 64, a lane finding and storing two
// consecutive ones (in chunks of 32, a source per lane, the staging was 40 % of
// the instructions), the last chunk filled up with chargeless sources outside
// the root cube, so that two sources always share an instruction.  The split is
// a runtime shift and the kernel has two inner loops, for chunks that may hold a
// target itself and for the others: a loop for each split measured up to twice
// slower on adaptive trees, waiting for instructions.
//
// Displacements: positions are two-float offsets from the system's root
// centre; the high parts of two nearby particles subtract exactly (Sterbenz)
// or with one rounding, and the low parts carry the rest, so the displacement
// keeps ~1e-7 relative accuracy even for very close pairs (three operations
// per axis, eighteen per interaction).
//
// Each chunk's contribution is summed in FP32 and folded into a
// Kahan-compensated FP32 total; the final per-particle near + far sum is FP64
// (k_finalize).  1/R is the hardware approximation (relative error ~1e-7, the
// size of the FP32 displacement's own rounding).  The potential is summed only
// when it is an output.
// Measured (one GB300, kernel alone, one target per lane and chunks of 32 sources
// before, and now): 10^6 uniform charges, 30 per leaf, field: 4.15 and 3.84 ms;
// 3x10^5, 73 per leaf: 3.54 and 2.39; 2x10^6 clustered: 16.4 and 13.6; 2x10^6 Plummer
// dipoles, 18 per leaf: 13.4 and 11.8; 10^4, 20 per leaf: 0.19 and 0.09.  (Sources a
// leaf width away as one FP32 number per axis in the target leaf's frame: 3.09, 2.02,
// 11.1, 10.7 and 0.11 ms, with operands of half the bits, which no caller has asked
// for.)  Median field error against FP64 over uniform, clustered and Plummer
// systems: 1.46-1.78e-7 before, 1.46-1.60e-7 now (dipoles 2.02-2.05e-7 and
// 2.00-2.05e-7).
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
  float y = v - c;
  float t = s + y;
  c = (t - s) - y;
  s = t;
}
// (s, c) += (s', c') for running sums s - c: the sum of the high parts with
// its rounding error
__device__ __forceinline__ void pair_add(float &s, float &c, float s2, float c2) {
  const float t = s + s2, z = t - s;
  const float e = (s - (t - z)) + (s2 - z);
  s = t;
  c = (c + c2) - e;
}
// x in FP64, by the integer pipe: the FP64 pipe would take 16 clocks of the SM for
// each.  (It does take subnormal numbers, which have no leading one.)
__device__ __forceinline__ double f2d(float x) {
  const unsigned b = __float_as_uint(x), e = (b >> 23) & 255u, m = b & 0x7fffffu;
  if (e == 0u && m) return (double)x;
  const unsigned E = e == 0u ? 0u : e == 255u ? 2047u : e + 896u;
  return __hiloint2double((int)((b & 0x80000000u) | (E << 20) | (m >> 3)), (int)(m << 29));
}

// ---- two sources per instruction (packed FP32x2) ----
// Pair k of staged sources (2k, 2k + 1) is four 16-byte words
//   X[k] = (xh, xh', yh, yh'), Z[k] = (zh, zh', q, q'),
//   XL[k] = (xl, xl', yl, yl'), ZL[k] = (zl, zl', index, index'),
// and for dipoles D[k] = (mx, mx', my, my'), DZ[k] = (mz, mz', -, -)
// (primes: source 2k + 1).
typedef unsigned long long u64;
__device__ __forceinline__ u64 padd(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 psub(u64 a, u64 b) {
  u64 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 pmul(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 pfma(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ u64 pk2(float a, float b) {
  return ((u64)__float_as_uint(b) << 32) | (u64)__float_as_uint(a);
}
__device__ __forceinline__ float plo(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float phi_(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }

// staged chunk of one warp (64 sources)
struct P2PStage {
  ulonglong2 X[32], Z[32], XL[32], ZL[32];
};
struct P2PStageD {
  ulonglong2 D[32], DZ[32];
};
// One of the lane's two targets.
struct P2PTarget {
  int i;
  float hx, hy, hz, lx, ly, lz;  // offset from the root centre
  float s0 = 0, s1 = 0, s2 = 0, s3 = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0;
};

// The lane's targets on the staged pairs slice, slice + (1 << lf), ...: nb blocks
// of two.  SELF: the chunk may hold the targets.
template <bool SELF, bool POT, int SO>
__device__ __forceinline__ void p2p_pairs(const P2PStage &sg, const P2PStageD &sd, int slice, int lf, int nb,
                                          P2PTarget (&g)[2]) {
  u64 ph[2] = {}, ex[2] = {}, ey[2] = {}, ez[2] = {};
  u64 hx[2], hy[2], hz[2], lx[2], ly[2], lz[2];
#pragma unroll
  for (int t = 0; t < 2; t++) {
    hx[t] = pk2(g[t].hx, g[t].hx); hy[t] = pk2(g[t].hy, g[t].hy); hz[t] = pk2(g[t].hz, g[t].hz);
    lx[t] = pk2(g[t].lx, g[t].lx); ly[t] = pk2(g[t].ly, g[t].ly); lz[t] = pk2(g[t].lz, g[t].lz);
  }
  int k = slice;
#pragma unroll 1
  for (int b = 0; b < nb; b++)
#pragma unroll
    for (int u = 0; u < 2; u++, k += 1 << lf) {
      const ulonglong2 X = sg.X[k], Z = sg.Z[k], XL = sg.XL[k], ZL = sg.ZL[k];
      ulonglong2 D;
      u64 mz;
      if (SO) {
        D = sd.D[k];
        mz = sd.DZ[k].x;
      }
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const u64 dx = padd(psub(hx[t], X.x), psub(lx[t], XL.x));
        const u64 dy = padd(psub(hy[t], X.y), psub(ly[t], XL.y));
        const u64 dz = padd(psub(hz[t], Z.x), psub(lz[t], ZL.x));
        const u64 r2 = pfma(dx, dx, pfma(dy, dy, pmul(dz, dz)));
        float ra = rsqrt_approx(plo(r2)), rb = rsqrt_approx(phi_(r2));
        if (SELF) {  // l2 != l1
          ra = (int)(unsigned)ZL.y == g[t].i ? 0.f : ra;
          rb = (int)(unsigned)(ZL.y >> 32) == g[t].i ? 0.f : rb;
        }
        const u64 rinv = pk2(ra, rb);
        const u64 rr = pmul(rinv, rinv);
        if (SO == 0) {
          const u64 qr = pmul(Z.y, rinv);
          const u64 qr3 = pmul(qr, rr);
          if (POT) ph[t] = padd(ph[t], qr);
          ex[t] = pfma(qr3, dx, ex[t]);
          ey[t] = pfma(qr3, dy, ey[t]);
          ez[t] = pfma(qr3, dz, ez[t]);
        } else {
          const u64 r3 = pmul(rr, rinv);
          const u64 v = pmul(pfma(D.x, dx, pfma(D.y, dy, pmul(mz, dz))), r3);
          if (POT) ph[t] = psub(ph[t], v);
          const u64 r5 = pmul(pmul(pk2(-3.f, -3.f), rr), v);
          ex[t] = padd(ex[t], pfma(D.x, r3, pmul(r5, dx)));
          ey[t] = padd(ey[t], pfma(D.y, r3, pmul(r5, dy)));
          ez[t] = padd(ez[t], pfma(mz, r3, pmul(r5, dz)));
        }
      }
    }
#pragma unroll
  for (int t = 0; t < 2; t++) {
    if (POT) kahan_add(g[t].s0, g[t].c0, plo(ph[t]) + phi_(ph[t]));
    kahan_add(g[t].s1, g[t].c1, plo(ex[t]) + phi_(ex[t]));
    kahan_add(g[t].s2, g[t].c2, plo(ey[t]) + phi_(ey[t]));
    kahan_add(g[t].s3, g[t].c3, plo(ez[t]) + phi_(ez[t]));
  }
}

struct P2PArgs {
  const int4 *units;               // (cell, first target, targets, leaf)
  const int *pstart, *pcount, *off, *src;
  const float4 *phi4, *plo4, *sdip;
  const float *lpad;
  double *Fnear;
};

// The near field of the targets [tb, tb + m) of leaf cell A by one warp (sg, sd:
// its staging area; pad: a coordinate outside the root cube).
template <bool POT, int SO>
__device__ __forceinline__ void p2p_targets(const P2PArgs &P, int A, float pad, int tb, int m, P2PStage &sg,
                                            P2PStageD &sd) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int a0 = P.pstart[A];
  const int k0 = P.off[A], k1 = P.off[A + 1];
  const int lf = m > 16 ? 1 : m > 8 ? 2 : 3, half = 32 >> lf;  // targets tl and tl + half
  const int tl = lane >> lf, slice = lane - (tl << lf);
  P2PTarget g[2];
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const int tt = tl + t * half;
    g[t].i = a0 + tb + (tt < m ? tt : 0);
    const float4 h = P.phi4[g[t].i], l = P.plo4[g[t].i];
    g[t].hx = h.x; g[t].hy = h.y; g[t].hz = h.z;
    g[t].lx = l.x; g[t].ly = l.y; g[t].lz = l.z;
  }
  for (int kb = k0; kb < k1; kb += 32) {
    // up to 32 source leaves: lane q holds leaf kb + q's particle range
    const int nbat = min(32, k1 - kb);
    int B = -1, start = 0, cnt = 0;
    if (lane < nbat) {
      B = P.src[kb + lane];
      start = P.pstart[B];
      cnt = P.pcount[B];
    }
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += v;
    }
    const int excl = incl - cnt;
    const int total = __shfl_sync(FULL, incl, 31);
    const int shift = start - excl;  // stream place -> particle
    const int next = __shfl_down_sync(FULL, start, 1);  // of the next leaf
    // the targets' own places in the stream
    const unsigned selfq = __ballot_sync(FULL, B == A);
    const int self_lo = selfq ? __shfl_sync(FULL, excl, __ffs(selfq) - 1) + tb : 1 << 30;
#pragma unroll 1
    for (int cb = 0; cb < total; cb += 64) {
      // the lane's sources: s lies in the last leaf q whose stream offset is <= s
      const int s = cb + 2 * lane;
      int q = 0;
#pragma unroll
      for (int stp = 16; stp; stp >>= 1) {
        const int v = __shfl_sync(FULL, excl, q + stp);
        if (v <= s) q += stp;
      }
      const int j0 = s + __shfl_sync(FULL, shift, q), end = __shfl_sync(FULL, incl, q);
      const int jn = __shfl_sync(FULL, next, q);
      const int j1 = s + 1 < end ? j0 + 1 : jn;
      float4 h0 = make_float4(pad, pad, pad, 0.f), h1 = h0;
      float4 l0 = make_float4(0.f, 0.f, 0.f, __int_as_float(-1)), l1 = l0;
      float4 d0 = make_float4(0.f, 0.f, 0.f, 0.f), d1 = d0;
      if (s < total) {
        h0 = P.phi4[j0];
        l0 = P.plo4[j0];
        if (SO) d0 = P.sdip[j0];
      }
      if (s + 1 < total) {
        h1 = P.phi4[j1];
        l1 = P.plo4[j1];
        if (SO) d1 = P.sdip[j1];
      }
      __syncwarp();
      sg.X[lane] = make_ulonglong2(pk2(h0.x, h1.x), pk2(h0.y, h1.y));
      sg.Z[lane] = make_ulonglong2(pk2(h0.z, h1.z), pk2(h0.w, h1.w));
      sg.XL[lane] = make_ulonglong2(pk2(l0.x, l1.x), pk2(l0.y, l1.y));
      sg.ZL[lane] = make_ulonglong2(pk2(l0.z, l1.z), pk2(l0.w, l1.w));
      if (SO) {
        sd.D[lane] = make_ulonglong2(pk2(d0.x, d1.x), pk2(d0.y, d1.y));
        sd.DZ[lane].x = pk2(d0.z, d1.z);
      }
      __syncwarp();
      // blocks of 2 << lf pairs that hold the chunk's sources
      const int nb = (min(64, total - cb) + (4 << lf) - 1) >> (2 + lf);
      if (self_lo < cb + 64 && self_lo + m > cb) p2p_pairs<true, POT, SO>(sg, sd, slice, lf, nb, g);
      else p2p_pairs<false, POT, SO>(sg, sd, slice, lf, nb, g);
    }
  }
  // the lanes of each target
#pragma unroll
  for (int t = 0; t < 2; t++) {
    P2PTarget &r = g[t];
    for (int o = 1; o < 1 << lf; o <<= 1) {
      if (POT) pair_add(r.s0, r.c0, __shfl_xor_sync(FULL, r.s0, o), __shfl_xor_sync(FULL, r.c0, o));
      pair_add(r.s1, r.c1, __shfl_xor_sync(FULL, r.s1, o), __shfl_xor_sync(FULL, r.c1, o));
      pair_add(r.s2, r.c2, __shfl_xor_sync(FULL, r.s2, o), __shfl_xor_sync(FULL, r.c2, o));
      pair_add(r.s3, r.c3, __shfl_xor_sync(FULL, r.s3, o), __shfl_xor_sync(FULL, r.c3, o));
    }
    if (slice == t && tl + t * half < m) {
      double *F = P.Fnear + 4 * (size_t)r.i;
      F[0] = f2d(r.s0) - f2d(r.c0);
      F[1] = f2d(r.s1) - f2d(r.c1);
      F[2] = f2d(r.s2) - f2d(r.c2);
      F[3] = f2d(r.s3) - f2d(r.c3);
    }
  }
}

// Warps an SM: charges 16 (24: 10^6 uniform 3.98 ms, 10^4 0.10), dipoles 24 (16: 12.0 ms).
template <bool POT, int SO>
__global__ void __launch_bounds__(32, SO ? 24 : 16) k_p2p32(const P2PArgs P) {
  __shared__ P2PStage sg;
  __shared__ P2PStageD sd;
  const int4 u = P.units[blockIdx.x];
  p2p_targets<POT, SO>(P, u.x, P.lpad[u.w], u.y, u.z, sg, sd);
}

// ---------------------------------------------------------------------------
// launchers used by eval.cu
// ---------------------------------------------------------------------------
int fmm_p2p_launch(DevTree *t, bool mixed, const double *S, cudaStream_t st) {
  const int nl = t->nleaves, so = t->so;
  t->p64_last = !mixed;
  if (mixed && so <= 1) {  // quadrupole sources take the FP64 kernel in every precision
    const bool pot = t->pass_potential;
    decltype(&k_p2p32<true, 0>) k = so ? (pot ? k_p2p32<true, 1> : k_p2p32<false, 1>)
                                       : (pot ? k_p2p32<true, 0> : k_p2p32<false, 0>);
    const P2PArgs P = {t->p2p_units.p, t->pstart.p, t->pcount.p, t->p2p_off.p, t->p2p_src.p, t->phi4.p, t->plo4.p,
                       t->sdip.p, t->lpad.p, t->Fnear.p};
    if (int rc = fmm_mark_kernel(t, 2, st)) return rc;
    fmm_note_launch(), k<<<t->np2p_units, 32, 0, st>>>(P);
    FMM_CUDA_TRY(cudaGetLastError());
    return fmm_mark_kernel(t, 3, st);
  }
  const bool pot = t->pass_potential;
  bool once = so <= 1;
  if (once) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    FMM_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    if (cap == cudaStreamCaptureStatusNone)
      if (int rc = p64_layout(t, st)) return rc;
    once = t->sym_serial == t->build_serial && t->sym_places >= 0;  // a captured first pass may have none: one way
  }
  if (once) {
    const P64Args P = {t->sym_units.p, t->leaf_cells.p, t->pstart.p, t->pcount.p, t->p2p_off.p, t->p2p_src.p, t->px.p,
                       t->py.p, t->pz.p, t->perm.p, S, t->sym_own.p, t->sym_get.p,
                       t->sym_place.p + std::max(t->np2p, 1L), t->sym_shares.p, t->Fnear.p};
    decltype(&k_p2p64_sym<0, true>) k = so == 0 ? (pot ? k_p2p64_sym<0, true> : k_p2p64_sym<0, false>)
                                                : (pot ? k_p2p64_sym<1, true> : k_p2p64_sym<1, false>);
    if (int rc = fmm_mark_kernel(t, 2, st)) return rc;
    if (t->sym_nunits > 0) fmm_note_launch(), k<<<(unsigned)t->sym_nunits, 32, 0, st>>>(P);
    const unsigned grid = fmm_blocks(nl, 4);
    if (pot)
      fmm_note_launch(), k_p2p64_gather<true><<<grid, 128, 0, st>>>(P, nl);
    else
      fmm_note_launch(), k_p2p64_gather<false><<<grid, 128, 0, st>>>(P, nl);
  } else {
    const int nub = (int)fmm_blocks(t->np2p_units, P2P_WARPS);
    decltype(&k_p2p64<0, true>) k = so == 0   ? (pot ? k_p2p64<0, true> : k_p2p64<0, false>)
                                    : so == 1 ? (pot ? k_p2p64<1, true> : k_p2p64<1, false>)
                                              : k_p2p64<2, true>;
    if (int rc = fmm_mark_kernel(t, 2, st)) return rc;
    fmm_note_launch(), k<<<3 * (unsigned)nub, 32 * P2P_WARPS, 0, st>>>(
        t->p2p_units.p, t->np2p_units, nub, t->pstart.p, t->pcount.p, t->p2p_off.p, t->p2p_src.p, t->px.p, t->py.p,
        t->pz.p, t->perm.p, S, t->Fnear.p);
  }
  FMM_CUDA_TRY(cudaGetLastError());
  return fmm_mark_kernel(t, 3, st);
}

int fmm_stage_particles(DevTree *t, const double *S, cudaStream_t st) {
  if (t->so > 1) return FMM_OK;  // the FP64 P2P reads the sources directly
  if (int rc = fmm_reserve(t->lpad, t->nleaves)) return rc;
  fmm_note_launch(), k_stage_particles<<<fmm_blocks(t->N, 256), 256, 0, st>>>(
      t->N, t->leaf_cells.p, t->nleaves, t->csys.p, t->nsys > 1 ? t->psys.p : nullptr, t->roots.p, t->px.p, t->py.p,
      t->pz.p, t->perm.p, S, t->so, t->phi4.p, t->plo4.p, t->sdip.p, t->lpad.p);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

// ---------------------------------------------------------------------------
// direct O(N^2) sum in FP64 (example/calculate.cpp:252-264)
// ---------------------------------------------------------------------------
// FP64-bound like k_p2p64.  A group of 32 targets (one per lane; fewer than 32
// targets in all share the lanes) is one cluster of blocks: its 8 warps per block
// take the source chunks in turn, and the partial sums are added in a fixed
// order through (distributed) shared memory.  The cluster is as large as it
// takes to give every SM its share of warps: one thread per target over all
// sources was 235 blocks of 128 threads at 30,011 targets, two waves of which
// the second was half empty.  30,011 x 30,011 charges: 57.8 -> 32.9 ms (the square
// root and division of every pair became one reciprocal square root).
#define DIR_WARPS 8
template <int SO>
__global__ void __launch_bounds__(32 * DIR_WARPS) k_direct(const double *pos, const double *S, long N,
                                                           const long *targets, long nt, int m, int potential,
                                                           int field, double *F) {
  constexpr int NQ = p64_nq(SO);
  constexpr unsigned FULL = 0xffffffffu;
  // one warp's staged sources, later its 32 lanes' sums
  constexpr int AREA = (3 + NQ) * P64_CHUNK;
  static_assert(AREA >= 4 * 32, "the sums reuse the staging area");
  __shared__ double sm[DIR_WARPS][AREA];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned nrank = cluster.num_blocks(), rank = cluster.block_rank();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double(*sp)[P64_CHUNK] = (double(*)[P64_CHUNK])sm[w];
  double(*sq)[P64_CHUNK] = sp + 3;
  // m targets per group, f = 32 / m lanes per target
  const int f = 32 / m, tl = lane / f, slice = lane - tl * f;
  const long t = (long)(blockIdx.x / nrank) * m + tl;
  const long i = tl < m && t < nt ? (targets ? targets[t] : t) : -1;
  const bool ok = i >= 0;  // a negative target has no particle: its row stays as it is
  double xi = 0, yi = 0, zi = 0;
  if (ok) {
    xi = pos[3 * i];
    yi = pos[3 * i + 1];
    zi = pos[3 * i + 2];
  }
  double phi = 0, ex = 0, ey = 0, ez = 0;
  for (long b = (long)(rank * DIR_WARPS + w) * P64_CHUNK; b < N; b += (long)nrank * DIR_WARPS * P64_CHUNK) {
    const int n = (int)min((long)P64_CHUNK, N - b);
    __syncwarp();
    for (int j = lane; j < n; j += 32) {
#pragma unroll
      for (int k = 0; k < 3; k++) sp[k][j] = pos[3 * (b + j) + k];
#pragma unroll
      for (int k = 0; k < NQ; k++) sq[k][j] = S[NQ * (b + j) + k];
    }
    __syncwarp();
    if (!ok) continue;
    const int me = i >= b && i < b + n ? (int)(i - b) : -1;
#pragma unroll 2
    for (int jj = slice; jj < n; jj += f)
      p64_one<SO, true, true>(xi - sp[0][jj], yi - sp[1][jj], zi - sp[2][jj], sq, jj, jj == me, phi, ex, ey, ez);
  }
  __syncwarp();
  double v[4] = {phi, ex, ey, ez};
  for (int o = 16; o; o >>= 1) {
    if (o >= f) continue;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double u = __shfl_down_sync(FULL, v[k], o);
      if (slice < o && slice + o < f) v[k] += u;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; k++) sm[w][32 * k + lane] = v[k];
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k] = sm[0][32 * k + lane];
      for (int u = 1; u < DIR_WARPS; u++) v[k] += sm[u][32 * k + lane];
      sm[0][32 * k + lane] = v[k];
    }
  }
  cluster.sync();
  if (rank == 0 && w == 0) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      for (unsigned r = 1; r < nrank; r++) v[k] += cluster.map_shared_rank(&sm[0][0], r)[32 * k + lane];
    if (ok && slice == 0) {
      double *o = F + (size_t)t * ((potential ? 1 : 0) + (field ? 3 : 0));
      if (potential) *o++ = v[0];
      if (field) {
        o[0] = v[1];
        o[1] = v[2];
        o[2] = v[3];
      }
    }
  }
  cluster.sync();  // the sums stay readable until rank 0 has added them
}

// All particles on all others, each pair once (as k_p2p64_sym): a block takes a
// pair of tiles of 256 particles, a warp 32 of the first tile's as targets, and
// the block goes over the second tile's in chunks of 32; each warp adds the
// chunk's side up in shared memory of its own.  Both sides' sums go into
// parts[tile][other tile][256], which k_direct_sum adds up in order.  The line: 16
// tiles, whose 136 pairs come near the number of SMs.  Charges, one way and each pair
// once: 3,000 0.52 and 0.56 ms, 4,096 0.69 and 0.57, 5,000 1.25 and 0.97, 12,000 4.87 and
// 3.36, 30,011 32.9 and 18.6 ms; 4,096 dipoles 1.09 and 0.95.
constexpr int DIR_TILE = 32 * DIR_WARPS;
constexpr long DIR_SYM_MIN = 16 * DIR_TILE;
template <int SO>
__global__ void __launch_bounds__(DIR_TILE) k_direct_sym(const double *pos, const double *S, long N, int nt,
                                                         double *parts) {
  constexpr int NQ = p64_nq(SO);
  __shared__ double sp[3][32], sq[NQ][P64_CHUNK], acc[DIR_WARPS][4][32];
  // block -> tiles I <= J: J (J + 1) / 2 + I
  const long b = blockIdx.x;
  long J = (long)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
  while (J * (J + 1) / 2 > b) J--;
  while ((J + 1) * (J + 2) / 2 <= b) J++;
  const long I = b - J * (J + 1) / 2;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long i = I * DIR_TILE + threadIdx.x;
  const bool ok = i < N;
  const long ii = ok ? i : N - 1;
  const double xi = pos[3 * ii], yi = pos[3 * ii + 1], zi = pos[3 * ii + 2];
  double si[NQ];
#pragma unroll
  for (int k = 0; k < NQ; k++) si[k] = S[NQ * ii + k];
  double phi = 0, ex = 0, ey = 0, ez = 0;
  double *const side = parts + 4 * DIR_TILE * (J * nt + I);  // tile J's from tile I
  for (int c = 0; c < DIR_WARPS; c++) {
    const long j0 = J * DIR_TILE + 32 * c;
    const int n = (int)min(32L, N - j0);
    if (n <= 0) break;
    __syncthreads();
    if (w == 0 && lane < n) {
#pragma unroll
      for (int k = 0; k < 3; k++) sp[k][lane] = pos[3 * (j0 + lane) + k];
#pragma unroll
      for (int k = 0; k < NQ; k++) sq[k][lane] = S[NQ * (j0 + lane) + k];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) acc[w][k][lane] = 0.0;
    __syncthreads();
    if (I == J) {  // a tile on itself: one way
      const int me = i >= j0 && i < j0 + n ? (int)(i - j0) : -1;
      if (ok)
        for (int jj = 0; jj < n; jj++)
          p64_one<SO, true, true>(xi - sp[0][jj], yi - sp[1][jj], zi - sp[2][jj], sq, jj, jj == me, phi, ex, ey, ez);
      continue;
    }
    for (int st = 0; st < 32; st++) {
      const int jj = (st + lane) & 31;
      if (ok && jj < n)
        p64_both<SO, true, 32>(xi - sp[0][jj], yi - sp[1][jj], zi - sp[2][jj], sq, jj, si, phi, ex, ey, ez, acc[w], jj);
      __syncwarp();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 128; e += DIR_TILE) {
      const int j = e >> 2, k = e & 3;
      double v = acc[0][k][j];
#pragma unroll
      for (int u = 1; u < DIR_WARPS; u++) v += acc[u][k][j];
      side[4 * (32 * c + j) + k] = v;
    }
  }
  double *o = parts + 4 * (DIR_TILE * (I * nt + J) + threadIdx.x);
  o[0] = phi;
  o[1] = ex;
  o[2] = ey;
  o[3] = ez;
}

__global__ void k_direct_sum(const double *parts, long N, int nt, int potential, int field, double *F) {
  const long i = blockIdx.x * (long)DIR_TILE + threadIdx.x;
  if (i >= N) return;
  const double *p = parts + 4 * ((long)DIR_TILE * nt * blockIdx.x + threadIdx.x);
  double v[4] = {0, 0, 0, 0};
  for (int j = 0; j < nt; j++, p += 4 * DIR_TILE)
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] += p[k];
  double *o = F + (size_t)i * ((potential ? 1 : 0) + (field ? 3 : 0));
  if (potential) *o++ = v[0];
  if (field) {
    o[0] = v[1];
    o[1] = v[2];
    o[2] = v[3];
  }
}

int fmm_direct(const double *pos, const double *S, long N, const long *targets, long ntargets, int so,
               int potential, int field, double *F, cudaStream_t st) {
  if (!pos || !S || !F || N < 1 || (!potential && !field) || so < 0 || so > 2) return FMM_ERR_ARG;
  const long nt = targets ? ntargets : N;
  if (nt < 1) return FMM_OK;
  // each pair once where both sides are asked for and the parts (N^2 / 8 bytes, from the stream's memory pool
  // for the call) can be had; a capture would keep them with its graph
  const long tiles = (N + DIR_TILE - 1) / DIR_TILE;
  const size_t bytes = sizeof(double) * 4 * DIR_TILE * (size_t)(tiles * tiles);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FMM_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
  if (!targets && so <= 1 && N >= DIR_SYM_MIN && bytes <= P64_SHARES && cap == cudaStreamCaptureStatusNone) {
    double *parts = nullptr;
    if (cudaMallocAsync((void **)&parts, bytes, st) == cudaSuccess) {
      const unsigned nb = (unsigned)(tiles * (tiles + 1) / 2);
      if (so == 0) fmm_note_launch(), k_direct_sym<0><<<nb, DIR_TILE, 0, st>>>(pos, S, N, (int)tiles, parts);
      else fmm_note_launch(), k_direct_sym<1><<<nb, DIR_TILE, 0, st>>>(pos, S, N, (int)tiles, parts);
      fmm_note_launch(), k_direct_sum<<<(unsigned)tiles, DIR_TILE, 0, st>>>(parts, N, (int)tiles, potential, field, F);
      const cudaError_t e = cudaGetLastError();
      FMM_CUDA_TRY(cudaFreeAsync(parts, st));
      FMM_CUDA_TRY(e);
      return FMM_OK;
    }
    cudaGetLastError();  // no memory: one way
  }
  const int m = (int)std::min(nt, 32L);
  const long groups = (nt + m - 1) / m;
  // at least four blocks of warps per SM, as long as every warp has sources to take
  int c = 1;
  while (c < 8 && groups * c < 4 * 152 && (long)c * DIR_WARPS * P64_CHUNK < N) c *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups * c));
  cfg.blockDim = dim3(32 * DIR_WARPS);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)c;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  fmm_note_launch();
  FMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, so == 0 ? k_direct<0> : so == 1 ? k_direct<1> : k_direct<2>, pos, S, N,
                                  targets, nt, m, potential, field, F));
  return FMM_OK;
}
