// p2p.cu -- near-field particle-particle interactions (P2P) over the P2P list
// (P2P_Cells / evaluate_P2P_lazy, example/calculate.cpp:24-40, 208-216), in FP64
// and in the mixed-precision form, plus the per-evaluate FP32 staging.
#include <algorithm>
#include <cooperative_groups.h>
#include "internal.h"

// ---------------------------------------------------------------------------
// P2P in FP64 (example/calculate.cpp:24-40, 208-216)
// ---------------------------------------------------------------------------
// Bound by the FP64 pipe: 1.60 operations per clock and SM measured on this
// part (FP32: 120), so a warp's FP64 instruction takes 20 clocks of its SM and
// everything else -- shared-memory reads, index arithmetic, shuffles, staging
// the sources again -- hides behind it.  What counts is that no lane idles.
// A leaf's targets are therefore cut into groups that fill the warp: chunks of
// 32, then 16 and 8 targets with 2 and 4 lanes each, then the last m <= 7 with
// floor(32 / m) lanes each; the f lanes of a target take every f-th source of
// the stream and their sums are added at the end.  One warp per (leaf, group):
// the groups of a leaf are independent warps, so leaves of several chunks do
// not make a tail of long warps.  With one lane per target and chunks of 32 a
// leaf of 14 left 56 % of the lanes idle and one of 40 took two full passes.
// The sources of the leaf's list are one stream (the leaves' particle ranges
// one after the other), staged 64 at a time.
// Measured (one GB300): 10^6 uniform charges, 30 per leaf, 4.79e9 interactions:
// 229 -> 158 ms; 100,003 clustered charges, 14 per leaf: the whole step 28.0 -> 17.1 ms; 86,400 dipoles, 11 per
// leaf: 25.8 -> 10.2 ms.
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
__global__ void __launch_bounds__(32 * P2P_WARPS) k_p2p64(const int *leaf_cells, int nleaves, int nlb, int nchunk,
                                                          const int *pstart, const int *pcount, const int *off_,
                                                          const int *src, const double *px, const double *py,
                                                          const double *pz, const uint32_t *perm, const double *S,
                                                          double *Fnear) {
  constexpr int NQ = p64_nq(SO);
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ double sp[P2P_WARPS][3][P64_CHUNK], sq[P2P_WARPS][NQ][P64_CHUNK];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int y = blockIdx.x / nlb;  // blocks by group: every leaf's first chunk, then the second ones, ...
  const int leaf = (blockIdx.x - y * nlb) * P2P_WARPS + w;
  if (leaf >= nleaves) return;
  const int A = leaf_cells[leaf];
  const int a0 = pstart[A], na = pcount[A];
  // this warp's group of targets: [tb, tb + m)
  const int full = na & ~31, rest = na & 31;
  int tb, m;
  if (y < nchunk) {  // a chunk of 32
    tb = 32 * y;
    m = tb < full ? 32 : 0;
  } else if (y == nchunk) {
    tb = full;
    m = rest & 16;
  } else if (y == nchunk + 1) {
    tb = full + (rest & 16);
    m = rest & 8;
  } else {
    tb = full + (rest & 24);
    m = rest & 7;
  }
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

// Per evaluate: positions as two-float offsets from the particle's system root
// centre (hi in .xyz, the charge in .w; lo in .xyz, the particle's own index
// in .w for the self test); dipole moments in FP32.
__global__ void k_stage_particles(const int *leaf_cells, int nleaves, const int *pstart, const int *pcount,
                                  const int *csys, const double *roots, const double *px, const double *py,
                                  const double *pz, const uint32_t *perm, const double *S, int so, float4 *phi4,
                                  float4 *plo4, float4 *sdip) {
  int leaf = blockIdx.x;
  if (leaf >= nleaves) return;
  int c = leaf_cells[leaf];
  const double *root = roots + 4 * (size_t)csys[c];
  const double ox = root[0], oy = root[1], oz = root[2];
  for (int j = threadIdx.x; j < pcount[c]; j += blockDim.x) {
    int i = pstart[c] + j;
    double dx = px[i] - ox, dy = py[i] - oy, dz = pz[i] - oz;
    float hx = (float)dx, hy = (float)dy, hz = (float)dz;
    uint32_t o = perm[i];
    phi4[i] = make_float4(hx, hy, hz, so == 0 ? (float)S[o] : 0.f);
    plo4[i] = make_float4((float)(dx - (double)hx), (float)(dy - (double)hy), (float)(dz - (double)hz),
                          __int_as_float(i));
    if (so) sdip[i] = make_float4((float)S[3 * (size_t)o], (float)S[3 * (size_t)o + 1], (float)S[3 * (size_t)o + 2], 0.f);
  }
}


// ---------------------------------------------------------------------------
// P2P in FP32 with compensated accumulation (mixed precision)
// ---------------------------------------------------------------------------
// One warp per target leaf, in chunks of up to 32 target particles.  The
// source particles of the leaf's P2P list are taken as one stream -- the
// concatenation of the source leaves' particle ranges, up to 32 leaves at a
// time -- and staged in full chunks of 32, so that the per-chunk work (finding
// each lane's source through a prefix sum of the leaves' counts, the staging
// copy, the compensated fold) is spread over 32 sources rather than one leaf's
// ~30.  A chunk of m targets uses f = the largest power of two with f*m <= 32
// lanes per target, each lane taking every f-th source, so a small chunk (a
// leaf's last few particles) does not leave most lanes idle; the f partial sums
// of a target are combined with shuffles.
// Positions are two-float offsets from the system's root centre: the high
// parts of two nearby particles subtract exactly (Sterbenz) or with one
// rounding of the difference, and the low parts carry the rest, so the
// displacement keeps ~1e-7 relative accuracy even for very close pairs.  Each
// chunk's contribution is summed in FP32 and folded into a Kahan-compensated
// FP32 total; the final per-particle near + far sum is FP64 (k_finalize).
// 1/R is the hardware approximation (relative error ~1e-7, the size of the
// FP32 displacement's own rounding).  The potential is summed only when it is
// an output.
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

template <bool SELF, bool POT>
__device__ __forceinline__ void coulomb_one(const float4 &q, const float4 &ql, int i, float txh, float txl, float tyh,
                                            float tyl, float tzh, float tzl, float &phi, float &ex, float &ey,
                                            float &ez) {
  const float dx = (txh - q.x) + (txl - ql.x);
  const float dy = (tyh - q.y) + (tyl - ql.y);
  const float dz = (tzh - q.z) + (tzl - ql.z);
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  float rinv = rsqrt_approx(r2);
  if (SELF) rinv = __float_as_int(ql.w) == i ? 0.f : rinv;  // l2 != l1
  const float qr = q.w * rinv;
  const float qr3 = qr * (rinv * rinv);
  if (POT) phi += qr;
  ex = fmaf(qr3, dx, ex);
  ey = fmaf(qr3, dy, ey);
  ez = fmaf(qr3, dz, ez);
}

template <bool SELF>
__device__ __forceinline__ void dipole_one(const float4 &q, const float4 &ql, const float4 &d, int i, float txh,
                                           float txl, float tyh, float tyl, float tzh, float tzl, float &phi,
                                           float &ex, float &ey, float &ez) {
  const float dx = (txh - q.x) + (txl - ql.x);
  const float dy = (tyh - q.y) + (tyl - ql.y);
  const float dz = (tzh - q.z) + (tzl - ql.z);
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  float rinv = rsqrt_approx(r2);
  if (SELF) rinv = __float_as_int(ql.w) == i ? 0.f : rinv;
  const float r3 = rinv * rinv * rinv;
  const float sr = fmaf(d.x, dx, fmaf(d.y, dy, d.z * dz));
  const float r5 = 3.f * sr * r3 * rinv * rinv;
  phi -= sr * r3;
  ex += d.x * r3 - r5 * dx;
  ey += d.y * r3 - r5 * dy;
  ez += d.z * r3 - r5 * dz;
}

// ---- two sources per instruction (packed FP32x2) ----
// A full chunk with one lane per target (the common case) runs two sources at a
// time through add/sub/mul/fma.rn.f32x2: the same operations, in the same
// precision, as coulomb_one / dipole_one for each source of the pair, with half
// the instructions (the kernel is issue-bound).  Staged chunks are laid out for
// this: pair k of sources (2k, 2k+1) is four 16-byte words
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

// staged chunk of one warp (32 sources)
struct P2PStage {
  ulonglong2 X[16], Z[16], XL[16], ZL[16];
};
struct P2PStageD {
  ulonglong2 D[16], DZ[16];
};
__device__ __forceinline__ float *sf(ulonglong2 *a) { return (float *)a; }
__device__ __forceinline__ const float *sf(const ulonglong2 *a) { return (const float *)a; }

// the target's coordinates (hi, lo) duplicated into both halves
struct P2PTgt {
  u64 xh, xl, yh, yl, zh, zl;
};

template <bool SELF, bool POT>
__device__ __forceinline__ void coulomb_two(const P2PStage &sg, int k, int i, const P2PTgt &t, u64 &phi, u64 &ex,
                                            u64 &ey, u64 &ez) {
  const ulonglong2 X = sg.X[k], Z = sg.Z[k], XL = sg.XL[k], ZL = sg.ZL[k];
  const u64 dx = padd(psub(t.xh, X.x), psub(t.xl, XL.x));
  const u64 dy = padd(psub(t.yh, X.y), psub(t.yl, XL.y));
  const u64 dz = padd(psub(t.zh, Z.x), psub(t.zl, ZL.x));
  const u64 r2 = pfma(dx, dx, pfma(dy, dy, pmul(dz, dz)));
  float ra = rsqrt_approx(plo(r2)), rb = rsqrt_approx(phi_(r2));
  if (SELF) {  // l2 != l1
    ra = (int)(unsigned)ZL.y == i ? 0.f : ra;
    rb = (int)(unsigned)(ZL.y >> 32) == i ? 0.f : rb;
  }
  const u64 rinv = pk2(ra, rb);
  const u64 qr = pmul(Z.y, rinv);
  const u64 qr3 = pmul(qr, pmul(rinv, rinv));
  if (POT) phi = padd(phi, qr);
  ex = pfma(qr3, dx, ex);
  ey = pfma(qr3, dy, ey);
  ez = pfma(qr3, dz, ez);
}

template <bool SELF>
__device__ __forceinline__ void dipole_two(const P2PStage &sg, const P2PStageD &sd, int k, int i, const P2PTgt &t,
                                           u64 &phi, u64 &ex, u64 &ey, u64 &ez) {
  const ulonglong2 X = sg.X[k], Z = sg.Z[k], XL = sg.XL[k], ZL = sg.ZL[k], D = sd.D[k];
  const u64 mz = sd.DZ[k].x;
  const u64 dx = padd(psub(t.xh, X.x), psub(t.xl, XL.x));
  const u64 dy = padd(psub(t.yh, X.y), psub(t.yl, XL.y));
  const u64 dz = padd(psub(t.zh, Z.x), psub(t.zl, ZL.x));
  const u64 r2 = pfma(dx, dx, pfma(dy, dy, pmul(dz, dz)));
  float ra = rsqrt_approx(plo(r2)), rb = rsqrt_approx(phi_(r2));
  if (SELF) {
    ra = (int)(unsigned)ZL.y == i ? 0.f : ra;
    rb = (int)(unsigned)(ZL.y >> 32) == i ? 0.f : rb;
  }
  const u64 rinv = pk2(ra, rb);
  const u64 rr = pmul(rinv, rinv);
  const u64 r3 = pmul(rr, rinv);
  const u64 sr = pfma(D.x, dx, pfma(D.y, dy, pmul(mz, dz)));
  const u64 r5 = pmul(pmul(pmul(pk2(3.f, 3.f), sr), r3), rr);
  phi = psub(phi, pmul(sr, r3));
  ex = padd(ex, psub(pmul(D.x, r3), pmul(r5, dx)));
  ey = padd(ey, psub(pmul(D.y, r3), pmul(r5, dy)));
  ez = padd(ez, psub(pmul(mz, r3), pmul(r5, dz)));
}

// one source of the packed layout, for partial chunks
__device__ __forceinline__ void stage_get(const P2PStage &sg, int j, float4 &h, float4 &l) {
  const int o = 4 * (j >> 1) + (j & 1);
  const float *x = sf(sg.X) + o, *z = sf(sg.Z) + o, *xl = sf(sg.XL) + o, *zl = sf(sg.ZL) + o;
  h = make_float4(x[0], x[2], z[0], z[2]);
  l = make_float4(xl[0], xl[2], zl[0], zl[2]);
}
__device__ __forceinline__ float4 stage_getd(const P2PStageD &sd, int j) {
  const int o = 4 * (j >> 1) + (j & 1);
  const float *d = sf(sd.D) + o, *dz = sf(sd.DZ) + o;
  return make_float4(d[0], d[2], dz[0], 0.f);
}

// Sources first, first + step, ... < cnt of the staged chunk.
template <bool SELF, bool POT, int SO>
__device__ __forceinline__ void p2p_chunk(const P2PStage &sg, const P2PStageD &sd, int first, int cnt, int step,
                                          int i, const P2PTgt &t, float txh, float txl, float tyh, float tyl,
                                          float tzh, float tzl, float &phi, float &ex, float &ey, float &ez) {
  if (step == 1 && cnt == 32) {
    u64 p2 = 0, x2 = 0, y2 = 0, z2 = 0;
#pragma unroll 4
    for (int k = 0; k < 16; k++) {
      if (SO == 0)
        coulomb_two<SELF, POT>(sg, k, i, t, p2, x2, y2, z2);
      else
        dipole_two<SELF>(sg, sd, k, i, t, p2, x2, y2, z2);
    }
    if (POT || SO) phi += plo(p2) + phi_(p2);
    ex += plo(x2) + phi_(x2);
    ey += plo(y2) + phi_(y2);
    ez += plo(z2) + phi_(z2);
    return;
  }
#pragma unroll 4
  for (int jj = first; jj < cnt; jj += step) {
    float4 h, l;
    stage_get(sg, jj, h, l);
    if (SO == 0)
      coulomb_one<SELF, POT>(h, l, i, txh, txl, tyh, tyl, tzh, tzl, phi, ex, ey, ez);
    else
      dipole_one<SELF>(h, l, stage_getd(sd, jj), i, txh, txl, tyh, tyl, tzh, tzl, phi, ex, ey, ez);
  }
}

// The near field of target leaf A by one warp (sg, sd: its staging area).
template <bool POT, int SO>
__device__ __forceinline__ void p2p_leaf(int A, const int *pstart, const int *pcount, const int *off_,
                                         const int *src, const float4 *phi4, const float4 *plo4,
                                         const float4 *sdip, P2PStage &sg, P2PStageD &sd, double *Fnear) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int a0 = pstart[A], na = pcount[A];
  const int k0 = off_[A], k1 = off_[A + 1];
  const int sk = 4 * (lane >> 1) + (lane & 1);  // this lane's slot when it stages source `lane` of a chunk
  for (int tb = 0; tb < na; tb += 32) {
    const int m = min(32, na - tb);
    int lf = 0;  // f = 2^lf lanes per target
    while ((2 << lf) * m <= 32) lf++;
    const int f = 1 << lf;
    const int tl = lane >> lf, slice = lane & (f - 1);
    const bool ok = tl < m;
    const int i = a0 + tb + (ok ? tl : 0);
    const float4 th = phi4[i], tlo = plo4[i];
    const P2PTgt tg = {pk2(th.x, th.x), pk2(tlo.x, tlo.x), pk2(th.y, th.y),
                       pk2(tlo.y, tlo.y), pk2(th.z, th.z), pk2(tlo.z, tlo.z)};
    float s0 = 0, s1 = 0, s2 = 0, s3 = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    for (int kb = k0; kb < k1; kb += 32) {
      // up to 32 source leaves: lane q holds leaf kb + q's particle range and
      // the exclusive prefix of the counts (its offset in the stream)
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
      // the target leaf's own range in the stream (self pairs skip i == j)
      const unsigned selfq = __ballot_sync(FULL, B == A);
      const int self_lo = selfq ? __shfl_sync(FULL, excl, __ffs(selfq) - 1) : -1;
      for (int cb = 0; cb < total; cb += 32) {
        // the lane's source: the last leaf q whose stream offset is <= s
        const int s = cb + lane;
        int q = 0;
#pragma unroll
        for (int stp = 16; stp; stp >>= 1) {
          const int cand = q + stp;
          const int v = __shfl_sync(FULL, excl, cand & 31);
          if (cand < nbat && v <= s) q = cand;
        }
        const int jb = __shfl_sync(FULL, start, q), je = __shfl_sync(FULL, excl, q);
        __syncwarp();
        if (s < total) {
          const int j = jb + (s - je);
          const float4 h = phi4[j], l = plo4[j];
          sf(sg.X)[sk] = h.x; sf(sg.X)[sk + 2] = h.y;
          sf(sg.Z)[sk] = h.z; sf(sg.Z)[sk + 2] = h.w;
          sf(sg.XL)[sk] = l.x; sf(sg.XL)[sk + 2] = l.y;
          sf(sg.ZL)[sk] = l.z; sf(sg.ZL)[sk + 2] = l.w;
          if (SO) {
            const float4 d = sdip[j];
            sf(sd.D)[sk] = d.x; sf(sd.D)[sk + 2] = d.y;
            sf(sd.DZ)[sk] = d.z;
          }
        }
        __syncwarp();
        const int n = min(32, total - cb);
        const bool self = self_lo >= 0 && self_lo < cb + n && self_lo + na > cb;
        float phi = 0, ex = 0, ey = 0, ez = 0;
        if (self)
          p2p_chunk<true, POT, SO>(sg, sd, slice, n, f, i, tg, th.x, tlo.x, th.y, tlo.y, th.z, tlo.z, phi, ex, ey,
                                   ez);
        else
          p2p_chunk<false, POT, SO>(sg, sd, slice, n, f, i, tg, th.x, tlo.x, th.y, tlo.y, th.z, tlo.z, phi, ex, ey,
                                    ez);
        if (POT) kahan_add(s0, c0, phi);
        kahan_add(s1, c1, ex); kahan_add(s2, c2, ey); kahan_add(s3, c3, ez);
      }
    }
    // combine the f lanes of each target in FP64
    double r0 = (double)s0 - (double)c0, r1 = (double)s1 - (double)c1;
    double r2 = (double)s2 - (double)c2, r3 = (double)s3 - (double)c3;
    for (int o = 1; o < f; o <<= 1) {
      r0 += __shfl_xor_sync(FULL, r0, o);
      r1 += __shfl_xor_sync(FULL, r1, o);
      r2 += __shfl_xor_sync(FULL, r2, o);
      r3 += __shfl_xor_sync(FULL, r3, o);
    }
    if (ok && slice == 0) {
      Fnear[4 * (size_t)i] = r0;
      Fnear[4 * (size_t)i + 1] = r1;
      Fnear[4 * (size_t)i + 2] = r2;
      Fnear[4 * (size_t)i + 3] = r3;
    }
  }
}

template <bool POT, int WARPS, int SO>
__global__ void __launch_bounds__(32 * WARPS) k_p2p32(const int *leaf_cells, int nleaves, const int *pstart,
                                                      const int *pcount, const int *off_, const int *src,
                                                      const float4 *phi4, const float4 *plo4, const float4 *sdip,
                                                      double *Fnear) {
  __shared__ P2PStage sg[WARPS];
  __shared__ P2PStageD sd[SO ? WARPS : 1];
  const int w = threadIdx.x >> 5;
  const int leaf = blockIdx.x * WARPS + w;
  if (leaf < nleaves)
    p2p_leaf<POT, SO>(leaf_cells[leaf], pstart, pcount, off_, src, phi4, plo4, sdip, sg[w], sd[SO ? w : 0], Fnear);
}

// ---------------------------------------------------------------------------
// launchers used by eval.cu
// ---------------------------------------------------------------------------
int fmm_p2p_launch(DevTree *t, bool mixed, const double *S, cudaStream_t st, bool narrow) {
  const int nl = t->nleaves, so = t->so;
  if (mixed && so <= 1) {  // quadrupole sources take the FP64 kernel in every precision
    // narrow blocks (2 warps) when running beside the tensor-core M2L: they
    // fit in the registers its CTA leaves free
    const bool pot = t->pass_potential || so;
    const int wp = narrow ? 2 : P2P_WARPS;
    decltype(&k_p2p32<true, 2, 0>) k;
    if (so)
      k = narrow ? k_p2p32<true, 2, 1> : k_p2p32<true, P2P_WARPS, 1>;
    else
      k = narrow ? (pot ? k_p2p32<true, 2, 0> : k_p2p32<false, 2, 0>)
                 : (pot ? k_p2p32<true, P2P_WARPS, 0> : k_p2p32<false, P2P_WARPS, 0>);
    const unsigned grid = fmm_blocks(nl, wp);
    if (int rc = fmm_mark_kernel(t, 2, st)) return rc;
    fmm_note_launch(), k<<<grid, 32 * wp, 0, st>>>(t->leaf_cells.p, nl, t->pstart.p, t->pcount.p, t->p2p_off.p,
                                                   t->p2p_src.p, t->phi4.p, t->plo4.p, t->sdip.p, t->Fnear.p);
  } else {
    // a leaf holds fewer than ncrit particles (a root leaf fewer than N): its full chunks of 32, then three groups
    const bool pot = t->pass_potential;
    const int nchunk = (int)(std::min(t->ncrit - 1, t->N) / 32);
    const int nlb = (int)fmm_blocks(nl, P2P_WARPS);
    decltype(&k_p2p64<0, true>) k = so == 0   ? (pot ? k_p2p64<0, true> : k_p2p64<0, false>)
                                    : so == 1 ? (pot ? k_p2p64<1, true> : k_p2p64<1, false>)
                                              : k_p2p64<2, true>;
    if (int rc = fmm_mark_kernel(t, 2, st)) return rc;
    fmm_note_launch(), k<<<(unsigned)nlb * (nchunk + 3), 32 * P2P_WARPS, 0, st>>>(
        t->leaf_cells.p, nl, nlb, nchunk, t->pstart.p, t->pcount.p, t->p2p_off.p, t->p2p_src.p, t->px.p, t->py.p, t->pz.p,
        t->perm.p, S, t->Fnear.p);
  }
  FMM_CUDA_TRY(cudaGetLastError());
  return fmm_mark_kernel(t, 3, st);
}

int fmm_stage_particles(DevTree *t, const double *S, cudaStream_t st) {
  if (t->so > 1) return FMM_OK;  // the FP64 P2P reads the sources directly
  fmm_note_launch(), k_stage_particles<<<t->nleaves, 128, 0, st>>>(
      t->leaf_cells.p, t->nleaves, t->pstart.p, t->pcount.p, t->csys.p, t->roots.p, t->px.p, t->py.p, t->pz.p,
      t->perm.p, S, t->so, t->phi4.p, t->plo4.p, t->sdip.p);
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
  const bool ok = tl < m && t < nt;
  const long i = ok ? (targets ? targets[t] : t) : -1;
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

int fmm_direct(const double *pos, const double *S, long N, const long *targets, long ntargets, int so,
               int potential, int field, double *F, cudaStream_t st) {
  if (!pos || !S || !F || N < 1 || (!potential && !field) || so < 0 || so > 2) return FMM_ERR_ARG;
  const long nt = targets ? ntargets : N;
  if (nt < 1) return FMM_OK;
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
