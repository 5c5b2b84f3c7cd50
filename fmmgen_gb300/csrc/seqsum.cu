// seqsum.cu -- the reference's sequential FP64 sum, reproduced bit for bit in
// parallel.
//
// build_tree centres the root cube on the mean position, accumulated as
//   s = 0; for i in 0..N-1: s = fl(s + x_i)                 (example/tree.cpp:148-156)
// Every tree decision downstream depends on the bits of that sum, so it must be
// reproduced exactly, not merely accurately.  A single dependent chain of FP64
// adds costs ~70 cycles per element on GB300's narrow FP64 pipe (~40 ms for
// 10^6 particles), so the chain is broken up:
//
//  While s stays inside one binade [2^e, 2^(e+1)) its ulp u = 2^(e-52) is fixed
//  and s is an integer S in units of u.  Adding x then rounds the exact sum to
//  the u grid:  S' = S + round(x / u), with the tie (x/u exactly half-way)
//  going to the even neighbour, i.e. depending only on the parity of S.  So
//  over a chunk of elements the whole chain is an integer map
//      S -> S + A[S mod 2]
//  valid while every intermediate S stays in [2^52, 2^53) (or its negative
//  mirror).  Chunks are analysed in parallel (integer arithmetic on the
//  mantissa bits, no FP64 pipe), with the binade guessed from an ordinary
//  parallel prefix sum.
//
//  A chunk that leaves its binade has no such map, but the prefix sum tells
//  where: the guess is off by rounding errors (~1e-12 of the terms), the running
//  sum passes the powers of two at distances of the size of the terms.  Take two
//  starts that differ by d, a multiple of 2^5 ulps of the start, and let no
//  result within the chunk lie above the start's binade by more than four.  Then d
//  is a multiple of twice every result's ulp, and if no result comes closer to a
//  power of two than |d|, every exact sum of the two runs is rounded to the same
//  grid, with the same parity: the results differ by exactly d.  So 32 runs of
//  plain FP64 adds, one for each value of the start's last five bits (a lane
//  each), are a table of the chunk for every start near the guess; the closest
//  approach to a power of two is kept beside it (k_ss_tables).
//
//  One warp then chains the chunks, checks each map's or table's validity against
//  the exact sum, and falls back to element scans with plain FP64 adds where
//  neither holds (the first chunk; sums passing zero).  The result equals the
//  sequential loop exactly.  A forest's systems are chained side by side.
//
//  Measured (one GB300): 2x10^6 centred positions (Plummer), whose sums leave
//  their binade in 1,740 of 7,813 chunks per axis: 19.1 -> 2.4 ms (those chunks took
//  26,000 clocks each as element scans); 10^6 positions in the unit cube: 0.31
//  -> 0.30 ms; 512 systems of 1,000 to 65,536: 7.1 -> 0.9 ms (a thread per sum).
#include "internal.h"

#define SS_C 256  // elements per chunk
#define SS_PER_LANE (SS_C / 32)

struct ChunkMap {
  long long A0, A1;      // total increment in ulps for start parity 0 / 1
  long long pmin, pmax;  // range of intermediate increments (with margin)
  int e;                 // binade the map is valid in
  int ok;                // 0: no map, run the chunk sequentially
};

// The systems' elements and chunks: system s holds elements [sys_off[s],
// sys_off[s + 1]) and chunks [chunk_off[s], chunk_off[s + 1]); one system has
// neither array.
struct SsArgs {
  const double *pos;
  long N, nchunks;
  int nsys;
  const long *sys_off;
  const int *chunk_off;
  __device__ __forceinline__ void chunks(int s, long &k0, long &k1) const {
    k0 = nsys > 1 ? chunk_off[s] : 0;
    k1 = nsys > 1 ? chunk_off[s + 1] : nchunks;
  }
  // elements [i0, i1) of chunk k
  __device__ __forceinline__ void range(long k, long &i0, long &i1) const {
    long end = N;
    i0 = k * SS_C;
    if (nsys > 1) {
      int lo = 0, hi = nsys - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunk_off[mid] <= k) lo = mid; else hi = mid - 1;
      }
      i0 = sys_off[lo] + (k - chunk_off[lo]) * SS_C;
      end = sys_off[lo + 1];
    }
    i1 = min(end, i0 + SS_C);
  }
};

// approximate chunk sums (FP64, any order)
__global__ void k_ss_chunksum(const SsArgs A, double *csum) {
  const long nchunks = A.nchunks;
  long k = blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  int a = blockIdx.y, lane = threadIdx.x & 31;
  if (k >= nchunks) return;
  long i0, i1;
  A.range(k, i0, i1);
  double s = 0;
  for (int j = 0; j < SS_PER_LANE; j++) {
    long i = i0 + lane * SS_PER_LANE + j;
    if (i < i1) s += A.pos[3 * i + a];
  }
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0) csum[a * nchunks + k] = s;
}

// exclusive prefix of a system's chunk sums (approximate start values), one block
// per axis and system
__global__ void k_ss_prefix(const SsArgs A, const double *csum, double *start) {
  __shared__ double wsum[32];
  const long nchunks = A.nchunks;
  long k0, k1;
  const int a = blockIdx.x % 3;
  A.chunks(blockIdx.x / 3, k0, k1);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, nt = blockDim.x;
  long per = (k1 - k0 + nt - 1) / nt;
  long b0 = min(k1, k0 + t * per), b1 = min(k1, b0 + per);
  double s = 0;
  for (long k = b0; k < b1; k++) s += csum[a * nchunks + k];
  double inc = s;
  for (int d = 1; d < 32; d <<= 1) {
    double o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (w == 0) {
    double x = lane < (nt >> 5) ? wsum[lane] : 0.0;
    for (int d = 1; d < 32; d <<= 1) {
      double o = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += o;
    }
    wsum[lane] = x;
  }
  __syncthreads();
  double run = (w > 0 ? wsum[w - 1] : 0.0) + inc - s;
  for (long k = b0; k < b1; k++) {
    start[a * nchunks + k] = run;
    run += csum[a * nchunks + k];
  }
}

// element effect in ulps of binade e: non-tie increment, or tie base
struct Elem {
  long long inc;  // rounded increment (non-tie) or the lower candidate (tie)
  int tie;        // 1: exactly half-way, increment is inc or inc+1 by parity
  int bad;        // 1: cannot be expressed (too large, NaN, Inf)
};

__device__ __forceinline__ Elem elem_in_ulps(double x, int e) {
  Elem r{0, 0, 0};
  unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  int ex = (int)((bits >> 52) & 0x7ff);
  unsigned long long m = bits & ((1ull << 52) - 1);
  bool neg = bits >> 63;
  if (ex == 0x7ff) { r.bad = 1; return r; }
  if (ex == 0) ex = 1;       // subnormal: no implicit bit
  else m |= 1ull << 52;
  // x = +-m * 2^(ex - 1075); x / u = +-m * 2^(ex - 1075 - (e - 52)) = +-m * 2^(ex - 1023 - e)
  int sh = ex - 1023 - e;
  long long a = 0;
  if (m == 0) return r;
  if (sh >= 0) {
    if (sh > 9) { r.bad = 1; return r; }  // |x| >= 2^(e+10): leaves the binade anyway
    a = (long long)(m << sh);
  } else {
    int s = -sh;
    if (s >= 64) {
      a = 0;  // |x/u| < 2^-11 < 1/2
    } else {
      unsigned long long q = m >> s;
      unsigned long long rem = m & ((1ull << s) - 1);
      unsigned long long half = 1ull << (s - 1);
      if (rem > half) q += 1;
      else if (rem == half) r.tie = 1;
      a = (long long)q;
    }
  }
  if (neg) {
    // -(q + t): for a tie the candidates are -q and -(q+1); keep the lower one as base
    a = -a;
    if (r.tie) a -= 1;
  }
  r.inc = a;
  return r;
}

// Map of one chunk for start parity p0/p1: (increment, end parity) composed
struct Map2 {
  long long i0, i1;
  int q0, q1;
};
__device__ __forceinline__ Map2 compose(Map2 g, Map2 f) {  // g first, then f
  Map2 r;
  r.i0 = g.i0 + (g.q0 ? f.i1 : f.i0);
  r.q0 = g.q0 ? f.q1 : f.q0;
  r.i1 = g.i1 + (g.q1 ? f.i1 : f.i0);
  r.q1 = g.q1 ? f.q1 : f.q0;
  return r;
}
__device__ __forceinline__ Map2 elem_map(const Elem &el) {
  Map2 m;
  if (!el.tie) {
    m.i0 = m.i1 = el.inc;
    int par = (int)(el.inc & 1);
    m.q0 = par;
    m.q1 = par ^ 1;
  } else {
    // S + inc even: parity p -> increment inc + ((p + inc) & 1), end parity 0
    int b = (int)(el.inc & 1);
    m.i0 = el.inc + (b ? 1 : 0);
    m.i1 = el.inc + (b ? 0 : 1);
    m.q0 = m.q1 = 0;
  }
  return m;
}

__global__ void k_ss_maps(const SsArgs A, const double *start, ChunkMap *maps) {
  const long nchunks = A.nchunks;
  long k = blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  int a = blockIdx.y, lane = threadIdx.x & 31;
  if (k >= nchunks) return;
  long i0, i1;
  A.range(k, i0, i1);
  double s0 = start[a * nchunks + k];
  ChunkMap cm{0, 0, 0, 0, 0, 0};
  if (s0 == 0.0 || !isfinite(s0)) {
    if (lane == 0) maps[a * nchunks + k] = cm;
    return;
  }
  int e = ilogb(fabs(s0));
  Map2 acc{0, 0, 0, 1};  // identity
  long long run = 0, lmin = 0, lmax = 0;
  int bad = 0;
  for (int j = 0; j < SS_PER_LANE; j++) {
    long i = i0 + lane * SS_PER_LANE + j;
    if (i >= i1) break;
    Elem el = elem_in_ulps(A.pos[3 * i + a], e);
    bad |= el.bad;
    acc = compose(acc, elem_map(el));
    run += el.inc;
    lmin = min(lmin, run);
    lmax = max(lmax, run);
  }
  // inclusive warp scan of the lane maps
  Map2 inc = acc;
  long long base = run;  // parity-0 path approximation for the range
  for (int d = 1; d < 32; d <<= 1) {
    Map2 o;
    o.i0 = __shfl_up_sync(0xffffffffu, inc.i0, d);
    o.i1 = __shfl_up_sync(0xffffffffu, inc.i1, d);
    o.q0 = __shfl_up_sync(0xffffffffu, inc.q0, d);
    o.q1 = __shfl_up_sync(0xffffffffu, inc.q1, d);
    long long ob = __shfl_up_sync(0xffffffffu, base, d);
    if (lane >= d) {
      inc = compose(o, inc);
      base += ob;
    }
  }
  long long excl = base - run;  // increments before this lane
  long long mn = excl + lmin, mx = excl + lmax;
  for (int d = 16; d; d >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, d));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    bad |= __shfl_xor_sync(0xffffffffu, bad, d);
  }
  if (lane == 31) {
    cm.A0 = inc.i0;
    cm.A1 = inc.i1;
    // ties can move the parity-1 path by at most one ulp per element
    cm.pmin = mn - SS_C - 1;
    cm.pmax = mx + SS_C + 1;
    cm.e = e;
    cm.ok = !bad;
    maps[a * nchunks + k] = cm;
  }
}

// S * 2^(e-52) for |S| in [2^52, 2^53), assembled from its bits (integer
// operations only: the chain runs on one warp per axis, where every FP64
// instruction costs the narrow FP64 pipe a full warp's worth of cycles)
__device__ __forceinline__ double ss_to_double(long long S, int e) {
  const unsigned long long m = (unsigned long long)(S < 0 ? -S : S);
  unsigned long long bits = ((unsigned long long)(e + 1023) << 52) | (m & ((1ull << 52) - 1));
  if (S < 0) bits |= 1ull << 63;
  return __longlong_as_double((long long)bits);
}
// binade e and S = s / 2^(e-52) of a normal double; false for zero,
// subnormals, infinities and NaN (which take plain FP64 adds)
__device__ __forceinline__ bool ss_from_double(double s, int &e, long long &S) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
  const int ex = (int)((bits >> 52) & 0x7ff);
  if (ex == 0 || ex == 0x7ff) return false;
  e = ex - 1023;
  const long long m = (long long)((bits & ((1ull << 52) - 1)) | (1ull << 52));
  S = (bits >> 63) ? -m : m;
  return true;
}

// Tables of the chunks whose map will not hold for the guessed start: for each
// value r of its last SS_TBITS bits the sum after the chunk, then the closest any
// of the runs' results came to a power of two, in ulps of the start (0: no table).
#define SS_TBITS 5
#define SS_TAB ((1 << SS_TBITS) + 1)
__global__ void k_ss_tables(const SsArgs A, const double *start, const ChunkMap *maps, double *tab) {
  constexpr unsigned FULL = 0xffffffffu;
  const long nchunks = A.nchunks;
  const long k = blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int a = blockIdx.y, lane = threadIdx.x & 31;
  if (k >= nchunks) return;
  const long at = a * nchunks + k;
  double *t = tab + at * SS_TAB;
  const double s0 = start[at];
  const ChunkMap m = maps[at];
  int e0 = 0;
  long long S0 = 0;
  bool want = ss_from_double(s0, e0, S0);
  if (want && m.ok) {  // the map holds with room to spare: no table
    const long long LO = 1ll << 52, HI = 1ll << 53, room = 1ll << 24;
    want = !(S0 > 0 ? (S0 + m.pmin >= LO + room && S0 + m.pmax < HI - room)
                    : (S0 + m.pmax <= -LO - room && S0 + m.pmin > -HI + room));
  }
  if (!want) {
    if (lane == 0) t[SS_TAB - 1] = 0.0;
    return;
  }
  long i0, i1;
  A.range(k, i0, i1);
  const int n = (int)(i1 - i0);
  double x[SS_PER_LANE];
#pragma unroll
  for (int j = 0; j < SS_PER_LANE; j++) x[j] = lane + 32 * j < n ? A.pos[3 * (i0 + lane + 32 * j) + a] : 0.0;
  const unsigned long long mask = (1ull << SS_TBITS) - 1, b0 = (unsigned long long)__double_as_longlong(s0);
  double s = __longlong_as_double((long long)((b0 & ~mask) | (unsigned)lane));
  const int ex0 = (int)((b0 >> 52) & 0x7ff);
  float room = 3e38f;
#pragma unroll
  for (int j = 0; j < SS_PER_LANE; j++) {
    const int cnt = min(32, n - 32 * j);
    for (int c = 0; c < cnt; c++) {
      s = __dadd_rn(s, __shfl_sync(FULL, x[j], c));
      const unsigned long long b = (unsigned long long)__double_as_longlong(s);
      const int ex = (int)((b >> 52) & 0x7ff), d = ex - ex0;
      const unsigned long long f = b & ((1ull << 52) - 1);
      // distance to the nearer power of two, four ulps short of it
      const float near = __ull2float_rd(min(f, (1ull << 52) - f)) - 4.f;
      const bool good = ex > 0 && ex < 0x7ff && d <= SS_TBITS - 1 && d > -64;
      room = fminf(room, good ? near * __int_as_float((d + 127) << 23) : 0.f);
    }
  }
  for (int d = 16; d; d >>= 1) room = fminf(room, __shfl_xor_sync(FULL, room, d));
  t[lane] = s;
  if (lane == 0) t[SS_TAB - 1] = (double)fmaxf(room, 0.f);
}

// Chunk maps compose: chunk a then chunk b (same binade) is again
//   S -> S + B[S mod 2],  B[p] = A_a[p] + A_b[(p + A_a[p]) mod 2]
// (the parity after a is that of p + A_a[p]), valid while every intermediate
// increment stays in [min(pmin_a, min A_a + pmin_b), max(pmax_a, max A_a + pmax_b)]
// -- a conservative range, so a composite that checks valid is valid.  e ==
// SS_ANY marks the identity.
#define SS_ANY (-100000)
__device__ __forceinline__ ChunkMap cm_identity() {
  ChunkMap m;
  m.A0 = m.A1 = m.pmin = m.pmax = 0;
  m.e = SS_ANY;
  m.ok = 1;
  return m;
}
__device__ __forceinline__ ChunkMap cm_compose(const ChunkMap &a, const ChunkMap &b) {
  if (a.e == SS_ANY) return b;
  if (b.e == SS_ANY) return a;
  ChunkMap c;
  c.ok = a.ok && b.ok && a.e == b.e;
  c.e = a.e;
  c.A0 = a.A0 + ((a.A0 & 1) ? b.A1 : b.A0);
  c.A1 = a.A1 + ((a.A1 & 1) ? b.A0 : b.A1);
  c.pmin = min(a.pmin, min(a.A0, a.A1) + b.pmin);
  c.pmax = max(a.pmax, max(a.A0, a.A1) + b.pmax);
  return c;
}
__device__ __forceinline__ ChunkMap cm_shfl_up(const ChunkMap &m, int d) {
  const unsigned FULL = 0xffffffffu;
  ChunkMap o;
  o.A0 = __shfl_up_sync(FULL, m.A0, d);
  o.A1 = __shfl_up_sync(FULL, m.A1, d);
  o.pmin = __shfl_up_sync(FULL, m.pmin, d);
  o.pmax = __shfl_up_sync(FULL, m.pmax, d);
  o.e = __shfl_up_sync(FULL, m.e, d);
  o.ok = __shfl_up_sync(FULL, m.ok, d);
  return o;
}

// Chains the chunk maps in order, exactly: one warp per axis and system, 32
// chunks at a time.  The state (s, or S in ulps of binade e) is kept identical in every
// lane.  From the current chunk j of a block, the lanes compose the maps of
// chunks j..lane (a warp scan); the longest run of composites that is valid
// for the exact S is applied in one step.  A chunk with a table takes that when
// the state is close enough to its guess.  A chunk that neither covers is run 32
// elements at a time: the lanes scan the element maps from the exact S, a ballot finds the
// first element whose result leaves the binade, and only that element takes a
// plain sequential FP64 add.
__global__ void k_ss_chain(const SsArgs A, const double *start, const ChunkMap *maps, const double *tab, double *out) {
  __shared__ double sx[1][SS_C];
  const unsigned FULL = 0xffffffffu;
  const int a = blockIdx.x % 3, sys = blockIdx.x / 3, lane = threadIdx.x & 31;  // one axis of one system per block
  const double *__restrict__ pos = A.pos;
  long kb, ke;
  A.chunks(sys, kb, ke);
  const long nchunks = ke - kb, all = A.nchunks;
  maps += a * all + kb;
  start += a * all + kb;
  if (tab) tab += (a * all + kb) * SS_TAB;
  const long e0 = A.nsys > 1 ? A.sys_off[sys] : 0, N = (A.nsys > 1 ? A.sys_off[sys + 1] : A.N) - e0;
  pos += 3 * e0;
  const long long LO = 1ll << 52, HI = 1ll << 53;
  double s = 0.0;
  bool imode = false;
  long long S = 0;
  int e = 0;
  // elements of the chunk after the last chunk that ran element by element
  // (such chunks come in runs: their loads overlap the previous one's work)
  long pref_k = -1;
  double pr[SS_PER_LANE];
  ChunkMap nxt = lane < nchunks ? maps[lane] : cm_identity();
  double nguess = lane < nchunks ? start[lane] : 0.0;
  double nroom = tab && lane < nchunks ? tab[lane * SS_TAB + SS_TAB - 1] : 0.0;
  for (long k0 = 0; k0 < nchunks; k0 += 32) {
    const ChunkMap mo = nxt;  // this lane's chunk k0 + lane
    const double guess = nguess, room = nroom;  // its guessed start; its table's room (0: none)
    const long kn = k0 + 32 + lane;
    if (kn < nchunks) {  // the next block's, ahead
      nxt = maps[kn];
      nguess = start[kn];
      nroom = tab ? tab[kn * SS_TAB + SS_TAB - 1] : 0.0;
    }
    const int nb = (int)min(32L, nchunks - k0);
    // the block's chunks with a table; the first one's rows are requested now, each next one's with its turn
    unsigned tabs = __ballot_sync(FULL, lane < nb && room > 0.0);
    double after = tabs ? tab[(k0 + __ffs(tabs) - 1) * SS_TAB + lane] : 0.0;
    int j = 0;
    while (j < nb) {
      const long k = k0 + j;
      while (tabs && __ffs(tabs) - 1 < j) {  // passed by
        tabs &= tabs - 1;
        after = tabs ? tab[(k0 + __ffs(tabs) - 1) * SS_TAB + lane] : 0.0;
      }
      if (tabs && __ffs(tabs) - 1 == j) {  // ---- chunk j's table ----
        const double row = after;
        tabs &= tabs - 1;
        after = tabs ? tab[(k0 + __ffs(tabs) - 1) * SS_TAB + lane] : 0.0;
        const unsigned long long cur =
            (unsigned long long)__double_as_longlong(imode ? ss_to_double(S, e) : s);
        const unsigned long long g = (unsigned long long)__double_as_longlong(__shfl_sync(FULL, guess, j));
        const unsigned long long mask = (1ull << SS_TBITS) - 1;
        // distance to the run with the same last bits, in ulps of the start (a multiple of 32)
        const long long d = (long long)(cur & ~mask) - (long long)(g & ~mask);
        // sign and binade of the guess, and near enough to it
        if ((cur >> 52) == (g >> 52) && (float)(d < 0 ? -d : d) < (float)__shfl_sync(FULL, room, j) * 0.999999f) {
          const unsigned long long r =
              (unsigned long long)__double_as_longlong(__shfl_sync(FULL, row, (int)(cur & mask)));
          // the same distance in ulps of the result, whose magnitude grows with it where the signs agree
          const int sh = (int)((g >> 52) & 0x7ff) - (int)((r >> 52) & 0x7ff);
          const long long dr = sh >= 0 ? d << sh : d >> -sh;  // exact
          s = __longlong_as_double((long long)(((g ^ r) >> 63) ? r - (unsigned long long)dr
                                                               : r + (unsigned long long)dr));
          imode = false;
          j++;
          continue;
        }
      }
      // the state in the binade of chunk j's map, when it has one
      const int ej = __shfl_sync(FULL, mo.e, j), okj = __shfl_sync(FULL, mo.ok, j);
      if (okj && (!imode || e != ej)) {
        double cur = imode ? ss_to_double(S, e) : s;
        int ce;
        long long cS;
        if (ss_from_double(cur, ce, cS) && ce == ej) {
          S = cS;  // exact: cur is a multiple of its ulp
          e = ej;
          imode = true;
        } else {
          s = cur;
          imode = false;
        }
      }
      if (okj && imode) {
        ChunkMap c = lane >= j && lane < nb ? mo : cm_identity();
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const ChunkMap o = cm_shfl_up(c, d);
          if (lane >= d) c = cm_compose(o, c);
        }
        const bool inr = S > 0 ? (S + c.pmin >= LO && S + c.pmax < HI) : (S + c.pmax <= -LO && S + c.pmin > -HI);
        const bool v = lane >= j && lane < nb && c.ok && c.e == e && inr;
        const unsigned inv = ~__ballot_sync(FULL, v) & (FULL << j);
        const int f = inv ? __ffs(inv) - 1 : 32;  // first chunk not covered
        if (f > j) {
          const long long B0 = __shfl_sync(FULL, c.A0, f - 1), B1 = __shfl_sync(FULL, c.A1, f - 1);
          S += (S & 1) ? B1 : B0;
          j = f;
          continue;
        }
      }
      // ---- warp-parallel exact fallback over chunk k ----
      long i0 = k * SS_C;
      int n = (int)(min(N, (k + 1) * SS_C) - i0);
      __syncwarp();
      if (pref_k == k) {
#pragma unroll
        for (int t = 0; t < SS_PER_LANE; t++) sx[0][lane + 32 * t] = pr[t];
      } else {
        for (int i = lane; i < n; i += 32) sx[0][i] = pos[3 * (i0 + i) + a];
      }
      pref_k = k + 1;
#pragma unroll
      for (int t = 0; t < SS_PER_LANE; t++) {
        const long i = pref_k * SS_C + lane + 32 * t;
        pr[t] = i < N ? pos[3 * i + a] : 0.0;
      }
      __syncwarp();
      for (int b = 0; b < n; b += 32) {
        int cnt = min(32, n - b);
        double xj = lane < cnt ? sx[0][b + lane] : 0.0;
        int c = 0;
        while (c < cnt) {
          if (!imode) {
            if (!ss_from_double(s, e, S)) {
              s = __dadd_rn(s, sx[0][b + c]);
              c++;
              continue;
            }
            imode = true;
          }
          bool act = lane >= c && lane < cnt;
          Elem el = act ? elem_in_ulps(xj, e) : Elem{0, 0, 0};
          Map2 mp = act ? elem_map(el) : Map2{0, 0, 0, 1};
          for (int d = 1; d < 32; d <<= 1) {
            Map2 o;
            o.i0 = __shfl_up_sync(FULL, mp.i0, d);
            o.i1 = __shfl_up_sync(FULL, mp.i1, d);
            o.q0 = __shfl_up_sync(FULL, mp.q0, d);
            o.q1 = __shfl_up_sync(FULL, mp.q1, d);
            if (lane >= d) mp = compose(o, mp);
          }
          long long Sj = S + ((S & 1) ? mp.i1 : mp.i0);
          // strictly inside the binade: a result of exactly 2^52 ulps may be the rounding of a sum
          // just below the power of two, whose true rounding is on the finer grid below it
          bool leaves = el.bad || !(S > 0 ? (Sj > LO && Sj < HI) : (Sj < -LO && Sj > -HI));
          unsigned bal = __ballot_sync(FULL, act && leaves);
          if (bal == 0) {
            S = __shfl_sync(FULL, Sj, cnt - 1);
            c = cnt;
          } else {
            int x = __ffs(bal) - 1;
            long long Sb = __shfl_sync(FULL, Sj, x > 0 ? x - 1 : 0);
            if (x == c) Sb = S;
            s = __dadd_rn(ss_to_double(Sb, e), sx[0][b + x]);
            imode = false;
            c = x + 1;
          }
        }
      }
      j++;
    }
  }
  if (lane == 0) {
    if (imode) s = ss_to_double(S, e);
    out[3 * (long)sys + a] = s;
  }
}

// Scratch of fmm_seqsum3, without and with the tables.
size_t fmm_seqsum_scratch(long N) {
  long nch = (N + SS_C - 1) / SS_C;
  return (size_t)nch * 3 * (2 * sizeof(double) + sizeof(ChunkMap)) + 256;
}
long fmm_seqsum_chunks(long n) { return (n + SS_C - 1) / SS_C; }
size_t fmm_seqsum_scratch_tables(long chunks) {
  return (size_t)chunks * 3 * (2 * sizeof(double) + sizeof(ChunkMap) + SS_TAB * sizeof(double)) + 256;
}

static int seqsum_run(const SsArgs &A, double *out, void *scratch, bool tables, cudaStream_t st) {
  const long nch = A.nchunks;
  double *csum = (double *)scratch;
  double *start = csum + 3 * nch;
  ChunkMap *maps = (ChunkMap *)(start + 3 * nch);
  double *tab = tables ? (double *)(maps + 3 * nch) : nullptr;
  const dim3 g((unsigned)((nch + 3) / 4), 3);
  const unsigned per = 3u * (unsigned)A.nsys;
  fmm_note_launch(), k_ss_chunksum<<<g, 128, 0, st>>>(A, csum);
  fmm_note_launch(), k_ss_prefix<<<per, A.nsys > 1 ? 128 : 1024, 0, st>>>(A, csum, start);
  fmm_note_launch(), k_ss_maps<<<g, 128, 0, st>>>(A, start, maps);
  if (tables) fmm_note_launch(), k_ss_tables<<<g, 128, 0, st>>>(A, start, maps, tab);
  fmm_note_launch(), k_ss_chain<<<per, 32, 0, st>>>(A, start, maps, tab, out);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

// out[0..2] = the three sequential sums; scratch must hold fmm_seqsum_scratch(N)
// bytes, or with `tables` fmm_seqsum_scratch_tables(fmm_seqsum_chunks(N))
int fmm_seqsum3(const double *pos, long N, double *out, void *scratch, bool tables, cudaStream_t st) {
  return seqsum_run({pos, N, fmm_seqsum_chunks(N), 1, nullptr, nullptr}, out, scratch, tables, st);
}

// out[3 s .. 3 s + 2] = the sums of system s, whose chunks are [chunk_off[s], chunk_off[s + 1]) (device arrays);
// scratch as with tables
int fmm_seqsum3_systems(const double *pos, const long *sys_off, const int *chunk_off, int nsys, long chunks,
                        double *out, void *scratch, cudaStream_t st) {
  return seqsum_run({pos, 0, chunks, nsys, sys_off, chunk_off}, out, scratch, true, st);
}
