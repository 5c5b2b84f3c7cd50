// bh.cu -- Barnes-Hut (Tree::compute_field_bh, example/tree.cpp:273-293) in FP64.
#include "internal.h"
#include "m2l_h.cuh"

#define TRY(x) do { int _rc = (x); if (_rc) return _rc; } while (0)

namespace {

// Per cell, degree n = 0 .. p + 1 and harmonic coefficient k of it (layout of
// gen_m2l_h.py: k_z = 0, 1), four weights (V, X, Y, Z) of tau_k(y), y = (x_i - c) / s:
//   phi = (1/s) sum V_k tau_k,   E = -(1/s^2) sum (X, Y, Z)_k tau_k
// is fmmgen's M2P (fmmgen/generator.py:174-206), the potential sum_m D_m M~_m
// with its exact gradient sum_m D_(m+e) M~_m.  tau_k = D_k / (k! gamma_n) with
// gamma_n = (-1)^n (2n-1)!! / n! takes the constants out of the recurrence
//   n r^2 D_k/k! = -(2n-1) sum_a y_a D_(k-e_a)/(k-e_a)! - (n-1) sum_a D_(k-2e_a)/(k-2e_a)!
// which becomes
//   tau_k = sum_a (y_a / r^2) tau_(k-e_a) + c_n / r^2 sum_a tau_(k-2e_a),  c_n = -(n-1)^2 / ((2n-1)(2n-3)),
// at most five operations an entry, and only the (p+2)^2 entries with k_z <= 1
// are needed: D is harmonic, so M~ is folded as for the M2L (m2l_h.cu) and a
// z-derivative that reaches k_z = 2 is folded again.
__global__ void k_bh_weights(int ncells, int p, const double *Mh, int hstr, BhWeight *W) {
  const int nw = h_terms(p + 1);
  const long g = blockIdx.x * 256l + threadIdx.x;
  const long c = g / nw;
  const int i = (int)(g - c * nw);
  if (c >= ncells) return;
  int n = 0;
  while (h_terms(n) <= i) n++;
  int r = i - h_terms(n - 1);
  const int z = r > n ? 1 : 0;
  r -= z ? n + 1 : 0;
  const int x = n - z - r, y = n - z - x;
  const double *M = Mh + (size_t)c * hstr;
  double f = 1.0;  // k! gamma_n
  for (int q = 2; q <= x; q++) f *= q;
  for (int q = 2; q <= y; q++) f *= q;
  for (int q = 1; q <= n; q++) f *= -(double)(2 * q - 1) / q;
  BhWeight w = {0, 0, 0, 0};
  if (n <= p) w.v = f * M[i];
  if (x > 0) w.x = f * M[h_index(x - 1, y, z)];
  if (y > 0) w.y = f * M[h_index(x, y - 1, z)];
  if (z) w.z = f * M[h_index(x, y, 0)];
  else w.z = -f * ((x > 1 ? M[h_index(x - 2, y, 1)] : 0.0) + (y > 1 ? M[h_index(x, y - 2, 1)] : 0.0));
  W[(size_t)c * nw + i] = w;
}

// v += W (V, X, Y, Z) . tau(y) for a cell's weights; y' = y / r^2, ir2 = 1 / r^2.
template <int P>
__device__ __forceinline__ void m2p(const BhWeight *__restrict__ W, double yx, double yy, double yz, double rinv,
                                    double ir2, double &v, double &gx, double &gy, double &gz) {
  constexpr int MAXN = 2 * (P + 1) + 1;
  double t0[MAXN], t1[MAXN], t2[MAXN];  // degrees n, n - 1, n - 2
#pragma unroll
  for (int n = 0; n <= P + 1; n++) {
    const double cn = n > 1 ? -(double)((n - 1) * (n - 1)) / (double)((2 * n - 1) * (2 * n - 3)) : 0.0;
    const double b = cn * ir2;
#pragma unroll
    for (int j = 0; j < 2 * n + 1; j++) {
      const int z = j > n ? 1 : 0, i = j - z * (n + 1);  // i: place among the entries of this z
      const int x = n - z - i, y = i;
      // places in degree n - 1: z = 0 entries have length n, z = 1 entries follow;
      // k - e_x keeps the place (y), k - e_y moves it down by one
      double s = 0;
      if (n == 0) {
        s = rinv;
      } else {
        const int o1 = z * n, o2 = z * (n - 1);
        if (x >= 1) s += yx * t1[o1 + y];
        if (y >= 1) s += yy * t1[o1 + y - 1];
        if (z) s += yz * t1[i];
        if (x >= 2) s += b * t2[o2 + y];
        if (y >= 2) s += b * t2[o2 + y - 2];
      }
      t0[j] = s;
      const BhWeight w = W[n * n + j];
      if (n <= P) v += w.v * s;
      if (x >= 1) gx += w.x * s;
      if (y >= 1) gy += w.y * s;
      if (z || x >= 2 || y >= 2) gz += w.z * s;
    }
#pragma unroll
    for (int j = 0; j < MAXN; j++) {
      t2[j] = t1[j];
      t1[j] = t0[j];
    }
  }
}

// One warp walks for 32 consecutive sorted particles: the stack holds (cell,
// lanes that opened it), and a child is tested by those lanes -- for every
// particle exactly the cells of evaluate_M2P_and_P2P
// (example/calculate.cpp:266-314).  The cells that a lane's particle accepts and
// the leaves it opens go into queues of its own, which the warp works off
// together, each lane on its own next cell or source: neighbours accept much
// the same number of cells, but half of them not the same ones.
// Bound by the FP64 pipe (16 clocks of an SM per instruction, whatever its
// active lanes): hence the queues (a thread per particle with its own stack ran
// with 15 of 32 lanes active, the common walk without them with 17), ~260
// operations per M2P at p = 4 (all derivatives in local memory took ~1,200), tests
// without a square root unless they are close, and one reciprocal square root
// per pair.  10^5 clustered charges, p = 4: 37.5 -> 7.1 ms (common walk without
// the queues 10.1).
constexpr int BH_STACK = 8 * 22;  // a depth-first walk of 21 levels holds at most 7 * 21 + 8 cells
constexpr int BH_QM = 64, BH_QL = 32;

struct BhCells {
  const double *cx, *cy, *cz, *cr;
  const unsigned char *clevel;
  const int *child_first;
  const unsigned char *child_mask;
  const int *pstart, *pcount;
};
struct BhBodies {
  long N;
  const double *px, *py, *pz;
  const uint32_t *perm;
  const double *S;
};

template <int P, int SO>
__global__ void __launch_bounds__(32) k_bh64(int nsys, const long *sys_off, const BhBodies B, const BhCells C,
                                             double theta, const BhWeight *W, int potential, int field, double *F,
                                             uint32_t *eflag) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int2 stack[BH_STACK];
  __shared__ int qm[BH_QM][32], ql[BH_QL][32];  // lane's accepted cells; opened leaves
  const int lane = threadIdx.x;
  const long i = blockIdx.x * 32l + lane;
  const bool in = i < B.N;
  int root = 0;
  if (in && nsys > 1) {  // the system holding sorted particle i: sys_off[s] <= i < sys_off[s + 1]
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sys_off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    root = lo;
  }
  const double xi = in ? B.px[i] : 0, yi = in ? B.py[i] : 0, zi = in ? B.pz[i] : 0;
  double phi = 0, ex = 0, ey = 0, ez = 0;
  double iroot = 0;
  int nm = 0, nl = 0;  // queue lengths
  const float th2 = (float)(theta * theta);

  // the multipoles queued by every lane, as long as `most` lanes have one
  auto multipoles = [&](int most) {
    while (__popc(__ballot_sync(FULL, nm > 0)) >= most) {
      if (nm > 0) {
        const int c = qm[--nm][lane];
        const double s = C.cr[c], is = iroot * h_exp2<double>((int)C.clevel[c]);  // half-widths halve exactly: 1 / s
        const double dx = xi - C.cx[c], dy = yi - C.cy[c], dz = zi - C.cz[c];
        const double rinv = rsqrt(dx * dx + dy * dy + dz * dz) * s, ir2 = rinv * rinv, f = is * ir2;
        double v = 0, gx = 0, gy = 0, gz = 0;
        m2p<P>(W + (size_t)c * ((P + 2) * (P + 2)), dx * f, dy * f, dz * f, rinv, ir2, v, gx, gy, gz);
        const double is2 = is * is;
        phi += v * is;
        ex -= gx * is2;
        ey -= gy * is2;
        ez -= gz * is2;
      }
    }
  };
  // the sources of the queued leaves, one per lane and round
  auto leaves = [&]() {
    int j = 0, j1 = 0;
    for (;;) {
      while (j == j1 && nl > 0) {
        const int c = ql[--nl][lane];
        j = C.pstart[c];
        j1 = j + C.pcount[c];
      }
      if (!__any_sync(FULL, j < j1)) break;
      if (j < j1 && j != i) {
        const double dx = xi - B.px[j], dy = yi - B.py[j], dz = zi - B.pz[j];
        const size_t oj = B.perm[j];
        if (SO == 2) {
          quadrupole_p2p<double>(dx, dy, dz, B.S + 6 * oj, phi, ex, ey, ez);
        } else {
          const double r2 = dx * dx + dy * dy + dz * dz;
          const double rinv = rsqrt(r2), rr = rinv * rinv;
          if (SO == 0) {
            const double qr = B.S[oj] * rinv, q3 = qr * rr;
            phi += qr;
            ex += q3 * dx;
            ey += q3 * dy;
            ez += q3 * dz;
          } else {
            const double sx = B.S[3 * oj], sy = B.S[3 * oj + 1], sz = B.S[3 * oj + 2];
            const double r3 = rr * rinv, u = (sx * dx + sy * dy + sz * dz) * r3, r5 = (3.0 * rr) * u;
            phi -= u;
            ex += sx * r3 - r5 * dx;
            ey += sy * r3 - r5 * dy;
            ez += sz * r3 - r5 * dz;
          }
        }
      }
      j += j < j1;
    }
  };

  unsigned todo = __ballot_sync(FULL, in);
  while (todo) {  // the particles of one system after the other
    const int r0 = __shfl_sync(FULL, root, __ffs(todo) - 1);
    const bool here = in && root == r0;
    const unsigned mine = __ballot_sync(FULL, here);
    todo &= ~mine;
    if (here) iroot = 1.0 / C.cr[r0];
    int sp = 1;
    if (lane == 0) stack[0] = make_int2(r0, (int)mine);
    while (sp > 0) {
      __syncwarp();
      const int2 top = stack[--sp];
      const int c0 = top.x;
      const bool on = ((unsigned)top.y >> lane) & 1u;
      const unsigned mask = C.child_mask[c0];
      if (!mask) {
        if (on) ql[nl++][lane] = c0;
        if (__any_sync(FULL, nl == BH_QL)) leaves();
        continue;
      }
      const int first = C.child_first[c0], nch = __popc(mask);
      for (int q = 0; q < nch; q++) {
        const int c = first + q;
        const double dx = xi - C.cx[c], dy = yi - C.cy[c], dz = zi - C.cz[c];
        const double s = C.cr[c];
        const double r2 = dx * dx + dy * dy + dz * dz;
        // s > theta r: in FP32 where more than 1e-5 decides, else as written
        const float a = __double2float_rn(s), d = __double2float_rn(r2), l = a * a, rr = th2 * d;
        bool open = l > rr;
        if (!(fabsf(l - rr) > 1e-5f * rr) || !(l > 1e-30f && l < 1e30f && rr > 1e-30f && rr < 1e30f))
          open = s > theta * sqrt(r2);
        const unsigned mo = __ballot_sync(FULL, open && on);
        if (on && !open) qm[nm++][lane] = c;
        if (mo) {
          if (sp < BH_STACK) {
            if (lane == 0) stack[sp] = make_int2(c, (int)mo);
            sp++;
          } else if (lane == 0) {
            atomicOr(eflag, 1u);  // deeper than the stack: reported, not walked
          }
        }
        // a full queue: work off what most lanes have, then what it takes
        if (__any_sync(FULL, nm == BH_QM)) {
          multipoles(24);
          if (__any_sync(FULL, nm >= BH_QM - 8)) multipoles(1);
        }
        __syncwarp();
      }
    }
  }
  multipoles(1);
  leaves();
  if (!in) return;
  double *f = F + (size_t)B.perm[i] * ((potential ? 1 : 0) + (field ? 3 : 0));
  if (potential) *f++ = phi;
  if (field) {
    f[0] = ex;
    f[1] = ey;
    f[2] = ez;
  }
}

template <int P> int walk(DevTree *t, const double *S, const BhWeight *W, double *F, int potential, int field,
                          cudaStream_t st) {
  if (t->order != P) {
    if constexpr (P < FMM_PMAX) return walk<P + 1>(t, S, W, F, potential, field, st);
    return FMM_ERR_ARG;
  } else {
    decltype(&k_bh64<P, 0>) k = t->so == 0 ? k_bh64<P, 0> : t->so == 1 ? k_bh64<P, 1> : k_bh64<P, 2>;
    const BhBodies B = {t->N, t->px.p, t->py.p, t->pz.p, t->perm.p, S};
    const BhCells C = {t->cx.p, t->cy.p, t->cz.p, t->cr.p, t->clevel.p, t->child_first.p, t->child_mask.p,
                       t->pstart.p, t->pcount.p};
    fmm_note_launch(), k<<<(unsigned)((t->N + 31) / 32), 32, 0, st>>>(t->nsys, t->nsys > 1 ? t->sys_off.p : nullptr, B,
                                                                      C, t->theta, W, potential, field, F,
                                                                      t->d_eflags.p);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
  }
}

}  // namespace

// The walk on the FP64 multipoles M (row length msize) of the cells; d_eflags is
// set when a walk was deeper than its stack.
int fmm_bh_walk(DevTree *t, const double *S, double *F, int potential, int field, cudaStream_t st) {
  const int p = t->order, hstr = h_terms(p), nw = h_terms(p + 1);
  TRY(fmm_reserve(t->bhM, (size_t)t->ncells * hstr));
  TRY(fmm_reserve(t->bhW, (size_t)t->ncells * nw));
  TRY(fmm_h_fold(t, t->M.p, fmm_nterms(p) - fmm_nterms(t->so - 1), t->bhM.p, hstr, st));
  const long n = (long)t->ncells * nw;
  fmm_note_launch(), k_bh_weights<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(t->ncells, p, t->bhM.p, hstr, t->bhW.p);
  FMM_CUDA_TRY(cudaGetLastError());
  return walk<1>(t, S, t->bhW.p, F, potential, field, st);
}
