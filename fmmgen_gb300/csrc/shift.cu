// shift.cu -- M2M and L2L of one level (example/calculate.cpp:163-187 and
// :219-234 with fmmgen's M2M_p / L2L_p, fmmgen/expansions.py:42-78 and :175-194),
// FP32 and FP64.
//
// In the scaled expansions (M~ = M / s^|m|, L^ = s^(|n|+1) L, s a cell's half-width)
//   M2M:  M~_parent[n] += sum_{k <= n} mono(k) 2^-|n-k| M~_child[n-k],  mono(k) = (d/s)^k / k!,
//         d = parent - child
//   L2L:  L^_child[n]  += 2^-(|n|+1) sum_{|n|+|k| <= p-so} mono(k) L^_parent[n+k],  d = child - parent
// and mono(k) is a product of the axes' powers, so a shift is one shift along
// each axis.  The eight children lie on a grid of two places per axis: children
// that differ in x only share their y and z shifts.  The M2M therefore shifts eight
// multipoles along x, adds them up in pairs, four along y and two along z; the L2L
// splits up in the same way, two, four and eight.  That is 14 shifts of C(p+4, 4)
// multiply-adds (p = 12: 1,820) for eight full ones of C(p+6, 6) (18,564).  A block of
// eight warps takes a parent, all stages in shared memory.
// Bound by the barriers between the stages and the index arithmetic (two warps a
// block for short rows measured the same).  Against a thread per output term with
// coefficient tables in FP32, and a warp per cell in the contraction engine in FP64,
// M2M and L2L: 2x10^6 clustered charges, p = 12, FP32: 4.1 and 1.45 ms, now 0.72 and
// 0.55; 10^6 uniform charges, p = 8, FP64: 2.20 and 1.34 ms, now 0.25 and 0.19.  Mean
// error of a mixed field against FP64, p = 8: 1.97e-7, now 1.85e-7 (uniform), 2.15e-7
// and 1.89e-7 (clustered).
// The axes' displacements are the cells' own (FP64 centres, each rounded when its
// cell was made), the same for all children on one side.
#include <algorithm>
#include "internal.h"
#include "mi_table.cuh"

namespace {

constexpr int SH_BS = 256;

static __constant__ double c_rfact[FMM_PMAX + 1] = {1.,       1.,        1. / 2,     1. / 6,      1. / 24,
                                                    1. / 120, 1. / 720,  1. / 5040,  1. / 40320,  1. / 362880,
                                                    1. / 3628800, 1. / 39916800, 1. / 479001600};

template <typename T> struct ShiftShared {
  T tab[3][2][FMM_PMAX + 1];  // v^k / k! per axis and side (0: the child at the smaller coordinate)
  T half[FMM_PMAX + 2];       // 2^-d
  uchar4 mi[FMM_NTMAX];       // the multi-indices (x, y, z, degree)
  int nt[FMM_PMAX + 2];       // nt[d + 1] = fmm_nterms(d)
};

template <typename T> __device__ __forceinline__ void shift_init(ShiftShared<T> &S, int p) {
  for (int e = threadIdx.x; e < fmm_nterms(p); e += SH_BS)
    S.mi[e] = make_uchar4(c_mi[e][0], c_mi[e][1], c_mi[e][2], c_mi[e][3]);
  if (threadIdx.x < FMM_PMAX + 2) {
    S.nt[threadIdx.x] = fmm_nterms((int)threadIdx.x - 1);
    S.half[threadIdx.x] = (T)ldexp(1.0, -(int)threadIdx.x);
  }
}
// The powers of parent c's displacements: sign * (child - parent) / s.
template <typename T>
__device__ __forceinline__ void shift_powers(ShiftShared<T> &S, int p, int c, const double *cx, const double *cy,
                                             const double *cz, const double *cr, double sign) {
  const int e = threadIdx.x;
  if (e >= 6 * (p + 1)) return;
  const int a = e / (2 * (p + 1)), r = e - a * 2 * (p + 1), side = r / (p + 1), k = r - side * (p + 1);
  const double s = cr[c], h = __ddiv_rn(s, 2.0), x = a == 0 ? cx[c] : a == 1 ? cy[c] : cz[c];
  const T v = (T)(sign * (__dadd_rn(x, side ? h : -h) - x) * (1.0 / s));
  T q = k > 0 ? v : T(1);
  for (int i = 2; i <= k; i++) q *= v;
  S.tab[a][side][k] = q * (T)c_rfact[k];
}

// Walks the terms of one output of a shift along axis a, (na, b, c) its component on
// the axis and the other two in their order: f(k, place of term k), k = 0 .. len.
template <bool L2L, typename F>
__device__ __forceinline__ void shift_terms(const int *nt, int a, int na, int b, int c, int len, F f) {
  const int deg = na + b + c;
  for (int k = 0; k <= len; k++) {
    const int q = L2L ? na + k : na - k, g = L2L ? deg + k : deg - k;
    // place of an index (x, y, z) of degree g: nt[g] + j (j + 1) / 2 + z, j = y + z
    const int j = a == 0 ? b + c : a == 1 ? q + c : c + q, z = a == 2 ? q : c;
    f(k, nt[g] + j * (j + 1) / 2 + z);
  }
}

template <typename T>
__global__ void __launch_bounds__(SH_BS) k_m2m(int lo, int hi, int p, int so, const unsigned char *child_mask,
                                               const int *child_first, const double *cx, const double *cy,
                                               const double *cz, const double *cr, T *M, int mstr) {
  extern __shared__ double shift_smem[];
  __shared__ ShiftShared<T> S;
  const int NT = fmm_nterms(p), off = fmm_nterms(so - 1);
  T *b0 = (T *)shift_smem, *b1 = b0 + 8 * NT;  // [8][NT] each
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  shift_init(S, p);
  // Outputs with equally long sums side by side: entry e of the multi-index table,
  // of degree d, stands for the component p - d on the axis and the others y and z.
  auto outputs = [&](int a, int e0, int step, auto body) {
    for (int e = e0; e < NT; e += step) {
      const uchar4 m = S.mi[e];
      const int na = p - m.w, deg = na + m.y + m.z;
      if (deg >= so) body(na, (int)m.y, (int)m.z, min(na, deg - so));
    }
  };
  for (int c = lo + (int)blockIdx.x; c < hi; c += gridDim.x) {
    const unsigned mask = child_mask[c];
    if (!mask) continue;
    __syncthreads();
    shift_powers(S, p, c, cx, cy, cz, cr, -1.0);
    const bool here = (mask >> w) & 1u;
    const T *child = M + (size_t)(child_first[c] + __popc(mask & ((1u << w) - 1u))) * mstr;
    for (int j = off + lane; j < NT; j += 32) {
      b0[w * NT + j] = here ? child[j - off] * S.half[S.mi[j].w] : T(0);
      if (!here) b1[w * NT + j] = T(0);
    }
    __syncthreads();
    if (here)
      outputs(0, lane, 32, [&](int na, int b, int cc, int len) {
        T s = T(0);
        int o = 0;
        shift_terms<false>(S.nt, 0, na, b, cc, len, [&](int k, int at) {
          if (k == 0) o = at;
          s += S.tab[0][w & 1][k] * b0[w * NT + at];
        });
        b1[w * NT + o] = s;
      });
    __syncthreads();
    {
      const int q = w >> 1;
      const T *u = b1 + 2 * q * NT;
      outputs(1, 32 * (w & 1) + lane, 64, [&](int na, int b, int cc, int len) {
        T s = T(0);
        int o = 0;
        shift_terms<false>(S.nt, 1, na, b, cc, len, [&](int k, int at) {
          if (k == 0) o = at;
          s += S.tab[1][q & 1][k] * (u[at] + u[NT + at]);
        });
        b0[q * NT + o] = s;
      });
    }
    __syncthreads();
    outputs(2, threadIdx.x, SH_BS, [&](int na, int b, int cc, int len) {
      T s = T(0);
      int o = 0;
      shift_terms<false>(S.nt, 2, na, b, cc, len, [&](int k, int at) {
        if (k == 0) o = at;
        s += S.tab[2][0][k] * (b0[at] + b0[NT + at]) + S.tab[2][1][k] * (b0[2 * NT + at] + b0[3 * NT + at]);
      });
      M[(size_t)c * mstr + o - off] = s;
    });
  }
}

template <typename T>
__global__ void __launch_bounds__(SH_BS) k_l2l(int lo, int hi, int p, const unsigned char *child_mask,
                                               const int *child_first, const double *cx, const double *cy,
                                               const double *cz, const double *cr, T *L, int lstr) {
  extern __shared__ double shift_smem[];
  __shared__ ShiftShared<T> S;
  const int NT = fmm_nterms(p);
  T *b0 = (T *)shift_smem, *bx = b0 + NT, *by = bx + 2 * NT;  // the parent; by side in x; by sides in x and y
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  shift_init(S, p);
  // one output (the lanes of a warp: mostly of one degree, sums of one length)
  auto sum = [&](int a, const uchar4 m, const T *t, const T *u) {
    const int na = a == 0 ? m.x : a == 1 ? m.y : m.z, b = a == 0 ? m.y : m.x, c = a == 2 ? m.y : m.z;
    T s = T(0);
    shift_terms<true>(S.nt, a, na, b, c, p - m.w, [&](int k, int at) { s += t[k] * u[at]; });
    return s;
  };
  for (int c = lo + (int)blockIdx.x; c < hi; c += gridDim.x) {
    const unsigned mask = child_mask[c];
    if (!mask) continue;
    __syncthreads();
    shift_powers(S, p, c, cx, cy, cz, cr, 1.0);
    for (int j = threadIdx.x; j < NT; j += SH_BS) b0[j] = L[(size_t)c * lstr + j];
    __syncthreads();
    for (int e = threadIdx.x & 127; e < NT; e += 128) bx[(w >> 2) * NT + e] = sum(0, S.mi[e], S.tab[0][w >> 2], b0);
    __syncthreads();
    for (int e = threadIdx.x & 63; e < NT; e += 64)
      by[(w >> 1) * NT + e] = sum(1, S.mi[e], S.tab[1][w >> 2], bx + ((w >> 1) & 1) * NT);
    __syncthreads();
    if ((mask >> w) & 1u) {
      T *child = L + (size_t)(child_first[c] + __popc(mask & ((1u << w) - 1u))) * lstr;
      for (int e = lane; e < NT; e += 32) {
        const uchar4 m = S.mi[e];
        child[e] += sum(2, m, S.tab[2][w >> 2], by + (w & 3) * NT) * S.half[m.w + 1];
      }
    }
  }
}

constexpr long SH_GRID = 152 * 8;

// The M2M's rows.  Its limit is that of the longest ones: it holds for the process, and another thread may be about to
// launch them.
template <typename T> constexpr size_t m2m_bytes(int nterms) { return 16 * sizeof(T) * (size_t)nterms; }

}  // namespace

// the multipoles of the parents in [lo, hi), the cells of one level, from their children's
template <typename T> int fmm_m2m(DevTree *t, int lo, int hi, T *M, int mstr, cudaStream_t st) {
  if (hi <= lo) return FMM_OK;
  const size_t bytes = m2m_bytes<T>(fmm_nterms(t->order));
  if (bytes > 32 * 1024)
    FMM_CUDA_TRY(cudaFuncSetAttribute(k_m2m<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)m2m_bytes<T>(FMM_NTMAX)));
  fmm_note_launch(), k_m2m<T><<<(unsigned)std::min<long>(hi - lo, SH_GRID), SH_BS, bytes, st>>>(
      lo, hi, t->order, t->so, t->child_mask.p, t->child_first.p, t->cx.p, t->cy.p, t->cz.p, t->cr.p, M, mstr);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

// L2L into the children [lo, hi) of one level, from their parents (the level above)
template <typename T> int fmm_l2l(DevTree *t, int lo, int hi, T *L, int lstr, cudaStream_t st) {
  if (hi <= lo) return FMM_OK;
  int l = 1;
  while (l < t->nlevels && t->level_off[l] != lo) l++;
  if (l >= t->nlevels) return FMM_ERR_STATE;
  const int plo = t->level_off[l - 1], phi = t->level_off[l], p = t->order - t->so;
  const size_t bytes = 7 * sizeof(T) * (size_t)fmm_nterms(p);
  static_assert(7 * sizeof(T) * FMM_NTMAX <= 32 * 1024, "within every kernel's limit");
  fmm_note_launch(), k_l2l<T><<<(unsigned)std::min<long>(phi - plo, SH_GRID), SH_BS, bytes, st>>>(
      plo, phi, p, t->child_mask.p, t->child_first.p, t->cx.p, t->cy.p, t->cz.p, t->cr.p, L, lstr);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

template int fmm_m2m<float>(DevTree *, int, int, float *, int, cudaStream_t);
template int fmm_m2m<double>(DevTree *, int, int, double *, int, cudaStream_t);
template int fmm_l2l<float>(DevTree *, int, int, float *, int, cudaStream_t);
template int fmm_l2l<double>(DevTree *, int, int, double *, int, cudaStream_t);
