// m2l_h.cu -- M2L over harmonic coefficients: the foldings around the
// generated kernels (m2l_h_*.cu) and the pass that runs them.
#include "m2l_h.cuh"

namespace {

constexpr int H_BLOCK = 256;

// binomial coefficients up to j = 6 (degree 12 folds six times)
__constant__ float c_binom[7][7] = {{1}, {1, 1}, {1, 2, 1}, {1, 3, 3, 1}, {1, 4, 6, 4, 1}, {1, 5, 10, 10, 5, 1},
                                    {1, 6, 15, 20, 15, 6, 1}};

// the coefficient at place i of the harmonic layout
__device__ __forceinline__ void h_decode(int i, int &x, int &y, int &z) {
  int d = 0;
  while (h_terms(d) <= i) d++;
  int r = i - h_terms(d - 1);
  z = r > d ? 1 : 0;
  r -= z ? d + 1 : 0;
  x = d - z - r;
  y = d - z - x;
}

// M'_(x,y,e) = sum_j (-1)^j sum_i C(j,i) M~_(x-2i, y-2(j-i), e+2j); zeros below
// the source order.  One thread per (cell, coefficient): a few reads of one row
// of the cell, which the row's other threads share in L1; bound by HBM.
template <typename T>
__global__ void k_h_fold(int ncells, int p, int so, const T *M, int mstr, T *Mh, int hstr) {
  const int nh = h_terms(p);
  const long g = blockIdx.x * (long)H_BLOCK + threadIdx.x;
  const long c = g / nh;
  const int i = (int)(g - c * nh);
  if (c >= ncells) return;
  int x, y, e;
  h_decode(i, x, y, e);
  T v = T(0);
  if (x + y + e >= so) {
    const T *row = M + (size_t)c * mstr - fmm_nterms(so - 1);
    for (int j = 0; 2 * j <= x + y; j++) {
      T s = T(0);
      for (int k = 0; k <= j; k++)
        if (2 * k <= x && 2 * (j - k) <= y)
          s += T(c_binom[j][k]) * row[fmm_idx3(x - 2 * k, y - 2 * (j - k), e + 2 * j)];
      v += (j & 1) ? -s : s;
    }
  }
  Mh[(size_t)c * hstr + i] = v;
}

// L_(x,y,e+2j) = (-1)^j sum_i C(j,i) L'_(x+2i, y+2(j-i), e)
template <typename T>
__global__ void k_h_unfold(int ncells, int pl, const T *Lh, int hstr, T *L, int lstr) {
  const int nl = fmm_nterms(pl);
  const long g = blockIdx.x * (long)H_BLOCK + threadIdx.x;
  const long c = g / nl;
  const int i = (int)(g - c * nl);
  if (c >= ncells) return;
  const MI n = fmm_decode(i);
  const int e = n.z & 1, j = n.z >> 1;
  const T *row = Lh + (size_t)c * hstr;
  T v = T(0);
  for (int k = 0; k <= j; k++) v += T(c_binom[j][k]) * row[h_index(n.x + 2 * k, n.y + 2 * (j - k), e)];
  L[(size_t)c * lstr + i] = (j & 1) ? -v : v;
}

// the operator entries with k_z <= 2 of every class; FP32: zeros for the classes that k_h_wide takes
template <typename T>
__global__ void k_h_operators(int ncls, int p, const int *key4, const double *D, T *Dh, int hstr) {
  const int nt = fmm_nterms(p);
  const long g = blockIdx.x * (long)H_BLOCK + threadIdx.x;
  const long c = g / nt;
  const int i = (int)(g - c * nt);
  if (c >= ncls) return;
  const MI k = fmm_decode(i);
  const bool none = sizeof(T) == 4 && -key4[4 * c] > fmm_wide_levels(p);
  if (k.z <= 2) Dh[(size_t)c * hstr + h_dindex(k.x, k.y, k.z)] = none ? T(0) : (T)D[(size_t)c * nt + i];
}

// The pairs of a mixed pass whose source is a cell so much larger than the target
// that FP32 holds neither 2^(degree x levels) nor the operator of high degree
// (fmm_wide_levels), in FP64 and added to L: few in any tree (coarse leaves that a
// deep cluster just accepts), so the plain contraction, a warp per target cell.  The
// other direction needs nothing: a much smaller source's higher degrees vanish.
constexpr int WIDE_WARPS = 4;
__global__ void __launch_bounds__(32 * WIDE_WARPS) k_h_wide(int ncells, int p, int so, const unsigned char *clevel,
                                                            const int *off, const int *src, const int *cls,
                                                            const unsigned char *ord, const double *D, const float *M,
                                                            int mstr, float *L, int lstr) {
  __shared__ double sM[WIDE_WARPS][FMM_NTMAX], sL[WIDE_WARPS][FMM_NTMAX];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int A = blockIdx.x * WIDE_WARPS + w;
  if (A >= ncells) return;
  const int la = clevel[A], wide = fmm_wide_levels(p);
  if (la <= wide) return;
  const int moff = fmm_nterms(so - 1), nl = fmm_nterms(p - so), nt = fmm_nterms(p);
  const int k0 = off[A], k1 = off[A + 1];
  bool some = false;
  for (int kb = k0; kb < k1; kb += 32) {
    const int k = kb + lane;
    unsigned todo = __ballot_sync(0xffffffffu, k < k1 && la - (int)clevel[src[min(k, k1 - 1)]] > wide);
    while (todo) {
      const int j = kb + __ffs(todo) - 1;
      todo &= todo - 1;
      const int B = src[j], dl = la - (int)clevel[B], q = ord ? min(max((int)ord[j], so + 1), p) : p;
      const double *Dc = D + (size_t)cls[j] * nt;
      if (!some)
        for (int i = lane; i < nl; i += 32) sL[w][i] = 0.0;
      some = true;
      __syncwarp();
      for (int i = moff + lane; i < fmm_nterms(q); i += 32)
        sM[w][i] = (double)M[(size_t)B * mstr + i - moff] * h_exp2<double>(dl * (int)fmm_decode(i).d);
      __syncwarp();
      for (int i = lane; i < nl; i += 32) {
        const MI n = fmm_decode(i);
        double v = 0;
        int m = moff;
        for (int d = so; d <= q - n.d; d++)
          for (int x = d; x >= 0; x--)
            for (int y = d - x; y >= 0; y--, m++) v += Dc[fmm_idx3(n.x + x, n.y + y, n.z + d - x - y)] * sM[w][m];
        sL[w][i] += v;
      }
    }
  }
  if (some)
    for (int i = lane; i < nl; i += 32) {
      float *o = L + (size_t)A * lstr + i;
      *o = (float)((double)*o + sL[w][i]);
    }
}

unsigned grid_of(long n) { return (unsigned)((n + H_BLOCK - 1) / H_BLOCK); }

// row length in elements, padded to a 128-byte line
template <typename T> int line_stride(int n) {
  constexpr int per = 128 / sizeof(T);
  return (n + per - 1) / per * per;
}

}  // namespace

bool fmm_m2l_h_supported(int p, int so) { return so >= 0 && so <= 2 && p >= so + 1 && p <= FMM_PMAX; }

template <typename T>
static int run(DevTree *t, const T *M, int mstr, T *L, int lstr, const unsigned char *ord, cudaStream_t st) {
  const int p = t->order, so = t->so, nc = t->ncells, pl = p - so;
  if (!fmm_m2l_h_supported(p, so)) return FMM_ERR_STATE;
  if (t->nm2l == 0) {
    int rc = fmm_mark_kernel(t, 0, st);  // no kernel, and not the time of an earlier pass
    FMM_CUDA_TRY(cudaMemset2DAsync(L, sizeof(T) * lstr, 0, sizeof(T) * fmm_nterms(pl), nc, st));
    return rc ? rc : fmm_mark_kernel(t, 1, st);
  }
  if (int rc = fmm_m2l_csr(t, st)) return rc;
  const int mh = line_stride<T>(h_terms(p)), lh = line_stride<T>(h_terms(pl)), dh = line_stride<T>(h_dterms(p));
  DevBuf<char> &hM = t->hM[sizeof(T) == 8], &hL = t->hL[sizeof(T) == 8], &hD = t->hD[sizeof(T) == 8];
  if (fmm_reserve(hM, sizeof(T) * (size_t)nc * mh) || fmm_reserve(hL, sizeof(T) * (size_t)nc * lh) ||
      fmm_reserve(hD, sizeof(T) * (size_t)t->nclasses * dh))
    return FMM_ERR_CUDA;
  if (int rc = fmm_m2l_targets(t, ord, st)) return rc;
  T *Mh = (T *)hM.p, *Lh = (T *)hL.p, *Dh = (T *)hD.p;
  fmm_note_launch(), k_h_operators<T><<<grid_of((long)t->nclasses * fmm_nterms(p)), H_BLOCK, 0, st>>>(
      t->nclasses, p, t->cls_key4.p, t->cls_D.p, Dh, dh);
  fmm_note_launch(), k_h_fold<T><<<grid_of((long)nc * h_terms(p)), H_BLOCK, 0, st>>>(nc, p, so, M, mstr, Mh, mh);
  HParams<T> P;
  P.tgt = t->tp_tgt.p;
  P.ntgt = nc;
  P.off = t->m2l_off.p;
  P.src = t->m2l_src.p;
  P.cls = t->m2l_cls.p;
  P.perm = ord ? t->tp_perm.p : nullptr;
  P.ord = ord;
  P.p = p;
  P.qlo = so + 1;
  P.D = Dh;
  P.dstr = (int)sizeof(T) * dh;
  P.clevel = t->clevel.p;
  P.M = Mh;
  P.mstr = (int)sizeof(T) * mh;
  P.L = Lh;
  P.lstr = lh;
  P.lsize = h_terms(pl);
  int rc = fmm_mark_kernel(t, 0, st);
  if (!rc) rc = h_run(P, st);
  if (!rc) rc = fmm_mark_kernel(t, 1, st);
  if (rc) return rc;
  fmm_note_launch(), k_h_unfold<T><<<grid_of((long)nc * fmm_nterms(pl)), H_BLOCK, 0, st>>>(nc, pl, Lh, lh, L, lstr);
  if constexpr (sizeof(T) == 4)
    if (t->eflags & FMM_EFLAG_WIDE)
      fmm_note_launch(), k_h_wide<<<fmm_blocks(nc, WIDE_WARPS), 32 * WIDE_WARPS, 0, st>>>(
          nc, p, so, t->clevel.p, t->m2l_off.p, t->m2l_src.p, t->m2l_cls.p, ord, t->cls_D.p, M, mstr, L, lstr);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

int fmm_m2l_h(DevTree *t, const float *M, int mstr, float *L, int lstr, const unsigned char *ord, cudaStream_t st) {
  return run<float>(t, M, mstr, L, lstr, ord, st);
}
int fmm_m2l_h(DevTree *t, const double *M, int mstr, double *L, int lstr, const unsigned char *ord, cudaStream_t st) {
  return run<double>(t, M, mstr, L, lstr, ord, st);
}
int fmm_h_fold(DevTree *t, const double *M, int mstr, double *Mh, int hstr, cudaStream_t st) {
  fmm_note_launch(), k_h_fold<double><<<grid_of((long)t->ncells * h_terms(t->order)), H_BLOCK, 0, st>>>(
      t->ncells, t->order, t->so, M, mstr, Mh, hstr);
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}
