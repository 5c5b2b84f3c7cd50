// m2l_h.cuh -- M2L over harmonic coefficients (example/calculate.cpp:190-206 with
// fmmgen's M2L, fmmgen/expansions.py:144-172): parameters, the pair loop's
// pieces and the launch rule of the generated kernels (m2l_h_*.cu, written by
// gen_m2l_h.py, which has the mathematics and the layouts).
#pragma once
#include <cooperative_groups.h>
#include "internal.h"

// coefficients / operator entries up to degree d
__host__ __device__ __forceinline__ constexpr int h_terms(int d) { return d < 0 ? 0 : (d + 1) * (d + 1); }
__host__ __device__ __forceinline__ constexpr int h_dterms(int d) { return d < 0 ? 0 : 1 + 3 * d * (d + 1) / 2; }
__host__ __device__ __forceinline__ int h_index(int x, int y, int z) {  // z <= 1
  const int d = x + y + z;
  return d * d + (z ? (d + 1) + (d - 1 - x) : d - x);
}
__host__ __device__ __forceinline__ int h_dindex(int x, int y, int z) {  // z <= 2
  const int d = x + y + z;
  return h_dterms(d - 1) + (z == 0 ? d - x : z == 1 ? (d + 1) + (d - 1 - x) : (2 * d + 1) + (d - 2 - x));
}
// 16-byte words that hold n elements of `SIZE` bytes
template <int SIZE> __host__ __device__ __forceinline__ constexpr int h_words(int n) { return (n * SIZE + 15) / 16; }

template <typename T> struct HParams {
  const int *tgt;               // [ntgt] target cells
  int ntgt;
  const int *off, *src, *cls;   // target lists: pairs of cell A are off[A] .. off[A + 1] - 1
  const int *perm;              // pair indices of each list by descending order, or null (list order)
  const unsigned char *ord;     // per-pair orders (list order, needs perm), or null: every pair at order p
  int p, qlo;                   // the order; the lowest order a pair can have
  const T *D;                   // [classes] operator rows of dstr bytes
  int dstr;
  const unsigned char *clevel;  // [ncells]
  const T *M;                   // [ncells] source rows of mstr bytes (degrees below the source order: zeros)
  int mstr;
  T *L;                         // [ncells][lstr] outputs
  int lstr, lsize;
};

__device__ __forceinline__ void h_copy16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void h_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void h_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
template <typename T> __device__ __forceinline__ T h_exp2(int e);
template <> __device__ __forceinline__ float h_exp2<float>(int e) {  // e <= 127; zero below FP32's normal numbers
  return e < -126 ? 0.f : __int_as_float((e + 127) << 23);
}
template <> __device__ __forceinline__ double h_exp2<double>(int e) {
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// Copies the 16-byte words [LO, HI) of the 32 lanes' rows (lane r's row number
// in lane r's `row`; none when negative) that lie below `need`; word q of row r
// lands in dst[r * STRIDE + q - BASE].  Eight lanes take a row's consecutive
// words, four rows per instruction.
template <int LO, int HI, int BASE, int STRIDE, typename T>
__device__ __forceinline__ void h_stage(float4 *dst, const T *rows, int rowbytes, int row, int lane, int need) {
  const int sub = lane & 7;
  need = min(need, HI);
#pragma unroll
  for (int g = 0; g < 8; g++) {
    const int r = 4 * g + (lane >> 3);
    const int R = __shfl_sync(0xffffffffu, row, r);
    const char *s = (const char *)rows + (size_t)max(R, 0) * rowbytes + 16 * (LO + sub);
    float4 *d = dst + r * STRIDE + (LO - BASE) + sub;
    const int have = R >= 0 ? need - LO - sub : 0;
#pragma unroll
    for (int c = 0; c < (HI - LO + 7) / 8; c++)
      if (8 * c < have) h_copy16(d + 8 * c, s + 128 * c);
  }
}

// The lane's staged rows.
template <int MSTR, int DSTR> struct HF32Row {
  const float4 *pm, *pd;
  __device__ __forceinline__ HF32Row(const float4 *mb, const float4 *db, int lane)
      : pm(mb + lane * MSTR), pd(db + lane * DSTR) {}
  __device__ __forceinline__ float4 m(int q) const { return pm[q]; }
  __device__ __forceinline__ float4 d(int q) const { return pd[q]; }
};
template <int MSTR, int DSTR> struct HF64Row {
  double *pm;
  const double *pd;
  unsigned am;
  __device__ __forceinline__ HF64Row(float4 *mb, const float4 *db, int lane)
      : pm((double *)(mb + lane * MSTR)), pd((const double *)(db + lane * DSTR)),
        am((unsigned)__cvta_generic_to_shared(mb + lane * MSTR)) {}
  __device__ __forceinline__ double d(int k) const { return pd[k]; }
  // acc += D * row[J]; a load of its own each time: kept in registers, the row would not fit beside the outputs
  template <int J> __device__ __forceinline__ void fma(double &acc, double D) const {
    double m;
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(m) : "r"(am + 8 * J));
    acc = __fma_rn(D, m, acc);
  }
  __device__ __forceinline__ void scale(int j0, int j1, double s) const {
    for (int j = j0; j < j1; j++) pm[j] *= s;
  }
};

// A lane's share of its target's list: entries w, w + W, ... (the W warps of a
// block share 32 targets).  `cur` is the pair being multiplied, its rows
// staged; the next pair's indices are loaded, and the list position of the one
// after it (a permuted list is a chain of two loads).
struct HList {
  const int *src, *cls, *perm;
  const unsigned char *ord, *clevel;
  int A, la, k0, n, W, p, qlo, j;  // j: list position of the pair after next
  int B, c, q;                     // current pair: source, class, order (-1: none)
  int Bn, cn, qn, k2;              // next pair; list index of the pair after it
  int Bs, cs;                      // next pair's rows to stage (-1: none)
  int ql, qmax, qmaxn, dl;
  bool on_any, on_next, rescale;
  template <typename T>
  __device__ __forceinline__ HList(const HParams<T> &P, int lane, int w, int W_)
      : src(P.src), cls(P.cls), perm(P.perm), ord(P.ord), clevel(P.clevel), W(W_), p(P.p), qlo(P.qlo) {
    // a cluster's blocks share 32 targets too
    const unsigned nb = cooperative_groups::this_cluster().num_blocks();
    const int t = (int)(blockIdx.x / nb) * 32 + lane;
    w += (int)cooperative_groups::this_cluster().block_rank() * W;
    W *= (int)nb;
    A = t < P.ntgt ? P.tgt[t] : -1;
    la = A >= 0 ? (int)clevel[A] : 0;
    k0 = A >= 0 ? P.off[A] : 0;
    n = A >= 0 ? P.off[A + 1] - k0 : 0;
    j = w;
    load(index(), B, c, q);
    j += W;
    load(index(), Bn, cn, qn);
    j += W;
    k2 = index();
  }
  __device__ __forceinline__ int index() const { return j < n ? (perm ? perm[k0 + j] : k0 + j) : -1; }
  __device__ __forceinline__ void load(int k, int &B_, int &c_, int &q_) const {
    B_ = k >= 0 ? src[k] : -1;
    c_ = k >= 0 ? cls[k] : -1;
    q_ = k < 0 ? -1 : ord ? min(max((int)ord[k], qlo), p) : p;
  }
  __device__ __forceinline__ bool begin(int dmin) {
    const bool on = q >= dmin;
    on_any = __any_sync(0xffffffffu, on);
    qmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)(on ? q : 0));
    if (!on) B = c = -1;
    return on_any;
  }
  // orders and level difference of the current pair; whether a next one follows.  A pair across more than `wide`
  // levels has an operator of zeros (k_h_operators): its source stays as it is.
  __device__ __forceinline__ void look_ahead(int dmin, int wide = 1 << 20) {
    const bool on = q >= dmin, onn = qn >= dmin;
    ql = on ? q : -1;
    dl = on ? la - (int)clevel[B] : 0;
    if (dl > wide) dl = 0;
    rescale = __any_sync(0xffffffffu, dl != 0);
    on_next = __any_sync(0xffffffffu, onn);  // lists go by descending order: no lane on, none later
    qmaxn = (int)__reduce_max_sync(0xffffffffu, (unsigned)(onn ? qn : 0));
    Bs = onn ? Bn : -1;
    cs = onn ? cn : -1;
  }
  __device__ __forceinline__ void advance() {
    B = Bn;
    c = cn;
    q = qn;
    on_any = on_next;
    load(k2, Bn, cn, qn);
    j += W;
    k2 = index();
  }
};

// The targets' outputs: the warps' sums ([warp][output][lane], `STRIDE` elements
// per warp) of the cluster's blocks added in a fixed order, stored in (or added
// to) the targets' rows; the blocks share the work.
template <typename T, int NOUT, int STRIDE, bool ADD>
__device__ __forceinline__ void h_store(const HParams<T> &P, T *sum, int i0, int W) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int t0 = (int)(blockIdx.x / nb) * 32;
  if (nb == 1) __syncthreads();
  else cl.sync();
  for (int e = rank * blockDim.x + threadIdx.x; e < 32 * NOUT; e += nb * blockDim.x) {
    const int r = e / NOUT, i = e - r * NOUT;
    if (t0 + r >= P.ntgt || i0 + i >= P.lsize) continue;
    T v = T(0);
    for (int b = 0; b < nb; b++) {
      const T *s = nb == 1 ? sum : cl.map_shared_rank(sum, b);
      for (int u = 0; u < W; u++) v += s[u * STRIDE + 32 * i + r];
    }
    T *o = P.L + (size_t)P.tgt[t0 + r] * P.lstr + i0 + i;
    *o = ADD ? *o + v : v;
  }
  if (nb > 1) cl.sync();  // the sums stay readable until every block has added them
}

// The lists of 32 targets are split over the four warps of a block and, in small
// trees, over the C blocks of a cluster: up to 28 warps per SM in all, about
// four rounds of the eight that are resident (FP64: seven of four), so that the
// longest lists do not decide alone and no SM idles.  Measured, FP32 (one
// GB300), C = 1 / 2 / 4 / 8: 585 cells, p = 4: 63 / 39 / 27 / 25 us; 4,681 cells,
// p = 8: 301 / 217 / 205 / 366 us; 8,357 cells, p = 6: 262 / 164 / 147 / 312 us;
// 37,449 cells, p = 8: 1.63 / 1.68 / 2.09 / 3.15 ms (one and two warps per block
// with C = 1: 1.89, 1.84).
template <typename T>
static int h_launch(void (*k)(const HParams<T>), const HParams<T> &P, int smem, int maxw, cudaStream_t st) {
  const long groups = ((long)P.ntgt + 31) / 32;
  if (groups == 0) return FMM_OK;
  const int W = maxw < 4 ? maxw : 4;
  int C = 1;
  while (C < 8 && groups * W * 2 * C <= 28L * 152) C *= 2;
  FMM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem * W));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups * C));
  cfg.blockDim = dim3(32 * W);
  cfg.dynamicSmemBytes = (size_t)smem * W;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  fmm_note_launch();
  FMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, P));
  return FMM_OK;
}

// the family with the smallest largest order >= P.p
int fmm_m2lh_f32_p4(const HParams<float> &P, cudaStream_t st);
int fmm_m2lh_f32_p6(const HParams<float> &P, cudaStream_t st);
int fmm_m2lh_f32_p8(const HParams<float> &P, cudaStream_t st);
int fmm_m2lh_f32_p12(const HParams<float> &P, cudaStream_t st);
int fmm_m2lh_f64_p4(const HParams<double> &P, cudaStream_t st);
int fmm_m2lh_f64_p6(const HParams<double> &P, cudaStream_t st);
int fmm_m2lh_f64_p8(const HParams<double> &P, cudaStream_t st);
int fmm_m2lh_f64_p12(const HParams<double> &P, cudaStream_t st);
static inline int h_run(const HParams<float> &P, cudaStream_t st) {
  return P.p <= 4   ? fmm_m2lh_f32_p4(P, st)
         : P.p <= 6 ? fmm_m2lh_f32_p6(P, st)
         : P.p <= 8 ? fmm_m2lh_f32_p8(P, st)
                    : fmm_m2lh_f32_p12(P, st);
}
static inline int h_run(const HParams<double> &P, cudaStream_t st) {
  return P.p <= 4   ? fmm_m2lh_f64_p4(P, st)
         : P.p <= 6 ? fmm_m2lh_f64_p6(P, st)
         : P.p <= 8 ? fmm_m2lh_f64_p8(P, st)
                    : fmm_m2lh_f64_p12(P, st);
}
