// ops.cu -- batched device versions of fmmgen's generated operators.
//
// Each entry applies one operator to n independent (displacement, input,
// output) triples with the generated code's "+=" semantics and unscaled
// coefficients, in FP64 (or FP32 through the _f32 entries).  They replace n calls of P2M_p / M2M_p / M2L_p /
// L2L_p / L2P_p / P2P from fmmgen/writer.py:142-264 (signatures
// fmmgen/printers.py:296-313), one warp per application.
#include "internal.h"
#include "deriv.cuh"

// Every kernel here but P2P and M2P takes one warp per application and, in FP64,
// is bound by the FP64 pipe (16 clocks of an SM per warp instruction): what
// counts is the number of those.  20,000 applications, p = 8, FP64, one GB300:
// P2M 1.48 -> 0.045 ms, M2M and L2L 1.77 -> 0.12 and 0.14 ms, M2L 0.59 -> 0.50 ms,
// L2P 1.54 -> 0.07 ms.

// The warp contraction engine on one application: every (lane, output) segment
// of the plan is finished once and stored -- adding into the slot would double
// the FP64 instructions (some lane ends a segment in almost every round).
template <typename T>
__device__ __forceinline__ void engine_run_op(const Plan &P, const T *A, const T *B, T *slots, int lane) {
  T acc = T(0);
  for (int it = 0; it < P.iters; ++it) {
    uint32_t w = __ldg(&P.task[it * 32 + lane]);
    if (w == 0xffffffffu) break;
    acc += A[w & 1023u] * B[(w >> 10) & 1023u];
    if (w >> 31) {
      slots[(w >> 20) & 2047u] = acc;
      acc = T(0);
    }
  }
}
template <typename T> __device__ __forceinline__ T engine_out_op(const Plan &P, const T *slots, int n) {
  const int k0 = __ldg(&P.out_seg[n]), k1 = __ldg(&P.out_seg[n + 1]);
  T s = slots[k0];
  for (int k = k0 + 1; k < k1; k++) s += slots[k];
  return s;
}

// Multi-indices (x, y, z, degree) up to order p in shared memory: the lanes read
// different ones, which the constant bank would serve one at a time.
__device__ __forceinline__ void op_indices(int p, uchar4 *mi) {
  for (int e = threadIdx.x; e < fmm_nterms(p); e += blockDim.x)
    mi[e] = make_uchar4(c_mi[e][0], c_mi[e][1], c_mi[e][2], c_mi[e][3]);
  __syncthreads();
}

// 1/k!
static __constant__ double c_rfact[FMM_PMAX + 1] = {1.,       1.,        1. / 2,     1. / 6,      1. / 24,
                                                    1. / 120, 1. / 720,  1. / 5040,  1. / 40320,  1. / 362880,
                                                    1. / 3628800, 1. / 39916800, 1. / 479001600};

// tab[a][k] = v_a^k / k! of the three axes, k <= pmax: an entry per lane, one chain
// of multiplications for all of them instead of a division per power of every
// monomial.
template <typename T>
__device__ __forceinline__ void op_powers(T vx, T vy, T vz, int pmax, T (*tab)[FMM_PMAX + 1], int lane) {
  for (int e = lane; e < 3 * (pmax + 1); e += 32) {
    const int a = e / (pmax + 1), k = e - a * (pmax + 1);
    const T v = a == 0 ? vx : a == 1 ? vy : vz;
    T r = k > 0 ? v : T(1);
    for (int q = 2; q <= pmax; q++)
      if (q <= k) r *= v;
    tab[a][k] = r * (T)c_rfact[k];
  }
}

#define OPW 4

// P2M_p: M[n] += (-1)^|n| q x^n/n!  (fmmgen/expansions.py:22-39)
template <typename T>
__global__ void k_op_p2m(int n, const T *d, const T *q, T *M, int order, int so) {
  __shared__ T tab[OPW][3][FMM_PMAX + 1];
  __shared__ uchar4 mi[FMM_NTMAX];
  op_indices(order, mi);
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int i = blockIdx.x * OPW + w;
  if (i >= n) return;
  op_powers(-d[3 * i], -d[3 * i + 1], -d[3 * i + 2], order, tab[w], lane);
  __syncwarp();
  int off = fmm_nterms(so - 1), ms = fmm_nterms(order) - off;
  const T qi = q[i];
  for (int j = lane; j < ms; j += 32) {
    const uchar4 m = mi[j + off];
    M[(size_t)i * ms + j] += qi * (tab[w][0][m.x] * tab[w][1][m.y] * tab[w][2][m.z]);
  }
}

// M2M_p (fmmgen/expansions.py:42-78) and L2L_p (fmmgen/expansions.py:175-194), one
// axis after the other:
//   M2M  out_n = sum_k v_a^k / k! in_(n - k e_a), k <= n_a, |n| - k >= the source order
//   L2L  out_n = sum_k v_a^k / k! in_(n + k e_a), |n| + k <= order - source order
// A shift monomial is the product of its axes' powers, so the three passes
// together are the full sum: 3 x 495 multiply-adds at p = 8 instead of 3,003, and
// no plan to decode.  The lanes of a round take outputs with equally long sums: in
// the L2L those of one degree, in the M2M those of one n_a (entry e of the
// multi-index table, of degree d, stands for n_a = p - d and the other two
// components y and z: p - d is met by as many outputs as there are indices of
// degree d).
template <typename T, bool L2L>
__global__ void k_op_shift(int n, const T *d, const T *in, T *out, int order, int so) {
  __shared__ T buf[OPW][2][FMM_NTMAX], tab[OPW][3][FMM_PMAX + 1];
  __shared__ uchar4 mi[FMM_NTMAX];
  __shared__ int nt[FMM_PMAX + 2];  // nt[d + 1] = fmm_nterms(d)
  if (threadIdx.x < FMM_PMAX + 2) nt[threadIdx.x] = fmm_nterms((int)threadIdx.x - 1);
  op_indices(order, mi);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * OPW + w;
  if (i >= n) return;
  const int p = L2L ? order - so : order, lo = L2L ? 0 : so;  // degrees lo .. p
  const int off = nt[lo], size = nt[p + 1] - off;
  op_powers(d[3 * i], d[3 * i + 1], d[3 * i + 2], order - so, tab[w], lane);
  for (int j = lane; j < size; j += 32) buf[w][0][j + off] = in[(size_t)i * size + j];
  __syncwarp();
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const T *src = buf[w][a & 1], *t = tab[w][a];
    for (int e = lane; e < nt[p + 1]; e += 32) {
      const uchar4 m = mi[e];
      // the output's component along the axis, and the other two in their order
      const int na = L2L ? (a == 0 ? m.x : a == 1 ? m.y : m.z) : p - m.w;
      const int b = L2L ? (a == 0 ? m.y : m.x) : m.y, c = L2L ? (a == 2 ? m.y : m.z) : m.z;
      const int deg = na + b + c;
      if (deg < lo) continue;
      const int len = L2L ? p - deg : min(na, deg - lo);
      // place of an index (x, y, z) of degree g: nt[g] + j (j + 1) / 2 + z, j = y + z
      T s = T(0);
      int o = 0;
      for (int k = 0; k <= len; k++) {
        const int q = L2L ? na + k : na - k, g = L2L ? deg + k : deg - k;
        const int j = a == 0 ? b + c : a == 1 ? q + c : c + q;
        const int z = a == 2 ? q : c;
        const int at = nt[g] + j * (j + 1) / 2 + z;
        if (k == 0) o = at;
        s += t[k] * src[at];
      }
      if (a == 2) out[(size_t)i * size + o - off] += s;
      else buf[w][(a & 1) ^ 1][o] = s;
    }
    __syncwarp();
  }
}

// M2L_p (fmmgen/expansions.py:144-172): derivatives at d, then the contraction
template <typename T>
__global__ void k_op_m2l(Plan P, int n, const T *d, const T *M, T *L, int order, int so) {
  // sT is the recurrence's scratch, then holds the source multipole
  __shared__ T sD[OPW][FMM_NTMAX], sT[OPW][FMM_NTMAX], sS[OPW][FMM_NTMAX + 32];
  __shared__ T sb[OPW][FMM_PMAX + 1];
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int i = blockIdx.x * OPW + w;
  if (i >= n) return;
  warp_derivs<T>(d[3 * i], d[3 * i + 1], d[3 * i + 2], order, sD[w], sT[w], sb[w]);
  T *sB = sT[w];
  int ms = fmm_nterms(order) - fmm_nterms(so - 1), ls = fmm_nterms(order - so);
  for (int j = lane; j < ms; j += 32) sB[j] = M[(size_t)i * ms + j];
  __syncwarp();
  engine_run_op<T>(P, sD[w], sB, sS[w], lane);
  __syncwarp();
  for (int j = lane; j < ls; j += 32) L[(size_t)i * ls + j] += engine_out_op(P, sS[w], j);
}

// L2P_p (fmmgen/expansions.py:197-207)
template <typename T>
__global__ void k_op_l2p(int n, const T *d, const T *L, T *F, int order, int so, int potential,
                         int field) {
  __shared__ T mon[OPW][FMM_NTMAX], tab[OPW][3][FMM_PMAX + 1];
  __shared__ uchar4 mi[FMM_NTMAX];
  op_indices(order, mi);
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int i = blockIdx.x * OPW + w;
  if (i >= n) return;
  int pl = order - so, ls = fmm_nterms(pl);
  op_powers(d[3 * i], d[3 * i + 1], d[3 * i + 2], pl, tab[w], lane);
  __syncwarp();
  for (int j = lane; j < ls; j += 32) {
    const uchar4 m = mi[j];
    mon[w][j] = tab[w][0][m.x] * tab[w][1][m.y] * tab[w][2][m.z];
  }
  __syncwarp();
  T phi = 0, ex = 0, ey = 0, ez = 0;
  const T *Li = L + (size_t)i * ls;
  for (int j = lane; j < ls; j += 32) {
    const int nx = mi[j].x, ny = mi[j].y, nz = mi[j].z;
    T l = Li[j];
    phi += l * mon[w][j];
    if (nx) ex -= l * mon[w][fmm_idx3(nx - 1, ny, nz)];
    if (ny) ey -= l * mon[w][fmm_idx3(nx, ny - 1, nz)];
    if (nz) ez -= l * mon[w][fmm_idx3(nx, ny, nz - 1)];
  }
  // the warp's sums: two exchanges that halve the number of values a lane holds
  // (phi, ex | ey, ez, then one each), then one value per lane to add
  const bool up = lane & 16, odd = lane & 8;
  T v0 = up ? ey : phi, v1 = up ? ez : ex;
  v0 += __shfl_xor_sync(0xffffffffu, up ? phi : ey, 16);
  v1 += __shfl_xor_sync(0xffffffffu, up ? ex : ez, 16);
  T v = odd ? v1 : v0;
  v += __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 8);
  for (int o = 4; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  // lanes 0, 8, 16, 24 hold phi, ex, ey, ez
  if ((lane & 7) == 0) {
    const int k = lane >> 3;
    const int os = (potential ? 1 : 0) + (field ? 3 : 0);
    T *Fi = F + (size_t)i * os;
    if (k == 0) {
      if (potential) Fi[0] += v;
    } else if (field) {
      Fi[k - 1 + (potential ? 1 : 0)] += v;
    }
  }
}

// P2P (Coulomb form of example/operators.cpp:54-66; dipole and quadrupole
// fields restated as the gradients of the generated potentials)
template <typename T>
__global__ void k_op_p2p(int n, const T *d, const T *S, T *F, int so, int potential, int field) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  T x = d[3 * i], y = d[3 * i + 1], z = d[3 * i + 2];
  T R = sqrt(x * x + y * y + z * z);
  T phi = 0, ex = 0, ey = 0, ez = 0;
  if (so == 2) {
    quadrupole_p2p<T>(x, y, z, S + 6 * (size_t)i, phi, ex, ey, ez);
  } else if (so == 0) {
    T q = S[i];
    T r3 = T(1) / (R * R * R);
    phi = q / R;
    ex = q * x * r3; ey = q * y * r3; ez = q * z * r3;
  } else {
    const T *s = S + 3 * (size_t)i;
    T rinv = T(1) / R, r3 = rinv * rinv * rinv, r5 = r3 * rinv * rinv;
    T sr = s[0] * x + s[1] * y + s[2] * z;
    phi = -sr * r3;
    ex = s[0] * r3 - T(3) * sr * x * r5; ey = s[1] * r3 - T(3) * sr * y * r5; ez = s[2] * r3 - T(3) * sr * z * r5;
  }
  int os = (potential ? 1 : 0) + (field ? 3 : 0);
  T *Fi = F + (size_t)i * os;
  int k = 0;
  if (potential) Fi[k++] += phi;
  if (field) { Fi[k] += ex; Fi[k + 1] += ey; Fi[k + 2] += ez; }
}

// op: 0 P2M, 1 M2M, 2 M2L, 3 L2L, 4 L2P, 5 P2P
// M2P_p (fmmgen/generator.py:174-206), one thread per application: the
// potential V = sum_m D_m(d) M_m of fmmgen's M2P and its exact gradient
// E = -sum_m D_(m+e)(d) M_m (the generated field is not that gradient);
// d = particle - cell.  NTQ holds the derivatives to order + 1.
template <typename T, int NTQ>
__global__ void k_op_m2p(int n, const T *d, const T *M, T *F, int order, int so, int potential,
                         int field) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  T D[NTQ];
  thread_derivs(d[3 * i], d[3 * i + 1], d[3 * i + 2], order + 1, D);
  const int moff = fmm_nterms(so - 1), ms = fmm_nterms(order) - moff;
  const T *Mi = M + (size_t)i * ms;
  T v = 0, gx = 0, gy = 0, gz = 0;
  int j = moff;
  for (int dg = so; dg <= order; dg++)
    for (int mx = dg; mx >= 0; mx--)
      for (int my = dg - mx; my >= 0; my--, j++) {
        const int mz = dg - mx - my;
        const T w = Mi[j - moff];
        v += D[j] * w;
        gx += D[fmm_idx3(mx + 1, my, mz)] * w;
        gy += D[fmm_idx3(mx, my + 1, mz)] * w;
        gz += D[fmm_idx3(mx, my, mz + 1)] * w;
      }
  const int os = (potential ? 1 : 0) + (field ? 3 : 0);
  T *Fi = F + (size_t)i * os;
  int k = 0;
  if (potential) Fi[k++] += v;
  if (field) {
    Fi[k] -= gx;
    Fi[k + 1] -= gy;
    Fi[k + 2] -= gz;
  }
}

template <typename T>
static int op_batch(int op, int n, const T *d, const T *in, T *out, int order, int so, int potential, int field,
                    cudaStream_t st) {
  if (n < 0 || so < 0 || so > 2 || !d || !in || !out) return FMM_ERR_ARG;
  if (op != 5 && (order < 0 || order > FMM_PMAX || order < so)) return FMM_ERR_ARG;
  if ((op == 4 || op == 5 || op == 6) && !potential && !field) return FMM_ERR_ARG;
  if (n == 0) return FMM_OK;
  unsigned nb = fmm_blocks(n, OPW);
  const PlanSet *ps = nullptr;
  if (op == 2) {
    ps = fmm_get_plans(order, so);
    if (!ps) return FMM_ERR_CUDA;
  }
  switch (op) {
    case 0: fmm_note_launch(), k_op_p2m<T><<<nb, 32 * OPW, 0, st>>>(n, d, in, out, order, so); break;
    case 1: fmm_note_launch(), k_op_shift<T, false><<<nb, 32 * OPW, 0, st>>>(n, d, in, out, order, so); break;
    case 2: fmm_note_launch(), k_op_m2l<T><<<nb, 32 * OPW, 0, st>>>(ps->m2l, n, d, in, out, order, so); break;
    case 3: fmm_note_launch(), k_op_shift<T, true><<<nb, 32 * OPW, 0, st>>>(n, d, in, out, order, so); break;
    case 4: fmm_note_launch(), k_op_l2p<T><<<nb, 32 * OPW, 0, st>>>(n, d, in, out, order, so, potential, field); break;
    case 5: fmm_note_launch(), k_op_p2p<T><<<fmm_blocks(n, 128), 128, 0, st>>>(n, d, in, out, so, potential, field); break;
    case 6:
      if (order + 1 <= 6) fmm_note_launch(), k_op_m2p<T, 84><<<fmm_blocks(n, 128), 128, 0, st>>>(n, d, in, out, order, so, potential, field);
      else if (order + 1 <= 9) fmm_note_launch(), k_op_m2p<T, 220><<<fmm_blocks(n, 128), 128, 0, st>>>(n, d, in, out, order, so, potential, field);
      else fmm_note_launch(), k_op_m2p<T, 560><<<fmm_blocks(n, 128), 128, 0, st>>>(n, d, in, out, order, so, potential, field);
      break;
    default: return FMM_ERR_ARG;
  }
  FMM_CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

int fmm_op_batch(int op, int n, const double *d, const double *in, double *out, int order, int so, int potential,
                 int field, cudaStream_t st) {
  return op_batch<double>(op, n, d, in, out, order, so, potential, field, st);
}

// The same operators in FP32 (the generator's precision="float" variant,
// fmmgen/writer.py:105): float buffers, float arithmetic throughout.
int fmm_op_batch_f32(int op, int n, const float *d, const float *in, float *out, int order, int so, int potential,
                     int field, cudaStream_t st) {
  return op_batch<float>(op, n, d, in, out, order, so, potential, field, st);
}
