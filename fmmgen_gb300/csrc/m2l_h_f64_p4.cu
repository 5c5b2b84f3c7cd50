// m2l_h_f64_p4.cu -- generated by fmmgen_gb300/gen_m2l_h.py; do not edit.
// M2L over harmonic coefficients in double, orders up to 4 (see m2l_h.cuh).
#include "m2l_h.cuh"

// outputs of degree 0..4, multipole degrees 0..4: 25 accumulators, 1 per-pair sums, 155 multiply-adds at order 4
__global__ void __launch_bounds__(256, 1) k_m2lh_f64_p4_0(const HParams<double> P) {
  extern __shared__ float4 h_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  float4 *const mb = h_smem + w * 960, *const db = mb + 416;
  const HF64Row<13, 17> row(mb, db, lane);
  HList it(P, lane, w, W);
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0, a7 = 0, a8 = 0, a9 = 0, a10 = 0, a11 = 0, a12 = 0, a13 = 0, a14 = 0, a15 = 0, a16 = 0, a17 = 0, a18 = 0, a19 = 0, a20 = 0, a21 = 0, a22 = 0, a23 = 0, a24 = 0;
  if (it.begin(0)) {
    h_stage<0, 13, 0, 13>(mb, P.M, P.mstr, it.B, lane, h_words<8>(h_terms(min(4, it.qmax - 0))));
    h_stage<0, 8, 0, 17>(db, P.D, P.dstr, it.c, lane, h_words<8>(h_dterms(min(4, it.qmax))));
    h_commit();
    h_stage<8, 16, 0, 17>(db, P.D, P.dstr, it.c, lane, h_words<8>(h_dterms(min(4, it.qmax))));
    h_commit();
  }
  while (it.on_any) {
    it.look_ahead(0);
    const int ql = it.ql;
    h_wait<0>();
    __syncwarp();
    if (it.rescale) {  // the lane's own row
      row.scale(1, 4, h_exp2<double>(1 * it.dl));
      row.scale(4, 9, h_exp2<double>(2 * it.dl));
      row.scale(9, 16, h_exp2<double>(3 * it.dl));
      row.scale(16, 25, h_exp2<double>(4 * it.dl));
    }
    __syncwarp();
    double t0 = 0;
    if (ql >= 0) {
      const double d0 = row.d(0); row.fma<0>(t0, d0);
      if (ql >= 1) {
        const double d1 = row.d(1); row.fma<1>(t0, d1); row.fma<0>(a1, d1); const double d2 = row.d(2); row.fma<2>(t0, d2);
        row.fma<0>(a2, d2); const double d3 = row.d(3); row.fma<3>(t0, d3); row.fma<0>(a3, d3);
        if (ql >= 2) {
          const double d4 = row.d(4); row.fma<4>(t0, d4); row.fma<1>(a1, d4); row.fma<0>(a4, d4);
          const double d5 = row.d(5); row.fma<5>(t0, d5); row.fma<2>(a1, d5); row.fma<1>(a2, d5);
          row.fma<0>(a5, d5); const double d6 = row.d(6); row.fma<6>(t0, d6); row.fma<2>(a2, d6);
          row.fma<0>(a6, d6); const double d7 = row.d(7); row.fma<7>(t0, d7); row.fma<3>(a1, d7);
          row.fma<1>(a3, d7); row.fma<0>(a7, d7); const double d8 = row.d(8); row.fma<8>(t0, d8);
          row.fma<3>(a2, d8); row.fma<2>(a3, d8); row.fma<0>(a8, d8); const double d9 = row.d(9); row.fma<3>(a3, d9);
          if (ql >= 3) {
            const double d10 = row.d(10); row.fma<9>(t0, d10); row.fma<4>(a1, d10); row.fma<1>(a4, d10);
            row.fma<0>(a9, d10); const double d11 = row.d(11); row.fma<10>(t0, d11); row.fma<5>(a1, d11);
            row.fma<4>(a2, d11); row.fma<2>(a4, d11); row.fma<1>(a5, d11); row.fma<0>(a10, d11);
            const double d12 = row.d(12); row.fma<11>(t0, d12); row.fma<6>(a1, d12); row.fma<5>(a2, d12);
            row.fma<2>(a5, d12); row.fma<1>(a6, d12); row.fma<0>(a11, d12); const double d13 = row.d(13); row.fma<12>(t0, d13);
            row.fma<6>(a2, d13); row.fma<2>(a6, d13); row.fma<0>(a12, d13); const double d14 = row.d(14); row.fma<13>(t0, d14);
            row.fma<7>(a1, d14); row.fma<4>(a3, d14); row.fma<3>(a4, d14); row.fma<1>(a7, d14);
            row.fma<0>(a13, d14); const double d15 = row.d(15); row.fma<14>(t0, d15); row.fma<8>(a1, d15);
            row.fma<7>(a2, d15); row.fma<5>(a3, d15); row.fma<3>(a5, d15); row.fma<2>(a7, d15);
            row.fma<1>(a8, d15); row.fma<0>(a14, d15);
          }
        }
      }
    }
    __syncwarp();
    if (it.on_next)
      h_stage<0, 8, 0, 17>(db, P.D, P.dstr, it.cs, lane, h_words<8>(h_dterms(min(4, it.qmaxn))));
    h_commit();
    if (ql >= 3) {
      const double d16 = row.d(16); row.fma<15>(t0, d16); row.fma<8>(a2, d16); row.fma<6>(a3, d16);
      row.fma<3>(a6, d16); row.fma<2>(a8, d16); row.fma<0>(a15, d16); const double d17 = row.d(17); row.fma<7>(a3, d17);
      row.fma<3>(a7, d17); const double d18 = row.d(18); row.fma<8>(a3, d18); row.fma<3>(a8, d18);
      if (ql >= 4) {
        const double d19 = row.d(19); row.fma<16>(t0, d19); row.fma<9>(a1, d19); row.fma<4>(a4, d19);
        row.fma<1>(a9, d19); row.fma<0>(a16, d19); const double d20 = row.d(20); row.fma<17>(t0, d20);
        row.fma<10>(a1, d20); row.fma<9>(a2, d20); row.fma<5>(a4, d20); row.fma<4>(a5, d20);
        row.fma<2>(a9, d20); row.fma<1>(a10, d20); row.fma<0>(a17, d20); const double d21 = row.d(21); row.fma<18>(t0, d21);
        row.fma<11>(a1, d21); row.fma<10>(a2, d21); row.fma<6>(a4, d21); row.fma<5>(a5, d21);
        row.fma<4>(a6, d21); row.fma<2>(a10, d21); row.fma<1>(a11, d21); row.fma<0>(a18, d21);
        const double d22 = row.d(22); row.fma<19>(t0, d22); row.fma<12>(a1, d22); row.fma<11>(a2, d22);
        row.fma<6>(a5, d22); row.fma<5>(a6, d22); row.fma<2>(a11, d22); row.fma<1>(a12, d22);
        row.fma<0>(a19, d22); const double d23 = row.d(23); row.fma<20>(t0, d23); row.fma<12>(a2, d23);
        row.fma<6>(a6, d23); row.fma<2>(a12, d23); row.fma<0>(a20, d23); const double d24 = row.d(24); row.fma<21>(t0, d24);
        row.fma<13>(a1, d24); row.fma<9>(a3, d24); row.fma<7>(a4, d24); row.fma<4>(a7, d24);
        row.fma<3>(a9, d24); row.fma<1>(a13, d24); row.fma<0>(a21, d24); const double d25 = row.d(25); row.fma<22>(t0, d25);
        row.fma<14>(a1, d25); row.fma<13>(a2, d25); row.fma<10>(a3, d25); row.fma<8>(a4, d25);
        row.fma<7>(a5, d25); row.fma<5>(a7, d25); row.fma<4>(a8, d25); row.fma<3>(a10, d25);
        row.fma<2>(a13, d25); row.fma<1>(a14, d25); row.fma<0>(a22, d25); const double d26 = row.d(26); row.fma<23>(t0, d26);
        row.fma<15>(a1, d26); row.fma<14>(a2, d26); row.fma<11>(a3, d26); row.fma<8>(a5, d26);
        row.fma<7>(a6, d26); row.fma<6>(a7, d26); row.fma<5>(a8, d26); row.fma<3>(a11, d26);
        row.fma<2>(a14, d26); row.fma<1>(a15, d26); row.fma<0>(a23, d26); const double d27 = row.d(27); row.fma<24>(t0, d27);
        row.fma<15>(a2, d27); row.fma<12>(a3, d27); row.fma<8>(a6, d27); row.fma<6>(a8, d27);
        row.fma<3>(a12, d27); row.fma<2>(a15, d27); row.fma<0>(a24, d27); const double d28 = row.d(28); row.fma<13>(a3, d28);
        row.fma<7>(a7, d28); row.fma<3>(a13, d28); const double d29 = row.d(29); row.fma<14>(a3, d29);
        row.fma<8>(a7, d29); row.fma<7>(a8, d29); row.fma<3>(a14, d29); const double d30 = row.d(30); row.fma<15>(a3, d30);
        row.fma<8>(a8, d30); row.fma<3>(a15, d30);
      }
    }
    a0 += t0;
    __syncwarp();
    if (it.on_next) {
      h_stage<0, 13, 0, 13>(mb, P.M, P.mstr, it.Bs, lane, h_words<8>(h_terms(min(4, it.qmaxn - 0))));
      h_stage<8, 16, 0, 17>(db, P.D, P.dstr, it.cs, lane, h_words<8>(h_dterms(min(4, it.qmaxn))));
    }
    h_commit();
    it.advance();
  }
  h_wait<0>();
  // the warps' sums, in shared memory
  double *const sum = (double *)(h_smem + w * 960) + lane;
  __syncwarp();
  sum[0] = a0; sum[32] = a1; sum[64] = a2; sum[96] = a3;
  sum[128] = a4; sum[160] = a5; sum[192] = a6; sum[224] = a7;
  sum[256] = a8; sum[288] = a9; sum[320] = a10; sum[352] = a11;
  sum[384] = a12; sum[416] = a13; sum[448] = a14; sum[480] = a15;
  sum[512] = a16; sum[544] = a17; sum[576] = a18; sum[608] = a19;
  sum[640] = a20; sum[672] = a21; sum[704] = a22; sum[736] = a23;
  sum[768] = a24;
  h_store<double, 25, 1920, false>(P, (double *)h_smem, 0, W);
}

int fmm_m2lh_f64_p4(const HParams<double> &P, cudaStream_t st) {
  if (P.p >= 0)
    if (int rc = h_launch(k_m2lh_f64_p4_0, P, 15360, 8, st)) return rc;
  return FMM_OK;
}
