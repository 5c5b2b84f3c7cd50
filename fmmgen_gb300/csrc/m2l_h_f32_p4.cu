// m2l_h_f32_p4.cu -- generated by fmmgen_gb300/gen_m2l_h.py; do not edit.
// M2L over harmonic coefficients in float, orders up to 4 (see m2l_h.cuh).
#include "m2l_h.cuh"

// outputs of degree 0..4, multipole degrees 0..4: 25 accumulators, 1 per-pair sums, 155 multiply-adds at order 4
__global__ void __launch_bounds__(256, 1) k_m2lh_f32_p4_0(const HParams<float> P) {
  extern __shared__ float4 h_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  float4 *const mb = h_smem + w * 512, *const db = mb + 224;
  const HF32Row<7, 9> row(mb, db, lane);
  HList it(P, lane, w, W);
  float a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0, a7 = 0, a8 = 0, a9 = 0, a10 = 0, a11 = 0, a12 = 0, a13 = 0, a14 = 0, a15 = 0, a16 = 0, a17 = 0, a18 = 0, a19 = 0, a20 = 0, a21 = 0, a22 = 0, a23 = 0, a24 = 0;
  if (it.begin(0)) {
    h_stage<0, 7, 0, 7>(mb, P.M, P.mstr, it.B, lane, h_words<4>(h_terms(min(4, it.qmax - 0))));
    h_stage<0, 8, 0, 9>(db, P.D, P.dstr, it.c, lane, h_words<4>(h_dterms(min(4, it.qmax))));
    h_commit();

    h_commit();
  }
  while (it.on_any) {
    it.look_ahead(0, fmm_wide_levels(4));
    const int ql = it.ql;
    h_wait<1>();  // the source row and the operator's first half
    __syncwarp();
    const float4 mq0 = row.m(0);
    const float4 mq1 = row.m(1);
    const float4 mq2 = row.m(2);
    const float4 mq3 = row.m(3);
    const float4 mq4 = row.m(4);
    const float4 mq5 = row.m(5);
    const float4 mq6 = row.m(6);
    float m0 = mq0.x, m1 = mq0.y, m2 = mq0.z, m3 = mq0.w, m4 = mq1.x, m5 = mq1.y, m6 = mq1.z, m7 = mq1.w, m8 = mq2.x, m9 = mq2.y, m10 = mq2.z, m11 = mq2.w, m12 = mq3.x, m13 = mq3.y, m14 = mq3.z, m15 = mq3.w, m16 = mq4.x, m17 = mq4.y, m18 = mq4.z, m19 = mq4.w, m20 = mq5.x, m21 = mq5.y, m22 = mq5.z, m23 = mq5.w, m24 = mq6.x;
    if (it.rescale) {
      const float s1 = h_exp2<float>(1 * it.dl);
      m1 *= s1; m2 *= s1; m3 *= s1;
      const float s2 = h_exp2<float>(2 * it.dl);
      m4 *= s2; m5 *= s2; m6 *= s2; m7 *= s2; m8 *= s2;
      const float s3 = h_exp2<float>(3 * it.dl);
      m9 *= s3; m10 *= s3; m11 *= s3; m12 *= s3; m13 *= s3; m14 *= s3; m15 *= s3;
      const float s4 = h_exp2<float>(4 * it.dl);
      m16 *= s4; m17 *= s4; m18 *= s4; m19 *= s4; m20 *= s4; m21 *= s4; m22 *= s4; m23 *= s4; m24 *= s4;
    }
    __syncwarp();
    if (it.on_next)
      h_stage<0, 7, 0, 7>(mb, P.M, P.mstr, it.Bs, lane, h_words<4>(h_terms(min(4, it.qmaxn - 0))));
    h_commit();
    float t0 = 0;
    if (ql >= 0) {
      const float4 d0 = row.d(0); t0 = fmaf(d0.x, m0, t0);
      if (ql >= 1) {
        t0 = fmaf(d0.y, m1, t0); a1 = fmaf(d0.y, m0, a1); t0 = fmaf(d0.z, m2, t0); a2 = fmaf(d0.z, m0, a2);
        t0 = fmaf(d0.w, m3, t0); a3 = fmaf(d0.w, m0, a3);
        if (ql >= 2) {
          const float4 d1 = row.d(1); t0 = fmaf(d1.x, m4, t0); a1 = fmaf(d1.x, m1, a1); a4 = fmaf(d1.x, m0, a4);
          t0 = fmaf(d1.y, m5, t0); a1 = fmaf(d1.y, m2, a1); a2 = fmaf(d1.y, m1, a2); a5 = fmaf(d1.y, m0, a5);
          t0 = fmaf(d1.z, m6, t0); a2 = fmaf(d1.z, m2, a2); a6 = fmaf(d1.z, m0, a6); t0 = fmaf(d1.w, m7, t0);
          a1 = fmaf(d1.w, m3, a1); a3 = fmaf(d1.w, m1, a3); a7 = fmaf(d1.w, m0, a7); const float4 d2 = row.d(2); t0 = fmaf(d2.x, m8, t0);
          a2 = fmaf(d2.x, m3, a2); a3 = fmaf(d2.x, m2, a3); a8 = fmaf(d2.x, m0, a8); a3 = fmaf(d2.y, m3, a3);
          if (ql >= 3) {
            t0 = fmaf(d2.z, m9, t0); a1 = fmaf(d2.z, m4, a1); a4 = fmaf(d2.z, m1, a4); a9 = fmaf(d2.z, m0, a9);
            t0 = fmaf(d2.w, m10, t0); a1 = fmaf(d2.w, m5, a1); a2 = fmaf(d2.w, m4, a2); a4 = fmaf(d2.w, m2, a4);
            a5 = fmaf(d2.w, m1, a5); a10 = fmaf(d2.w, m0, a10); const float4 d3 = row.d(3); t0 = fmaf(d3.x, m11, t0);
            a1 = fmaf(d3.x, m6, a1); a2 = fmaf(d3.x, m5, a2); a5 = fmaf(d3.x, m2, a5); a6 = fmaf(d3.x, m1, a6);
            a11 = fmaf(d3.x, m0, a11); t0 = fmaf(d3.y, m12, t0); a2 = fmaf(d3.y, m6, a2); a6 = fmaf(d3.y, m2, a6);
            a12 = fmaf(d3.y, m0, a12); t0 = fmaf(d3.z, m13, t0); a1 = fmaf(d3.z, m7, a1); a3 = fmaf(d3.z, m4, a3);
            a4 = fmaf(d3.z, m3, a4); a7 = fmaf(d3.z, m1, a7); a13 = fmaf(d3.z, m0, a13); t0 = fmaf(d3.w, m14, t0);
            a1 = fmaf(d3.w, m8, a1); a2 = fmaf(d3.w, m7, a2); a3 = fmaf(d3.w, m5, a3); a5 = fmaf(d3.w, m3, a5);
            a7 = fmaf(d3.w, m2, a7); a8 = fmaf(d3.w, m1, a8); a14 = fmaf(d3.w, m0, a14); const float4 d4 = row.d(4); t0 = fmaf(d4.x, m15, t0);
            a2 = fmaf(d4.x, m8, a2); a3 = fmaf(d4.x, m6, a3); a6 = fmaf(d4.x, m3, a6); a8 = fmaf(d4.x, m2, a8);
            a15 = fmaf(d4.x, m0, a15); a3 = fmaf(d4.y, m7, a3); a7 = fmaf(d4.y, m3, a7); a3 = fmaf(d4.z, m8, a3);
            a8 = fmaf(d4.z, m3, a8);
            if (ql >= 4) {
              t0 = fmaf(d4.w, m16, t0); a1 = fmaf(d4.w, m9, a1); a4 = fmaf(d4.w, m4, a4); a9 = fmaf(d4.w, m1, a9);
              a16 = fmaf(d4.w, m0, a16); const float4 d5 = row.d(5); t0 = fmaf(d5.x, m17, t0); a1 = fmaf(d5.x, m10, a1);
              a2 = fmaf(d5.x, m9, a2); a4 = fmaf(d5.x, m5, a4); a5 = fmaf(d5.x, m4, a5); a9 = fmaf(d5.x, m2, a9);
              a10 = fmaf(d5.x, m1, a10); a17 = fmaf(d5.x, m0, a17); t0 = fmaf(d5.y, m18, t0); a1 = fmaf(d5.y, m11, a1);
              a2 = fmaf(d5.y, m10, a2); a4 = fmaf(d5.y, m6, a4); a5 = fmaf(d5.y, m5, a5); a6 = fmaf(d5.y, m4, a6);
              a10 = fmaf(d5.y, m2, a10); a11 = fmaf(d5.y, m1, a11); a18 = fmaf(d5.y, m0, a18); t0 = fmaf(d5.z, m19, t0);
              a1 = fmaf(d5.z, m12, a1); a2 = fmaf(d5.z, m11, a2); a5 = fmaf(d5.z, m6, a5); a6 = fmaf(d5.z, m5, a6);
              a11 = fmaf(d5.z, m2, a11); a12 = fmaf(d5.z, m1, a12); a19 = fmaf(d5.z, m0, a19); t0 = fmaf(d5.w, m20, t0);
              a2 = fmaf(d5.w, m12, a2); a6 = fmaf(d5.w, m6, a6); a12 = fmaf(d5.w, m2, a12); a20 = fmaf(d5.w, m0, a20);
              const float4 d6 = row.d(6); t0 = fmaf(d6.x, m21, t0); a1 = fmaf(d6.x, m13, a1); a3 = fmaf(d6.x, m9, a3);
              a4 = fmaf(d6.x, m7, a4); a7 = fmaf(d6.x, m4, a7); a9 = fmaf(d6.x, m3, a9); a13 = fmaf(d6.x, m1, a13);
              a21 = fmaf(d6.x, m0, a21); t0 = fmaf(d6.y, m22, t0); a1 = fmaf(d6.y, m14, a1); a2 = fmaf(d6.y, m13, a2);
              a3 = fmaf(d6.y, m10, a3); a4 = fmaf(d6.y, m8, a4); a5 = fmaf(d6.y, m7, a5); a7 = fmaf(d6.y, m5, a7);
              a8 = fmaf(d6.y, m4, a8); a10 = fmaf(d6.y, m3, a10); a13 = fmaf(d6.y, m2, a13); a14 = fmaf(d6.y, m1, a14);
              a22 = fmaf(d6.y, m0, a22); t0 = fmaf(d6.z, m23, t0); a1 = fmaf(d6.z, m15, a1); a2 = fmaf(d6.z, m14, a2);
              a3 = fmaf(d6.z, m11, a3); a5 = fmaf(d6.z, m8, a5); a6 = fmaf(d6.z, m7, a6); a7 = fmaf(d6.z, m6, a7);
              a8 = fmaf(d6.z, m5, a8); a11 = fmaf(d6.z, m3, a11); a14 = fmaf(d6.z, m2, a14); a15 = fmaf(d6.z, m1, a15);
              a23 = fmaf(d6.z, m0, a23); t0 = fmaf(d6.w, m24, t0); a2 = fmaf(d6.w, m15, a2); a3 = fmaf(d6.w, m12, a3);
              a6 = fmaf(d6.w, m8, a6); a8 = fmaf(d6.w, m6, a8); a12 = fmaf(d6.w, m3, a12); a15 = fmaf(d6.w, m2, a15);
              a24 = fmaf(d6.w, m0, a24); const float4 d7 = row.d(7); a3 = fmaf(d7.x, m13, a3); a7 = fmaf(d7.x, m7, a7);
              a13 = fmaf(d7.x, m3, a13); a3 = fmaf(d7.y, m14, a3); a7 = fmaf(d7.y, m8, a7); a8 = fmaf(d7.y, m7, a8);
              a14 = fmaf(d7.y, m3, a14); a3 = fmaf(d7.z, m15, a3); a8 = fmaf(d7.z, m8, a8); a15 = fmaf(d7.z, m3, a15);
            }
          }
        }
      }
    }
    __syncwarp();
    if (it.on_next)
      h_stage<0, 8, 0, 9>(db, P.D, P.dstr, it.cs, lane, h_words<4>(h_dterms(min(4, it.qmaxn))));
    h_commit();
    h_wait<2>();  // the operator's second half
    __syncwarp();
    a0 += t0;
    __syncwarp();
    if (it.on_next) {
    }
    h_commit();
    it.advance();
  }
  h_wait<0>();
  // the warps' sums, in shared memory
  float *const sum = (float *)(h_smem + w * 512) + lane;
  __syncwarp();
  sum[0] = a0; sum[32] = a1; sum[64] = a2; sum[96] = a3;
  sum[128] = a4; sum[160] = a5; sum[192] = a6; sum[224] = a7;
  sum[256] = a8; sum[288] = a9; sum[320] = a10; sum[352] = a11;
  sum[384] = a12; sum[416] = a13; sum[448] = a14; sum[480] = a15;
  sum[512] = a16; sum[544] = a17; sum[576] = a18; sum[608] = a19;
  sum[640] = a20; sum[672] = a21; sum[704] = a22; sum[736] = a23;
  sum[768] = a24;
  h_store<float, 25, 2048, false>(P, (float *)h_smem, 0, W);
}

int fmm_m2lh_f32_p4(const HParams<float> &P, cudaStream_t st) {
  if (P.p >= 0)
    if (int rc = h_launch(k_m2lh_f32_p4_0, P, 8192, 8, st)) return rc;
  return FMM_OK;
}
