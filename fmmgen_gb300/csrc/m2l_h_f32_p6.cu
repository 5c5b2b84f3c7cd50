// m2l_h_f32_p6.cu -- generated by fmmgen_gb300/gen_m2l_h.py; do not edit.
// M2L over harmonic coefficients in float, orders up to 6 (see m2l_h.cuh).
#include "m2l_h.cuh"

// outputs of degree 0..6, multipole degrees 0..6: 49 accumulators, 9 per-pair sums, 532 multiply-adds at order 6
__global__ void __launch_bounds__(256, 1) k_m2lh_f32_p6_0(const HParams<float> P) {
  extern __shared__ float4 h_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  float4 *const mb = h_smem + w * 960, *const db = mb + 416;
  const HF32Row<13, 17> row(mb, db, lane);
  HList it(P, lane, w, W);
  float a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0, a7 = 0, a8 = 0, a9 = 0, a10 = 0, a11 = 0, a12 = 0, a13 = 0, a14 = 0, a15 = 0, a16 = 0, a17 = 0, a18 = 0, a19 = 0, a20 = 0, a21 = 0, a22 = 0, a23 = 0, a24 = 0, a25 = 0, a26 = 0, a27 = 0, a28 = 0, a29 = 0, a30 = 0, a31 = 0, a32 = 0, a33 = 0, a34 = 0, a35 = 0, a36 = 0, a37 = 0, a38 = 0, a39 = 0, a40 = 0, a41 = 0, a42 = 0, a43 = 0, a44 = 0, a45 = 0, a46 = 0, a47 = 0, a48 = 0;
  if (it.begin(0)) {
    h_stage<0, 13, 0, 13>(mb, P.M, P.mstr, it.B, lane, h_words<4>(h_terms(min(6, it.qmax - 0))));
    h_stage<0, 8, 0, 17>(db, P.D, P.dstr, it.c, lane, h_words<4>(h_dterms(min(6, it.qmax))));
    h_commit();
    h_stage<8, 16, 0, 17>(db, P.D, P.dstr, it.c, lane, h_words<4>(h_dterms(min(6, it.qmax))));
    h_commit();
  }
  while (it.on_any) {
    it.look_ahead(0, fmm_wide_levels(6));
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
    const float4 mq7 = row.m(7);
    const float4 mq8 = row.m(8);
    const float4 mq9 = row.m(9);
    const float4 mq10 = row.m(10);
    const float4 mq11 = row.m(11);
    const float4 mq12 = row.m(12);
    float m0 = mq0.x, m1 = mq0.y, m2 = mq0.z, m3 = mq0.w, m4 = mq1.x, m5 = mq1.y, m6 = mq1.z, m7 = mq1.w, m8 = mq2.x, m9 = mq2.y, m10 = mq2.z, m11 = mq2.w, m12 = mq3.x, m13 = mq3.y, m14 = mq3.z, m15 = mq3.w, m16 = mq4.x, m17 = mq4.y, m18 = mq4.z, m19 = mq4.w, m20 = mq5.x, m21 = mq5.y, m22 = mq5.z, m23 = mq5.w, m24 = mq6.x, m25 = mq6.y, m26 = mq6.z, m27 = mq6.w, m28 = mq7.x, m29 = mq7.y, m30 = mq7.z, m31 = mq7.w, m32 = mq8.x, m33 = mq8.y, m34 = mq8.z, m35 = mq8.w, m36 = mq9.x, m37 = mq9.y, m38 = mq9.z, m39 = mq9.w, m40 = mq10.x, m41 = mq10.y, m42 = mq10.z, m43 = mq10.w, m44 = mq11.x, m45 = mq11.y, m46 = mq11.z, m47 = mq11.w, m48 = mq12.x;
    if (it.rescale) {
      const float s1 = h_exp2<float>(1 * it.dl);
      m1 *= s1; m2 *= s1; m3 *= s1;
      const float s2 = h_exp2<float>(2 * it.dl);
      m4 *= s2; m5 *= s2; m6 *= s2; m7 *= s2; m8 *= s2;
      const float s3 = h_exp2<float>(3 * it.dl);
      m9 *= s3; m10 *= s3; m11 *= s3; m12 *= s3; m13 *= s3; m14 *= s3; m15 *= s3;
      const float s4 = h_exp2<float>(4 * it.dl);
      m16 *= s4; m17 *= s4; m18 *= s4; m19 *= s4; m20 *= s4; m21 *= s4; m22 *= s4; m23 *= s4; m24 *= s4;
      const float s5 = h_exp2<float>(5 * it.dl);
      m25 *= s5; m26 *= s5; m27 *= s5; m28 *= s5; m29 *= s5; m30 *= s5; m31 *= s5; m32 *= s5; m33 *= s5; m34 *= s5; m35 *= s5;
      const float s6 = h_exp2<float>(6 * it.dl);
      m36 *= s6; m37 *= s6; m38 *= s6; m39 *= s6; m40 *= s6; m41 *= s6; m42 *= s6; m43 *= s6; m44 *= s6; m45 *= s6; m46 *= s6; m47 *= s6; m48 *= s6;
    }
    __syncwarp();
    if (it.on_next)
      h_stage<0, 13, 0, 13>(mb, P.M, P.mstr, it.Bs, lane, h_words<4>(h_terms(min(6, it.qmaxn - 0))));
    h_commit();
    float t0 = 0, t1 = 0, t2 = 0, t3 = 0, t4 = 0, t5 = 0, t6 = 0, t7 = 0, t8 = 0;
    if (ql >= 0) {
      const float4 d0 = row.d(0); t0 = fmaf(d0.x, m0, t0);
      if (ql >= 1) {
        t0 = fmaf(d0.y, m1, t0); t1 = fmaf(d0.y, m0, t1); t0 = fmaf(d0.z, m2, t0); t2 = fmaf(d0.z, m0, t2);
        t0 = fmaf(d0.w, m3, t0); t3 = fmaf(d0.w, m0, t3);
        if (ql >= 2) {
          const float4 d1 = row.d(1); t0 = fmaf(d1.x, m4, t0); t1 = fmaf(d1.x, m1, t1); t4 = fmaf(d1.x, m0, t4);
          t0 = fmaf(d1.y, m5, t0); t1 = fmaf(d1.y, m2, t1); t2 = fmaf(d1.y, m1, t2); t5 = fmaf(d1.y, m0, t5);
          t0 = fmaf(d1.z, m6, t0); t2 = fmaf(d1.z, m2, t2); t6 = fmaf(d1.z, m0, t6); t0 = fmaf(d1.w, m7, t0);
          t1 = fmaf(d1.w, m3, t1); t3 = fmaf(d1.w, m1, t3); t7 = fmaf(d1.w, m0, t7); const float4 d2 = row.d(2); t0 = fmaf(d2.x, m8, t0);
          t2 = fmaf(d2.x, m3, t2); t3 = fmaf(d2.x, m2, t3); t8 = fmaf(d2.x, m0, t8); t3 = fmaf(d2.y, m3, t3);
          if (ql >= 3) {
            t0 = fmaf(d2.z, m9, t0); t1 = fmaf(d2.z, m4, t1); t4 = fmaf(d2.z, m1, t4); a9 = fmaf(d2.z, m0, a9);
            t0 = fmaf(d2.w, m10, t0); t1 = fmaf(d2.w, m5, t1); t2 = fmaf(d2.w, m4, t2); t4 = fmaf(d2.w, m2, t4);
            t5 = fmaf(d2.w, m1, t5); a10 = fmaf(d2.w, m0, a10); const float4 d3 = row.d(3); t0 = fmaf(d3.x, m11, t0);
            t1 = fmaf(d3.x, m6, t1); t2 = fmaf(d3.x, m5, t2); t5 = fmaf(d3.x, m2, t5); t6 = fmaf(d3.x, m1, t6);
            a11 = fmaf(d3.x, m0, a11); t0 = fmaf(d3.y, m12, t0); t2 = fmaf(d3.y, m6, t2); t6 = fmaf(d3.y, m2, t6);
            a12 = fmaf(d3.y, m0, a12); t0 = fmaf(d3.z, m13, t0); t1 = fmaf(d3.z, m7, t1); t3 = fmaf(d3.z, m4, t3);
            t4 = fmaf(d3.z, m3, t4); t7 = fmaf(d3.z, m1, t7); a13 = fmaf(d3.z, m0, a13); t0 = fmaf(d3.w, m14, t0);
            t1 = fmaf(d3.w, m8, t1); t2 = fmaf(d3.w, m7, t2); t3 = fmaf(d3.w, m5, t3); t5 = fmaf(d3.w, m3, t5);
            t7 = fmaf(d3.w, m2, t7); t8 = fmaf(d3.w, m1, t8); a14 = fmaf(d3.w, m0, a14); const float4 d4 = row.d(4); t0 = fmaf(d4.x, m15, t0);
            t2 = fmaf(d4.x, m8, t2); t3 = fmaf(d4.x, m6, t3); t6 = fmaf(d4.x, m3, t6); t8 = fmaf(d4.x, m2, t8);
            a15 = fmaf(d4.x, m0, a15); t3 = fmaf(d4.y, m7, t3); t7 = fmaf(d4.y, m3, t7); t3 = fmaf(d4.z, m8, t3);
            t8 = fmaf(d4.z, m3, t8);
            if (ql >= 4) {
              t0 = fmaf(d4.w, m16, t0); t1 = fmaf(d4.w, m9, t1); t4 = fmaf(d4.w, m4, t4); a9 = fmaf(d4.w, m1, a9);
              a16 = fmaf(d4.w, m0, a16); const float4 d5 = row.d(5); t0 = fmaf(d5.x, m17, t0); t1 = fmaf(d5.x, m10, t1);
              t2 = fmaf(d5.x, m9, t2); t4 = fmaf(d5.x, m5, t4); t5 = fmaf(d5.x, m4, t5); a9 = fmaf(d5.x, m2, a9);
              a10 = fmaf(d5.x, m1, a10); a17 = fmaf(d5.x, m0, a17); t0 = fmaf(d5.y, m18, t0); t1 = fmaf(d5.y, m11, t1);
              t2 = fmaf(d5.y, m10, t2); t4 = fmaf(d5.y, m6, t4); t5 = fmaf(d5.y, m5, t5); t6 = fmaf(d5.y, m4, t6);
              a10 = fmaf(d5.y, m2, a10); a11 = fmaf(d5.y, m1, a11); a18 = fmaf(d5.y, m0, a18); t0 = fmaf(d5.z, m19, t0);
              t1 = fmaf(d5.z, m12, t1); t2 = fmaf(d5.z, m11, t2); t5 = fmaf(d5.z, m6, t5); t6 = fmaf(d5.z, m5, t6);
              a11 = fmaf(d5.z, m2, a11); a12 = fmaf(d5.z, m1, a12); a19 = fmaf(d5.z, m0, a19); t0 = fmaf(d5.w, m20, t0);
              t2 = fmaf(d5.w, m12, t2); t6 = fmaf(d5.w, m6, t6); a12 = fmaf(d5.w, m2, a12); a20 = fmaf(d5.w, m0, a20);
              const float4 d6 = row.d(6); t0 = fmaf(d6.x, m21, t0); t1 = fmaf(d6.x, m13, t1); t3 = fmaf(d6.x, m9, t3);
              t4 = fmaf(d6.x, m7, t4); t7 = fmaf(d6.x, m4, t7); a9 = fmaf(d6.x, m3, a9); a13 = fmaf(d6.x, m1, a13);
              a21 = fmaf(d6.x, m0, a21); t0 = fmaf(d6.y, m22, t0); t1 = fmaf(d6.y, m14, t1); t2 = fmaf(d6.y, m13, t2);
              t3 = fmaf(d6.y, m10, t3); t4 = fmaf(d6.y, m8, t4); t5 = fmaf(d6.y, m7, t5); t7 = fmaf(d6.y, m5, t7);
              t8 = fmaf(d6.y, m4, t8); a10 = fmaf(d6.y, m3, a10); a13 = fmaf(d6.y, m2, a13); a14 = fmaf(d6.y, m1, a14);
              a22 = fmaf(d6.y, m0, a22); t0 = fmaf(d6.z, m23, t0); t1 = fmaf(d6.z, m15, t1); t2 = fmaf(d6.z, m14, t2);
              t3 = fmaf(d6.z, m11, t3); t5 = fmaf(d6.z, m8, t5); t6 = fmaf(d6.z, m7, t6); t7 = fmaf(d6.z, m6, t7);
              t8 = fmaf(d6.z, m5, t8); a11 = fmaf(d6.z, m3, a11); a14 = fmaf(d6.z, m2, a14); a15 = fmaf(d6.z, m1, a15);
              a23 = fmaf(d6.z, m0, a23); t0 = fmaf(d6.w, m24, t0); t2 = fmaf(d6.w, m15, t2); t3 = fmaf(d6.w, m12, t3);
              t6 = fmaf(d6.w, m8, t6); t8 = fmaf(d6.w, m6, t8); a12 = fmaf(d6.w, m3, a12); a15 = fmaf(d6.w, m2, a15);
              a24 = fmaf(d6.w, m0, a24); const float4 d7 = row.d(7); t3 = fmaf(d7.x, m13, t3); t7 = fmaf(d7.x, m7, t7);
              a13 = fmaf(d7.x, m3, a13); t3 = fmaf(d7.y, m14, t3); t7 = fmaf(d7.y, m8, t7); t8 = fmaf(d7.y, m7, t8);
              a14 = fmaf(d7.y, m3, a14); t3 = fmaf(d7.z, m15, t3); t8 = fmaf(d7.z, m8, t8); a15 = fmaf(d7.z, m3, a15);
              if (ql >= 5) {
                t0 = fmaf(d7.w, m25, t0); t1 = fmaf(d7.w, m16, t1); t4 = fmaf(d7.w, m9, t4); a9 = fmaf(d7.w, m4, a9);
                a16 = fmaf(d7.w, m1, a16); a25 = fmaf(d7.w, m0, a25);
              }
            }
          }
        }
      }
    }
    __syncwarp();
    if (it.on_next)
      h_stage<0, 8, 0, 17>(db, P.D, P.dstr, it.cs, lane, h_words<4>(h_dterms(min(6, it.qmaxn))));
    h_commit();
    h_wait<2>();  // the operator's second half
    __syncwarp();
    if (ql >= 5) {
      const float4 d8 = row.d(8); t0 = fmaf(d8.x, m26, t0); t1 = fmaf(d8.x, m17, t1); t2 = fmaf(d8.x, m16, t2);
      t4 = fmaf(d8.x, m10, t4); t5 = fmaf(d8.x, m9, t5); a9 = fmaf(d8.x, m5, a9); a10 = fmaf(d8.x, m4, a10);
      a16 = fmaf(d8.x, m2, a16); a17 = fmaf(d8.x, m1, a17); a26 = fmaf(d8.x, m0, a26); t0 = fmaf(d8.y, m27, t0);
      t1 = fmaf(d8.y, m18, t1); t2 = fmaf(d8.y, m17, t2); t4 = fmaf(d8.y, m11, t4); t5 = fmaf(d8.y, m10, t5);
      t6 = fmaf(d8.y, m9, t6); a9 = fmaf(d8.y, m6, a9); a10 = fmaf(d8.y, m5, a10); a11 = fmaf(d8.y, m4, a11);
      a17 = fmaf(d8.y, m2, a17); a18 = fmaf(d8.y, m1, a18); a27 = fmaf(d8.y, m0, a27); t0 = fmaf(d8.z, m28, t0);
      t1 = fmaf(d8.z, m19, t1); t2 = fmaf(d8.z, m18, t2); t4 = fmaf(d8.z, m12, t4); t5 = fmaf(d8.z, m11, t5);
      t6 = fmaf(d8.z, m10, t6); a10 = fmaf(d8.z, m6, a10); a11 = fmaf(d8.z, m5, a11); a12 = fmaf(d8.z, m4, a12);
      a18 = fmaf(d8.z, m2, a18); a19 = fmaf(d8.z, m1, a19); a28 = fmaf(d8.z, m0, a28); t0 = fmaf(d8.w, m29, t0);
      t1 = fmaf(d8.w, m20, t1); t2 = fmaf(d8.w, m19, t2); t5 = fmaf(d8.w, m12, t5); t6 = fmaf(d8.w, m11, t6);
      a11 = fmaf(d8.w, m6, a11); a12 = fmaf(d8.w, m5, a12); a19 = fmaf(d8.w, m2, a19); a20 = fmaf(d8.w, m1, a20);
      a29 = fmaf(d8.w, m0, a29); const float4 d9 = row.d(9); t0 = fmaf(d9.x, m30, t0); t2 = fmaf(d9.x, m20, t2);
      t6 = fmaf(d9.x, m12, t6); a12 = fmaf(d9.x, m6, a12); a20 = fmaf(d9.x, m2, a20); a30 = fmaf(d9.x, m0, a30);
      t0 = fmaf(d9.y, m31, t0); t1 = fmaf(d9.y, m21, t1); t3 = fmaf(d9.y, m16, t3); t4 = fmaf(d9.y, m13, t4);
      t7 = fmaf(d9.y, m9, t7); a9 = fmaf(d9.y, m7, a9); a13 = fmaf(d9.y, m4, a13); a16 = fmaf(d9.y, m3, a16);
      a21 = fmaf(d9.y, m1, a21); a31 = fmaf(d9.y, m0, a31); t0 = fmaf(d9.z, m32, t0); t1 = fmaf(d9.z, m22, t1);
      t2 = fmaf(d9.z, m21, t2); t3 = fmaf(d9.z, m17, t3); t4 = fmaf(d9.z, m14, t4); t5 = fmaf(d9.z, m13, t5);
      t7 = fmaf(d9.z, m10, t7); t8 = fmaf(d9.z, m9, t8); a9 = fmaf(d9.z, m8, a9); a10 = fmaf(d9.z, m7, a10);
      a13 = fmaf(d9.z, m5, a13); a14 = fmaf(d9.z, m4, a14); a17 = fmaf(d9.z, m3, a17); a21 = fmaf(d9.z, m2, a21);
      a22 = fmaf(d9.z, m1, a22); a32 = fmaf(d9.z, m0, a32); t0 = fmaf(d9.w, m33, t0); t1 = fmaf(d9.w, m23, t1);
      t2 = fmaf(d9.w, m22, t2); t3 = fmaf(d9.w, m18, t3); t4 = fmaf(d9.w, m15, t4); t5 = fmaf(d9.w, m14, t5);
      t6 = fmaf(d9.w, m13, t6); t7 = fmaf(d9.w, m11, t7); t8 = fmaf(d9.w, m10, t8); a10 = fmaf(d9.w, m8, a10);
      a11 = fmaf(d9.w, m7, a11); a13 = fmaf(d9.w, m6, a13); a14 = fmaf(d9.w, m5, a14); a15 = fmaf(d9.w, m4, a15);
      a18 = fmaf(d9.w, m3, a18); a22 = fmaf(d9.w, m2, a22); a23 = fmaf(d9.w, m1, a23); a33 = fmaf(d9.w, m0, a33);
      const float4 d10 = row.d(10); t0 = fmaf(d10.x, m34, t0); t1 = fmaf(d10.x, m24, t1); t2 = fmaf(d10.x, m23, t2);
      t3 = fmaf(d10.x, m19, t3); t5 = fmaf(d10.x, m15, t5); t6 = fmaf(d10.x, m14, t6); t7 = fmaf(d10.x, m12, t7);
      t8 = fmaf(d10.x, m11, t8); a11 = fmaf(d10.x, m8, a11); a12 = fmaf(d10.x, m7, a12); a14 = fmaf(d10.x, m6, a14);
      a15 = fmaf(d10.x, m5, a15); a19 = fmaf(d10.x, m3, a19); a23 = fmaf(d10.x, m2, a23); a24 = fmaf(d10.x, m1, a24);
      a34 = fmaf(d10.x, m0, a34); t0 = fmaf(d10.y, m35, t0); t2 = fmaf(d10.y, m24, t2); t3 = fmaf(d10.y, m20, t3);
      t6 = fmaf(d10.y, m15, t6); t8 = fmaf(d10.y, m12, t8); a12 = fmaf(d10.y, m8, a12); a15 = fmaf(d10.y, m6, a15);
      a20 = fmaf(d10.y, m3, a20); a24 = fmaf(d10.y, m2, a24); a35 = fmaf(d10.y, m0, a35); t3 = fmaf(d10.z, m21, t3);
      t7 = fmaf(d10.z, m13, t7); a13 = fmaf(d10.z, m7, a13); a21 = fmaf(d10.z, m3, a21); t3 = fmaf(d10.w, m22, t3);
      t7 = fmaf(d10.w, m14, t7); t8 = fmaf(d10.w, m13, t8); a13 = fmaf(d10.w, m8, a13); a14 = fmaf(d10.w, m7, a14);
      a22 = fmaf(d10.w, m3, a22); const float4 d11 = row.d(11); t3 = fmaf(d11.x, m23, t3); t7 = fmaf(d11.x, m15, t7);
      t8 = fmaf(d11.x, m14, t8); a14 = fmaf(d11.x, m8, a14); a15 = fmaf(d11.x, m7, a15); a23 = fmaf(d11.x, m3, a23);
      t3 = fmaf(d11.y, m24, t3); t8 = fmaf(d11.y, m15, t8); a15 = fmaf(d11.y, m8, a15); a24 = fmaf(d11.y, m3, a24);
      if (ql >= 6) {
        t0 = fmaf(d11.z, m36, t0); t1 = fmaf(d11.z, m25, t1); t4 = fmaf(d11.z, m16, t4); a9 = fmaf(d11.z, m9, a9);
        a16 = fmaf(d11.z, m4, a16); a25 = fmaf(d11.z, m1, a25); a36 = fmaf(d11.z, m0, a36); t0 = fmaf(d11.w, m37, t0);
        t1 = fmaf(d11.w, m26, t1); t2 = fmaf(d11.w, m25, t2); t4 = fmaf(d11.w, m17, t4); t5 = fmaf(d11.w, m16, t5);
        a9 = fmaf(d11.w, m10, a9); a10 = fmaf(d11.w, m9, a10); a16 = fmaf(d11.w, m5, a16); a17 = fmaf(d11.w, m4, a17);
        a25 = fmaf(d11.w, m2, a25); a26 = fmaf(d11.w, m1, a26); a37 = fmaf(d11.w, m0, a37); const float4 d12 = row.d(12); t0 = fmaf(d12.x, m38, t0);
        t1 = fmaf(d12.x, m27, t1); t2 = fmaf(d12.x, m26, t2); t4 = fmaf(d12.x, m18, t4); t5 = fmaf(d12.x, m17, t5);
        t6 = fmaf(d12.x, m16, t6); a9 = fmaf(d12.x, m11, a9); a10 = fmaf(d12.x, m10, a10); a11 = fmaf(d12.x, m9, a11);
        a16 = fmaf(d12.x, m6, a16); a17 = fmaf(d12.x, m5, a17); a18 = fmaf(d12.x, m4, a18); a26 = fmaf(d12.x, m2, a26);
        a27 = fmaf(d12.x, m1, a27); a38 = fmaf(d12.x, m0, a38); t0 = fmaf(d12.y, m39, t0); t1 = fmaf(d12.y, m28, t1);
        t2 = fmaf(d12.y, m27, t2); t4 = fmaf(d12.y, m19, t4); t5 = fmaf(d12.y, m18, t5); t6 = fmaf(d12.y, m17, t6);
        a9 = fmaf(d12.y, m12, a9); a10 = fmaf(d12.y, m11, a10); a11 = fmaf(d12.y, m10, a11); a12 = fmaf(d12.y, m9, a12);
        a17 = fmaf(d12.y, m6, a17); a18 = fmaf(d12.y, m5, a18); a19 = fmaf(d12.y, m4, a19); a27 = fmaf(d12.y, m2, a27);
        a28 = fmaf(d12.y, m1, a28); a39 = fmaf(d12.y, m0, a39); t0 = fmaf(d12.z, m40, t0); t1 = fmaf(d12.z, m29, t1);
        t2 = fmaf(d12.z, m28, t2); t4 = fmaf(d12.z, m20, t4); t5 = fmaf(d12.z, m19, t5); t6 = fmaf(d12.z, m18, t6);
        a10 = fmaf(d12.z, m12, a10); a11 = fmaf(d12.z, m11, a11); a12 = fmaf(d12.z, m10, a12); a18 = fmaf(d12.z, m6, a18);
        a19 = fmaf(d12.z, m5, a19); a20 = fmaf(d12.z, m4, a20); a28 = fmaf(d12.z, m2, a28); a29 = fmaf(d12.z, m1, a29);
        a40 = fmaf(d12.z, m0, a40); t0 = fmaf(d12.w, m41, t0); t1 = fmaf(d12.w, m30, t1); t2 = fmaf(d12.w, m29, t2);
        t5 = fmaf(d12.w, m20, t5); t6 = fmaf(d12.w, m19, t6); a11 = fmaf(d12.w, m12, a11); a12 = fmaf(d12.w, m11, a12);
        a19 = fmaf(d12.w, m6, a19); a20 = fmaf(d12.w, m5, a20); a29 = fmaf(d12.w, m2, a29); a30 = fmaf(d12.w, m1, a30);
        a41 = fmaf(d12.w, m0, a41); const float4 d13 = row.d(13); t0 = fmaf(d13.x, m42, t0); t2 = fmaf(d13.x, m30, t2);
        t6 = fmaf(d13.x, m20, t6); a12 = fmaf(d13.x, m12, a12); a20 = fmaf(d13.x, m6, a20); a30 = fmaf(d13.x, m2, a30);
        a42 = fmaf(d13.x, m0, a42); t0 = fmaf(d13.y, m43, t0); t1 = fmaf(d13.y, m31, t1); t3 = fmaf(d13.y, m25, t3);
        t4 = fmaf(d13.y, m21, t4); t7 = fmaf(d13.y, m16, t7); a9 = fmaf(d13.y, m13, a9); a13 = fmaf(d13.y, m9, a13);
        a16 = fmaf(d13.y, m7, a16); a21 = fmaf(d13.y, m4, a21); a25 = fmaf(d13.y, m3, a25); a31 = fmaf(d13.y, m1, a31);
        a43 = fmaf(d13.y, m0, a43); t0 = fmaf(d13.z, m44, t0); t1 = fmaf(d13.z, m32, t1); t2 = fmaf(d13.z, m31, t2);
        t3 = fmaf(d13.z, m26, t3); t4 = fmaf(d13.z, m22, t4); t5 = fmaf(d13.z, m21, t5); t7 = fmaf(d13.z, m17, t7);
        t8 = fmaf(d13.z, m16, t8); a9 = fmaf(d13.z, m14, a9); a10 = fmaf(d13.z, m13, a10); a13 = fmaf(d13.z, m10, a13);
        a14 = fmaf(d13.z, m9, a14); a16 = fmaf(d13.z, m8, a16); a17 = fmaf(d13.z, m7, a17); a21 = fmaf(d13.z, m5, a21);
        a22 = fmaf(d13.z, m4, a22); a26 = fmaf(d13.z, m3, a26); a31 = fmaf(d13.z, m2, a31); a32 = fmaf(d13.z, m1, a32);
        a44 = fmaf(d13.z, m0, a44); t0 = fmaf(d13.w, m45, t0); t1 = fmaf(d13.w, m33, t1); t2 = fmaf(d13.w, m32, t2);
        t3 = fmaf(d13.w, m27, t3); t4 = fmaf(d13.w, m23, t4); t5 = fmaf(d13.w, m22, t5); t6 = fmaf(d13.w, m21, t6);
        t7 = fmaf(d13.w, m18, t7); t8 = fmaf(d13.w, m17, t8); a9 = fmaf(d13.w, m15, a9); a10 = fmaf(d13.w, m14, a10);
        a11 = fmaf(d13.w, m13, a11); a13 = fmaf(d13.w, m11, a13); a14 = fmaf(d13.w, m10, a14); a15 = fmaf(d13.w, m9, a15);
        a17 = fmaf(d13.w, m8, a17); a18 = fmaf(d13.w, m7, a18); a21 = fmaf(d13.w, m6, a21); a22 = fmaf(d13.w, m5, a22);
        a23 = fmaf(d13.w, m4, a23); a27 = fmaf(d13.w, m3, a27); a32 = fmaf(d13.w, m2, a32); a33 = fmaf(d13.w, m1, a33);
        a45 = fmaf(d13.w, m0, a45); const float4 d14 = row.d(14); t0 = fmaf(d14.x, m46, t0); t1 = fmaf(d14.x, m34, t1);
        t2 = fmaf(d14.x, m33, t2); t3 = fmaf(d14.x, m28, t3); t4 = fmaf(d14.x, m24, t4); t5 = fmaf(d14.x, m23, t5);
        t6 = fmaf(d14.x, m22, t6); t7 = fmaf(d14.x, m19, t7); t8 = fmaf(d14.x, m18, t8); a10 = fmaf(d14.x, m15, a10);
        a11 = fmaf(d14.x, m14, a11); a12 = fmaf(d14.x, m13, a12); a13 = fmaf(d14.x, m12, a13); a14 = fmaf(d14.x, m11, a14);
        a15 = fmaf(d14.x, m10, a15); a18 = fmaf(d14.x, m8, a18); a19 = fmaf(d14.x, m7, a19); a22 = fmaf(d14.x, m6, a22);
        a23 = fmaf(d14.x, m5, a23); a24 = fmaf(d14.x, m4, a24); a28 = fmaf(d14.x, m3, a28); a33 = fmaf(d14.x, m2, a33);
        a34 = fmaf(d14.x, m1, a34); a46 = fmaf(d14.x, m0, a46); t0 = fmaf(d14.y, m47, t0); t1 = fmaf(d14.y, m35, t1);
        t2 = fmaf(d14.y, m34, t2); t3 = fmaf(d14.y, m29, t3); t5 = fmaf(d14.y, m24, t5); t6 = fmaf(d14.y, m23, t6);
        t7 = fmaf(d14.y, m20, t7); t8 = fmaf(d14.y, m19, t8); a11 = fmaf(d14.y, m15, a11); a12 = fmaf(d14.y, m14, a12);
        a14 = fmaf(d14.y, m12, a14); a15 = fmaf(d14.y, m11, a15); a19 = fmaf(d14.y, m8, a19); a20 = fmaf(d14.y, m7, a20);
        a23 = fmaf(d14.y, m6, a23); a24 = fmaf(d14.y, m5, a24); a29 = fmaf(d14.y, m3, a29); a34 = fmaf(d14.y, m2, a34);
        a35 = fmaf(d14.y, m1, a35); a47 = fmaf(d14.y, m0, a47); t0 = fmaf(d14.z, m48, t0); t2 = fmaf(d14.z, m35, t2);
        t3 = fmaf(d14.z, m30, t3); t6 = fmaf(d14.z, m24, t6); t8 = fmaf(d14.z, m20, t8); a12 = fmaf(d14.z, m15, a12);
        a15 = fmaf(d14.z, m12, a15); a20 = fmaf(d14.z, m8, a20); a24 = fmaf(d14.z, m6, a24); a30 = fmaf(d14.z, m3, a30);
        a35 = fmaf(d14.z, m2, a35); a48 = fmaf(d14.z, m0, a48); t3 = fmaf(d14.w, m31, t3); t7 = fmaf(d14.w, m21, t7);
        a13 = fmaf(d14.w, m13, a13); a21 = fmaf(d14.w, m7, a21); a31 = fmaf(d14.w, m3, a31); const float4 d15 = row.d(15); t3 = fmaf(d15.x, m32, t3);
        t7 = fmaf(d15.x, m22, t7); t8 = fmaf(d15.x, m21, t8); a13 = fmaf(d15.x, m14, a13); a14 = fmaf(d15.x, m13, a14);
        a21 = fmaf(d15.x, m8, a21); a22 = fmaf(d15.x, m7, a22); a32 = fmaf(d15.x, m3, a32); t3 = fmaf(d15.y, m33, t3);
        t7 = fmaf(d15.y, m23, t7); t8 = fmaf(d15.y, m22, t8); a13 = fmaf(d15.y, m15, a13); a14 = fmaf(d15.y, m14, a14);
        a15 = fmaf(d15.y, m13, a15); a22 = fmaf(d15.y, m8, a22); a23 = fmaf(d15.y, m7, a23); a33 = fmaf(d15.y, m3, a33);
        t3 = fmaf(d15.z, m34, t3); t7 = fmaf(d15.z, m24, t7); t8 = fmaf(d15.z, m23, t8); a14 = fmaf(d15.z, m15, a14);
        a15 = fmaf(d15.z, m14, a15); a23 = fmaf(d15.z, m8, a23); a24 = fmaf(d15.z, m7, a24); a34 = fmaf(d15.z, m3, a34);
        t3 = fmaf(d15.w, m35, t3); t8 = fmaf(d15.w, m24, t8); a15 = fmaf(d15.w, m15, a15); a24 = fmaf(d15.w, m8, a24);
        a35 = fmaf(d15.w, m3, a35);
      }
    }
    a0 += t0; a1 += t1; a2 += t2; a3 += t3; a4 += t4; a5 += t5; a6 += t6; a7 += t7; a8 += t8;
    __syncwarp();
    if (it.on_next) {
      h_stage<8, 16, 0, 17>(db, P.D, P.dstr, it.cs, lane, h_words<4>(h_dterms(min(6, it.qmaxn))));
    }
    h_commit();
    it.advance();
  }
  h_wait<0>();
  // the warps' sums, in shared memory
  float *const sum = (float *)(h_smem + w * 960) + lane;
  __syncwarp();
  sum[0] = a0; sum[32] = a1; sum[64] = a2; sum[96] = a3;
  sum[128] = a4; sum[160] = a5; sum[192] = a6; sum[224] = a7;
  sum[256] = a8; sum[288] = a9; sum[320] = a10; sum[352] = a11;
  sum[384] = a12; sum[416] = a13; sum[448] = a14; sum[480] = a15;
  sum[512] = a16; sum[544] = a17; sum[576] = a18; sum[608] = a19;
  sum[640] = a20; sum[672] = a21; sum[704] = a22; sum[736] = a23;
  sum[768] = a24; sum[800] = a25; sum[832] = a26; sum[864] = a27;
  sum[896] = a28; sum[928] = a29; sum[960] = a30; sum[992] = a31;
  sum[1024] = a32; sum[1056] = a33; sum[1088] = a34; sum[1120] = a35;
  sum[1152] = a36; sum[1184] = a37; sum[1216] = a38; sum[1248] = a39;
  sum[1280] = a40; sum[1312] = a41; sum[1344] = a42; sum[1376] = a43;
  sum[1408] = a44; sum[1440] = a45; sum[1472] = a46; sum[1504] = a47;
  sum[1536] = a48;
  h_store<float, 49, 3840, false>(P, (float *)h_smem, 0, W);
}

int fmm_m2lh_f32_p6(const HParams<float> &P, cudaStream_t st) {
  if (P.p >= 0)
    if (int rc = h_launch(k_m2lh_f32_p6_0, P, 15360, 8, st)) return rc;
  return FMM_OK;
}
