// m2l_h_f64_p6.cu -- generated by fmmgen_gb300/gen_m2l_h.py; do not edit.
// M2L over harmonic coefficients in double, orders up to 6 (see m2l_h.cuh).
#include "m2l_h.cuh"

// outputs of degree 0..6, multipole degrees 0..6: 49 accumulators, 9 per-pair sums, 532 multiply-adds at order 6
__global__ void __launch_bounds__(256, 1) k_m2lh_f64_p6_0(const HParams<double> P) {
  extern __shared__ float4 h_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  float4 *const mb = h_smem + w * 1344, *const db = mb + 800;
  const HF64Row<25, 17> row(mb, db, lane);
  HList it(P, lane, w, W);
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0, a7 = 0, a8 = 0, a9 = 0, a10 = 0, a11 = 0, a12 = 0, a13 = 0, a14 = 0, a15 = 0, a16 = 0, a17 = 0, a18 = 0, a19 = 0, a20 = 0, a21 = 0, a22 = 0, a23 = 0, a24 = 0, a25 = 0, a26 = 0, a27 = 0, a28 = 0, a29 = 0, a30 = 0, a31 = 0, a32 = 0, a33 = 0, a34 = 0, a35 = 0, a36 = 0, a37 = 0, a38 = 0, a39 = 0, a40 = 0, a41 = 0, a42 = 0, a43 = 0, a44 = 0, a45 = 0, a46 = 0, a47 = 0, a48 = 0;
  if (it.begin(0)) {
    h_stage<0, 25, 0, 25>(mb, P.M, P.mstr, it.B, lane, h_words<8>(h_terms(min(6, it.qmax - 0))));
    h_stage<0, 16, 0, 17>(db, P.D, P.dstr, it.c, lane, h_words<8>(h_dterms(min(6, it.qmax))));
    h_commit();

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
      row.scale(25, 36, h_exp2<double>(5 * it.dl));
      row.scale(36, 49, h_exp2<double>(6 * it.dl));
    }
    __syncwarp();
    double t0 = 0, t1 = 0, t2 = 0, t3 = 0, t4 = 0, t5 = 0, t6 = 0, t7 = 0, t8 = 0;
    if (ql >= 0) {
      const double d0 = row.d(0); row.fma<0>(t0, d0);
      if (ql >= 1) {
        const double d1 = row.d(1); row.fma<1>(t0, d1); row.fma<0>(t1, d1); const double d2 = row.d(2); row.fma<2>(t0, d2);
        row.fma<0>(t2, d2); const double d3 = row.d(3); row.fma<3>(t0, d3); row.fma<0>(t3, d3);
        if (ql >= 2) {
          const double d4 = row.d(4); row.fma<4>(t0, d4); row.fma<1>(t1, d4); row.fma<0>(t4, d4);
          const double d5 = row.d(5); row.fma<5>(t0, d5); row.fma<2>(t1, d5); row.fma<1>(t2, d5);
          row.fma<0>(t5, d5); const double d6 = row.d(6); row.fma<6>(t0, d6); row.fma<2>(t2, d6);
          row.fma<0>(t6, d6); const double d7 = row.d(7); row.fma<7>(t0, d7); row.fma<3>(t1, d7);
          row.fma<1>(t3, d7); row.fma<0>(t7, d7); const double d8 = row.d(8); row.fma<8>(t0, d8);
          row.fma<3>(t2, d8); row.fma<2>(t3, d8); row.fma<0>(t8, d8); const double d9 = row.d(9); row.fma<3>(t3, d9);
          if (ql >= 3) {
            const double d10 = row.d(10); row.fma<9>(t0, d10); row.fma<4>(t1, d10); row.fma<1>(t4, d10);
            row.fma<0>(a9, d10); const double d11 = row.d(11); row.fma<10>(t0, d11); row.fma<5>(t1, d11);
            row.fma<4>(t2, d11); row.fma<2>(t4, d11); row.fma<1>(t5, d11); row.fma<0>(a10, d11);
            const double d12 = row.d(12); row.fma<11>(t0, d12); row.fma<6>(t1, d12); row.fma<5>(t2, d12);
            row.fma<2>(t5, d12); row.fma<1>(t6, d12); row.fma<0>(a11, d12); const double d13 = row.d(13); row.fma<12>(t0, d13);
            row.fma<6>(t2, d13); row.fma<2>(t6, d13); row.fma<0>(a12, d13); const double d14 = row.d(14); row.fma<13>(t0, d14);
            row.fma<7>(t1, d14); row.fma<4>(t3, d14); row.fma<3>(t4, d14); row.fma<1>(t7, d14);
            row.fma<0>(a13, d14); const double d15 = row.d(15); row.fma<14>(t0, d15); row.fma<8>(t1, d15);
            row.fma<7>(t2, d15); row.fma<5>(t3, d15); row.fma<3>(t5, d15); row.fma<2>(t7, d15);
            row.fma<1>(t8, d15); row.fma<0>(a14, d15); const double d16 = row.d(16); row.fma<15>(t0, d16);
            row.fma<8>(t2, d16); row.fma<6>(t3, d16); row.fma<3>(t6, d16); row.fma<2>(t8, d16);
            row.fma<0>(a15, d16); const double d17 = row.d(17); row.fma<7>(t3, d17); row.fma<3>(t7, d17);
            const double d18 = row.d(18); row.fma<8>(t3, d18); row.fma<3>(t8, d18);
            if (ql >= 4) {
              const double d19 = row.d(19); row.fma<16>(t0, d19); row.fma<9>(t1, d19); row.fma<4>(t4, d19);
              row.fma<1>(a9, d19); row.fma<0>(a16, d19); const double d20 = row.d(20); row.fma<17>(t0, d20);
              row.fma<10>(t1, d20); row.fma<9>(t2, d20); row.fma<5>(t4, d20); row.fma<4>(t5, d20);
              row.fma<2>(a9, d20); row.fma<1>(a10, d20); row.fma<0>(a17, d20); const double d21 = row.d(21); row.fma<18>(t0, d21);
              row.fma<11>(t1, d21); row.fma<10>(t2, d21); row.fma<6>(t4, d21); row.fma<5>(t5, d21);
              row.fma<4>(t6, d21); row.fma<2>(a10, d21); row.fma<1>(a11, d21); row.fma<0>(a18, d21);
              const double d22 = row.d(22); row.fma<19>(t0, d22); row.fma<12>(t1, d22); row.fma<11>(t2, d22);
              row.fma<6>(t5, d22); row.fma<5>(t6, d22); row.fma<2>(a11, d22); row.fma<1>(a12, d22);
              row.fma<0>(a19, d22); const double d23 = row.d(23); row.fma<20>(t0, d23); row.fma<12>(t2, d23);
              row.fma<6>(t6, d23); row.fma<2>(a12, d23); row.fma<0>(a20, d23); const double d24 = row.d(24); row.fma<21>(t0, d24);
              row.fma<13>(t1, d24); row.fma<9>(t3, d24); row.fma<7>(t4, d24); row.fma<4>(t7, d24);
              row.fma<3>(a9, d24); row.fma<1>(a13, d24); row.fma<0>(a21, d24); const double d25 = row.d(25); row.fma<22>(t0, d25);
              row.fma<14>(t1, d25); row.fma<13>(t2, d25); row.fma<10>(t3, d25); row.fma<8>(t4, d25);
              row.fma<7>(t5, d25); row.fma<5>(t7, d25); row.fma<4>(t8, d25); row.fma<3>(a10, d25);
              row.fma<2>(a13, d25); row.fma<1>(a14, d25); row.fma<0>(a22, d25); const double d26 = row.d(26); row.fma<23>(t0, d26);
              row.fma<15>(t1, d26); row.fma<14>(t2, d26); row.fma<11>(t3, d26); row.fma<8>(t5, d26);
              row.fma<7>(t6, d26); row.fma<6>(t7, d26); row.fma<5>(t8, d26); row.fma<3>(a11, d26);
              row.fma<2>(a14, d26); row.fma<1>(a15, d26); row.fma<0>(a23, d26); const double d27 = row.d(27); row.fma<24>(t0, d27);
              row.fma<15>(t2, d27); row.fma<12>(t3, d27); row.fma<8>(t6, d27); row.fma<6>(t8, d27);
              row.fma<3>(a12, d27); row.fma<2>(a15, d27); row.fma<0>(a24, d27); const double d28 = row.d(28); row.fma<13>(t3, d28);
              row.fma<7>(t7, d28); row.fma<3>(a13, d28); const double d29 = row.d(29); row.fma<14>(t3, d29);
              row.fma<8>(t7, d29); row.fma<7>(t8, d29); row.fma<3>(a14, d29); const double d30 = row.d(30); row.fma<15>(t3, d30);
              row.fma<8>(t8, d30); row.fma<3>(a15, d30);
              if (ql >= 5) {
                const double d31 = row.d(31); row.fma<25>(t0, d31); row.fma<16>(t1, d31); row.fma<9>(t4, d31);
                row.fma<4>(a9, d31); row.fma<1>(a16, d31); row.fma<0>(a25, d31);
              }
            }
          }
        }
      }
    }
    __syncwarp();
    h_stage<16, 32, 16, 17>(db, P.D, P.dstr, it.c, lane, h_words<8>(h_dterms(min(6, it.qmax))));
    h_commit();
    h_wait<0>();
    __syncwarp();
    if (ql >= 5) {
      const double d32 = row.d(0); row.fma<26>(t0, d32); row.fma<17>(t1, d32); row.fma<16>(t2, d32);
      row.fma<10>(t4, d32); row.fma<9>(t5, d32); row.fma<5>(a9, d32); row.fma<4>(a10, d32);
      row.fma<2>(a16, d32); row.fma<1>(a17, d32); row.fma<0>(a26, d32); const double d33 = row.d(1); row.fma<27>(t0, d33);
      row.fma<18>(t1, d33); row.fma<17>(t2, d33); row.fma<11>(t4, d33); row.fma<10>(t5, d33);
      row.fma<9>(t6, d33); row.fma<6>(a9, d33); row.fma<5>(a10, d33); row.fma<4>(a11, d33);
      row.fma<2>(a17, d33); row.fma<1>(a18, d33); row.fma<0>(a27, d33); const double d34 = row.d(2); row.fma<28>(t0, d34);
      row.fma<19>(t1, d34); row.fma<18>(t2, d34); row.fma<12>(t4, d34); row.fma<11>(t5, d34);
      row.fma<10>(t6, d34); row.fma<6>(a10, d34); row.fma<5>(a11, d34); row.fma<4>(a12, d34);
      row.fma<2>(a18, d34); row.fma<1>(a19, d34); row.fma<0>(a28, d34); const double d35 = row.d(3); row.fma<29>(t0, d35);
      row.fma<20>(t1, d35); row.fma<19>(t2, d35); row.fma<12>(t5, d35); row.fma<11>(t6, d35);
      row.fma<6>(a11, d35); row.fma<5>(a12, d35); row.fma<2>(a19, d35); row.fma<1>(a20, d35);
      row.fma<0>(a29, d35); const double d36 = row.d(4); row.fma<30>(t0, d36); row.fma<20>(t2, d36);
      row.fma<12>(t6, d36); row.fma<6>(a12, d36); row.fma<2>(a20, d36); row.fma<0>(a30, d36);
      const double d37 = row.d(5); row.fma<31>(t0, d37); row.fma<21>(t1, d37); row.fma<16>(t3, d37);
      row.fma<13>(t4, d37); row.fma<9>(t7, d37); row.fma<7>(a9, d37); row.fma<4>(a13, d37);
      row.fma<3>(a16, d37); row.fma<1>(a21, d37); row.fma<0>(a31, d37); const double d38 = row.d(6); row.fma<32>(t0, d38);
      row.fma<22>(t1, d38); row.fma<21>(t2, d38); row.fma<17>(t3, d38); row.fma<14>(t4, d38);
      row.fma<13>(t5, d38); row.fma<10>(t7, d38); row.fma<9>(t8, d38); row.fma<8>(a9, d38);
      row.fma<7>(a10, d38); row.fma<5>(a13, d38); row.fma<4>(a14, d38); row.fma<3>(a17, d38);
      row.fma<2>(a21, d38); row.fma<1>(a22, d38); row.fma<0>(a32, d38); const double d39 = row.d(7); row.fma<33>(t0, d39);
      row.fma<23>(t1, d39); row.fma<22>(t2, d39); row.fma<18>(t3, d39); row.fma<15>(t4, d39);
      row.fma<14>(t5, d39); row.fma<13>(t6, d39); row.fma<11>(t7, d39); row.fma<10>(t8, d39);
      row.fma<8>(a10, d39); row.fma<7>(a11, d39); row.fma<6>(a13, d39); row.fma<5>(a14, d39);
      row.fma<4>(a15, d39); row.fma<3>(a18, d39); row.fma<2>(a22, d39); row.fma<1>(a23, d39);
      row.fma<0>(a33, d39); const double d40 = row.d(8); row.fma<34>(t0, d40); row.fma<24>(t1, d40);
      row.fma<23>(t2, d40); row.fma<19>(t3, d40); row.fma<15>(t5, d40); row.fma<14>(t6, d40);
      row.fma<12>(t7, d40); row.fma<11>(t8, d40); row.fma<8>(a11, d40); row.fma<7>(a12, d40);
      row.fma<6>(a14, d40); row.fma<5>(a15, d40); row.fma<3>(a19, d40); row.fma<2>(a23, d40);
      row.fma<1>(a24, d40); row.fma<0>(a34, d40); const double d41 = row.d(9); row.fma<35>(t0, d41);
      row.fma<24>(t2, d41); row.fma<20>(t3, d41); row.fma<15>(t6, d41); row.fma<12>(t8, d41);
      row.fma<8>(a12, d41); row.fma<6>(a15, d41); row.fma<3>(a20, d41); row.fma<2>(a24, d41);
      row.fma<0>(a35, d41); const double d42 = row.d(10); row.fma<21>(t3, d42); row.fma<13>(t7, d42);
      row.fma<7>(a13, d42); row.fma<3>(a21, d42); const double d43 = row.d(11); row.fma<22>(t3, d43);
      row.fma<14>(t7, d43); row.fma<13>(t8, d43); row.fma<8>(a13, d43); row.fma<7>(a14, d43);
      row.fma<3>(a22, d43); const double d44 = row.d(12); row.fma<23>(t3, d44); row.fma<15>(t7, d44);
      row.fma<14>(t8, d44); row.fma<8>(a14, d44); row.fma<7>(a15, d44); row.fma<3>(a23, d44);
      const double d45 = row.d(13); row.fma<24>(t3, d45); row.fma<15>(t8, d45); row.fma<8>(a15, d45);
      row.fma<3>(a24, d45);
      if (ql >= 6) {
        const double d46 = row.d(14); row.fma<36>(t0, d46); row.fma<25>(t1, d46); row.fma<16>(t4, d46);
        row.fma<9>(a9, d46); row.fma<4>(a16, d46); row.fma<1>(a25, d46); row.fma<0>(a36, d46);
        const double d47 = row.d(15); row.fma<37>(t0, d47); row.fma<26>(t1, d47); row.fma<25>(t2, d47);
        row.fma<17>(t4, d47); row.fma<16>(t5, d47); row.fma<10>(a9, d47); row.fma<9>(a10, d47);
        row.fma<5>(a16, d47); row.fma<4>(a17, d47); row.fma<2>(a25, d47); row.fma<1>(a26, d47);
        row.fma<0>(a37, d47); const double d48 = row.d(16); row.fma<38>(t0, d48); row.fma<27>(t1, d48);
        row.fma<26>(t2, d48); row.fma<18>(t4, d48); row.fma<17>(t5, d48); row.fma<16>(t6, d48);
        row.fma<11>(a9, d48); row.fma<10>(a10, d48); row.fma<9>(a11, d48); row.fma<6>(a16, d48);
        row.fma<5>(a17, d48); row.fma<4>(a18, d48); row.fma<2>(a26, d48); row.fma<1>(a27, d48);
        row.fma<0>(a38, d48); const double d49 = row.d(17); row.fma<39>(t0, d49); row.fma<28>(t1, d49);
        row.fma<27>(t2, d49); row.fma<19>(t4, d49); row.fma<18>(t5, d49); row.fma<17>(t6, d49);
        row.fma<12>(a9, d49); row.fma<11>(a10, d49); row.fma<10>(a11, d49); row.fma<9>(a12, d49);
        row.fma<6>(a17, d49); row.fma<5>(a18, d49); row.fma<4>(a19, d49); row.fma<2>(a27, d49);
        row.fma<1>(a28, d49); row.fma<0>(a39, d49); const double d50 = row.d(18); row.fma<40>(t0, d50);
        row.fma<29>(t1, d50); row.fma<28>(t2, d50); row.fma<20>(t4, d50); row.fma<19>(t5, d50);
        row.fma<18>(t6, d50); row.fma<12>(a10, d50); row.fma<11>(a11, d50); row.fma<10>(a12, d50);
        row.fma<6>(a18, d50); row.fma<5>(a19, d50); row.fma<4>(a20, d50); row.fma<2>(a28, d50);
        row.fma<1>(a29, d50); row.fma<0>(a40, d50); const double d51 = row.d(19); row.fma<41>(t0, d51);
        row.fma<30>(t1, d51); row.fma<29>(t2, d51); row.fma<20>(t5, d51); row.fma<19>(t6, d51);
        row.fma<12>(a11, d51); row.fma<11>(a12, d51); row.fma<6>(a19, d51); row.fma<5>(a20, d51);
        row.fma<2>(a29, d51); row.fma<1>(a30, d51); row.fma<0>(a41, d51); const double d52 = row.d(20); row.fma<42>(t0, d52);
        row.fma<30>(t2, d52); row.fma<20>(t6, d52); row.fma<12>(a12, d52); row.fma<6>(a20, d52);
        row.fma<2>(a30, d52); row.fma<0>(a42, d52); const double d53 = row.d(21); row.fma<43>(t0, d53);
        row.fma<31>(t1, d53); row.fma<25>(t3, d53); row.fma<21>(t4, d53); row.fma<16>(t7, d53);
        row.fma<13>(a9, d53); row.fma<9>(a13, d53); row.fma<7>(a16, d53); row.fma<4>(a21, d53);
        row.fma<3>(a25, d53); row.fma<1>(a31, d53); row.fma<0>(a43, d53); const double d54 = row.d(22); row.fma<44>(t0, d54);
        row.fma<32>(t1, d54); row.fma<31>(t2, d54); row.fma<26>(t3, d54); row.fma<22>(t4, d54);
        row.fma<21>(t5, d54); row.fma<17>(t7, d54); row.fma<16>(t8, d54); row.fma<14>(a9, d54);
        row.fma<13>(a10, d54); row.fma<10>(a13, d54); row.fma<9>(a14, d54); row.fma<8>(a16, d54);
        row.fma<7>(a17, d54); row.fma<5>(a21, d54); row.fma<4>(a22, d54); row.fma<3>(a26, d54);
        row.fma<2>(a31, d54); row.fma<1>(a32, d54); row.fma<0>(a44, d54); const double d55 = row.d(23); row.fma<45>(t0, d55);
        row.fma<33>(t1, d55); row.fma<32>(t2, d55); row.fma<27>(t3, d55); row.fma<23>(t4, d55);
        row.fma<22>(t5, d55); row.fma<21>(t6, d55); row.fma<18>(t7, d55); row.fma<17>(t8, d55);
        row.fma<15>(a9, d55); row.fma<14>(a10, d55); row.fma<13>(a11, d55); row.fma<11>(a13, d55);
        row.fma<10>(a14, d55); row.fma<9>(a15, d55); row.fma<8>(a17, d55); row.fma<7>(a18, d55);
        row.fma<6>(a21, d55); row.fma<5>(a22, d55); row.fma<4>(a23, d55); row.fma<3>(a27, d55);
        row.fma<2>(a32, d55); row.fma<1>(a33, d55); row.fma<0>(a45, d55); const double d56 = row.d(24); row.fma<46>(t0, d56);
        row.fma<34>(t1, d56); row.fma<33>(t2, d56); row.fma<28>(t3, d56); row.fma<24>(t4, d56);
        row.fma<23>(t5, d56); row.fma<22>(t6, d56); row.fma<19>(t7, d56); row.fma<18>(t8, d56);
        row.fma<15>(a10, d56); row.fma<14>(a11, d56); row.fma<13>(a12, d56); row.fma<12>(a13, d56);
        row.fma<11>(a14, d56); row.fma<10>(a15, d56); row.fma<8>(a18, d56); row.fma<7>(a19, d56);
        row.fma<6>(a22, d56); row.fma<5>(a23, d56); row.fma<4>(a24, d56); row.fma<3>(a28, d56);
        row.fma<2>(a33, d56); row.fma<1>(a34, d56); row.fma<0>(a46, d56); const double d57 = row.d(25); row.fma<47>(t0, d57);
        row.fma<35>(t1, d57); row.fma<34>(t2, d57); row.fma<29>(t3, d57); row.fma<24>(t5, d57);
        row.fma<23>(t6, d57); row.fma<20>(t7, d57); row.fma<19>(t8, d57); row.fma<15>(a11, d57);
        row.fma<14>(a12, d57); row.fma<12>(a14, d57); row.fma<11>(a15, d57); row.fma<8>(a19, d57);
        row.fma<7>(a20, d57); row.fma<6>(a23, d57); row.fma<5>(a24, d57); row.fma<3>(a29, d57);
        row.fma<2>(a34, d57); row.fma<1>(a35, d57); row.fma<0>(a47, d57); const double d58 = row.d(26); row.fma<48>(t0, d58);
        row.fma<35>(t2, d58); row.fma<30>(t3, d58); row.fma<24>(t6, d58); row.fma<20>(t8, d58);
        row.fma<15>(a12, d58); row.fma<12>(a15, d58); row.fma<8>(a20, d58); row.fma<6>(a24, d58);
        row.fma<3>(a30, d58); row.fma<2>(a35, d58); row.fma<0>(a48, d58); const double d59 = row.d(27); row.fma<31>(t3, d59);
        row.fma<21>(t7, d59); row.fma<13>(a13, d59); row.fma<7>(a21, d59); row.fma<3>(a31, d59);
        const double d60 = row.d(28); row.fma<32>(t3, d60); row.fma<22>(t7, d60); row.fma<21>(t8, d60);
        row.fma<14>(a13, d60); row.fma<13>(a14, d60); row.fma<8>(a21, d60); row.fma<7>(a22, d60);
        row.fma<3>(a32, d60); const double d61 = row.d(29); row.fma<33>(t3, d61); row.fma<23>(t7, d61);
        row.fma<22>(t8, d61); row.fma<15>(a13, d61); row.fma<14>(a14, d61); row.fma<13>(a15, d61);
        row.fma<8>(a22, d61); row.fma<7>(a23, d61); row.fma<3>(a33, d61); const double d62 = row.d(30); row.fma<34>(t3, d62);
        row.fma<24>(t7, d62); row.fma<23>(t8, d62); row.fma<15>(a14, d62); row.fma<14>(a15, d62);
        row.fma<8>(a23, d62); row.fma<7>(a24, d62); row.fma<3>(a34, d62); const double d63 = row.d(31); row.fma<35>(t3, d63);
        row.fma<24>(t8, d63); row.fma<15>(a15, d63); row.fma<8>(a24, d63); row.fma<3>(a35, d63);
      }
    }
    a0 += t0; a1 += t1; a2 += t2; a3 += t3; a4 += t4; a5 += t5; a6 += t6; a7 += t7; a8 += t8;
    __syncwarp();
    if (it.on_next) {
      h_stage<0, 25, 0, 25>(mb, P.M, P.mstr, it.Bs, lane, h_words<8>(h_terms(min(6, it.qmaxn - 0))));
      h_stage<0, 16, 0, 17>(db, P.D, P.dstr, it.cs, lane, h_words<8>(h_dterms(min(6, it.qmaxn))));
    }
    h_commit();
    it.advance();
  }
  h_wait<0>();
  // the warps' sums, in shared memory
  double *const sum = (double *)(h_smem + w * 1344) + lane;
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
  h_store<double, 49, 2688, false>(P, (double *)h_smem, 0, W);
}

int fmm_m2lh_f64_p6(const HParams<double> &P, cudaStream_t st) {
  if (P.p >= 0)
    if (int rc = h_launch(k_m2lh_f64_p6_0, P, 21504, 8, st)) return rc;
  return FMM_OK;
}
