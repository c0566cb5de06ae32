// GENERATED by gen_ops.py -- do not edit by hand.
// Register-unrolled small-matrix products for the Kalman hot path.
#pragma once

namespace mkfg {

// Cout = J * C * J^T for the barrel helix Jacobian (C, Cout packed symmetric)
// Algorithmic FLOPs (FMA = 2): 317
__device__ __forceinline__ void similarity_barrel(const float (&J)[36], const float (&C)[21], float (&Cout)[21])
{
  float T[36];
  T[0] = fmaf(J[4], C[10], fmaf(J[3], C[6], fmaf(J[0], C[0], J[1] * C[1])));
  T[1] = fmaf(J[4], C[11], fmaf(J[3], C[7], fmaf(J[0], C[1], J[1] * C[2])));
  T[2] = fmaf(J[4], C[12], fmaf(J[3], C[8], fmaf(J[0], C[3], J[1] * C[4])));
  T[3] = fmaf(J[4], C[13], fmaf(J[3], C[9], fmaf(J[0], C[6], J[1] * C[7])));
  T[4] = fmaf(J[4], C[14], fmaf(J[3], C[13], fmaf(J[0], C[10], J[1] * C[11])));
  T[5] = fmaf(J[4], C[19], fmaf(J[3], C[18], fmaf(J[0], C[15], J[1] * C[16])));
  T[6] = fmaf(J[10], C[10], fmaf(J[9], C[6], fmaf(J[6], C[0], J[7] * C[1])));
  T[7] = fmaf(J[10], C[11], fmaf(J[9], C[7], fmaf(J[6], C[1], J[7] * C[2])));
  T[8] = fmaf(J[10], C[12], fmaf(J[9], C[8], fmaf(J[6], C[3], J[7] * C[4])));
  T[9] = fmaf(J[10], C[13], fmaf(J[9], C[9], fmaf(J[6], C[6], J[7] * C[7])));
  T[10] = fmaf(J[10], C[14], fmaf(J[9], C[13], fmaf(J[6], C[10], J[7] * C[11])));
  T[11] = fmaf(J[10], C[19], fmaf(J[9], C[18], fmaf(J[6], C[15], J[7] * C[16])));
  T[12] = fmaf(J[17], C[15], fmaf(J[16], C[10], fmaf(J[15], C[6], fmaf(J[12], C[0], J[13] * C[1]) + C[3])));
  T[13] = fmaf(J[17], C[16], fmaf(J[16], C[11], fmaf(J[15], C[7], fmaf(J[12], C[1], J[13] * C[2]) + C[4])));
  T[14] = fmaf(J[17], C[17], fmaf(J[16], C[12], fmaf(J[15], C[8], fmaf(J[12], C[3], J[13] * C[4]) + C[5])));
  T[15] = fmaf(J[17], C[18], fmaf(J[16], C[13], fmaf(J[15], C[9], fmaf(J[12], C[6], J[13] * C[7]) + C[8])));
  T[16] = fmaf(J[17], C[19], fmaf(J[16], C[14], fmaf(J[15], C[13], fmaf(J[12], C[10], J[13] * C[11]) + C[12])));
  T[17] = fmaf(J[17], C[20], fmaf(J[16], C[19], fmaf(J[15], C[18], fmaf(J[12], C[15], J[13] * C[16]) + C[17])));
  T[18] = C[6];
  T[19] = C[7];
  T[20] = C[8];
  T[21] = C[9];
  T[22] = C[13];
  T[23] = C[18];
  T[24] = fmaf(J[28], C[10], fmaf(J[27], C[6], fmaf(J[24], C[0], J[25] * C[1])));
  T[25] = fmaf(J[28], C[11], fmaf(J[27], C[7], fmaf(J[24], C[1], J[25] * C[2])));
  T[26] = fmaf(J[28], C[12], fmaf(J[27], C[8], fmaf(J[24], C[3], J[25] * C[4])));
  T[27] = fmaf(J[28], C[13], fmaf(J[27], C[9], fmaf(J[24], C[6], J[25] * C[7])));
  T[28] = fmaf(J[28], C[14], fmaf(J[27], C[13], fmaf(J[24], C[10], J[25] * C[11])));
  T[29] = fmaf(J[28], C[19], fmaf(J[27], C[18], fmaf(J[24], C[15], J[25] * C[16])));
  T[30] = C[15];
  T[31] = C[16];
  T[32] = C[17];
  T[33] = C[18];
  T[34] = C[19];
  T[35] = C[20];
  Cout[0] = fmaf(T[4], J[4], fmaf(T[3], J[3], fmaf(T[0], J[0], T[1] * J[1])));
  Cout[1] = fmaf(T[10], J[4], fmaf(T[9], J[3], fmaf(T[6], J[0], T[7] * J[1])));
  Cout[2] = fmaf(T[10], J[10], fmaf(T[9], J[9], fmaf(T[6], J[6], T[7] * J[7])));
  Cout[3] = fmaf(T[16], J[4], fmaf(T[15], J[3], fmaf(T[12], J[0], T[13] * J[1])));
  Cout[4] = fmaf(T[16], J[10], fmaf(T[15], J[9], fmaf(T[12], J[6], T[13] * J[7])));
  Cout[5] = fmaf(T[17], J[17], fmaf(T[16], J[16], fmaf(T[15], J[15], fmaf(T[12], J[12], T[13] * J[13]) + T[14])));
  Cout[6] = fmaf(T[22], J[4], fmaf(T[21], J[3], fmaf(T[18], J[0], T[19] * J[1])));
  Cout[7] = fmaf(T[22], J[10], fmaf(T[21], J[9], fmaf(T[18], J[6], T[19] * J[7])));
  Cout[8] = fmaf(T[23], J[17], fmaf(T[22], J[16], fmaf(T[21], J[15], fmaf(T[18], J[12], T[19] * J[13]) + T[20])));
  Cout[9] = T[21];
  Cout[10] = fmaf(T[28], J[4], fmaf(T[27], J[3], fmaf(T[24], J[0], T[25] * J[1])));
  Cout[11] = fmaf(T[28], J[10], fmaf(T[27], J[9], fmaf(T[24], J[6], T[25] * J[7])));
  Cout[12] = fmaf(T[29], J[17], fmaf(T[28], J[16], fmaf(T[27], J[15], fmaf(T[24], J[12], T[25] * J[13]) + T[26])));
  Cout[13] = T[27];
  Cout[14] = fmaf(T[28], J[28], fmaf(T[27], J[27], fmaf(T[24], J[24], T[25] * J[25])));
  Cout[15] = fmaf(T[34], J[4], fmaf(T[33], J[3], fmaf(T[30], J[0], T[31] * J[1])));
  Cout[16] = fmaf(T[34], J[10], fmaf(T[33], J[9], fmaf(T[30], J[6], T[31] * J[7])));
  Cout[17] = fmaf(T[35], J[17], fmaf(T[34], J[16], fmaf(T[33], J[15], fmaf(T[30], J[12], T[31] * J[13]) + T[32])));
  Cout[18] = T[33];
  Cout[19] = fmaf(T[34], J[28], fmaf(T[33], J[27], fmaf(T[30], J[24], T[31] * J[25])));
  Cout[20] = T[35];
}

// Cout = J * C * J^T for the endcap (propagate-to-z) Jacobian
// Algorithmic FLOPs (FMA = 2): 216
__device__ __forceinline__ void similarity_endcap(const float (&J)[36], const float (&C)[21], float (&Cout)[21])
{
  float T[36];
  T[0] = fmaf(J[5], C[15], fmaf(J[4], C[10], fmaf(J[3], C[6], fmaf(J[2], C[3], C[0]))));
  T[1] = fmaf(J[5], C[16], fmaf(J[4], C[11], fmaf(J[3], C[7], fmaf(J[2], C[4], C[1]))));
  T[2] = fmaf(J[5], C[17], fmaf(J[4], C[12], fmaf(J[3], C[8], fmaf(J[2], C[5], C[3]))));
  T[3] = fmaf(J[5], C[18], fmaf(J[4], C[13], fmaf(J[3], C[9], fmaf(J[2], C[8], C[6]))));
  T[4] = fmaf(J[5], C[19], fmaf(J[4], C[14], fmaf(J[3], C[13], fmaf(J[2], C[12], C[10]))));
  T[5] = fmaf(J[5], C[20], fmaf(J[4], C[19], fmaf(J[3], C[18], fmaf(J[2], C[17], C[15]))));
  T[6] = fmaf(J[11], C[15], fmaf(J[10], C[10], fmaf(J[9], C[6], fmaf(J[8], C[3], C[1]))));
  T[7] = fmaf(J[11], C[16], fmaf(J[10], C[11], fmaf(J[9], C[7], fmaf(J[8], C[4], C[2]))));
  T[8] = fmaf(J[11], C[17], fmaf(J[10], C[12], fmaf(J[9], C[8], fmaf(J[8], C[5], C[4]))));
  T[9] = fmaf(J[11], C[18], fmaf(J[10], C[13], fmaf(J[9], C[9], fmaf(J[8], C[8], C[7]))));
  T[10] = fmaf(J[11], C[19], fmaf(J[10], C[14], fmaf(J[9], C[13], fmaf(J[8], C[12], C[11]))));
  T[11] = fmaf(J[11], C[20], fmaf(J[10], C[19], fmaf(J[9], C[18], fmaf(J[8], C[17], C[16]))));
  T[12] = 0.f;
  T[13] = 0.f;
  T[14] = 0.f;
  T[15] = 0.f;
  T[16] = 0.f;
  T[17] = 0.f;
  T[18] = C[6];
  T[19] = C[7];
  T[20] = C[8];
  T[21] = C[9];
  T[22] = C[13];
  T[23] = C[18];
  T[24] = fmaf(J[29], C[15], fmaf(J[26], C[3], J[27] * C[6]) + C[10]);
  T[25] = fmaf(J[29], C[16], fmaf(J[26], C[4], J[27] * C[7]) + C[11]);
  T[26] = fmaf(J[29], C[17], fmaf(J[26], C[5], J[27] * C[8]) + C[12]);
  T[27] = fmaf(J[29], C[18], fmaf(J[26], C[8], J[27] * C[9]) + C[13]);
  T[28] = fmaf(J[29], C[19], fmaf(J[26], C[12], J[27] * C[13]) + C[14]);
  T[29] = fmaf(J[29], C[20], fmaf(J[26], C[17], J[27] * C[18]) + C[19]);
  T[30] = C[15];
  T[31] = C[16];
  T[32] = C[17];
  T[33] = C[18];
  T[34] = C[19];
  T[35] = C[20];
  Cout[0] = fmaf(T[5], J[5], fmaf(T[4], J[4], fmaf(T[3], J[3], fmaf(T[2], J[2], T[0]))));
  Cout[1] = fmaf(T[11], J[5], fmaf(T[10], J[4], fmaf(T[9], J[3], fmaf(T[8], J[2], T[6]))));
  Cout[2] = fmaf(T[11], J[11], fmaf(T[10], J[10], fmaf(T[9], J[9], fmaf(T[8], J[8], T[7]))));
  Cout[3] = 0.f;
  Cout[4] = 0.f;
  Cout[5] = 0.f;
  Cout[6] = fmaf(T[23], J[5], fmaf(T[22], J[4], fmaf(T[21], J[3], fmaf(T[20], J[2], T[18]))));
  Cout[7] = fmaf(T[23], J[11], fmaf(T[22], J[10], fmaf(T[21], J[9], fmaf(T[20], J[8], T[19]))));
  Cout[8] = 0.f;
  Cout[9] = T[21];
  Cout[10] = fmaf(T[29], J[5], fmaf(T[28], J[4], fmaf(T[27], J[3], fmaf(T[26], J[2], T[24]))));
  Cout[11] = fmaf(T[29], J[11], fmaf(T[28], J[10], fmaf(T[27], J[9], fmaf(T[26], J[8], T[25]))));
  Cout[12] = 0.f;
  Cout[13] = T[27];
  Cout[14] = fmaf(T[29], J[29], fmaf(T[26], J[26], T[27] * J[27]) + T[28]);
  Cout[15] = fmaf(T[35], J[5], fmaf(T[34], J[4], fmaf(T[33], J[3], fmaf(T[32], J[2], T[30]))));
  Cout[16] = fmaf(T[35], J[11], fmaf(T[34], J[10], fmaf(T[33], J[9], fmaf(T[32], J[8], T[31]))));
  Cout[17] = 0.f;
  Cout[18] = T[33];
  Cout[19] = fmaf(T[35], J[29], fmaf(T[32], J[26], T[33] * J[27]) + T[34]);
  Cout[20] = T[35];
}

// Out = KH * C (KH with three live columns; Out packed symmetric)
// Algorithmic FLOPs (FMA = 2): 105
__device__ __forceinline__ void khc_barrel(const float (&KH)[36], const float (&C)[21], float (&Out)[21])
{
  Out[0] = fmaf(KH[2], C[3], fmaf(KH[0], C[0], KH[1] * C[1]));
  Out[1] = fmaf(KH[8], C[3], fmaf(KH[6], C[0], KH[7] * C[1]));
  Out[2] = fmaf(KH[8], C[4], fmaf(KH[6], C[1], KH[7] * C[2]));
  Out[3] = fmaf(KH[14], C[3], fmaf(KH[12], C[0], KH[13] * C[1]));
  Out[4] = fmaf(KH[14], C[4], fmaf(KH[12], C[1], KH[13] * C[2]));
  Out[5] = fmaf(KH[14], C[5], fmaf(KH[12], C[3], KH[13] * C[4]));
  Out[6] = fmaf(KH[20], C[3], fmaf(KH[18], C[0], KH[19] * C[1]));
  Out[7] = fmaf(KH[20], C[4], fmaf(KH[18], C[1], KH[19] * C[2]));
  Out[8] = fmaf(KH[20], C[5], fmaf(KH[18], C[3], KH[19] * C[4]));
  Out[9] = fmaf(KH[20], C[8], fmaf(KH[18], C[6], KH[19] * C[7]));
  Out[10] = fmaf(KH[26], C[3], fmaf(KH[24], C[0], KH[25] * C[1]));
  Out[11] = fmaf(KH[26], C[4], fmaf(KH[24], C[1], KH[25] * C[2]));
  Out[12] = fmaf(KH[26], C[5], fmaf(KH[24], C[3], KH[25] * C[4]));
  Out[13] = fmaf(KH[26], C[8], fmaf(KH[24], C[6], KH[25] * C[7]));
  Out[14] = fmaf(KH[26], C[12], fmaf(KH[24], C[10], KH[25] * C[11]));
  Out[15] = fmaf(KH[32], C[3], fmaf(KH[30], C[0], KH[31] * C[1]));
  Out[16] = fmaf(KH[32], C[4], fmaf(KH[30], C[1], KH[31] * C[2]));
  Out[17] = fmaf(KH[32], C[5], fmaf(KH[30], C[3], KH[31] * C[4]));
  Out[18] = fmaf(KH[32], C[8], fmaf(KH[30], C[6], KH[31] * C[7]));
  Out[19] = fmaf(KH[32], C[12], fmaf(KH[30], C[10], KH[31] * C[11]));
  Out[20] = fmaf(KH[32], C[17], fmaf(KH[30], C[15], KH[31] * C[16]));
}

// Out = K * C[0:2,:] (K is 6x2; Out packed symmetric)
// Algorithmic FLOPs (FMA = 2): 63
__device__ __forceinline__ void khc_endcap(const float (&K)[12], const float (&C)[21], float (&Out)[21])
{
  Out[0] = fmaf(K[0], C[0], K[1] * C[1]);
  Out[1] = fmaf(K[2], C[0], K[3] * C[1]);
  Out[2] = fmaf(K[2], C[1], K[3] * C[2]);
  Out[3] = fmaf(K[4], C[0], K[5] * C[1]);
  Out[4] = fmaf(K[4], C[1], K[5] * C[2]);
  Out[5] = fmaf(K[4], C[3], K[5] * C[4]);
  Out[6] = fmaf(K[6], C[0], K[7] * C[1]);
  Out[7] = fmaf(K[6], C[1], K[7] * C[2]);
  Out[8] = fmaf(K[6], C[3], K[7] * C[4]);
  Out[9] = fmaf(K[6], C[6], K[7] * C[7]);
  Out[10] = fmaf(K[8], C[0], K[9] * C[1]);
  Out[11] = fmaf(K[8], C[1], K[9] * C[2]);
  Out[12] = fmaf(K[8], C[3], K[9] * C[4]);
  Out[13] = fmaf(K[8], C[6], K[9] * C[7]);
  Out[14] = fmaf(K[8], C[10], K[9] * C[11]);
  Out[15] = fmaf(K[10], C[0], K[11] * C[1]);
  Out[16] = fmaf(K[10], C[1], K[11] * C[2]);
  Out[17] = fmaf(K[10], C[3], K[11] * C[4]);
  Out[18] = fmaf(K[10], C[6], K[11] * C[7]);
  Out[19] = fmaf(K[10], C[10], K[11] * C[11]);
  Out[20] = fmaf(K[10], C[15], K[11] * C[16]);
}

}  // namespace mkfg
