// Coarse-level operators on the solver's hot path (loadpath/mg.py:174-346 for the level kinds,
// loadpath/mgops.py:106-146 for the products they replace).
//
// Level 1 ("weights"): K_c = sum_k w[k, c] M_k with M_k = P_k^T Ke P_k, the reference's first
// Galerkin level. With the child moduli's Walsh transform c = H w, sum_k w_k M_k =
// sum_t c_t G_t, G_t = sum_k H[t, k] M_k / 8, and in the corner-parity basis of the coarse cell
// the eight G_t together have 279 non-zeros, each (row, col) entry belonging to exactly one t.
// The kernel marches z like the fine kernel (four cells per step, x neighbours by shuffles, y
// neighbours through shared memory) and forms each cell's product in that basis: ~450 flops
// against the 4608 of the dense sum. Cells touching held dofs ("patch" cells: weights zero,
// an explicit masked matrix instead) are taken in the same march, a warp's lanes sharing a cell's
// dense product, or by a launch behind it.
//
// Levels >= 2 ("explicit"): K_c stored per cell, symmetric, as the 300 upper-triangle entries
// in entry-major order (entry p of consecutive cells contiguous, so a warp's loads coalesce).
// Two passes: a cell pass forms the 24 corner forces f_c = K_c u_c into a caller-provided
// (24, cells) buffer, a node pass sums each node's eight cells' rows and applies the mask.
#include <cstring>
#include <numeric>

#include "lp_common.cuh"
#include "lp_modal.cuh"
#include "lp_tma.cuh"

#include <mutex>

namespace {

template <typename T>
struct G1 {
  T c[279];
};

// f = sum_t c_t G^_t v on the corner-parity modes (index 3 * mode + component)
template <typename T>
__device__ __forceinline__ void g1_product(const G1<T>& g, const T (&c)[8], const T (&v)[24], T (&f)[24]) {
  f[0] = f[1] = f[2] = T(0);
  f[3] = c[0] * (g.c[0] * v[3] + g.c[1] * v[7] + g.c[2] * v[14])
         + c[1] * (g.c[3] * v[10] + g.c[4] * v[17])
         + c[2] * (g.c[5] * v[9] + g.c[6] * v[20])
         + c[3] * (g.c[7] * v[23])
         + c[4] * (g.c[8] * v[15] + g.c[9] * v[19])
         + c[5] * (g.c[10] * v[22])
         + c[6] * (g.c[11] * v[21]);
  f[4] = c[0] * (g.c[12] * v[4] + g.c[13] * v[6])
         + c[1] * (g.c[14] * v[9])
         + c[2] * (g.c[15] * v[10])
         + c[4] * (g.c[16] * v[16] + g.c[17] * v[18])
         + c[5] * (g.c[18] * v[21])
         + c[6] * (g.c[19] * v[22]);
  f[5] = c[0] * (g.c[20] * v[5] + g.c[21] * v[12])
         + c[1] * (g.c[22] * v[15])
         + c[2] * (g.c[23] * v[11] + g.c[24] * v[18])
         + c[3] * (g.c[25] * v[21])
         + c[4] * (g.c[26] * v[17])
         + c[6] * (g.c[27] * v[23]);
  f[6] = c[0] * (g.c[28] * v[4] + g.c[29] * v[6])
         + c[1] * (g.c[30] * v[9])
         + c[2] * (g.c[31] * v[10])
         + c[4] * (g.c[32] * v[16] + g.c[33] * v[18])
         + c[5] * (g.c[34] * v[21])
         + c[6] * (g.c[35] * v[22]);
  f[7] = c[0] * (g.c[36] * v[3] + g.c[37] * v[7] + g.c[38] * v[14])
         + c[1] * (g.c[39] * v[10] + g.c[40] * v[17])
         + c[2] * (g.c[41] * v[9] + g.c[42] * v[20])
         + c[3] * (g.c[43] * v[23])
         + c[4] * (g.c[44] * v[15] + g.c[45] * v[19])
         + c[5] * (g.c[46] * v[22])
         + c[6] * (g.c[47] * v[21]);
  f[8] = c[0] * (g.c[48] * v[8] + g.c[49] * v[13])
         + c[1] * (g.c[50] * v[11] + g.c[51] * v[16])
         + c[2] * (g.c[52] * v[19])
         + c[3] * (g.c[53] * v[22])
         + c[4] * (g.c[54] * v[20])
         + c[5] * (g.c[55] * v[23]);
  f[9] = c[0] * (g.c[56] * v[9] + g.c[57] * v[20])
         + c[1] * (g.c[58] * v[4] + g.c[59] * v[6] + g.c[60] * v[23])
         + c[2] * (g.c[61] * v[3] + g.c[62] * v[7] + g.c[63] * v[14])
         + c[3] * (g.c[64] * v[10] + g.c[65] * v[17])
         + c[4] * (g.c[66] * v[21])
         + c[5] * (g.c[67] * v[16] + g.c[68] * v[18])
         + c[6] * (g.c[69] * v[15] + g.c[70] * v[19])
         + c[7] * (g.c[71] * v[22]);
  f[10] = c[0] * (g.c[72] * v[10] + g.c[73] * v[17])
         + c[1] * (g.c[74] * v[3] + g.c[75] * v[7] + g.c[76] * v[14])
         + c[2] * (g.c[77] * v[4] + g.c[78] * v[6] + g.c[79] * v[23])
         + c[3] * (g.c[80] * v[9] + g.c[81] * v[20])
         + c[4] * (g.c[82] * v[22])
         + c[5] * (g.c[83] * v[15] + g.c[84] * v[19])
         + c[6] * (g.c[85] * v[16] + g.c[86] * v[18])
         + c[7] * (g.c[87] * v[21]);
  f[11] = c[0] * (g.c[88] * v[11] + g.c[89] * v[16] + g.c[90] * v[18])
         + c[1] * (g.c[91] * v[8] + g.c[92] * v[13] + g.c[93] * v[21])
         + c[2] * (g.c[94] * v[5] + g.c[95] * v[12] + g.c[96] * v[22])
         + c[3] * (g.c[97] * v[15] + g.c[98] * v[19])
         + c[4] * (g.c[99] * v[23])
         + c[5] * (g.c[100] * v[20])
         + c[6] * (g.c[101] * v[17]);
  f[12] = c[0] * (g.c[102] * v[5] + g.c[103] * v[12])
         + c[1] * (g.c[104] * v[15])
         + c[2] * (g.c[105] * v[11] + g.c[106] * v[18])
         + c[3] * (g.c[107] * v[21])
         + c[4] * (g.c[108] * v[17])
         + c[6] * (g.c[109] * v[23]);
  f[13] = c[0] * (g.c[110] * v[8] + g.c[111] * v[13])
         + c[1] * (g.c[112] * v[11] + g.c[113] * v[16])
         + c[2] * (g.c[114] * v[19])
         + c[3] * (g.c[115] * v[22])
         + c[4] * (g.c[116] * v[20])
         + c[5] * (g.c[117] * v[23]);
  f[14] = c[0] * (g.c[118] * v[3] + g.c[119] * v[7] + g.c[120] * v[14])
         + c[1] * (g.c[121] * v[10] + g.c[122] * v[17])
         + c[2] * (g.c[123] * v[9] + g.c[124] * v[20])
         + c[3] * (g.c[125] * v[23])
         + c[4] * (g.c[126] * v[15] + g.c[127] * v[19])
         + c[5] * (g.c[128] * v[22])
         + c[6] * (g.c[129] * v[21]);
  f[15] = c[0] * (g.c[130] * v[15] + g.c[131] * v[19])
         + c[1] * (g.c[132] * v[5] + g.c[133] * v[12] + g.c[134] * v[22])
         + c[2] * (g.c[135] * v[21])
         + c[3] * (g.c[136] * v[11] + g.c[137] * v[18])
         + c[4] * (g.c[138] * v[3] + g.c[139] * v[7] + g.c[140] * v[14])
         + c[5] * (g.c[141] * v[10] + g.c[142] * v[17])
         + c[6] * (g.c[143] * v[9] + g.c[144] * v[20])
         + c[7] * (g.c[145] * v[23]);
  f[16] = c[0] * (g.c[146] * v[11] + g.c[147] * v[16] + g.c[148] * v[18])
         + c[1] * (g.c[149] * v[8] + g.c[150] * v[13] + g.c[151] * v[21])
         + c[2] * (g.c[152] * v[22])
         + c[3] * (g.c[153] * v[19])
         + c[4] * (g.c[154] * v[4] + g.c[155] * v[6] + g.c[156] * v[23])
         + c[5] * (g.c[157] * v[9] + g.c[158] * v[20])
         + c[6] * (g.c[159] * v[10]);
  f[17] = c[0] * (g.c[160] * v[10] + g.c[161] * v[17])
         + c[1] * (g.c[162] * v[3] + g.c[163] * v[7] + g.c[164] * v[14])
         + c[2] * (g.c[165] * v[23])
         + c[3] * (g.c[166] * v[9] + g.c[167] * v[20])
         + c[4] * (g.c[168] * v[5] + g.c[169] * v[12] + g.c[170] * v[22])
         + c[5] * (g.c[171] * v[15] + g.c[172] * v[19])
         + c[6] * (g.c[173] * v[11] + g.c[174] * v[18])
         + c[7] * (g.c[175] * v[21]);
  f[18] = c[0] * (g.c[176] * v[11] + g.c[177] * v[16] + g.c[178] * v[18])
         + c[1] * (g.c[179] * v[21])
         + c[2] * (g.c[180] * v[5] + g.c[181] * v[12] + g.c[182] * v[22])
         + c[3] * (g.c[183] * v[15])
         + c[4] * (g.c[184] * v[4] + g.c[185] * v[6] + g.c[186] * v[23])
         + c[5] * (g.c[187] * v[9])
         + c[6] * (g.c[188] * v[10] + g.c[189] * v[17]);
  f[19] = c[0] * (g.c[190] * v[15] + g.c[191] * v[19])
         + c[1] * (g.c[192] * v[22])
         + c[2] * (g.c[193] * v[8] + g.c[194] * v[13] + g.c[195] * v[21])
         + c[3] * (g.c[196] * v[11] + g.c[197] * v[16])
         + c[4] * (g.c[198] * v[3] + g.c[199] * v[7] + g.c[200] * v[14])
         + c[5] * (g.c[201] * v[10] + g.c[202] * v[17])
         + c[6] * (g.c[203] * v[9] + g.c[204] * v[20])
         + c[7] * (g.c[205] * v[23]);
  f[20] = c[0] * (g.c[206] * v[9] + g.c[207] * v[20])
         + c[1] * (g.c[208] * v[23])
         + c[2] * (g.c[209] * v[3] + g.c[210] * v[7] + g.c[211] * v[14])
         + c[3] * (g.c[212] * v[10] + g.c[213] * v[17])
         + c[4] * (g.c[214] * v[8] + g.c[215] * v[13] + g.c[216] * v[21])
         + c[5] * (g.c[217] * v[11] + g.c[218] * v[16])
         + c[6] * (g.c[219] * v[15] + g.c[220] * v[19])
         + c[7] * (g.c[221] * v[22]);
  f[21] = c[0] * (g.c[222] * v[21])
         + c[1] * (g.c[223] * v[11] + g.c[224] * v[16] + g.c[225] * v[18])
         + c[2] * (g.c[226] * v[15] + g.c[227] * v[19])
         + c[3] * (g.c[228] * v[5] + g.c[229] * v[12] + g.c[230] * v[22])
         + c[4] * (g.c[231] * v[9] + g.c[232] * v[20])
         + c[5] * (g.c[233] * v[4] + g.c[234] * v[6] + g.c[235] * v[23])
         + c[6] * (g.c[236] * v[3] + g.c[237] * v[7] + g.c[238] * v[14])
         + c[7] * (g.c[239] * v[10] + g.c[240] * v[17]);
  f[22] = c[0] * (g.c[241] * v[22])
         + c[1] * (g.c[242] * v[15] + g.c[243] * v[19])
         + c[2] * (g.c[244] * v[11] + g.c[245] * v[16] + g.c[246] * v[18])
         + c[3] * (g.c[247] * v[8] + g.c[248] * v[13] + g.c[249] * v[21])
         + c[4] * (g.c[250] * v[10] + g.c[251] * v[17])
         + c[5] * (g.c[252] * v[3] + g.c[253] * v[7] + g.c[254] * v[14])
         + c[6] * (g.c[255] * v[4] + g.c[256] * v[6] + g.c[257] * v[23])
         + c[7] * (g.c[258] * v[9] + g.c[259] * v[20]);
  f[23] = c[0] * (g.c[260] * v[23])
         + c[1] * (g.c[261] * v[9] + g.c[262] * v[20])
         + c[2] * (g.c[263] * v[10] + g.c[264] * v[17])
         + c[3] * (g.c[265] * v[3] + g.c[266] * v[7] + g.c[267] * v[14])
         + c[4] * (g.c[268] * v[11] + g.c[269] * v[16] + g.c[270] * v[18])
         + c[5] * (g.c[271] * v[8] + g.c[272] * v[13] + g.c[273] * v[21])
         + c[6] * (g.c[274] * v[5] + g.c[275] * v[12] + g.c[276] * v[22])
         + c[7] * (g.c[277] * v[15] + g.c[278] * v[19]);
}

// row r of the level-1 modal product (the rows g1_product forms together), so a caller can
// consume each row as it is produced
template <int R, typename T>
__device__ __forceinline__ T g1_row(const G1<T>& g, const T (&c)[8], const T (&v)[24]);
template <>
__device__ __forceinline__ float g1_row<0, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return 0.0f;
}
template <>
__device__ __forceinline__ double g1_row<0, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return 0.0;
}
template <>
__device__ __forceinline__ float g1_row<1, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return 0.0f;
}
template <>
__device__ __forceinline__ double g1_row<1, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return 0.0;
}
template <>
__device__ __forceinline__ float g1_row<2, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return 0.0f;
}
template <>
__device__ __forceinline__ double g1_row<2, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return 0.0;
}
template <>
__device__ __forceinline__ float g1_row<3, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[0] * v[3] + g.c[1] * v[7] + g.c[2] * v[14]) + c[1] * (g.c[3] * v[10] + g.c[4] * v[17]) + c[2] * (g.c[5] * v[9] + g.c[6] * v[20]) + c[3] * (g.c[7] * v[23]) + c[4] * (g.c[8] * v[15] + g.c[9] * v[19]) + c[5] * (g.c[10] * v[22]) + c[6] * (g.c[11] * v[21]);
}
template <>
__device__ __forceinline__ double g1_row<3, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[0] * v[3] + g.c[1] * v[7] + g.c[2] * v[14]) + c[1] * (g.c[3] * v[10] + g.c[4] * v[17]) + c[2] * (g.c[5] * v[9] + g.c[6] * v[20]) + c[3] * (g.c[7] * v[23]) + c[4] * (g.c[8] * v[15] + g.c[9] * v[19]) + c[5] * (g.c[10] * v[22]) + c[6] * (g.c[11] * v[21]);
}
template <>
__device__ __forceinline__ float g1_row<4, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[12] * v[4] + g.c[13] * v[6]) + c[1] * (g.c[14] * v[9]) + c[2] * (g.c[15] * v[10]) + c[4] * (g.c[16] * v[16] + g.c[17] * v[18]) + c[5] * (g.c[18] * v[21]) + c[6] * (g.c[19] * v[22]);
}
template <>
__device__ __forceinline__ double g1_row<4, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[12] * v[4] + g.c[13] * v[6]) + c[1] * (g.c[14] * v[9]) + c[2] * (g.c[15] * v[10]) + c[4] * (g.c[16] * v[16] + g.c[17] * v[18]) + c[5] * (g.c[18] * v[21]) + c[6] * (g.c[19] * v[22]);
}
template <>
__device__ __forceinline__ float g1_row<5, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[20] * v[5] + g.c[21] * v[12]) + c[1] * (g.c[22] * v[15]) + c[2] * (g.c[23] * v[11] + g.c[24] * v[18]) + c[3] * (g.c[25] * v[21]) + c[4] * (g.c[26] * v[17]) + c[6] * (g.c[27] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<5, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[20] * v[5] + g.c[21] * v[12]) + c[1] * (g.c[22] * v[15]) + c[2] * (g.c[23] * v[11] + g.c[24] * v[18]) + c[3] * (g.c[25] * v[21]) + c[4] * (g.c[26] * v[17]) + c[6] * (g.c[27] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<6, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[28] * v[4] + g.c[29] * v[6]) + c[1] * (g.c[30] * v[9]) + c[2] * (g.c[31] * v[10]) + c[4] * (g.c[32] * v[16] + g.c[33] * v[18]) + c[5] * (g.c[34] * v[21]) + c[6] * (g.c[35] * v[22]);
}
template <>
__device__ __forceinline__ double g1_row<6, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[28] * v[4] + g.c[29] * v[6]) + c[1] * (g.c[30] * v[9]) + c[2] * (g.c[31] * v[10]) + c[4] * (g.c[32] * v[16] + g.c[33] * v[18]) + c[5] * (g.c[34] * v[21]) + c[6] * (g.c[35] * v[22]);
}
template <>
__device__ __forceinline__ float g1_row<7, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[36] * v[3] + g.c[37] * v[7] + g.c[38] * v[14]) + c[1] * (g.c[39] * v[10] + g.c[40] * v[17]) + c[2] * (g.c[41] * v[9] + g.c[42] * v[20]) + c[3] * (g.c[43] * v[23]) + c[4] * (g.c[44] * v[15] + g.c[45] * v[19]) + c[5] * (g.c[46] * v[22]) + c[6] * (g.c[47] * v[21]);
}
template <>
__device__ __forceinline__ double g1_row<7, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[36] * v[3] + g.c[37] * v[7] + g.c[38] * v[14]) + c[1] * (g.c[39] * v[10] + g.c[40] * v[17]) + c[2] * (g.c[41] * v[9] + g.c[42] * v[20]) + c[3] * (g.c[43] * v[23]) + c[4] * (g.c[44] * v[15] + g.c[45] * v[19]) + c[5] * (g.c[46] * v[22]) + c[6] * (g.c[47] * v[21]);
}
template <>
__device__ __forceinline__ float g1_row<8, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[48] * v[8] + g.c[49] * v[13]) + c[1] * (g.c[50] * v[11] + g.c[51] * v[16]) + c[2] * (g.c[52] * v[19]) + c[3] * (g.c[53] * v[22]) + c[4] * (g.c[54] * v[20]) + c[5] * (g.c[55] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<8, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[48] * v[8] + g.c[49] * v[13]) + c[1] * (g.c[50] * v[11] + g.c[51] * v[16]) + c[2] * (g.c[52] * v[19]) + c[3] * (g.c[53] * v[22]) + c[4] * (g.c[54] * v[20]) + c[5] * (g.c[55] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<9, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[56] * v[9] + g.c[57] * v[20]) + c[1] * (g.c[58] * v[4] + g.c[59] * v[6] + g.c[60] * v[23]) + c[2] * (g.c[61] * v[3] + g.c[62] * v[7] + g.c[63] * v[14]) + c[3] * (g.c[64] * v[10] + g.c[65] * v[17]) + c[4] * (g.c[66] * v[21]) + c[5] * (g.c[67] * v[16] + g.c[68] * v[18]) + c[6] * (g.c[69] * v[15] + g.c[70] * v[19]) + c[7] * (g.c[71] * v[22]);
}
template <>
__device__ __forceinline__ double g1_row<9, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[56] * v[9] + g.c[57] * v[20]) + c[1] * (g.c[58] * v[4] + g.c[59] * v[6] + g.c[60] * v[23]) + c[2] * (g.c[61] * v[3] + g.c[62] * v[7] + g.c[63] * v[14]) + c[3] * (g.c[64] * v[10] + g.c[65] * v[17]) + c[4] * (g.c[66] * v[21]) + c[5] * (g.c[67] * v[16] + g.c[68] * v[18]) + c[6] * (g.c[69] * v[15] + g.c[70] * v[19]) + c[7] * (g.c[71] * v[22]);
}
template <>
__device__ __forceinline__ float g1_row<10, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[72] * v[10] + g.c[73] * v[17]) + c[1] * (g.c[74] * v[3] + g.c[75] * v[7] + g.c[76] * v[14]) + c[2] * (g.c[77] * v[4] + g.c[78] * v[6] + g.c[79] * v[23]) + c[3] * (g.c[80] * v[9] + g.c[81] * v[20]) + c[4] * (g.c[82] * v[22]) + c[5] * (g.c[83] * v[15] + g.c[84] * v[19]) + c[6] * (g.c[85] * v[16] + g.c[86] * v[18]) + c[7] * (g.c[87] * v[21]);
}
template <>
__device__ __forceinline__ double g1_row<10, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[72] * v[10] + g.c[73] * v[17]) + c[1] * (g.c[74] * v[3] + g.c[75] * v[7] + g.c[76] * v[14]) + c[2] * (g.c[77] * v[4] + g.c[78] * v[6] + g.c[79] * v[23]) + c[3] * (g.c[80] * v[9] + g.c[81] * v[20]) + c[4] * (g.c[82] * v[22]) + c[5] * (g.c[83] * v[15] + g.c[84] * v[19]) + c[6] * (g.c[85] * v[16] + g.c[86] * v[18]) + c[7] * (g.c[87] * v[21]);
}
template <>
__device__ __forceinline__ float g1_row<11, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[88] * v[11] + g.c[89] * v[16] + g.c[90] * v[18]) + c[1] * (g.c[91] * v[8] + g.c[92] * v[13] + g.c[93] * v[21]) + c[2] * (g.c[94] * v[5] + g.c[95] * v[12] + g.c[96] * v[22]) + c[3] * (g.c[97] * v[15] + g.c[98] * v[19]) + c[4] * (g.c[99] * v[23]) + c[5] * (g.c[100] * v[20]) + c[6] * (g.c[101] * v[17]);
}
template <>
__device__ __forceinline__ double g1_row<11, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[88] * v[11] + g.c[89] * v[16] + g.c[90] * v[18]) + c[1] * (g.c[91] * v[8] + g.c[92] * v[13] + g.c[93] * v[21]) + c[2] * (g.c[94] * v[5] + g.c[95] * v[12] + g.c[96] * v[22]) + c[3] * (g.c[97] * v[15] + g.c[98] * v[19]) + c[4] * (g.c[99] * v[23]) + c[5] * (g.c[100] * v[20]) + c[6] * (g.c[101] * v[17]);
}
template <>
__device__ __forceinline__ float g1_row<12, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[102] * v[5] + g.c[103] * v[12]) + c[1] * (g.c[104] * v[15]) + c[2] * (g.c[105] * v[11] + g.c[106] * v[18]) + c[3] * (g.c[107] * v[21]) + c[4] * (g.c[108] * v[17]) + c[6] * (g.c[109] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<12, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[102] * v[5] + g.c[103] * v[12]) + c[1] * (g.c[104] * v[15]) + c[2] * (g.c[105] * v[11] + g.c[106] * v[18]) + c[3] * (g.c[107] * v[21]) + c[4] * (g.c[108] * v[17]) + c[6] * (g.c[109] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<13, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[110] * v[8] + g.c[111] * v[13]) + c[1] * (g.c[112] * v[11] + g.c[113] * v[16]) + c[2] * (g.c[114] * v[19]) + c[3] * (g.c[115] * v[22]) + c[4] * (g.c[116] * v[20]) + c[5] * (g.c[117] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<13, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[110] * v[8] + g.c[111] * v[13]) + c[1] * (g.c[112] * v[11] + g.c[113] * v[16]) + c[2] * (g.c[114] * v[19]) + c[3] * (g.c[115] * v[22]) + c[4] * (g.c[116] * v[20]) + c[5] * (g.c[117] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<14, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[118] * v[3] + g.c[119] * v[7] + g.c[120] * v[14]) + c[1] * (g.c[121] * v[10] + g.c[122] * v[17]) + c[2] * (g.c[123] * v[9] + g.c[124] * v[20]) + c[3] * (g.c[125] * v[23]) + c[4] * (g.c[126] * v[15] + g.c[127] * v[19]) + c[5] * (g.c[128] * v[22]) + c[6] * (g.c[129] * v[21]);
}
template <>
__device__ __forceinline__ double g1_row<14, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[118] * v[3] + g.c[119] * v[7] + g.c[120] * v[14]) + c[1] * (g.c[121] * v[10] + g.c[122] * v[17]) + c[2] * (g.c[123] * v[9] + g.c[124] * v[20]) + c[3] * (g.c[125] * v[23]) + c[4] * (g.c[126] * v[15] + g.c[127] * v[19]) + c[5] * (g.c[128] * v[22]) + c[6] * (g.c[129] * v[21]);
}
template <>
__device__ __forceinline__ float g1_row<15, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[130] * v[15] + g.c[131] * v[19]) + c[1] * (g.c[132] * v[5] + g.c[133] * v[12] + g.c[134] * v[22]) + c[2] * (g.c[135] * v[21]) + c[3] * (g.c[136] * v[11] + g.c[137] * v[18]) + c[4] * (g.c[138] * v[3] + g.c[139] * v[7] + g.c[140] * v[14]) + c[5] * (g.c[141] * v[10] + g.c[142] * v[17]) + c[6] * (g.c[143] * v[9] + g.c[144] * v[20]) + c[7] * (g.c[145] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<15, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[130] * v[15] + g.c[131] * v[19]) + c[1] * (g.c[132] * v[5] + g.c[133] * v[12] + g.c[134] * v[22]) + c[2] * (g.c[135] * v[21]) + c[3] * (g.c[136] * v[11] + g.c[137] * v[18]) + c[4] * (g.c[138] * v[3] + g.c[139] * v[7] + g.c[140] * v[14]) + c[5] * (g.c[141] * v[10] + g.c[142] * v[17]) + c[6] * (g.c[143] * v[9] + g.c[144] * v[20]) + c[7] * (g.c[145] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<16, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[146] * v[11] + g.c[147] * v[16] + g.c[148] * v[18]) + c[1] * (g.c[149] * v[8] + g.c[150] * v[13] + g.c[151] * v[21]) + c[2] * (g.c[152] * v[22]) + c[3] * (g.c[153] * v[19]) + c[4] * (g.c[154] * v[4] + g.c[155] * v[6] + g.c[156] * v[23]) + c[5] * (g.c[157] * v[9] + g.c[158] * v[20]) + c[6] * (g.c[159] * v[10]);
}
template <>
__device__ __forceinline__ double g1_row<16, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[146] * v[11] + g.c[147] * v[16] + g.c[148] * v[18]) + c[1] * (g.c[149] * v[8] + g.c[150] * v[13] + g.c[151] * v[21]) + c[2] * (g.c[152] * v[22]) + c[3] * (g.c[153] * v[19]) + c[4] * (g.c[154] * v[4] + g.c[155] * v[6] + g.c[156] * v[23]) + c[5] * (g.c[157] * v[9] + g.c[158] * v[20]) + c[6] * (g.c[159] * v[10]);
}
template <>
__device__ __forceinline__ float g1_row<17, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[160] * v[10] + g.c[161] * v[17]) + c[1] * (g.c[162] * v[3] + g.c[163] * v[7] + g.c[164] * v[14]) + c[2] * (g.c[165] * v[23]) + c[3] * (g.c[166] * v[9] + g.c[167] * v[20]) + c[4] * (g.c[168] * v[5] + g.c[169] * v[12] + g.c[170] * v[22]) + c[5] * (g.c[171] * v[15] + g.c[172] * v[19]) + c[6] * (g.c[173] * v[11] + g.c[174] * v[18]) + c[7] * (g.c[175] * v[21]);
}
template <>
__device__ __forceinline__ double g1_row<17, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[160] * v[10] + g.c[161] * v[17]) + c[1] * (g.c[162] * v[3] + g.c[163] * v[7] + g.c[164] * v[14]) + c[2] * (g.c[165] * v[23]) + c[3] * (g.c[166] * v[9] + g.c[167] * v[20]) + c[4] * (g.c[168] * v[5] + g.c[169] * v[12] + g.c[170] * v[22]) + c[5] * (g.c[171] * v[15] + g.c[172] * v[19]) + c[6] * (g.c[173] * v[11] + g.c[174] * v[18]) + c[7] * (g.c[175] * v[21]);
}
template <>
__device__ __forceinline__ float g1_row<18, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[176] * v[11] + g.c[177] * v[16] + g.c[178] * v[18]) + c[1] * (g.c[179] * v[21]) + c[2] * (g.c[180] * v[5] + g.c[181] * v[12] + g.c[182] * v[22]) + c[3] * (g.c[183] * v[15]) + c[4] * (g.c[184] * v[4] + g.c[185] * v[6] + g.c[186] * v[23]) + c[5] * (g.c[187] * v[9]) + c[6] * (g.c[188] * v[10] + g.c[189] * v[17]);
}
template <>
__device__ __forceinline__ double g1_row<18, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[176] * v[11] + g.c[177] * v[16] + g.c[178] * v[18]) + c[1] * (g.c[179] * v[21]) + c[2] * (g.c[180] * v[5] + g.c[181] * v[12] + g.c[182] * v[22]) + c[3] * (g.c[183] * v[15]) + c[4] * (g.c[184] * v[4] + g.c[185] * v[6] + g.c[186] * v[23]) + c[5] * (g.c[187] * v[9]) + c[6] * (g.c[188] * v[10] + g.c[189] * v[17]);
}
template <>
__device__ __forceinline__ float g1_row<19, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[190] * v[15] + g.c[191] * v[19]) + c[1] * (g.c[192] * v[22]) + c[2] * (g.c[193] * v[8] + g.c[194] * v[13] + g.c[195] * v[21]) + c[3] * (g.c[196] * v[11] + g.c[197] * v[16]) + c[4] * (g.c[198] * v[3] + g.c[199] * v[7] + g.c[200] * v[14]) + c[5] * (g.c[201] * v[10] + g.c[202] * v[17]) + c[6] * (g.c[203] * v[9] + g.c[204] * v[20]) + c[7] * (g.c[205] * v[23]);
}
template <>
__device__ __forceinline__ double g1_row<19, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[190] * v[15] + g.c[191] * v[19]) + c[1] * (g.c[192] * v[22]) + c[2] * (g.c[193] * v[8] + g.c[194] * v[13] + g.c[195] * v[21]) + c[3] * (g.c[196] * v[11] + g.c[197] * v[16]) + c[4] * (g.c[198] * v[3] + g.c[199] * v[7] + g.c[200] * v[14]) + c[5] * (g.c[201] * v[10] + g.c[202] * v[17]) + c[6] * (g.c[203] * v[9] + g.c[204] * v[20]) + c[7] * (g.c[205] * v[23]);
}
template <>
__device__ __forceinline__ float g1_row<20, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[206] * v[9] + g.c[207] * v[20]) + c[1] * (g.c[208] * v[23]) + c[2] * (g.c[209] * v[3] + g.c[210] * v[7] + g.c[211] * v[14]) + c[3] * (g.c[212] * v[10] + g.c[213] * v[17]) + c[4] * (g.c[214] * v[8] + g.c[215] * v[13] + g.c[216] * v[21]) + c[5] * (g.c[217] * v[11] + g.c[218] * v[16]) + c[6] * (g.c[219] * v[15] + g.c[220] * v[19]) + c[7] * (g.c[221] * v[22]);
}
template <>
__device__ __forceinline__ double g1_row<20, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[206] * v[9] + g.c[207] * v[20]) + c[1] * (g.c[208] * v[23]) + c[2] * (g.c[209] * v[3] + g.c[210] * v[7] + g.c[211] * v[14]) + c[3] * (g.c[212] * v[10] + g.c[213] * v[17]) + c[4] * (g.c[214] * v[8] + g.c[215] * v[13] + g.c[216] * v[21]) + c[5] * (g.c[217] * v[11] + g.c[218] * v[16]) + c[6] * (g.c[219] * v[15] + g.c[220] * v[19]) + c[7] * (g.c[221] * v[22]);
}
template <>
__device__ __forceinline__ float g1_row<21, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[222] * v[21]) + c[1] * (g.c[223] * v[11] + g.c[224] * v[16] + g.c[225] * v[18]) + c[2] * (g.c[226] * v[15] + g.c[227] * v[19]) + c[3] * (g.c[228] * v[5] + g.c[229] * v[12] + g.c[230] * v[22]) + c[4] * (g.c[231] * v[9] + g.c[232] * v[20]) + c[5] * (g.c[233] * v[4] + g.c[234] * v[6] + g.c[235] * v[23]) + c[6] * (g.c[236] * v[3] + g.c[237] * v[7] + g.c[238] * v[14]) + c[7] * (g.c[239] * v[10] + g.c[240] * v[17]);
}
template <>
__device__ __forceinline__ double g1_row<21, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[222] * v[21]) + c[1] * (g.c[223] * v[11] + g.c[224] * v[16] + g.c[225] * v[18]) + c[2] * (g.c[226] * v[15] + g.c[227] * v[19]) + c[3] * (g.c[228] * v[5] + g.c[229] * v[12] + g.c[230] * v[22]) + c[4] * (g.c[231] * v[9] + g.c[232] * v[20]) + c[5] * (g.c[233] * v[4] + g.c[234] * v[6] + g.c[235] * v[23]) + c[6] * (g.c[236] * v[3] + g.c[237] * v[7] + g.c[238] * v[14]) + c[7] * (g.c[239] * v[10] + g.c[240] * v[17]);
}
template <>
__device__ __forceinline__ float g1_row<22, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[241] * v[22]) + c[1] * (g.c[242] * v[15] + g.c[243] * v[19]) + c[2] * (g.c[244] * v[11] + g.c[245] * v[16] + g.c[246] * v[18]) + c[3] * (g.c[247] * v[8] + g.c[248] * v[13] + g.c[249] * v[21]) + c[4] * (g.c[250] * v[10] + g.c[251] * v[17]) + c[5] * (g.c[252] * v[3] + g.c[253] * v[7] + g.c[254] * v[14]) + c[6] * (g.c[255] * v[4] + g.c[256] * v[6] + g.c[257] * v[23]) + c[7] * (g.c[258] * v[9] + g.c[259] * v[20]);
}
template <>
__device__ __forceinline__ double g1_row<22, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[241] * v[22]) + c[1] * (g.c[242] * v[15] + g.c[243] * v[19]) + c[2] * (g.c[244] * v[11] + g.c[245] * v[16] + g.c[246] * v[18]) + c[3] * (g.c[247] * v[8] + g.c[248] * v[13] + g.c[249] * v[21]) + c[4] * (g.c[250] * v[10] + g.c[251] * v[17]) + c[5] * (g.c[252] * v[3] + g.c[253] * v[7] + g.c[254] * v[14]) + c[6] * (g.c[255] * v[4] + g.c[256] * v[6] + g.c[257] * v[23]) + c[7] * (g.c[258] * v[9] + g.c[259] * v[20]);
}
template <>
__device__ __forceinline__ float g1_row<23, float>(const G1<float>& g, const float (&c)[8], const float (&v)[24]) {
  return c[0] * (g.c[260] * v[23]) + c[1] * (g.c[261] * v[9] + g.c[262] * v[20]) + c[2] * (g.c[263] * v[10] + g.c[264] * v[17]) + c[3] * (g.c[265] * v[3] + g.c[266] * v[7] + g.c[267] * v[14]) + c[4] * (g.c[268] * v[11] + g.c[269] * v[16] + g.c[270] * v[18]) + c[5] * (g.c[271] * v[8] + g.c[272] * v[13] + g.c[273] * v[21]) + c[6] * (g.c[274] * v[5] + g.c[275] * v[12] + g.c[276] * v[22]) + c[7] * (g.c[277] * v[15] + g.c[278] * v[19]);
}
template <>
__device__ __forceinline__ double g1_row<23, double>(const G1<double>& g, const double (&c)[8], const double (&v)[24]) {
  return c[0] * (g.c[260] * v[23]) + c[1] * (g.c[261] * v[9] + g.c[262] * v[20]) + c[2] * (g.c[263] * v[10] + g.c[264] * v[17]) + c[3] * (g.c[265] * v[3] + g.c[266] * v[7] + g.c[267] * v[14]) + c[4] * (g.c[268] * v[11] + g.c[269] * v[16] + g.c[270] * v[18]) + c[5] * (g.c[271] * v[8] + g.c[272] * v[13] + g.c[273] * v[21]) + c[6] * (g.c[274] * v[5] + g.c[275] * v[12] + g.c[276] * v[22]) + c[7] * (g.c[277] * v[15] + g.c[278] * v[19]);
}

// modes 1, s (per axis) of a pair: (a, b) -> (a + b, b - a)
template <typename T>
__device__ __forceinline__ void fwht8(const T (&w)[8], T (&c)[8]) {
  T a[8], b[8];
#pragma unroll
  for (int k = 0; k < 8; k += 2) { a[k] = w[k] + w[k + 1]; a[k + 1] = w[k + 1] - w[k]; }
#pragma unroll
  for (int k = 0; k < 8; k += 4) {
    b[k] = a[k] + a[k + 2]; b[k + 2] = a[k + 2] - a[k];
    b[k + 1] = a[k + 1] + a[k + 3]; b[k + 3] = a[k + 3] - a[k + 1];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) { c[k] = b[k] + b[k + 4]; c[k + 4] = b[k + 4] - b[k]; }
}

template <typename T>
__device__ __forceinline__ void xy4(T u00, T u10, T u01, T u11, T (&a)[4]) {
  T sx0 = u00 + u10, dx0 = u10 - u00, sx1 = u01 + u11, dx1 = u11 - u01;
  a[0] = sx0 + sx1;
  a[1] = dx0 + dx1;
  a[2] = sx1 - sx0;
  a[3] = dx1 - dx0;
}

// ---- level 1, TMA-staged march -------------------------------------------------------------
// The chunked Walsh layout: c = H w per cell (the coefficients of the eight G_t), stored
// (cpz / 4, ny, nx, 4, 8) so one cell column's four cells of a z chunk are 128 contiguous bytes
// (float32), each cell's eight coefficients 32 of them, and a row of x columns is one run.
// Formed once per hierarchy (after the patch cells' weights are zeroed).
template <typename T>
__global__ void k_walsh_chunks(T* __restrict__ wc, const T* __restrict__ w, LpGrid g) {
  lp_after_launch();
  const long long ncp = g.cells_padded();
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncp; c += (long long)gridDim.x * blockDim.x) {
    T wk[8], cw[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) wk[k] = w[k * ncp + c];
    fwht8(wk, cw);
    T* dst = wc + (c >> 2) * 32 + (c & 3) * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k] = cw[k];
  }
}

constexpr int LX = 16, LY = 8;          // cell columns per block: 15 x 7 owned node columns
constexpr int LBX = LX + 1, LBY = LY + 1;
constexpr int LCOL = LX * LY;
constexpr int LST = 2;                  // TMA ring depth
constexpr int L1_MAX_BLOCKS = 296;
constexpr int L1_PATCH = 64;            // patch cells of a tile's chunk taken together

template <typename T, int N>
struct alignas(128) WSlot {
  T v[(N * sizeof(T) + 127) / 128 * 128 / sizeof(T)];
};

// float32: the Walsh coefficients of the block's 16 x 8 cell columns arrive by TMA with the
// node values, one 128-byte row per column in the 128-byte swizzle (a warp's 16-byte reads of
// eight consecutive rows then meet no bank twice); float64 reads them from global memory
template <typename T>
struct WCoef {
  static constexpr int N = sizeof(T) == 4 ? 32 * LCOL : 32;
};

template <typename T>
struct L1Smem {
  alignas(1024) T w[LST][WCoef<T>::N];                // Walsh coefficients [y][x][cell][t] (float32)
  WSlot<T, 3 * LBX * LBY * 4> u[LST];                 // node values [comp][y][x][z]
  // by chunk parity, component and plane: corners 00 + 10 with the -x neighbour's, and corners 01 + 11
  // (to y + 1)
  T own[2][3][4][LCOL];
  T red[2][3][4][LCOL];
  // the chunk's patch cells: their modes, products, matrices and cells (thread, z)
  T pv[L1_PATCH][24];
  T pf[L1_PATCH][24];
  int pmat[L1_PATCH], pcell[L1_PATCH], npatch;
  alignas(8) uint64_t full[LST];
};

struct L1Maps {
  CUtensorMap u;    // (4 NX, NY, pz / 4, 3), box (4 * 17, 9, 1, 3)
  CUtensorMap w;    // float32 Walsh coefficients (32, nx, ny, cpz / 4), box (32, 16, 8, 1), 128-byte swizzle
};

// block b takes units [u0[b], u0[b + 1]) of (tile, chunk), tile-major
struct L1Split {
  int u0[L1_MAX_BLOCKS + 1];
};

// cell columns [x, hx) x [y, hy) that hold the patch cells
struct L1Box {
  int x, hx, y, hy;
};

// nodes of columns [x, hx) x [y, hy) and chunks [c, hc) whose patch cells' part comes from the launch behind
struct L1Nodes {
  int x, hx, y, hy, c, hc;
};

template <typename T>
struct L1Cheb {
  T* x;
  T* r;
  T* d;
  const T* b;
  const T* dinv;
  const double* coef;
};

// node-plane forces of one cell: rows (3q + cc, 3(q + 4) + cc) of the modal product give the
// lower face (f0 - f1) and upper face (f0 + f1) of mode (q, cc); fp = carry + lower face and the
// upper face becomes the next carry, row pair by row pair
template <int Q, int CC, typename T>
__device__ __forceinline__ void fold_pair(const G1<T>& g, const T (&c)[8], const T (&v)[24], T& fp, T& up) {
  const T f0 = g1_row<3 * Q + CC, T>(g, c, v), f1 = g1_row<3 * (Q + 4) + CC, T>(g, c, v);
  fp = up + (f0 - f1);
  up = f0 + f1;
}

template <typename T>
__device__ __forceinline__ void fold_rows(const G1<T>& g, const T (&c)[8], const T (&v)[24], T (&fp)[4][3],
                                          T (&up)[4][3]) {
  fold_pair<0, 0>(g, c, v, fp[0][0], up[0][0]); fold_pair<0, 1>(g, c, v, fp[0][1], up[0][1]);
  fold_pair<0, 2>(g, c, v, fp[0][2], up[0][2]); fold_pair<1, 0>(g, c, v, fp[1][0], up[1][0]);
  fold_pair<1, 1>(g, c, v, fp[1][1], up[1][1]); fold_pair<1, 2>(g, c, v, fp[1][2], up[1][2]);
  fold_pair<2, 0>(g, c, v, fp[2][0], up[2][0]); fold_pair<2, 1>(g, c, v, fp[2][1], up[2][1]);
  fold_pair<2, 2>(g, c, v, fp[2][2], up[2][2]); fold_pair<3, 0>(g, c, v, fp[3][0], up[3][0]);
  fold_pair<3, 1>(g, c, v, fp[3][1], up[3][1]); fold_pair<3, 2>(g, c, v, fp[3][2], up[3][2]);
}

// x-y modes of plane zz of this thread's four node columns, from a staged slot
template <typename T>
__device__ __forceinline__ void slot_modes(const T* __restrict__ slot, int i, int j, int zz, T (&a)[4][3]) {
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    const T* b = slot + cc * LBX * LBY * 4 + zz;
    T m[4];
    xy4(b[(j * LBX + i) * 4], b[(j * LBX + i + 1) * 4], b[((j + 1) * LBX + i) * 4],
        b[((j + 1) * LBX + i + 1) * 4], m);
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q][cc] = m[q];
  }
}

// The patch cells of a chunk in one go: f^ = K^ v with each cell's dense corner-parity matrix (patch_m,
// row by row), the block's threads sharing the modes (a thread per cell and component) and the
// rows (a thread per row), so their loads of the matrices are in flight together.
template <typename T>
__device__ __forceinline__ void patch_products(L1Smem<T>& sm, const T* us, const T* un, const T* __restrict__ pm) {
  const int n = min(sm.npatch, L1_PATCH);
  constexpr int H = sizeof(T) == 4 ? 3 : 1;   // rows a thread has in flight
  T k[H][24];
  // the first rows' loads are issued before the modes are formed
  auto load = [&](int e0) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int e = min(e0 + h * LCOL, 24 * n - 1), q = e / 24, r = e - 24 * q;
      const T* row = pm + (long long)sm.pmat[q] * 576 + 24 * r;
#pragma unroll
      for (int c = 0; c < 24; c += 4) lp_ldg4(row + c, &k[h][c]);
    }
  };
  if (n > 0) load(threadIdx.x);
  for (int e = threadIdx.x; e < 3 * n; e += LCOL) {
    const int q = e / 3, cc = e - 3 * q, th = sm.pcell[q] >> 2, t = sm.pcell[q] & 3;
    const int at = (cc * LBY + th / LX) * LBX + th % LX;
    T a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int col = 4 * (at + cx_(i) + LBX * cy_(i)), z = t + cz_(i);
      a[i] = z < 4 ? us[col + z] : (un ? un[col] : T(0));
    }
    lp_walsh8(a);
#pragma unroll
    for (int m = 0; m < 8; ++m) sm.pv[q][3 * m + cc] = a[m];
  }
  __syncthreads();
  for (int e0 = threadIdx.x; e0 < 24 * n; e0 += H * LCOL) {
    if (e0 >= H * LCOL) load(e0);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int e = e0 + h * LCOL;
      if (e < 24 * n) {
        const T* v = sm.pv[e / 24];
        T f0 = T(0), f1 = T(0);
#pragma unroll
        for (int c = 0; c < 24; c += 2) {
          f0 += k[h][c] * v[c];
          f1 += k[h][c + 1] * v[c + 1];
        }
        sm.pf[e / 24][e % 24] = f0 + f1;
      }
    }
  }
  __syncthreads();
}

// The dense product of a patch cell that found no place among those (more than L1_PATCH in a chunk),
// by its own thread: the same sums in the same order, so which cells are placed changes no bit.
template <typename T>
__device__ __noinline__ void patch_alone(const T* __restrict__ pm, int patch, const T* v, T* f) {
#pragma unroll 1
  for (int r = 0; r < 24; ++r) {
    T f0 = T(0), f1 = T(0);
#pragma unroll 1
    for (int c = 0; c < 24; c += 2) {
      f0 += __ldg(pm + (long long)patch * 576 + 24 * r + c) * v[c];
      f1 += __ldg(pm + (long long)patch * 576 + 24 * r + c + 1) * v[c + 1];
    }
    f[r] = f0 + f1;
  }
}

// Level-1 operator, u zero on masked dofs: out = m K u (MODE 0), or a degree-2 Chebyshev update formed
// where K u is stored (modes 1..3 as lpb_apply_fine_cheb_f32's, the vector kernels' expressions).
//
// What bounds it: instruction issue. A cell's product is 279 products in rows of 8 to 19 (about 560
// floating-point instructions with the modes and the corner sums) and keeps 230 registers busy, so two
// warps per scheduler issue them; what can be cut is the waiting and the rest: two blocks of four
// warps per SM, whose barriers do not meet, instead of one of eight; one barrier per chunk; masks and
// patch indices loaded a chunk ahead of their use; the patch cells (dense products) shared by a
// block's threads in the same launch, or in one behind it (launch_level1 says when); units split evenly over the SMs
// instead of whole z segments. Sharing a
// cell's rows between two warps (half the registers, twice the warps) ran 1.2x slower: the modes and
// indices formed twice cost more issue slots than the extra warps filled.
//
// A block runs 16 x 8 cell columns (15 x 7 owned node columns; halo on the low sides) in persistent
// segments of (tile, chunk) units, split evenly by weight (a tile with patch cells weighs more);
// a segment recomputes the top cell of the chunk below it. u and the Walsh coefficients arrive by
// TMA into a two-stage ring; the next chunk's first plane is waited for only when the last cell of a
// chunk needs it. Waits are bounded and a block that gives up sets *err.
template <typename T, int MODE>
__global__ void __launch_bounds__(LCOL, 2)
k_level1(const __grid_constant__ L1Maps maps, const __grid_constant__ L1Split split, T* __restrict__ out,
         const T* __restrict__ wc, const int* __restrict__ pid, const T* __restrict__ pm,
         const uint8_t* __restrict__ mask, const __grid_constant__ G1<T> gc, LpGrid g, int nchunks, int* __restrict__ err,
         const L1Cheb<T> ch, const L1Box pbox, const L1Nodes apart) {
  // nothing global is touched before lp_after_launch: the set-up overlaps the launch ahead
  extern __shared__ unsigned char wsm_raw[];
  const uint32_t raw_off = lp_smem_addr(wsm_raw);
  L1Smem<T>& sm = *reinterpret_cast<L1Smem<T>*>(wsm_raw + ((1024u - (raw_off & 1023u)) & 1023u));
  constexpr bool staged_w = sizeof(T) == 4;
  const int tid = threadIdx.x;
  const int i = tid % LX, j = tid / LX;
  const int gx = (g.NX() + LX - 2) / (LX - 1);
  const long long u0 = split.u0[blockIdx.x], u1 = split.u0[blockIdx.x + 1];
  constexpr uint32_t UBYTES = 3 * LBX * LBY * 4 * sizeof(T);
  constexpr uint32_t WBYTES = staged_w ? 32 * LCOL * sizeof(T) : 0;
  if (u0 >= u1) {
    lp_after_launch();
    return;
  }
  __shared__ int bad;
  if (tid == 0) {
    int code = 0;
    uint32_t so = 0, sw = 0;
    for (int s = 0; s < LST; ++s) {
      so |= lp_smem_addr(sm.u[s].v);
      sw |= lp_smem_addr(sm.w[s]);
    }
    if ((so & 127) || (staged_w && (sw & 1023))) code = 20;
    else if (staged_w && (reinterpret_cast<uintptr_t>(&maps.w) & 63)) code = 26;
    else if (reinterpret_cast<uintptr_t>(&maps.u) & 63) code = 21;
    else if ((MODE == 0 || apart.hx > apart.x) && (reinterpret_cast<uintptr_t>(out) & 15)) code = 22;
    else if (MODE != 0 && ((reinterpret_cast<uintptr_t>(ch.x) | reinterpret_cast<uintptr_t>(ch.r) |
                            reinterpret_cast<uintptr_t>(ch.d) | reinterpret_cast<uintptr_t>(ch.b) |
                            reinterpret_cast<uintptr_t>(ch.dinv)) & 15)) code = 27;
    else if (lp_smem_addr(&sm.full[0]) & 7) code = 23;
    else if (reinterpret_cast<uintptr_t>(mask) & 3) code = 24;
    else if ((reinterpret_cast<uintptr_t>(wc) & 15) || (reinterpret_cast<uintptr_t>(pid) & 15)) code = 25;
    bad = code;
    if (code) atomicExch(err, code);
  }
  __syncthreads();
  if (bad) {
    lp_after_launch();
    return;
  }
  // thread 0 issues the block's loads in order: its segment, the loads issued in it and in all
  int total = 0, issued = 0, pk = 0;
  long long pu = u0;
  LpSeg ps = lp_seg(u0, u1, nchunks);
  if (tid == 0) {
    for (long long u = u0; u < u1;) {
      const LpSeg q = lp_seg(u, u1, nchunks);
      total += q.nload;
      u += q.ce - q.cb;
    }
    for (int s = 0; s < LST; ++s) lp_mbar_init(&sm.full[s], 1);
    lp_fence_barrier_init();
  }
  __syncthreads();
  lp_after_launch();
  T cs_s = T(0), cs_c1 = T(0), cs_c2 = T(0);
  if constexpr (MODE != 0) {
    cs_s = (T)ch.coef[1];
    cs_c1 = (T)ch.coef[2];
    cs_c2 = (T)ch.coef[3];
  }
  auto issue_next = [&]() {
    if (pk == ps.nload) {
      pu += ps.ce - ps.cb;
      ps = lp_seg(pu, u1, nchunks);
      pk = 0;
    }
    const int s = issued % LST;
    const int x0 = (ps.tile % gx) * (LX - 1), y0 = (ps.tile / gx) * (LY - 1);
    lp_mbar_expect_tx(&sm.full[s], UBYTES + WBYTES);
    lp_tma_load_4d(sm.u[s].v, &maps.u, 4 * (x0 - 1), y0 - 1, ps.cstart + pk, 3 * (int)blockIdx.y, &sm.full[s]);
    if constexpr (staged_w) lp_tma_load_4d(sm.w[s], &maps.w, 0, x0 - 1, y0 - 1, ps.cstart + pk, &sm.full[s]);
    ++pk;
    ++issued;
  };
  if (tid == 0)
    while (issued < LST && issued < total) issue_next();
  const long long wstride = 32LL * g.nx * g.ny, cs = g.comp_stride(), zcs = g.node_zc_stride();
  const long long co = 3 * cs * blockIdx.y;   // the column's fields (a launch of several right-hand sides)
  bool ok = true, failed = false;
  int n = 0, it = 0;   // the load in hand, chunks processed
  for (long long u = u0; u < u1 && !failed;) {
    const LpSeg sg = lp_seg(u, u1, nchunks);
    u += sg.ce - sg.cb;
    const int x0 = (sg.tile % gx) * (LX - 1), y0 = (sg.tile / gx) * (LY - 1);
    const int cx = x0 - 1 + i, cy = y0 - 1 + j;
    const bool cell_ok = cx >= 0 && cx < g.nx && cy >= 0 && cy < g.ny;
    const T* wcol = wc + (cell_ok ? ((long long)cy * g.nx + cx) * 32 : 0);
    // the tile's cells reach into the box of the patch cells
    const bool tile_patches = pid && x0 - 1 < pbox.hx && x0 - 1 + LX > pbox.x && y0 - 1 < pbox.hy && y0 - 1 + LY > pbox.y;
    const bool writer = i >= 1 && j >= 1 && cx < g.NX() && cy < g.NY();   // owns the node column (cx, cy)
    const bool raw_col = MODE != 0 && cx >= apart.x && cx < apart.hx && cy >= apart.y && cy < apart.hy;
    const long long obase = writer ? g.node(cx, cy, 0) : 0;               // chunk c at obase + c * zcs
    const long long pstride = g.cell_zc_stride();
    const int* pcol = pid + (cell_ok ? g.cell(cx, cy, 0) : 0);
    int4 p_next = make_int4(-1, -1, -1, -1);   // the next chunk's patch cells of this column
    if (tile_patches && cell_ok) p_next = __ldg(reinterpret_cast<const int4*>(pcol + sg.cstart * pstride));
    T up[4][3], a_lo[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) up[q][c] = T(0);
    ok = ok && lp_mbar_wait(&sm.full[n % LST], (n / LST) & 1);
    slot_modes(sm.u[n % LST].v, i, j, sg.cb > sg.cstart ? 3 : 0, a_lo);
    for (int k = 0; k < sg.nproc; ++k, ++n, ++it) {
      const int c = sg.cstart + k;
      const bool halo = c < sg.cb, has_next = k + 1 < sg.nload;
      const int s = n % LST, s1 = (n + 1) % LST;
      const uint32_t mb = writer && !halo ? __ldg(reinterpret_cast<const uint32_t*>(mask + obase + c * zcs)) : 0u;
      const int4 p4 = p_next;   // the column's patch cells
      int4 sl = make_int4(-1, -1, -1, -1);   // and their places in pf
      if (tile_patches && cell_ok && k + 1 < sg.nproc) p_next = __ldg(reinterpret_cast<const int4*>(pcol + (c + 1) * pstride));
      ok = ok && lp_mbar_wait(&sm.full[s], (n / LST) & 1);
      if (tile_patches) {   // uniform across the block
        if (tid == 0) sm.npatch = 0;
        __syncthreads();
        auto place = [&](int p, int t) {
          if (p < 0 || (halo && t < 3)) return -1;
          const int q = atomicAdd(&sm.npatch, 1);   // (the order of the places changes no bit)
          if (q < L1_PATCH) {
            sm.pmat[q] = p;
            sm.pcell[q] = 4 * tid + t;
          }
          return q;
        };
        sl = make_int4(place(p4.x, 0), place(p4.y, 1), place(p4.z, 2), place(p4.w, 3));
        if (has_next) ok = ok && lp_mbar_wait(&sm.full[s1], ((n + 1) / LST) & 1);
        __syncthreads();
        patch_products<T>(sm, sm.u[s].v, has_next ? sm.u[s1].v : nullptr, pm);
      }
      const T* us = sm.u[s].v;
      const T* wch = wcol + (long long)c * wstride;   // this chunk's Walsh run
#pragma unroll 1
      for (int t = halo ? 3 : 0; t < 4; ++t) {
        T cw[8];
        if constexpr (staged_w) {
          // this cell's eight coefficients: two 16-byte reads of the column's swizzled row
          const unsigned char* wb = reinterpret_cast<const unsigned char*>(sm.w[s]);
          const float4 c0 = *reinterpret_cast<const float4*>(wb + lp_swz128((uint32_t)tid * 128u + (uint32_t)t * 32u));
          const float4 c1 = *reinterpret_cast<const float4*>(wb + lp_swz128((uint32_t)tid * 128u + (uint32_t)t * 32u + 16u));
          cw[0] = c0.x; cw[1] = c0.y; cw[2] = c0.z; cw[3] = c0.w;
          cw[4] = c1.x; cw[5] = c1.y; cw[6] = c1.z; cw[7] = c1.w;
        } else {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) cw[kk] = __ldg(wch + t * 8 + kk);
        }
        T a_hi[4][3];
        if (t < 3) {
          slot_modes(us, i, j, t + 1, a_hi);
        } else if (has_next) {
          ok = ok && lp_mbar_wait(&sm.full[s1], ((n + 1) / LST) & 1);
          slot_modes(sm.u[s1].v, i, j, 0, a_hi);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) a_hi[q][cc] = T(0);
        }
        T v[24];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) {
            const T lo = a_lo[q][cc], hi = a_hi[q][cc];
            v[3 * q + cc] = lo + hi;
            v[3 * (q + 4) + cc] = hi - lo;
            a_lo[q][cc] = hi;
          }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) cw[kk] = cell_ok ? cw[kk] : T(0);
        T fp[4][3];
        fold_rows<T>(gc, cw, v, fp, up);
        if (tile_patches) {
          const int slot = t == 0 ? sl.x : t == 1 ? sl.y : t == 2 ? sl.z : sl.w;
          if (slot >= 0) {
            if (slot < L1_PATCH) {
              const T* f = sm.pf[slot];
#pragma unroll
              for (int q = 0; q < 12; ++q) {
                fp[q / 3][q % 3] += f[q] - f[12 + q];
                up[q / 3][q % 3] += f[q] + f[12 + q];
              }
            } else {
              const int patch = t == 0 ? p4.x : t == 1 ? p4.y : t == 2 ? p4.z : p4.w;
              T vv[24], f[24];
#pragma unroll
              for (int q = 0; q < 24; ++q) vv[q] = v[q];
              patch_alone<T>(pm, patch, vv, f);
#pragma unroll
              for (int q = 0; q < 12; ++q) {
                fp[q / 3][q % 3] += f[q] - f[12 + q];
                up[q / 3][q % 3] += f[q] + f[12 + q];
              }
            }
          }
        }
        if (!halo) {
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) {
            const T t0 = fp[0][cc] - fp[2][cc], t1 = fp[1][cc] - fp[3][cc];
            const T t2 = fp[0][cc] + fp[2][cc], t3 = fp[1][cc] + fp[3][cc];
            const T c10 = __shfl_up_sync(0xffffffffu, t0 + t1, 1, LX);
            const T c11 = __shfl_up_sync(0xffffffffu, t2 + t3, 1, LX);
            sm.own[it & 1][cc][t][tid] = (t0 - t1) + c10;
            sm.red[it & 1][cc][t][tid] = (t2 - t3) + c11;
          }
        }
      }
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {
          atomicExch(err, 1);
          // let the loads already issued land before the block exits (bounded as well)
          for (int kk = n; kk < issued; ++kk) lp_mbar_wait(&sm.full[kk % LST], (kk / LST) & 1);
        }
        failed = true;
        break;
      }
      // this chunk's stage is read (its last plane's modes are in registers): the load after the next
      if (tid == 0 && issued < total && issued < n + 1 + LST) issue_next();
      if (halo) continue;   // uniform across the block
      if (!writer) continue;
      const bool raw = raw_col && c >= apart.c && c < apart.hc;
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        T o[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const T val = sm.own[it & 1][cc][t][tid] + sm.red[it & 1][cc][t][tid - LX];
          o[t] = ((mb >> (8 * t + cc)) & 1u) ? val : T(0);
        }
        const long long at = cc * cs + obase + c * zcs, idx = co + at;
        if (MODE == 0 || raw) {
          lp_st4(out + idx, o);
        } else {
          T dv[4], d[4];
          lp_ld4(ch.dinv + at, dv);
          if constexpr (MODE == 1) {
            T b[4], x[4];
            lp_ld4(ch.d + idx, d);
            lp_ld4(ch.b + idx, b);
#pragma unroll
            for (int t = 0; t < 4; ++t) x[t] = lp_cheb2_zero_v(d[t], b[t], o[t], dv[t], cs_c1, cs_c2);
            lp_st4(ch.x + idx, x);
          } else if constexpr (MODE == 2) {
            T b[4], r[4];
            lp_ld4(ch.b + idx, b);
#pragma unroll
            for (int t = 0; t < 4; ++t) lp_residual_scaled_v(b[t], o[t], dv[t], cs_s, r[t], d[t]);
            lp_st4(ch.r + idx, r);
            lp_st4(ch.d + idx, d);
          } else {
            T x[4], r[4], y[4];
            lp_ld4(ch.x + idx, x);   // read, then written, by this thread
            lp_ld4(ch.d + idx, d);
            lp_ld4(ch.r + idx, r);
#pragma unroll
            for (int t = 0; t < 4; ++t) y[t] = lp_cheb2_v(x[t], d[t], r[t], o[t], dv[t], cs_c1, cs_c2);
            lp_st4(ch.x + idx, y);
          }
        }
      }
    }
    // the segment's last load (the chunk above) was only read as the next chunk's first plane
    if (!failed && sg.nload > sg.nproc) {
      ++n;
      __syncthreads();
      if (tid == 0 && issued < total && issued < n + LST) issue_next();
    }
  }
}

// a patch cell's matrix in the corner-parity basis, K^ = T K T^T / 64 with T = kron(H, I3); one block per
// cell, float64 inside
template <typename T>
__global__ void __launch_bounds__(192) k_patch_modal(T* __restrict__ pm, const T* __restrict__ pk) {
  lp_after_launch();
  __shared__ double a[24][25], b[24][25];
  const long long p = blockIdx.x;
  for (int e = threadIdx.x; e < 576; e += 192) a[e / 24][e % 24] = (double)pk[p * 576 + e];
  __syncthreads();
  // rows, then columns: b[3 m + c][.] = sum_k H[m][k] a[3 k + c][.]
  for (int e = threadIdx.x; e < 576; e += 192) {
    const int r = e / 24, c = e % 24, m = r / 3, cc = r % 3;
    double s = 0.0;
    for (int k = 0; k < 8; ++k) s += lp_walsh_h(m, k) * a[3 * k + cc][c];
    b[r][c] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 576; e += 192) {
    const int c = e / 24, r = e % 24, m = c / 3, cc = c % 3;
    double s = 0.0;
    for (int k = 0; k < 8; ++k) s += lp_walsh_h(m, k) * b[r][3 * k + cc];
    pm[p * 576 + r * 24 + c] = (T)(s / 64.0);
  }
}

// Patch cells (weights zero, an explicit masked matrix) after a march without them, over the nodes of a box of
// columns and whole chunks: MODE 0 out += m * sum of their rows times u; modes 1..3 the Chebyshev update from
// out, which the march left there, and that sum (the vector kernels' expressions). All they read but out is
// older than the march, the launch ahead, so only the finish waits for that one. Two forms, the same bits:
//   k_patch_quads   a warp per P planes of a quad (a node column's four planes of a chunk): its lanes load the
//                   patch indices around and split the 8 cells x 24 columns of each solved node that a
//                   patch cell touches; three lanes finish the components
//   k_patch_nodes   for boxes of which such cells are a small part (supports on opposite faces, scattered ones):
//                   a thread per quad looks for them and lists their nodes, the block's warps take the
//                   listed nodes, and a thread per quad and component finishes
// Bound by the latency of their loads. A float32 smoothing (two updates) of 96 x 48 x 48 level-1 cells, march
// included, against a warp per node of the box: held on two opposite x faces 74 us (221), at 40 points 65
// (205), on one z face 53 (61), on one x face 45 (45).
constexpr int PN_QUADS = 32;     // most quads of a block of k_patch_nodes
constexpr int PN_THREADS = 128;
constexpr int PQ_THREADS = 256;
// quads from which a box takes k_patch_nodes (float32 smoothing, k_patch_quads and k_patch_nodes: two x faces of 64 x
// 32 x 32 cells, 19305 quads, 43.1 and 42.9 us; of 96 x 48 x 48, 61789 quads, 96.4 and 71.4)
constexpr long long PN_FROM = 32768;

template <int P, typename T>
__device__ __forceinline__ void ldcg_planes(const T* p, T (&v)[P]) {
  if constexpr (P == 1) {
    v[0] = __ldcg(p);
  } else if constexpr (sizeof(T) == 4) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}

// a warp's part of the sum at node (x, y, z): lane -> (cell corner kk = lane / 4, column block of 6 = lane % 4),
// p the patch cell at that corner (-1: none); u: the column's field
template <typename T>
__device__ __forceinline__ void patch_node_part(T (&a)[3], const T* __restrict__ u, const T* __restrict__ pk, const LpGrid& g,
                                                int x, int y, int z, int p) {
  a[0] = a[1] = a[2] = T(0);
  if (p < 0) return;
  const int lane = threadIdx.x & 31, kk = lane >> 2, cb = lane & 3;
  const int cx = x - cx_(kk), cy = y - cy_(kk), cz = z - cz_(kk);
  const T* kp = pk + (long long)p * 576;
#pragma unroll
  for (int c6 = 0; c6 < 6; ++c6) {
    const int col = 6 * cb + c6, q2 = col / 3, c2 = col % 3;
    const T uv = __ldcg(u + c2 * g.comp_stride() + g.node(cx + cx_(q2), cy + cy_(q2), cz + cz_(q2)));
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) a[cc] += __ldcg(kp + (3 * kk + cc) * 24 + col) * uv;
  }
}
// the warp's sum of component lane (of lane 0..2)
template <typename T>
__device__ __forceinline__ T patch_node_sum(T (&a)[3]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int cc = 0; cc < 3; ++cc)
    for (int o = 16; o > 0; o >>= 1) a[cc] += __shfl_xor_sync(0xffffffffu, a[cc], o);
  return lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
}

// what a component's finish of P planes reads beside out, and the finish: ad = out with the sums added
template <typename T, int MODE, int P>
struct PatchFinish {
  T dv[P], v0[P], v1[P], v2[P], s, c1, c2;
  __device__ __forceinline__ void load(const L1Cheb<T>& ch, long long at, long long i) {
    if constexpr (MODE != 0) {
      s = (T)__ldcg(ch.coef + 1);
      c1 = (T)__ldcg(ch.coef + 2);
      c2 = (T)__ldcg(ch.coef + 3);
      ldcg_planes<P>(ch.dinv + at, dv);
      ldcg_planes<P>((MODE == 1 ? ch.d : MODE == 2 ? ch.b : ch.x) + i, v0);
      if constexpr (MODE != 2) ldcg_planes<P>((MODE == 1 ? ch.b : ch.d) + i, v1);
      if constexpr (MODE == 3) ldcg_planes<P>(ch.r + i, v2);
    }
  }
  static __device__ __forceinline__ void save(T* p, const T (&v)[P]) {
    if constexpr (P == 1) *p = v[0];
    else lp_st4(p, v);
  }
  __device__ __forceinline__ void store(T* __restrict__ out, const L1Cheb<T>& ch, long long i, const T (&ad)[P]) const {
    T a[P], b[P];
#pragma unroll
    for (int z = 0; z < P; ++z) {
      if constexpr (MODE == 1) a[z] = lp_cheb2_zero_v(v0[z], v1[z], ad[z], dv[z], c1, c2);
      else if constexpr (MODE == 2) lp_residual_scaled_v(v0[z], ad[z], dv[z], s, a[z], b[z]);
      else if constexpr (MODE == 3) a[z] = lp_cheb2_v(v0[z], v1[z], v2[z], ad[z], dv[z], c1, c2);
    }
    if constexpr (MODE == 0) {
      save(out + i, ad);
    } else if constexpr (MODE == 2) {
      save(ch.r + i, a);
      save(ch.d + i, b);
    } else {
      save(ch.x + i, a);
    }
  }
};

template <typename T, int MODE, int P>
__global__ void __launch_bounds__(PQ_THREADS)
k_patch_quads(T* __restrict__ out, const T* __restrict__ u, const int* __restrict__ pid, const T* __restrict__ pk,
              const uint8_t* __restrict__ mask, LpGrid g, int bx0, int by0, int bc0, int bnx, int bny, int bnc,
              L1Cheb<T> ch) {
  constexpr int H = sizeof(T) == 4 ? P : (P + 1) / 2;   // nodes whose loads are in flight together
  const int item = (int)((blockIdx.x * (unsigned)PQ_THREADS + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const int quad = item / (4 / P), zb = (item % (4 / P)) * P;   // the planes zb .. zb + P - 1 of the quad
  if (quad >= bnx * bny * bnc) {
    lp_after_launch();
    return;
  }
  const long long cs = g.comp_stride(), co = 3 * cs * blockIdx.y;   // (the column)
  const int x = bx0 + quad % bnx, y = by0 + (quad / bnx) % bny, c = bc0 + quad / (bnx * bny);
  const long long n = g.node(x, y, 4 * c);
  const uint32_t mb = __ldcg(reinterpret_cast<const unsigned*>(mask + n));
  // lane -> cell of column lane % 4 (x - bit 0, y - bit 1) and plane 4 c - 1 + lane / 4
  int pc = -1;
  {
    const int cx = x - (lane & 1), cy = y - ((lane >> 1) & 1), cz = 4 * c - 1 + (lane >> 2);
    if (lane < 20 && cx >= 0 && cy >= 0 && cz >= 0 && cx < g.nx && cy < g.ny && cz < g.nz) pc = __ldcg(pid + g.cell(cx, cy, cz));
  }
  const unsigned have = __ballot_sync(0xffffffffu, pc >= 0);
  unsigned todo = 0;   // the planes whose node is solved and touched: by the cells of its plane or of the one below
#pragma unroll
  for (int z = 0; z < P; ++z)
    if (((mb >> (8 * (zb + z))) & 7) && ((have >> (4 * (zb + z))) & 0xff)) todo |= 1u << z;
  T sum[P] = {};   // lane cc < 3: component cc of each plane
  if (todo) {
#pragma unroll
    for (int z0 = 0; z0 < P; z0 += H) {
      T a[H][3];
#pragma unroll
      for (int h = 0; h < H; ++h) {   // (the cell at corner kk: one column and plane down per set bit)
        const int kk = lane >> 2, z = zb + z0 + h, p = __shfl_sync(0xffffffffu, pc, (kk & 3) + 4 * (z + 1 - (kk >> 2)));
        patch_node_part<T>(a[h], u + co, pk, g, x, y, 4 * c + z, (todo >> (z0 + h)) & 1 ? p : -1);
      }
#pragma unroll
      for (int h = 0; h < H; ++h)
        if ((todo >> (z0 + h)) & 1) sum[z0 + h] = patch_node_sum<T>(a[h]);
    }
  }
  const int cc = lane < 3 ? lane : 0;
  const long long at = cc * cs + n + zb, i = co + at;
  PatchFinish<T, MODE, P> fin;
  fin.load(ch, at, i);
  lp_wait_prior();
  lp_release_next();
  if (lane >= 3 || (MODE == 0 && !todo)) return;
  T ad[P];
  if constexpr (P == 1) ad[0] = out[i];
  else lp_ld4(out + i, ad);
#pragma unroll
  for (int z = 0; z < P; ++z)
    if (((todo >> z) & 1) && ((mb >> (8 * (zb + z) + cc)) & 1)) ad[z] += sum[z];
  fin.store(out, ch, i, ad);
}

template <typename T, int MODE>
__global__ void __launch_bounds__(PN_THREADS)
k_patch_nodes(T* __restrict__ out, const T* __restrict__ u, const int* __restrict__ pid, const T* __restrict__ pk,
              const uint8_t* __restrict__ mask, LpGrid g, int bx0, int by0, int bc0, int bnx, int bny, int bnc, int quads,
              unsigned stride, L1Cheb<T> ch) {
  __shared__ T sums[4 * PN_QUADS][3];
  __shared__ int cells[PN_QUADS][20];      // column k (x - bit 0, y - bit 1) and plane 4 c - 1 + z at 5 k + z
  __shared__ uint8_t touched[PN_QUADS];    // a bit per plane
  __shared__ uint8_t list[4 * PN_QUADS];   // 4 quad + plane
  __shared__ int count;
  const int total = bnx * bny * bnc, tid = threadIdx.x, lane = tid & 31;
  const long long cs = g.comp_stride(), co = 3 * cs * blockIdx.y;   // (the column)
  // this thread's quad and component (a component past the third: none)
  const int first = (int)((unsigned long long)blockIdx.x * stride % gridDim.x) * quads;
  const int q = tid & (quads - 1), cc = tid / quads, quad = first + q;
  const bool in = cc < 3 && quad < total;
  const int x = bx0 + quad % bnx, y = by0 + (quad / bnx) % bny, c = bc0 + quad / (bnx * bny);
  const long long n = in ? g.node(x, y, 4 * c) : 0, at = cc * cs + n, i = co + at;
  if (tid == 0) count = 0;
  __syncthreads();
  const uint32_t mb = in ? __ldcg(reinterpret_cast<const unsigned*>(mask + n)) : 0;
  if (cc == 0) {
    unsigned bits = 0;   // bit z + 1: a patch cell in plane 4 c + z of the columns around
    int p[4][5];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int cx = x - (k & 1), cy = y - (k >> 1);
      const bool col = in && cx >= 0 && cy >= 0 && cx < g.nx && cy < g.ny;
      const int* pc = pid + (col ? g.cell(cx, cy, 4 * c) : 0);
      p[k][0] = col && c > 0 ? __ldcg(pc - g.cell_zc_stride() + 3) : -1;
#pragma unroll
      for (int z = 0; z < 4; ++z) p[k][z + 1] = col && 4 * c + z < g.nz ? __ldcg(pc + z) : -1;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int z = 0; z < 5; ++z) {
        cells[q][5 * k + z] = p[k][z];
        bits |= (p[k][z] >= 0 ? 1u : 0u) << z;
      }
    bits = (bits | bits >> 1) & 15;   // a node: the cells of its plane and of the one below
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      if (!((mb >> (8 * z)) & 7)) bits &= ~(1u << z);
      if ((bits >> z) & 1) list[atomicAdd(&count, 1)] = 4 * q + z;   // (their order changes no bit)
    }
    touched[q] = bits;
  }
  PatchFinish<T, MODE, 4> fin;
  if (in) fin.load(ch, at, i);
  __syncthreads();
  const int listed = count;
  for (int e = tid >> 5; e < listed; e += PN_THREADS / 32) {
    const int node = list[e], nq = first + (node >> 2), z = node & 3;
    const int kk = lane >> 2;
    T a[3];
    patch_node_part<T>(a, u + co, pk, g, bx0 + nq % bnx, by0 + (nq / bnx) % bny, 4 * (bc0 + nq / (bnx * bny)) + z,
                       cells[node >> 2][5 * (kk & 3) + z + 1 - (kk >> 2)]);
    const T sum = patch_node_sum<T>(a);
    if (lane < 3) sums[node][lane] = sum;
  }
  if (listed) __syncthreads();   // the sums are there
  lp_wait_prior();
  lp_release_next();
  if (!in || (MODE == 0 && !touched[q])) return;
  T ad[4];
  lp_ld4(out + i, ad);
#pragma unroll
  for (int z = 0; z < 4; ++z)
    if (((touched[q] >> z) & 1) && ((mb >> (8 * z + cc)) & 1)) ad[z] += sums[4 * q + z][cc];
  fin.store(out, ch, i, ad);
}

// ---- explicit levels: packed symmetric matrices, entry-major ---------------------------------
__host__ __device__ __forceinline__ int sym_index(int i, int j) {  // i <= j
  return i * 24 - (i * (i - 1)) / 2 + (j - i);
}

// A block takes 32 consecutive cells, a lane per cell, and its eight warps share the 300 entries of their
// matrices (entry p of consecutive cells coalesced): each warp loads its 37 or 38 entries before the
// corner values are staged, forms its part of the 24 corner forces, and the parts are added in order. Where the
// matrices are older than the launch ahead (lpb_pack_sym_* see to it) they are loaded while it runs; where the
// caller may have written them by the launch ahead, the launch is in stream order.
// What bounds it is how many of those loads are in flight: with one thread per cell (a few
// thousand cells on a coarse level) the apply of 32 x 16 x 16 cells took 25.7 us in float64, shared by
// eight warps 11.7 us, of 64 x 32 x 32 cells 69 and 50 us (157 MB of entries from DRAM: 22 us); with the
// loads ahead 9.3 us.
constexpr int EX_WARPS = 8;
template <typename T>
struct ExCells {
  T u[24][32];
  T part[EX_WARPS][24][32];
};
template <int W, typename T>
__device__ __forceinline__ void sym_part(const T* __restrict__ kc, long long ncp, T (&k)[38]) {
  constexpr int LO = 300 * W / EX_WARPS, HI = 300 * (W + 1) / EX_WARPS;
#pragma unroll
  for (int p = LO; p < HI; ++p) k[p - LO] = __ldcg(kc + (long long)p * ncp);
}
template <int W, typename T>
__device__ __forceinline__ void sym_forces(const T (&k)[38], const T (&u)[24][32], T (&f)[24]) {
  constexpr int LO = 300 * W / EX_WARPS, HI = 300 * (W + 1) / EX_WARPS;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < 24; ++a)
#pragma unroll
    for (int b = a; b < 24; ++b) {
      const int p = sym_index(a, b);
      if (p < LO || p >= HI) continue;
      f[a] += k[p - LO] * u[b][lane];
      if (b != a) f[b] += k[p - LO] * u[a][lane];
    }
}
template <int W, typename T>
__device__ __forceinline__ void sym_warp(ExCells<T>& sm, const T* __restrict__ kc, long long ncp,
                                         const T* __restrict__ u, long long cs, bool in) {
  const int lane = threadIdx.x & 31;
  T k[38], f[24];
  sym_part<W, T>(kc, ncp, k);
  lp_wait_prior();
  lp_release_next();
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) sm.u[3 * W + cc][lane] = in ? u[cc * cs] : T(0);   // corner W
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 24; ++r) f[r] = T(0);
  sym_forces<W, T>(k, sm.u, f);
#pragma unroll
  for (int r = 0; r < 24; ++r) sm.part[W][r][lane] = f[r];
}

template <typename T>
__global__ void __launch_bounds__(32 * EX_WARPS)
k_explicit_cells(T* __restrict__ ft, const T* __restrict__ u, const T* __restrict__ kp, LpGrid g) {
  extern __shared__ __align__(16) unsigned char ex_raw[];
  ExCells<T>& sm = *reinterpret_cast<ExCells<T>*>(ex_raw);
  const long long ncp = g.cells_padded(), cs = g.comp_stride();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long c = blockIdx.x * 32LL + lane;
  int x = 0, y = 0, z = 0;
  const bool in = c < ncp && g.cell_at(c, x, y, z);
  // corner k at n0 + x step (4) + y step (4 NX) + z step (1, or to the next chunk): warp k stages corner k
  const long long n0 = in ? g.node(x, y, z) : 0;
  const long long oy = 4LL * g.NX(), oz = (z & 3) == 3 ? g.node_zc_stride() - 3 : 1;
  const long long n = n0 + (w & 1 ? 4 : 0) + (w & 2 ? oy : 0) + (w & 4 ? oz : 0);
  const T* kc = kp + (in ? c : 0);
  switch (w) {
    case 0: sym_warp<0, T>(sm, kc, ncp, u + n, cs, in); break;
    case 1: sym_warp<1, T>(sm, kc, ncp, u + n, cs, in); break;
    case 2: sym_warp<2, T>(sm, kc, ncp, u + n, cs, in); break;
    case 3: sym_warp<3, T>(sm, kc, ncp, u + n, cs, in); break;
    case 4: sym_warp<4, T>(sm, kc, ncp, u + n, cs, in); break;
    case 5: sym_warp<5, T>(sm, kc, ncp, u + n, cs, in); break;
    case 6: sym_warp<6, T>(sm, kc, ncp, u + n, cs, in); break;
    default: sym_warp<7, T>(sm, kc, ncp, u + n, cs, in); break;
  }
  __syncthreads();
  if (!in) return;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int r = 3 * w + q;
    T s = sm.part[0][r][lane];
#pragma unroll
    for (int p = 1; p < EX_WARPS; ++p) s += sm.part[p][r][lane];
    ft[(long long)r * ncp + c] = s;
  }
}

// ---- explicit levels in the corner-parity basis ------------------------------------------------
// A Galerkin level's cell matrix K, in the modes of its cell (K^ = T K T^T / 64, T = kron(H, I3)),
// has the level-1 pattern: 279 non-zeros, 150 in the upper triangle, at every level of the plain
// hierarchy (the pattern is kept by the child Galerkin product). Those cells are stored as the
// 150 entries (entry-major, (150, cells)) and applied as f = T^T (K^ (T u)): half the bytes of the
// 300-entry node-basis form. Cells with weight off the pattern (children carrying masked patch
// matrices) are listed and applied from the node-basis form.
constexpr int MODAL_UP = 150;
__constant__ int c_mup_r[MODAL_UP] = {3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5, 5, 5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 8, 8, 8, 8, 8, 8, 8, 8, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 12, 12, 12, 12, 12, 12, 13, 13, 13, 13, 13, 13, 14, 14, 14, 14, 14, 14, 14, 14, 15, 15, 15, 15, 15, 15, 15, 15, 16, 16, 16, 16, 16, 16, 16, 17, 17, 17, 17, 17, 17, 17, 18, 18, 18, 18, 19, 19, 19, 19, 19, 20, 20, 20, 20, 21, 21, 21, 22, 22, 23};
__constant__ int c_mup_c[MODAL_UP] = {3, 7, 9, 10, 14, 15, 17, 19, 20, 21, 22, 23, 4, 6, 9, 10, 16, 18, 21, 22, 5, 11, 12, 15, 17, 18, 21, 23, 6, 9, 10, 16, 18, 21, 22, 7, 9, 10, 14, 15, 17, 19, 20, 21, 22, 23, 8, 11, 13, 16, 19, 20, 22, 23, 9, 10, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 10, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 11, 12, 13, 15, 16, 17, 18, 19, 20, 21, 22, 23, 12, 15, 17, 18, 21, 23, 13, 16, 19, 20, 22, 23, 14, 15, 17, 19, 20, 21, 22, 23, 15, 17, 18, 19, 20, 21, 22, 23, 16, 18, 19, 20, 21, 22, 23, 17, 18, 19, 20, 21, 22, 23, 18, 21, 22, 23, 19, 20, 21, 22, 23, 20, 21, 22, 23, 21, 22, 23, 22, 23, 23};
// bit i % 32 of word i / 32: entry i = 24 r + c of K^ is on the pattern
__constant__ unsigned c_mpat[18] = {0x00000000u, 0x00000000u, 0xfac68800u, 0x20650650u, 0x0650a698u, 0xfac68865u, 0xd8d92900u, 0xc6d8ffc6u, 0xffb920ffu, 0x00a69820u, 0xc688d929u, 0xfedea8fau, 0xa8fd2f50u, 0x9e70fedeu, 0xfbef88e7u, 0xf8fbef88u, 0xefd8ffdeu, 0xffffa8ffu};
#define MUP_ROWS {3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5, 5, 5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 8, 8, 8, 8, 8, 8, 8, 8, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 12, 12, 12, 12, 12, 12, 13, 13, 13, 13, 13, 13, 14, 14, 14, 14, 14, 14, 14, 14, 15, 15, 15, 15, 15, 15, 15, 15, 16, 16, 16, 16, 16, 16, 16, 17, 17, 17, 17, 17, 17, 17, 18, 18, 18, 18, 19, 19, 19, 19, 19, 20, 20, 20, 20, 21, 21, 21, 22, 22, 23}
#define MUP_COLS {3, 7, 9, 10, 14, 15, 17, 19, 20, 21, 22, 23, 4, 6, 9, 10, 16, 18, 21, 22, 5, 11, 12, 15, 17, 18, 21, 23, 6, 9, 10, 16, 18, 21, 22, 7, 9, 10, 14, 15, 17, 19, 20, 21, 22, 23, 8, 11, 13, 16, 19, 20, 22, 23, 9, 10, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 10, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 11, 12, 13, 15, 16, 17, 18, 19, 20, 21, 22, 23, 12, 15, 17, 18, 21, 23, 13, 16, 19, 20, 22, 23, 14, 15, 17, 19, 20, 21, 22, 23, 15, 17, 18, 19, 20, 21, 22, 23, 16, 18, 19, 20, 21, 22, 23, 17, 18, 19, 20, 21, 22, 23, 18, 21, 22, 23, 19, 20, 21, 22, 23, 20, 21, 22, 23, 21, 22, 23, 22, 23, 23}

__device__ __forceinline__ float walsh_h(int m, int k) {
  float v = 1.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if ((m >> a) & 1) v *= ((k >> a) & 1) ? 1.0f : -1.0f;
  return v;
}

// one warp per cell: K^ of the cell's (24 x 24) matrix in float64, its symmetric part on the
// pattern into km; a cell with off-pattern weight above tol of its largest entry is listed
template <typename Ti>
__global__ void __launch_bounds__(128) k_pack_modal(float* __restrict__ km, int* __restrict__ glist,
                                                    int* __restrict__ gcount, float* __restrict__ kpc,
                                                    const Ti* __restrict__ k, long long ncp, double tol) {
  lp_after_launch();
  __shared__ double sk[4][576];
  __shared__ double sa[4][576];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* K = sk[w];
  double* A = sa[w];
  for (long long cell = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; cell < ncp;
       cell += (long long)gridDim.x * (blockDim.x >> 5)) {
    for (int i = lane; i < 576; i += 32) K[i] = (double)k[cell * 576 + i];
    __syncwarp();
    // A = T K
    for (int i = lane; i < 576; i += 32) {
      const int r = i / 24, c = i % 24, mr = r / 3, cr = r % 3;
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) s += (double)walsh_h(mr, q) * K[(3 * q + cr) * 24 + c];
      A[i] = s;
    }
    __syncwarp();
    // K^ = A T^T / 64 into K (reused)
    double amax = 0.0, off = 0.0;
    for (int i = lane; i < 576; i += 32) {
      const int r = i / 24, c = i % 24, mc = c / 3, cc = c % 3;
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) s += A[r * 24 + 3 * q + cc] * (double)walsh_h(mc, q);
      s /= 64.0;
      K[i] = s;
      amax = fmax(amax, fabs(s));
    }
    __syncwarp();
    for (int i = lane; i < 576; i += 32)
      if (!((c_mpat[i >> 5] >> (i & 31)) & 1u)) off = fmax(off, fabs(K[i]));
    for (int o = 16; o > 0; o >>= 1) {
      amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      off = fmax(off, __shfl_xor_sync(0xffffffffu, off, o));
    }
    const bool general = off > tol * amax;
    for (int p = lane; p < MODAL_UP; p += 32) {
      const int r = c_mup_r[p], c = c_mup_c[p];
      // a listed cell's entries are zero, its entry 0 a NaN marker the apply skips it by
      km[(long long)p * ncp + cell] =
          general ? (p == 0 ? __int_as_float(0x7fc00001) : 0.0f) : (float)(0.5 * (K[r * 24 + c] + K[c * 24 + r]));
    }
    if (general) {   // listed: the node-basis symmetric part, cell-major, at the cell's slot
      int slot = 0;
      if (lane == 0) slot = atomicAdd(gcount, 1);
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (lane == 0) glist[slot] = (int)cell;
      for (int p = lane; p < 300; p += 32) {
        int a = 0, rem = p;
        while (rem >= 24 - a) { rem -= 24 - a; ++a; }
        const int b2 = a + rem;
        kpc[(long long)slot * 300 + p] =
            (float)(0.5 * ((double)k[cell * 576 + a * 24 + b2] + (double)k[cell * 576 + b2 * 24 + a]));
      }
    }
    __syncwarp();
  }
}

// in-place a[k] <- sum_m H[m][k] a[m] (the transpose of lp's Walsh transform H a)
__device__ __forceinline__ void walsh8t(float (&a)[8]) {
#pragma unroll
  for (int b = 1; b < 8; b <<= 1)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (!(k & b)) {
        const float lo = a[k], hi = a[k | b];
        a[k] = lo - hi;
        a[k | b] = lo + hi;
      }
}

__device__ __forceinline__ void walsh8(float (&a)[8]) {
#pragma unroll
  for (int b = 1; b < 8; b <<= 1)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (!(k & b)) {
        const float lo = a[k], hi = a[k | b];
        a[k] = lo + hi;
        a[k | b] = hi - lo;
      }
}

// ft (24, cells) = T^T (K^ (T u_c)) for every cell (listed cells are rewritten afterwards). Where the matrices
// are older than the launch ahead (lpb_pack_modal_f32 sees to it) a cell's first MODAL_AHEAD entries
// are loaded while that launch still runs (elsewhere the launch is in stream order); u is read after it (an update of 32 x 16 x 16 cells 7.3 -> 6.6 us,
// and 8.2 -> 7.3 by the gather's loads ahead; a cell's entries shared by four warps
// won 0.4 us there and lost 2.0 us at 64 x 32 x 32).
constexpr int MODAL_AHEAD = 64;
__device__ __forceinline__ void modal_cell(float* __restrict__ ft, const float* __restrict__ u,
                                           const float* __restrict__ km, const LpGrid& g, long long t) {
  const long long ncp = g.cells_padded();
  const long long cs = g.comp_stride();
  int x, y, z;
  const bool on = t < ncp && g.cell_at(t, x, y, z);
  constexpr int MUP_R[MODAL_UP] = MUP_ROWS;
  constexpr int MUP_C[MODAL_UP] = MUP_COLS;
  const float* kc = km + t;
  float ahead[MODAL_AHEAD];
  if (on)
#pragma unroll
    for (int p = 0; p < MODAL_AHEAD; ++p) ahead[p] = __ldcg(kc + (long long)p * ncp);
  lp_wait_prior();
  lp_release_next();
  if (!on || isnan(ahead[0])) return;              // a listed cell's entry 0 holds the marker
  const long long n0 = g.node(x, y, z);
  const long long oy = 4LL * g.NX(), oz = (z & 3) == 3 ? g.node_zc_stride() - 3 : 1;
  float uh[24], fh[24];
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    float a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      a[q] = u[cc * cs + n0 + (q & 1 ? 4 : 0) + (q & 2 ? oy : 0) + (q & 4 ? oz : 0)];
    walsh8(a);
#pragma unroll
    for (int m = 0; m < 8; ++m) uh[3 * m + cc] = a[m];
  }
#pragma unroll
  for (int r = 0; r < 24; ++r) fh[r] = 0.0f;
#pragma unroll
  for (int p = 0; p < MODAL_UP; ++p) {
    const float v = p < MODAL_AHEAD ? ahead[p < MODAL_AHEAD ? p : 0] : __ldg(kc + (long long)p * ncp);
    fh[MUP_R[p]] += v * uh[MUP_C[p]];
    if (MUP_R[p] != MUP_C[p]) fh[MUP_C[p]] += v * uh[MUP_R[p]];
  }
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    float a[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) a[m] = fh[3 * m + cc];
    walsh8t(a);
#pragma unroll
    for (int q = 0; q < 8; ++q) ft[(long long)(3 * q + cc) * ncp + t] = a[q];
  }
}

// the listed cells from their node-basis entries (kpc: 300 per listed cell, cell-major): one warp
// per cell, its 300 entries and 24 corner values staged in shared memory, lane r < 24 forms row r
__device__ __forceinline__ void listed_cells(float* __restrict__ ft, const float* __restrict__ u,
                                             const float* __restrict__ kpc, const int* __restrict__ glist,
                                             const int* __restrict__ gcount, const LpGrid& g, int block, int nblocks,
                                             float (*sk)[300], float (*su)[24]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long ncp = g.cells_padded();
  const long long cs = g.comp_stride();
  const int cnt = *gcount;
  for (int slot = (block * blockDim.x + threadIdx.x) >> 5; slot < cnt; slot += (nblocks * blockDim.x) >> 5) {
    const long long c = glist[slot];
    int x, y, z;
    g.cell_at(c, x, y, z);
    for (int p = lane; p < 300; p += 32) sk[w][p] = __ldg(kpc + (long long)slot * 300 + p);
    if (lane < 24) {
      const int q = lane / 3, cc = lane % 3;
      su[w][lane] = u[cc * cs + g.node(x + cx_(q), y + cy_(q), z + cz_(q))];
    }
    __syncwarp();
    if (lane < 24) {
      float f = 0.0f;
#pragma unroll
      for (int b = 0; b < 24; ++b) {
        const int lo = lane < b ? lane : b, hi = lane < b ? b : lane;
        f += sk[w][sym_index(lo, hi)] * su[w][b];
      }
      ft[(long long)lane * ncp + c] = f;
    }
    __syncwarp();
  }
}

// the cell rows of an explicit level in one launch: blocks below modal_blocks apply the modal
// form to one cell per thread (listed cells skipped), the blocks past them the listed cells
__global__ void __launch_bounds__(128, 4) k_explicit_modal_cells(float* __restrict__ ft, const float* __restrict__ u,
                                                                const float* __restrict__ km,
                                                                const float* __restrict__ kpc,
                                                                const int* __restrict__ glist,
                                                                const int* __restrict__ gcount, LpGrid g,
                                                                int modal_blocks) {
  ft += 24 * g.cells_padded() * blockIdx.y;   // the column
  u += 3 * g.comp_stride() * blockIdx.y;
  __shared__ float sk[4][300];
  __shared__ float su[4][24];
  if ((int)blockIdx.x < modal_blocks) {
    modal_cell(ft, u, km, g, blockIdx.x * (long long)blockDim.x + threadIdx.x);
  } else {
    lp_after_launch();
    listed_cells(ft, u, kpc, glist, gcount, g, blockIdx.x - modal_blocks, gridDim.x - modal_blocks, sk, su);
  }
}

// nothing: a launch of its own behind lpb_pack_modal_f32's and lpb_pack_sym_*'s, after which that one is complete for whatever is
// launched next, started early or not
__global__ void k_settled() { lp_after_launch(); }

template <typename T>
__global__ void k_explicit_gather(T* __restrict__ out, const T* __restrict__ ft, const uint8_t* __restrict__ mask,
                                  LpGrid g) {
  lp_after_launch();
  const long long total = g.nodes_padded();
  const long long ncp = g.cells_padded(), cs = g.comp_stride();
  ft += 24 * ncp * blockIdx.y;   // the column
  out += 3 * cs * blockIdx.y;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    if (!g.node_at(t, x, y, z)) continue;
    T a[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int cx = x - cx_(k), cy = y - cy_(k), cz = z - cz_(k);
      if (cx < 0 || cy < 0 || cz < 0 || cx >= g.nx || cy >= g.ny || cz >= g.nz) continue;
      const long long c = g.cell(cx, cy, cz);
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) a[cc] += ft[(long long)(3 * k + cc) * ncp + c];
    }
    const long long n = g.node(x, y, z);
    const uint8_t mb = mask[n];
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) out[cc * cs + n] = ((mb >> cc) & 1) ? a[cc] : T(0);
  }
}

// The explicit gather with a degree-2 Chebyshev update applied to each node's A u as it is formed
// (the standalone kernels' expressions): mode 1 x = d + (c1 d + c2 dinv (b - A d)); mode 2 r = b - A x,
// d = s dinv r; mode 3 x = (x + d) + (c1 d + c2 dinv (r - A d)). Padding is left as it is (zero).
template <typename T>
struct ChebArgs {
  T* x;
  T* r;
  T* d;
  const T* b;
  const T* dinv;
  const double* coef;
};

template <typename T, int MODE>
__global__ void __launch_bounds__(128)
k_explicit_gather_cheb(const T* __restrict__ ft, const uint8_t* __restrict__ mask, LpGrid g, ChebArgs<T> a) {
  const long long ncp = g.cells_padded(), cs = g.comp_stride(), co = 3 * cs * blockIdx.y;
  ft += 24 * ncp * blockIdx.y;   // the column
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int x, y, z;
  const bool on = t < g.nodes_padded() && g.node_at(t, x, y, z);
  const T s = (T)__ldcg(a.coef + 1), c1 = (T)__ldcg(a.coef + 2), c2 = (T)__ldcg(a.coef + 3);
  // all but the cells' forces was complete before the launch ahead (the cells')
  uint8_t mb = 0;
  T dv[3], v0[3], v1[3], v2[3];   // mode 1: d, b; mode 2: b; mode 3: x, d, r
  if (on) {
    mb = __ldcg(mask + t);
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
      const long long i = co + cc * cs + t;
      dv[cc] = __ldcg(a.dinv + i - co);
      v0[cc] = __ldcg((MODE == 1 ? a.d : MODE == 2 ? a.b : a.x) + i);
      if (MODE != 2) v1[cc] = __ldcg((MODE == 1 ? a.b : a.d) + i);
      if (MODE == 3) v2[cc] = __ldcg(a.r + i);
    }
  }
  lp_wait_prior();
  lp_release_next();
  if (!on) return;
  T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int cx = x - cx_(k), cy = y - cy_(k), cz = z - cz_(k);
    if (cx < 0 || cy < 0 || cz < 0 || cx >= g.nx || cy >= g.ny || cz >= g.nz) continue;
    const long long c = g.cell(cx, cy, cz);
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) acc[cc] += ft[(long long)(3 * k + cc) * ncp + c];
  }
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    const long long i = co + cc * cs + t;
    const T adi = ((mb >> cc) & 1) ? acc[cc] : T(0);
    if (MODE == 1) {
      a.x[i] = lp_cheb2_zero_v(v0[cc], v1[cc], adi, dv[cc], c1, c2);
    } else if (MODE == 2) {
      T ri, di;
      lp_residual_scaled_v(v0[cc], adi, dv[cc], s, ri, di);
      a.r[i] = ri;
      a.d[i] = di;
    } else {
      a.x[i] = lp_cheb2_v(v0[cc], v1[cc], v2[cc], adi, dv[cc], c1, c2);
    }
  }
}

// full (cells, 576) matrices -> packed symmetric entry-major (the average of K and K^T)
template <typename Ti, typename To>
__global__ void k_pack_sym(To* __restrict__ kp, const Ti* __restrict__ k, long long ncp) {
  lp_after_launch();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 300 * ncp; t += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(t / ncp);
    const long long c = t % ncp;
    int a = 0, rem = p;
    while (rem >= 24 - a) { rem -= 24 - a; ++a; }
    const int b = a + rem;
    kp[t] = (To)(0.5 * ((double)k[c * 576 + a * 24 + b] + (double)k[c * 576 + b * 24 + a]));
  }
}

}  // namespace

#define LP_GRID_ARGS int nx, int ny, int nz, int pz, int cpz
#define LP_GRID lp_grid(nx, ny, nz, pz, cpz)
#define LP_ST ((cudaStream_t)stream)

static double pw_host(int k, int q, int r) {
  double w = 1.0;
  for (int a = 0; a < 3; ++a) {
    const int p = ((k >> a) & 1) + ((q >> a) & 1);
    const double t = 0.5 * p;
    w *= ((r >> a) & 1) ? t : 1.0 - t;
  }
  return w;
}

static const int G1_ROWS[279] = {3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5, 5, 5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 6, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 7, 8, 8, 8, 8, 8, 8, 8, 8, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 9, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 10, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 12, 12, 12, 12, 12, 12, 12, 12, 13, 13, 13, 13, 13, 13, 13, 13, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 17, 18, 18, 18, 18, 18, 18, 18, 18, 18, 18, 18, 18, 18, 18, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 19, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 21, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 22, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23, 23};
static const int G1_TS[279] = {0, 0, 0, 1, 1, 2, 2, 3, 4, 4, 5, 6, 0, 0, 1, 2, 4, 4, 5, 6, 0, 0, 1, 2, 2, 3, 4, 6, 0, 0, 1, 2, 4, 4, 5, 6, 0, 0, 0, 1, 1, 2, 2, 3, 4, 4, 5, 6, 0, 0, 1, 1, 2, 3, 4, 5, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 4, 5, 5, 6, 6, 7, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 4, 5, 5, 6, 6, 7, 0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 4, 5, 6, 0, 0, 1, 2, 2, 3, 4, 6, 0, 0, 1, 1, 2, 3, 4, 5, 0, 0, 0, 1, 1, 2, 2, 3, 4, 4, 5, 6, 0, 0, 1, 1, 1, 2, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 0, 0, 0, 1, 1, 1, 2, 3, 4, 4, 4, 5, 5, 6, 0, 0, 1, 1, 1, 2, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 0, 0, 0, 1, 2, 2, 2, 3, 4, 4, 4, 5, 6, 6, 0, 0, 1, 2, 2, 2, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 0, 0, 1, 2, 2, 2, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 0, 1, 1, 1, 2, 2, 3, 3, 3, 4, 4, 5, 5, 5, 6, 6, 6, 7, 7, 0, 1, 1, 2, 2, 2, 3, 3, 3, 4, 4, 5, 5, 5, 6, 6, 6, 7, 7, 0, 1, 1, 2, 2, 3, 3, 3, 4, 4, 4, 5, 5, 5, 6, 6, 6, 7, 7};
static const int G1_COLS[279] = {3, 7, 14, 10, 17, 9, 20, 23, 15, 19, 22, 21, 4, 6, 9, 10, 16, 18, 21, 22, 5, 12, 15, 11, 18, 21, 17, 23, 4, 6, 9, 10, 16, 18, 21, 22, 3, 7, 14, 10, 17, 9, 20, 23, 15, 19, 22, 21, 8, 13, 11, 16, 19, 22, 20, 23, 9, 20, 4, 6, 23, 3, 7, 14, 10, 17, 21, 16, 18, 15, 19, 22, 10, 17, 3, 7, 14, 4, 6, 23, 9, 20, 22, 15, 19, 16, 18, 21, 11, 16, 18, 8, 13, 21, 5, 12, 22, 15, 19, 23, 20, 17, 5, 12, 15, 11, 18, 21, 17, 23, 8, 13, 11, 16, 19, 22, 20, 23, 3, 7, 14, 10, 17, 9, 20, 23, 15, 19, 22, 21, 15, 19, 5, 12, 22, 21, 11, 18, 3, 7, 14, 10, 17, 9, 20, 23, 11, 16, 18, 8, 13, 21, 22, 19, 4, 6, 23, 9, 20, 10, 10, 17, 3, 7, 14, 23, 9, 20, 5, 12, 22, 15, 19, 11, 18, 21, 11, 16, 18, 21, 5, 12, 22, 15, 4, 6, 23, 9, 10, 17, 15, 19, 22, 8, 13, 21, 11, 16, 3, 7, 14, 10, 17, 9, 20, 23, 9, 20, 23, 3, 7, 14, 10, 17, 8, 13, 21, 11, 16, 15, 19, 22, 21, 11, 16, 18, 15, 19, 5, 12, 22, 9, 20, 4, 6, 23, 3, 7, 14, 10, 17, 22, 15, 19, 11, 16, 18, 8, 13, 21, 10, 17, 3, 7, 14, 4, 6, 23, 9, 20, 23, 9, 20, 10, 17, 3, 7, 14, 11, 16, 18, 8, 13, 21, 5, 12, 22, 15, 19};

// The patch cells' launch over the chunks of pbox (host, 6 ints: their node box). Nothing on fields that it cannot
// read by four: the march has reported those (*err).
template <typename T, int MODE>
static void launch_patch_nodes(T* out, const T* u, const int* pid, const T* pk, const uint8_t* mask, const int* pbox,
                               const LpGrid& g, const L1Cheb<T>& ch, int cols, cudaStream_t st) {
  const uintptr_t fields = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(ch.x) | reinterpret_cast<uintptr_t>(ch.r) |
                           reinterpret_cast<uintptr_t>(ch.d) | reinterpret_cast<uintptr_t>(ch.b) |
                           reinterpret_cast<uintptr_t>(ch.dinv);
  if ((MODE ? fields & 15 : reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(mask) & 3)) return;
  const int c0 = pbox[2] >> 2, nc = ((pbox[2] + pbox[5] + 3) >> 2) - c0;
  const long long total = (long long)pbox[3] * pbox[4] * nc;
  if (total > PN_FROM) {
    int quads = 4;   // few quads a block while that leaves the GPU short of blocks
    while (quads < PN_QUADS && total * cols > quads * 148 * 32LL) quads *= 2;
    // neighbouring blocks, whose quads have the same share of patch cells, go to different SMs
    const unsigned nb = (unsigned)((total + quads - 1) / quads);
    unsigned stride = (unsigned)(0.618 * nb) | 1;
    while (std::gcd(stride, nb) != 1) stride += 2;
    lp_launch(k_patch_nodes<T, MODE>, dim3(nb, cols), PN_THREADS, 0, st, out, u, pid, pk, mask, g, pbox[0], pbox[1], c0, pbox[3],
              pbox[4], nc, quads, stride, ch);
    return;
  }
  // on an x or y face most nodes of the box are touched: a warp each while they are few (96 x 48 x 48 cells,
  // float32 smoothing: x face 45.2 us, a warp per quad 55.8; y face, twice the nodes, 62.5 and 56.1)
  const bool face = std::min(pbox[3], pbox[4]) <= 3 && total <= 2048;
  lp_launch(face ? k_patch_quads<T, MODE, 1> : k_patch_quads<T, MODE, 4>,
            dim3(lp_blocks(32 * total * (face ? 4 : 1), PQ_THREADS), cols), PQ_THREADS, 0, st, out, u, pid, pk, mask, g, pbox[0],
            pbox[1], c0, pbox[3], pbox[4], nc, ch);
}

// pbox: the node box of the patch cells (host, 6 ints), which the split weighs
template <typename T, int MODE>
static int launch_level1(T* out, const T* u, const T* wc, const int* pid, const T* pm, const T* pk, const uint8_t* mask,
                         const double* g1_host, const int* pbox, int* err, LpGrid g, cudaStream_t st,
                         const L1Cheb<T>& ch, int cols = 1) {
  if (cols < 1 || cols > 65535) return LP_ERR_ARG;
  if (!lp_grid_ok(g) || g.pz % 4 || g.cpz != g.pz || (MODE == 0 && !out) || !u || !wc || !mask || !g1_host || !err)
    return LP_ERR_ARG;
  G1<T> gc;
  for (int i = 0; i < 279; ++i) gc.c[i] = (T)g1_host[i];
  L1Maps maps;
  const uint64_t nd[4] = {4 * (uint64_t)g.NX(), (uint64_t)g.NY(), (uint64_t)g.pz / 4, 3 * (uint64_t)cols};
  const uint32_t bin[4] = {4 * LBX, LBY, 1, 3};
  if (!lp_make_map(&maps.u, u, 4, nd, bin, sizeof(T))) return LP_ERR_ARG;
  memset(&maps.w, 0, sizeof(maps.w));
  if (sizeof(T) == 4) {
    const uint64_t wd[4] = {32, (uint64_t)g.nx, (uint64_t)g.ny, (uint64_t)g.cpz / 4};
    const uint32_t wb[4] = {32, LX, LY, 1};
    if (!lp_make_map(&maps.w, wc, 4, wd, wb, sizeof(T), 128)) return LP_ERR_ARG;
  }
  const int smem = (int)sizeof(L1Smem<T>) + 1024;
  const long long slots = lp_resident_blocks((const void*)k_level1<T, MODE>, LCOL, smem);
  if (slots < 1) return LP_ERR_LAUNCH;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int gx = (g.NX() + LX - 2) / (LX - 1), gy = (g.NY() + LY - 2) / (LY - 1), nchunks = g.pz / 4;
  // persistent blocks: all resident ones (or the tuned number per SM)
  long long nb = slots < L1_MAX_BLOCKS ? slots : L1_MAX_BLOCKS;
  const int tuned = lp_tune_lookup(sizeof(T) == 4 ? LP_KNOB_L1_F32 : LP_KNOB_L1_F64, g.nx, g.ny, g.nz);
  if (tuned >= 1 && (long long)tuned * nsm < nb) nb = (long long)tuned * nsm;
  const long long units = (long long)gx * gy * nchunks;
  if (units > 2147483647LL) return LP_ERR_SIZE;
  // The patch cells' products are a chunk's latency over again, which a march of a few units a block does not
  // hide: their own launch, overlapping the march, is then the faster form (applies in us, in the march and
  // apart: 64 x 32 x 32 cells 13.8 and 9.7 in float32, 27.2 and 17.0 in float64; 96 x 48 x 48, 2.2
  // units a block, 21.0 and 19.7, 41.7 and 34.4; 128 x 64 x 64, 5.2 units, 32.7 and 35.8, 69.7 and 71.4). So it
  // is where a tile's chunk may hold more cells than the block takes together, which a thread each then takes
  // alone (in float32, on a grid of 128 x 64 x 64 cells: a z face held 93.4 and 40.7, two z faces 162.7 and
  // 72.2; two x faces, whose box says the same, 50.6 and 50.2).
  const bool have_patches = pid && pm && pbox && pbox[3] > 0 && pbox[4] > 0 && pbox[5] > 0;
  const bool crowded = have_patches && (long long)std::min(LX, pbox[3] - 1) * std::min(LY, pbox[4] - 1) *
                                               std::min(4, pbox[5] - 1) > L1_PATCH;
  const bool apart = have_patches && pk && out && out != u && (units <= 3 * nb || crowded);
  if (nb > units) nb = units;
  // block b starts where b / nb of the total weight is reached: a chunk weighs 4, 8 in a tile that holds
  // patch cells (measured: with equal weights the support face's blocks ran 1.8x as long as the mean,
  // 47 us against 36 at 128 x 64 x 64)
  const bool patches = have_patches && !apart;
  const L1Box box = patches ? L1Box{pbox[0], pbox[0] + pbox[3] - 1, pbox[1], pbox[1] + pbox[4] - 1} : L1Box{};
  auto weight = [&](int tile) {
    const int x0 = (tile % gx) * (LX - 1) - 1, y0 = (tile / gx) * (LY - 1) - 1;
    return patches && x0 < box.hx && x0 + LX > box.x && y0 < box.hy && y0 + LY > box.y ? 8 : 4;
  };
  L1Split split;
  long long sum = 0;
  for (int t = 0; t < gx * gy; ++t) sum += weight(t);
  sum *= nchunks;
  int b = 0;
  long long done = 0;
  for (int t = 0; t < gx * gy; ++t) {
    const int w = weight(t);
    for (; b < nb && sum * b < (done + (long long)w * nchunks) * nb; ++b) {
      const long long into = (sum * b - done * nb + (long long)w * nb - 1) / ((long long)w * nb);
      split.u0[b] = (int)((long long)t * nchunks + into);
    }
    done += (long long)w * nchunks;
  }
  for (; b <= nb; ++b) split.u0[b] = (int)units;
  L1Nodes nodes{};
  if (apart && MODE)
    nodes = L1Nodes{pbox[0], pbox[0] + pbox[3], pbox[1], pbox[1] + pbox[4], pbox[2] >> 2, (pbox[2] + pbox[5] + 3) >> 2};
  lp_launch(k_level1<T, MODE>, dim3((unsigned)nb, cols), LCOL, smem, st, maps, split, out, wc, patches ? pid : nullptr, pm, mask,
            gc, g, nchunks, err, ch, box, nodes);
  if (apart) launch_patch_nodes<T, MODE>(out, u, pid, pk, mask, pbox, g, ch, cols, st);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// lpb_apply_weights_tma_*: the march without the patch cells, then their node-basis matrices node by node
template <typename T>
static int apply_weights_tma(T* out, const T* u, const T* wc, const int* pid, const T* pk, const uint8_t* mask,
                             const double* g1, const int* pbox, int* err, LpGrid g, cudaStream_t st) {
  if (out == u || (reinterpret_cast<uintptr_t>(out) & 15)) return LP_ERR_ARG;
  const int rc = launch_level1<T, 0>(out, u, wc, nullptr, nullptr, nullptr, mask, g1, nullptr, err, g, st, L1Cheb<T>{});
  if (rc != LP_OK) return rc;
  if (pid && pk && pbox && pbox[3] > 0 && pbox[4] > 0 && pbox[5] > 0) {
    launch_patch_nodes<T, 0>(out, u, pid, pk, mask, pbox, g, L1Cheb<T>{}, 1, st);
    LP_LAUNCH_CHECK();
  }
  return LP_OK;
}

template <typename T>
static int apply_level1(int mode, T* out, T* x, T* r, T* d, const T* u, const T* b, const T* dinv, const double* coef,
                        const T* wc, const int* pid, const T* pm, const T* pk, const uint8_t* mask, const double* g1,
                        const int* pbox, int* err, LpGrid g, int cols, cudaStream_t st) {
  if (!u || mode < 0 || mode > 3 || (mode && (!dinv || !coef))) return LP_ERR_ARG;
  const L1Cheb<T> ch{x, r, d, b, dinv, coef};
  if (mode == 0 && out && out != u)
    return launch_level1<T, 0>(out, u, wc, pid, pm, pk, mask, g1, pbox, err, g, st, ch, cols);
  if (mode == 1 && x && d && b && u == d && x != d)
    return launch_level1<T, 1>(out, u, wc, pid, pm, pk, mask, g1, pbox, err, g, st, ch, cols);
  if (mode == 2 && r && d && b && u == x && r != u && d != u && r != d)
    return launch_level1<T, 2>(out, u, wc, pid, pm, pk, mask, g1, pbox, err, g, st, ch, cols);
  if (mode == 3 && x && d && r && u == d && x != d && r != d && r != x)
    return launch_level1<T, 3>(out, u, wc, pid, pm, pk, mask, g1, pbox, err, g, st, ch, cols);
  return LP_ERR_ARG;
}

// settled: kp was complete before the launch ahead began, so the cells may load it beside that launch
template <typename T>
static int launch_explicit(bool settled, T* out, const T* u, const T* kp, T* ft, const uint8_t* mask, LpGrid g,
                           cudaStream_t st, int mode = 0, const ChebArgs<T>* ch = nullptr) {
  if (!lp_grid_ok(g) || !u || !kp || !ft || !mask) return LP_ERR_ARG;
  if (mode == 0 && (!out || out == u)) return LP_ERR_ARG;
  constexpr int smem = (int)sizeof(ExCells<T>);   // above the 48 KB default in float64
  if (cudaFuncSetAttribute(k_explicit_cells<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return LP_ERR_LAUNCH;
  lp_launch_as(settled, k_explicit_cells<T>, lp_blocks(g.cells_padded(), 32), 32 * EX_WARPS, smem, st, ft, u, kp, g);
  if (mode == 0) {
    lp_launch(k_explicit_gather<T>, lp_blocks(g.nodes_padded(), 256), 256, 0, st, out, ft, mask, g);
  } else {
    const ChebArgs<T> a = *ch;
    const int nb = lp_blocks(g.nodes_padded(), 128);
    if (mode == 1) lp_launch(k_explicit_gather_cheb<T, 1>, nb, 128, 0, st, ft, mask, g, a);
    else if (mode == 2) lp_launch(k_explicit_gather_cheb<T, 2>, nb, 128, 0, st, ft, mask, g, a);
    else lp_launch(k_explicit_gather_cheb<T, 3>, nb, 128, 0, st, ft, mask, g, a);
  }
  LP_LAUNCH_CHECK();
  return LP_OK;
}

template <typename T>
static bool explicit_cheb_ok(int mode, const ChebArgs<T>& a, const T* u) {
  if (mode < 1 || mode > 3 || !a.dinv || !a.coef) return false;
  if (mode == 1) return a.x && a.d && a.b && u == a.d && a.x != a.d;
  if (mode == 2) return a.r && a.d && a.b && u != a.r && u != a.d && a.r != a.d;
  return a.x && a.d && a.r && u == a.d && a.x != a.d;
}

// settled: as launch_explicit's, of km, kpc, glist and gcount
static int launch_explicit_modal(bool settled, int mode, float* out, float* x, float* r, float* d, const float* u, const float* b,
                                 const float* dinv, const double* coef, const float* km, const float* kpc,
                                 const int* glist, const int* gcount, float* ft, const uint8_t* mask, LpGrid g, int cols,
                                 cudaStream_t st) {
  if (!lp_grid_ok(g) || !u || !km || !kpc || !glist || !gcount || !ft || !mask) return LP_ERR_ARG;
  if (cols < 1 || cols > 65535) return LP_ERR_ARG;
  if (mode == 0 && (!out || out == u)) return LP_ERR_ARG;
  const ChebArgs<float> a{x, r, d, b, dinv, coef};
  if (mode != 0 && !explicit_cheb_ok(mode, a, u)) return LP_ERR_ARG;
  const int modal_blocks = lp_blocks(g.cells_padded(), 128);
  lp_launch_as(settled, k_explicit_modal_cells, dim3(modal_blocks + 148, cols), 128, 0, st, ft, u, km, kpc, glist, gcount,
               g, modal_blocks);
  const dim3 nb(lp_blocks(g.nodes_padded(), 256), cols), nbc(lp_blocks(g.nodes_padded(), 128), cols);
  if (mode == 0) lp_launch(k_explicit_gather<float>, nb, 256, 0, st, out, ft, mask, g);
  else if (mode == 1) lp_launch(k_explicit_gather_cheb<float, 1>, nbc, 128, 0, st, ft, mask, g, a);
  else if (mode == 2) lp_launch(k_explicit_gather_cheb<float, 2>, nbc, 128, 0, st, ft, mask, g, a);
  else lp_launch(k_explicit_gather_cheb<float, 3>, nbc, 128, 0, st, ft, mask, g, a);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// ---- the explicit-level apply without caller scratch -----------------------------------------
// For callers that cannot allocate device memory: a host application or language binding that
// owns every device allocation and hands this library only the pointers it needs, or a loop
// that must never call cudaMalloc / cudaFree (they synchronize the device). The cell pass's
// (24, cells) intermediate lives in this file-scope array instead of a caller buffer. Every GPU
// that loads the library holds it (6 MB) until the process exits.
#define LP_NOALLOC_MAX_CELLS (1 << 16)   // padded cells (nx * ny * cpz) one call may cover
#define LP_NOALLOC_MAX_DEVICES 64
static __device__ __align__(256) float g_explicit_scratch[24 * LP_NOALLOC_MAX_CELLS];

// the array's device address on the current device, looked up once per device ordinal and kept
// for the life of the process: the caller's stream must belong to the current device, and a
// cudaDeviceReset invalidates the kept address (callers must not reset a device they use it on)
static float* explicit_scratch_address() {
  static std::mutex mu;
  static float* addr[LP_NOALLOC_MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= LP_NOALLOC_MAX_DEVICES) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_explicit_scratch) != cudaSuccess || !p) return nullptr;
    addr[dev] = static_cast<float*>(p);
  }
  return addr[dev];
}

extern "C" {

// the 279 corner-parity coefficients of the eight G_t = sum_k H[t, k] P_k^T Ke P_k / 8 (host)
int lpb_modal_g1(const double* ke, double* g1_out) {
  if (!ke || !g1_out) return LP_ERR_ARG;
  double h[8][8];
  for (int m = 0; m < 8; ++m)
    for (int k = 0; k < 8; ++k) {
      double v = 1.0;
      for (int a = 0; a < 3; ++a)
        if ((m >> a) & 1) v *= ((k >> a) & 1) ? 1.0 : -1.0;
      h[m][k] = v;
    }
  // M_k = P_k^T Ke P_k
  static double mk[8][24][24];
  for (int k = 0; k < 8; ++k)
    for (int i = 0; i < 24; ++i)
      for (int jj = 0; jj < 24; ++jj) {
        const int ri = i / 3, ci = i % 3, rj = jj / 3, cj = jj % 3;
        double s = 0.0;
        for (int q1 = 0; q1 < 8; ++q1) {
          const double p1 = pw_host(k, q1, ri);
          if (p1 == 0.0) continue;
          for (int q2 = 0; q2 < 8; ++q2) {
            const double p2 = pw_host(k, q2, rj);
            if (p2 == 0.0) continue;
            s += p1 * ke[(3 * q1 + ci) * 24 + 3 * q2 + cj] * p2;
          }
        }
        mk[k][i][jj] = s;
      }
  double amax = 0.0;
  static double gh[8][24][24];
  for (int t = 0; t < 8; ++t)
    for (int r = 0; r < 24; ++r)
      for (int c = 0; c < 24; ++c) {
        const int mr = r / 3, cr = r % 3, mc = c / 3, cc = c % 3;
        double s = 0.0;
        for (int k1 = 0; k1 < 8; ++k1)
          for (int k2 = 0; k2 < 8; ++k2) {
            double gsum = 0.0;
            for (int k = 0; k < 8; ++k) gsum += h[t][k] * mk[k][3 * k1 + cr][3 * k2 + cc];
            s += h[mr][k1] * gsum * h[mc][k2];
          }
        gh[t][r][c] = s / (8.0 * 64.0);
        if (fabs(gh[t][r][c]) > amax) amax = fabs(gh[t][r][c]);
      }
  static bool used[8][24][24];
  for (int t = 0; t < 8; ++t)
    for (int r = 0; r < 24; ++r)
      for (int c = 0; c < 24; ++c) used[t][r][c] = false;
  for (int i = 0; i < 279; ++i) used[G1_TS[i]][G1_ROWS[i]][G1_COLS[i]] = true;
  for (int t = 0; t < 8; ++t)
    for (int r = 0; r < 24; ++r)
      for (int c = 0; c < 24; ++c)
        if (!used[t][r][c] && fabs(gh[t][r][c]) > 1e-12 * amax) return -1;
  for (int i = 0; i < 279; ++i) g1_out[i] = gh[G1_TS[i]][G1_ROWS[i]][G1_COLS[i]];
  return 279;
}

// pbox (host, 6 ints): node box x0, y0, z0, nx, ny, nz holding every node a patch cell touches
int lpb_walsh_chunks_f32(float* wc, const float* w, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || g.cpz % 4 || !wc || !w) return LP_ERR_ARG;
  lp_launch(k_walsh_chunks<float>, lp_blocks(g.cells_padded(), 256), 256, 0, LP_ST, wc, w, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_walsh_chunks_f64(double* wc, const double* w, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || g.cpz % 4 || !wc || !w) return LP_ERR_ARG;
  lp_launch(k_walsh_chunks<double>, lp_blocks(g.cells_padded(), 256), 256, 0, LP_ST, wc, w, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// level-1 apply, its patch cells from their node-basis matrices in a second launch: wc from
// lpb_walsh_chunks_*; g1 and pbox are HOST arrays; err: a device int set when a wait gave up
// (or to an alignment code, 20..27)
int lpb_apply_weights_tma_f32(float* out, const float* u, const float* wc, const int* patch_id, const float* patch_k,
                              const uint8_t* mask, const double* g1, const int* pbox, int* err, LP_GRID_ARGS,
                              void* stream) {
  return apply_weights_tma<float>(out, u, wc, patch_id, patch_k, mask, g1, pbox, err, LP_GRID, LP_ST);
}

int lpb_apply_weights_tma_f64(double* out, const double* u, const double* wc, const int* patch_id,
                              const double* patch_k, const uint8_t* mask, const double* g1, const int* pbox, int* err,
                              LP_GRID_ARGS, void* stream) {
  return apply_weights_tma<double>(out, u, wc, patch_id, patch_k, mask, g1, pbox, err, LP_GRID, LP_ST);
}

// the patch cells' matrices (npatch, 24, 24) in the corner-parity basis
int lpb_patch_modal_f32(float* pm, const float* pk, long long npatch, void* stream) {
  if (!pm || !pk || npatch < 1 || npatch > 2147483647LL) return LP_ERR_ARG;
  lp_launch(k_patch_modal<float>, (unsigned)npatch, 192, 0, LP_ST, pm, pk);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_patch_modal_f64(double* pm, const double* pk, long long npatch, void* stream) {
  if (!pm || !pk || npatch < 1 || npatch > 2147483647LL) return LP_ERR_ARG;
  lp_launch(k_patch_modal<double>, (unsigned)npatch, 192, 0, LP_ST, pm, pk);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// the level-1 apply with its patch cells (patch_m from lpb_patch_modal_*): mode 0 out = m K u;
// modes 1..3 the Chebyshev updates of lpb_apply_fine_cheb_f32 (out not used; the fields a mode does
// not name may be NULL)
int lpb_apply_level1_f32(int mode, float* out, float* x, float* r, float* d, const float* u, const float* b,
                         const float* dinv, const double* coef, const float* wc, const int* patch_id,
                         const float* patch_m, const float* patch_k, const uint8_t* mask, const double* g1, const int* pbox, int* err,
                         LP_GRID_ARGS, void* stream) {
  return apply_level1<float>(mode, out, x, r, d, u, b, dinv, coef, wc, patch_id, patch_m, patch_k, mask, g1, pbox, err, LP_GRID, 1,
                             LP_ST);
}

// the same for cols columns (each field's columns one after the other)
int lpb_apply_level1_cols_f32(int mode, float* out, float* x, float* r, float* d, const float* u, const float* b,
                         const float* dinv, const double* coef, const float* wc, const int* patch_id,
                         const float* patch_m, const float* patch_k, const uint8_t* mask, const double* g1, const int* pbox, int* err,
                         LP_GRID_ARGS, int cols, void* stream) {
  return apply_level1<float>(mode, out, x, r, d, u, b, dinv, coef, wc, patch_id, patch_m, patch_k, mask, g1, pbox, err, LP_GRID, cols,
                             LP_ST);
}

int lpb_apply_level1_f64(int mode, double* out, double* x, double* r, double* d, const double* u, const double* b,
                         const double* dinv, const double* coef, const double* wc, const int* patch_id,
                         const double* patch_m, const double* patch_k, const uint8_t* mask, const double* g1, const int* pbox, int* err,
                         LP_GRID_ARGS, void* stream) {
  return apply_level1<double>(mode, out, x, r, d, u, b, dinv, coef, wc, patch_id, patch_m, patch_k, mask, g1, pbox, err, LP_GRID, 1,
                              LP_ST);
}

// the same for cols columns (each field's columns one after the other)
int lpb_apply_level1_cols_f64(int mode, double* out, double* x, double* r, double* d, const double* u, const double* b,
                         const double* dinv, const double* coef, const double* wc, const int* patch_id,
                         const double* patch_m, const double* patch_k, const uint8_t* mask, const double* g1, const int* pbox, int* err,
                         LP_GRID_ARGS, int cols, void* stream) {
  return apply_level1<double>(mode, out, x, r, d, u, b, dinv, coef, wc, patch_id, patch_m, patch_k, mask, g1, pbox, err, LP_GRID, cols,
                              LP_ST);
}

int lpb_apply_explicit_sym_f32(float* out, const float* u, const float* kp, float* ft, const uint8_t* mask,
                               LP_GRID_ARGS, void* stream) {
  return launch_explicit<float>(false, out, u, kp, ft, mask, LP_GRID, LP_ST);
}

int lpb_apply_explicit_sym_f64(double* out, const double* u, const double* kp, double* ft, const uint8_t* mask,
                               LP_GRID_ARGS, void* stream) {
  return launch_explicit<double>(false, out, u, kp, ft, mask, LP_GRID, LP_ST);
}

// lpb_apply_explicit_sym_f64 with a degree-2 Chebyshev update in its gather (modes 1..3, as
// lpb_apply_explicit_modal_cheb_f32), kp loaded before the launch ahead has ended: it must have been complete
// when that one began (lpb_pack_sym_f64 ends with a launch that sees to it)
int lpb_apply_explicit_sym_cheb_f64(int mode, double* x, double* r, double* d, const double* u, const double* b,
                                    const double* dinv, const double* coef, const double* kp, double* ft,
                                    const uint8_t* mask, LP_GRID_ARGS, void* stream) {
  const ChebArgs<double> a{x, r, d, b, dinv, coef};
  if (!explicit_cheb_ok(mode, a, u)) return LP_ERR_ARG;
  return launch_explicit<double>(true, nullptr, u, kp, ft, mask, LP_GRID, LP_ST, mode, &a);
}

// lpb_apply_explicit_sym_f32 with its (24, cells) scratch in the library's static array: no
// allocation by the caller or the library. Grids with more than LP_NOALLOC_MAX_CELLS padded
// cells return LP_ERR_SIZE. The first call on a device looks the array's address up (it should
// come before any stream capture); calls that overlap on the GPU share the array and race. The
// cell pass writes every entry the node pass reads, so stale contents from an earlier call are
// never used and nothing needs clearing.
int lpb_apply_explicit_sym_noalloc_f32(float* out, const float* u, const float* kp, const uint8_t* mask, LP_GRID_ARGS,
                                       void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g)) return LP_ERR_ARG;
  if (g.cells_padded() > LP_NOALLOC_MAX_CELLS) return LP_ERR_SIZE;
  float* ft = explicit_scratch_address();
  if (!ft) return LP_ERR_LAUNCH;
  return launch_explicit<float>(false, out, u, kp, ft, mask, g, LP_ST);
}

// km (150, ncells) = the pattern entries of each cell's K^ = T K T^T / 64 (symmetric part); cells
// with off-pattern weight above tol of their largest entry get zeros and are listed in glist
// (*gcount of them), their 300 node-basis symmetric entries in kpc at their list slot (glist and
// kpc hold up to ncells cells)
int lpb_pack_modal_f32(float* km, int* glist, int* gcount, float* kpc, const float* k, long long ncells, double tol,
                       void* stream) {
  if (!km || !glist || !gcount || !kpc || !k || ncells < 1) return LP_ERR_ARG;
  if (cudaMemsetAsync(gcount, 0, sizeof(int), LP_ST) != cudaSuccess) return LP_ERR_LAUNCH;
  const long long blocks = (ncells + 3) / 4;
  lp_launch(k_pack_modal<float>, (unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 128, 0, LP_ST, km, glist, gcount, kpc,
                                                                                          k, ncells, tol);
  lp_launch(k_settled, 1, 32, 0, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// out = m K u on an explicit level from the modal form km and, for the listed cells, their
// node-basis entries kpc (both from lpb_pack_modal_f32); ft: 24 * cells scratch
int lpb_apply_explicit_modal_f32(float* out, const float* u, const float* km, const float* kpc, const int* glist,
                                 const int* gcount, float* ft, const uint8_t* mask, LP_GRID_ARGS, void* stream) {
  return launch_explicit_modal(false, 0, out, nullptr, nullptr, nullptr, u, nullptr, nullptr, nullptr, km, kpc, glist, gcount, ft,
                               mask, LP_GRID, 1, LP_ST);
}

// the explicit level's A u (modal form, as lpb_apply_explicit_modal_f32) with a degree-2 Chebyshev
// update in its gather: mode 1 (u = d) x = d + (c1 d + c2 dinv (b - A d)); mode 2 (u = x)
// r = b - A x, d = s dinv r; mode 3 (u = d) x = (x + d) + (c1 d + c2 dinv (r - A d)); the fields
// a mode does not name may be NULL; coef: the level's Chebyshev coefficients (device)
int lpb_apply_explicit_modal_cheb_f32(int mode, float* x, float* r, float* d, const float* u, const float* b,
                                      const float* dinv, const double* coef, const float* km, const float* kpc,
                                      const int* glist, const int* gcount, float* ft, const uint8_t* mask,
                                      LP_GRID_ARGS, void* stream) {
  if (mode < 1) return LP_ERR_ARG;
  return launch_explicit_modal(false, mode, nullptr, x, r, d, u, b, dinv, coef, km, kpc, glist, gcount, ft, mask, LP_GRID,
                               1, LP_ST);
}

// both (mode 0: out = m K u) for cols columns, each field's columns one after the other; ft: 24 * cells
// scratch per column. km, kpc, glist and gcount are loaded before the launch ahead has ended: they must have been
// complete when that one began (lpb_pack_modal_f32 ends with a launch that sees to it)
int lpb_apply_explicit_modal_cols_f32(int mode, float* out, float* x, float* r, float* d, const float* u, const float* b,
                                      const float* dinv, const double* coef, const float* km, const float* kpc,
                                      const int* glist, const int* gcount, float* ft, const uint8_t* mask,
                                      LP_GRID_ARGS, int cols, void* stream) {
  return launch_explicit_modal(true, mode, out, x, r, d, u, b, dinv, coef, km, kpc, glist, gcount, ft, mask, LP_GRID, cols,
                               LP_ST);
}

int lpb_pack_sym_f32(float* kp, const float* k, long long ncells, void* stream) {
  if (!kp || !k || ncells < 0) return LP_ERR_ARG;
  lp_launch(k_pack_sym<float, float>, lp_blocks(300 * ncells, 256), 256, 0, LP_ST, kp, k, ncells);
  lp_launch(k_settled, 1, 32, 0, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_pack_sym_f64(double* kp, const double* k, long long ncells, void* stream) {
  if (!kp || !k || ncells < 0) return LP_ERR_ARG;
  lp_launch(k_pack_sym<double, double>, lp_blocks(300 * ncells, 256), 256, 0, LP_ST, kp, k, ncells);
  lp_launch(k_settled, 1, 32, 0, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

}  // extern "C"
