// mw_pow.cuh -- x^gamma for the row constants (the background pressure
// C0 (rho theta)^gamma) in 25 FP64 operations.
//
// A row's constants sit at the head of a kernel, where their serial FP64 chain
// is latency (a warp's FP64 instruction takes 64 cycles): CUDA's pow takes 5900
// cycles there, this about 1900.  Table-driven logarithm and exponential after
// P. T. P. Tang (ACM TOMS 15(2), 1989, and 16(4), 1990) for the one exponent:
// x = 2^E m, m in [1, 2), c ~ 1/m from the leading 6 bits of m, r = m c - 1
// (one FMA, |r| < 2^-7), log2 x = (E - log2 c) + log2(1 + r) with the first term
// exact and the series' sum as a correction; gamma log2 x as a head and a tail
// by an FMA; 2^that by the nearest multiple of 1/64 and a series.  At most 0.86
// ulp off on 4 million arguments in [1e-4, 1e5], 0.77 in [20, 400] where the
// atmosphere's lie, 0.93 over the range it takes (against 113-bit arithmetic).  Arguments outside the positive normal range, or whose
// power is near its ends, take pow itself.
#pragma once

#include "mw_common.cuh"

namespace mw {

struct PowTables {
  double c[64], hi[64], lo[64], t[64], tl[64];
};
// log2 and 2^x of the table points, from their definitions in 200-bit arithmetic.
static __device__ const PowTables g_pow_tables = {
    // c[j] ~ 1 / (1 + (j + 1/2) / 64)
    {0x1.fc07f01fc07f0p-1, 0x1.f44659e4a4271p-1, 0x1.ecc07b301ecc0p-1, 0x1.e573ac901e574p-1, 0x1.de5d6e3f8868ap-1,
     0x1.d77b654b82c34p-1, 0x1.d0cb58f6ec074p-1, 0x1.ca4b3055ee191p-1, 0x1.c3f8f01c3f8f0p-1, 0x1.bdd2b899406f7p-1,
     0x1.b7d6c3dda338bp-1, 0x1.b2036406c80d9p-1, 0x1.ac5701ac5701bp-1, 0x1.a6d01a6d01a6dp-1, 0x1.a16d3f97a4b02p-1,
     0x1.9c2d14ee4a102p-1, 0x1.970e4f80cb872p-1, 0x1.920fb49d0e229p-1, 0x1.8d3018d3018d3p-1, 0x1.886e5f0abb04ap-1,
     0x1.83c977ab2beddp-1, 0x1.7f405fd017f40p-1, 0x1.7ad2208e0ecc3p-1, 0x1.767dce434a9b1p-1, 0x1.724287f46debcp-1,
     0x1.6e1f76b4337c7p-1, 0x1.6a13cd1537290p-1, 0x1.661ec6a5122f9p-1, 0x1.623fa77016240p-1, 0x1.5e75bb8d015e7p-1,
     0x1.5ac056b015ac0p-1, 0x1.571ed3c506b3ap-1, 0x1.5390948f40febp-1, 0x1.5015015015015p-1, 0x1.4cab88725af6ep-1,
     0x1.49539e3b2d067p-1, 0x1.460cbc7f5cf9ap-1, 0x1.42d6625d51f87p-1, 0x1.3fb013fb013fbp-1, 0x1.3c995a47babe7p-1,
     0x1.3991c2c187f63p-1, 0x1.3698df3de0748p-1, 0x1.33ae45b57bcb2p-1, 0x1.30d190130d190p-1, 0x1.2e025c04b8097p-1,
     0x1.2b404ad012b40p-1, 0x1.288b01288b013p-1, 0x1.25e22708092f1p-1, 0x1.23456789abcdfp-1, 0x1.20b470c67c0d9p-1,
     0x1.1e2ef3b3fb874p-1, 0x1.1bb4a4046ed29p-1, 0x1.19453808ca29cp-1, 0x1.16e0689427379p-1, 0x1.1485f0e0acd3bp-1,
     0x1.12358e75d3033p-1, 0x1.0fef010fef011p-1, 0x1.0db20a88f4696p-1, 0x1.0b7e6ec259dc8p-1, 0x1.0953f39010954p-1,
     0x1.073260a47f7c6p-1, 0x1.05197f7d73404p-1, 0x1.03091b51f5e1ap-1, 0x1.0101010101010p-1},
    // hi[j]: -log2 c[j] to a multiple of 2^-38
    {0x1.6fe50b6e00000p-7, 0x1.11cd1d5100000p-5, 0x1.c4dfab9080000p-5, 0x1.3aa2fdd280000p-4, 0x1.918a16e480000p-4,
     0x1.e72ec11800000p-4, 0x1.1dcd197560000p-3, 0x1.476a9f9840000p-3, 0x1.70742d4f00000p-3, 0x1.98edd077e0000p-3,
     0x1.c0db6cdda0000p-3, 0x1.e840be74e0000p-3, 0x1.0790adbb00000p-2, 0x1.1ac05b2920000p-2, 0x1.2db10fc4e0000p-2,
     0x1.406463b1b0000p-2, 0x1.52dbdfc4d0000p-2, 0x1.6518fe4670000p-2, 0x1.771d2ba7f0000p-2, 0x1.88e9c72e10000p-2,
     0x1.9a802391e0000p-2, 0x1.abe18797f0000p-2, 0x1.bd0f2e9e80000p-2, 0x1.ce0a4923a0000p-2, 0x1.ded3fd4420000p-2,
     0x1.ef6d673290000p-2, 0x1.ffd799a840000p-2, 0x1.0809cf27f8000p-1, 0x1.10113b1540000p-1, 0x1.18028cf728000p-1,
     0x1.1fde3d30e8000p-1, 0x1.27a4c05860000p-1, 0x1.2f56875eb0000p-1, 0x1.36f3ffb6d8000p-1, 0x1.3e7d9379f8000p-1,
     0x1.45f3a98a20000p-1, 0x1.4d56a5b340000p-1, 0x1.54a6e8ca58000p-1, 0x1.5be4d0cb50000p-1, 0x1.6310b8f550000p-1,
     0x1.6a2af9e5a0000p-1, 0x1.7133e9b158000p-1, 0x1.782bdbfdd8000p-1, 0x1.7f13221830000p-1, 0x1.85ea0b0b28000p-1,
     0x1.8cb0e3b4b0000p-1, 0x1.9367f6da08000p-1, 0x1.9a0f8d3b10000p-1, 0x1.a0a7eda4c0000p-1, 0x1.a7315d02f0000p-1,
     0x1.adac1e7120000p-1, 0x1.b418734a90000p-1, 0x1.ba769b39e8000p-1, 0x1.c0c6d447c8000p-1, 0x1.c7095ae920000p-1,
     0x1.cd3e6a0ca8000p-1, 0x1.d3663b27f0000p-1, 0x1.d9810643d8000p-1, 0x1.df8f020868000p-1, 0x1.e59063c880000p-1,
     0x1.eb855f8ca8000p-1, 0x1.f16e281db8000p-1, 0x1.f74aef0ef8000p-1, 0x1.fd1be4c7f0000p-1},
    // lo[j]: the rest of it
    {0x1.e10ba1463d48cp-40, 0x1.9a0d857e2f4b2p-40, 0x1.55b53fce557fdp-40, -0x1.c823f46e8a2bep-45,
     -0x1.cca1e46534b24p-40, -0x1.694d30fc17716p-42, -0x1.a906bc63888e5p-40, -0x1.1658678e6180cp-44,
     -0x1.fb003b2b4fb7ap-40, 0x1.c383cd11362f4p-41, -0x1.64213d272bed9p-40, 0x1.a9334d525e1edp-41,
     0x1.804528474da30p-41, -0x1.f1f4f5c753fabp-43, -0x1.95477e8443f5bp-40, 0x1.1203fa482900bp-44,
     -0x1.a52b0046bb944p-40, 0x1.ee99254b5c0b9p-40, -0x1.310572b05468cp-44, -0x1.376fbcf7f316cp-40,
     0x1.197e845877c95p-41, 0x1.f4a52f8e8a811p-42, -0x1.bf382f3266ecdp-40, 0x1.61f33c897020dp-40,
     0x1.b2632e8306321p-41, -0x1.de05866d2bf99p-42, -0x1.90c4d0a037194p-48, -0x1.f85558435ec8ap-42,
     -0x1.b8b1ec6aebd76p-40, 0x1.76b100b1f6c61p-41, 0x1.26faeb9870946p-45, -0x1.a046240f0ea2dp-40,
     0x1.f92cc0a9688d0p-40, 0x1.162432a1b8df7p-41, -0x1.fd122dbea4062p-42, 0x1.ce1cf2b20a4a8p-43,
     -0x1.89dbb0bc5d818p-40, -0x1.e3939e8e4d05ep-40, 0x1.434adcde7edc8p-41, 0x1.8246f8e527755p-40,
     0x1.e1513c28e180ep-42, -0x1.38518d3919b17p-41, 0x1.32b9861ab04c9p-40, -0x1.875005351ded5p-40,
     -0x1.367b25968abd8p-43, 0x1.ddf360962d7acp-40, 0x1.596b9cb373ea6p-40, -0x1.faff05d54fe46p-41,
     0x1.12ce913d7a827p-41, 0x1.063444cb7ab64p-40, -0x1.be640c51d93c5p-40, 0x1.17b8b6c4f846cp-46,
     -0x1.b4df2be6eb7abp-40, -0x1.11669fc6ff575p-40, -0x1.e378761633cc4p-41, 0x1.20fbfd5902a1ep-42,
     0x1.8ea934ac76088p-40, -0x1.9ec5700a3ac0fp-41, 0x1.7958fed540c9ap-40, 0x1.16719bc9348fdp-40,
     0x1.1f87e4a9cc778p-42, -0x1.39f165275ede4p-42, 0x1.7d75c58973ce6p-40, 0x1.57cb86e584c32p-40},
    // t[j]: 2^(j/64)
    {0x1.0000000000000p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0874518759bc8p+0, 0x1.0b5586cf9890fp+0,
     0x1.0e3ec32d3d1a2p+0, 0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0, 0x1.172b83c7d517bp+0, 0x1.1a35beb6fcb75p+0,
     0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0, 0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0,
     0x1.2d285a6e4030bp+0, 0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0, 0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0,
     0x1.3dea64c123422p+0, 0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0, 0x1.4bfdad5362a27p+0,
     0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0, 0x1.56f4736b527dap+0, 0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0,
     0x1.6247eb03a5585p+0, 0x1.6623882552225p+0, 0x1.6a09e667f3bcdp+0, 0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0,
     0x1.75feb564267c9p+0, 0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0, 0x1.868d99b4492edp+0,
     0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0, 0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0, 0x1.9c49182a3f090p+0,
     0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0, 0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0,
     0x1.b7f76f2fb5e47p+0, 0x1.bcc1e904bc1d2p+0, 0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0, 0x1.cb720dcef9069p+0,
     0x1.d072d4a07897cp+0, 0x1.d5818dcfba487p+0, 0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
     0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0, 0x1.fa7c1819e90d8p+0},
    // tl[j]: the rest of it
    {0x0.0p+0, -0x1.19083535b085dp-56, 0x1.d73e2a475b465p-55, 0x1.186be4bb284ffp-57, 0x1.8a62e4adc610bp-54,
     0x1.03a1727c57b53p-59, -0x1.6c51039449b3ap-54, -0x1.32fbf9af1369ep-54, -0x1.19041b9d78a76p-55,
     0x1.e5b4c7b4968e4p-55, 0x1.e016e00a2643cp-54, 0x1.dc775814a8495p-55, 0x1.9b07eb6c70573p-54,
     0x1.2bd339940e9d9p-55, 0x1.612e8afad1255p-55, 0x1.0024754db41d5p-54, 0x1.6f46ad23182e4p-55,
     0x1.32721843659a6p-54, -0x1.63aeabf42eae2p-54, -0x1.5e436d661f5e3p-56, 0x1.ada0911f09ebcp-55,
     -0x1.ef3691c309278p-58, 0x1.89b7a04ef80d0p-59, 0x1.3c1a3b69062f0p-56, 0x1.d4397afec42e2p-56,
     -0x1.4b309d25957e3p-54, -0x1.07abe1db13cadp-55, 0x1.9bb2c011d93adp-54, 0x1.6324c054647adp-54,
     0x1.ba6f93080e65ep-54, -0x1.383c17e40b497p-54, -0x1.bb60987591c34p-54, -0x1.bdd3413b26456p-54,
     -0x1.bbe3a683c88abp-57, -0x1.16e4786887a99p-55, -0x1.0245957316dd3p-54, -0x1.41577ee04992fp-55,
     0x1.05d02ba15797ep-56, -0x1.d4c1dd41532d8p-54, -0x1.fc6f89bd4f6bap-54, 0x1.6e9f156864b27p-54,
     0x1.5cc13a2e3976cp-55, -0x1.75fc781b57ebcp-57, -0x1.d185b7c1b85d1p-54, 0x1.c7c46b071f2bep-56,
     -0x1.359495d1cd533p-54, -0x1.d2f6edb8d41e1p-54, 0x1.0fac90ef7fd31p-54, 0x1.7a1cd345dcc81p-54,
     -0x1.2805e3084d708p-57, -0x1.5584f7e54ac3bp-56, 0x1.23dd07a2d9e84p-55, 0x1.11065895048ddp-55,
     0x1.2884dff483cadp-54, 0x1.503cbd1e949dbp-56, -0x1.cbc3743797a9cp-54, 0x1.2ed02d75b3707p-55,
     0x1.c2300696db532p-54, -0x1.1a5cd4f184b5cp-54, 0x1.39e8980a9cc8fp-55, -0x1.e9c23179c2893p-54,
     0x1.dc7f486a4b6b0p-54, 0x1.9d3e12dd8a18bp-54, 0x1.74853f3a5931ep-55},
};

// Copies the tables into shared memory (every thread of the CTA calls it; a
// barrier is needed before they are used).
__device__ __forceinline__ void load_pow_tables(PowTables& sm) {
  constexpr int n = sizeof(PowTables) / sizeof(double);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    reinterpret_cast<double*>(&sm)[i] = reinterpret_cast<const double*>(&g_pow_tables)[i];
}

__device__ __forceinline__ double pow_gamma(double x, const PowTables& T) {
  // log2(1 + r) / r and (2^f - 1) / f: (-1)^(k+1) / (k ln 2) and (ln 2)^k / k!
  constexpr double L[8] = {0x1.71547652b82fep+0,  -0x1.71547652b82fep-1, 0x1.ec709dc3a03fdp-2,  -0x1.71547652b82fep-2,
                           0x1.2776c50ef9bfep-2,  -0x1.ec709dc3a03fdp-3, 0x1.a61762a7aded9p-3,  -0x1.71547652b82fep-3};
  constexpr double X[6] = {0x1.62e42fefa39efp-1, 0x1.ebfbdff82c58fp-3, 0x1.c6b08d704a0c0p-5,
                           0x1.3b2ab6fba4e77p-7, 0x1.5d87fe78a6731p-10, 0x1.430912f86c787p-13};
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(b >> 52);  // sign and exponent
  // 2^-650 < x < 2^650: the power stays normal
  if (ex < 1023 - 650 || ex > 1023 + 649) return pow(x, kGamma);
  const double m = __longlong_as_double((long long)((b & 0xfffffffffffffull) | 0x3ff0000000000000ull));
  const int j = (int)(b >> 46) & 63;
  const double r = fma(m, T.c[j], -1.0);
  double p = L[7];
#pragma unroll
  for (int k = 6; k >= 0; --k) p = fma(p, r, L[k]);
  const double yl = fma(r, p, T.lo[j]);
  // E as a double by its bits: 2^52 + 2^51 + E less 2^52 + 2^51
  const double E = __longlong_as_double(0x4338000000000000ll + (ex - 1023)) - 0x1.8p52;
  const double H = E + T.hi[j];  // exact
  const double z = kGamma * H, zl = fma(kGamma, yl, fma(kGamma, H, -z));
  const double s = fma(z, 64.0, 0x1.8p52);
  const int n = (int)(unsigned)__double_as_longlong(s);  // 64 z to the nearest integer
  const double f = fma(s - 0x1.8p52, -1.0 / 64, z) + zl;
  double q = X[5];
#pragma unroll
  for (int k = 4; k >= 0; --k) q = fma(q, f, X[k]);
  q *= f;
  const double v = fma(T.t[n & 63], q, T.tl[n & 63]) + T.t[n & 63];
  return __longlong_as_double(__double_as_longlong(v) + ((long long)(n >> 6) << 52));
}

}  // namespace mw
