// ziv64.cuh -- correctly rounded pow(x, 1/3), acos, cos and sin in two phases.
//
// crmath.cuh evaluates these functions to about 100 bits, which takes
// hundreds of FP64 operations.  Here a first phase evaluates them to about 70
// bits in a tenth of that and rounds, if no FP64 rounding boundary lies
// within its error (Ziv, "Fast evaluation of elementary mathematical
// functions with correctly rounded last bit", ACM TOMS 17 (1991)); where one
// does (about one argument in 10^4), it clears `ok` and the caller takes the
// functions of crmath.cuh.  Where the first phase decides, both give the
// correctly rounded result, so the same bits.
//
// Methods:
//   * sine and cosine of t in [0, 1.57]: angle addition from the values at
//     k/64 (double-double table) and the Taylor series of t - k/64, its
//     leading products and sums exact (TwoProd by fused multiply-add, TwoSum);
//   * arc cosine: two Newton steps on cos(t) = |z| from an FP32 value, the
//     second from a residual of the accuracy of the cosine above; for z < 0,
//     pi minus that; next to z = -1 its series;
//   * cube root: the series of (1 + rho)^(1/3) about an FP32 cube root, whose
//     cube is exact, and the factor a^(y - 1/3) = 1 + e for the exponent
//     y = fl(1/3) = (1 - 2^-54) / 3, e from an FP32 logarithm.
#pragma once

#include <math.h>

#include "crmath.cuh"
#include "ieee64.cuh"

namespace ziv64 {

using crm::add;
using crm::dd;
using crm::fmad;
using crm::mul;
using crm::sub;
using crm::two_sum;

// sin(k/64) and cos(k/64) as double-double: hi, lo, hi, lo
#if defined(__CUDACC__)
__device__
#endif
static const double SINCOS[102][4] = {
    {0x0.0p+0, 0x0.0p+0, 0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.fffaaaaeeeed5p-7, -0x1.2ab639a9f0776p-63, 0x1.fff000155549fp-1, 0x1.28a28a03a5ef3p-55},
    {0x1.ffeaaaeeee86fp-6, -0x1.cd406fb224ae2p-60, 0x1.ffc00155527d3p-1, -0x1.3b54492d89b5bp-55},
    {0x1.7fdc01032fba9p-5, -0x1.599bdf46e997ap-59, 0x1.ff7006bfdf99fp-1, -0x1.8b3b560648d5fp-56},
    {0x1.ffaaaeeed4edbp-5, -0x1.2d16d32684b69p-59, 0x1.ff0015549f4d3p-1, 0x1.328387b99426fp-55},
    {0x1.3facb12d1755bp-4, -0x1.921915299468bp-58, 0x1.fe7034129ef6fp-1, -0x1.cbf4337c96f97p-57},
    {0x1.7f701032550e4p-4, 0x1.afc2d1800501ap-60, 0x1.fdc06bf7e6b9bp-1, 0x1.31902b535f8dbp-55},
    {0x1.bf1b78568391dp-4, 0x1.e91841dea4cc8p-58, 0x1.fcf0c800e99b1p-1, 0x1.ea3d786d186acp-57},
    {0x1.feaaeee86ee36p-4, -0x1.afcb2bcc6f03bp-59, 0x1.fc015527d5bd3p-1, 0x1.b68f35094efb8p-55},
    {0x1.1f0d3d7afceafp-3, -0x1.6ef95099769a5p-57, 0x1.faf22263c4bd3p-1, -0x1.52ace133a2769p-58},
    {0x1.3eb312c5d66cbp-3, 0x1.47d666b66cb91p-57, 0x1.f9c340a7cc428p-1, 0x1.c5b6b063b7462p-55},
    {0x1.5e44fcfa126f3p-3, -0x1.6f443063f89b6p-57, 0x1.f874c2e1eecf6p-1, -0x1.c6514e1332b16p-55},
    {0x1.7dc102fbaf2b5p-3, 0x1.5ab50e23c97c3p-59, 0x1.f706bdf9ece1cp-1, -0x1.698c80c36dcb4p-55},
    {0x1.9d252d0cec312p-3, 0x1.9c43d80b1137dp-58, 0x1.f57948cff6797p-1, 0x1.e3a0d3e03b1d4p-57},
    {0x1.bc6f84edc6199p-3, 0x1.9c1a56a7b0cabp-57, 0x1.f3cc7c3b3d16ep-1, -0x1.21a3ad28a3494p-57},
    {0x1.db9e15fb5a5d0p-3, -0x1.32e20d6cc6fc2p-57, 0x1.f20073086649fp-1, 0x1.b940416c1984bp-56},
    {0x1.faaeed4f31577p-3, -0x1.15d88508e32b8p-57, 0x1.f01549f7deea1p-1, 0x1.d3c1e99e5cafdp-55},
    {0x1.0cd00cef36436p-2, -0x1.9fb0a0c93e2b4p-56, 0x1.ee0b1fbc0f11cp-1, -0x1.bfd2380bbc3b1p-59},
    {0x1.1c37d64c6b876p-2, 0x1.46076fe0dcff4p-56, 0x1.ebe214f76efa8p-1, -0x1.02f9f12ba543ep-55},
    {0x1.2b8ddc43eb49fp-2, 0x1.1553899f2d807p-57, 0x1.e99a4c3a7cd83p-1, -0x1.2264b1bc53ce8p-55},
    {0x1.3ad129769d3d8p-2, 0x1.03d550487839ap-63, 0x1.e733ea0193d40p-1, -0x1.6428b3546ce13p-55},
    {0x1.4a00c9b0f3d20p-2, 0x1.823ba6bb08eadp-56, 0x1.e4af14b2a449cp-1, -0x1.68ca02e8a6833p-55},
    {0x1.591bc9fa2f597p-2, 0x1.7c74bac3fe0cbp-57, 0x1.e20bf49acd6c1p-1, -0x1.660aec7ef636bp-58},
    {0x1.682138a38d7f7p-2, -0x1.d889202444aadp-56, 0x1.df4ab3ebd875ep-1, -0x1.e2d8a7e6736c4p-55},
    {0x1.7710255764214p-2, -0x1.6ead7314bb6cep-57, 0x1.dc6b7eb995912p-1, 0x1.4b364776dcd35p-58},
    {0x1.85e7a12826949p-2, 0x1.8a40e9b5face0p-56, 0x1.d96e82f71a9dcp-1, 0x1.ff61bd5d2039dp-55},
    {0x1.94a6be9f546c5p-2, -0x1.69ce13e683f58p-56, 0x1.d653f073e4040p-1, -0x1.76236434bec37p-55},
    {0x1.a34c91cc50ccap-2, -0x1.a310e3b50cecdp-58, 0x1.d31bf8d8d7c06p-1, 0x1.e60dd3089cbddp-56},
    {0x1.b1d8305321617p-2, -0x1.ae242cb99f519p-56, 0x1.cfc6cfa52ad9fp-1, 0x1.8b5b5508f2a0dp-55},
    {0x1.c048b17b140a3p-2, 0x1.19fe6757e9fa7p-57, 0x1.cc54aa2b2972ep-1, 0x1.4ee162ba83a98p-57},
    {0x1.ce9d2e3d4a51fp-2, -0x1.2fc8a12dae298p-57, 0x1.c8c5bf8ce1a84p-1, 0x1.ab3d1a1590123p-56},
    {0x1.dcd4c15329c9ap-2, 0x1.0d4c6e171fd9ap-56, 0x1.c51a48b8b175ep-1, -0x1.1bbb43b9aa880p-57},
    {0x1.eaee8744b05f0p-2, -0x1.789b43c9b027dp-58, 0x1.c1528065b7d50p-1, -0x1.892111312e828p-55},
    {0x1.f8e99e76abc97p-2, 0x1.9d950af2d00a3p-58, 0x1.bd6ea310294f5p-1, 0x1.31bbcc88c109dp-56},
    {0x1.0362939c69955p-1, -0x1.2d8cd78397b01p-55, 0x1.b96eeef58840ep-1, 0x1.45a3cc78fade0p-58},
    {0x1.0a4021e9e1001p-1, -0x1.6f643a13914f6p-55, 0x1.b553a410c104ep-1, 0x1.8ff7947027a15p-58},
    {0x1.110d0c4b69c3bp-1, 0x1.d918998809981p-55, 0x1.b11d04162a4c6p-1, 0x1.1dd561efbc0c2p-56},
    {0x1.17c8e5f2eedb0p-1, 0x1.35e57102e2488p-57, 0x1.accb526f69de5p-1, 0x1.8fb6a8dd6b6ccp-55},
    {0x1.1e7343236574cp-1, 0x1.22a3fa4f41d5ap-56, 0x1.a85ed4373e02dp-1, 0x1.9be06385ec792p-57},
    {0x1.250bb93788bbbp-1, 0x1.ea3d02457bccep-56, 0x1.a3d7d0352bdcfp-1, -0x1.68dbaeca19669p-55},
    {0x1.2b91dea88421ep-1, -0x1.fa371db216ab0p-55, 0x1.9f368ed912f85p-1, -0x1.1d200c5791606p-55},
    {0x1.32054b148bc4fp-1, 0x1.f6b42095a135bp-55, 0x1.9a7b5a36a6514p-1, 0x1.722cfcc9fa7a9p-55},
    {0x1.386597456282bp-1, -0x1.10fada93b07a8p-56, 0x1.95a67e00cb1fdp-1, -0x1.0befda21f862dp-55},
    {0x1.3eb25d36cd53ap-1, -0x1.be570e1570fc0p-58, 0x1.90b84784ddaf7p-1, -0x1.0feb10ab93b87p-56},
    {0x1.44eb381cf386bp-1, -0x1.3ed6c1e6a5505p-55, 0x1.8bb105a5dc900p-1, 0x1.863e03e9474c1p-55},
    {0x1.4b0fc46aab761p-1, 0x1.0da05738cc59cp-61, 0x1.869108d77a6c6p-1, 0x1.338ffe2bfe9ddp-56},
    {0x1.511f9fd7b351cp-1, -0x1.5c0e861c48831p-55, 0x1.8158a31916d5dp-1, -0x1.de8b90b8228dep-57},
    {0x1.571a6966d59b3p-1, 0x1.c843b4d0fb197p-58, 0x1.7c0827f09e54fp-1, -0x1.c73d6d72aee68p-57},
    {0x1.5cffc16bf8f0dp-1, 0x1.96cb370eb578ap-55, 0x1.769fec655211fp-1, -0x1.827d5cf8c68c5p-57},
    {0x1.62cf49921ac79p-1, -0x1.edd9855b6241ap-55, 0x1.712046fa77678p-1, 0x1.425b0a5029c81p-55},
    {0x1.6888a4e134b2fp-1, -0x1.6b7d37644d5e6p-55, 0x1.6b898fa9efb5dp-1, 0x1.15ac786ccf4b2p-56},
    {0x1.6e2b77c40bde1p-1, -0x1.0e729857fad53p-56, 0x1.65dc1fdeb8cbap-1, -0x1.97c1b47337c77p-58},
    {0x1.73b7680dea578p-1, -0x1.2248306dc12a2p-56, 0x1.6018526f563dfp-1, 0x1.46ca5e0e432d0p-55},
    {0x1.792c1d0041d52p-1, -0x1.abf05eeb354ebp-55, 0x1.5a3e839824077p-1, 0x1.428aa2759be62p-55},
    {0x1.7e893f5037959p-1, 0x1.0eefbaa650c4cp-55, 0x1.544f10f592ca5p-1, -0x1.e7ae8e6c7a62fp-55},
    {0x1.83ce792c1906ep-1, -0x1.f3899682b4a7dp-56, 0x1.4e4a597e4e10ep-1, 0x1.ccd992849f6c8p-56},
    {0x1.88fb7640b8da2p-1, -0x1.49987c11efaa3p-55, 0x1.4830bd7d4ceb3p-1, 0x1.df77ff20d5448p-55},
    {0x1.8e0fe3beb42f8p-1, 0x1.324c55de9ed0bp-55, 0x1.42029e8bcd474p-1, 0x1.995705e2a2526p-55},
    {0x1.930b705f9f85ap-1, -0x1.09ae60f413f40p-61, 0x1.3bc05f8b3a656p-1, 0x1.dab7124aa8c6dp-55},
    {0x1.97edcc6b1b193p-1, 0x1.93523ce2c8213p-55, 0x1.356a649efec9dp-1, -0x1.500caf33eb802p-60},
    {0x1.9cb6a9bbce64bp-1, -0x1.4f3e7a32f8d0cp-56, 0x1.2f011326420e4p-1, 0x1.8e30efe9e96c2p-56},
    {0x1.a165bbc44a6f1p-1, -0x1.25d120e45579ap-55, 0x1.2884d1b592f81p-1, -0x1.099bbe3a4f76bp-55},
    {0x1.a5fab793d29c8p-1, 0x1.7482b1e8e6d85p-55, 0x1.21f608107e37ap-1, -0x1.0a3f22ad63580p-55},
    {0x1.aa7553db0bb41p-1, -0x1.ddb562ca148f2p-56, 0x1.1b551f2312386p-1, 0x1.a85cdf15867a6p-55},
    {0x1.aed548f090ceep-1, 0x1.06374f484e288p-59, 0x1.14a280fb5068cp-1, -0x1.b71edcc9344bcp-55},
    {0x1.b31a50d56de8fp-1, -0x1.4d46c15ba8ea7p-55, 0x1.0dde98c28c628p-1, -0x1.b0e8e5bebb55bp-55},
    {0x1.b74427397fca2p-1, 0x1.da351af253ee4p-55, 0x1.0709d2b6b95eep-1, -0x1.71cc4ee678c32p-55},
    {0x1.bb52897fb9032p-1, 0x1.953ad2e7b7f06p-55, 0x1.00249c23a6603p-1, -0x1.9b0cfbef87821p-57},
    {0x1.bf4536c24bb85p-1, 0x1.97632053703f0p-55, 0x1.f25ec6b852fc2p-2, 0x1.445cbca9a80a8p-56},
    {0x1.c31befd6b7f98p-1, -0x1.767b85f1a5287p-55, 0x1.e4552f6675828p-2, -0x1.027885c508dc9p-56},
    {0x1.c6d67751be646p-1, 0x1.d163b7b4fe389p-56, 0x1.d62d52e9fdfa9p-2, 0x1.f6eae4ae67d35p-58},
    {0x1.ca74918b36d3dp-1, -0x1.01b062b75945ep-55, 0x1.c7e813bf862f7p-2, 0x1.909f60366377fp-56},
    {0x1.cdf604a1cadcep-1, -0x1.6b50757f2fa40p-56, 0x1.b9865639d0596p-2, -0x1.931bd06786cb9p-56},
    {0x1.d15a987e93dfcp-1, 0x1.7d89c8d349c80p-55, 0x1.ab09007382047p-2, 0x1.14a41d3d11354p-57},
    {0x1.d4a216d89c717p-1, 0x1.d4810b29c8736p-55, 0x1.9c70fa40c279dp-2, -0x1.6346cef9b5fa7p-58},
    {0x1.d7cc4b3844e67p-1, 0x1.3f6e971be3f02p-55, 0x1.8dbf2d20bd903p-2, 0x1.0ce77f57be8cbp-56},
    {0x1.dad902fa8ac87p-1, 0x1.ea5e370875907p-58, 0x1.7ef4842f0bccdp-2, 0x1.83529407722f1p-56},
    {0x1.ddc80d5433024p-1, -0x1.5a6ac4bf29104p-55, 0x1.7011ec1500bd6p-2, 0x1.21c45557ddc22p-56},
    {0x1.e0993b54d68f6p-1, -0x1.f26cc0d6a7cecp-58, 0x1.611852fae0769p-2, -0x1.71272938d7ae8p-57},
    {0x1.e34c5fe9d17ebp-1, 0x1.f2ef95683b7d1p-61, 0x1.5208a878fd239p-2, 0x1.c83eff91c5e12p-58},
    {0x1.e5e14fe11418cp-1, 0x1.f26492c1c25a0p-57, 0x1.42e3dd88bd952p-2, -0x1.353a9f74bf255p-57},
    {0x1.e857e1ebd5fd5p-1, -0x1.9d8e945823d2ap-56, 0x1.33aae4758dbefp-2, -0x1.d058881847909p-57},
    {0x1.eaafeea12b0c4p-1, 0x1.d7af5fa4a5c74p-57, 0x1.245eb0cdba154p-2, -0x1.c4555428fdfb4p-57},
    {0x1.ece9508079f14p-1, 0x1.2b2c513ff0cf6p-55, 0x1.1500375336bc5p-2, 0x1.9a39da062c982p-57},
    {0x1.ef03e3f3d42a2p-1, 0x1.0572b0573c404p-59, 0x1.05906dec537dap-2, 0x1.12c3f77448473p-61},
    {0x1.f0ff87522f62cp-1, -0x1.fd676d1225f8cp-55, 0x1.ec209728baee8p-3, -0x1.c4601d778aa03p-58},
    {0x1.f2dc1ae18002ep-1, -0x1.be7521dc7c740p-58, 0x1.cd0190985ef77p-3, -0x1.11be2ffbeed45p-58},
    {0x1.f49980d8b4cc7p-1, -0x1.881ca7411b5f8p-56, 0x1.adc5ba1564320p-3, -0x1.6c8ed88c3e7a8p-60},
    {0x1.f6379d619369dp-1, 0x1.6b296ac1928abp-55, 0x1.8e6f075a987d6p-3, 0x1.a57e7fd1918d8p-62},
    {0x1.f7b6569a75cf8p-1, -0x1.14cbbb7799b36p-56, 0x1.6eff6dd08af8dp-3, -0x1.1bb80ce3b15c7p-57},
    {0x1.f9159497e853fp-1, 0x1.66c77a4219a37p-56, 0x1.4f78e46e35a46p-3, -0x1.82bbe6c49f2b0p-59},
    {0x1.fa55416628652p-1, 0x1.c8aa2f23a4669p-55, 0x1.2fdd63998e1b6p-3, 0x1.09edc7d2bed7dp-58},
    {0x1.fb75490a83c2cp-1, 0x1.d9fbeed39ae46p-55, 0x1.102ee507ff5f0p-3, -0x1.77ec7eee89a9bp-57},
    {0x1.fc7599849827bp-1, 0x1.feee53c5da7cfp-56, 0x1.e0dec73d9d533p-4, 0x1.698b2d527d376p-59},
    {0x1.fd5622cf734eap-1, 0x1.576f5c33de713p-55, 0x1.a141b6a6da89dp-4, 0x1.dd0de04944ab6p-58},
    {0x1.fe16d6e293400p-1, -0x1.53fdcb5496323p-55, 0x1.618a921772ba3p-4, -0x1.2e89936f086fap-58},
    {0x1.feb7a9b2c6d8bp-1, -0x1.0c8f40129a886p-56, 0x1.21bd54fc5f9a7p-4, 0x1.0fcb936b1ce7ep-58},
    {0x1.ff389132ee7c6p-1, 0x1.400f472356ae9p-55, 0x1.c3bbf8484388ap-5, -0x1.52bb3d8120de5p-59},
    {0x1.ff9985549ce69p-1, 0x1.57aa6cfbfc93dp-55, 0x1.43e10afde8436p-5, -0x1.fc499d21a9320p-60},
    {0x1.ffda80089810bp-1, -0x1.e60e93f33d826p-56, 0x1.87e3bf7bb4f99p-6, 0x1.4aa5c3ca7c944p-61},
    {0x1.fffb7d3f3a253p-1, -0x1.2d4934e6c1f3dp-56, 0x1.0fd9d5c093df5p-7, -0x1.50076d7383a18p-64},
    {0x1.fffc7ae8b279cp-1, -0x1.1fa8b32bcbba5p-55, -0x1.e049a1f9ed9acp-8, 0x1.3baca337c3df0p-63},
};

struct SinCos {
    dd s, c;    // sin(k/64), cos(k/64)
};
CRM_FN SinCos table(int k)
{
    return {{SINCOS[k][0], SINCOS[k][1]}, {SINCOS[k][2], SINCOS[k][3]}};
}

// hi + lo rounded; ok cleared unless every value within err of it rounds alike
CRM_FN double round_checked(double hi, double lo, double err, bool& ok)
{
    const double r = add(hi, add(lo, err));
    ok = ok && ieee64::bits(r) == ieee64::bits(add(hi, sub(lo, err)));
    return r;
}

// x a - y b for |d| <= 1/128, with a = 1 - d^2/2 + ..., b = d - d^3/6 + ... the
// cosine and sine of d: cos(t + d) for x = cos t, y = sin t, and
// sin(t + d) = cos-like with y = -cos t.  hi + lo to 2^-73 (2^-74.5 measured).
CRM_FN void rotate(dd x, dd y, double d, double& hi, double& lo)
{
    const double d2 = mul(d, d), e2 = fmad(d, d, -d2);
    // d^3/6 (1 - d^2/20 (1 - d^2/42)) and d^4/24 (1 - d^2/30 (1 - d^2/56)) with the square's rounding
    const double ps = fmad(d2, fmad(d2, -0x1.a01a01a01a01ap-13, 0x1.1111111111111p-7), -0x1.5555555555555p-3);
    const double sd = mul(mul(d, d2), ps);                  // sin d - d
    const double pc = fmad(d2, fmad(d2, 0x1.a01a01a01a01ap-16, -0x1.6c16c16c16c17p-10), 0x1.5555555555555p-5);
    const double cd = fmad(mul(d2, d2), pc, mul(-0.5, e2)); // cos d - (1 - d2/2)
    const double h = mul(-0.5, d2);
    const double p = mul(y.hi, d), pe = fmad(y.hi, d, -p);
    const double m = mul(x.hi, h), me = fmad(x.hi, h, -m);
    const dd s = two_sum(x.hi, -p);
    const dd t = two_sum(s.hi, m);
    hi = t.hi;
    // the small terms, largest (about 2^-24) last
    double z = fmad(x.lo, h, sub(me, pe));
    z = fmad(-y.lo, d, add(z, x.lo));
    z = add(z, fmad(-y.hi, sd, mul(x.hi, cd)));
    lo = add(add(s.lo, t.lo), z);
}

// cos and sin of t in [0, 1.05] (a third of an arc cosine)
CRM_FN void sincos_third(double t, double& c, double& s, bool& ok)
{
    const bool in = t >= 0x1p-8 && t <= 1.5;
    ok = ok && in;
    const int k = in ? (int) rintf((float) t * 64.0f) : 1;
    const double d = sub(t, mul((double) k, 0x1p-6));
    const SinCos T = table(k);
    double hi, lo;
    rotate(T.c, T.s, d, hi, lo);
    c = round_checked(hi, lo, 0x1p-72, ok);
    rotate(T.s, crm::dd_neg(T.c), d, hi, lo);
    s = round_checked(hi, lo, 0x1p-72, ok);
}

// arc cosine of -1 < z < 1
CRM_FN double arccos(double z, bool& ok)
{
    const double w = fabs(z);
    if (z < -1.0 + 0x1p-30 && z >= -1.0) {
        // two coinciding roots of the resolvent: pi - sqrt(2 u) (1 + u / 12 + ...), u = 1 + z exact
        const double u = sub(1.0, w), v = ieee64::sqrt_rn(mul(2.0, u), ok);
        const dd q = two_sum(0x1.921fb54442d18p+1, -fmad(mul(v, u), 0x1.5555555555555p-4, v));
        return round_checked(q.hi, add(q.lo, 0x1.1a62633145c07p-53), 0x1p-66, ok);
    }
    const bool in = w < 1.0 - 0x1p-34;
    ok = ok && in;
    // t0 = 2 asin(sqrt((1 - w) / 2)): to FP32's relative accuracy also near w = 1
    const float t0 = in ? 2.0f * asinf(sqrtf(0.5f * (float) sub(1.0, w))) : 1.0f;
    const int k = (int) rintf(t0 * 64.0f);
    const double t64 = mul((double) k, 0x1p-6);
    const SinCos T = table(k);
    double d = sub((double) t0, t64);
    // Newton: d + (cos(t64 + d) - w) / sin(t64 + d), first in plain FP64
    const double d2 = mul(d, d);
    const double v = mul(d2, fmad(d2, -0x1.5555555555555p-5, 0.5));             // 1 - cos d
    const double u = fmad(mul(d, d2), fmad(d2, 0x1.1111111111111p-7, -0x1.5555555555555p-3), d);   // sin d
    const float sf = (float) fmad(T.c.hi, u, fmad(-T.s.hi, v, T.s.hi));         // sin(t64 + d)
    const double inv = (double) (1.0f / sf);
    const double f = fmad(-T.s.hi, u, fmad(-T.c.hi, v, sub(T.c.hi, w)));
    d = fmad(f, inv, d);
    // then with an accurate residual
    double hi, lo;
    rotate(T.c, T.s, d, hi, lo);
    const double g = add(sub(hi, w), lo);
    const dd t = two_sum(t64, d);
    const double tail = fmad(g, inv, t.lo);
    // the residual's error over the sine, and what the second step leaves
    const double err = fmad(inv, 0x1p-73, fmad(mul(fabs(g), inv), 0x1p-20, 0x1p-74));
    if (z > 0.0) return round_checked(t.hi, tail, err, ok);
    const dd q = two_sum(0x1.921fb54442d18p+1, -t.hi);
    return round_checked(q.hi, add(q.lo, sub(0x1.1a62633145c07p-53, tail)), err, ok);
}

// pow(x, fl(1/3)) for x of 2^-300 to 2^300
CRM_FN double pow_third(double x, bool& ok)
{
    const ieee64::u64 b = ieee64::bits(x);
    const int e = (int) (b >> 52);                       // sign and exponent field
    ok = ok && (unsigned) (e - 723) <= 600u;
    // x = m 2^(3 j), m in [1, 8)
    const int j = (e - 1023 + 3 * 400) / 3 - 400;
    const double m = ieee64::from_bits((b & 0xfffffffffffffull) | ((ieee64::u64) (e - 3 * j) << 52));
    const float c = cbrtf((float) m);
    const double c0 = (double) c;
    const double q2 = mul(c0, c0);                       // exact: 48 bits
    const double p = mul(q2, c0), pe = fmad(q2, c0, -p);
    const double rho = ieee64::div(sub(sub(m, p), pe), p, ok);   // (m - c0^3) / c0^3, about 2^-22
    // c0 ((1 + rho)^(1/3) - 1) and the exponent's e = -(2^-54 / 3) ln x
    const double s = fmad(rho, fmad(rho, fmad(rho, -0x1.511e8d2b3183bp-5, 0x1.f9add3c0ca458p-5), -0x1.c71c71c71c71cp-4),
                          0x1.5555555555555p-2);
    const double lnx = (double) (logf((float) m) + (float) (3 * j) * 0.693147181f);
    const double corr = mul(c0, fmad(rho, s, mul(lnx, -0x1.5555555555555p-56)));
    const double y = round_checked(c0, corr, 0x1p-68, ok);
    return ieee64::from_bits(ieee64::bits(y) + ((ieee64::u64) (ieee64::i64) j << 52));
}

} // namespace ziv64
