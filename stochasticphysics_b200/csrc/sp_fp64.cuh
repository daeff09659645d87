// sp_fp64.cuh — double-precision sines, cosines and Box-Muller pairs of the step kernels.
//
// Inlined straight-line code for the arguments an SDE step produces.  The library's sincos,
// log and sincospi accept every double: inlined, their range reduction and special cases
// overflow the instruction cache, and called (the form these replace) the five angles of a
// Brown+Neel step and the pairs of its noise run one after another, each waiting out its
// own chain of 8-cycle FP64 operations.  Inlined and branch-free they interleave.
// Brown+Neel Euler/spherical, FP64: see step_min_blocks in sp_kernels.cuh for the figures.
//
// Methods: Cody-Waite reduction by pi/2 in three parts and minimax polynomials (W. J. Cody,
// W. Waite, Software Manual for the Elementary Functions, 1980); P. T. P. Tang's
// table-driven logarithm (ACM TOMS 16, 1990) in the layout of log() in ARM's Optimized
// Routines (table index and exponent from the high word's offset, one exact fused product per
// argument, the order of the last additions); Goldschmidt's square root iteration with a
// final residual correction; Newton's iteration for reciprocals, P. Markstein's quotient.  The
// coefficients are Remez fits computed for this file with 300-bit arithmetic; the table's rows
// are c ~ 1 / centre with 18 fraction bits and -ln c as a multiple of 2^-42 plus a remainder.
// Largest errors against 113-bit arithmetic: tests/test_fp64_math_cpu.py compiles this file for
// the host and checks them (tests/test_fp64_nan_cpu.py: and that all are finite).  Against
// CUDA's own on the device (tests/test_gpu_fp64_math.py): sine and cosine of a step's angles
// 0.350 and 0.365 ulp root mean square, CUDA's sincos 0.350 and 0.367, largest 1.30 and 1.38,
// CUDA's 1.31 and 1.35; reciprocals and quotients equal bit for bit.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define SP_HD __host__ __device__ __forceinline__
#else
#define SP_HD inline
#endif

namespace sp {

SP_HD int fp64_hi(double x) {
#ifdef __CUDA_ARCH__
    return __double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return static_cast<int>(u >> 32);
#endif
}
SP_HD int fp64_lo(double x) {
#ifdef __CUDA_ARCH__
    return __double2loint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return static_cast<int>(static_cast<uint32_t>(u));
#endif
}
SP_HD double fp64_make(int hi, int lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(hi, lo);
#else
    const uint64_t u = (static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32) | static_cast<uint32_t>(lo);
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
// products that must not be fused into a later addition: every kernel that draws a Wiener
// increment has to round it the same way
SP_HD double fp64_mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
// first approximation of 1/sqrt(x), x normal and positive
SP_HD double fp64_rsqrt_seed(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
#else
    return static_cast<double>(1.0f / sqrtf(static_cast<float>(x)));
#endif
}

// first approximation of 1/x, x normal
SP_HD double fp64_rcp_seed(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
#else
    return static_cast<double>(1.0f / static_cast<float>(x));
#endif
}

struct SinCosD {
    double s, c;
};

// sin and cos of r + q pi/2, |r| <= pi/4 (a little more is harmless)
SP_HD SinCosD sincos_quadrant(double r, int q) {
    const double z = r * r;
    double p = fma(z, 0x1.5d9300f0397f2p-33, -0x1.ae5e663a6459ep-26);
    p = fma(z, p, 0x1.71de3577b65eep-19);
    p = fma(z, p, -0x1.a01a019c11990p-13);
    p = fma(z, p, 0x1.111111110f87ap-7);
    p = fma(z, p, -0x1.5555555555549p-3);
    double t = fma(z, -0x1.8fae9c69b38f2p-37, 0x1.1ee9ebe913ef4p-29);
    t = fma(z, t, -0x1.27e4f809f07b0p-22);
    t = fma(z, t, 0x1.a01a019cb1bd8p-16);
    t = fma(z, t, -0x1.6c16c16c1517ep-10);
    t = fma(z, t, 0x1.555555555554cp-5);
    t = fma(z, t, -0.5);
    const double s = fma(r * z, p, r), c = fma(z, t, 1.0);
    // odd quadrants exchange the two; signs: sin negative in quadrants 2, 3, cos in 1, 2
    const bool odd = q & 1;
    const double a = odd ? c : s, b = odd ? s : c;
    SinCosD o;
    o.s = fp64_make(fp64_hi(a) ^ ((q << 30) & static_cast<int>(0x80000000u)), fp64_lo(a));
    o.c = fp64_make(fp64_hi(b) ^ (((q + 1) << 30) & static_cast<int>(0x80000000u)), fp64_lo(b));
    return o;
}

// |x| < 8192: angles of a step stay within a few turns.  The quadrant number
// (|k| < 2^13) times the 40-bit parts is exact.
constexpr int kSincosRangeHigh = 0x40c00000;  // high word of 8192
SP_HD SinCosD sincos_reduced(double x) {
    const double magic = 0x1.8p52;  // adding it rounds to an integer held in the low word
    const double k = fma(x, 0x1.45f306dc9c883p-1, magic);
    const int q = fp64_lo(k);
    const double kd = k - magic;
    double r = fma(-kd, 0x1.921fb54442000p+0, x);
    r = fma(-kd, 0x1.a308d31318000p-41, r);
    r = fma(-kd, 0x1.8a2e03707344ap-81, r);
    return sincos_quadrant(r, q);
}

// sin and cos of 2 pi (b + 1/2) 2^-32: the quadrant is b's nearest multiple of 2^30, the
// rest is an integer, so the reduction is exact
SP_HD SinCosD sincos_turn(uint32_t b) {
    const uint32_t q = (b + 0x20000000u) >> 30;
    const uint32_t n = 2u * (b - (q << 30)) + 1u;             // odd integer in [-2^30, 2^30], units of half an ulp of b
    const double d = fp64_make(0x43200000, static_cast<int>(n ^ 0x80000000u)) - (0x1p51 + 0x1p30);  // n / 2
    // 2 pi 2^-32 as 22 bits, whose product with d is exact, and the rest
    return sincos_quadrant(fma(d, 0x1.5110b4611a626p-52, d * 0x1.921fb00000000p-30), static_cast<int>(q));
}

// {c, ln-part multiple of 2^-42, remainder} of the 128 intervals of [0.75, 1.5): steps 2^-8
// below 1 and 2^-7 above; the interval that ends at 1 has c = 1, so that the logarithm
// keeps its relative accuracy there
constexpr int kLogRows = 128;
struct LogTab {
    double c[kLogRows];
    double l[kLogRows][2];
};
#define SP_LOG_TABLE \
    {0x1.5472400000000p+0, -0x1.23ebfe11e8000p-2, 0x1.c7df3de8a7086p-44}, \
    {0x1.52b0000000000p+0, -0x1.1e9e367889000p-2, -0x1.f45475b87c132p-46}, \
    {0x1.50f2400000000p+0, -0x1.19570a39bb000p-2, 0x1.0e881177921f3p-44}, \
    {0x1.4f39000000000p+0, -0x1.14169cf367000p-2, -0x1.ec080eeda7de4p-48}, \
    {0x1.4d84400000000p+0, -0x1.0edd128b78000p-2, 0x1.6f64a811a7574p-47}, \
    {0x1.4bd4000000000p+0, -0x1.09aa8f2e6b000p-2, 0x1.abd6a2f88de5cp-46}, \
    {0x1.4a28000000000p+0, -0x1.047e70cde8000p-2, -0x1.b7be26fc852cep-46}, \
    {0x1.4880400000000p+0, -0x1.feb1b23e9e000p-3, 0x1.427f73c62b26fp-44}, \
    {0x1.46dd000000000p+0, -0x1.f4756534d8000p-3, 0x1.8ce3b1d0075a6p-44}, \
    {0x1.453d800000000p+0, -0x1.ea438bf042000p-3, 0x1.07bec3832dcaap-46}, \
    {0x1.43a2800000000p+0, -0x1.e0211e6234000p-3, -0x1.c50220342ba25p-49}, \
    {0x1.420b400000000p+0, -0x1.d609a2f900000p-3, 0x1.91c904f373cc5p-49}, \
    {0x1.4078400000000p+0, -0x1.cc00859db0000p-3, -0x1.90ab9a8182e44p-46}, \
    {0x1.3ee9000000000p+0, -0x1.c202d6b17e000p-3, -0x1.923e6ac71954ep-46}, \
    {0x1.3d5d800000000p+0, -0x1.b810d10b7c000p-3, 0x1.58fc30415b970p-46}, \
    {0x1.3bd6000000000p+0, -0x1.ae2c4ef670000p-3, -0x1.b28d3f2aa3c59p-44}, \
    {0x1.3a52400000000p+0, -0x1.a453f12e6a000p-3, -0x1.1e877c0339c0ap-44}, \
    {0x1.38d2400000000p+0, -0x1.9a87f3deb6000p-3, -0x1.e3efefa7f0cfep-44}, \
    {0x1.3755c00000000p+0, -0x1.90c6ee9fcc000p-3, 0x1.23efab29e16a0p-45}, \
    {0x1.35dd000000000p+0, -0x1.8712bf7508000p-3, 0x1.3f707cc3c768bp-44}, \
    {0x1.3467800000000p+0, -0x1.7d6851caee000p-3, 0x1.e843e3991aedep-48}, \
    {0x1.32f5c00000000p+0, -0x1.73cb2d74fa000p-3, -0x1.607547b4b6373p-44}, \
    {0x1.3187800000000p+0, -0x1.6a39e3abbc000p-3, -0x1.7d97f1c91e95bp-49}, \
    {0x1.301c800000000p+0, -0x1.60b2fe0b0a000p-3, 0x1.99c56cd54f81ap-44}, \
    {0x1.2eb5000000000p+0, -0x1.5738609014000p-3, 0x1.165501abd3fc3p-44}, \
    {0x1.2d50c00000000p+0, -0x1.4dc89197b0000p-3, -0x1.3ad50bde659e3p-44}, \
    {0x1.2bef800000000p+0, -0x1.44620fdc94000p-3, -0x1.7be6b6970cca0p-46}, \
    {0x1.2a91c00000000p+0, -0x1.3b0877757e000p-3, -0x1.94059aa896d0fp-46}, \
    {0x1.2937400000000p+0, -0x1.31ba49d39c000p-3, -0x1.f179df82632d7p-44}, \
    {0x1.27dfc00000000p+0, -0x1.287600c112000p-3, 0x1.7e89e58f98edcp-44}, \
    {0x1.268b400000000p+0, -0x1.1f3bcb5f26000p-3, 0x1.edfd32e309011p-44}, \
    {0x1.2539c00000000p+0, -0x1.160bd924ac000p-3, 0x1.5014507687f4fp-45}, \
    {0x1.23eb800000000p+0, -0x1.0ce81adccc000p-3, 0x1.6dd68ab4302aap-45}, \
    {0x1.22a0000000000p+0, -0x1.03cd40a51a000p-3, -0x1.81a979c146707p-44}, \
    {0x1.2157800000000p+0, -0x1.f57a73d8f4000p-4, 0x1.bed7156e7f063p-44}, \
    {0x1.2012000000000p+0, -0x1.e3706ee304000p-4, -0x1.fed09cb978024p-46}, \
    {0x1.1ecf400000000p+0, -0x1.d179428218000p-4, -0x1.b6467523e7d9ap-45}, \
    {0x1.1d8f400000000p+0, -0x1.bf954569f0000p-4, 0x1.c51158e95114fp-50}, \
    {0x1.1c52400000000p+0, -0x1.adc868e5a8000p-4, 0x1.96b7dc2f16c6cp-50}, \
    {0x1.1b17c00000000p+0, -0x1.9c0bd4d4d0000p-4, -0x1.4063f1de4a319p-44}, \
    {0x1.19e0000000000p+0, -0x1.8a6377a914000p-4, -0x1.c28bb5a46418ap-44}, \
    {0x1.18ab000000000p+0, -0x1.78cfaa63d8000p-4, 0x1.94c959a092f20p-44}, \
    {0x1.1778c00000000p+0, -0x1.6750c6934c000p-4, -0x1.5f7b580601012p-44}, \
    {0x1.1648c00000000p+0, -0x1.55dfca50d4000p-4, -0x1.f4694249067ccp-46}, \
    {0x1.151b800000000p+0, -0x1.44845c3dac000p-4, 0x1.96b2ea2c0f153p-46}, \
    {0x1.13f1000000000p+0, -0x1.333ed78174000p-4, -0x1.82b773b88fdbep-44}, \
    {0x1.12c8c00000000p+0, -0x1.220823c784000p-4, 0x1.82394bcf07e29p-47}, \
    {0x1.11a3000000000p+0, -0x1.10e4433cb0000p-4, 0x1.8ef69296a3466p-44}, \
    {0x1.107fc00000000p+0, -0x1.ffa70d1ab8000p-5, -0x1.fe465f8137b9fp-48}, \
    {0x1.0f5ec00000000p+0, -0x1.dda4f1c648000p-5, 0x1.c6be3a99f455cp-46}, \
    {0x1.0e40800000000p+0, -0x1.bbd1e7c668000p-5, 0x1.2df32b39d0555p-46}, \
    {0x1.0d24400000000p+0, -0x1.9a17d75740000p-5, 0x1.de42e7ba3af0fp-44}, \
    {0x1.0c0a800000000p+0, -0x1.78867da358000p-5, 0x1.e6ac2c308269bp-44}, \
    {0x1.0af3000000000p+0, -0x1.5716d4c038000p-5, -0x1.abb976786d0a2p-47}, \
    {0x1.09ddc00000000p+0, -0x1.35c96baa10000p-5, -0x1.386fb257a2a1fp-45}, \
    {0x1.08cac00000000p+0, -0x1.149ed24008000p-5, 0x1.d6b8a79473ec5p-44}, \
    {0x1.07ba000000000p+0, -0x1.e72f328120000p-6, -0x1.f145a379992cep-44}, \
    {0x1.06ab400000000p+0, -0x1.a5590c8c10000p-6, 0x1.52499ece30e1ap-45}, \
    {0x1.059f000000000p+0, -0x1.63db778650000p-6, -0x1.bd58b61f506a8p-44}, \
    {0x1.0494800000000p+0, -0x1.2288a1fe40000p-6, 0x1.bf15e37a27d2ep-47}, \
    {0x1.038c800000000p+0, -0x1.c321584c00000p-7, -0x1.ed8d6d2fba1cdp-44}, \
    {0x1.0286400000000p+0, -0x1.418acf9640000p-7, -0x1.897d9bbc5ea9fp-45}, \
    {0x1.0182400000000p+0, -0x1.811dc14580000p-8, -0x1.0340d3d54fa95p-48}, \
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0}, \
    {0x1.fe02000000000p-1, 0x1.fefeaa2b00000p-9, 0x1.1bc049fdc0ac0p-45}, \
    {0x1.fa12000000000p-1, 0x1.7db6f5f8c0000p-7, 0x1.b9d840748ca0ep-45}, \
    {0x1.f631000000000p-1, 0x1.3ceba43470000p-6, -0x1.e0b0fed853743p-46}, \
    {0x1.f25f800000000p-1, 0x1.b9f8727b10000p-6, 0x1.3dbf6611b2c35p-45}, \
    {0x1.ee9c800000000p-1, 0x1.1b0d909240000p-5, -0x1.3381e9ae9df10p-44}, \
    {0x1.eae8000000000p-1, 0x1.58a63afc90000p-5, -0x1.656e6d58c041cp-46}, \
    {0x1.e741800000000p-1, 0x1.95caf8ecb0000p-5, -0x1.68232f42b6559p-44}, \
    {0x1.e3a9000000000p-1, 0x1.d27848adb8000p-5, 0x1.3c90b7ced5baep-44}, \
    {0x1.e01e000000000p-1, 0x1.0759935990000p-4, -0x1.b0ecfe4604432p-44}, \
    {0x1.dca0000000000p-1, 0x1.254062f0a8000p-4, 0x1.416fe50bf3c56p-44}, \
    {0x1.d92f000000000p-1, 0x1.42eef3ea70000p-4, -0x1.bdf780dab787dp-45}, \
    {0x1.d5cb000000000p-1, 0x1.6063a29394000p-4, -0x1.e1c73129d989ep-44}, \
    {0x1.d273000000000p-1, 0x1.7da58ed7cc000p-4, 0x1.7b18b5c395b6dp-46}, \
    {0x1.cf27000000000p-1, 0x1.9ab33c6208000p-4, 0x1.cccd7f48e9da5p-44}, \
    {0x1.cbe7000000000p-1, 0x1.b78b2abb1c000p-4, 0x1.4c0fb52fc9e19p-44}, \
    {0x1.c8b2800000000p-1, 0x1.d4305166d4000p-4, -0x1.fdaa5ea3827fbp-44}, \
    {0x1.c589800000000p-1, 0x1.f0a1400130000p-4, -0x1.1bd746d48b542p-52}, \
    {0x1.c26b800000000p-1, 0x1.0670872cb0000p-3, -0x1.cb781892645a7p-45}, \
    {0x1.bf58000000000p-1, 0x1.1479784688000p-3, 0x1.ab21c0820b429p-45}, \
    {0x1.bc50000000000p-1, 0x1.22663190ae000p-3, 0x1.596e8a3e0d005p-44}, \
    {0x1.b952000000000p-1, 0x1.303ce98e4c000p-3, 0x1.025f6c31cabb9p-44}, \
    {0x1.b65e000000000p-1, 0x1.3dfd030ed8000p-3, -0x1.cb144b686618fp-46}, \
    {0x1.b374800000000p-1, 0x1.4ba38539a6000p-3, -0x1.06d4bad036f2cp-44}, \
    {0x1.b094800000000p-1, 0x1.59347f9990000p-3, 0x1.527952cb3b9c2p-45}, \
    {0x1.adbe800000000p-1, 0x1.66acfa272c000p-3, -0x1.a16421c7fe2a6p-44}, \
    {0x1.aaf2000000000p-1, 0x1.740eb7540e000p-3, 0x1.bc979c6007c5bp-44}, \
    {0x1.a82e800000000p-1, 0x1.815b88143a000p-3, -0x1.844b11eed06f5p-45}, \
    {0x1.a574000000000p-1, 0x1.8e92dde888000p-3, 0x1.902abfd25a3dcp-45}, \
    {0x1.a2c2800000000p-1, 0x1.9bb428e7ea000p-3, -0x1.6b1409341998ep-44}, \
    {0x1.a01a000000000p-1, 0x1.a8bed7c882000p-3, 0x1.eb185cf770f25p-44}, \
    {0x1.9d7a000000000p-1, 0x1.b5b4d1e8fc000p-3, 0x1.3c8dc20fee737p-44}, \
    {0x1.9ae2800000000p-1, 0x1.c2958f58d0000p-3, 0x1.49240691b4804p-45}, \
    {0x1.9853000000000p-1, 0x1.cf6308e09e000p-3, -0x1.c9dbd431ae023p-46}, \
    {0x1.95cb800000000p-1, 0x1.dc1cc00ace000p-3, -0x1.c7a30fb9f9430p-45}, \
    {0x1.934c800000000p-1, 0x1.e8bfab2aaa000p-3, -0x1.6f8325ea59404p-44}, \
    {0x1.90d5000000000p-1, 0x1.f5505964ba000p-3, -0x1.c71f2ee13a436p-44}, \
    {0x1.8e65000000000p-1, 0x1.00e72a5ada000p-2, 0x1.64cbf31b474cap-46}, \
    {0x1.8bfd000000000p-1, 0x1.071b47fcd7000p-2, 0x1.c546f82d573a3p-44}, \
    {0x1.899c000000000p-1, 0x1.0d46dd79ac000p-2, 0x1.e5906872c81ffp-45}, \
    {0x1.8742800000000p-1, 0x1.136865293b000p-2, -0x1.97684a0c51bbfp-44}, \
    {0x1.84f0000000000p-1, 0x1.1980f2dd43000p-2, -0x1.24262183a4308p-44}, \
    {0x1.82a4800000000p-1, 0x1.1f904ee48e000p-2, -0x1.26dbd7f67844ep-44}, \
    {0x1.8060000000000p-1, 0x1.2596410df9000p-2, 0x1.8e7c177a43938p-44}, \
    {0x1.7e22800000000p-1, 0x1.2b9290ab90000p-2, 0x1.1da57a3696d89p-44}, \
    {0x1.7beb000000000p-1, 0x1.3187b69550000p-2, -0x1.4cbcacc8e9521p-44}, \
    {0x1.79ba800000000p-1, 0x1.3772cf2c03000p-2, -0x1.8307c7c1781d4p-46}, \
    {0x1.7790800000000p-1, 0x1.3d54fd5c1f000p-2, 0x1.c861cd9c795e3p-44}, \
    {0x1.756c800000000p-1, 0x1.432f6ba056000p-2, -0x1.6290588328ea0p-44}, \
    {0x1.734f000000000p-1, 0x1.49008a0401000p-2, 0x1.6c6619d3695c5p-45}, \
    {0x1.7137800000000p-1, 0x1.4ec9862600000p-2, 0x1.4eebd7b3bbe57p-44}, \
    {0x1.6f26000000000p-1, 0x1.548a303add000p-2, 0x1.4167e63b2c7a2p-45}, \
    {0x1.6d1a800000000p-1, 0x1.5a42580f50000p-2, 0x1.6ce65a13a2b76p-44}, \
    {0x1.6b14800000000p-1, 0x1.5ff3360a7a000p-2, 0x1.45723ec46e565p-44}, \
    {0x1.6914800000000p-1, 0x1.659b34303f000p-2, -0x1.1edf97322c132p-44}, \
    {0x1.671a000000000p-1, 0x1.6b3b8e235a000p-2, -0x1.a276de1b31cc1p-46}, \
    {0x1.6525000000000p-1, 0x1.70d4182789000p-2, 0x1.7f756624a1cd3p-44}, \
    {0x1.6335800000000p-1, 0x1.7664a6239f000p-2, 0x1.c030067665be0p-44}, \
    {0x1.614b000000000p-1, 0x1.7bee7ea387000p-2, 0x1.63d917710b7fap-45}, \
    {0x1.5f66800000000p-1, 0x1.816e90da1d000p-2, -0x1.aa199f5276493p-44}, \
    {0x1.5d86800000000p-1, 0x1.86e90ea331000p-2, -0x1.b6fb02717958bp-45}, \
    {0x1.5bac000000000p-1, 0x1.8c5ae48597000p-2, -0x1.bd6281df29608p-44}, \
    {0x1.59d6000000000p-1, 0x1.91c6dab45f000p-2, -0x1.689d109026758p-44}, \
    {0x1.5805800000000p-1, 0x1.9729d51139000p-2, 0x1.f69944f1fb0c2p-44}, \
    {0x1.5639800000000p-1, 0x1.9c86a32dc1000p-2, -0x1.92d918a5cbf17p-44}

// ln((a + 1/2) 2^-32) < 0, laid out as ARM's log() is (see above)
SP_HD double log_unit(uint32_t a, const LogTab& tab) {
    // (2^52 + a) 2^-32 - 2^20 + 2^-33, exact
    const double u = fma(fp64_make(0x43300000, static_cast<int>(a)), 0x1p-32, -0x1p20 + 0x1p-33);
    const int hi = fp64_hi(u), off = hi - 0x3fe80000;
    const int i = (off >> 13) & (kLogRows - 1);
    const double kd = fp64_make(0x43300000, (off >> 20) + 1024) - (0x1p52 + 1024.0);
    const double m = fp64_make(hi - (off & static_cast<int>(0xfff00000u)), fp64_lo(u));  // u = 2^k m
    const double r = fma(m, tab.c[i], -1.0);  // exact: 33 bits times 19
    const double w = fma(kd, 0x1.62e42fefa3800p-1, tab.l[i][0]);  // exact: multiples of 2^-42
    const double low = fma(kd, 0x1.ef35793c76730p-45, tab.l[i][1]);
    // ln(1 + r), |r| <= 2^-8, by its series
    const double z = r * r;
    double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    p = fma(r, p, 0.2);
    p = fma(r, p, -0.25);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -0.5);
    return w + (r + fma(z, p, low));
}

// sqrt(x) of a normal x > 0
SP_HD double sqrt_normal(double x) {
    const double y = fp64_rsqrt_seed(x);
    double g = x * y;
    const double h = 0.5 * y;
    g = fma(g, fma(-g, h, 0.5), g);
    return fma(fma(-g, g, x), h, g);
}

// 1/x of an x in [2^-1022, 2^1022]: two steps of Newton's iteration y <- y + y (1 - x y).  A step
// squares the relative error: below 2^-19 in the first approximation (the hardware's: 9.8e-7),
// 2^-38 after one step (with its rounding), 2^-76 after two, so the result is the exact
// reciprocal rounded once, 2^-23 ulp apart at most (in place of a division, which cannot be
// interleaved with its neighbours: it branches on its operands).
SP_HD double rcp_normal(double x) {
    double y = fp64_rcp_seed(x);
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

// a / b from b's reciprocal: quotient and residual correction (P. Markstein, IBM J. Res. Dev.
// 34, 1990).  The correctly rounded quotient where nothing over- or underflows.
SP_HD double quotient(double a, double b, double reciprocal) {
    const double q = fp64_mul(a, reciprocal);
    return fma(fma(-b, q, a), reciprocal, q);
}

// 1/x of the sine of an angle, 0 for x = 0 (and for a subnormal x, whose reciprocal only
// overflows what it multiplies)
SP_HD double rcp_or_zero(double x) {
    const double y = rcp_normal(x);
    return (fp64_hi(x) & 0x7ff00000) == 0 ? 0.0 : y;
}

// one Box-Muller pair on the words (a, b): u = (w + 1/2) 2^-32, r = sqrt(scale ln u_a) with
// scale < 0, (r sin 2 pi u_b, r cos 2 pi u_b)
SP_HD SinCosD box_muller_pair(uint32_t a, uint32_t b, double scale, const LogTab& tab) {
    const double r = sqrt_normal(scale * log_unit(a, tab));
    const SinCosD t = sincos_turn(b);
    return SinCosD{fp64_mul(r, t.s), fp64_mul(r, t.c)};
}

}  // namespace sp
