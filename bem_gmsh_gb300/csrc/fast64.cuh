// FP64 log, quotient and square root with few FP64 instructions.
//
// GB300 runs a warp's FP64 instruction in 64 cycles of its scheduler (2
// lanes per clock and SM, measured with one to sixteen warps), an FP32 or
// integer one in one or two: an FP64 kernel's time is its count of FP64
// instructions, and everything else is nearly free.  Measured in FP64
// multiply-adds (512 threads, independent chains): the compiler's quotient
// 5.5, its square root 9, its logarithm about 20.  Here a quotient is 5, a
// square root 7 and a logarithm 10, with these errors:
//   quotient     the rounded value of a result within 2^-75 of the quotient
//   square root  within 0.51 ulp
//   log          within 0.51 ulp of the result, or 2^-61 where that is larger
//                than half an ulp (|log x| < 2^-8: within 2 ulp, 1.33
//                measured; the argument's own rounding, in a squared distance
//                near 1, is 2^8 times that)
// Methods: quotient and square root from the hardware's approximation by
// Newton and a remainder correction (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990); the logarithm
// by Tang's table reduction ("Table-driven implementation of the logarithm
// function in IEEE floating-point arithmetic", 1990): x = 2^E m,
// m rc = 1 + r with rc = 1/c to 16 bits (c the nearest of 1 + i/128, so
// |r| < 2^-7.9), log x = E log 2 - log rc + log1p(r).  The terms of log1p from
// r^5 on need 24 bits only and take FP32; conversions go through the integer
// pipes.  Arguments that are not positive, normal and finite take the
// platform's functions.
//
// On the host (tests) the approximations are replaced by 1/x and 1/sqrt(x)
// without their low 32 bits, which the hardware's do not have either.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef BEM_HD
#ifdef __CUDACC__
#define BEM_HD __host__ __device__ __forceinline__
#else
#define BEM_HD inline
#endif
#endif

namespace bem {
namespace f64 {

// {rc, high part of -log rc (a multiple of 2^-42), low part}, centre 1 + i/128
#ifdef __CUDA_ARCH__
static __device__ const
#else
static const
#endif
double kLogTab[129][3] = {
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0},
    {0x1.fc08000000000p-1, 0x1.fdfaa6b100000p-8, 0x1.33c478c65f4c7p-43},
    {0x1.f820000000000p-1, 0x1.fbea8b13c0000p-7, 0x1.ec927b17e4e13p-50},
    {0x1.f446000000000p-1, 0x1.7b9d307e60000p-6, 0x1.c8e520ec779f0p-45},
    {0x1.f07c000000000p-1, 0x1.f82db0e7a0000p-6, 0x1.980312729348fp-45},
    {0x1.ecc0000000000p-1, 0x1.39f07ba0e8000p-5, 0x1.eb129d642e577p-44},
    {0x1.e914000000000p-1, 0x1.77368f66b0000p-5, 0x1.ceab23b20a79dp-45},
    {0x1.e574000000000p-1, 0x1.b428571210000p-5, 0x1.bde4b7dc0b00bp-49},
    {0x1.e1e2000000000p-1, 0x1.f0a10c0120000p-5, 0x1.8a995b487d1b1p-43},
    {0x1.de5e000000000p-1, 0x1.164e8eeaf4000p-4, 0x1.cde7e7ae94a9fp-44},
    {0x1.dae6000000000p-1, 0x1.341db961bc000p-4, 0x1.9d092aed8cba6p-44},
    {0x1.d77c000000000p-1, 0x1.51ab33f13c000p-4, 0x1.01e32b4262a3cp-43},
    {0x1.d41e000000000p-1, 0x1.6f06a8afa8000p-4, 0x1.68bc6775aa563p-45},
    {0x1.d0cc000000000p-1, 0x1.8c2e9d6420000p-4, 0x1.18e7fe18d63d6p-43},
    {0x1.cd86000000000p-1, 0x1.a92193a588000p-4, 0x1.d60614c9016aap-44},
    {0x1.ca4c000000000p-1, 0x1.c5de08f760000p-4, 0x1.e764adc3ff039p-45},
    {0x1.c71c000000000p-1, 0x1.e27476e32c000p-4, 0x1.9739fa00eaaa2p-43},
    {0x1.c3f8000000000p-1, 0x1.fed1932000000p-4, 0x1.58eeb117feaf2p-45},
    {0x1.c0e0000000000p-1, 0x1.0d79e7cd48000p-3, 0x1.cb422847849e4p-44},
    {0x1.bdd2000000000p-1, 0x1.1b75fd53a6000p-3, 0x1.4660db3fc0841p-48},
    {0x1.bad0000000000p-1, 0x1.29532f823e000p-3, 0x1.522a15b51c651p-43},
    {0x1.b7d6000000000p-1, 0x1.37235202b4000p-3, 0x1.e0016b63aa4bdp-49},
    {0x1.b4e8000000000p-1, 0x1.44d336ccba000p-3, 0x1.d1e6a7e841ba3p-43},
    {0x1.b204000000000p-1, 0x1.526b7e3a9e000p-3, 0x1.835a7ef352587p-43},
    {0x1.af28000000000p-1, 0x1.5ff5070ab8000p-3, 0x1.3d4731eacb4b8p-43},
    {0x1.ac58000000000p-1, 0x1.6d5c3e7306000p-3, 0x1.09cf818d9389ep-46},
    {0x1.a98e000000000p-1, 0x1.7abd302262000p-3, 0x1.d115a71a8f7dcp-43},
    {0x1.a6d0000000000p-1, 0x1.87fa865210000p-3, 0x1.2212595679851p-44},
    {0x1.a41a000000000p-1, 0x1.9526e9cf5e000p-3, 0x1.ad27faf800790p-45},
    {0x1.a16e000000000p-1, 0x1.a23811ff04000p-3, 0x1.cbdd713b1a053p-44},
    {0x1.9ec8000000000p-1, 0x1.af4114e94e000p-3, 0x1.ffa70d1943aa9p-43},
    {0x1.9c2e000000000p-1, 0x1.bc23d74424000p-3, 0x1.dce3fdbdbd76fp-43},
    {0x1.999a000000000p-1, 0x1.c8fd7c79e8000p-3, 0x1.a21017b4d7442p-43},
    {0x1.970e000000000p-1, 0x1.d5c3a6b522000p-3, 0x1.92359e4dd4e25p-44},
    {0x1.948c000000000p-1, 0x1.e26bb6e418000p-3, 0x1.6e7dcc9665548p-46},
    {0x1.9210000000000p-1, 0x1.ef095cbde8000p-3, 0x1.9360a18e87436p-43},
    {0x1.8f9c000000000p-1, 0x1.fb9206d5e6000p-3, 0x1.e2a8ffff136e2p-43},
    {0x1.8d30000000000p-1, 0x1.0402994b4f000p-2, 0x1.0370df44d82d4p-48},
    {0x1.8acc000000000p-1, 0x1.0a312e2761000p-2, 0x1.1c5cbe8228225p-43},
    {0x1.886e000000000p-1, 0x1.1059b79b02000p-2, 0x1.6aacc68b2daf6p-43},
    {0x1.8618000000000p-1, 0x1.1676cabada000p-2, 0x1.83963c8b4ab26p-44},
    {0x1.83ca000000000p-1, 0x1.1c882416d8000p-2, 0x1.cf41cf19a0e7fp-43},
    {0x1.8182000000000p-1, 0x1.2292cfbd2e000p-2, 0x1.6c9c2a5697156p-43},
    {0x1.7f40000000000p-1, 0x1.2896a13e08000p-2, 0x1.a8ed027e16952p-44},
    {0x1.7d06000000000p-1, 0x1.2e8e0bae12000p-2, 0x1.4c2700879c369p-44},
    {0x1.7ad2000000000p-1, 0x1.347e31a98b000p-2, 0x1.3a9b37979bce8p-43},
    {0x1.78a4000000000p-1, 0x1.3a66e55724000p-2, 0x1.bd9f40ba2c8a8p-43},
    {0x1.767e000000000p-1, 0x1.4042806873000p-2, 0x1.0c760817cddc1p-43},
    {0x1.745e000000000p-1, 0x1.46163c228d000p-2, 0x1.d7a8f712dc24bp-43},
    {0x1.7242000000000p-1, 0x1.4be77157bc000p-2, 0x1.243d358722946p-43},
    {0x1.702e000000000p-1, 0x1.51aae872df000p-2, 0x1.45a139d256c6ap-43},
    {0x1.6e20000000000p-1, 0x1.5765f1749d000p-2, 0x1.4d669360f93ebp-43},
    {0x1.6c16000000000p-1, 0x1.5d1dfbf611000p-2, 0x1.cd836429a6520p-46},
    {0x1.6a14000000000p-1, 0x1.62c79f2ba6000p-2, 0x1.32a407ec1796cp-43},
    {0x1.6816000000000p-1, 0x1.686df1e9f3000p-2, 0x1.abf06f6b4338dp-44},
    {0x1.661e000000000p-1, 0x1.6e0b22a357000p-2, 0x1.4ce6048d85e73p-43},
    {0x1.642c000000000p-1, 0x1.739eff6c05000p-2, 0x1.ef38a75504c83p-52},
    {0x1.6240000000000p-1, 0x1.792955fdf4000p-2, 0x1.e889b0253ca88p-44},
    {0x1.6058000000000p-1, 0x1.7eafc3b82c000p-2, 0x1.f86cc11f69a14p-43},
    {0x1.5e76000000000p-1, 0x1.842c55a1fc000p-2, 0x1.cb904537d88b4p-45},
    {0x1.5c98000000000p-1, 0x1.89a4b86c5c000p-2, 0x1.2dead3b4c0944p-45},
    {0x1.5ac0000000000p-1, 0x1.8f12e87386000p-2, 0x1.63e9b66795610p-45},
    {0x1.58ee000000000p-1, 0x1.9476b1c2e3000p-2, 0x1.1ea3ce9c89502p-43},
    {0x1.571e000000000p-1, 0x1.99dbd01241000p-2, 0x1.0fcfa02becd8ap-46},
    {0x1.5556000000000p-1, 0x1.9f303ecc79000p-2, 0x1.0929019c596bcp-43},
    {0x1.5390000000000p-1, 0x1.a485c90ebd000p-2, 0x1.617eaa5243931p-43},
    {0x1.51d0000000000p-1, 0x1.a9d049a9e8000p-2, 0x1.0955a9141ea8fp-43},
    {0x1.5016000000000p-1, 0x1.af0f8b259d000p-2, 0x1.1c390f040eb72p-43},
    {0x1.4e5e000000000p-1, 0x1.b44f97bcc9000p-2, 0x1.d8a33a6615a51p-44},
    {0x1.4cac000000000p-1, 0x1.b984196973000p-2, 0x1.7d2e0aa57b6d5p-45},
    {0x1.4afe000000000p-1, 0x1.beb309dada000p-2, 0x1.af3f6d83e73a5p-43},
    {0x1.4954000000000p-1, 0x1.c3dc4a7d07000p-2, 0x1.e99c99d178e5bp-43},
    {0x1.47ae000000000p-1, 0x1.c8ffbc79ab000p-2, 0x1.4435af65b0891p-43},
    {0x1.460c000000000p-1, 0x1.ce1d40b90a000p-2, 0x1.7be6b112abf98p-44},
    {0x1.4470000000000p-1, 0x1.d32e67e056000p-2, 0x1.7a883be3397a7p-43},
    {0x1.42d6000000000p-1, 0x1.d83faa58d2000p-2, 0x1.efbab2dfbbf59p-44},
    {0x1.4142000000000p-1, 0x1.dd44404cd0000p-2, 0x1.9388f7af21401p-43},
    {0x1.3fb0000000000p-1, 0x1.e248c1a7c8000p-2, 0x1.84c3c25c955d5p-43},
    {0x1.3e22000000000p-1, 0x1.e746b61e3a000p-2, 0x1.31afeb5fffab2p-43},
    {0x1.3c9a000000000p-1, 0x1.ec378524f5000p-2, 0x1.3d0821772418ep-46},
    {0x1.3b14000000000p-1, 0x1.f127f5fb10000p-2, 0x1.bb1781cf96eeap-44},
    {0x1.3992000000000p-1, 0x1.f61177a716000p-2, 0x1.2c3894c787ec3p-46},
    {0x1.3814000000000p-1, 0x1.faf3e8f7e3000p-2, 0x1.63ad70af19637p-43},
    {0x1.3698000000000p-1, 0x1.ffd5c08687000p-2, 0x1.94082e2d55e2dp-43},
    {0x1.3522000000000p-1, 0x1.0254da5a63000p-1, 0x1.3faf0c6ffad50p-43},
    {0x1.33ae000000000p-1, 0x1.04be6dda9f800p-1, 0x1.1285be71109f5p-45},
    {0x1.323e000000000p-1, 0x1.07243dc1d5800p-1, 0x1.0170d3b55dbabp-47},
    {0x1.30d2000000000p-1, 0x1.098638f595800p-1, 0x1.580c7c15493a9p-43},
    {0x1.2f68000000000p-1, 0x1.0be7ae4262800p-1, 0x1.4170a1a532f01p-44},
    {0x1.2e02000000000p-1, 0x1.0e45345d34800p-1, 0x1.98884fef0a16cp-46},
    {0x1.2ca0000000000p-1, 0x1.109eb9e2e4800p-1, 0x1.25b4ce527c17dp-43},
    {0x1.2b40000000000p-1, 0x1.12f799594e800p-1, 0x1.ef1f6af5711d0p-43},
    {0x1.29e4000000000p-1, 0x1.154c5d2f4e000p-1, 0x1.7a6a8e7795904p-43},
    {0x1.288c000000000p-1, 0x1.179cf3be46800p-1, 0x1.4cfd5be0637efp-44},
    {0x1.2736000000000p-1, 0x1.19ecc3472c000p-1, 0x1.345ec995d8965p-44},
    {0x1.25e2000000000p-1, 0x1.1c3bc5f718000p-1, 0x1.1930bea90eaacp-43},
    {0x1.2492000000000p-1, 0x1.1e8675e714000p-1, 0x1.a0d12e18a1405p-46},
    {0x1.2346000000000p-1, 0x1.20ccc11970800p-1, 0x1.6b02eca05de22p-43},
    {0x1.21fc000000000p-1, 0x1.23121d7c24000p-1, 0x1.a0b4cf4cb3beep-44},
    {0x1.20b4000000000p-1, 0x1.255684e9b6800p-1, 0x1.97bd8e2a69253p-46},
    {0x1.1f70000000000p-1, 0x1.27966128ab000p-1, 0x1.1b1622f1e865bp-45},
    {0x1.1e2e000000000p-1, 0x1.29d533ece4800p-1, 0x1.68af4eb08bb0bp-44},
    {0x1.1cf0000000000p-1, 0x1.2c0f5ed46c800p-1, 0x1.a3125eb12c719p-43},
    {0x1.1bb4000000000p-1, 0x1.2e486b6e95800p-1, 0x1.b527fbd87c975p-44},
    {0x1.1a7c000000000p-1, 0x1.307cb33515000p-1, 0x1.7b1f6b7243d28p-46},
    {0x1.1946000000000p-1, 0x1.32afc791a3000p-1, 0x1.d6ae688647ba6p-44},
    {0x1.1812000000000p-1, 0x1.34e1a1da02800p-1, 0x1.690c6f49eccc9p-44},
    {0x1.16e0000000000p-1, 0x1.37123b5498000p-1, 0x1.ed95774ab2144p-43},
    {0x1.15b2000000000p-1, 0x1.393ddd3564800p-1, 0x1.8669e110a22dbp-43},
    {0x1.1486000000000p-1, 0x1.3b6828a000800p-1, 0x1.8abc7225c382fp-47},
    {0x1.135c000000000p-1, 0x1.3d9116a74d800p-1, 0x1.7ddea2448ed7fp-44},
    {0x1.1236000000000p-1, 0x1.3fb4e44d42800p-1, 0x1.60665d4bb62dap-43},
    {0x1.1112000000000p-1, 0x1.41d73e852b000p-1, 0x1.539f8a0bf52b6p-44},
    {0x1.0ff0000000000p-1, 0x1.43f81e307d800p-1, 0x1.97ac1e2a67afap-43},
    {0x1.0ed0000000000p-1, 0x1.46177c2229800p-1, 0x1.aff89882431b1p-43},
    {0x1.0db2000000000p-1, 0x1.4835511ea8800p-1, 0x1.c7dcffe4d9c4dp-43},
    {0x1.0c98000000000p-1, 0x1.4a4dc5dbc7800p-1, 0x1.acf735c69bc25p-43},
    {0x1.0b7e000000000p-1, 0x1.4c686efcfa800p-1, 0x1.1e9cd0b4eec23p-43},
    {0x1.0a68000000000p-1, 0x1.4e7da11b76800p-1, 0x1.d84eada184782p-44},
    {0x1.0954000000000p-1, 0x1.509124c017000p-1, 0x1.6b4b833a5d935p-45},
    {0x1.0842000000000p-1, 0x1.52a2f265bd000p-1, 0x1.6abbc89cd8701p-43},
    {0x1.0732000000000p-1, 0x1.54b30279bb800p-1, 0x1.360c11449c268p-43},
    {0x1.0624000000000p-1, 0x1.56c14d5bf5000p-1, 0x1.e7ea581c049ccp-43},
    {0x1.051a000000000p-1, 0x1.58c9df5d15800p-1, 0x1.c7eafe6a8ce43p-45},
    {0x1.0410000000000p-1, 0x1.5ad484c369800p-1, 0x1.cb49751754272p-43},
    {0x1.030a000000000p-1, 0x1.5cd959c788800p-1, 0x1.e74d8d8542e79p-43},
    {0x1.0204000000000p-1, 0x1.5ee03a9241800p-1, 0x1.3ab875af5ad3dp-44},
    {0x1.0102000000000p-1, 0x1.60e1334574800p-1, 0x1.0e5f59f4bd8f2p-45},
    {0x1.0000000000000p-1, 0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45},
};
#define BEM_LN2_HI 0x1.62e42fefa3800p-1
#define BEM_LN2_LO 0x1.ef35793c76730p-45

BEM_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
BEM_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
BEM_HD float from_bits32(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}
BEM_HD uint32_t bits32(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return u;
#endif
}
BEM_HD uint32_t hi32(double x) { return (uint32_t)(bits(x) >> 32); }

// 2^-499 <= |x| < 2^500: quotients, squares and their corrections stay normal
BEM_HD bool plain(double x) { return (((hi32(x) & 0x7fffffffu) - 0x20c00000u) < 0x3e700000u); }

BEM_HD double rcp_approx(double x) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
#else
  return from_bits(bits(1.0 / x) & ~0xffffffffull);
#endif
}
BEM_HD double rsqrt_approx(double x) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
#else
  return from_bits(bits(1.0 / std::sqrt(x)) & ~0xffffffffull);
#endif
}

// about 2^-40 of 1/d (plain d)
BEM_HD double rcp40(double d) {
  const double y = rcp_approx(d);
  return fma(fma(-d, y, 1.0), y, y);
}

BEM_HD double div(double n, double d) {
  if (!plain(d) || !(plain(n) || (bits(n) << 1) == 0)) return n / d;
  const double y = rcp40(d);
  const double q = n * y;
  return fma(fma(-q, d, n), y, q);
}

// 1/d to half an ulp and a little
BEM_HD double rcp(double d) {
  if (!plain(d)) return 1.0 / d;
  const double y = rcp40(d);
  return fma(fma(-d, y, 1.0), y, y);
}

BEM_HD double sqrt(double x) {
  if (!plain(x) || x < 0.0) return ::sqrt(x);
  const double y = rsqrt_approx(x);
  double s = x * y, h = 0.5 * y;
  const double r = fma(-s, h, 0.5);
  s = fma(s, r, s);
  h = fma(h, r, h);
  return fma(fma(-s, s, x), h, s);
}

// small integer (|i| < 2^21) and positive normal float to double
BEM_HD double small_int(int i) {
  const float f = from_bits32(0x4B400000u + (uint32_t)i) - 12582912.0f;
  const uint32_t b = bits32(f);
  const uint32_t h = (b & 0x7fffffffu) ? (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u) : 0u;
  return from_bits((uint64_t)h << 32);
}
BEM_HD double widen_positive(float f) {
  const uint32_t b = bits32(f);
  return from_bits(((uint64_t)((b >> 3) + 0x38000000u) << 32) | (uint64_t)(b << 29));
}

BEM_HD double log(double x) {
  const uint64_t u = bits(x);
  const uint32_t h = (uint32_t)(u >> 32);
  if (h - 0x00100000u >= 0x7fe00000u) return ::log(x);  // not positive, normal and finite
  const int E = (int)(h >> 20) - 1023;
  const int i = (int)(((h >> 12) & 0xffu) + 1u) >> 1;
  const double m = from_bits((u & 0xFFFFFFFFFFFFFull) | 0x3FF0000000000000ull);
  const double rc = kLogTab[i][0], lh = kLogTab[i][1], ll = kLogTab[i][2];
  const double r = fma(m, rc, -1.0);
  // r as FP32 (|r| < 2^-7: the low seven exponent bits)
  const uint64_t rb = bits(r);
  const uint32_t t = (uint32_t)(rb >> 29);
  const float rf = from_bits32((t & 0x3fffffffu) | ((uint32_t)(rb >> 32) & 0x80000000u));
  const float q5 = fmaf(rf, fmaf(rf, 0.142857142857142857f, -0.166666666666666667f), 0.2f);
  double q = fma(widen_positive(q5), r, -0.25);
  q = fma(q, r, 0.33333333333333333);
  q = fma(q, r, -0.5);
  const double l = fma(q, r * r, r);
  const double Ed = small_int(E);
  return fma(Ed, BEM_LN2_HI, lh) + (fma(Ed, BEM_LN2_LO, ll) + l);
}

}  // namespace f64
}  // namespace bem
