/*
 * sflow_pow.h -- x^y of the FP64 form, with the bits of sfm_pow
 * (sflow_math.h) and a fraction of its cost (device code).
 *
 * sfm_pow carries some 600 FP64 operations of double-double arithmetic; GB300
 * executes FP64 at 1/64 of the FP32 rate, and the settling closure calls it
 * once per fixed-point iteration, class and cell.  sfm_pow_int, the function
 * the kernels call, evaluates x^y in 64-bit fixed point on the integer
 * pipes; sfm_pow_quick in about 70 FP64 operations to a relative error below
 * 2^-68.  Each returns when its value is further than its error from every
 * rounding boundary of FP64: the rounding is then that of the exact x^y,
 * which is also what sfm_pow returns (relative error below 2^-70 before its
 * one rounding).  The first passes the rest, about one argument in two
 * hundred, to the second, and that about one in a thousand to sfm_pow (A. Ziv,
 * Fast evaluation of elementary mathematical functions with correctly rounded
 * last bit, ACM TOMS 17(3), 1991).  So all three give the same bits
 * (tests/test_pow.py, tests/test_gpu_math.py).
 * Measured: 8 steps of a 512^2 FP64 current with settling of 2 classes took
 * 54.4 ms with sfm_pow, 32.8 ms with sfm_pow_quick.
 *
 * Method of sfm_pow_quick:
 *  log x   x = 2^k m, m in [1, 2), c_i = 1/m rounded to 8 bits at the centre
 *          of the i-th of 128 intervals; r = m c - 1 is exact (|r| <= 2^-7,
 *          a multiple of 2^-60); log x = k ln 2 - log c + log1p(r).
 *          k ln 2 and -log c have high parts that are multiples of 2^-42, so
 *          their sum is exact; r and r^2/2 enter without error; the terms
 *          r^3/3 ... r^9/9 in double (next term below 2^-73).
 *  exp z   z = (128 k' + j) ln2/128 + r', |r'| <= 2^-8.5; 2^(j/128) from a
 *          table in double-double, exp(r') - 1 by its series to r'^6/720
 *          (next term below 2^-71), the product with r' without error.
 * The tables are the exact values split into a high double and the nearest
 * double of the remainder; tests/test_pow.py recomputes them.
 */
#ifndef SFLOW_POW_H
#define SFLOW_POW_H

#include "sflow_math.h"

#if defined(__CUDACC__)
#define SFM_TAB static __device__ const double
#define SFM_LD(p) __ldg(p)
#define SFM_COLD static __device__ __noinline__
#else
#define SFM_TAB static const double
#define SFM_LD(p) (*(p))
#define SFM_COLD static inline
#endif

/* per interval: c, -log c rounded to a multiple of 2^-42, the rest */
SFM_TAB sfm_pow_log_tab[128 * 3] = {
    0x1.fe00000000000p-1, 0x1.0080559580000p-8, 0x1.166afcb31c67bp-45,
    0x1.fa00000000000p-1, 0x1.82448a3880000p-7, 0x1.4554412c584e0p-44,
    0x1.f600000000000p-1, 0x1.432a925980000p-6, 0x1.98139928637fep-47,
    0x1.f200000000000p-1, 0x1.c63d2ec150000p-6, -0x1.5439ce030a687p-44,
    0x1.ee00000000000p-1, 0x1.252f32f8d0000p-5, 0x1.83e9ae021b67bp-45,
    0x1.ea00000000000p-1, 0x1.67c94f2d48000p-5, 0x1.dac20827cca0cp-44,
    0x1.e800000000000p-1, 0x1.894aa149f8000p-5, 0x1.9a19a8be97661p-44,
    0x1.e400000000000p-1, 0x1.ccb73cddd8000p-5, 0x1.965c36e09f5fep-44,
    0x1.e000000000000p-1, 0x1.08598b59e4000p-4, -0x1.7e5dd7009902cp-46,
    0x1.dc00000000000p-1, 0x1.2aa04a4470000p-4, 0x1.7a48ba8b1cb41p-44,
    0x1.da00000000000p-1, 0x1.3bdf5a7d20000p-4, -0x1.19bd0ad125895p-44,
    0x1.d600000000000p-1, 0x1.5e95a4d978000p-4, 0x1.1cb7ce1d17171p-44,
    0x1.d200000000000p-1, 0x1.8197e2f410000p-4, -0x1.c0fe460d20041p-44,
    0x1.d000000000000p-1, 0x1.9335e5d594000p-4, 0x1.3115c3abd47dap-45,
    0x1.cc00000000000p-1, 0x1.b6ac88dad4000p-4, 0x1.b1bdff50225c7p-44,
    0x1.c800000000000p-1, 0x1.da72763844000p-4, 0x1.a89401fa71733p-46,
    0x1.c600000000000p-1, 0x1.ec739830a0000p-4, 0x1.11fcba80cdd10p-44,
    0x1.c200000000000p-1, 0x1.08598b59e4000p-3, -0x1.7e5dd7009902cp-45,
    0x1.c000000000000p-1, 0x1.1178e8227e000p-3, 0x1.1ef78ce2d07f2p-45,
    0x1.bc00000000000p-1, 0x1.23d712a49c000p-3, 0x1.00d238fd3df5cp-46,
    0x1.ba00000000000p-1, 0x1.2d1610c868000p-3, 0x1.39d6ccb81b4a1p-47,
    0x1.b600000000000p-1, 0x1.3fb45a5992000p-3, 0x1.19713c0cae559p-44,
    0x1.b400000000000p-1, 0x1.4913d8333c000p-3, -0x1.53e43558124c4p-44,
    0x1.b000000000000p-1, 0x1.5bf406b544000p-3, -0x1.27023eb68981cp-46,
    0x1.ae00000000000p-1, 0x1.6574ebe8c2000p-3, -0x1.98c1d34f0f462p-44,
    0x1.aa00000000000p-1, 0x1.7898d85444000p-3, 0x1.8e67be3dbaf3fp-44,
    0x1.a800000000000p-1, 0x1.823c16551a000p-3, 0x1.e0ddb9a631e83p-46,
    0x1.a600000000000p-1, 0x1.8beafeb390000p-3, -0x1.73d54aae92cd1p-47,
    0x1.a200000000000p-1, 0x1.9f6c40708a000p-3, -0x1.337d94bcd3f43p-44,
    0x1.a000000000000p-1, 0x1.a93ed3c8ae000p-3, -0x1.8724350562169p-45,
    0x1.9e00000000000p-1, 0x1.b31d8575bc000p-3, 0x1.c794e562a63cbp-44,
    0x1.9a00000000000p-1, 0x1.c6ffbc6f00000p-3, 0x1.ee138d3a69d43p-44,
    0x1.9800000000000p-1, 0x1.d1037f2656000p-3, -0x1.84a7e75b6f6e4p-47,
    0x1.9600000000000p-1, 0x1.db13db0d48000p-3, 0x1.2806a847527e6p-44,
    0x1.9400000000000p-1, 0x1.e530effe72000p-3, -0x1.fdbdbb13f7c18p-44,
    0x1.9000000000000p-1, 0x1.f991c6cb3c000p-3, -0x1.90d04cd7cc834p-44,
    0x1.8e00000000000p-1, 0x1.01eae5626c000p-2, 0x1.a43dcfade85aep-44,
    0x1.8c00000000000p-1, 0x1.07138604d6000p-2, -0x1.e76324e912b17p-44,
    0x1.8a00000000000p-1, 0x1.0c42d67616000p-2, 0x1.7188b163ceae9p-45,
    0x1.8800000000000p-1, 0x1.1178e8227e000p-2, 0x1.1ef78ce2d07f2p-44,
    0x1.8400000000000p-1, 0x1.1bf99635a7000p-2, -0x1.1ac89575c2125p-44,
    0x1.8200000000000p-1, 0x1.214456d0ec000p-2, -0x1.caf0428b728a3p-44,
    0x1.8000000000000p-1, 0x1.269621134e000p-2, -0x1.1b61f10522625p-44,
    0x1.7e00000000000p-1, 0x1.2bef07cdc9000p-2, 0x1.a9cfa4a5004f4p-45,
    0x1.7c00000000000p-1, 0x1.314f1e1d36000p-2, -0x1.8e27ad3213cb8p-45,
    0x1.7a00000000000p-1, 0x1.36b6776be1000p-2, 0x1.16ecdb0f177c8p-46,
    0x1.7800000000000p-1, 0x1.3c25277333000p-2, 0x1.83b54b606bd5cp-46,
    0x1.7600000000000p-1, 0x1.419b423d5f000p-2, -0x1.ce379226de3ecp-44,
    0x1.7400000000000p-1, 0x1.4718dc271c000p-2, 0x1.06c18fb4c14c5p-44,
    0x1.7200000000000p-1, 0x1.4c9e09e173000p-2, -0x1.e20891b0ad8a4p-45,
    0x1.7000000000000p-1, 0x1.522ae0738a000p-2, 0x1.ebe708164c759p-45,
    0x1.6e00000000000p-1, 0x1.57bf753c8d000p-2, 0x1.fadedee5d40efp-46,
    0x1.6c00000000000p-1, 0x1.5d5bddf596000p-2, -0x1.a0b2a08a465dcp-47,
    0x1.6a00000000000p-1, 0x1.630030b3ab000p-2, -0x1.db623e731ae00p-45,
    0x1.6800000000000p-1, 0x1.68ac83e9c7000p-2, -0x1.7af966c548a30p-44,
    0x1.6600000000000p-1, 0x1.6e60ee6af2000p-2, -0x1.a37a6a0f7749ep-44,
    0x1.6400000000000p-1, 0x1.741d876c68000p-2, -0x1.13a7b5b11cfa7p-44,
    0x1.6200000000000p-1, 0x1.79e26687d0000p-2, -0x1.309c168817444p-44,
    0x1.6000000000000p-1, 0x1.7fafa3bd81000p-2, 0x1.46fb79bf6d4cbp-44,
    0x1.5e00000000000p-1, 0x1.85855776dd000p-2, -0x1.015486666443bp-44,
    0x1.5c00000000000p-1, 0x1.8b639a88b3000p-2, -0x1.05ae1e5e70470p-45,
    0x1.5a00000000000p-1, 0x1.914a8635bf000p-2, 0x1.a2652b44673e1p-44,
    0x1.5800000000000p-1, 0x1.973a343135000p-2, 0x1.ab73b16bf4984p-44,
    0x1.5600000000000p-1, 0x1.9d32bea15f000p-2, -0x1.6279e10d0c0b0p-45,
    0x1.5400000000000p-1, 0x1.a334402250000p-2, -0x1.61cdd40314305p-44,
    0x1.5200000000000p-1, 0x1.a93ed3c8ae000p-2, -0x1.8724350562169p-44,
    0x1.5000000000000p-1, 0x1.af5295248d000p-2, -0x1.17cc552774458p-45,
    0x1.5000000000000p-1, 0x1.af5295248d000p-2, -0x1.17cc552774458p-45,
    0x1.4e00000000000p-1, 0x1.b56fa04463000p-2, -0x1.bdab6b49ef99bp-44,
    0x1.4c00000000000p-1, 0x1.bb9611b80e000p-2, 0x1.7d85bf40a666dp-45,
    0x1.4a00000000000p-1, 0x1.c1c60693fa000p-2, 0x1.cec807fe8e180p-45,
    0x1.4800000000000p-1, 0x1.c7ff9c7455000p-2, 0x1.324911f56db29p-44,
    0x1.4600000000000p-1, 0x1.ce42f18064000p-2, 0x1.d0d0798270b2ap-44,
    0x1.4600000000000p-1, 0x1.ce42f18064000p-2, 0x1.d0d0798270b2ap-44,
    0x1.4400000000000p-1, 0x1.d490246df0000p-2, -0x1.652280b2c4c2cp-44,
    0x1.4200000000000p-1, 0x1.dae75484c9000p-2, 0x1.856f4a7c8e7a6p-44,
    0x1.4000000000000p-1, 0x1.e148a1a272000p-2, 0x1.b36537e3375b2p-44,
    0x1.3e00000000000p-1, 0x1.e7b42c3ddb000p-2, -0x1.465505372bd08p-45,
    0x1.3e00000000000p-1, 0x1.e7b42c3ddb000p-2, -0x1.465505372bd08p-45,
    0x1.3c00000000000p-1, 0x1.ee2a156b41000p-2, 0x1.f27f45a470251p-45,
    0x1.3a00000000000p-1, 0x1.f4aa7ee032000p-2, -0x1.b4c86a43fad5dp-44,
    0x1.3800000000000p-1, 0x1.fb358af7a5000p-2, -0x1.def40b87d36d9p-44,
    0x1.3800000000000p-1, 0x1.fb358af7a5000p-2, -0x1.def40b87d36d9p-44,
    0x1.3600000000000p-1, 0x1.00e5ae5b20800p-1, -0x1.53ba3b1727b1cp-47,
    0x1.3400000000000p-1, 0x1.04360be760000p-1, 0x1.d6774030d58c4p-44,
    0x1.3200000000000p-1, 0x1.078bf0533c800p-1, -0x1.4bf6edf090501p-44,
    0x1.3200000000000p-1, 0x1.078bf0533c800p-1, -0x1.4bf6edf090501p-44,
    0x1.3000000000000p-1, 0x1.0ae76e2d05800p-1, -0x1.82de51de06076p-44,
    0x1.2e00000000000p-1, 0x1.0e4898611d000p-1, -0x1.8f599fe1ffa30p-44,
    0x1.2e00000000000p-1, 0x1.0e4898611d000p-1, -0x1.8f599fe1ffa30p-44,
    0x1.2c00000000000p-1, 0x1.11af823c75800p-1, 0x1.53cdc223111a7p-44,
    0x1.2a00000000000p-1, 0x1.151c3f6f29800p-1, -0x1.edd97a293ae49p-45,
    0x1.2a00000000000p-1, 0x1.151c3f6f29800p-1, -0x1.edd97a293ae49p-45,
    0x1.2800000000000p-1, 0x1.188ee40f24000p-1, -0x1.accec41d52e6cp-44,
    0x1.2600000000000p-1, 0x1.1c07849ae6000p-1, 0x1.cacdeed70e667p-51,
    0x1.2600000000000p-1, 0x1.1c07849ae6000p-1, 0x1.cacdeed70e667p-51,
    0x1.2400000000000p-1, 0x1.1f8635fc61800p-1, -0x1.a7242c9fe81d3p-45,
    0x1.2200000000000p-1, 0x1.230b0d8bec000p-1, -0x1.b40fe646de661p-44,
    0x1.2200000000000p-1, 0x1.230b0d8bec000p-1, -0x1.b40fe646de661p-44,
    0x1.2000000000000p-1, 0x1.269621134d800p-1, 0x1.c93c1df5bb3b6p-44,
    0x1.1e00000000000p-1, 0x1.2a2786d0ec000p-1, 0x1.06d2be797882dp-45,
    0x1.1e00000000000p-1, 0x1.2a2786d0ec000p-1, 0x1.06d2be797882dp-45,
    0x1.1c00000000000p-1, 0x1.2dbf557b0e000p-1, -0x1.7a6e507b9dc11p-46,
    0x1.1c00000000000p-1, 0x1.2dbf557b0e000p-1, -0x1.7a6e507b9dc11p-46,
    0x1.1a00000000000p-1, 0x1.315da44340800p-1, -0x1.74e93c5a0ed9cp-45,
    0x1.1800000000000p-1, 0x1.35028ad9d9000p-1, -0x1.bd1f01ab60655p-44,
    0x1.1800000000000p-1, 0x1.35028ad9d9000p-1, -0x1.bd1f01ab60655p-44,
    0x1.1600000000000p-1, 0x1.38ae217197800p-1, -0x1.18b7abb5569a4p-45,
    0x1.1600000000000p-1, 0x1.38ae217197800p-1, -0x1.18b7abb5569a4p-45,
    0x1.1400000000000p-1, 0x1.3c6080c36c000p-1, -0x1.2b7367cfe13c2p-47,
    0x1.1200000000000p-1, 0x1.4019c2125c800p-1, 0x1.498c367879c5ap-44,
    0x1.1200000000000p-1, 0x1.4019c2125c800p-1, 0x1.498c367879c5ap-44,
    0x1.1000000000000p-1, 0x1.43d9ff2f92000p-1, 0x1.e267b0b7efae1p-44,
    0x1.1000000000000p-1, 0x1.43d9ff2f92000p-1, 0x1.e267b0b7efae1p-44,
    0x1.0e00000000000p-1, 0x1.47a1527e8a000p-1, 0x1.69a4a83594fabp-44,
    0x1.0e00000000000p-1, 0x1.47a1527e8a000p-1, 0x1.69a4a83594fabp-44,
    0x1.0c00000000000p-1, 0x1.4b6fd6f971000p-1, -0x1.f047750959d5fp-44,
    0x1.0a00000000000p-1, 0x1.4f45a835a5000p-1, -0x1.e6c516d93b8fbp-45,
    0x1.0a00000000000p-1, 0x1.4f45a835a5000p-1, -0x1.e6c516d93b8fbp-45,
    0x1.0800000000000p-1, 0x1.5322e26867800p-1, 0x1.5ccc45d257531p-47,
    0x1.0800000000000p-1, 0x1.5322e26867800p-1, 0x1.5ccc45d257531p-47,
    0x1.0600000000000p-1, 0x1.5707a26bb9000p-1, -0x1.cccfe80199f84p-44,
    0x1.0600000000000p-1, 0x1.5707a26bb9000p-1, -0x1.cccfe80199f84p-44,
    0x1.0400000000000p-1, 0x1.5af405c364800p-1, 0x1.dfa63ac10c9fbp-45,
    0x1.0400000000000p-1, 0x1.5af405c364800p-1, 0x1.dfa63ac10c9fbp-45,
    0x1.0200000000000p-1, 0x1.5ee82aa241800p-1, 0x1.202380cda46bep-45,
    0x1.0200000000000p-1, 0x1.5ee82aa241800p-1, 0x1.202380cda46bep-45,
    0x1.0000000000000p-1, 0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45,
};
/* 2^(j/128): nearest double, the rest */
SFM_TAB sfm_pow_exp_tab[128 * 2] = {
    0x1.0000000000000p+0, 0.0,
    0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54,
    0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56,
    0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54,
    0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55,
    0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55,
    0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57,
    0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54,
    0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54,
    0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54,
    0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59,
    0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57,
    0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54,
    0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58,
    0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54,
    0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55,
    0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55,
    0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54,
    0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55,
    0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54,
    0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54,
    0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54,
    0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55,
    0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55,
    0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54,
    0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55,
    0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55,
    0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54,
    0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55,
    0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59,
    0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54,
    0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56,
    0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55,
    0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55,
    0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54,
    0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55,
    0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54,
    0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54,
    0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56,
    0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54,
    0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55,
    0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54,
    0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58,
    0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55,
    0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59,
    0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54,
    0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56,
    0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54,
    0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56,
    0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54,
    0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54,
    0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55,
    0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55,
    0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55,
    0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54,
    0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55,
    0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54,
    0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60,
    0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54,
    0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54,
    0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54,
    0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55,
    0x1.6623882552225p+0, -0x1.bb60987591c34p-54,
    0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57,
    0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54,
    0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56,
    0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57,
    0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55,
    0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55,
    0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54,
    0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54,
    0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54,
    0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55,
    0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54,
    0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56,
    0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54,
    0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54,
    0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55,
    0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54,
    0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54,
    0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54,
    0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56,
    0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55,
    0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54,
    0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57,
    0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56,
    0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54,
    0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54,
    0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56,
    0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56,
    0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54,
    0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54,
    0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54,
    0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54,
    0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54,
    0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55,
    0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54,
    0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54,
    0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57,
    0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54,
    0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56,
    0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54,
    0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55,
    0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54,
    0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55,
    0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54,
    0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54,
    0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56,
    0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56,
    0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55,
    0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54,
    0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54,
    0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55,
    0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54,
    0x1.da9e603db3285p+0, 0x1.c2300696db532p-54,
    0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54,
    0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54,
    0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54,
    0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55,
    0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54,
    0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54,
    0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54,
    0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54,
    0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54,
    0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54,
    0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54,
    0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55,
    0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57,
};
#define SFM_POW_LN2_HI 0x1.62e42fefa3800p-1   /* ln 2, a multiple of 2^-42 */
#define SFM_POW_LN2_LO 0x1.ef35793c76730p-45
#define SFM_POW_L_HI 0x1.62e42fefa4000p-8   /* ln 2 / 128, a multiple of 2^-46 */
#define SFM_POW_L_LO -0x1.8432a1b0e2634p-50
#define SFM_POW_INV_L 0x1.71547652b82fep+7   /* 128 / ln 2 */

/* x^y of the slow evaluation, out of line */
SFM_COLD double sfm_pow_slow(double x, double y) { return sfm_pow(x, y); }

/* x^y; the bits of sfm_pow(x, y) for every x and y */
SFM_FN double sfm_pow_quick(double x, double y) {
  const int64_t bx = sfm_bits(x), by = sfm_bits(y) & 0x7fffffffffffffffLL;
  /* x positive and normal, |y| below 2^10 (NaN and infinities are not) */
  if (bx < 0x0010000000000000LL || bx >= 0x7ff0000000000000LL || by >= 0x4090000000000000LL) return sfm_pow_slow(x, y);
  const int i = (int)((bx >> 45) & 127);
  const double kd = (double)(int)((bx >> 52) - 1023);
  const double m = sfm_from_bits((bx & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);
  const double* lt = sfm_pow_log_tab + 3 * i;
  const double r = SFM_FMA(m, SFM_LD(lt), -1.0);
  const double p = SFM_MUL(r, r), pe = SFM_FMA(r, r, -p);
  double w = SFM_FMA(r, 0x1.c71c71c71c71cp-4, -0.125);
  w = SFM_FMA(r, w, 0x1.2492492492492p-3);
  w = SFM_FMA(r, w, -0x1.5555555555555p-3);
  w = SFM_FMA(r, w, 0x1.999999999999ap-3);
  w = SFM_FMA(r, w, -0.25);
  w = SFM_FMA(r, w, 0x1.5555555555555p-2);
  const double cub = SFM_MUL(SFM_MUL(p, r), w);
  const double a = SFM_FMA(kd, SFM_POW_LN2_HI, SFM_LD(lt + 1));
  const sfm_dd s1 = sfm_two_sum(a, r);
  const sfm_dd s2 = sfm_two_sum(s1.hi, SFM_MUL(-0.5, p));
  double lo = SFM_FMA(kd, SFM_POW_LN2_LO, SFM_LD(lt + 2));
  lo = SFM_ADD(lo, cub);
  lo = SFM_FMA(-0.5, pe, lo);
  lo = SFM_ADD(SFM_ADD(lo, s2.lo), s1.lo);
  const sfm_dd l = sfm_two_sum(s2.hi, lo);
  const sfm_dd z0 = sfm_two_prod(y, l.hi);
  const double zl = SFM_FMA(y, l.lo, z0.lo);
  /* |y log x| below 700: the scaling by a power of two stays normal */
  if ((sfm_bits(z0.hi) & 0x7fffffffffffffffLL) >= 0x4085e00000000000LL) return sfm_pow_slow(x, y);
  const double t = SFM_FMA(z0.hi, SFM_POW_INV_L, 0x1.8p52);
  const double nd = SFM_SUB(t, 0x1.8p52);
  const int n = (int)(uint32_t)sfm_bits(t);
  const double rh = SFM_FMA(-nd, SFM_POW_L_HI, z0.hi);
  const double rl = SFM_FMA(-nd, SFM_POW_L_LO, zl);
  const double rr = SFM_ADD(rh, rl);
  double e = SFM_FMA(rr, 0x1.6c16c16c16c17p-10, 0x1.1111111111111p-7);
  e = SFM_FMA(rr, e, 0x1.5555555555555p-5);
  e = SFM_FMA(rr, e, 0x1.5555555555555p-3);
  e = SFM_FMA(rr, e, 0.5);
  const double q = SFM_FMA(SFM_MUL(rr, rr), e, rl);
  const double* et = sfm_pow_exp_tab + 2 * (n & 127);
  const double th = SFM_LD(et), tl = SFM_LD(et + 1);
  const sfm_dd pr = sfm_two_prod(th, rh);
  const sfm_dd s = sfm_fast_two_sum(th, pr.hi);
  double g = SFM_FMA(th, q, pr.lo);
  g = SFM_FMA(tl, rh, g);
  g = SFM_ADD(s.lo, SFM_ADD(g, tl));
  /* the value lies in (0.99, 2.01): 2^-64 is above 2^-65 of it */
  const double u = SFM_ADD(s.hi, SFM_SUB(g, 0x1p-64)), v = SFM_ADD(s.hi, SFM_ADD(g, 0x1p-64));
  if (sfm_bits(u) != sfm_bits(v)) return sfm_pow_slow(x, y);
  return sfm_from_bits(sfm_bits(u) + ((int64_t)(n >> 7) << 52));
}

/* the FP64 evaluation, out of line */
SFM_COLD double sfm_pow_quick_cold(double x, double y) { return sfm_pow_quick(x, y); }

/*
 * The same power on the integer pipes.  An FP64 instruction of a warp holds
 * an SM's FP64 pipe for 16 cycles on GB300, in which the SM issues up to 64
 * others, so 64-bit fixed point beats FP64 arithmetic: log2 x and 2^f by the
 * reductions above with series in 64 x 64 -> 128 bit products (base 2, so
 * that y log2 x splits into integer and fraction exactly), the result to
 * 2^-61 (|y| < 1) or 2^-59 (|y| < 8).  The rounding test then leaves about
 * one argument in two hundred (|y| < 1) to the FP64 evaluation above.
 * log2 x = k + L_i + log2(1 + r), r = m c - 1 exact, L_i in [-1/2, 1/2] to
 * 2^-64; log2(1 + r) = r P(r) to r^8 (next term below 2^-68); y log2 x exact
 * in 128 bits; 2^f = 1 + f Q(f), |f| <= 2^-8, to f^6 (next below 2^-71).
 * Coefficients: of P and Q at the scales 2^(62 - 6 n), so that a Horner step
 * is one high product.
 */
#if defined(__CUDACC__)
#define SFM_ITAB static __device__ const int64_t
SFM_FN int64_t sfm_mulhi(int64_t a, int64_t b) { return __mul64hi(a, b); }
SFM_FN int32_t sfm_mulhi32(int32_t a, int32_t b) { return __mulhi(a, b); }
#else
#define SFM_ITAB static const int64_t
SFM_FN int64_t sfm_mulhi(int64_t a, int64_t b) { return (int64_t)(((__int128)a * b) >> 64); }
SFM_FN int32_t sfm_mulhi32(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
#endif
/* per interval: L_i 2^63 (-log2 c, less 1 from the interval of 1/sqrt(2) on), 256 c */
SFM_ITAB sfm_powi_log_tab[128 * 2] = {
    52080352580344565LL, 255,
    156856587611359393LL, 253,
    262464388758716179LL, 251,
    368917061291480011LL, 249,
    476228232387282600LL, 247,
    584411861601177296LL, 245,
    638835303920586374LL, 244,
    748354548482425863LL, 242,
    858782676832593460LL, 240,
    970134900679354152LL, 238,
    1026162407023108733LL, 237,
    1138930142077825653LL, 235,
    1252661715613151172LL, 233,
    1309894118242293459LL, 232,
    1425102743535505569LL, 230,
    1541317570432119309LL, 228,
    1599807832071135499LL, 227,
    1717565353665186919LL, 225,
    1776837224931603046LL, 224,
    1896178949527447616LL, 222,
    1956253602797536653LL, 221,
    2077222736812378418LL, 219,
    2138122216557105918LL, 218,
    2260763758429090961LL, 216,
    2322511029776656571LL, 215,
    2446871870455587345LL, 213,
    2509490871181947108LL, 212,
    2572405943934259308LL, 211,
    2699135598006097888LL, 209,
    2762955927049785547LL, 208,
    2827083825132003070LL, 207,
    2956274287476944212LL, 205,
    3021342940842373362LL, 204,
    3086731343173896505LL, 203,
    3152442652505152648LL, 202,
    3284846860330718215LL, 200,
    3351546313759202669LL, 199,
    3418581786003069540LL, 198,
    3485956679806199380LL, 197,
    3553674449863206093LL, 196,
    3690152703675950302LL, 194,
    3758920366278535087LL, 193,
    3828045265094622256LL, 192,
    3897531131076026346LL, 191,
    3967381753930244064LL, 190,
    4037600983360694007LL, 189,
    4108192730339854449LL, 188,
    4179160968416351941LL, 187,
    4250509735057093000LL, 186,
    4322243133025572372LL, 185,
    4394365331797534366LL, 184,
    4466880569015208631LL, 183,
    4539793151981388594LL, 182,
    -4610264577660106100LL, 181,
    -4536544094927560092LL, 180,
    -4462412911008301306LL, 179,
    -4387866424172454937LL, 178,
    -4312899954913613981LL, 177,
    -4237508744186174972LL, 176,
    -4161687951592454547LL, 175,
    -4085432653517860093LL, 174,
    -4008737841212318039LL, 173,
    -3931598418816090440LL, 172,
    -3854009201328034243LL, 171,
    -3775964912514277691LL, 170,
    -3697460182755204713LL, 169,
    -3618489546828550505LL, 168,
    -3618489546828550505LL, 168,
    -3539047441626319689LL, 167,
    -3459128203803142245LL, 166,
    -3378726067353581513LL, 165,
    -3297835161115802799LL, 164,
    -3216449506198900170LL, 163,
    -3216449506198900170LL, 163,
    -3134563013331062591LL, 162,
    -3052169480125638396LL, 161,
    -2969262588262028797LL, 160,
    -2885835900578206443LL, 159,
    -2885835900578206443LL, 159,
    -2801882858071513523LL, 158,
    -2717396776804245214LL, 157,
    -2632370844710368005LL, 156,
    -2632370844710368005LL, 156,
    -2546798118299558053LL, 155,
    -2460671519254571926LL, 154,
    -2373983830917780190LL, 153,
    -2373983830917780190LL, 153,
    -2286727694662502948LL, 152,
    -2198895606144584904LL, 151,
    -2198895606144584904LL, 151,
    -2110479911429435337LL, 150,
    -2021472802989534785LL, 149,
    -2021472802989534785LL, 149,
    -1931866315567174640LL, 148,
    -1841652321896947459LL, 147,
    -1841652321896947459LL, 147,
    -1750822528282243838LL, 146,
    -1659368470019735338LL, 145,
    -1659368470019735338LL, 145,
    -1567281506665531296LL, 144,
    -1474552817136389425LL, 143,
    -1474552817136389425LL, 143,
    -1381173394639034911LL, 142,
    -1381173394639034911LL, 142,
    -1287134041420299103LL, 141,
    -1192425363330425750LL, 140,
    -1192425363330425750LL, 140,
    -1097037764191508750LL, 139,
    -1097037764191508750LL, 139,
    -1000961439962619186LL, 138,
    -904186372692749655LL, 137,
    -904186372692749655LL, 137,
    -806702324252248894LL, 136,
    -806702324252248894LL, 136,
    -708498829832937836LL, 135,
    -708498829832937836LL, 135,
    -609565191206587738LL, 134,
    -509890469730899901LL, 133,
    -509890469730899901LL, 133,
    -409463479091552716LL, 132,
    -409463479091552716LL, 132,
    -308272777768273083LL, 131,
    -308272777768273083LL, 131,
    -206306661212243249LL, 130,
    -206306661212243249LL, 130,
    -103553153721468184LL, 129,
    -103553153721468184LL, 129,
    0LL, 128,
};
#define SFM_POWI_J 53
/* 2^(j/128) 2^63 - 2^63 */
SFM_ITAB sfm_powi_exp_tab[128] = {
    0LL,
    50081998086712172LL,
    100435936470566771LL,
    151063291760485868LL,
    201965548583231959LL,
    253144199626944055LL,
    304600745684910150LL,
    356336695699577385LL,
    408353566806801173LL,
    460652884380334596LL,
    513236182076559376LL,
    566105001879459730LL,
    619260894145840423LL,
    672705417650790365LL,
    726440139633393050LL,
    780466635842685220LL,
    834786490583865063LL,
    889401296764751326LL,
    944312655942494694LL,
    999522178370542806LL,
    1055031483045860288LL,
    1110842197756405188LL,
    1166955959128863196LL,
    1223374412676641067LL,
    1280099212848120630LL,
    1337132023075174828LL,
    1394474515821947180LL,
    1452128372633896118LL,
    1510095284187105633LL,
    1568376950337863663LL,
    1626975080172509696LL,
    1685891392057553038LL,
    1745127613690063215LL,
    1804685482148333994LL,
    1864566743942822501LL,
    1924773155067364938LL,
    1985306481050670393LL,
    2046168497008094253LL,
    2107360987693692753LL,
    2168885747552560160LL,
    2230744580773450158LL,
    2292939301341682950LL,
    2355471733092339650LL,
    2418343709763745508LL,
    2481557075051243545LL,
    2545113682661260179LL,
    2609015396365664414LL,
    2673264090056422201LL,
    2737861647800547562LL,
    2802809963895352094LL,
    2868110942923994474LL,
    2933766499811331593LL,
    2999778559880072952LL,
    3066149058907239977LL,
    3132879943180931895LL,
    3199973169557399849LL,
    3267430705518430918LL,
    3335254529229043726LL,
    3403446629595497333LL,
    3472009006323615108LL,
    3540943669977425296LL,
    3610252642038119995LL,
    3679937954963334281LL,
    3750001652246747201LL,
    3820445788478006404LL,
    3891272429402978156LL,
    3962483651984324497LL,
    4034081544462409340LL,
    4106068206416535273LL,
    4178445748826512875LL,
    4251216294134564347LL,
    4324381976307563277LL,
    4397944940899612351LL,
    4471907345114960866LL,
    4546271357871263875LL,
    4621039159863184816LL,
    4696212943626343510LL,
    4771794913601611379LL,
    4847787286199755783LL,
    4924192289866435379LL,
    5001012165147548381LL,
    5078249164754935673LL,
    5155905553632440669LL,
    5233983609022327877LL,
    5312485620532062115LL,
    5391413890201450318LL,
    5470770732570147933LL,
    5550558474745531858LL,
    5630779456470941924LL,
    5711436030194292929LL,
    5792530561137059221LL,
    5874065427363633862LL,
    5956043019851064410LL,
    6038465742559167353LL,
    6121336012501023263LL,
    6204656259813854727LL,
    6288428927830289140LL,
    6372656473150008452LL,
    6457341365711787958LL,
    6542486088865926258LL,
    6628093139447068501LL,
    6714165027847425056LL,
    6800704278090387748LL,
    6887713427904545824LL,
    6975195028798103825LL,
    7063151646133703529LL,
    7151585859203652177LL,
    7240500261305559181LL,
    7329897459818383528LL,
    7419780076278894114LL,
    7510150746458545256LL,
    7601012120440769623LL,
    7692366862698690863LL,
    7784217652173258204LL,
    7876567182351805316LL,
    7969418161347035739LL,
    8062773311976437195LL,
    8156635371842127113LL,
    8251007093411131706LL,
    8345891244096100955LL,
    8441290606336461868LL,
    8537207977680012398LL,
    8633646170864958393LL,
    8730608013902396020LL,
    8828096350159242042LL,
    8926114038441614409LL,
    9024663953078665589LL,
    9123748984006871116LL,
};
#define SFM_POWI_P0 (6653256548922161246LL)
#define SFM_POWI_P1 (-51978566788454385LL)
#define SFM_POWI_P2 (541443404046400LL)
#define SFM_POWI_P3 (-6345039891169LL)
#define SFM_POWI_P4 (79312998640LL)
#define SFM_POWI_P5 (-1032721336)
#define SFM_POWI_P6 (13831089)
#define SFM_POWI_P7 (-189097)
#define SFM_POWI_Q0 (3196577161300663915LL)
#define SFM_POWI_Q1 (17310144115608349LL)
#define SFM_POWI_Q2 (62492070775105LL)
#define SFM_POWI_Q3 (169203916661LL)
#define SFM_POWI_Q4 (366510056)
#define SFM_POWI_Q5 (661577)

/* x^y; the bits of sfm_pow(x, y) for every x and y */
SFM_COLD double sfm_pow_int(double x, double y) {
  const int64_t bx = sfm_bits(x), by = sfm_bits(y);
  const int ey = (int)((by >> 52) & 0x7ff) - 1023;
  /* x positive and normal, |y| in [2^-3, 8) */
  if (bx < 0x0010000000000000LL || bx >= 0x7ff0000000000000LL || (unsigned)(ey + 3) > 5u) return sfm_pow_quick_cold(x, y);
  const int i = (int)((bx >> 45) & 127);
  const int k = (int)((bx >> 52) - 1023) + (i >= SFM_POWI_J ? 1 : 0);
  const int64_t ya = ((by & 0x000fffffffffffffLL) | 0x0010000000000000LL) << (ey + 3);   /* |y| 2^55 */
  /* |y log2 x| below 500 */
  if (((int)(ya >> 55) + 1) * ((k < 0 ? -k : k) + 1) > 480) return sfm_pow_quick_cold(x, y);
  const int64_t yf = by < 0 ? -ya : ya;
  const int64_t c8 = SFM_LD(sfm_powi_log_tab + 2 * i + 1);
  /* r 2^70 */
  const int64_t rs = ((((bx & 0x000fffffffffffffLL) | 0x0010000000000000LL) * c8) - 0x1000000000000000LL) << 10;
  const int32_t rh = (int32_t)(rs >> 32);
  const int32_t p5 = SFM_POWI_P5 + sfm_mulhi32(rh, SFM_POWI_P6 + sfm_mulhi32(rh, SFM_POWI_P7));
  int64_t p = SFM_POWI_P4 + sfm_mulhi32(rh, p5);
  p = SFM_POWI_P3 + sfm_mulhi(rs, p);
  p = SFM_POWI_P2 + sfm_mulhi(rs, p);
  p = SFM_POWI_P1 + sfm_mulhi(rs, p);
  p = SFM_POWI_P0 + sfm_mulhi(rs, p);
  const int64_t L = SFM_LD(sfm_powi_log_tab + 2 * i) + ((sfm_mulhi(rs, p) + 16) >> 5);   /* (log2 x - k) 2^63 */
  /* E = y log2 x at 2^118 in (eh, el) */
  const uint64_t el0 = (uint64_t)yf * (uint64_t)L;
  const int64_t eh0 = sfm_mulhi(yf, L);
  const uint64_t kl = (uint64_t)yf * (uint64_t)(int64_t)k;
  const int64_t kh = sfm_mulhi(yf, (int64_t)k);
  const uint64_t el = el0 + (kl << 63);
  int64_t eh = eh0 + (int64_t)((kl >> 1) | ((uint64_t)kh << 63)) + (el < el0 ? 1 : 0);
  const int64_t n = (eh + 0x0000400000000000LL) >> 47;      /* 128 E rounded */
  eh -= (int64_t)((uint64_t)n << 47);
  const int64_t fs = (int64_t)(((uint64_t)eh << 16) | (el >> 48));   /* f 2^70 */
  const int32_t fh = (int32_t)(fs >> 32);
  int64_t q = SFM_POWI_Q3 + sfm_mulhi32(fh, SFM_POWI_Q4 + sfm_mulhi32(fh, SFM_POWI_Q5));
  q = SFM_POWI_Q2 + sfm_mulhi(fs, q);
  q = SFM_POWI_Q1 + sfm_mulhi(fs, q);
  q = SFM_POWI_Q0 + sfm_mulhi(fs, q);
  const int64_t fq = sfm_mulhi(fs, q);                      /* (2^f - 1) 2^68 */
  const uint64_t T = (uint64_t)SFM_LD(sfm_powi_exp_tab + (int)(n & 127)) + 0x8000000000000000ULL;
  uint64_t G = T + (uint64_t)((sfm_mulhi((int64_t)(T >> 1), fq) + 4) >> 3);   /* 2^(f + j/128) 2^63 */
  int e = (int)(n >> 7) + 1022;
  if (!(G >> 63)) {
    G <<= 1;
    e -= 1;
  }
  /* G is off by at most 1.1 |y| ln 2 2^(j/128) units of 2^-63 from log2 x and
     1.2 from the table and the last product (twice that in units below 1):
     3.3 for |y| < 1, 13 for |y| < 8.  Round unless the midpoint is that close */
  const int err = ey < 0 ? 4 : 14;
  const int low = (int)(G & 2047u) - 1024;
  if (low <= err && low >= -err) return sfm_pow_quick_cold(x, y);
  return sfm_from_bits((int64_t)(((uint64_t)e << 52) + (G >> 11) + (low > 0 ? 1u : 0u)));
}

#endif /* SFLOW_POW_H */
