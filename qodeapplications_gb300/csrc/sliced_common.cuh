// Exact digit slices of FP64 numbers for the tensor cores, shared by the sliced kernels: a number x
// with |x| < 2^e becomes V = round(x 2^(62 - e)) = sum_t d_t 256^(7 - t) with |d_t| <= 128, |d_0| <= 65
// (each digit exact in BF16), and sums of digit products S_w (w = i + j < 8) collected as the integer
// T = sum_w S_w 256^(7 - w) give the dot product T 2^(ea + eb - 68).
#pragma once
#include "xrh_common.cuh"

namespace xrh_sliced {

constexpr int NS = XRH_SLICES;

// (hi 2^32 + lo) 2^(x - 68) rounded to FP64 (nearest, ties to even), |hi 2^32 + lo| < 2^94, by about
// 45 integer operations without a branch (a branch per element serialises the 32 conversions of
// a thread: 52 000 cycles a tile; the FP64 pipe would need 16 000).  Results outside the normal
// range are formed by scalbn.
__device__ __forceinline__ double sliced_to_double(int64_t hi, uint32_t lo, int x) {
    const uint32_t sg = (uint32_t)(hi >> 63);           // all ones for a negative value
    uint32_t w0 = lo ^ sg, w1 = (uint32_t)hi ^ sg, w2 = (uint32_t)(hi >> 32) ^ sg;
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, %2, 0;"
        : "+r"(w0), "+r"(w1), "+r"(w2)
        : "r"(sg & 1u));
    // leading zeros of the 96 bits (w2 < 2^30); the leading one goes to bit 62 of (a : b), c behind
    const bool z2 = w2 == 0u, z1 = z2 && w1 == 0u;
    const uint32_t top = z1 ? w0 : (z2 ? w1 : w2);
    const int z = __clz((int)top);
    const int lz = z + (z1 ? 64 : (z2 ? 32 : 0));
    uint32_t a = z1 ? w0 : (z2 ? w1 : w2), b = z1 ? 0u : (z2 ? w0 : w1), c = z2 ? 0u : w0;
    a = __funnelshift_l(b, a, z);
    b = __funnelshift_l(c, b, z);
    c = c << (z & 31);
    const uint32_t sticky = (c != 0u) | (b & 1u);
    b = __funnelshift_r(b, a, 1) | sticky;
    a >>= 1;
    asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, 0;" : "+r"(b), "+r"(a) : "r"(0x1ffu + ((b >> 10) & 1u)));
    // 53 bits above bit 10; e - 1 is added above the implicit one
    const int e = 95 - lz + x - 68 + 1023;
    const uint32_t mh = a >> 10, ml = __funnelshift_r(b, a, 10);
    double v = __hiloint2double((int)((mh + ((uint32_t)(e - 1) << 20)) | (sg & 0x80000000u)), (int)ml);
    if (top == 0u) v = 0.0;
    else if ((unsigned)(e - 1) >= 2044u) {
        v = scalbn((double)(((uint64_t)mh << 32) | ml), e - 1075);
        if (sg) v = -v;
    }
    return v;
}

__device__ __forceinline__ int exp_of(uint32_t hi) {   // |x| < 2^exp_of for the row's largest high word
    const int E = (int)(hi >> 20);
    return (E < 1 ? 1 : E) - 1022;
}

__device__ __forceinline__ uint32_t abs_hi(double x) { return (uint32_t)__double2hiint(x) & 0x7fffffffu; }

// V = round(x 2^(62 - e)) for |x| < 2^e, with 128 added to its low seven digits: byte t of the
// result (t = 0 lowest) is digit 7 - t plus 128, the top byte (signed) is digit 0.
__device__ __forceinline__ uint64_t fixed62(double x, int E) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    uint64_t m = b & 0xfffffffffffffull;
    if (ex) m |= 1ull << 52;
    const int s = 9 - (E - (ex ? ex : 1));             // shift of the 53-bit mantissa
    uint64_t v;
    if (s >= 0) v = m << s;
    else if (s > -54) v = ((m >> (-s - 1)) + 1ull) >> 1;   // nearest, ties away
    else v = 0;
    const int64_t sv = (b >> 63) ? -(int64_t)v : (int64_t)v;
    return (uint64_t)sv + 0x0080808080808080ull;
}

// Digit t of such a V as the bits of a float (its upper half is the BF16).
__device__ __forceinline__ uint32_t digit_float(uint64_t v, int t) {
    const uint32_t word = t < 4 ? (uint32_t)(v >> 32) : (uint32_t)v;
    const uint32_t byte = (word >> (8 * (3 - (t & 3)))) & 0xffu;
    // 2^23 + byte exactly, minus 2^23 and the digit's bias
    if (t == 0) return __float_as_uint((float)(int)(int8_t)byte);
    return __float_as_uint(__uint_as_float(0x4b000000u | byte) - 8388736.0f);
}

}  // namespace xrh_sliced
