// Exact digit slices of FP64 numbers for the tensor cores, shared by the sliced kernels: a number x
// with |x| < 2^e becomes V = round(x 2^(62 - e)) = sum_t d_t 256^(7 - t) with |d_t| <= 128, |d_0| <= 65
// (each digit exact in BF16), and sums of digit products S_w (w = i + j < 8) collected as the integer
// T = sum_w S_w 256^(7 - w) give the dot product T 2^(ea + eb - 68).
#pragma once
#include "xrh_common.cuh"

namespace xrh_sliced {

constexpr int NS = XRH_SLICES;

// A 96-bit two's complement sum T (w0 lowest).
struct Sum96 {
    uint32_t w0, w1, w2;
};

__device__ __forceinline__ void add96(Sum96& s, uint32_t a0, uint32_t a1, uint32_t a2) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(s.w0), "+r"(s.w1), "+r"(s.w2)
        : "r"(a0), "r"(a1), "r"(a2));
}

// s[j] += S_w 256^(7 - w) for the accumulators v[j] of weight w < 8 (integers below 2^24 in magnitude).
// Conversions (16 lanes/clk/SM) bound it; a 32 x 32 + 64 bit multiply-add also runs at 16 lanes/clk/SM,
// on another pipe, so the weights that need 64 bits take one and those that need 96 shifts and carries.
template <int N>
__device__ __forceinline__ void add_weight(Sum96* s, const float (&v)[N], int w) {
    const int sh = 8 * (3 - (w & 3));
    if (w < 4) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int x = __float2int_rn(v[j]);
            const uint64_t h = (((uint64_t)s[j].w2 << 32) | s[j].w1) + (uint64_t)((int64_t)x * (1 << sh));
            s[j].w1 = (uint32_t)h;
            s[j].w2 = (uint32_t)(h >> 32);
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int x = __float2int_rn(v[j]);
            const uint32_t g = (uint32_t)(x >> 31);
            add96(s[j], (uint32_t)x << sh, __funnelshift_l((uint32_t)x, g, sh), g);
        }
    }
}

// All eight weights of a sum over at most K <= 64 products a pair: T = sum_w v[w] 256^(7 - w).  With
// |S_w| <= K ((w - 1) 2^14 + 2 * 65 * 128) a sum below 2^22 becomes an integer by an addition on the FP32
// pipe (1.5 2^23 + S has it in its low bits) instead of a conversion at 16 lanes/clk/SM, and two
// neighbouring weights fit 32 bits.
template <int K>
__device__ __forceinline__ Sum96 collect_weights(const float (&v)[8]) {
    static_assert(K <= 64, "two weights in 32 bits");
    int y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (K <= 32 || i < 2) {
            const uint32_t a = __float_as_uint(v[2 * i] + 12582912.0f), b = __float_as_uint(v[2 * i + 1] + 12582912.0f);
            y[i] = (int)((a << 8) + b + 0x74c00000u);              // minus 0x4b400000 (256 + 1)
        } else {
            y[i] = (int)(((uint32_t)__float2int_rn(v[2 * i]) << 8) + (uint32_t)__float2int_rn(v[2 * i + 1]));
        }
    }
    const int64_t lo = (int64_t)y[2] * 65536 + y[3], hi = (int64_t)y[0] * 65536 + y[1];
    const uint32_t g = (uint32_t)(lo >> 63);
    Sum96 s;
    s.w0 = (uint32_t)lo;
    const uint64_t h = (uint64_t)hi + (((uint64_t)g << 32) | (uint32_t)(lo >> 32));
    s.w1 = (uint32_t)h;
    s.w2 = (uint32_t)(h >> 32);
    return s;
}

// T 2^(x - 68) rounded to FP64 (nearest, ties to even), |T| < 2^94, by about 45 integer operations
// without a branch (a branch per element serialises a thread's conversions; the FP64 pipe, conversions
// included, runs at 2 lanes/clk/SM).  `rare` is set, and the result is not valid, where it lies outside
// the normal range (sliced_to_double_rare).
__device__ __forceinline__ double sliced_to_double_fast(const Sum96& t, int x, bool& rare) {
    const uint32_t sg = (uint32_t)((int)t.w2 >> 31);    // all ones for a negative value
    uint32_t w0 = t.w0 ^ sg, w1 = t.w1 ^ sg, w2 = t.w2 ^ sg;
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
    rare = rare || (top != 0u && (unsigned)(e - 1) >= 2044u);
    return top == 0u ? 0.0 : v;
}

// The same for results that may lie anywhere: two roundings below the normal range, infinite above.
static __device__ __noinline__ double sliced_to_double_rare(const Sum96& t, int x) {
    bool rare = false;
    const int64_t hi = (int64_t)(((uint64_t)t.w2 << 32) | t.w1), mag = hi < 0 ? ~hi : hi;
    const int bits = 32 + 64 - __clzll(mag | 1);
    return scalbn(sliced_to_double_fast(t, 68 - bits, rare), x - 68 + bits);
}

// N sums at once: one branch for all of them, so that their operations interleave.
template <int N>
__device__ __forceinline__ void sliced_to_doubles(const Sum96 (&t)[N], const int (&x)[N], double (&v)[N]) {
    bool rare = false;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sliced_to_double_fast(t[i], x[i], rare);
    if (rare) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = sliced_to_double_rare(t[i], x[i]);
    }
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

// |x| 2^-e rounded down to BF16 (bits), at least 2^-60 for x != 0, for an x of a row with |x| < 2^e.  A sum
// of products of magnitudes bounds sum |a||b| 2^-(ea + eb) from below, and is zero only where every
// product is (2^-60 adds nothing at the threshold below).
__device__ __forceinline__ uint32_t magnitude(double x, int E) {
    const uint32_t hi = abs_hi(x);
    const int m = hi < 0x00100000u ? 0 : (int)(hi >> 13) - ((E - 126) << 7);       // (subnormal: the least one)
    return hi == 0u && __double2loint(x) == 0 ? 0u : (uint32_t)max(m, 67 << 7);
}

// Lanes that share one of `elements` sums of `terms` terms, for `threads` threads: a power of two, so that few
// elements keep the threads busy (and neighbouring lanes read neighbouring terms).
__device__ __forceinline__ int lanes_per_sum(int elements, int threads, int64_t terms, int least = 1) {
    int n = least;
    while (n < 32 && 2 * n * elements <= threads && 2 * n <= terms) n *= 2;
    return n;
}
// The sum over a group of n lanes (a power of two, whole warps call), in every lane.
__device__ __forceinline__ double sum_lanes(double x, int n) {
    for (int o = n / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Where a sum needs FP64 arithmetic.  What the digits leave out of K products, 2^-63 2^e of an element and
// the pairs with i + j >= 8 (7 2^14 256^-1 + .. units of 2^-68), is at most K 1.003 2^-59 2^(ea + eb); an FP64
// sum has the bound K 2^-53 sum |a||b|.  So the digits are as good where sum |a||b| >= 1.003 2^-6
// 2^(ea + eb): everywhere for rows of elements of like size (there it is about K / 16 and more), not where
// the large elements of one row meet zeros or small elements of the other.
constexpr float LOW_SUM = 1.01f / 64.0f;
__device__ __forceinline__ bool low_sum(float magnitudes) { return magnitudes > 0.0f && magnitudes < LOW_SUM; }

}  // namespace xrh_sliced
