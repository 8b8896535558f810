// FP64 transition densities with exact digit products on the tensor cores (sm_103a).
//
//   rho[idx, I, J] = sum_c s_c zb[P_c, I] zk[Q_c, J]   over the couplings c of operator index idx
//
// is for every idx a product of two gathered matrices with the couplings as contraction index; on
// CUDA cores it runs at GB300's FP64 rate (2 DFMA/clk/SM).  Here every state's coefficients are scaled
// by the power of two above the largest of them and kept as eight BF16 digits per determinant
// (sliced_common.cuh), rows [8 slices][NPAD states] (NPAD = 16, 32, 64; larger state counts in blocks
// of 64), so that a coupling is two contiguous rows of 16 NPAD bytes.  They are gathered into
// shared memory as MN-major operands (128-byte swizzle: 64 elements x 8 couplings per KB) and every
// digit pair with i + j < 8 comes out of a few wide MMAs: the 128 rows of A tile t are its slices
// t G .. t G + G - 1 (G = 128 / NPAD), the columns all slices of B, and the accumulator column block
// t G + j takes A tile t x B slice j, so that lane group g of column block b holds the pairs of weight
// b + g with i = g mod G.  The sums stay below 2^24, so exact, for GROUP stages; they are collected in
// 96-bit integers, added over the lane groups and rounded once at the end of the index.
//
// The digits are relative to a state's largest coefficient: an error of at most count 1.003 2^-59 2^(eI + eJ)
// (gemm_sliced.cu) where an FP64 sum has count 2^-53 sum |zb||zk|.  Elements that need it are formed by FP64
// FMAs over their couplings, listed first so that all epilogue threads share them (low_sum in
// sliced_common.cuh: indices without a large coefficient in their couplings, as in the tails of a
// wave function).  Which ones is decided from below: one MMA over the magnitudes of 64 couplings spread over
// the list (all of a shorter one) finds most elements large enough, masks of the determinants' nonzero
// states find those without any product, and the rest are formed in FP64.  Gathering every coupling's
// magnitudes instead cost 18 % (14 orbitals, 40 states: 4.80 ms without, 4.94 with the sample, 5.70 with all;
// 5.06 with the sample and the masks).
//
// A CTA (persistent over a work list ordered by length), 16 warps:
//   * warps 8-11: cp.async gathers of stages of 32 couplings of one sign (positive ones first: the MMA
//     negates A for the negative ones);
//   * warp 12: MMAs;  * warps 0-7: collection and conversion.
// Bounds: the gathers, 2 x 16 NPAD bytes of L2 per coupling, against 640 / 192 / 64 cycles of the tensor
// pipe per 16 couplings at NPAD = 64 / 32 / 16, and the collection (8 NPAD columns a group).  Measured,
// all blocks of a fragment, no element in FP64: 28 spin orbitals, 60 states 115 -> 5.1 ms (97 GFLOP of
// canonical couplings, 19 TFLOP/s FP64 against the pipe's 1.1); 22, 27 states 0.47; 18, 10 states 3.4 -> 0.11.
// Every wait is bounded; on timeout *status is set and all roles leave after their copies and MMAs
// have completed.
#include "sliced_common.cuh"
#include "tc_common.cuh"
#include "xrh_common.cuh"

namespace {
using namespace xrh_tc;
using namespace xrh_sliced;

constexpr int DS_KS = 32;                              // couplings per stage
constexpr int DS_EPI = 256, DS_PROD = 128, DS_THREADS = DS_EPI + DS_PROD + 128;
constexpr int DS_SAMPLE = 64;                          // couplings whose magnitudes are summed
constexpr uint32_t DS_ATOM = DS_KS * 128;              // bytes between 64-element atoms of a stage side

template <int NPAD>
struct Cfg {
    static constexpr int G = 128 / NPAD;                               // slices per A tile
    static constexpr int TILES = NS / G;                               // A tiles
    static constexpr int COLS = NS * NPAD;                             // accumulator columns
    static constexpr uint32_t SIDE = (uint32_t)DS_KS * NS * NPAD * 2;  // bytes of one side of a stage
    static constexpr int STAGES = NPAD == 64 ? 3 : (NPAD == 32 ? 2 : 4);
    static constexpr int CTAS = NPAD == 64 ? 1 : 2;                    // per SM
    // TILES pairs of |d d| <= 2^14 fall on one accumulator: 2^24 / (TILES 2^14) couplings
    static constexpr int GROUP = (1 << 10) / TILES / DS_KS;            // stages per exact group
    static constexpr int CW = NPAD / 2;                                // output columns per epilogue thread
    // registers: 512 threads x 128 at launch = 65536 >= 256 x 168 + 256 x 72 (NPAD 64, one CTA an SM);
    // 512 x 64 = 32768 = 256 x 88 + 256 x 40 (two CTAs)
    static constexpr int EPI_REGS = CTAS == 1 ? 168 : 88, IO_REGS = CTAS == 1 ? 72 : 40;
    static_assert(DS_EPI * EPI_REGS + (DS_THREADS - DS_EPI) * IO_REGS <= DS_THREADS * (CTAS == 1 ? 128 : 64),
                  "register split exceeds the launch");
};

__device__ __forceinline__ void epi_bar() { named_bar<1, DS_EPI>(); }
__device__ __forceinline__ int epi_bar_or(int pred) { return named_bar_or<1, DS_EPI>(pred); }

// MN-major operand: 64-element atoms DS_ATOM apart, 8-coupling groups 1024 B apart.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(DS_ATOM >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Coupling i of the sample of an index with n couplings: spread over the list (which is ordered by sign and
// ket, so that every kind of determinant is met), or all of them.
__device__ __forceinline__ int sampled(int i, int n) { return n > DS_SAMPLE ? (int)((int64_t)i * n / DS_SAMPLE) : i; }

__device__ __forceinline__ int stages_of(int n) { return (n + DS_KS - 1) / DS_KS; }

// columns [c, c + n) of an accumulator, n = 8, 16, 32
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t ta, float (&v)[N]) {
    uint32_t r[N];
    if constexpr (N == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(ta)
                     : "memory");
    } else {
        static_assert(N == 16, "8 or 16 columns");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(ta)
                     : "memory");
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
}

// The magnitudes of a side's states, [block of 64 states][determinant][NPAD], behind its digits.
template <int NPAD>
__device__ __forceinline__ const uint8_t* magnitudes(const xrh_dens_sliced_task& T, int side) {
    const int64_t rows = (((side ? T.nk : T.nb) + 63) / 64) * (side ? T.conf_k : T.conf_b);
    return reinterpret_cast<const uint8_t*>(side ? T.digk : T.digb) + rows * (NS * NPAD * 2);
}

// Which of its block's states a determinant has a coefficient of, [block of 64 states][determinant], behind those.
template <int NPAD>
__device__ __forceinline__ const uint64_t* nonzero(const xrh_dens_sliced_task& T, int side) {
    const int64_t rows = (((side ? T.nk : T.nb) + 63) / 64) * (side ? T.conf_k : T.conf_b);
    return reinterpret_cast<const uint64_t*>(reinterpret_cast<const uint8_t*>(side ? T.digk : T.digb) + rows * ((NS + 1) * NPAD * 2));
}

template <int NPAD>
__global__ void __launch_bounds__(DS_THREADS, Cfg<NPAD>::CTAS)
    density_sliced_kernel(const xrh_dens_sliced_task* __restrict__ tasks, const xrh_dens_sliced_unit* __restrict__ units,
                          int64_t n_units, int32_t* status) {
    using C = Cfg<NPAD>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;       // [STAGES][bra, ket][atoms][couplings]
    __shared__ __align__(8) uint64_t full_bar[C::STAGES], empty_bar[C::STAGES];
    __shared__ __align__(8) uint64_t ready_bar, drained_bar, mag_ready_bar, mag_drained_bar, done_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_sh;
    __shared__ uint4 s_raw[128][9];
    __shared__ uint32_t s_eb[64], s_ek[64];
    __shared__ int s_count;                            // elements to form in FP64
    __shared__ unsigned long long s_nz[64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), DS_PROD);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&ready_bar), 1);
        mbar_init(smem_u32(&drained_bar), DS_EPI / 32);
        mbar_init(smem_u32(&mag_ready_bar), 1);
        mbar_init(smem_u32(&mag_drained_bar), DS_EPI / 32);
        mbar_init(smem_u32(&done_bar), 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(C::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh;

    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::IO_REGS));
        if (warp == 12 && lane == 0) {
            // ------------------------------------------------------------------------ MMA --
            constexpr uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (8u << 24);
            uint32_t st = 0, grp = 0, un = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++un) {
                const int np = units[u].n_pos, nn = units[u].count - np;
                const int s_pos = stages_of(np), n_st = s_pos + stages_of(nn);
                for (int q = 0; q < n_st && ok; ++q, ++st) {
                    const int in_group = q % C::GROUP;
                    const uint32_t s = st % C::STAGES;
                    if (in_group == 0 && q > 0 && !mbar_wait(smem_u32(&drained_bar), (grp - 1) & 1u, &abort_sh)) ok = false;
                    if (ok && !mbar_wait(smem_u32(&full_bar[s]), (st / C::STAGES) & 1u, &abort_sh)) ok = false;
                    if (!ok) break;
                    fence_copies();
                    tc_fence_after();
                    const uint32_t id = idesc0 | (q >= s_pos ? 1u << 13 : 0u);
                    const uint64_t da = desc_mn_sw128(ring + s * 2 * C::SIDE), db = desc_mn_sw128(ring + s * 2 * C::SIDE + C::SIDE);
                    // tile t, columns [c0, COLS) of its 128 t ..: slices of B from column c0 on
                    auto tile = [&](int t, int ks, int c0, int cols, uint32_t acc) {
                        umma<0>(tmem + 128 * t + c0, da + (uint64_t)((t * 2 * DS_ATOM + ks * 2048) >> 4),
                                db + (uint64_t)((c0 / 64 * DS_ATOM + ks * 2048) >> 4), id | ((uint32_t)(cols / 8) << 17), acc);
                    };
                    // the first 64 columns of a unit's first stage come last: the sums of the magnitudes of the
                    // unit before are read from there meanwhile
                    const int skip = q == 0 ? 64 : 0;
#pragma unroll
                    for (int ks = 0; ks < DS_KS / 16; ++ks) {
#pragma unroll
                        for (int t = 0; t < C::TILES; ++t) {
                            const int c0 = t == 0 ? skip : 0, n = C::COLS - 128 * t - c0;
                            const uint32_t acc = (in_group > 0 || ks > 0 || t > 0) ? 1u : 0u;
                            tile(t, ks, c0, n < 256 ? n : 256, acc);
                            if (n > 256) tile(t, ks, c0 + 256, n - 256, acc);
                        }
                    }
                    if (q == 0) {
                        if (un > 0 && !mbar_wait(smem_u32(&mag_drained_bar), (un - 1) & 1u, &abort_sh)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int ks = 0; ks < DS_KS / 16; ++ks) tile(0, ks, 0, 64, ks > 0 ? 1u : 0u);
                    }
                    umma_commit(smem_u32(&empty_bar[s]));
                    if (in_group == C::GROUP - 1 || q == n_st - 1) {
                        umma_commit(smem_u32(&ready_bar));
                        ++grp;
                    }
                }
                // the products of the magnitudes (the rows of A from NPAD on are not written, their sums not read)
                const uint32_t s = st % C::STAGES;
                if (ok && (!mbar_wait(smem_u32(&drained_bar), (grp - 1) & 1u, &abort_sh) ||
                           !mbar_wait(smem_u32(&full_bar[s]), (st / C::STAGES) & 1u, &abort_sh)))
                    ok = false;
                if (ok) {
                    fence_copies();
                    tc_fence_after();
                    const uint64_t da = desc_mn_sw128(ring + s * 2 * C::SIDE), db = desc_mn_sw128(ring + s * 2 * C::SIDE + C::SIDE);
#pragma unroll
                    for (int k = 0; k < DS_SAMPLE / 16; ++k)
                        umma<0>(tmem, da + (uint64_t)((k * 2048) >> 4), db + (uint64_t)((k * 2048) >> 4),
                                idesc0 | ((uint32_t)(NPAD / 8) << 17), k > 0 ? 1u : 0u);
                    umma_commit(smem_u32(&empty_bar[s]));
                    ++st;
                }
                if (ok) umma_commit(smem_u32(&mag_ready_bar));
            }
            if (!ok) {
                abort_sh = 1;
                atomicExch(status, XRH_ERR_TIMEOUT);
            }
            umma_commit(smem_u32(&done_bar));
            mbar_wait(smem_u32(&done_bar), 0u, nullptr);
        }
    } else if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::IO_REGS));
        // -------------------------------------------------------------------- gathers --
        // warps 8, 9 the bra side, 10, 11 the ket side; a lane per 16-byte chunk of a row
        const int pw = warp - 8, side = pw >> 1;
        uint32_t st = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            const xrh_dens_sliced_unit U = units[u];
            const xrh_dens_sliced_task& T = tasks[U.task];
            const int32_t* list = (side ? T.Q : T.P) + U.c0;
            const int blk = side ? U.jblk : U.iblk;
            const uint8_t* rows = reinterpret_cast<const uint8_t*>(side ? T.digk : T.digb) +
                                  (int64_t)blk * (side ? T.conf_k : T.conf_b) * (NS * NPAD * 2);
            const int s_pos = stages_of(U.n_pos), n_st = s_pos + stages_of(U.count - U.n_pos);
            int sample[DS_SAMPLE / 32];
#pragma unroll
            for (int i = 0; i < DS_SAMPLE / 32; ++i) {
                const int c = sampled(i * 32 + lane, U.count);
                sample[i] = c < U.count ? __ldg(list + c) : -1;
            }
            for (int q = 0; q < n_st; ++q, ++st) {
                const uint32_t s = st % C::STAGES;
                const int c = (q < s_pos ? q * DS_KS : U.n_pos + (q - s_pos) * DS_KS) + lane;
                const int mine = c < (q < s_pos ? U.n_pos : U.count) ? __ldg(list + c) : -1;
                if (st >= C::STAGES) {
                    const bool free = mbar_wait(smem_u32(&empty_bar[s]), (st / C::STAGES - 1) & 1u, &abort_sh);
                    if (!__all_sync(0xffffffffu, free)) {
                        ok = false;
                        break;
                    }
                }
                const uint32_t base = ring + s * 2 * C::SIDE + side * C::SIDE;
#pragma unroll 8
                for (int i = 0; i < NPAD / 2; ++i) {
                    const int item = i * 64 + (pw & 1) * 32 + lane;
                    const int cc = item / NPAD, chunk = item % NPAD;           // NPAD 16-byte chunks per row
                    const int row = __shfl_sync(0xffffffffu, mine, cc);
                    const uint32_t dst = base + (uint32_t)(chunk >> 3) * DS_ATOM + (uint32_t)(cc >> 3) * 1024u +
                                         (uint32_t)(cc & 7) * 128u + (uint32_t)(((chunk & 7) ^ (cc & 7)) << 4);
                    cp_async16_or_zero(dst, rows + (int64_t)(row < 0 ? 0 : row) * (NS * NPAD * 2) + chunk * 16, row >= 0);
                }
                cp_async_arrive(smem_u32(&full_bar[s]));
            }
            // the magnitudes of the sample, 128 bytes a coupling of which NPAD / 8 chunks are written
            if (ok) {
                constexpr int CH = NPAD / 8;
                const uint32_t s = st % C::STAGES;
                const uint8_t* mags = magnitudes<NPAD>(T, side) + (int64_t)blk * (side ? T.conf_k : T.conf_b) * (NPAD * 2);
                if (st >= C::STAGES) {
                    const bool free = mbar_wait(smem_u32(&empty_bar[s]), (st / C::STAGES - 1) & 1u, &abort_sh);
                    if (!__all_sync(0xffffffffu, free)) {
                        ok = false;
                        break;
                    }
                }
                ++st;
                const uint32_t base = ring + s * 2 * C::SIDE + side * C::SIDE;
#pragma unroll
                for (int i = 0; i < DS_SAMPLE * CH / 64; ++i) {
                    const int item = i * 64 + (pw & 1) * 32 + lane, cc = item / CH, chunk = item % CH;
                    int row = __shfl_sync(0xffffffffu, sample[0], cc & 31);
#pragma unroll
                    for (int k = 1; k < DS_SAMPLE / 32; ++k) {
                        const int x = __shfl_sync(0xffffffffu, sample[k], cc & 31);
                        if (cc >> 5 == k) row = x;
                    }
                    const uint32_t dst = base + (uint32_t)(cc >> 3) * 1024u + (uint32_t)(cc & 7) * 128u + (uint32_t)((chunk ^ (cc & 7)) << 4);
                    cp_async16_or_zero(dst, mags + (int64_t)(row < 0 ? 0 : row) * (NPAD * 2) + chunk * 16, row >= 0);
                }
                cp_async_arrive(smem_u32(&full_bar[s]));
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        if (!ok) {
            abort_sh = 1;
            if (lane == 0) atomicExch(status, XRH_ERR_TIMEOUT);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::EPI_REGS));
        // ------------------------------------------------------------------- epilogue --
        const int quarter = warp & 3, part = warp >> 2;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int row = quarter * 32 + lane;
        const int g = row / NPAD;                      // lane group: weight = column block + g
        uint32_t grp = 0, un = 0;
        bool failed = false;
        for (int64_t u = blockIdx.x; u < n_units && !failed; u += gridDim.x, ++un) {
            const int np = units[u].n_pos, count = units[u].count;
            const int n_st = stages_of(np) + stages_of(count - np);
            const bool partial = count > DS_SAMPLE;
            if (partial) {
                // s_nz[row]: columns with a product that is not zero.  The determinants' nonzero states come as
                // masks, few different pairs of them in an index (spin and spatial symmetry)
                const xrh_dens_sliced_unit U = units[u];
                const xrh_dens_sliced_task& T = tasks[U.task];
                const uint64_t *nb_ = nonzero<NPAD>(T, 0) + (int64_t)U.iblk * T.conf_b, *nk_ = nonzero<NPAD>(T, 1) + (int64_t)U.jblk * T.conf_k;
                if (tid < 64) s_nz[tid] = 0ull;
                epi_bar();
                uint64_t done_b = 0ull, done_k = 0ull;
                for (int c = tid; c - lane < count; c += DS_EPI) {
                    const uint64_t b = c < count ? __ldg(nb_ + __ldg(T.P + U.c0 + c)) : 0ull, k = c < count ? __ldg(nk_ + __ldg(T.Q + U.c0 + c)) : 0ull;
                    uint32_t todo = __ballot_sync(0xffffffffu, b != 0ull && k != 0ull && !(b == done_b && k == done_k));
                    while (todo) {
                        const int src = __ffs((int)todo) - 1;
                        done_b = __shfl_sync(0xffffffffu, b, src);
                        done_k = __shfl_sync(0xffffffffu, k, src);
#pragma unroll
                        for (int r = lane; r < 64; r += 32)
                            if ((done_b >> r) & 1ull) atomicOr(&s_nz[r], (unsigned long long)done_k);
                        todo &= ~__ballot_sync(0xffffffffu, b == done_b && k == done_k);
                    }
                }
            }
            Sum96 sum[C::CW];
#pragma unroll
            for (int j = 0; j < C::CW; ++j) sum[j] = Sum96{0u, 0u, 0u};
            for (int q = 0; q < n_st; q += C::GROUP, ++grp) {
                if (!failed && !mbar_wait(smem_u32(&ready_bar), grp & 1u, &abort_sh)) {
                    failed = true;
                    abort_sh = 1;
                }
                if (failed) break;
                tc_fence_after();
#pragma unroll 1
                for (int b = 0; b < NS; ++b) {
                    constexpr int CH = C::CW < 16 ? C::CW : 16;
                    const int w = b + g;               // above 7: not needed
#pragma unroll
                    for (int h = 0; h < C::CW; h += CH) {
                        float v[CH];
                        tmem_ld<CH>(tmem + lane_base + (uint32_t)(b * NPAD + part * C::CW + h), v);
                        if (w < NS) add_weight<CH>(sum + h, v, w);
                        __syncwarp();                  // (w differs within a warp for NPAD = 16)
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&drained_bar));
            }
            uint32_t low = 0u;                         // bit j: column j of this row may need FP64 arithmetic
            if (!failed && !mbar_wait(smem_u32(&mag_ready_bar), un & 1u, &abort_sh)) {
                failed = true;
                abort_sh = 1;
            }
            if (!failed) {
                constexpr int CH = 8;                  // (16 spill)
                tc_fence_after();
#pragma unroll 1
                for (int h = 0; h < C::CW && quarter * 32 < NPAD; h += CH) {
                    float v[CH];
                    tmem_ld<CH>(tmem + lane_base + (uint32_t)(part * C::CW + h), v);
#pragma unroll
                    for (int j = 0; j < CH; ++j) low |= ((partial ? v[j] < LOW_SUM : low_sum(v[j])) ? 1u << j : 0u) << h;
                }
                const xrh_dens_sliced_task& T = tasks[units[u].task];
                const int cols = T.nk - units[u].jblk * 64 - part * C::CW;
                if (row >= NPAD || units[u].iblk * 64 + row >= T.nb || cols <= 0) low = 0u;
                else if (cols < 32) low &= (1u << cols) - 1u;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&mag_drained_bar));
            }
            if (epi_bar_or(failed)) {                  // (also: s_eb, s_ek of the unit before are read)
                failed = true;
                abort_sh = 1;
                if (tid == 0) atomicExch(status, XRH_ERR_TIMEOUT);
                break;
            }
            const xrh_dens_sliced_unit U = units[u];
            const xrh_dens_sliced_task& T = tasks[U.task];
            const int i0 = U.iblk * 64, j0 = U.jblk * 64;
            if (tid < 64) s_eb[tid] = i0 + tid < T.nb ? T.eb[i0 + tid] : 0u;
            else if (tid < 128) s_ek[tid - 64] = j0 + tid - 64 < T.nk ? T.ek[j0 + tid - 64] : 0u;
            if (tid == 0) s_count = 0;
            if (partial && row < NPAD) low &= (uint32_t)(s_nz[row] >> (part * C::CW));
            epi_bar();
            const bool any_odd = epi_bar_or(low != 0u || (tid < 64 && ((s_eb[tid] >> 20) >= 2047u || (s_ek[tid] >> 20) >= 2047u))) != 0;
            // 4 columns of each part at a time: the lane groups of an element are added, converted, stored
#pragma unroll 1
            for (int p = 0; p < C::CW / 4; ++p) {
#pragma unroll
                for (int v = 0; v < C::CW / 4; ++v) {
                    if (v != p) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        s_raw[row][part * 4 + j] = make_uint4(sum[4 * v + j].w0, sum[4 * v + j].w1, sum[4 * v + j].w2, 0u);
                }
                epi_bar();
#pragma unroll
                for (int e = 0; e < (NPAD * 8 + DS_EPI - 1) / DS_EPI; ++e) {
                    const int item = e * DS_EPI + tid, slot = item & 7, I = item >> 3;
                    const int J = (slot >> 2) * C::CW + 4 * p + (slot & 3);
                    if (I >= NPAD || i0 + I >= T.nb || j0 + J >= T.nk) continue;
                    Sum96 t[1] = {Sum96{0u, 0u, 0u}};
#pragma unroll
                    for (int k = 0; k < C::G; ++k) {
                        const uint4 r = s_raw[k * NPAD + I][slot];
                        add96(t[0], r.x, r.y, r.z);
                    }
                    const int te[1] = {exp_of(s_eb[I]) + exp_of(s_ek[J])};
                    double tv[1];
                    sliced_to_doubles<1>(t, te, tv);
                    T.rhoT[((int64_t)U.idx * T.nb + i0 + I) * T.nk + j0 + J] = tv[0];
                }
                __syncwarp();
                epi_bar();
            }
            if (any_odd) {
                // sums the digits are too coarse for, states with an infinity or a NaN: the couplings in FP64
                // (in place of what has been stored), listed first, so that all threads share them
                uint16_t* odd = reinterpret_cast<uint16_t*>(s_raw);
                // the couplings' determinants staged behind the list, so that only the coefficients are waited for;
                // behind those the marked columns of a row and the tiles that begin at it
                constexpr int CH = 1024;
                int *s_p = reinterpret_cast<int*>(odd + 4096), *s_q = s_p + CH;
                uint32_t* s_m = reinterpret_cast<uint32_t*>(s_q + CH);
                int* s_n = reinterpret_cast<int*>(s_m + 2 * NPAD);
                static_assert(sizeof(s_raw) >= 4096 * 2 + 2 * CH * 4 + 3 * NPAD * 4, "list, couplings and masks share the buffer of the sums");
                if (row < NPAD) {
                    const bool bad = (s_eb[row] >> 20) >= 2047u;
#pragma unroll 1
                    for (int j = 0; j < C::CW; ++j) {
                        const int J = part * C::CW + j;
                        if (i0 + row < T.nb && j0 + J < T.nk && (bad || (s_ek[J] >> 20) >= 2047u)) low |= 1u << j;
                    }
                    s_m[2 * row + part] = low;
                    int at = atomicAdd(&s_count, __popc(low));
                    for (; low; low &= low - 1u) odd[at++] = (uint16_t)(row * 64 + part * C::CW + __ffs((int)low) - 1);
                }
                epi_bar();
                auto marked = [&](int r) { return (uint64_t)s_m[2 * r] | ((uint64_t)s_m[2 * r + 1] << C::CW); };
                if (tid < NPAD) {
                    const uint64_t m = marked(tid);
                    int rank = 0;
                    for (int r = 0; r < tid; ++r) rank += marked(r) == m;
                    s_n[tid] = rank % 4 == 0 ? (__popcll(m) + 1) / 2 : 0;
                }
                epi_bar();
                const int32_t *P = T.P + U.c0, *Q = T.Q + U.c0;
                const int n_odd = s_count;
                auto stage = [&](int c0, int n) {
                    epi_bar();
                    for (int i = tid; i < n; i += DS_EPI) {
                        s_p[i] = __ldg(P + c0 + i);
                        s_q[i] = __ldg(Q + c0 + i);
                    }
                    epi_bar();
                };
                const int rows = T.nb - i0 < NPAD ? T.nb - i0 : NPAD, cols = T.nk - j0 < NPAD ? T.nk - j0 : NPAD;
                int grouped = 0;
                for (int r = 0; r < NPAD; ++r) grouped += s_n[r];
                const int tk = (cols + 1) / 2, all = (rows + 3) / 4 * tk;
                const bool whole = grouped > all;
                const int tiles = whole ? all : grouped;
                if (2 * 8 * tiles <= 3 * n_odd) {
                    // tiles of 4 x 2 elements, a group of lanes each: 6 loads for 8 FMAs.  Four rows with the same marked
                    // columns (a symmetry marks whole classes of states) and two of these columns, or, where the rows
                    // differ too much, all of the block.  Where they are mostly filled: an element by itself
                    // costs 1.5 times one of a tile.  Evolved states of two Sz classes, all indices of two
                    // fragments, ms, by elements / whole blocks / tiles of this kind: 28 spin orbitals, 60 states - / 290 /
                    // 167, 40 - / 141 / 79, 30 52.2 / - / 40.3; 24, 21 states (tiles filled to 0.8) 11.3 / - /
                    // 10.6, 16 6.2 / - / 4.8; 18, 10 states (tiles filled to 0.5) 0.61 / - / 0.75
                    const int lanes = lanes_per_sum(tiles, DS_EPI, count), sub = tid % lanes;
#pragma unroll 1
                    for (int t0 = 0; t0 < tiles; t0 += DS_EPI / lanes) {
                        const int t = t0 + tid / lanes;
                        int I[4], J[2], n_r = 0, n_c = 0;
#pragma unroll
                        for (int r = 0; r < 4; ++r) I[r] = 0;
                        J[0] = J[1] = 0;
                        if (t < tiles && whole) {
                            const int a = t / tk * 4, b = t % tk * 2;
                            n_r = rows - a < 4 ? rows - a : 4;
                            n_c = cols - b < 2 ? cols - b : 2;
#pragma unroll
                            for (int r = 0; r < 4; ++r) I[r] = r < n_r ? a + r : a;
                            J[0] = b;
                            J[1] = n_c > 1 ? b + 1 : b;
                        } else if (t < tiles) {
                            int r0 = 0, c = t;
                            for (; c >= s_n[r0]; ++r0) c -= s_n[r0];
                            const uint64_t m = marked(r0);
                            uint64_t left = m;
                            for (int k = 0; k < 2 * c; ++k) left &= left - 1ull;
                            J[0] = J[1] = __ffsll((long long)left) - 1;
                            left &= left - 1ull;
                            n_c = left ? 2 : 1;
                            if (left) J[1] = __ffsll((long long)left) - 1;
                            I[0] = I[1] = I[2] = I[3] = r0;
                            n_r = 1;
                            for (int r = r0 + 1; r < NPAD && n_r < 4; ++r) {
                                if (marked(r) != m) continue;
#pragma unroll
                                for (int k = 1; k < 4; ++k)
                                    if (k == n_r) I[k] = r;
                                ++n_r;
                            }
                        }
                        const double *zb = T.zbT + i0, *zk = T.zkT + j0;
                        double x[4][2];
#pragma unroll
                        for (int r = 0; r < 4; ++r) x[r][0] = x[r][1] = 0.0;
#pragma unroll 1
                        for (int c0 = 0; c0 < count; c0 += CH) {
                            const int n = count - c0 < CH ? count - c0 : CH;
                            if (t0 == 0 || count > CH) stage(c0, n);
                            if (t >= tiles) continue;
#pragma unroll 4
                            for (int c = sub; c < n; c += lanes) {
                                const double *p = zb + (int64_t)s_p[c] * T.nb, *q = zk + (int64_t)s_q[c] * T.nk;
                                const double k0 = __ldg(q + J[0]), k1 = __ldg(q + J[1]);
                                const bool neg = c0 + c >= np;
#pragma unroll
                                for (int r = 0; r < 4; ++r) {
                                    const double a = neg ? -__ldg(p + I[r]) : __ldg(p + I[r]);
                                    x[r][0] = fma(a, k0, x[r][0]);
                                    x[r][1] = fma(a, k1, x[r][1]);
                                }
                            }
                        }
#pragma unroll
                        for (int r = 0; r < 4; ++r)
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const double y = sum_lanes(x[r][k], lanes);
                                if (sub == 0 && r < n_r && k < n_c)
                                    T.rhoT[((int64_t)U.idx * T.nb + i0 + I[r]) * T.nk + j0 + J[k]] = y;
                            }
                    }
                } else {
                    const int lanes = lanes_per_sum(n_odd, DS_EPI, count), sub = tid % lanes;
#pragma unroll 1
                    for (int e0 = 0; e0 < n_odd; e0 += DS_EPI / lanes) {
                        const int e = e0 + tid / lanes, at = odd[e < n_odd ? e : 0];
                        const int I = i0 + (at >> 6), J = j0 + (at & 63);
                        const double *zb = T.zbT + I, *zk = T.zkT + J;
                        double x = 0.0;
#pragma unroll 1
                        for (int c0 = 0; c0 < count; c0 += CH) {
                            const int n = count - c0 < CH ? count - c0 : CH;
                            if (e0 == 0 || count > CH) stage(c0, n);
                            if (e < n_odd) {
#pragma unroll 8
                                for (int c = sub; c < n; c += lanes) {
                                    const double a = __ldg(zb + (int64_t)s_p[c] * T.nb);
                                    x = fma(c0 + c < np ? a : -a, __ldg(zk + (int64_t)s_q[c] * T.nk), x);
                                }
                            }
                        }
                        x = sum_lanes(x, lanes);
                        if (e < n_odd && sub == 0) T.rhoT[((int64_t)U.idx * T.nb + I) * T.nk + J] = x;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
}

// ---- digits of the state coefficients ------------------------------------------------------
constexpr int CD_ROWS = 64;                            // determinants per CTA

__device__ __forceinline__ const xrh_coeff_digit_task& find_coeff(const xrh_coeff_digit_task* __restrict__ tasks, int n_tasks) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].cta_begin <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    return tasks[lo];
}

// exps[state] = high word of the largest |coefficient| (zero on entry)
__global__ void __launch_bounds__(256) coeff_max_kernel(const xrh_coeff_digit_task* __restrict__ tasks, int n_tasks) {
    const xrh_coeff_digit_task& T = find_coeff(tasks, n_tasks);
    const int64_t r0 = ((int64_t)blockIdx.x - T.cta_begin) * CD_ROWS;
    const int rows = T.n_conf - r0 < CD_ROWS ? (int)(T.n_conf - r0) : CD_ROWS;
    const int lanes = T.n <= 8 ? 8 : (T.n <= 16 ? 16 : (T.n <= 32 ? 32 : 64));   // threads along the states
    for (int s0 = 0; s0 < T.n; s0 += lanes) {
        const int s = s0 + threadIdx.x % lanes;
        uint32_t m = 0;
        if (s < T.n)
            for (int r = threadIdx.x / lanes; r < rows; r += 256 / lanes) m = max(m, abs_hi(__ldg(T.zT + (r0 + r) * T.n + s)));
        if (m) atomicMax(T.exps + s, m);
    }
}

// rows [block of 64 states][determinant][slice][NPAD]: a thread per (determinant, 8 states)
__global__ void __launch_bounds__(256) coeff_digits_kernel(const xrh_coeff_digit_task* __restrict__ tasks, int n_tasks) {
    const xrh_coeff_digit_task& T = find_coeff(tasks, n_tasks);
    const int64_t r0 = ((int64_t)blockIdx.x - T.cta_begin) * CD_ROWS;
    const int rows = T.n_conf - r0 < CD_ROWS ? (int)(T.n_conf - r0) : CD_ROWS;
    const int blocks = (T.n + T.npad - 1) / T.npad, oct = T.npad / 8, per = blocks * oct;
    for (int x = threadIdx.x; x < rows * per; x += 256) {
        const int r = x / per, o = x - r * per, blk = o / oct, s0 = blk * T.npad + (o - blk * oct) * 8;
        const double* z = T.zT + (r0 + r) * T.n;
        uint64_t v[8];
        uint32_t m[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int s = s0 + k;
            v[k] = 0x0080808080808080ull;
            m[k] = 0u;
            if (s < T.n) {
                const uint32_t w = T.exps[s] >> 20;
                const int E = w < 1u ? 1 : (int)w;
                if (w < 2047u) {
                    const double x = __ldg(z + s);
                    v[k] = fixed62(x, E);
                    m[k] = magnitude(x, E);
                }
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(T.digits) +
                                              ((int64_t)blk * T.n_conf + r0 + r) * (T.slices * T.npad)) + (o - blk * oct);
#pragma unroll
        for (int t = 0; t < NS; ++t) {
            if (t >= T.slices) break;
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = __byte_perm(digit_float(v[2 * k], t), digit_float(v[2 * k + 1], t), 0x7632);
            dst[t * oct] = make_uint4(q[0], q[1], q[2], q[3]);
        }
        if (T.slices == NS)                            // behind the digits of all blocks
            *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(T.digits) +
                                      ((int64_t)blocks * T.n_conf * NS + (int64_t)blk * T.n_conf + r0 + r) * T.npad + (o - blk * oct) * 8) =
                make_uint4(m[0] | (m[1] << 16), m[2] | (m[3] << 16), m[4] | (m[5] << 16), m[6] | (m[7] << 16));
        if (T.slices == NS) {
            uint8_t bits = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) bits |= m[k] ? 1u << k : 0u;
            uint8_t* nz = reinterpret_cast<uint8_t*>(reinterpret_cast<uint16_t*>(T.digits) + (int64_t)blocks * T.n_conf * (NS + 1) * T.npad) +
                          ((int64_t)blk * T.n_conf + r0 + r) * 8;
            nz[o - blk * oct] = bits;                  // (little-endian: state k is bit k)
            if (oct < 8 && o == 0)
                for (int k = oct; k < 8; ++k) nz[k] = 0;
        }
    }
}

template <int NPAD>
int launch(const xrh_dens_sliced_task* tasks, const xrh_dens_sliced_unit* units, int64_t n_units, int32_t* status,
           cudaStream_t s) {
    using C = Cfg<NPAD>;
    int dev = 0, n_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = (size_t)C::STAGES * 2 * C::SIDE + 1024;
    cudaFuncSetAttribute(density_sliced_kernel<NPAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int64_t grid = n_units < (int64_t)n_sm * C::CTAS ? n_units : (int64_t)n_sm * C::CTAS;
    density_sliced_kernel<NPAD><<<(unsigned)grid, DS_THREADS, smem, s>>>(tasks, units, n_units, status);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

}  // namespace

extern "C" int64_t xrh_coeff_digit_ctas(int64_t n_conf) { return n_conf > 0 ? (n_conf + CD_ROWS - 1) / CD_ROWS : 0; }

extern "C" int xrh_coeff_digits(const xrh_coeff_digit_task* tasks_dev, int n_tasks, int64_t total_ctas, void* stream) {
    if (n_tasks < 0 || total_ctas < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_ctas == 0) return XRH_OK;
    if (!tasks_dev) return XRH_ERR_ARG;
    if (total_ctas > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    coeff_max_kernel<<<(unsigned)total_ctas, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
    XRH_CHECK_LAUNCH();
    coeff_digits_kernel<<<(unsigned)total_ctas, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

extern "C" int xrh_density_sliced_grouped(const xrh_dens_sliced_task* tasks_dev, int n_tasks,
                                          const xrh_dens_sliced_unit* units_dev, int64_t n_units, int npad,
                                          int32_t* status_dev, void* stream) {
    if (n_tasks < 0 || n_units < 0 || (npad != 16 && npad != 32 && npad != 64)) return XRH_ERR_ARG;
    if (n_tasks == 0 || n_units == 0) return XRH_OK;
    if (!tasks_dev || !units_dev || !status_dev) return XRH_ERR_ARG;
    if (npad == 16) return launch<16>(tasks_dev, units_dev, n_units, status_dev, (cudaStream_t)stream);
    if (npad == 32) return launch<32>(tasks_dev, units_dev, n_units, status_dev, (cudaStream_t)stream);
    return launch<64>(tasks_dev, units_dev, n_units, status_dev, (cudaStream_t)stream);
}
