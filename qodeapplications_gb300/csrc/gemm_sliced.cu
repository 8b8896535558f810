// FP64 grouped GEMM with exact digit products on the 5th-generation tensor cores (sm_103a).
//
// GB300 runs FP64 at about 2 DFMA/clk/SM (1.1 TFLOP/s), a two-thousandth of its BF16 tensor rate, so
// the FP64 contractions are rebuilt from integer products (the error-free slicing of Ozaki, Ogita,
// Oishi and Rump, Numer. Algorithms 59, 95 (2012)): a row x of an operand with |x| < 2^e is the
// integer V = round(x 2^(62 - e)), written in balanced base-256 digits V = sum_t d_t 256^(7 - t),
// |d_t| <= 128, |d_0| <= 65, each digit exact in BF16.  With S_w = sum_(i+j=w) sum_k d_i(a_k) d_j(b_k),
//     sum_k a_k b_k = 2^(ea + eb - 68) sum_(w<8) S_w 256^(7 - w)   (+ what the 36 digit pairs leave out)
// |d_i d_j| <= 2^14 and a weight has at most 8 pairs, so 128 K elements keep every FP32 accumulator at or
// below 2^24, where integers are exact: the order and the rounding of the tensor core's additions do
// not matter.  The eight sums of such a group go into one 96-bit integer per output element, rounded
// to FP64 once per segment.
//
// Error: an element within 2^-9 of its row's largest is represented exactly, a smaller one to 2^-63
// of 2^e, and the pairs with i + j >= 8 left out are below 2^-59.1 2^(ea + eb) a product: K 1.003 2^-59 2^(ea + eb)
// in all, K 2^-62 as a rule.  That is relative to the largest elements of the row and the column, an
// FP64 sum's K 2^-53 sum |a||b| to the products themselves.  So a ninth image holds the magnitudes of
// the elements as BF16 numbers, one more MMA a K step gives sum |a||b| from below, and the elements where
// the first bound could exceed the second (low_sum: rows that span many orders of magnitude, whose
// large elements meet zeros or small ones) are formed by FP64 FMAs from the operands, as those of
// rows with infinities and NaN are (odd_products_kernel).  Rows of one size have none of them; the
// magnitudes cost 3 % at 3 600 x 21 952 x 28, the spin blocks and near identities of an integral
// transformation of 28 spin orbitals 15 % (2.8 -> 3.2 ms; CUDA cores 15.4).
//
// What bounds it: 36 pairs of BF16 MMAs are 2 304 cycles of the tensor pipe per 128 x 64 x 32 stage; the
// integer collection of a group (8 x 8 192 conversions) and the flush of a tile (about 25 000 cycles)
// overlap with it in part.  Measured, whole launches with their digits: M = N = 3 600, K = 784 0.82 ms, 25 TFLOP/s
// of FP64 products (CUDA cores: 20.8 ms, 1.0); 3 600 x 784 x 784 0.26 ms against 4.64; one tile of 128 K 39 us
// against 158 us.
//
// Per CTA (persistent over 128 x BN tiles, BN = 64, or 32 for N <= 32), 12 warps:
//   * warp 8: bulk copies of all eight slices of A and B for 32 K (96 KB: two stages), at the end of a
//     segment of the magnitudes of 256 K; the digits lie in global memory as the swizzled shared-memory
//     image of a stage, so a stage is two contiguous copies;
//   * warp 9: the tcgen05.mma of a stage into eight TMEM accumulators (weight w at column BN w; see
//     stage_mmas), handed to the epilogue in pairs of weights, the next group starting behind it; the
//     products of the magnitudes on the first pair's accumulators once they are drained;
//   * warps 0-7: tcgen05.ld of two weights (32 columns a warp), integer accumulation, release; at the
//     end of a segment conversion by integer operations (the FP64 pipe is needed only for alpha
//     and for additions) and the store, scatter or atomic epilogue through shared memory.
// Every mbarrier wait is bounded; on timeout *status is set, all roles leave, copies and MMAs in
// flight are waited for (bounded), TMEM is freed.
#include "sliced_common.cuh"
#include "tc_common.cuh"

namespace {
using namespace xrh_tc;
using namespace xrh_sliced;

constexpr int SL_BM = 128;
constexpr int SL_KS = 32;                              // K elements per stage (64-byte rows)
constexpr int SL_GROUP = 4;                            // stages per exact accumulation group
constexpr int SL_STAGES = 2;
constexpr int SL_EPI_WARPS = 8;
constexpr int SL_EPI_THREADS = SL_EPI_WARPS * 32;
constexpr int SL_THREADS = SL_EPI_THREADS + 128;       // + a warpgroup: loads, MMA, two idle warps
// registers: 384 threads x 168 at launch = 64512 = 256 x 208 (epilogue) + 128 x 88; 16 epilogue
// warps of 104 registers spill and are 20 % slower
constexpr int SL_EPI_REGS = 208, SL_IO_REGS = 88;
static_assert(SL_EPI_THREADS * SL_EPI_REGS + 128 * SL_IO_REGS <= SL_THREADS * 168, "register split exceeds the launch");
constexpr int SL_CW = 64 / (SL_EPI_WARPS / 4);         // columns per epilogue warp
constexpr int SL_SUB = SL_CW / 8;                      // of them per pass of a flush (8 passes, 8 slots a row)
constexpr int SL_NEL = 1024 / SL_EPI_THREADS;          // elements a thread converts per pass
constexpr int NP = NS / 2;                             // weight pairs: the unit handed to the epilogue
constexpr uint32_t SL_A_SLICE = SL_BM * 64;            // bytes of one slice of a stage
constexpr uint32_t SL_A_BYTES = NS * SL_A_SLICE;
constexpr uint32_t SL_B_BYTES = NS * 64 * 64;
constexpr uint32_t SL_STAGE_BYTES = SL_A_BYTES + SL_B_BYTES;
constexpr int SL_RUN_GROUPS = 4096;                    // groups collected in 96 bits before a flush (< 2^93)
static_assert(NS == 8, "digit weights and shifts below are written for eight slices");
static_assert((long long)SL_GROUP * SL_KS * NS * (1 << 14) <= (1 << 24), "a group must stay exact in FP32");

__device__ __forceinline__ void epi_bar() { named_bar<1, SL_EPI_THREADS>(); }
__device__ __forceinline__ int epi_bar_or(int pred) { return named_bar_or<1, SL_EPI_THREADS>(pred); }

// A persistent CTA's tile: task, batch, output corner, N tile, range of K stages.
struct Tile {
    int task, m0, n0, BN;
    int sb, left;                 // first stage (over the concatenated segments) and their number
    int64_t batch;
};

__device__ __forceinline__ Tile tile_of(const xrh_gemm_task* __restrict__ tasks, int n_tasks,
                                        const xrh_sliced_segment* __restrict__ segs, int64_t tile) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    const xrh_gemm_task& T = tasks[lo];
    Tile r;
    r.task = lo;
    r.BN = T.N <= 32 ? 32 : 64;
    const int64_t tiles_m = (T.M + SL_BM - 1) / SL_BM, tiles_n = (T.N + r.BN - 1) / r.BN, mn = tiles_m * tiles_n;
    int64_t local = tile - T.tile_begin;
    r.batch = local / (mn * T.splitk);
    local -= r.batch * mn * T.splitk;
    const int64_t split = local / mn;
    local -= split * mn;
    // concurrent CTAs walk the N tiles of one M tile, or the M tiles of one N tile where those are
    // the fewer, so that the smaller operand is the one re-read (from L2)
    if (tiles_m < tiles_n) {
        r.m0 = (int)((local % tiles_m) * SL_BM);
        r.n0 = (int)((local / tiles_m) * r.BN);
    } else {
        r.m0 = (int)((local / tiles_n) * SL_BM);
        r.n0 = (int)((local % tiles_n) * r.BN);
    }
    int64_t total = 0;
    for (int64_t s = 0; s < T.seg_count; ++s) total += segs[T.seg_begin + s].stages;
    const int64_t per = (total + T.splitk - 1) / T.splitk;
    const int64_t sb = split * per, se = sb + per < total ? sb + per : total;
    r.sb = (int)sb;
    r.left = (int)(se > sb ? se - sb : 0);
    return r;
}

// What the epilogue needs of its tile, in shared memory: its registers hold 32 96-bit sums.
struct EpiTile {
    double* C;
    const xrh_sliced_segment* segs;
    uint32_t* odd;                // marks of the tile's runs
    int64_t ldc, batch;
    int M, N, m0, n0, mode, BN, sb, left, task;
};

// The stages of a tile as groups: at most SL_GROUP consecutive stages of one segment.  Every role
// walks the same sequence.
struct Groups {
    const xrh_sliced_segment* segs;
    int si, c, left;              // segment, next stage in it, stages left in the tile
    int g0;                       // first stage of the current run (stages flushed together)
    int run;                      // groups in the run so far
    int take;                     // stages of the current group
    bool flush;                   // the current group ends its run

    __device__ __forceinline__ Groups(const xrh_sliced_segment* s, int first, int stages)
        : segs(s), si(0), c(first), left(stages), g0(0), run(0), take(0), flush(true) {}
    __device__ __forceinline__ bool next() {
        c += take;
        left -= take;
        if (left <= 0) return false;
        while (c >= segs[si].stages) {
            c -= (int)segs[si].stages;
            ++si;
        }
        if (flush) {
            g0 = c;
            run = 0;
        }
        const int in_seg = (int)segs[si].stages - c;
        int n = in_seg < SL_GROUP ? in_seg : SL_GROUP;
        if (n > left) n = left;
        take = n;
        flush = n == in_seg || n == left || ++run == SL_RUN_GROUPS;
        return true;
    }
};

// The MMAs of one stage (two K steps of 16).  The B slices of a stage are consecutive rows and the
// accumulators consecutive columns (weight w at column BN w), so A_i x [B_j .. B_j+c] adds to the
// weights i+j .. i+j+c in one MMA of N = BN (c + 1): 12 MMAs a K step for BN = 64 (8 for 32) instead
// of 36 of N = 64, whose operand reads and dependent additions (about 110 cycles between two
// MMAs on one accumulator) would bound them: 8 300 cycles a stage against 2 304 of the tensor pipe.
// The first stage of a group goes weight pair by weight pair instead, each as soon as the epilogue
// has drained it from the group before; at the last stage a pair is handed over after its own
// last product.
template <int BN>
__device__ __forceinline__ bool stage_mmas(uint32_t tmem, uint64_t dA, uint64_t dB, bool first, bool last,
                                           uint32_t drained, bool wait_drained, uint32_t drained_parity,
                                           uint32_t ready, volatile int* abort_flag) {
    constexpr uint32_t id0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(SL_BM >> 4) << 24);
    constexpr uint64_t a_step = SL_A_SLICE >> 4, b_step = (uint64_t)(BN * 64) >> 4;
    auto mma = [&](int i, int j, int cnt, int ks, uint32_t acc) {       // A_i x [B_j .. B_j+cnt-1]
        umma<0>(tmem + (uint32_t)(BN * (i + j)), dA + i * a_step + 2 * ks, dB + j * b_step + 2 * ks,
                id0 | ((uint32_t)(BN * cnt / 8) << 17), acc);
    };
    if (first) {
#pragma unroll
        for (int p = 0; p < NS / 2; ++p) {
            if (wait_drained) {
                if (!mbar_wait(drained + 8u * p, drained_parity, abort_flag)) return false;
                tc_fence_after();
            }
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
                for (int i = 0; i <= 2 * p; ++i) mma(i, 2 * p - i, 2, ks, (ks || i) ? 1u : 0u);
                mma(2 * p + 1, 0, 1, ks, 1u);
            }
            if (last) umma_commit(ready + 8u * p);
        }
        return true;
    }
    constexpr int WIDE = 256 / BN;                 // slices of B in the widest MMA
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            mma(i, 0, NS - i < WIDE ? NS - i : WIDE, ks, 1u);
            if (NS - i > WIDE) mma(i, WIDE, NS - i - WIDE, ks, 1u);
            if (ks && last && (i & 1)) umma_commit(ready + 8u * (i >> 1));
        }
    }
    return true;
}

__global__ void __launch_bounds__(SL_THREADS, 1)
    gemm_sliced_kernel(const xrh_gemm_task* __restrict__ tasks, int n_tasks, int64_t total_tiles,
                       const xrh_sliced_segment* __restrict__ segs, const xrh_odd_range* __restrict__ odd_ranges,
                       uint32_t* __restrict__ odd_bits, uint32_t* __restrict__ odd_list, int32_t* status) {
    extern __shared__ unsigned char smem_raw[];
    uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[SL_STAGES], empty_bar[SL_STAGES];
    __shared__ __align__(8) uint64_t ready_bar[NP], drained_bar[NP];
    __shared__ __align__(8) uint64_t mag_ready_bar, mag_drained_bar;
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_sh;
    __shared__ uint4 s_raw[SL_BM][9];
    __shared__ int64_t s_roff[SL_BM], s_coff[64];      // element (m, n) lies at C[s_roff[m] + s_coff[n]]
    __shared__ double s_DA[SL_BM], s_DB[64];
    __shared__ uint32_t s_eA[SL_BM], s_eB[64];
    __shared__ uint32_t s_low[SL_EPI_WARPS / 4][SL_BM];
    __shared__ unsigned char s_diagA[SL_BM], s_diagB[64];
    __shared__ EpiTile s_t;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < SL_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int w = 0; w < NP; ++w) {
            mbar_init(smem_u32(&ready_bar[w]), 1);
            mbar_init(smem_u32(&drained_bar[w]), SL_EPI_WARPS);
        }
        mbar_init(smem_u32(&mag_ready_bar), 1);
        mbar_init(smem_u32(&mag_drained_bar), SL_EPI_WARPS);
        mbar_init(smem_u32(&done_bar), 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh;

    if (warp >= SL_EPI_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SL_IO_REGS));
        if (warp == SL_EPI_WARPS && lane == 0) {
            // -------------------------------------------------------------------- TMA loads --
            uint64_t g = 0;
            bool ok = true;
            for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const Tile I = tile_of(tasks, n_tasks, segs, tile);
                const uint32_t b_bytes = (uint32_t)NS * (uint32_t)I.BN * 64u;
                Groups G(segs + tasks[I.task].seg_begin, I.sb, I.left);
                while (ok && G.next()) {
                    const xrh_sliced_segment& S = G.segs[G.si];
                    const int64_t blk_a = I.batch * ((S.rA + SL_BM - 1) / SL_BM) + I.m0 / SL_BM;
                    const int64_t blk_b = I.batch * ((S.rB + I.BN - 1) / I.BN) + I.n0 / I.BN;
                    const uint32_t b_slice = (uint32_t)I.BN * 64u;
                    const uint8_t* pa = reinterpret_cast<const uint8_t*>(S.digA) + blk_a * S.stages * (int64_t)(SL_A_BYTES + SL_A_SLICE);
                    const uint8_t* pb = reinterpret_cast<const uint8_t*>(S.digB) + blk_b * S.stages * (int64_t)(b_bytes + b_slice);
                    // n slices of either operand into the next slot
                    auto load = [&](int64_t slice, int n) {
                        const int s = (int)(g % SL_STAGES);
                        if (g >= SL_STAGES &&
                            !mbar_wait(smem_u32(&empty_bar[s]), (uint32_t)(g / SL_STAGES - 1) & 1u, &abort_sh))
                            return false;
                        uint8_t* st = stages + (size_t)s * SL_STAGE_BYTES;
                        const uint32_t bar = smem_u32(&full_bar[s]);
                        mbar_expect_tx(bar, (uint32_t)n * (SL_A_SLICE + b_slice));
                        bulk_load(smem_u32(st), pa + slice * SL_A_SLICE, (uint32_t)n * SL_A_SLICE, bar);
                        bulk_load(smem_u32(st + SL_A_BYTES), pb + slice * b_slice, (uint32_t)n * b_slice, bar);
                        ++g;
                        return true;
                    };
                    for (int q = 0; q < G.take && ok; ++q) ok = load((int64_t)(G.c + q) * NS, NS);
                    if (G.flush)                                 // the magnitudes of the run, NS stages a slot
                        for (int q = G.g0; q < G.c + G.take && ok; q += NS)
                            ok = load(S.stages * NS + q, min(NS, G.c + G.take - q));
                }
            }
            if (!ok) {
                abort_sh = 1;
                atomicExch(status, XRH_ERR_TIMEOUT);
            }
            // every copy issued has landed before shared memory goes away
            for (uint64_t q = g > SL_STAGES ? g - SL_STAGES : 0; q < g; ++q)
                mbar_wait(smem_u32(&full_bar[q % SL_STAGES]), (uint32_t)(q / SL_STAGES) & 1u, nullptr);
        } else if (warp == SL_EPI_WARPS + 1 && lane == 0) {
            // -------------------------------------------------------------------------- MMA --
            uint64_t g = 0, grp = 0, runs = 0;
            bool behind_mag = false;                             // the group before ended its run
            int bn = 0;                                          // N tile of the previous group
            bool ok = true;
            for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const Tile I = tile_of(tasks, n_tasks, segs, tile);
                Groups G(segs + tasks[I.task].seg_begin, I.sb, I.left);
                for (; ok && G.next(); ++grp) {
                    for (int q = 0; q < G.take && ok; ++q, ++g) {
                        const int s = (int)(g % SL_STAGES);
                        if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(g / SL_STAGES) & 1u, &abort_sh)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_u32(stages + (size_t)s * SL_STAGE_BYTES);
                        const uint64_t dA = umma_desc_sw64(st), dB = umma_desc_sw64(st + SL_A_BYTES);
                        const bool wait_d = q == 0 && grp > 0, last = q == G.take - 1;
                        const uint32_t par = (uint32_t)(grp - 1) & 1u;
                        if (wait_d && I.BN != bn) {
                            // the accumulators of the two tile widths overlap: all must be drained
                            for (int w = 0; w < NP && ok; ++w)
                                ok = mbar_wait(smem_u32(&drained_bar[w]), par, &abort_sh);
                            if (!ok) break;
                        }
                        bn = I.BN;
                        if (q == 0 && behind_mag && !mbar_wait(smem_u32(&mag_drained_bar), (uint32_t)(runs - 1) & 1u, &abort_sh)) {
                            ok = false;
                            break;
                        }
                        ok = I.BN == 64
                                 ? stage_mmas<64>(tmem, dA, dB, q == 0, last, smem_u32(drained_bar), wait_d, par,
                                                  smem_u32(ready_bar), &abort_sh)
                                 : stage_mmas<32>(tmem, dA, dB, q == 0, last, smem_u32(drained_bar), wait_d, par,
                                                  smem_u32(ready_bar), &abort_sh);
                        umma_commit(smem_u32(&empty_bar[s]));
                    }
                    behind_mag = G.flush;
                    if (!ok || !G.flush) continue;
                    // the products of the magnitudes, on the accumulators of the first weight pair (a sum
                    // for either K step, so that two MMAs are in flight)
                    if (!mbar_wait(smem_u32(&drained_bar[0]), (uint32_t)grp & 1u, &abort_sh)) {
                        ok = false;
                        continue;
                    }
                    for (int q = G.g0; q < G.c + G.take; q += NS, ++g) {
                        const int s = (int)(g % SL_STAGES), n = min(NS, G.c + G.take - q);
                        if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(g / SL_STAGES) & 1u, &abort_sh)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_u32(stages + (size_t)s * SL_STAGE_BYTES);
                        const uint64_t dA = umma_desc_sw64(st), dB = umma_desc_sw64(st + SL_A_BYTES);
                        for (int j = 0; j < n; ++j)
#pragma unroll
                            for (int ks = 0; ks < 2; ++ks)
                                umma<0>(tmem + (uint32_t)(ks * I.BN), dA + (uint64_t)(j * (SL_A_SLICE >> 4) + 2 * ks),
                                        dB + (uint64_t)(j * ((I.BN * 64) >> 4) + 2 * ks), make_idesc(1u, SL_BM, (uint32_t)I.BN, false),
                                        q > G.g0 || j > 0 ? 1u : 0u);
                        umma_commit(smem_u32(&empty_bar[s]));
                    }
                    if (ok) umma_commit(smem_u32(&mag_ready_bar));
                    ++runs;
                }
            }
            if (!ok) {
                abort_sh = 1;
                atomicExch(status, XRH_ERR_TIMEOUT);
            }
            umma_commit(smem_u32(&done_bar));          // every MMA issued has completed
            mbar_wait(smem_u32(&done_bar), 0u, nullptr);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SL_EPI_REGS));
        // --------------------------------------------------------------------- epilogue --
        const int quarter = warp & 3, part = warp >> 2;          // TMEM lanes 32*quarter.., columns 16*part..
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int row = quarter * 32 + lane;
        uint64_t grp = 0;
        uint32_t runs = 0;
        bool failed = false;
        for (int64_t tile = blockIdx.x; tile < total_tiles && !failed; tile += gridDim.x) {
            if (tid == 0) {
                const Tile I = tile_of(tasks, n_tasks, segs, tile);
                const xrh_gemm_task& T = tasks[I.task];
                s_t.C = T.C + I.batch * T.sC;
                s_t.segs = segs + T.seg_begin;
                s_t.ldc = T.ldc;
                s_t.batch = I.batch;
                s_t.M = (int)T.M;
                s_t.N = (int)T.N;
                s_t.m0 = I.m0;
                s_t.n0 = I.n0;
                s_t.mode = (int)T.mode;
                s_t.BN = I.BN;
                s_t.sb = I.sb;
                s_t.left = I.left;
                s_t.task = I.task;
                s_t.odd = odd_bits + (odd_ranges[I.task].begin + (tile - T.tile_begin) * odd_ranges[I.task].runs) * (2 * SL_BM);
            }
            epi_bar();
            if (s_t.left == 0) {                                 // (uniform)
                epi_bar();                                       // read before the next tile's is written
                continue;
            }
            const int BN = s_t.BN;
            const bool mine = part * SL_CW < BN;
            {
                const xrh_gemm_task& T = tasks[s_t.task];
                const bool scatter = s_t.mode == 2;
                for (int j = tid; j < BN; j += SL_EPI_THREADS) {
                    const int64_t n = s_t.n0 + j;
                    const bool ok = scatter && n < s_t.N;
                    s_coff[j] = ok ? (int64_t)T.rowB[n] * s_t.ldc + T.colB[n] : n;
                    s_diagB[j] = ok ? T.diagB[n] : 0;
                    s_DB[j] = (ok && T.DB) ? T.DB[n] : 0.0;
                }
                for (int r = tid; r < SL_BM; r += SL_EPI_THREADS) {
                    const int64_t m = s_t.m0 + r;
                    const bool ok = scatter && m < s_t.M;
                    s_roff[r] = ok ? (int64_t)T.rowA[m] * s_t.ldc + T.colA[m] : m * s_t.ldc;
                    s_diagA[r] = ok ? T.diagA[m] : 0;
                    s_DA[r] = (ok && T.DA) ? T.DA[m] : 0.0;
                }
            }
            bool first = true;                                   // first flush of the tile
            bool tile_odd = false;                               // it has elements for odd_products_kernel
            int run = 0;
            Sum96 sum[SL_CW];
#pragma unroll
            for (int j = 0; j < SL_CW; ++j) sum[j] = Sum96{0u, 0u, 0u};
            Groups G(s_t.segs, s_t.sb, s_t.left);
            while (G.next()) {
                const uint32_t ph = (uint32_t)grp & 1u;
                ++grp;
                // a rolled loop over the weight pairs: the code of a group stays small (an unrolled one does
                // not stay in the instruction cache beside the flush)
#pragma unroll 1
                for (int p = 0; p < NP; ++p) {
                    if (!failed && !mbar_wait(smem_u32(&ready_bar[p]), ph, &abort_sh)) {
                        failed = true;
                        abort_sh = 1;
                    }
                    if (failed) break;
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < SL_CW; h += 16) {
                        float v[16], u[16];
                        if (mine)
                            tmem_ld16_pair(tmem + lane_base + (uint32_t)(2 * p * BN + part * SL_CW + h),
                                           tmem + lane_base + (uint32_t)((2 * p + 1) * BN + part * SL_CW + h), v, u);
                        if (h + 16 == SL_CW) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(smem_u32(&drained_bar[p]));
                        }
                        if (mine) {
                            add_weight<16>(sum + h, v, 2 * p);
                            add_weight<16>(sum + h, u, 2 * p + 1);
                        }
                    }
                }
                if (!G.flush) continue;
                uint32_t low = 0u;                               // bit j: column j needs FP64 arithmetic (s_low)
                if (!failed && !mbar_wait(smem_u32(&mag_ready_bar), runs & 1u, &abort_sh)) {
                    failed = true;
                    abort_sh = 1;
                }
                ++runs;
                if (!failed) {
                    tc_fence_after();
#pragma unroll 1
                    for (int h = 0; h < SL_CW && mine; h += 16) {
                        float v[16], u[16];
                        tmem_ld16_pair(tmem + lane_base + (uint32_t)(part * SL_CW + h),
                                       tmem + lane_base + (uint32_t)(BN + part * SL_CW + h), v, u);
#pragma unroll
                        for (int j = 0; j < 16; ++j) low |= (low_sum(v[j] + u[j]) ? 1u << j : 0u) << h;
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&mag_drained_bar));
                }
                // one decision of all epilogue warps per flush (also the barrier before s_eB is reused)
                if (epi_bar_or(failed)) {
                    failed = true;
                    abort_sh = 1;
                    if (tid == 0) atomicExch(status, XRH_ERR_TIMEOUT);
                    break;
                }
                const xrh_sliced_segment& S = G.segs[G.si];
                bool bad = false;                                // an infinity or a NaN
                if (tid < BN) {
                    const uint32_t wb = s_t.n0 + tid < s_t.N ? S.eB[s_t.batch * S.rB + s_t.n0 + tid] : 0u;
                    s_eB[tid] = wb;
                    bad = (wb >> 20) >= 2047u;
                }
                const uint32_t wa = s_t.m0 + row < s_t.M ? S.eA[s_t.batch * S.rA + s_t.m0 + row] : 0u;
                if (part == 0) s_eA[row] = wa;
                if (epi_bar_or(bad || (wa >> 20) >= 2047u) && s_t.m0 + row < s_t.M) {
#pragma unroll 1
                    for (int j = 0; j < SL_CW; ++j) {
                        const int jj = part * SL_CW + j;
                        if (jj < BN && s_t.n0 + jj < s_t.N && ((wa >> 20) >= 2047u || (s_eB[jj] >> 20) >= 2047u)) low |= 1u << j;
                    }
                }
                s_low[part][row] = low;
                s_t.odd[run * (2 * SL_BM) + 2 * row + part] = low;
                ++run;
                // the integer sums of 4 columns of each warp at a time through shared memory; a thread
                // converts and writes four elements, lanes on consecutive columns.  The register
                // arrays need constant indices, everything behind them is one rolled body.
                const double alpha = S.alpha;
                const bool scale = alpha != 1.0;
                // the elements of s_low: nothing here, odd_products_kernel adds what they are
                const bool any_odd = epi_bar_or(low != 0u) != 0;
                tile_odd = tile_odd || any_odd;
                const int slot = lane & 7, rr = warp * (4 * SL_NEL) + (lane >> 3);       // rows rr, rr + 4, ..
                #pragma unroll 1
                for (int p = 0; p < 8; ++p) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (u != p) continue;
#pragma unroll
                        for (int j = 0; j < SL_SUB; ++j)
                            s_raw[row][part * SL_SUB + j] =
                                make_uint4(sum[SL_SUB * u + j].w0, sum[SL_SUB * u + j].w1, sum[SL_SUB * u + j].w2, 0u);
                    }
                    epi_bar();
                    Sum96 raw[SL_NEL];
#pragma unroll
                    for (int it = 0; it < SL_NEL; ++it) {
                        const uint4 r = s_raw[rr + 4 * it][slot];
                        raw[it] = Sum96{r.x, r.y, r.z};
                    }
                    epi_bar();                                   // buffer free
                    const int jj = slot / SL_SUB * SL_CW + SL_SUB * p + slot % SL_SUB;
                    if (jj < BN && s_t.n0 + jj < s_t.N) {
                        const uint32_t wb = s_eB[jj];
                        const int eb = exp_of(wb);
                        double x[SL_NEL];
                        int te[SL_NEL];
#pragma unroll
                        for (int it = 0; it < SL_NEL; ++it) te[it] = exp_of(s_eA[rr + 4 * it]) + eb;
                        sliced_to_doubles<SL_NEL>(raw, te, x);
                        if (any_odd) {
#pragma unroll
                            for (int it = 0; it < SL_NEL; ++it)
                                if ((s_low[jj / SL_CW][rr + 4 * it] >> (jj % SL_CW)) & 1u) x[it] = 0.0;
                        }
                        if (scale) {
#pragma unroll
                            for (int it = 0; it < SL_NEL; ++it) x[it] *= alpha;
                        }
                        double* d[SL_NEL];
#pragma unroll
                        for (int it = 0; it < SL_NEL; ++it) d[it] = s_t.C + s_roff[rr + 4 * it] + s_coff[jj];
                        if (first && s_t.mode == 2) {
#pragma unroll
                            for (int it = 0; it < SL_NEL; ++it) {
                                if (s_diagB[jj]) x[it] += s_DA[rr + 4 * it];
                                if (s_diagA[rr + 4 * it]) x[it] += s_DB[jj];
                            }
                        }
                        if (s_t.mode == 1) {
#pragma unroll
                            for (int it = 0; it < SL_NEL; ++it)
                                if (s_t.m0 + rr + 4 * it < s_t.M) atomicAdd(d[it], x[it]);
                        } else {
                            // later segments add to what the same thread stored for the first one
                            if (!first) {
#pragma unroll
                                for (int it = 0; it < SL_NEL; ++it)
                                    if (s_t.m0 + rr + 4 * it < s_t.M) x[it] = *d[it] + x[it];
                            }
#pragma unroll
                            for (int it = 0; it < SL_NEL; ++it)
                                if (s_t.m0 + rr + 4 * it < s_t.M) *d[it] = x[it];
                        }
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int j = 0; j < SL_CW; ++j) sum[j] = Sum96{0u, 0u, 0u};
                first = false;
            }
            if (tile_odd && !failed && tid == 0) odd_list[1 + atomicAdd(odd_list, 1u)] = (uint32_t)tile;
            if (!failed) epi_bar();                              // metadata reads done before the next tile
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---- the elements in FP64 -------------------------------------------------------------------
// A tile's marked elements: sums of the marked runs of stages by FP64 FMAs, added to C, where the tile left
// nothing (delta terms apart).  Eight rows of a tile per CTA and step, or 32 where there are many tiles, the
// elements listed so that all threads share them: a few tiles that are marked throughout spread over the chip
// (in the GEMM's own epilogue they took 1.9 ms of an FP64 iteration of 18 spin orbitals, here 0.85).
constexpr int OD_ROWS = 8, OD_MORE_ROWS = 32, OD_THREADS = 256;

__global__ void __launch_bounds__(OD_THREADS, 4) odd_products_kernel(const xrh_gemm_task* __restrict__ tasks, int n_tasks,
                                                                  const xrh_sliced_segment* __restrict__ segs,
                                                                  const xrh_odd_range* __restrict__ odd_ranges,
                                                                  const uint32_t* __restrict__ odd_bits, const uint32_t* __restrict__ odd_list) {
    __shared__ uint16_t list[OD_MORE_ROWS * 64];
    __shared__ double s_part[OD_THREADS];
    __shared__ int s_count;
    __shared__ Tile s_tile;
    const int64_t n_odd = odd_list[0];
    const int rows = n_odd * (SL_BM / OD_ROWS) <= 8 * (int64_t)gridDim.x ? OD_ROWS : OD_MORE_ROWS, steps = SL_BM / rows;
    for (int64_t w = blockIdx.x; w < n_odd * steps; w += gridDim.x) {
        const int64_t tile = odd_list[1 + w / steps];
        const int r0 = (int)(w % steps) * rows;
        __syncthreads();
        if (threadIdx.x == 0) {
            s_tile = tile_of(tasks, n_tasks, segs, tile);
            s_count = 0;
        }
        __syncthreads();
        const Tile I = s_tile;
        const xrh_gemm_task& T = tasks[I.task];
        const xrh_sliced_segment* S0 = segs + T.seg_begin;
        const int runs = (int)odd_ranges[I.task].runs;
        const uint32_t* bits = odd_bits + (odd_ranges[I.task].begin + (tile - T.tile_begin) * runs) * (2 * SL_BM);
        // the runs of the tile (Groups): f(run, segment, first K, behind the last K)
        auto each_run = [&](auto&& f) {
            int si = 0, c = I.sb, run = 0;
            for (int left = I.left; left > 0; ++run) {
                while (c >= S0[si].stages) {
                    c -= (int)S0[si].stages;
                    ++si;
                }
                int k = (int)S0[si].stages - c;
                if (k > left) k = left;
                if (k > SL_RUN_GROUPS * SL_GROUP) k = SL_RUN_GROUPS * SL_GROUP;
                const int64_t end = (int64_t)(c + k) * SL_KS;
                f(run, S0[si], (int64_t)c * SL_KS, end < S0[si].K ? end : S0[si].K);
                c += k;
                left -= k;
            }
        };
        if (threadIdx.x < rows * 2) {
            const int r = r0 + (threadIdx.x >> 1), part = threadIdx.x & 1;
            uint32_t any = 0u;
            each_run([&](int run, const xrh_sliced_segment&, int64_t, int64_t) { any |= bits[run * (2 * SL_BM) + 2 * r + part]; });
            int at = atomicAdd(&s_count, __popc(any));
            for (; any; any &= any - 1u) list[at++] = (uint16_t)(r * 64 + part * SL_CW + __ffs((int)any) - 1);
        }
        __syncthreads();
        // a group of threads per element: neighbours, which read neighbouring K of stored rows (a lane a row would
        // touch 32 lines an instruction, twice the time of its FMAs), or, both operands stored [k][row], one of
        // every `step` threads, so that neighbours read neighbouring elements
        const bool trans = (S0->flags & 3) == 3;
        const int count = s_count, lanes = lanes_per_sum(count, OD_THREADS, S0->K, trans ? 1 : S0->K >= 64 ? 8 : 2);
        const int step = OD_THREADS / lanes;
        const bool across = lanes > 1 && trans;
        const int sub = across ? threadIdx.x / step : threadIdx.x % lanes;
        for (int e0 = 0; e0 < count; e0 += step) {
            const int e = e0 + (across ? threadIdx.x % step : threadIdx.x / lanes), at = list[e < count ? e : 0];
            const int r = at >> 6, j = at & 63;
            const int64_t m = I.m0 + r, col = I.n0 + j;
            double x = 0.0;
            each_run([&](int run, const xrh_sliced_segment& S, int64_t k0, int64_t k1) {
                if (e >= count || !((bits[run * (2 * SL_BM) + 2 * r + j / SL_CW] >> (j % SL_CW)) & 1u)) return;
                const double* a = S.A + I.batch * S.sA + m * ((S.flags & 1) ? 1 : S.lda);
                const double* b = S.B + I.batch * S.sB + col * ((S.flags & 2) ? 1 : S.ldb);
                const int64_t ka = (S.flags & 1) ? S.lda : 1, kb = (S.flags & 2) ? S.ldb : 1;
                double y = 0.0;
#pragma unroll 8
                for (int64_t k = k0 + sub; k < k1; k += lanes) y = fma(a[k * ka], b[k * kb], y);
                x += S.alpha * y;
            });
            if (across) {
                s_part[threadIdx.x] = x;
                __syncthreads();
                if (sub == 0)
                    for (int i = 1; i < lanes; ++i) x += s_part[threadIdx.x + i * step];
                __syncthreads();
            } else {
                x = sum_lanes(x, lanes);
            }
            if (e >= count || sub != 0) continue;
            double* d = T.C + I.batch * T.sC +
                        (T.mode == 2 ? (int64_t)(T.rowA[m] + T.rowB[col]) * T.ldc + T.colA[m] + T.colB[col] : m * T.ldc + col);
            if (T.mode == 1) atomicAdd(d, x);
            else *d += x;
        }
    }
}

// ---- digits -------------------------------------------------------------------------------
constexpr int DG_THREADS = 256;
constexpr int DG_WARP_K = 1024;        // rows up to this K: a warp each; longer ones a CTA each
constexpr int DG_TK = 64;              // transposed operands: 32 rows x 64 K per CTA
constexpr int DG_MAX_K = 512;          // K per CTA of the row-maximum pass

// Digit slices and magnitudes of four consecutive K elements of a row: nine 8-byte stores into the stage
// images (blocks of `block` rows; per block and 32 K: [slice][row][32 K], 64-byte rows, 64-byte swizzle:
// 16-byte chunk index xor bits 1..2 of the row; behind the digits of a block its magnitudes, [32 K][row]).
__device__ __forceinline__ void put_digits(const double (&x)[4], int E, const xrh_slice_task& T, int64_t blk, int r, int64_t k) {
    const int64_t stages = T.Kp / SL_KS, st = k / SL_KS, slice_stride = T.block * 64;
    const int kk = (int)(k & (SL_KS - 1));
    uint8_t* base = reinterpret_cast<uint8_t*>(T.digits) + blk * stages * (slice_stride * (NS + 1)) + r * 64 +
                    (((kk >> 3) ^ ((r >> 1) & 3)) << 4) + (kk & 7) * 2;
    uint8_t* dst = base + st * NS * slice_stride;
    const bool bad = E >= 2047;                        // an infinity or a NaN in the row
    uint64_t v[4];
    uint32_t m[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        v[e] = bad ? 0x0080808080808080ull : fixed62(x[e], E);
        m[e] = bad ? 0u : magnitude(x[e], E);
    }
    *reinterpret_cast<uint2*>(base + (stages * NS + st) * slice_stride) = make_uint2(m[0] | (m[1] << 16), m[2] | (m[3] << 16));
#pragma unroll
    for (int t = 0; t < NS; ++t) {
        uint32_t f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            f[e] = digit_float(v[e], t);
        }
        uint2 o;
        o.x = __byte_perm(f[0], f[1], 0x7632);          // upper halves: BF16
        o.y = __byte_perm(f[2], f[3], 0x7632);
        *reinterpret_cast<uint2*>(dst + t * slice_stride) = o;
    }
}

__device__ __forceinline__ int find_slice_task(const xrh_slice_task* __restrict__ tasks, int n_tasks, int64_t cta, bool max_pass) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((max_pass ? tasks[mid].max_begin : tasks[mid].cta_begin) <= cta) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Largest |element| of every row of the transposed operands: 32 rows x DG_MAX_K per CTA.
__global__ void __launch_bounds__(DG_THREADS) slice_max_kernel(const xrh_slice_task* __restrict__ tasks, int n_tasks) {
    __shared__ uint32_t part[8][32];
    const xrh_slice_task& T = tasks[find_slice_task(tasks, n_tasks, blockIdx.x, true)];
    int64_t local = (int64_t)blockIdx.x - T.max_begin;
    const int64_t nr = (T.rows + 31) / 32, nk = (T.K + DG_MAX_K - 1) / DG_MAX_K;
    const int64_t b = local / (nr * nk);
    local -= b * nr * nk;
    const int64_t r = (local % nr) * 32 + (threadIdx.x & 31), k0 = (local / nr) * DG_MAX_K;
    const int64_t ke = k0 + DG_MAX_K < T.K ? k0 + DG_MAX_K : T.K;
    uint32_t m = 0;
    if (r < T.rows) {
        const double* p = T.src + b * T.sbatch + r;
#pragma unroll 4
        for (int64_t k = k0 + (threadIdx.x >> 5); k < ke; k += 8) m = max(m, abs_hi(__ldg(p + k * T.ld)));
    }
    part[threadIdx.x >> 5][threadIdx.x & 31] = m;
    __syncthreads();
    if (threadIdx.x < 32 && r < T.rows) {
        for (int w = 1; w < 8; ++w) m = max(m, part[w][threadIdx.x]);
        atomicMax(T.exps + b * T.rows + r, m);
    }
}

__global__ void __launch_bounds__(DG_THREADS) slice_digits_kernel(const xrh_slice_task* __restrict__ tasks, int n_tasks,
                                                                  uint32_t* odd_list) {
    __shared__ uint32_t part[8];
    __shared__ double tile[DG_TK][33];
    const xrh_slice_task& T = tasks[find_slice_task(tasks, n_tasks, blockIdx.x, false)];
    int64_t local = (int64_t)blockIdx.x - T.cta_begin;
    if (blockIdx.x == 0 && threadIdx.x == 0) odd_list[0] = 0u;         // of the GEMM that follows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // rows are padded with zero digits to whole blocks (block: 32, 64 or 128)
    const int64_t blocks = (T.rows + T.block - 1) / T.block, rows_p = blocks * T.block;
    if (T.trans) {
        const int64_t nr = rows_p / 32, nk = (T.Kp + DG_TK - 1) / DG_TK;
        const int64_t b = local / (nr * nk);
        local -= b * nr * nk;
        const int64_t r0 = (local % nr) * 32, k0 = (local / nr) * DG_TK;
        const double* p = T.src + b * T.sbatch;
#pragma unroll
        for (int i = 0; i < DG_TK / 8; ++i) {
            const int64_t k = k0 + warp + 8 * i;
            tile[warp + 8 * i][lane] = (k < T.K && r0 + lane < T.rows) ? __ldg(p + k * T.ld + r0 + lane) : 0.0;
        }
        __syncthreads();
        // 16 threads take the 64 K of a row, four each; 16 rows at a time
        for (int rr = threadIdx.x >> 4; rr < 32; rr += DG_THREADS / 16) {
            const int64_t r = r0 + rr, k = k0 + 4 * (threadIdx.x & 15);
            if (k >= T.Kp) continue;
            const uint32_t w = r < T.rows ? T.exps[b * T.rows + r] >> 20 : 0u;
            const int E = w < 1u ? 1 : (int)w;
            double x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = tile[4 * (threadIdx.x & 15) + e][rr];
            put_digits(x, E, T, b * blocks + r / T.block, (int)(r % T.block), k);
        }
        return;
    }
    // K-contiguous rows: a warp, or the whole CTA, takes one row: its largest element, then the
    // digits (the second read of the row hits in cache)
    const bool wide = T.K > DG_WARP_K;
    const int64_t row = wide ? local : local * 8 + warp;
    const int64_t b = row / rows_p, r = row - b * rows_p;
    const bool ok = b < T.batch && r < T.rows;
    const double* p = T.src + b * T.sbatch + r * T.ld;
    const int step = wide ? DG_THREADS : 32, me = wide ? (int)threadIdx.x : lane;
    uint32_t m = 0;
    if (ok) {
#pragma unroll 4
        for (int64_t k = me; k < T.K; k += step) m = max(m, abs_hi(__ldg(p + k)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (wide) {
        if (lane == 0) part[warp] = m;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) m = max(m, part[w]);
    }
    if (b >= T.batch) return;
    if (ok && me == 0) T.exps[b * T.rows + r] = m;
    const uint32_t w = m >> 20;
    const int E = w < 1u ? 1 : (int)w;
    for (int64_t k = 4 * me; k < T.Kp; k += 4 * step) {
        double x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = ok && k + e < T.K ? __ldg(p + k + e) : 0.0;
        put_digits(x, E, T, b * blocks + r / T.block, (int)(r % T.block), k);
    }
}

}  // namespace

extern "C" int64_t xrh_slice_ctas(int64_t rows, int64_t K, int64_t batch, int trans, int block, int max_pass) {
    if (rows <= 0 || K <= 0 || batch <= 0 || (block != 32 && block != 64 && block != 128)) return 0;
    const int64_t rows_p = (rows + block - 1) / block * block;
    if (trans) {
        if (max_pass) return batch * ((rows + 31) / 32) * ((K + DG_MAX_K - 1) / DG_MAX_K);
        return batch * (rows_p / 32) * (((K + SL_KS - 1) / SL_KS * SL_KS + DG_TK - 1) / DG_TK);
    }
    if (max_pass) return 0;
    return K > DG_WARP_K ? rows_p * batch : rows_p * batch / 8;
}

extern "C" int xrh_slice_grouped(const xrh_slice_task* tasks_dev, int n_tasks, int64_t total_ctas, int64_t max_ctas,
                                 uint32_t* odd_list_dev, void* stream) {
    if (n_tasks < 0 || total_ctas < 0 || max_ctas < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_ctas == 0) return XRH_OK;
    if (!tasks_dev || !odd_list_dev) return XRH_ERR_ARG;
    if (total_ctas > 0x7fffffffLL || max_ctas > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    if (max_ctas > 0) {
        slice_max_kernel<<<(unsigned)max_ctas, DG_THREADS, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
        XRH_CHECK_LAUNCH();
    }
    slice_digits_kernel<<<(unsigned)total_ctas, DG_THREADS, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks, odd_list_dev);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

extern "C" int xrh_gemm_sliced_grouped(const xrh_gemm_task* tasks_dev, int n_tasks, int64_t total_tiles,
                                       const xrh_sliced_segment* segs_dev, const xrh_odd_range* odd_ranges_dev,
                                       uint32_t* odd_bits_dev, uint32_t* odd_list_dev, int32_t* status_dev, void* stream) {
    if (n_tasks < 0 || total_tiles < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_tiles == 0) return XRH_OK;
    if (!tasks_dev || !segs_dev || !odd_ranges_dev || !odd_bits_dev || !odd_list_dev || !status_dev) return XRH_ERR_ARG;
    if (total_tiles > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    int dev = 0, n_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = (size_t)SL_STAGES * SL_STAGE_BYTES + 1024;
    cudaFuncSetAttribute(gemm_sliced_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int64_t grid = total_tiles < n_sm ? total_tiles : n_sm;
    gemm_sliced_kernel<<<(unsigned)grid, SL_THREADS, smem, (cudaStream_t)stream>>>(
        tasks_dev, n_tasks, total_tiles, segs_dev, odd_ranges_dev, odd_bits_dev, odd_list_dev, status_dev);
    XRH_CHECK_LAUNCH();
    const int64_t odd_grid = total_tiles * (SL_BM / OD_ROWS) < 4 * n_sm ? total_tiles * (SL_BM / OD_ROWS) : 4 * n_sm;
    odd_products_kernel<<<(unsigned)odd_grid, OD_THREADS, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks, segs_dev, odd_ranges_dev,
                                                                                     odd_bits_dev, odd_list_dev);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}
