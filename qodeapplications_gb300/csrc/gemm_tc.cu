// Split-precision grouped GEMM on the 5th-generation tensor cores (tcgen05, sm_103a).
//
// Same task model as the FP64 path (gemm_fp64.cu): every output block of the XR-H build is
// one task whose K-concatenated segments are the density x integral contractions that land
// in it.  Each FP64 operand X is split once per build into hi = round(X) and
// lo = round(X - hi) in BF16 (XRH_BF16X3) or TF32 (XRH_TF32X3); a segment contributes
//     A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T.
//
// Accuracy: the tensor core's FP32 accumulation is not round-to-nearest, and its error grows
// with the number of MMA steps summed into one accumulator.  So no accumulator outlives a K
// chunk (128 bytes of K: 64 BF16 / 32 TF32 elements): every chunk writes a fresh main slot
// (hi*hi, 4 MMA steps) and a fresh correction slot (hi*lo + lo*hi, 8 steps, 2^-8 smaller),
// and the epilogue warps drain both into FP32 registers with ordinary round-to-nearest adds
// while the tensor core works on the next chunk.  The tile is converted to FP64 once, where
// the segment-independent delta terms are added and the result is scattered like the FP64
// path.
//
// Per CTA (persistent over 128 x BN output tiles, one CTA per SM), 18 warps:
//   * warp 16, one thread: TMA loads (cp.async.bulk.tensor, 128B swizzle) of the four operand
//     tiles of a chunk into a 3-stage shared-memory ring, prefetched across tile boundaries;
//   * warp 17, one thread: the 8 tcgen05.mma of each chunk into one of two TMEM chunk buffers (main +
//     correction slot, 2 BN columns): A_hi x [B_hi; B_lo] goes to both slots at once, then A_lo x B_hi
//     (12 MMAs of half the width wait longer for their accumulators); tcgen05.commit releases the
//     ring stage (empty) and hands the buffer to the epilogue (ready);
//   * warps 0-15: per chunk, tcgen05.ld of both slots (warp w reads TMEM lanes 32(w%4).. = rows, a
//     quarter of the columns), add into registers, release the buffer (drained); at the end of the
//     tile, the FP64 epilogue.
// What bounds it: for short K the store of C, for long K the operand tiles (64 KB a chunk from L2).
// Measured, TF32 x 3: 3600 x 21952, K = 28 374 -> 227 us (2.8 TB/s of C); 3600 x 3600, K = 784 257 -> 157 us (42
// bytes/clk/SM of operands; without its drains or a third of its MMAs the same); 1600 x 1120 over 40
// segments of K = 28 71 -> 45 us; before: one thread for loads and MMAs, 8 epilogue warps that converted on the
// FP64 pipe and stored 8 bytes a lane behind barriers.
// Every mbarrier wait is bounded; on timeout the kernel records XRH_ERR_TIMEOUT in *status,
// every warp leaves its loop (the epilogue warps decide together through bar.red.or once per
// tile), the producer waits (bounded) for its copies and MMAs in flight, TMEM is freed and the
// kernel returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "tc_common.cuh"
#include "xrh_common.cuh"

namespace {
using namespace xrh_tc;

constexpr int TC_BM = 128;
constexpr int TC_STAGES = 3;
constexpr int TC_EPI_WARPS = 16;
constexpr int TC_EPI_THREADS = TC_EPI_WARPS * 32;
constexpr int TC_THREADS = TC_EPI_THREADS + 64;    // + a warp that loads, a warp that multiplies
constexpr int TC_TILES = 4;                         // tiles announced to the epilogue
constexpr uint32_t TC_TMEM_COLS = 512;             // 2 chunk buffers x (main, correction) x 128
constexpr uint32_t TC_A_BYTES = TC_BM * 128;       // 128 rows x 128 B (one swizzle width of K)
constexpr uint32_t TC_B_MAX_BYTES = 128 * 128;
constexpr uint32_t TC_STAGE_BYTES = 2 * TC_A_BYTES + 2 * TC_B_MAX_BYTES;

// Named barrier 1 over the epilogue warps, returning the OR of a predicate over them.
__device__ __forceinline__ int epi_bar_or(int pred) { return named_bar_or<1, TC_EPI_THREADS>(pred); }

__device__ __forceinline__ int find_task(const xrh_tc_task* __restrict__ tasks, int n_tasks, int64_t tile) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Where a persistent CTA's tile lies: its task, output corner, N tile and K-chunk range.
struct TileInfo {
    int task, m0, n0, BN, nk;
    int64_t cb;
};

__device__ __forceinline__ TileInfo tile_info(const xrh_tc_task* __restrict__ tasks, int n_tasks,
                                              const xrh_tc_segment* __restrict__ segs, int64_t tile) {
    TileInfo r;
    r.task = find_task(tasks, n_tasks, tile);
    const xrh_tc_task& T = tasks[r.task];
    r.BN = (int)T.bn;
    const int64_t tiles_m = (T.M + TC_BM - 1) / TC_BM, tiles_n = (T.N + r.BN - 1) / r.BN;
    int64_t local = tile - T.tile_begin;
    const int64_t split = local / (tiles_m * tiles_n);
    local -= split * tiles_m * tiles_n;
    // the CTAs running at once take consecutive tiles: they walk the M tiles of one N tile when
    // M < N, so the smaller operand (A, M x K) is the one every CTA re-reads (from L2) and each
    // tile of the larger one comes from HBM once; else the N tiles of one M tile
    if (T.M < T.N) {
        r.m0 = (int)((local % tiles_m) * TC_BM);
        r.n0 = (int)((local / tiles_m) * r.BN);
    } else {
        r.m0 = (int)((local / tiles_n) * TC_BM);
        r.n0 = (int)((local % tiles_n) * r.BN);
    }
    int64_t kc_total = 0;
#pragma unroll 8
    for (int64_t s = 0; s < T.seg_count; ++s) kc_total += segs[T.seg_begin + s].kchunks;
    const int64_t per = (kc_total + T.splitk - 1) / T.splitk;
    r.cb = split * per;
    const int64_t ce = (r.cb + per < kc_total) ? r.cb + per : kc_total;
    r.nk = (int)(ce > r.cb ? ce - r.cb : 0);
    return r;
}

template <int KIND>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_tc_kernel(const xrh_tc_task* __restrict__ tasks, int n_tasks, int64_t total_tiles,
                   const xrh_tc_segment* __restrict__ segs, const CUtensorMap* __restrict__ maps, int32_t* status) {
    extern __shared__ unsigned char smem_raw[];
    uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[TC_STAGES];
    __shared__ __align__(8) uint64_t empty_bar[TC_STAGES];
    __shared__ __align__(8) uint64_t ready_bar[2];
    __shared__ __align__(8) uint64_t drained_bar[2];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_sh;
    __shared__ int s_negate[TC_STAGES];                 // of the chunk in a stage
    // tiles announced by the MMA warp: where, first chunk and number of chunks (0: no more tiles)
    __shared__ __align__(8) uint64_t tile_bar[TC_TILES];
    __shared__ TileInfo s_tile[TC_TILES];
    // element (m, n) of the tile lies at C[s_roff[m] + s_coff[n]]
    __shared__ int64_t s_roff[128], s_coff[128];
    __shared__ double s_DA[128], s_DB[128];
    __shared__ unsigned char s_diagA[128], s_diagB[128];
    __shared__ __align__(8) float s_stage[TC_EPI_WARPS][16][18];      // 16 x 16 results of a warp, on their way to C
    constexpr int KCH = (KIND == 0) ? 64 : 32;          // elements of K per 128-byte chunk
    constexpr uint32_t FMT = (KIND == 0) ? 1u : 2u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&ready_bar[b]), 1);
            mbar_init(smem_u32(&drained_bar[b]), TC_EPI_WARPS);
        }
        for (int t = 0; t < TC_TILES; ++t) mbar_init(smem_u32(&tile_bar[t]), 1);
        mbar_init(smem_u32(&done_bar), 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh;

    if (warp == TC_EPI_WARPS) {
        // ---------------------------------------------------------------------- loads --
        if (lane == 0) {
            uint64_t g = 0;                    // chunks loaded
            bool ok = true;
            for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const TileInfo I = tile_info(tasks, n_tasks, segs, tile);
                if (I.nk == 0) continue;
                const uint32_t b_bytes = (uint32_t)I.BN * 128u;
                // the tile's first segment is located once (its split-K offset); the next one's fields
                // are read while this one's chunks are loaded
                const int64_t seg_end = tasks[I.task].seg_begin + tasks[I.task].seg_count;
                int64_t si = tasks[I.task].seg_begin, c = I.cb;
                xrh_tc_segment S = segs[si], nx = si + 1 < seg_end ? segs[si + 1] : S;
                for (int q = 0; q < I.nk; ++q, ++g) {
                    while (c >= S.kchunks) {
                        c -= S.kchunks;
                        ++si;
                        S = nx;
                        if (si + 1 < seg_end) nx = segs[si + 1];
                    }
                    const int s = (int)(g % TC_STAGES);
                    if (g >= TC_STAGES && !mbar_wait(smem_u32(&empty_bar[s]), (uint32_t)(g / TC_STAGES - 1) & 1u, &abort_sh)) {
                        ok = false;
                        break;
                    }
                    const int kcoord = (int)(c * KCH);
                    ++c;
                    uint8_t* st = stages + (size_t)s * TC_STAGE_BYTES;
                    const uint32_t bar = smem_u32(&full_bar[s]);
                    s_negate[s] = S.negate != 0;
                    mbar_expect_tx(bar, 2u * TC_A_BYTES + 2u * b_bytes);
                    tma_load_2d(smem_u32(st), maps + S.tmA, bar, kcoord, I.m0);
                    tma_load_2d(smem_u32(st + TC_A_BYTES), maps + S.tmA + 1, bar, kcoord, I.m0);
                    tma_load_2d(smem_u32(st + 2 * TC_A_BYTES), maps + S.tmB, bar, kcoord, I.n0);
                    tma_load_2d(smem_u32(st + 2 * TC_A_BYTES + b_bytes), maps + S.tmB + 1, bar, kcoord, I.n0);
                }
            }
            if (!ok) {
                abort_sh = 1;
                atomicExch(status, XRH_ERR_TIMEOUT);
            }
            // every copy issued has landed before shared memory goes away (bounded)
            for (uint64_t q = g > TC_STAGES ? g - TC_STAGES : 0; q < g; ++q)
                mbar_wait(smem_u32(&full_bar[q % TC_STAGES]), (uint32_t)(q / TC_STAGES) & 1u, nullptr);
        }
    } else if (warp == TC_EPI_WARPS + 1) {
        // ------------------------------------------------------------------------ MMA --
        if (lane == 0) {
            uint64_t g = 0;
            uint32_t k = 0;                    // tiles announced
            bool ok = true;
            // (entry k has been read before its chunk buffers let tile k + 3 begin)
            auto announce = [&](TileInfo I) {
                I.cb = (int64_t)g;
                s_tile[k % TC_TILES] = I;
                mbar_arrive(smem_u32(&tile_bar[k % TC_TILES]));
                ++k;
            };
            for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const TileInfo I = tile_info(tasks, n_tasks, segs, tile);
                if (I.nk == 0) continue;
                announce(I);
                const uint32_t bn = (uint32_t)I.BN;
                for (int q = 0; q < I.nk; ++q, ++g) {
                    // the MMAs of chunk g into chunk buffer g & 1
                    const int s = (int)(g % TC_STAGES);
                    const uint32_t b = (uint32_t)(g & 1);
                    if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(g / TC_STAGES) & 1u, &abort_sh) ||
                        (g >= 2 && !mbar_wait(smem_u32(&drained_bar[b]), (uint32_t)((g >> 1) - 1) & 1u, &abort_sh))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const bool neg = s_negate[s] != 0;
                    const uint32_t wide = make_idesc(FMT, TC_BM, 2 * bn, neg), narrow = make_idesc(FMT, TC_BM, bn, neg);
                    const uint32_t st = smem_u32(stages + (size_t)s * TC_STAGE_BYTES);
                    const uint64_t da_hi = umma_desc_sw128(st), da_lo = umma_desc_sw128(st + TC_A_BYTES);
                    const uint64_t db = umma_desc_sw128(st + 2 * TC_A_BYTES);
                    const uint32_t t_main = tmem + b * 256u, t_corr = t_main + bn;
                    // B_lo lies behind B_hi and the correction slot behind the main one: A_hi times both is
                    // one MMA a K step (32 bytes), with the same sums in either slot
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma<KIND>(t_main, da_hi + 2 * j, db + 2 * j, wide, j > 0 ? 1u : 0u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma<KIND>(t_corr, da_lo + 2 * j, db + 2 * j, narrow, 1u);
                    umma_commit(smem_u32(&empty_bar[s]));
                    umma_commit(smem_u32(&ready_bar[b]));
                }
            }
            if (ok) {
                announce(TileInfo{});
            } else {
                abort_sh = 1;
                atomicExch(status, XRH_ERR_TIMEOUT);
            }
            // every MMA issued has completed before TMEM goes away (bounded)
            umma_commit(smem_u32(&done_bar));
            mbar_wait(smem_u32(&done_bar), 0u, nullptr);
        }
    } else {
        // ------------------------------------------------------------------ epilogue --
        const int quarter = warp & 3, part = warp >> 2;      // TMEM lanes 32*quarter.., a quarter of the columns
        for (uint32_t k = 0;; ++k) {
            const bool here = mbar_wait(smem_u32(&tile_bar[k % TC_TILES]), (k / TC_TILES) & 1u, &abort_sh);
            const TileInfo I = s_tile[k % TC_TILES];
            // (also: the metadata of the tile before have been read)
            if (epi_bar_or(!here)) {
                abort_sh = 1;
                if (tid == 0) atomicExch(status, XRH_ERR_TIMEOUT);
                break;
            }
            if (I.nk == 0) break;
            uint64_t ge = (uint64_t)I.cb;
            const xrh_tc_task& T = tasks[I.task];
            const int BN = I.BN, m0 = I.m0, n0 = I.n0;
            // metadata of the tile (the decision barrier below is behind it)
            {
                const bool scatter = T.mode == 2;
                const int64_t ldc = T.ldc;
                const int M = (int)T.M, N = (int)T.N;
                for (int x = tid; x < TC_BM + BN; x += TC_EPI_THREADS) {
                    if (x < TC_BM) {
                        const int m = m0 + x;
                        const bool ok = scatter && m < M;
                        s_roff[x] = ok ? (int64_t)T.rowA[m] * ldc + T.colA[m] : m * ldc;
                        s_diagA[x] = ok ? T.diagA[m] : 0;
                        s_DA[x] = (ok && T.DA) ? T.DA[m] : 0.0;
                    } else {
                        const int j = x - TC_BM, n = n0 + j;
                        const bool ok = scatter && n < N;
                        s_coff[j] = ok ? (int64_t)T.rowB[n] * ldc + T.colB[n] : n;
                        s_diagB[j] = ok ? T.diagB[n] : 0;
                        s_DB[j] = (ok && T.DB) ? T.DB[n] : 0.0;
                    }
                }
            }
            float acc[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[j] = 0.f;
            const int cw = BN >> 2, cb = part * cw;              // this warp's columns: 8, 16 or 32
            // the warps drain their chunks independently; a wait that gives up raises abort_sh,
            // so the others' waits give up too, and all decide together once per tile below
            bool failed = false;
            for (int q = 0; q < I.nk; ++q, ++ge) {
                const uint32_t b = (uint32_t)(ge & 1);
                if (!mbar_wait(smem_u32(&ready_bar[b]), (uint32_t)(ge >> 1) & 1u, &abort_sh)) {
                    failed = true;
                    abort_sh = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
                const uint32_t at = tmem + lane_base + b * 256u + (uint32_t)cb;
#pragma unroll
                for (int h = 0; h < 32; h += 16) {
                    if (h < cw) {                                      // uniform
                        float vm[16], vc[16];
                        // (8 columns: the 8 behind them are read and not used)
                        tmem_ld16_pair(at + h, at + h + (uint32_t)BN, vm, vc);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[h + j] += vm[j] + vc[j];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&drained_bar[b]));
            }
            // one collective decision per tile (also the barrier after the column metadata)
            if (epi_bar_or(failed)) {
                abort_sh = 1;
                if (tid == 0) atomicExch(status, XRH_ERR_TIMEOUT);
                break;
            }
            // FP64 epilogue, 16 rows x 16 columns of a warp at a time, without the other warps: through its
            // own shared memory to lanes on pairs of columns, four rows an instruction.  16-byte stores
            // reach 6.7 TB/s here, 8-byte ones 4.4.  FP32 to FP64 by integer operations (the FP64 pipe
            // converts 2 lanes/clk/SM).
            double* C = T.C;
            const int mode = (int)T.mode, N = (int)T.N;
            const int64_t ldc = T.ldc;
            // a tile inside a plain matrix of 16-byte rows: no bounds, no offsets
            const bool whole = mode == 0 && m0 + TC_BM <= T.M && n0 + BN <= N && (ldc & 1) == 0 &&
                               (reinterpret_cast<uintptr_t>(C) & 15) == 0;
            const int col = 2 * (lane & 7), r_lane = lane >> 3;
#pragma unroll 1
            for (int p = 0; p < 4; ++p) {                              // columns 16 (p >> 1).., rows 16 (p & 1)..
                if (16 * (p >> 1) >= cw) break;                        // uniform
                if ((lane >> 4) == (p & 1)) {
                    // (selected value by value: an array indexed at run time would lie in local memory)
#pragma unroll
                    for (int j = 0; j < 16; ++j) s_stage[warp][lane & 15][j] = p < 2 ? acc[j] : acc[16 + j];
                }
                __syncwarp();
                const int jc = 16 * (p >> 1) + col, jj = cb + jc, row0 = quarter * 32 + 16 * (p & 1) + r_lane;
                if (jc < cw && n0 + jj < N) {
                    float f[8];
                    double x[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 v = *reinterpret_cast<const float2*>(&s_stage[warp][r_lane + 4 * i][col]);
                        f[2 * i] = v.x;
                        f[2 * i + 1] = v.y;
                    }
                    xrh_f32_to_f64s(f, x);
                    if (mode == 2) {
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const bool diag_col = s_diagB[jj + e];
                            const double db = s_DB[jj + e];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (diag_col) x[2 * i + e] += s_DA[row0 + 4 * i];
                                if (s_diagA[row0 + 4 * i]) x[2 * i + e] += db;
                            }
                        }
                    }
                    if (whole) {
                        double* d0 = C + (int64_t)(m0 + row0) * ldc + n0 + jj;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            *reinterpret_cast<double2*>(d0 + 4 * i * ldc) = make_double2(x[2 * i], x[2 * i + 1]);
                    } else {
                        const int64_t o0 = s_coff[jj], o1 = s_coff[jj + 1];
                        const bool two = n0 + jj + 1 < N, pair = two && o1 == o0 + 1;
                        const int left = (int)T.M - m0 - row0;             // rows from this lane's first one on
                        double* d[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) d[i] = C + o0 + s_roff[row0 + 4 * i];
                        if (mode == 1) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (4 * i < left) atomicAdd(d[i], x[2 * i]);
                                if (4 * i < left && two) atomicAdd(d[i] + (o1 - o0), x[2 * i + 1]);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (4 * i >= left) continue;
                                if (pair && (reinterpret_cast<uintptr_t>(d[i]) & 15) == 0) {
                                    *reinterpret_cast<double2*>(d[i]) = make_double2(x[2 * i], x[2 * i + 1]);
                                } else {
                                    *d[i] = x[2 * i];
                                    if (two) d[i][o1 - o0] = x[2 * i + 1];
                                }
                            }
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
    }
}

// ---- operand split --------------------------------------------------------------------
// One thread per group of 4 consecutive K elements of a row (one division per group), one
// 8- or 16-byte store per group and part.
template <int KIND>
__device__ __forceinline__ void split_store(const float (&x)[4], void* __restrict__ hi, void* __restrict__ lo, int64_t o);

template <int KIND>
__device__ __forceinline__ void split_group(const double* __restrict__ src, int64_t K, int64_t ld, int64_t Kp,
                                            void* __restrict__ hi, void* __restrict__ lo, int64_t t) {
    const int64_t groups = Kp >> 2;
    const int64_t r = t / groups;
    const int64_t k0 = (t - r * groups) * 4;
    const double* srow = src + r * ld;
    // x rounded to FP32 by integer operations; hi from it and lo = x32 - hi, exact in FP32 (it
    // keeps the low mantissa bits of x32); the part of x below FP32 (2^-24 |x|) lies under
    // lo's own resolution.  No FP64 arithmetic: the FP64 pipe is slow on this part.
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = (k0 + e < K) ? xrh_f64_to_f32(__ldg(srow + k0 + e)) : 0.f;
    split_store<KIND>(x, hi, lo, r * Kp + k0);
}

template <int KIND>
__device__ __forceinline__ void split_store(const float (&x)[4], void* __restrict__ hi, void* __restrict__ lo, int64_t o) {
    if constexpr (KIND == 0) {
        __nv_bfloat16 h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            h[e] = __float2bfloat16_rn(x[e]);
            l[e] = __float2bfloat16_rn(__fsub_rn(x[e], __bfloat162float(h[e])));
        }
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(hi) + o) = *reinterpret_cast<uint2*>(h);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(lo) + o) = *reinterpret_cast<uint2*>(l);
    } else {
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h[e]) : "f"(x[e]));
            const float rem = __fsub_rn(x[e], __uint_as_float(h[e]));
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l[e]) : "f"(rem));
        }
        *reinterpret_cast<uint4*>(reinterpret_cast<uint32_t*>(hi) + o) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(reinterpret_cast<uint32_t*>(lo) + o) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

template <int KIND>
__global__ void split_kernel(const double* __restrict__ src, int64_t rows, int64_t K, int64_t ld, int64_t Kp,
                             void* __restrict__ hi, void* __restrict__ lo) {
    const int64_t total = rows * (Kp >> 2);
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
        split_group<KIND>(src, K, ld, Kp, hi, lo, t);
}

// Every operand of a task table in one launch: global 4-element group g belongs to the task
// with the last group_begin <= g (binary search over the group_begin values staged in shared
// memory, SPLIT_SMEM_TASKS of them at most; larger tables search global memory).
constexpr int SPLIT_SMEM_TASKS = 512;

template <int KIND>
__global__ void __launch_bounds__(256) split_grouped_kernel(const xrh_split_task* __restrict__ tasks, int n_tasks,
                                                            int64_t total) {
    __shared__ int64_t s_begin[SPLIT_SMEM_TASKS];
    const bool in_smem = n_tasks <= SPLIT_SMEM_TASKS;
    if (in_smem)
        for (int i = threadIdx.x; i < n_tasks; i += blockDim.x) s_begin[i] = tasks[i].group_begin;
    __syncthreads();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = n_tasks - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const int64_t b = in_smem ? s_begin[mid] : tasks[mid].group_begin;
            if (b <= t) lo = mid; else hi = mid - 1;
        }
        const xrh_split_task& T = tasks[lo];
        split_group<KIND>(T.src, T.K, T.ld, T.Kp, T.hi, T.lo, t - T.group_begin);
    }
}

// Operands stored transposed, src [K][rows]: 32 rows x 64 K per CTA through shared memory, read along
// the rows, written in 16-byte groups along K (256 bytes a row).  In place of a transposed FP64 copy
// first: 16 bytes an element through memory instead of 32; bound by memory.
template <int KIND>
__global__ void __launch_bounds__(256) split_trans_grouped_kernel(const xrh_split_task* __restrict__ tasks, int n_tasks) {
    __shared__ __align__(16) double tile[32][66];
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].group_begin <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const xrh_split_task& T = tasks[lo];
    const int64_t local = (int64_t)blockIdx.x - T.group_begin, tr = (T.rows + 31) / 32;
    const int64_t r0 = (local % tr) * 32, k0 = (local / tr) * 64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t k = k0 + warp + 8 * i;
        v[i] = (k < T.K && r0 + lane < T.rows) ? __ldg(T.src + k * T.ld + r0 + lane) : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) tile[lane][warp + 8 * i] = v[i];
    __syncthreads();
#pragma unroll
    for (int item = threadIdx.x; item < 32 * 16; item += 256) {
        const int r = item >> 4, g = 4 * (item & 15);
        if (r0 + r >= T.rows || k0 + g >= T.Kp) continue;
        const double2 a = *reinterpret_cast<const double2*>(&tile[r][g]), b = *reinterpret_cast<const double2*>(&tile[r][g + 2]);
        const float x[4] = {xrh_f64_to_f32(a.x), xrh_f64_to_f32(a.y), xrh_f64_to_f32(b.x), xrh_f64_to_f32(b.y)};
        split_store<KIND>(x, T.hi, T.lo, (r0 + r) * T.Kp + k0 + g);
    }
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

}  // namespace

extern "C" int xrh_tc_chunk_elems(int precision) {
    return precision == XRH_BF16X3 ? 64 : (precision == XRH_TF32X3 ? 32 : 0);
}

extern "C" int xrh_split_operand(int precision, const double* src_dev, int64_t rows, int64_t K, int64_t ld,
                                 int64_t Kp, void* hi_dev, void* lo_dev, void* stream) {
    const int kch = xrh_tc_chunk_elems(precision);
    if (!kch) return XRH_ERR_UNSUPPORTED;
    if (rows < 0 || K < 0 || ld < K || Kp < K || Kp % kch) return XRH_ERR_ARG;
    if (rows == 0 || Kp == 0) return XRH_OK;
    if (!src_dev || !hi_dev || !lo_dev) return XRH_ERR_ARG;
    // the hi / lo arrays are [rows, Kp] with Kp a multiple of 32 elements: 16-byte row starts
    if ((reinterpret_cast<uintptr_t>(hi_dev) & 15) || (reinterpret_cast<uintptr_t>(lo_dev) & 15)) return XRH_ERR_ARG;
    const int64_t total = rows * (Kp / 4);
    const int64_t blocks64 = (total + 255) / 256;
    const unsigned blocks = (unsigned)(blocks64 < 152 * 64 ? blocks64 : 152 * 64);
    if (precision == XRH_BF16X3)
        split_kernel<0><<<blocks, 256, 0, (cudaStream_t)stream>>>(src_dev, rows, K, ld, Kp, hi_dev, lo_dev);
    else
        split_kernel<1><<<blocks, 256, 0, (cudaStream_t)stream>>>(src_dev, rows, K, ld, Kp, hi_dev, lo_dev);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

extern "C" int xrh_split_grouped(int precision, const xrh_split_task* tasks_dev, int n_tasks, int64_t total_groups,
                                 void* stream) {
    if (!xrh_tc_chunk_elems(precision)) return XRH_ERR_UNSUPPORTED;
    if (n_tasks < 0 || total_groups < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_groups == 0) return XRH_OK;
    if (!tasks_dev) return XRH_ERR_ARG;
    const int64_t blocks64 = (total_groups + 255) / 256;
    const unsigned blocks = (unsigned)(blocks64 < 152 * 32 ? blocks64 : 152 * 32);
    if (precision == XRH_BF16X3)
        split_grouped_kernel<0><<<blocks, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks, total_groups);
    else
        split_grouped_kernel<1><<<blocks, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks, total_groups);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

extern "C" int xrh_split_trans_grouped(int precision, const xrh_split_task* tasks_dev, int n_tasks, int64_t total_tiles,
                                       void* stream) {
    if (!xrh_tc_chunk_elems(precision)) return XRH_ERR_UNSUPPORTED;
    if (n_tasks < 0 || total_tiles < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_tiles == 0) return XRH_OK;
    if (!tasks_dev) return XRH_ERR_ARG;
    if (total_tiles > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    if (precision == XRH_BF16X3)
        split_trans_grouped_kernel<0><<<(unsigned)total_tiles, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
    else
        split_trans_grouped_kernel<1><<<(unsigned)total_tiles, 256, 0, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}

extern "C" int xrh_tc_encode_map(int precision, const void* base_dev, int64_t rows, int64_t Kp, int box_rows,
                                 void* map_out_host) {
    const int kch = xrh_tc_chunk_elems(precision);
    if (!kch) return XRH_ERR_UNSUPPORTED;
    if (!base_dev || !map_out_host || rows <= 0 || Kp <= 0 || Kp % kch) return XRH_ERR_ARG;
    if (box_rows != 32 && box_rows != 64 && box_rows != 128) return XRH_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(base_dev) & 15) != 0) return XRH_ERR_ARG;
    PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode();
    if (!enc) return XRH_ERR_UNSUPPORTED;
    const int esz = precision == XRH_BF16X3 ? 2 : 4;
    const cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)Kp * esz};
    const cuuint32_t box[2] = {(cuuint32_t)kch, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(reinterpret_cast<CUtensorMap*>(map_out_host),
                     precision == XRH_BF16X3 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                     const_cast<void*>(base_dev), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? XRH_OK : XRH_ERR_ARG;
}

extern "C" int xrh_gemm_tc_grouped(int precision, const xrh_tc_task* tasks_dev, int n_tasks, int64_t total_tiles,
                                   const xrh_tc_segment* segs_dev, const void* maps_dev, int32_t* status_dev,
                                   void* stream) {
    if (!xrh_tc_chunk_elems(precision)) return XRH_ERR_UNSUPPORTED;
    if (n_tasks < 0 || total_tiles < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_tiles == 0) return XRH_OK;
    if (!tasks_dev || !segs_dev || !maps_dev || !status_dev) return XRH_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(maps_dev) & 63) != 0) return XRH_ERR_ARG;
    int dev = 0, n_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = (size_t)TC_STAGES * TC_STAGE_BYTES + 1024;
    const int64_t grid64 = total_tiles < n_sm ? total_tiles : n_sm;
    const unsigned grid = (unsigned)(grid64 > 0 ? grid64 : 1);
    if (precision == XRH_BF16X3) {
        cudaFuncSetAttribute(gemm_tc_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        gemm_tc_kernel<0><<<grid, TC_THREADS, smem, (cudaStream_t)stream>>>(
            tasks_dev, n_tasks, total_tiles, segs_dev, reinterpret_cast<const CUtensorMap*>(maps_dev), status_dev);
    } else {
        cudaFuncSetAttribute(gemm_tc_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        gemm_tc_kernel<1><<<grid, TC_THREADS, smem, (cudaStream_t)stream>>>(
            tasks_dev, n_tasks, total_tiles, segs_dev, reinterpret_cast<const CUtensorMap*>(maps_dev), status_dev);
    }
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}
