// FP32 transition densities of blocks of many states (sm_103a): the sums of xrh_density_accumulate_f32
// for blocks that are one thread group there (more than 128 register tiles of 4 x 4, about 45 states a
// side), in the same order, so with the same bits.
//
//   rho[idx, I, J] = sum_c s_c zb[P_c, I] zk[Q_c, J]     (FP32 products, FP64 result of an FP32 pair)
//
// The couplings of an index come as stages of C (positive signs first); a stage is a chain of FP32 FMAs,
// stages are added to an FP32 (hi, lo) pair by TwoSum.  A CTA takes an index (or a split of one) and a
// block of 64 x 64 states, a lane 8 rows and 4 columns of them:
//   * 48 bytes of shared memory for 32 FMAs (4 x 4 tiles: 32 for 16, which bounded them; 16 x 2 is 4 %
//     slower, 8 x 8 does not fit the registers and is 25 % slower);
//   * the FMAs are packed pairs of rows (fma.rn.f32x2: the same rounding, half the issue slots);
//   * couplings are gathered 32 at a time, three buffers, a bra and a ket row per instruction, indexes
//     read one buffer ahead, and the first negative coupling of an index comes from the host instead
//     of a search by dependent loads (about 20 of them).
// Measured, all such blocks of a fragment of 28 spin orbitals, 60 states: 4.98 -> 2.94 ms (33 TFLOP/s; the
// FP32 pipe alone takes 1.5, everything else 1.3: indexes of about 640 couplings are short); 24 and 48
// states 2.6 -> 1.20 ms.
#include "xrh_common.cuh"

namespace {

constexpr int FW_SUB = 32, FW_RING = 3, FW_ROW = 128;  // floats of a staged coupling: bra 64 | ket 64
constexpr int FW_TN = 4;                               // a lane: 8 rows x 4 columns
constexpr int FW_THREADS = 64 * 8 / FW_TN, FW_WARPS = FW_THREADS / 32, FW_PER = FW_SUB / FW_WARPS;
constexpr int FW_CTAS = 3;                             // 168 registers (4 bytes spilled); four (128) spill more and are slower
constexpr int FW_STAGE_FLOATS = 8192;

__device__ __forceinline__ void copy16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ uint64_t both(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}

// The couplings of an index in pieces of at most FW_SUB: stages of `chunk` of either sign.
struct Pieces {
    int64_t c, end, split, last_end;
    int chunk, in_stage;
    bool neg;
    // the current piece
    int64_t c0;
    int n;
    bool ends_stage;

    __device__ __forceinline__ Pieces(int64_t begin, int64_t split_, int64_t end_, int chunk_)
        : c(begin), end(split_), split(split_), last_end(end_), chunk(chunk_), in_stage(0), neg(false), c0(0), n(0),
          ends_stage(false) {}
    __device__ __forceinline__ bool next() {
        n = 0;
        if (c >= end) {
            if (neg || split >= last_end) return false;
            neg = true;
            end = last_end;
        }
        int64_t m = end - c;
        if (m > chunk - in_stage) m = chunk - in_stage;
        if (m > FW_SUB) m = FW_SUB;
        c0 = c;
        n = (int)m;
        c += n;
        in_stage += n;
        ends_stage = in_stage == chunk || c == end;
        if (ends_stage) in_stage = 0;
        return true;
    }
};

__global__ void __launch_bounds__(FW_THREADS, FW_CTAS) density_f32_wide_kernel(const xrh_dens_wide_task* __restrict__ tasks, int n_tasks) {
    extern __shared__ __align__(16) float ring[];      // [FW_RING][FW_SUB][bra 64 | ket 64]
    int lo_t = 0, hi_t = n_tasks - 1;
    while (lo_t < hi_t) {
        const int mid = (lo_t + hi_t + 1) >> 1;
        if (tasks[mid].cta_begin <= (int64_t)blockIdx.x) lo_t = mid; else hi_t = mid - 1;
    }
    const xrh_dens_wide_task& T = tasks[lo_t];
    const int nb = T.nb, nk = T.nk, nbp = (nb + 3) & ~3, nkp = (nk + 3) & ~3;
    const int bj = (nk + 63) / 64, blocks = (nb + 63) / 64 * bj;
    int64_t local = (int64_t)blockIdx.x - T.cta_begin;
    const int blk = (int)(local % blocks);
    local /= blocks;
    const int64_t idx = local / T.splits;
    const int split = (int)(local - idx * T.splits);
    const int i0 = blk / bj * 64, j0 = blk % bj * 64;
    const int64_t cb0 = T.idx_ptr[idx], ce0 = T.idx_ptr[idx + 1];
    const int64_t per = (ce0 - cb0 + T.splits - 1) / T.splits;
    const int64_t c_begin = cb0 + split * per, c_end = c_begin + per < ce0 ? c_begin + per : ce0;
    double* out = T.rhoT + idx * (int64_t)nb * nk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows = nb - i0 < 64 ? nb - i0 : 64, cols = nk - j0 < 64 ? nk - j0 : 64;
    if (c_begin >= c_end) {
        if (T.splits == 1)
            for (int o = tid; o < rows * cols; o += FW_THREADS) out[(int64_t)(i0 + o / cols) * nk + j0 + o % cols] = 0.0;
        return;
    }
    int64_t c_split = cb0 + T.n_pos[idx];
    c_split = c_split < c_begin ? c_begin : (c_split > c_end ? c_end : c_split);
    const int cap = FW_STAGE_FLOATS / (nbp + nkp), chunk = cap < 64 ? (cap < 4 ? 4 : cap) : 64;

    // lanes 0 .. 15 copy the bra row of a coupling, 16 .. 31 the ket row, 16 bytes each
    const bool ket = lane >= 16;
    const int part = lane & 15;
    const bool copies = 4 * part < (ket ? nkp - j0 : nbp - i0);
    const float* src = (ket ? T.zk32 + j0 : T.zb32 + i0) + 4 * part;
    const int64_t ld = ket ? nkp : nbp;
    const int32_t* list = ket ? T.Q : T.P;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(ring);
    const uint32_t dst = base + (uint32_t)(warp * FW_PER) * (FW_ROW * 4) + (uint32_t)lane * 16u;
    // the index of one of this warp's couplings of a piece
    auto index_of = [&](const Pieces& p) {
        const int k = warp * FW_PER + (lane & (FW_PER - 1));
        return k < p.n ? __ldg(list + p.c0 + k) : 0;
    };
    auto load = [&](const Pieces& p, int mine, int slot) {
#pragma unroll
        for (int k = 0; k < FW_PER; ++k) {
            const int row = __shfl_sync(0xffffffffu, mine, (lane & 16) + k);
            if (warp * FW_PER + k < p.n && copies) copy16(dst + (uint32_t)(slot * FW_SUB + k) * (FW_ROW * 4), src + row * ld);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // 8 rows (four pairs) x FW_TN columns of the block
    constexpr int LANES_J = 64 / FW_TN;
    const int ri = (warp * (32 / LANES_J) + lane / LANES_J) * 8, rj = lane % LANES_J * FW_TN;
    uint64_t acc[4][FW_TN];                            // of the stage
    float hi[8][FW_TN], lo[8][FW_TN];
#pragma unroll
    for (int j = 0; j < FW_TN; ++j) {
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][j] = 0ull;
#pragma unroll
        for (int r = 0; r < 8; ++r) hi[r][j] = lo[r][j] = 0.f;
    }

    Pieces ahead(c_begin, c_split, c_end, chunk), now = ahead;
    ahead.next();
    int mine = index_of(ahead);
    for (int s = 0; s < FW_RING - 1; ++s) {
        load(ahead, mine, s);
        ahead.next();
        mine = index_of(ahead);
    }
    int slot = 0;
    while (now.next()) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FW_RING - 2) : "memory");
        __syncthreads();                               // this piece is there, the one before is used up
        load(ahead, mine, slot == 0 ? FW_RING - 1 : slot - 1);
        ahead.next();
        mine = index_of(ahead);
        const uint32_t at = base + (uint32_t)(slot * FW_SUB) * (FW_ROW * 4);
        const uint32_t a_at = at + (uint32_t)ri * 4u, b_at = at + 256u + (uint32_t)rj * 4u;
#pragma unroll 4
        for (int c = 0; c < now.n; ++c) {
            uint64_t a[4];
            float b[FW_TN];
#pragma unroll
            for (int q = 0; q < 2; ++q)
                asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];"
                             : "=l"(a[2 * q]), "=l"(a[2 * q + 1])
                             : "r"(a_at + (uint32_t)c * (FW_ROW * 4) + q * 16u));
#pragma unroll
            for (int q = 0; q < FW_TN / 4; ++q)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(b[4 * q]), "=f"(b[4 * q + 1]), "=f"(b[4 * q + 2]), "=f"(b[4 * q + 3])
                             : "r"(b_at + (uint32_t)c * (FW_ROW * 4) + q * 16u));
#pragma unroll
            for (int j = 0; j < FW_TN; ++j) {
                const uint64_t x = both(b[j]);
#pragma unroll
                for (int r = 0; r < 4; ++r) fma2(acc[r][j], a[r], x);
            }
        }
        if (now.ends_stage) {
            // (the sum of a stage of negative couplings is minus that of their products, rounding included)
            const uint32_t flip = now.neg ? 0x80000000u : 0u;
#pragma unroll
            for (int j = 0; j < FW_TN; ++j) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const float p = __uint_as_float((uint32_t)(acc[r >> 1][j] >> (32 * (r & 1))) ^ flip);
                    float sum, err;
                    xrh_two_sum(hi[r][j], p, sum, err);
                    hi[r][j] = sum;
                    lo[r][j] += err;
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r][j] = 0ull;
            }
        }
        slot = slot == FW_RING - 1 ? 0 : slot + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        if (ri + r >= rows) break;
        double* o = out + (int64_t)(i0 + ri + r) * nk + j0 + rj;
#pragma unroll
        for (int j = 0; j < FW_TN; ++j) {
            if (rj + j >= cols) break;
            const double v = xrh_f32_to_f64(__fadd_rn(hi[r][j], lo[r][j]));
            if (T.splits == 1) o[j] = v;
            else atomicAdd(o + j, v);
        }
    }
}

}  // namespace

extern "C" int xrh_density_accumulate_f32_wide(const xrh_dens_wide_task* tasks_dev, int n_tasks, int64_t total_ctas, void* stream) {
    if (n_tasks < 0 || total_ctas < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_ctas == 0) return XRH_OK;
    if (!tasks_dev) return XRH_ERR_ARG;
    if (total_ctas > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    const int smem = FW_RING * FW_SUB * FW_ROW * (int)sizeof(float);
    cudaFuncSetAttribute(density_f32_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    density_f32_wide_kernel<<<(unsigned)total_ctas, FW_THREADS, smem, (cudaStream_t)stream>>>(tasks_dev, n_tasks);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}
