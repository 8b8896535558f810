// Layout passes of the three-index density blocks (sm_103a): bound by memory, so each block is read
// once and everything derived from it is written from there.
//
// The coupling-list kernels work on [K][R] rows (K = N^3 operator index tuples f = (p, q, r), R = nb nk
// state pairs); the contractions want rho [R][K], and a block of the creation side is the
// annihilation side's with bra and ket swapped and the operator indices reversed,
//     rho_m[(j, i)][(r, q, p)] = rho[(i, j)][(p, q, r)].
//   expand:  rhoT -> rho, rho_m; rows with q > r are minus the rows (p, r, q) where the operators q, r
//            anticommute and the kernels ran over q < r only
//   collect: dE/drho, dE/drho_m -> d[K][R] = transpose(dE/drho) + their sum over the same map
// A CTA takes one q and `cols` state pairs: all (p, r) of them in shared memory, so that rho is read or
// written along r, rho_m along p and the K rows along the state pairs.
// Consecutive CTAs take consecutive q, so the rows read a second time (q, r swapped) come from L2.
// Separate passes (fill the rows, transpose, mirror by planes) move 5 blocks through memory against 2.5
// for expand (1.8 ms against 0.76 ms at the size below) and 5 against 3 for collect (1.7 against 0.91).
#include "xrh_common.cuh"

namespace {

constexpr int DL_THREADS = 256, DL_WARPS = DL_THREADS / 32;

// A tile is [column][p][r]; odd strides of p and of the columns: no direction has bank conflicts.
__host__ __device__ __forceinline__ int p_stride(int N) { return N | 1; }
__host__ __device__ __forceinline__ int c_stride(int N) { return (N * p_stride(N)) | 1; }

// State pairs per CTA, for `tiles` tiles: 4, one sector of a K row.  Many small CTAs an SM overlap their
// loads and stores; 8 or 16 pairs read longer pieces but are slower (two blocks of 60 x 60 states, N = 28:
// expand 0.76 / 0.91 / 1.01 ms, collect 0.91 / 0.91 / 1.22).  2 where 4 would leave no second CTA.
// 0: N out of range.
__host__ __device__ __forceinline__ int tile_cols(int N, int tiles) {
    if (N < 1 || N > 64) return 0;
    return (size_t)4 * tiles * c_stride(N) * sizeof(double) <= 112 * 1024 ? 4 : 2;
}
__host__ __device__ __forceinline__ size_t tile_bytes(int N, int tiles) {
    return (size_t)tile_cols(N, tiles) * tiles * c_stride(N) * sizeof(double);
}

// 8 bytes to shared memory: every load of a CTA in flight at once, without registers
__device__ __forceinline__ void copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

struct Tile {
    int64_t c0;                   // first state pair
    int q, cols, n;               // operator index, columns of the tile, of them in range
};

__device__ __forceinline__ Tile tile_at(const xrh_layout_task& T, int64_t local, int tiles) {
    Tile t;
    t.cols = tile_cols(T.N, tiles);
    const int64_t chunk = local / T.N;
    t.q = (int)(local - chunk * T.N);
    t.c0 = chunk * t.cols;
    const int64_t left = (int64_t)T.nb * T.nk - t.c0;
    t.n = left < t.cols ? (int)left : t.cols;
    return t;
}

// f(p, r, c) for every K row (p, q, r) and column c of the tile, lanes along c.
template <typename F>
__device__ __forceinline__ void along_columns(int N, const Tile& t, F&& f) {
    const int c = threadIdx.x % t.cols, step = DL_THREADS / t.cols;
    int e = threadIdx.x / t.cols, p = e / N, r = e - p * N;
    if (c >= t.n) return;
#pragma unroll 4
    while (p < N) {
        f(p, r, c);
        r += step;
        while (r >= N) {
            r -= N;
            ++p;
        }
    }
}

// f(row, c, outer, inner) with row = base(c), a warp per (column, outer index), lanes along the inner one.
template <typename B, typename F>
__device__ __forceinline__ void along_inner(int N, const Tile& t, B&& base, F&& f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = 0; c < t.n; ++c) {
        auto row = base(c);
#pragma unroll 4
        for (int o = warp; o < N; o += DL_WARPS)
            for (int in = lane; in < N; in += 32) f(row, c, o, in);
    }
}

__device__ __forceinline__ const xrh_layout_task& find_layout(const xrh_layout_task* __restrict__ tasks, int n_tasks, int64_t cta) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].cta_begin <= cta) lo = mid; else hi = mid - 1;
    }
    return tasks[lo];
}

// row (j, i) of the mirrored block for the state pair (i, j)
__device__ __forceinline__ int64_t mirrored(const xrh_layout_task& T, int64_t pair) {
    const int64_t i = pair / T.nk;
    return (pair - i * T.nk) * T.nb + i;
}

template <bool COLLECT>
__global__ void __launch_bounds__(DL_THREADS) density_layout_kernel(const xrh_layout_task* __restrict__ tasks, int n_tasks, int N) {
    extern __shared__ double tile[];                   // [column][p][r]
    const xrh_layout_task& T = find_layout(tasks, n_tasks, blockIdx.x);
    if (T.N != N) return;                              // (the host checks)
    const Tile t = tile_at(T, (int64_t)blockIdx.x - T.cta_begin, COLLECT ? 2 : 1);
    const int W = p_stride(N), S = c_stride(N);
    const int nn = N * N;
    const int64_t R = (int64_t)T.nb * T.nk, K = (int64_t)nn * N;
    auto at = [&](int p, int r, int c) -> double& { return tile[c * S + p * W + r]; };
    double* rows = T.rows + t.c0;
    auto rho_row = [&](int c) { return T.rho + (t.c0 + c) * K + t.q * N; };
    auto mirror_row = [&](int c) { return T.mirror + mirrored(T, t.c0 + c) * K + t.q * N; };
    if constexpr (!COLLECT) {
        const bool anti = T.anti != 0;
        along_columns(N, t, [&](int p, int r, int c) {
            const bool swap = anti && t.q > r;
            copy8(&at(p, r, c), rows + (int64_t)(p * nn + (swap ? r * N + t.q : t.q * N + r)) * R + c);
        });
        copies_done();
        auto value = [&](int p, int r, int c) { return anti && t.q > r ? -at(p, r, c) : at(p, r, c); };
        along_inner(N, t, rho_row, [&](double* row, int c, int p, int r) { row[p * nn + r] = value(p, r, c); });
        if (T.mirror) {
            along_inner(N, t, mirror_row, [&](double* row, int c, int r, int p) { row[r * nn + p] = value(p, r, c); });
        }
    } else {
        double* other = tile + t.cols * S;
        along_inner(N, t, rho_row, [&](double* row, int c, int p, int r) { copy8(&at(p, r, c), row + p * nn + r); });
        if (T.mirror) {
            along_inner(N, t, mirror_row, [&](double* row, int c, int r, int p) { copy8(other + c * S + p * W + r, row + r * nn + p); });
        }
        copies_done();
        along_columns(N, t, [&](int p, int r, int c) {
            double v = at(p, r, c);
            if (T.mirror) v += other[c * S + p * W + r];
            rows[(int64_t)(p * nn + t.q * N + r) * R + c] = v;
        });
    }
}

}  // namespace

extern "C" int64_t xrh_density_layout_ctas(int collect, int N, int64_t pairs) {
    const int c = tile_cols(N, collect ? 2 : 1);
    return c && pairs > 0 ? N * ((pairs + c - 1) / c) : 0;
}

extern "C" int xrh_density_layout_grouped(int collect, const xrh_layout_task* tasks_dev, int n_tasks, int64_t total_ctas,
                                          int N, void* stream) {
    if (n_tasks < 0 || total_ctas < 0 || N < 0) return XRH_ERR_ARG;
    if (n_tasks == 0 || total_ctas == 0) return XRH_OK;
    if (!tasks_dev || N < 1) return XRH_ERR_ARG;
    if (N > 64 || total_ctas > 0x7fffffffLL) return XRH_ERR_CAPACITY;
    const size_t smem = tile_bytes(N, collect ? 2 : 1);
    auto kernel = collect ? density_layout_kernel<true> : density_layout_kernel<false>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<(unsigned)total_ctas, DL_THREADS, smem, (cudaStream_t)stream>>>(tasks_dev, n_tasks, N);
    XRH_CHECK_LAUNCH();
    return XRH_OK;
}
