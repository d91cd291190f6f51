// C[M, N] = A[M, K] * W[N, K]^T with float32 multiply-add on the CUDA cores: the matrix product of
// the true 32-bit path (no tensor cores, no TF32) and the fallback of the bfloat16 path for
// shapes the tensor-core kernels refuse.
//
// `gemm_f32_rows` (up to 16 rows) and `gemm_f32_tile` take float32 operands whose rows are whole 16-byte vectors (K, the strides and
// the addresses multiples of four floats); `gemm_simt_kernel` takes everything else (bfloat16 storage, other strides and widths).
//
// The order of an output's sum follows from K alone.  gemm_f32_*: K is cut into slices of 64; a slice is summed over ascending k in one
// register; four slices are added up in their order to a group's sum, and the groups in theirs, whether one block walks all groups of a
// tile or the blocks of a cluster have them side by side.  gemm_simt_kernel: ascending k = 0..K-1 inside one thread.  A row's
// result therefore does not depend on M, on the tile it falls in or on what else is in the batch.
// Weight layout [out, in] row-major, no bias, as in the reference
// (src/module/linear.zig:48-82, src/backend/cpu/linear.zig:7-28); the reference's own CUDA path
// is a bfloat16 GEMV or cuBLAS (src/backend/cuda/linear/linear.cu:22-96) and has no float32
// product.
#define LLMK_MODULE_NAME "gemm_simt"
#include "common.cuh"
#include <algorithm>

LLMK_DEFINE_LAST_ERROR()

constexpr int BN = 64, BK = 16, THREADS = 256;      // gemm_simt_kernel

// Tile BM x BN per block, 16 x 16 threads, each thread TM x 4 outputs (BM = 16 * TM).
template <typename TA, typename TW, typename TC, int TM>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(TC* C, const TA* A, const TW* W, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, int accumulate) {
    constexpr int BM = 16 * TM;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // A tile: BM x BK values, W tile: BN x BK values; consecutive threads walk along k.
        for (int idx = threadIdx.x; idx < BM * BK; idx += THREADS) {
            const int r = idx / BK, c = idx % BK;
            const int gm = m0 + r, gk = k0 + c;
            As[c][r] = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
        }
        for (int idx = threadIdx.x; idx < BN * BK; idx += THREADS) {
            const int r = idx / BK, c = idx % BK;
            const int gn = n0 + r, gk = k0 + c;
            Ws[c][r] = (gn < N && gk < K) ? to_float(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[4];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            TC* c = C + (size_t)gm * ldc + gn;
            float v = acc[i][j];
            if (accumulate) v += to_float(*c);
            *c = from_float<TC>(v);
        }
    }
}

template <typename TA, typename TW, typename TC>
static void launch(void* C, const void* A, const void* W, int M, int N, int K, long long lda, long long ldw,
                   long long ldc, int accumulate, cudaStream_t s) {
    if (M <= 16) {
        dim3 grid(ceil_div(N, BN), ceil_div(M, 16));
        gemm_simt_kernel<TA, TW, TC, 1><<<grid, THREADS, 0, s>>>((TC*)C, (const TA*)A, (const TW*)W, M, N, K, lda,
                                                                  ldw, ldc, accumulate);
    } else {
        dim3 grid(ceil_div(N, BN), ceil_div(M, 64));
        gemm_simt_kernel<TA, TW, TC, 4><<<grid, THREADS, 0, s>>>((TC*)C, (const TA*)A, (const TW*)W, M, N, K, lda,
                                                                  ldw, ldc, accumulate);
    }
}

// ------------------------------------------------------------------------------------------------------------ gemm_f32
constexpr int SLICE = 64;       // k of one slice
constexpr int GROUP = 4;        // slices of a group

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct GemmF32Params {
    float* C;
    const float* A;
    const float* W;
    long long lda, ldw, ldc;
    int M, N, K, accumulate;
    int groups, per_block;      // groups of slices of K in all, and of one block of a cluster
};

__device__ __forceinline__ void store_f32(const GemmF32Params& p, int row, int col, float v) {
    if (row >= p.M || col >= p.N) return;
    float* c = p.C + (size_t)row * p.ldc + col;
    *c = p.accumulate ? v + *c : v;
}

// The groups' sums of one tile lie in the shared memory of a cluster's blocks, group g in block g / per_block at
// parts[g % per_block][rows * cols]: each block adds up its share of the tile's outputs, in the order of the groups.
__device__ __forceinline__ void add_groups(const GemmF32Params& p, uint32_t parts, int rows_held, int rows, int cols, int m0, int n0) {
    cluster_sync_all();
    const int rank = (int)cluster_ctarank(), blocks = gridDim.y;
    for (int idx = threadIdx.x + rank * (int)blockDim.x; idx < rows * cols; idx += (int)blockDim.x * blocks) {
        float v = 0.f;
        for (int g0 = 0; g0 < p.groups; g0 += 4) {                      // four reads on their way at a time
            float x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int g = min(g0 + u, p.groups - 1);
                x[u] = cluster_ld_f32(cluster_map_shared(parts + (uint32_t)((g % p.per_block) * rows_held * cols + idx) * 4u, g / p.per_block));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (g0 + u < p.groups) v = g0 + u == 0 ? x[u] : v + x[u];
        }
        store_f32(p, m0 + idx / cols, n0 + idx % cols, v);
    }
    cluster_sync_all();                                                // no block leaves while its sums may still be read
}

// Up to 16 rows.  Bound by the stream of W: a block takes 32 rows of W and a run of slices, its warps a slice each at a time (lane = row
// of W, read from shared memory once for all rows of A): a round of slices is a group.  The first two rounds (70 KB) are asked for before
// the wait for the kernel that makes A; three blocks share an SM.  One row on W of 4096 x 1024 / 1024 x 3072 / 6144 x 1024: 5.6 / 4.9 / 7.0 us
// (the kernel it took the place of, one tile of 16 x 64 a block: 162 / 440 / 164).
constexpr int LDS_ = SLICE + 4; // floats a row of a staged slice: eight threads that read 16 bytes of neighbouring rows touch all 32 banks once
constexpr int RCOLS = 32, RWARPS = GROUP, RROUND = RWARPS * RCOLS * LDS_;   // floats of one round of slices
template <int TM>
__global__ void __launch_bounds__(RWARPS * 32) gemm_f32_rows_kernel(GemmF32Params p) {
    extern __shared__ __align__(16) float sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * RCOLS;
    const int g_beg = blockIdx.y * p.per_block, rounds = min(p.per_block, p.groups - g_beg);
    const int k_beg = g_beg * GROUP * SLICE;
    const int count = min(rounds * GROUP, ceil_div(p.K - k_beg, SLICE));      // slices of this block
    const int k_width = p.per_block * GROUP * SLICE + 4;
    float* Ws = sm;                                                    // [2][RWARPS][RCOLS][LDS_]
    float* As = Ws + 2 * RROUND;                                       // [TM][k_width]
    float* parts = As + TM * k_width;                                  // [per_block][TM][RCOLS]: the groups' sums
    float* mine = parts + p.per_block * TM * RCOLS;                    // [2][GROUP][TM][RCOLS]: a round's slices
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
    // a warp fetches the slice that it will use itself: no other warp is waited for
    auto load_w = [&](int round) {
        const int i = round * RWARPS + warp;
        if (i < count) {
            const int k0 = k_beg + i * SLICE;
            const uint32_t dst = base + (uint32_t)(((round & 1) * RWARPS + warp) * RCOLS * LDS_) * 4u;
#pragma unroll 4
            for (int idx = lane; idx < RCOLS * (SLICE / 4); idx += 32) {
                const int r = idx / (SLICE / 4), c = idx % (SLICE / 4);
                const bool ok = n0 + r < p.N && k0 + 4 * c < p.K;
                cp_async16_zfill(dst + (uint32_t)(r * LDS_ + 4 * c) * 4u, ok ? p.W + (size_t)(n0 + r) * p.ldw + k0 + 4 * c : p.W, ok);
            }
        }
        cp_async_commit();
    };
    pdl_launch_dependents();
    load_w(0);
    load_w(1);
    pdl_wait();
    {
        const int vecs = count * (SLICE / 4);
        for (int idx = threadIdx.x; idx < TM * vecs; idx += blockDim.x) {
            const int r = idx / vecs, c = idx % vecs;
            const bool ok = r < p.M && k_beg + 4 * c < p.K;
            cp_async16_zfill(base + (uint32_t)(2 * RROUND + r * k_width + 4 * c) * 4u, ok ? p.A + (size_t)r * p.lda + k_beg + 4 * c : p.A, ok);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
    }
    for (int round = 0; round < rounds; ++round) {
        const int i = round * RWARPS + warp;
        cp_async_wait<1>();
        __syncwarp();
        if (i < count) {
            const float* w = Ws + ((round & 1) * RWARPS + warp) * RCOLS * LDS_ + lane * LDS_;
            const float* a = As + i * SLICE;
            float acc[TM];
#pragma unroll
            for (int m = 0; m < TM; ++m) acc[m] = 0.f;
#pragma unroll 4
            for (int k = 0; k < SLICE; k += 4) {
                const float4 b = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
                for (int m = 0; m < TM; ++m) {
                    const float4 x = *reinterpret_cast<const float4*>(a + m * k_width + k);
                    acc[m] = fmaf(x.x, b.x, acc[m]);
                    acc[m] = fmaf(x.y, b.y, acc[m]);
                    acc[m] = fmaf(x.z, b.z, acc[m]);
                    acc[m] = fmaf(x.w, b.w, acc[m]);
                }
            }
#pragma unroll
            for (int m = 0; m < TM; ++m) mine[(((round & 1) * GROUP + warp) * TM + m) * RCOLS + lane] = acc[m];
        }
        __syncthreads();                     // (the buffer of two rounds ago is free: everyone has passed the round between)
        load_w(round + 2);
        const int held = min(GROUP, count - round * GROUP);
        for (int idx = threadIdx.x; idx < TM * RCOLS; idx += blockDim.x) {
            const float* x = mine + (round & 1) * GROUP * TM * RCOLS + idx;
            float v = x[0];
            for (int u = 1; u < held; ++u) v += x[u * TM * RCOLS];
            parts[round * TM * RCOLS + idx] = v;
        }
    }
    cp_async_wait<0>();
    add_groups(p, base + (uint32_t)(2 * RROUND + TM * k_width) * 4u, TM, min(TM, p.M), RCOLS, 0, n0);
}

// More rows.  A block of 16 x 8 threads makes (8 TM) x (16 TN) outputs; thread (tx, ty) has rows ty + 8 i and columns tx + 16 j.  Both
// operands lie in shared memory as their rows are in memory, half a slice a stage, in a ring of three.  What bounds it: the issue of
// multiply-adds from three warps a scheduler (34.8 TFLOP/s at 512 rows on 6144 x 1024, where a loop of nothing but independent
// multiply-adds reaches 60; the kernel with 64 x 64 tiles and value-wise copies that it took the place of reached 17).
// fma.rn.f32x2 (34.9), 8 x 8 outputs a thread (25.8) and 4 x 4 (34.2) were measured there too.
constexpr int TBK = SLICE / 2, TLD = TBK + 4, TTHREADS = 128, TSTAGES = 3;
template <int TM, int TN>
struct TileF32 {
    static constexpr int BM = 8 * TM, BN_ = 16 * TN, STAGE = (BM + BN_) * TLD;
    static constexpr size_t RING = (size_t)TSTAGES * STAGE * sizeof(float);
};
template <int TM, int TN>
__global__ void __launch_bounds__(TTHREADS, 3) gemm_f32_tile_kernel(GemmF32Params p) {
    using L = TileF32<TM, TN>;
    constexpr int STAGES = TSTAGES, TCOLS = L::BN_;
    extern __shared__ __align__(16) float sm[];
    float* parts = sm + STAGES * L::STAGE;                             // [per_block][BM][TCOLS] where groups are side by side, else the running sum [BM][TCOLS]
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int n0 = blockIdx.x * TCOLS, m0 = blockIdx.z * L::BM;
    const int g_beg = blockIdx.y * p.per_block, k_beg = g_beg * GROUP * SLICE;
    const int steps = 2 * min(min(p.per_block, p.groups - g_beg) * GROUP, ceil_div(p.K - k_beg, SLICE));
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
    // a thread's vectors of a stage: rows r0 + 16 i, column c of 8
    const int r0 = threadIdx.x / (TBK / 4), c4 = 4 * (threadIdx.x % (TBK / 4));
    auto load_rows = [&](int step, const float* src, long long ld, int row0, int rows, int limit, int offset) {
        const uint32_t dst = base + (uint32_t)((step % STAGES) * L::STAGE + offset + r0 * TLD + c4) * 4u;
        const int k = k_beg + step * TBK + c4;
        const float* at = src + (size_t)(row0 + r0) * ld + k;
#pragma unroll
        for (int i = 0; i < rows / 16; ++i) {
            const bool ok = row0 + r0 + 16 * i < limit && k < p.K;
            cp_async16_zfill(dst + (uint32_t)(16 * i * TLD) * 4u, ok ? at + (size_t)(16 * i) * ld : src, ok);
        }
    };
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) load_rows(s, p.W, p.ldw, n0, TCOLS, p.N, L::BM * TLD);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_rows(s, p.A, p.lda, m0, L::BM, p.M, 0);
        cp_async_commit();
    }
    float acc[TM][TN], total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.f;
    const bool side_by_side = gridDim.y > 1;
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                               // the stage is filled, and the one before it is free
        if (step + STAGES - 1 < steps) {
            load_rows(step + STAGES - 1, p.W, p.ldw, n0, TCOLS, p.N, L::BM * TLD);
            load_rows(step + STAGES - 1, p.A, p.lda, m0, L::BM, p.M, 0);
        }
        cp_async_commit();
        const float* As = sm + (step % STAGES) * L::STAGE + ty * TLD;
        const float* Ws = sm + (step % STAGES) * L::STAGE + (L::BM + tx) * TLD;
#pragma unroll
        for (int kk = 0; kk < TBK; kk += 4) {
            float4 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(Ws + 16 * j * TLD + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(As + 8 * i * TLD + kk);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
                }
            }
        }
        if (step & 1) {                                                // a slice is done, perhaps a group
            const int slice = step / 2, group = slice / GROUP;
            const bool first = slice % GROUP == 0, last = slice % GROUP == GROUP - 1 || step + 1 == steps;
            float* at = parts + (side_by_side ? group * L::BM * TCOLS : 0) + ty * TCOLS + tx;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    total[i][j] = first ? acc[i][j] : total[i][j] + acc[i][j];
                    acc[i][j] = 0.f;
                    if (last) {
                        float* to = at + 8 * i * TCOLS + 16 * j;       // (this thread's own place)
                        if (side_by_side || group == 0) *to = total[i][j];
                        else *to = *to + total[i][j];
                    }
                }
        }
    }
    if (side_by_side) {
        add_groups(p, base + (uint32_t)(STAGES * L::STAGE) * 4u, L::BM, min(L::BM, p.M - m0), TCOLS, m0, n0);
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) store_f32(p, m0 + ty + 8 * i, n0 + tx + 16 * j, parts[(ty + 8 * i) * TCOLS + tx + 16 * j]);
}

constexpr size_t F32_SMEM_MAX = 200 * 1024;
template <void (*KERNEL)(GemmF32Params)>
static int launch_f32(const GemmF32Params& p, int tiles_n, int blocks, int tiles_m, size_t smem, cudaStream_t s) {
    // one bound for every size of this kernel, set once: launches recorded into graphs keep theirs
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F32_SMEM_MAX);
        if (e != cudaSuccess) LLMK_FAIL("gemm_simt: cannot raise shared memory to %zu: %s", F32_SMEM_MAX, cudaGetErrorString(e));
        configured = true;
    }
    LLMK_CHECK_LAUNCH_RC("gemm_simt", llmk_launch_cluster(KERNEL, dim3(tiles_n, blocks, tiles_m), dim3(RWARPS * 32), smem, s, true, (unsigned)blocks, p));
    return LLMK_OK;
}

static size_t rows_smem(int TM, int per_block) {
    return ((size_t)2 * RROUND + (size_t)TM * (per_block * GROUP * SLICE + 4) + (size_t)(per_block + 2 * GROUP) * TM * RCOLS) * sizeof(float);
}
static int blocks_by_smem(size_t smem, int most) {
    const int fit = (int)((size_t)(226 * 1024) / (smem + 1024));
    return std::max(1, std::min(fit, most));
}

// Few rows: as many blocks a tile as still find a place at once, three an SM (fewer where their shared memory is larger).
template <int TM>
static int launch_rows(GemmF32Params p, cudaStream_t s) {
    const int tiles = ceil_div(p.N, RCOLS), sms = device_sm_count();
    int best = 0;
    double best_cost = 1e30;
    for (int c = 1; c <= 8 && c <= p.groups; ++c) {
        const int per = ceil_div(p.groups, c);
        const size_t smem = rows_smem(TM, per);
        if (ceil_div(p.groups, per) != c || smem > F32_SMEM_MAX) continue;
        const int places = sms * blocks_by_smem(smem, 3);
        const double cost = (double)((tiles * (long long)c + places - 1) / places) * (per + 1.0);
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = c;
        }
    }
    if (best == 0) return -1;
    p.per_block = ceil_div(p.groups, best);
    return launch_f32<gemm_f32_rows_kernel<TM>>(p, tiles, best, 1, rows_smem(TM, p.per_block), s);
}

// More rows: the groups that an SM has to walk, with the cost of filling a ring (and of the exchange) for each of its blocks; one block
// alone on an SM keeps it about two thirds busy.
template <int TM, int TN>
static int launch_tile(GemmF32Params p, cudaStream_t s) {
    using L = TileF32<TM, TN>;
    const long long tiles = (long long)ceil_div(p.N, L::BN_) * ceil_div(p.M, L::BM);
    const int sms = device_sm_count();
    const size_t part = (size_t)L::BM * L::BN_ * sizeof(float);
    int best = 1;
    double best_cost = 1e30;
    for (int c = 1; c <= 8 && c <= p.groups; ++c) {
        const int per = ceil_div(p.groups, c);
        const size_t smem = L::RING + (c > 1 ? per : 1) * part;
        if (ceil_div(p.groups, per) != c || smem > F32_SMEM_MAX) continue;
        const long long each = (tiles * c + sms - 1) / sms;
        const int resident = (int)std::min<long long>(each, blocks_by_smem(smem, 3));
        const double busy = resident == 1 ? 1.5 : resident == 2 ? 1.1 : 1.0;
        const double cost = each * (per + (c > 1 ? 0.35 : 0.15)) * busy;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = c;
        }
    }
    p.per_block = ceil_div(p.groups, best);
    return launch_f32<gemm_f32_tile_kernel<TM, TN>>(p, ceil_div(p.N, L::BN_), best, ceil_div(p.M, L::BM), L::RING + (best > 1 ? p.per_block : 1) * part, s);
}

static int gemm_f32(void* C, const void* A, const void* W, int M, int N, int K, long long lda, long long ldw, long long ldc,
                    int accumulate, cudaStream_t s) {
    GemmF32Params p;
    p.C = (float*)C; p.A = (const float*)A; p.W = (const float*)W;
    p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.accumulate = accumulate;
    p.groups = ceil_div(K, GROUP * SLICE);
    p.per_block = p.groups;
    int rc = -1;
    if (M == 1) rc = launch_rows<1>(p, s);
    else if (M == 2) rc = launch_rows<2>(p, s);
    else if (M <= 4) rc = launch_rows<4>(p, s);
    else if (M <= 8) rc = launch_rows<8>(p, s);
    else if (M <= 16) rc = launch_rows<16>(p, s);
    if (rc != -1) return rc;                    // -1: K too wide for the few-rows kernel's shared memory
    // 32 x 128 outputs a block up to 128 rows, 64 x 64 beyond (us, 32 x 128 against 64 x 64: 64 rows on 4096 x 1024 24.8 / 30.3,
    // 128 on 1024 x 2048 24.1 / 29.3, 512 on 4096 x 1024 175 / 133 and on 1024 x 3072 130 / 119)
    return M <= 128 ? launch_tile<4, 8>(p, s) : launch_tile<8, 4>(p, s);
}

// dtype: storage of A and W; out_dtype: storage of C (float32 output of a bfloat16 product is
// what the logits use).  accumulate != 0 adds into C.
LLMK_EXPORT int llmk_gemm_simt(void* C, const void* A, const void* W, int M, int N, int K, long long lda,
                               long long ldw, long long ldc, int accumulate, int dtype, int out_dtype,
                               void* stream) {
    if (M <= 0 || N <= 0) return LLMK_OK;
    if (K <= 0) LLMK_FAIL("gemm_simt: K=%d", K);
    if (lda < K || ldw < K || ldc < N) LLMK_FAIL("gemm_simt: strides lda=%lld ldw=%lld ldc=%lld too small for K=%d N=%d", lda, ldw, ldc, K, N);
    if (ceil_div(M, 16) > 65535) LLMK_FAIL("gemm_simt: M=%d too large", M);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LLMK_F32 && out_dtype == LLMK_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && host_aligned16(A) && host_aligned16(W))
        return gemm_f32(C, A, W, M, N, K, lda, ldw, ldc, accumulate, s);
    if (dtype == LLMK_F32 && out_dtype == LLMK_F32)
        launch<float, float, float>(C, A, W, M, N, K, lda, ldw, ldc, accumulate, s);
    else if (dtype == LLMK_BF16 && out_dtype == LLMK_BF16)
        launch<bf16, bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, accumulate, s);
    else if (dtype == LLMK_BF16 && out_dtype == LLMK_F32)
        launch<bf16, bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, accumulate, s);
    else
        LLMK_FAIL("gemm_simt: unsupported dtypes in=%d out=%d", dtype, out_dtype);
    LLMK_CHECK_LAUNCH("gemm_simt");
    return LLMK_OK;
}
