// The products of a mixture of experts, out[m, :] = act(X[m, :] * W[expert of row m]^T) in bfloat16, on the 5th-generation tensor cores of
// sm_100a with the operands swapped: W's rows are the MMA's rows, the experts' rows of X its columns, so that an expert's rows are padded to
// a multiple of 32 and not of 128.
//
// X's rows are sorted by expert; `spans` (csrc/moe.cu, on the device: the launch has the same shape whatever the experts' counts are) lists
// runs of at most 256 rows of one expert, an expert's rows cut evenly.  A pair of blocks (a cluster of two, `tcgen05.mma.cta_group::2`) computes
// 256 rows of W by one span, one such tile after the other; 320 threads a block:
//   warp 0     TMA producer: per step of 64 along K this block's 128 rows of W and its half of the span's rows (boxes of 128, 64, 32 and
//              16 rows), in a ring of six stages; no multicast, every block loads what it holds.
//   warp 1     of rank 0 issues the MMAs (columns: the span's rows rounded up to 32), two accumulators of 256 columns in turn
//   warps 2-9  epilogue: a lane is a row of W, a column of tensor memory a row of X; two warps share 32 rows of W and take runs of 32 columns in
//              turn.  Gated units (W interleaves gate and up rows in groups of 16: the other of a pair is 16 lanes away) and relu squared
//              are applied here, in float32; 32 x 32 results turn round in shared memory and leave 16 bytes a thread.
//
// What bounds it: W from memory (32 experts of gate and up [2048, 2048]: 268 MB, 41 us at the copy rate) and, where many rows share it, what the
// SMs pull from L2: a block pulls 16 KB of W and at most 16 KB of X per step for 128 x (at most) 256 outputs.
//
// Every wait is bounded; a wait that gives up raises `*error_flag`.
#define LLMK_MODULE_NAME "gemm_grouped"
#include "common.cuh"
#include "tcgen05.cuh"

#include <algorithm>

LLMK_DEFINE_LAST_ERROR()

namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16, THREADS = 320;
constexpr int SPAN = 256;           // rows of X a tile has at the most: columns of an accumulator
constexpr int STAGES = 6;
constexpr int W_BYTES = BM * BK * 2, STAGE_BYTES = W_BYTES + SPAN / 2 * BK * 2;
constexpr int SLAB = 32 * 32 * 4;                       // an epilogue warp's 32 x 32 results on their way out
constexpr int SLAB_OFF = STAGES * STAGE_BYTES, BAR_OFF = SLAB_OFF + 8 * SLAB, NUM_BARS = 2 * STAGES + 4;
constexpr int SMEM = BAR_OFF + NUM_BARS * 8 + 16 + 1024;        // + alignment slack

enum { ACT_NONE = 0, ACT_RELU2 = 1, ACT_SILU_GLU = 2, ACT_CLAMPED_GLU = 3 };
constexpr bool is_glu(int act) { return act == ACT_SILU_GLU || act == ACT_CLAMPED_GLU; }

struct Params {
    const int4* spans;              // [0].x: how many; then (expert, first row, rows, columns of the MMA) each
    int N, K;                       // of an expert's matrix
    long long ldc;
    float alpha, limit;
    int* error_flag;
};

// gate and up of the same unit (see act_rows in csrc/rowwise.cu)
template <int ACT>
__device__ __forceinline__ float glu(float g, float u, float alpha, float limit) {
    if constexpr (ACT == ACT_CLAMPED_GLU) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return __fdividef(g, 1.f + __expf(-alpha * g)) * (u + 1.f);
    }
    return __fdividef(g, 1.f + __expf(-g)) * u;
}

template <typename TC, int ACT>
__global__ void __launch_bounds__(THREADS)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x128, const __grid_constant__ CUtensorMap map_x64,
                    const __grid_constant__ CUtensorMap map_x32, const __grid_constant__ CUtensorMap map_x16, TC* C, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;         // 2
    uint64_t* acc_empty = bars + 2 * STAGES + 2;    // 2, sixteen arrivals each (one per epilogue warp of either block)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same for all lanes, and known to be)
    const uint32_t rank = cluster_ctarank();
    const int unit = (int)blockIdx.x / 2, units = (int)gridDim.x / 2;
    const int num_kb = (p.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(tc::smem_u32(&full[s]), 1);
            tc::mbar_init(tc::smem_u32(&empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(tc::smem_u32(&acc_full[i]), 1);
            tc::mbar_init(tc::smem_u32(&acc_empty[i]), 16);
        }
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_w);
        tc::prefetch_tensormap(&map_x128);
        tc::prefetch_tensormap(&map_x64);
        tc::prefetch_tensormap(&map_x32);
        tc::prefetch_tensormap(&map_x16);
    }
    if (warp == 1) {
        tc::tmem_alloc_pair(tc::smem_u32(tmem_slot), 2 * SPAN);
        tc::tmem_relinquish_pair();
    }
    tc::tc_fence_before_sync();
    __syncwarp();
    cluster_sync_all();         // both blocks' barriers and tensor memory are ready before either uses the other's
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();    // (behind the allocation: the next kernel's blocks must not get their tensor memory first)
    pdl_wait();                 // the spans and X come from kernels before this one
    const int n_spans = p.spans[0].x;
    const int items = n_spans * ((p.N + 2 * BM - 1) / (2 * BM));

    // The whole warp walks the loops of both issuing roles and one lane issues: what the instructions are given is then known to be the same for
    // all lanes and kept where they read it.
    if (warp == 0) {
        {
            const bool issues = tc::elect_one();
            uint32_t it = 0;
            bool ok = true;
            for (int item = unit; item < items && ok; item += units) {
                const int4 span = p.spans[1 + item % n_spans];
                const int w_row = span.x * p.N + item / n_spans * 2 * BM + (int)rank * BM;
                const int rows = span.w / 2, x_row = span.y + (int)rank * rows;     // this block's half of the span: a multiple of 16 rows
                const uint32_t bytes = 2u * (uint32_t)(W_BYTES + rows * BK * 2);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!tc::mbar_wait_warp(tc::smem_u32(&empty[s]), ((it / STAGES) & 1) ^ 1, abort_flag)) { ok = false; break; }
                    if (!issues) continue;
                    // both blocks' bytes are counted on rank 0's barrier
                    if (rank == 0) tc::mbar_expect_tx(tc::smem_u32(&full[s]), bytes);
                    const uint32_t bar = cluster_map_shared(tc::smem_u32(&full[s]), 0), dst = tc::smem_u32(smem + s * STAGE_BYTES);
                    tc::tma_load_2d_pair(dst, &map_w, bar, kb * BK, w_row);
                    // rows <= 128 in boxes of the powers of two they are made of
                    if (rows & 128) tc::tma_load_2d_pair(dst + W_BYTES, &map_x128, bar, kb * BK, x_row);
                    if (rows & 64) tc::tma_load_2d_pair(dst + W_BYTES, &map_x64, bar, kb * BK, x_row);
                    if (rows & 32) tc::tma_load_2d_pair(dst + W_BYTES + (rows & 64) * 128, &map_x32, bar, kb * BK, x_row + (rows & 64));
                    if (rows & 16) tc::tma_load_2d_pair(dst + W_BYTES + (rows & 96) * 128, &map_x16, bar, kb * BK, x_row + (rows & 96));
                }
            }
            // the MMA's last arrivals on `empty` come from the other block and have to land while this block's memory is still its own
            for (uint32_t k = it > (uint32_t)STAGES ? it - STAGES : 0; k < it && ok; ++k)
                ok = tc::mbar_wait_warp(tc::smem_u32(&empty[k % STAGES]), (k / STAGES) & 1, abort_flag);
            if (*abort_flag && rank == 0) {
                // let the copies that are in flight land before the block's memory is given up (rank 0's barriers count both blocks')
                for (uint32_t k = it > (uint32_t)STAGES ? it - STAGES : 0; k < it; ++k) {
                    const long long t0 = clock64();
                    while (!tc::mbar_try_wait(tc::smem_u32(&full[k % STAGES]), (k / STAGES) & 1) &&
                           clock64() - t0 < tc::WAIT_LIMIT_CYCLES) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const bool issues = tc::elect_one();
            const uint64_t ring_desc = tc::smem_desc_sw128(tc::smem_u32(smem));
            uint32_t it = 0;
            bool ok = true;
            int tile_iter = 0;
            for (int item = unit; item < items && ok; item += units, ++tile_iter) {
                const uint32_t idesc = tc::idesc_bf16_f32(2 * BM, p.spans[1 + item % n_spans].w);
                const int buf = tile_iter & 1;
                ok = tc::mbar_wait_warp(tc::smem_u32(&acc_empty[buf]), ((tile_iter / 2) & 1) ^ 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after_sync();
                const uint32_t acc = tmem_base + (uint32_t)(buf * SPAN);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = tc::mbar_wait_warp(tc::smem_u32(&full[s]), (it / STAGES) & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                    if (!issues) continue;
                    const uint64_t w_desc = ring_desc + (uint64_t)((s * STAGE_BYTES) >> 4);
                    const uint64_t x_desc = w_desc + (uint64_t)(W_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        const uint64_t at = (uint64_t)((k * UMMA_K * 2) >> 4);
                        tc::mma_bf16_ss_pair(acc, w_desc + at, x_desc + at, idesc, kb != 0 || k != 0);
                    }
                    tc::mma_commit_pair(tc::smem_u32(&empty[s]), (uint16_t)3);
                }
                if (ok && issues) tc::mma_commit_pair(tc::smem_u32(&acc_full[buf]), (uint16_t)3);
            }
        }
    } else {
        // warp w may touch tensor-memory lanes 32 * (w % 4) .. + 31
        const int quarter = warp & 3, turn = (warp - 2) >> 2;
        constexpr int COLS = is_glu(ACT) ? 16 : 32;             // results of 32 rows of W
        constexpr int VEC = 16 / (int)sizeof(TC), LANES = COLS / VEC;        // vectors of a row of X
        TC* slab = reinterpret_cast<TC*>(smem + SLAB_OFF + (warp - 2) * SLAB);       // [32 rows of X][COLS]
        const int n_out = is_glu(ACT) ? p.N / 2 : p.N;
        const bool whole = p.ldc % VEC == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
        bool ok = true;
        int tile_iter = 0;
        for (int item = unit; item < items && ok; item += units, ++tile_iter) {
            const int4 span = p.spans[1 + item % n_spans];
            const int n0 = item / n_spans * 2 * BM + (int)rank * BM + quarter * 32;      // this warp's first row of the expert's W
            const int j0 = is_glu(ACT) ? n0 / 2 : n0, j_end = min(j0 + COLS, n_out);
            const int buf = tile_iter & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&acc_full[buf]), (tile_iter / 2) & 1, abort_flag));
            if (!ok) break;
            tc::tc_fence_after_sync();
            const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * SPAN);
            if (n0 < p.N) {                                     // uniform over the warp
#pragma unroll 1
                for (int c0 = turn * 32; c0 < span.z; c0 += 64) {
                    uint32_t r[32];
                    __syncwarp();                               // (the slab's results before these have been read)
                    tc::tmem_ld_32x32_wait(acc + (uint32_t)c0, r);
                    if constexpr (is_glu(ACT)) {
                        // lanes 0 .. 15 are gates, 16 .. 31 the matching ups; of two rows of X the lower lanes finish the first, the upper ones the second
                        const bool up = lane >= 16;
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float a = __uint_as_float(r[i]), b = __uint_as_float(r[i + 1]);
                            const float other = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
                            const float o = up ? glu<ACT>(other, b, p.alpha, p.limit) : glu<ACT>(a, other, p.alpha, p.limit);
                            slab[(i + (up ? 1 : 0)) * COLS + (lane & 15)] = from_float<TC>(o);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            float v = __uint_as_float(r[i]);
                            if constexpr (ACT == ACT_RELU2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
                            slab[i * COLS + lane] = from_float<TC>(v);
                        }
                    }
                    __syncwarp();
                    const int rows = min(32, span.z - c0);
                    TC* dst = C + (size_t)(span.y + c0) * p.ldc + j0;
#pragma unroll
                    for (int idx = lane; idx < 32 * LANES; idx += 32) {
                        const int m = idx / LANES, c = idx % LANES * VEC;
                        if (m >= rows || j0 + c >= j_end) continue;
                        if (whole && j0 + c + VEC <= j_end)
                            *reinterpret_cast<uint4*>(dst + (size_t)m * p.ldc + c) = *reinterpret_cast<const uint4*>(slab + m * COLS + c);
                        else
                            for (int u = 0; u < VEC && j0 + c + u < j_end; ++u) dst[(size_t)m * p.ldc + c + u] = slab[m * COLS + c + u];
                    }
                }
            }
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster(cluster_map_shared(tc::smem_u32(&acc_empty[buf]), 0));
        }
    }
    tc::tc_fence_before_sync();
    __syncwarp();
    cluster_sync_all();         // neither block leaves, or frees tensor memory, while the other may still use it
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc_pair(tmem_base, 2 * SPAN);
    }
    if (threadIdx.x == 0 && *abort_flag && p.error_flag) atomicExch(p.error_flag, 1);
}

template <typename TC, int ACT>
int launch(const CUtensorMap& mw, const CUtensorMap (&mx)[4], void* C, const Params& p, int most_items, cudaStream_t s) {
    auto kernel = gemm_grouped_kernel<TC, ACT>;
    static bool configured = false;   // per instantiation
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) LLMK_FAIL("gemm_grouped: cannot raise shared memory to %d: %s", SMEM, cudaGetErrorString(e));
        configured = true;
    }
    const int pairs = std::max(1, std::min(most_items, device_sm_count() / 2));
    LLMK_CHECK_LAUNCH_RC("gemm_grouped", llmk_launch_clusters(kernel, dim3(2 * pairs), dim3(THREADS), SMEM, s, true, dim3(2, 1, 1), mw, mx[0], mx[1],
                                                              mx[2], mx[3], (TC*)C, p));
    return LLMK_OK;
}

}  // namespace

// 1 if the kernel takes these operands.
LLMK_EXPORT int llmk_gemm_grouped_usable(const void* X, const void* W, int N, int K, long long ldx) {
    return N > 0 && K > 0 && K % 8 == 0 && ldx % 8 == 0 && host_aligned16(X) && host_aligned16(W);
}

// X [n_rows, K] sorted by expert, W [experts, N, K] contiguous, spans as llmk_moe_plan leaves them (at most `max_spans`).  C [n_rows, N], or with a
// gated unit (act 2: silu(gate) * up, 3: the clamped one; bfloat16; W interleaves gate and up rows in groups of 16) [n_rows, N / 2].  act 1:
// relu squared (bfloat16).  Rows of C that no span names are left as they are.
LLMK_EXPORT int llmk_gemm_grouped(void* C, const void* X, const void* W, const void* spans, int max_spans, int n_rows, int experts, int N, int K,
                                  long long ldx, long long ldc, int act, float alpha, float limit, int out_dtype, int* error_flag, void* stream) {
    if (n_rows <= 0 || max_spans <= 0) return LLMK_OK;
    if (!llmk_gemm_grouped_usable(X, W, N, K, ldx) || experts <= 0)
        LLMK_FAIL("gemm_grouped: operands not usable (K=%d ldx=%lld must be multiples of 8, bases 16-byte aligned)", K, ldx);
    if (!host_aligned16(spans)) LLMK_FAIL("gemm_grouped: spans must start on a 16-byte boundary");
    if (ldx < K || ldc < (is_glu(act) ? N / 2 : N)) LLMK_FAIL("gemm_grouped: strides ldx=%lld ldc=%lld too small", ldx, ldc);
    if (is_glu(act) && N % 32 != 0) LLMK_FAIL("gemm_grouped: a gated unit needs N=%d to be a multiple of 32", N);
    if (act != ACT_NONE && out_dtype != LLMK_BF16) LLMK_FAIL("gemm_grouped: activations are built for bfloat16 results");
    CUtensorMap mw, mx[4];
    bool made = tc_host::cached_map_bf16_2d(&mw, W, (uint64_t)experts * N, K, K, BM);
    for (int i = 0; i < 4; ++i) made = made && tc_host::cached_map_bf16_2d(&mx[i], X, n_rows, K, ldx, SPAN / 2 >> i);
    if (!made)
        LLMK_FAIL("gemm_grouped: cuTensorMapEncodeTiled failed (rows %d N=%d K=%d experts %d)", n_rows, N, K, experts);
    Params p;
    p.spans = static_cast<const int4*>(spans);
    p.N = N; p.K = K; p.ldc = ldc; p.alpha = alpha; p.limit = limit; p.error_flag = error_flag;
    const int most = (int)std::min<long long>((long long)max_spans * ceil_div(N, 2 * BM), 1 << 20);
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == LLMK_F32) return launch<float, ACT_NONE>(mw, mx, C, p, most, s);
    if (out_dtype != LLMK_BF16) LLMK_FAIL("gemm_grouped: unknown output dtype %d", out_dtype);
    switch (act) {
        case ACT_NONE: return launch<bf16, ACT_NONE>(mw, mx, C, p, most, s);
        case ACT_RELU2: return launch<bf16, ACT_RELU2>(mw, mx, C, p, most, s);
        case ACT_SILU_GLU: return launch<bf16, ACT_SILU_GLU>(mw, mx, C, p, most, s);
        case ACT_CLAMPED_GLU: return launch<bf16, ACT_CLAMPED_GLU>(mw, mx, C, p, most, s);
        default: LLMK_FAIL("gemm_grouped: unknown activation %d", act);
    }
}
