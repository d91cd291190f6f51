// C[M, N] = A[M, K] * W[N, K]^T in bfloat16 on the 5th-generation tensor cores of sm_100a:
// operand tiles arrive in shared memory through TMA (`cp.async.bulk.tensor`, 128-byte swizzle),
// one thread issues `tcgen05.mma` with the float32 accumulator in tensor memory, and four
// epilogue warps read it back with `tcgen05.ld`, round once and store.
//
// A block computes 128 x BN output tiles (BN = 64, 128 or 256) one after the other, 192 threads
// (or two blocks of a cluster compute tiles of 256 rows together, see `gemm_pair_kernel`):
//   warp 0     TMA producer: for every 64-wide slice of K, one A box [128, 64] and one W box
//              [BN, 64] into a ring of STAGES buffers; `full[s]` counts the bytes.
//   warp 1     owns the tensor memory (two accumulators of BN columns) and issues the MMAs: 4
//              instructions of K = 16 per slice; `tcgen05.commit` releases the buffer (`empty[s]`) when
//              they have read it, and signals `acc_full[i]` after a tile's last slice; the next tile
//              goes to the other accumulator once the epilogue has released it (`acc_empty[i]`).
//   warps 2-5  epilogue: each reads the 32 accumulator lanes its warp id allows, 32 columns at a
//              time.  bfloat16 results are rounded into a slab of shared memory (32 rows x 64
//              columns, 128-byte swizzle) that one lane hands to a TMA store, two slabs per warp in
//              turn; float32 results, and results TMA cannot address, are stored by the threads,
//              64 or 128 contiguous bytes per row.
// Rows of A beyond M, rows of W beyond N and columns beyond K are zero-filled by TMA, so any M and
// N are taken; K must be a multiple of 8 and the bases 16-byte aligned (TMA's rules), otherwise
// the launcher refuses and the caller uses the CUDA-core product.
//
// Optionally the epilogue applies the gated activation to a W whose rows interleave gate and up in
// groups of 16 (`GATED`): out[m, j] = silu(c[m, gate j]) * c[m, up j], N/2 columns wide.
//
// Every wait is bounded (see tcgen05.cuh); a wait that gives up raises `*error_flag`, and the
// block still frees its tensor memory before it returns.
//
// The reference calls `cublasGemmEx` for this product (src/backend/cuda/linear/linear.cu:89-96).
#define LLMK_MODULE_NAME "gemm_tc"
#include "common.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <mutex>
#include <unordered_map>

LLMK_DEFINE_LAST_ERROR()

namespace {

constexpr int BM = 128;
constexpr int BK = 64;           // one 128-byte swizzle row of bfloat16
constexpr int UMMA_K = 16;
constexpr int THREADS = 192;

template <int W_ROWS, int STAGES, int KS = 1>
struct Smem {
    static constexpr int A_BYTES = BM * BK * 2;        // one block of 128 rows of A
    static constexpr int B_BYTES = W_ROWS * BK * 2;
    static constexpr int SUB_BYTES = A_BYTES + B_BYTES;             // one step of 64 along K: A, then W
    static constexpr int STAGE_BYTES = KS * SUB_BYTES;              // a stage of the ring holds KS such steps
    // the epilogue's staging: per epilogue warp two slabs of 32 rows x 64 bfloat16 columns (128-byte swizzle)
    static constexpr int SLAB_BYTES = 32 * 128;
    static constexpr int STAGING_OFFSET = STAGES * STAGE_BYTES;
    static constexpr int STAGING_BYTES = 4 * 2 * SLAB_BYTES;
    static constexpr int BAR_OFFSET = STAGING_OFFSET + STAGING_BYTES;
    static constexpr int NUM_BARS = 2 * STAGES + 4;     // full, empty, acc_full[2], acc_empty[2]
    static constexpr int TOTAL = BAR_OFFSET + NUM_BARS * 8 + 16 + 1024;  // + alignment slack
};

// the division as a reciprocal and a product: the exact one is a call with a slow path, which keeps the
// compiler from overlapping the elements of a row (measured: 9 us against 2 us for the epilogue of a tile)
__device__ __forceinline__ float silu(float g) { return __fdividef(g, 1.0f + __expf(-g)); }
// The gated epilogue's activation is part of the kernel's type (`GATED`: 0 no gate, 1 silu, 2 the tanh form of gelu), so
// that the silu kernels are the code they were: z / 2 (1 + tanh(u)) = z sigmoid(2u), u = sqrt(2 / pi) (z + 0.044715 z^3),
// costs what silu costs.  (A selector passed at launch was built first: with it two cases of the replay tests of another
// architecture failed when the whole suite ran, though not alone; as a template parameter it leaves those kernels as
// they were.)
// ACT_RELU2 (grouped products only) is no gate: the epilogue leaves relu(c)^2, as many columns as W has rows.
enum { GATE_NONE = 0, GATE_SILU = 1, GATE_GELU_TANH = 2, ACT_RELU2 = 3 };
constexpr bool is_glu(int act) { return act == GATE_SILU || act == GATE_GELU_TANH; }
template <int ACT>
__device__ __forceinline__ float plain_act(float c) {
    if constexpr (ACT == ACT_RELU2) return fmaxf(c, 0.f) * fmaxf(c, 0.f);
    else return c;
}
template <int ACT>
__device__ __forceinline__ float gate_act(float g) {
    if constexpr (ACT == GATE_GELU_TANH) return __fdividef(g, 1.0f + __expf(-1.5957691216057308f * (g + 0.044715f * g * g * g)));
    else return silu(g);
}


// What the epilogue warps do with one tile: `acc` is the warp's 32 lanes of an accumulator of `width` columns (a multiple of 32), its
// rows are row0 .. row0 + 31 and its columns begin at n0.
template <typename TC, int ACT>
__device__ __forceinline__ void store_tile(const CUtensorMap& map_c, int store_by_tma, uint32_t slabs, uint32_t& box_iter, uint32_t acc,
                                           int row0, int n0, int width, int split, TC* __restrict__ C, int M, int N, long long ldc) {
    constexpr bool GATED = is_glu(ACT);
    constexpr int SLAB_BYTES = 32 * 128;
    const int lane = threadIdx.x & 31;
    if (row0 >= M) return;                                  // uniform over the warp
    int c0 = 0;
    if constexpr (sizeof(TC) == 2) {
        if (store_by_tma) {
            // Row-per-thread stores to global memory are slow and hold up the TMA loads of the next
            // tile (measured: 4.3 us a tile against 1 us without them).  Each warp rounds its 32
            // rows into a slab of shared memory, 64 output columns at a time, in the layout of a
            // 128-byte-swizzled box (a lane's 16-byte pieces then fall into different banks), and
            // one lane hands the slab to TMA, which writes whole rows and clips at M and N.
            constexpr int ACC_COLS = GATED ? 128 : 64;          // accumulator columns per 64 output columns
#pragma unroll 1
            for (; c0 + ACC_COLS <= width; c0 += ACC_COLS) {
                if (n0 + c0 >= N) return;
                const uint32_t slab = slabs + (uint32_t)(box_iter & 1) * SLAB_BYTES;
                if (lane == 0) tc::bulk_wait_read<1>();         // the store that read this slab two boxes ago
                __syncwarp();
#pragma unroll
                for (int h = 0; h < ACC_COLS / 32; ++h) {
                    uint32_t r[32];
                    tc::tmem_ld_32x32_wait(acc + (uint32_t)(c0 + 32 * h), r);
                    if constexpr (GATED) {
                        float o[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = gate_act<ACT>(__uint_as_float(r[i])) * __uint_as_float(r[16 + i]);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            Vec16<bf16> v;
                            v.pack(o + 8 * q);
                            const int chunk = 2 * h + q;
                            tc::st_shared_v4(slab + (uint32_t)lane * 128 + (uint32_t)((chunk ^ (lane & 7)) << 4), v.raw);
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float f[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) f[j] = plain_act<ACT>(__uint_as_float(r[8 * q + j]));
                            Vec16<bf16> v;
                            v.pack(f);
                            const int chunk = 4 * h + q;
                            tc::st_shared_v4(slab + (uint32_t)lane * 128 + (uint32_t)((chunk ^ (lane & 7)) << 4), v.raw);
                        }
                    }
                }
                tc::fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    tc::tma_store_2d(&map_c, slab, GATED ? (n0 + c0) / 2 : n0 + c0, row0);
                    tc::bulk_commit();
                }
                ++box_iter;
            }
        }
    }
    if constexpr (sizeof(TC) == 4 && !GATED) {
        if (store_by_tma) {
            // float32 slices: slabs of 32 rows x 32 columns (128 bytes a row), handed to TMA the same way
#pragma unroll 1
            for (; c0 < width; c0 += 32) {
                if (n0 + c0 >= N) return;
                const uint32_t slab = slabs + (uint32_t)(box_iter & 1) * SLAB_BYTES;
                if (lane == 0) tc::bulk_wait_read<1>();
                __syncwarp();
                uint32_t r[32];
                tc::tmem_ld_32x32_wait(acc + (uint32_t)c0, r);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    tc::st_shared_v4(slab + (uint32_t)lane * 128 + (uint32_t)((q ^ (lane & 7)) << 4),
                                     make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]));
                tc::fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    tc::tma_store_3d(&map_c, slab, n0 + c0, row0, split);
                    tc::bulk_commit();
                }
                ++box_iter;
            }
        }
    }
    // results TMA cannot address, and a last half of a box
    const int row = row0 + lane;
    const int n_out = GATED ? N / 2 : N;
    const bool vec_ok = (ldc % (16 / (int)sizeof(TC)) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
#pragma unroll 1
    for (; c0 < width; c0 += 32) {
        if (n0 + c0 >= N) return;                           // uniform over the warp
        uint32_t r[32];
        __syncwarp();
        tc::tmem_ld_32x32_wait(acc + (uint32_t)c0, r);
        if (row >= M) {
            // nothing to store for this lane; it still takes part in the loads above
        } else if constexpr (GATED) {
            // columns [c0, c0 + 16) are gates, [c0 + 16, c0 + 32) the matching ups
            const int j0 = (n0 + c0) / 2;
            float o[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = gate_act<ACT>(__uint_as_float(r[i])) * __uint_as_float(r[16 + i]);
            TC* dst = C + (size_t)row * ldc + j0;
            if (vec_ok && j0 + 16 <= n_out) {
                if constexpr (sizeof(TC) == 2) {
                    Vec16<bf16> v0, v1;
                    v0.pack(o);
                    v1.pack(o + 8);
                    reinterpret_cast<uint4*>(dst)[0] = v0.raw;
                    reinterpret_cast<uint4*>(dst)[1] = v1.raw;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        reinterpret_cast<float4*>(dst)[i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                }
            } else {
                for (int i = 0; i < 16; ++i)
                    if (j0 + i < n_out) dst[i] = from_float<TC>(o[i]);
            }
        } else {
            TC* dst = C + ((size_t)split * M + row) * ldc + n0 + c0;
            if (vec_ok && n0 + c0 + 32 <= N) {
                if constexpr (sizeof(TC) == 2) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float f[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) f[j] = plain_act<ACT>(__uint_as_float(r[8 * i + j]));
                        Vec16<bf16> v;
                        v.pack(f);
                        reinterpret_cast<uint4*>(dst)[i] = v.raw;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        reinterpret_cast<float4*>(dst)[i] =
                            make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                        __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                }
            } else {
                for (int i = 0; i < 32; ++i)
                    if (n0 + c0 + i < N) dst[i] = from_float<TC>(plain_act<ACT>(__uint_as_float(r[i])));
            }
        }
    }
}

// Persistent: block b computes tiles b, b + gridDim.x, ... (tile t = (t % m_tiles) rows, (t / m_tiles)
// columns, so blocks that run together share W tiles).  Two accumulators of BN columns are used in turn: while
// the epilogue warps read tile i out of one, the MMA warp fills the other with tile i + 1; the TMA
// ring runs on across tiles either way.
template <typename TC, int BN, int STAGES, int ACT, int KS = 1>
__global__ void __launch_bounds__(THREADS)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const __grid_constant__ CUtensorMap map_c, int store_by_tma, int splits,
               TC* __restrict__ C, int M, int N, int K, long long ldc, int* error_flag,
               const int* __restrict__ tile_group) {
    using L = Smem<BN, STAGES, KS>;
    constexpr int W_OFF = KS * L::A_BYTES;          // a stage: A's KS steps, then W's
    constexpr uint32_t TMEM_COLS = 2 * BN;                         // 128, 256 or 512: a power of two
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;         // 2
    uint64_t* acc_empty = bars + 2 * STAGES + 2;    // 2, four arrivals each (one per epilogue warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NUM_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same for all lanes, and known to be)
    const int num_kb = (K + BK - 1) / BK;
    const int m_tiles = (M + BM - 1) / BM;
    const int n_tiles = (N + BN - 1) / BN;
    const int total_tiles = m_tiles * n_tiles;
    // K may be cut into `splits` slices (float32 results only): work item i is slice i / total_tiles of tile
    // i % total_tiles and leaves its sum in slice `split` of C ([splits][M][ldc]) for the consumer to add up
    const int total_items = total_tiles * splits;
    // a stage of the ring holds KS steps of 64 along K under one barrier (the hand-over of a stage costs about as
    // much as the copy of a narrow tile's step, so narrow tiles take two steps a stage); a slice begins on a stage
    const int kb_per_split = ((num_kb + splits - 1) / splits + KS - 1) / KS * KS;
    const int unit = (int)blockIdx.x, units = (int)gridDim.x;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(tc::smem_u32(&full[s]), 1);
            tc::mbar_init(tc::smem_u32(&empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(tc::smem_u32(&acc_full[i]), 1);
            tc::mbar_init(tc::smem_u32(&acc_empty[i]), 4);
        }
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_a);
        tc::prefetch_tensormap(&map_w);
    }
    if (warp == 1) {
        tc::tmem_alloc(tc::smem_u32(tmem_slot), TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        {
            // The whole warp walks the loops of both issuing roles and one lane issues: what the instructions are given is then known to be the
            // same for all lanes and kept where they read it.
            const bool issues = tc::elect_one();
            if (issues) pdl_launch_dependents();
            // KS steps of 64 along K of an operand (what lies beyond K is filled with zeros and counts its bytes all the same)
            auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t step_bytes, uint32_t bar, int kb, int row) {
#pragma unroll
                for (int h = 0; h < KS; ++h) tc::tma_load_2d(dst + h * step_bytes, map, bar, (kb + h) * BK, row);
            };
            // W is a weight: no kernel of the stream writes it, so the first slices of it are asked for before the
            // wait for the kernel that makes A, and arrive while that kernel ends.
            uint32_t w_ahead = 0;
            if (unit < total_items && !tile_group) {      // (which rows of W a grouped tile reads is known only after the wait)
                const int tile = unit % total_tiles, kb0 = (unit / total_tiles) * kb_per_split;
                const int sts = (min(num_kb, kb0 + kb_per_split) - kb0 + KS - 1) / KS;     // stages of the first item
                w_ahead = (uint32_t)(sts < STAGES ? sts : STAGES);
                const int n0 = (tile / m_tiles) * BN;
                for (uint32_t i = 0; i < w_ahead; ++i) {
                    const uint32_t bar = tc::smem_u32(&full[i]);
                    if (issues) {
                        tc::mbar_expect_tx(bar, L::STAGE_BYTES);
                        load(&map_w, tc::smem_u32(smem + i * L::STAGE_BYTES) + W_OFF, L::B_BYTES, bar, kb0 + (int)i * KS, n0);
                    }
                }
            }
            pdl_wait();   // A was written by the kernel before this one
            uint32_t it = 0;        // k-slices loaded so far, over all tiles of this block
            bool ok = true;
            for (int item = unit; item < total_items && ok; item += units) {
                const int tile = item % total_tiles, split = item / total_tiles;
                const int m0 = (tile % m_tiles) * BM;
                int n0 = (tile / m_tiles) * BN;
                if (tile_group) {
                    // grouped: the 128 rows of this tile belong to one group, whose matrix is rows [g N, (g + 1) N) of W
                    const int g = tile_group[tile % m_tiles];
                    if (g < 0) continue;                       // a tile of padding: nobody computes, nobody stores it
                    n0 += g * N;
                }
                const int kb_end = min(num_kb, (split + 1) * kb_per_split);
                for (int kb = split * kb_per_split; kb < kb_end; kb += KS, ++it) {
                    const int s = it % STAGES;
                    const uint32_t round = it / STAGES;
                    if (!tc::mbar_wait_warp(tc::smem_u32(&empty[s]), (round & 1) ^ 1, abort_flag)) { ok = false; break; }
                    const uint32_t bar = tc::smem_u32(&full[s]);
                    const bool w_here = it < w_ahead;       // its bytes are expected and W is on its way
                    const uint32_t dst = tc::smem_u32(smem + s * L::STAGE_BYTES);
                    if (issues) {
                        if (!w_here) tc::mbar_expect_tx(bar, L::STAGE_BYTES);
                        load(&map_a, dst, L::A_BYTES, bar, kb, m0);
                        if (!w_here) load(&map_w, dst + W_OFF, L::B_BYTES, bar, kb, n0);
                    }
                }
            }
            if (*abort_flag) {
                // Let the copies that are in flight land before the block's memory is given up.
                for (uint32_t k = it > (uint32_t)STAGES ? it - STAGES : 0; k < it; ++k) {
                    const long long t0 = clock64();
                    while (!tc::mbar_try_wait(tc::smem_u32(&full[k % STAGES]), (k / STAGES) & 1) &&
                           clock64() - t0 < tc::WAIT_LIMIT_CYCLES) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        {
            const bool issues = tc::elect_one();
            constexpr uint32_t idesc = tc::idesc_bf16_f32(BM, BN);
            // The descriptor of the ring's first byte, built once: every operand tile's descriptor is this one plus
            // its byte offset in units of 16 (the start address is the descriptor's lowest field); built per
            // instruction they cost the one issuing thread a few per cent (11.1 -> 10.9 us, 15.2 -> 14.9 us on the
            // N = 1,024 products of a 2,048-token prompt).
            const uint64_t ring_desc = tc::smem_desc_sw128(tc::smem_u32(smem));
            uint32_t it = 0;
            bool ok = true;
            int tile_iter = 0;
            if (tile_group) pdl_wait();         // the list of groups comes from a kernel before this one
            for (int item = unit; item < total_items && ok; item += units, ++tile_iter) {
                if (tile_group && tile_group[(item % total_tiles) % m_tiles] < 0) {
                    --tile_iter;                // a tile of padding takes no turn with the accumulators
                    continue;
                }
                const int split = item / total_tiles;
                const int kb_begin = split * kb_per_split, kb_end = min(num_kb, (split + 1) * kb_per_split);
                const int buf = tile_iter & 1;
                // the epilogue must have read this accumulator before it is filled again
                ok = tc::mbar_wait_warp(tc::smem_u32(&acc_empty[buf]), ((tile_iter / 2) & 1) ^ 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after_sync();
                const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
                for (int kb = kb_begin; kb < kb_end; kb += KS, ++it) {
                    const int s = it % STAGES;
                    const uint32_t round = it / STAGES;
                    ok = tc::mbar_wait_warp(tc::smem_u32(&full[s]), round & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                    if (!issues) continue;
#pragma unroll
                    for (int h = 0; h < KS; ++h) {
                        if (kb + h >= kb_end) break;            // a step beyond K holds zeros: nothing to add
                        const uint64_t a_desc = ring_desc + (uint64_t)((s * L::STAGE_BYTES + h * L::A_BYTES) >> 4);
                        const uint64_t b_desc = ring_desc + (uint64_t)((s * L::STAGE_BYTES + W_OFF + h * L::B_BYTES) >> 4);
                        const bool first = kb + h == kb_begin;
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            const uint64_t at = (uint64_t)((k * UMMA_K * 2) >> 4);
                            tc::mma_bf16_ss(acc, a_desc + at, b_desc + at, idesc, !first || k != 0);
                        }
                    }
                    tc::mma_commit(tc::smem_u32(&empty[s]));
                }
                if (ok && issues) tc::mma_commit(tc::smem_u32(&acc_full[buf]));
            }
        }
    } else {
        // Epilogue: warp w may touch tensor-memory lanes 32 * (w % 4) .. + 31.
        const int quarter = warp & 3;
        const uint32_t slabs = tc::smem_u32(smem + L::STAGING_OFFSET) + (uint32_t)quarter * 2 * L::SLAB_BYTES;
        bool ok = true;
        int tile_iter = 0;
        uint32_t box_iter = 0;          // boxes this warp has handed to TMA
        if (tile_group) pdl_wait();
        for (int item = unit; item < total_items && ok; item += units, ++tile_iter) {
            const int tile = item % total_tiles, split = item / total_tiles;
            if (tile_group && tile_group[tile % m_tiles] < 0) {
                --tile_iter;
                continue;
            }
            const int buf = tile_iter & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&acc_full[buf]), (tile_iter / 2) & 1, abort_flag));
            if (!ok) break;
            tc::tc_fence_after_sync();
            store_tile<TC, ACT>(map_c, store_by_tma, slabs, box_iter, tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN),
                                (tile % m_tiles) * BM + quarter * 32, (tile / m_tiles) * BN, BN, split, C, M, N, ldc);
            // this warp has read its lanes of the accumulator: let the MMA warp fill it again
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(tc::smem_u32(&acc_empty[buf]));
        }
        if (lane == 0) tc::bulk_wait_read<0>();     // the slabs are read before the block's memory is given up
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag && error_flag) atomicExch(error_flag, 1);
}

// ------------------------------------------------------------------------------------------- pairs of blocks
// The same product by clusters of two blocks (an SM pair): a tile is 256 rows by up to 256 columns, computed by
// `tcgen05.mma.cta_group::2`.  Each block loads its 128 rows of A and its half of the tile's W rows (no multicast: every block
// loads what it holds), so a block pulls 32 KB per step of 64 along K for 128 x 256 outputs where a lone block pulls 48 KB: the
// products are bound by what the SMs pull from L2.  The bytes of both blocks are counted on the `full` barriers of the block of
// rank 0, which issues the MMAs; its commits arrive on the `empty` and `acc_full` barriers of both blocks; the epilogue warps of
// both release an accumulator on rank 0's `acc_empty`.  Each block reads its own 128 rows of the accumulator out of its own
// tensor memory.
//
// PairPlan: the tiles of a launch have two widths, so that the last round over the SM pairs is as full as the others: `wide` tiles of
// PAIR_BN columns from a panel's (256 rows') first column on, in whole rounds, and what is left of every panel in tiles of
// `narrow` columns.  A stage holds two steps of 64 along K (with one, tiles of 128 columns took 287 ns a step instead of 215).
constexpr int PAIR_BN = 256, PAIR_STAGES = 3, PAIR_KS = 2;
struct PairPlan {
    int panels;         // of 256 rows
    int panels_hi;      // the first of them have `wide_hi` wide tiles each, the others one less
    int wide_hi;
    int wide_items;     // wide tiles in all
    int narrow;         // width of the narrow tiles, a multiple of 32; 0: none
    int narrow_hi;      // narrow tiles of each of the first panels
    int total;          // tiles in all
};
struct PairTile { int m0, n0, width; };
__device__ __forceinline__ PairTile pair_tile(const PairPlan& p, int item) {
    PairTile t;
    if (item < p.wide_items) {
        t.m0 = item % p.panels * 2 * BM;
        t.n0 = item / p.panels * PAIR_BN;
        t.width = PAIR_BN;
        return t;
    }
    int j = item - p.wide_items, panel, c;
    if (j < p.panels * p.narrow_hi) {
        panel = j % p.panels;
        c = j / p.panels;
    } else {                                     // panels with one wide tile less have more narrow ones
        j -= p.panels * p.narrow_hi;
        const int lo = p.panels - p.panels_hi;
        panel = p.panels_hi + j % lo;
        c = p.narrow_hi + j / lo;
    }
    t.m0 = panel * 2 * BM;
    t.n0 = (p.wide_hi - (panel < p.panels_hi ? 0 : 1)) * PAIR_BN + c * p.narrow;
    t.width = p.narrow;
    return t;
}

template <typename TC, int ACT>
__global__ void __launch_bounds__(THREADS)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_w_narrow, const __grid_constant__ CUtensorMap map_c, int store_by_tma,
                 const PairPlan plan, TC* __restrict__ C, int M, int N, int K, long long ldc, int* error_flag) {
    constexpr int STAGES = PAIR_STAGES, KS = PAIR_KS;
    using L = Smem<PAIR_BN / 2, STAGES, KS>;
    constexpr int W_OFF = KS * L::A_BYTES;          // a stage: A's KS steps, then W's
    constexpr uint32_t TMEM_COLS = 2 * PAIR_BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;         // 2
    uint64_t* acc_empty = bars + 2 * STAGES + 2;    // 2, eight arrivals each (one per epilogue warp of either block)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NUM_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same for all lanes, and known to be)
    const int num_kb = (K + BK - 1) / BK;
    const uint32_t rank = cluster_ctarank();                        // which block of the pair
    const int unit = (int)blockIdx.x / 2, units = (int)gridDim.x / 2;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(tc::smem_u32(&full[s]), 1);
            tc::mbar_init(tc::smem_u32(&empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(tc::smem_u32(&acc_full[i]), 1);
            tc::mbar_init(tc::smem_u32(&acc_empty[i]), 8);
        }
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_a);
        tc::prefetch_tensormap(&map_w);
        if (plan.narrow) tc::prefetch_tensormap(&map_w_narrow);
    }
    if (warp == 1) {
        tc::tmem_alloc_pair(tc::smem_u32(tmem_slot), TMEM_COLS);
        tc::tmem_relinquish_pair();
    }
    tc::tc_fence_before_sync();
    __syncwarp();
    cluster_sync_all();         // both blocks' barriers and tensor memory are ready before either uses the other's
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        {
            const bool issues = tc::elect_one();
            if (issues) pdl_launch_dependents();
            // a stage is KS steps of 64 along K (what lies beyond K is filled with zeros and counts its bytes all the same)
            const int stages = (num_kb + KS - 1) / KS;
            auto stage_bytes = [](const PairTile& t) { return 2 * KS * (L::A_BYTES + t.width / 2 * BK * 2); };      // of both blocks
            auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t step_bytes, uint32_t bar, int st, int row) {
#pragma unroll
                for (int h = 0; h < KS; ++h) tc::tma_load_2d_pair(dst + h * step_bytes, map, bar, (st * KS + h) * BK, row);
            };
            auto load_w = [&](const PairTile& t, int s, int st) {
                load(t.width == PAIR_BN ? &map_w : &map_w_narrow, tc::smem_u32(smem + s * L::STAGE_BYTES) + W_OFF, (uint32_t)(t.width / 2 * BK * 2),
                     cluster_map_shared(tc::smem_u32(&full[s]), 0), st, t.n0 + (int)rank * (t.width / 2));
            };
            // the first stages of W before the wait for the kernel that makes A, as in `gemm_tc_kernel`
            const uint32_t w_ahead = (uint32_t)min(stages, STAGES);
            {
                const PairTile t = pair_tile(plan, unit);
                for (uint32_t i = 0; i < w_ahead; ++i) {
                    if (!issues) continue;
                    if (rank == 0) tc::mbar_expect_tx(tc::smem_u32(&full[i]), stage_bytes(t));
                    load_w(t, (int)i, (int)i);
                }
            }
            pdl_wait();   // A was written by the kernel before this one
            uint32_t it = 0;        // stages loaded so far, over all tiles of this block
            bool ok = true;
            for (int item = unit; item < plan.total && ok; item += units) {
                const PairTile t = pair_tile(plan, item);
                for (int st = 0; st < stages; ++st, ++it) {
                    const int s = it % STAGES;
                    if (!tc::mbar_wait_warp(tc::smem_u32(&empty[s]), ((it / STAGES) & 1) ^ 1, abort_flag)) { ok = false; break; }
                    if (!issues) continue;
                    const bool w_here = it < w_ahead;       // its bytes are expected and W is on its way
                    // both blocks' bytes are counted on rank 0's barrier
                    if (!w_here && rank == 0) tc::mbar_expect_tx(tc::smem_u32(&full[s]), stage_bytes(t));
                    load(&map_a, tc::smem_u32(smem + s * L::STAGE_BYTES), L::A_BYTES, cluster_map_shared(tc::smem_u32(&full[s]), 0), st,
                         t.m0 + (int)rank * BM);
                    if (!w_here) load_w(t, s, st);
                }
            }
            if (*abort_flag && rank == 0) {
                // Let the copies that are in flight land before the block's memory is given up (rank 0's
                // barriers count the other block's copies too, and that block leaves only after rank 0).
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
            for (int item = unit; item < plan.total && ok; item += units, ++tile_iter) {
                const int width = pair_tile(plan, item).width;
                const uint32_t idesc = tc::idesc_bf16_f32(2 * BM, width);
                const uint64_t w_step = (uint64_t)((width / 2 * BK * 2) >> 4);
                const int buf = tile_iter & 1;
                // the epilogue must have read this accumulator before it is filled again
                ok = tc::mbar_wait_warp(tc::smem_u32(&acc_empty[buf]), ((tile_iter / 2) & 1) ^ 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after_sync();
                const uint32_t acc = tmem_base + (uint32_t)(buf * PAIR_BN);
                for (int kb = 0; kb < num_kb; kb += KS, ++it) {
                    const int s = it % STAGES;
                    ok = tc::mbar_wait_warp(tc::smem_u32(&full[s]), (it / STAGES) & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                    if (!issues) continue;
#pragma unroll
                    for (int h = 0; h < KS; ++h) {
                        if (kb + h >= num_kb) break;            // a step beyond K holds zeros: nothing to add
                        const uint64_t a_desc = ring_desc + (uint64_t)((s * L::STAGE_BYTES + h * L::A_BYTES) >> 4);
                        const uint64_t b_desc = ring_desc + (uint64_t)((s * L::STAGE_BYTES + W_OFF) >> 4) + (uint64_t)h * w_step;
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            const uint64_t at = (uint64_t)((k * UMMA_K * 2) >> 4);
                            tc::mma_bf16_ss_pair(acc, a_desc + at, b_desc + at, idesc, kb + h != 0 || k != 0);
                        }
                    }
                    tc::mma_commit_pair(tc::smem_u32(&empty[s]), (uint16_t)3);
                }
                if (ok && issues) tc::mma_commit_pair(tc::smem_u32(&acc_full[buf]), (uint16_t)3);
            }
        }
    } else {
        const int quarter = warp & 3;
        const uint32_t slabs = tc::smem_u32(smem + L::STAGING_OFFSET) + (uint32_t)quarter * 2 * L::SLAB_BYTES;
        bool ok = true;
        int tile_iter = 0;
        uint32_t box_iter = 0;
        for (int item = unit; item < plan.total && ok; item += units, ++tile_iter) {
            const PairTile t = pair_tile(plan, item);
            const int buf = tile_iter & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&acc_full[buf]), (tile_iter / 2) & 1, abort_flag));
            if (!ok) break;
            tc::tc_fence_after_sync();
            store_tile<TC, ACT>(map_c, store_by_tma, slabs, box_iter, tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * PAIR_BN),
                                t.m0 + (int)rank * BM + quarter * 32, t.n0, t.width, 0, C, M, N, ldc);
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster(cluster_map_shared(tc::smem_u32(&acc_empty[buf]), 0));
        }
        if (lane == 0) tc::bulk_wait_read<0>();
    }
    tc::tc_fence_before_sync();
    __syncwarp();
    cluster_sync_all();         // neither block leaves, or frees tensor memory, while the other may still use it
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag && error_flag) atomicExch(error_flag, 1);
}

// ------------------------------------------------------------------------ tensor-map cache
struct MapKey {
    const void* base;
    uint64_t rows, cols, ld;
    uint32_t box_rows;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        size_t h = reinterpret_cast<size_t>(k.base);
        h = h * 1000003u ^ k.rows;
        h = h * 1000003u ^ k.cols;
        h = h * 1000003u ^ k.ld;
        return h * 1000003u ^ k.box_rows;
    }
};
std::mutex g_map_lock;
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;

bool get_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    MapKey key{base, rows, cols, ld, box_rows};
    std::lock_guard<std::mutex> guard(g_map_lock);
    auto it = g_maps.find(key);
    if (it != g_maps.end()) {
        *out = it->second;
        return true;
    }
    if (!tc_host::make_map_bf16_2d(out, base, rows, cols, ld, box_rows)) return false;
    if (g_maps.size() > 4096) g_maps.clear();
    g_maps.emplace(key, *out);
    return true;
}

int g_store_by_tma = 1;      // 0: the threads store their rows themselves (for measurements)

// float32 slices of C ([splits][M][ldc]) for TMA stores of [32 x 32] boxes
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_slice_maps;
bool get_slice_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t slices) {
    MapKey key{base, rows, cols, ld, slices};
    std::lock_guard<std::mutex> guard(g_map_lock);
    auto it = g_slice_maps.find(key);
    if (it != g_slice_maps.end()) {
        *out = it->second;
        return true;
    }
    if (!tc_host::make_map_f32_slices(out, base, rows, cols, ld, slices, 32)) return false;
    if (g_slice_maps.size() > 1024) g_slice_maps.clear();
    g_slice_maps.emplace(key, *out);
    return true;
}

// bfloat16 results leave through shared memory and TMA stores of [32 rows x 64 columns] boxes
// where TMA can address C (16-byte aligned base and rows), float32 slices in boxes of 32 columns; otherwise the threads store their rows.
// (A TMA store clips at the tensor's last column in units of 16 bytes, measured: with a width that is no
// multiple of 16 bytes it writes up to 7 bfloat16 columns beyond it, so such results are stored by the threads.)
template <typename TC, int ACT>
int store_map(CUtensorMap* mc, void* C, int M, int N, long long ldc, int splits) {
    constexpr bool GATED = is_glu(ACT);
    const int n_out = GATED ? N / 2 : N;
    if (!g_store_by_tma || !host_aligned16(C)) return 0;
    if (sizeof(TC) == 2 && ldc % 8 == 0 && n_out % 8 == 0) return get_map(mc, C, M, n_out, ldc, 32) ? 1 : 0;
    if (sizeof(TC) == 4 && !GATED && ldc % 4 == 0 && N % 4 == 0) return get_slice_map(mc, C, M, N, ldc, splits) ? 1 : 0;
    return 0;
}

// w_rows: rows of the array W (N, or those of all groups)
template <typename TC, int BN, int STAGES, int ACT, int KS = 1>
int launch(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
           int* error_flag, int pdl, cudaStream_t s, uint64_t w_rows, int splits = 1, const int* tile_group = nullptr) {
    static_assert(ACT != ACT_RELU2 || sizeof(TC) == 2, "the squared relu is built for bfloat16 results");
    using L = Smem<BN, STAGES, KS>;
    auto kernel = gemm_tc_kernel<TC, BN, STAGES, ACT, KS>;
    static bool configured = false;   // per instantiation
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
        if (e != cudaSuccess) LLMK_FAIL("gemm_tc: cannot raise shared memory to %d: %s", L::TOTAL, cudaGetErrorString(e));
        configured = true;
    }
    CUtensorMap ma, mw, mc{};
    if (!get_map(&ma, A, M, K, lda, BM) || !get_map(&mw, W, w_rows, K, ldw, BN))
        LLMK_FAIL("gemm_tc: cuTensorMapEncodeTiled failed (M=%d N=%d K=%d lda=%lld ldw=%lld)", M, N, K, lda, ldw);
    const int store_by_tma = store_map<TC, ACT>(&mc, C, M, N, ldc, splits);
    const int NUM_SMS = device_sm_count();
    const int tiles = ceil_div(N, BN) * ceil_div(M, BM) * splits;
    LLMK_CHECK_LAUNCH_RC("gemm_tc", llmk_launch(kernel, dim3(tiles < NUM_SMS ? tiles : NUM_SMS), dim3(THREADS), L::TOTAL, s,
                                                pdl != 0, ma, mw, mc, store_by_tma, splits, (TC*)C, M, N, K, ldc,
                                                error_flag, tile_group));
    return LLMK_OK;
}

// 0: lone blocks only.  1: pairs of blocks where they are the faster ones.
// 2, 3: pairs always, with tiles of two widths or all 128 columns wide (for measurements and tests).
int g_pair_mode = 1;

// Nanoseconds that a launch takes besides its rounds of tiles, and that a tile of `width` columns takes for 64 along K, by a pair of blocks and by lone
// ones.  Measured on products of 300 to 2,048 rows (K 1,024 to 12,288; graphs of 20 launches): a pair's tile of 128 / 160 / 192 / 224 / 256 columns
// 206-220 / 224-250 / 240-297 / 299-305 / 305-342, a lone block's of 128 / 256 200-215 / 352-400.
constexpr long long PAIR_LAUNCH = 5300, LONE_LAUNCH = 4300;
inline long long pair_time(int width) { return 115 + 82 * width / 100; }
inline long long lone_time(int width) { return width == 256 ? 370 : 205; }

// The plan of the least time over the SM pairs, and that time.
PairPlan pair_plan(int M, int N, int pairs, long long* time) {
    PairPlan best{};
    *time = -1;
    const int panels = ceil_div(M, 2 * BM), per_panel = ceil_div(N, PAIR_BN);
    auto consider = [&](int wide_items, int narrow) {
        PairPlan p{};
        p.panels = panels;
        p.wide_items = wide_items;
        const int lo = wide_items / panels, extra = wide_items % panels;
        p.panels_hi = extra ? extra : panels;
        p.wide_hi = extra ? lo + 1 : lo;
        p.narrow = narrow;
        p.total = wide_items;
        if (narrow) {
            const int rest_hi = N - p.wide_hi * PAIR_BN, rest_lo = N - lo * PAIR_BN;
            p.narrow_hi = rest_hi > 0 ? ceil_div(rest_hi, narrow) : 0;
            p.total += p.panels_hi * p.narrow_hi + (panels - p.panels_hi) * (rest_lo > 0 ? ceil_div(rest_lo, narrow) : 0);
        }
        const long long t = (long long)ceil_div(wide_items, pairs) * pair_time(PAIR_BN) +
                            (narrow ? (long long)ceil_div(p.total - wide_items, pairs) * pair_time(narrow) : 0);
        if (*time < 0 || t < *time) {
            *time = t;
            best = p;
        }
    };
    if (g_pair_mode == 3) {
        consider(0, 128);
        return best;
    }
    const int all = panels * per_panel;
    consider(all, 0);
    for (int k = 0; k * pairs < all; ++k)
        for (int w = 32; w < PAIR_BN; w += 32) consider(k * pairs, w);
    return best;
}

template <typename TC, int ACT>
int launch_pair(const PairPlan& plan, const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
                long long ldc, int* error_flag, int pdl, cudaStream_t s) {
    using L = Smem<PAIR_BN / 2, PAIR_STAGES, PAIR_KS>;
    auto kernel = gemm_pair_kernel<TC, ACT>;
    static bool configured = false;   // per instantiation
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
        if (e != cudaSuccess) LLMK_FAIL("gemm_tc: cannot raise shared memory to %d: %s", L::TOTAL, cudaGetErrorString(e));
        configured = true;
    }
    CUtensorMap ma, mw, mn, mc{};
    const int narrow = plan.narrow ? plan.narrow : PAIR_BN;
    if (!get_map(&ma, A, M, K, lda, BM) || !get_map(&mw, W, N, K, ldw, PAIR_BN / 2) || !get_map(&mn, W, N, K, ldw, narrow / 2))
        LLMK_FAIL("gemm_tc: cuTensorMapEncodeTiled failed (M=%d N=%d K=%d lda=%lld ldw=%lld)", M, N, K, lda, ldw);
    const int store_by_tma = store_map<TC, ACT>(&mc, C, M, N, ldc, 1);
    const int pairs = std::min(plan.total, device_sm_count() / 2);
    LLMK_CHECK_LAUNCH_RC("gemm_tc", llmk_launch_clusters(kernel, dim3(2 * pairs), dim3(THREADS), L::TOTAL, s, pdl != 0, dim3(2, 1, 1), ma, mw, mn,
                                                         mc, store_by_tma, plan, (TC*)C, M, N, K, ldc, error_flag));
    return LLMK_OK;
}

// ring depth of the narrower tiles (3, 4 and 6 were measured on a prompt's products: no difference
// beyond 4, the MMA instructions set the pace)
constexpr int STAGES_128 = 3, KS_128 = 2, STAGES_64 = 4;      // 128-wide tiles: three stages of two steps along K

template <typename TC, int GATED>
int dispatch_tile(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
                  long long ldc, int* error_flag, int pdl, cudaStream_t s) {
    // The tiles that take the least time in rounds over the SMs, lone blocks' or pairs'.  What the pairs gain (us, lone / pairs): 2,048 rows on 8,192 x 2,048
    // 55.5 / 48.1, 2,048 x 6,144 40.3 / 36.8, gated 6,144 x 1,024 21.7 / 20.1; 1,501 rows on 4,096 x 12,288 180 / 120, gated 24,576 x 4,096 212 / 192;
    // 700 rows on 4,096 x 4,096 28.9 / 23.5.  What stays with lone blocks: 2,048 rows on 1,024 x 2,048 10.7 / 11.5, 300 rows on 6,144 x 1,024 12.4 / 14.5.
    // (64 columns take as long as 128; they are for W of few rows.)
    const int NUM_SMS = device_sm_count();
    const long long steps = ceil_div(K, BK);
    int bn = GATED ? 128 : 64;
    long long best = -1;
    for (const int width : {256, 128, 64}) {
        if (GATED && width == 64) continue;          // the gated epilogue is built for the wider tiles only
        const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, width);
        const long long cost = LONE_LAUNCH + (tiles + NUM_SMS - 1) / NUM_SMS * steps * lone_time(width);
        if (best < 0 || cost < best) {
            best = cost;
            bn = width;
        }
    }
    if (g_pair_mode != 0) {
        long long pair = -1;
        const PairPlan plan = pair_plan(M, N, NUM_SMS / 2, &pair);
        if (g_pair_mode >= 2 || PAIR_LAUNCH + pair * steps < best)
            return launch_pair<TC, GATED>(plan, A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s);
    }
    switch (bn) {
        case 256: return launch<TC, 256, 4, GATED>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, N);
        case 128: return launch<TC, 128, STAGES_128, GATED, KS_128>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, N);
        default: return launch<TC, 64, STAGES_64, GATE_NONE>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, N);
    }
}

}  // namespace

// 1 if the tensor-core kernel takes these operands (TMA needs 16-byte aligned bases and row strides).
LLMK_EXPORT int llmk_gemm_tc_usable(const void* A, const void* W, int M, int N, int K, long long lda, long long ldw) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (K % 8 != 0 || lda % 8 != 0 || ldw % 8 != 0) return 0;
    if (!host_aligned16(A) || !host_aligned16(W)) return 0;
    return 1;
}

// Into how many slices of K a product is best cut when its tiles of 128 x 128 are too few for the SMs: about
// one work item per SM, at least 4 steps of 64 along K per item, at most 16 slices.  1: not cut.
LLMK_EXPORT int llmk_gemm_tc_splits(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 1;
    const int NUM_SMS = device_sm_count();
    const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, 128);
    if (tiles * 4 >= 3LL * NUM_SMS) return 1;           // the tiles alone keep three quarters of the SMs busy
    const int num_kb = ceil_div(K, BK);
    int splits = (int)(NUM_SMS / tiles);
    if (splits > num_kb / 4) splits = num_kb / 4;
    if (splits > 16) splits = 16;
    if (splits < 2) return 1;
    const int per = ceil_div(ceil_div(num_kb, splits), KS_128) * KS_128;      // a slice begins on a stage of the ring
    return ceil_div(num_kb, per);                        // no slice is left empty
}

// C (float32, [splits][M][ldc]) receives the sums over `splits` slices of K of A[M, K] * W[N, K]^T, in tiles of
// 128 x 128; the consumer adds the slices up in slice order.
LLMK_EXPORT int llmk_gemm_tc_sliced(float* C, const void* A, const void* W, int M, int N, int K, long long lda,
                                    long long ldw, long long ldc, int splits, int* error_flag, int pdl, void* stream) {
    if (M <= 0 || N <= 0) return LLMK_OK;
    if (K <= 0 || K % 8 != 0 || lda % 8 != 0 || ldw % 8 != 0 || !host_aligned16(A) || !host_aligned16(W))
        LLMK_FAIL("gemm_tc: operands not usable (K=%d lda=%lld ldw=%lld must be multiples of 8, bases 16-byte aligned)", K, lda, ldw);
    const int num_kb = ceil_div(K, BK);
    if (splits < 1 || splits > num_kb) LLMK_FAIL("gemm_tc: %d slices for K=%d", splits, K);
    if ((splits - 1) * (ceil_div(ceil_div(num_kb, splits), KS_128) * KS_128) >= num_kb)
        LLMK_FAIL("gemm_tc: %d slices of K=%d would leave one empty (slices are multiples of %d columns)", splits, K, KS_128 * BK);
    if (ldc < N) LLMK_FAIL("gemm_tc: ldc=%lld too small", ldc);
    return launch<float, 128, STAGES_128, false, KS_128>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, (cudaStream_t)stream, N, splits);
}

// Grouped product: the rows of A come in tiles of 128 that belong to one group each (`tile_group[i]` for rows
// [128 i, 128 i + 128); -1: a tile of padding, skipped), W stacks the groups' matrices ([groups * N, K]) and
// C[m, :] = A[m, :] * W[group of m's tile]^T.  The list of groups lives on the device, so the launch has the same
// shape whatever the groups' sizes are (a mixture of experts whose rows were sorted by expert on the device).
// relu2 != 0 (bfloat16 results): C = relu(.)^2 of that, applied in the epilogue.
LLMK_EXPORT int llmk_gemm_tc_grouped(void* C, const void* A, const void* W, int M, int N, int K, long long lda, long long ldw,
                                     long long ldc, int groups, const int* tile_group, int relu2, int out_dtype, int* error_flag, int pdl,
                                     void* stream) {
    if (M <= 0 || N <= 0 || groups <= 0) return LLMK_OK;
    if (!llmk_gemm_tc_usable(A, W, M, N, K, lda, ldw))
        LLMK_FAIL("gemm_tc_grouped: operands not usable (K=%d lda=%lld ldw=%lld must be multiples of 8, bases 16-byte aligned)", K, lda, ldw);
    if (M % BM != 0 || !tile_group) LLMK_FAIL("gemm_tc_grouped: %d rows are not whole tiles of %d with a group each", M, BM);
    if (ldc < N) LLMK_FAIL("gemm_tc_grouped: ldc=%lld too small", ldc);
    const int bn = N >= 256 ? 256 : N > 64 ? 128 : 64;
    const uint64_t w_rows = (uint64_t)groups * N;
    cudaStream_t s = (cudaStream_t)stream;
    if (relu2) {
        if (out_dtype != LLMK_BF16) LLMK_FAIL("gemm_tc_grouped: the squared relu is built for bfloat16 results");
        if (bn == 256) return launch<bf16, 256, 4, ACT_RELU2>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        if (bn == 128) return launch<bf16, 128, STAGES_128, ACT_RELU2, KS_128>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        return launch<bf16, 64, STAGES_64, ACT_RELU2>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
    }
    if (out_dtype == LLMK_BF16) {
        if (bn == 256) return launch<bf16, 256, 4, false>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        if (bn == 128) return launch<bf16, 128, STAGES_128, false, KS_128>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        return launch<bf16, 64, STAGES_64, false>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
    }
    if (out_dtype == LLMK_F32) {
        if (bn == 256) return launch<float, 256, 4, false>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        if (bn == 128) return launch<float, 128, STAGES_128, false, KS_128>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
        return launch<float, 64, STAGES_64, false>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s, w_rows, 1, tile_group);
    }
    LLMK_FAIL("gemm_tc_grouped: unknown output dtype %d", out_dtype);
}

LLMK_EXPORT void llmk_gemm_tc_set_pair_mode(int mode) { g_pair_mode = mode; }
LLMK_EXPORT void llmk_gemm_tc_set_store_by_tma(int on) { g_store_by_tma = on; }

// out_dtype: storage of C (bfloat16, or float32 for logits).  gated != 0: W interleaves gate and up
// rows in groups of 16 and C is [M, N / 2] = act(gate) * up, act = silu (gated 1) or the tanh form of gelu (gated 2).  error_flag (device int, may be null) is raised if a
// wait inside the kernel gave up.
LLMK_EXPORT int llmk_gemm_tc(void* C, const void* A, const void* W, int M, int N, int K, long long lda,
                             long long ldw, long long ldc, int gated, int out_dtype, int* error_flag, int pdl,
                             void* stream) {
    if (M <= 0 || N <= 0) return LLMK_OK;
    if (!llmk_gemm_tc_usable(A, W, M, N, K, lda, ldw))
        LLMK_FAIL("gemm_tc: operands not usable (K=%d lda=%lld ldw=%lld must be multiples of 8, bases 16-byte aligned)", K, lda, ldw);
    if (gated && N % 32 != 0) LLMK_FAIL("gemm_tc: gated epilogue needs N=%d to be a multiple of 32", N);
    if (gated != GATE_NONE && gated != GATE_SILU && gated != GATE_GELU_TANH) LLMK_FAIL("gemm_tc: unknown gated activation %d", gated);
    if (ldc < (gated ? N / 2 : N)) LLMK_FAIL("gemm_tc: ldc=%lld too small", ldc);
    if (ceil_div(M, BM) > 65535) LLMK_FAIL("gemm_tc: M=%d too large", M);
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == LLMK_BF16)
        return gated == GATE_GELU_TANH ? dispatch_tile<bf16, GATE_GELU_TANH>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s)
               : gated             ? dispatch_tile<bf16, GATE_SILU>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s)
                                   : dispatch_tile<bf16, GATE_NONE>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s);
    if (out_dtype == LLMK_F32)
        return gated == GATE_GELU_TANH ? dispatch_tile<float, GATE_GELU_TANH>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s)
               : gated             ? dispatch_tile<float, GATE_SILU>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s)
                                   : dispatch_tile<float, GATE_NONE>(A, W, C, M, N, K, lda, ldw, ldc, error_flag, pdl, s);
    LLMK_FAIL("gemm_tc: unknown output dtype %d", out_dtype);
}

