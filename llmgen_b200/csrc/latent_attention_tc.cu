// The latent attention of whole portions of prompts (csrc/latent_attention.cu: softmax attention of absorbed queries over one cached vector z a
// token, whose first `rank` entries are also the values) on the 5th-generation tensor cores of sm_100a.
//
// Block = 128 rows (128 / heads queries x heads) of one tile of queries and 256 of the `rank` value columns: with rank 512 two blocks
// make a tile's two halves and both compute its scores, because 128 rows x 512 columns of float32 sums would be all of tensor memory.
// Tiles of 64 keys.  384 threads:
//   warp 0     TMA producer: a tile's cached vectors in boxes of 8 keys x 4 blocks of 64 entries (128-byte swizzle; a page of 16 keys in boxes of one
//              block each was bound by the number of boxes), so that a tile's four blocks that are also this block's values, and the four that only
//              the scores read, lie as groups of eight keys 4 KB apart; the rotated part apart from them.  Values: a ring of two tiles (three
//              where there is room), the others one tile, the rotated parts two.
//   warp 1     owns tensor memory and issues the MMAs: S = Q Z^T (both K-major; QT blocks of Q lie in tensor memory, the others in
//              shared memory, which does not hold all of Q beside the rings), and, with P as the operand in tensor memory,
//              P V (V read MN-major) into an accumulator that starts anew with every tile.  S of the next tile is issued
//              before P V of this one, and its softmax runs beside it.
//   warps 4-11 two threads a row, 32 keys and 128 value columns each.  Softmax: the running maximum (the two threads exchange theirs
//              through shared memory), weights as powers of two, which go to tensor memory as three bfloat16 terms
//              p = p1 + p2 + p3 (24 bits of mantissa: they are not rounded).  The sums O stay in registers: a tile's P V is read
//              from tensor memory and added in rounded float32 arithmetic, O = O 2^(m_old - m_new) + P V, so that the accumulator,
//              which cuts off what it cannot hold, is never longer than a tile, and a new maximum costs nothing.
// Queries come as float32 [tokens, heads, za] (rounded to bfloat16 here) or as bfloat16 [heads, tq_pad, za]; the result leaves as
// bfloat16 [heads, t_pad, rank] or float32 [tokens, heads, rank].
//
// What bounds it: the MMAs.  A tile of 64 keys is 36 MMAs of 64 columns for the scores (32 cycles each, about 48 where Q comes from shared
// memory, which serves 128 bytes a clock) and 12 of 256 columns for the sums (128 cycles): 3,100 cycles; the softmax of the
// next tile and the sums of the last run beside them (measured: 3,300 cycles a tile; a block's queries cost 14,000 cycles once, read as float32).
// Prompts of 666 and 1,333 tokens, 16 heads, rank 512: 476 us with mma.sync (csrc/latent_attention.cu), 129 us here.
//
// Rows of z behind a sequence's last key are cleared before they are multiplied by weights of zero, so that what another request left
// there is nothing to this one.  Every wait is bounded; a wait that gives up raises `*error_flag`.
#define LLMK_MODULE_NAME "latent_attention_tc"
#include "common.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <type_traits>

LLMK_DEFINE_LAST_ERROR()

namespace {

constexpr int BM = 128;         // rows of a block
constexpr int KT = 64;          // keys of a tile
constexpr int VB = 4;           // blocks of 64 value columns of a block
constexpr int NV = 64 * VB;
constexpr int THREADS = 384, ROW_THREADS = 256;
constexpr int RS = 2;           // ring of rotated parts
constexpr int TERMS = 3;

struct Params {
    const float* qa;            // [tokens, heads, za]
    const bf16* qa_hm;          // or, if set, [heads, tq_pad, za]
    float* out;                 // [tokens, heads, rank]
    bf16* out_hm;               // or, if set, [heads, t_pad, rank]
    const int* block_tables;
    const int* ctx_len;
    const int* cu_q;
    const int* tile_seq;
    const int* tile_q0;
    int* error_flag;
    int tq_pad, t_pad, max_blocks, heads, rank, window, bq, halves, page_shift;
    float scale_log2;
};

// ZB: blocks of 64 entries of a cached vector (4 or 8 of the latent, one of the rotated part); QT: blocks of Q in tensor memory
template <int ZB, int QT>
struct Layout {
    static constexpr int Q_BLOCK = BM * 128, Z_BLOCK = KT * 128, QUAD = VB * Z_BLOCK;
    static constexpr int OTHERS = ZB - 1 - VB;                                  // blocks of the latent that are no values of this block: 0 or 4
    static constexpr int VS = OTHERS ? 2 : 3;                                   // ring of values
    static constexpr int Q_OFF = 0;
    static constexpr int N_OFF = Q_OFF + (ZB - QT) * Q_BLOCK;
    static constexpr int V_OFF = N_OFF + (OTHERS ? QUAD : 0);
    static constexpr int R_OFF = V_OFF + VS * QUAD;
    static constexpr int XCHG_OFF = R_OFF + RS * Z_BLOCK;                       // float [2][2][BM]
    static constexpr int TURN_OFF = XCHG_OFF + 2 * 2 * BM * 4;                  // QT: 2 KB a warp, where rows of Q turn from lanes side by side to lanes of their own
    static constexpr int BAR_OFF = TURN_OFF + (QT ? ROW_THREADS / 32 * 2048 : 0);
    static constexpr int NUM_BARS = 2 + 2 * VS + 2 * RS + 5;
    static constexpr int TOTAL = BAR_OFF + NUM_BARS * 8 + 16;                   // (no static shared memory: the base lies on 1024 bytes)
    // tensor memory
    static constexpr uint32_t O_COL = 0, S_COL = NV, P_COL = S_COL + KT, Q_COL = P_COL + TERMS * KT / 2;
    static_assert(Q_COL + QT * 32 <= 512, "tensor memory");
    static_assert(OTHERS == 0 || OTHERS == VB, "blocks of a cached vector");
};

// The entry block that is read at place `pos` of the scores' order: the blocks that are no values of this block, the rotated part, its values.
template <int ZB, int QT>
__device__ __forceinline__ int block_at(int pos, int half) {
    using L = Layout<ZB, QT>;
    if (pos < L::OTHERS) return (half ^ 1) * VB + pos;
    return pos == L::OTHERS ? ZB - 1 : half * VB + pos - L::OTHERS - 1;
}

// Where key `key` of block `b` lies in four blocks that came in boxes of eight keys
__device__ __forceinline__ int quad_row(int key, int b) { return (key / 8 * VB + b) * 1024 + key % 8 * 128; }

__device__ __forceinline__ float pow2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int ZB, int QT>
__global__ void __launch_bounds__(THREADS, 1) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_r,
                                                                       const Params p) {
    using L = Layout<ZB, QT>;
    constexpr uint32_t TMEM_COLS = 512;
    constexpr int VS = L::VS, GROUPS = KT / 8;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (p.tile_seq[blockIdx.y] < 0) {       // padding of a list of fixed length
        pdl_wait();
        return;
    }
    if ((tc::smem_u32(smem) & 1023u) != 0) {      // uniform over the block: nothing has been set up yet
        if (threadIdx.x == 0 && p.error_flag) atomicExch(p.error_flag, 2);
        return;
    }
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint64_t* n_full = bars;                // 1
    uint64_t* n_empty = n_full + 1;         // 1
    uint64_t* r_full = n_empty + 1;         // RS
    uint64_t* r_empty = r_full + RS;        // RS
    uint64_t* v_full = r_empty + RS;        // VS
    uint64_t* v_empty = v_full + VS;        // VS
    uint64_t* q_full = v_empty + VS;        // every row thread
    uint64_t* s_full = q_full + 1;
    uint64_t* s_read = s_full + 1;          // every row thread
    uint64_t* p_full = s_read + 1;          // every row thread
    uint64_t* o_full = p_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NUM_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same for all lanes, and known to be)
    const int half = blockIdx.x;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < L::NUM_BARS; ++i) {
            const uint64_t* b = bars + i;
            tc::mbar_init(tc::smem_u32(b), b == q_full || b == s_read || b == p_full ? ROW_THREADS : 1);
        }
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_z);
        tc::prefetch_tensormap(&map_r);
    }
    if (warp == 1) {
        tc::tmem_alloc(tc::smem_u32(tmem_slot), TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) pdl_launch_dependents();      // (behind the allocation: the next kernel's blocks must not get their tensor memory first)
    pdl_wait();

    const int s = p.tile_seq[blockIdx.y];
    const int q0 = p.tile_q0[blockIdx.y];
    const int q_beg = p.cu_q[s];
    const int q_len = p.cu_q[s + 1] - q_beg;
    const int ctx = p.ctx_len[s];
    const int nq_tile = min(p.bq, q_len - q0);
    const int first_pos = ctx - q_len + q0;
    int kt0 = 0, n_tiles = 0, k_beg = 0;
    if (ctx >= q_len && nq_tile > 0) {
        k_beg = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
        kt0 = k_beg / KT * KT;
        n_tiles = (first_pos + nq_tile - kt0 + KT - 1) / KT;
    }

    // Registers: the launch's 3 x 128 x 168 are shared out anew, 72 a thread for warps 0 to 3 and 216 for the rows (504 of 504)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        // The whole warp walks the loops of both issuing roles and one lane issues: what the instructions are given is then known to be the same for all
        // lanes and kept where they read it.
        const bool issues = tc::elect_one();
        if (warp == 0) {
            if (n_tiles > 0) {
                const int* bt = p.block_tables + (size_t)s * p.max_blocks;
                const int last_page = (ctx - 1) >> p.page_shift, in_page = (1 << p.page_shift) - 1;
                // The cache rows of a tile's groups of eight keys; pages past the sequence's last one, or given back by a window (id -1), are replaced by
                // the last page: their keys are masked.  The ids of the next tile are asked for while this one's copies are sent.
                int rows[GROUPS], next[GROUPS];
                auto look_up = [&](int k0) {
#pragma unroll
                    for (int g = 0; g < GROUPS; ++g) next[g] = __ldg(bt + min((k0 + g * 8) >> p.page_shift, last_page));
                };
                look_up(kt0);
                bool ok = true;
                auto load_quad = [&](uint32_t dst, uint32_t bar, int block) {
                    if (!issues) return;
                    tc::mbar_expect_tx(bar, L::QUAD);
#pragma unroll
                    for (int g = 0; g < GROUPS; ++g) tc::tma_load_3d(dst + g * VB * 1024, &map_z, bar, 0, rows[g], block);
                };
                int loaded = 0;
                for (int j = 0; j < n_tiles && ok; ++j) {
                    const int k0 = kt0 + j * KT;
#pragma unroll
                    for (int g = 0; g < GROUPS; ++g) {
                        const int page = next[g] < 0 ? __ldg(bt + last_page) : next[g];
                        rows[g] = (page << p.page_shift) + ((k0 + g * 8) & in_page);
                    }
                    if (j + 1 < n_tiles) look_up(k0 + KT);
                    if constexpr (L::OTHERS > 0) {
                        ok = tc::mbar_wait_warp(tc::smem_u32(n_empty), (j & 1) ^ 1, abort_flag);
                        if (!ok) break;
                        load_quad(tc::smem_u32(smem + L::N_OFF), tc::smem_u32(n_full), (half ^ 1) * VB);
                    }
                    const int rs = j % RS, st = j % VS;
                    ok = tc::mbar_wait_warp(tc::smem_u32(&r_empty[rs]), ((j / RS) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    if (issues) tc::mbar_expect_tx(tc::smem_u32(&r_full[rs]), L::Z_BLOCK);
#pragma unroll
                    for (int g = 0; g < KT / 16; ++g)
                        if (issues) tc::tma_load_3d(tc::smem_u32(smem + L::R_OFF + rs * L::Z_BLOCK + g * 16 * 128), &map_r, tc::smem_u32(&r_full[rs]), 0,
                                        rows[2 * g], ZB - 1);
                    ok = tc::mbar_wait_warp(tc::smem_u32(&v_empty[st]), ((j / VS) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    load_quad(tc::smem_u32(smem + L::V_OFF + st * L::QUAD), tc::smem_u32(&v_full[st]), half * VB);
                    loaded = j + 1;
                }
                if (*abort_flag) {
                    // let the copies that are in flight land before the block's memory is given up (of the tile that was not finished too)
                    auto drain = [](uint32_t bar, uint32_t parity) {
                        const long long t0 = clock64();
                        while (!tc::mbar_try_wait(bar, parity) && clock64() - t0 < tc::WAIT_LIMIT_CYCLES / 8) {
                        }
                    };
                    for (int k = max(loaded - 2, 0); k < loaded + 1; ++k) {
                        if (L::OTHERS > 0) drain(tc::smem_u32(n_full), k & 1);
                        drain(tc::smem_u32(&r_full[k % RS]), (k / RS) & 1);
                        drain(tc::smem_u32(&v_full[k % VS]), (k / VS) & 1);
                    }
                }
            }
        } else if (warp == 1) {
            if (n_tiles > 0) {
                constexpr uint32_t idesc_s = tc::idesc_bf16_f32(BM, KT);
                constexpr uint32_t idesc_o = tc::idesc_bf16_f32_b_mn(BM, NV);
                const uint64_t q_desc = tc::smem_desc_sw128(tc::smem_u32(smem + L::Q_OFF));
                // groups of eight keys: 4 KB apart in four blocks, 1 KB in the rotated part
                constexpr uint64_t APART = (uint64_t)((VB * 1024 - 1024) >> 4) << 32;
                const uint64_t n_desc = tc::smem_desc_sw128(tc::smem_u32(smem + L::N_OFF)) + APART;
                const uint64_t vk_desc = tc::smem_desc_sw128(tc::smem_u32(smem + L::V_OFF)) + APART;
                const uint64_t r_desc = tc::smem_desc_sw128(tc::smem_u32(smem + L::R_OFF));
                const uint64_t v_desc = tc::smem_desc_sw128_mn(tc::smem_u32(smem + L::V_OFF), 1024, VB * 1024);
                auto issue_scores = [&](int j) -> bool {
                    const int rs = j % RS, st = j % VS;
#pragma unroll
                    for (int pos = 0; pos < ZB; ++pos) {
                        uint64_t b_desc;
                        if (pos < L::OTHERS) {
                            if (pos == 0 && !tc::mbar_wait_warp(tc::smem_u32(n_full), j & 1, abort_flag)) return false;
                            b_desc = n_desc + (uint64_t)((pos * 1024) >> 4);
                        } else if (pos == L::OTHERS) {
                            if (!tc::mbar_wait_warp(tc::smem_u32(&r_full[rs]), (j / RS) & 1, abort_flag)) return false;
                            b_desc = r_desc + (uint64_t)((rs * L::Z_BLOCK) >> 4);
                        } else {
                            if (pos == L::OTHERS + 1 && !tc::mbar_wait_warp(tc::smem_u32(&v_full[st]), (j / VS) & 1, abort_flag)) return false;
                            b_desc = vk_desc + (uint64_t)((st * L::QUAD + (pos - L::OTHERS - 1) * 1024) >> 4);
                        }
                        tc::tc_fence_after_sync();
                        if (!issues) continue;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint64_t at = (uint64_t)((k * 32) >> 4);
                            if (pos < QT)
                                tc::mma_bf16_ts(tmem_base + L::S_COL, tmem_base + L::Q_COL + (uint32_t)(pos * 32 + k * 8), b_desc + at, idesc_s,
                                                pos != 0 || k != 0);
                            else
                                tc::mma_bf16_ss(tmem_base + L::S_COL, q_desc + (uint64_t)(((pos - QT) * L::Q_BLOCK) >> 4) + at, b_desc + at, idesc_s,
                                                pos != 0 || k != 0);
                        }
                        if (pos == L::OTHERS - 1) tc::mma_commit(tc::smem_u32(n_empty));
                        if (pos == L::OTHERS) tc::mma_commit(tc::smem_u32(&r_empty[rs]));
                    }
                    if (issues) tc::mma_commit(tc::smem_u32(s_full));
                    return true;
                };
                bool ok = tc::mbar_wait_warp(tc::smem_u32(q_full), 0, abort_flag);
                if (ok) tc::tc_fence_after_sync();
                ok = ok && issue_scores(0);
                for (int j = 0; j < n_tiles && ok; ++j) {
                    // the next tile's scores in front of P V, beside which their softmax then runs; its values arrive beside the scores of the other blocks
                    if (j + 1 < n_tiles) {
                        ok = tc::mbar_wait_warp(tc::smem_u32(s_read), j & 1, abort_flag);
                        if (!ok) break;
                        tc::tc_fence_after_sync();
                        ok = issue_scores(j + 1);
                    }
                    ok = ok && tc::mbar_wait_warp(tc::smem_u32(p_full), j & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                    const uint64_t v_tile = v_desc + (uint64_t)((j % VS * L::QUAD) >> 4);
                    if (issues) {
#pragma unroll
                        for (int term = TERMS - 1; term >= 0; --term)           // the smaller terms first
#pragma unroll
                            for (int kk = 0; kk < KT / 16; ++kk)
                                tc::mma_bf16_ts(tmem_base + L::O_COL, tmem_base + L::P_COL + (uint32_t)(term * (KT / 2) + kk * 8),
                                                v_tile + (uint64_t)((kk * 2 * VB * 1024) >> 4), idesc_o, term != TERMS - 1 || kk != 0);
                        tc::mma_commit(tc::smem_u32(o_full));
                        tc::mma_commit(tc::smem_u32(&v_empty[j % VS]));
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        // Warp w may touch tensor-memory lanes 32 * (w % 4) .. + 31; a row belongs to two warps: `side` 0 has its first 32 keys of a tile and
        // the first half of this block's value columns, `side` 1 the others.
        const int quarter = warp & 3, side = (warp - 4) >> 2;
        const int r = quarter * 32 + lane, tid = threadIdx.x - 128;
        // index of this lane's row among the queries and among the results (tokens x heads in either layout); -1: nobody's row
        int source = -1, place = -1;
        {
            const int qi = r / p.heads, hh = r % p.heads, tok = q_beg + q0 + qi;
            if (r < p.bq * p.heads && qi < nq_tile) {
                source = p.qa_hm ? hh * p.tq_pad + tok : tok * p.heads + hh;
                place = p.out_hm ? hh * p.t_pad + tok : tok * p.heads + hh;
            }
        }
        const bool live = source >= 0;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        if (n_tiles > 0) {
            constexpr int ZA = ZB * 64;
            // Q: all of a thread's vectors of a part are asked for before the first is used (a branch around each load made this 20,000 cycles, half of
            // what a block took on the average); rows of nobody read the first query and are cleared
            auto load_q = [&](auto head_major) {
                using Vec = std::conditional_t<decltype(head_major)::value, uint2, float4>;         // four entries
                auto entries = [&](int src, int col) -> Vec {
                    const size_t at = (size_t)max(src, 0) * ZA + col;
                    if constexpr (decltype(head_major)::value) return *reinterpret_cast<const uint2*>(p.qa_hm + at);
                    else return *reinterpret_cast<const float4*>(p.qa + at);
                };
                auto rounded = [&](int src, const Vec& f) -> uint2 {
                    if (src < 0) return make_uint2(0u, 0u);
                    if constexpr (decltype(head_major)::value) return f;
                    else {
                        const __nv_bfloat162 a = __floats2bfloat162_rn(f.x, f.y), b = __floats2bfloat162_rn(f.z, f.w);
                        return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
                    }
                };
                // In tensor memory: a lane's row, two entries a column; this warp has 32 rows and 32 entries of each block.  Eight lanes read a row's 32
                // entries side by side, a lane then takes its own row.
                if constexpr (QT > 0) {
                    Vec v[QT][8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int src = __shfl_sync(0xffffffffu, source, i * 4 + lane / 8);
#pragma unroll
                        for (int pos = 0; pos < QT; ++pos) v[pos][i] = entries(src, block_at<ZB, QT>(pos, half) * 64 + side * 32 + lane % 8 * 4);
                    }
                    uint8_t* turn = smem + L::TURN_OFF + (warp - 4) * 2048;
#pragma unroll
                    for (int pos = 0; pos < QT; ++pos) {
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            *reinterpret_cast<uint2*>(turn + (i * 4 + lane / 8) * 64 + lane % 8 * 8) =
                                rounded(__shfl_sync(0xffffffffu, source, i * 4 + lane / 8), v[pos][i]);
                        __syncwarp();
                        uint32_t w[16];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 x = *reinterpret_cast<const uint4*>(turn + lane * 64 + i * 16);
                            w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
                        }
                        tc::tmem_st_32x16(tmem_base + lane_addr + L::Q_COL + (uint32_t)(pos * 32 + side * 16), w);
                    }
                }
                // In shared memory, in the layout of 128-byte-swizzled rows: 16 of this warp's 32 rows, 16 lanes take 64 entries of a row, four each
                const int c4 = lane & 15;
#pragma unroll 1
                for (int k0 = 0; k0 < 8; k0 += 4) {
                    Vec v[4][ZB - QT];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int src = __shfl_sync(0xffffffffu, source, side * 16 + (k0 + u) * 2 + lane / 16);
#pragma unroll
                        for (int pos = QT; pos < ZB; ++pos) v[u][pos - QT] = entries(src, block_at<ZB, QT>(pos, half) * 64 + c4 * 4);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int in_warp = side * 16 + (k0 + u) * 2 + lane / 16, row = quarter * 32 + in_warp;
                        const int src = __shfl_sync(0xffffffffu, source, in_warp);
#pragma unroll
                        for (int pos = QT; pos < ZB; ++pos)
                            *reinterpret_cast<uint2*>(smem + L::Q_OFF + (pos - QT) * L::Q_BLOCK + row * 128 + (((c4 >> 1) ^ (row & 7)) << 4) +
                                                      (c4 & 1) * 8) = rounded(src, v[u][pos - QT]);
                    }
                }
            };
            if (p.qa_hm) load_q(std::true_type());
            else load_q(std::false_type());
            tc::tmem_st_wait();
            tc::fence_proxy_async();
            tc::tc_fence_before_sync();
            tc::mbar_arrive(tc::smem_u32(q_full));
        }
        const int qpos = first_pos + r / p.heads;
        const int lo = p.window > 0 ? qpos - p.window : -1;      // keys at positions > lo are seen
        const uint32_t s_addr = tmem_base + lane_addr + L::S_COL + (uint32_t)(side * 32);
        const uint32_t p_addr = tmem_base + lane_addr + L::P_COL + (uint32_t)(side * 16);
        const uint32_t o_addr = tmem_base + lane_addr + L::O_COL + (uint32_t)(side * (NV / 2));
        float* xchg = reinterpret_cast<float*>(smem + L::XCHG_OFF);      // [2 tiles][2 sides][128 rows]
        const int pair_barrier = 1 + quarter;                    // a row's two warps
        const float scale2 = p.scale_log2;
        float o[NV / 2];
#pragma unroll
        for (int i = 0; i < NV / 2; ++i) o[i] = 0.f;
        float m = -INFINITY, l = 0.f, alpha = 0.f;
        // O = O alpha + P V of the last tile
        auto add_tile = [&]() {
#pragma unroll
            for (int c = 0; c < NV / 64; ++c) {
                uint32_t t[32];
                tc::tmem_ld_32x32_wait(o_addr + (uint32_t)(c * 32), t);
#pragma unroll
                for (int i = 0; i < 32; ++i) o[c * 32 + i] = fmaf(o[c * 32 + i], alpha, __uint_as_float(t[i]));
            }
        };
        for (int j = 0; j < n_tiles; ++j) {
            const int k0 = kt0 + j * KT + side * 32;             // this thread's first key
            ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(s_full), j & 1, abort_flag));
            uint32_t v[32];
            tc::tc_fence_after_sync();
            if (ok) {
                tc::tmem_ld_32x32_wait(s_addr, v);
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = 0u;
            }
            tc::tc_fence_before_sync();
            if (ok) tc::mbar_arrive(tc::smem_u32(s_read));
            if (__any_sync(0xffffffffu, live && (k0 + 31 > qpos || k0 <= lo))) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (live && (k0 + i > qpos || k0 + i <= lo)) v[i] = 0xff800000u;         // -inf
            }
            float mx4[4] = {__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3])};
#pragma unroll
            for (int i = 4; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[i]));
            const float mx_own = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            float* x = xchg + (j & 1) * 2 * BM;
            x[side * BM + r] = mx_own;
            asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
            const float m_new = fmaxf(m, fmaxf(mx_own, x[(side ^ 1) * BM + r]));
            const float base = m_new > -INFINITY ? m_new * scale2 : 0.f;         // a row that has seen nothing: every weight 2^-inf
            const float alpha_new = pow2(fmaf(m, scale2, -base));
            m = m_new;
            float pv[32], sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                pv[i] = pow2(fmaf(__uint_as_float(v[i]), scale2, -base));
                sum4[i & 3] += pv[i];
            }
            l = l * alpha_new + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            uint32_t w[TERMS][16];
#pragma unroll
            for (int term = 0; term < TERMS; ++term)
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(pv[2 * i], pv[2 * i + 1]);
                    w[term][i] = *reinterpret_cast<const uint32_t*>(&h);
                    if (term + 1 < TERMS) {                      // what is left of them (exact)
                        pv[2 * i] -= __uint_as_float(w[term][i] << 16);
                        pv[2 * i + 1] -= __uint_as_float(w[term][i] & 0xffff0000u);
                    }
                }
            if (!ok) continue;          // (both warps of a row meet at the barrier above in every turn, whatever happens)
            if (j == 0 || j == n_tiles - 1) {
                // Keys of this tile that no row of it sees, in front of a window or behind the last query: their vectors are cleared.  (The scores of
                // this tile are there, so its vectors are, and nothing reads these rows of them but P V.)
                const int seen = first_pos + nq_tile - (kt0 + j * KT), gone = j == 0 ? k_beg - kt0 : 0;
                uint8_t* vt = smem + L::V_OFF + j % VS * L::QUAD;
                for (int idx = tid; idx < KT * VB * 8; idx += ROW_THREADS) {
                    const int key = idx / (VB * 8), at = idx % (VB * 8);
                    if (key < gone || key >= seen) *reinterpret_cast<uint4*>(vt + quad_row(key, at / 8) + at % 8 * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                tc::fence_proxy_async();
            }
            // P V of the tile before has been computed: its operand may be replaced and its result read
            if (j > 0) {
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(o_full), (j - 1) & 1, abort_flag));
                tc::tc_fence_after_sync();
                if (!ok) continue;
            }
#pragma unroll
            for (int term = 0; term < TERMS; ++term) tc::tmem_st_32x16(p_addr + (uint32_t)(term * (KT / 2)), w[term]);
            if (j > 0) add_tile();
            alpha = alpha_new;
            tc::tmem_st_wait();
            tc::tc_fence_before_sync();
            tc::mbar_arrive(tc::smem_u32(p_full));
        }
        if (ok && n_tiles > 0) {
            ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(o_full), (n_tiles - 1) & 1, abort_flag));
            tc::tc_fence_after_sync();
            if (ok) add_tile();
        }
        // the row's sum is its two threads' sums (both were kept against the same maxima)
        asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");       // every read of the last tiles' maxima is done
        xchg[side * BM + r] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
        const float l_row = l + xchg[(side ^ 1) * BM + r];
        float inv = l_row > 0.f ? 1.0f / l_row : 0.f;
        if (l_row != l_row) inv = l_row;                         // a score that is no number: its row is none
        if (ok) {
            // A warp's 32 rows of 128 columns turn round where Q was (every score has been computed): a row's columns then leave side by side.
            const int col = half * NV + side * (NV / 2);
            uint8_t* own = smem + L::Q_OFF + (warp - 4) * (32 * 256);
            if (p.out_hm) {
#pragma unroll
                for (int i = 0; i < NV / 16; ++i) {
                    float f[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = o[8 * i + e] * inv;
                    Vec16<bf16> pk;
                    pk.pack(f);
                    *reinterpret_cast<uint4*>(own + lane * 256 + ((i ^ (lane & 15)) << 4)) = pk.raw;
                }
                __syncwarp();
#pragma unroll 4
                for (int i = 0; i < 16; ++i) {
                    const int row = 2 * i + lane / 16, c = lane % 16;
                    const int to = __shfl_sync(0xffffffffu, place, row);
                    if (to >= 0) *reinterpret_cast<uint4*>(p.out_hm + (size_t)to * p.rank + col + c * 8) = *reinterpret_cast<const uint4*>(own + row * 256 + ((c ^ (row & 15)) << 4));
                }
            } else {
#pragma unroll
                for (int part = 0; part < 2; ++part) {           // 64 columns at a time
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float* x = o + part * 64 + 4 * i;
                        *reinterpret_cast<float4*>(own + lane * 256 + ((i ^ (lane & 15)) << 4)) = make_float4(x[0] * inv, x[1] * inv, x[2] * inv, x[3] * inv);
                    }
                    __syncwarp();
#pragma unroll 4
                    for (int i = 0; i < 16; ++i) {
                        const int row = 2 * i + lane / 16, c = lane % 16;
                        const int to = __shfl_sync(0xffffffffu, place, row);
                        if (to >= 0)
                            *reinterpret_cast<float4*>(p.out + (size_t)to * p.rank + col + part * 64 + c * 4) =
                                *reinterpret_cast<const float4*>(own + row * 256 + ((c ^ (row & 15)) << 4));
                    }
                }
            }
        }
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag && p.error_flag) atomicExch(p.error_flag, 1);
}

template <int ZB, int QT>
int launch(const CUtensorMap& mz, const CUtensorMap& mr, const Params& p, dim3 grid, cudaStream_t s) {
    using L = Layout<ZB, QT>;
    auto kernel = latent_attention_tc_kernel<ZB, QT>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
        if (e != cudaSuccess) LLMK_FAIL("latent_attention_tc: cannot raise shared memory to %d: %s", L::TOTAL, cudaGetErrorString(e));
        configured = true;
    }
    LLMK_CHECK_LAUNCH_RC("latent_attention_tc", llmk_launch(kernel, grid, dim3(THREADS), L::TOTAL, s, true, mz, mr, p));
    return LLMK_OK;
}

}  // namespace

// Queries per tile (128 rows of queries x heads), or 0: these sizes are not taken.  (rank 256 and 512 with a rotated part of 64: sums of
// 256 columns a block, one block or two a tile.)
LLMK_EXPORT int llmk_latent_attention_tc_tile_queries(int heads, int rank, int rot, int page_size, int dtype) {
    if (dtype != LLMK_BF16 || heads <= 0 || heads > BM || rot != 64 || (rank != 256 && rank != 512)) return 0;
    if (page_size != 16 && page_size != 32 && page_size != 64 && page_size != 128) return 0;
    return BM / heads;
}

// The arguments of `llmk_latent_attention` (csrc/latent_attention.cu) for whole key ranges; tiles of `llmk_latent_attention_tc_tile_queries`
// queries; `cache_rows`: tokens that the cache array holds.  Exactly one of qa / qa_hm and of out / out_hm is given.
LLMK_EXPORT int llmk_latent_attention_tc(float* out, const float* qa, const void* cache, long long cache_rows, const int* block_tables,
                                         int max_blocks, const int* ctx_len, const int* cu_q, const int* tile_seq, const int* tile_q0, int n_tiles,
                                         int n_tokens, int heads, int rank, int rot, int page_size, float scale, int window, void* out_hm, int t_pad,
                                         const void* qa_hm, int tq_pad, int* error_flag, void* stream) {
    if (n_tiles <= 0 || n_tokens <= 0) return LLMK_OK;
    const int bq = llmk_latent_attention_tc_tile_queries(heads, rank, rot, page_size, LLMK_BF16);
    if (bq == 0) LLMK_FAIL("latent_attention_tc: sizes not taken (heads %d, rank %d, rot %d, pages of %d)", heads, rank, rot, page_size);
    if ((long long)heads * std::max(std::max(t_pad, tq_pad), n_tokens) > 0x7fffffffLL) LLMK_FAIL("latent_attention_tc: %d tokens of %d heads", n_tokens, heads);
    if (n_tiles > 65535) LLMK_FAIL("latent_attention_tc: %d tiles", n_tiles);
    if (!(scale > 0.f)) LLMK_FAIL("latent_attention_tc: scale %g (the maxima are those of unscaled scores)", (double)scale);
    if (!qa_hm == !qa || !out_hm == !out) LLMK_FAIL("latent_attention_tc: one array of queries and one of results");
    if (!host_aligned16(cache) || !host_aligned16(qa) || !host_aligned16(qa_hm) || !host_aligned16(out) || !host_aligned16(out_hm))
        LLMK_FAIL("latent_attention_tc: arrays must start on 16-byte boundaries");
    if ((qa_hm && tq_pad < n_tokens) || (out_hm && t_pad < n_tokens)) LLMK_FAIL("latent_attention_tc: head-major arrays need room for %d tokens", n_tokens);
    Params p;
    p.qa = qa; p.qa_hm = static_cast<const bf16*>(qa_hm); p.out = out; p.out_hm = static_cast<bf16*>(out_hm);
    p.block_tables = block_tables; p.ctx_len = ctx_len; p.cu_q = cu_q; p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.error_flag = error_flag;
    p.tq_pad = tq_pad; p.t_pad = t_pad; p.max_blocks = max_blocks; p.heads = heads; p.rank = rank; p.window = window > 0 ? window : 0;
    p.bq = bq; p.halves = rank / NV;
    p.page_shift = page_size == 16 ? 4 : page_size == 32 ? 5 : page_size == 64 ? 6 : 7;
    p.scale_log2 = scale * 1.4426950408889634f;
    // the cache as [blocks of 64 entries][tokens][64]
    const uint64_t za = (uint64_t)(rank + rot);
    CUtensorMap mz, mr;
    if (!tc_host::make_map_bf16_3d(&mz, cache, 64, (uint64_t)cache_rows, za / 64, za, 64, 8, VB) ||
        !tc_host::make_map_bf16_3d(&mr, cache, 64, (uint64_t)cache_rows, za / 64, za, 64, 16, 1))
        LLMK_FAIL("latent_attention_tc: cuTensorMapEncodeTiled failed (%lld rows of %d)", cache_rows, rank + rot);
    // the halves of a tile side by side in the order of the list
    const dim3 grid(p.halves, n_tiles);
    return rank == 512 ? launch<9, 3>(mz, mr, p, grid, (cudaStream_t)stream) : launch<5, 0>(mz, mr, p, grid, (cudaStream_t)stream);
}
