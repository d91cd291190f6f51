// Matrix memories with one decay per head and token, over prompts, on the tensor cores:
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T      o_t = S_t^T q_t
//
// with a per-head constant a and b = 1 (CM_CONST: the linear attention of linear_attention.cu), or with the gates of a memory under a
// running maximum (CM_MAX: memory_scan.cu's mlstm, a = exp(f + m_before - m), b = exp(i - m), and a vector n that decays with S and takes b k).
//
// A sequence's tokens are taken in chunks of 64.  With A(i, j) the weight of token j in the output of token i >= j (the decays between
// them times b_j), g_i the decays from the chunk's start through i, w_j the weight of token j in the state after the chunk:
//   chunk_memory_local   dS = K^T diag(w) V of every chunk by itself, and the chunk's whole decay
//   chunk_memory_scan    the state before each chunk, S <- decay S + dS, a thread per entry; the request's state afterwards
//   chunk_memory_out     o_i = g_i S_before^T q_i + sum_(j <= i) A(i, j) (q_i . k_j) v_j
// so nothing but the scan's one multiply-add per entry and chunk runs along the sequence.
//
// Everything is 32-bit arithmetic although the products run on `mma.sync.m16n8k16`: a float32 operand enters as THREE bfloat16 terms
// x = x1 + x2 + x3 (24 bits of mantissa), a product of two such operands as the six products of terms whose places add up to at
// most the third (what is left out is 2^-25 of the product), an operand that is bfloat16 to begin with as itself; the sums are
// float32, rounded.  What bounds it: a third of the time the tensor cores (for 2,048 tokens on 16 heads of 128 x 128, whose float32 operands take
// six products, 4 M of them), the rest the conversion of what is staged, and the latency of one block an SM.
//
// Measured (us, one sequence, 16 heads of 128 x 128, bfloat16 rows, before -> now), and the error against float64 of the rows:
//   linear attention   2,048 tokens 353 -> 115 (segments of 256 tokens walked 32 at a time on the CUDA cores), 1.9e-7 -> 0.9e-7;  512: 203 -> 45
//   running maximum    2,048 tokens 1,139 -> 106 with its gates (a walk token by token), 7.4e-7 -> 6.5e-7;  512: 324 -> 43
// What a sequence brings decides, not what the step brings: sequences of up to few_of(form) tokens keep the walks (one launch, and no state but the
// request's own to write), in steps of any size, so that a token's sums do not depend on which other requests share its step.  The walk is
// launched behind the chunks and skips the sequences that they took.  Walk -> chunks
// (us, constant decay / running maximum): one sequence of 96 tokens 50 -> 37 / 68 -> 39, 8 of 60 tokens - / 124 -> 73, 32 of 64 - / 478 -> 248; a step that counted
// its rows instead took 417 -> 1,090 / 185 -> 1,051 for a token each of 128 sequences and 729 -> 2,069 / 697 -> 2,015 for 10 tokens each of 200.
// Terms of bfloat16 are made of ordinary numbers only: an infinity would fall apart into inf - inf, and products of sixteen keys at a time would
// carry what is no number to tokens before it.  A head of a sequence whose tokens or state hold a value beyond 1e38, an infinity or a NaN, or whose
// gates add up to more than two floats can tell apart, is left to the walk too (the check reads the queries once more, and the state once).
#pragma once
#include "common.cuh"
#include <algorithm>

namespace chunk_memory {

constexpr int C = 64;           // tokens a chunk
constexpr int EB = 64;          // value columns at a time
constexpr int THREADS = 256;
constexpr int LDE = EB + 8, LDP = C + 8;      // rows of 144 bytes: eight rows' 16 bytes lie in different banks
enum { CM_CONST = 0, CM_MAX = 1 };
__host__ __device__ constexpr int few_of(int form) { return form == CM_CONST ? 64 : 48; }       // sequences of more tokens are taken in chunks

struct Params {
    const void *q, *k, *v;      // storage type, rows ldq / ldk / ldv apart, heads side by side
    long long ldq, ldk, ldv;
    float* out;                 // [tokens, H E]
    float* state;               // CM_CONST [slots, H, D, E]; CM_MAX rows `state_ld` apart: S [H, D, E], then n [H, D]
    long long state_ld;
    const float* decay;         // CM_CONST: [H]
    const float4* gates;        // CM_MAX: [tokens, H] = (i, f, -, m before the token)
    const int *cu_q, *state_slots;
    float* scratch;             // [chunks][H][entries], the chunks' decays [chunks][H], and as ints [chunks][H] and [n_seqs][H]: left to the walk
    int H, D, E, n_seqs, silu;
    int chunks, longs;          // the most chunks, and sequences taken in chunks, that the step can have
    int entries;                // of a head's state: D E, CM_MAX D E + D
    float q_scale, den_eps;
    __host__ __device__ float* decays() const { return scratch + (size_t)chunks * H * entries; }
    __host__ __device__ int* chunk_odd() const { return reinterpret_cast<int*>(decays() + (size_t)chunks * H); }
    __host__ __device__ int* odd() const { return chunk_odd() + (size_t)chunks * H; }
};

inline bool sizes_usable(int D, int E) { return (D == 64 || D == 128) && E % EB == 0; }
inline int most_longs(int form, int n_tokens, int n_seqs) { return std::min(n_seqs, n_tokens / (few_of(form) + 1)); }
// What the step's shape says: a sequence's chunks are at most its tokens / C and one more.
inline void shape(Params& p, int form, int n_tokens) {
    p.longs = most_longs(form, n_tokens, p.n_seqs);
    p.chunks = n_tokens / C + p.longs;
    p.entries = p.D * p.E + (form == CM_MAX ? p.D : 0);
}
// (0: no sequence can be long enough)
inline long long scratch_floats(int form, int n_tokens, int n_seqs, int H, int D, int E) {
    if (n_tokens <= few_of(form) || n_seqs <= 0 || !sizes_usable(D, E)) return 0;
    const long long chunks = n_tokens / C + most_longs(form, n_tokens, n_seqs);
    return chunks * H * ((long long)D * E + (form == CM_MAX ? D : 0) + 2) + (long long)n_seqs * H;
}
// What the walk behind the chunks skips: head h of sequence s.  odd: Params::odd(), null where no chunks were launched.
template <int FORM>
__device__ __forceinline__ bool taken(const int* odd, int n_tokens, int s, int h, int H) {
    return odd && n_tokens > few_of(FORM) && !odd[(size_t)s * H + h];
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const bf16* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// No ordinary number, or one beyond what a bfloat16 can hold (3.3e38) with room to spare.
__device__ __forceinline__ bool odd_value(float x) { return !(fabsf(x) < 1e38f); }
// (x, y) as NT pairs of bfloat16, the most significant first.
template <int NT>
__device__ __forceinline__ void terms(uint32_t (&t)[NT], float x, float y) {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        t[i] = *reinterpret_cast<const uint32_t*>(&v);
        if (i + 1 < NT) {
            const float2 f = __bfloat1622float2(v);
            x -= f.x;
            y -= f.y;
        }
    }
}
// Sums of products: `main` takes the products of the first terms, one MMA after the other added in rounded float32 arithmetic (the tensor cores
// cut off what an accumulator cannot hold, and always towards zero: 48 products of a sum on one accumulator were 6 times further off), `rest` the
// products of the other terms, which are 2^-8 of them and below, on an accumulator.
template <int N8>
struct Sums {
    float main[N8][4], rest[N8][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < N8; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) main[i][u] = rest[i][u] = 0.f;
    }
    __device__ __forceinline__ float at(int i, int u) const { return main[i][u] + rest[i][u]; }
};
// The products of term ta of A and term tb of B that count: places that add up to at most the last, smallest first.
template <int NA, int NB, int N8>
__device__ __forceinline__ void mma_terms(Sums<N8>& s, int n, const uint32_t (&a)[NA][4], const uint32_t (&b)[NB][4]) {
    constexpr int LAST = (NA > NB ? NA : NB) - 1;
#pragma unroll
    for (int sum = LAST; sum >= 1; --sum)
#pragma unroll
        for (int ta = 0; ta < NA; ++ta) {
            const int tb = sum - ta;
            if (tb < 0 || tb >= NB) continue;
            mma(s.rest[n], a[ta], b[tb][0], b[tb][1]);
            mma(s.rest[n + 1], a[ta], b[tb][2], b[tb][3]);
        }
    float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
    mma(x, a[0], b[0][0], b[0][1]);
    mma(y, a[0], b[0][2], b[0][3]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        s.main[n][u] += x[u];
        s.main[n + 1][u] += y[u];
    }
}

__device__ __forceinline__ float act(float x, int silu) { return silu ? __fdividef(x, 1.0f + __expf(-x)) : x; }

// Which sequence and which of its chunks chunk number `c` of the step is (s = -1: the step has fewer); or, with BY_SEQUENCE, which sequence the
// c-th of those taken in chunks is.  All threads of a warp.
struct Place {
    int s, chunk, base;         // base: number of the sequence's first chunk
};
template <int FORM>
__device__ __forceinline__ int chunks_of(const int* cu_q, int s) {
    const int tokens = cu_q[s + 1] - cu_q[s];
    return tokens > few_of(FORM) ? ceil_div(tokens, C) : 0;
}
template <int FORM, bool BY_SEQUENCE>
__device__ __forceinline__ Place place_of(const int* cu_q, int n_seqs, int c) {
    const int lane = threadIdx.x & 31, each = ceil_div(n_seqs, 32), s0 = lane * each, s1 = min(n_seqs, s0 + each);      // a run of sequences a lane
    int count = 0, found = 0;                   // their chunks, and what is counted: chunks, or sequences that have any
#pragma unroll 4
    for (int s = s0; s < s1; ++s) {
        const int n = chunks_of<FORM>(cu_q, s);
        count += n;
        found += BY_SEQUENCE ? n > 0 : n;
    }
    int base = count, upto = found;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, base, o), y = BY_SEQUENCE ? __shfl_up_sync(0xffffffffu, upto, o) : x;
        if (lane >= o) {
            base += x;
            upto += y;
        }
    }
    const unsigned holds = __ballot_sync(0xffffffffu, upto > c);
    if (!holds) return {-1, 0, 0};
    const int owner = __ffs(holds) - 1;
    base -= count;
    int s = s0, left = c - (upto - found);      // (the owner's are used)
    if (lane == owner)
        for (;; ++s) {
            const int n = chunks_of<FORM>(cu_q, s), step = BY_SEQUENCE ? n > 0 : n;
            if (left < step) break;
            left -= step;
            base += n;
        }
    base = __shfl_sync(0xffffffffu, base, owner);
    return {__shfl_sync(0xffffffffu, s, owner), c - base, base};
}

// What the weights of a chunk follow from, per token i: CM_MAX the sums F_i = f_1 + .. + f_i as two floats, i and m; CM_CONST powers of the decay.
struct Weights {
    float hi[C], lo[C], gate[C], top[C];    // CM_MAX
    float pw[C + 1];                        // CM_CONST
    float m_before;
};
template <int FORM>
__device__ __forceinline__ void make_weights(Weights& w, const Params& p, int h, int t0, int n) {
    const int tid = threadIdx.x;
    if (FORM == CM_CONST) {
        if (tid <= C) w.pw[tid] = powf(p.decay[h], (float)tid);
        return;
    }
    if (tid >= 32) return;
    double f[2], sum = 0.0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = 2 * tid + u;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) g = p.gates[(size_t)(t0 + i) * p.H + h];
        if (i == 0) w.m_before = g.w;
        w.gate[i] = i < n ? g.x : 0.f;
        w.top[i] = i < n ? fmaxf(g.y + g.w, g.x) : 0.f;
        sum += (double)g.y;
        f[u] = sum;
    }
    double upto = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, upto, o);
        if (tid >= o) upto += x;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const double F = upto - sum + f[u];
        w.hi[2 * tid + u] = (float)F;
        w.lo[2 * tid + u] = (float)(F - (double)(float)F);
    }
}
// Whether a thread's token has gates that are no numbers, or sums of them of which `hi` and `lo` keep too little: up to 2^20 they hold 2^-28, and
// differences of two sums are exponents.
template <int FORM>
__device__ __forceinline__ bool weights_odd(const Weights& w, int n) {
    const int i = threadIdx.x;
    if (i >= n) return false;
    if (FORM == CM_CONST) return odd_value(w.pw[C]);
    return !(fabsf(w.hi[i]) <= 1048576.f) || odd_value(w.gate[i]) || odd_value(w.top[i]) || odd_value(w.m_before);
}
// The weight of token j in what token i (or the state after it) holds, i >= j.
template <int FORM>
__device__ __forceinline__ float weight(const Weights& w, int i, int j) {
    if (FORM == CM_CONST) return w.pw[i - j];
    return expf((w.hi[i] - w.hi[j]) + (w.lo[i] - w.lo[j]) + (w.gate[j] - w.top[i]));
}
// The decays from the chunk's start through token i.
template <int FORM>
__device__ __forceinline__ float from_start(const Weights& w, int i) {
    if (FORM == CM_CONST) return w.pw[i + 1];
    return expf((w.hi[i] + (w.m_before - w.top[i])) + w.lo[i]);
}

// COLS columns of a chunk's rows on their way into shared memory: `ask` sends for a thread's 16-byte vectors, all at once, and `put` writes them
// as NT terms, times `scale` per row (null: 1), zeros beyond the chunk's n tokens.
// `odd`: whether one of the thread's values is none that terms can be made of.
template <typename T, int NT, int COLS, int NTHREADS = THREADS>
struct Rows {
    static constexpr int VN = Vec16<T>::N, LD = COLS + 8, EACH = C * COLS / VN / NTHREADS;
    static_assert(EACH * VN * NTHREADS == C * COLS, "whole vectors a thread");
    Vec16<T> held[EACH];
    __device__ __forceinline__ void ask(const T* src, long long ld, int n) {
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            const int idx = threadIdx.x + i * NTHREADS, r = idx / (COLS / VN), c = idx % (COLS / VN) * VN;
            if (r < n) held[i].raw = *reinterpret_cast<const decltype(held[i].raw)*>(src + (size_t)r * ld + c);
        }
    }
    __device__ __forceinline__ bool odd(int n) const {
        bool any = false;
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            float f[VN];
            held[i].unpack(f);
            const bool row = (threadIdx.x + i * NTHREADS) / (COLS / VN) < n;
#pragma unroll
            for (int u = 0; u < VN; ++u) any |= row && odd_value(f[u]);
        }
        return any;
    }
    __device__ __forceinline__ void put(bf16* dst, int n, int silu, const float* scale) {
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            const int idx = threadIdx.x + i * NTHREADS, r = idx / (COLS / VN), c = idx % (COLS / VN) * VN;
            float f[VN];
            if (r < n) {
                if constexpr (NT == 1) {        // (bfloat16 as it is)
                    *reinterpret_cast<decltype(held[i].raw)*>(dst + r * LD + c) = held[i].raw;
                    continue;
                }
                held[i].unpack(f);
                const float s = scale ? scale[r] : 1.f;
#pragma unroll
                for (int u = 0; u < VN; ++u) f[u] = act(f[u], silu) * s;
            } else {
#pragma unroll
                for (int u = 0; u < VN; ++u) f[u] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < VN; u += 4) {
                uint32_t a[NT], b[NT];
                terms<NT>(a, f[u], f[u + 1]);
                terms<NT>(b, f[u + 2], f[u + 3]);
#pragma unroll
                for (int t = 0; t < NT; ++t) *reinterpret_cast<uint2*>(dst + (t * C + r) * LD + c + u) = make_uint2(a[t], b[t]);
            }
        }
    }
};

// Terms of q, k and v: one where they are bfloat16 values as they are stored.
template <typename T, int FORM> constexpr int input_terms() { return sizeof(T) == 2 && FORM == CM_MAX ? 1 : 3; }

// ---------------------------------------------------------------------------------------------------------------- local
// Block (chunk, head): dS [D, E], 64 columns at a time; warp w has rows 16 (w % (D / 16)) of D and, with D = 64, half of the columns.  It also looks
// for values that the terms cannot hold, in the chunk's rows, its gates and its share of the state that the sequence comes with.
template <typename T, int FORM, int D>
__global__ void __launch_bounds__(THREADS, 2) chunk_memory_local_kernel(Params p) {
    constexpr int NT = input_terms<T, FORM>(), LDD = D + 8;
    constexpr int ROW_WARPS = D / 16, COL_WARPS = 8 / ROW_WARPS, N8 = EB / 8 / COL_WARPS;
    extern __shared__ __align__(16) bf16 smem[];
    bf16* Ks = smem;                            // [NT][C][LDD]
    bf16* Vs = Ks + NT * C * LDD;               // [3][C][LDE]: the values times their weights
    __shared__ Weights w;
    __shared__ float wj[C];
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    pdl_wait();
    const Place at = place_of<FORM, false>(p.cu_q, p.n_seqs, blockIdx.x);
    if (at.s < 0) return;
    const int slot = p.state_slots[at.s];
    if (FORM == CM_CONST && slot < 0) return;
    const int q_beg = p.cu_q[at.s], q_end = p.cu_q[at.s + 1], t0 = q_beg + at.chunk * C, n = min(C, q_end - t0);
    Rows<T, NT, D> keys;
    Rows<T, 3, EB> values;
    const T* vp = static_cast<const T*>(p.v) + (size_t)t0 * p.ldv + (size_t)h * p.E;
    keys.ask(static_cast<const T*>(p.k) + (size_t)t0 * p.ldk + (size_t)h * D, p.ldk, n);
    values.ask(vp, p.ldv, n);
    make_weights<FORM>(w, p, h, t0, n);
    bool odd = keys.odd(n);
    keys.put(Ks, n, p.silu, nullptr);
    {
        Rows<T, NT, D> queries;
        queries.ask(static_cast<const T*>(p.q) + (size_t)t0 * p.ldq + (size_t)h * D, p.ldq, n);
        if (slot >= 0) {
            const float* Sg = p.state + (size_t)slot * p.state_ld;
            const int DE = D * p.E, step = ceil_div(q_end - q_beg, C) * THREADS;
            for (int i0 = at.chunk * THREADS + tid; i0 < p.entries; i0 += 16 * step) {       // sixteen asked for at once
                float x[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int i = i0 + u * step;
                    x[u] = i < p.entries ? Sg[i < DE ? (size_t)h * DE + i : (size_t)p.H * DE + (size_t)h * D + (i - DE)] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 16; ++u) odd |= odd_value(x[u]);
            }
        }
        odd |= queries.odd(n);
    }
    __syncthreads();
    odd |= weights_odd<FORM>(w, n);
    if (tid < C) wj[tid] = tid < n ? weight<FORM>(w, n - 1, tid) : 0.f;
    float* dst = p.scratch + ((size_t)blockIdx.x * p.H + h) * p.entries;
    if (tid == 0) p.decays()[(size_t)blockIdx.x * p.H + h] = from_start<FORM>(w, n - 1);
    __syncthreads();
    const int d0 = 16 * (warp % ROW_WARPS), e_warp = (warp / ROW_WARPS) * (N8 * 8);
    for (int e0 = 0; e0 < p.E; e0 += EB) {
        if (e0 > 0) __syncthreads();            // the columns before are used
        odd |= values.odd(n);
        values.put(Vs, n, p.silu, wj);
        __syncthreads();
        if (e0 + EB < p.E) values.ask(vp + e0 + EB, p.ldv, n);
        Sums<N8> acc;
        acc.clear();
        for (int j0 = 0; j0 < n; j0 += 16) {
            uint32_t a[NT][4];
#pragma unroll
            for (int t = 0; t < NT; ++t)
                ldsm4t(a[t], Ks + (t * C + j0 + (lane & 7) + (lane >> 4) * 8) * LDD + d0 + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int n8 = 0; n8 < N8; n8 += 2) {
                uint32_t b[3][4];
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    ldsm4t(b[t], Vs + (t * C + j0 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDE + e_warp + n8 * 8 + (lane >> 4) * 8);
                mma_terms(acc, n8, a, b);
            }
        }
#pragma unroll
        for (int n8 = 0; n8 < N8; ++n8) {
            float* o = dst + (size_t)(d0 + lane / 4) * p.E + e0 + e_warp + n8 * 8 + 2 * (lane & 3);
            *reinterpret_cast<float2*>(o) = make_float2(acc.at(n8, 0), acc.at(n8, 1));
            *reinterpret_cast<float2*>(o + (size_t)8 * p.E) = make_float2(acc.at(n8, 2), acc.at(n8, 3));
        }
    }
    if (FORM == CM_MAX && tid < D) {            // n's own sum
        float s = 0.f;
        for (int j = 0; j < n; ++j) {
            float k = 0.f;
#pragma unroll
            for (int t = NT - 1; t >= 0; --t) k += to_float(Ks[(t * C + j) * LDD + tid]);
            s = fmaf(wj[j], k, s);
        }
        dst[(size_t)D * p.E + tid] = s;
    }
    const int any = __syncthreads_or(odd);
    if (tid == 0) p.chunk_odd()[(size_t)blockIdx.x * p.H + h] = any;
}

// ----------------------------------------------------------------------------------------------------------------- scan
// A thread per entry of the state (CM_MAX: of n too): a chunk's sum is replaced by the state before it, eight chunks' values asked for at once.
// Blocks take (sequence, head, 256 entries) one after the other, those of sequences in chunks only: the most that a shape can have would be
// 262,144 blocks for 256 sequences of 16 heads of 128 x 128.
template <int FORM>
__global__ void __launch_bounds__(THREADS) chunk_memory_scan_kernel(Params p) {
    const int per_head = ceil_div(p.entries, THREADS);
    pdl_launch_dependents();
    pdl_wait();
    for (int item = blockIdx.x; item < p.longs * p.H * per_head; item += gridDim.x) {
        const Place seq = place_of<FORM, true>(p.cu_q, p.n_seqs, item / (per_head * p.H));
        if (seq.s < 0) return;
        const int s = seq.s, h = item / per_head % p.H, part = item % per_head, entry = part * THREADS + (int)threadIdx.x;
        const int slot = p.state_slots[s];
        if (FORM == CM_CONST && slot < 0) continue;
        const int count = ceil_div(p.cu_q[s + 1] - p.cu_q[s], C);
        const bool on = entry < p.entries;
        float* Sg = nullptr;
        if (slot >= 0 && on) {
            const int DE = p.D * p.E;
            Sg = p.state + (size_t)slot * p.state_ld + (entry < DE ? (size_t)h * DE + entry : (size_t)p.H * DE + (size_t)h * p.D + (entry - DE));
        }
        const size_t stride = (size_t)p.H * p.entries;
        float* at = p.scratch + ((size_t)seq.base * p.H + h) * p.entries + entry;
        const float* gain = p.decays() + (size_t)seq.base * p.H + h;
        float S = Sg ? *Sg : 0.f;
        float add[8], g[8];
        auto ask = [&](int c0) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                add[u] = on && c0 + u < count ? at[(size_t)(c0 + u) * stride] : 0.f;
                g[u] = c0 + u < count ? gain[(size_t)(c0 + u) * p.H] : 0.f;
            }
        };
        ask(0);
        bool any = false;
        for (int c = threadIdx.x & 31; c < count; c += 32) any |= p.chunk_odd()[(size_t)(seq.base + c) * p.H + h] != 0;
        any = __any_sync(0xffffffffu, any);
        if (part == 0 && threadIdx.x == 0) p.odd()[(size_t)s * p.H + h] = any;
        if (any) continue;
        for (int c0 = 0; c0 < count; c0 += 8) {
            if (c0 > 0) ask(c0);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (c0 + u >= count) break;
                if (on) at[(size_t)(c0 + u) * stride] = S;
                S = fmaf(g[u], S, add[u]);
            }
        }
        if (Sg) *Sg = S;
    }
}

// ------------------------------------------------------------------------------------------------------------------ out
// Block (chunk, head): warp w has rows 16 (w % 4) of the chunk and, as number w / 4 of `GROUPS`, that part of the keys (scores) or of 64 value columns
// (outputs).  Sixteen warps an SM hide more of the MMAs' and loads' chains than eight: as two blocks of eight where the operands are one term and two
// blocks' shared memory fits (a prompt of 2,048 under a running maximum, 8 heads: 28.4 -> 23.8 us; the layer's pass 296 -> 290, with one block of
// sixteen 294), as one block of sixteen where they are three (constant decay, 16 heads: 70.1 -> 66.8 us, the pass 355 -> 350).  What holds the second
// form is not its warps: the MMAs of its terms take 19 us at the rate `mma.sync` reaches alone.
// BLOCKS: blocks an SM has to have room for.  Room for two takes half of the registers from a block's chain, so where the SMs have a chunk and head each at the most
// a block has its SM for itself (`lone_blocks`): under a running maximum, the three launches, us with room for two / for one: 8 heads of 128 x 128, 100 tokens
// 33.3 / 27.8, 600 35.5 / 31.1, 1,200 40.0 / 43.1, eight of 100 53.9 / 47.8; 16 heads, 300 tokens 35.5 / 33.0, 600 41.7 / 44.0, 64 single tokens beside
// 300 143 / 127.
template <typename T, int FORM> constexpr int out_warps() { return input_terms<T, FORM>() == 1 ? 8 : 16; }
template <typename T, int FORM, int D>
struct OutLayout {
    static constexpr int NT = input_terms<T, FORM>(), LDD = D + 8;
    static constexpr int Q = NT * C * LDD, KS = (NT * C * LDD > 3 * D * LDE ? NT * C * LDD : 3 * D * LDE), P = 3 * C * LDP, V = NT * C * LDE;
    static constexpr size_t bytes() { return (size_t)(Q + KS + P + V) * sizeof(bf16); }
};
template <typename T, int FORM, int D, int BLOCKS>
__global__ void __launch_bounds__(32 * out_warps<T, FORM>(), BLOCKS) chunk_memory_out_kernel(Params p) {
    using L = OutLayout<T, FORM, D>;
    constexpr int NT = L::NT, LDD = L::LDD, WARPS = out_warps<T, FORM>(), NTHREADS = 32 * WARPS, GROUPS = WARPS / 4, N8 = 8 / GROUPS;
    extern __shared__ __align__(16) bf16 smem[];
    bf16* Qs = smem;                            // [NT][C][LDD]
    bf16* Ks = Qs + L::Q;                       // [NT][C][LDD], then the state's columns [3][D][LDE]
    bf16* Ps = Ks + L::KS;                      // [3][C][LDP]: the weighted scores
    bf16* Vs = Ps + L::P;                       // [NT][C][LDE]
    __shared__ Weights w;
    __shared__ float start[C], sums[GROUPS][C], n_dot[C];
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    pdl_wait();
    const Place at = place_of<FORM, false>(p.cu_q, p.n_seqs, blockIdx.x);
    if (at.s < 0 || (FORM == CM_CONST && p.state_slots[at.s] < 0)) return;
    const int left = p.odd()[(size_t)at.s * p.H + h];
    const int q_beg = p.cu_q[at.s], t0 = q_beg + at.chunk * C, n = min(C, p.cu_q[at.s + 1] - t0);
    const float* before = p.scratch + ((size_t)blockIdx.x * p.H + h) * p.entries;
    // the state's entries of 64 columns, float4 a thread and turn: asked for early, put down where the keys were
    constexpr int SV = D * EB / 4 / NTHREADS;
    float4 held[SV];
    auto ask = [&](int e0) {
#pragma unroll
        for (int i = 0; i < SV; ++i) {
            const int idx = tid + i * NTHREADS, d = idx / (EB / 4), c = idx % (EB / 4) * 4;
            held[i] = *reinterpret_cast<const float4*>(before + (size_t)d * p.E + e0 + c);
        }
    };
    const T* vp = static_cast<const T*>(p.v) + (size_t)t0 * p.ldv + (size_t)h * p.E;
    Rows<T, NT, EB, NTHREADS> values;
    {
        Rows<T, NT, D, NTHREADS> queries, keys;
        queries.ask(static_cast<const T*>(p.q) + (size_t)t0 * p.ldq + (size_t)h * D, p.ldq, n);
        keys.ask(static_cast<const T*>(p.k) + (size_t)t0 * p.ldk + (size_t)h * D, p.ldk, n);
        values.ask(vp, p.ldv, n);
        ask(0);
        if (left) return;                       // (all threads of the block)
        make_weights<FORM>(w, p, h, t0, n);
        queries.put(Qs, n, p.silu, nullptr);
        keys.put(Ks, n, p.silu, nullptr);
    }
    __syncthreads();
    if (tid < C) start[tid] = tid < n ? from_start<FORM>(w, tid) * p.q_scale : 0.f;
    const int r0 = 16 * (warp & 3), group = warp >> 2;
    // scores of 16 rows and the group's keys, those of keys behind all rows left out
    {
        Sums<N8> s;
        s.clear();
        const int j0 = 8 * N8 * group;
        if (j0 <= r0 + 15) {
#pragma unroll 2
            for (int d = 0; d < D; d += 16) {
                uint32_t a[NT][4];
#pragma unroll
                for (int t = 0; t < NT; ++t) ldsm4(a[t], Qs + (t * C + r0 + (lane & 15)) * LDD + d + (lane >> 4) * 8);
#pragma unroll
                for (int n8 = 0; n8 < N8; n8 += 2) {
                    if (j0 + 8 * n8 > r0 + 15) continue;
                    uint32_t b[NT][4];
#pragma unroll
                    for (int t = 0; t < NT; ++t)
                        ldsm4(b[t], Ks + (t * C + j0 + 8 * n8 + (lane & 7) + (lane >> 4) * 8) * LDD + d + ((lane >> 3) & 1) * 8);
                    mma_terms(s, n8, a, b);
                }
            }
        }
        float row_sum[2] = {0.f, 0.f};
#pragma unroll
        for (int n8 = 0; n8 < N8; ++n8)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = r0 + lane / 4 + 8 * u, j = j0 + 8 * n8 + 2 * (lane & 3);
                float x = 0.f, y = 0.f;
                if (j <= i && i < n) x = s.at(n8, 2 * u) * (weight<FORM>(w, i, j) * p.q_scale);
                if (j + 1 <= i && i < n) y = s.at(n8, 2 * u + 1) * (weight<FORM>(w, i, j + 1) * p.q_scale);
                row_sum[u] += x + y;
                uint32_t t[3];
                terms<3>(t, x, y);
#pragma unroll
                for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(Ps + (k * C + i) * LDP + j) = t[k];
            }
        if (FORM == CM_MAX) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                row_sum[u] += __shfl_xor_sync(0xffffffffu, row_sum[u], 1);
                row_sum[u] += __shfl_xor_sync(0xffffffffu, row_sum[u], 2);
                if ((lane & 3) == 0) sums[group][r0 + lane / 4 + 8 * u] = row_sum[u];
            }
            // q . n, a row a warp in turn
            const float* nb = before + (size_t)D * p.E;
            for (int i = warp; i < n; i += WARPS) {
                float x = 0.f;
#pragma unroll
                for (int d = lane; d < D; d += 32) {
                    float q = 0.f;
#pragma unroll
                    for (int t = NT - 1; t >= 0; --t) q += to_float(Qs[(t * C + i) * LDD + d]);
                    x = fmaf(q, nb[d], x);
                }
                x = warp_sum(x);
                if (lane == 0) n_dot[i] = x;
            }
        }
    }
    for (int e0 = 0; e0 < p.E; e0 += EB) {
        __syncthreads();                        // the keys, or the columns before, are used
#pragma unroll
        for (int i = 0; i < SV; ++i) {
            const int idx = tid + i * NTHREADS, d = idx / (EB / 4), c = idx % (EB / 4) * 4;
            uint32_t a[3], b[3];
            terms<3>(a, held[i].x, held[i].y);
            terms<3>(b, held[i].z, held[i].w);
#pragma unroll
            for (int t = 0; t < 3; ++t) *reinterpret_cast<uint2*>(Ks + (t * D + d) * LDE + c) = make_uint2(a[t], b[t]);
        }
        values.put(Vs, n, p.silu, nullptr);
        __syncthreads();
        if (e0 + EB < p.E) {
            ask(e0 + EB);
            values.ask(vp + e0 + EB, p.ldv, n);
        }
        Sums<N8> o;
        o.clear();
#pragma unroll 2
        for (int d = 0; d < D; d += 16) {
            uint32_t a[NT][4];
#pragma unroll
            for (int t = 0; t < NT; ++t) ldsm4(a[t], Qs + (t * C + r0 + (lane & 15)) * LDD + d + (lane >> 4) * 8);
#pragma unroll
            for (int n8 = 0; n8 < N8; n8 += 2) {
                uint32_t b[3][4];
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    ldsm4t(b[t], Ks + (t * D + d + (lane & 7) + ((lane >> 3) & 1) * 8) * LDE + 8 * N8 * group + 8 * n8 + (lane >> 4) * 8);
                mma_terms(o, n8, a, b);
            }
        }
        const float g[2] = {start[r0 + lane / 4], start[r0 + lane / 4 + 8]};
#pragma unroll
        for (int n8 = 0; n8 < N8; ++n8)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                o.main[n8][u] *= g[u / 2];
                o.rest[n8][u] *= g[u / 2];
            }
        for (int j = 0; j <= r0; j += 16) {      // keys behind the rows weigh nothing
            uint32_t a[3][4];
#pragma unroll
            for (int t = 0; t < 3; ++t) ldsm4(a[t], Ps + (t * C + r0 + (lane & 15)) * LDP + j + (lane >> 4) * 8);
#pragma unroll
            for (int n8 = 0; n8 < N8; n8 += 2) {
                uint32_t b[NT][4];
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    ldsm4t(b[t], Vs + (t * C + j + (lane & 7) + ((lane >> 3) & 1) * 8) * LDE + 8 * N8 * group + 8 * n8 + (lane >> 4) * 8);
                mma_terms(o, n8, a, b);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = r0 + lane / 4 + 8 * u;
            if (i >= n) continue;
            float inv = 1.f;
            if (FORM == CM_MAX) {
                float keys_sum = sums[0][i];
#pragma unroll
                for (int k = 1; k < GROUPS; ++k) keys_sum += sums[k][i];
                const float dot = fmaf(start[i], n_dot[i], keys_sum);
                inv = 1.0f / (fmaxf(fabsf(dot), expf(-w.top[i])) + p.den_eps);
            }
            float* to = p.out + (size_t)(t0 + i) * ((size_t)p.H * p.E) + (size_t)h * p.E + e0 + 8 * N8 * group + 2 * (lane & 3);
#pragma unroll
            for (int n8 = 0; n8 < N8; ++n8) *reinterpret_cast<float2*>(to + 8 * n8) = make_float2(o.at(n8, 2 * u) * inv, o.at(n8, 2 * u + 1) * inv);
        }
    }
}

// Whether the kernels above take these sizes and addresses: key widths of 64 and 128, value widths in whole runs of 64 columns, rows of 16-byte vectors.
inline bool usable(const Params& p, int elem) {
    const int v = 16 / elem;
    return sizes_usable(p.D, p.E) && p.ldq % v == 0 && p.ldk % v == 0 && p.ldv % v == 0 && host_aligned16(p.q) && host_aligned16(p.k) &&
           host_aligned16(p.v) && host_aligned16(p.out) && host_aligned16(p.scratch);
}

// Whether a step's chunks and heads, with half a chunk more for every sequence that may be long, are no more than the SMs.
inline bool lone_blocks(const Params& p, int n_tokens) {
    return (2LL * n_tokens + (long long)p.longs * C) * p.H <= 2LL * C * device_sm_count();
}
template <typename T, int FORM, int D>
static int launch_width(const Params& p, int n_tokens, cudaStream_t s) {
    constexpr int NT = input_terms<T, FORM>();
    const size_t local = (size_t)(NT * C * (D + 8) + 3 * C * LDE) * sizeof(bf16), out = OutLayout<T, FORM, D>::bytes();
    auto k1 = chunk_memory_local_kernel<T, FORM, D>;
    constexpr int MOST = 16 / out_warps<T, FORM>();
    auto k3 = chunk_memory_out_kernel<T, FORM, D, MOST>;
    auto k3_lone = chunk_memory_out_kernel<T, FORM, D, 1>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)local);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k3_lone, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out);
        if (e != cudaSuccess) LLMK_FAIL("chunk_memory: cannot raise shared memory: %s", cudaGetErrorString(e));
        configured = true;
    }
    const dim3 grid(p.chunks, p.H);
    const long long items = (long long)p.longs * p.H * ceil_div(p.entries, THREADS);
    const dim3 scan((unsigned)std::min<long long>(items, 8 * device_sm_count()));
    LLMK_CHECK_LAUNCH_RC("chunk_memory_local", llmk_launch(k1, grid, dim3(THREADS), local, s, true, p));
    LLMK_CHECK_LAUNCH_RC("chunk_memory_scan", llmk_launch(chunk_memory_scan_kernel<FORM>, scan, dim3(THREADS), 0, s, true, p));
    LLMK_CHECK_LAUNCH_RC("chunk_memory_out", llmk_launch(lone_blocks(p, n_tokens) ? k3_lone : k3, grid, dim3(32 * out_warps<T, FORM>()), out, s, true, p));
    return LLMK_OK;
}
template <typename T, int FORM>
static int launch(const Params& p, int n_tokens, cudaStream_t s) {
    return p.D == 64 ? launch_width<T, FORM, 64>(p, n_tokens, s) : launch_width<T, FORM, 128>(p, n_tokens, s);
}

}  // namespace chunk_memory
