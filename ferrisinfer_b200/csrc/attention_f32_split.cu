// Attention of prompts on the 32-bit path, heads of 64: products on tensor cores with operands and sums of 32 bits.
//
// Every operand (queries, keys, softmax weights, values), times 2^40, is the sum of three bf16 numbers, v = v1 + v2 + v3 (each the rest
// rounded to nearest, the third exact: also for the smallest subnormal numbers), and a product the six of their products that reach into
// 32 bits; what is left out is at most 2^-24 of it and some 2^-27 on average.
// The tensor core's additions cut off, so the four steps of large products (v1 v1) of a tile have an accumulator of their own, the
// twenty of small ones another, and a tile's weighted values join the output by rounded fp32 additions.  Softmax in fp32.
// Error against 64 bits (2-norm, relative, 1e-7; here / the FMA kernel): 777 tokens 1.4 / 3.0, 2,048 1.6 / 4.0, 512 behind 4,096 keys 2.8 / 12.
//
// A block takes 64 query rows (the g query heads of one kv head for floor(64 / g) consecutive tokens of a request), a warp 16 of
// them, and walks the keys in tiles of 64: each warp brings 16 keys and values of the next tile in by cp.async while this one is
// multiplied, splits them once for all warps and stores the parts in rows of 144 bytes, from which ldmatrix reads without conflicts.
// Queries stay split in registers, weights are split where the scores lie.  Bound by the chain of a block's tiles at two blocks of four
// warps an SM: 2,048 tokens keep the tensor pipe busy 41 % of the time; 777 tokens, whose 174 blocks leave most SMs one, 14 %, and last as
// long as the block that walks 13 tiles (4 x 384 products of 16 x 8 x 16 each, which the pipe alone would take in some 52 us).  Before, FMAs
// bound by what shared memory returns to the lanes (attention_simt.cu, which takes every other form).  14 heads over 2 (us, before /
// here): 777 tokens 123 / 83, 2,048 339 / 213, 512 behind 4,096 keys 521 / 367, 31 single tokens beside 481 of a prompt 456 / 149 (a block a
// request; with a block's requests one after the other much longer), 4 prompts of 96 21 / 20.
//
// A row whose output is not finite (an infinity times a part of zero, an operand from 2^88 on, sums from 2^48 on), or that has a score of
// minus infinity, is formed again key by key with FMAs.
#include <math.h>

#include "attention_f32_split.cuh"
#include "attention_general.cuh"
#include "common.cuh"
#include "sm100.cuh"

namespace {

constexpr int AF_D = 64, AF_KEYS = 64, AF_ROWS = 64, AF_THREADS = 128;
constexpr int AF_PITCH = (AF_D + 8) * 2;        // bytes of a row of parts
constexpr int AF_PART = AF_KEYS * AF_PITCH;
constexpr int AF_RAW = AF_KEYS * AF_D * 4;      // bytes of a tile's keys as they come
constexpr int AF_SMEM = 6 * AF_PART + 2 * AF_RAW;
constexpr float AF_UP = 0x1p40f, AF_DOWN = 0x1p-80f;  // operands are split times 2^40, their products come back times 2^-80

struct SplitAttArgs {
    const float* q;
    float* out;
    const float* k_cache;
    const float* v_cache;
    const int* block_tables;
    const int* token_seq;
    const int* positions;
    int ldq, ldo, max_blocks, tokens, nh, nkv, page_size, window;
    float scale;
};

// Two values, times AF_UP, as three packed pairs of bf16.
__device__ __forceinline__ void split2(float lo, float hi, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    lo *= AF_UP, hi *= AF_UP;
    p1 = pack_bf16(lo, hi);
    lo -= __uint_as_float(p1 << 16), hi -= __uint_as_float(p1 & 0xffff0000u);
    p2 = pack_bf16(lo, hi);
    lo -= __uint_as_float(p2 << 16), hi -= __uint_as_float(p2 & 0xffff0000u);
    p3 = pack_bf16(lo, hi);
}

// B operands of four tiles of eight columns from two places `step` bytes apart; and their products with one A operand.
template <bool TRANS>
__device__ __forceinline__ void load_parts(uint32_t (&b)[2][4], uint32_t at, int step) {
    if (TRANS) {
        ldmatrix_x4_trans(b[0], at);
        ldmatrix_x4_trans(b[1], at + step);
    } else {
        ldmatrix_x4(b[0], at);
        ldmatrix_x4(b[1], at + step);
    }
}
template <int N>
__device__ __forceinline__ void products(float (&c)[N][4], int first, const uint32_t (&a)[4], const uint32_t (&b)[2][4]) {
#pragma unroll
    for (int t = 0; t < 4; ++t) mma_bf16_16816(c[first + t], a, b[t >> 1][2 * (t & 1)], b[t >> 1][2 * (t & 1) + 1]);
}

__device__ __forceinline__ const float* cache_row(const SplitAttArgs& p, const float* cache, int seq, int hk, int j) {
    const int page = p.block_tables[(size_t)seq * p.max_blocks + j / p.page_size];
    return cache + (((size_t)page * p.nkv + hk) * p.page_size + j % p.page_size) * AF_D;
}

// One row key by key, by a warp: two columns a lane.
__device__ __noinline__ void row_by_keys(const SplitAttArgs& p, int t, int head, int hk) {
    const int lane = threadIdx.x & 31, seq = p.token_seq[t], P = p.positions[t];
    const float* q = p.q + (size_t)t * p.ldq + (size_t)head * AF_D;
    const float q0 = q[lane], q1 = q[lane + 32];
    float* o = p.out + (size_t)t * p.ldo + (size_t)head * AF_D;
    if (__any_sync(0xffffffffu, q0 != q0 || q1 != q1)) {  // whatever the keys are
        o[lane] = o[lane + 32] = __int_as_float(0x7fffffff);
        return;
    }
    float m = -INFINITY, l = 0.0f, a0 = 0.0f, a1 = 0.0f;
    for (int j = first_key(P, p.window); j <= P; ++j) {
        const float* k = cache_row(p, p.k_cache, seq, hk, j);
        const float* v = cache_row(p, p.v_cache, seq, hk, j);
        const float s = warp_sum(fmaf(q0, k[lane], q1 * k[lane + 32])) * p.scale;
        const float m_new = fmaxf(m, s);
        const float alpha = (m_new == -INFINITY || m == m_new) ? 1.0f : expf(m - m_new);
        const float w = s == -INFINITY ? 0.0f : expf(s - m_new);
        l = l * alpha + w;
        a0 = fmaf(w, v[lane], a0 * alpha);
        a1 = fmaf(w, v[lane + 32], a1 * alpha);
        m = m_new;
    }
    o[lane] = a0 / l;
    o[lane + 32] = a1 / l;
}

__global__ void __launch_bounds__(AF_THREADS, 2) prefill_attention_f32_kernel(const SplitAttArgs p) {
    extern __shared__ __align__(128) uint8_t af_smem[];
    uint8_t* kparts = af_smem;                  // [part][key][64], rows of AF_PITCH
    uint8_t* vparts = kparts + 3 * AF_PART;
    uint8_t* raw = vparts + 3 * AF_PART;        // [keys, values][key][64] fp32
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = p.nh / p.nkv, qt = AF_ROWS / g, hk = blockIdx.y;
    const int tile_first = (gridDim.x - 1 - blockIdx.x) * qt;  // the last tokens, which see most keys, first
    const int tile_end = min(tile_first + qt, p.tokens);
    // of the requests that the tile's tokens belong to, block z takes the z-th: single tokens of many requests stand side by side
    int t_first = tile_first, t_end = tile_first;
    for (int z = 0; z <= (int)blockIdx.z; ++z) {
        t_first = t_end;
        if (t_first == tile_end) return;
        while (t_end < tile_end && p.token_seq[t_end] == p.token_seq[t_first]) ++t_end;
    }
    const int seq = p.token_seq[t_first];

    // this lane's rows (of the accumulators): two tokens' heads, their queries in parts as A operands
    int rt[2], rpos[2], rlo[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int r = warp * 16 + (lane >> 2) + 8 * a;
        rt[a] = r < qt * g ? tile_first + r / g : p.tokens;
        if (rt[a] < t_first) rt[a] = p.tokens;
        const bool there = rt[a] < t_end;
        rpos[a] = there ? p.positions[rt[a]] : -1;
        rlo[a] = there ? first_key(rpos[a], p.window) : 0;
    }
    uint32_t qp[3][4][4];  // [part][16 columns][register]
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int r = warp * 16 + (lane >> 2) + 8 * a;
        const float* row = p.q + (size_t)(rt[a] < t_end ? rt[a] : t_first) * p.ldq + (size_t)(hk * g + (r < qt * g ? r % g : 0)) * AF_D;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float2 v = *reinterpret_cast<const float2*>(row + 16 * k + 8 * half + 2 * (lane & 3));
                if (rt[a] >= t_end) v = make_float2(0.0f, 0.0f);
                split2(v.x, v.y, qp[0][k][2 * half + a], qp[1][k][2 * half + a], qp[2][k][2 * half + a]);
            }
    }

    // of the first token: no later one of the request sees an earlier key
    const int kmin = first_key(p.positions[t_first], p.window), kmax = p.positions[t_end - 1];
    const uint32_t raw_at = smem_u32(raw);
    auto request = [&](int j0) {  // 16 keys a warp, half a row of 16-byte pieces a lane
        if (j0 <= kmax) {
            const int j = j0 + warp * 16 + (lane & 15);
            long long row = -1;
            if (j >= kmin && j <= kmax) {
                const int page = p.block_tables[(size_t)seq * p.max_blocks + j / p.page_size];
                row = ((long long)page * p.nkv + hk) * p.page_size + j % p.page_size;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int key = 2 * i + (lane >> 4);
                const long long r = __shfl_sync(0xffffffffu, row, key);
                const size_t at = (size_t)(r < 0 ? 0 : r) * AF_D + 4 * (lane & 15);
                const uint32_t to = raw_at + ((warp * 16 + key) * AF_D + 4 * (lane & 15)) * 4;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(p.k_cache + at), "r"(r < 0 ? 0 : 16) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + AF_RAW), "l"(p.v_cache + at), "r"(r < 0 ? 0 : 16)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float o[8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
    bool over[2] = {false, false};  // whether a score beyond the range came out as minus infinity (any other makes the row's sums not finite)
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.0f;
    // ldmatrix: lanes 0-7 the rows of the first matrix, 8-15 of the second, ..
    const uint32_t k_frag = smem_u32(kparts) + ((lane & 7) + ((lane >> 4) << 3)) * AF_PITCH + ((lane >> 3) & 1) * 16;
    const uint32_t v_frag = smem_u32(vparts) + ((lane & 7) + ((lane >> 3) & 1) * 8) * AF_PITCH + (lane >> 4) * 16;

    request(kmin & ~(AF_KEYS - 1));
    for (int j0 = kmin & ~(AF_KEYS - 1); j0 <= kmax; j0 += AF_KEYS) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the tile before has been used (and every lane's copies are seen by its warp)
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {  // this warp's 16 keys, then their values
            const int key = warp * 16 + 2 * (i & 7) + (lane >> 4), c = lane & 15;
            const float4 v = *reinterpret_cast<const float4*>(raw + (i >> 3) * AF_RAW + (key * AF_D + 4 * c) * 4);
            uint2 p1, p2, p3;
            split2(v.x, v.y, p1.x, p2.x, p3.x);
            split2(v.z, v.w, p1.y, p2.y, p3.y);
            uint8_t* to = (i < 8 ? kparts : vparts) + key * AF_PITCH + 8 * c;
            *reinterpret_cast<uint2*>(to) = p1;
            *reinterpret_cast<uint2*>(to + AF_PART) = p2;
            *reinterpret_cast<uint2*>(to + 2 * AF_PART) = p3;
        }
        __syncwarp();
        request(j0 + AF_KEYS);
        __syncthreads();

        // scores of 16 rows x 64 keys; the products of a sum lie four others apart
        float s[8][4], low[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = low[n][e] = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int n = 0; n < 4; n += 2) {  // 32 keys
                uint32_t b1[2][4], b2[2][4], b3[2][4];
                const uint32_t at = k_frag + n * 16 * AF_PITCH + k * 32;
                load_parts<false>(b1, at, 16 * AF_PITCH);
                load_parts<false>(b2, at + AF_PART, 16 * AF_PITCH);
                load_parts<false>(b3, at + 2 * AF_PART, 16 * AF_PITCH);
                products(low, 2 * n, qp[1][k], b2);
                products(s, 2 * n, qp[0][k], b1);
                products(low, 2 * n, qp[0][k], b3);
                products(low, 2 * n, qp[2][k], b1);
                products(low, 2 * n, qp[0][k], b2);
                products(low, 2 * n, qp[1][k], b1);
            }
        float alpha[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int lo = rlo[a], hi = rpos[a];
            float best = -INFINITY;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = j0 + 8 * n + 2 * (lane & 3) + e;
                    float& v = s[n][2 * a + e];
                    const bool seen = j >= lo && j <= hi;
                    v = seen ? (v + low[n][2 * a + e]) * AF_DOWN * p.scale : -INFINITY;
                    over[a] |= seen && v == -INFINITY;
                    best = fmaxf(best, v);
                }
            best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 1));
            best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 2));
            const float m_new = fmaxf(m[a], best);
            alpha[a] = (m_new == -INFINITY || m[a] == m_new) ? 1.0f : expf(m[a] - m_new);  // exp(-inf) = 0 at a row's first keys
            float sum = 0.0f;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float& v = s[n][2 * a + e];
                    v = v == -INFINITY ? 0.0f : expf(v - m_new);
                    sum += v;
                }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[a] = l[a] * alpha[a] + sum;
            m[a] = m_new;
        }
        // the tile's weighted values, 32 columns at a time
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float big[4][4], small[4][4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) big[n][e] = small[n][e] = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // 16 keys
                uint32_t w1[4], w2[4], w3[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) split2(s[2 * k + (i >> 1)][2 * (i & 1)], s[2 * k + (i >> 1)][2 * (i & 1) + 1], w1[i], w2[i], w3[i]);
                uint32_t b1[2][4], b2[2][4], b3[2][4];
                const uint32_t at = v_frag + k * 16 * AF_PITCH + half * 64;
                load_parts<true>(b1, at, 32);
                load_parts<true>(b2, at + AF_PART, 32);
                load_parts<true>(b3, at + 2 * AF_PART, 32);
                products(small, 0, w2, b2);
                products(big, 0, w1, b1);
                products(small, 0, w1, b3);
                products(small, 0, w3, b1);
                products(small, 0, w1, b2);
                products(small, 0, w2, b1);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    o[4 * half + n][e] = fmaf(o[4 * half + n][e], alpha[e >> 1], big[n][e] + small[n][e]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int r = warp * 16 + (lane >> 2) + 8 * a;
        const bool there = rt[a] < t_end;
        const int head = hk * g + (there ? r % g : 0);
        bool odd = there && over[a];
        if (there) {
            float* row = p.out + (size_t)rt[a] * p.ldo + (size_t)head * AF_D;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float v = o[n][2 * a + e] / l[a] * AF_DOWN;
                    odd |= !(fabsf(v) <= 3.402823466e38f);
                    row[8 * n + 2 * (lane & 3) + e] = v;
                }
        }
        unsigned left = __ballot_sync(0xffffffffu, odd);
        __syncwarp();
        while (left) {  // rows that are not finite, one after the other
            const int src = __ffs(left) - 1;
            row_by_keys(p, __shfl_sync(0xffffffffu, rt[a], src), __shfl_sync(0xffffffffu, head, src), hk);
            left &= ~(0xfu << (src & ~3));  // (the four lanes of the row)
        }
    }
}

}  // namespace

bool ferris_attention_f32_split_takes(int nh, int nkv, int d, int dv) {
    return d == AF_D && dv == AF_D && nkv > 0 && nh % nkv == 0 && nh / nkv <= AF_ROWS;
}

int ferris_attention_f32_split(const float* q, int ldq, float* out, int ldo, const float* k_cache, const float* v_cache,
                               const int* block_tables, int max_blocks, const int* token_seq, const int* positions, int tokens, int nh,
                               int nkv, int page_size, int window, float scale, int seqs, cudaStream_t s) {
    const SplitAttArgs p = {q, out, k_cache, v_cache, block_tables, token_seq, positions, ldq, ldo, max_blocks, tokens, nh, nkv, page_size,
                            window, scale};
    if (int rc = ferris_allow_dynamic_smem((const void*)prefill_attention_f32_kernel, AF_SMEM)) return rc;
    const int qt = AF_ROWS / (nh / nkv);
    ferris_launch(prefill_attention_f32_kernel, dim3((tokens + qt - 1) / qt, nkv, seqs < qt ? seqs : qt), dim3(AF_THREADS), AF_SMEM, s, p);
    FERRIS_LAUNCH_CHECK();
}
