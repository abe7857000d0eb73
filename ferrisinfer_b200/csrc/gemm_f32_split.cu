// The 32-bit path's products of many tokens on the tensor cores: out[t, n] (+)= sum_k x[t, k] * w[n, k] (+ bias[n]) with operands and
// sums of 32 bits.
//
// Every operand, times 2^40, is written as the sum of three bf16 numbers, v = v1 + v2 + v3 (each the rest rounded to nearest; the third
// is exact), so that every fp32 number below 2^88 keeps all its bits, the smallest subnormal ones too (bf16 ends at 2^-133: without the
// factor a number of 2^-120 would keep 14 bits).  Sums come back times 2^-80; an operand from 2^88 on or a sum from 2^48 on is no longer
// finite there (see below).  A product is the six of their nine products that reach into 32 bits: x1 w1, x1 w2, x2 w1, x2 w2, x1 w3,
// x3 w1.  What is left out, x2 w3 + x3 w2 + x3 w3, is at most 2^-24 of |x w| and some 2^-27 of it on average.  The products
// themselves are exact.  The tensor core's own additions cut off instead of rounding, so a sum stays there for 32 k's only, the
// small products first (the cuts then fall on sums a 256th as large) and the two steps of large ones last; after that it is
// added to sums in registers, rounded to nearest, and these every 1,280 k's to a sum of their own.  Error against 64 bits
// (2-norm, relative; this kernel / the FMA kernels of gemm_f32.cu): K = 64 0.7 / 1.1, 896 0.9 to 1.15 / 1.55, 4,864
// 1.2 to 1.3 / 1.6, 9,220 1.3 / 1.65, each 1e-7.
//
// A cluster of two CTAs (cta_group::2) takes 256 weight rows x NT tokens.  Nothing reads the fp32 operands from shared memory: sixteen
// warps load runs of 8 k's straight into registers (a warp: 4 rows x 64 k's, whole 128-byte lines), split them, take the next slice's into
// the same registers and store three 16-byte chunks into bf16 tiles in the 128-byte swizzle that the MMA reads; one lane issues the
// MMAs; eight warps add the sums up.  Three slices of 64 k's stand in shared memory, because a slot's way around (split, its arrival at the
// leader, MMAs, their commit) is longer than any of its parts: with two slots it took 2.45 us a slice at 128 tokens, of which the MMAs
// are 0.8 and everything else without them 1.65; with three (and the MMAs issued by a warp of their own) 1.8.  Before that: one set of
// warps that split and drained 4.2, two 3.1, two accumulators in turn 2.45.
// Measured (us, tokens: 96 / 200 / 777 / 2,048; in brackets the FMA kernels): 9,728 x 896 29 / 51 / 105 / 229 (84 / 131 / 351 / 817; 155
// TFLOP/s), 896 x 4,864 32 / 37 / 80 / 199 (61 / 79 / 218 / 564); 200 / 777 / 2,048: 1,152 x 896 24 / 26 / 50 (29 / 61 / 109), 896 x 896 24 / 26 / 32 (28 / 54 /
// 108).
//
// K SPLITS: where rows are long and few a cluster of up to four pairs takes one tile, each a run of slices; the sums meet through
// shared memory and are added in the runs' order.  SwiGLU: a CTA's rows 0..63 are gate rows, 64..127 their up rows.
//
// Infinities and overflow: a part of an infinity times a part that is zero is not a number, so a result that is not finite is
// formed again with FMAs in the order of gemm_f32.cuh.
#include <atomic>

#include "common.cuh"
#include "gemm_f32.cuh"
#include "sm100.cuh"

namespace {

constexpr int SP_DRAINERS = 8;    // warps that add the accumulators up and write
constexpr int SP_SPLITTERS = 16;  // warps that load and split the operands
constexpr int SP_ISSUERS = 4;     // and a group of four of which one lane (of the leader) issues the MMAs
constexpr int SP_THREADS = (SP_DRAINERS + SP_SPLITTERS + SP_ISSUERS) * 32;
// Registers a thread: 72 at the launch, then so many for either kind of warp, which together are no more.
constexpr int SP_LAUNCH_REGS = 72, SP_DRAIN_REGS = 128, SP_SPLIT_REGS = 56, SP_ISSUE_REGS = 24;
static_assert(SP_DRAINERS * SP_DRAIN_REGS + SP_SPLITTERS * SP_SPLIT_REGS + SP_ISSUERS * SP_ISSUE_REGS <= SP_THREADS / 32 * SP_LAUNCH_REGS &&
                  SP_THREADS * SP_LAUNCH_REGS <= 65536 && SP_DRAINERS % 4 == 0 && SP_SPLITTERS % 4 == 0 && SP_ISSUERS % 4 == 0,
              "the shares come out of the launch's registers, by groups of four warps");
constexpr int SP_ROWS = SP_SPLITTERS * 4;  // rows that the splitting warps take at a time, eight threads a row
constexpr int SP_SLOTS = 3;                // slices in shared memory
constexpr int SP_M = 128;                  // weight rows of a CTA, 256 of a pair
constexpr int SP_K = 64;                   // k's of a slice: two runs of 32
constexpr int SP_LEVEL = 20;               // slices whose runs are added up before they join the outer sum
constexpr int SP_MAX_SPLITS = 4;
constexpr int SP_MAX_LD = 1 << 24;         // elements between rows (offsets of a thread's rows are 32-bit numbers)
constexpr int SP_EXCHANGE = 4 * 16 * 32 * 4;  // SwiGLU: sums of up rows on their way, of sixteen tokens for each pair of warps
constexpr int SP_A_PART = SP_M * 128;      // bytes of one part of a slice of the weights
constexpr float SP_UP = 0x1p40f, SP_DOWN = 0x1p-80f;  // operands are split times 2^40, sums come back times 2^-80

struct SplitParams {
    const float* x;
    const float* w;
    const float* bias;
    float* out;
    int M, N, K, ldx, ldw, ldo, accumulate;
    int up_offset;  // > 0: SwiGLU of weight rows n and up_offset + n; N outputs
    int m_tiles, n_tiles, slices, slices_per, splits;
    int early_weights;
    int* status;
};

// a + b and a - b of two pairs, an instruction each.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    const float2 minus = make_float2(-1.0f, -1.0f);  // (a - b in one rounding: -b is exact)
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(r)
        : "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<const unsigned long long&>(minus)),
          "l"(reinterpret_cast<unsigned long long&>(a)));
    return reinterpret_cast<float2&>(r);
}

// Eight fp32 values times SP_UP as three runs of eight bf16: the value rounded, the rest rounded, what then is left.
__device__ __forceinline__ float2 unpack2(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
__device__ __forceinline__ void split8(const float4 a, const float4 b, uint4& p1, uint4& p2, uint4& p3) {
    const float2 up = make_float2(SP_UP, SP_UP);
    const float2 v[4] = {mul2(make_float2(a.x, a.y), up), mul2(make_float2(a.z, a.w), up), mul2(make_float2(b.x, b.y), up),
                         mul2(make_float2(b.z, b.w), up)};
    uint32_t o1[4], o2[4], o3[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o1[i] = pack_bf16(v[i].x, v[i].y);
        float2 rest = sub2(v[i], unpack2(o1[i]));
        o2[i] = pack_bf16(rest.x, rest.y);
        rest = sub2(rest, unpack2(o2[i]));
        o3[i] = pack_bf16(rest.x, rest.y);
    }
    p1 = make_uint4(o1[0], o1[1], o1[2], o1[3]);
    p2 = make_uint4(o2[0], o2[1], o2[2], o2[3]);
    p3 = make_uint4(o3[0], o3[1], o3[2], o3[3]);
}

// Two tokens' outputs of one weight row in the order of the FMA kernels.
__device__ __forceinline__ float2 dots_in_order(const float* x0, const float* x1, const float* w, int K) {
    const int runs = (K + F32_CHUNK - 1) / F32_CHUNK, per = f32_runs_per_part(runs);
    float2 total = make_float2(0.0f, 0.0f), part = total;
    for (int c = 0; c < runs; ++c) {
        float2 even = make_float2(0.0f, 0.0f), odd = even;  // (of the two tokens)
        const int k1 = min(K, (c + 1) * F32_CHUNK);
#pragma unroll 4
        for (int k = c * F32_CHUNK; k < k1; k += 4) {
            const float4 v = *reinterpret_cast<const float4*>(w + k);
            const float4 a = *reinterpret_cast<const float4*>(x0 + k), b = *reinterpret_cast<const float4*>(x1 + k);
            even.x = fmaf(a.x, v.x, even.x), odd.x = fmaf(a.y, v.y, odd.x), even.y = fmaf(b.x, v.x, even.y), odd.y = fmaf(b.y, v.y, odd.y);
            even.x = fmaf(a.z, v.z, even.x), odd.x = fmaf(a.w, v.w, odd.x), even.y = fmaf(b.z, v.z, even.y), odd.y = fmaf(b.w, v.w, odd.y);
        }
        part.x += even.x + odd.x, part.y += even.y + odd.y;
        if ((c + 1) % per == 0 || c + 1 == runs) {
            total.x += part.x, total.y += part.y;
            part = make_float2(0.0f, 0.0f);
        }
    }
    return total;
}

// Outputs whose sums are not finite: those of weight row n of the tokens t0 + i, i the bits of `odd`, two at a time; by a warp (a lane
// without any: odd = 0).  A token that has a NaN makes nothing else of it, and is not multiplied again (777 tokens of nothing but NaN,
// 9,728 x 896: 35,000 us number by number, 490 so, 122 of finite numbers; one infinity 184, 141).
template <bool SWIGLU>
__device__ __forceinline__ void write_in_order(const SplitParams& p, int t0, uint32_t odd, int n) {
    for (uint32_t any = __reduce_or_sync(0xffffffffu, odd); any; any &= any - 1) {
        const int t = __ffs(any) - 1;
        bool nan = false;
        for (int k = 4 * (threadIdx.x & 31); k < p.K; k += 128) {
            const float4 v = *reinterpret_cast<const float4*>(p.x + (size_t)(t0 + t) * p.ldx + k);
            nan |= v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
        }
        if (__any_sync(0xffffffffu, nan) && (odd >> t & 1)) {
            p.out[(size_t)(t0 + t) * p.ldo + n] = __int_as_float(0x7fffffff);
            odd &= ~(1u << t);
        }
    }
    while (odd) {
        const int first = t0 + __ffs(odd) - 1;
        odd &= odd - 1;
        const int second = odd ? t0 + __ffs(odd) - 1 : first;
        if (odd) odd &= odd - 1;
        const float *x0 = p.x + (size_t)first * p.ldx, *x1 = p.x + (size_t)second * p.ldx;
        float2 v = dots_in_order(x0, x1, p.w + (size_t)n * p.ldw, p.K);
        float *o0 = p.out + (size_t)first * p.ldo + n, *o1 = p.out + (size_t)second * p.ldo + n;
        if (SWIGLU) {
            const float2 u = dots_in_order(x0, x1, p.w + (size_t)(n + p.up_offset) * p.ldw, p.K);
            *o0 = u.x * (v.x * (1.0f / (1.0f + expf(-v.x))));
            *o1 = u.y * (v.y * (1.0f / (1.0f + expf(-v.y))));
        } else {
            if (p.bias) v.x += p.bias[n], v.y += p.bias[n];
            if (p.accumulate) v.x += *o0, v.y += *o1;
            *o0 = v.x;
            *o1 = v.y;
        }
    }
}

__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

__device__ __forceinline__ void tmem_load_32x8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_store_32x8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// All of an SM's tensor memory, for both CTAs of a pair.
__device__ __forceinline__ void take_tensor_memory(uint32_t* dst) { tmem_alloc_pair(dst, 512); }

template <int NT>  // tokens of a tile
struct SplitShape {
    static constexpr int CW = NT / 2;  // columns of a draining warp
    static constexpr int XR = NT / 2;  // token rows that a CTA holds
    static constexpr int B_PART = XR * 128;
    static constexpr int SLOT = 3 * (SP_A_PART + B_PART);
};

template <int NT, bool SWIGLU>
__global__ void __launch_bounds__(SP_THREADS, 1) gemm_f32_split_kernel(const SplitParams p) {
    using S = SplitShape<NT>;
    constexpr int CW = S::CW;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[SP_SLOTS], slot_free[SP_SLOTS], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta = cluster_ctarank(), rank = cta & 1, leader = cta & ~1u;
    const int splits = SWIGLU ? 1 : p.splits, split = SWIGLU ? 0 : (int)(cta >> 1);
    const int first = (int)blockIdx.x / (2 * splits), stride = (int)gridDim.x / (2 * splits);  // clusters
    const int s0 = split * p.slices_per, per_tile = min(p.slices, s0 + p.slices_per) - s0;
    const int tiles = p.m_tiles * p.n_tiles;
    const int total = first < tiles ? (tiles - first + stride - 1) / stride * per_tile : 0;  // slices of this CTA
    const uint16_t both = (uint16_t)(3u << leader);
    if (tid == 0) {
        for (int i = 0; i < SP_SLOTS; ++i) {
            mbar_init(&full[i], 2 * SP_SPLITTERS);  // the splitting warps of both CTAs (used in the leader only)
            mbar_init(&slot_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * SP_DRAINERS);  // (the leader's only)
        }
        mbar_fence_init();
    }
    if (warp == 0) take_tensor_memory(&tmem_base);  // ahead of the dependents: a launch that had it could wait for this one
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_base;
    pdl_launch_dependents();

    int ok = 1;  // 0: a wait ran out; nothing is waited for any more, every barrier is still met
    if (warp >= SP_DRAINERS && warp < SP_DRAINERS + SP_SPLITTERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SP_SPLIT_REGS));
        // -------------------------------------------------------------------------------- operands: fp32 -> three bf16 tiles
        constexpr int WG = SP_M / SP_ROWS, XG = (S::XR + SP_ROWS - 1) / SP_ROWS;  // rows of a thread, SP_ROWS apart
        const int ct = tid - SP_DRAINERS * 32, lr = ct >> 3, ch = ct & 7;         // its first row, its 8 k's of a slice
        const uint32_t full_at = map_to_cta(smem_u32(&full[0]), leader);
        float4 wa[WG][2], xb[XG][2];
        int l_tile = first, l_slice = 0, l_it = 0;  // the slice that is loaded next
        const float* w_row = nullptr;               // its tile's first row of this thread (the product's first where there is none)
        const float* x_row = nullptr;
        int w_left = 0, x_left = 0;                 // the operand's rows from there on
        const int w_step = SP_ROWS * p.ldw, x_step = SP_ROWS * p.ldx;
        const size_t w_up = SWIGLU ? (size_t)p.up_offset * p.ldw - (size_t)64 * p.ldw : 0;  // from a row 64 further to the up row
        auto rows_of_tile = [&]() {
            const int nt = l_tile / p.m_tiles, n = nt * (SWIGLU ? SP_M : 2 * SP_M) + (int)rank * (SWIGLU ? 64 : SP_M) + lr;
            const int t = (l_tile - nt * p.m_tiles) * NT + (int)rank * S::XR + lr;
            w_left = p.N - n, x_left = p.M - t;
            w_row = p.w + (w_left > 0 ? (size_t)n * p.ldw : 0) + 8 * ch;
            x_row = p.x + (x_left > 0 ? (size_t)t * p.ldx : 0) + 8 * ch;
        };
        auto load8 = [&](float4 (&v)[2], const float* at, bool lo, bool hi) {
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            v[0] = lo ? *reinterpret_cast<const float4*>(at) : none;
            v[1] = hi ? *reinterpret_cast<const float4*>(at + 4) : none;
        };
        bool w_lo = false, w_hi = false, w_far = false;  // which of this thread's k's the slice has, and whether the one two further on
        int w_k = 0;
        // Turns to the slice that is loaded next; then its rows may be loaded, in any order (none beyond the last slice).
        auto turn = [&]() {
            if (l_it > 0 && ++l_slice == per_tile) {
                l_slice = 0;
                l_tile += stride;
            }
            const bool any = l_it++ < total;
            if (any && l_slice == 0) rows_of_tile();
            w_k = (s0 + l_slice) * SP_K;
            const int left = p.K - w_k - 8 * ch;  // k's from this thread's first on
            w_lo = any && left > 0, w_hi = any && left > 4, w_far = any && left > 2 * SP_K && (ch & 3) == 0;
        };
        auto load_w = [&](int j) {
            const bool there = (SWIGLU ? SP_ROWS * j % 64 : SP_ROWS * j) < w_left;
            const float* at = w_row + w_k + j * w_step + (SWIGLU && SP_ROWS * j >= 64 ? w_up : 0);
            load8(wa[j], at, there && w_lo, there && w_hi);
            if (there && w_far) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 2 * SP_K));  // from HBM into L2
        };
        auto load_x = [&](int j) {
            const bool there = SP_ROWS * j < x_left && SP_ROWS * j + lr < S::XR;
            load8(xb[j], x_row + w_k + j * x_step, there && w_lo, there && w_hi);
        };
        const uint32_t at0 = swizzle128(lr, ch);  // (rows a multiple of eight further: the same swizzle)
        turn();
        if (!p.early_weights) pdl_wait();
#pragma unroll
        for (int j = 0; j < WG; ++j) load_w(j);
        if (p.early_weights) pdl_wait();
#pragma unroll
        for (int j = 0; j < XG; ++j) load_x(j);
        int s = 0, phase = 1;  // the slot that is filled next, and the phase of its barrier that frees it
        for (int it = 0; it < total; ++it) {
            uint8_t* slot = smem + s * S::SLOT + at0;
            if (it >= SP_SLOTS && ok) ok = __all_sync(0xffffffffu, mbar_wait(&slot_free[s], phase, p.status, 0x73));
            turn();
            uint4 p1, p2, p3;
            // a run of rows is split and stored, and its registers take the next slice's at once
#pragma unroll
            for (int j = 0; j < WG; ++j) {
                split8(wa[j][0], wa[j][1], p1, p2, p3);
                load_w(j);
                uint8_t* at = slot + j * SP_ROWS * 128;
                *reinterpret_cast<uint4*>(at) = p1;
                *reinterpret_cast<uint4*>(at + SP_A_PART) = p2;
                *reinterpret_cast<uint4*>(at + 2 * SP_A_PART) = p3;
            }
#pragma unroll
            for (int j = 0; j < XG; ++j) {
                split8(xb[j][0], xb[j][1], p1, p2, p3);
                load_x(j);
                if (SP_ROWS * j + lr >= S::XR) continue;
                uint8_t* at = slot + 3 * SP_A_PART + j * SP_ROWS * 128;
                *reinterpret_cast<uint4*>(at) = p1;
                *reinterpret_cast<uint4*>(at + S::B_PART) = p2;
                *reinterpret_cast<uint4*>(at + 2 * S::B_PART) = p3;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads what every lane wrote
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(full_at + 8u * s);
            if (++s == SP_SLOTS) s = 0, phase ^= 1;
        }
        if (!SWIGLU && splits > 1) {  // (the draining warps' exchange)
            __syncwarp();
            cluster_sync();
            cluster_sync();
        }
    } else if (warp >= SP_DRAINERS) {
        // ---------------------------------------------------------------------------------------- MMAs
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SP_ISSUE_REGS));
        if (warp == SP_DRAINERS + SP_SPLITTERS && lane == 0 && rank == 0) {
            // A slice: its two runs of 32 k's into the two accumulators of its set, the smallest products first.  A product waits for the one
            // before it in the same accumulator, so the runs take turns.
            const uint32_t idesc = umma_idesc_bf16(2 * SP_M, NT);
            int s = 0, phase = 0;
            for (int it = 0; it < total; ++it) {
                const int set = it & 1;
                if (!mbar_wait(&full[s], phase, p.status, 0x70)) break;
                if (it >= 2 && !mbar_wait(&acc_empty[set], ((it >> 1) - 1) & 1, p.status, 0x71)) break;
                tcgen05_fence_after();
                constexpr int PA[6] = {1, 0, 2, 0, 1, 0}, PB[6] = {1, 2, 0, 1, 0, 0};
                const uint32_t at = smem_u32(smem + s * S::SLOT), d = tmem + set * 2 * NT;
                const uint64_t a = umma_desc_k_major_sw128(at), b = umma_desc_k_major_sw128(at + 3 * SP_A_PART);
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint64_t step = (uint64_t)(2 * (2 * h + k));
                            tcgen05_mma_bf16_pair(d + h * NT, a + (uint64_t)(PA[i] * (SP_A_PART >> 4)) + step,
                                                  b + (uint64_t)(PB[i] * (S::B_PART >> 4)) + step, idesc, (i | k) ? 1u : 0u);
                        }
                tcgen05_commit_pair(&slot_free[s], both);
                tcgen05_commit_pair(&acc_full[set], both);
                if (++s == SP_SLOTS) s = 0, phase ^= 1;
            }
        }
        if (!SWIGLU && splits > 1) {  // (the draining warps' exchange)
            __syncwarp();
            cluster_sync();
            cluster_sync();
        }
    } else {
        // ---------------------------------------------------------------------------------------- sums, outputs
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SP_DRAIN_REGS));
        const int quarter = warp & 3, wc = warp >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + wc * CW;
        const uint32_t empty_at = map_to_cta(smem_u32(&acc_empty[0]), leader);
        pdl_wait();  // (an accumulating product reads what the launch before wrote)
        float acc[CW];
#pragma unroll
        for (int c = 0; c < CW; ++c) acc[c] = 0.0f;
        int tile = first, slice = 0;
        for (int it = 0; it < total; ++it) {
            const int set = it & 1;
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[set], (it >> 1) & 1, p.status, 0x72));
            tcgen05_fence_after();
            const uint32_t from = lane_addr + set * 2 * NT;
#pragma unroll
            for (int c0 = 0; c0 < CW; c0 += 16) {
                uint32_t r[16], q[16];
                tmem_load_32x16(from + c0, r);
                tmem_load_32x16(from + NT + c0, q);
                tmem_load_wait();
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    float2 sum = add2(make_float2(acc[c0 + c], acc[c0 + c + 1]), make_float2(__uint_as_float(r[c]), __uint_as_float(r[c + 1])));
                    sum = add2(sum, make_float2(__uint_as_float(q[c]), __uint_as_float(q[c + 1])));
                    acc[c0 + c] = sum.x;
                    acc[c0 + c + 1] = sum.y;
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty_at + 8u * set);
            const bool last = slice + 1 == per_tile;
            if ((slice + 1) % SP_LEVEL == 0 || (last && slice >= SP_LEVEL)) {  // the runs so far join the outer sum
#pragma unroll
                for (int c = 0; c < CW; c += 8) {
                    uint32_t r[8];
                    if (slice >= SP_LEVEL) {
                        tmem_load_32x8(lane_addr + 4 * NT + c, r);
                        tmem_load_wait();
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float sum = slice >= SP_LEVEL ? __uint_as_float(r[i]) + acc[c + i] : acc[c + i];
                        r[i] = __float_as_uint(sum);
                        acc[c + i] = last ? sum : 0.0f;
                    }
                    if (!last) tmem_store_32x8(lane_addr + 4 * NT + c, r);
                }
                if (!last) tmem_store_wait();
            }
            ++slice;
            if (!last) continue;
            slice = 0;
            if (!SWIGLU && splits > 1) break;  // one tile to a cluster: its sums meet below
            const int t0 = (tile % p.m_tiles) * NT + wc * CW, nt = tile / p.m_tiles;
            const int n = SWIGLU ? nt * SP_M + (int)rank * 64 + (quarter & 1) * 32 + lane : nt * 2 * SP_M + (int)rank * SP_M + quarter * 32 + lane;
            // sixteen tokens at a time; those whose sums are not finite are left for the loop behind
            float* up = reinterpret_cast<float*>(smem + SP_SLOTS * S::SLOT) + (wc * 2 + (quarter & 1)) * (16 * 32) + lane;
            const int bar = 1 + wc * 2 + (quarter & 1);  // the warp of the gate rows and that of their up rows
            const float bias = !SWIGLU && p.bias && n < p.N ? p.bias[n] : 0.0f;
#pragma unroll
            for (int c0 = 0; c0 < CW; c0 += 16) {
                uint32_t odd = 0;
                if (SWIGLU) {
                    if (quarter >= 2) {
#pragma unroll
                        for (int c = 0; c < 16; ++c) up[c * 32] = acc[c0 + c];
                    }
                    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
                }
                if (n < p.N && (!SWIGLU || quarter < 2)) {
                    float* o = p.out + (size_t)(t0 + c0) * p.ldo + n;
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        if (t0 + c0 + c >= p.M) continue;
                        const float v = acc[c0 + c] * SP_DOWN;
                        float* at = o + (size_t)c * p.ldo;
                        if (SWIGLU) {
                            const float u = up[c * 32] * SP_DOWN;
                            if (is_finite(v) && is_finite(u))
                                *at = u * (v * (1.0f / (1.0f + expf(-v))));
                            else
                                odd |= 1u << c;
                        } else if (is_finite(v)) {
                            const float sum = p.bias ? v + bias : v;
                            *at = p.accumulate ? *at + sum : sum;
                        } else {
                            odd |= 1u << c;
                        }
                    }
                }
                if (SWIGLU) asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
                if (!SWIGLU || quarter < 2) write_in_order<SWIGLU>(p, t0 + c0, odd, n);
            }
#pragma unroll
            for (int c = 0; c < CW; ++c) acc[c] = 0.0f;
            tile += stride;
        }
        if (!SWIGLU && splits > 1) {
            // groups of four tokens of a warp belong to the pairs in turn; a pair sends the others theirs
            constexpr int GROUPS = CW / 4, THREADS = SP_DRAINERS * 32;
            const int each = (GROUPS + splits - 1) / splits;  // groups of an owner
            const uint32_t ring = smem_u32(smem);
            __syncwarp();
            cluster_sync();  // every MMA of the cluster is done: the slots take partial sums now
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                const int owner = g % splits;
                if (owner == split) continue;
                const int place = (split < owner ? split : split - 1) * each + g / splits;
                uint32_t v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = __float_as_uint(acc[4 * g + i]);
                st_cluster_x4(map_to_cta(ring + (place * THREADS + tid) * 16, 2 * owner + rank), v);
            }
            __syncwarp();
            cluster_sync();
            const int t0 = (first % p.m_tiles) * NT + wc * CW;
            const int n = first / p.m_tiles * 2 * SP_M + (int)rank * SP_M + quarter * 32 + lane;
            const float bias = p.bias && n < p.N ? p.bias[n] : 0.0f;
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                if (g % splits != split) continue;
                float sum[4];
                for (int from = 0; from < splits; ++from) {
                    float4 v = make_float4(acc[4 * g], acc[4 * g + 1], acc[4 * g + 2], acc[4 * g + 3]);
                    if (from != split) {
                        const int place = (from < split ? from : from - 1) * each + g / splits;
                        v = *reinterpret_cast<const float4*>(smem + (size_t)(place * THREADS + tid) * 16);
                    }
                    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[i] = from ? sum[i] + f[i] : f[i];
                }
                uint32_t odd = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int t = t0 + 4 * g + i;
                    if (n >= p.N || t >= p.M) continue;
                    float* o = p.out + (size_t)t * p.ldo + n;
                    const float dot = sum[i] * SP_DOWN, v = p.bias ? dot + bias : dot;
                    if (is_finite(dot))
                        *o = p.accumulate ? *o + v : v;
                    else
                        odd |= 1u << i;
                }
                write_in_order<false>(p, t0 + 4 * g, odd, n);
            }
        }
    }
    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();  // neither CTA frees tensor memory or leaves while the pair's MMAs or arrivals may still come
    if (warp == 0) {
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
}

// ------------------------------------------------------------------------------------------------- launching
template <int NT, bool SWIGLU>
int launch_split(const SplitParams& p, int clusters, cudaStream_t s) {
    const size_t smem = SP_SLOTS * SplitShape<NT>::SLOT + (SWIGLU ? SP_EXCHANGE : 0) + 1024;
    if (int rc = ferris_allow_dynamic_smem((const void*)gemm_f32_split_kernel<NT, SWIGLU>, smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * p.splits * clusters);
    cfg.blockDim = dim3(SP_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ferris_pdl_enabled() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<NT, SWIGLU>, p);
    if (e != cudaSuccess) {
        ferris_set_error("32-bit gemm: %s", cudaGetErrorString(e));
        return (int)e;
    }
    FERRIS_LAUNCH_CHECK();
}
template <bool SWIGLU>
int launch_split_of(int nt, const SplitParams& p, int clusters, cudaStream_t s) {
    if (nt == 32) return launch_split<32, SWIGLU>(p, clusters, s);
    if (nt == 64) return launch_split<64, SWIGLU>(p, clusters, s);
    if (nt == 96) return launch_split<96, SWIGLU>(p, clusters, s);
    return launch_split<128, SWIGLU>(p, clusters, s);
}

// Clusters of so many pairs that the current GPU holds at once, a CTA an SM (a cluster keeps to a GPC); asked for once on each GPU, and where
// two threads ask at once they write the same.
int active_clusters(int pairs) {
    constexpr int DEVICES = 16;
    static std::atomic<int> known[DEVICES][SP_MAX_SPLITS + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError(), dev = DEVICES;
    const bool keep = dev >= 0 && dev < DEVICES;
    if (keep)
        if (const int n = known[dev][pairs].load(std::memory_order_relaxed)) return n;
    constexpr int UNKNOWN[SP_MAX_SPLITS + 1] = {0, 74, 32, 20, 12};
    const size_t smem = SP_SLOTS * SplitShape<128>::SLOT + 1024;
    int n = 0;
    if (ferris_allow_dynamic_smem((const void*)gemm_f32_split_kernel<128, false>, smem) == FERRIS_OK) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * pairs);
        cfg.blockDim = dim3(SP_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2 * pairs;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_split_kernel<128, false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
    }
    if (n <= 0) n = UNKNOWN[pairs];
    if (keep) known[dev][pairs].store(n, std::memory_order_relaxed);
    return n;
}

struct SplitPlan {
    int nt, splits, clusters, m_tiles, n_tiles, slices_per;
    double us;
};
// K splits regroup an output's sum, so they are chosen without a look at the number of tokens: a row's bits do not depend on what else is in
// the step.  Long rows and few of them gain from splits where tokens are few too, and lose the less by them where tokens are many; with
// many weight rows there are tiles enough.  Against the splits that are best for each of up to ten numbers of tokens from 48 to 4,096 (times the
// time on average, at worst): 896 x 896 and 1,152 x 896 1.09 and 1.10, 1.7 (192 tokens 24 us instead of 14; FMAs 29); 896 x 4,864 1.07, 1.40;
// 1,536 x 1,536 1.10, 1.39; 1,536 x 8,960 1.17, 1.46; 2,048 x 2,048 1.13, 1.47; 3,584 x 3,584 1.08, 1.31; 3,584 x 18,944 1.10, 1.23; 9,728 x 896 none.
int split_count(int slices, int n_tiles) {
    if (n_tiles >= 20 || slices < 24) return 1;
    if (slices < 48) return 2;
    return slices >= 72 && n_tiles <= 8 ? 4 : 3;
}
// The cut of a product: its splits, and the token tile of the least time, from what a slice was measured to take (us, token tiles of 32 to
// 128), a tile's end, the launch and a cluster's exchange.
SplitPlan split_plan(int M, int rows, int K, bool swiglu, int nt_only = 0, int splits_only = 0) {
    constexpr double SLICE[4] = {1.3, 1.55, 1.7, 1.8};
    SplitPlan best = {};
    const int slices = (K + SP_K - 1) / SP_K, n_tiles = (rows + 2 * SP_M - 1) / (2 * SP_M);
    const int sp = splits_only ? splits_only : swiglu ? 1 : split_count(slices, n_tiles), per = (slices + sp - 1) / sp;
    if (sp > 1 && (per < 4 || (sp - 1) * per >= slices)) return best;
    const int at_once = active_clusters(sp);
    for (int nt = 32; nt <= 128; nt += 32) {
        if ((nt_only && nt != nt_only) || (nt == 128 && per > SP_LEVEL)) continue;  // (128: no tensor memory left for the outer sums)
        const long long m_tiles = (M + nt - 1) / nt, tiles = m_tiles * n_tiles, rounds = (tiles + at_once - 1) / at_once;
        const double us = rounds * (per * SLICE[nt / 32 - 1] + (sp > 1 ? 5.0 : 1.0)) + 3.0;
        if (best.nt && us >= best.us) continue;
        best = {nt, sp, (int)(sp > 1 || tiles < at_once ? tiles : at_once), (int)m_tiles, n_tiles, per, us};
    }
    return best;
}

int run_split(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx, int ldw, int ldo,
              int accumulate, int up_offset, int early_weights, const SplitPlan& q, cudaStream_t s) {
    const SplitParams p = {x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, up_offset, q.m_tiles, q.n_tiles, (K + SP_K - 1) / SP_K,
                           q.slices_per, q.splits, early_weights, ferris_status_ptr()};
    return up_offset > 0 ? launch_split_of<true>(q.nt, p, q.clusters, s) : launch_split_of<false>(q.nt, p, q.clusters, s);
}

}  // namespace

// More than 32 tokens and 150 million multiply-adds.  Up to there every form of the product adds in one order, and a row's bits do not depend
// on how many others the step brings, nor do they beyond (split_count): only on which side of the line the product lies.  From 33 tokens on this
// kernel would win below it too, by 5 to 14 us of 18 to 27, with other bits for the products of short steps.
bool ferris_gemm_f32_split_takes(int M, int rows, int K, int ldx, int ldw) {
    return M > 32 && (long long)M * rows * K >= 150000000LL && (long long)((M + 31) / 32) * ((rows + 255) / 256) < (1 << 28) &&
           ldx <= SP_MAX_LD && ldw <= SP_MAX_LD;
}

int ferris_gemm_f32_split(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx, int ldw,
                          int ldo, int accumulate, int up_offset, int early_weights, cudaStream_t s) {
    return run_split(x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, up_offset, early_weights,
                     split_plan(M, up_offset > 0 ? 2 * N : N, K, up_offset > 0), s);
}

// The product on the tensor cores whatever its size, cut as told (token_tile 32 to 128 in steps of 32, splits 1 to 4; 0: by the plan).  Rows aligned as
// ferris_gemm_f32_takes has it; swiglu: N outputs of 2 N weight rows, gate rows first.
FERRIS_API int ferris_gemm_f32_split_run(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx,
                                         int ldw, int ldo, int accumulate, int swiglu, int token_tile, int splits, void* stream) {
    if (M <= 0 || N <= 0) return FERRIS_OK;
    if (K <= 0 || ldx < K || ldw < K || ldo < N) FERRIS_REFUSE("gemm: K=%d, row strides %d, %d, %d", K, ldx, ldw, ldo);
    if (!ferris_gemm_f32_takes(x, w, out, K, ldx, ldw)) FERRIS_REFUSE("gemm: rows that do not begin on 16 bytes");
    if ((long long)((M + 31) / 32) * ((2LL * N + 255) / 256) >= (1 << 28) || ldx > SP_MAX_LD || ldw > SP_MAX_LD) FERRIS_REFUSE("gemm: %d x %d outputs", M, N);
    if (token_tile % 32 || token_tile < 0 || token_tile > 128 || splits < 0 || splits > SP_MAX_SPLITS || (swiglu && (splits > 1 || bias || accumulate)))
        FERRIS_REFUSE("gemm: token tile %d, %d splits", token_tile, splits);
    const SplitPlan q = split_plan(M, swiglu ? 2 * N : N, K, swiglu != 0, token_tile, splits);
    if (!q.nt) FERRIS_REFUSE("gemm: %d k's in %d splits", K, splits);
    return run_split(x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, swiglu ? N : 0, 0, q, (cudaStream_t)stream);
}
