// Linear attention with a fixed decay per head over portions of prompts, 64 tokens at a time (linear_attention.cu holds the
// formulas and the walk token by token, which single tokens, short portions and the 32-bit path keep).
//
// With S_0 the state at the start of a chunk of n tokens, everything in it is a matrix product:
//     o_t = decay^(t+1) S_0^T q_t + sum_(i<=t) decay^(t-i) (q_t . k_i) v_i
//     S_n = decay^n S_0 + sum_i decay^(n-1-i) k_i v_i^T
// Four kernels: q, k and v of every token as they enter, in fp32; each chunk's own sum of k v^T, all side by side; the states at the chunks' starts, an elementwise walk over the
// chunks; the outputs, all side by side.
//
// The products are tf32 fragments with fp32 sums.  What enters is fp32 (q, k, v after SiLU or rotation, the state, the weights
// between tokens), so every operand is cut into its leading eleven bits and the rest, both rounded to nearest, and big x big, big
// x rest and rest x big are added; the big products leave the tensor core after eight of them and are added by fp32 additions (its
// own additions cut off).  Powers of the decay come from doubles.  Against 64 bits, 16 heads of 128, errors of the outputs / of the
// last state in units of 1e-7 of their norm, before (the walk): with SiLU 2,048 tokens 1.4 / 2.8, 300 tokens 0.8 / 2.3, without
// 2.1 / 2.1 and 1.9 / 1.9; now 1.1 / 0.9 and 1.1 / 0.9, 1.3 / 0.9 and 1.2 / 0.9.
// What bounds it: the instructions around the products (two loads, six cuts and four additions for three products) at sixteen
// warps an SM; the tensor pipe is a quarter busy.  64 tokens and 64 columns a block: 104 KB of shared memory and less than 128
// registers, so that two blocks share an SM and one's rows come in while the other multiplies; the columns' two halves form q . k
// twice, which costs 16 % of the products.  q, k and v are activated and turned once by a kernel of their own, not by each of the
// four blocks that read them (166 -> 137 us).  us, 16 heads of 128 / 128, the walk (in segments of 128 tokens side by side) and
// the chunks: one request of 2,048 tokens 428 / 137, four of 512 392 / 132, one of 256 197 / 30, of 64 57 / 26, of 48 43 / 25, of 32
// 30 / 30 (the walk's last); 31 single tokens beside 481 331 / 102.
#include "common.cuh"
#include "linear_attention.cuh"
#include "sm100.cuh"

namespace {

constexpr int LC_TOKENS = 64;  // of a chunk
constexpr int LC_COLS = 64;    // value columns of a block
constexpr int LC_THREADS = 256;
constexpr int A_PITCH = LC_TOKENS + 4, V_PITCH = LC_COLS + 8;  // pitches 4 (8) modulo 32: fragments read along rows (columns)

struct ChunkArgs {
    const bf16* qkv;
    float* rows;  // what enters the recurrence, fp32: [tokens][q heads | k heads | v heads]
    float* out;
    float* state;
    float* scratch;
    const float* decay;
    const int* seq_q_start;
    const int* seq_state_slot;
    int ld, q_off, k_off, v_off, ldo, heads, dim, vdim, silu, write_state, chunks_max, above;  // above: requests of at most so many tokens are not taken
    RotaryArgs rot;
};

__device__ __forceinline__ void cut_tf32(float x, uint32_t& big, uint32_t& rest) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(big) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(rest) : "f"(x - __uint_as_float(big)));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// Sums of products: the tensor core adds by cutting off, so it sums eight big products at a time from zero, and those sums are
// added by rounded fp32 additions; the small products (2^-11 of the big ones) stay in its accumulator.
template <int TILES>
struct CutSums {
    float big[TILES][4] = {}, small[TILES][4] = {};
    __device__ __forceinline__ float get(int j, int e) const { return big[j][e] + small[j][e]; }
};
// c += a b over eight inner indices for up to TILES tiles of eight columns; B's element (k, n) of tile j lies at
// b[k * bk + (tile_step * j + n) * bn], A's (row, k) at a[row * am + k * ak], times factor[k] with SCALED.
template <int TILES, bool SCALED = false>
__device__ __forceinline__ void cut_products(CutSums<TILES>& c, const float* a, int am, int ak, const float* b, int bk, int bn,
                                             int tile_step, int tiles, const float* factor = nullptr) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float f0 = SCALED ? factor[t] : 1.0f, f1 = SCALED ? factor[t + 4] : 1.0f;
    uint32_t ab[4], ar[4];
    cut_tf32(f0 * a[g * am + t * ak], ab[0], ar[0]);
    cut_tf32(f0 * a[(g + 8) * am + t * ak], ab[1], ar[1]);
    cut_tf32(f1 * a[g * am + (t + 4) * ak], ab[2], ar[2]);
    cut_tf32(f1 * a[(g + 8) * am + (t + 4) * ak], ab[3], ar[3]);
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
        if (j < tiles) {
            uint32_t bb[2], br[2];
            const float* at = b + (tile_step * j + g) * bn + t * bk;
            cut_tf32(at[0], bb[0], br[0]);
            cut_tf32(at[4 * bk], bb[1], br[1]);
            float eight[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_tf32(eight, ab, bb);
            mma_tf32(c.small[j], ar, bb);
            mma_tf32(c.small[j], ab, br);
#pragma unroll
            for (int e = 0; e < 4; ++e) c.big[j][e] += eight[e];
        }
    }
}

// base^n: a few roundings in 64 bits
__device__ __forceinline__ float power(float base, int n) {
    double r = 1.0, b = base;
    for (; n; n >>= 1, b *= b)
        if (n & 1) r *= b;
    return (float)r;
}

// q, k and v of a token as they enter the recurrence, activated, turned and scaled, once for all blocks that need them.
constexpr int LP_THREADS = 256;
__global__ void __launch_bounds__(LP_THREADS) linear_chunk_rows_kernel(const ChunkArgs p) {
    extern __shared__ __align__(16) float lc_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const size_t t = blockIdx.x;
    const int qk = p.heads * p.dim, width = 2 * qk + p.heads * p.vdim;
    const bf16* src = p.qkv + t * p.ld;
    for (int x = threadIdx.x * 8; x < width; x += LP_THREADS * 8) {
        const bf16* at = src + (x < qk ? p.q_off + x : x < 2 * qk ? p.k_off + x - qk : p.v_off + x - 2 * qk);
        const uint4 u = *reinterpret_cast<const uint4*>(at);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        float f[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) f[2 * i] = __uint_as_float(w[i] << 16), f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        if (p.silu) {
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = silu_f(f[i]);
        }
        float4* to = reinterpret_cast<float4*>(lc_smem + x);
        to[0] = make_float4(f[0], f[1], f[2], f[3]);
        to[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    __syncthreads();
    const RotaryArgs& rot = p.rot;
    const int rotary = rot.positions ? rot.rotary : 0, half = rotary >> 1;
    if (half > 0) {
        const float pos = (float)rot.positions[t];
        for (int f = threadIdx.x; f < half; f += LP_THREADS) {
            float sn, cs;
            sincosf(pos * rot.freq[f], &sn, &cs);
            sn *= rot.mag, cs *= rot.mag;
            const int iu = rot.interleaved ? 2 * f : f, iv = rot.interleaved ? 2 * f + 1 : f + half;
            for (int h = 0; h < p.heads; ++h) {
                float *qr = lc_smem + h * p.dim, *kr = qr + qk;
                const float qu = qr[iu], qv = qr[iv], ku = kr[iu], kv = kr[iv];
                qr[iu] = qu * cs - qv * sn;
                qr[iv] = qv * cs + qu * sn;
                kr[iu] = ku * cs - kv * sn;
                kr[iv] = kv * cs + ku * sn;
            }
        }
        __syncthreads();
    }
    float* dst = p.rows + t * width;
    for (int x = threadIdx.x * 4; x < width; x += LP_THREADS * 4) {
        float4 v = *reinterpret_cast<const float4*>(lc_smem + x);
        if (x >= qk && x < 2 * qk) v.x *= rot.k_scale, v.y *= rot.k_scale, v.z *= rot.k_scale, v.w *= rot.k_scale;
        *reinterpret_cast<float4*>(dst + x) = v;
    }
}

// Requests the n rows of `cols` floats (a multiple of four) that begin at src into rows of `pitch` floats; rows from n to LC_TOKENS
// and columns from `cols` to `fill` are zeros.
__device__ __forceinline__ void request_rows(float* dst, int pitch, const float* src, size_t ld, int n, int cols, int fill) {
    const int pieces = fill >> 2;
    const uint32_t to = smem_u32(dst);
    for (int x = threadIdx.x; x < LC_TOKENS * pieces; x += LC_THREADS) {
        const int t = x / pieces, c = (x - t * pieces) * 4;
        const bool there = t < n && c < cols;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + 4 * (t * pitch + c)),
                     "l"(there ? src + (size_t)t * ld + c : src), "r"(there ? 16 : 0)
                     : "memory");
    }
}
__device__ __forceinline__ void commit_rows() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_rows() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A block's chunk: its first row, its tokens (0: none), whether the request ends with it, its place in scratch.
struct Chunk {
    int row0, n;
    bool last;
    float* state;  // [vdim][dim] of the head
};
__device__ __forceinline__ Chunk chunk_of(const ChunkArgs& p, int head) {
    const int seq = blockIdx.x / p.chunks_max;
    const int first = p.seq_q_start[seq], row1 = p.seq_q_start[seq + 1];
    const int row0 = first + (blockIdx.x % p.chunks_max) * LC_TOKENS;
    Chunk c = {row0, row1 - first > p.above ? min(LC_TOKENS, row1 - row0) : 0, row0 + LC_TOKENS >= row1, nullptr};
    c.state = p.scratch + ((size_t)(row0 / LC_TOKENS + seq) * p.heads + head) * p.vdim * p.dim;
    return c;
}

// A chunk whose products are not finite, token by token as the walk does it: an infinity cut into parts leaves inf - inf, a
// weight of zero meets a later token's, a power of the decay that falls to zero an earlier one's.  `cols` columns of one head,
// four threads each: their values begin at v and the keys and queries at k and q, rows of `width`; the state goes from `start`
// (null: zeros) to `end` (null: not wanted), the outputs to rows of `ldo` at `out` (null: not wanted).  Not inlined: the kernels
// keep their registers.
template <int D>
__device__ __noinline__ void walk_chunk(const float* q, const float* k, const float* v, int width, int n, int dim, int cols, float lam,
                                        const float* start, float* end, float* out, int ldo) {
    const int col = threadIdx.x >> 2, part = threadIdx.x & 3;
    const bool mine = col < cols;
    const size_t at = (size_t)col * dim;
    float S[D / 4];
#pragma unroll
    for (int i = 0; i < D / 4; ++i) S[i] = start && mine && part + 4 * i < dim ? start[at + part + 4 * i] : 0.0f;
    for (int t = 0; t < n; ++t, q += width, k += width, v += width) {
        const float value = mine ? v[col] : 0.0f;
        float o = 0.0f;
#pragma unroll
        for (int i = 0; i < D / 4; ++i) {
            const int d = part + 4 * i;
            if (d < dim) {
                S[i] = fmaf(k[d], value, lam * S[i]);
                o = fmaf(S[i], q[d], o);
            }
        }
        o += __shfl_xor_sync(0xffffffffu, o, 1);
        o += __shfl_xor_sync(0xffffffffu, o, 2);
        if (out && mine && part == 0) out[(size_t)t * ldo + col] = o;
    }
    if (end && mine) {
#pragma unroll
        for (int i = 0; i < D / 4; ++i)
            if (part + 4 * i < dim) end[at + part + 4 * i] = S[i];
    }
}
__device__ __forceinline__ bool is_finite(float x) { return fabsf(x) <= 3.402823466e38f; }

template <int D>
__global__ void __launch_bounds__(LC_THREADS, 2) linear_chunk_sums_kernel(const ChunkArgs p) {
    extern __shared__ __align__(16) float lc_smem[];
    constexpr int K_PITCH = D + 8;
    float* ks = lc_smem;
    float* vs = ks + LC_TOKENS * K_PITCH;
    float* pw = vs + LC_TOKENS * V_PITCH;
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.y, col0 = blockIdx.z * LC_COLS;
    const Chunk c = chunk_of(p, head);
    if (c.n <= 0 || (c.last && !p.write_state)) return;  // nobody starts from the end of the last chunk but the request's state
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int cols = min(LC_COLS, p.vdim - col0);
    const int qk = p.heads * p.dim;
    const size_t width = 2 * qk + p.heads * p.vdim;
    const float* row = p.rows + c.row0 * width;
    request_rows(ks, K_PITCH, row + qk + head * p.dim, width, c.n, p.dim, D);
    request_rows(vs, V_PITCH, row + 2 * qk + head * p.vdim + col0, width, c.n, cols, LC_COLS);
    commit_rows();
    if (tid < LC_TOKENS) pw[tid] = tid < c.n ? power(p.decay[head], c.n - 1 - tid) : 0.0f;
    wait_rows<0>();
    __syncthreads();
    // 16 columns of v and half of the rows of k a warp
    const int m0 = (warp & 3) * 16, d0 = (warp >> 2) * (D / 2);
    CutSums<D / 16> acc;
    for (int t = 0; t < c.n; t += 8)
        cut_products<D / 16, true>(acc, vs + t * V_PITCH + m0, 1, V_PITCH, ks + t * K_PITCH + d0, K_PITCH, 1, 8, D / 16, pw + t);
    bool odd = false;
#pragma unroll
    for (int j = 0; j < D / 16; ++j) {
        const int d = d0 + 8 * j + 2 * t4;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int v = m0 + g + 8 * a;
            const float2 sum = make_float2(acc.get(j, 2 * a), acc.get(j, 2 * a + 1));
            if (v < cols && d < p.dim) {
                odd |= !is_finite(sum.x) || !is_finite(sum.y);
                *reinterpret_cast<float2*>(c.state + (size_t)(col0 + v) * p.dim + d) = sum;
            }
        }
    }
    if (__syncthreads_or(odd))
        walk_chunk<D>(row + head * p.dim, row + qk + head * p.dim, row + 2 * qk + head * p.vdim + col0, (int)width, c.n, p.dim, cols,
                      p.decay[head], nullptr, c.state + (size_t)col0 * p.dim, nullptr, 0);
}

// scratch holds each chunk's own sum; afterwards it holds the state at each chunk's start, and the request's slot its new state.
__global__ void __launch_bounds__(256) linear_chunk_starts_kernel(const ChunkArgs p) {
    constexpr int AHEAD = 8;
    pdl_wait();
    pdl_launch_dependents();
    const int seq = blockIdx.y;
    const size_t per_state = (size_t)p.heads * p.vdim * p.dim;
    const size_t e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const int row0 = p.seq_q_start[seq], row1 = p.seq_q_start[seq + 1];
    if (e >= per_state || row1 - row0 <= p.above) return;
    const float lam = p.decay[e / ((size_t)p.vdim * p.dim)];
    const float step = power(lam, LC_TOKENS);
    // for a power of zero: an infinity stays one however often it decays, also where the power is too small for 32 bits
    auto decayed = [lam](float f, float x) { return lam != 0.0f && isinf(x) ? copysignf(1.0f, f) * x : f * x; };
    float4* slot = reinterpret_cast<float4*>(p.state + (size_t)p.seq_state_slot[seq] * per_state + e);
    float4 S = *slot;
    const int chunks = (row1 - row0 + LC_TOKENS - 1) / LC_TOKENS;
    float* first = p.scratch + e;
    auto place = [&](int c) { return reinterpret_cast<float4*>(first + (size_t)((row0 + c * LC_TOKENS) / LC_TOKENS + seq) * per_state); };
    const int sums = p.write_state ? chunks : chunks - 1;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 own[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < sums) own[i] = *place(c0 + i);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c0 + i < chunks) *place(c0 + i) = S;
            if (c0 + i < sums) {
                const float f = c0 + i + 1 < chunks ? step : power(lam, row1 - row0 - (chunks - 1) * LC_TOKENS);
                if (f != 0.0f) {
                    S.x = fmaf(f, S.x, own[i].x), S.y = fmaf(f, S.y, own[i].y), S.z = fmaf(f, S.z, own[i].z), S.w = fmaf(f, S.w, own[i].w);
                } else {
                    S.x = decayed(f, S.x) + own[i].x, S.y = decayed(f, S.y) + own[i].y;
                    S.z = decayed(f, S.z) + own[i].z, S.w = decayed(f, S.w) + own[i].w;
                }
            }
        }
    }
    if (p.write_state) *slot = S;
}

template <int D>
__global__ void __launch_bounds__(LC_THREADS, 2) linear_chunk_outputs_kernel(const ChunkArgs p) {
    extern __shared__ __align__(16) float lc_smem[];
    constexpr int K_PITCH = D + 4;
    float* qs = lc_smem;
    float* ks = qs + LC_TOKENS * K_PITCH;  // the keys, then the state's columns
    float* vs = ks + LC_TOKENS * K_PITCH;
    float* as = vs + LC_TOKENS * V_PITCH;  // weights between the tokens
    float* pw = as + LC_TOKENS * A_PITCH;  // decay^0 .. decay^64
    static_assert(LC_COLS == LC_TOKENS, "the state's columns stand where the keys stood");
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.y, col0 = blockIdx.z * LC_COLS;
    const Chunk c = chunk_of(p, head);
    if (c.n <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int cols = min(LC_COLS, p.vdim - col0);
    if (tid <= LC_TOKENS) pw[tid] = power(p.decay[head], tid);
    const int qk = p.heads * p.dim;
    const size_t width = 2 * qk + p.heads * p.vdim;
    const float* row = p.rows + c.row0 * width;
    request_rows(qs, K_PITCH, row + head * p.dim, width, c.n, p.dim, D);
    request_rows(ks, K_PITCH, row + qk + head * p.dim, width, c.n, p.dim, D);
    commit_rows();
    request_rows(vs, V_PITCH, row + 2 * qk + head * p.vdim + col0, width, c.n, cols, LC_COLS);
    commit_rows();
    wait_rows<1>();
    __syncthreads();
    // 16 tokens and every other tile of eight columns a warp; a scheduler's two warps have the strips s and 3 - s, whose
    // shares of the triangle add up to the same
    const int strip = warp < 4 ? warp : 7 - warp, odd = warp >> 2, m0 = 16 * strip;
    {
        CutSums<4> acc;
        for (int d = 0; d < D; d += 8)  // tiles 2 j + odd up to the diagonal: j <= strip
            cut_products<4>(acc, qs + m0 * K_PITCH + d, K_PITCH, 1, ks + 8 * odd * K_PITCH + d, 1, K_PITCH, 16, strip + 1);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = m0 + g + 8 * (e >> 1), i = 16 * j + 8 * odd + 2 * t4 + (e & 1);
                as[t * A_PITCH + i] = i <= t ? acc.get(j, e) * pw[t - i] : 0.0f;
            }
    }
    wait_rows<0>();
    __syncthreads();  // v is there, and the keys have been read
    request_rows(ks, K_PITCH, c.state + (size_t)col0 * p.dim, p.dim, cols, p.dim, D);  // the state's columns as rows
    commit_rows();
    const int v0 = 8 * odd;  // tiles 2 j + odd of the columns
    CutSums<4> within, before;
    for (int i = 0; i < m0 + 16; i += 8)
        cut_products<4>(within, as + m0 * A_PITCH + i, A_PITCH, 1, vs + i * V_PITCH + v0, V_PITCH, 1, 16, 4);
    wait_rows<0>();
    __syncthreads();
    for (int d = 0; d < D; d += 8) cut_products<4>(before, qs + m0 * K_PITCH + d, K_PITCH, 1, ks + v0 * K_PITCH + d, 1, K_PITCH, 16, 4);
    bool odd_sum = false;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int t = m0 + g + 8 * a;
        if (t >= c.n) continue;
        float* orow = p.out + (size_t)(c.row0 + t) * p.ldo + (size_t)head * p.vdim + col0;
        const float f = pw[t + 1];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int v = 16 * j + v0 + 2 * t4;
            const float2 o = make_float2(fmaf(f, before.get(j, 2 * a), within.get(j, 2 * a)), fmaf(f, before.get(j, 2 * a + 1), within.get(j, 2 * a + 1)));
            if (v < cols) {
                odd_sum |= !is_finite(o.x) || !is_finite(o.y);
                *reinterpret_cast<float2*>(orow + v) = o;
            }
        }
    }
    if (__syncthreads_or(odd_sum))
        walk_chunk<D>(row + head * p.dim, row + qk + head * p.dim, row + 2 * qk + head * p.vdim + col0, (int)width, c.n, p.dim, cols,
                      p.decay[head], c.state + (size_t)col0 * p.dim, nullptr,
                      p.out + (size_t)c.row0 * p.ldo + (size_t)head * p.vdim + col0, p.ldo);
}

template <int D>
int launch_chunks(const ChunkArgs& p, int tokens, int seqs, cudaStream_t s) {
    constexpr size_t sums = (size_t)(LC_TOKENS * (D + 8) + LC_TOKENS * V_PITCH + LC_TOKENS) * 4;
    constexpr size_t outputs = (size_t)(2 * LC_TOKENS * (D + 4) + LC_TOKENS * V_PITCH + LC_TOKENS * A_PITCH + LC_TOKENS + 1) * 4;
    if (int rc = ferris_allow_dynamic_smem((const void*)linear_chunk_sums_kernel<D>, sums)) return rc;
    if (int rc = ferris_allow_dynamic_smem((const void*)linear_chunk_outputs_kernel<D>, outputs)) return rc;
    const dim3 grid((unsigned)(seqs * p.chunks_max), p.heads, (p.vdim + LC_COLS - 1) / LC_COLS);
    const size_t row_bytes = (size_t)(2 * p.heads * p.dim + p.heads * p.vdim) * 4;
    if (int rc = ferris_allow_dynamic_smem((const void*)linear_chunk_rows_kernel, row_bytes)) return rc;
    const size_t quads = (size_t)p.heads * p.vdim * p.dim / 4;
    ferris_launch(linear_chunk_rows_kernel, dim3(tokens), dim3(LP_THREADS), row_bytes, s, p);
    ferris_launch(linear_chunk_sums_kernel<D>, grid, dim3(LC_THREADS), sums, s, p);
    ferris_launch(linear_chunk_starts_kernel, dim3((unsigned)((quads + 255) / 256), seqs), dim3(256), 0, s, p);
    ferris_launch(linear_chunk_outputs_kernel<D>, grid, dim3(LC_THREADS), outputs, s, p);
    FERRIS_LAUNCH_CHECK();
}

bool chunks_take(const void* qkv, int ld, int q_off, int k_off, int v_off, const void* out, int ldo, const void* state, int seqs,
                 long long longest, int heads, int dim, int vdim) {
    if (dim <= 0 || dim > 128 || vdim <= 0 || heads <= 0 || seqs <= 0 || seqs > 65535 || heads > 65535 || vdim > 65535 * LC_COLS) return false;
    if ((dim | vdim | ld | q_off | k_off | v_off) & 7 || ldo & 1) return false;
    if (heads * (2LL * dim + vdim) * 4 > 200 * 1024) return false;  // a token's row stands in shared memory
    if (((uintptr_t)qkv | (uintptr_t)state) & 15 || (uintptr_t)out & 7) return false;
    return seqs * ((longest + LC_TOKENS - 1) / LC_TOKENS) <= 0x7fffffff;
}

}  // namespace

// Whether ferris_linear_attention_chunks takes a step (bf16 rows; `longest`: the most tokens a request brings).
FERRIS_API int ferris_linear_attention_chunks_takes(const void* qkv, int ld, int q_off, int k_off, int v_off, const void* out, int ldo,
                                                    const void* state, int seqs, int longest, int heads, int dim, int vdim) {
    return chunks_take(qkv, ld, q_off, k_off, v_off, out, ldo, state, seqs, longest, heads, dim, vdim) ? 1 : 0;
}

// Arguments as ferris_linear_attention's, bf16 rows; no request brings more than `longest` tokens, and those that bring
// at most `above` are left alone; scratch: fp32
// [tokens / 64 + seqs + 1, heads, vdim, dim]; rows: scratch, fp32 [tokens, heads x (2 dim + vdim)]; both 16-byte aligned.
FERRIS_API int ferris_linear_attention_chunks(const void* qkv, int ld, int q_off, int k_off, int v_off, float* out, int ldo,
                                              float* state, const float* decay, const int* seq_q_start, const int* seq_state_slot,
                                              int tokens, int seqs, int longest, int above, int heads, int dim, int vdim, int silu,
                                              int write_state, float* scratch, float* rows, const int* positions, const float* freq, int rotary, int interleaved,
                                              float mag, float k_scale, void* stream) {
    if (seqs <= 0 || longest <= 0 || longest <= above) return FERRIS_OK;
    if (above < 0) FERRIS_REFUSE("linear attention: requests above %d tokens", above);
    if (positions && (rotary < 0 || rotary > dim || (rotary & 1) || (rotary > 0 && !freq)))
        FERRIS_REFUSE("linear attention: %d rotated elements of heads of %d", rotary, dim);
    if (!chunks_take(qkv, ld, q_off, k_off, v_off, out, ldo, state, seqs, longest, heads, dim, vdim))
        FERRIS_REFUSE("linear attention: chunks do not take %d heads of %d / %d", heads, dim, vdim);
    if (!state || !decay || !scratch || !rows || ((uintptr_t)scratch | (uintptr_t)rows) & 15 || tokens <= 0)
        FERRIS_REFUSE("linear attention: no state, no decay or no scratch");
    const ChunkArgs p = {(const bf16*)qkv, rows, out, state, scratch, decay, seq_q_start, seq_state_slot, ld, q_off, k_off, v_off, ldo,
                         heads, dim, vdim, silu, write_state, (longest + LC_TOKENS - 1) / LC_TOKENS, above,
                         {positions, freq, rotary, interleaved, mag, k_scale}};
    return dim <= 64 ? launch_chunks<64>(p, tokens, seqs, (cudaStream_t)stream) : launch_chunks<128>(p, tokens, seqs, (cudaStream_t)stream);
}
