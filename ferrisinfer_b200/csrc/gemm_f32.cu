// The 32-bit path's matrix products of up to 150 million multiply-adds or 32 rows (gemm_f32_split.cu takes the larger ones): out[t, n] (+)=
// sum_k x[t, k] * w[n, k] (+ bias[n]), every product and sum an fp32 FMA
// or an fp32 add on the CUDA cores (no tensor cores, no reduced precision), in ONE order of summation for every number of
// rows that comes here, so that a row's result does not depend on what else is in the batch: within runs of F32_CHUNK the even and the odd k's
// ascending, each a chain of FMAs, and the two added; the runs added in ascending order within at most F32_PARTS parts of K, the parts in ascending order (gemm_simt.cu, which takes
// what is not aligned, sums in the same order).  Runs that add up by themselves are what lets several lanes, warps
// and CTAs work on one output; they also halve the rounding error of one long chain.
//
// gemm_f32_rows_kernel: few tokens (decode steps).  Bound by reading the weights once.  The weight ROWS are divided among
// the CTAs; a producer warp streams them through a ring of stages (bulk copies, a row a copy; a model's weights before the
// launch wait), the step's rows lie in shared memory, and a lane sums one run of one weight row for all tokens: eight
// lanes take eight rows, four such groups four runs, so that every shared-memory read of weights is free of conflicts and
// every read of a token's values is shared by eight lanes.  The runs' sums meet in shared memory and are added in order.
// What binds it beside HBM is what shared memory returns to the lanes: 16 bytes a lane take four cycles, shared or not, so a
// step of 16 KB of weights takes 32 x 4 x (1 + tokens) cycles.  Measured (us, 24 layers' weights in turn; 1 / 4 / 8 tokens; before,
// one 64 x 64 tile kernel for all sizes, 250 on the average product of a step of four): 1152 x 896 3.4 / 4.2 / 5.8, 896 x 896
// 3.4 / 4.1 / 5.7, 9728 x 896 12.3 / 15.7 / 22.9, 896 x 4864 10.1 / 10.6 / 19.8, 151936 x 896 98 / 142 / 203 (5.5 TB/s at one).
// Two or four weight rows a lane (a ring twice as large and one CTA an SM): 17 / 22 / 28 at 9728 x 896.
// SwiGLU rides in it: a CTA takes the gate rows and the up rows of its outputs, eight by eight in turn (four requests
// of 96 + 24 tokens at the 0.5B sizes 44.0 -> 40.4 ms; the RMSNorm formed in every CTA as well: 42.5, what its launch cost the wait for
// the rows took twice).
//
// gemm_f32_tile_kernel: prompts.  Bound by the FMA pipes and, as closely, by what shared memory returns to the lanes (16
// bytes a lane take four cycles of an SM a warp, whether lanes share them or not).  64 x 64 tiles, k-slices of 32 through a
// cp.async ring; a thread holds 8 x 4 outputs and reads both operands four k at a time, two FMAs an instruction (the even and
// the odd k's); where tiles are few, the parts of K are divided among the CTAs of a cluster and added through its shared
// memory.  Measured at 777 / 2,048 tokens (us; before: 240 / 215 / 1,030 / 960 at 777): 1152 x 896 60 / 108, 896 x 896 52 /
// 108, 9728 x 896 350 / 815 (44 TFLOP/s of 74), 896 x 4864 216 / 562.  8 x 8 outputs a thread in 64 x 64 or 128 x 64 tiles: the
// same within 3 % at many rows, slower at few.
#include "common.cuh"
#include "gemm_f32.cuh"
#include "sm100.cuh"

namespace {

// ------------------------------------------------------------------------------------------------ few tokens
constexpr int ROWS_WARPS = 4;
constexpr int ROWS_THREADS = ROWS_WARPS * 32 + 32;
constexpr int ROWS_MAX_STAGES = 32;
constexpr int PHASE = 4 * F32_CHUNK;  // k's of a weight row in a stage: a run for each of a warp's four groups of lanes
constexpr int W_PITCH = PHASE + 4;    // floats between a stage's rows: eight rows meet eight bank groups
constexpr int RS = 8;                 // weight rows in a stage
constexpr int ROWS_CAP = 64;          // most weight rows of a CTA: an output head's CTAs come in several rounds
constexpr int ROWS_SMEM = 110 * 1024; // two CTAs to an SM where the sizes allow it: one streams while the other's ends meet
constexpr int X_PITCH = F32_CHUNK + 4;  // floats between a token's runs: the four runs of a warp meet four bank groups

struct RowsParams {
    const float* x;
    const float* w;
    const float* bias;
    float* out;
    int M, N, K, ldx, ldw, ldo, accumulate;
    int rows_per_cta, phases, stages;  // stages: a multiple of ROWS_WARPS, so that one warp takes a stage every time
    int* status;
    int early_weights;  // no launch that may still run writes w: its rows are requested ahead of the launch wait
    int up_offset;  // > 0: SwiGLU, out[t, n] of gate row n and up row up_offset + n; N outputs of 2 N weight rows
};

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Two fp32 FMAs of one instruction: the even k's and the odd k's of a run are two chains.
__device__ __forceinline__ void fma4(float4 a, float4 b, float2& c) {
    unsigned long long& c2 = reinterpret_cast<unsigned long long&>(c);
    const unsigned long long* a2 = reinterpret_cast<const unsigned long long*>(&a);
    const unsigned long long* b2 = reinterpret_cast<const unsigned long long*>(&b);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c2) : "l"(a2[0]), "l"(b2[0]));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c2) : "l"(a2[1]), "l"(b2[1]));
}

template <int TT>  // tokens of a CTA
__global__ void __launch_bounds__(ROWS_THREADS) gemm_f32_rows_kernel(const RowsParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + ROWS_MAX_STAGES;
    float* ring = reinterpret_cast<float*>(smem + 2 * ROWS_MAX_STAGES * sizeof(uint64_t));
    constexpr int stage_floats = RS * W_PITCH;
    const int runs = (p.K + F32_CHUNK - 1) / F32_CHUNK;
    float* xs = ring + p.stages * stage_floats;
    const int xp = runs * X_PITCH;
    float* part = xs + TT * xp;  // [run][row of the CTA][token]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool pairs = p.up_offset > 0;  // groups of eight weight rows: gate, up, gate, up, ...
    const int outs_per_cta = pairs ? p.rows_per_cta / 2 : p.rows_per_cta;
    const int n0 = blockIdx.x * outs_per_cta, m0 = blockIdx.y * TT;
    const int outs = min(outs_per_cta, p.N - n0), mt = min(TT, p.M - m0);
    const int groups = (outs + RS - 1) / RS * (pairs ? 2 : 1);
    auto group_outs = [&](int g) { return min(RS, outs - (pairs ? g >> 1 : g) * RS); };
    auto group_row = [&](int g) { return n0 + (pairs ? (g & 1) * p.up_offset + (g >> 1) * RS : g * RS); };
    const int rowsp = p.rows_per_cta;
    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();
    if (warp == ROWS_WARPS) {
        if (!p.early_weights) pdl_wait();
        const int total = groups * p.phases;
        for (int it = 0; it < total; ++it) {
            const int s = it % p.stages, round = it / p.stages;
            const int g = it / p.phases, k0 = (it % p.phases) * PHASE;
            if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, p.status, 0x60)) break;
            const int nr = group_outs(g);
            const uint32_t bytes = 4u * min(PHASE, p.K - k0);
            if (lane == 0) mbar_expect_tx(&full[s], bytes * nr);
            __syncwarp();
            if (lane < nr)
                bulk_load(ring + s * stage_floats + lane * W_PITCH, p.w + (size_t)(group_row(g) + lane) * p.ldw + k0, bytes,
                          &full[s]);
        }
        return;
    }
    pdl_wait();
    const int k4s = p.K >> 2;
    for (int k4 = tid; k4 < k4s; k4 += ROWS_WARPS * 32) {
        float4 v[TT];
#pragma unroll
        for (int t = 0; t < TT; ++t)
            v[t] = t < mt ? *reinterpret_cast<const float4*>(p.x + (size_t)(m0 + t) * p.ldx + 4 * k4)
                          : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float* at = xs + (k4 / (F32_CHUNK / 4)) * X_PITCH + 4 * (k4 % (F32_CHUNK / 4));
#pragma unroll
        for (int t = 0; t < TT; ++t) *reinterpret_cast<float4*>(at + t * xp) = v[t];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(ROWS_WARPS * 32) : "memory");
    const int r = lane & 7, sub = lane >> 3;
    const int tasks = groups * p.phases;
    for (int it = warp; it < tasks; it += ROWS_WARPS) {
        const int s = it % p.stages;
        const int g = it / p.phases, ph = it % p.phases;
        if (!mbar_wait(&full[s], (it / p.stages) & 1, p.status, 0x61)) break;
        const int kl = sub * F32_CHUNK, k0 = ph * PHASE + kl;
        const int len = min(F32_CHUNK, p.K - k0);
        const int run = k0 / F32_CHUNK;
        float2 acc[TT];
#pragma unroll
        for (int t = 0; t < TT; ++t) acc[t] = make_float2(0.0f, 0.0f);
        const float* wr = ring + s * stage_floats + r * W_PITCH + kl;
        const float* xr = xs + run * X_PITCH;
#pragma unroll 4
        for (int k = 0; k < len; k += 4) {
            const float4 wv = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
            for (int t = 0; t < TT; ++t)
                fma4(*reinterpret_cast<const float4*>(xr + t * xp + k), wv, acc[t]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        const int row = g * RS + r;
        if (len > 0 && r < group_outs(g)) {
#pragma unroll
            for (int t = 0; t < TT; ++t) part[((size_t)run * rowsp + row) * TT + t] = acc[t].x + acc[t].y;
        }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(ROWS_WARPS * 32) : "memory");
    const int per = f32_runs_per_part(runs);
    auto total_of = [&](int row, int t) {
        float total = 0.0f;
        for (int c0 = 0; c0 < runs; c0 += per) {
            float sum = 0.0f;
            const int c1 = min(runs, c0 + per);
            for (int c = c0; c < c1; ++c) sum += part[((size_t)c * rowsp + row) * TT + t];
            total += sum;
        }
        return total;
    };
    for (int i = tid; i < outs * mt; i += ROWS_WARPS * 32) {
        const int row = i % outs, t = i / outs;
        const int n = n0 + row;
        float* o = p.out + (size_t)(m0 + t) * p.ldo + n;
        if (pairs) {
            const int at = row / RS * 2 * RS + row % RS;
            const float g = total_of(at, t), u = total_of(at + RS, t);
            const float sg = g * (1.0f / (1.0f + expf(-g)));
            *o = u * sg;
            continue;
        }
        const float old = p.accumulate ? *o : 0.0f;
        float total = total_of(row, t);
        if (p.bias) total += p.bias[n];
        *o = p.accumulate ? old + total : total;
    }
}

// --------------------------------------------------------------------------------------------------- prompts
constexpr int BM = 64, BN = 64, BK = 32, TM = 8, TN = 4, TILE_STAGES = 3;
constexpr int T_PITCH = BK + 4;  // floats: consecutive rows lie 16 bytes apart modulo 128

struct TileParams {
    const float* x;
    const float* w;
    const float* bias;
    float* out;
    int M, N, K, ldx, ldw, ldo, accumulate;
    int parts, part_k;  // parts of K and the k's of each but the last
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(BM * BN / (TM * TN), 3) gemm_f32_tile_kernel(const TileParams p) {
    constexpr int THREADS = BM * BN / (TM * TN), WN = BN / (8 * TN);  // warps of 32 x (8 TN) outputs, WN of them along n
    constexpr int STAGE = (BM + BN) * T_PITCH;
    extern __shared__ __align__(128) unsigned char smem[];
    float* ring = reinterpret_cast<float*>(smem);
    float* kept = ring + TILE_STAGES * STAGE;  // [output of a thread][thread]: a part's sums, or the parts' so far
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int splits = gridDim.z, rank = blockIdx.z;  // 1, or a CTA of the cluster for every part
    const int ln = (lane & 7) + (warp % WN) * 8 * TN, lm = (lane >> 3) + (warp / WN) * 32;
    pdl_launch_dependents();
    pdl_wait();
    // a thread's pieces of a slice: one 16-byte column of every THREADS / (BK / 4)th row
    const int lk = 4 * (tid % (BK / 4)), lrow = tid / (BK / 4);
    float tot[TM][TN];
    for (int part = rank; part < p.parts; part += splits) {
        const int kbeg = part * p.part_k, kend = min(p.K, kbeg + p.part_k);
        const int slices = (kend - kbeg + BK - 1) / BK;
        auto request = [&](int sl) {
            if (sl < slices) {
                float* st = ring + (sl % TILE_STAGES) * STAGE;
                const int k = kbeg + sl * BK + lk;
#pragma unroll
                for (int row = 0; row < BM + BN; row += THREADS / (BK / 4)) {
                    const bool ofx = row < BM;  // (a multiple of the rows that the threads take together)
                    const int at = ofx ? m0 + row + lrow : n0 + row - BM + lrow;
                    const bool there = k < kend && at < (ofx ? p.M : p.N);
                    const float* src = ofx ? p.x + (size_t)(there ? at : 0) * p.ldx : p.w + (size_t)(there ? at : 0) * p.ldw;
                    cp_async16(st + (row + lrow) * T_PITCH + lk, src + (there ? k : 0), there);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float2 acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                acc[i][j] = make_float2(0.0f, 0.0f);
                tot[i][j] = 0.0f;
            }
        __syncthreads();
        for (int sl = 0; sl < TILE_STAGES - 1; ++sl) request(sl);
        for (int sl = 0; sl < slices; ++sl) {
            asm volatile("cp.async.wait_group %0;" ::"n"(TILE_STAGES - 2) : "memory");
            __syncthreads();
            request(sl + TILE_STAGES - 1);
            const float* st = ring + (sl % TILE_STAGES) * STAGE;
            const float* xa = st + lm * T_PITCH;
            const float* wb = st + (BM + ln) * T_PITCH;
#pragma unroll 2
            for (int k = 0; k < BK; k += 4) {
                float4 b[TN];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(wb + 8 * j * T_PITCH + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(xa + 4 * i * T_PITCH + k);
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma4(a, b[j], acc[i][j]);
                }
            }
            if ((sl + 1) % (F32_CHUNK / BK) == 0 || sl + 1 == slices) {  // a run ends
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        tot[i][j] += acc[i][j].x + acc[i][j].y;
                        acc[i][j] = make_float2(0.0f, 0.0f);
                    }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (splits > 1) {
#pragma unroll
            for (int i = 0; i < TM * TN; ++i) kept[i * THREADS + tid] = tot[i / TN][i % TN];
        } else if (p.parts > 1) {
#pragma unroll
            for (int i = 0; i < TM * TN; ++i) {
                float* k = kept + i * THREADS + tid;
                tot[i / TN][i % TN] = *k = part ? *k + tot[i / TN][i % TN] : tot[i / TN][i % TN];
            }
        }
    }
    auto store = [&](int i, int j, float v) {
        const int m = m0 + 4 * i + lm, n = n0 + 8 * j + ln;
        if (m >= p.M || n >= p.N) return;
        if (p.bias) v += p.bias[n];
        float* o = p.out + (size_t)m * p.ldo + n;
        *o = p.accumulate ? *o + v : v;
    };
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) store(i, j, tot[i][j]);
        return;
    }
    cluster_sync();
    // a thread's outputs are divided among the CTAs of the cluster; each adds the parts in ascending order
    const uint32_t base = smem_u32(kept);
    for (int i = rank; i < TM * TN; i += splits) {
        float v = 0.0f;
        for (int part = 0; part < splits; ++part) v += ld_peer_shared_f32(base + 4u * (i * THREADS + tid), part);
        store(i / TN, i % TN, v);
    }
    cluster_sync();  // nobody leaves while a peer reads
}

// ------------------------------------------------------------------------------------------------- launching
template <int TT>
int launch_rows(RowsParams& p, size_t smem, cudaStream_t s) {
    if (int rc = ferris_allow_dynamic_smem((const void*)gemm_f32_rows_kernel<TT>, smem)) return rc;
    const int outs = p.up_offset > 0 ? p.rows_per_cta / 2 : p.rows_per_cta;
    dim3 grid((p.N + outs - 1) / outs, (p.M + TT - 1) / TT);
    ferris_launch(gemm_f32_rows_kernel<TT>, grid, dim3(ROWS_THREADS), smem, s, p);
    FERRIS_LAUNCH_CHECK();
}

struct RowsPlan {
    int TT, rows_per_cta, phases, stages;
    size_t smem;
};
int launch_rows_of(RowsParams& p, const RowsPlan& q, cudaStream_t s) {
    if (q.TT == 8) return launch_rows<8>(p, q.smem, s);
    if (q.TT == 4) return launch_rows<4>(p, q.smem, s);
    if (q.TT == 2) return launch_rows<2>(p, q.smem, s);
    return launch_rows<1>(p, q.smem, s);
}

int launch_tile(TileParams& p, dim3 grid, cudaStream_t s) {
    const size_t smem = (size_t)TILE_STAGES * (BM + BN) * T_PITCH * 4 + (p.parts > 1 ? (size_t)BM * BN * 4 : 0);
    if (int rc = ferris_allow_dynamic_smem((const void*)gemm_f32_tile_kernel, smem)) return rc;
    if (grid.z > 1)
        ferris_launch_cluster(gemm_f32_tile_kernel, grid, dim3(BM * BN / (TM * TN)), smem, s, grid.z, p);
    else
        ferris_launch(gemm_f32_tile_kernel, grid, dim3(BM * BN / (TM * TN)), smem, s, p);
    FERRIS_LAUNCH_CHECK();
}

constexpr size_t MAX_SMEM = 227 * 1024;
constexpr int SMS = 148;
constexpr int TILE_SPLIT = 2 * SMS;  // fewer tiles than two an SM: the parts of K side by side

// How few tokens are cut (N weight rows; unit: a CTA's are a multiple of so many); false: they do not fit.
bool rows_plan(int M, int N, int K, int unit, RowsPlan& q) {
    const int runs = (K + F32_CHUNK - 1) / F32_CHUNK;
    q.phases = (K + PHASE - 1) / PHASE;
    for (int tt = M >= 5 ? 8 : M >= 3 ? 4 : M; tt >= 1; tt /= 2) {
        q.TT = tt;
        const int rows = ((N + SMS - 1) / SMS + unit - 1) / unit * unit;
        q.rows_per_cta = rows > ROWS_CAP ? ROWS_CAP : rows;
        const size_t round = (size_t)ROWS_WARPS * RS * W_PITCH * 4;  // a stage for every warp
        const size_t fixed = 2 * ROWS_MAX_STAGES * sizeof(uint64_t) + (size_t)tt * runs * X_PITCH * 4 +
                             (size_t)runs * q.rows_per_cta * tt * 4;
        const int wanted = (q.rows_per_cta / RS * q.phases + ROWS_WARPS - 1) / ROWS_WARPS;
        const size_t room = ROWS_SMEM >= fixed + round ? ROWS_SMEM : MAX_SMEM;
        if (fixed + round > room) continue;
        int rounds = (int)((room - fixed) / round);
        rounds = rounds > ROWS_MAX_STAGES / ROWS_WARPS ? ROWS_MAX_STAGES / ROWS_WARPS : rounds;
        q.stages = ROWS_WARPS * (rounds > wanted ? wanted : rounds);
        q.smem = fixed + q.stages / ROWS_WARPS * round;
        return true;
    }
    return false;
}

// Whether few tokens are better off with the rows kernel, cut so, than with the tiles.  The rows kernel goes over the weights
// once for every q.TT tokens, and the longer K is the fewer tokens' rows fit (eight up to K = 3,584 or so, four at 4,864 to 8,960 and for
// 37,888 rows of 3,584, one at 18,944); the tiles do the work of 64 tokens whatever their number.  Both from estimates: a round of the
// rows kernel's CTAs takes in weights at the rates below (KB a microsecond a CTA; two share an SM where their memory allows), a
// tile's CTA 0.09 us a k, three to an SM.  They are within a fifth or so, and the rows kernel is left only where it loses by more
// (us, rows / tiles, tokens: 3,584 x 18,944 three 263 / 280, four 351 / 280, eight 614 / 281, sixteen 1,139 / 280; 37,888 x 3,584 eight 282 / 409, twelve
// 423 / 409, sixteen 563 / 409; sixteen tokens: 9,728 x 896 38 / 44, 896 x 4,864 35 / 51, 17,920 x 1,536 85 / 98, 1,536 x 8,960 82 / 92, 4,608 x 3,584
// 55 / 79, 3,584 x 3,584 53 / 50).
bool rows_pay(int M, int N, int K, const RowsPlan& q) {
    const int each = q.smem <= ROWS_SMEM ? 2 : 1;
    const long long ctas = (long long)((N + q.rows_per_cta - 1) / q.rows_per_cta) * ((M + q.TT - 1) / q.TT);
    const double rate = each == 2 ? 12.5e3 : q.TT == 8 ? 17.5e3 : q.TT == 4 ? 23e3 : 27e3;
    const double t_rows = (double)((ctas + SMS * each - 1) / (SMS * each)) * q.rows_per_cta * K * 4.0 / rate;
    const int runs = (K + F32_CHUNK - 1) / F32_CHUNK, per = f32_runs_per_part(runs);
    long long tiles = (long long)((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    double k = K;
    if (tiles < TILE_SPLIT) {
        tiles *= (runs + per - 1) / per;
        k = runs > per ? per * F32_CHUNK : K;
    }
    const double t_tiles = 0.09 * k * (tiles > 3 * SMS ? (double)tiles / (3 * SMS) : 1.0);
    return t_rows <= 1.25 * t_tiles;
}

// The rows kernel up to 16 tokens, and up to 32 where the weights are few (us at 32 / 33 tokens: 9728 x 896 62 / 44, 896 x 4864 67 / 49,
// 151936 x 896 730 / 422, but 1152 x 896 11 / 18), where it pays.
bool rows_take(int M, int N, int K, int unit, RowsPlan& q) {
    return (M <= 16 || (M <= 32 && (long long)N * K <= (1 << 21))) && rows_plan(M, N, K, unit, q) && rows_pay(M, N, K, q);
}

}  // namespace

// How a 32-bit product of aligned rows is cut: tokens of a CTA of the rows kernel, 0 where the tiles take it (swiglu: N outputs of
// 2 N weight rows; 0 also where SwiGLU does not ride along).
FERRIS_API int ferris_gemm_f32_plan(int M, int N, int K, int swiglu) {
    RowsPlan q;
    if (M <= 0 || N <= 0 || K <= 0 || K & 3) return 0;
    return rows_take(M, swiglu ? 2 * N : N, K, swiglu ? 2 * RS : RS, q) ? q.TT : 0;
}

bool ferris_gemm_f32_takes(const void* x, const void* w, const void* out, int K, int ldx, int ldw) {
    return !(K & 3) && !(ldx & 3) && !(ldw & 3) && !(((uintptr_t)x | (uintptr_t)w) & 15) && K <= 65536;
}

int ferris_gemm_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx, int ldw,
                    int ldo, int accumulate, int early_weights, cudaStream_t s, bool* taken) {
    *taken = true;
    RowsPlan q;
    if (rows_take(M, N, K, RS, q)) {
        RowsParams p = {x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, q.rows_per_cta, q.phases, q.stages, ferris_status_ptr(),
                        early_weights, 0};
        return launch_rows_of(p, q, s);
    }
    if (ferris_gemm_f32_split_takes(M, N, K, ldx, ldw))
        return ferris_gemm_f32_split(x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, 0, early_weights, s);
    const int runs = (K + F32_CHUNK - 1) / F32_CHUNK, per = f32_runs_per_part(runs);
    const int parts = (runs + per - 1) / per;
    if ((M + BM - 1) / BM > 65535) {
        *taken = false;
        return FERRIS_OK;
    }
    TileParams p = {x, w, bias, out, M, N, K, ldx, ldw, ldo, accumulate, parts, per * F32_CHUNK};
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if ((int)(grid.x * grid.y) < TILE_SPLIT) grid.z = parts;
    return launch_tile(p, grid, s);
}

constexpr int SWIGLU_MAX_TOKENS = 16;  // (beyond, the plain product may run the tiles)

// Whether ferris_gemm_f32_swiglu takes a product of M tokens and N outputs, of rows that begin on 16 bytes: few tokens whose weights the
// rows kernel reads in fewer microseconds than the tiles, and what goes to the tensor cores.
FERRIS_API int ferris_gemm_f32_swiglu_takes(const void* x, const void* w, int M, int N, int K, int ldx, int ldw) {
    RowsPlan q;
    if (M <= 0 || N <= 0 || N > (1 << 30) || !ferris_gemm_f32_takes(x, w, nullptr, K, ldx, ldw)) return 0;
    return M <= SWIGLU_MAX_TOKENS ? rows_take(M, 2 * N, K, 2 * RS, q) : ferris_gemm_f32_split_takes(M, 2 * N, K, ldx, ldw);
}
// out[t, n] = silu(x[t] . w[n]) (x[t] . w[N + n]), fp32 throughout, with the sums of the plain product (on the tensor cores: of one without K
// splits, which the 2 N rows have where there are many of them).
// early_weights: no launch that may still run writes w.
FERRIS_API int ferris_gemm_f32_swiglu(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldw, int ldo,
                                      int early_weights, void* stream) {
    if (M <= 0 || N <= 0) return FERRIS_OK;
    if (K <= 0 || ldx < K || ldw < K || ldo < N) FERRIS_REFUSE("gemm: K=%d, row strides %d, %d, %d", K, ldx, ldw, ldo);
    if (!ferris_gemm_f32_swiglu_takes(x, w, M, N, K, ldx, ldw))
        FERRIS_REFUSE("gemm: %d tokens x %d outputs of %d do not take SwiGLU on the way", M, N, K);
    if (M > SWIGLU_MAX_TOKENS)
        return ferris_gemm_f32_split(x, w, nullptr, out, M, N, K, ldx, ldw, ldo, 0, N, early_weights, (cudaStream_t)stream);
    RowsPlan q;
    rows_plan(M, 2 * N, K, 2 * RS, q);
    RowsParams p = {x, w, nullptr, out, M, N, K, ldx, ldw, ldo, 0, q.rows_per_cta, q.phases, q.stages, ferris_status_ptr(), early_weights, N};
    return launch_rows_of(p, q, (cudaStream_t)stream);
}
