// y[t][n] = sum_k x[t][k] * w[n][k] in float32 on the 5th-generation tensor cores, for the float32 path.
//
// Arithmetic.  Every float32 operand is the exact sum of three bfloat16 values: its upper 16 bits, the upper 16 bits
// of what is left, and what is left then (8 + 8 + 8 bits of the 24; truncation, so nothing overflows).  Of the nine
// products of the pieces the six largest are formed (tcgen05.mma multiplies bfloat16 exactly and adds in float32):
//   w0 x0  |  w0 x1 + w1 x0  |  w0 x2 + w1 x1 + w2 x0
// The three dropped ones are below 2^-24 of a product.  Weights, activations and sums are 32-bit in memory: the pieces
// exist in shared and tensor memory only.  The tensor core truncates when it adds, so its chain is kept short: the
// sum of w0 x0 over 64 k is taken out of tensor memory and added with rounding in registers; the small terms (2^-8 and
// 2^-16 of the products) run over a whole segment of the reduction.  Error against float64 (norm of the difference
// over norm of the result, normal operands) beside that of one fmaf chain per output (gemm_simt.cu):
//   inner 64: 1.2e-7, 1.5e-7;  2,048: 1.4e-7, 8.0e-7;  4,096 in one segment: 2.2e-7, 1.2e-6;  12,288: 1.9e-7, 2.0e-6.
//
// An output's sum is formed in an order that depends on (outs, inner) alone: 64-wide k blocks in ascending order
// within a segment, segments in ascending order, whether the segments of a tile run one after the other in a CTA or
// side by side in the CTAs of a cluster.  A row's bits therefore do not depend on what else is in the batch.
// A sum that comes out infinite or NaN (a piece of an infinity is NaN) is formed again with fmaf in ascending k.
//
// Orientation and roles follow the bfloat16 product (gemm_tcgen05.cu): 128 weight rows are the A operand, the tokens
// the narrow B operand.  Warp 0 loads raw float32 tiles with TMA, warp 1 issues the MMAs, eight converter warps make the
// pieces (weights: a thread's row goes to tensor memory, where A is read from; tokens: three stacked bfloat16 tiles in
// shared memory, so that one MMA multiplies a piece of the weights by several pieces of the tokens), eight taker warps add
// the sums of a block up while the MMAs of the next run.
//
// What bounds it: a block takes about 1,500 cycles whatever its tokens: the 16 MMAs hold the thread that issues them
// 58 cycles each, waits for the other roles come on top, and the converters need 1,000 to 1,100.  Beside the CUDA-core
// kernel: 256 x 24,576 x 4,096 (tokens, outs, inner) 2,378 -> 431 us (120 TFLOP/s), 256 x 4,096 x 12,288 1,714 -> 207,
// 512 x 2,048 x 5,632 760 -> 102; 8 x 24,576 x 4,096 807 -> 92 (4.4 TB/s of weights), 8 x 4,096 x 4,096 377 -> 24,
// 1 x 151,936 x 1,024 919 -> 110 (5.7 TB/s).
#include "tcgen05.cuh"

constexpr int SPLIT_ROWS = 128;  // output features per CTA
constexpr int SPLIT_K = 64;      // k per block: two 128-byte rows of float32, one of bfloat16
constexpr int CONVERTERS = 256;  // threads: two warps per quarter of tensor memory's lanes
constexpr int TAKERS = 256;      // threads: two warps per quarter
constexpr int SPLIT_THREADS = 64 + CONVERTERS + TAKERS;
constexpr int MAX_SEGMENTS = 8;

__device__ int g_split_error = 0;  // 0 ok; else (role << 8) | detail of the first failure seen

// NT: tokens per CTA.
template <int NT>
struct SplitConfig {
    static constexpr int W_BYTES = SPLIT_ROWS * SPLIT_K * 4;
    static constexpr int X_BYTES = NT * SPLIT_K * 4;
    static constexpr int RAW_BYTES = W_BYTES + X_BYTES;
    static constexpr int PIECES_BYTES = 3 * NT * SPLIT_K * 2;
    // 16 tokens: 36 KB raw blocks, two CTAs to an SM (one CTA with five blocks in flight was 30 % slower: a block's
    // way through the roles is what takes the time); 64 tokens: 48 KB, one CTA
    static constexpr int STAGES = NT > 16 ? 3 : 2;
    // tensor memory: two buffers of w0 x0, the 2^-8 and the 2^-16 terms, two buffers of the weights' pieces
    static constexpr int SMALL_COLUMN = 2 * NT, A_COLUMN = 4 * NT, A_COLUMNS = 3 * SPLIT_K / 2;
    static constexpr int TMEM_COLUMNS = 4 * NT + 2 * A_COLUMNS <= 256 ? 256 : 512;
    static constexpr int SMEM_BYTES = STAGES * RAW_BYTES + 2 * PIECES_BYTES + 1024 + 128;
};
static_assert(SplitConfig<16>::RAW_BYTES * SplitConfig<16>::STAGES >= 16 * SPLIT_ROWS * 4, "the cluster's exchange reuses the raw tiles");

struct SplitParams {
    const float* x;
    const float* w;
    float* out;
    int tokens, outs, inner;
    int k_blocks, per_segment;
    int clustered;  // the segments of a tile are the CTAs of a cluster along z
    // Grouped product: the weight holds `group_rows` rows per group, one group after the other, and token tile b belongs to
    // group group_of_block[b] (negative: it holds no rows and its CTAs return at once).  `outs` counts one group's features.
    const int* group_of_block;
    int group_rows;
};

__device__ __forceinline__ uint32_t upper_pair(float even, float odd) {  // bfloat16 pair, the even k in the low half
    return __byte_perm(__float_as_uint(even), __float_as_uint(odd), 0x7632);
}
__device__ __forceinline__ float below_upper(float v) { return v - __uint_as_float(__float_as_uint(v) & 0xffff0000u); }

__device__ __forceinline__ float4 lds128(uint32_t address) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t address, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t address, uint32_t rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(address), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ void tcgen05_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tcgen05_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// The sum of one output again, for one that came out infinite or NaN.
__device__ __noinline__ float plain_sum(const float* x, const float* w, int inner) {
    float sum = 0.0f;
    for (int k = 0; k < inner; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        sum = fmaf(a.x, b.x, sum);
        sum = fmaf(a.y, b.y, sum);
        sum = fmaf(a.z, b.z, sum);
        sum = fmaf(a.w, b.w, sum);
    }
    return sum;
}
__device__ __forceinline__ float finite_or_again(const SplitParams& p, int t, int w_row, float v) {
    if (fabsf(v) <= 3.402823466e38f) return v;
    return plain_sum(p.x + static_cast<size_t>(t) * p.inner, p.w + static_cast<size_t>(w_row) * p.inner, p.inner);
}

template <int NT>
__global__ void __launch_bounds__(SPLIT_THREADS, NT <= 16 ? 2 : 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, SplitParams p) {
    using C = SplitConfig<NT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* pieces = raw + C::STAGES * C::RAW_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(pieces + 2 * C::PIECES_BYTES);  // raw tiles arrived
    uint64_t* empty = full + C::STAGES;                                          // raw tiles read by the workers
    uint64_t* ready = empty + C::STAGES;                                         // [2] pieces written
    uint64_t* done = ready + 2;                                                  // [2] MMAs retired
    uint64_t* taken = done + 2;                                                  // [2] sums out of tensor memory
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(taken + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * NT, n0 = blockIdx.y * SPLIT_ROWS;
    const int kb_begin = p.clustered ? blockIdx.z * p.per_segment : 0;
    const int kb_end = p.clustered ? min(kb_begin + p.per_segment, p.k_blocks) : p.k_blocks;
    const int blocks = kb_end - kb_begin;
    int w0 = n0;  // first weight row of the tile
    if (p.group_of_block != nullptr) {
        pdl_wait();  // a kernel before this one wrote the groups
        const int group = p.group_of_block[blockIdx.x];
        if (group < 0) return;  // every CTA of the tile (and of its cluster): nothing has been set up yet
        w0 = group * p.group_rows + n0;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], CONVERTERS / 32); }
        for (int b = 0; b < 2; ++b) { mbar_init(&ready[b], CONVERTERS / 32); mbar_init(&done[b], 1); mbar_init(&taken[b], TAKERS / 32); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tcgen05_alloc(tmem_holder, C::TMEM_COLUMNS);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    const int quarter = warp & 3;  // tensor memory lanes [32 * quarter, +32) of the converters and takers
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);

    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------- TMA producer
        if (lane == 0) {
            pdl_trigger();
            auto load_w = [&](int i) {
                uint8_t* at = raw + (i % C::STAGES) * C::RAW_BYTES;
                mbar_expect_tx(&full[i % C::STAGES], C::RAW_BYTES);
                const int k = (kb_begin + i) * SPLIT_K;
                tma_load_2d(at, &map_w, k, w0, &full[i % C::STAGES]);
                tma_load_2d(at + C::W_BYTES / 2, &map_w, k + SPLIT_K / 2, w0, &full[i % C::STAGES]);
            };
            auto load_x = [&](int i) {
                uint8_t* at = raw + (i % C::STAGES) * C::RAW_BYTES + C::W_BYTES;
                const int k = (kb_begin + i) * SPLIT_K;
                tma_load_2d(at, &map_x, k, t0, &full[i % C::STAGES]);
                tma_load_2d(at + C::X_BYTES / 2, &map_x, k + SPLIT_K / 2, t0, &full[i % C::STAGES]);
            };
            const int early = min(blocks, C::STAGES);  // weights are written by no kernel: ahead of the wait
            for (int i = 0; i < early; ++i) load_w(i);
            pdl_wait();
            for (int i = 0; i < early; ++i) load_x(i);
            int issued = early;
            for (int i = early; i < blocks; ++i, ++issued) {
                if (!mbar_wait(&empty[i % C::STAGES], ((i / C::STAGES) & 1) ^ 1)) { atomicCAS(&g_split_error, 0, (1 << 8)); break; }
                load_w(i);
                load_x(i);
            }
            // Copies in flight must land before the shared memory is released; on the normal path the converters saw them.
            if (issued < blocks || g_split_error != 0) {
                for (int i = max(issued - C::STAGES, 0); i < issued; ++i) mbar_wait(&full[i % C::STAGES], (i / C::STAGES) & 1);
            }
        }
    } else if (warp == 1) {
        // --------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            constexpr uint32_t one = make_idesc(NT), two = make_idesc(2 * NT);
            const uint32_t small = tmem_base + C::SMALL_COLUMN;
            for (int i = 0, at = 0; i < blocks; ++i) {
                bool go = mbar_wait(&ready[i & 1], (i >> 1) & 1);
                if (i >= 2) go = go && mbar_wait(&taken[i & 1], ((i >> 1) & 1) ^ 1);
                if (i > 0 && at == 0) go = go && mbar_wait(&taken[(i - 1) & 1], ((i - 1) >> 1) & 1);  // the small terms too
                if (!go) { atomicCAS(&g_split_error, 0, (2 << 8)); break; }
                tcgen05_fence_after();
                const uint32_t a = tmem_base + C::A_COLUMN + (i & 1) * C::A_COLUMNS, main_sum = tmem_base + (i & 1) * NT;
                const uint64_t x0 = smem_desc_sw128(smem_u32(pieces + (i & 1) * C::PIECES_BYTES));
                const uint64_t x1 = x0 + ((NT * 128) >> 4);
                // one kind of product after the other: MMAs into the same columns follow each other without a gap
                const uint32_t w1 = a + SPLIT_K / 2, w2 = w1 + SPLIT_K / 2;
                constexpr int STEPS = SPLIT_K / 16;  // 8 columns of the weights' pieces, 32 bytes of the tokens'
#pragma unroll
                for (int k = 0; k < STEPS; ++k) tcgen05_mma_bf16_ts(small, a + 8 * k, x1 + 2 * k, two, at > 0 || k > 0);
#pragma unroll
                for (int k = 0; k < STEPS; ++k) tcgen05_mma_bf16_ts(small, w1 + 8 * k, x0 + 2 * k, two, 1);
#pragma unroll
                for (int k = 0; k < STEPS; ++k) tcgen05_mma_bf16_ts(small + NT, w2 + 8 * k, x0 + 2 * k, one, 1);
#pragma unroll
                for (int k = 0; k < STEPS; ++k) tcgen05_mma_bf16_ts(main_sum, a + 8 * k, x0 + 2 * k, one, k > 0);
                tcgen05_commit(&done[i & 1]);
                if (++at == p.per_segment) at = 0;  // a new segment starts its own sums
            }
        }
    } else if (warp < 2 + CONVERTERS / 32) {
        // ----------------------------------------------------------------- converters
        const int worker = threadIdx.x - 64, half = worker >> 7;  // which half of a block's k
        const int row = quarter * 32 + lane;
        for (int i = 0; i < blocks; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(&full[i % C::STAGES], (i / C::STAGES) & 1));
            if (!ok) break;
            const uint32_t w_tile = smem_u32(raw + (i % C::STAGES) * C::RAW_BYTES), x_tile = w_tile + C::W_BYTES;
            const uint32_t x_pieces = smem_u32(pieces + (i & 1) * C::PIECES_BYTES);
            // 32 of the row's 64 weights, 16 at a time; TMA put 16-byte chunk c of row r at c ^ (r % 8)
            const uint32_t from = w_tile + half * (C::W_BYTES / 2) + row * 128;
            const uint32_t to = lanes + C::A_COLUMN + (i & 1) * C::A_COLUMNS + half * 16;
#pragma unroll
            for (int run = 0; run < 2; ++run) {
                uint32_t w0[8], w1[8], w2[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = lds128(from + (((4 * run + c) ^ (row & 7)) << 4));
                    const float4 r = make_float4(below_upper(v.x), below_upper(v.y), below_upper(v.z), below_upper(v.w));
                    w0[2 * c] = upper_pair(v.x, v.y), w0[2 * c + 1] = upper_pair(v.z, v.w);
                    w1[2 * c] = upper_pair(r.x, r.y), w1[2 * c + 1] = upper_pair(r.z, r.w);
                    w2[2 * c] = upper_pair(below_upper(r.x), below_upper(r.y));
                    w2[2 * c + 1] = upper_pair(below_upper(r.z), below_upper(r.w));
                }
                if (run == 0 && i >= 2) {  // the MMAs of block i - 2 have read these buffers
                    ok = __all_sync(0xffffffffu, mbar_wait(&done[i & 1], ((i >> 1) & 1) ^ 1));
                    if (!ok) break;
                    tcgen05_fence_after();
                }
                tcgen05_st8(to + 8 * run, w0);
                tcgen05_st8(to + 8 * run + SPLIT_K / 2, w1);
                tcgen05_st8(to + 8 * run + SPLIT_K, w2);
            }
            if (!ok) break;
#pragma unroll
            for (int unit = worker; unit < NT * 8; unit += CONVERTERS) {
                // 8 k values of a token: two raw chunks to one 16-byte chunk of each piece
                const int t = unit >> 3, chunk = unit & 7, side = chunk >> 2;
                const uint32_t x_from = x_tile + side * (C::X_BYTES / 2) + t * 128;
                float4 v[2];
                // the sides take their chunks in opposite order: the eight lanes of a row then meet all banks
                const float4 first = lds128(x_from + (((2 * (chunk & 3) + side) ^ (t & 7)) << 4));
                const float4 second = lds128(x_from + (((2 * (chunk & 3) + (side ^ 1)) ^ (t & 7)) << 4));
                v[0] = side ? second : first;
                v[1] = side ? first : second;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    sts128(x_pieces + q * NT * 128 + t * 128 + ((chunk ^ (t & 7)) << 4),
                           make_uint4(upper_pair(v[0].x, v[0].y), upper_pair(v[0].z, v[0].w), upper_pair(v[1].x, v[1].y),
                                      upper_pair(v[1].z, v[1].w)));
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        v[h] = make_float4(below_upper(v[h].x), below_upper(v[h].y), below_upper(v[h].z), below_upper(v[h].w));
                }
            }
            tcgen05_wait_st();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read shared memory as the async proxy
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&ready[i & 1]);
                mbar_arrive(&empty[i % C::STAGES]);
            }
        }
        if (!ok && lane == 0) atomicCAS(&g_split_error, 0, (3 << 8));
    } else {
        // ------------------------------------------------------------------- takers
        // The sums of a block out of tensor memory and added up; at the end of a segment the small terms join them.
        constexpr int COLUMNS = NT / 2;
        const int row = quarter * 32 + lane, n = n0 + row, column = (warp - 2 - CONVERTERS / 32) / 4 * COLUMNS;
        float sum[COLUMNS], total[COLUMNS];  // of the running segment, of the finished ones
        int at = 0;
        bool first = true;
#pragma unroll
        for (int c = 0; c < COLUMNS; ++c) sum[c] = total[c] = 0.0f;
        for (int i = 0; i < blocks; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(&done[i & 1], (i >> 1) & 1));
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLUMNS; c0 += 8) {
                float got[8];
                tcgen05_ld8(lanes + (i & 1) * NT + column + c0, got);
#pragma unroll
                for (int c = 0; c < 8; ++c) sum[c0 + c] += got[c];
            }
            if (++at == p.per_segment || i + 1 == blocks) {
                at = 0;
#pragma unroll
                for (int c0 = 0; c0 < COLUMNS; c0 += 8) {
                    float low[8], lower[8];
                    tcgen05_ld8(lanes + C::SMALL_COLUMN + column + c0, low);
                    tcgen05_ld8(lanes + C::SMALL_COLUMN + NT + column + c0, lower);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float part = sum[c0 + c] + (low[c] + lower[c]);
                        total[c0 + c] = first ? part : total[c0 + c] + part;
                        sum[c0 + c] = 0.0f;
                    }
                }
                first = false;
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&taken[i & 1]);
        }
        if (!ok && lane == 0) atomicCAS(&g_split_error, 0, (4 << 8));
        pdl_wait();  // the output may still be read by a kernel before this one
        if (p.clustered && ok) {
            // every MMA and load of this CTA has ended: the raw tiles make room for the exchange
            float* exchange = reinterpret_cast<float*>(raw);
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) exchange[(column + c) * SPLIT_ROWS + row] = total[c];
        } else if (ok && n < p.outs) {
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) {
                const int t = t0 + column + c;
                if (t < p.tokens) p.out[static_cast<size_t>(t) * p.outs + n] = finite_or_again(p, t, w0 + row, total[c]);
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) tcgen05_dealloc(tmem_base, C::TMEM_COLUMNS);
    if (p.clustered) {
        cluster_sync();
        if (warp >= 2 && warp < 2 + CONVERTERS / 32 && ok) {
            pdl_wait();
            const int worker = threadIdx.x - 64, row = worker & 127, segments = gridDim.z;
            for (int c = 2 * blockIdx.z + (worker >> 7); c < NT; c += 2 * segments) {
                const int t = t0 + c, n = n0 + row;
                if (t >= p.tokens || n >= p.outs) continue;
                const uint32_t from = smem_u32(raw) + (c * SPLIT_ROWS + row) * 4;
                float part[MAX_SEGMENTS];
#pragma unroll
                for (int s = 0; s < MAX_SEGMENTS; ++s)
                    if (s < segments) part[s] = ld_cluster_f32(from, s);
#pragma unroll
                for (int s = 1; s < MAX_SEGMENTS; ++s)
                    if (s < segments) part[0] += part[s];
                p.out[static_cast<size_t>(t) * p.outs + n] = finite_or_again(p, t, w0 + row, part[0]);
            }
        }
        cluster_sync();  // the others may still read this CTA's part
    }
}

// -------------------------------------------------------------------------------- host

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &status) == cudaSuccess &&
            status == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(entry);
    }
    return fn;
}

// A [rows][inner] float32 matrix, tiles of box_rows x 32 in the 128-byte swizzle; elements outside read as zero.
ME_EXPORT int me_make_tensor_map_f32(void* out, const void* base, unsigned long long rows, unsigned long long inner, unsigned int box_rows) {
    EncodeTiledFn encode = encode_tiled();
    if (!encode) return ME_ERR_UNSUPPORTED;
    if (inner % 4 != 0 || reinterpret_cast<uintptr_t>(base) % 16 != 0 || box_rows > 256) return ME_ERR_ARGUMENT;
    alignas(64) CUtensorMap map;
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {inner * 4};
    const cuuint32_t box[2] = {SPLIT_K / 2, box_rows};
    const cuuint32_t element_strides[2] = {1, 1};
    const CUresult result = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box,
                                   element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (result != CUDA_SUCCESS) return ME_ERR_ARGUMENT;
    memcpy(out, &map, sizeof(map));
    return 0;
}

template <int NT>
static int launch_split(const CUtensorMap& map_w, const CUtensorMap& map_x, const SplitParams& p, int segments, cudaStream_t stream) {
    using C = SplitConfig<NT>;
    auto kernel = gemm_split_kernel<NT>;
    static SharedMemoryOptIn opt_in;
    if (const int e = opt_in(kernel, C::SMEM_BYTES)) return e;
    const dim3 grid((p.tokens + NT - 1) / NT, (p.outs + SPLIT_ROWS - 1) / SPLIT_ROWS, p.clustered ? segments : 1);
    if (grid.y > 65535) return ME_ERR_UNSUPPORTED;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = dim3(SPLIT_THREADS);
    config.dynamicSmemBytes = C::SMEM_BYTES;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    int count = 0;
    if (p.clustered) {
        attributes[count].id = cudaLaunchAttributeClusterDimension;
        attributes[count].val.clusterDim.x = attributes[count].val.clusterDim.y = 1;
        attributes[count++].val.clusterDim.z = segments;
    }
    if (g_programmatic_launch) {
        attributes[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attributes[count++].val.programmaticStreamSerializationAllowed = 1;
    }
    config.attrs = attributes;
    config.numAttrs = count;
    return static_cast<int>(cudaLaunchKernelEx(&config, kernel, map_w, map_x, p));
}

// out[t][n] = sum_k x[t][k] * w[n][k]; `segments` ranges of k blocks whose sums are added in ascending order, in one
// CTA or (`clustered`) in a cluster's CTAs.  With `group_of_block` a grouped product: `tile` rows of x to a group.  `map_x` has boxes of `tile` (16 or 64) rows.
ME_EXPORT int me_gemm_split(const void* map_w, const void* map_x, const float* x, const float* w, float* out, int tokens, int outs,
                            int inner, int tile, int segments, int clustered, const int* group_of_block, int group_rows, cudaStream_t stream) {
    if (tokens <= 0 || outs <= 0) return 0;
    if (group_of_block != nullptr && (group_rows < outs || tokens % tile)) return ME_ERR_ARGUMENT;
    if (inner <= 0 || inner % 4 != 0 || segments < 1 || segments > MAX_SEGMENTS) return ME_ERR_ARGUMENT;
    SplitParams p = {};
    p.x = x, p.w = w, p.out = out;
    p.tokens = tokens, p.outs = outs, p.inner = inner;
    p.k_blocks = (inner + SPLIT_K - 1) / SPLIT_K;
    p.per_segment = (p.k_blocks + segments - 1) / segments;
    p.clustered = clustered && segments > 1;
    p.group_of_block = group_of_block, p.group_rows = group_rows;
    if ((segments - 1) * p.per_segment >= p.k_blocks) return ME_ERR_ARGUMENT;  // a segment would be empty
    alignas(64) CUtensorMap w_map, x_map;
    memcpy(&w_map, map_w, sizeof(w_map));
    memcpy(&x_map, map_x, sizeof(x_map));
    if (tile == 16) return launch_split<16>(w_map, x_map, p, segments, stream);
    if (tile == 64) return launch_split<64>(w_map, x_map, p, segments, stream);
    return ME_ERR_ARGUMENT;
}

ME_EXPORT int me_gemm_split_take_error(int* code) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_split_error, sizeof(int));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (*code != 0) e = cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int));
    return static_cast<int>(e);
}
