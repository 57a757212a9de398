// y[t][n] = sum_k x[t][k] * w[n][k] in float32 on the 5th-generation tensor cores, for the float32 path.
//
// Arithmetic.  A float32 operand of 2^-110 and more (or zero) is the exact sum of three bfloat16 values: the operand rounded to
// nearest, what is left rounded to nearest, and what is left then (8 + 8 + 8 bits and two signs).  A piece is at most 2^-8,
// the third 2^-17 of the operand.  Of the nine products of the pieces the six largest are formed (tcgen05.mma multiplies
// bfloat16 exactly and adds in float32):
//   w0 x0  |  w0 x1 + w1 x0  |  w0 x2 + w1 x1 + w2 x0
// The three dropped ones are together at most 2^-24 of a product, of either sign (0.09 x 2^-24 in the mean square over all
// mantissas; pieces that are cut instead of rounded have the operand's sign and drop up to 2^-21).  Weights, activations and
// sums are 32-bit in memory: the pieces exist in shared and tensor memory only.  The tensor core truncates when it adds, so its
// chain is kept short: the sum of w0 x0 over 64 k is taken out of tensor memory and added with rounding in registers; the
// small terms (2^-8 and 2^-16 of the products) run over a whole segment of the reduction.  Error against float64 (norm of the
// difference over norm of the result, 64 x 512 outputs) | that of one fmaf chain per output (gemm_simt.cu), by inner size:
//                        64                  2,048               12,288
//   normal operands      6.9e-8 | 1.5e-7     9.9e-8 | 8.1e-7     1.3e-7 | 2.0e-6
//   one sign             9.0e-8 | 1.2e-7     9.3e-8 | 7.0e-7     9.1e-8 | 1.5e-6
//   sums that cancel     4.6e-4 | 1.4e-3     7.3e-4 | 8.2e-3     1.1e-3 | 2.0e-2
//   one operand in ten   3.8e-8 | 4.4e-8     7.3e-8 | 1.8e-7     9.8e-8 | 4.4e-7
//   one operand 1e4 of the others
//                        1.1e-7 | 1.3e-7     1.4e-7 | 8.0e-7     1.6e-7 | 2.0e-6
//   one operand alone    2.6e-8 | 2.6e-8     2.6e-8 | 2.5e-8     2.6e-8 | 2.5e-8 (at most 8.6e-8 | 6.0e-8 of an output)
// Smaller operands lose what falls under 2^-134, so an output below 2^-90 is formed again as below.
//
// An output's sum is formed in an order that depends on (outs, inner) alone: 64-wide k blocks in ascending order
// within a segment, segments in ascending order, whether the segments of a tile run one after the other in a CTA or
// side by side in the CTAs of a cluster.  A row's bits therefore do not depend on what else is in the batch.
// A sum that comes out infinite or NaN (a piece of an infinity is NaN, and that of a value that rounds to one) is formed again
// with fmaf in ascending k.
//
// Orientation and roles follow the bfloat16 product (gemm_tcgen05.cu): 128 weight rows are the A operand, the tokens
// the narrow B operand.  Warp 0 loads raw float32 tiles with TMA, warp 1 issues the MMAs, eight converter warps make the
// pieces (weights: a thread's row goes to tensor memory, where A is read from; tokens: three stacked bfloat16 tiles in
// shared memory, so that one MMA multiplies a piece of the weights by several pieces of the tokens), eight taker warps add
// the sums of a block up while the MMAs of the next run.
//
// What bounds it: a k block takes about 2,000 cycles with 16 or 64 tokens and 2,500 with 128.  The MMAs take 85 to 90 cycles
// each beside the converters, 58 alone (both work on tensor memory and shared memory), the converters 1,050 to 1,100 a block,
// and the waits between the roles come on top.  Beside the CUDA-core kernel (tokens x outs x inner): 256 x 24,576 x 4,096
// 2,378 -> 324 us (159 TFLOP/s), 256 x 4,096 x 12,288 1,714 -> 202, 512 x 2,048 x 5,632 760 -> 107; 8 x 24,576 x 4,096
// 807 -> 94 (4.3 TB/s of weights), 8 x 4,096 x 4,096 377 -> 25, 1 x 151,936 x 1,024 919 -> 112 (5.6 TB/s); these with pieces that were cut.  Rounded ones against cut ones, in turn and
// behind a flushed L2: 256 x 24,576 x 4,096 338 -> 325, 256 x 4,096 x 12,288 215 -> 205, 8 x 24,576 x 4,096 106 -> 102, others the same.
#include "tcgen05.cuh"

constexpr int SPLIT_ROWS = 128;  // output features per CTA
constexpr int SPLIT_K = 64;      // k per block: two 128-byte rows of float32, one of bfloat16
constexpr int CONVERTERS = 256;  // threads: two warps per quarter of tensor memory's lanes
constexpr int TAKERS = 256;      // threads: two warps per quarter
constexpr int SPLIT_THREADS = 64 + CONVERTERS + TAKERS;
constexpr int MAX_SEGMENTS = 8;

__device__ int g_split_error = 0;  // 0 ok; else (role << 8) | detail of the first failure seen

// NT: tokens per CTA.  The tiles pass through the roles in units, whole k blocks or (128 tokens, for which tensor memory has
// no room otherwise) halves of 32 k; two buffers of pieces, so that the converters write one while the MMAs read the other.
template <int NT>
struct SplitConfig {
    static constexpr int UNITS = NT >= 128 ? 2 : 1, UNIT_K = SPLIT_K / UNITS;  // units to a block
    static constexpr int BOXES = UNIT_K / 32;                                  // a TMA box is 32 k wide
    static constexpr int W_BYTES = SPLIT_ROWS * UNIT_K * 4, X_BYTES = NT * UNIT_K * 4, RAW_BYTES = W_BYTES + X_BYTES;  // raw tiles of a unit
    static constexpr int PIECES_BYTES = 3 * NT * SPLIT_K * 2;  // of a block: rows of 128 bytes, of which a half takes 64
    static constexpr int PIECES_BUFFERS = 2 / UNITS;
    // 16 tokens: 36 KB a unit, two CTAs to an SM (one CTA with five units in flight was 30 % slower: a unit's way through the
    // roles is what takes the time); 64 tokens: 48 KB; 128: 32 KB
    static constexpr int STAGES = NT <= 16 ? 2 : NT <= 64 ? 3 : 5;
    // tensor memory: w0 x0 of one or two blocks, the 2^-8 and the 2^-16 terms, the weights' pieces of two units
    static constexpr int MAINS = UNITS == 1 ? 2 : 1;
    static constexpr int SMALL_COLUMN = MAINS * NT, A_COLUMN = SMALL_COLUMN + 2 * NT, A_PIECE = UNIT_K / 2, A_COLUMNS = 3 * A_PIECE;
    static constexpr int TMEM_COLUMNS = A_COLUMN + 2 * A_COLUMNS <= 256 ? 256 : 512;
    static constexpr int SMEM_BYTES = STAGES * RAW_BYTES + PIECES_BUFFERS * PIECES_BYTES + 1024 + 256;
    static_assert(A_COLUMN + 2 * A_COLUMNS <= TMEM_COLUMNS, "tensor memory");
    static_assert(STAGES * RAW_BYTES >= NT * SPLIT_ROWS * 4, "the cluster's exchange reuses the raw tiles");
};

struct SplitParams {
    const float* x;
    const float* w;
    float* out;
    int tokens, outs, inner;
    int k_blocks, per_segment;
    int vector_out;  // rows of the output start on 16 bytes and hold whole float4
    int clustered;  // the segments of a tile are the CTAs of a cluster along z
    // Grouped product: the weight holds `group_rows` rows per group, one group after the other, and token tile b belongs to
    // group group_of_block[b] (negative: it holds no rows and its CTAs return at once).  `outs` counts one group's features.
    const int* group_of_block;
    int group_rows;
};

__device__ __forceinline__ uint32_t upper_pair(float even, float odd) {  // bfloat16 pair, the even k in the low half
    return __byte_perm(__float_as_uint(even), __float_as_uint(odd), 0x7632);
}
__device__ __forceinline__ uint32_t rounded_pair(float even, float odd) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(even, odd);
    return *reinterpret_cast<const uint32_t*>(&pair);
}
// What a pair of pieces leaves of four values.
__device__ __forceinline__ float4 without(float4 v, uint32_t xy, uint32_t zw) {
    return make_float4(v.x - __uint_as_float(xy << 16), v.y - __uint_as_float(xy & 0xffff0000u), v.z - __uint_as_float(zw << 16),
                       v.w - __uint_as_float(zw & 0xffff0000u));
}

__device__ __forceinline__ float4 lds128(uint32_t address) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t address, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t address, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(address), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
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

// The sum of one output again, for one that came out infinite, NaN or so small that pieces may have fallen under the range.
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
__device__ __forceinline__ float sound_or_again(const SplitParams& p, int t, int w_row, float v) {
    if (fabsf(v) <= 3.402823466e38f && (fabsf(v) >= 0x1p-90f || v == 0.0f)) return v;
    return plain_sum(p.x + static_cast<size_t>(t) * p.inner, p.w + static_cast<size_t>(w_row) * p.inner, p.inner);
}

// WITHHELD: no tile is ever loaded and waits end after a few polls, so that a test can take the way of a kernel that gives up.
template <int NT, bool WITHHELD = false>
__global__ void __launch_bounds__(SPLIT_THREADS, NT <= 16 ? 2 : 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, SplitParams p) {
    using C = SplitConfig<NT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* pieces = raw + C::STAGES * C::RAW_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(pieces + C::PIECES_BUFFERS * C::PIECES_BYTES);  // raw tiles arrived
    uint64_t* empty = full + C::STAGES;                                                         // raw tiles read by the converters
    uint64_t* ready = empty + C::STAGES;                                                        // [2] a unit's pieces written
    uint64_t* done = ready + 2;                                                                 // [2] its MMAs retired
    uint64_t* taken = done + 2;                                                                 // [MAINS] a block's sums out of tensor memory
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(taken + C::MAINS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * NT, n0 = blockIdx.y * SPLIT_ROWS;
    const int kb_begin = p.clustered ? blockIdx.z * p.per_segment : 0;
    const int kb_end = p.clustered ? min(kb_begin + p.per_segment, p.k_blocks) : p.k_blocks;
    const int blocks = kb_end - kb_begin, units = C::UNITS * blocks;
    int w0 = n0;  // first weight row of the tile
    if (p.group_of_block != nullptr) {
        pdl_wait();  // a kernel before this one wrote the groups
        const int group = p.group_of_block[blockIdx.x];
        if (group < 0) return;  // every CTA of the tile (and of its cluster): nothing has been set up yet
        w0 = group * p.group_rows + n0;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], CONVERTERS / 32); }
        for (int b = 0; b < 2; ++b) { mbar_init(&ready[b], CONVERTERS / 32); mbar_init(&done[b], 1); }
        for (int b = 0; b < C::MAINS; ++b) mbar_init(&taken[b], TAKERS / 32);
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
    auto wait = [](uint64_t* bar, uint32_t parity) { return WITHHELD ? mbar_wait(bar, parity, 512) : mbar_wait(bar, parity); };

    if (warp == 0) {
        // ------------------------------------------------------------- TMA producer
        if (elect_one()) {
            pdl_trigger();
            auto load_w = [&](int u) {
                if (WITHHELD) return;
                mbar_expect_tx(&full[u % C::STAGES], C::RAW_BYTES);
                for (int box = 0; box < C::BOXES; ++box)
                    tma_load_2d(raw + (u % C::STAGES) * C::RAW_BYTES + box * SPLIT_ROWS * 128, &map_w, kb_begin * SPLIT_K + u * C::UNIT_K + 32 * box, w0,
                                &full[u % C::STAGES]);
            };
            auto load_x = [&](int u) {
                if (WITHHELD) return;
                for (int box = 0; box < C::BOXES; ++box)
                    tma_load_2d(raw + (u % C::STAGES) * C::RAW_BYTES + C::W_BYTES + box * NT * 128, &map_x, kb_begin * SPLIT_K + u * C::UNIT_K + 32 * box, t0,
                                &full[u % C::STAGES]);
            };
            const int early = min(units, C::STAGES);  // weights are written by no kernel: ahead of the wait
            for (int u = 0; u < early; ++u) load_w(u);
            pdl_wait();
            for (int u = 0; u < early; ++u) load_x(u);
            int issued = early;
            for (int u = early; u < units; ++u, ++issued) {
                if (!wait(&empty[u % C::STAGES], ((u / C::STAGES) & 1) ^ 1)) { atomicCAS(&g_split_error, 0, (1 << 8)); break; }
                load_w(u);
                load_x(u);
            }
            // Copies in flight must land before the shared memory is released, also when another role has given up.
            for (int u = max(issued - C::STAGES, 0); u < issued; ++u) wait(&full[u % C::STAGES], (u / C::STAGES) & 1);
        }
    } else if (warp == 1) {
        // --------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t one = make_idesc(NT), two = make_idesc(2 * NT);
            const uint32_t small = tmem_base + C::SMALL_COLUMN;
            int sent = 0;  // units whose MMAs were issued
            auto wait_taken = [&](int block) { return block < 0 || wait(&taken[block % C::MAINS], (block / C::MAINS) & 1); };
            for (int u = 0, at = 0; u < units; ++u) {
                const int half = u % C::UNITS, block = u / C::UNITS;
                const bool fresh = half == 0 && at == 0;  // a segment starts its own sums: the last one's must be out
                if (!wait(&ready[u & 1], (u >> 1) & 1) || (fresh && !wait_taken(block - 1))) { atomicCAS(&g_split_error, 0, (2 << 8)); break; }
                tcgen05_fence_after();
                const uint32_t a = tmem_base + C::A_COLUMN + (u & 1) * C::A_COLUMNS, main_sum = tmem_base + block % C::MAINS * NT;
                const uint64_t b = smem_desc_sw128(smem_u32(pieces + (C::UNITS == 1 ? (u & 1) * C::PIECES_BYTES : 0))) + 4 * half;
                // The small terms of 32 k, then of the next: MMAs into the same columns follow each other without a gap, and the
                // widest come last, so that the next unit's waits pass while they run.  A step of 16 k is 8 columns of the weights'
                // pieces and 32 bytes of the tokens'.
                bool go = true;
#pragma unroll
                for (int box = 0; box < C::BOXES; ++box) {
                    const uint32_t w0_piece = a + 16 * box, w1_piece = w0_piece + C::A_PIECE, w2_piece = w1_piece + C::A_PIECE;
                    const uint64_t x0 = b + 4 * box, x1 = x0 + ((NT * 128) >> 4);
                    tcgen05_mma_bf16_ts(small, w1_piece, x0, two, !fresh || box > 0);
                    tcgen05_mma_bf16_ts(small, w1_piece + 8, x0 + 2, two, 1);
                    tcgen05_mma_bf16_ts(small + NT, w2_piece, x0, one, 1);
                    tcgen05_mma_bf16_ts(small + NT, w2_piece + 8, x0 + 2, one, 1);
                    if (box == C::BOXES - 1) {
                        if (half == 0 && !wait_taken(block - C::MAINS)) { go = false; break; }  // the takers have had their time
                        tcgen05_fence_after();
#pragma unroll
                        for (int k = 0; k < C::UNIT_K / 16; ++k) tcgen05_mma_bf16_ts(main_sum, a + 8 * k, b + 2 * k, one, half > 0 || k > 0);
                    }
                    tcgen05_mma_bf16_ts(small, w0_piece, x1, two, 1);
                    tcgen05_mma_bf16_ts(small, w0_piece + 8, x1 + 2, two, 1);
                }
                tcgen05_commit(&done[u & 1]);
                ++sent;
                if (!go) { atomicCAS(&g_split_error, 0, (2 << 8)); break; }
                if (half == C::UNITS - 1 && ++at == p.per_segment) at = 0;
            }
            // MMAs in flight read shared memory and write tensor memory: they end before either is given back.
            for (int u = max(sent - 2, 0); u < sent; ++u) wait(&done[u & 1], (u >> 1) & 1);
        }
    } else if (warp < 2 + CONVERTERS / 32) {
        // ----------------------------------------------------------------- converters
        // A thread takes 16 or 32 weights of a row.
        const int worker = threadIdx.x - 64, run = worker >> 7;
        const int row = quarter * 32 + lane;
        for (int u = 0; u < units; ++u) {
            ok = __all_sync(0xffffffffu, wait(&full[u % C::STAGES], (u / C::STAGES) & 1));
            if (!ok) break;
            const uint32_t w_tile = smem_u32(raw + (u % C::STAGES) * C::RAW_BYTES), x_tile = w_tile + C::W_BYTES;
            const uint32_t from_row = w_tile + (C::BOXES == 2 ? run * SPLIT_ROWS * 128 : 0) + row * 128;
            const uint32_t to = lanes + C::A_COLUMN + (u & 1) * C::A_COLUMNS + run * (C::UNIT_K / 4);
#pragma unroll
            for (int part = 0; part < C::BOXES; ++part) {  // 16 weights; TMA put 16-byte chunk c of row r at c ^ (r % 8)
                const int first_chunk = 4 * (C::BOXES == 2 ? part : run);
                uint32_t piece0[8], piece1[8], piece2[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = lds128(from_row + (((first_chunk + c) ^ (row & 7)) << 4));
                    piece0[2 * c] = rounded_pair(v.x, v.y), piece0[2 * c + 1] = rounded_pair(v.z, v.w);
                    const float4 r = without(v, piece0[2 * c], piece0[2 * c + 1]);
                    piece1[2 * c] = rounded_pair(r.x, r.y), piece1[2 * c + 1] = rounded_pair(r.z, r.w);
                    const float4 rest = without(r, piece1[2 * c], piece1[2 * c + 1]);
                    piece2[2 * c] = upper_pair(rest.x, rest.y), piece2[2 * c + 1] = upper_pair(rest.z, rest.w);
                }
                if (part == 0 && u >= 2) {  // the MMAs of two units ago have read these buffers
                    ok = __all_sync(0xffffffffu, wait(&done[u & 1], ((u >> 1) & 1) ^ 1));
                    if (!ok) break;
                    tcgen05_fence_after();
                }
                tcgen05_st8(to + 8 * part, piece0);
                tcgen05_st8(to + 8 * part + C::A_PIECE, piece1);
                tcgen05_st8(to + 8 * part + 2 * C::A_PIECE, piece2);
            }
            if (!ok) break;
            const uint32_t x_pieces = smem_u32(pieces + (C::UNITS == 1 ? (u & 1) * C::PIECES_BYTES : 0));
#pragma unroll
            for (int item = worker; item < NT * C::UNIT_K / 8; item += CONVERTERS) {
                // 8 k values of a token: two raw chunks to one 16-byte chunk of each piece.  Eight lanes are four chunks of tokens t
                // and t + 4, whose pieces fall into different banks; so do their raw chunks, read in opposite order.
                const int box = item / (NT * 4), chunk = item & 3, upper = (item >> 2) & 1, t = ((item >> 3) & 3) + 4 * upper + 8 * (item % (NT * 4) >> 5);
                const uint32_t from = x_tile + box * NT * 128 + t * 128;
                const float4 one = lds128(from + (((2 * chunk + upper) ^ (t & 7)) << 4));
                const float4 other = lds128(from + (((2 * chunk + (upper ^ 1)) ^ (t & 7)) << 4));
                float4 v[2];
                v[0] = upper ? other : one;
                v[1] = upper ? one : other;
                const int to_chunk = 4 * (C::UNITS == 1 ? box : u & 1) + chunk;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    uint32_t pair[4];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        pair[2 * h] = q < 2 ? rounded_pair(v[h].x, v[h].y) : upper_pair(v[h].x, v[h].y);
                        pair[2 * h + 1] = q < 2 ? rounded_pair(v[h].z, v[h].w) : upper_pair(v[h].z, v[h].w);
                        v[h] = without(v[h], pair[2 * h], pair[2 * h + 1]);
                    }
                    sts128(x_pieces + q * NT * 128 + t * 128 + ((to_chunk ^ (t & 7)) << 4), make_uint4(pair[0], pair[1], pair[2], pair[3]));
                }
            }
            tcgen05_wait_st();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read shared memory as the async proxy
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&ready[u & 1]);
                mbar_arrive(&empty[u % C::STAGES]);
            }
        }
        if (!ok && lane == 0) atomicCAS(&g_split_error, 0, (3 << 8));
    } else {
        // ------------------------------------------------------------------- takers
        // The sums of a block out of tensor memory and added up; at the end of a segment the small terms join them.
        constexpr int COLUMNS = NT / 2;
        const int row = quarter * 32 + lane, n = n0 + row, column = (warp - 2 - CONVERTERS / 32) / 4 * COLUMNS;
        // With 128 tokens a thread's registers hold one sum per column: its CTA runs one segment (see me_gemm_split).
        constexpr bool MANY = NT < 128;
        float sum[COLUMNS], total[MANY ? COLUMNS : 1] = {};  // of the running segment, of the finished ones
        int at = 0;
        bool first = true;
#pragma unroll
        for (int c = 0; c < COLUMNS; ++c) sum[c] = 0.0f;
        for (int i = 0; i < blocks; ++i) {
            const int u = i * C::UNITS + C::UNITS - 1;  // the block's last unit
            ok = __all_sync(0xffffffffu, wait(&done[u & 1], (u >> 1) & 1));
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLUMNS; c0 += 8) {
                float got[8];
                tcgen05_ld8(lanes + i % C::MAINS * NT + column + c0, got);
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
                        if constexpr (MANY) {
                            total[c0 + c] = first ? part : total[c0 + c] + part;
                            sum[c0 + c] = 0.0f;
                        } else {
                            sum[c0 + c] = part;
                        }
                    }
                }
                first = false;
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&taken[i % C::MAINS]);
        }
        auto result = [&](int c) { return MANY ? total[MANY ? c : 0] : sum[c]; };
        if (!ok && lane == 0) atomicCAS(&g_split_error, 0, (4 << 8));
        pdl_wait();  // the output may still be read by a kernel before this one
        if (p.clustered && ok) {
            // every MMA and load of this CTA has ended: the raw tiles make room for the exchange
            float* exchange = reinterpret_cast<float*>(raw);
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) exchange[(column + c) * SPLIT_ROWS + row] = result(c);
        } else if (ok && n < p.outs) {
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) {
                const int t = t0 + column + c;
                if (t < p.tokens) p.out[static_cast<size_t>(t) * p.outs + n] = sound_or_again(p, t, w0 + row, result(c));
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
            // Four rows of a column at a time, shared out among the cluster's CTAs.
            const int segments = gridDim.z;
            for (int item = threadIdx.x - 64 + CONVERTERS * blockIdx.z; item < NT * (SPLIT_ROWS / 4); item += CONVERTERS * segments) {
                const int c = item / (SPLIT_ROWS / 4), row = item % (SPLIT_ROWS / 4) * 4, t = t0 + c, n = n0 + row;
                if (t >= p.tokens || n >= p.outs) continue;
                const uint32_t from = smem_u32(raw) + (c * SPLIT_ROWS + row) * 4;
                float4 part[MAX_SEGMENTS];
#pragma unroll
                for (int s = 0; s < MAX_SEGMENTS; ++s)
                    if (s < segments) part[s] = ld_cluster_f32x4(from, s);
                float4 y = part[0];
#pragma unroll
                for (int s = 1; s < MAX_SEGMENTS; ++s)
                    if (s < segments) y.x += part[s].x, y.y += part[s].y, y.z += part[s].z, y.w += part[s].w;
                const float v[4] = {sound_or_again(p, t, w0 + row, y.x), n + 1 < p.outs ? sound_or_again(p, t, w0 + row + 1, y.y) : 0.0f,
                                    n + 2 < p.outs ? sound_or_again(p, t, w0 + row + 2, y.z) : 0.0f, n + 3 < p.outs ? sound_or_again(p, t, w0 + row + 3, y.w) : 0.0f};
                float* to = p.out + static_cast<size_t>(t) * p.outs + n;
                if (p.vector_out) {
                    *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (n + i < p.outs) to[i] = v[i];
                }
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

template <int NT, bool WITHHELD = false>
static int launch_split(const CUtensorMap& map_w, const CUtensorMap& map_x, const SplitParams& p, int segments, cudaStream_t stream) {
    using C = SplitConfig<NT>;
    auto kernel = gemm_split_kernel<NT, WITHHELD>;
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
// CTA or (`clustered`) in a cluster's CTAs.  With `group_of_block` a grouped product: `tile` rows of x to a group.  `map_x` has boxes
// of `tile` rows: 16, 64, or 128 where a CTA runs one segment (one in all, or `clustered`).  `withheld`: every wait runs out (for tests).
ME_EXPORT int me_gemm_split(const void* map_w, const void* map_x, const float* x, const float* w, float* out, int tokens, int outs,
                            int inner, int tile, int segments, int clustered, const int* group_of_block, int group_rows, int withheld,
                            cudaStream_t stream) {
    if (tokens <= 0 || outs <= 0) return 0;
    if (group_of_block != nullptr && (group_rows < outs || tokens % tile)) return ME_ERR_ARGUMENT;
    if (inner <= 0 || inner % 4 != 0 || segments < 1 || segments > MAX_SEGMENTS) return ME_ERR_ARGUMENT;
    SplitParams p = {};
    p.x = x, p.w = w, p.out = out;
    p.tokens = tokens, p.outs = outs, p.inner = inner;
    p.k_blocks = (inner + SPLIT_K - 1) / SPLIT_K;
    p.per_segment = (p.k_blocks + segments - 1) / segments;
    p.clustered = clustered && segments > 1;
    p.vector_out = outs % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
    p.group_of_block = group_of_block, p.group_rows = group_rows;
    if ((segments - 1) * p.per_segment >= p.k_blocks) return ME_ERR_ARGUMENT;  // a segment would be empty
    alignas(64) CUtensorMap w_map, x_map;
    memcpy(&w_map, map_w, sizeof(w_map));
    memcpy(&x_map, map_x, sizeof(x_map));
    if (withheld) return tile == 16 ? launch_split<16, true>(w_map, x_map, p, segments, stream) : ME_ERR_ARGUMENT;
    if (tile == 16) return launch_split<16>(w_map, x_map, p, segments, stream);
    if (tile == 64) return launch_split<64>(w_map, x_map, p, segments, stream);
    if (tile == 128 && (p.clustered || segments == 1)) return launch_split<128>(w_map, x_map, p, segments, stream);
    return ME_ERR_ARGUMENT;
}

ME_EXPORT int me_gemm_split_take_error(int* code) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_split_error, sizeof(int));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (*code != 0) e = cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int));
    return static_cast<int>(e);
}
