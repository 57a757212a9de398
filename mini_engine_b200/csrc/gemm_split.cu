// y[t][n] = sum_k x[t][k] * w[n][k] in float32 on the 5th-generation tensor cores, for the float32 path.
//
// Arithmetic.  A float32 operand of 2^-110 and more (or zero) is the exact sum of three bfloat16 values: the operand rounded to
// nearest, what is left rounded to nearest, and what is left then (8 + 8 + 8 bits and two signs).  A piece is at most 2^-8,
// the third 2^-17 of the operand.  Of the nine products of the pieces the six largest are formed (tcgen05.mma multiplies
// bfloat16 exactly and adds in float32):
//   w0 x0  |  w0 x1 + w1 x0  |  w0 x2 + w1 x1 + w2 x0
// The three dropped ones are together at most 2^-24 of a product, of either sign (0.09 x 2^-24 in the mean square over all
// mantissas; pieces that are cut instead of rounded have the operand's sign and drop up to 2^-21).  Weights, activations and
// sums are 32-bit in memory; the weights' pieces exist in tensor memory only, the tokens' ones (all three, so every bit of a token) in
// shared memory or a scratch buffer.  The tensor core truncates when it adds, so its
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
// the narrow B operand.  Warp 0 loads raw float32 tiles with TMA, warp 1 issues the MMAs, converter warps make the pieces of the
// weights (a thread's row goes to tensor memory, where A is read from), taker warps add the sums of a block up while the MMAs of the
// next run.  The tokens' pieces are three stacked bfloat16 tiles in shared memory, so that one MMA multiplies a piece of the weights
// by several pieces of the tokens.  With 16 tokens to a CTA the converters make them too; with 64 and 128 a kernel before this one makes
// them once for all feature tiles (split_rows_kernel) and they arrive by TMA.  Which form a product takes is the caller's choice.
//
// What bounds it: the issuing thread.  Alone, the MMAs of a k block take 768 cycles with 64 tokens and 1,536 with 128.  A look at a barrier takes
// the thread 198 cycles, also when the barrier has long completed, and only the MMAs issued before run meanwhile (`kernel_bench mma-rate`, an
// idle SM: four MMAs of 16 or 64 columns 36 and 128 cycles, with a look behind them 198 either way, of 128 columns 256 with and without).
// A block takes 1,380 cycles with 64 tokens, 2,390 with 128, and 2,830 in both CTAs of an SM with 16 (what each of 64 blocks more takes, with a
// CTA or two on every SM, at 1,965 MHz).  So the thread looks once a unit, at one barrier that takes the arrivals of converters, takers and TMA
// together, and the widest MMAs come last.  Two groups of eight converter warps work on alternate units: one group (with the tokens to convert as
// well) took 2,000 to 2,700 cycles a block from the arrival of a tile to its last piece (clock stamps in a copy).  us of a product (plain stream order, behind a flushed L2; one group of
// converters and waits of their own | this form; of the 64-token and wider ones 5 are split_rows_kernel and its launch): 256 x 24,576 x 4,096 320 | 260
// (198 TFLOP/s), 256 x 4,096 x 12,288 199 | 149, 512 x 2,048 x 6,144 115 | 78, 512 x 2,048 x 2,048 46 | 33, 1,024 sorted rows in 8 groups x 6,144 x 2,048
// 259 | 185, 64 x 2,048 x 9,216 55 | 41, 8 x 24,576 x 4,096 92 | 81 (5.0 TB/s of weights), 8 x 2,048 x 2,048 13.7 | 11.2.
#include "tcgen05.cuh"

constexpr int SPLIT_ROWS = 128;  // output features per CTA
constexpr int SPLIT_K = 64;      // k per block: two 128-byte rows of float32, one of bfloat16
constexpr int CONVERTERS = 256;  // threads of a group of converters: two warps per quarter of tensor memory's lanes
constexpr int MAX_SEGMENTS = 8;
constexpr int RING = 4;          // barriers of units in flight

__device__ int g_split_error = 0;  // 0 ok; else (role << 8) | detail of the first failure seen

// NT: tokens per CTA.  The tiles pass through the roles in units, whole k blocks or (128 tokens, for which tensor memory has
// no room otherwise) halves of 32 k; the weights' pieces have two buffers, so that the converters write one while the MMAs read the other.
// PRE: the tokens' pieces were made by split_rows_kernel and arrive by TMA, a block at a time; with 16 tokens the raw tokens arrive with
// the raw weights and the converters make their pieces too.
template <int NT>
struct SplitConfig {
    static constexpr bool PRE = NT > 16;
    static constexpr int GROUPS = NT <= 16 ? 1 : 2;  // of converters: unit u is group u % GROUPS's
    static constexpr int TAKERS = NT <= 16 ? 128 : 256, COLUMNS = NT * 128 / TAKERS;  // threads; columns of one
    static constexpr int FIRST_CONVERTER = GROUPS == 2 ? 4 : 2, FIRST_TAKER = FIRST_CONVERTER + GROUPS * CONVERTERS / 32;  // warps
    static constexpr int THREADS = FIRST_TAKER * 32 + TAKERS, CTAS = NT <= 16 ? 2 : 1;
    // Registers of a thread at launch (the most that so many threads leave, what launch_split checks) and in the roles of two groups: the
    // shares are what the launch has, since more than that would be waited for in vain.
    static constexpr int LAUNCH_REGISTERS = 65536 / (THREADS * CTAS) / 8 * 8, HELPER_REGISTERS = 56, TAKER_REGISTERS = 112;
    static_assert(GROUPS == 1 || (THREADS - TAKERS) * HELPER_REGISTERS + TAKERS * TAKER_REGISTERS <= THREADS * LAUNCH_REGISTERS, "register shares");
    static constexpr int UNITS = NT >= 128 ? 2 : 1, UNIT_K = SPLIT_K / UNITS;  // units to a block
    static constexpr int BOXES = UNIT_K / 32;                                  // a TMA box of float32 is 32 k wide
    static constexpr int W_BYTES = SPLIT_ROWS * UNIT_K * 4, X_BYTES = PRE ? 0 : NT * UNIT_K * 4, RAW_BYTES = W_BYTES + X_BYTES;  // of a unit
    static constexpr int PIECES_BYTES = 3 * NT * SPLIT_K * 2;  // of a block's tokens
    static constexpr int X_BUFFERS = NT == 64 ? 3 : 2;  // blocks of them
    static constexpr int STAGES = NT <= 16 ? 2 : NT <= 64 ? 4 : 8;
    // tensor memory: w0 x0 of one or two blocks, the 2^-8 and the 2^-16 terms, the weights' pieces of two units
    static constexpr int MAINS = UNITS == 1 ? 2 : 1;
    static constexpr int SMALL_COLUMN = MAINS * NT, A_COLUMN = SMALL_COLUMN + 2 * NT, A_PIECE = UNIT_K / 2, A_COLUMNS = 3 * A_PIECE;
    static constexpr int TMEM_COLUMNS = A_COLUMN + 2 * A_COLUMNS <= 256 ? 256 : 512;
    static constexpr int SMEM_BYTES = STAGES * RAW_BYTES + X_BUFFERS * PIECES_BYTES + 1024 + 384;
    static_assert((2 * STAGES + 2 * RING + MAINS + 1) * 8 + (2 + THREADS / 32) * 4 <= 384, "barriers, what the roles leave behind");
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
__device__ __forceinline__ float2 without(float2 v, uint32_t pair) {  // both at once; exact, as a piece is a part of its value
    const float2 piece = make_float2(__uint_as_float(pair << 16), __uint_as_float(pair & 0xffff0000u)), minus = make_float2(-1.0f, -1.0f);
    float2 rest;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(rest))
        : "l"(reinterpret_cast<const unsigned long long&>(piece)), "l"(reinterpret_cast<const unsigned long long&>(minus)),
          "l"(reinterpret_cast<const unsigned long long&>(v)));
    return rest;
}
__device__ __forceinline__ float4 without(float4 v, uint32_t xy, uint32_t zw) {
    const float2 a = without(make_float2(v.x, v.y), xy), b = without(make_float2(v.z, v.w), zw);
    return make_float4(a.x, a.y, b.x, b.y);
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
__device__ __forceinline__ float plain_sum(const float* x, const float* w, int inner) {
    float sum = 0.0f;
#pragma unroll 1
    for (int k = 0; k < inner; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        sum = fmaf(a.x, b.x, sum);
        sum = fmaf(a.y, b.y, sum);
        sum = fmaf(a.z, b.z, sum);
        sum = fmaf(a.w, b.w, sum);
    }
    return sum;
}
__device__ __forceinline__ bool sound(float v) { return fabsf(v) <= 3.402823466e38f && (fabsf(v) >= 0x1p-90f || v == 0.0f); }
__device__ __forceinline__ void form_again(const SplitParams& p, int t, int w_row, int n) {
    p.out[static_cast<size_t>(t) * p.outs + n] = plain_sum(p.x + static_cast<size_t>(t) * p.inner, p.w + static_cast<size_t>(w_row) * p.inner, p.inner);
}
// What the threads of four warps hold at most from now on; the roles' shares stand in SplitConfig.
template <int REGISTERS>
__device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGISTERS)); }
template <int REGISTERS>
__device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGISTERS)); }

// The three pieces of four values, each as two pairs.
__device__ __forceinline__ void pieces_of(float4 v, uint32_t* p0, uint32_t* p1, uint32_t* p2) {
    p0[0] = rounded_pair(v.x, v.y), p0[1] = rounded_pair(v.z, v.w);
    const float4 r = without(v, p0[0], p0[1]);
    p1[0] = rounded_pair(r.x, r.y), p1[1] = rounded_pair(r.z, r.w);
    const float4 rest = without(r, p1[0], p1[1]);
    p2[0] = upper_pair(rest.x, rest.y), p2[1] = upper_pair(rest.z, rest.w);
}

// Where a warp meets ahead of each instruction that is warp-wide (.aligned), since lanes go apart at every wait and every arrival of lane 0:
//   tcgen05.alloc           the branch before it is another warp's (thread 0 is in warp 0)
//   setmaxnreg, at roles    __syncthreads behind alloc, then branches on the warp's number alone; at the end __syncthreads again
//   tcgen05.st              __all_sync of the wait for the raw tile, and of the wait for the unit that read these columns before
//   tcgen05.wait::st        nothing divides lanes between the stores and it: the loop over tokens has as many turns in every lane of a warp
//   tcgen05.ld, wait::ld    __all_sync of the wait for the block, and at the end of a segment of the wait for its last unit
//   tcgen05.dealloc         __syncthreads and the __syncwarp behind the producer's last waits
//   barrier.cluster         __syncwarp in cluster_sync
// An elected thread's role ends in the branch of its own warp; arrivals on barriers, loads, MMAs and commits are single threads' instructions.
//
// WITHHELD: no weights are ever loaded (the tokens' pieces are) and waits end after a few polls, so that a test can take the way of a kernel
// that gives up, with copies in flight where pieces are made ahead.
template <int NT, bool WITHHELD = false>
__global__ void __launch_bounds__(SplitConfig<NT>::THREADS, SplitConfig<NT>::CTAS)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, SplitParams p) {
    using C = SplitConfig<NT>;
    constexpr bool PRE = C::PRE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* pieces = raw + C::STAGES * C::RAW_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(pieces + C::X_BUFFERS * C::PIECES_BYTES);  // raw tiles arrived
    uint64_t* empty = full + C::STAGES;   // raw tiles read by the converters
    uint64_t* ready = empty + C::STAGES;  // [RING] all that a unit's MMAs need is there
    uint64_t* done = ready + RING;        // [RING] its MMAs retired
    uint64_t* mains = done + RING;        // [MAINS] a block's w0 x0 complete
    uint64_t* taken = mains + C::MAINS;   // a segment's small terms out of tensor memory
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(taken + 1);
    int* gave_up = reinterpret_cast<int*>(tmem_holder + 1);  // whether some role did
    int* reached = gave_up + 1;                              // [warps] PRE: the unit or block at which a converter or taker ended

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
        *gave_up = 0;
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], CONVERTERS / 32); }
        // The issuer waits once a unit: a look holds it for 198 cycles, which only the last MMAs before it cover.  So a unit's
        // barrier also takes the arrivals of the tokens' pieces and of the takers who have emptied the sums that it overwrites:
        // in the first unit of a block if that is a unit of its own (barriers 0 and 2 of four if a block has two units).
        for (int b = 0; b < RING; ++b) {
            const bool opens = b % C::UNITS == 0;
            mbar_init(&ready[b], CONVERTERS / 32 + (opens ? C::TAKERS / 32 + (PRE ? 1 : 0) : 0));
            mbar_init(&done[b], 1);
        }
        for (int b = 0; b < C::MAINS; ++b) mbar_init(&mains[b], 1);
        mbar_init(taken, C::TAKERS / 32);
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
    int x_issued = 0;  // of the producer: blocks whose pieces it has asked for
    auto give_up = [&](int role) {
        atomicCAS(&g_split_error, 0, role << 8);
        *gave_up = 1;
    };
    auto wait = [](uint64_t* bar, uint32_t parity) { return WITHHELD ? mbar_wait(bar, parity, 512) : mbar_wait(bar, parity); };

    if (C::GROUPS == 2 && warp < C::FIRST_CONVERTER) registers_down<C::HELPER_REGISTERS>();
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
            auto load_x = [&](int u) {  // raw tokens
                if (WITHHELD) return;
                for (int box = 0; box < C::BOXES; ++box)
                    tma_load_2d(raw + (u % C::STAGES) * C::RAW_BYTES + C::W_BYTES + box * NT * 128, &map_x, kb_begin * SPLIT_K + u * C::UNIT_K + 32 * box, t0,
                                &full[u % C::STAGES]);
            };
            auto load_pieces = [&](int b) {
                uint64_t* bar = &ready[b * C::UNITS % RING];
                mbar_expect_tx(bar, C::PIECES_BYTES);
                for (int q = 0; q < 3; ++q)
                    tma_load_2d(pieces + b % C::X_BUFFERS * C::PIECES_BYTES + q * NT * 128, &map_x, (kb_begin + b) * SPLIT_K, q * p.tokens + t0, bar);
            };
            const int early = min(units, C::STAGES);  // weights are written by no kernel: ahead of the wait
            for (int u = 0; u < early; ++u) load_w(u);
            pdl_wait();
            int issued = early;
            bool go = true;
            if constexpr (PRE) {
                for (; x_issued < min(blocks, C::X_BUFFERS); ++x_issued) load_pieces(x_issued);
                // A block's pieces take the place of the block X_BUFFERS before, whose last unit must be done.  Weights go first: their
                // room comes free with a unit's conversion, ahead of its MMAs.  A unit is converted at most two units ahead of
                // them, so whenever this thread waits for room for weights, all pieces that the MMAs need until then are on their way.
                auto room_for_pieces = [&]() { return (x_issued - C::X_BUFFERS + 1) * C::UNITS - 1; };  // the unit that gives it
                for (int u = early; u < units || x_issued < blocks;) {
                    if (u < units) {
                        if (!wait(&empty[u % C::STAGES], ((u / C::STAGES) & 1) ^ 1)) { go = false; break; }
                        load_w(u);
                        issued = ++u;
                    } else {
                        const int last = room_for_pieces();
                        if (!wait(&done[last % RING], (last / RING) & 1)) { go = false; break; }
                    }
                    while (x_issued < blocks) {
                        const int last = room_for_pieces();
                        if (!mbar_try_wait(&done[last % RING], (last / RING) & 1)) break;
                        load_pieces(x_issued);
                        ++x_issued;
                    }
                }
            } else {
                for (int u = 0; u < early; ++u) load_x(u);
                for (int u = early; u < units; ++u, ++issued) {
                    if (!wait(&empty[u % C::STAGES], ((u / C::STAGES) & 1) ^ 1)) { go = false; break; }
                    load_w(u);
                    load_x(u);
                }
            }
            if (!go) give_up(1);
            // Copies in flight must land before the shared memory is released, also when another role has given up (pieces: behind the join).
            for (int u = max(issued - C::STAGES, 0); u < issued; ++u) wait(&full[u % C::STAGES], (u / C::STAGES) & 1);
        }
    } else if (warp == 1) {
        // --------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t one = make_idesc(NT), two = make_idesc(2 * NT);
            constexpr uint64_t PIECE = (NT * 128) >> 4;  // from a piece of the tokens to the next, in descriptor units
            const uint32_t small = tmem_base + C::SMALL_COLUMN;
            const uint64_t x_pieces = smem_desc_sw128(smem_u32(pieces));
            int sent = 0;  // units whose MMAs were issued
            for (int u = 0, at = 0, segment = 0; u < units; ++u) {
                const int half = u % C::UNITS, block = u / C::UNITS;
                const bool fresh = half == 0 && at == 0;  // a segment starts its own small terms
                if (!wait(&ready[u % RING], (u / RING) & 1)) { give_up(2); break; }
                tcgen05_fence_after();
                const uint32_t a = tmem_base + C::A_COLUMN + (u & 1) * C::A_COLUMNS, main_sum = tmem_base + block % C::MAINS * NT;
                const uint64_t b = x_pieces + block % C::X_BUFFERS * (C::PIECES_BYTES >> 4) + 4 * half;
                // A step of 16 k is 8 columns of the weights' pieces and 32 bytes of the tokens'.  The block's own sums come first, so
                // that the takers have them while the small terms run; MMAs of both small sums come last: while the last of them run
                // the wait for the next unit passes.  MMAs into the same columns follow each other without a gap.
#pragma unroll
                for (int k = 0; k < C::UNIT_K / 16; ++k) tcgen05_mma_bf16_ts(main_sum, a + 8 * k, b + 2 * k, one, half > 0 || k > 0);
                if (half == C::UNITS - 1) tcgen05_commit(&mains[block % C::MAINS]);
                bool go = true;
                if (fresh && segment > 0) {
                    go = wait(taken, (segment & 1) ^ 1);
                    tcgen05_fence_after();
                }
                if (go) {
#pragma unroll
                    for (int k = 0; k < C::UNIT_K / 16; k += 2) {  // 32 k after 32 k: the order is the same in every form
                        tcgen05_mma_bf16_ts(small, a + C::A_PIECE + 8 * k, b + 2 * k, two, !fresh || k > 0);
                        tcgen05_mma_bf16_ts(small, a + C::A_PIECE + 8 * k + 8, b + 2 * k + 2, two, 1);
                        tcgen05_mma_bf16_ts(small + NT, a + 2 * C::A_PIECE + 8 * k, b + 2 * k, one, 1);
                        tcgen05_mma_bf16_ts(small + NT, a + 2 * C::A_PIECE + 8 * k + 8, b + 2 * k + 2, one, 1);
                        tcgen05_mma_bf16_ts(small, a + 8 * k, b + PIECE + 2 * k, two, 1);
                        tcgen05_mma_bf16_ts(small, a + 8 * k + 8, b + PIECE + 2 * k + 2, two, 1);
                    }
                }
                tcgen05_commit(&done[u % RING]);
                ++sent;
                if (!go) { give_up(2); break; }
                if (half == C::UNITS - 1 && ++at == p.per_segment) at = 0, ++segment;
            }
            // MMAs in flight read shared memory and write tensor memory: they end before either is given back.
            for (int u = max(sent - RING, 0); u < sent; ++u) wait(&done[u % RING], (u / RING) & 1);
        }
    } else if (warp < C::FIRST_CONVERTER) {
        // warps that fill the first group of four up
    } else if (warp < C::FIRST_TAKER) {
        // ----------------------------------------------------------------- converters
        // A thread takes 16 or 32 weights of a row.
        if constexpr (C::GROUPS == 2) registers_down<C::HELPER_REGISTERS>();
        const int group = (warp - C::FIRST_CONVERTER) / (CONVERTERS / 32);
        const int worker = threadIdx.x - C::FIRST_CONVERTER * 32 - group * CONVERTERS, run = worker >> 7;
        const int row = quarter * 32 + lane;
        int u = group;
        for (; u < units; u += C::GROUPS) {
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
                for (int c = 0; c < 4; ++c)
                    pieces_of(lds128(from_row + (((first_chunk + c) ^ (row & 7)) << 4)), piece0 + 2 * c, piece1 + 2 * c, piece2 + 2 * c);
                if (part == 0 && u >= 2) {  // the MMAs of two units ago have read these buffers
                    ok = __all_sync(0xffffffffu, wait(&done[(u - 2) % RING], ((u - 2) / RING) & 1));
                    if (!ok) break;
                    tcgen05_fence_after();
                }
                tcgen05_st8(to + 8 * part, piece0);
                tcgen05_st8(to + 8 * part + C::A_PIECE, piece1);
                tcgen05_st8(to + 8 * part + 2 * C::A_PIECE, piece2);
            }
            if (!ok) break;
            if constexpr (!PRE) {
                const uint32_t x_pieces = smem_u32(pieces + u % C::X_BUFFERS * C::PIECES_BYTES);
#pragma unroll
                for (int item = worker; item < NT * C::UNIT_K / 8; item += CONVERTERS) {
                    // 8 k values of a token: two raw chunks to one 16-byte chunk of each piece.  Eight lanes are four chunks of tokens t
                    // and t + 4, whose pieces fall into different banks; so do their raw chunks, read in opposite order.
                    const int box = item / (NT * 4), chunk = item & 3, upper = (item >> 2) & 1, t = ((item >> 3) & 3) + 4 * upper + 8 * (item % (NT * 4) >> 5);
                    const uint32_t from = x_tile + box * NT * 128 + t * 128;
                    const float4 one = lds128(from + (((2 * chunk + upper) ^ (t & 7)) << 4));
                    const float4 other = lds128(from + (((2 * chunk + (upper ^ 1)) ^ (t & 7)) << 4));
                    uint32_t out[3][4];
                    pieces_of(upper ? other : one, out[0], out[1], out[2]);
                    pieces_of(upper ? one : other, out[0] + 2, out[1] + 2, out[2] + 2);
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        sts128(x_pieces + q * NT * 128 + t * 128 + (((4 * box + chunk) ^ (t & 7)) << 4), make_uint4(out[q][0], out[q][1], out[q][2], out[q][3]));
                }
            }
            tcgen05_wait_st();
            if (!PRE) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read shared memory as the async proxy
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&ready[u % RING]);
                mbar_arrive(&empty[u % C::STAGES]);
            }
        }
        if (!ok && lane == 0) give_up(3);
        if (PRE && lane == 0) reached[warp] = u;
    } else {
        // ------------------------------------------------------------------- takers
        // The sums of a block out of tensor memory and added up; at the end of a segment the small terms join them.
        if constexpr (C::GROUPS == 2) registers_up<C::TAKER_REGISTERS>();
        constexpr int COLUMNS = C::COLUMNS;
        const int row = quarter * 32 + lane, n = n0 + row, column = (warp - C::FIRST_TAKER) / 4 * COLUMNS;
        // With 128 tokens a thread's registers hold one sum per column: its CTA runs one segment (see me_gemm_split).
        constexpr bool MANY = NT < 128;
        float sum[COLUMNS], total[MANY ? COLUMNS : 1] = {};  // of the running segment, of the finished ones
        int at = 0, segment = 0;
#pragma unroll
        for (int c = 0; c < COLUMNS; ++c) sum[c] = 0.0f;
        if (lane == 0)
            for (int b = 0; b < C::MAINS; ++b) mbar_arrive(&ready[b * C::UNITS]);  // nothing lies in tensor memory yet
        int taken_blocks = 0;
        for (int i = 0; i < blocks; ++i) {
            ok = __all_sync(0xffffffffu, wait(&mains[i % C::MAINS], (i / C::MAINS) & 1));
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLUMNS; c0 += 16) {
                float got[16];
                tcgen05_ld16(lanes + i % C::MAINS * NT + column + c0, got);
#pragma unroll
                for (int c = 0; c < 16; ++c) sum[c0 + c] += got[c];
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[(i + C::MAINS) * C::UNITS % RING]);  // for the block that takes this one's columns
            ++taken_blocks;
            if (++at == p.per_segment || i + 1 == blocks) {
                at = 0;
                const int u = i * C::UNITS + C::UNITS - 1;  // the block's last unit
                ok = __all_sync(0xffffffffu, wait(&done[u % RING], (u / RING) & 1));
                if (!ok) break;
                tcgen05_fence_after();
#pragma unroll
                for (int c0 = 0; c0 < COLUMNS; c0 += 8) {
                    float low[8], lower[8];
                    tcgen05_ld8(lanes + C::SMALL_COLUMN + column + c0, low);
                    tcgen05_ld8(lanes + C::SMALL_COLUMN + NT + column + c0, lower);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float part = sum[c0 + c] + (low[c] + lower[c]);
                        if constexpr (MANY) {
                            total[c0 + c] = segment == 0 ? part : total[c0 + c] + part;
                            sum[c0 + c] = 0.0f;
                        } else {
                            sum[c0 + c] = part;
                        }
                    }
                }
                ++segment;
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(taken);
            }
        }
        auto result = [&](int c) { return MANY ? total[MANY ? c : 0] : sum[c]; };
        if (!ok && lane == 0) give_up(4);
        if (PRE && lane == 0) reached[warp] = taken_blocks;
        pdl_wait();  // the output may still be read by a kernel before this one
        if (p.clustered && ok) {
            // every MMA and load of this CTA has ended: the raw tiles make room for the exchange
            float* exchange = reinterpret_cast<float*>(raw);
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) exchange[(column + c) * SPLIT_ROWS + row] = result(c);
        } else if (ok && n < p.outs) {
            unsigned long long odd = 0;  // columns to be formed again
#pragma unroll
            for (int c = 0; c < COLUMNS; ++c) {
                const int t = t0 + column + c;
                if (t < p.tokens) {
                    p.out[static_cast<size_t>(t) * p.outs + n] = result(c);
                    if (!sound(result(c))) odd |= 1ull << c;
                }
            }
#pragma unroll 1
            for (; odd != 0; odd &= odd - 1) form_again(p, t0 + column + __ffsll(odd) - 1, w0 + row, n);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    // What follows is every warp's code, so it must not name a register that the smallest share lacks.  All come back to what they were
    // launched with: the takers give first, behind the barrier above, so nobody waits for registers that do not come.
    if constexpr (C::GROUPS == 2) {
        if (warp >= C::FIRST_TAKER) registers_down<C::LAUNCH_REGISTERS>();
        else registers_up<C::LAUNCH_REGISTERS>();
    }
    if (PRE && warp == 0 && *gave_up && x_issued > 0) {
        // Some role gave up, so pieces may still be on their way behind barriers that also wait for arrivals which never come.  Behind the
        // join nobody else arrives any more: this thread (the producer; the others have asked for none) makes up what is missing, after which a barrier
        // completes when its bytes have landed.
        for (int b = max(x_issued - C::X_BUFFERS, 0); b < x_issued; ++b) {
            const int u = b * C::UNITS;
            uint64_t* bar = &ready[u % RING];
            if (mbar_try_wait(bar, (u / RING) & 1)) continue;
            for (int w = 0; w < CONVERTERS / 32; ++w)
                if (reached[C::FIRST_CONVERTER + u % C::GROUPS * (CONVERTERS / 32) + w] <= u) mbar_arrive(bar);
            for (int w = 0; w < C::TAKERS / 32; ++w)
                if (reached[C::FIRST_TAKER + w] <= b - C::MAINS) mbar_arrive(bar);
            if (!mbar_wait(bar, (u / RING) & 1)) atomicExch(&g_split_error, 5 << 8);
        }
    }
    __syncwarp();
    if (warp == 1) tcgen05_dealloc(tmem_base, C::TMEM_COLUMNS);
    if (p.clustered) {
        cluster_sync();
        if (warp >= C::FIRST_CONVERTER && warp < C::FIRST_CONVERTER + CONVERTERS / 32 && ok) {
            pdl_wait();
            // Four rows of a column at a time, shared out among the cluster's CTAs.
            const int segments = gridDim.z;
            for (int item = threadIdx.x - C::FIRST_CONVERTER * 32 + CONVERTERS * blockIdx.z; item < NT * (SPLIT_ROWS / 4); item += CONVERTERS * segments) {
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
                const float v[4] = {y.x, y.y, y.z, y.w};
                float* to = p.out + static_cast<size_t>(t) * p.outs + n;
                if (p.vector_out) {
                    *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (n + i < p.outs) to[i] = v[i];
                }
                unsigned odd = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) odd |= sound(v[i]) ? 0u : 1u << i;
#pragma unroll 1
                for (int i = 0; i < 4 && n + i < p.outs; ++i)
                    if (odd >> i & 1) form_again(p, t, w0 + row + i, n + i);
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

static int make_map(void* out, const void* base, CUtensorMapDataType type, int element, unsigned long long rows, unsigned long long inner,
                    unsigned long long pitch, unsigned int box_rows) {
    EncodeTiledFn encode = encode_tiled();
    if (!encode) return ME_ERR_UNSUPPORTED;
    if (pitch % 16 != 0 || reinterpret_cast<uintptr_t>(base) % 16 != 0 || box_rows > 256) return ME_ERR_ARGUMENT;
    alignas(64) CUtensorMap map;
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {pitch};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / element), box_rows};
    const cuuint32_t element_strides[2] = {1, 1};
    const CUresult result = encode(&map, type, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (result != CUDA_SUCCESS) return ME_ERR_ARGUMENT;
    memcpy(out, &map, sizeof(map));
    return 0;
}

// A [rows][inner] float32 matrix, tiles of box_rows x 32 in the 128-byte swizzle; elements outside read as zero.
ME_EXPORT int me_make_tensor_map_f32(void* out, const void* base, unsigned long long rows, unsigned long long inner, unsigned int box_rows) {
    return make_map(out, base, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, rows, inner, inner * 4, box_rows);
}

// The pieces that split_rows_kernel wrote of `rows` tokens, tiles of box_rows x 64.
ME_EXPORT int me_make_tensor_map_pieces(void* out, const void* base, unsigned long long rows, unsigned long long inner, unsigned int box_rows) {
    return make_map(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 3 * rows, inner, (inner + 7) / 8 * 16, box_rows);
}

// pieces[q][t][k] of x[t][k], rows of the pieces padded to whole 16 bytes.  A thread makes 8 values' pieces; bound by the
// latency of one load and of the launch.
constexpr int ROWS_THREADS = 256;
__global__ void __launch_bounds__(ROWS_THREADS)
split_rows_kernel(const float* __restrict__ x, uint4* __restrict__ pieces, int tokens, int inner) {
    pdl_trigger();
    pdl_wait();
    const int chunks = (inner + 7) / 8;
    const long long total = static_cast<long long>(tokens) * chunks;
    for (long long i = static_cast<long long>(blockIdx.x) * ROWS_THREADS + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * ROWS_THREADS) {
        const long long t = i / chunks;
        const int k = static_cast<int>(i - t * chunks) * 8;
        const float* from = x + t * inner + k;  // inner is a multiple of 4
        const float4 a = *reinterpret_cast<const float4*>(from);
        const float4 b = k + 4 < inner ? *reinterpret_cast<const float4*>(from + 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint32_t out[3][4];
        pieces_of(a, out[0], out[1], out[2]);
        pieces_of(b, out[0] + 2, out[1] + 2, out[2] + 2);
#pragma unroll
        for (int q = 0; q < 3; ++q) pieces[q * total + i] = make_uint4(out[q][0], out[q][1], out[q][2], out[q][3]);
    }
}

static int split_rows(const float* x, void* pieces, int tokens, int inner, cudaStream_t stream) {
    if (reinterpret_cast<uintptr_t>(x) % 16 != 0 || reinterpret_cast<uintptr_t>(pieces) % 16 != 0) return ME_ERR_ARGUMENT;
    const long long total = static_cast<long long>(tokens) * ((inner + 7) / 8);
    const long long wanted = (total + ROWS_THREADS - 1) / ROWS_THREADS;
    const int blocks = static_cast<int>(wanted < 148 * 8 ? wanted : 148 * 8);
    return launch_kernel(split_rows_kernel, dim3(blocks), dim3(ROWS_THREADS), 0, stream, x, static_cast<uint4*>(pieces), tokens, inner);
}

template <int NT, bool WITHHELD = false>
static int launch_split(const CUtensorMap& map_w, const CUtensorMap& map_x, const SplitParams& p, int segments, cudaStream_t stream) {
    using C = SplitConfig<NT>;
    auto kernel = gemm_split_kernel<NT, WITHHELD>;
    static SharedMemoryOptIn opt_in;
    if (const int e = opt_in(kernel, C::SMEM_BYTES)) return e;
    if (C::GROUPS == 2) {  // launched with fewer registers, the takers would wait for a share that does not exist
        static const int registers = [kernel] {
            cudaFuncAttributes of = {};
            return cudaFuncGetAttributes(&of, kernel) == cudaSuccess ? of.numRegs : 0;
        }();
        if (registers != C::LAUNCH_REGISTERS) return ME_ERR_UNSUPPORTED;
    }
    const dim3 grid((p.tokens + NT - 1) / NT, (p.outs + SPLIT_ROWS - 1) / SPLIT_ROWS, p.clustered ? segments : 1);
    if (grid.y > 65535) return ME_ERR_UNSUPPORTED;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = dim3(C::THREADS);
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
// CTA or (`clustered`) in a cluster's CTAs.  With `group_of_block` a grouped product: `tile` rows of x to a group.  `tile` tokens to a CTA: 16
// (`map_x` has boxes of as many rows of x), or 64, or 128 where a CTA runs one segment (one in all, or `clustered`): these come with room for the
// tokens' `pieces` (3 x tokens x inner bfloat16, rows padded to 16 bytes), which are made first, and `map_x` is that of the pieces.
// `withheld`: every wait runs out (for tests).
ME_EXPORT int me_gemm_split(const void* map_w, const void* map_x, const float* x, const float* w, float* out, int tokens, int outs,
                            int inner, int tile, void* pieces, int segments, int clustered, const int* group_of_block, int group_rows, int withheld,
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
    if (pieces != nullptr)
        if (const int e = split_rows(x, pieces, tokens, inner, stream)) return e;
    if (tile == 16 && !pieces) return withheld ? launch_split<16, true>(w_map, x_map, p, segments, stream) : launch_split<16>(w_map, x_map, p, segments, stream);
    if (tile == 64 && pieces) return withheld ? launch_split<64, true>(w_map, x_map, p, segments, stream) : launch_split<64>(w_map, x_map, p, segments, stream);
    if (tile == 128 && pieces && (p.clustered || segments == 1))
        return withheld ? launch_split<128, true>(w_map, x_map, p, segments, stream) : launch_split<128>(w_map, x_map, p, segments, stream);
    return ME_ERR_ARGUMENT;
}

ME_EXPORT int me_gemm_split_take_error(int* code) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_split_error, sizeof(int));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (*code != 0) e = cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int));
    return static_cast<int>(e);
}
