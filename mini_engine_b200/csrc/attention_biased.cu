// Softmax attention over the paged cache with the options that the plain kernels do not have:
//
//   * value heads of another width than query/key heads;
//   * a window that also keeps the first tokens of the sequence: the query at position p sees key j
//     when j <= p and (p - j < window or j < keep_first); window 0 keeps every key;
//   * a distance bias taken off the score: s = (q . k) * scale - r1[h] * ln(1 + r2[h] * (p - j));
//   * mixing of the heads' weights after the softmax: w'_h = sum_g talk[h][g] * w_g, head h then reads
//     the values of its own KV head with w'_h.
//
// One warp per (token, query head).  Keys are visited in tiles of 32 whose boundaries are multiples of 32
// in absolute position, first the kept tokens that lie behind the window, then the window, so the
// arithmetic of a query depends on its own position only (the same bits however the prompt was cut
// and whatever else is in the batch).
//
// Mixing after the softmax needs every head's normalised weights over all keys.  Instead of keeping them,
// head g's warp applies its weights to the values of EVERY KV head c: A[g][c] = sum_j w_g(j) v_c(j).
// The mixed output of head h is then sum_g talk[h][g] * A[g][kv(h)], which a second small kernel forms.
// The weights themselves are never stored and one pass over the keys suffices.
#include "mma_sync.cuh"

#include <algorithm>
#include <type_traits>

struct BiasedArgs {
    const void* q;           // [tokens][heads][dim]
    const void* k_pages;     // [pages][kv_heads][page_size][dim]
    const void* v_pages;     // [pages][kv_heads][page_size][vdim]
    const int* block_table;  // [entries][table_width]
    const int* entry_of_token;
    const int* positions;
    const float* r1;  // [heads] or null: no distance bias
    const float* r2;
    void* out;        // spread == 1: float32 [tokens][heads][kv_heads][vdim]; else [tokens][heads][vdim] of T
    float scale;
    int tokens, heads, kv_heads, dim, vdim, page_size, table_width, window, keep_first;
    int spread;  // 1: every KV head's values (for mixing); 0: the head's own
};

constexpr int BIASED_WARPS = 4;

template <typename T, int NACC>
__global__ void __launch_bounds__(BIASED_WARPS * 32) biased_attention_kernel(BiasedArgs a) {
    extern __shared__ float q_staged[];  // [BIASED_WARPS][dim]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = static_cast<long long>(blockIdx.x) * BIASED_WARPS + warp;
    if (item >= static_cast<long long>(a.tokens) * a.heads) return;
    const int token = static_cast<int>(item / a.heads), head = static_cast<int>(item % a.heads);
    const int d = a.dim, vd = a.vdim;
    const int vchunks = (vd + 31) / 32;
    pdl_trigger();
    const float r1 = a.r1 ? a.r1[head] : 0.0f, r2 = a.r1 ? a.r2[head] : 0.0f;
    pdl_wait();
    const int own_kv = head / (a.heads / a.kv_heads);
    const int first_value_head = a.spread ? 0 : own_kv;
    const int value_heads = a.spread ? a.kv_heads : 1;
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const T* k_pages = static_cast<const T*>(a.k_pages);
    const T* v_pages = static_cast<const T*>(a.v_pages);

    float* q = q_staged + warp * d;
    const T* q_src = static_cast<const T*>(a.q) + (static_cast<size_t>(token) * a.heads + head) * d;
    for (int i = lane; i < d; i += 32) q[i] = to_float(q_src[i]);
    __syncwarp();

    const int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    const int kept_end = a.window > 0 ? min(a.keep_first, lowest) : 0;  // keys [0, kept_end) lie behind the window and stay
    float running_max = -INFINITY, denom = 0.0f;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.0f;

    // Two runs of tiles: the kept first tokens, then the window.
    for (int run = 0; run < 2; ++run) {
        const int from = run == 0 ? 0 : lowest, to = run == 0 ? kept_end - 1 : position;  // inclusive
        for (int tile = (from / 32) * 32; tile <= to; tile += 32) {
            const int key = tile + lane;
            const bool valid = key >= from && key <= to;
            long long slot = -1;  // page * page_size + offset of this lane's key, -1 when masked
            if (valid) {
                const int page = table[key / a.page_size];
                if (page >= 0) slot = static_cast<long long>(page) * a.page_size + key % a.page_size;
            }
            float score = -INFINITY;
            if (slot >= 0) {
                const long long page = slot / a.page_size, offset = slot % a.page_size;
                const T* k_row = k_pages + ((page * a.kv_heads + own_kv) * a.page_size + offset) * d;
                float dot = 0.0f;
                for (int i = 0; i < d; ++i) dot = fmaf(q[i], to_float(k_row[i]), dot);
                score = dot * a.scale;
                if (a.r1) score -= r1 * logf(1.0f + r2 * static_cast<float>(position - key));
            }
            const float new_max = fmaxf(running_max, warp_max(score));
            if (new_max == -INFINITY) continue;  // nothing visible yet (uniform across the warp)
            const float p = slot >= 0 ? expf(score - new_max) : 0.0f;
            const float rescale = expf(running_max - new_max);  // 0 on the first tile (exp(-inf))
            denom = denom * rescale + warp_sum(p);
            running_max = new_max;
#pragma unroll
            for (int i = 0; i < NACC; ++i) acc[i] *= rescale;
            for (int j = 0; j < 32; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j);
                const long long sj = __shfl_sync(0xffffffffu, slot, j);
                if (sj < 0) continue;  // uniform across the warp
                const long long page = sj / a.page_size, offset = sj % a.page_size;
#pragma unroll
                for (int i = 0; i < NACC; ++i) {
                    const int c = i / vchunks, e = lane + 32 * (i % vchunks);
                    if (c < value_heads && e < vd) {
                        const T* v_row = v_pages + ((page * a.kv_heads + first_value_head + c) * a.page_size + offset) * vd;
                        acc[i] = fmaf(pj, to_float(v_row[e]), acc[i]);
                    }
                }
            }
        }
    }
    const float inv = 1.0f / denom;
    if (a.spread) {
        float* out = static_cast<float*>(a.out) + (static_cast<size_t>(token) * a.heads + head) * a.kv_heads * vd;
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int c = i / vchunks, e = lane + 32 * (i % vchunks);
            if (c < value_heads && e < vd) out[c * vd + e] = acc[i] * inv;
        }
    } else {
        T* out = static_cast<T*>(a.out) + (static_cast<size_t>(token) * a.heads + head) * vd;
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int e = lane + 32 * i;
            if (i < vchunks && e < vd) out[e] = from_float<T>(acc[i] * inv);
        }
    }
}

// ---- the same with 16-byte loads: head widths that are multiples of 8 (bfloat16) or 4 (float32)

template <typename T>
struct Packed;
template <>
struct Packed<float> {
    static constexpr int N = 4;
    __device__ static void load(const float* p, float (&v)[4]) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    }
};
template <>
struct Packed<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static void load(const __nv_bfloat16* p, float (&v)[8]) {
        const uint4 x = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // a bfloat16 is the upper half of a float
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

// One block of VEC_WARPS warps per (token, query head): 4 in float32 always (the same bits for a token in a
// prompt and decoded alone), in bfloat16 1 when the step has items enough to fill the GPU and 16 when it has few.  Warp w takes the key tiles whose number (absolute
// position / 32) is w modulo VEC_WARPS, keeps its own running maximum, denominator and sums, and warp 0 adds
// the warps' results in ascending order: which warp visits which tile, and the order of every sum, depend on
// the query's position only.  A lane owns NV segments of N consecutive value elements among the (value
// heads x vdim) values of a key: segment u = lane + 32 * i is elements (u % per_row) * N .. of value head
// u / per_row.  Values are fetched for four keys at a time, all loads ahead of the arithmetic.
template <typename T, int NV, int VEC_WARPS>
__global__ void __launch_bounds__(VEC_WARPS * 32) biased_attention_vec_kernel(BiasedArgs a) {
    constexpr int N = Packed<T>::N;
    extern __shared__ __align__(16) float vec_shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int token = blockIdx.x / a.heads, head = blockIdx.x % a.heads;
    const int d = a.dim, vd = a.vdim;
    float* q = vec_shared;                                  // [dim]
    float* part_stat = q + ((d + 3) / 4) * 4;               // [VEC_WARPS][2] maximum, denominator
    float* part_acc = part_stat + VEC_WARPS * 2;            // [VEC_WARPS][NV][N][32]
    pdl_trigger();
    const float r1 = a.r1 ? a.r1[head] : 0.0f, r2 = a.r1 ? a.r2[head] : 0.0f;
    pdl_wait();
    const int own_kv = head / (a.heads / a.kv_heads);
    const int first_value_head = a.spread ? 0 : own_kv;
    const int value_heads = a.spread ? a.kv_heads : 1;
    const int per_row = vd / N, segments = value_heads * per_row;
    long long segment_offset[NV];  // where the lane's segments lie behind a key's first value head
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int u = lane + 32 * i;
        segment_offset[i] = u < segments ? (static_cast<long long>(first_value_head + u / per_row) * a.page_size) * vd + (u % per_row) * N : -1;
    }
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const T* k_pages = static_cast<const T*>(a.k_pages);
    const T* v_pages = static_cast<const T*>(a.v_pages);

    const T* q_src = static_cast<const T*>(a.q) + (static_cast<size_t>(token) * a.heads + head) * d;
    for (int i = threadIdx.x; i < d; i += VEC_WARPS * 32) q[i] = to_float(q_src[i]);
    __syncthreads();

    const int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    const int kept_end = a.window > 0 ? min(a.keep_first, lowest) : 0;
    float running_max = -INFINITY, denom = 0.0f;
    float acc[NV][N];
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int e = 0; e < N; ++e) acc[i][e] = 0.0f;

    for (int run = 0; run < 2; ++run) {
        const int from = run == 0 ? 0 : lowest, to = run == 0 ? kept_end - 1 : position;  // inclusive
        for (int tile = (from / 32) * 32; tile <= to; tile += 32) {
            if ((tile >> 5) % VEC_WARPS != warp) continue;
            const int key = tile + lane;
            const bool valid = key >= from && key <= to;
            int page = -1, offset = 0;
            if (valid) {
                page = table[key / a.page_size];
                offset = key % a.page_size;
            }
            float score = -INFINITY;
            if (page >= 0) {
                const T* k_row = k_pages + ((static_cast<long long>(page) * a.kv_heads + own_kv) * a.page_size + offset) * d;
                float dot = 0.0f;
#pragma unroll 4
                for (int i = 0; i < d; i += N) {
                    float k[N];
                    Packed<T>::load(k_row + i, k);
#pragma unroll
                    for (int e = 0; e < N; ++e) dot = fmaf(q[i + e], k[e], dot);
                }
                score = dot * a.scale;
                if (a.r1) score -= r1 * logf(1.0f + r2 * static_cast<float>(position - key));
            }
            const float new_max = fmaxf(running_max, warp_max(score));
            if (new_max == -INFINITY) continue;  // nothing visible in this tile (uniform across the warp)
            const float p = page >= 0 ? expf(score - new_max) : 0.0f;
            const float rescale = expf(running_max - new_max);  // 0 on the warp's first tile (exp(-inf))
            denom = denom * rescale + warp_sum(p);
            running_max = new_max;
#pragma unroll
            for (int i = 0; i < NV; ++i)
#pragma unroll
                for (int e = 0; e < N; ++e) acc[i][e] *= rescale;
            // element offset of the key's value row in value head 0, -1 when masked
            const long long row = page >= 0 ? (static_cast<long long>(page) * a.kv_heads * a.page_size + offset) * vd : -1;
            // Values: for KEYS keys at a time, all loads ahead of the arithmetic.  One warp per item (a step
            // with items enough to fill every SM) takes one key at a time: fewer registers, more warps per SM.
            constexpr int KEYS = VEC_WARPS == 1 ? 1 : 4;
#pragma unroll 4
            for (int j0 = 0; j0 < 32; j0 += KEYS) {
                float pj[KEYS];
                long long rj[KEYS];
                float v[KEYS][NV][N];
#pragma unroll
                for (int u = 0; u < KEYS; ++u) {
                    pj[u] = __shfl_sync(0xffffffffu, p, j0 + u);
                    rj[u] = __shfl_sync(0xffffffffu, row, j0 + u);
                }
#pragma unroll
                for (int u = 0; u < KEYS; ++u)
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        if (rj[u] >= 0 && segment_offset[i] >= 0) {
                            Packed<T>::load(v_pages + rj[u] + segment_offset[i], v[u][i]);
                        } else {
#pragma unroll
                            for (int e = 0; e < N; ++e) v[u][i][e] = 0.0f;  // a masked key has weight 0 as well
                        }
                    }
#pragma unroll
                for (int u = 0; u < KEYS; ++u)
#pragma unroll
                    for (int i = 0; i < NV; ++i)
#pragma unroll
                        for (int e = 0; e < N; ++e) acc[i][e] = fmaf(pj[u], v[u][i][e], acc[i][e]);
            }
        }
    }
    // The warps' partial results meet in shared memory; warp 0 adds them in ascending order.
    if (lane == 0) {
        part_stat[warp * 2] = running_max;
        part_stat[warp * 2 + 1] = denom;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int e = 0; e < N; ++e) part_acc[((warp * NV + i) * N + e) * 32 + lane] = acc[i][e];
    __syncthreads();
    if (warp != 0) return;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < VEC_WARPS; ++w) top = fmaxf(top, part_stat[w * 2]);
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int e = 0; e < N; ++e) acc[i][e] = 0.0f;
#pragma unroll
    for (int w = 0; w < VEC_WARPS; ++w) {
        const float m = part_stat[w * 2];
        if (m == -INFINITY) continue;  // this warp saw no key
        const float factor = expf(m - top);
        total = fmaf(part_stat[w * 2 + 1], factor, total);
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < N; ++e) acc[i][e] = fmaf(part_acc[((w * NV + i) * N + e) * 32 + lane], factor, acc[i][e]);
    }
    const float inv = 1.0f / total;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int u = lane + 32 * i;
        if (u >= segments) continue;
        const int c = u / per_row, e0 = (u % per_row) * N;
        if (a.spread) {
            float* out = static_cast<float*>(a.out) + ((static_cast<size_t>(token) * a.heads + head) * a.kv_heads + c) * vd + e0;
#pragma unroll
            for (int e = 0; e < N; ++e) out[e] = acc[i][e] * inv;
        } else {
            T* out = static_cast<T*>(a.out) + (static_cast<size_t>(token) * a.heads + head) * vd + e0;
#pragma unroll
            for (int e = 0; e < N; ++e) out[e] = from_float<T>(acc[i][e] * inv);
        }
    }
}

template <typename T, int NV, int VEC_WARPS>
static int launch_biased_vec_with(const BiasedArgs& a, cudaStream_t stream) {
    static SharedMemoryOptIn opt_in;
    constexpr int N = Packed<T>::N;
    const size_t smem = (static_cast<size_t>((a.dim + 3) / 4) * 4 + VEC_WARPS * 2 + static_cast<size_t>(VEC_WARPS) * NV * N * 32) * sizeof(float);
    if (smem > 200 * 1024) return ME_ERR_UNSUPPORTED;
    if (smem > 48 * 1024) {
        const int code = opt_in(biased_attention_vec_kernel<T, NV, VEC_WARPS>, static_cast<int>(smem));
        if (code) return code;
    }
    const long long items = static_cast<long long>(a.tokens) * a.heads;
    if (items > 0x7fffffffll) return ME_ERR_UNSUPPORTED;
    return launch_kernel_in_order(biased_attention_vec_kernel<T, NV, VEC_WARPS>, static_cast<int>(items), VEC_WARPS * 32, smem, stream, a);
}

constexpr long long ITEMS_THAT_FILL_THE_GPU = 2048;

template <typename T, int NV>
static int launch_biased_vec_as(const BiasedArgs& a, cudaStream_t stream) {
    if constexpr (sizeof(T) == 4) {
        return launch_biased_vec_with<T, NV, 4>(a, stream);
    } else {
        if (static_cast<long long>(a.tokens) * a.heads >= ITEMS_THAT_FILL_THE_GPU) return launch_biased_vec_with<T, NV, 1>(a, stream);
        return launch_biased_vec_with<T, NV, 16>(a, stream);
    }
}

template <typename T>
static int launch_biased_vec(const BiasedArgs& a, cudaStream_t stream, bool& taken) {
    constexpr int N = Packed<T>::N;
    const int segments = (a.spread ? a.kv_heads : 1) * (a.vdim / N);
    const int per_lane = (segments + 31) / 32;
    taken = true;
    if (per_lane <= 1) return launch_biased_vec_as<T, 1>(a, stream);
    if (per_lane <= 2) return launch_biased_vec_as<T, 2>(a, stream);
    if (per_lane <= 4) return launch_biased_vec_as<T, 4>(a, stream);
    if constexpr (N == 4) {
        if (per_lane <= 8) return launch_biased_vec_as<T, 8>(a, stream);
    }
    taken = false;
    return 0;
}

template <typename T>
static int launch_biased(const BiasedArgs& a, cudaStream_t stream) {
    // Which kernel runs depends on the model's sizes and the alignment of the engine's buffers only.
    constexpr int N = Packed<T>::N;
    const bool aligned = reinterpret_cast<uintptr_t>(a.k_pages) % 16 == 0 && reinterpret_cast<uintptr_t>(a.v_pages) % 16 == 0;
    if (a.dim % N == 0 && a.vdim % N == 0 && aligned) {
        bool taken = false;
        const int code = launch_biased_vec<T>(a, stream, taken);
        if (taken) return code;
    }
    const int per_lane = (a.spread ? a.kv_heads : 1) * ((a.vdim + 31) / 32);
    const long long items = static_cast<long long>(a.tokens) * a.heads;
    const int blocks = static_cast<int>((items + BIASED_WARPS - 1) / BIASED_WARPS);
    const size_t smem = static_cast<size_t>(BIASED_WARPS) * a.dim * sizeof(float);
    if (per_lane <= 2) return launch_kernel_in_order(biased_attention_kernel<T, 2>, blocks, BIASED_WARPS * 32, smem, stream, a);
    if (per_lane <= 4) return launch_kernel_in_order(biased_attention_kernel<T, 4>, blocks, BIASED_WARPS * 32, smem, stream, a);
    if (per_lane <= 8) return launch_kernel_in_order(biased_attention_kernel<T, 8>, blocks, BIASED_WARPS * 32, smem, stream, a);
    if (per_lane <= 16) return launch_kernel_in_order(biased_attention_kernel<T, 16>, blocks, BIASED_WARPS * 32, smem, stream, a);
    if (per_lane <= 32) return launch_kernel_in_order(biased_attention_kernel<T, 32>, blocks, BIASED_WARPS * 32, smem, stream, a);
    if (per_lane <= 64) return launch_kernel_in_order(biased_attention_kernel<T, 64>, blocks, BIASED_WARPS * 32, smem, stream, a);
    return ME_ERR_UNSUPPORTED;
}

ME_EXPORT int me_biased_attention(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                  const int* entry_of_token, const int* positions, const float* r1, const float* r2,
                                  void* out, int type, float scale, int tokens, int heads, int kv_heads, int dim,
                                  int vdim, int page_size, int table_width, int window, int keep_first, int spread,
                                  cudaStream_t stream) {
    if (tokens <= 0) return 0;
    if (heads % kv_heads || dim < 1 || vdim < 1 || dim > 2048) return ME_ERR_UNSUPPORTED;
    if ((r1 == nullptr) != (r2 == nullptr) || window < 0 || keep_first < 0) return ME_ERR_ARGUMENT;
    BiasedArgs a{q, k_pages, v_pages, block_table, entry_of_token, positions, r1, r2, out, scale,
                 tokens, heads, kv_heads, dim, vdim, page_size, table_width, window, keep_first, spread};
    return type == ME_BF16 ? launch_biased<__nv_bfloat16>(a, stream) : launch_biased<float>(a, stream);
}

// ------------------------------------------------------------- mixing in two kernels (fewer multiply-adds)
//
// The one-pass form above pays kv_heads times the value arithmetic for mixing after the softmax.  The form
// below keeps the scores instead: kernel 1 writes every (token, head)'s scores of its visible keys (32-bit,
// compacted: kept tokens first, then the window) and the softmax's maximum and denominator; kernel 2, one block
// per (token, KV head), turns the scores of ALL heads into normalised weights key by key, mixes them for the
// heads of its own group and applies the mixed weights to its values.  Per (token, key): heads x dim for the
// scores, heads x group for the mixing, group x vdim for the values, each once.  Tiles go to warps by tile
// number and partial results are added in ascending order, as above.

// Which entries of a step the tile kernel below takes, for a step that runs both forms: those that bring at least `eighths` / 8 of
// the keys that their last token sees, or `most` tokens.  An entry's few tokens behind many keys fill few blocks of tiles, each of
// which walks all of the keys; see me_mixed_attention_tiles.
struct TileRule {
    const int* cu_tokens;  // [entries + 1]; null: the kernel takes every entry
    int eighths, most;
};

constexpr int TILE_Q = 8, TILE_K = 32, TILE_DIM = 128;  // of the tile kernel

__device__ __forceinline__ bool takes_tiles(const TileRule& rule, const BiasedArgs& a, int entry) {
    const int begin = rule.cu_tokens[entry], count = rule.cu_tokens[entry + 1] - begin;
    if (count < TILE_Q) return false;
    const long long keys = min(static_cast<long long>(a.positions[begin + count - 1]) + 1, static_cast<long long>(a.window) + a.keep_first);
    return count >= rule.most || 8ll * count >= keys * rule.eighths;
}

struct ScoreArgs {
    BiasedArgs a;
    float* scores;  // [tokens][heads][stride]
    float* stats;   // [tokens][heads][2] maximum, denominator
    int stride;     // most keys a query can see
    TileRule tiles;  // entries that are left to the tile kernel
};

template <typename T, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) attention_scores_kernel(ScoreArgs s) {
    constexpr int N = Packed<T>::N;
    const BiasedArgs& a = s.a;
    extern __shared__ __align__(16) float score_shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int token = blockIdx.x / a.heads, head = blockIdx.x % a.heads;
    const int d = a.dim;
    float* q = score_shared;                         // [dim]
    float* part_stat = q + ((d + 3) / 4) * 4;        // [WARPS][2]
    pdl_trigger();
    const float r1 = a.r1 ? a.r1[head] : 0.0f, r2 = a.r1 ? a.r2[head] : 0.0f;
    pdl_wait();
    if (s.tiles.cu_tokens && takes_tiles(s.tiles, a, a.entry_of_token[token])) return;
    const int own_kv = head / (a.heads / a.kv_heads);
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const T* k_pages = static_cast<const T*>(a.k_pages);
    const T* q_src = static_cast<const T*>(a.q) + (static_cast<size_t>(token) * a.heads + head) * d;
    for (int i = threadIdx.x; i < d; i += WARPS * 32) q[i] = to_float(q_src[i]);
    __syncthreads();
    const bool packed = d % N == 0 && reinterpret_cast<uintptr_t>(a.k_pages) % 16 == 0;
    const int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    const int kept_end = a.window > 0 ? min(a.keep_first, lowest) : 0;
    float* row = s.scores + (static_cast<size_t>(token) * a.heads + head) * s.stride;
    float running_max = -INFINITY, denom = 0.0f;
    for (int run = 0; run < 2; ++run) {
        const int from = run == 0 ? 0 : lowest, to = run == 0 ? kept_end - 1 : position;  // inclusive
        for (int tile = (from / 32) * 32; tile <= to; tile += 32) {
            if ((tile >> 5) % WARPS != warp) continue;
            const int key = tile + lane;
            const bool valid = key >= from && key <= to;
            int page = -1;
            if (valid) page = table[key / a.page_size];
            float score = -INFINITY;
            if (page >= 0) {
                const T* k_row = k_pages + ((static_cast<long long>(page) * a.kv_heads + own_kv) * a.page_size + key % a.page_size) * d;
                float dot = 0.0f;
                if (packed) {
#pragma unroll 4
                    for (int i = 0; i < d; i += N) {
                        float k[N];
                        Packed<T>::load(k_row + i, k);
#pragma unroll
                        for (int e = 0; e < N; ++e) dot = fmaf(q[i + e], k[e], dot);
                    }
                } else {
                    for (int i = 0; i < d; ++i) dot = fmaf(q[i], to_float(k_row[i]), dot);
                }
                score = dot * a.scale;
                if (a.r1) score -= r1 * logf(1.0f + r2 * static_cast<float>(position - key));
            }
            if (valid) row[run == 0 ? key : kept_end + (key - lowest)] = score;
            const float new_max = fmaxf(running_max, warp_max(score));
            if (new_max == -INFINITY) continue;
            const float p = page >= 0 ? expf(score - new_max) : 0.0f;
            denom = denom * expf(running_max - new_max) + warp_sum(p);
            running_max = new_max;
        }
    }
    if (lane == 0) {
        part_stat[warp * 2] = running_max;
        part_stat[warp * 2 + 1] = denom;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    float top = -INFINITY;
    for (int w = 0; w < WARPS; ++w) top = fmaxf(top, part_stat[w * 2]);
    float total = 0.0f;
    for (int w = 0; w < WARPS; ++w)
        if (part_stat[w * 2] != -INFINITY) total = fmaf(part_stat[w * 2 + 1], expf(part_stat[w * 2] - top), total);
    float* out = s.stats + (static_cast<size_t>(token) * a.heads + head) * 2;
    out[0] = top;
    out[1] = total;
}

constexpr int MIX_GROUP = 8;    // query heads per KV head, at most
constexpr int MIX_COLUMNS = 8;  // value elements per lane, at most: vdim <= 256

// GROUP and COLUMNS: MIX_GROUP and MIX_COLUMNS, or as many as the sizes need, so that nothing is shuffled and added for heads
// and columns that are not there.  What the warps of a block wait for is memory: AT_ONCE heads' scores and KEYS keys' values are
// fetched ahead of the arithmetic, whose order is that of one at a time.  Four keys pay while their values and the sums leave
// registers for many warps: with 4 x 4 or more sums a lane, one key at a time is faster but for sixteen warps of 8 x 4.  Both
// kernels, us, every head and key at full width and one by one | this form (decoded tokens of 1,088 visible keys, bfloat16 unless
// said): 16 heads in 8 KV heads of 128, 32 tokens: 243 | 127; 32 heads in 8: 298 | 179; 16 in 4: 124 | 99; 16 in 2: 118 | 101; 16 in
// 8 with values of 256: 290 | 169 (four keys at a time: 570), float32 429 | 400; 8 in 1 with values of 192: 93 | 93 (151).
template <typename T, int WARPS, int GROUP, int COLUMNS>
__global__ void __launch_bounds__(WARPS * 32) attention_mix_values_kernel(ScoreArgs s, const float* __restrict__ talk) {
    constexpr int KEYS = COLUMNS == 4 && (GROUP == 2 || (GROUP == 8 && WARPS == 16)) ? 4 : 1;
    constexpr int AT_ONCE = GROUP == 8 && COLUMNS == 8 ? 4 : 8;
    const BiasedArgs& a = s.a;
    extern __shared__ __align__(16) float mix_shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int token = blockIdx.x / a.kv_heads, kv = blockIdx.x % a.kv_heads;
    const int heads = a.heads, group = heads / a.kv_heads, vd = a.vdim;
    float* top = mix_shared;                 // [heads]
    float* inverse = top + heads;            // [heads] 1 / denominator
    float* mixing = inverse + heads;         // [group][heads] rows of the mixing matrix for this group's heads
    float* partial = mixing + group * heads; // [WARPS][group][vd]
    pdl_trigger();
    for (int i = threadIdx.x; i < group * heads; i += WARPS * 32) mixing[i] = talk[(kv * group + i / heads) * heads + i % heads];
    pdl_wait();
    if (s.tiles.cu_tokens && takes_tiles(s.tiles, a, a.entry_of_token[token])) return;
    for (int g = threadIdx.x; g < heads; g += WARPS * 32) {
        const float* st = s.stats + (static_cast<size_t>(token) * heads + g) * 2;
        top[g] = st[0];
        inverse[g] = 1.0f / st[1];
    }
    __syncthreads();
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const T* v_pages = static_cast<const T*>(a.v_pages);
    const int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    const int kept_end = a.window > 0 ? min(a.keep_first, lowest) : 0;
    const float* rows = s.scores + static_cast<size_t>(token) * heads * s.stride;
    float acc[GROUP][COLUMNS];
#pragma unroll
    for (int h = 0; h < GROUP; ++h)
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) acc[h][i] = 0.0f;
    for (int run = 0; run < 2; ++run) {
        const int from = run == 0 ? 0 : lowest, to = run == 0 ? kept_end - 1 : position;  // inclusive
        for (int tile = (from / 32) * 32; tile <= to; tile += 32) {
            if ((tile >> 5) % WARPS != warp) continue;
            const int key = tile + lane;
            const bool valid = key >= from && key <= to;
            long long value_row = -1;  // element offset of this key's values in this KV head
            float mixed[GROUP];
#pragma unroll
            for (int h = 0; h < GROUP; ++h) mixed[h] = 0.0f;
            if (valid) {
                const int page = table[key / a.page_size];
                if (page >= 0) {
                    value_row = ((static_cast<long long>(page) * a.kv_heads + kv) * a.page_size + key % a.page_size) * vd;
                    const float* column = rows + (run == 0 ? key : kept_end + (key - lowest));
                    for (int g0 = 0; g0 < heads; g0 += AT_ONCE) {  // ascending g: the order of the mixed sum
                        float score[AT_ONCE];
#pragma unroll
                        for (int i = 0; i < AT_ONCE; ++i) score[i] = g0 + i < heads ? column[static_cast<size_t>(g0 + i) * s.stride] : 0.0f;
#pragma unroll
                        for (int i = 0; i < AT_ONCE; ++i) {
                            const int g = g0 + i;
                            if (g >= heads) break;
                            const float w = expf(score[i] - top[g]) * inverse[g];
#pragma unroll
                            for (int h = 0; h < GROUP; ++h)
                                if (h < group) mixed[h] = fmaf(mixing[h * heads + g], w, mixed[h]);
                        }
                    }
                }
            }
            for (int j0 = 0; j0 < 32; j0 += KEYS) {
                long long rj[KEYS];
                float v[KEYS][COLUMNS];
#pragma unroll
                for (int u = 0; u < KEYS; ++u) rj[u] = __shfl_sync(0xffffffffu, value_row, j0 + u);
#pragma unroll
                for (int u = 0; u < KEYS; ++u)
#pragma unroll
                    for (int i = 0; i < COLUMNS; ++i) v[u][i] = rj[u] >= 0 && lane + 32 * i < vd ? to_float(v_pages[rj[u] + lane + 32 * i]) : 0.0f;
#pragma unroll
                for (int u = 0; u < KEYS; ++u) {
                    float wj[GROUP];
#pragma unroll
                    for (int h = 0; h < GROUP; ++h) wj[h] = __shfl_sync(0xffffffffu, mixed[h], j0 + u);
                    if (rj[u] < 0) continue;  // uniform across the warp
#pragma unroll
                    for (int i = 0; i < COLUMNS; ++i)
#pragma unroll
                        for (int h = 0; h < GROUP; ++h) acc[h][i] = fmaf(wj[h], v[u][i], acc[h][i]);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < GROUP; ++h)
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) {
            const int e = lane + 32 * i;
            if (h < group && e < vd) partial[(warp * group + h) * vd + e] = acc[h][i];
        }
    __syncthreads();
    T* out = static_cast<T*>(a.out) + (static_cast<size_t>(token) * heads + kv * group) * vd;
    for (int i = threadIdx.x; i < group * vd; i += WARPS * 32) {
        float sum = 0.0f;
        for (int w = 0; w < WARPS; ++w) sum += partial[w * group * vd + i];
        out[i] = from_float<T>(sum);
    }
}

// The same for bfloat16 values in rows of whole 16-byte pieces, up to 128 wide, when few blocks of sixteen warps run (decoded tokens): a tile's values
// are on their way into shared memory, all 32 keys at once, while its weights are formed, and a lane adds four neighbouring
// columns up, so that a key costs a warp one load of values and one of weights instead of four loads and a shuffle per head.  The kernel above fetches four keys at a
// time, eight trips to memory a tile, behind the scores.  The order of every sum is the same, so are the bits.  16 heads in 8 KV heads of 128, eight tokens behind 16 to
// 2,048 keys (window 1,024, 64 kept): 61 -> 27 us.
constexpr int STAGED_WARPS = 16;

template <int GROUP>
__global__ void __launch_bounds__(STAGED_WARPS * 32) mix_values_staged_kernel(ScoreArgs s, const float* __restrict__ talk) {
    constexpr int AT_ONCE = 8;
    const BiasedArgs& a = s.a;
    extern __shared__ __align__(16) float mix_shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int token = blockIdx.x / a.kv_heads, kv = blockIdx.x % a.kv_heads;
    const int heads = a.heads, group = heads / a.kv_heads, vd = a.vdim, pieces = vd / 8;
    float* weights = mix_shared + warp * 32 * GROUP;                                                               // [32][GROUP] of this warp
    __nv_bfloat16* values = reinterpret_cast<__nv_bfloat16*>(mix_shared + STAGED_WARPS * 32 * GROUP) + warp * 32 * vd;  // [32][vd] of this warp
    float* partial = mix_shared + STAGED_WARPS * 32 * GROUP;                                                       // [WARPS][group][vd], when all is added
    float* top = partial + STAGED_WARPS * 16 * vd;                                                                 // [heads]
    float* inverse = top + heads;                                                                                  // [heads] 1 / denominator
    float* mixing = inverse + heads;                                                                               // [heads][GROUP] columns of the mixing matrix for this group's heads
    pdl_trigger();
    for (int i = threadIdx.x; i < GROUP * heads; i += STAGED_WARPS * 32) mixing[i] = i % GROUP < group ? talk[(kv * group + i % GROUP) * heads + i / GROUP] : 0.0f;
    pdl_wait();
    if (s.tiles.cu_tokens && takes_tiles(s.tiles, a, a.entry_of_token[token])) return;
    for (int g = threadIdx.x; g < heads; g += STAGED_WARPS * 32) {
        const float* st = s.stats + (static_cast<size_t>(token) * heads + g) * 2;
        top[g] = st[0];
        inverse[g] = 1.0f / st[1];
    }
    __syncthreads();
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const __nv_bfloat16* v_pages = static_cast<const __nv_bfloat16*>(a.v_pages);
    const int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    const int kept_end = a.window > 0 ? min(a.keep_first, lowest) : 0;
    const float* rows = s.scores + static_cast<size_t>(token) * heads * s.stride;
    float acc[GROUP][4];
#pragma unroll
    for (int h = 0; h < GROUP; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[h][i] = 0.0f;
    for (int run = 0; run < 2; ++run) {
        const int from = run == 0 ? 0 : lowest, to = run == 0 ? kept_end - 1 : position;  // inclusive
        for (int tile = (from / 32) * 32; tile <= to; tile += 32) {
            if ((tile >> 5) % STAGED_WARPS != warp) continue;
            const int key = tile + lane;
            long long value_row = -1;  // element offset of this key's values in this KV head
            if (key >= from && key <= to) {
                const int page = table[key / a.page_size];
                if (page >= 0) value_row = ((static_cast<long long>(page) * a.kv_heads + kv) * a.page_size + key % a.page_size) * vd;
            }
            const unsigned there = __ballot_sync(0xffffffffu, value_row >= 0);
            __syncwarp();  // the values of the tile before are read
            for (int c = lane; c < 32 * pieces; c += 32) {  // all lanes in every turn
                const int j = c / pieces, piece = c % pieces;
                const long long row = __shfl_sync(0xffffffffu, value_row, j);
                cp_async_16(values + j * vd + piece * 8, v_pages + max(row, 0ll) + piece * 8, row >= 0);
            }
            cp_async_commit();
            float mixed[GROUP];
#pragma unroll
            for (int h = 0; h < GROUP; ++h) mixed[h] = 0.0f;
            if (value_row >= 0) {
                const float* column = rows + (run == 0 ? key : kept_end + (key - lowest));
                for (int g0 = 0; g0 < heads; g0 += AT_ONCE) {  // ascending g: the order of the mixed sum
                    float score[AT_ONCE];
#pragma unroll
                    for (int i = 0; i < AT_ONCE; ++i) score[i] = g0 + i < heads ? column[static_cast<size_t>(g0 + i) * s.stride] : 0.0f;
#pragma unroll
                    for (int i = 0; i < AT_ONCE; ++i) {
                        const int g = g0 + i;
                        if (g >= heads) break;
                        const float w = expf(score[i] - top[g]) * inverse[g];
#pragma unroll
                        for (int h = 0; h < GROUP; ++h) mixed[h] = fmaf(mixing[g * GROUP + h], w, mixed[h]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < GROUP; ++h) weights[lane * GROUP + h] = mixed[h];
            cp_async_wait<0>();
            __syncwarp();
            if (lane * 4 < vd) {
#pragma unroll 8
                for (int j = 0; j < 32; ++j) {
                    float w[GROUP];
#pragma unroll
                    for (int h = 0; h < GROUP; ++h) w[h] = weights[j * GROUP + h];
                    const uint2 pair = *reinterpret_cast<const uint2*>(values + j * vd + lane * 4);
                    if (!(there >> j & 1)) continue;  // uniform across the warp
                    const float v[4] = {__uint_as_float(pair.x << 16), __uint_as_float(pair.x & 0xffff0000u), __uint_as_float(pair.y << 16), __uint_as_float(pair.y & 0xffff0000u)};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int h = 0; h < GROUP; ++h) acc[h][i] = fmaf(w[h], v[i], acc[h][i]);
                }
            }
        }
    }
    __syncthreads();  // the partial sums take the values' place
    if (lane * 4 < vd)
#pragma unroll
        for (int h = 0; h < GROUP; ++h)
            if (h < group) *reinterpret_cast<float4*>(partial + (warp * group + h) * vd + lane * 4) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
    __syncthreads();
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + (static_cast<size_t>(token) * heads + kv * group) * vd;
    for (int i = threadIdx.x; i < group * vd; i += STAGED_WARPS * 32) {
        float sum = 0.0f;
        for (int w = 0; w < STAGED_WARPS; ++w) sum += partial[w * group * vd + i];
        out[i] = __float2bfloat16_rn(sum);
    }
}

// Whether the staged kernel takes these sizes; its partial sums lie where the values were.  At widths of 128 one of its blocks fits an SM (135 KB) where
// two of the other kernel's do, and it is ahead all the same wherever sixteen warps run (up to 1,023 blocks).  Both kernels of the attention, us, the
// other form | this one, behind 64 keys and behind 2,048: 16 heads in 8 KV heads, 8 tokens 36 | 22 and 85 | 50, 32 44 | 36 and 124 | 112, 127 126 | 99
// and 413 | 362; 32 in 8, 127 tokens 170 | 140 and 616 | 560; 64 in 8 376 | 255 and 1,379 | 1,072; 8 in 1 60 | 36 and 181 | 126.  Beside a portion of 512
// that runs in tiles, whose blocks here return at once, 32 in 8: 8 decoded tokens 149 | 120, 32 233 | 226.
static bool staged_takes(const ScoreArgs& s) {
    const BiasedArgs& a = s.a;
    return a.vdim % 8 == 0 && a.vdim <= 128 && reinterpret_cast<uintptr_t>(a.v_pages) % 16 == 0 && a.heads <= 128;
}

template <int GROUP>
static int launch_staged(const ScoreArgs& s, const float* talk, cudaStream_t stream) {
    const size_t smem = (static_cast<size_t>(STAGED_WARPS) * 32 * GROUP + static_cast<size_t>(STAGED_WARPS) * 16 * s.a.vdim + (2 + GROUP) * s.a.heads) * sizeof(float);
    static SharedMemoryOptIn opt_in;
    if (const int code = opt_in(mix_values_staged_kernel<GROUP>, 200 * 1024)) return code;
    return launch_kernel_in_order(mix_values_staged_kernel<GROUP>, s.a.tokens * s.a.kv_heads, STAGED_WARPS * 32, smem, stream, s, talk);
}

template <typename T, int WARPS, int GROUP, int COLUMNS>
static int launch_mix_values(const ScoreArgs& s, const float* talk, size_t smem, cudaStream_t stream) {
    static SharedMemoryOptIn opt_in;
    if (smem > 48 * 1024) {
        const int code = opt_in(attention_mix_values_kernel<T, WARPS, GROUP, COLUMNS>, 200 * 1024);
        if (code) return code;
    }
    return launch_kernel_in_order(attention_mix_values_kernel<T, WARPS, GROUP, COLUMNS>, s.a.tokens * s.a.kv_heads, WARPS * 32, smem, stream, s, talk);
}

template <typename T, int WARPS>
static int launch_two_kernels(const ScoreArgs& s, const float* talk, cudaStream_t stream) {
    const BiasedArgs& a = s.a;
    const int group = a.heads / a.kv_heads;
    const size_t smem1 = (static_cast<size_t>((a.dim + 3) / 4) * 4 + WARPS * 2) * sizeof(float);
    const size_t smem2 = (static_cast<size_t>(2) * a.heads + static_cast<size_t>(group) * a.heads + static_cast<size_t>(WARPS) * group * a.vdim) * sizeof(float);
    if (smem1 > 48 * 1024 || smem2 > 200 * 1024) return ME_ERR_UNSUPPORTED;
    int code = launch_kernel_in_order(attention_scores_kernel<T, WARPS>, a.tokens * a.heads, WARPS * 32, smem1, stream, s);
    if (code) return code;
    if constexpr (std::is_same<T, __nv_bfloat16>::value && WARPS == STAGED_WARPS) {
        if (staged_takes(s)) {
            if (group <= 2) return launch_staged<2>(s, talk, stream);
            if (group <= 4) return launch_staged<4>(s, talk, stream);
            return launch_staged<MIX_GROUP>(s, talk, stream);
        }
    }
    if (a.vdim > 128) {
        if (group <= 2) return launch_mix_values<T, WARPS, 2, MIX_COLUMNS>(s, talk, smem2, stream);
        if (group <= 4) return launch_mix_values<T, WARPS, 4, MIX_COLUMNS>(s, talk, smem2, stream);
        return launch_mix_values<T, WARPS, MIX_GROUP, MIX_COLUMNS>(s, talk, smem2, stream);
    }
    if (group <= 2) return launch_mix_values<T, WARPS, 2, 4>(s, talk, smem2, stream);
    if (group <= 4) return launch_mix_values<T, WARPS, 4, 4>(s, talk, smem2, stream);
    return launch_mix_values<T, WARPS, MIX_GROUP, 4>(s, talk, smem2, stream);
}

// Mixed attention in two kernels.  `scores` holds tokens * heads * stride floats, `stats` tokens * heads * 2;
// `stride` is the most keys a query of this step can see.  out: [tokens][heads][vdim] of the pages' type.  With `cu_tokens` the
// entries that TileRule gives to the tile kernel are left alone; `expected`: about how many tokens then remain, else all.
ME_EXPORT int me_mixed_attention(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                 const int* entry_of_token, const int* positions, const float* r1, const float* r2,
                                 const float* talk, float* scores, float* stats, int stride, void* out, int type,
                                 float scale, int tokens, int heads, int kv_heads, int dim, int vdim, int page_size,
                                 int table_width, int window, int keep_first, const int* cu_tokens, int eighths, int most,
                                 int expected, cudaStream_t stream) {
    if (tokens <= 0) return 0;
    if (heads % kv_heads || heads / kv_heads > MIX_GROUP || vdim > 32 * MIX_COLUMNS || dim < 1 || vdim < 1) return ME_ERR_UNSUPPORTED;
    if ((r1 == nullptr) != (r2 == nullptr) || window < 0 || keep_first < 0 || talk == nullptr || stride < 1) return ME_ERR_ARGUMENT;
    if (static_cast<long long>(tokens) * heads > 0x7fffffffll) return ME_ERR_UNSUPPORTED;
    ScoreArgs s{{q, k_pages, v_pages, block_table, entry_of_token, positions, r1, r2, out, scale, tokens, heads,
                 kv_heads, dim, vdim, page_size, table_width, window, keep_first, 0},
                scores, stats, stride, {cu_tokens, eighths, most}};
    // float32: four warps always (the same bits for a token in a prompt and decoded alone); bfloat16: two
    // warps when the step has blocks enough to fill the GPU, sixteen when it has few.
    if (type != ME_BF16) return launch_two_kernels<float, 4>(s, talk, stream);
    if (static_cast<long long>(expected) * kv_heads >= 1024) return launch_two_kernels<__nv_bfloat16, 2>(s, talk, stream);
    return launch_two_kernels<__nv_bfloat16, 16>(s, talk, stream);
}

// ------------------------------------------------- mixing on tensor cores (portions of prompts, bfloat16)
//
// A block takes eight consecutive tokens of an entry and all heads; a warp one KV head with its GROUP query heads, two heads
// to the 16 rows of a product, so its keys, values, scores and output stay with it.  The first walk over the key tiles
// gives every row's maximum and denominator, the second forms the normalised weights, leaves them in shared memory as three
// bfloat16 terms (their sum is the float32 weight, all 24 bits), mixes them there as products [heads x heads] . [heads x
// (query, key)], each warp its own columns and in place, and applies the mixed weights, again three terms, to the values.
// Nothing but the output is written.  The distance bias is taken per (head, distance), 39 distances a tile of 32 keys, instead
// of per score.  Products are m16n8k16 with float32 sums.
//
// The terms are rounded to nearest, so a term is at most 2^-8 of the number before it: of the nine products of the mixing
// matrix's and the weights' terms the six largest are formed, the others are below 2^-24 of a product.  The tensor core
// truncates when it adds: the products with 16 keys' values leave it and are added to the output with rounding.
//
// A key that a query does not see has the weight zero in a product, which an infinity or NaN among its values would carry to
// that query.  So a block whose output holds one walks again: keys with such values are then taken out of the product and
// added to the queries that see them alone.
//
// Bound by the latency of a warp's own chains: registers and shared memory leave one block and two warps a scheduler, of which
// one issues every 4.6 cycles (1.9 of them the fixed latency of the instruction before); the tensor pipe is active 30 % of the
// time (profiles/mixed_attention_tiles_kernel_prefill_2048.md); figures at launch_mixed_tiles.  A tile of eight tokens, since the
// output of four heads and 16 tokens would take every register of a warp.
constexpr int BIAS_SPAN = TILE_Q + TILE_K;  // distances within a tile, one spare
constexpr int TERMS = 3;                    // bfloat16 terms of a float32 number

template <int KV, int GROUP>
struct MixTile {
    static constexpr int HEADS = KV * GROUP;
    static constexpr int PITCH = TILE_Q * TILE_K + 8;  // weights of a head, 16 bytes of padding: rows fall into different banks
    static constexpr int TALK_PITCH = HEADS + 8;
    static constexpr int KV_BYTES = TILE_K * TILE_DIM * 2;
    static constexpr int SMEM = 2 * KV * KV_BYTES + TERMS * HEADS * PITCH * 2 + TERMS * HEADS * TALK_PITCH * 2 + HEADS * BIAS_SPAN * 4;
};

struct MixTileArgs {
    BiasedArgs a;
    const float* talk;
    const int* cu_tokens;  // [entries + 1]
    TileRule rule;         // which entries, all without its own cu_tokens
};

// x and y as pairs of bfloat16 terms, the largest first
__device__ __forceinline__ void terms_of(float x, float y, uint32_t (&term)[TERMS]) {
#pragma unroll
    for (int i = 0; i < TERMS; ++i) {
        term[i] = pack_bf16(x, y);
        x -= __uint_as_float(term[i] << 16), y -= __uint_as_float(term[i] & 0xffff0000u);
    }
}

template <int KV, int GROUP>
__global__ void __launch_bounds__(KV * 32, 1) mixed_attention_tiles_kernel(MixTileArgs m) {
    using C = MixTile<KV, GROUP>;
    constexpr int HEADS = C::HEADS, ROWS = GROUP / 2;  // ROWS: products of 16 rows per warp
    static_assert(GROUP % 2 == 0 && (HEADS == 16 || HEADS == 32), "two heads to a product, 16 or 32 heads to mix");
    const BiasedArgs& a = m.a;
    extern __shared__ __align__(16) uint8_t mix_tile_shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, q = lane >> 2;
    __nv_bfloat16* keys = reinterpret_cast<__nv_bfloat16*>(mix_tile_shared) + warp * (C::KV_BYTES / 2);
    __nv_bfloat16* values = keys + KV * (C::KV_BYTES / 2);
    __nv_bfloat16* weights = reinterpret_cast<__nv_bfloat16*>(mix_tile_shared) + 2 * KV * (C::KV_BYTES / 2);  // [TERMS][HEADS][PITCH]
    __nv_bfloat16* talk = weights + TERMS * HEADS * C::PITCH;                                           // [TERMS][HEADS][TALK_PITCH]
    float* bias = reinterpret_cast<float*>(talk + TERMS * HEADS * C::TALK_PITCH) + warp * GROUP * BIAS_SPAN;
    constexpr int PLANE = HEADS * C::PITCH, TALK_PLANE = HEADS * C::TALK_PITCH;

    const int entry = blockIdx.y, begin = m.cu_tokens[entry];
    const int first = static_cast<int>(gridDim.x - 1 - blockIdx.x) * TILE_Q;  // the last tokens see the most keys: they go first
    const int count = min(m.cu_tokens[entry + 1] - begin - first, TILE_Q);
    if (count <= 0 || (m.rule.cu_tokens && !takes_tiles(m.rule, a, entry))) return;
    const int head0 = warp * GROUP;
    for (int i = threadIdx.x; i < HEADS * HEADS; i += KV * 32) {
        uint32_t term[TERMS];
        terms_of(m.talk[i], 0.0f, term);
#pragma unroll
        for (int plane = 0; plane < TERMS; ++plane)
            talk[plane * TALK_PLANE + i / HEADS * C::TALK_PITCH + i % HEADS] = __ushort_as_bfloat16(static_cast<unsigned short>(term[plane]));
    }
    const int p0 = a.positions[begin + first], p_last = p0 + count - 1;
    const int* table = a.block_table + static_cast<size_t>(entry) * a.table_width;
    const __nv_bfloat16* k_pages = static_cast<const __nv_bfloat16*>(a.k_pages);
    const __nv_bfloat16* v_pages = static_cast<const __nv_bfloat16*>(a.v_pages);

    uint32_t query[ROWS][TILE_DIM / 16][4];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int k = 0; k < TILE_DIM / 16; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.q) +
                    (static_cast<size_t>(begin + first + q) * HEADS + head0 + 2 * r + (i & 1)) * TILE_DIM + 16 * k + 8 * (i >> 1) + 2 * quad;
                query[r][k][i] = q < count ? *reinterpret_cast<const uint32_t*>(src) : 0u;
            }

    // Tiles: the kept keys behind every window of the block, then from the first window on.
    const int lowest = max(p0 - a.window + 1, 0);
    const int kept = min(a.keep_first, lowest);
    const int kept_tiles = (kept + TILE_K - 1) / TILE_K, tiles = kept_tiles + p_last / TILE_K - lowest / TILE_K + 1;
    auto tile_start = [&](int i) { return i < kept_tiles ? i * TILE_K : (lowest / TILE_K + i - kept_tiles) * TILE_K; };
    // This warp's 32 rows of a page array into shared memory (asynchronous); which keys there are.
    auto fetch = [&](const __nv_bfloat16* pages, __nv_bfloat16* to, int i) -> uint32_t {
        const int key = tile_start(i) + lane;
        long long row = -1;
        if (i < kept_tiles ? key < kept : key >= lowest && key <= p_last) {
            const int page = table[key / a.page_size];
            if (page >= 0) row = ((static_cast<long long>(page) * KV + warp) * a.page_size + key % a.page_size) * TILE_DIM;
        }
#pragma unroll
        for (int j = 0; j < TILE_K / 2; ++j) {
            const int r = 2 * j + (lane >> 4), chunk = lane & 15;
            const long long from = __shfl_sync(0xffffffffu, row, r);
            cp_async_16(to + swizzled<TILE_DIM>(r, chunk) * 8, pages + max(from, 0ll) + chunk * 8, from >= 0);
        }
        cp_async_commit();
        return __ballot_sync(0xffffffffu, row >= 0);
    };
    // bias[h][x]: distance x - 31 from the tile's first key to the block's first query
    auto distances = [&](int i) {
        const int base = p0 - tile_start(i) - (TILE_K - 1);
        __syncwarp();
        for (int x = lane; x < GROUP * BIAS_SPAN; x += 32) {
            const int h = head0 + x / BIAS_SPAN;
            bias[x] = a.r1 ? a.r1[h] * logf(1.0f + a.r2[h] * static_cast<float>(max(base + x % BIAS_SPAN, 0))) : 0.0f;
        }
        __syncwarp();
    };
    // Scores of 16 keys of a tile (`half`), -inf where the query does not see the key.
    auto scores = [&](const __nv_bfloat16* from, int i, int half, uint32_t there, float (&s)[ROWS][2][4]) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[r][n][c] = 0.0f;
#pragma unroll
        for (int k = 0; k < TILE_DIM / 16; ++k) {
            uint32_t b[4];
            ldmatrix_x4(b, from + swizzled<TILE_DIM>(half * 16 + (lane >> 4) * 8 + (lane & 7), 2 * k + ((lane >> 3) & 1)) * 8);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                mma_bf16(s[r][0], query[r][k], b[0], b[1]);
                mma_bf16(s[r][1], query[r][k], b[2], b[3]);
            }
        }
        const int start = tile_start(i);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int place = half * 16 + n * 8 + 2 * quad + e, distance = p0 + q - start - place;
                const bool seen = (there >> place & 1u) && distance >= 0 && (distance < a.window || start + place < a.keep_first) && q < count;
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float& v = s[r][n][2 * h + e];
                        v = seen ? v * a.scale - bias[(2 * r + h) * BIAS_SPAN + q + TILE_K - 1 - place] : -INFINITY;
                    }
            }
    };

    // First walk: maximum and denominator of every row (a lane's own columns, then the four lanes of a row).
    float top[ROWS][2], total[ROWS][2];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) top[r][0] = top[r][1] = -INFINITY, total[r][0] = total[r][1] = 0.0f;
    uint32_t there = fetch(k_pages, keys, 0);
    for (int i = 0; i < tiles; ++i) {
        __nv_bfloat16* held = i & 1 ? values : keys;
        uint32_t there_next = 0;
        if (i + 1 < tiles) there_next = fetch(k_pages, i & 1 ? keys : values, i + 1);
        else cp_async_commit();
        cp_async_wait<1>();
        distances(i);  // and the warp meets: every lane's copies are there
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float s[ROWS][2][4];
            scores(held, i, half, there, s);
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float peak = fmaxf(top[r][h], fmaxf(fmaxf(s[r][0][2 * h], s[r][0][2 * h + 1]), fmaxf(s[r][1][2 * h], s[r][1][2 * h + 1])));
                    if (peak == -INFINITY) continue;
                    total[r][h] = total[r][h] * expf(top[r][h] - peak) + ((expf(s[r][0][2 * h] - peak) + expf(s[r][0][2 * h + 1] - peak)) +
                                                                            (expf(s[r][1][2 * h] - peak) + expf(s[r][1][2 * h + 1] - peak)));
                    top[r][h] = peak;
                }
        }
        there = there_next;
        __syncwarp();  // the next copies overwrite this tile
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float peak = fmaxf(top[r][h], __shfl_xor_sync(0xffffffffu, top[r][h], 1));
            peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, 2));
            float sum = peak == -INFINITY ? 0.0f : total[r][h] * expf(top[r][h] - peak);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            top[r][h] = peak;
            total[r][h] = sum > 0.0f ? 1.0f / sum : 0.0f;
        }

    // Second walk.
    float out[ROWS][TILE_DIM / 8][4];
    // Values that hold an infinity or NaN: out of the product, and to the queries that see their key.
    auto add_apart = [&](int start) {
        bool odd_lane = false;
        for (int chunk = 0; chunk < TILE_DIM / 8; ++chunk) {
            const uint4 x = *reinterpret_cast<const uint4*>(values + swizzled<TILE_DIM>(lane, chunk) * 8);
            for (const uint32_t pair : {x.x, x.y, x.z, x.w}) odd_lane = odd_lane || (pair & 0x7f80u) == 0x7f80u || (pair & 0x7f800000u) == 0x7f800000u;
        }
        for (uint32_t odd = __ballot_sync(0xffffffffu, odd_lane); odd; odd &= odd - 1) {
            const int j = __ffs(odd) - 1, distance = p0 + q - start - j;
            if (q < count && distance >= 0 && (distance < a.window || start + j < a.keep_first)) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const __nv_bfloat16* from = weights + (head0 + 2 * r + h) * C::PITCH + ((j >> 3) * TILE_Q + q) * 8 + (j & 7);
                        const float w = __bfloat162float(from[0]) + (__bfloat162float(from[PLANE]) + __bfloat162float(from[2 * PLANE]));
#pragma unroll
                        for (int n = 0; n < TILE_DIM / 8; ++n) {
                            const uint32_t v = *reinterpret_cast<const uint32_t*>(values + swizzled<TILE_DIM>(j, n) * 8 + 2 * quad);
                            out[r][n][2 * h] = fmaf(w, __uint_as_float(v << 16), out[r][n][2 * h]);
                            out[r][n][2 * h + 1] = fmaf(w, __uint_as_float(v & 0xffff0000u), out[r][n][2 * h + 1]);
                        }
                    }
            }
            __syncwarp();
            if (lane < TILE_DIM / 8) *reinterpret_cast<uint4*>(values + swizzled<TILE_DIM>(j, lane) * 8) = make_uint4(0u, 0u, 0u, 0u);
            __syncwarp();
        }
    };
    auto walk = [&](auto apart) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int n = 0; n < TILE_DIM / 8; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) out[r][n][c] = 0.0f;
        there = fetch(k_pages, keys, 0);
        fetch(v_pages, values, 0);
        for (int i = 0; i < tiles; ++i) {
            cp_async_wait<1>();
            distances(i);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float s[ROWS][2][4];
                scores(keys, i, half, there, s);
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float w[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const float v = s[r][n][2 * h + e];
                                w[e] = v == -INFINITY ? 0.0f : expf(v - top[r][h]) * total[r][h];
                            }
                            uint32_t term[TERMS];
                            terms_of(w[0], w[1], term);
                            // columns of a head: (8 keys, query, key), so that a query's eight keys are one 16-byte row
                            __nv_bfloat16* to = weights + (head0 + 2 * r + h) * C::PITCH + ((half * 2 + n) * TILE_Q + q) * 8 + 2 * quad;
#pragma unroll
                            for (int plane = 0; plane < TERMS; ++plane) *reinterpret_cast<uint32_t*>(to + plane * PLANE) = term[plane];
                        }
            }
            __syncwarp();
            if (i + 1 < tiles) there = fetch(k_pages, keys, i + 1);
            else cp_async_commit();
            __syncthreads();  // every head's weights
#pragma unroll
            for (int column = warp; column < TILE_Q * TILE_K / 8; column += KV) {
                uint32_t b[TERMS][HEADS / 8];  // B operands: eight (query, key) columns of all heads
#pragma unroll
                for (int plane = 0; plane < TERMS; ++plane) {
                    if constexpr (HEADS == 32) ldmatrix_x4_trans(b[plane], weights + plane * PLANE + lane * C::PITCH + column * 8);
                    else ldmatrix_x2_trans(b[plane], weights + plane * PLANE + (lane & 15) * C::PITCH + column * 8);
                }
                __syncwarp();  // the columns are read before their mixed weights take their place
#pragma unroll
                for (int r = 0; r < HEADS / 16; ++r) {
                    uint32_t t[TERMS][HEADS / 16][4];
#pragma unroll
                    for (int plane = 0; plane < TERMS; ++plane)
#pragma unroll
                        for (int k = 0; k < HEADS / 16; ++k)
                            ldmatrix_x4(t[plane][k], talk + plane * TALK_PLANE + (r * 16 + (lane & 15)) * C::TALK_PITCH + k * 16 + (lane >> 4) * 8);
                    float mixed[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int level = TERMS - 1; level >= 0; --level)  // the smallest products first
#pragma unroll
                        for (int k = 0; k < HEADS / 16; ++k)
#pragma unroll
                            for (int plane = 0; plane <= level; ++plane) mma_bf16(mixed, t[plane][k], b[level - plane][2 * k], b[level - plane][2 * k + 1]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t term[TERMS];
                        terms_of(mixed[2 * h], mixed[2 * h + 1], term);
                        __nv_bfloat16* to = weights + (r * 16 + q + 8 * h) * C::PITCH + column * 8 + 2 * quad;
#pragma unroll
                        for (int plane = 0; plane < TERMS; ++plane) *reinterpret_cast<uint32_t*>(to + plane * PLANE) = term[plane];
                    }
                }
            }
            cp_async_wait<1>();
            __syncthreads();  // every column's mixed weights; each warp reads its own heads' and overwrites them alone
            if constexpr (decltype(apart)::value) add_apart(tile_start(i));
#pragma unroll
            for (int k = 0; k < TILE_K / 16; ++k) {
                uint32_t w[ROWS][TERMS][4];
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int plane = 0; plane < TERMS; ++plane)
                        ldmatrix_x4(w[r][plane], weights + plane * PLANE + (head0 + 2 * r + ((lane >> 3) & 1)) * C::PITCH +
                                                     ((2 * k + (lane >> 4)) * TILE_Q + (lane & 7)) * 8);
#pragma unroll
                for (int n = 0; n < TILE_DIM / 16; ++n) {
                    uint32_t b[4];
                    ldmatrix_x4_trans(b, values + swizzled<TILE_DIM>(k * 16 + (lane & 15), 2 * n + (lane >> 4)) * 8);
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        float part[2][4] = {};
#pragma unroll
                        for (int plane = TERMS - 1; plane >= 0; --plane) {
                            mma_bf16(part[0], w[r][plane], b[0], b[1]);
                            mma_bf16(part[1], w[r][plane], b[2], b[3]);
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c) out[r][2 * n][c] += part[0][c], out[r][2 * n + 1][c] += part[1][c];
                    }
                }
            }
            __syncwarp();
            if (i + 1 < tiles) fetch(v_pages, values, i + 1);
            else cp_async_commit();
        }
        cp_async_wait<0>();
    };
    walk(std::false_type{});
    bool finite = true;
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int n = 0; n < TILE_DIM / 8; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) finite = finite && fabsf(out[r][n][c]) < INFINITY;
    if (__syncthreads_or(!finite)) walk(std::true_type{});
    if (q >= count) return;
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            __nv_bfloat16* to = static_cast<__nv_bfloat16*>(a.out) + (static_cast<size_t>(begin + first + q) * HEADS + head0 + 2 * r + h) * TILE_DIM + 2 * quad;
#pragma unroll
            for (int n = 0; n < TILE_DIM / 8; ++n) *reinterpret_cast<uint32_t*>(to + 8 * n) = pack_bf16(out[r][n][2 * h], out[r][n][2 * h + 1]);
        }
}

// Against the two kernels above as they were, on one prompt of 2,048 tokens (window 1,024, 64 kept): 32 heads of 8 KV heads
// 7,795 -> 699 us, 16 heads 5,294 -> 376 us; 700 tokens behind 800: 3,448 -> 455 and 2,363 -> 245 us (with weights and mixing
// matrix in two terms, 17 bits, 569, 330, 377 and 216 us: the third term's products cost a fifth and are what keeps 32 bits).  Error
// against float64 the same (1.66e-3, the output's rounding to bfloat16), also where the heads' weights cancel.
template <int KV, int GROUP>
static int launch_mixed_tiles(const MixTileArgs& m, int entries, int longest, cudaStream_t stream) {
    static SharedMemoryOptIn opt_in;
    if (const int code = opt_in(mixed_attention_tiles_kernel<KV, GROUP>, MixTile<KV, GROUP>::SMEM)) return code;
    const dim3 grid((longest + TILE_Q - 1) / TILE_Q, entries);
    return launch_kernel_in_order(mixed_attention_tiles_kernel<KV, GROUP>, grid, KV * 32, MixTile<KV, GROUP>::SMEM, stream, m);
}

// The same result from tiles of tokens; bfloat16, 128-wide heads, the (kv_heads, group) pairs below.  The tokens of entry e are
// cu_tokens[e] .. cu_tokens[e + 1], at consecutive positions; none has more than `longest`.  `most` > 0: only the entries that
// TileRule gives to this kernel, which the two kernels above then leave alone.
ME_EXPORT int me_mixed_attention_tiles(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                       const int* cu_tokens, const int* positions, const float* r1, const float* r2,
                                       const float* talk, void* out, float scale, int entries, int longest, int heads, int kv_heads,
                                       int dim, int vdim, int page_size, int table_width, int window, int keep_first, int eighths,
                                       int most, cudaStream_t stream) {
    if (entries <= 0 || longest <= 0) return 0;
    if (dim != TILE_DIM || vdim != TILE_DIM || kv_heads < 1 || heads % kv_heads || entries > 65535) return ME_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(k_pages) % 16 || reinterpret_cast<uintptr_t>(v_pages) % 16 || reinterpret_cast<uintptr_t>(q) % 4 || reinterpret_cast<uintptr_t>(out) % 4)
        return ME_ERR_UNSUPPORTED;
    if ((r1 == nullptr) != (r2 == nullptr) || window < 1 || keep_first < 0 || talk == nullptr) return ME_ERR_ARGUMENT;
    MixTileArgs m{{q, k_pages, v_pages, block_table, nullptr, positions, r1, r2, out, scale, 0, heads, kv_heads, dim, vdim,
                   page_size, table_width, window, keep_first, 0},
                  talk, cu_tokens, {most > 0 ? cu_tokens : nullptr, eighths, most}};
    const int group = heads / kv_heads;
    if (kv_heads == 8 && group == 4) return launch_mixed_tiles<8, 4>(m, entries, longest, stream);
    if (kv_heads == 8 && group == 2) return launch_mixed_tiles<8, 2>(m, entries, longest, stream);
    if (kv_heads == 4 && group == 4) return launch_mixed_tiles<4, 4>(m, entries, longest, stream);
    return ME_ERR_UNSUPPORTED;
}

// out[t][h][e] = sum_g talk[h][g] * spread[t][g][kv(h)][e], ascending g.
template <typename T>
__global__ void mix_heads_kernel(const float* __restrict__ spread, const float* __restrict__ talk, T* __restrict__ out,
                                 int tokens, int heads, int kv_heads, int vdim) {
    pdl_trigger();
    pdl_wait();
    const size_t total = static_cast<size_t>(tokens) * heads * vdim;
    const int group = heads / kv_heads;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int e = static_cast<int>(idx % vdim);
        const int h = static_cast<int>((idx / vdim) % heads);
        const size_t t = idx / (static_cast<size_t>(vdim) * heads);
        const float* row = spread + t * heads * kv_heads * vdim + static_cast<size_t>(h / group) * vdim + e;
        float sum = 0.0f;
        for (int g = 0; g < heads; ++g) sum = fmaf(talk[h * heads + g], row[static_cast<size_t>(g) * kv_heads * vdim], sum);
        out[idx] = from_float<T>(sum);
    }
}

ME_EXPORT int me_mix_heads(const float* spread, const float* talk, void* out, int type, int tokens, int heads,
                           int kv_heads, int vdim, cudaStream_t stream) {
    if (tokens <= 0) return 0;
    const size_t total = static_cast<size_t>(tokens) * heads * vdim;
    const int threads = 256;
    const int blocks = static_cast<int>(std::min<size_t>((total + threads - 1) / threads, 148 * 16));
    if (type == ME_BF16)
        return launch_kernel(mix_heads_kernel<__nv_bfloat16>, blocks, threads, 0, stream, spread, talk,
                             static_cast<__nv_bfloat16*>(out), tokens, heads, kv_heads, vdim);
    return launch_kernel(mix_heads_kernel<float>, blocks, threads, 0, stream, spread, talk, static_cast<float*>(out),
                         tokens, heads, kv_heads, vdim);
}
