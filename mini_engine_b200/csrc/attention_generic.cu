// Causal grouped-query attention over the paged cache for any head size: one warp per
// (token, query head).  It is the attention of the float32 path and of bfloat16 head sizes
// that the tensor-core kernels do not take.
//
// Formula (YuvGev00/mini-engine, src/mini_engine/attention.py:84-86,160-175 and the online
// softmax of src/mini_engine/triton_attention.py:56-82): query head h reads KV head h / group;
// s = (q . k) * scale; the query at position p sees keys at positions <= p (and > p - window
// when a window is given); out = softmax(s) V.  Options: value heads of their own width (`value_dim`); a
// softmax with one more, silent participant of score zero that has no value (`sink`: p_j = exp(s_j) /
// (1 + sum exp(s))), or of a learned score per head (`sink_values`: exp(sink_h) in place of the 1); a multiplier
// on the output (`gate`, float32 [tokens][heads][gate_width] with gate_width 1, one per head, or value_dim, one per
// element); a distance bias that is linear in the distance (`slopes`, one per head: s -= slope_h * (p - j), after
// the scale); a cap on the scaled scores (`softcap`: s becomes softcap * tanh(s / softcap)); and values that are the first value_dim elements of the key rows (`value_stride`: elements between
// two value rows; pass the key pages as value pages and head_dim as the stride); chunks (`chunk`: the query at position p sees
// keys from floor(p / chunk) * chunk on); and weights without a softmax (`sigmoid_bias`, one per head: the weight of a visible
// key is sigmoid(s + bias_h), not normalised over the keys).
//
// Keys are visited in tiles of 32 whose boundaries are multiples of 32 in *absolute position*
// and are combined in ascending order, so the arithmetic of a query depends only on its own
// position: the same bits come out whether the token arrived in a whole prompt, in a
// two-token portion or as a decoded token, and whatever else is in the batch.
#include "mma_sync.cuh"

struct AttnArgs {
    const void* q;         // [tokens][heads][head_dim]
    const void* k_pages;   // [pages][kv_heads][page_size][head_dim]
    const void* v_pages;
    const int* block_table;  // [entries][table_width]
    const int* entry_of_token;
    const int* positions;
    void* out;  // [tokens][heads][value_dim]
    float scale;
    int tokens, heads, kv_heads, head_dim, page_size, table_width, window;
    int value_dim, sink;
    const float* gate;  // [tokens][heads][gate_width] or null
    int gate_width, value_stride;
    const float* slopes;       // [heads] or null
    const float* sink_values;  // [heads] or null (with sink: the silent participant's score, zero when null)
    float softcap;             // > 0: the scaled score s becomes softcap * tanh(s / softcap)
    int chunk;                  // > 0: keys of the query's own chunk of positions only
    const float* sigmoid_bias;  // [heads] weights sigmoid(s + bias) in the place of a softmax, or null
};

constexpr int ATTN_WARPS = 4;
constexpr int MAX_DIM_PER_LANE = 16;  // value_dim <= 512
constexpr int MAX_KEY_DIM = 2048;     // the query is staged in shared memory

template <typename T>
__global__ void __launch_bounds__(ATTN_WARPS * 32) paged_attention_generic_kernel(AttnArgs a) {
    extern __shared__ float q_staged[];  // [ATTN_WARPS][head_dim]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = static_cast<long long>(blockIdx.x) * ATTN_WARPS + warp;
    if (item >= static_cast<long long>(a.tokens) * a.heads) return;
    const int token = static_cast<int>(item / a.heads), head = static_cast<int>(item % a.heads);
    const int d = a.head_dim, dv = a.value_dim;
    pdl_trigger();
    pdl_wait();
    const int kv_head = head / (a.heads / a.kv_heads);
    const int position = a.positions[token];
    const int* table = a.block_table + static_cast<size_t>(a.entry_of_token[token]) * a.table_width;
    const T* k_pages = static_cast<const T*>(a.k_pages);
    const T* v_pages = static_cast<const T*>(a.v_pages);

    float* q = q_staged + warp * d;
    const T* q_src = static_cast<const T*>(a.q) + (static_cast<size_t>(token) * a.heads + head) * d;
    for (int i = lane; i < d; i += 32) q[i] = to_float(q_src[i]);
    __syncwarp();

    const float slope = a.slopes ? a.slopes[head] : 0.0f;
    const size_t v_stride = static_cast<size_t>(a.value_stride);
    int lowest = a.window > 0 ? max(position - a.window + 1, 0) : 0;
    if (a.chunk > 0) lowest = max(lowest, position / a.chunk * a.chunk);
    const bool sigmoid = a.sigmoid_bias != nullptr;
    const float weight_bias = sigmoid ? a.sigmoid_bias[head] : 0.0f;
    float running_max = -INFINITY, denom = 0.0f;
    float acc[MAX_DIM_PER_LANE];
#pragma unroll
    for (int i = 0; i < MAX_DIM_PER_LANE; ++i) acc[i] = 0.0f;

    for (int tile = (lowest / 32) * 32; tile <= position; tile += 32) {
        const int key = tile + lane;
        const bool valid = key >= lowest && key <= position;
        long long base = -1;  // row of this lane's key in the pages, -1 when masked
        if (valid) {
            const int page = table[key / a.page_size];
            if (page >= 0)
                base = (static_cast<long long>(page) * a.kv_heads + kv_head) * a.page_size + key % a.page_size;
        }
        float score = -INFINITY;
        if (base >= 0) {
            const T* k_row = k_pages + base * d;
            float dot = 0.0f;
            for (int i = 0; i < d; ++i) dot = fmaf(q[i], to_float(k_row[i]), dot);
            score = dot * a.scale;
            if (a.softcap > 0.0f) score = a.softcap * tanhf(score / a.softcap);
            if (a.slopes) score -= slope * static_cast<float>(position - key);
        }
        float p;
        if (sigmoid) {
            p = base >= 0 ? 1.0f / (1.0f + expf(-(score + weight_bias))) : 0.0f;
        } else {
            const float new_max = fmaxf(running_max, warp_max(score));
            if (new_max == -INFINITY) continue;  // nothing visible yet (uniform across the warp)
            p = base >= 0 ? expf(score - new_max) : 0.0f;
            const float rescale = expf(running_max - new_max);  // 0 on the first tile (exp(-inf))
            denom = denom * rescale + warp_sum(p);
            running_max = new_max;
#pragma unroll
            for (int i = 0; i < MAX_DIM_PER_LANE; ++i) acc[i] *= rescale;
        }
        for (int j = 0; j < 32; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const long long bj = __shfl_sync(0xffffffffu, base, j);
            if (bj < 0) continue;  // uniform across the warp
            const T* v_row = v_pages + bj * v_stride;
#pragma unroll
            for (int i = 0; i < MAX_DIM_PER_LANE; ++i) {
                const int e = lane + 32 * i;
                if (e < dv) acc[i] = fmaf(pj, to_float(v_row[e]), acc[i]);
            }
        }
    }
    T* out = static_cast<T*>(a.out) + (static_cast<size_t>(token) * a.heads + head) * dv;
    if (a.sink) denom += expf((a.sink_values ? a.sink_values[head] : 0.0f) - running_max);  // the silent participant
    float inv = sigmoid ? 1.0f : 1.0f / denom;
    const float* gate = a.gate ? a.gate + (static_cast<size_t>(token) * a.heads + head) * a.gate_width : nullptr;
    if (gate && a.gate_width == 1) inv *= gate[0];
#pragma unroll
    for (int i = 0; i < MAX_DIM_PER_LANE; ++i) {
        const int e = lane + 32 * i;
        if (e < dv) {
            float y = acc[i] * inv;
            if (gate && a.gate_width > 1) y *= gate[e];
            out[e] = from_float<T>(y);
        }
    }
}

// ------------------------------------------------------------------ float32, keys shared by many rows
//
// The same attention in float32 with every key and value fetched once for a block of R rows, a row being a (token, query
// head) pair of one entry and KV head: row r of an entry is its token r / group, head r % group of the group.  The
// arithmetic of a row is the kernel's above, operation by operation (a score is one fmaf chain over the head; maximum and sum of
// a tile by the same butterflies over its 32 keys; a value element one fmaf chain over the keys), so the bits are the same
// whichever kernel and whichever R a step takes.  Tiles of 32 keys arrive by asynchronous copies, two buffers; 256 threads form
// R x 32 scores (a thread 2 rows x 4 keys, or 1 x 2), a warp takes whole rows for the softmax, and a thread keeps one quad
// of value elements of R * QP / 256 rows.  A tile that some row sees in part marks the weights of unseen keys, and
// their values are left out (they may be anything); a tile that all rows see whole is not looked at twice.
// Bound by latency: eight warps to an SM for steps of this size (512 tokens are 128 blocks), each of which issues every 4.8 cycles
// at R = 64 and every 6 at R = 16 and waits for shared memory most (1.5 and 2.2 cycles; profiles/paged_attention_rows_kernel.md);
// figures at launch_rows.
constexpr int ROW_THREADS = 256;
constexpr uint32_t UNSEEN = 0x80000000u;  // the weight -0: a key that the row does not see

struct RowArgs {
    AttnArgs a;
    const int* cu_tokens;
};

template <int R, int QP>
__global__ void __launch_bounds__(ROW_THREADS) paged_attention_rows_kernel(RowArgs m) {
    constexpr int KEYS = R == 64 ? 4 : 2, KEY_LANES = 32 / KEYS, ROWS = R * KEY_LANES / ROW_THREADS;  // a thread's scores
    constexpr int HELD = R * QP / ROW_THREADS;                                                      // its rows of values
    static_assert(ROWS >= 1 && HELD >= 1, "every thread has work");
    constexpr int SP = 36;  // floats between two rows of weights
    const AttnArgs& a = m.a;
    extern __shared__ __align__(16) float row_shared[];
    __shared__ int key_there[2][32];
    __shared__ float row_max[R], row_sum[R], row_scale[R];
    const int d = a.head_dim, dv = a.value_dim, kp = d + 4, vp = dv + 4;
    const bool shared_rows = a.k_pages == a.v_pages;  // values are the first elements of the key rows
    float* q = row_shared;                                   // [R][kp]
    float* keys = q + R * kp;                                // [2][32][kp]
    float* values = shared_rows ? keys : keys + 2 * 32 * kp; // [2][32][vp]
    const int v_pitch = shared_rows ? kp : vp;
    float* weights = shared_rows ? keys + 2 * 32 * kp : values + 2 * 32 * vp;  // [R][SP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    pdl_wait();
    const int entry = blockIdx.z, kv = blockIdx.y, group = a.heads / a.kv_heads;
    const int begin = m.cu_tokens[entry], rows = (m.cu_tokens[entry + 1] - begin) * group;
    const int row0 = static_cast<int>(gridDim.x - 1 - blockIdx.x) * R;  // the last rows see the most keys: they go first
    if (row0 >= rows) return;
    const int live = min(R, rows - row0);
    const int* table = a.block_table + static_cast<size_t>(entry) * a.table_width;
    const float *k_pages = static_cast<const float*>(a.k_pages), *v_pages = static_cast<const float*>(a.v_pages);
    auto position_of = [&](int r) { return a.positions[begin + (row0 + r) / group]; };
    auto lowest_of = [&](int position) {
        const int low = a.window > 0 ? max(position - a.window + 1, 0) : 0;
        return a.chunk > 0 ? max(low, position / a.chunk * a.chunk) : low;
    };
    const int first_position = position_of(0), last_position = position_of(live - 1);
    const int lowest = lowest_of(first_position), highest_low = lowest_of(last_position);

    for (int i = tid; i < R * (d / 4); i += ROW_THREADS) {
        const int r = i / (d / 4), e = i % (d / 4) * 4;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < live)
            x = *reinterpret_cast<const float4*>(static_cast<const float*>(a.q) +
                                                 (static_cast<size_t>(begin + (row0 + r) / group) * a.heads + kv * group + (row0 + r) % group) * d + e);
        *reinterpret_cast<float4*>(q + r * kp + e) = x;
    }
    for (int r = tid; r < R; r += ROW_THREADS) row_max[r] = -INFINITY, row_sum[r] = 0.0f;

    // Eight threads fetch a key's row and its values.
    auto fetch = [&](int tile, int buffer) {
        const int j = tid >> 3, key = tile + j;
        int page = -1;
        if (key >= lowest && key <= last_position) page = table[key / a.page_size];
        const size_t row = page >= 0 ? (static_cast<size_t>(page) * a.kv_heads + kv) * a.page_size + key % a.page_size : 0;
        float* to = keys + (buffer * 32 + j) * kp;
        for (int e = (tid & 7) * 4; e < d; e += 32) cp_async_16(to + e, k_pages + row * d + e, page >= 0);
        if (!shared_rows) {
            float* v_to = values + (buffer * 32 + j) * vp;
            for (int e = (tid & 7) * 4; e < dv; e += 32) cp_async_16(v_to + e, v_pages + row * a.value_stride + e, page >= 0);
        }
        if ((tid & 7) == 0) key_there[buffer][j] = page >= 0;
        cp_async_commit();
    };

    const int quad = tid % QP * 4, held0 = tid / QP * HELD;  // value elements, first row
    float4 acc[HELD];
#pragma unroll
    for (int i = 0; i < HELD; ++i) acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int key_lane = tid % KEY_LANES, score_row = tid / KEY_LANES * ROWS;
    const bool sigmoid = a.sigmoid_bias != nullptr;

    int buffer = 0;
    fetch(lowest / 32 * 32, 0);
    for (int tile = lowest / 32 * 32; tile <= last_position; tile += 32, buffer ^= 1) {
        if (tile + 32 <= last_position) fetch(tile + 32, buffer ^ 1);
        else cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* k_tile = keys + buffer * 32 * kp;
        {
            float dot[ROWS][KEYS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int k = 0; k < KEYS; ++k) dot[r][k] = 0.0f;
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                float4 qq[ROWS], kk[KEYS];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) qq[r] = *reinterpret_cast<const float4*>(q + (score_row + r) * kp + e);
#pragma unroll
                for (int k = 0; k < KEYS; ++k) kk[k] = *reinterpret_cast<const float4*>(k_tile + (key_lane + KEY_LANES * k) * kp + e);
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int k = 0; k < KEYS; ++k) {
                        dot[r][k] = fmaf(qq[r].x, kk[k].x, dot[r][k]);
                        dot[r][k] = fmaf(qq[r].y, kk[k].y, dot[r][k]);
                        dot[r][k] = fmaf(qq[r].z, kk[k].z, dot[r][k]);
                        dot[r][k] = fmaf(qq[r].w, kk[k].w, dot[r][k]);
                    }
            }
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int k = 0; k < KEYS; ++k) weights[(score_row + r) * SP + key_lane + KEY_LANES * k] = dot[r][k];
        }
        __syncthreads();
        const bool there = key_there[buffer][lane] != 0;
        const bool whole = __all_sync(0xffffffffu, there) && tile >= highest_low && tile + 31 <= first_position;
#pragma unroll 4
        for (int r = warp; r < R; r += ROW_THREADS / 32) {
            if (r >= live) break;
            const int position = position_of(r), head = kv * group + (row0 + r) % group, key = tile + lane;
            const bool seen = there && key >= lowest_of(position) && key <= position;
            float score = -INFINITY;
            if (seen) {
                score = weights[r * SP + lane] * a.scale;
                if (a.softcap > 0.0f) score = a.softcap * tanhf(score / a.softcap);
                if (a.slopes) score -= a.slopes[head] * static_cast<float>(position - key);
            }
            float p = __uint_as_float(UNSEEN);
            if (sigmoid) {
                if (seen) p = 1.0f / (1.0f + expf(-(score + a.sigmoid_bias[head])));
            } else {
                const float old_max = row_max[r], new_max = fmaxf(old_max, warp_max(score));
                float rescale = 1.0f;
                if (new_max != -INFINITY) {  // uniform across the warp
                    rescale = expf(old_max - new_max);
                    const float weight = seen ? expf(score - new_max) : 0.0f;
                    const float sum = row_sum[r] * rescale + warp_sum(weight);
                    if (seen) p = weight;
                    __syncwarp();
                    if (lane == 0) row_max[r] = new_max, row_sum[r] = sum;
                }
                if (lane == 0) row_scale[r] = rescale;
            }
            weights[r * SP + lane] = p;
        }
        __syncthreads();
        if (quad < dv) {
            if (!sigmoid) {
#pragma unroll
                for (int i = 0; i < HELD; ++i) {
                    const float f = row_scale[held0 + i];
                    acc[i].x *= f, acc[i].y *= f, acc[i].z *= f, acc[i].w *= f;
                }
            }
            const float* v_tile = values + buffer * 32 * v_pitch + quad;
#pragma unroll 2
            for (int j = 0; j < 32; j += 4) {
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(v_tile + (j + u) * v_pitch);
#pragma unroll
                for (int i = 0; i < HELD; ++i) {
                    const float4 w4 = *reinterpret_cast<const float4*>(weights + (held0 + i) * SP + j);
                    const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (!whole && __float_as_uint(w[u]) == UNSEEN) continue;
                        acc[i].x = fmaf(w[u], v[u].x, acc[i].x);
                        acc[i].y = fmaf(w[u], v[u].y, acc[i].y);
                        acc[i].z = fmaf(w[u], v[u].z, acc[i].z);
                        acc[i].w = fmaf(w[u], v[u].w, acc[i].w);
                    }
                }
            }
        }
        __syncthreads();  // the next copies overwrite this buffer
    }
    cp_async_wait<0>();
    if (quad >= dv) return;
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        const int r = held0 + i;
        if (r >= live) break;
        const int token = begin + (row0 + r) / group, head = kv * group + (row0 + r) % group;
        float denom = row_sum[r];
        if (a.sink) denom += expf((a.sink_values ? a.sink_values[head] : 0.0f) - row_max[r]);  // the silent participant
        float inv = sigmoid ? 1.0f : 1.0f / denom;
        const size_t at = static_cast<size_t>(token) * a.heads + head;
        if (a.gate && a.gate_width == 1) inv *= a.gate[at];
        float4 y = make_float4(acc[i].x * inv, acc[i].y * inv, acc[i].z * inv, acc[i].w * inv);
        if (a.gate && a.gate_width > 1) {
            const float* g = a.gate + at * a.gate_width + quad;
            y.x *= g[0], y.y *= g[1], y.z *= g[2], y.w *= g[3];
        }
        *reinterpret_cast<float4*>(static_cast<float*>(a.out) + at * dv + quad) = y;
    }
}

// ------------------------------------------------------------------ float32, few rows an entry (decoded tokens)
//
// The same bits for entries of at most 16 (token, head) rows per KV head, in two kernels.  In the kernel above such an entry is one block, whose tiles
// follow each other: a tile of 32 keys takes the latency of a chain over the head, of a softmax and of a chain over its keys, 4 us
// at heads of 128 and 11 over latent rows of 576, while most SMs are idle.  Only what a row's order of operations demands is serial here:
// the scores of all tiles are independent (first kernel, a block to a tile), a tile's maximum needs its own scores, its weights the
// running maximum, and the chains over the keys are separate for every value element (second kernel, a block to 64 value columns).
// Eight decoded tokens, us, the kernel above | these two: 16 heads in 8 KV heads of 128 behind 512 68 | 38, behind 2,048 250 | 114; 16 heads over
// latent rows of 576 with 512 values 176 | 69 and 666 | 220.  Of the 114 the second kernel takes 76: a step of four tiles takes the
// latencies of its softmax and of 128 keys' chain, 5 us, in blocks of eight warps of which few are resident.  More entries, and where the one kernel
// is faster: ops.few_rows_pay.
constexpr int FEW_ROWS = 16, FEW_TILES = 4, FEW_KEYS = 32 * FEW_TILES, FEW_COLUMNS = 64;  // rows of a block; tiles and keys of a step of the second kernel

struct FewRows {
    const AttnArgs& a;
    int begin, rows, group, kv, lowest, last, tile0;  // of the block's entry and KV head
    __device__ FewRows(const RowArgs& m, int entry, int kv_head) : a(m.a), group(m.a.heads / m.a.kv_heads), kv(kv_head) {
        begin = m.cu_tokens[entry];
        rows = (m.cu_tokens[entry + 1] - begin) * group;
        if (rows <= 0) return;
        lowest = lowest_of(position_of(0)), last = position_of(rows - 1);
        tile0 = lowest / 32 * 32;
    }
    __device__ int position_of(int r) const { return a.positions[begin + r / group]; }
    __device__ int head_of(int r) const { return kv * group + r % group; }
    __device__ size_t item_of(int r) const { return static_cast<size_t>(begin + r / group) * a.heads + head_of(r); }
    __device__ int lowest_of(int position) const {
        const int low = a.window > 0 ? max(position - a.window + 1, 0) : 0;
        return a.chunk > 0 ? max(low, position / a.chunk * a.chunk) : low;
    }
    __device__ int page_of(const int* table, int key) const { return key >= lowest && key <= last ? table[key / a.page_size] : -1; }
    __device__ size_t cached_row(int page, int key) const { return (static_cast<size_t>(page) * a.kv_heads + kv) * a.page_size + key % a.page_size; }
};

// scores[token][head][key - tile0] = q . k, for the tiles blockIdx.x, + gridDim.x, ... of the entry.
__global__ void __launch_bounds__(ROW_THREADS) few_rows_scores_kernel(RowArgs m, float* scores, int capacity) {
    extern __shared__ __align__(16) float few_shared[];
    const AttnArgs& a = m.a;
    const int d = a.head_dim, kp = d + 4;
    float *q = few_shared, *keys = q + FEW_ROWS * kp;  // [FEW_ROWS][kp], [32][kp]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    pdl_wait();
    const FewRows e(m, blockIdx.z, blockIdx.y);
    if (e.rows <= 0 || e.tile0 + 32 * static_cast<int>(blockIdx.x) > e.last) return;
    const int* table = a.block_table + static_cast<size_t>(blockIdx.z) * a.table_width;
    for (int i = tid; i < e.rows * (d / 4); i += ROW_THREADS) {
        const int r = i / (d / 4), x = i % (d / 4) * 4;
        *reinterpret_cast<float4*>(q + r * kp + x) = *reinterpret_cast<const float4*>(static_cast<const float*>(a.q) + e.item_of(r) * d + x);
    }
    for (int tile = e.tile0 + 32 * blockIdx.x; tile <= e.last; tile += 32 * gridDim.x) {
        __syncthreads();  // the keys of the tile before are read
        const int key = tile + (tid >> 3), page = e.page_of(table, key);
        const float* from = static_cast<const float*>(a.k_pages) + (page >= 0 ? e.cached_row(page, key) * d : 0);
        for (int x = (tid & 7) * 4; x < d; x += 32) cp_async_16(keys + (tid >> 3) * kp + x, from + x, page >= 0);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        for (int r = warp; r < e.rows; r += 2 * (ROW_THREADS / 32)) {  // a key to a lane, two rows at a time
            const int other = r + ROW_THREADS / 32 < e.rows ? r + ROW_THREADS / 32 : r;
            const float *k = keys + lane * kp, *q0 = q + r * kp, *q1 = q + other * kp;
            float dot0 = 0.0f, dot1 = 0.0f;
#pragma unroll 8
            for (int x = 0; x < d; x += 4) {
                const float4 kk = *reinterpret_cast<const float4*>(k + x), u = *reinterpret_cast<const float4*>(q0 + x), v = *reinterpret_cast<const float4*>(q1 + x);
                dot0 = fmaf(u.x, kk.x, dot0), dot1 = fmaf(v.x, kk.x, dot1);
                dot0 = fmaf(u.y, kk.y, dot0), dot1 = fmaf(v.y, kk.y, dot1);
                dot0 = fmaf(u.z, kk.z, dot0), dot1 = fmaf(v.z, kk.z, dot1);
                dot0 = fmaf(u.w, kk.w, dot0), dot1 = fmaf(v.w, kk.w, dot1);
            }
            scores[e.item_of(r) * capacity + (tile - e.tile0) + lane] = dot0;
            scores[e.item_of(other) * capacity + (tile - e.tile0) + lane] = dot1;
        }
    }
}

// Softmax and values of 64 value columns.  A step is four tiles: every (row, tile) gets a warp of its own for the scores' maximum and, with the
// running maximum known, for the weights; then a thread adds a quad of columns of one row up over the step's keys.
__global__ void __launch_bounds__(ROW_THREADS) few_rows_values_kernel(RowArgs m, const float* scores, int capacity) {
    extern __shared__ __align__(16) float few_values[];
    float(*values)[FEW_KEYS][FEW_COLUMNS] = reinterpret_cast<float(*)[FEW_KEYS][FEW_COLUMNS]>(few_values);  // [2]
    __shared__ __align__(16) float weights[FEW_ROWS][FEW_KEYS];
    __shared__ float tile_max[FEW_ROWS][FEW_TILES], tile_sum[FEW_ROWS][FEW_TILES], tile_scale[FEW_ROWS][FEW_TILES], row_max[FEW_ROWS], row_sum[FEW_ROWS];
    __shared__ int key_there[2][FEW_KEYS];
    const AttnArgs& a = m.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, column0 = blockIdx.x * FEW_COLUMNS, columns = min(FEW_COLUMNS, a.value_dim - column0);
    pdl_trigger();
    pdl_wait();
    const FewRows e(m, blockIdx.z, blockIdx.y);
    if (e.rows <= 0) return;
    const int* table = a.block_table + static_cast<size_t>(blockIdx.z) * a.table_width;
    const bool sigmoid = a.sigmoid_bias != nullptr;
    if (tid < FEW_ROWS) row_max[tid] = -INFINITY, row_sum[tid] = 0.0f;
    auto fetch = [&](int first, int buffer) {  // two threads to a key
        const int j = tid >> 1, key = first + j, page = e.page_of(table, key);
        const float* from = static_cast<const float*>(a.v_pages) + (page >= 0 ? e.cached_row(page, key) * a.value_stride + column0 : 0);
        for (int x = (tid & 1) * 4; x < columns; x += 8) cp_async_16(&values[buffer][j][x], from + x, page >= 0);
        if ((tid & 1) == 0) key_there[buffer][j] = page >= 0;
        cp_async_commit();
    };
    const int my_row = tid / (FEW_COLUMNS / 4), quad = tid % (FEW_COLUMNS / 4) * 4;
    const bool adds = my_row < e.rows && quad < columns;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int buffer = 0;
    fetch(e.tile0, 0);
    for (int first = e.tile0; first <= e.last; first += FEW_KEYS, buffer ^= 1) {
        if (first + FEW_KEYS <= e.last) fetch(first + FEW_KEYS, buffer ^ 1);
        else cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        for (int i = warp; i < e.rows * FEW_TILES; i += ROW_THREADS / 32) {
            const int r = i / FEW_TILES, t = i % FEW_TILES, key = first + 32 * t + lane, position = e.position_of(r), head = e.head_of(r);
            const bool seen = key_there[buffer][32 * t + lane] != 0 && key >= e.lowest_of(position) && key <= position;
            float score = -INFINITY;
            if (seen) {
                score = scores[e.item_of(r) * capacity + (key - e.tile0)] * a.scale;
                if (a.softcap > 0.0f) score = a.softcap * tanhf(score / a.softcap);
                if (a.slopes) score -= a.slopes[head] * static_cast<float>(position - key);
            }
            if (sigmoid) {
                weights[r][32 * t + lane] = seen ? 1.0f / (1.0f + expf(-(score + a.sigmoid_bias[head]))) : __uint_as_float(UNSEEN);
            } else {
                weights[r][32 * t + lane] = seen ? score : __uint_as_float(UNSEEN);
                const float best = warp_max(score);
                if (lane == 0) tile_max[r][t] = best;
            }
            const unsigned mask = __ballot_sync(0xffffffffu, seen);
            if (lane == 0) tile_sum[r][t] = __uint_as_float(mask);  // which keys the row sees, until the sums take its place
        }
        __syncthreads();
        if (!sigmoid) {
            for (int i = warp; i < e.rows * FEW_TILES; i += ROW_THREADS / 32) {
                const int r = i / FEW_TILES, t = i % FEW_TILES;
                float old_max = row_max[r];
                for (int before = 0; before < t; ++before) old_max = fmaxf(old_max, tile_max[r][before]);
                const float new_max = fmaxf(old_max, tile_max[r][t]);
                float rescale = 1.0f, sum = 0.0f;
                if (new_max != -INFINITY) {  // uniform across the warp
                    const bool seen = __float_as_uint(tile_sum[r][t]) >> lane & 1;
                    rescale = expf(old_max - new_max);
                    const float weight = seen ? expf(weights[r][32 * t + lane] - new_max) : 0.0f;
                    sum = warp_sum(weight);
                    if (seen) weights[r][32 * t + lane] = weight;
                } else {
                    weights[r][32 * t + lane] = __uint_as_float(UNSEEN);
                }
                __syncwarp();
                if (lane == 0) tile_scale[r][t] = rescale, tile_sum[r][t] = sum;
            }
            __syncthreads();
            if (tid < e.rows) {
                float best = row_max[tid], sum = row_sum[tid];
                for (int t = 0; t < FEW_TILES; ++t) {
                    best = fmaxf(best, tile_max[tid][t]);
                    if (best != -INFINITY) sum = sum * tile_scale[tid][t] + tile_sum[tid][t];
                }
                row_max[tid] = best, row_sum[tid] = sum;
            }
        }
        if (adds) {
            for (int t = 0; t < FEW_TILES; ++t) {
                if (!sigmoid) {
                    const float f = tile_scale[my_row][t];
                    acc.x *= f, acc.y *= f, acc.z *= f, acc.w *= f;
                }
#pragma unroll 8
                for (int j = 32 * t; j < 32 * t + 32; ++j) {
                    const float w = weights[my_row][j];
                    const float4 v = *reinterpret_cast<const float4*>(&values[buffer][j][quad]);
                    if (__float_as_uint(w) == UNSEEN) continue;
                    acc.x = fmaf(w, v.x, acc.x), acc.y = fmaf(w, v.y, acc.y), acc.z = fmaf(w, v.z, acc.z), acc.w = fmaf(w, v.w, acc.w);
                }
            }
        }
        __syncthreads();  // the next copies overwrite this buffer, the next step the weights
    }
    cp_async_wait<0>();
    if (!adds) return;
    const int head = e.head_of(my_row);
    float denom = row_sum[my_row];
    if (a.sink) denom += expf((a.sink_values ? a.sink_values[head] : 0.0f) - row_max[my_row]);  // the silent participant
    float inv = sigmoid ? 1.0f : 1.0f / denom;
    const size_t at = e.item_of(my_row);
    if (a.gate && a.gate_width == 1) inv *= a.gate[at];
    float4 y = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    if (a.gate && a.gate_width > 1) {
        const float* g = a.gate + at * a.gate_width + column0 + quad;
        y.x *= g[0], y.y *= g[1], y.z *= g[2], y.w *= g[3];
    }
    *reinterpret_cast<float4*>(static_cast<float*>(a.out) + at * a.value_dim + column0 + quad) = y;
}

static size_t rows_shared_bytes(const AttnArgs& a, int rows) {
    const size_t kp = a.head_dim + 4, vp = a.k_pages == a.v_pages ? 0 : a.value_dim + 4;
    return (rows * kp + 64 * (kp + vp) + static_cast<size_t>(rows) * 36) * sizeof(float);
}

// Against one warp per (token, head), a prompt of 512 tokens, 16 heads of 128 in 8 KV heads: 1,361 -> 165 us; 256 tokens, 32
// heads: 826 -> 143; eight decoded tokens behind 17 to 512 (which now take the two kernels above): 768 -> 68, over latent rows of 576 with 512
// values 768 -> 179 us.
template <int R, int QP>
static int launch_rows(const RowArgs& m, int entries, int longest, cudaStream_t stream) {
    static SharedMemoryOptIn opt_in;
    if (const int e = opt_in(paged_attention_rows_kernel<R, QP>, 200 * 1024)) return e;
    const int group = m.a.heads / m.a.kv_heads;
    const long long blocks = (static_cast<long long>(longest) * group + R - 1) / R;
    if (blocks > 0x7fffffffll || m.a.kv_heads > 65535 || entries > 65535) return ME_ERR_UNSUPPORTED;
    return launch_kernel(paged_attention_rows_kernel<R, QP>, dim3(static_cast<unsigned>(blocks), m.a.kv_heads, entries), ROW_THREADS,
                         rows_shared_bytes(m.a, R), stream, m);
}

template <int R>
static int launch_rows_of(const RowArgs& m, int entries, int longest, cudaStream_t stream) {
    if (m.a.value_dim <= 64) return launch_rows<R, 16>(m, entries, longest, stream);
    if (m.a.value_dim <= 128) return launch_rows<R, 32>(m, entries, longest, stream);
    if (m.a.value_dim <= 256) return launch_rows<R, 64>(m, entries, longest, stream);
    return launch_rows<R, 128>(m, entries, longest, stream);
}

// Whether the kernel takes these sizes (float32; everything else takes the one above): rows of whole 16-byte pieces, and 16 rows'
// queries, weights and two tiles in shared memory.
ME_EXPORT int me_paged_attention_rows_supports(int head_dim, int value_dim, int value_stride, int values_in_keys) {
    AttnArgs a = {};
    a.head_dim = head_dim, a.value_dim = value_dim, a.value_stride = value_stride;
    a.v_pages = values_in_keys ? nullptr : &a;  // compared with k_pages, not read
    return head_dim >= 4 && head_dim % 4 == 0 && value_dim >= 4 && value_dim % 4 == 0 && value_dim <= 32 * MAX_DIM_PER_LANE &&
           value_stride % 4 == 0 && rows_shared_bytes(a, 16) <= 200 * 1024;
}

// The attention of me_paged_attention_generic in float32, with its bits.  The tokens of entry e are cu_tokens[e] ..
// cu_tokens[e + 1], in ascending position; no entry has more than `longest`.  With `scores` (room for tokens x heads x `capacity`
// floats, a multiple of 32 that no entry's visible keys, from their tile's start on, pass) entries of at most 16 rows take the two kernels for few rows.
ME_EXPORT int me_paged_attention_rows(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                      const int* cu_tokens, const int* positions, void* out, float scale, int entries, int longest,
                                      int heads, int kv_heads, int head_dim, int page_size, int table_width, int window,
                                      int value_dim, int sink, const float* gate, int gate_width, int value_stride,
                                      const float* slopes, const float* sink_values, float softcap, int chunk,
                                      const float* sigmoid_bias, float* scores, int capacity, cudaStream_t stream) {
    if (entries <= 0 || longest <= 0) return 0;
    if (gate && gate_width != 1 && gate_width != value_dim) return ME_ERR_ARGUMENT;
    if (value_stride < value_dim || chunk < 0 || (sigmoid_bias && sink)) return ME_ERR_ARGUMENT;
    if (heads < 1 || kv_heads < 1 || heads % kv_heads || !me_paged_attention_rows_supports(head_dim, value_dim, value_stride, k_pages == v_pages)) return ME_ERR_UNSUPPORTED;
    for (const void* p : {q, k_pages, v_pages, static_cast<const void*>(out)})
        if (reinterpret_cast<uintptr_t>(p) % 16) return ME_ERR_UNSUPPORTED;
    RowArgs m{{q, k_pages, v_pages, block_table, nullptr, positions, out, scale, 0, heads, kv_heads, head_dim, page_size,
               table_width, window, value_dim, sink, gate, gate_width, value_stride, slopes, sink_values, softcap, chunk, sigmoid_bias},
              cu_tokens};
    // 64 rows share a key where an entry brings that many; else 16, whose tiles take a third of the time.  Two blocks of
    // 64 rows fit an SM up to heads of 128.
    const long long rows = static_cast<long long>(longest) * (heads / kv_heads);
    if (scores != nullptr) {
        const size_t bytes = (FEW_ROWS + 32) * static_cast<size_t>(head_dim + 4) * sizeof(float);
        if (rows > FEW_ROWS || capacity < 32 || capacity % 32 || kv_heads > 65535 || entries > 65535 || bytes > 200 * 1024) return ME_ERR_ARGUMENT;
        static SharedMemoryOptIn opt_in, values_opt_in;
        if (const int e = opt_in(few_rows_scores_kernel, 200 * 1024)) return e;
        if (const int e = values_opt_in(few_rows_values_kernel, 2 * FEW_KEYS * FEW_COLUMNS * sizeof(float))) return e;
        const int tiles = capacity / 32 < 64 ? capacity / 32 : 64;
        if (const int e = launch_kernel(few_rows_scores_kernel, dim3(tiles, kv_heads, entries), ROW_THREADS, bytes, stream, m, scores, capacity)) return e;
        return launch_kernel(few_rows_values_kernel, dim3((value_dim + FEW_COLUMNS - 1) / FEW_COLUMNS, kv_heads, entries), ROW_THREADS,
                             2 * FEW_KEYS * FEW_COLUMNS * sizeof(float), stream, m, scores, capacity);
    }
    if (rows > 32 && rows_shared_bytes(m.a, 64) <= 113 * 1024) return launch_rows_of<64>(m, entries, longest, stream);
    return launch_rows_of<16>(m, entries, longest, stream);
}

ME_EXPORT int me_paged_attention_generic(const void* q, const void* k_pages, const void* v_pages,
                                         const int* block_table, const int* entry_of_token,
                                         const int* positions, void* out, int type, float scale, int tokens,
                                         int heads, int kv_heads, int head_dim, int page_size, int table_width,
                                         int window, int value_dim, int sink, const float* gate, int gate_width,
                                         int value_stride, const float* slopes, const float* sink_values,
                                         float softcap, int chunk, const float* sigmoid_bias, cudaStream_t stream) {
    if (tokens <= 0) return 0;
    if (gate && gate_width != 1 && gate_width != value_dim) return ME_ERR_ARGUMENT;
    if (value_stride < value_dim || chunk < 0 || (sigmoid_bias && sink)) return ME_ERR_ARGUMENT;
    if (head_dim > MAX_KEY_DIM || value_dim < 1 || value_dim > 32 * MAX_DIM_PER_LANE || heads % kv_heads)
        return ME_ERR_UNSUPPORTED;
    AttnArgs a{q, k_pages, v_pages, block_table, entry_of_token, positions, out, scale,
               tokens, heads, kv_heads, head_dim, page_size, table_width, window, value_dim, sink, gate,
               gate_width, value_stride, slopes, sink_values, softcap, chunk, sigmoid_bias};
    const long long items = static_cast<long long>(tokens) * heads;
    const int blocks = static_cast<int>((items + ATTN_WARPS - 1) / ATTN_WARPS);
    const size_t smem = static_cast<size_t>(ATTN_WARPS) * head_dim * sizeof(float);
    if (type == ME_BF16)
        return launch_kernel(paged_attention_generic_kernel<__nv_bfloat16>, blocks, ATTN_WARPS * 32, smem, stream, a);
    return launch_kernel(paged_attention_generic_kernel<float>, blocks, ATTN_WARPS * 32, smem, stream, a);
}
