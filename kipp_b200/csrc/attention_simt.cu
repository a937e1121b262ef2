// Causal grouped-query attention over the paged cache on the CUDA cores, for
// any mix of prompt portions and single decoded tokens.
//
// This is the attention of the true 32-bit path and the fallback of the
// bfloat16 path for head sizes the tensor-core kernels refuse.  Reference
// counterpart: cached_gqa_kernel (cuda/kipp_kernels.cu:160), formula
// src/kipp.c:2882-2922: s_j = (q . k_j) / sqrt(head_dim) for the keys j the
// query may see, softmax with the maximum subtracted, o = sum_j p_j v_j, the
// kv head of query head h being h / (n_q / n_kv).
//
// A block handles one token and the query heads of one kv head (at most MAX_HEADS of them), a warp
// one query head.  Keys are walked in tiles of 32 aligned to absolute positions, one key per lane, with a
// running maximum and sum (all float32).  The order of every sum depends only on the token's own
// position and window, never on the batch it is in.
//
// The tiles go through shared memory, the next one on its way while the present one is worked on: a
// lane that walks its own key row in global memory waits a trip to the L2 for every few values, and every
// head of a group fetched the same rows (four layers of 16 heads of 128 over prompts of 400 tokens and eight steps
// of three tokens: 36 launches in 10.6 ms, 1.35 with two stages, 1.63 while each 16 bytes copied looked its page up).  What bounds it
// now is the chain of head_dim FMAs per key tile and the 32 weighted rows after it.
//
// A window of w (0 = none) lets position p see keys j with p - w < j <= p.
#include "common.cuh"
#include <math.h>
#include <algorithm>

namespace {
constexpr int MAX_ACC = 8;         // head_dim <= 256
constexpr int MAX_HEADS = 8;       // query heads (warps) of a block
constexpr int TILE = 32;           // keys of a tile: one per lane

// Bytes of a row of a tile: padded so that 32 lanes reading 16 bytes of 32 rows meet every bank.
template <typename T> __host__ __device__ inline int tile_row_bytes(int head_dim) {
    return (head_dim * (int)sizeof(T) + 15) / 16 * 16 + 16;
}

// 16 bytes of a key row against the query, in the order of the elements.
__device__ __forceinline__ float dot16(const float* q, const float* k, float dot) {
    const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(k);
    dot = fmaf(a.x, b.x, dot);
    dot = fmaf(a.y, b.y, dot);
    dot = fmaf(a.z, b.z, dot);
    return fmaf(a.w, b.w, dot);
}
__device__ __forceinline__ float dot16(const float* q, const bf16* k, float dot) {
    const uint4 raw = *reinterpret_cast<const uint4*>(k);
    const bf16* b = reinterpret_cast<const bf16*>(&raw);
    const float4 lo = *reinterpret_cast<const float4*>(q), hi = *reinterpret_cast<const float4*>(q + 4);
    const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) dot = fmaf(a[i], to_f32(b[i]), dot);
    return dot;
}

// VEC: rows of whole 16-byte pieces that start on 16 bytes, moved by asynchronous copies; else element by element.
// NACC: head_dim <= 32 NACC.
template <typename T, bool VEC, int NACC>
__global__ void __launch_bounds__(MAX_HEADS * 32)
paged_attention_simt_kernel(T* __restrict__ out, const T* __restrict__ q,
                            const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                            const int* __restrict__ positions, const int* __restrict__ entry_of_token,
                            const int* __restrict__ block_table, int table_width, int page_size,
                            int n_q, int n_kv, int head_dim, float scale, int window, int stages, int* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t smem[];   // q [warps][head_dim padded], then the stages, a key and a value tile each
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int group = n_q / n_kv, parts = (group + warps - 1) / warps;
    const int t = (int)(blockIdx.x / (unsigned)(n_kv * parts)), rest = (int)(blockIdx.x % (unsigned)(n_kv * parts));
    const int g = rest / parts, in_group = (rest % parts) * warps + warp;
    const bool live = in_group < group;               // the last block of a group may have warps left over
    const int h = g * group + min(in_group, group - 1);
    const int pos = positions[t];
    const int e = entry_of_token[t];
    const int* table = block_table + (size_t)e * table_width;
    const int first = window > 0 ? max(0, pos - window + 1) : 0;
    const int row_bytes = tile_row_bytes<T>(head_dim), q_stride = (head_dim + 3) & ~3;
    uint8_t* tiles = smem + (size_t)warps * q_stride * 4;

    float* qs = reinterpret_cast<float*>(smem) + warp * q_stride;
    const T* qrow = q + ((size_t)t * n_q + h) * head_dim;
    for (int i = lane; i < head_dim; i += 32) qs[i] = to_f32(qrow[i]);

    // the page row of key j of kv head g, or null: outside what the token sees, or not mapped
    auto row_of = [&](int j) -> long long {
        if (j < first || j > pos) return -1;
        const int page = j / page_size < table_width ? table[j / page_size] : -1;
        return page < 0 ? -2 : (((long long)page * n_kv + g) * page_size + (j % page_size)) * head_dim;
    };
    // a warp copies whole rows, every `warps`-th of the tile; `rows`: this lane's key's page row, looked up once a tile
    auto fetch = [&](long long rows, int stage) {
        uint8_t* kt = tiles + (size_t)stage * 2 * TILE * row_bytes;
        uint8_t* vt = kt + (size_t)TILE * row_bytes;
        for (int key = warp; key < TILE; key += warps) {
            const long long row = __shfl_sync(0xffffffffu, rows, key);
            if (VEC) {
                const int bytes = row < 0 ? 0 : 16;
                const size_t off = row < 0 ? 0 : (size_t)row * sizeof(T);
                for (int at = lane * 16; at < head_dim * (int)sizeof(T); at += 512) {
                    cp_async16(smem_address(kt + key * row_bytes + at), (const uint8_t*)k_pages + off + (row < 0 ? 0 : at), bytes);
                    cp_async16(smem_address(vt + key * row_bytes + at), (const uint8_t*)v_pages + off + (row < 0 ? 0 : at), bytes);
                }
            } else {
                for (int at = lane; at < head_dim; at += 32) {
                    reinterpret_cast<T*>(kt + key * row_bytes)[at] = row < 0 ? from_f32<T>(0.f) : k_pages[row + at];
                    reinterpret_cast<T*>(vt + key * row_bytes)[at] = row < 0 ? from_f32<T>(0.f) : v_pages[row + at];
                }
            }
        }
        cp_async_commit();
    };

    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;

    const int begin = (first / TILE) * TILE;
    long long row_next = row_of(begin + lane);
    fetch(row_next, 0);
    int stage = 0;
    for (int j0 = begin; j0 <= pos; j0 += TILE, stage ^= stages - 1) {
        const long long row = row_next;
        const bool more = j0 + TILE <= pos;
        if (more) row_next = row_of(j0 + TILE + lane);
        if (stages == 1) {
            cp_async_wait<0>();
        } else {
            if (more) fetch(row_next, stage ^ 1);
            else cp_async_commit();
            cp_async_wait<1>();
        }
        __syncthreads();
        const uint8_t* kt = tiles + (size_t)stage * 2 * TILE * row_bytes;
        const uint8_t* vt = kt + (size_t)TILE * row_bytes;
        if (row == -2) atomicExch(status, 3);         // a needed key is not mapped
        float s = -INFINITY;
        if (row >= 0) {
            const T* krow = reinterpret_cast<const T*>(kt + lane * row_bytes);
            float dot = 0.f;
            if (VEC) {
#pragma unroll 8
                for (int d = 0; d < head_dim; d += 16 / (int)sizeof(T)) dot = dot16(qs + d, krow + d, dot);
            } else {
                for (int d = 0; d < head_dim; ++d) dot = fmaf(qs[d], to_f32(krow[d]), dot);
            }
            s = dot * scale;
        }
        const float tile_max = warp_max(s);
        const float m_new = fmaxf(m, tile_max);
        if (m_new != -INFINITY) {                      // something is visible
            const float p = (s == -INFINITY) ? 0.f : expf(s - m_new);
            const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
            l = l * corr + warp_sum(p);
#pragma unroll
            for (int i = 0; i < NACC; ++i) acc[i] *= corr;
            m = m_new;
            const unsigned seen = __ballot_sync(0xffffffffu, row >= 0);
#pragma unroll 8
            for (int jj = 0; jj < TILE; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, p, jj);
                if (!(seen >> jj & 1u)) continue;
                const T* vr = reinterpret_cast<const T*>(vt + jj * row_bytes);
#pragma unroll
                for (int i = 0; i < NACC; ++i) {
                    const int d = lane + 32 * i;
                    if (d < head_dim) acc[i] = fmaf(pj, to_f32(vr[d]), acc[i]);
                }
            }
        }
        __syncthreads();                              // the tile is read: its place may be filled again
        if (stages == 1 && more) fetch(row_next, 0);
    }
    cp_async_wait<0>();
    if (!live) return;
    T* orow = out + ((size_t)t * n_q + h) * head_dim;
    const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
    for (int i = 0; i < NACC; ++i) {
        const int d = lane + 32 * i;
        if (d < head_dim) orow[d] = from_f32<T>(acc[i] * inv);
    }
}

// ---------------------------------------------------------------------------------------
// The same for few blocks, where a block's chain of tiles is what the launch lasts: FEW_TILES tiles at a time and what of
// them depends on nothing else side by side.  A warp scores a tile for every fourth head of the block (as many chains of FMAs
// as it has heads, a key's 16 bytes read once for all of them); the tiles' maxima meet in shared memory, which gives each
// tile the running maximum it has in the order of the tiles, and so its weights; then a thread per value of the
// result walks the keys.  Every sum has the terms and the order it has in the kernel above: the same bits.  What is left of a
// chain is a head's FMAs once per FEW_TILES tiles and one FMA per key.  The next tiles' keys travel beside the weighted
// sums, their values beside the scores, and the first ones before the dependency wait where the caller says that they are
// there (`early`).  Bound by the instructions of a block's
// warps, one after the other: 3 tokens of up to 211 keys, 16 heads of 128: 11.5 us a launch, 35 in the kernel above.
constexpr int FEW_TILES = 4, FEW_KEYS = FEW_TILES * TILE, FEW_THREADS = 512, FEW_WARPS = FEW_THREADS / 32;
struct FewStats {
    float tile_max[MAX_HEADS][FEW_TILES], running[MAX_HEADS][FEW_TILES], sum[MAX_HEADS][FEW_TILES];
    unsigned seen[FEW_TILES];
    long long rows[FEW_KEYS];
    int own[FEW_WARPS];          // by warp: the first position of the entry's tokens in this step
};
// heads of the block at most 4 NH; NACC as above: a thread's value is number tid % (32 NACC) of heads tid / (32 NACC), + HEAD_STEP, ...
template <typename T, int NACC, int NH>
__global__ void __launch_bounds__(FEW_THREADS, 1)
paged_attention_few_kernel(T* __restrict__ out, const T* __restrict__ q, const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                           const int* __restrict__ positions, const int* __restrict__ entry_of_token, const int* __restrict__ block_table,
                           int table_width, int page_size, int n_q, int n_kv, int head_dim, float scale, int window, int block_heads,
                           bool early, int* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t smem[];   // q [heads][head_dim padded], weights [heads][FEW_KEYS], keys, values
    __shared__ FewStats st;
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = n_q / n_kv, parts = (group + block_heads - 1) / block_heads;
    const int t = (int)(blockIdx.x / (unsigned)(n_kv * parts)), rest = (int)(blockIdx.x % (unsigned)(n_kv * parts));
    const int g = rest / parts, h0 = (rest % parts) * block_heads, heads = min(block_heads, group - h0);
    const int pos = positions[t];                     // (the step's lists)
    const int* table = block_table + (size_t)entry_of_token[t] * table_width;
    const int first = window > 0 ? max(0, pos - window + 1) : 0, begin = first / TILE * TILE;
    const int row_bytes = tile_row_bytes<T>(head_dim), q_stride = (head_dim + 3) & ~3;
    float* qs = reinterpret_cast<float*>(smem);
    float* weights = qs + (size_t)block_heads * q_stride;
    uint8_t* kt = reinterpret_cast<uint8_t*>(weights + (size_t)block_heads * FEW_KEYS);
    uint8_t* vt = kt + (size_t)FEW_KEYS * row_bytes;

    // the page rows of FEW_KEYS keys from j0 on: -1 outside what the token sees, -2 not mapped
    auto look_up = [&](int j0) {
        if (tid < FEW_KEYS) {
            const int j = j0 + tid;
            long long row = -1;
            if (j >= first && j <= pos) {
                const int page = j / page_size < table_width ? table[j / page_size] : -1;
                row = page < 0 ? -2 : (((long long)page * n_kv + g) * page_size + (j % page_size)) * head_dim;
            }
            st.rows[tid] = row;
        }
    };
    // a warp takes whole rows; of keys [from, to) of the FEW_KEYS
    auto fetch = [&](const T* pages, uint8_t* tile, int from, int to) {
        for (int key = from + warp; key < to; key += FEW_WARPS) {
            const long long row = st.rows[key];
            const uint32_t dst = smem_address(tile + key * row_bytes);
            const uint8_t* src = (const uint8_t*)pages + (row < 0 ? 0 : (size_t)row * sizeof(T));
            for (int at = lane * 16; at < head_dim * (int)sizeof(T); at += 512) cp_async16(dst + at, src + (row < 0 ? 0 : at), row < 0 ? 0 : 16);
        }
    };
    auto whole_tiles = [&](int j0) { return min(FEW_KEYS, (pos - j0) / TILE * TILE + TILE); };     // keys of the tiles from j0 on
    // With `early` the first keys and values come before the dependency wait, all but those of this step's own tokens: the
    // entry's tokens up to this one, which follow one another.
    look_up(begin);
    if (early) {                                      // (a thread per token; walking back one by one, 148 tokens of one entry: 26.8 us, 15.3 so)
        int own = pos;
        for (int u = tid; u < t; u += FEW_THREADS)
            if (entry_of_token[u] == entry_of_token[t]) own = min(own, positions[u]);
        own = __reduce_min_sync(0xffffffffu, own);
        if (lane == 0) st.own[warp] = own;
    }
    __syncthreads();
    int own = early ? pos : 0;
    for (int w = 0; early && 32 * w < t && w < FEW_WARPS; ++w) own = min(own, st.own[w]);
    const int n_first = whole_tiles(begin), kept = min(max(own - begin, 0), n_first);
    fetch(k_pages, kt, 0, kept);
    fetch(v_pages, vt, 0, kept);
    pdl_wait();
    fetch(k_pages, kt, kept, n_first);
    cp_async_commit();
    fetch(v_pages, vt, kept, n_first);
    cp_async_commit();
    const T* q_rows = q + ((size_t)t * n_q + g * group + h0) * head_dim;
    for (int i = tid; i < heads * head_dim; i += FEW_THREADS) qs[i / head_dim * q_stride + i % head_dim] = to_f32(q_rows[i]);

    constexpr int VALUES = 32 * NACC, HEAD_STEP = FEW_THREADS / VALUES, PER = (FEW_WARPS / FEW_TILES * NH + HEAD_STEP - 1) / HEAD_STEP;
    const int d = tid % VALUES, my_head = tid / VALUES;
    float acc[PER], m[PER], l[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) { acc[i] = 0.f; m[i] = -INFINITY; l[i] = 0.f; }
    float m_before[NH];                               // the scoring warps' running maxima
#pragma unroll
    for (int i = 0; i < NH; ++i) m_before[i] = -INFINITY;
    const int tile = warp & (FEW_TILES - 1), first_head = warp / FEW_TILES;
    constexpr int SCORE_STEP = FEW_WARPS / FEW_TILES;

    for (int j0 = begin; j0 <= pos; j0 += FEW_KEYS) {
        const int tiles = whole_tiles(j0) / TILE;
        cp_async_wait<1>();                           // the keys; the values may still be on their way
        __syncthreads();
        const long long row = st.rows[tile * TILE + lane];
        float s[NH];
#pragma unroll
        for (int i = 0; i < NH; ++i) s[i] = -INFINITY;
        if (tile < tiles) {
            if (row == -2) atomicExch(status, 3);     // a needed key is not mapped
            const T* krow = reinterpret_cast<const T*>(kt + (size_t)(tile * TILE + lane) * row_bytes);
            float dot[NH];
#pragma unroll
            for (int i = 0; i < NH; ++i) dot[i] = 0.f;
#pragma unroll 4
            for (int x = 0; x < head_dim; x += 16 / (int)sizeof(T))
#pragma unroll
                for (int i = 0; i < NH; ++i) dot[i] = dot16(qs + min(first_head + SCORE_STEP * i, heads - 1) * q_stride + x, krow + x, dot[i]);
#pragma unroll
            for (int i = 0; i < NH; ++i) {
                s[i] = row >= 0 ? dot[i] * scale : -INFINITY;
                const float most = warp_max(s[i]);
                if (lane == 0 && first_head + SCORE_STEP * i < heads) st.tile_max[first_head + SCORE_STEP * i][tile] = most;
            }
            const unsigned seen = __ballot_sync(0xffffffffu, row >= 0);
            if (lane == 0) st.seen[tile] = seen;
        }
        __syncthreads();
        const bool more = j0 + FEW_KEYS <= pos;
        if (more) look_up(j0 + FEW_KEYS);
#pragma unroll
        for (int i = 0; i < NH; ++i) {
            const int h = min(first_head + SCORE_STEP * i, heads - 1);
            float m_new = m_before[i];
            for (int x = 0; x < tiles; ++x) {
                m_before[i] = fmaxf(m_before[i], st.tile_max[h][x]);
                if (x <= tile) m_new = m_before[i];
            }
            const float p = m_new == -INFINITY || s[i] == -INFINITY ? 0.f : expf(s[i] - m_new);
            const float sum = warp_sum(p);
            if (tile < tiles && first_head + SCORE_STEP * i < heads) {
                weights[h * FEW_KEYS + tile * TILE + lane] = p;
                if (lane == 0) { st.sum[h][tile] = sum; st.running[h][tile] = m_new; }
            }
        }
        cp_async_wait<0>();                           // the values
        __syncthreads();
        if (more) fetch(k_pages, kt, 0, whole_tiles(j0 + FEW_KEYS));
        cp_async_commit();
        for (int x = 0; x < tiles; ++x) {
            const unsigned seen = st.seen[x];
            const float* p[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int h = min(my_head + HEAD_STEP * i, heads - 1);
                p[i] = weights + h * FEW_KEYS + x * TILE;
                const float m_new = st.running[h][x];
                if (m_new == -INFINITY) continue;     // nothing visible yet: the weights are 0
                const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
                l[i] = l[i] * corr + st.sum[h][x];
                acc[i] *= corr;
                m[i] = m_new;
            }
            const T* v = reinterpret_cast<const T*>(vt + (size_t)x * TILE * row_bytes) + min(d, head_dim - 1);
            const size_t pitch = (size_t)row_bytes / sizeof(T);
            if (seen == 0xffffffffu) {
#pragma unroll 4
                for (int jj = 0; jj < TILE; jj += 4) {
                    const float value[4] = {to_f32(v[jj * pitch]), to_f32(v[(jj + 1) * pitch]), to_f32(v[(jj + 2) * pitch]), to_f32(v[(jj + 3) * pitch])};
#pragma unroll
                    for (int i = 0; i < PER; ++i) {
                        const float4 w = *reinterpret_cast<const float4*>(p[i] + jj);
                        acc[i] = fmaf(w.w, value[3], fmaf(w.z, value[2], fmaf(w.y, value[1], fmaf(w.x, value[0], acc[i]))));
                    }
                }
            } else {
                for (int jj = 0; jj < TILE; ++jj) {
                    if (!(seen >> jj & 1u)) continue;
                    const float value = to_f32(v[jj * pitch]);
#pragma unroll
                    for (int i = 0; i < PER; ++i) acc[i] = fmaf(p[i][jj], value, acc[i]);
                }
            }
            // (where a head has seen nothing yet the tile counts for nothing, infinite values and all)
#pragma unroll
            for (int i = 0; i < PER; ++i)
                if (m[i] == -INFINITY) acc[i] = 0.f;
        }
        __syncthreads();                              // the values, weights and maxima are read
        if (more) fetch(v_pages, vt, 0, whole_tiles(j0 + FEW_KEYS));
        cp_async_commit();
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int h = my_head + HEAD_STEP * i;
        if (h < heads && d < head_dim)
            out[((size_t)t * n_q + g * group + h0 + h) * head_dim + d] = from_f32<T>(acc[i] * (l[i] > 0.f ? 1.0f / l[i] : 0.f));
    }
}

constexpr int SM_SMEM = 227 * 1024, SM_THREADS = 2048, SM_BLOCKS = 32;         // what an SM has for blocks

template <typename T, bool VEC, int NACC>
int launch(void* out, const void* q, const void* k_pages, const void* v_pages, const int* positions,
           const int* entry_of_token, const int* block_table, int table_width, int page_size, int tokens, int n_q,
           int n_kv, int head_dim, float scale, int window, bool early, int* status, cudaStream_t s) {
    const int group = n_q / n_kv, warps = group < MAX_HEADS ? group : MAX_HEADS;
    const long long blocks = (long long)tokens * n_kv * ((group + warps - 1) / warps);
    if (blocks > 0x7fffffffLL) return KIPP_ERR_ARG;
    if constexpr (VEC && NACC <= 4) {
        // a block for each SM at most: the chain of a block's tiles is all that counts
        if (blocks <= kipp_sm_count()) {
            const size_t few = ((size_t)warps * (((head_dim + 3) & ~3) + FEW_KEYS)) * 4 + (size_t)2 * FEW_KEYS * tile_row_bytes<T>(head_dim);
            const auto kernel = warps <= 4 ? paged_attention_few_kernel<T, NACC, 1> : paged_attention_few_kernel<T, NACC, 2>;
            if (const int e = kipp_allow_smem(kernel, few + sizeof(FewStats))) return e;      // (what it declares counts too)
            return kipp_launch(kernel, dim3((unsigned)blocks), dim3(FEW_THREADS), few, s, 1, (T*)out, (const T*)q, (const T*)k_pages,
                               (const T*)v_pages, positions, entry_of_token, block_table, table_width, page_size, n_q, n_kv, head_dim,
                               scale, window, warps, early, status);
        }
    }
    const size_t queries = (size_t)warps * ((head_dim + 3) & ~3) * 4, tiles = (size_t)2 * TILE * tile_row_bytes<T>(head_dim);
    // Two stages where every block is on an SM at once even so, and a block's chain of tiles is what the launch lasts; else
    // one, which makes room for more blocks (float32 heads of 256 that share no keys, 16 of them, 400 tokens: 2,749 us with one
    // block an SM and two stages, 952 with three and one; with 3 tokens of 1,000 keys, four heads of 128 a group, 158 us with two
    // stages and 166 with one).
    const int sms = kipp_sm_count(), fit = std::min(SM_SMEM / (int)(queries + 2 * tiles + 1024), SM_THREADS / (32 * warps));
    const int stages = blocks <= (long long)sms * std::min(fit, SM_BLOCKS) ? 2 : 1;
    const size_t smem = queries + stages * tiles;
    if (const int e = kipp_allow_smem(paged_attention_simt_kernel<T, VEC, NACC>, smem)) return e;
    return kipp_launch(paged_attention_simt_kernel<T, VEC, NACC>, dim3((unsigned)blocks), dim3(warps * 32), smem, s, 1,
                       (T*)out, (const T*)q, (const T*)k_pages, (const T*)v_pages, positions, entry_of_token, block_table,
                       table_width, page_size, n_q, n_kv, head_dim, scale, window, stages, status);
}

template <typename T, typename... Args>
int launch_for(bool vec, int head_dim, Args... args) {
    if (head_dim <= 64) return vec ? launch<T, true, 2>(args...) : launch<T, false, 2>(args...);
    if (head_dim <= 128) return vec ? launch<T, true, 4>(args...) : launch<T, false, 4>(args...);
    return vec ? launch<T, true, MAX_ACC>(args...) : launch<T, false, MAX_ACC>(args...);
}
}  // namespace

namespace {
int run_simt(void* out, const void* q, const void* k_pages, const void* v_pages, int dtype, const int* positions, const int* entry_of_token,
             const int* block_table, int table_width, int page_size, int tokens, int n_q, int n_kv, int head_dim, float scale, int window,
             bool early, int* status, void* stream) {
    if (tokens <= 0) return 0;
    if (head_dim <= 0 || head_dim > 32 * MAX_ACC || n_q <= 0 || n_kv <= 0 || n_q % n_kv ||
        page_size <= 0 || window < 0)
        return KIPP_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const int item = dtype == KIPP_DT_F32 ? 4 : 2;
    const bool vec = head_dim * item % 16 == 0 && (((uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0;
    if (dtype == KIPP_DT_F32)
        return launch_for<float>(vec, head_dim, out, q, k_pages, v_pages, positions, entry_of_token, block_table, table_width,
                                 page_size, tokens, n_q, n_kv, head_dim, scale, window, early, status, s);
    if (dtype == KIPP_DT_BF16)
        return launch_for<bf16>(vec, head_dim, out, q, k_pages, v_pages, positions, entry_of_token, block_table, table_width,
                                page_size, tokens, n_q, n_kv, head_dim, scale, window, early, status, s);
    return KIPP_ERR_DTYPE;
}
}  // namespace

extern "C" int kipp_paged_attention_simt(
    void* out, const void* q, const void* k_pages, const void* v_pages, int dtype,
    const int* positions, const int* entry_of_token, const int* block_table, int table_width,
    int page_size, int tokens, int n_q, int n_kv, int head_dim, float scale, int window,
    int* status, void* stream) {
    return run_simt(out, q, k_pages, v_pages, dtype, positions, entry_of_token, block_table, table_width, page_size, tokens, n_q, n_kv,
                    head_dim, scale, window, false, status, stream);
}
// The same within a step of the engine, all of whose tokens of an entry are here and follow one another: the keys and values before
// an entry's first token are from earlier steps, which ended before this step's lists came, so they may be read before
// the kernel ahead in the stream has ended.  (The entry above takes whatever that kernel has written: a
// few of the tokens it put into the cache, say.)
extern "C" int kipp_paged_attention_simt_of_step(
    void* out, const void* q, const void* k_pages, const void* v_pages, int dtype,
    const int* positions, const int* entry_of_token, const int* block_table, int table_width,
    int page_size, int tokens, int n_q, int n_kv, int head_dim, float scale, int window,
    int* status, void* stream) {
    return run_simt(out, q, k_pages, v_pages, dtype, positions, entry_of_token, block_table, table_width, page_size, tokens, n_q, n_kv,
                    head_dim, scale, window, true, status, stream);
}
