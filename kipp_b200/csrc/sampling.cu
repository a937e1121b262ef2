// Greedy and temperature sampling on the device.  A row of logits is worked on by a team:
// one thread block, or for long rows a thread-block cluster of eight whose blocks take an
// eighth of the row each and put their counts and sums together through distributed shared
// memory (every block reads all eight and decides alike, so nothing is broadcast; the
// cluster's hardware barrier stands between writing and reading).  One block alone scanned a
// 151,936-entry row some fifteen times at 40 to 70 us a scan.
//
// The token drawn is the one the reference's host sampler draws from the same
// logits and the same uniform number (kipp_sample_ex, src/kipp.c:3433-3559):
//   * greedy (temperature <= 0): first index of the maximum, strict '>';
//   * else scaled = logit * (1/T); candidates are scaled >= max - 20; they are
//     ordered by scaled value descending, ties by token id ascending; top-k
//     keeps the first k; weights w = expf(scaled - max) in float32, sums in
//     double; min-p keeps w >= min_p * w_top; the nucleus is the shortest
//     prefix whose sum reaches top_p * total; draw = u * kept picks the first
//     candidate whose inclusive prefix sum exceeds it.
// The reference sorts the candidates.  Here nothing is sorted: a position in
// that order is found by radix selection over the (value, token) keys, with
// per-bucket counts and weight sums, four 8-bit passes over the value and,
// only among equal values, four over the token id.  Bucket sums add the same
// float32 weights as integers in units of 2^-40 (see peers_units) where the
// reference keeps a running double sum, so a draw that lies within 2^-23 of a
// boundary may pick the neighbour.
//
// A pass over the row is what costs (a 151,936-entry row is 600 KB, and each of its entries takes some
// forty instructions in a pass that adds weights), so there are few: the first pass of a selection also
// gives the total that its target is a share of; its second pass, which looks at one bucket of the
// first, puts that bucket's elements into a list in shared memory, and the passes after it walk the
// list; what top-k leaves is listed once for everything that follows; a rank is looked for without weights; and the
// draw within a nucleus takes its first pass from the selection that found the nucleus; and a pass over a long part
// that adds weights has a histogram for each lane.  64 rows of 151,936, top-p 0.95: 207 us, 158 with top-k 50 (519 and 158
// before the histograms by lane; with half the rows of either kind 488, 934 with all passes over the rows and the loads
// one at a time); a single such row by eight blocks: 92 us (138), 148 of them by a block each 351 (1,013).  Rows that all have a top-k
// that fits the list go without (kipp_sample_rows_of): as before them.  What is left is six walks of some forty instructions an
// element.
//
// Also here: the penalties and logit bias the reference applies before
// sampling (apply_bias_and_penalties, src/kipp.c:3386-3431).
#include "common.cuh"
#include <math.h>

namespace {
constexpr int THREADS = 1024;

__device__ __forceinline__ unsigned desc_key(float x) {
    // Ascending unsigned order of the result == descending float order of x.
    unsigned k = __float_as_uint(x);
    k = (k & 0x80000000u) ? ~k : (k | 0x80000000u);
    return ~k;
}

// ---- the team of blocks that shares a row (a cluster along x; one block when launched without)
__device__ __forceinline__ int team_size() { unsigned n; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n)); return (int)n; }
__device__ __forceinline__ int team_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return (int)r; }
// all threads of all blocks of the team: what was written to shared memory before is visible after
__device__ __forceinline__ void team_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t team_addr(const void* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ unsigned team_ld_u32(const void* p, int rank) {
    unsigned v; asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(team_addr(p, rank)) : "memory"); return v;
}
__device__ __forceinline__ float team_ld_f32(const void* p, int rank) {
    float v; asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(team_addr(p, rank)) : "memory"); return v;
}
__device__ __forceinline__ unsigned long long team_ld_u64(const void* p, int rank) {
    unsigned long long v; asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(team_addr(p, rank)) : "memory"); return v;
}

constexpr int LIST_CAP = 4096;  // elements a block lists: 16 KB
constexpr int FEW_ELEMENTS = 2048;
constexpr int COPIES = 4;       // histograms of a block, one for every fourth warp: most elements of a first pass meet a
                                // handful of buckets, and atomics on one word run one after the other
constexpr int COPIES_FROM = 2048;   // elements from which a block has them; clearing and adding four costs a short row more

// A pass over a long part of a row: a histogram for each lane of a warp, shared by the block's warps ([what][bucket][lane]
// words: counts, then the two pieces of the weights' units), so that no two lanes of an atomic meet in a word or a bank.
// Finding the lanes of equal buckets and adding them as one, which serves lists and counts without weights, took most of a
// long pass: the lanes' buckets are few in a selection's first pass and many in its second, and their groups add their
// weights one after the other.  BY_LANE_FROM: 16 rows of 10,000 101 us with the groups, 64 so; below that a kernel that
// clears and adds up 24,576 words a pass has little to win.  A lane's sum of a piece of the units must not pass 2^32: after
// BY_LANE_TO elements the lanes' sums are added up and start anew.  (Kernels of their own for the two: four rows of 700 in one
// kernel for both 37 us, 33 so.)
constexpr int LANE_WORDS = 256 * 32, BY_LANE_BYTES = 3 * LANE_WORDS * 4;
constexpr int BY_LANE_FROM = 8192, BY_LANE_TO = 32 * 4095;
struct RowCtx {
    unsigned* by_lane;          // [3][256][32] in shared memory (LONG)
    const float* v;
    int n;
    int lo, hi;                 // this block's part of the row
    int* list;                  // [LIST_CAP] in shared memory
    int listed;                 // >= 0: the elements to walk are the first `listed` of the list
    int copies;                 // histograms in use
    float inv_t, smax, cutoff;
    // filters
    bool has_topk;   unsigned topk_key, topk_tok;
    bool has_minp;   double minp_threshold;
    bool has_nucleus; unsigned nuc_key, nuc_tok;
};

__device__ __forceinline__ bool before_or_at(unsigned key, unsigned tok, unsigned bkey, unsigned btok) {
    return key < bkey || (key == bkey && tok <= btok);
}

// Whether element i of value x passes every filter but min-p, which wants the weight; gives its key.
__device__ __forceinline__ bool candidate(const RowCtx& c, int i, float x, unsigned& key) {
    const float scaled = x * c.inv_t;
    if (!(scaled >= c.cutoff)) return false;
    key = desc_key(scaled);
    if (c.has_topk && !before_or_at(key, (unsigned)i, c.topk_key, c.topk_tok)) return false;
    return !c.has_nucleus || before_or_at(key, (unsigned)i, c.nuc_key, c.nuc_tok);
}
__device__ __forceinline__ bool weighs(const RowCtx& c, float x, float& w) {
    w = expf(x * c.inv_t - c.smax);
    return !c.has_minp || !((double)w < c.minp_threshold);
}

struct Shared {
    unsigned cnt[COPIES][256];  // this block's part of the row
    unsigned long long wfix[COPIES][256];   // weight sums in units of 2^-40 (see peers_units)
    unsigned cnt_all[256];      // the team's: the blocks' parts added in block order
    double wsum_all[256];
    unsigned long long units_all[256];
    unsigned cnt_first[256], part_first[256];   // cnt_all, cnt[0] and wsum_all after the first pass of a selection by share
    double wsum_first[256];
    int listed;                 // elements appended to the list
    double total;
    float red_val[32];
    int red_idx[32];
    // results broadcast
    unsigned sel_digit; unsigned long long sel_cnt_before; double sel_w_before;
    unsigned sel_bucket_cnt; int found;
    int i_val; float f_val; double d_val;
};

enum { MODE_COUNT = 0, MODE_W_GE = 1, MODE_W_GT = 2 };

// Weights are summed as integers, in units of 2^-40 of the top weight (1): integer sums do not
// depend on their order, so a row's draw is the same whichever block or lane adds first, and
// the lanes of a warp that hit the same bucket add their weights with the warp's integer
// reduction and ONE atomic instead of 32 that the hardware runs one after the other (with
// float64 atomics the passes were bound by exactly that).  A weight is at least e^-20 = 2^-29,
// so it keeps eleven bits and more; a row's sums stay below 2^58.  Against the reference's
// running float64 sum a draw within 2^-23 of a boundary may pick the neighbour.
constexpr double WEIGHT_UNIT = 1.0 / 1099511627776.0;      // 2^-40
struct Units { unsigned whole, rest; };      // whole 2^20 + rest
__device__ __forceinline__ Units units_of(float w) {
    const float scaled = w * 1048576.0f;
    const unsigned whole = (unsigned)scaled;
    return Units{whole, (unsigned)((scaled - (float)whole) * 1048576.0f)};
}
// Sum of the units of `w` (0 <= w <= 1, cut to a whole number of them) over the lanes of `peers` (all of them call this
// with the same mask).  The units leave the float in two pieces of 20 bits, every step exact.
__device__ __forceinline__ unsigned long long peers_units(unsigned peers, float w) {
    const Units u = units_of(w);
    const unsigned hi = __reduce_add_sync(peers, u.whole);                                                  // 32 x 2^20 < 2^32
    const unsigned lo = __reduce_add_sync(peers, u.rest);
    return ((unsigned long long)hi << 20) + lo;
}

// Calls f(i, x, there) for every element of this block's part (or list), by whole warps: all lanes
// of a warp together, `there` false where a lane has none.  Several loads are on their way at a time.
template <typename F> __device__ __forceinline__ void walk(const RowCtx& c, F f) {
    constexpr int AT_ONCE = 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const bool list = c.listed >= 0;
    const int n = list ? c.listed : c.hi - c.lo;
    // (few elements one by one: eight copies of a pass's code are more to fetch than they save there; four rows of 700 with a nucleus
    // of 0.9: 36 us with eight at a time and four histograms, 30 so)
    if (n <= FEW_ELEMENTS) {
#pragma unroll 1
        for (int base = warp * 32; base < n; base += warps * 32) {
            const int at = base + lane, i = at >= n ? -1 : list ? c.list[at] : c.lo + at;
            f(i, i < 0 ? 0.f : c.v[i], i >= 0);
        }
        return;
    }
    for (int base = warp * 32; base < n; base += warps * 32 * AT_ONCE) {
        int i[AT_ONCE]; float x[AT_ONCE];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const int at = base + 32 * warps * u + lane;
            i[u] = at >= n ? -1 : list ? c.list[at] : c.lo + at;
            x[u] = i[u] < 0 ? 0.f : c.v[i[u]];
        }
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            if (base + 32 * warps * u >= n) break;
            f(i[u], x[u], i[u] >= 0);
        }
    }
}
// Appends the lanes' elements to the block's list (the caller knows that they fit; whole warps).
__device__ __forceinline__ void append(const RowCtx& c, Shared& sh, int i, bool there) {
    const int lane = threadIdx.x & 31;
    const unsigned who = __ballot_sync(0xffffffffu, there);
    if (who == 0) return;
    int at = 0;
    if (lane == __ffs(who) - 1) at = atomicAdd(&sh.listed, __popc(who));
    at = __shfl_sync(0xffffffffu, at, __ffs(who) - 1) + __popc(who & ((1u << lane) - 1u));
    if (there) c.list[at] = i;
}

// One histogram pass.  level 0..3: value key digits (high to low); level 4..7:
// token digits among elements whose key == prefix_key.  `gather`: what lies under the prefix is listed too.
// Without `weigh` only the counts are formed (no min-p is in force then).
template <bool LONG>
__device__ void histogram_pass(const RowCtx& c, Shared& sh, int level, unsigned prefix_key,
                               unsigned prefix_tok, bool gather, bool weigh) {
    const bool by_lane = LONG && weigh && c.listed < 0;
    if (by_lane) {
        for (int b = threadIdx.x; b < 256; b += blockDim.x) { sh.cnt[0][b] = 0; sh.wfix[0][b] = 0ull; }
    } else {
        for (int b = threadIdx.x; b < c.copies * 256; b += blockDim.x) { (&sh.cnt[0][0])[b] = 0; (&sh.wfix[0][0])[b] = 0ull; }
    }
    if (threadIdx.x == 0) sh.listed = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, copy = (threadIdx.x >> 5) & (c.copies - 1);
    auto digit_of = [&](int i, float x, bool there, float& w) {
        unsigned key = 0;
        unsigned digit = 256u;                                  // no bucket: not in the set at this level
        w = 0.f;
        if (there && candidate(c, i, x, key)) {
            if (level < 4) {
                const int shift = 24 - 8 * level;
                if (level == 0 || (key >> (shift + 8)) == (prefix_key >> (shift + 8))) digit = (key >> shift) & 0xffu;
            } else if (key == prefix_key) {
                const int shift = 24 - 8 * (level - 4);
                const unsigned tok = (unsigned)i;
                if (level == 4 || (tok >> (shift + 8)) == (prefix_tok >> (shift + 8))) digit = (tok >> shift) & 0xffu;
            }
            if (weigh && digit < 256u && !weighs(c, x, w)) { digit = 256u; w = 0.f; }
        }
        return digit;
    };
    // (two walks rather than one with both forms in it: 64 rows of 151,936 203 us instead of 239)
    if (by_lane) {
        RowCtx piece = c;
#pragma unroll 1
        for (piece.lo = c.lo; piece.lo < c.hi; piece.lo += BY_LANE_TO) {
            piece.hi = min(c.hi, piece.lo + BY_LANE_TO);
            for (int i = threadIdx.x; i < 3 * LANE_WORDS / 4; i += blockDim.x) reinterpret_cast<uint4*>(c.by_lane)[i] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            walk(piece, [&](int i, float x, bool there) {
                float w;
                const unsigned digit = digit_of(i, x, there, w);
                if (gather) append(c, sh, i, digit < 256u);
                if (digit < 256u) {
                    unsigned* at = c.by_lane + digit * 32 + lane;
                    const Units u = units_of(w);
                    atomicAdd(at, 1u);
                    atomicAdd(at + LANE_WORDS, u.whole);
                    atomicAdd(at + 2 * LANE_WORDS, u.rest);
                }
            });
            __syncthreads();
            // four neighbouring threads a bucket, eight lanes' words each
            for (int at = threadIdx.x; at < 1024; at += blockDim.x) {
                unsigned long long sum[3] = {0ull, 0ull, 0ull};
#pragma unroll
                for (int what = 0; what < 3; ++what) {
                    const uint4* words = reinterpret_cast<const uint4*>(c.by_lane + what * LANE_WORDS + at * 8);
                    const uint4 x = words[0], y = words[1];
                    sum[what] = (unsigned long long)x.x + x.y + x.z + x.w + y.x + y.y + y.z + y.w;
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) sum[what] += __shfl_xor_sync(0xffffffffu, sum[what], o);
                }
                if ((at & 3) == 0) { sh.cnt[0][at >> 2] += (unsigned)sum[0]; sh.wfix[0][at >> 2] += (sum[1] << 20) + sum[2]; }
            }
            __syncthreads();
        }
    } else {
        // the lanes of a round that fall into one bucket are found with match.any and add as one
        walk(c, [&](int i, float x, bool there) {
            float w;
            const unsigned digit = digit_of(i, x, there, w);
            if (gather) append(c, sh, i, digit < 256u);
            if (!__any_sync(0xffffffffu, digit < 256u)) return;
            const unsigned peers = __match_any_sync(0xffffffffu, digit);
            const unsigned long long units = weigh ? peers_units(peers, w) : 0ull;
            if (digit < 256u && lane == __ffs(peers) - 1) {
                atomicAdd(&sh.cnt[copy][digit], (unsigned)__popc(peers));
                if (weigh) atomicAdd(&sh.wfix[copy][digit], units);
            }
        });
    }
    __syncthreads();
    if (!by_lane) for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        for (int k = 1; k < c.copies; ++k) { sh.cnt[0][b] += sh.cnt[k][b]; sh.wfix[0][b] += sh.wfix[k][b]; }
    }
    // the team's histogram: every block adds the blocks' parts in block order
    team_sync();
    const int blocks = team_size();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        unsigned n8[8]; unsigned long long w8[8];    // all loads first: they travel together
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            n8[r] = r < blocks ? team_ld_u32(&sh.cnt[0][b], r) : 0u;
            w8[r] = r < blocks ? team_ld_u64(&sh.wfix[0][b], r) : 0ull;
        }
        unsigned n = 0; unsigned long long w = 0ull;
#pragma unroll
        for (int r = 0; r < 8; ++r) { n += n8[r]; w += w8[r]; }
        sh.cnt_all[b] = n; sh.wsum_all[b] = (double)w * WEIGHT_UNIT; sh.units_all[b] = w;
    }
    team_sync();                                   // nobody clears its part while another still reads it
}

// Position selection in the (value desc, token asc) order of the current set.
//   MODE_COUNT: the element with 1-based rank `target_count`;
//   MODE_W_GE : the first element whose inclusive weight sum >= target_w;
//   MODE_W_GT : the first element whose inclusive weight sum >  target_w.
// With `of_total` target_w is a share of the set's total weight, which `total` gives in any case.
// If no element qualifies, the last element of the set is returned.
// `again`: the set is the nucleus that the selection before has found in its own set (`nuc_key`).  It is a prefix of
// that set's order, so the counts and sums of the first pass are those found then: exactly in the buckets before
// the one where the nucleus ends, in that one too much, which decides nothing (it is the last either way),
// and none after it.
// Outputs (uniform over the block): key, token, inclusive weight sum at it.
template <bool LONG>
__device__ void select(RowCtx& c, Shared& sh, int mode, unsigned long long target_count, double target_w, bool of_total,
                       bool again, unsigned& out_key, unsigned& out_tok, double& out_cum, double& total) {
    const int listed_before = c.listed;
    unsigned part_cnt = 0;                            // elements of this block's part under the prefix
    unsigned prefix_key = 0, prefix_tok = 0;
    unsigned long long cnt_before = 0;
    double w_before = 0.0;
    for (int level = 0; level < 8; ++level) {
        const bool gather = level > 0 && c.listed < 0 && part_cnt <= LIST_CAP;
        if (level == 0 && again) {
            for (int b = threadIdx.x; b < 256; b += blockDim.x) {
                sh.cnt_all[b] = b <= (int)(c.nuc_key >> 24) ? sh.cnt_first[b] : 0u;
                sh.wsum_all[b] = b <= (int)(c.nuc_key >> 24) ? sh.wsum_first[b] : 0.0;
                sh.cnt[0][b] = sh.part_first[b];
            }
            __syncthreads();
        } else {
            histogram_pass<LONG>(c, sh, level, prefix_key, prefix_tok, gather, mode != MODE_COUNT);
        }
        if (gather) c.listed = sh.listed;
        if (level == 0 && mode == MODE_W_GE)                      // (a bucket's own thread has formed all three)
            for (int b = threadIdx.x; b < 256; b += blockDim.x) {
                sh.cnt_first[b] = sh.cnt_all[b]; sh.part_first[b] = sh.cnt[0][b]; sh.wsum_first[b] = sh.wsum_all[b];
            }
        if (threadIdx.x < 32) {
            if (level == 0) {
                unsigned long long all = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) all += sh.units_all[8 * threadIdx.x + j];
                // Below an infinite largest value every member weighs e^(inf - inf).  Its conversion to units gives 2^63 and
                // sums are taken modulo 2^64: with an odd number of members a share of the total lies behind all of them,
                // so that the last is taken; with an even number it is 0.
                if (isinf(c.smax))
#pragma unroll
                    for (int j = 0; j < 8; ++j) all += (unsigned long long)sh.cnt_all[8 * threadIdx.x + j] << 63;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
                const double sum = (double)all * WEIGHT_UNIT;
                if (of_total) target_w *= sum;
                if (threadIdx.x == 0) sh.total = sum;
            }
            // The first bucket (in order) at which the running count or weight reaches the target,
            // else the last bucket that is not empty.  One warp: a lane walks over its eight
            // buckets from the sums of the lanes before it (one thread alone took 256 dependent
            // steps, some 5 us a level).
            const int lane = threadIdx.x;
            unsigned n8[8]; double w8[8];
            unsigned long long ln = 0; double lw = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                n8[j] = sh.cnt_all[8 * lane + j]; w8[j] = sh.wsum_all[8 * lane + j];
                ln += n8[j]; lw += w8[j];
            }
            unsigned long long pn = ln; double pw = lw;             // inclusive over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long tn = __shfl_up_sync(0xffffffffu, pn, o);
                const double tw = __shfl_up_sync(0xffffffffu, pw, o);
                if (lane >= o) { pn += tn; pw += tw; }
            }
            unsigned long long cb = __shfl_up_sync(0xffffffffu, pn, 1);
            double wb = __shfl_up_sync(0xffffffffu, pw, 1);
            if (lane == 0) { cb = 0; wb = 0.0; }
            cb += cnt_before; wb += w_before;
            int chosen = -1, last_nonempty = -1;
            unsigned long long cb_hit = 0, cb_last = 0; double wb_hit = 0.0, wb_last = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (n8[j] == 0 || chosen >= 0) continue;
                last_nonempty = 8 * lane + j; cb_last = cb; wb_last = wb;
                bool hit;
                if (mode == MODE_COUNT) hit = cb + n8[j] >= target_count;
                else if (mode == MODE_W_GE) hit = wb + w8[j] >= target_w;
                else hit = wb + w8[j] > target_w;
                if (hit) { chosen = 8 * lane + j; cb_hit = cb; wb_hit = wb; }
                else { cb += n8[j]; wb += w8[j]; }
            }
            const unsigned hits = __ballot_sync(0xffffffffu, chosen >= 0);
            const unsigned some = __ballot_sync(0xffffffffu, last_nonempty >= 0);
            int src = -1;                                            // the lane whose answer counts
            if (hits) src = __ffs(hits) - 1;
            else if (some) { src = 31 - __clz(some); chosen = last_nonempty; cb_hit = cb_last; wb_hit = wb_last; }
            if (lane == src) {
                sh.found = chosen;
                sh.sel_cnt_before = cb_hit; sh.sel_w_before = wb_hit;
                sh.sel_bucket_cnt = sh.cnt_all[chosen];
                sh.d_val = wb_hit + sh.wsum_all[chosen];
            } else if (src < 0 && lane == 0) {
                sh.found = -1;
                sh.sel_cnt_before = cnt_before; sh.sel_w_before = w_before;
                sh.sel_bucket_cnt = 0;
                sh.d_val = w_before;
            }
        }
        __syncthreads();
        const int chosen = sh.found;
        cnt_before = sh.sel_cnt_before; w_before = sh.sel_w_before;
        const double cum_incl = sh.d_val;
        const unsigned bucket_cnt = sh.sel_bucket_cnt;
        if (level == 0) total = sh.total;
        part_cnt = chosen < 0 ? 0 : sh.cnt[0][chosen];
        __syncthreads();
        if (chosen < 0) { out_key = 0xffffffffu; out_tok = 0; out_cum = w_before; break; }  // empty set
        const int shift = 24 - 8 * (level & 3);
        if (level < 4) prefix_key |= (unsigned)chosen << shift;
        else prefix_tok |= (unsigned)chosen << shift;
        if (level == 7) { out_key = prefix_key; out_tok = prefix_tok; out_cum = cum_incl; break; }
        if (level == 3 && bucket_cnt == 1) {
            // One element has this value: find its token in one pass.
            if (threadIdx.x == 0) sh.i_val = 0x7fffffff;
            __syncthreads();
            walk(c, [&](int i, float x, bool there) {
                unsigned key; float w;
                if (there && candidate(c, i, x, key) && key == prefix_key && weighs(c, x, w)) atomicMin(&sh.i_val, i);
            });
            __syncthreads();
            team_sync();
            int first = 0x7fffffff;
            for (int r = 0; r < team_size(); ++r) first = min(first, (int)team_ld_u32(&sh.i_val, r));
            team_sync();
            out_key = prefix_key; out_tok = (unsigned)first; out_cum = cum_incl;
            break;
        }
    }
    c.listed = listed_before;
}

// best_i = 0x7fffffff when the row holds no number (NaN only)
__device__ void block_argmax_raw(const float* v, int n, Shared& sh, float& best_v, int& best_i) {
    float bv = -INFINITY; int bi = 0x7fffffff;
    constexpr int AT_ONCE = 8;                        // loads on their way
    for (int i0 = threadIdx.x; i0 < n; i0 += AT_ONCE * blockDim.x) {
        float x[AT_ONCE];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const int i = i0 + u * (int)blockDim.x;
            x[u] = i < n ? v[i] : -INFINITY;
        }
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const int i = i0 + u * (int)blockDim.x;
            if (i < n && (x[u] > bv || (x[u] == bv && i < bi))) { bv = x[u]; bi = i; }
        }
    }
    // A row of NaNs or -inf leaves bi unset in some threads; index 0 then wins
    // as in the reference (argmax starts at 0 and only '>' replaces it).
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sh.red_val[warp] = bv; sh.red_idx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        bv = lane < nw ? sh.red_val[lane] : -INFINITY;
        bi = lane < nw ? sh.red_idx[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { sh.f_val = bv; sh.i_val = bi; }
    }
    __syncthreads();
    best_v = sh.f_val; best_i = sh.i_val;
    __syncthreads();
}

__device__ void block_argmax(const float* v, int n, Shared& sh, float& best_v, int& best_i) {
    block_argmax_raw(v, n, sh, best_v, best_i);
    if (best_i == 0x7fffffff) best_i = 0;
}

__global__ void __launch_bounds__(THREADS)
argmax_rows_kernel(const float* __restrict__ logits, long long ld, int n, int* __restrict__ out) {
    __shared__ Shared sh;
    pdl_launch_dependents();
    pdl_wait();
    float bv; int bi;
    block_argmax(logits + (size_t)blockIdx.x * ld, n, sh, bv, bi);
    if (threadIdx.x == 0) out[blockIdx.x] = bi;
}

// A long row by many blocks: block (c, r) leaves the first maximum of its share of row r, the
// second kernel takes the first maximum of the shares (in share order, so the lowest index wins
// a tie as in the one-block kernel).  One block per row would scan a 150,000-entry row alone
// for 70 us; the shares take a few.
struct ArgmaxPart { float v; int i; };

__global__ void __launch_bounds__(THREADS)
argmax_parts_kernel(const float* __restrict__ logits, long long ld, int n, int per, ArgmaxPart* __restrict__ parts) {
    __shared__ Shared sh;
    pdl_launch_dependents();
    pdl_wait();
    const int first = blockIdx.x * per;
    const int count = min(per, n - first);
    float bv = -INFINITY; int bi = 0x7fffffff;
    if (count > 0) block_argmax_raw(logits + (size_t)blockIdx.y * ld + first, count, sh, bv, bi);
    if (threadIdx.x == 0)
        parts[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = ArgmaxPart{bv, bi == 0x7fffffff ? bi : first + bi};
}

__global__ void argmax_merge_kernel(const ArgmaxPart* __restrict__ parts, int n_parts, int* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    // one warp per row; lane l takes shares l, l + 32, ... in order, then the lanes in order
    const ArgmaxPart* row = parts + (size_t)blockIdx.x * n_parts;
    float bv = -INFINITY; int bi = 0x7fffffff;
    for (int c = threadIdx.x; c < n_parts; c += 32) {
        const ArgmaxPart p = row[c];
        if (p.v > bv || (p.v == bv && p.i < bi)) { bv = p.v; bi = p.i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    // a row without any number (NaN only) leaves every share without an index: index 0 then
    if (threadIdx.x == 0) out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
}

// The token drawn from a row (temperature above 0) whose first maximum is `best_i`.  (Its options are read where they are used: held
// from the start they cost the kernel its last registers, and 64 rows of 151,936 with top-k 4,096 191 us instead of 187.)
template <bool LONG>
__device__ int draw(RowCtx& c, Shared& sh, int k, const float* top_p, const float* min_p, const double* uniform, int best_i) {
    unsigned key, tok; double cum, total;
    if (k > 0) {
        // rank k in the order, or the last candidate when there are fewer
        select<LONG>(c, sh, MODE_COUNT, (unsigned long long)k, 0.0, false, false, key, tok, cum, total);
        c.has_topk = true; c.topk_key = key; c.topk_tok = tok;
        if (k <= LIST_CAP) {                           // what is left is k elements at most
            if (threadIdx.x == 0) sh.listed = 0;
            __syncthreads();
            walk(c, [&](int i, float x, bool there) {
                unsigned kk;
                append(c, sh, i, there && candidate(c, i, x, kk));
            });
            __syncthreads();
            c.listed = sh.listed;
            __syncthreads();                           // read by all before the next pass counts anew
        }
    }
    const float mp = *min_p;
    if (mp > 0.0f) {
        // The top weight is expf(smax - smax) = 1.
        c.has_minp = true;
        c.minp_threshold = (double)mp * (double)expf(0.0f);
    }
    // with a nucleus, the prefix that is kept, and a share of its weight; else a share of the set's
    const float tp = *top_p;
    double kept;
    if (tp < 1.0f) {
        select<LONG>(c, sh, MODE_W_GE, 0, (double)tp, true, false, key, tok, cum, total);
        c.has_nucleus = true; c.nuc_key = key; c.nuc_tok = tok;
        kept = cum;
        select<LONG>(c, sh, MODE_W_GT, 0, *uniform * kept, false, true, key, tok, cum, total);
    } else {
        select<LONG>(c, sh, MODE_W_GT, 0, *uniform, true, false, key, tok, cum, total);
        kept = total;
    }
    return (key == 0xffffffffu && tok == 0 && kept == 0.0) ? best_i : (int)tok;
}

// LONG: a block's part of a row is long enough for the histograms by lane.
template <bool LONG>
__global__ void __launch_bounds__(THREADS)
sample_rows_kernel(const float* __restrict__ logits, long long ld, int n,
                   const float* __restrict__ temperature, const int* __restrict__ top_k,
                   const float* __restrict__ top_p, const float* __restrict__ min_p,
                   const double* __restrict__ uniform, int* __restrict__ out) {
    __shared__ Shared sh;
    __shared__ int list[LIST_CAP];
    extern __shared__ __align__(16) unsigned by_lane[];     // BY_LANE_BYTES with LONG, else nothing
    pdl_launch_dependents();
    pdl_wait();
    const int blocks = team_size(), rank = team_rank();
    const int r = blockIdx.x / blocks;
    const float* v = logits + (size_t)r * ld;
    const int part = ((n + blocks - 1) / blocks + 3) & ~3;
    const int lo = min(n, rank * part), hi = min(n, lo + part);
    // the row's first maximum: each block's over its part, then the first of those
    float best_v; int best_i;
    block_argmax_raw(v + lo, hi - lo, sh, best_v, best_i);
    if (threadIdx.x == 0) { sh.f_val = best_v; sh.i_val = best_i == 0x7fffffff ? best_i : lo + best_i; }
    __syncthreads();
    team_sync();
    best_v = -INFINITY; best_i = 0x7fffffff;
    for (int b = 0; b < blocks; ++b) {
        const float ov = team_ld_f32(&sh.f_val, b);
        const int oi = (int)team_ld_u32(&sh.i_val, b);
        if (ov > best_v || (ov == best_v && oi < best_i)) { best_v = ov; best_i = oi; }
    }
    if (best_i == 0x7fffffff) best_i = 0;
    team_sync();
    const float T = temperature[r];
    if (!(T > 0.0f)) {
        if (threadIdx.x == 0 && rank == 0) out[r] = best_i;
        return;
    }
    RowCtx c;
    c.by_lane = by_lane;
    c.v = v; c.n = n; c.lo = lo; c.hi = hi; c.list = list; c.listed = -1; c.copies = hi - lo > COPIES_FROM ? COPIES : 1;
    c.inv_t = 1.0f / T;
    c.smax = v[best_i] * c.inv_t;
    c.cutoff = c.smax - 20.0f;
    c.has_topk = c.has_minp = c.has_nucleus = false;
    c.topk_key = c.topk_tok = c.nuc_key = c.nuc_tok = 0;
    c.minp_threshold = 0.0;

    // (Rows whose top-k leaves no more than the list holds walk long parts without weights only: they take the code of the short
    // parts.  Sharing the other's, with its second kind of walk, cost them another 2 to 3 us of code to fetch.)
    const int k = top_k[r];
    const int token = LONG && !(k > 0 && k <= LIST_CAP) ? draw<true>(c, sh, k, top_p + r, min_p + r, uniform + r, best_i)
                                                        : draw<false>(c, sh, k, top_p + r, min_p + r, uniform + r, best_i);
    if (threadIdx.x == 0 && rank == 0) out[r] = token;
}

// Logit bias, then repetition / presence / frequency penalties over each row's
// window of recent tokens; each distinct token is adjusted once
// (src/kipp.c:3386-3431).  One block per row; the window is short.
__global__ void apply_penalties_kernel(float* __restrict__ logits, long long ld, int n,
                                       const int* __restrict__ recent, int recent_width,
                                       const int* __restrict__ recent_count,
                                       const float* __restrict__ repetition,
                                       const float* __restrict__ presence,
                                       const float* __restrict__ frequency,
                                       const int* __restrict__ bias_tokens,
                                       const float* __restrict__ bias_values, int bias_width,
                                       const int* __restrict__ bias_count) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x;
    float* v = logits + (size_t)r * ld;
    if (bias_tokens != nullptr && threadIdx.x == 0) {
        // sequential: the same token may be listed twice and both add up
        const int nb = bias_count[r];
        for (int i = 0; i < nb; ++i) {
            const int tok = bias_tokens[(size_t)r * bias_width + i];
            if (tok >= 0 && tok < n) v[tok] += bias_values[(size_t)r * bias_width + i];
        }
    }
    __syncthreads();
    if (recent == nullptr) return;
    const float rep = repetition[r], pres = presence[r], freq = frequency[r];
    const bool has = freq != 0.0f || pres != 0.0f || (rep != 0.0f && rep != 1.0f);
    const int nr = recent_count[r];
    if (!has || nr == 0) return;
    const int* win = recent + (size_t)r * recent_width;
    for (int p = threadIdx.x; p < nr; p += blockDim.x) {
        const int tok = win[p];
        if (tok < 0 || tok >= n) continue;
        bool seen = false;
        for (int e = 0; e < p; ++e) if (win[e] == tok) { seen = true; break; }
        if (seen) continue;
        int count = 0;
        for (int o = 0; o < nr; ++o) count += win[o] == tok;
        float x = v[tok];
        if (rep != 0.0f && rep != 1.0f) x = x > 0.0f ? x / rep : x * rep;
        x -= pres;
        x -= freq * (float)count;
        v[tok] = x;
    }
}
}  // namespace

// Between two greedy decode steps that run without the host (captured in one CUDA
// graph with the step itself): the tokens just chosen become the next step's
// tokens and go into row `*counter` of the ring; every request moves on by one
// position.  What a mixer's kernels derive from the lengths (the keys per split of
// the decode attention) is made anew by that mixer's own kernel after this one.
// One block.  What follows may read the lists before its dependency wait (see common.cuh), so this kernel lets
// nothing start before it has ended.
namespace {
__global__ void burst_advance_kernel(int* tokens, int* positions, int* context_len, const int* next, int* ring,
                                     int* counter, int n, int ring_rows) {
    pdl_wait();                                      // the tokens are chosen, every kernel of the step is through
    const int c = *counter;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int t = next[i];
        tokens[i] = t;
        if (c < ring_rows) ring[(size_t)c * n + i] = t;
        positions[i] += 1;
        context_len[i] += 1;                         // cached tokens before the next step's token
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = c + 1;
}
}  // namespace

extern "C" int kipp_argmax_rows(const float* logits, long long ld, int rows, int n, int* out,
                                void* stream) {
    if (rows <= 0) return 0;
    if (n <= 0) return KIPP_ERR_ARG;
    return kipp_launch(argmax_rows_kernel, dim3(rows), dim3(THREADS), 0, (cudaStream_t)stream, 1, logits, ld, n, out);
}

// How a row of n entries is shared among blocks: shares of at least ARGMAX_SHARE entries, at most 64.
namespace {
constexpr int ARGMAX_SHARE = 4096;
inline int argmax_shares(int n) { return n >= 2 * ARGMAX_SHARE ? (n / ARGMAX_SHARE > 64 ? 64 : n / ARGMAX_SHARE) : 1; }
}  // namespace

// Bytes of scratch kipp_argmax_rows_split wants for rows of n entries (0: the one-block kernel does it).
extern "C" long long kipp_argmax_scratch_bytes(int rows, int n) {
    const int shares = argmax_shares(n);
    return shares > 1 ? (long long)rows * shares * (long long)sizeof(ArgmaxPart) : 0;
}

// kipp_argmax_rows with long rows shared among blocks; `scratch` of kipp_argmax_scratch_bytes,
// 8-byte aligned, is the caller's and holds nothing between calls.
extern "C" int kipp_argmax_rows_split(const float* logits, long long ld, int rows, int n, int* out, void* scratch,
                                      long long scratch_bytes, void* stream) {
    if (rows <= 0) return 0;
    if (n <= 0) return KIPP_ERR_ARG;
    const int shares = argmax_shares(n);
    if (shares <= 1) return kipp_argmax_rows(logits, ld, rows, n, out, stream);
    if (scratch == nullptr || ((uintptr_t)scratch & 7) || scratch_bytes < kipp_argmax_scratch_bytes(rows, n) || rows > 65535)
        return KIPP_ERR_ARG;
    const int per = (n + shares - 1) / shares;
    int rc = kipp_launch(argmax_parts_kernel, dim3(shares, rows), dim3(THREADS), 0, (cudaStream_t)stream, 1, logits, ld,
                         n, per, (ArgmaxPart*)scratch);
    if (rc) return rc;
    return kipp_launch(argmax_merge_kernel, dim3(rows), dim3(32), 0, (cudaStream_t)stream, 1,
                       (const ArgmaxPart*)scratch, shares, out);
}

namespace {
// Long rows: a cluster of up to eight blocks a row (at most eight: the kernel's loops over the team are unrolled to that), as many as
// keep all rows' blocks within one wave of the GPU.
int sample_blocks(int rows, int n) {
    int blocks = 1;
    while (blocks < 8 && n >= 16384 * blocks && (long long)rows * blocks * 2 <= kipp_sm_count()) blocks *= 2;
    return blocks;
}
}  // namespace

// Whether kipp_sample_rows_of launches the kernel with histograms by lane: where a block's part of a row is long and a row may be
// without a top-k that fits the list.  (Rows that all have one walk long parts without weights only, and the kernel's 96 KB of shared
// memory and second kind of walk cost them for nothing: top-k 50, 128 rows of 32,000 79.0 us, 76.9 without; 148 of 151,936 222 and 217, 8
// of 10,000 57.8 and 55.6.)
extern "C" int kipp_sample_rows_by_lane(int rows, int n, int largest_top_k) {
    const int blocks = sample_blocks(rows, n), part = ((n + blocks - 1) / blocks + 3) & ~3;                // (the last block of a row may have less)
    return part >= BY_LANE_FROM && !(largest_top_k > 0 && largest_top_k <= LIST_CAP);
}
// largest_top_k: the largest top_k of the rows that are drawn from (temperature above 0) where each of them has one; 0 where one has
// none, or where nobody says.  It chooses between two forms with the same draws.
extern "C" int kipp_sample_rows_of(const float* logits, long long ld, int rows, int n, const float* temperature, const int* top_k,
                                   const float* top_p, const float* min_p, const double* uniform, int largest_top_k, int* out,
                                   void* stream) {
    if (rows <= 0) return 0;
    if (n <= 0) return KIPP_ERR_ARG;
    const int blocks = sample_blocks(rows, n);
    if ((long long)rows * blocks > 0x7fffffffLL) return KIPP_ERR_ARG;
    const bool by_lane = kipp_sample_rows_by_lane(rows, n, largest_top_k) != 0;
    const auto kernel = by_lane ? sample_rows_kernel<true> : sample_rows_kernel<false>;
    const size_t smem = by_lane ? BY_LANE_BYTES : 0;
    if (const int e = kipp_allow_smem(kernel, smem)) return e;
    return kipp_launch_cluster(kernel, dim3((unsigned)(rows * blocks)), dim3(THREADS), smem, (cudaStream_t)stream,
                               dim3(blocks, 1, 1), logits, ld, n, temperature, top_k, top_p, min_p, uniform, out);
}
extern "C" int kipp_sample_rows(const float* logits, long long ld, int rows, int n,
                                const float* temperature, const int* top_k, const float* top_p,
                                const float* min_p, const double* uniform, int* out, void* stream) {
    return kipp_sample_rows_of(logits, ld, rows, n, temperature, top_k, top_p, min_p, uniform, 0, out, stream);
}

extern "C" int kipp_apply_penalties(float* logits, long long ld, int rows, int n, const int* recent,
                                    int recent_width, const int* recent_count,
                                    const float* repetition, const float* presence,
                                    const float* frequency, const int* bias_tokens,
                                    const float* bias_values, int bias_width, const int* bias_count,
                                    void* stream) {
    if (rows <= 0) return 0;
    if (n <= 0) return KIPP_ERR_ARG;
    return kipp_launch(apply_penalties_kernel, dim3(rows), dim3(64), 0, (cudaStream_t)stream, 1, logits, ld, n,
                       recent, recent_width, recent_count, repetition, presence, frequency, bias_tokens,
                       bias_values, bias_width, bias_count);
}

// See burst_advance_kernel.  `next` holds the n tokens just chosen.
extern "C" int kipp_burst_advance(int* tokens, int* positions, int* context_len, const int* next, int* ring,
                                  int* counter, int n, int ring_rows, void* stream) {
    if (n <= 0) return 0;
    if (ring_rows <= 0) return KIPP_ERR_ARG;
    return kipp_launch(burst_advance_kernel, dim3(1), dim3(128), 0, (cudaStream_t)stream, 1, tokens, positions,
                       context_len, next, ring, counter, n, ring_rows);
}
