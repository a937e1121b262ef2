// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores with float32 accumulation.
//
// This is the matrix product of the true 32-bit path (float32 operands, plain
// FMA, no tensor-core mode) and the fallback of the bfloat16 path for shapes
// the tensor-core kernels refuse.  The reference computes the same product
// one output row per block and one token per launch (matvec_kernel,
// cuda/kipp_kernels.cu:93; src/kipp.c:2233-2243).
//
// The sum over k runs in the same order for every output element whatever M is, so a token's result does
// not depend on what else is in the batch: K is cut into at most 16 runs whose length depends on K alone
// (run_length), a run is one chain of FMAs in the order of k, the sums of four neighbouring runs are added in
// their order, and so are then the up to four sums of those.  The runs are what lets a few tokens be multiplied by
// many threads at once, the groups of four what lets a small product of many tokens be shared by more blocks.
//
// Three kernels, chosen by shape and alignment alone, with that one order for 32-bit weights whose rows start on 16 bytes:
//   few   float32, up to FEW_MAX tokens (16 of many features): bound by the weights' bytes (a token is 2 operations per 4
//         bytes) and, of several tokens, by shared memory's reads.  A block holds 16 features, a thread one feature and one
//         run, so a 2,048-feature matrix still gives 128 blocks of 256 chains; weights and tokens travel by asynchronous copies,
//         the weights' first ones before the wait for the kernel before (few_stages).
//         12,288 x 2,048 with 1, 3 and 16 tokens: 20, 27 and 48 us (100 MB: 15 us of copy rate; the kernel below, which ran
//         once: 334, 339 and 353); 2,048 x 6,144 with 3: 17 us.  From 17 tokens on it needs two passes, which win where the features
//         are few: 32 tokens, 2,048 and 3,072 x 2,048 16 and 30 us, 8,192 x 2,048 60, 2,048 x 6,144 43 (33 tokens in tiles: 49,
//         57, 93 and 128); from many_features() on they are tiles'.
//   tile  float32, more tokens: 128 or 256 features x 64 tokens per block of 128 threads, 8 or 16 x 8 per thread in float32
//         pairs, operands in shared memory with k outermost, so that a k's values cost a thread four or six 16-byte reads
//         (with four bytes copied at a time); the groups of runs are blocks of their own, a cluster that meets in its
//         shared memory.  Bound by the issue around the multiply-adds and shared memory's reads: 407 tokens,
//         12,288 x 2,048 in tiles of 128: FMA pipes 57 % busy, shared memory's data pipe 62 %.  1,024 tokens: 37.7 of 74 TFLOP/s
//         in tiles of 128, 40.2 in 256.
//   any   what is left: tokens whose float32 rows do not start on 16 bytes, in the order above; and what no other kernel
//         here takes, bfloat16 operands of shapes that the tensor-core kernels refuse and float32 weights off 16 bytes: one
//         chain of FMAs in the order of k, without the 38 registers and the extra sums of the runs (bfloat16, 2,050 features
//         of 2,056: 1 and 200 tokens 154 and 152 us, 186 and 180 in runs).
//
// Epilogues:
//   STORE   C[m,n]    = acc                 (C in float32 or bfloat16)
//   ADD     C[m,n]   += acc                 (C float32: the residual stream)
//   SWIGLU  C[m,n/2]  = silu(acc[n]) * acc[n+1] for even n, W holding gate and
//           up rows interleaved (src/kipp.c:2402-2404, 3002-3005)
#include "common.cuh"

#define EPI_STORE 0
#define EPI_ADD 1
#define EPI_SWIGLU 2

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// K in runs: at most MAX_RUNS of them, each of a length that is a multiple of BK, in groups of GROUP_RUNS.
constexpr int MAX_RUNS = 16, GROUP_RUNS = 4;
__host__ __device__ inline int run_length(int K) {
    const int per = (K + MAX_RUNS - 1) / MAX_RUNS;
    return (per + BK - 1) / BK * BK;
}

// One finished sum per element, or a gate and up pair of it, into C.
template <typename TC, int EPI>
__device__ __forceinline__ void put(TC* C, int ldc, int m, int n, float v) {
    const size_t idx = (size_t)m * ldc + n;
    if (EPI == EPI_ADD) C[idx] = from_f32<TC>(to_f32(C[idx]) + v);
    else C[idx] = from_f32<TC>(v);
}
__device__ __forceinline__ float swiglu(float g, float u) { return g / (1.0f + expf(-g)) * u; }

// RUNS: the sum in runs and groups of them (see the head of the file), else one chain.
template <typename TA, typename TW, typename TC, int EPI, bool RUNS>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W,
                 int M, int N, int K, int lda, int ldw, int ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int run = RUNS ? run_length(K) : 0;
    float acc[TM][TN], group[RUNS ? TM : 1][TN], sum[RUNS ? TM : 1][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = 0.f;
            if constexpr (RUNS) group[i][j] = sum[i][j] = 0.f;
        }

    // 64x16 tile = 1024 elements, 256 threads -> 4 each; thread loads row
    // (tid / 4), k columns (tid % 4) * 4 .. + 3.
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int am = m0 + lrow, wn = n0 + lrow;
            As[lk + i][lrow] = (am < M && k < K) ? to_f32(A[(size_t)am * lda + k]) : 0.f;
            Ws[lk + i][lrow] = (wn < N && k < K) ? to_f32(W[(size_t)wn * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
        if constexpr (RUNS) {
            if ((k0 + BK) % run == 0 || k0 + BK >= K) {
                const bool whole = (k0 + BK) % (GROUP_RUNS * run) == 0 || k0 + BK >= K;
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        group[i][j] += acc[i][j];
                        acc[i][j] = 0.f;
                        if (whole) {
                            sum[i][j] += group[i][j];
                            group[i][j] = 0.f;
                        }
                    }
            }
        }
    }

    auto total = [&](int i, int j) {
        if constexpr (RUNS) return sum[i][j];
        else return acc[i][j];
    };
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (EPI == EPI_SWIGLU) {
                if ((j & 1) == 0 && n + 1 < N) put<TC, EPI_STORE>(C, ldc, m, n >> 1, swiglu(total(i, j), total(i, j + 1)));
            } else if (n < N) {
                put<TC, EPI>(C, ldc, m, n, total(i, j));
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Few tokens (see the head of the file).  Warp w of a block holds runs 2w and 2w + 1 of the block's 16
// features; a warp copies only what its own lanes read, so its ring needs no block-wide barrier.
// PAIR: a thread has two features (f and f + 16 of the block's 32), so that a token's values, which every lane of a
// run reads, serve both: of several tokens those reads are what an SM is busy with.
constexpr int FEW_F = 16, FEW_THREADS = 16 * MAX_RUNS, FEW_MAX = 32;
inline int many_features() { return 64 * kipp_sm_count(); }         // two blocks of pairs of features for each SM
inline bool few_tokens(int M, int N) { return M <= (N >= many_features() ? FEW_MAX / 2 : FEW_MAX); }
constexpr int FEW_CHUNK = BK * 4 + 16;              // 64 bytes of a feature's row, padded against bank conflicts
// A warp's stage: its chunks of weights, then 16 values of each of MT tokens for its two runs.  (The tokens' values came
// from global memory before, four at a time and the next four on their way: a trip to the L2 for every four, since a
// block reads each of them once.)
template <bool PAIR, int MT> struct Few {
    static constexpr int PER = PAIR ? 2 : 1, F = FEW_F * PER, CHUNKS = 32 * PER;
    static constexpr int X_AT = CHUNKS * FEW_CHUNK, STAGE = X_AT + MT * 2 * BK * 4;
    static constexpr int BLOCK_STAGE = (FEW_THREADS / 32) * STAGE;        // bytes of a stage of the block's eight warps
};

constexpr int FEW_STAGES_MAX = 6;
// Waits until at most `n` of the thread's groups of copies are on their way, n from 0 to FEW_STAGES_MAX - 2 (else for all).
__device__ __forceinline__ void cp_async_wait_most(int n) {
    static_assert(FEW_STAGES_MAX - 2 == 4, "the cases below");
    switch (n) {
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    case 4: cp_async_wait<4>(); break;
    default: cp_async_wait<0>(); break;
    }
}
// (One function for all epilogues: a layer's four products then find its code where the one before left it.)
template <int MT, bool PAIR>
__global__ void __launch_bounds__(FEW_THREADS)
gemm_few_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                int M, int N, int K, int lda, int ldw, int ldc, int epi, int stages) {
    using Form = Few<PAIR, MT>;
    extern __shared__ __align__(16) uint8_t ring[];
    __shared__ float parts[MAX_RUNS][MT][Form::F + 1];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * Form::F, m0 = blockIdx.y * MT;
    const int run = run_length(K), steps = run / BK;
    uint8_t* mine = ring + (size_t)warp * stages * Form::STAGE;
    // copy j of a step: 16 bytes (lane & 3) of chunk 8 j + lane / 4; chunk c is feature c & 15 (the second 32: 16 + c & 15)
    // of run 2 warp + c / 16 & 1
    auto fetch = [&](int step, int stage) {
#pragma unroll
        for (int j = 0; j < 4 * Form::PER; ++j) {
            const int c = 8 * j + (lane >> 2), n = n0 + (c & 15) + (c >> 5) * FEW_F;
            const int k = (2 * warp + (c >> 4 & 1)) * run + step * BK + (lane & 3) * 4;
            const bool in = n < N && k < K;
            cp_async16(smem_address(mine + (size_t)stage * Form::STAGE + c * FEW_CHUNK + (lane & 3) * 16),
                               in ? W + (size_t)n * ldw + k : W, in ? 16 : 0);
        }
    };
    // piece i of a step's tokens: 16 bytes (i & 3) of run 2 warp + (i / 4 & 1) of token i / 8
    auto fetch_x = [&](int step, int stage) {
#pragma unroll
        for (int j = 0; j < (MT * 8 + 31) / 32; ++j) {
            const int i = lane + 32 * j, k = (2 * warp + (i >> 2 & 1)) * run + step * BK + (i & 3) * 4;
            if (i >= MT * 8) break;
            cp_async16(smem_address(mine + (size_t)stage * Form::STAGE + Form::X_AT + i * 16),
                       k < K ? A + (size_t)min(m0 + (i >> 3), M - 1) * lda + k : A, k < K ? 16 : 0);
        }
    };
    for (int s = 0; s < min(stages - 1, steps); ++s) fetch(s, s);
    pdl_wait();
    const int r = 2 * warp + (lane >> 4);                 // this thread's run of feature lane & 15
    for (int s = 0; s < stages - 1; ++s) {
        if (s < steps) fetch_x(s, s);
        cp_async_commit();                                // (the first group holds all the weights)
    }
    float acc[Form::PER][MT];
#pragma unroll
    for (int f = 0; f < Form::PER; ++f)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[f][m] = 0.f;
    int stage_at = 0;
    for (int step = 0; step < steps; ++step) {
        cp_async_wait_most(stages - 2);
        __syncwarp();
        const int k0 = r * run + step * BK;
        const uint8_t* stage = mine + (size_t)stage_at * Form::STAGE;
        const uint8_t* chunk = stage + lane * FEW_CHUNK;
        const uint8_t* x = stage + Form::X_AT + (lane >> 4) * (BK * 4);
#pragma unroll
        for (int q = 0; q < BK / 4; ++q) {
            if (k0 + 4 * q >= K) break;                   // whole quarters: K is a multiple of 4
            float4 w[Form::PER];
#pragma unroll
            for (int f = 0; f < Form::PER; ++f) w[f] = *reinterpret_cast<const float4*>(chunk + 32 * f * FEW_CHUNK + 16 * q);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 v = *reinterpret_cast<const float4*>(x + m * 2 * BK * 4 + 16 * q);
#pragma unroll
                for (int f = 0; f < Form::PER; ++f)
                    acc[f][m] = fmaf(v.w, w[f].w, fmaf(v.z, w[f].z, fmaf(v.y, w[f].y, fmaf(v.x, w[f].x, acc[f][m]))));
            }
        }
        __syncwarp();                                     // the stage before this one is read: fill it again
        if (step + stages - 1 < steps) {
            const int free = stage_at == 0 ? stages - 1 : stage_at - 1;
            fetch(step + stages - 1, free);
            fetch_x(step + stages - 1, free);
        }
        cp_async_commit();
        if (++stage_at == stages) stage_at = 0;
    }
    cp_async_wait<0>();
#pragma unroll
    for (int f = 0; f < Form::PER; ++f)
#pragma unroll
        for (int m = 0; m < MT; ++m) parts[r][m][(lane & 15) + FEW_F * f] = acc[f][m];
    __syncthreads();
    const int runs = (K + run - 1) / run;
    for (int i = threadIdx.x; i < MT * Form::F; i += FEW_THREADS) {
        const int f = i % Form::F, m = i / Form::F, n = n0 + f;
        if (m0 + m >= M) break;
        auto total = [&](int at) {
            float v = 0.f;
            for (int s0 = 0; s0 < runs; s0 += GROUP_RUNS) {
                float group = 0.f;
                for (int s = s0; s < min(runs, s0 + GROUP_RUNS); ++s) group += parts[s][m][at];
                v += group;
            }
            return v;
        };
        if (epi == EPI_SWIGLU) {
            if ((f & 1) || n + 1 >= N) continue;
            put<float, EPI_STORE>(C, ldc, m0 + m, n >> 1, swiglu(total(f), total(f + 1)));
        } else if (n < N) {
            if (epi == EPI_ADD) put<float, EPI_ADD>(C, ldc, m0 + m, n, total(f));
            else put<float, EPI_STORE>(C, ldc, m0 + m, n, total(f));
        }
    }
}

// ---------------------------------------------------------------------------------------
// Many tokens.  Thread (r, c) has features r .. r + 3, 64 + r .., (128 + r .., 192 + r ..) of the block's 64 FG, tokens
// c .. c + 3 and 32 + c .. of its 64.  A block has one group of runs; the blocks of the groups are a cluster along z, and each of them finishes a
// share of the tokens.  A group's sums lie in shared memory (one word per thread and value: 64 registers fewer).
constexpr int TILE_T = 64, TILE_K = 16, TILE_THREADS = 128;
template <int FG> struct Tile {                                       // FG groups of four features a thread
    static constexpr int F = 64 * FG, PER = 4 * FG, STAGES = FG == 2 ? 3 : 2, BLOCKS = FG == 2 ? 3 : 2;
    static constexpr int W = F + 4, X = TILE_T + 4;                   // padded: eight k's of four rows meet every bank once
    static constexpr int STAGE = TILE_K * (W + X), VALUES = 8 * PER;
    static constexpr int SMEM = (STAGES * STAGE + VALUES * TILE_THREADS) * 4;
};
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
          "l"(reinterpret_cast<const unsigned long long&>(c)));
    return d;
}

template <int EPI, int FG>
__global__ void __launch_bounds__(TILE_THREADS, Tile<FG>::BLOCKS)
gemm_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                 int M, int N, int K, int lda, int ldw, int ldc) {
    using Form = Tile<FG>;
    constexpr int TILE_F = Form::F, TILE_W = Form::W, TILE_X = Form::X, TILE_STAGE = Form::STAGE, TILE_STAGES = Form::STAGES;
    constexpr int PER = Form::PER, TILE_VALUES = Form::VALUES;
    extern __shared__ __align__(16) float tiles[];        // [stage][W by k, X by k], then [value][thread]: a group's sum
    float* sums = tiles + TILE_STAGES * TILE_STAGE;
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * TILE_T, n0 = blockIdx.x * TILE_F;
    const int run = run_length(K), per_group = GROUP_RUNS * run;
    const int k_begin = (int)blockIdx.z * per_group, k_end = min(K, k_begin + per_group);
    const int steps = (k_end - k_begin + TILE_K - 1) / TILE_K;
    // copy j of a step: k = (tid & 7) + 8 (j & 1), row (tid >> 3) + 16 (j >> 1): eight neighbouring k of a row are one sector
    const int ck = tid & 7, crow = tid >> 3;
    auto fetch = [&](int step, int stage) {
        float* to = tiles + stage * TILE_STAGE;
#pragma unroll
        for (int j = 0; j < TILE_F / 8; ++j) {
            const int k = ck + 8 * (j & 1), row = crow + 16 * (j >> 1), at = k_begin + step * TILE_K + k;
            const bool in = at < k_end && n0 + row < N;
            cp_async4(smem_address(to + k * TILE_W + row), in ? W + (size_t)(n0 + row) * ldw + at : W, in ? 4 : 0);
        }
#pragma unroll
        for (int j = 0; j < TILE_T / 8; ++j) {
            const int k = ck + 8 * (j & 1), row = crow + 16 * (j >> 1), at = k_begin + step * TILE_K + k;
            const bool in = at < k_end && m0 + row < M;
            cp_async4(smem_address(to + TILE_K * TILE_W + k * TILE_X + row), in ? A + (size_t)(m0 + row) * lda + at : A, in ? 4 : 0);
        }
    };
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < steps) fetch(s, s);
        cp_async_commit();
    }
    // acc[i][j]: features 2 i, 2 i + 1 of the thread's, token j of its eight
    float2 acc[PER / 2][8];
#pragma unroll
    for (int i = 0; i < PER / 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
    // value v of a thread: token v / PER, feature v % PER
#pragma unroll
    for (int v = 0; v < TILE_VALUES; ++v) sums[v * TILE_THREADS + tid] = 0.f;
    const int r = (tid >> 3) * 4, c = (tid & 7) * 4;
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<TILE_STAGES - 2>();
        __syncthreads();                                  // this stage has landed, the one before is read by all
        if (step + TILE_STAGES - 1 < steps) fetch(step + TILE_STAGES - 1, (step + TILE_STAGES - 1) % TILE_STAGES);
        cp_async_commit();
        const float* w = tiles + (step % TILE_STAGES) * TILE_STAGE;
        const float* x = w + TILE_K * TILE_W;
        // (a k's values are on their way while the one before is multiplied)
        struct Values { float2 f[PER / 2]; float t[8]; } even, odd;
        auto take = [&](int k, Values& v) {
#pragma unroll
            for (int g = 0; g < FG; ++g) {
                const float4 w4 = *reinterpret_cast<const float4*>(w + k * TILE_W + 64 * g + r);
                v.f[2 * g] = make_float2(w4.x, w4.y);
                v.f[2 * g + 1] = make_float2(w4.z, w4.w);
            }
            const float4 x0 = *reinterpret_cast<const float4*>(x + k * TILE_X + c), x1 = *reinterpret_cast<const float4*>(x + k * TILE_X + 32 + c);
            v.t[0] = x0.x; v.t[1] = x0.y; v.t[2] = x0.z; v.t[3] = x0.w;
            v.t[4] = x1.x; v.t[5] = x1.y; v.t[6] = x1.z; v.t[7] = x1.w;
        };
        auto multiply = [&](const Values& v) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < PER / 2; ++i) acc[i][j] = fma_pair(v.f[i], make_float2(v.t[j], v.t[j]), acc[i][j]);
        };
        take(0, even);
#pragma unroll 2
        for (int k = 0; k < TILE_K; k += 2) {
            take(k + 1, odd);
            multiply(even);
            take(k + 2 < TILE_K ? k + 2 : k, even);
            multiply(odd);
        }
        const int done = k_begin + (step + 1) * TILE_K;
        if (done % run == 0 || step + 1 == steps) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < PER / 2; ++i) {
                    float* at = sums + (PER * j + 2 * i) * TILE_THREADS + tid;
                    at[0] += acc[i][j].x;
                    at[TILE_THREADS] += acc[i][j].y;
                    acc[i][j] = make_float2(0.f, 0.f);
                }
        }
    }
    cp_async_wait<0>();
    const int groups = (int)gridDim.z;
    if (groups > 1)                                       // all blocks' sums are there
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    uint32_t of[MAX_RUNS / GROUP_RUNS];
#pragma unroll
    for (int z = 0; z < MAX_RUNS / GROUP_RUNS; ++z)
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(of[z]) : "r"(smem_address(sums + tid)), "r"(z < groups ? z : 0));
    const int per = (8 + groups - 1) / groups, j0 = (int)blockIdx.z * per, j1 = min(8, j0 + per);
    const bool vectors = (EPI == EPI_SWIGLU ? ldc % 2 == 0 && ((uintptr_t)C & 7) == 0 : ldc % 4 == 0 && ((uintptr_t)C & 15) == 0);
    for (int j = j0; j < j1; ++j) {
        float g[PER][MAX_RUNS / GROUP_RUNS];
#pragma unroll
        for (int i = 0; i < PER; ++i)
#pragma unroll
            for (int z = 0; z < MAX_RUNS / GROUP_RUNS; ++z) {
                g[i][z] = 0.f;
                if (z < groups)
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(g[i][z]) : "r"(of[z] + (uint32_t)((PER * j + i) * TILE_THREADS * 4)) : "memory");
            }
        float v[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            v[i] = 0.f;
#pragma unroll
            for (int z = 0; z < MAX_RUNS / GROUP_RUNS; ++z) v[i] += g[i][z];
        }
        const int m = m0 + (j < 4 ? c + j : 28 + c + j);
        if (m >= M) continue;
#pragma unroll
        for (int half = 0; half < FG; ++half) {
            const int n = n0 + 64 * half + r;
            const float* q = v + 4 * half;
            if (EPI == EPI_SWIGLU) {
                float* at = C + (size_t)m * ldc + (n >> 1);
                if (vectors && n + 3 < N) {
                    *reinterpret_cast<float2*>(at) = make_float2(swiglu(q[0], q[1]), swiglu(q[2], q[3]));
                } else {
                    if (n + 1 < N) at[0] = swiglu(q[0], q[1]);
                    if (n + 3 < N) at[1] = swiglu(q[2], q[3]);
                }
            } else if (vectors && n + 3 < N) {
                float4* at = reinterpret_cast<float4*>(C + (size_t)m * ldc + n);
                float4 o = EPI == EPI_ADD ? *at : make_float4(0.f, 0.f, 0.f, 0.f);
                *at = EPI == EPI_ADD ? make_float4(o.x + q[0], o.y + q[1], o.z + q[2], o.w + q[3]) : make_float4(q[0], q[1], q[2], q[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (n + i < N) put<float, EPI>(C, ldc, m, n + i, q[i]);
            }
        }
    }
    if (groups > 1)                                       // nobody's sums may go away while a neighbour reads them
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Stages of a warp's ring.  A block that has its SM to itself takes what shared memory there is, so that enough of the weights
// is on its way; where blocks follow one another on an SM, several at once hide one's start and end behind the others', the
// more of them the more follow.  us per launch with 2 / 3 / 4 / 5 stages and more, weights in rotation: 3 tokens, 2,048 x
// 2,048: - / 9.1 / 8.7 / 7.3, x 6,144: - / 23.2 / 22.9 / 17.3, 12,288 x 2,048: - / 27.0 / 27.5 / 40.1, 32,000 x 2,048:
// 53.9 / 60.8 / 61.2 / 96; one token, 12,288 and 32,000: 23.1 / 20.1 / 22.2 / 21.8 and 42.0 / 43.2 / 45.8 / 45.9.
inline int few_stages(long long blocks, int stage_bytes, int static_bytes) {
    const long long per_sm = (blocks + kipp_sm_count() - 1) / kipp_sm_count();
    const int at_once = per_sm <= 1 ? 1 : per_sm <= 8 ? 2 : 4, most = per_sm <= 2 ? FEW_STAGES_MAX : 3;
    const int fit = (227 * 1024 / at_once - static_bytes - 1024) / stage_bytes;
    return fit < 2 ? 2 : fit > most ? most : fit;
}
template <int MT, bool PAIR>
int launch_few_form(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int epi, cudaStream_t s) {
    using F = Few<PAIR, MT>;
    const dim3 grid((N + F::F - 1) / F::F, (M + MT - 1) / MT);
    constexpr int parts = MAX_RUNS * MT * (F::F + 1) * 4;                 // what the kernel declares beside the ring
    const int stages = few_stages((long long)grid.x * grid.y, F::BLOCK_STAGE, parts);
    const size_t smem = (size_t)stages * F::BLOCK_STAGE;
    if (const int e = kipp_allow_smem(gemm_few_kernel<MT, PAIR>, smem + parts)) return e;
    return kipp_launch(gemm_few_kernel<MT, PAIR>, grid, dim3(FEW_THREADS), smem, s, 1, C, A, W, M, N, K, lda, ldw, ldc, epi, stages);
}
template <int MT>
int launch_few(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int epi, cudaStream_t s) {
    // pairs of features for 5 to 8 tokens of many features (6 tokens, 32,000 x 2,048: 58.0 us, 64.5 with one a thread; 12,288: level;
    // 3 tokens: 55.3 and 53.9, 29.4 and 27.0)
    constexpr bool MAY_PAIR = MT == 8;
    if (MAY_PAIR && N >= many_features()) return launch_few_form<MT, MAY_PAIR>(C, A, W, M, N, K, lda, ldw, ldc, epi, s);
    return launch_few_form<MT, false>(C, A, W, M, N, K, lda, ldw, ldc, epi, s);
}

template <int EPI, int FG>
int launch_tile(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int groups, cudaStream_t s) {
    using Form = Tile<FG>;
    const dim3 grid((N + Form::F - 1) / Form::F, (M + TILE_T - 1) / TILE_T, groups);
    if (grid.y > 65535) return KIPP_ERR_ARG;
    if (const int e = kipp_allow_smem(gemm_tile_kernel<EPI, FG>, Form::SMEM)) return e;
    return kipp_launch(gemm_tile_kernel<EPI, FG>, grid, dim3(TILE_THREADS), Form::SMEM, s, groups, C, A, W, M, N, K, lda, ldw, ldc);
}
// 128 or 256 features a block, by what the SM with the most blocks has to do: a block of 256 takes 1.88 of 128's time beside
// another one, 2.3 alone.  us a product in tiles of 128 / 256: 399 tokens, 12,288 x 2,048: 617 / 588, 3,072 x 2,048: 173 / 175,
// 2,048 x 6,144: 369 / 348; 64 tokens: 104 / 131, 58 / 70, 118 / 194; 1,024 tokens: 1,366 / 1,282, 355 / 338, 713 / 708.  The one
// chosen is within 7 % of the better everywhere that was measured (64 to 1,024 tokens).
inline int run_groups(int K) { return (K + GROUP_RUNS * run_length(K) - 1) / (GROUP_RUNS * run_length(K)); }
inline int tile_features(int M, int N, int groups) {
    const long long t_tiles = (M + TILE_T - 1) / TILE_T, sms = kipp_sm_count();
    auto per_sm = [&](int f) { return (t_tiles * ((N + f - 1) / f) * groups + sms - 1) / sms; };
    const double narrow = (double)per_sm(Tile<2>::F), wide = (double)per_sm(Tile<4>::F);
    return (wide <= 1 ? 2.3 : 1.88 * wide) < narrow ? Tile<4>::F : Tile<2>::F;
}

// float32 rows that start on 16 bytes and hold whole groups of four: the kernels that copy 16 bytes at a time.
template <int EPI>
int launch_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
    if (few_tokens(M, N)) {
        // tokens of a block: as many as there are, up to 16 (the accumulators of a thread)
        if (M == 1) return launch_few<1>(C, A, W, M, N, K, lda, ldw, ldc, EPI, s);
        if (M == 2) return launch_few<2>(C, A, W, M, N, K, lda, ldw, ldc, EPI, s);
        if (M <= 4) return launch_few<4>(C, A, W, M, N, K, lda, ldw, ldc, EPI, s);
        if (M <= 8) return launch_few<8>(C, A, W, M, N, K, lda, ldw, ldc, EPI, s);
        return launch_few<16>(C, A, W, M, N, K, lda, ldw, ldc, EPI, s);
    }
    const int groups = run_groups(K);
    return tile_features(M, N, groups) == Tile<4>::F ? launch_tile<EPI, 4>(C, A, W, M, N, K, lda, ldw, ldc, groups, s)
                                                     : launch_tile<EPI, 2>(C, A, W, M, N, K, lda, ldw, ldc, groups, s);
}

template <typename TA, typename TW, typename TC, bool RUNS>
int launch(void* C, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldc,
           int epi, cudaStream_t s) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return KIPP_ERR_ARG;
    switch (epi) {
    case EPI_STORE:
        return kipp_launch(gemm_simt_kernel<TA, TW, TC, EPI_STORE, RUNS>, grid, dim3(256), 0, s, 1, (TC*)C, (const TA*)A,
                           (const TW*)W, M, N, K, lda, ldw, ldc);
    case EPI_ADD:
        return kipp_launch(gemm_simt_kernel<TA, TW, TC, EPI_ADD, RUNS>, grid, dim3(256), 0, s, 1, (TC*)C, (const TA*)A,
                           (const TW*)W, M, N, K, lda, ldw, ldc);
    case EPI_SWIGLU:
        if (N & 1) return KIPP_ERR_ARG;
        return kipp_launch(gemm_simt_kernel<TA, TW, TC, EPI_SWIGLU, RUNS>, grid, dim3(256), 0, s, 1, (TC*)C, (const TA*)A,
                           (const TW*)W, M, N, K, lda, ldw, ldc);
    default:
        return KIPP_ERR_ARG;
    }
}
}  // namespace

// in_dtype: dtype of A and W (both float32 or both bfloat16); out_dtype: dtype of C.
// Features of the tiles that a 32-bit product of this size is made in (128 or 256), or 0 where the kernel for few tokens makes it.
extern "C" int kipp_gemm_simt_tile_features(int M, int N, int K) {
    if (few_tokens(M, N)) return 0;
    return tile_features(M, N, run_groups(K));
}
extern "C" int kipp_gemm_simt(void* C, int out_dtype, const void* A, const void* W, int in_dtype,
                              int M, int N, int K, int lda, int ldw, int ldc, int epilogue,
                              void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return KIPP_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (epilogue == EPI_ADD && out_dtype != KIPP_DT_F32) return KIPP_ERR_DTYPE;
    // `shared`: weights that all three kernels may be given, and so have one order of sums for
    const bool shared = K % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)W & 15) == 0;
    const bool vectors = shared && lda % 4 == 0 && ((uintptr_t)A & 15) == 0;
    if (in_dtype == KIPP_DT_F32 && out_dtype == KIPP_DT_F32 && vectors) {
        if (epilogue == EPI_STORE) return launch_f32<EPI_STORE>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, s);
        if (epilogue == EPI_ADD) return launch_f32<EPI_ADD>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, s);
        if (epilogue == EPI_SWIGLU && N % 2 == 0)
            return launch_f32<EPI_SWIGLU>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, s);
    }
    if (in_dtype == KIPP_DT_F32 && out_dtype == KIPP_DT_F32)
        return shared ? launch<float, float, float, true>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, s)
                      : launch<float, float, float, false>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, s);
    if (in_dtype == KIPP_DT_BF16 && out_dtype == KIPP_DT_F32)
        return launch<bf16, bf16, float, false>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, s);
    if (in_dtype == KIPP_DT_BF16 && out_dtype == KIPP_DT_BF16)
        return launch<bf16, bf16, bf16, false>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, s);
    return KIPP_ERR_DTYPE;
}
