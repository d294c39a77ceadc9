// y[M, N] = x[M, K] * w[N, K]^T on the CUDA cores, float32 multiply-add, one fixed order.
//
// Every output element is the sum, in ascending order, of its blocks of 128 of K, and a block is the sum over its even k plus
// the sum over its odd k, each a chain of multiply-adds in ascending order, whatever M and N are and wherever the element lies
// in its tile, so a row's result does not depend on the batch it is in, nor on which of the kernels below computed it.  Blocks
// let several warps work on one output (a single chain over K bounds a product of few outputs: 4 x 1024 x 3072 took 12.9 us as
// one chain a thread, 8.4 now) and err less than one chain does (logits of the 0.6B shape against 64 bits: 2.1e-6 -> 6.6e-7);
// even and odd k are what one packed multiply-add takes.  No tensor cores and no reduced-precision mode: this is the
// matrix product of the 32-bit path (the reference's exact-order F32 kernels: src/matvec_q.hip:837-991), the plain
// reference of the tensor-core kernels, and the product for shapes they refuse.  x and w may be float32 or bfloat16
// (widened exactly), y float32 or bfloat16.
//
// Four kernels, one order of additions:
//   gemm_rows_f32        float32 with at most 16 rows: the weight streams through a ring in shared memory (decoding)
//   gemm_rows_split_f32  the same where the columns are few: the warps of a CTA share out K
//   gemm_tile_f32        float32 with more rows: register tiles, operands by cp.async with k left contiguous
//   gemm_simple          any other type, K not a multiple of 4 or an operand off 16 bytes
// The float32 kernels start early only where their CTAs are few (at most one for every second SM:
// a tiny model's three streams of 12 tokens 1.78 -> 1.64 ms).  Elsewhere, started early, their CTAs pile up on the SMs that the kernel in
// front leaves first, and with one or two CTAs an SM that imbalance cost a 256-row layer of a 0.6B
// model 61 us (428 against 367).
#include "async_copy.cuh"
#include "common.cuh"
#include "shared_limit.cuh"

namespace {

using namespace ph;

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
constexpr int KC = 128;                                            // a block of K

// Two neighbouring k in one packed multiply-add, and the two sums added.
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ float sum_of(uint64_t acc) {
    return __fadd_rn(__uint_as_float((uint32_t)acc), __uint_as_float((uint32_t)(acc >> 32)));
}

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256) gemm_simple_kernel(const TX* __restrict__ x, const TW* __restrict__ w,
                                                          TY* __restrict__ y, int M, int N, int K) {
    __shared__ float xs[BK][BM + 1];
    __shared__ float ws[BK][BN + 1];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tr = tid / (BN / TN), tc = tid % (BN / TN);      // 16 x 16 threads
    float total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) total[i][j] = 0.0f;

    // 64 rows x 16 k = 1024 elements of each operand, 4 per thread, on their way while the 16 k in front of them are multiplied: few
    // CTAs wait for little else (bfloat16, us with one chain an output, with blocks of K, and now: 1 x 4096 x 1020 185, 195 and 78;
    // 512 x 4096 x 1020 317, 336 and 251; 1024 x 4096 x 1020 456, 480 and 434)
    float xv[4], wv[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = (tid + e * 256) / BK, k = k0 + tid % BK;
            xv[e] = k < K && m0 + r < M ? to_float<TX>(x[(size_t)(m0 + r) * K + k]) : 0.0f;
            wv[e] = k < K && n0 + r < N ? to_float<TW>(w[(size_t)(n0 + r) * K + k]) : 0.0f;
        }
    };
    fetch(0);
    for (int block = 0; block < K; block += KC) {
        float acc[TM][TN][2];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0f;
        const int end = min(block + KC, K);
        for (int k0 = block; k0 < end; k0 += BK) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                xs[tid % BK][(tid + e * 256) / BK] = xv[e];
                ws[tid % BK][(tid + e * 256) / BK] = wv[e];
            }
            __syncthreads();
            fetch(k0 + BK);
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[TM], b[TN];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = xs[kk][tr * TM + i];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = ws[kk][tc * TN + j];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j][kk & 1] = fmaf(a[i], b[j], acc[i][j][kk & 1]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) total[i][j] += __fadd_rn(acc[i][j][0], acc[i][j][1]);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + tr * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tc * TN + j;
            if (n < N) y[(size_t)m * N + n] = from_float<TY>(total[i][j]);
        }
    }
}


// ---- float32: 16-byte asynchronous copies --------------------------------------------------------------------------
// A row of an operand in shared memory holds its k side by side, padded by 16 bytes: eight neighbouring rows then start
// in eight different groups of four banks, so lanes that read float4s of eight rows (the same k) ask for every bank once.
// (The counters show about three wavefronts for such a read in gemm_tile_f32 all the same.)

// Few rows.  A CTA owns BN_ columns and all MB rows: its 128 threads keep STAGES chunks of KC numbers of its weight rows (and
// of x) on their way, and BN_ * MB / RM of them multiply, one column and RM rows each.  What bounds it: the chain of K / 2
// dependent multiply-adds of an output and the weight's way from memory.
constexpr int KC_STRIDE = KC + 4;
// One block of K: acc[i] += the products of row i of xs with ws, even and odd k apart.  G float4s of each operand are fetched
// while the G in front of them are multiplied: left to the compiler, the chain waits for shared memory.
template <int RM>
__device__ __forceinline__ void multiply_block(const float* xs, const float* ws, uint64_t (&acc)[RM]) {
    constexpr int G = RM == 1 ? 4 : RM <= 4 ? 2 : 1;
    ulonglong2 a[2][RM][G], b[2][G];
    auto fetch = [&](int group, int to) {
#pragma unroll
        for (int j = 0; j < G; ++j) {
            b[to][j] = *(const ulonglong2*)(ws + (group * G + j) * 4);
#pragma unroll
            for (int i = 0; i < RM; ++i) a[to][i][j] = *(const ulonglong2*)(xs + i * KC_STRIDE + (group * G + j) * 4);
        }
    };
    fetch(0, 0);
#pragma unroll
    for (int group = 0; group < KC / 4 / G; ++group) {
        const int now = group & 1;
        if (group + 1 < KC / 4 / G) fetch(group + 1, now ^ 1);
#pragma unroll
        for (int j = 0; j < G; ++j)
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                fma2(acc[i], a[now][i][j].x, b[now][j].x);
                fma2(acc[i], a[now][i][j].y, b[now][j].y);
            }
    }
}

template <int BN_, int MB, int RM, int STAGES>
__global__ void __launch_bounds__(128) gemm_rows_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                            int M, int N, int K) {
    extern __shared__ __align__(16) float ring[];                  // [STAGES][BN_ + MB][KC_STRIDE]
    constexpr int ROWS = BN_ + MB, WORKERS = BN_ * (MB / RM);
    static_assert(WORKERS <= 128 && MB % RM == 0, "one CTA holds every output");
    const int tid = threadIdx.x, n0 = blockIdx.x * BN_;
    const int chunks = (K + KC - 1) / KC;
    pdl_wait();
    auto request = [&](int c) {
        if (c < chunks) {
            float* dst = ring + (size_t)(c % STAGES) * ROWS * KC_STRIDE;
            const int k0 = c * KC;
#pragma unroll
            for (int e = 0; e < (ROWS * (KC / 4) + 127) / 128; ++e) {
                const int i = tid + e * 128, r = i / (KC / 4), k = i % (KC / 4) * 4;
                if (ROWS * (KC / 4) % 128 && r >= ROWS) break;
                const bool is_w = r < BN_;
                const bool valid = k0 + k < K && (is_w ? n0 + r < N : r - BN_ < M);
                const float* src = is_w ? w + (size_t)(n0 + r) * K : x + (size_t)(r - BN_) * K;
                copy16(dst + r * KC_STRIDE + k, valid ? src + k0 + k : w, valid);
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) request(c);
    const int n = tid % BN_, mg = tid / BN_;                       // this thread's column, and its rows mg * RM ...
    float total[RM];
#pragma unroll
    for (int i = 0; i < RM; ++i) total[i] = 0.0f;
    for (int c = 0; c < chunks; ++c) {
        copies_wait<STAGES - 2>();
        __syncthreads();
        request(c + STAGES - 1);                                   // into the place that chunk c - 1 has left
        if (tid < WORKERS) {
            const float* ws = ring + ((size_t)(c % STAGES) * ROWS + n) * KC_STRIDE;
            const float* xs = ring + ((size_t)(c % STAGES) * ROWS + BN_ + mg * RM) * KC_STRIDE;
            uint64_t acc[RM];
#pragma unroll
            for (int i = 0; i < RM; ++i) acc[i] = 0;
            multiply_block<RM>(xs, ws, acc);
#pragma unroll
            for (int i = 0; i < RM; ++i) total[i] += sum_of(acc[i]);
        }
    }
    copies_wait<0>();
    pdl_launch_dependents();
    if (tid >= WORKERS || n0 + n >= N) return;
#pragma unroll
    for (int i = 0; i < RM; ++i)
        if (mg * RM + i < M) y[(size_t)(mg * RM + i) * N + n0 + n] = total[i];
}

// Few rows and few columns.  A CTA owns BN_ columns and all MB rows, and its W warps share out K: a warp takes CH neighbouring
// blocks of 128 at a time, its lanes an output (or RM rows of a column) of one of them, through a ring of its own that no other
// warp waits for.  The sums of blocks meet in shared memory after every round and are added in ascending order.  What bounded
// such a product was the chain of K multiply-adds of an output in one thread; a chain is 64 long here, whatever K is.
template <int BN_, int MB, int RM, int W, int STAGES>
__global__ void __launch_bounds__(W * 32) gemm_rows_split_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                                     int M, int N, int K) {
    extern __shared__ __align__(16) float ring[];                  // [W][STAGES][CH][BN_ + MB][KC_STRIDE], then the sums
    constexpr int ROWS = BN_ + MB, LANES = BN_ * (MB / RM), CH = 32 / LANES, OUT = BN_ * MB, HELD = (OUT + W * 32 - 1) / (W * 32);
    static_assert(LANES * CH == 32 && MB % RM == 0, "a warp's lanes share out its blocks");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n0 = blockIdx.x * BN_;
    const int blocks = (K + KC - 1) / KC, rounds = (blocks + W * CH - 1) / (W * CH);
    float* mine = ring + (size_t)warp * STAGES * CH * ROWS * KC_STRIDE;
    float* sums = ring + (size_t)W * STAGES * CH * ROWS * KC_STRIDE;               // [2][W * CH][OUT]
    pdl_wait();
    auto request = [&](int i) {
        if (i < rounds) {
            float* dst = mine + (size_t)(i % STAGES) * CH * ROWS * KC_STRIDE + lane * 4;
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) {
                const int k = ((i * W + warp) * CH + ch) * KC + lane * 4;
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const bool is_w = r < BN_, valid = k < K && (is_w ? n0 + r < N : r - BN_ < M);
                    const float* src = is_w ? w + (size_t)(n0 + r) * K : x + (size_t)(r - BN_) * K;
                    copy16(dst + (ch * ROWS + r) * KC_STRIDE, valid ? src + k : w, valid);
                }
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) request(i);
    const int n = lane % BN_, mg = lane / BN_ % (MB / RM), ch = lane / LANES;
    float total[HELD];
#pragma unroll
    for (int u = 0; u < HELD; ++u) total[u] = 0.0f;
    for (int i = 0; i < rounds; ++i) {
        copies_wait<STAGES - 2>();
        __syncwarp();
        request(i + STAGES - 1);                                   // into the place that round i - 1 has left
        const float* at = mine + ((size_t)(i % STAGES) * CH + ch) * ROWS * KC_STRIDE;
        const float *ws = at + n * KC_STRIDE, *xs = at + (BN_ + mg * RM) * KC_STRIDE;
        uint64_t acc[RM];
#pragma unroll
        for (int j = 0; j < RM; ++j) acc[j] = 0;
        multiply_block<RM>(xs, ws, acc);
        float* to = sums + ((size_t)(i & 1) * W * CH + warp * CH + ch) * OUT + mg * RM * BN_ + n;
#pragma unroll
        for (int j = 0; j < RM; ++j) to[j * BN_] = sum_of(acc[j]);
        __syncthreads();
        const int here = min(W * CH, blocks - i * W * CH);
#pragma unroll
        for (int u = 0; u < HELD; ++u) {
            const int o = tid + u * W * 32;
            if (OUT % (W * 32) && o >= OUT) break;
            const float* from = sums + (size_t)(i & 1) * W * CH * OUT + o;
            for (int b = 0; b < here; ++b) total[u] += from[b * OUT];
        }
    }
    copies_wait<0>();
    pdl_launch_dependents();
#pragma unroll
    for (int u = 0; u < HELD; ++u) {
        const int o = tid + u * W * 32, m = o / BN_, nn = n0 + o % BN_;
        if (o < OUT && m < M && nn < N) y[(size_t)m * N + nn] = total[u];
    }
}

// Many rows.  A CTA owns 32 x 32 outputs and GROUPS groups of 64 threads that share out K: group g takes every GROUPS-th block of
// 128, through a ring of its own; after each round the groups' sums of an output meet in shared memory and are added in
// ascending order.  A thread holds 4 x 4 outputs, rows and columns interleaved with its neighbours' (lanes: 8 columns x 4 rows),
// with k contiguous in shared memory, where cp.async puts it without a transposition and where two neighbouring k are one
// operand of a packed multiply-add.  What bounds it: the shared-memory reads (1024 x 6144 x 1024: 330 us, 39 TFLOP/s; 64 x 32
// tiles, which read less, hold too few warps an SM and take 364 to 388).
constexpr int BK32 = 32, BK32_STRIDE = BK32 + 4, TILE_STAGES = 2, TILE = 32, SUM_STRIDE = TILE + 8;
__host__ __device__ constexpr int tile_floats(int groups) { return groups * (TILE_STAGES * 2 * TILE * BK32_STRIDE + TILE * SUM_STRIDE); }
template <int GROUPS>
__global__ void __launch_bounds__(64 * GROUPS, 8 / GROUPS) gemm_tile_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                                float* __restrict__ y, int M, int N, int K) {
    constexpr int RM = TM, ROWS = 2 * TILE, PER = KC / BK32, HELD = TILE * TILE / (64 * GROUPS);
    extern __shared__ __align__(16) float ring[];                  // [GROUPS][TILE_STAGES][ROWS][BK32_STRIDE], [GROUPS][TILE][SUM_STRIDE]
    const int tid = threadIdx.x, group = tid >> 6, gt = tid & 63, lane = tid & 31, tx = lane & 7, ty = gt >> 5 << 2 | lane >> 3;
    const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
    const int blocks = (K + KC - 1) / KC, rounds = (blocks + GROUPS - 1) / GROUPS;
    float* mine = ring + (size_t)group * TILE_STAGES * ROWS * BK32_STRIDE;
    float* sums = ring + (size_t)GROUPS * TILE_STAGES * ROWS * BK32_STRIDE;
    pdl_wait();
    // part c of this group: block group + GROUPS * (c / PER), its k from 32 * (c % PER)
    auto request = [&](int c) {
        const int k0 = (group + GROUPS * (c / PER)) * KC + c % PER * BK32;
        if (k0 < K) {
            float* dst = mine + (size_t)(c % TILE_STAGES) * ROWS * BK32_STRIDE + (gt & 7) * 4;
            const int k = k0 + (gt & 7) * 4;
#pragma unroll
            for (int e = 0; e < ROWS / 8; ++e) {                   // eight threads a row
                const int r = gt / 8 + e * 8;
                const bool is_x = r < TILE, valid = k < K && (is_x ? m0 + r < M : n0 + r - TILE < N);
                const float* src = is_x ? x + (size_t)(m0 + r) * K : w + (size_t)(n0 + r - TILE) * K;
                copy16(dst + r * BK32_STRIDE, valid ? src + k : w, valid);
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int c = 0; c < TILE_STAGES - 1; ++c) request(c);
    float total[HELD];
#pragma unroll
    for (int u = 0; u < HELD; ++u) total[u] = 0.0f;
    for (int round = 0; round < rounds; ++round) {
        const int block = group + GROUPS * round;
        if (block < blocks) {
            uint64_t acc[RM][TN];
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = 0;
            for (int c = round * PER; c < (round + 1) * PER; ++c) {
                copies_wait<TILE_STAGES - 2>();
                asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory");
                request(c + TILE_STAGES - 1);                      // into the place that part c - 1 has left
                if (block * KC + c % PER * BK32 >= K) continue;
                const float* xs = mine + ((size_t)(c % TILE_STAGES) * ROWS + ty) * BK32_STRIDE;
                const float* ws = mine + ((size_t)(c % TILE_STAGES) * ROWS + TILE + tx) * BK32_STRIDE;
#pragma unroll
                for (int k = 0; k < BK32; k += 4) {
                    ulonglong2 a[RM], b[TN];
#pragma unroll
                    for (int i = 0; i < RM; ++i) a[i] = *(const ulonglong2*)(xs + i * 8 * BK32_STRIDE + k);
#pragma unroll
                    for (int j = 0; j < TN; ++j) b[j] = *(const ulonglong2*)(ws + j * 8 * BK32_STRIDE + k);
#pragma unroll
                    for (int i = 0; i < RM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i].x, b[j].x);
#pragma unroll
                    for (int i = 0; i < RM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i].y, b[j].y);
                }
            }
            float* to = sums + ((size_t)group * TILE + ty) * SUM_STRIDE + tx;
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) to[i * 8 * SUM_STRIDE + j * 8] = sum_of(acc[i][j]);
        }
        __syncthreads();
        const int here = min(GROUPS, blocks - round * GROUPS);
#pragma unroll
        for (int u = 0; u < HELD; ++u) {
            const int o = tid + u * 64 * GROUPS;
            const float* from = sums + (size_t)(o / TILE) * SUM_STRIDE + o % TILE;
            for (int g = 0; g < here; ++g) total[u] += from[(size_t)g * TILE * SUM_STRIDE];
        }
        __syncthreads();
    }
    copies_wait<0>();
    pdl_launch_dependents();
#pragma unroll
    for (int u = 0; u < HELD; ++u) {
        const int o = tid + u * 64 * GROUPS, m = m0 + o / TILE, n = n0 + o % TILE;
        if (m < M && n < N) y[(size_t)m * N + n] = total[u];
    }
}

template <int BN_, int MB, int RM, int STAGES>
int launch_rows(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    const size_t bytes = (size_t)STAGES * (BN_ + MB) * KC_STRIDE * sizeof(float);
    constexpr auto kernel = gemm_rows_f32_kernel<BN_, MB, RM, STAGES>;
    if (int e = allow_shared<kernel>(bytes, "gemm_simple")) return e;
    const int ctas = (N + BN_ - 1) / BN_;
    if (2 * ctas <= multiprocessors()) launch_overlapped(kernel, dim3(ctas), dim3(128), bytes, stream, x, w, y, M, N, K);
    else kernel<<<ctas, 128, bytes, stream>>>(x, w, y, M, N, K);
    return check_launch("gemm_simple");
}

template <int BN_, int MB, int RM, int W, int STAGES>
int launch_rows_split(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    constexpr int CH = 32 / (BN_ * (MB / RM));
    constexpr size_t bytes = ((size_t)W * STAGES * CH * (BN_ + MB) * KC_STRIDE + 2 * W * CH * BN_ * MB) * sizeof(float);
    constexpr auto kernel = gemm_rows_split_f32_kernel<BN_, MB, RM, W, STAGES>;
    if (int e = allow_shared<kernel>(bytes, "gemm_simple")) return e;
    const int ctas = (N + BN_ - 1) / BN_;
    if (2 * ctas <= multiprocessors()) launch_overlapped(kernel, dim3(ctas), dim3(W * 32), bytes, stream, x, w, y, M, N, K);
    else kernel<<<ctas, W * 32, bytes, stream>>>(x, w, y, M, N, K);
    return check_launch("gemm_simple");
}

// Columns a CTA takes: 8 while there are at most two such CTAs an SM; 32 with a row or a few per thread beyond; 64 for two to four
// rows of more columns than that is good for (4 x 151936 x 1024, which streams 622 MB: 121 against 140 us).  With 8, K is shared out
// among the warps where it has three blocks or more (4 x 1024 x 3072: 8.4 us, 12.9 as one chain a thread; 8 x 1024 x 3072: 10.4 and
// 18.1; with one block seven of eight warps would stand by).  A CTA of that form has an SM to itself, so more CTAs than SMs are two
// rounds of it, and with 16 rows a warp has little of K at a time: those gain from a longer K only (us, a chain a thread and shared
// out: 8 x 2048 x 384 3.98 and 5.19, x 768 6.9 and 6.7, x 6144 39.3 and 27.0; 4 x 2368 x 384 3.58 and 4.37, x 896 5.84 and 6.21,
// x 1024 6.72 and 6.61; 16 x 1024 x 384 3.10 and 3.98, x 768 4.98 and 4.90).
template <int MB>
int plan_rows(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    const long long sms = multiprocessors();
    if (N <= 16 * sms) {
        const bool one_round = N <= 8 * sms && MB <= 8;
        if (K > 2 * KC && (one_round || K >= (MB >= 8 ? 768 : 1024)))
            return launch_rows_split<8, MB, MB <= 4 ? 1 : MB / 4, MB == 1 ? 4 : 8, MB == 4 ? 3 : 2>(x, w, y, M, N, K, stream);
        return launch_rows<8, MB, 1, MB <= 8 ? 10 : 8>(x, w, y, M, N, K, stream);
    }
    if constexpr (MB == 2 || MB == 4)
        if (N > 32 * sms) return launch_rows<64, MB, MB / 2, 3>(x, w, y, M, N, K, stream);
    return launch_rows<32, MB, MB <= 4 ? 1 : MB / 4, 4>(x, w, y, M, N, K, stream);
}

template <int GROUPS> int launch_tile(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    constexpr size_t bytes = tile_floats(GROUPS) * sizeof(float);
    constexpr auto kernel = gemm_tile_f32_kernel<GROUPS>;
    if (int e = allow_shared<kernel>(bytes, "gemm_simple")) return e;
    const dim3 grid((N + TILE - 1) / TILE, (M + TILE - 1) / TILE);
    if (2ll * grid.x * grid.y <= multiprocessors()) launch_overlapped(kernel, grid, dim3(64 * GROUPS), bytes, stream, x, w, y, M, N, K);
    else kernel<<<grid, 64 * GROUPS, bytes, stream>>>(x, w, y, M, N, K);
    return check_launch("gemm_simple");
}

int gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M == 1) return plan_rows<1>(x, w, y, M, N, K, stream);
    if (M == 2) return plan_rows<2>(x, w, y, M, N, K, stream);
    if (M <= 4) return plan_rows<4>(x, w, y, M, N, K, stream);
    if (M <= 8) return plan_rows<8>(x, w, y, M, N, K, stream);
    if (M <= 16) return plan_rows<16>(x, w, y, M, N, K, stream);
    // An SM holds eight groups whatever the split.  Few tiles want every group at work on each of them (256 x 1024 x 3072: 61.6 us
    // with four groups a tile, 66 with two, 72 with one).  Beyond, a tile of one group is two warps, so an odd number of them an SM
    // leaves two of its four partitions idle at the end, and two groups a tile do not; else one group reads and adds less
    // (x 1024 x 3072, us with one and with two: 608 rows, five tiles an SM, 147 and 139; 768, six, 152 and 161; 1024, seven, 191 and
    // 184; 1184, eight, 197 and 210; 1536, eleven, 288 and 284; from thirteen on the odd numbers are level, and 2048, fourteen, takes
    // 335 and 358).
    const long long sms = multiprocessors(), tiles = (long long)((M + TILE - 1) / TILE) * ((N + TILE - 1) / TILE);
    if (tiles <= 2 * sms && K > 2 * KC) return launch_tile<4>(x, w, y, M, N, K, stream);
    const long long most = (tiles + sms - 1) / sms;
    if (most % 2 && most < 13 && K > KC) return launch_tile<2>(x, w, y, M, N, K, stream);
    return launch_tile<1>(x, w, y, M, N, K, stream);
}

}  // namespace

PH_EXPORT int ph_gemm_simple(const void* x, int x_dtype, const void* w, int w_dtype, void* y, int y_dtype, int M,
                             int N, int K, cudaStream_t stream) {
    if (!x || !w || !y || M < 0 || N < 1 || K < 1 || !valid_dtype(x_dtype) || !valid_dtype(w_dtype) ||
        !valid_dtype(y_dtype))
        return fail(PH_ERR_ARG, "gemm_simple: bad arguments (M %d, N %d, K %d)", M, N, K);
    if (M == 0) return PH_OK;
    // (rows of whole 16 bytes: K a multiple of 4 and both operands on 16 bytes)
    if (x_dtype == PH_F32 && w_dtype == PH_F32 && y_dtype == PH_F32 && K % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0 &&
        (M + TILE - 1) / TILE <= 65535)
        return gemm_f32((const float*)x, (const float*)w, (float*)y, M, N, K, stream);
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return fail(PH_ERR_UNSUPPORTED, "gemm_simple: %d rows exceed the supported %d", M, 65535 * BM);
#define LAUNCH(TX, TW, TY) \
    gemm_simple_kernel<TX, TW, TY><<<grid, 256, 0, stream>>>((const TX*)x, (const TW*)w, (TY*)y, M, N, K)
    PH_DISPATCH(x_dtype, TX, PH_DISPATCH(w_dtype, TW, PH_DISPATCH(y_dtype, TY, LAUNCH(TX, TW, TY))));
#undef LAUNCH
    return check_launch("gemm_simple");
}
