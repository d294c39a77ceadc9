// y[M, N] = x[M, K] * w[N, K]^T on the CUDA cores, float32 multiply-add, one fixed order.
//
// Every output element is the sum over k = 0, 1, ..., K-1 taken in that order by one thread, whatever M
// and N are and wherever the element lies in its tile, so a row's result does not depend on the batch it
// is in, nor on which of the kernels below computed it.  No tensor cores and no reduced-precision mode: this is the
// matrix product of the 32-bit path (the reference's exact-order F32 kernels: src/matvec_q.hip:837-991), the plain
// reference of the tensor-core kernels, and the product for shapes they refuse.  x and w may be float32 or bfloat16
// (widened exactly), y float32 or bfloat16.
//
// Three kernels, one order of additions:
//   gemm_rows_f32   float32 with at most 16 rows: the weight streams through a ring in shared memory (decoding)
//   gemm_tile_f32   float32 with more rows: register tiles, operands by cp.async with k left contiguous
//   gemm_simple     any other type, K not a multiple of 4 or an operand off 16 bytes
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

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256) gemm_simple_kernel(const TX* __restrict__ x, const TW* __restrict__ w,
                                                          TY* __restrict__ y, int M, int N, int K) {
    __shared__ float xs[BK][BM + 1];
    __shared__ float ws[BK][BN + 1];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tr = tid / (BN / TN), tc = tid % (BN / TN);      // 16 x 16 threads
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k = 1024 elements of each operand, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;
            const int r = idx / BK, kk = idx % BK;
            const int k = k0 + kk;
            float xv = 0.0f, wv = 0.0f;
            if (k < K) {
                if (m0 + r < M) xv = to_float<TX>(x[(size_t)(m0 + r) * K + k]);
                if (n0 + r < N) wv = to_float<TW>(w[(size_t)(n0 + r) * K + k]);
            }
            xs[kk][r] = xv;
            ws[kk][r] = wv;
        }
        __syncthreads();
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
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + tr * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tc * TN + j;
            if (n < N) y[(size_t)m * N + n] = from_float<TY>(acc[i][j]);
        }
    }
}


// ---- float32: 16-byte asynchronous copies --------------------------------------------------------------------------
// A row of an operand in shared memory holds its k side by side, padded by 16 bytes: eight neighbouring rows then start
// in eight different groups of four banks, so lanes that read float4s of eight rows (the same k) ask for every bank once.
// (The counters show about three wavefronts for such a read in gemm_tile_f32 all the same.)

// Few rows.  A CTA owns BN_ columns and all MB rows: its 128 threads keep STAGES chunks of KC numbers of its weight rows (and
// of x) on their way, and BN_ * MB / RM of them multiply, one column and RM rows each.  What bounds it: the chain of K
// dependent multiply-adds of an output (4 cycles each: 1.1 us per 512 numbers) where the columns are few, the weight's way
// from memory where they are many.
constexpr int KC = 128, KC_STRIDE = KC + 4;
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
    float acc[RM];
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[i] = 0.0f;
    for (int c = 0; c < chunks; ++c) {
        copies_wait<STAGES - 2>();
        __syncthreads();
        request(c + STAGES - 1);                                   // into the place that chunk c - 1 has left
        if (tid < WORKERS) {
            const float* ws = ring + ((size_t)(c % STAGES) * ROWS + n) * KC_STRIDE;
            const float* xs = ring + ((size_t)(c % STAGES) * ROWS + BN_ + mg * RM) * KC_STRIDE;
            // G float4s of each operand are fetched while the G in front of them are multiplied: left to the compiler, the
            // chain waits for shared memory (4 x 1024 x 3072: 13 to 22 us by the unrolling alone)
            constexpr int G = RM == 1 ? 4 : 2;
            float4 a[2][RM][G], b[2][G];
            auto fetch = [&](int group, int to) {
#pragma unroll
                for (int j = 0; j < G; ++j) {
                    b[to][j] = load4(ws + (group * G + j) * 4);
#pragma unroll
                    for (int i = 0; i < RM; ++i) a[to][i][j] = load4(xs + i * KC_STRIDE + (group * G + j) * 4);
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
                        acc[i] = fmaf(a[now][i][j].x, b[now][j].x, acc[i]);
                        acc[i] = fmaf(a[now][i][j].y, b[now][j].y, acc[i]);
                        acc[i] = fmaf(a[now][i][j].z, b[now][j].z, acc[i]);
                        acc[i] = fmaf(a[now][i][j].w, b[now][j].w, acc[i]);
                    }
            }
        }
    }
    copies_wait<0>();
    pdl_launch_dependents();
    if (tid >= WORKERS || n0 + n >= N) return;
#pragma unroll
    for (int i = 0; i < RM; ++i)
        if (mg * RM + i < M) y[(size_t)(mg * RM + i) * N + n0 + n] = acc[i];
}

// Many rows.  A CTA of two warps owns 32 x 32 outputs, a thread 4 x 4 of them, its rows and columns interleaved with its
// neighbours' (lanes: 8 columns x 4 rows), so that a read takes four k of eight rows and no bank twice.  Both operands keep k
// contiguous in shared memory, which cp.async can write without a transposition through registers.  What bounds it: the
// shared-memory reads (81 % of their rate at 1024 x 6144 x 1024) and the issue of the multiply-adds (68 %).  Many small CTAs
// that wait for their own copies only are as fast as larger tiles where there are many outputs (1024 x 6144 x 1024: 319 us,
// 41 TFLOP/s, 313 to 333 with tiles of 64 x 64, 128 x 128 and 32 x 64; the plain kernel 680) and faster where there are few
// (256 x 1024 x 3072: 60 us, 74 to 320; the plain kernel 302).
constexpr int BK32 = 32, BK32_STRIDE = BK32 + 4, TILE_STAGES = 3, TILE = 32;
__global__ void __launch_bounds__(64) gemm_tile_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                           int M, int N, int K) {
    constexpr int ROWS = 2 * TILE;                                 // of the ring: TILE of x, then TILE of w
    extern __shared__ __align__(16) float ring[];                  // [TILE_STAGES][ROWS][BK32_STRIDE]
    const int tid = threadIdx.x, lane = tid & 31, tx = lane & 7, ty = tid >> 5 << 2 | lane >> 3;
    const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
    const int chunks = (K + BK32 - 1) / BK32;
    pdl_wait();
    auto request = [&](int c) {
        if (c < chunks) {
            float* dst = ring + (size_t)(c % TILE_STAGES) * ROWS * BK32_STRIDE;
            const int k = c * BK32 + (tid & 7) * 4;
#pragma unroll
            for (int e = 0; e < ROWS / 8; ++e) {                   // eight threads a row
                const int r = tid / 8 + e * 8;
                const bool is_x = r < TILE;
                const bool valid = k < K && (is_x ? m0 + r < M : n0 + r - TILE < N);
                const float* src = is_x ? x + (size_t)(m0 + r) * K : w + (size_t)(n0 + r - TILE) * K;
                copy16(dst + r * BK32_STRIDE + (tid & 7) * 4, valid ? src + k : w, valid);
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int c = 0; c < TILE_STAGES - 1; ++c) request(c);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    for (int c = 0; c < chunks; ++c) {
        copies_wait<TILE_STAGES - 2>();
        __syncthreads();
        request(c + TILE_STAGES - 1);                              // into the place that chunk c - 1 has left
        const float* xs = ring + ((size_t)(c % TILE_STAGES) * ROWS + ty) * BK32_STRIDE;
        const float* ws = ring + ((size_t)(c % TILE_STAGES) * ROWS + TILE + tx) * BK32_STRIDE;
#pragma unroll
        for (int k = 0; k < BK32; k += 4) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = load4(xs + i * 8 * BK32_STRIDE + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = load4(ws + j * 8 * BK32_STRIDE + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    copies_wait<0>();
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * 8;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * 8;
            if (n < N) y[(size_t)m * N + n] = acc[i][j];
        }
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

// Columns a CTA takes: 8 while there are at most two such CTAs an SM (a product as narrow as that is as long as its chains:
// 4 x 1024 x 3072 takes 10.8 us with 8 columns and a deep ring, 12 with 16, 20 with 32); 32 with a row or a few per thread
// beyond (4 x 4096 x 1024: 6.7 us, 11.3 with 8, 9.2 with 64); 64 for two to four rows of more columns than that is good for
// (4 x 6144 x 1024: 9.6 against 10.8 us; 4 x 151936 x 1024, which streams 622 MB: 121 against 140 us).  The plain kernel took
// 291, 99, 171 and 1,224 us.
template <int MB>
int plan_rows(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    const long long sms = multiprocessors();
    if (N <= 16 * sms) return launch_rows<8, MB, 1, MB <= 8 ? 10 : 8>(x, w, y, M, N, K, stream);
    if constexpr (MB == 2 || MB == 4)
        if (N > 32 * sms) return launch_rows<64, MB, MB / 2, 3>(x, w, y, M, N, K, stream);
    return launch_rows<32, MB, MB <= 4 ? 1 : MB / 4, 4>(x, w, y, M, N, K, stream);
}

int gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M == 1) return plan_rows<1>(x, w, y, M, N, K, stream);
    if (M == 2) return plan_rows<2>(x, w, y, M, N, K, stream);
    if (M <= 4) return plan_rows<4>(x, w, y, M, N, K, stream);
    if (M <= 8) return plan_rows<8>(x, w, y, M, N, K, stream);
    if (M <= 16) return plan_rows<16>(x, w, y, M, N, K, stream);
    // (16 rows as tiles: 20.5 against 18.9 us at 6144 x 1024, 52 against 17.5 at 1024 x 3072)
    constexpr size_t bytes = (size_t)TILE_STAGES * 2 * TILE * BK32_STRIDE * sizeof(float);
    if (int e = allow_shared<gemm_tile_f32_kernel>(bytes, "gemm_simple")) return e;
    const dim3 grid((N + TILE - 1) / TILE, (M + TILE - 1) / TILE);
    if (2ll * grid.x * grid.y <= multiprocessors()) launch_overlapped(gemm_tile_f32_kernel, grid, dim3(64), bytes, stream, x, w, y, M, N, K);
    else gemm_tile_f32_kernel<<<grid, 64, bytes, stream>>>(x, w, y, M, N, K);
    return check_launch("gemm_simple");
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
