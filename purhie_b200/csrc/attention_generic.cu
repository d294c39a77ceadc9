// Attention over cache pages, the plain kernel: any head size, any number of heads and groups, float32
// arithmetic.  It is the whole attention of the 32-bit path, the reference the fast kernels are tested
// against, and the refuge for head sizes the fast kernels do not take.
//
// Values may have another width (DV) than keys (D); the output row of a head is DV wide.  A value row may also be the
// first DV elements of a wider row (v_stride elements from one token's to the next's): values kept inside the key rows.
// One warp per (token row, query head).  The row at absolute position z of a request sees the cached
// positions lo .. z, lo = max(0, z - window + 1) (window 0: lo = 0); with a block mask (chunk > 0) it sees only
// the positions of its own block of `chunk` positions counted from 0, lo = max(lo, floor(z / chunk) * chunk).
// Keys are taken 32 at a time
// starting from lo: each lane scores one key (the whole dot product in one lane, in d order), the warp
// keeps a running maximum and sum (online softmax) and each lane owns the output dimensions d = lane,
// lane + 32, ...  The order of every addition depends on (z, window) only, never on how the request was
// cut into steps or on what else is in the batch.
// A sink (one float32 number per query head, or none) is one more term exp(sink) in the softmax's denominator: it has no
// key and no value, is not scaled, and counts once whatever the window holds.
// A cap (0: none) bends the scaled score s to cap * tanh(s / cap).
// A distance bias (one slope per query head, or none) takes slope_h * (z - p) off the scaled score of the key at p.  A gate
// (rows of HQ * DV logits, or none) multiplies the output by sigmoid(gate), element by element.
// Formulas (reference): src/qwen_ops.cpp:26-51 (scores * scale, max-subtracted softmax, weighted sum of
// V; query head h uses kv head h / (HQ / HKV)); window: src/attention.h:73.
#include "async_copy.cuh"
#include "common.cuh"
#include "shared_limit.cuh"

#include <math.h>

#include <algorithm>

namespace {

using namespace ph;

constexpr int WARPS = 4;
constexpr int MAX_D = 640;

template <typename TQ, typename TKV, typename TO>
__global__ void attention_generic_kernel(const TQ* __restrict__ q, const TKV* __restrict__ k_base,
                                         const TKV* __restrict__ v_base, long long page_stride, int page_size,
                                         const int32_t* __restrict__ block_table, int table_stride,
                                         const int32_t* __restrict__ row_seg, const int32_t* __restrict__ positions,
                                         TO* __restrict__ out, int T, int HQ, int HKV, int D, int window, float scale, int DV, int chunk, int VS,
                                         const float* __restrict__ sink, const float* __restrict__ slopes, const TQ* __restrict__ gate,
                                         long long gate_stride, float cap) {
    __shared__ float qs[WARPS][MAX_D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)T * HQ) return;
    const int t = (int)(item / HQ), h = (int)(item % HQ);
    const int g = h / (HQ / HKV);
    const int z = positions[t];
    int lo = (window > 0 && z - window + 1 > 0) ? z - window + 1 : 0;
    if (chunk > 0 && z / chunk * chunk > lo) lo = z / chunk * chunk;
    const int32_t* table = block_table + (size_t)row_seg[t] * table_stride;
    const TQ* qr = q + ((size_t)t * HQ + h) * D;
    for (int d = lane; d < D; d += 32) qs[warp][d] = to_float<TQ>(qr[d]);
    __syncwarp();

    const float slope = slopes ? slopes[h] : 0.0f;
    float m = -INFINITY, l = 0.0f;
    float acc[MAX_D / 32];
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) acc[i] = 0.0f;

    for (int base = lo; base <= z; base += 32) {
        const int p = base + lane;
        float s = -INFINITY;
        const TKV* vrow = nullptr;
        if (p <= z) {
            const int page = table[p / page_size];
            const size_t at = (size_t)g * page_size + p % page_size;
            const TKV* krow = k_base + (size_t)page * page_stride + at * D;
            vrow = v_base + (size_t)page * page_stride + at * VS;
            float dot = 0.0f;
            for (int d = 0; d < D; ++d) dot += qs[warp][d] * to_float<TKV>(krow[d]);
            s = dot * scale;
            if (cap > 0.0f) s = cap * tanhf(s / cap);
            if (slopes) s -= slope * (float)(z - p);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float pexp = (p <= z) ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);            // m = -inf on the first chunk: corr = 0, l and acc are 0
        l = l * corr + warp_sum(pexp);
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) acc[i] *= corr;
        const int n = (z - base + 1) < 32 ? (z - base + 1) : 32;
        for (int j = 0; j < n; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pexp, j);
            const unsigned long long vp = __shfl_sync(0xffffffffu, (unsigned long long)vrow, j);
            const TKV* vj = (const TKV*)vp;
#pragma unroll
            for (int i = 0; i < MAX_D / 32; ++i) {
                const int d = lane + 32 * i;
                if (d < DV) acc[i] += pj * to_float<TKV>(vj[d]);
            }
        }
        m = m_new;
    }
    TO* o = out + ((size_t)t * HQ + h) * DV;
    if (sink) {
        // the sink joins the denominator under the larger of the two maxima
        const float sk = sink[h], top = fmaxf(m, sk), corr = expf(m - top);
        l = l * corr + expf(sk - top);
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) acc[i] *= corr;
    }
    const float inv = 1.0f / l;
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) {
        const int d = lane + 32 * i;
        if (d >= DV) continue;
        float v = acc[i] * inv;
        if (gate) v *= 1.0f / (1.0f + expf(-to_float<TQ>(gate[(size_t)t * gate_stride + (size_t)h * DV + d])));
        o[d] = from_float<TO>(v);
    }
}


// ---- float32, head sizes 32, 64 and 128 ----------------------------------------------------------------------------
struct F32Params {
    const float *q, *k_base, *v_base;
    long long page_stride;
    const int32_t *block_table, *row_seg, *positions;
    float* out;
    const float *sink, *slopes, *gate;
    long long gate_stride;
    int page_size, table_stride, T, HQ, HKV, window, chunk, v_stride;
    float scale, cap;
    int tiles;                       // tokens of a CTA of the tile kernel, which has the rows of runs of at least RUN_MIN (0: no tiles)
};

constexpr int RUN_MIN = 4;           // tokens of one request side by side that the tile kernel takes
constexpr int FEW_ROWS_PER_SM = 64;  // (token, head) rows an SM below which a warp of the tile kernel takes four instead of eight
constexpr int KEYS = 128;            // keys a CTA of the rows kernel scores at once

// The score of a key from its dot product, every operation rounded by itself as in the plain kernel.
__device__ __forceinline__ float bent_score(float dot, float scale, float cap, bool biased, float slope, int distance) {
    float s = __fmul_rn(dot, scale);
    if (cap > 0.0f) s = cap * tanhf(s / cap);
    if (biased) s = fmaf(-slope, (float)distance, s);
    return s;
}

// Bit i: the token lo + i (of at most 32, below `end`) belongs to request `seg`.  All lanes of a warp call it.
__device__ __forceinline__ unsigned tokens_of(const int32_t* row_seg, int lo, int end, int seg) {
    const int t = lo + (threadIdx.x & 31);
    return __ballot_sync(0xffffffffu, t < end && row_seg[t] == seg);
}
// Ones of the mask from bit b on, side by side (b up to 32).
__device__ __forceinline__ int ones_from(unsigned mask, int b) {
    if (b > 31) return 0;
    const unsigned gap = ~mask >> b;
    return gap ? __ffs(gap) - 1 : 32 - b;
}
// The tokens, in order, that lie in a run shorter than RUN_MIN, runs being cut at multiples of `tile` tokens (8, 16 or 32).
struct Leftovers {
    const int32_t* row_seg;
    int T, tile;
    int base = 0, before = 0;                          // the tokens from `base` on have `before` such tokens in front of them
    // The wanted-th (from 0; no smaller than in the call before) of them; -1: there are fewer.  All lanes of a warp call it.
    __device__ int token(int wanted) {
        const int lane = threadIdx.x & 31;
        for (; base < T; base += 128) {
            int seg[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = base + 32 * i + lane;
                seg[i] = t < T ? row_seg[t] : -1;
            }
            int count = before;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int front = __shfl_up_sync(0xffffffffu, seg[i], 1);
                const unsigned joined = __ballot_sync(0xffffffffu, lane % tile != 0 && seg[i] == front);      // to the token in front
                const int start = lane - ones_from(__brev(joined), 31 - lane);
                const bool left = base + 32 * i + lane < T && 1 + ones_from(joined, start + 1) < RUN_MIN;
                const unsigned lefts = __ballot_sync(0xffffffffu, left);
                if (wanted < count + __popc(lefts)) return base + 32 * i + (int)__fns(lefts, 0, wanted - count + 1);
                count += __popc(lefts);
            }
            before = count;
        }
        return -1;
    }
};

// One CTA of 128 threads per (token row, query head), or one for every SM for what the tile kernel leaves.  KEYS keys at a
// time: their rows come by cp.async (the values of a block under its scores, the keys of the next block under the values'
// sums), thread j scores key j, every warp takes the maximum and the sum of its 32 keys, and thread d adds up output d over
// the keys in order.  What bounds it: the chain of KEYS dependent multiply-adds of a score's D numbers and of an output's
// KEYS keys per block, one warp a scheduler.  Four rows of 256 keys, 16 heads of 128: 9.4 us (the plain kernel 214); eight rows of
// 1,024: 31 us (836).
// LEFT: only the rows that the tile kernel leaves (the search costs registers, and with them a tenth of the speed at D = 32).
template <int D, bool LEFT>
__global__ void __launch_bounds__(128, 1) attention_rows_f32_kernel(const F32Params p) {
    constexpr int KS = D + 4;
    extern __shared__ __align__(16) float smem[];
    float* ks = smem;                                  // [KEYS][D + 4]
    float* vs = ks + KEYS * KS;                        // [KEYS][D]
    float* qs = vs + KEYS * D;                         // [D]
    float* ps = qs + D;                                // [KEYS]
    float* tops = ps + KEYS;                           // [KEYS / 32] maxima, then sums
    float* sums = tops + KEYS / 32;
    long long* at = reinterpret_cast<long long*>(sums + KEYS / 32);   // [2][KEYS] where each key row and value row starts
    const int h = blockIdx.x % p.HQ, g = h / (p.HQ / p.HKV);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    pdl_wait();
    Leftovers leftovers{p.row_seg, p.T, p.tiles};
    for (int row = blockIdx.x / p.HQ;; row += gridDim.x / p.HQ) {
        // this CTA's next row: of all, or of those that the tile kernel leaves
        const int t = LEFT ? leftovers.token(row) : row < p.T ? row : -1;
        if (t < 0) return;
        const int z = p.positions[t], lo = first_seen(z, p.window, p.chunk);
        const int32_t* table = p.block_table + (size_t)p.row_seg[t] * p.table_stride;
        long long page = 0, slot = 0;                  // of key `base + tid` of the block that is fetched next
        auto place = [&](int base) {
            const int key = base + tid;
            if (key <= z) {
                page = table[key / p.page_size];
                slot = (long long)g * p.page_size + key % p.page_size;
            }
        };
        auto places = [&]() {
            at[tid] = page * p.page_stride + slot * D;
            at[KEYS + tid] = page * p.page_stride + slot * p.v_stride;
        };
        // rows of D numbers: D / 4 threads a row
        constexpr int PER_ROW = D / 4, STEP = 128 / PER_ROW;
        const int r0 = tid / PER_ROW, c4 = tid % PER_ROW * 4;
        auto fetch = [&](float* dst, int stride, const float* base_ptr, const long long* where, int n) {
#pragma unroll 8
            for (int r = r0; r < n; r += STEP) copy16(dst + r * stride + c4, base_ptr + where[r] + c4);
            copies_commit();
        };
        place(lo);
        places();
        if (tid < D) qs[tid] = p.q[((size_t)t * p.HQ + h) * D + tid];
        __syncthreads();
        int n = min(KEYS, z - lo + 1);
        fetch(ks, KS, p.k_base, at, n);
        fetch(vs, D, p.v_base, at + KEYS, n);
        const bool biased = p.slopes != nullptr;
        const float slope = biased ? p.slopes[h] : 0.0f;
        float m = -INFINITY, l = 0.0f, acc = 0.0f;
        for (int base = lo; base <= z; base += KEYS) {
            n = min(KEYS, z - base + 1);
            const int next = min(KEYS, z - base - KEYS + 1);           // keys of the block behind (none: <= 0)
            place(base + KEYS);
            copies_wait<1>();                                          // this block's keys
            __syncthreads();
            float s = -INFINITY;
            if (tid < n) {
                const float* kr = ks + tid * KS;
                // four float4s of the key and of q are fetched while the four in front are multiplied
                float dot = 0.0f;
                float4 a[2][4], b[2][4];
                auto take = [&](int d, int to) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) { a[to][i] = load4(qs + d + 4 * i); b[to][i] = load4(kr + d + 4 * i); }
                };
                take(0, 0);
#pragma unroll
                for (int d = 0; d < D; d += 16) {
                    const int now = d / 16 & 1;
                    if (d + 16 < D) take(d + 16, now ^ 1);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        dot = fmaf(a[now][i].x, b[now][i].x, dot);
                        dot = fmaf(a[now][i].y, b[now][i].y, dot);
                        dot = fmaf(a[now][i].z, b[now][i].z, dot);
                        dot = fmaf(a[now][i].w, b[now][i].w, dot);
                    }
                }
                s = bent_score(dot, p.scale, p.cap, biased, slope, z - (base + tid));
            }
            const float top = warp_max(s);
            if (lane == 0) tops[warp] = top;
            __syncthreads();                                           // (every score is made: the key rows may be overwritten)
            float run[KEYS / 32 + 1], mine = 0.0f;                     // the running maximum in front of and behind every 32 keys
            run[0] = m;
#pragma unroll
            for (int i = 0; i < KEYS / 32; ++i) {
                run[i + 1] = fmaxf(run[i], tops[i]);
                if (i == warp) mine = run[i + 1];
            }
            const float pe = tid < n ? expf(s - mine) : 0.0f;
            ps[tid] = pe;
            const float sum = warp_sum(pe);
            if (lane == 0) sums[warp] = sum;
            if (next > 0) places();
            copies_wait<0>();                                          // this block's values
            __syncthreads();
            if (next > 0) fetch(ks, KS, p.k_base, at, next);
#pragma unroll
            for (int i = 0; i < KEYS / 32; ++i) {
                if (i * 32 >= n) break;
                const float corr = expf(run[i] - run[i + 1]);
                l = fmaf(l, corr, sums[i]);
                if (tid < D) {
                    acc *= corr;
                    if (n >= (i + 1) * 32) {
                        const float* v = vs + i * 32 * D + tid;
                        float4 w4[8];
                        float vj[32];
#pragma unroll
                        for (int j = 0; j < 8; ++j) w4[j] = load4(ps + i * 32 + 4 * j);
#pragma unroll
                        for (int j = 0; j < 32; ++j) vj[j] = v[j * D];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            acc = fmaf(w4[j].x, vj[4 * j], acc);
                            acc = fmaf(w4[j].y, vj[4 * j + 1], acc);
                            acc = fmaf(w4[j].z, vj[4 * j + 2], acc);
                            acc = fmaf(w4[j].w, vj[4 * j + 3], acc);
                        }
                    } else {
                        for (int j = i * 32; j < n; ++j) acc = fmaf(ps[j], vs[j * D + tid], acc);
                    }
                }
                m = run[i + 1];
            }
            if (next > 0) {
                __syncthreads();                                       // the value rows, weights, maxima and sums are read
                fetch(vs, D, p.v_base, at + KEYS, next);
            }
        }
        if (tid < D) {
            if (p.sink) {
                const float sk = p.sink[h], top = fmaxf(m, sk), corr = expf(m - top);
                l = fmaf(l, corr, expf(sk - top));
                acc *= corr;
            }
            float v = acc * (1.0f / l);
            if (p.gate) v *= 1.0f / (1.0f + expf(-p.gate[(size_t)t * p.gate_stride + (size_t)h * D + tid]));
            p.out[((size_t)t * p.HQ + h) * D + tid] = v;
        }
        __syncthreads();                                               // the row's buffers are read
    }
}

// One CTA of 128 threads per (4 R / HH tokens side by side, HH heads of one kv head), for rows that see every position up to
// their own.  Runs of one request in turn; per run 32 keys at a time from position 0 on (two buffers), every warp for its own
// R rows: scores and softmax with a lane per key, sums over the values with D / 32 outputs a lane.  What bounds it: a warp's
// chain of blocks (few rows), the shared-memory reads beside the multiply-adds (many rows: 9 float4s for 32 of them in the
// scores, 3 in the sums at R = 8).
template <int D, int HH, int R>
__global__ void __launch_bounds__(128, 2) attention_tile_f32_kernel(const F32Params p) {
    constexpr int ROWS = 4 * R, TT = ROWS / HH, KS = D + 4, V = D / 32;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                  // [ROWS][D]
    float* ks = qs + ROWS * D;                         // [2][32][D + 4]
    float* vs = ks + 2 * 32 * KS;                      // [2][32][D]
    float* ss = vs + 2 * 32 * D;                       // [4 warps][32 keys][R rows] weights
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int heads = p.HQ / HH, t0 = (int)(gridDim.x / heads - 1 - blockIdx.x / heads) * TT;      // the last tokens first
    const int h0 = blockIdx.x % heads * HH, g = h0 / (p.HQ / p.HKV);
    const int t_end = min(t0 + TT, p.T);
    // row r: token t0 + r / HH, head h0 + r % HH
    constexpr int PER_ROW = D / 4, STEP = 128 / PER_ROW;
    const int r0 = tid / PER_ROW, c4 = tid % PER_ROW * 4;
#pragma unroll 4
    for (int r = r0; r < ROWS; r += STEP) {
        const int t = t0 + r / HH;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (t < t_end) v = load4(p.q + ((size_t)t * p.HQ + h0 + r % HH) * D + c4);
        *reinterpret_cast<float4*>(qs + r * D + c4) = v;
    }
    const bool biased = p.slopes != nullptr;
    const float* qw = qs + warp * R * D;
    float* sw = ss + warp * 32 * R;
    for (int first = t0; first < t_end;) {
        const int seg = p.row_seg[first], from = first;
        const int last = first + ones_from(tokens_of(p.row_seg, t0, t_end, seg), first - t0);
        first = last;
        if (last - from < RUN_MIN) continue;                       // the rows kernel's
        const int32_t* table = p.block_table + (size_t)seg * p.table_stride;
        const int z_lane = p.positions[min(from + lane, last - 1)];
        const int zmax = __reduce_max_sync(0xffffffffu, z_lane), zmin = __reduce_min_sync(0xffffffffu, z_lane);
        int zr[R];                                                 // the last position each of the warp's rows sees (-1: not in this run)
        float m[R], l[R], acc[R][V];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int t = t0 + (warp * R + i) / HH;
            zr[i] = t >= from && t < last ? p.positions[t] : -1;
            m[i] = -INFINITY;
            l[i] = 0.0f;
#pragma unroll
            for (int e = 0; e < V; ++e) acc[i][e] = 0.0f;
        }
        int page = 0, slot = 0;                                    // of key `lane` of the block that is fetched next
        auto place = [&](int base) {
            const int key = base + lane;
            if (key <= zmax) {
                page = table[key / p.page_size];
                slot = g * p.page_size + key % p.page_size;
            }
        };
        auto fetch = [&](int base, int buffer) {
            if (base <= zmax) {
#pragma unroll
                for (int i = 0; i < 32 / STEP; ++i) {
                    const int r = r0 + i * STEP;
                    const long long at = (long long)__shfl_sync(0xffffffffu, page, r) * p.page_stride, s = __shfl_sync(0xffffffffu, slot, r);
                    if (base + r <= zmax) {
                        copy16(ks + (buffer * 32 + r) * KS + c4, p.k_base + at + s * D + c4);
                        copy16(vs + (buffer * 32 + r) * D + c4, p.v_base + at + s * p.v_stride + c4);
                    }
                }
            }
            copies_commit();
        };
        __syncthreads();                                           // q is in place; the run in front has read its buffers
        place(0);
        fetch(0, 0);
        place(32);
        // rows of this warp that are all in the run and see a whole block take the plain loop, else key by key
        const bool inside = t0 + warp * R / HH >= from && t0 + (warp * R + R - 1) / HH < last;
        for (int base = 0; base <= zmax; base += 32) {
            const int buffer = base / 32 & 1;
            copies_wait<0>();
            __syncthreads();
            fetch(base + 32, buffer ^ 1);
            place(base + 64);
            const float* kr = ks + (buffer * 32 + lane) * KS;
            const float* vb = vs + buffer * 32 * D + lane * V;
            float pe[R];                                           // this lane's key: dot products, then weights
#pragma unroll
            for (int i = 0; i < R; ++i) pe[i] = 0.0f;
            float4 a[2][R], b[2];
            auto take = [&](int d, int to) {
                b[to] = load4(kr + d);
#pragma unroll
                for (int i = 0; i < R; ++i) a[to][i] = load4(qw + i * D + d);
            };
            take(0, 0);
#pragma unroll
            for (int d = 0; d < D; d += 4) {
                const int now = d / 4 & 1;
                if (d + 4 < D) take(d + 4, now ^ 1);
#pragma unroll
                for (int i = 0; i < R; ++i) pe[i] = fmaf(a[now][i].x, b[now].x, pe[i]);
#pragma unroll
                for (int i = 0; i < R; ++i) pe[i] = fmaf(a[now][i].y, b[now].y, pe[i]);
#pragma unroll
                for (int i = 0; i < R; ++i) pe[i] = fmaf(a[now][i].z, b[now].z, pe[i]);
#pragma unroll
                for (int i = 0; i < R; ++i) pe[i] = fmaf(a[now][i].w, b[now].w, pe[i]);
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                // (a row that sees none of the block keeps its maximum: its factor is 1, its weights are 0)
                const int key = base + lane, h = h0 + (warp * R + i) % HH;
                const bool seen = key <= zr[i];
                const float s = seen ? bent_score(pe[i], p.scale, p.cap, biased, biased ? p.slopes[h] : 0.0f, zr[i] - key) : -INFINITY;
                const float m_new = fmaxf(m[i], warp_max(s));
                pe[i] = seen ? expf(s - m_new) : 0.0f;
                const float corr = expf(m[i] - m_new);
                l[i] = fmaf(l[i], corr, warp_sum(pe[i]));
                m[i] = m_new;
#pragma unroll
                for (int e = 0; e < V; ++e) acc[i][e] *= corr;
            }
            __syncwarp();                                          // the last block's weights are read
#pragma unroll
            for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(sw + lane * R + i) = make_float4(pe[i], pe[i + 1], pe[i + 2], pe[i + 3]);
            __syncwarp();
            auto add = [&](int j, bool check) {
                float v[V], w[R];
                const float* vj = vb + j * D;
                if constexpr (V == 4) {
                    const float4 x = load4(vj);
                    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
                } else if constexpr (V == 2) {
                    const float2 x = *reinterpret_cast<const float2*>(vj);
                    v[0] = x.x; v[1] = x.y;
                } else {
                    v[0] = vj[0];
                }
#pragma unroll
                for (int i = 0; i < R; i += 4) {
                    const float4 x = load4(sw + j * R + i);
                    w[i] = x.x; w[i + 1] = x.y; w[i + 2] = x.z; w[i + 3] = x.w;
                }
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (check && base + j > zr[i]) continue;
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[i][e] = fmaf(w[i], v[e], acc[i][e]);
                }
            };
            if (inside && base + 31 <= zmin) {
#pragma unroll 16
                for (int j = 0; j < 32; ++j) add(j, false);
            } else {
                const int n = min(32, zmax - base + 1);
#pragma unroll 4
                for (int j = 0; j < n; ++j) add(j, true);
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (zr[i] < 0) continue;
            const int r = warp * R + i, t = t0 + r / HH, h = h0 + r % HH;
            float ls = l[i], corr = 1.0f;
            if (p.sink) {
                const float sk = p.sink[h], top = fmaxf(m[i], sk);
                corr = expf(m[i] - top);
                ls = fmaf(ls, corr, expf(sk - top));
            }
            const float inv = 1.0f / ls;
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int d = lane * V + e;
                float v = acc[i][e];
                if (p.sink) v *= corr;
                v *= inv;
                if (p.gate) v *= 1.0f / (1.0f + expf(-p.gate[(size_t)t * p.gate_stride + (size_t)h * D + d]));
                p.out[((size_t)t * p.HQ + h) * D + d] = v;
            }
        }
    }
}

template <int D, int HH, int R>
int launch_tiles_f32(F32Params& p, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)(4 * R * D + 2 * 32 * (D + 4) + 2 * 32 * D + 4 * 32 * R) * sizeof(float);
    constexpr auto kernel = attention_tile_f32_kernel<D, HH, R>;
    if (int e = allow_shared<kernel>(bytes, "attention_generic")) return e;
    p.tiles = 4 * R / HH;
    kernel<<<(unsigned)((p.T + p.tiles - 1) / p.tiles * (p.HQ / HH)), 128, bytes, stream>>>(p);
    return check_launch("attention_generic");
}

template <int D, bool LEFT>
int launch_rows_f32(const F32Params& p, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)(KEYS * (D + 4) + KEYS * D + D + KEYS + 2 * (KEYS / 32)) * sizeof(float) + 2 * KEYS * sizeof(long long);
    constexpr auto kernel = attention_rows_f32_kernel<D, LEFT>;
    if (int e = allow_shared<kernel>(bytes, "attention_generic")) return e;
    long long rows = p.T;
    if (LEFT) {
        // How many rows the tiles leave is known on the device only: all of a batch of decoded tokens, none of a prompt.  So a CTA for
        // every SM takes them in turn.  512 decoded tokens of 200 keys, 4 heads of 32: 87 us (with 16 CTAs a head 214, the plain
        // kernel 176); 256 portions of three: 83 (249, 105); 64 tokens of 1,024 keys, one head of 128: 44 (140, 1,708); a prompt of
        // 512, which leaves none, one head of 128: 62 (62).  As many CTAs as an SM holds (five at D = 32) would take 38 us for the
        // first of these, but where nothing is left, as behind a prompt, the kernel behind them then stood still for 13 us (a tiny
        // model's prompt of 97 tokens and two answers: 381 -> 409 us).
        rows = std::min<long long>(rows, std::max(1, multiprocessors() / p.HQ));
    }
    // (started early only where its CTAs are few, as the float32 product; behind the tile kernel, which lets nothing start before
    // its own CTAs have ended, always)
    if (LEFT || 2 * rows * p.HQ <= multiprocessors()) launch_overlapped(kernel, dim3((unsigned)(rows * p.HQ)), dim3(128), bytes, stream, p);
    else kernel<<<(unsigned)(rows * p.HQ), 128, bytes, stream>>>(p);
    return check_launch("attention_generic");
}

// Portions of at least RUN_MIN tokens go to the tile kernel in steps of more than 32 rows without a window; the rows kernel
// takes the rest of such a step (all of it, where every portion is short) and every other step whole.  Four rows a warp while
// tiles of eight would leave the schedulers with one or two warps each (16 heads of 128: 39 against 63 us at 256 tokens, 76
// against 123 at 512; 242 both ways at 1,024).
template <int D>
int launch_f32(F32Params p, cudaStream_t stream) {
    if (p.T > 32 && !p.window && !p.chunk) {
        const bool two = (p.HQ / p.HKV) % 2 == 0, eight = (long long)p.T * p.HQ >= (long long)FEW_ROWS_PER_SM * multiprocessors();
        const int e = two ? (eight ? launch_tiles_f32<D, 2, 8>(p, stream) : launch_tiles_f32<D, 2, 4>(p, stream))
                          : (eight ? launch_tiles_f32<D, 1, 8>(p, stream) : launch_tiles_f32<D, 1, 4>(p, stream));
        if (e) return e;
    }
    return p.tiles ? launch_rows_f32<D, true>(p, stream) : launch_rows_f32<D, false>(p, stream);
}

}  // namespace

// sink, slopes: [HQ] float32 or null.  gate: rows of HQ * DV logits in q's dtype, gate_stride elements apart, or null.
PH_EXPORT int ph_attention_generic_capped(const void* q, int q_dtype, const void* k_base, const void* v_base, int kv_dtype,
                                          long long page_stride, int page_size, const int32_t* block_table,
                                          int table_stride, const int32_t* row_seg, const int32_t* positions, void* out,
                                          int out_dtype, int T, int HQ, int HKV, int D, int window, float scale, int DV,
                                          int chunk, int v_stride, const float* sink, const float* slopes, const void* gate,
                                          long long gate_stride, float cap, cudaStream_t stream) {
    if (!q || !k_base || !v_base || !block_table || !row_seg || !positions || !out || T < 0 || HQ < 1 || HKV < 1 ||
        D < 1 || page_size < 1 || window < 0 || chunk < 0 || cap < 0.0f || !valid_dtype(q_dtype) || !valid_dtype(kv_dtype) ||
        !valid_dtype(out_dtype))
        return fail(PH_ERR_ARG, "attention_generic: bad arguments (T %d, HQ %d, HKV %d, D %d)", T, HQ, HKV, D);
    if (HQ % HKV) return fail(PH_ERR_ARG, "attention_generic: %d query heads are not a multiple of %d kv heads", HQ, HKV);
    if (DV <= 0) DV = D;                     // values as wide as keys
    if (v_stride <= 0) v_stride = DV;        // value rows lie side by side (else: v_stride elements apart, inside wider rows)
    if (D > MAX_D || DV > MAX_D) return fail(PH_ERR_UNSUPPORTED, "attention_generic: head_dim %d / %d exceeds the supported %d", D, DV, MAX_D);
    if (T == 0) return PH_OK;
    const long long items = (long long)T * HQ;
    // the float32 kernels read rows of whole 16 bytes
    const bool on16 = ((uintptr_t)q | (uintptr_t)k_base | (uintptr_t)v_base) % 16 == 0 && page_stride % 4 == 0 && v_stride % 4 == 0;
    if (q_dtype == PH_F32 && kv_dtype == PH_F32 && out_dtype == PH_F32 && D == DV && (D == 32 || D == 64 || D == 128) && on16 &&
        items <= 0x7fffffff) {
        const F32Params p = {(const float*)q, (const float*)k_base, (const float*)v_base, page_stride, block_table, row_seg, positions,
                             (float*)out, sink, slopes, (const float*)gate, gate_stride, page_size, table_stride, T, HQ, HKV, window, chunk,
                             v_stride, scale, cap, 0};
        return D == 128 ? launch_f32<128>(p, stream) : D == 64 ? launch_f32<64>(p, stream) : launch_f32<32>(p, stream);
    }
    const unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
#define LAUNCH(TQ, TKV, TO)                                                                                    \
    attention_generic_kernel<TQ, TKV, TO><<<blocks, WARPS * 32, 0, stream>>>(                                  \
        (const TQ*)q, (const TKV*)k_base, (const TKV*)v_base, page_stride, page_size, block_table, table_stride, \
        row_seg, positions, (TO*)out, T, HQ, HKV, D, window, scale, DV, chunk, v_stride, sink, slopes, (const TQ*)gate, gate_stride, cap)
    PH_DISPATCH(q_dtype, TQ, PH_DISPATCH(kv_dtype, TKV, PH_DISPATCH(out_dtype, TO, LAUNCH(TQ, TKV, TO))));
#undef LAUNCH
    return check_launch("attention_generic");
}

PH_EXPORT int ph_attention_generic_biased(const void* q, int q_dtype, const void* k_base, const void* v_base, int kv_dtype,
                                          long long page_stride, int page_size, const int32_t* block_table,
                                          int table_stride, const int32_t* row_seg, const int32_t* positions, void* out,
                                          int out_dtype, int T, int HQ, int HKV, int D, int window, float scale, int DV,
                                          int chunk, int v_stride, const float* sink, const float* slopes, const void* gate,
                                          long long gate_stride, cudaStream_t stream) {
    return ph_attention_generic_capped(q, q_dtype, k_base, v_base, kv_dtype, page_stride, page_size, block_table, table_stride, row_seg,
                                       positions, out, out_dtype, T, HQ, HKV, D, window, scale, DV, chunk, v_stride, sink, slopes, gate,
                                       gate_stride, 0.0f, stream);
}

PH_EXPORT int ph_attention_generic_sink(const void* q, int q_dtype, const void* k_base, const void* v_base, int kv_dtype,
                                        long long page_stride, int page_size, const int32_t* block_table,
                                        int table_stride, const int32_t* row_seg, const int32_t* positions, void* out,
                                        int out_dtype, int T, int HQ, int HKV, int D, int window, float scale, int DV,
                                        int chunk, int v_stride, const float* sink, cudaStream_t stream) {
    return ph_attention_generic_biased(q, q_dtype, k_base, v_base, kv_dtype, page_stride, page_size, block_table, table_stride, row_seg,
                                       positions, out, out_dtype, T, HQ, HKV, D, window, scale, DV, chunk, v_stride, sink, nullptr, nullptr,
                                       0, stream);
}

PH_EXPORT int ph_attention_generic(const void* q, int q_dtype, const void* k_base, const void* v_base, int kv_dtype,
                                   long long page_stride, int page_size, const int32_t* block_table,
                                   int table_stride, const int32_t* row_seg, const int32_t* positions, void* out,
                                   int out_dtype, int T, int HQ, int HKV, int D, int window, float scale, int DV,
                                   int chunk, int v_stride, cudaStream_t stream) {
    return ph_attention_generic_sink(q, q_dtype, k_base, v_base, kv_dtype, page_stride, page_size, block_table, table_stride, row_seg,
                                     positions, out, out_dtype, T, HQ, HKV, D, window, scale, DV, chunk, v_stride, nullptr, stream);
}
