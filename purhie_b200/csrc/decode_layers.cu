// All layers of a decode step of at most eight rows in one cooperative launch.
//
// A step of few rows reads every weight once and computes little, so its floor is the time of that read; as nine launches a
// layer it spent most of its time between them: each kernel's start, its dependent round trip to memory, its end (0.6B shape,
// one row, 28 layers: 39 us a layer for 40 MB, 6 us at the copy rate).  Here one CTA per SM stays for the whole stack and a
// warp of it does nothing but ask for what the CTA will need, in order, through a ring of shared-memory stages: weights and
// cached keys do not depend on the step's results, so the memory keeps streaming while the CTAs wait for one another.
//
// A layer is five parts with a counter behind each: [q|k|v] product; norm, rotation, cache write and attention; output product
// and addition; gate/up product and activation; down product and addition.  The norms' row factors are applied where a product
// ends (a product is linear in its rows), from sums of squares that the addition leaves.
//
// Products: groups of 16 output rows are dealt to the CTAs so that every CTA streams the same bytes per layer (`shares`); K
// stays whole in a CTA, so a result is written once, by one CTA, and nothing is added up between CTAs.  A stage is 16 weight
// rows x 512 of K, one box of eight blocks of 64, 128-byte swizzled (as 16 copies of 1 KB the same bytes came at 2.6 TB/s, the copy
// engine bound by their number; as a box with the rows outermost two rows meet in a bank: 8B shape 85.7 us).  Eight warps take
// 64 of the 512 each on mma.sync.m16n8k16 with the weights as the 16 rows and the tokens as the 8 columns: the work is a stream from memory (8 rows:
// 16 flops a byte), and this instruction takes both operands from registers as 16-byte reads deliver them, where a
// tensor-memory accumulator would add its own round trip to each of 5 parts.  The eight partial sums are added in ascending
// order of K.
//
// Attention: a (row, kv head) pair's blocks of 32 keys are shared by CTAs of its own, and merged by the last of them to arrive
// (a counter per pair), in ascending order of the keys.  Keys and values come
// as one box per page as in attention_decode_bulk.cu; the step's own key and value are made by the CTA that holds the pair's last
// block, which writes them to the cache and over their row of the stage.
//
// Measured (us a layer behind 2,048 tokens, a launch per operation -> this): 0.6B shape 38.9 -> 27.6 at one row, 51.1 -> 40.6 at eight;
// width 2,048 48.1 -> 36.4 and 61.2 -> 50.1; 8B shape 86.2 -> 79.1 and 98.8 -> 92.6.  What bounds a layer now is the way of a
// result to the other CTAs, five times: barrier and release 1.2 us, the poll 0.7, the rows' way to shared memory 1.2, and in the
// attention twice that for the merge; with larger weights also the copying thread's turn (a stage in 390 ns, 42 GB/s an SM).
//
// Waiting: results pass between CTAs through global memory behind counters (release adds, acquire polls), which is safe
// because the launch is cooperative: all CTAs are resident.  Every wait is bounded; one that runs out reports through the error
// word, and its CTA's threads run on without waiting as they notice, so that no other CTA is held up and the launch ends.  Such a
// thread frees no place of a ring any more (nothing is asked for twice over), and a CTA leaves when all that it asked for has landed.
#include "attention_mma.cuh"
#include "decode_layers.h"
#include "mbarrier.cuh"

#include <cuda.h>

#include <mutex>
#include <vector>

namespace {

using namespace ph;
using namespace ph_attn;
namespace mb = ph_mbar;

constexpr int WARPS = 8;                        // consumer warps; one more for the ring, one for the activations
constexpr int NTHREADS = (WARPS + 2) * 32;
constexpr int CONSUMERS = WARPS * 32;
constexpr int ROWS = 8;                         // most rows of a step
constexpr int SEG = 512;                        // K of a stage
constexpr int STAGE = 16 * SEG * 2;             // a multiple of 1,024, which the swizzle needs
constexpr int PITCH = SEG * 2 + 16;             // bytes between the rows of activations
constexpr int MAPS = 5;                         // descriptors per layer: the four weights, the cache entry
constexpr int MAX_STAGES = 12, MAX_SLOTS = 32;
constexpr int KEYS = 32;                        // keys of a stage
constexpr int D = 128;
constexpr int QPITCH = D * 2 + 16;
constexpr int RED = 20;                         // floats between the tokens of a warp's 16 x 8 partial sums
constexpr int PAGES = 1024;                     // page coordinates kept in shared memory (DecodeStack asks for no more of 148 CTAs)
constexpr int MAX_GROUP = 8;                    // query heads per kv head
constexpr int PARTS = 5;                        // counters per layer
constexpr int MERGE = 20;                       // pieces of a pair that are merged at once

#define PH_ERR_WAIT_LAYERS_RING 131
#define PH_ERR_WAIT_LAYERS_DATA 132
#define PH_ERR_WAIT_LAYERS_PEERS 133

struct Plan {
    int stages, slots, acc_groups;              // ring stages, places for 512 of K of the rows, groups with sums that wait
    size_t x_bytes, bytes;
};

struct Params {
    PhDecodeLayersArgs a;
    int stages, slots, acc_groups, x_bytes, page_shift;
    long long rows_per_page;
    float scale_log2;
    long long wait_cycles;
};

__host__ __device__ inline int segments(int k) { return (k + SEG - 1) / SEG; }
// Segments of K whose rows are in shared memory at once: all of them, or halves of the places in turn.
__host__ __device__ inline int chunk_of(int nseg, int slots) { return nseg <= slots ? nseg : slots / 2; }

// How the blocks of keys of all (row, kv head) pairs are dealt, from the rows' lengths, the same by every CTA.  A piece costs its
// blocks and about 13 more (5 us: queries, the chain of waits, what its warps and then its pair's pieces add up).
//   Whole CTAs: a pair has CTAs of its own, more of them where a row is longer, and a CTA has one piece at most (0.6B shape, one row
//   of 2,048: with pieces of two pairs in a CTA the others waited 5 us a layer for it).  A row gets whole multiples of the kv heads,
//   so the largest piece can be far from the even share.
//   Even shares: the pairs end to end, each as 13 and its blocks, cut into one range per CTA.  For rows that are long and do not
//   divide well, or unequal (and for more pairs than CTAs).
// The one with the shorter longest piece is taken.  us a layer with a launch per operation, with whole CTAs only, and now: width 2,048
// with 16 kv heads, six rows of 2,048 70, 71 and 62, five of 8,192 106, 141 and 99, one of 32,768 beside seven of 256 110, 247 and 98;
// 8B shape, seven rows of 8,192 130, 154 and 129, one of 32,768 beside seven of 256 158, 140 and 117.
constexpr int PIECE = 13;
// Most pieces of a pair: a merge asks for MERGE of them at once, twice a group's heads over two, each round about three blocks long
// (16 heads over 2, one row of 2,048: 65.6 us a layer in 64 pieces, 47.6 in 20, a launch per operation 52.0).
constexpr int ROUND = 3;
__host__ __device__ inline int rounds_of(int parts, int group) { return parts > 1 ? (group * D + CONSUMERS - 1) / CONSUMERS * ((parts + MERGE - 1) / MERGE) : 0; }
struct Deal {
    int rows, kv_heads, ctas;
    const int32_t *blocks, *before;             // per row: blocks of keys, first CTA (place, with even shares) of its pairs
    int total;                                  // even shares: the length of all pairs end to end (0: whole CTAs)
};
struct Piece {
    int row, head, b0, n, blocks;               // blocks b0 .. b0 + n - 1 of the pair's
    int parts, index, first;                    // of the pair: its pieces, which one this is, the CTA of the first
    int next;                                   // even shares: where the pair behind this begins
};
__host__ __device__ inline long long share_begin(const Deal& d, int cta) { return (long long)cta * d.total / d.ctas; }
__host__ __device__ inline int share_of(const Deal& d, int at) { return (int)(((long long)(at + 1) * d.ctas - 1) / d.total); }
// A CTA's i-th piece, asked for in order.
__host__ __device__ inline bool piece_at(const Deal& d, int cta, int i, Piece& s) {
    const int M = d.rows, HKV = d.kv_heads;
    if (!d.total) {
        if (i || cta >= d.before[M]) return false;
        s.row = 0;
        while (s.row + 1 < M && cta >= d.before[s.row + 1]) ++s.row;
        s.blocks = d.blocks[s.row];
        s.parts = (d.before[s.row + 1] - d.before[s.row]) / HKV;
        const int rest = cta - d.before[s.row];
        s.head = rest / s.parts;
        s.index = rest - s.head * s.parts;
        s.first = cta - s.index;
        s.b0 = s.index * s.blocks / s.parts;
        s.n = (s.index + 1) * s.blocks / s.parts - s.b0;
        return true;
    }
    const int begin = (int)share_begin(d, cta), end = (int)share_begin(d, cta + 1);
    if (!i) s.next = begin;
    while (s.next < end) {
        s.row = 0;
        while (s.row + 1 < M && s.next >= d.before[s.row + 1]) ++s.row;
        s.blocks = d.blocks[s.row];
        const int length = PIECE + s.blocks;
        s.head = (s.next - d.before[s.row]) / length;
        const int pair = d.before[s.row] + s.head * length, keys = pair + PIECE;
        s.b0 = begin > keys ? begin - keys : 0;
        s.n = (end - keys < s.blocks ? end - keys : s.blocks) - s.b0;
        s.next = pair + length;
        if (s.n > 0) {
            s.first = share_of(d, keys);
            s.parts = share_of(d, keys + s.blocks - 1) - s.first + 1;
            s.index = cta - s.first;
            return true;
        }
    }
    return false;
}
// Fills in `before` ([rows + 1]) from `blocks`; returns Deal::total.
__host__ __device__ inline int deal_out(int M, int HKV, int group, int ctas, const int32_t* blocks, int32_t* before) {
    int whole = 0x7fffffff;                                              // the longest piece with whole CTAs, in blocks
    if (M * HKV <= ctas) {
        // one CTA a pair, then the rest to the rows with the most blocks per CTA, as long as the merge does not eat it up
        int used = M * HKV, parts[ROWS], most_parts[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            int rounds = 1;
            if (i < M)
                while (blocks[i] > MERGE * rounds * (rounds + 1) * ROUND * rounds_of(2, group)) ++rounds;
            parts[i] = 1;
            most_parts[i] = MERGE * rounds;
        }
        while (used + HKV <= ctas) {
            int best = -1, most = 1;
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                if (i < M && parts[i] < most_parts[i]) {
                    const int per = (blocks[i] + parts[i] - 1) / parts[i];
                    if (per > most) { most = per; best = i; }
                }
            if (best < 0) break;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) parts[i] += i == best;
            used += HKV;
        }
        int at = 0;
        whole = 0;
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
            if (i < M) {
                before[i] = at;
                at += parts[i] * HKV;
                const int piece = (blocks[i] + parts[i] - 1) / parts[i] + ROUND * rounds_of(parts[i], group);
                if (piece > whole) whole = piece;
            }
        before[M] = at;
    }
    int total = 0, longest = 0;
    for (int i = 0; i < M; ++i) {
        total += HKV * (PIECE + blocks[i]);
        if (blocks[i] > longest) longest = blocks[i];
    }
    // (every share has a length, so every CTA between a pair's first and its last has a piece of it)
    const int share = total / ctas;
    if (share < 1 || whole <= share + ROUND * rounds_of(longest / share + 2, group)) return 0;
    before[0] = 0;
    for (int i = 0; i < M; ++i) before[i + 1] = before[i] + HKV * (PIECE + blocks[i]);
    return total;
}

__device__ __forceinline__ void add_release(int32_t* p, int v) { asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ int load_acquire(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int add_acq_rel(int32_t* p, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CONSUMERS) : "memory"); }
// A copy from the host wrote the map, which the copy engine reads through a proxy and cache of its own: nothing else orders the two.
__device__ __forceinline__ void acquire_map(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}
__device__ __forceinline__ void load_weights(void* dst, const CUtensorMap* map, uint64_t* bar, int row, int block) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(block) : "memory");
}
__device__ __forceinline__ void load_page(void* dst, const CUtensorMap* map, uint64_t* bar, int row) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %3}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row) : "memory");
}

// Byte offset of 16-byte chunk `chunk` of key (value) `row` (0 .. 31) in a stage: pages as the box arrives,
// [K, V][half of 64 elements][row in page][128 bytes], swizzled.
__device__ __forceinline__ uint32_t key_off(int row, int chunk, int is_v, int page_size, int page_shift) {
    const int region = page_size * 128;
    return (uint32_t)((row >> page_shift) * (4 * region) + (is_v * 2 + (chunk >> 3)) * region + (row & (page_size - 1)) * 128 +
                      (((chunk & 7) ^ (row & 7)) << 4));
}

struct Ring {
    int stage = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int n) { if (++stage == n) { stage = 0; phase ^= 1; } }
};

// What every warp of the CTA shares.
struct Cta {
    unsigned char *ring, *x;
    float *red, *acc, *fac;
    unsigned char *q_tile, *k_new, *v_new;
    int32_t *z, *blocks, *before;               // per row: position, blocks of keys, first CTA (place, with even shares) of its pairs
    int32_t* pages;
    PhDecodeLayer* layers;
    uint64_t *full, *empty, *x_full, *x_empty, *ready;
    volatile int* dead;                         // a wait ran out: nobody waits any more
    mutable bool gone;                          // ... and this thread knows: it neither waits nor frees places
    int* flag;
    int g0[4], ng[4];                           // this CTA's groups in each product
    Deal deal;
    bool attends;
};

// Looks again and again, the first few hundred times without a look at the clock; gives up for the whole CTA when the limit
// passes (4e9 cycles: two seconds at the highest clock).  False: nobody waits any more.
constexpr long long WAIT_CYCLES = 4000000000ll;
template <typename Done> __device__ __forceinline__ bool wait_until(Done done, const Cta& c, const Params& p, int code) {
    if (c.gone) return false;
    long long t0 = 0;
    for (uint32_t i = 1; !done(); ++i) {
        if (i & 255u) continue;
        if (!*c.dead) {
            const long long now = clock64();
            if (i == 256u) t0 = now;
            if (now - t0 <= p.wait_cycles) continue;
            atomicExch(p.a.error_flag, code);
            *c.dead = 1;
        }
        c.gone = true;
        return false;
    }
    return true;
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, const Cta& c, const Params& p, int code) {
    return wait_until([&] { return mb::try_wait(bar, parity); }, c, p, code);
}
__device__ __forceinline__ bool wait_count(const int32_t* counter, int target, const Cta& c, const Params& p) {
    return wait_until([&] { return load_acquire(counter) >= target; }, c, p, PH_ERR_WAIT_LAYERS_PEERS);
}
// A warp's answer for a place that it has read.
__device__ __forceinline__ void free_place(uint64_t* bar, const Cta& c) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && !c.gone) mb::arrive(bar);
}

// The results that this part wrote are complete: every consumer's stores, then one add.
__device__ __forceinline__ void publish(int32_t* counter) {
    consumers_sync();
    if (threadIdx.x == 0) {                      // (one thread's release covers what the barrier has ordered before it)
        fence_async();                           // the next part's copies read them
        add_release(counter, 1);
    }
}

__device__ __forceinline__ int page_row(const Cta& c, const Params& p, int row, int head, int block, int page) {
    const int pos = block * KEYS + (page << p.page_shift);
    if (pos > c.z[row]) return p.a.total_rows;                       // zeros
    const int32_t id = p.a.block_table[(size_t)p.a.row_seg[row] * p.a.table_width + (pos >> p.page_shift)];
    return (int)((long long)id * p.rows_per_page + (long long)head * p.a.page_size);
}

enum { QKV, RESIDUAL, GATE_UP };

// One product over this CTA's groups of 16 output rows.
//   QKV: out (float32) = factor * sum.   RESIDUAL: x += sum; xw = bf16(x * next norm's weight), sums of squares per group.
//   GATE_UP: act = silu(gate) * up of the factored sums.
template <int KIND>
__device__ __forceinline__ void product(const Cta& c, const Params& p, Ring& ring, uint32_t& x_parity, uint32_t& ready, int which, int K,
                                        const float* next_norm) {
    const int g0 = c.g0[which], ng = c.ng[which];
    if (!ng) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int M = p.a.rows, E = p.a.width;
    wait_for(c.ready, ready, c, p, PH_ERR_WAIT_LAYERS_DATA);
    ready ^= 1;
    if (KIND != RESIDUAL && warp < M) {
        float s = 0.0f;
        const int parts = E / 16;
        const float* src = p.a.sumsq + (size_t)warp * parts;
        for (int j = lane; j < parts; j += 32) s += __ldcg(src + j);
        s = warp_sum(s);
        if (lane == 0) c.fac[warp] = rsqrtf(s / (float)E + p.a.norm_eps);
    }
    const int nseg = segments(K), cs = chunk_of(nseg, p.slots);
    const bool whole = cs == nseg;
    const int slot_bytes = M * PITCH;
    const int g = lane >> 2, t = lane & 3;
    // 16-byte chunks 2t and 2t + 1 of the warp's 64 of K, so that two rows of a swizzled stage meet different banks
    const uint32_t w_off = (uint32_t)(warp * 2048 + g * 128), w_chunk = (uint32_t)(((2 * t) ^ (g & 7)) << 4);
    const uint32_t x_off = (uint32_t)(min(g, M - 1) * PITCH + warp * 128 + t * 32);
    const int e = threadIdx.x & 127, token = e >> 4, row = e & 15;      // of the epilogue
    int unit = 0;
    for (int c0 = 0, half = 0; c0 < nseg; c0 += cs, half ^= 1) {
        const int c1 = min(c0 + cs, nseg);
        const bool last = c1 == nseg;
        for (int gi = 0; gi < ng; ++gi, ++unit) {
            const bool mine = (warp >> 2) == (unit & 1);
            const int feature = (g0 + gi) * 16 + row;
            float xv = 0.0f, nw = 0.0f;
            if (KIND == RESIDUAL && mine && last && token < M) {
                xv = __ldcg(p.a.x + (size_t)token * E + feature);
                if (next_norm) nw = next_norm[feature];
            }
            float s[2][4] = {};
            for (int seg = c0; seg < c1; ++seg) {
                const int slot = whole ? seg : half * cs + seg - c0;
                wait_for(&c.full[ring.stage], ring.phase, c, p, PH_ERR_WAIT_LAYERS_DATA);
                if (gi == 0) wait_for(&c.x_full[slot], (x_parity >> slot) & 1u, c, p, PH_ERR_WAIT_LAYERS_DATA);
                if (seg * SEG + warp * 64 < K) {
                    const unsigned char* w = c.ring + ring.stage * STAGE + w_off;
                    const unsigned char* x = c.x + slot * slot_bytes + x_off;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint4 a = *(const uint4*)(w + (w_chunk ^ (h << 4))), b = *(const uint4*)(w + 1024 + (w_chunk ^ (h << 4)));
                        const uint4 v = *(const uint4*)(x + (h << 4));
                        mma_bf16(s[h], a.x, b.x, a.y, b.y, v.x, v.y);
                        mma_bf16(s[h], a.z, b.z, a.w, b.w, v.z, v.w);
                    }
                }
                free_place(&c.empty[ring.stage], c);
                ring.next(p.stages);
            }
            float* red = c.red + (unit & 1) * (WARPS * ROWS * RED);
            {
                float* r = red + warp * (ROWS * RED) + 2 * t * RED + g;
                r[0] = s[0][0] + s[1][0]; r[RED] = s[0][1] + s[1][1];
                r[8] = s[0][2] + s[1][2]; r[RED + 8] = s[0][3] + s[1][3];
            }
            consumers_sync();
            if (!mine) continue;
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) v += red[w * (ROWS * RED) + token * RED + row];
            if (!whole) {
                float* a = c.acc + gi * 128 + e;
                if (c0) v += *a;
                if (!last) { *a = v; continue; }
            }
            if (KIND == QKV) {
                if (token < M) p.a.qkv[(size_t)token * ((p.a.heads + 2 * p.a.kv_heads) * D) + feature] = v * c.fac[token];
            } else if (KIND == GATE_UP) {
                const float f = token < M ? c.fac[token] : 0.0f;
                v *= f;
                const float u = __shfl_xor_sync(0xffffffffu, v, 1);
                if (!(row & 1) && token < M)
                    ((__nv_bfloat16*)p.a.act)[(size_t)token * p.a.inner + (feature >> 1)] = __float2bfloat16_rn(v / (1.0f + __expf(-v)) * u);
            } else {
                const float sum = xv + v;
                if (token < M) {
                    p.a.x[(size_t)token * E + feature] = sum;
                    if (next_norm) ((__nv_bfloat16*)p.a.xw)[(size_t)token * E + feature] = __float2bfloat16_rn(sum * nw);
                }
                float q = sum * sum;
#pragma unroll
                for (int o = 8; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                if (row == 0 && token < M) p.a.sumsq[(size_t)token * (E / 16) + g0 + gi] = q;
            }
        }
        // the places of this chunk are free
        const uint32_t used = (c1 - c0 == 32 ? 0xffffffffu : ((1u << (c1 - c0)) - 1u)) << (whole ? 0 : half * cs);
        x_parity ^= used;
        if (whole || half == 0) free_place(&c.x_empty[0], c);
        if (whole || half == 1) free_place(&c.x_empty[1], c);
    }
}

// Attention over this CTA's share of the blocks of keys.
__device__ __forceinline__ void attention(const Cta& c, const Params& p, Ring& ring, uint32_t& ready, const PhDecodeLayer& L, int32_t* counter,
                                          int32_t* pairs) {
    if (!c.attends) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int HQ = p.a.heads, HKV = p.a.kv_heads, G = HQ / HKV;
    const int width = (HQ + 2 * HKV) * D;
    const int ps = p.a.page_size, psh = p.page_shift;
    constexpr int RS = D + 2;
    float* red = (float*)c.x;                                            // [warps][G][D + 2]: the activations' place is free here
    float* mine = red + (size_t)warp * G * RS;
    const int r0 = lane >> 2;
    Piece s;
    for (int i = 0; piece_at(c.deal, blockIdx.x, i, s); ++i) {
        const int z = c.z[s.row], pair = s.row * HKV + s.head;
        // (the rotation does not wait for the product in front)
        const int pos = min(max(p.a.rotation_positions[s.row], 0), p.a.max_position - 1);
        const float4* cs = (const float4*)(p.a.rotation + (size_t)pos * D) + (lane & 15);
        const float4 co = cs[0], si = cs[16];
        if (!i) {
            wait_for(c.ready, ready, c, p, PH_ERR_WAIT_LAYERS_DATA);
            ready ^= 1;
        }
        const bool tail = s.b0 + s.n == s.blocks;
        // the group's queries, normed and rotated, and with the last block the step's own key and value
        for (int task = warp; task < G + (tail ? 2 : 0); task += WARPS) {
            const int head = task < G ? s.head * G + task : task == G ? HQ + s.head : HQ + HKV + s.head;
            float4 v = __ldcg((const float4*)(p.a.qkv + (size_t)s.row * width + head * D) + lane);
            if (task <= G) {
                const float4 w = ((const float4*)(task < G ? L.q_norm : L.k_norm))[lane];
                const float ss = warp_sum(fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x))));
                const float inv = rsqrtf(ss / (float)D + p.a.qk_eps);
                v.x *= inv * w.x; v.y *= inv * w.y; v.z *= inv * w.z; v.w *= inv * w.w;
                float4 o;
                o.x = __shfl_xor_sync(0xffffffffu, v.x, 16); o.y = __shfl_xor_sync(0xffffffffu, v.y, 16);
                o.z = __shfl_xor_sync(0xffffffffu, v.z, 16); o.w = __shfl_xor_sync(0xffffffffu, v.w, 16);
                const float sign = lane < 16 ? -1.0f : 1.0f;             // (a, b) -> (a c - b s, b c + a s)
                v.x = fmaf(v.x, co.x, sign * o.x * si.x); v.y = fmaf(v.y, co.y, sign * o.y * si.y);
                v.z = fmaf(v.z, co.z, sign * o.z * si.z); v.w = fmaf(v.w, co.w, sign * o.w * si.w);
            }
            uint2 h;
            h.x = pack_bf16(v.x, v.y); h.y = pack_bf16(v.z, v.w);
            if (task < G) *(uint2*)(c.q_tile + task * QPITCH + lane * 8) = h;
            else {
                *(uint2*)((task == G ? c.k_new : c.v_new) + lane * 8) = h;
                const int slot = p.a.slots[s.row];
                __nv_bfloat16* base = (__nv_bfloat16*)(task == G ? L.k_base : L.v_base);
                if (slot >= 0)
                    *(uint2*)(base + (size_t)(slot >> psh) * p.a.page_stride + ((size_t)s.head * ps + (slot & (ps - 1))) * D + lane * 4) = h;
            }
        }
        consumers_sync();
        uint32_t qf[D / 16][4];
        {   // rows beyond the group repeat a real row; their results are never stored
            const uint32_t q = smem_u32(c.q_tile) + min(lane & 15, G - 1) * QPITCH + (lane >> 4) * 16;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) ldmatrix_x4(q + ks * 32, qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3]);
        }
        float o[D / 8][4];
        float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
#pragma unroll
        for (int dt = 0; dt < D / 8; ++dt)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[dt][i] = 0.0f;
        // Four blocks at a time, two warps a block, 16 keys each.  Every warp sees every stage and answers for it: a warp that
        // passed over stages could ask for one whose fill before the last has the parity it waits for.
        for (int j = 0; j < s.n; ++j, ring.next(p.stages)) {
            wait_for(&c.full[ring.stage], ring.phase, c, p, PH_ERR_WAIT_LAYERS_DATA);
            if ((j & 3) != (warp >> 1)) {
                free_place(&c.empty[ring.stage], c);
                continue;
            }
            unsigned char* st_ptr = c.ring + ring.stage * STAGE;
            const uint32_t st = smem_u32(st_ptr);
            const int k0 = (warp & 1) * 16, key0 = (s.b0 + j) * KEYS + k0;
            if (key0 <= z) {
                const bool edge = key0 + 15 >= z;                        // the step's own token, and nothing behind it, is here
                if (edge) {
                    const int zr = z - key0;
                    *(uint4*)(st_ptr + key_off(k0 + zr, lane & 15, lane >> 4, ps, psh)) = *(const uint4*)((lane < 16 ? c.k_new : c.v_new) + (lane & 15) * 16);
                    for (int i = (zr + 1) * 16 + lane; i < 256; i += 32)
                        *(uint4*)(st_ptr + key_off(k0 + (i >> 4), i & 15, 1, ps, psh)) = make_uint4(0, 0, 0, 0);
                    __syncwarp();
                }
                float sc[2][4], s2[2][4];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) { sc[nt][i] = 0.0f; s2[nt][i] = 0.0f; }
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4(st + key_off(k0 + (lane & 7) + ((lane >> 4) << 3), ks * 2 + ((lane >> 3) & 1), 0, ps, psh), b0, b1, b2, b3);
                    mma_bf16(ks & 1 ? s2[0] : sc[0], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b0, b1);
                    mma_bf16(ks & 1 ? s2[1] : sc[1], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b2, b3);
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) sc[nt][i] += s2[nt][i];
                softmax_update<D, 16>(sc, key0, z, z, 0, 0, edge, p.scale_log2, m, l, o);
                const uint32_t a0 = pack_bf16(sc[0][0], sc[0][1]), a1 = pack_bf16(sc[0][2], sc[0][3]);
                const uint32_t a2 = pack_bf16(sc[1][0], sc[1][1]), a3 = pack_bf16(sc[1][2], sc[1][3]);
#pragma unroll
                for (int dt = 0; dt < D / 8; dt += 2) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(st + key_off(k0 + (lane & 7) + (((lane >> 3) & 1) << 3), dt + (lane >> 4), 1, ps, psh), b0, b1, b2, b3);
                    mma_bf16(o[dt], a0, a1, a2, a3, b0, b1);
                    mma_bf16(o[dt + 1], a0, a1, a2, a3, b2, b3);
                }
                if (edge) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // our stores, before the next copy lands there
            }
            free_place(&c.empty[ring.stage], c);
        }
        // merge the eight warps (a group has at most eight heads: fragment rows 8 .. 15 are padding)
        if (r0 < G) {
#pragma unroll
            for (int dt = 0; dt < D / 8; ++dt) *(float2*)(mine + r0 * RS + dt * 8 + (lane & 3) * 2) = make_float2(o[dt][0], o[dt][1]);
            if ((lane & 3) == 0) *(float2*)(mine + r0 * RS + D) = make_float2(m[0], l[0]);
        }
        consumers_sync();
        for (int idx = threadIdx.x; idx < G * D; idx += CONSUMERS) {
            const int r = idx / D, d = idx % D;
            float mm = -INFINITY;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, red[((size_t)w * G + r) * RS + D]);
            const float use = mm == -INFINITY ? 0.0f : mm;
            float acc = 0.0f, ll = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const float* src = red + ((size_t)w * G + r) * RS;
                const float f = exp2f(src[D] - use);
                acc += f * src[d];
                ll += f * src[D + 1];
            }
            if (s.parts == 1) {
                ((__nv_bfloat16*)p.a.attn)[(size_t)s.row * HQ * D + (s.head * G + r) * D + d] = __float2bfloat16_rn(ll == 0.0f ? 0.0f : acc / ll);
            } else {
                const size_t at = (size_t)(2 * blockIdx.x + (s.index == 0)) * G + r;     // (the end of one pair, the start of another)
                p.a.part_o[at * D + d] = acc;
                if (d == 0) *(float2*)(p.a.part_ml + at * 2) = make_float2(mm, ll);
            }
        }
        if (s.parts == 1) publish(counter);
        else {
            consumers_sync();
            if (threadIdx.x == 0) *c.flag = add_acq_rel(pairs + pair, 1) == s.parts - 1;
            consumers_sync();
            if (*c.flag) {
                // the last of the pair's CTAs: every reference and sum, and eight parts of the output, on their way at once
                const size_t at = (size_t)2 * s.first * G;
                for (int idx = threadIdx.x; idx < G * D; idx += CONSUMERS) {
                    const int r = idx / D, d = idx % D;
                    const float* po = p.a.part_o + (at + r) * D + d;
                    const float2* pml = (const float2*)p.a.part_ml + at + r;
                    float mm = -INFINITY, acc = 0.0f, ll = 0.0f;
                    for (int j = 0; j < s.parts; j += MERGE) {
                        float2 ml[MERGE];
                        float v[MERGE];
#pragma unroll
                        for (int u = 0; u < MERGE; ++u) {
                            const int part = min(j + u, s.parts - 1), k = (2 * part + (part == 0)) * G;
                            ml[u] = __ldcg(pml + k);
                            v[u] = __ldcg(po + (size_t)k * D);
                        }
                        float top = mm;
#pragma unroll
                        for (int u = 0; u < MERGE; ++u) top = fmaxf(top, ml[u].x);       // (the last part again: no harm)
                        const float use = top == -INFINITY ? 0.0f : top, old = exp2f(mm - use);
                        acc *= old; ll *= old;
#pragma unroll
                        for (int u = 0; u < MERGE; ++u) {
                            const float f = exp2f(ml[u].x - use);
                            if (j + u < s.parts) { acc = fmaf(f, v[u], acc); ll = fmaf(f, ml[u].y, ll); }
                        }
                        mm = top;
                    }
                    ((__nv_bfloat16*)p.a.attn)[(size_t)s.row * HQ * D + (s.head * G + r) * D + d] = __float2bfloat16_rn(ll == 0.0f ? 0.0f : acc / ll);
                }
                if (threadIdx.x == 0) pairs[pair] = 0;
                publish(counter);
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // the merge's stores, before activations land there
}

__global__ void __launch_bounds__(NTHREADS, 1) decode_layers_kernel(const Params p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);      // (an offset: the compiler still sees shared memory)
    const int M = p.a.rows, E = p.a.width, HKV = p.a.kv_heads;
    const int CTAS = gridDim.x;
    Cta c;
    c.gone = false;
    c.ring = smem;
    c.x = c.ring + p.stages * STAGE;
    c.red = (float*)(c.x + p.x_bytes);
    c.acc = c.red + 2 * WARPS * ROWS * RED;
    c.q_tile = (unsigned char*)(c.acc + p.acc_groups * 128);
    c.k_new = c.q_tile + 16 * QPITCH;
    c.v_new = c.k_new + D * 2;
    c.layers = (PhDecodeLayer*)(c.v_new + D * 2);
    c.full = (uint64_t*)(c.layers + p.a.n_layers);
    c.empty = c.full + MAX_STAGES;
    c.x_full = c.empty + MAX_STAGES;
    c.x_empty = c.x_full + MAX_SLOTS;
    c.ready = c.x_empty + 2;
    c.fac = (float*)(c.ready + 1);
    c.z = (int32_t*)(c.fac + ROWS);
    c.blocks = c.z + ROWS;
    c.before = c.blocks + ROWS;
    c.pages = c.before + ROWS + 1;
    c.dead = (volatile int*)(c.pages + PAGES);
    c.flag = (int*)(c.pages + PAGES) + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < p.a.n_layers * (int)(sizeof(PhDecodeLayer) / 8); i += NTHREADS)
        ((uint64_t*)c.layers)[i] = ((const uint64_t*)p.a.layers)[i];
    // (an engine's maps may lie where those of a closed one lay; a map a thread, in front of the barriers before the first copy)
    for (int i = threadIdx.x; i < p.a.n_layers * MAPS; i += NTHREADS) acquire_map((const CUtensorMap*)p.a.maps + i);
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) { mb::init(&c.full[s], 1); mb::init(&c.empty[s], WARPS); }
        for (int s = 0; s < p.slots; ++s) mb::init(&c.x_full[s], 1);
        for (int s = 0; s < 2; ++s) mb::init(&c.x_empty[s], WARPS);
        mb::init(c.ready, 1);
        *c.dead = 0;
        mb::fence_init();
        for (int i = 0; i < M; ++i) {
            c.z[i] = p.a.positions[i];
            c.blocks[i] = c.z[i] / KEYS + 1;
        }
        *c.flag = deal_out(M, HKV, p.a.heads / HKV, CTAS, c.blocks, c.before);
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int32_t* s = p.a.shares + w * (CTAS + 1) + blockIdx.x;
        c.g0[w] = s[0];
        c.ng[w] = s[1] - s[0];
    }
    __syncthreads();
    c.deal = Deal{M, HKV, CTAS, c.blocks, c.before, *c.flag};
    const int ppb = KEYS >> p.page_shift;                                // pages per block
    {
        Piece s;
        c.attends = piece_at(c.deal, blockIdx.x, 0, s);
        for (int n = 0, at = 0; at < PAGES && piece_at(c.deal, blockIdx.x, n, s); ++n, at += s.n * ppb)
            for (int i = threadIdx.x; i < s.n * ppb && at + i < PAGES; i += NTHREADS)
                c.pages[at + i] = page_row(c, p, s.row, s.head, s.b0 + i / ppb, i % ppb);
    }
    __syncthreads();

    int32_t* counters = p.a.counters + 1;                                // [0]: CTAs that are done
    int32_t* pairs = counters + 1 + PARTS * p.a.n_layers;
    const int widths[4] = {E, p.a.heads * D, E, p.a.inner};

    if (warp == WARPS) {
        // ---- the ring: weights and cached keys in the order of their use, whatever the other CTAs are at ----
        // One thread, with as little as possible between two copies: a stage's time is the longer of its bytes' and of this
        // loop's turn.
        if (lane == 0) {
            Ring ring;
            int filled = 0;
            unsigned char* to = c.ring;
            auto fill = [&](uint32_t bytes) {                            // a free stage, with so many bytes announced
                if (!mb::try_wait(&c.empty[ring.stage], ring.phase ^ 1) &&
                    !wait_for(&c.empty[ring.stage], ring.phase ^ 1, c, p, PH_ERR_WAIT_LAYERS_RING))
                    return false;
                mb::arrive_expect_tx(&c.full[ring.stage], bytes);
                return true;
            };
            auto filled_one = [&] {
                ++filled;
                to += STAGE;
                if (++ring.stage == p.stages) { ring.stage = 0; ring.phase ^= 1; to = c.ring; }
            };
            auto weights = [&](const CUtensorMap* map, int g0, int ng, int K) {
                const int nseg = segments(K), cs = chunk_of(nseg, p.slots);
                for (int c0 = 0; c0 < nseg; c0 += cs) {
                    const int end = min(c0 + cs, nseg) * (SEG / 64);
                    for (int row = g0 * 16; row < (g0 + ng) * 16; row += 16)
                        for (int block = c0 * (SEG / 64); block < end; block += SEG / 64) {
                            if (!fill(STAGE)) return false;              // (K's end counts in full: zeros)
                            load_weights(to, map, &c.full[ring.stage], row, block);
                            filled_one();
                        }
                }
                return true;
            };
            auto keys = [&](const CUtensorMap* map) {
                int at = 0;
                Piece s;
                for (int n = 0; piece_at(c.deal, blockIdx.x, n, s); ++n)
                    for (int j = 0; j < s.n; ++j) {
                        if (!fill(KEYS * D * 4)) return false;
                        for (int i = 0; i < ppb; ++i, ++at)
                            load_page(to + i * p.a.page_size * 512, map, &c.full[ring.stage],
                                      at < PAGES ? c.pages[at] : page_row(c, p, s.row, s.head, s.b0 + j, i));
                        filled_one();
                    }
                return true;
            };
            const CUtensorMap* maps = (const CUtensorMap*)p.a.maps;
            for (int i = 0; i < MAPS; ++i) asm volatile("prefetch.tensormap [%0];" ::"l"(maps + i) : "memory");
            for (int l = 0; l < p.a.n_layers; ++l, maps += MAPS) {
                if (l + 1 < p.a.n_layers)
                    for (int i = 0; i < MAPS; ++i) asm volatile("prefetch.tensormap [%0];" ::"l"(maps + MAPS + i) : "memory");
                if (!weights(maps, c.g0[0], c.ng[0], widths[0]) || !keys(maps + 4) || !weights(maps + 1, c.g0[1], c.ng[1], widths[1]) ||
                    !weights(maps + 2, c.g0[2], c.ng[2], widths[2]) || !weights(maps + 3, c.g0[3], c.ng[3], widths[3]))
                    break;
            }
            // do not leave before the last of it has landed: consumers that are gone do not wait for it
            for (int i = min(filled, p.stages); i; --i) {
                if (ring.stage == 0) { ring.stage = p.stages; ring.phase ^= 1; }
                --ring.stage;
                mb::wait(&c.full[ring.stage], ring.phase, p.a.error_flag, PH_ERR_WAIT_LAYERS_RING);
            }
        }
    } else if (warp == WARPS + 1) {
        // ---- the activations: when a part's input is complete, its rows go to shared memory ----
        uint32_t x_free[2] = {1, 1}, x_parity = 0, pending = 0;
        bool ok = true;
        auto alive = [&] { return __shfl_sync(0xffffffffu, lane == 0 ? *c.dead : 0, 0) == 0; };
        auto begin = [&](const int32_t* counter, int target) {           // every lane looks, so every lane may go on
            wait_count(counter, target, c, p);
            fence_async();
            if (lane == 0) mb::arrive(c.ready);
            ok = alive();
        };
        // places for n segments from slot0 on are free, and their bytes announced
        auto make_room = [&](bool whole, int half, int slot0, int c0, int n, int K) {
            for (int h = 0; h < 2; ++h)
                if (whole || h == half) {
                    wait_for(&c.x_empty[h], x_free[h], c, p, PH_ERR_WAIT_LAYERS_RING);
                    x_free[h] ^= 1;
                }
            ok = alive();
            if (ok && lane < n) mb::arrive_expect_tx(&c.x_full[slot0 + lane], M * min(SEG, K - (c0 + lane) * SEG) * 2);
            __syncwarp();
        };
        auto load = [&](const int32_t* counter, int target, const void* src, int K) {
            const int nseg = segments(K), cs = chunk_of(nseg, p.slots);
            const bool whole = cs == nseg;
            for (int c0 = 0, half = 0; c0 < nseg && ok; c0 += cs, half ^= 1) {
                const int n = min(cs, nseg - c0), slot0 = whole ? 0 : half * cs;
                make_room(whole, half, slot0, c0, n, K);
                if (ok && c0 == 0) begin(counter, target);
                if (!ok) break;
                for (int i = lane; i < n * M; i += 32) {
                    const int seg = i / M, row = i - seg * M;
                    mb::bulk_copy(c.x + (slot0 + seg) * M * PITCH + row * PITCH, (const __nv_bfloat16*)src + (size_t)row * K + (c0 + seg) * SEG,
                                  min(SEG, K - (c0 + seg) * SEG) * 2, &c.x_full[slot0 + seg]);
                }
                const uint32_t used = (n == 32 ? 0xffffffffu : ((1u << n) - 1u)) << slot0;
                x_parity ^= used;
                pending |= used;
            }
        };
        for (int l = 0; l < p.a.n_layers && ok; ++l) {
            const int32_t* k = counters + PARTS * l;
            if (ok && c.ng[0]) load(k, CTAS, p.a.xw, E);
            if (ok && c.attends) begin(k + 1, CTAS);
            if (ok && c.ng[1]) load(k + 2, M * HKV, p.a.attn, widths[1]);
            if (ok && c.ng[2]) load(k + 3, CTAS, p.a.xw, E);
            if (ok && c.ng[3]) load(k + 4, CTAS, p.a.act, widths[3]);
        }
        if (lane == 0)                                                   // (as the ring's thread)
            for (int s = 0; s < p.slots; ++s)
                if ((pending >> s) & 1u) mb::wait(&c.x_full[s], ((x_parity >> s) & 1u) ^ 1u, p.a.error_flag, PH_ERR_WAIT_LAYERS_RING);
    } else {
        // ---- the work ----
        Ring ring;
        uint32_t x_parity = 0, ready = 0;
        {   // the embedding's rows for the first layer's norm
            const float* w = c.layers[0].norm1;
            const int e = threadIdx.x & 127, token = e >> 4, row = e & 15;
            for (int grp = 2 * blockIdx.x + (threadIdx.x >> 7); grp < E / 16; grp += 2 * CTAS) {
                const int feature = grp * 16 + row;
                const float v = token < M ? p.a.x[(size_t)token * E + feature] : 0.0f;
                if (token < M) ((__nv_bfloat16*)p.a.xw)[(size_t)token * E + feature] = __float2bfloat16_rn(v * w[feature]);
                float q = v * v;
#pragma unroll
                for (int o = 8; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                if (row == 0 && token < M) p.a.sumsq[(size_t)token * (E / 16) + grp] = q;
            }
            publish(counters);
        }
        for (int l = 0; l < p.a.n_layers; ++l) {
            int32_t* k = counters + PARTS * l;
            const PhDecodeLayer& L = c.layers[l];
            product<QKV>(c, p, ring, x_parity, ready, 0, widths[0], nullptr);
            publish(k + 1);
            attention(c, p, ring, ready, L, k + 2, pairs);
            product<RESIDUAL>(c, p, ring, x_parity, ready, 1, widths[1], L.norm2);
            publish(k + 3);
            product<GATE_UP>(c, p, ring, x_parity, ready, 2, widths[2], nullptr);
            publish(k + 4);
            product<RESIDUAL>(c, p, ring, x_parity, ready, 3, widths[3], l + 1 < p.a.n_layers ? c.layers[l + 1].norm1 : nullptr);
            publish(k + 5);
        }
    }
    __syncthreads();
    // the last CTA leaves the counters as it found them
    if (threadIdx.x == 0) *c.flag = add_acq_rel(p.a.counters, 1) == CTAS - 1;
    __syncthreads();
    if (*c.flag)
        for (int i = threadIdx.x; i < 2 + PARTS * p.a.n_layers + M * HKV; i += NTHREADS) p.a.counters[i] = 0;
}

size_t fixed_bytes(int n_layers) {
    return 1024 + 2 * WARPS * ROWS * RED * 4 + 16 * QPITCH + 2 * D * 2 + (size_t)n_layers * sizeof(PhDecodeLayer) +
           (2 * MAX_STAGES + MAX_SLOTS + 3) * 8 + (ROWS * 4 + 1 + PAGES + 2) * 4 + 64;
}

// How shared memory is shared out: places for the rows' activations (all of the widest product's K where that leaves the ring
// most of the memory, at most 70 KB), the rest to the ring.
Plan make_plan(int rows, int width, int heads, int kv_heads, int inner, int n_layers, int most_groups) {
    Plan q{};
    const int k[4] = {width, heads * D, width, inner};
    int most = 0;
    for (int i = 0; i < 4; ++i) most = most > segments(k[i]) ? most : segments(k[i]);
    int slots = 70 * 1024 / (rows * PITCH);
    slots = slots < most ? slots : most;
    slots = slots < MAX_SLOTS ? slots : MAX_SLOTS;
    if (slots < most) slots &= ~1;
    if (slots < 2) slots = 2;
    q.slots = slots;
    q.acc_groups = most > slots ? most_groups : 0;
    const size_t merge = (size_t)WARPS * (heads / kv_heads) * (D + 2) * 4;
    q.x_bytes = (size_t)slots * rows * PITCH;
    if (q.x_bytes < merge) q.x_bytes = merge;
    q.x_bytes = (q.x_bytes + 15) & ~(size_t)15;
    const size_t rest = fixed_bytes(n_layers) + q.x_bytes + (size_t)q.acc_groups * 512;
    constexpr size_t SM = 227 * 1024;
    q.stages = rest >= SM ? 0 : (int)((SM - rest) / STAGE);
    if (q.stages > MAX_STAGES) q.stages = MAX_STAGES;
    q.bytes = rest + (size_t)q.stages * STAGE;
    return q;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)q;
    });
    return fn;
}

}  // namespace

PH_DEFINE_LAST_ERROR(ph_layers)

// 1 if the kernel takes layers of these sizes for a step of `rows` rows.
PH_EXPORT int ph_decode_layers_supports(int rows, int width, int heads, int kv_heads, int head_dim, int inner, int page_size, int n_layers,
                                        int most_groups) {
    if (rows < 1 || rows > ROWS || n_layers < 1 || head_dim != D || kv_heads < 1 || heads < 1 || heads % kv_heads || heads / kv_heads > MAX_GROUP) return 0;
    if (width < 64 || width % 64 || inner < 64 || inner % 64) return 0;
    if (page_size != 8 && page_size != 16 && page_size != 32) return 0;
    return make_plan(rows, width, heads, kv_heads, inner, n_layers, most_groups).stages >= 4 ? 1 : 0;
}

// Deals each product's groups of 16 output rows to the CTAs, [4][ctas + 1] first groups: every CTA gets the whole part of an
// equal share, and what is left over goes one each to the CTAs with the least so far, so that all stream about the same bytes
// per layer although no product divides evenly.  Returns the largest share.
PH_EXPORT int ph_decode_layers_shares(int width, int heads, int kv_heads, int inner, int ctas, int32_t* out) {
    const int n[4] = {(heads + 2 * kv_heads) * D / 16, width / 16, 2 * inner / 16, width / 16};
    const int k[4] = {width, heads * D, width, inner};
    std::vector<long long> load(ctas, 0);
    std::vector<int> share(ctas);
    int most = 0;
    for (int w = 0; w < 4; ++w) {
        for (int i = 0; i < ctas; ++i) share[i] = n[w] / ctas;
        std::vector<bool> taken(ctas, false);
        for (int r = 0; r < n[w] % ctas; ++r) {
            int best = -1;
            for (int i = 0; i < ctas; ++i)
                if (!taken[i] && (best < 0 || load[i] < load[best])) best = i;
            taken[best] = true;
            share[best]++;
        }
        int at = 0;
        for (int i = 0; i < ctas; ++i) {
            out[w * (ctas + 1) + i] = at;
            at += share[i];
            load[i] += (long long)share[i] * k[w];
            most = most > share[i] ? most : share[i];
        }
        out[w * (ctas + 1) + ctas] = at;
    }
    return most;
}

// The copy engine's view of a weight [rows, K], 128 bytes to `out` (host memory): blocks of 64 of K, a box of 16 rows x 8 blocks.
PH_EXPORT int ph_decode_layers_weight_map(void* out, const void* w, int rows, int K) {
    EncodeTiledFn fn = encode_fn();
    const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(K / 64)};
    const cuuint64_t strides[2] = {(cuuint64_t)K * 2, 128};
    const cuuint32_t box[3] = {64, 16, SEG / 64}, elem[3] = {1, 1, 1};
    CUtensorMap m;
    if (K % 64 || !fn || fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return fail(PH_ERR_UNSUPPORTED, "decode_layers: the copy engine does not take a weight of %d x %d", rows, K);
    memcpy(out, &m, sizeof(m));
    return PH_OK;
}

// The deal of the keys for rows at these positions: nine numbers a piece (CTA, row, kv head, first block, blocks, the pair's blocks, its
// pieces, which of them, the CTA of the first) to `out`, room for `most` pieces.  Returns how many there are.
PH_EXPORT int ph_decode_layers_deal(int rows, int heads, int kv_heads, const int32_t* positions, int ctas, int32_t* out, int most) {
    if (rows < 1 || rows > ROWS || kv_heads < 1 || heads < kv_heads || ctas < 1 || !positions || !out)
        return fail(PH_ERR_ARG, "decode_layers: no deal of %d rows, %d heads over %d, to %d CTAs", rows, heads, kv_heads, ctas);
    int32_t blocks[ROWS], before[ROWS + 1];
    for (int i = 0; i < rows; ++i) blocks[i] = positions[i] / KEYS + 1;
    const int total = deal_out(rows, kv_heads, heads / kv_heads, ctas, blocks, before);
    const Deal d{rows, kv_heads, ctas, blocks, before, total};
    int n = 0;
    for (int cta = 0; cta < ctas; ++cta) {
        Piece s;
        for (int i = 0; piece_at(d, cta, i, s); ++i, ++n)
            if (n < most) {
                const int32_t v[9] = {cta, s.row, s.head, s.b0, s.n, s.blocks, s.parts, s.index, s.first};
                memcpy(out + (size_t)n * 9, v, sizeof(v));
            }
    }
    return n;
}

// 1 if the current device takes cooperative launches and all `ctas` of them can be resident.
PH_EXPORT int ph_decode_layers_resident(int ctas) {
    int dev = 0, sms = 0, cooperative = 0, per_sm = 0;
    const bool ok = cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
                    cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess &&
                    cudaFuncSetAttribute(decode_layers_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_layers_kernel, NTHREADS, 227 * 1024) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok && cooperative && per_sm >= 1 && sms >= ctas ? 1 : 0;
}

PH_EXPORT int ph_decode_layers_counters(int n_layers, int kv_heads) { return 2 + PARTS * n_layers + ROWS * kv_heads; }

// The copy engine's view of one cache entry, 128 bytes to `out` (host memory); as in attention_decode_bulk.cu.
PH_EXPORT int ph_decode_layers_map(void* out, const void* k_base, const void* v_base, long long page_stride, int page_size, int num_pages, int kv_heads,
                                   int* total_rows) {
    const long long rows = (long long)(num_pages - 1) * (page_stride / D) + (long long)kv_heads * page_size;
    const long long kv = (const char*)v_base - (const char*)k_base;
    if (page_stride % D || rows >= 0x7fffffffLL || kv <= 0 || kv % 16 || (((uintptr_t)k_base) & 15))
        return fail(PH_ERR_UNSUPPORTED, "decode_layers: the cache is not laid out in whole, 16-byte aligned rows");
    EncodeTiledFn fn = encode_fn();
    const cuuint64_t dims[4] = {64, (cuuint64_t)rows, 2, 2};
    const cuuint64_t strides[3] = {(cuuint64_t)D * 2, 128, (cuuint64_t)kv};
    const cuuint32_t box[4] = {64, (cuuint32_t)page_size, 2, 2}, elem[4] = {1, 1, 1, 1};
    CUtensorMap m;
    if (!fn || fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(k_base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return fail(PH_ERR_UNSUPPORTED, "decode_layers: the copy engine does not take this cache layout");
    memcpy(out, &m, sizeof(m));
    *total_rows = (int)rows;
    return PH_OK;
}

PH_EXPORT int ph_decode_layers(const PhDecodeLayersArgs* args, cudaStream_t stream) {
    const PhDecodeLayersArgs& a = *args;
    if (!a.layers || !a.maps || !a.shares || !a.counters || !a.rotation || !a.block_table || !a.row_seg || !a.positions || !a.rotation_positions ||
        !a.slots || !a.x || !a.xw || !a.sumsq || !a.qkv || !a.attn || !a.act || !a.part_o || !a.part_ml || !a.error_flag)
        return fail(PH_ERR_ARG, "decode_layers: a pointer is missing");
    if (!ph_decode_layers_supports(a.rows, a.width, a.heads, a.kv_heads, D, a.inner, a.page_size, a.n_layers, a.most_groups))
        return fail(PH_ERR_UNSUPPORTED, "decode_layers: %d rows of %d, %d heads over %d, %d inner, pages of %d", a.rows, a.width, a.heads, a.kv_heads,
                    a.inner, a.page_size);
    const Plan q = make_plan(a.rows, a.width, a.heads, a.kv_heads, a.inner, a.n_layers, a.most_groups);
    Params p;
    p.a = a;
    p.stages = q.stages; p.slots = q.slots; p.acc_groups = q.acc_groups; p.x_bytes = (int)q.x_bytes;
    p.page_shift = a.page_size == 8 ? 3 : a.page_size == 16 ? 4 : 5;
    p.rows_per_page = a.page_stride / D;
    p.scale_log2 = a.scale * LOG2E;
    p.wait_cycles = a.wait_cycles > 0 ? a.wait_cycles : WAIT_CYCLES;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(decode_layers_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
        return fail(PH_ERR_LAUNCH, "decode_layers: cannot reserve %zu bytes of shared memory", q.bytes);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = q.bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_layers_kernel, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        // (a process may hold a part of the device only)
        const bool refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported;
        return fail(refused ? PH_LAYERS_REFUSED : PH_ERR_LAUNCH, "decode_layers: launch failed: %s", cudaGetErrorString(e));
    }
    return check_launch("decode_layers");
}
