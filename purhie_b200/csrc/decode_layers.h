// The layers of a decode step as one launch: what the host hands to the kernel of decode_layers.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// One layer's vectors (float32) and where its cache entry lies.  Its matrices (bfloat16, [out, in]) are w_qkv [(HQ + 2 HKV) 128, E],
// w_o [E, HQ 128], w_gate_up [2 F, E] with (gate, up) row pairs, and w_down [E, F], read through `maps`.
struct PhDecodeLayer {
    const float* norm1;          // [E]
    const float* norm2;          // [E]
    const float* q_norm;         // [128]
    const float* k_norm;         // [128]
    void* k_base;                // the entry's keys and values in page 0
    void* v_base;
};

// ph_decode_layers: the device did not let all CTAs be resident at once; nothing was launched.
#define PH_LAYERS_REFUSED 134

struct PhDecodeLayersArgs {
    // fixed for a model and its cache
    const PhDecodeLayer* layers;       // [n_layers] on the device
    const void* maps;                  // [n_layers][5] copy-engine descriptors on the device: w_qkv, w_o, w_gate_up, w_down, the cache entry
    const int32_t* shares;             // [4][CTAs + 1] first group of 16 output rows of every CTA in each product, on the device
    int32_t* counters;                 // ph_decode_layers_counters() words on the device, zero before the first launch
    int n_layers, width, heads, kv_heads, inner, page_size, total_rows, max_position;
    int most_groups;                   // largest share of any CTA in any product
    long long page_stride;             // elements
    float norm_eps, qk_eps, scale;
    const float* rotation;             // [max_position, 128]
    // of the step
    int rows;
    const int32_t* block_table;
    int table_width;
    const int32_t* row_seg;
    const int32_t* positions;
    const int32_t* rotation_positions;
    const int32_t* slots;
    // scratch, and the residual [rows, width] that is updated in place
    float* x;
    void* xw;                          // [rows, width] bfloat16
    float* sumsq;                      // [rows, width / 16]
    float* qkv;                        // [rows, (HQ + 2 HKV) 128]
    void* attn;                        // [rows, HQ 128] bfloat16
    void* act;                         // [rows, F] bfloat16
    float* part_o;                     // [2 CTAs][HQ / HKV][128]
    float* part_ml;                    // [2 CTAs][HQ / HKV][2]
    int* error_flag;
    long long wait_cycles;             // limit of every wait (0: two seconds)
};
