#include "decode_stack.h"

#include <algorithm>

#include "../csrc/decode_layers.h"

namespace qe {

namespace {
constexpr int kMostRows = 8;
DeviceBuffer upload(const void* host, size_t bytes, cudaStream_t stream) {
    DeviceBuffer b(bytes);
    QE_CUDA(cudaMemcpyAsync(b.data(), host, bytes, cudaMemcpyHostToDevice, stream));
    QE_CUDA(cudaStreamSynchronize(stream));
    return b;
}
// The launches that a layer saves, about twelve microseconds, against what it loses where a product's groups do not divide among
// the CTAs: each product waits for its largest share, which streams at 44 GB/s an SM.  us a layer at one and eight rows
// behind 2,048 tokens, a launch per operation and one launch: 0.6B shape (loses 2.6) 39.8 / 52.4 and 29.5 / 42.6; width 2,048 (2.4)
// 49.2 / 62.1 and 38.2 / 51.5; 8B shape (6.3) 88.8 / 103.4 and 85.7 / 100.7; width 5,120 with 17,408 inner and 40 heads (18.5)
// 133 / 150 and 144 / 168; with 25,600 and 64 (24.5) 187 / 207 and 194 / 218.  Width 2,560 with 32 heads (11.5) lies between and is
// left out: 63.8 / 76.5 and 59.6 / 75.8, one to eight percent, which the form that the line was drawn for did not have.
constexpr double kMostUnevenUs = 9.0;
double uneven_us(const std::vector<int32_t>& shares, int ctas, const DecodeLayerSpec& a) {
    const double k[4] = {(double)a.width, (double)a.heads * a.head_dim, (double)a.width, (double)a.inner};
    double us = 0.0;
    for (int w = 0; w < 4; w++) {
        const int32_t* first = shares.data() + (size_t)w * (ctas + 1);
        int most = 0;
        for (int i = 0; i < ctas; i++) most = std::max(most, first[i + 1] - first[i]);
        us += (most - (double)first[ctas] / ctas) * 16 * 2 * k[w] / 44e3;
    }
    return us;
}
}  // namespace

std::unique_ptr<DecodeStack> DecodeStack::make(const std::vector<DecodeLayerSpec>& layers, const std::vector<CacheView>& views, cudaStream_t stream) {
    if (layers.empty() || layers.size() != views.size()) return nullptr;
    const DecodeLayerSpec& a = layers[0];
    const CacheView& v = views[0];
    for (size_t i = 0; i < layers.size(); i++) {
        const DecodeLayerSpec& b = layers[i];
        const CacheView& w = views[i];
        if (b.width != a.width || b.inner != a.inner || b.heads != a.heads || b.kv_heads != a.kv_heads || b.head_dim != a.head_dim ||
            b.norm_eps != a.norm_eps || b.qk_eps != a.qk_eps || b.scale != a.scale || b.rotation != a.rotation ||
            b.max_position != a.max_position || b.position_column != a.position_column)
            return nullptr;
        if (w.kind != CacheNeed::Pages || !w.writable || w.kv_dtype != DType::BF16 || w.group != v.group || w.page_size != v.page_size ||
            w.page_stride != v.page_stride || w.num_pages != v.num_pages || w.num_pages < 1 || w.kv_heads != a.kv_heads || w.key_dim != a.head_dim ||
            w.value_dim != a.head_dim || w.state.defined())
            return nullptr;
    }
    const LayersKernels& k = layers_kernels();
    std::unique_ptr<DecodeStack> s(new DecodeStack());
    s->first_ = a;
    s->n_layers_ = (int)layers.size();
    s->group_ = v.group; s->page_size_ = v.page_size; s->page_stride_ = v.page_stride;
    s->num_ctas_ = sm_count();
    // Every pair of eight rows a CTA of its own, at least: with more kv heads keys are most of a step, the attention kernel streams
    // them 5 % faster than the ring does, and rows of 32,768 lost more than the launches cost (width 4,096 with 32 kv heads, us a layer
    // with a launch per operation and with one: one row of 2,048 107 and 103, eight 144 and 155, one of 32,768 177 and 182).
    if (a.kv_heads * kMostRows > s->num_ctas_ || !k.resident(s->num_ctas_)) return nullptr;
    std::vector<int32_t> shares((size_t)4 * (s->num_ctas_ + 1));
    s->most_groups_ = k.shares((int)a.width, a.heads, a.kv_heads, (int)a.inner, s->num_ctas_, shares.data());
    if (uneven_us(shares, s->num_ctas_, a) > kMostUnevenUs) return nullptr;
    if (!k.supports(1, (int)a.width, a.heads, a.kv_heads, a.head_dim, (int)a.inner, v.page_size, s->n_layers_, s->most_groups_)) return nullptr;
    std::vector<PhDecodeLayer> records;
    constexpr int kMaps = 5;                              // of a layer: four weights, the cache entry; 128 bytes each
    std::vector<uint8_t> maps((size_t)kMaps * 128 * layers.size());
    const int qkv = (a.heads + 2 * a.kv_heads) * a.head_dim, q = a.heads * a.head_dim, E = (int)a.width, F = (int)a.inner;
    for (size_t i = 0; i < layers.size(); i++) {
        const DecodeLayerSpec& b = layers[i];
        records.push_back({b.norm1, b.norm2, b.q_norm, b.k_norm, views[i].k_base, views[i].v_base});
        uint8_t* m = maps.data() + (size_t)kMaps * 128 * i;
        if (k.weight_map(m, b.w_qkv, qkv, E) != 0 || k.weight_map(m + 128, b.w_o, E, q) != 0 || k.weight_map(m + 256, b.w_gate_up, 2 * F, E) != 0 ||
            k.weight_map(m + 384, b.w_down, E, F) != 0 ||
            k.map(m + 512, views[i].k_base, views[i].v_base, v.page_stride, v.page_size, v.num_pages, a.kv_heads, &s->total_rows_) != 0)
            return nullptr;
    }
    s->layers_ = upload(records.data(), records.size() * sizeof(PhDecodeLayer), stream);
    s->maps_ = upload(maps.data(), maps.size(), stream);
    s->shares_ = upload(shares.data(), shares.size() * 4, stream);
    const std::vector<int32_t> zeros((size_t)k.counters(s->n_layers_, a.kv_heads), 0);
    s->counters_ = upload(zeros.data(), zeros.size() * 4, stream);
    return s;
}

// Keys times kv heads of a step.  The ring streams keys at 5.8 TB/s and the attention kernel at 6.3, so beyond some 150 us of them a
// layer what the launch saves is lost again: us a layer with a launch per operation and with one, 0.6B shape, five rows of 32,768
// (1.3 million) 143 and 138, eight of 65,536 (4.2) 363 and 422; 8B shape, eight rows of 8,192 (0.5) 136 and 135, five of 32,768 195
// and 198; width 2,048 with 16 kv heads, eight rows of 8,192 (1.05) 137 and 137, of 16,384 (2.1) 213 and 222.
constexpr long long kMostKeys = 1 << 20;

bool DecodeStack::short_enough(const std::vector<int>& lengths) const {
    long long keys = 0;
    for (int n : lengths) keys += n;
    return keys * first_.kv_heads <= kMostKeys;
}

bool DecodeStack::takes(const StepContext& ctx) const {
    if (refused_ || !ctx.decode_only || ctx.T > kMostRows || ctx.T != ctx.S || ctx.n_decode_rows != ctx.T || !short_enough(ctx.ctx_lens)) return false;
    // (a profile says what each operation takes, which one launch for all of them cannot)
    if (LaunchProfile::get().on() || ctx.option("decode_stack") == "off") return false;
    for (const char* choice : {"decode_kernel", "decode_splits", "row_factor", "norm_ahead"})
        if (ctx.options && ctx.options->find(choice)) return false;
    return layers_kernels().supports(ctx.T, (int)first_.width, first_.heads, first_.kv_heads, first_.head_dim, (int)first_.inner, page_size_, n_layers_,
                                     most_groups_) != 0;
}

bool DecodeStack::run(ResidualStream& stream, StepContext& ctx) const {
    const int T = ctx.T, group = first_.heads / first_.kv_heads;
    const int64_t E = first_.width, D = first_.head_dim, pieces = 2 * num_ctas_;
    Workspace& ws = *ctx.workspace;
    const GroupStep& g = ctx.groups.at(group_);
    PhDecodeLayersArgs a{};
    a.layers = static_cast<const PhDecodeLayer*>(layers_.data());
    a.maps = maps_.data();
    a.shares = static_cast<const int32_t*>(shares_.data());
    a.counters = static_cast<int32_t*>(counters_.data());
    a.n_layers = n_layers_; a.width = (int)E; a.heads = first_.heads; a.kv_heads = first_.kv_heads; a.inner = (int)first_.inner;
    a.page_size = page_size_; a.total_rows = total_rows_; a.max_position = (int)first_.max_position;
    a.most_groups = most_groups_; a.page_stride = page_stride_;
    a.norm_eps = first_.norm_eps; a.qk_eps = first_.qk_eps; a.scale = first_.scale;
    a.rotation = first_.rotation;
    a.rows = T;
    a.block_table = g.block_table; a.table_width = g.table_width;
    a.row_seg = ctx.row_seg;
    a.positions = ctx.position_column(0);
    a.rotation_positions = ctx.position_column(first_.position_column);
    a.slots = g.slot_mapping;
    a.x = stream.x.as<float>();
    a.xw = ws.get("stack_xw", {T, E}, DType::BF16).data;
    a.sumsq = ws.get("stack_sumsq", {T, E / 16}, DType::F32).as<float>();
    a.qkv = ws.get("stack_qkv", {T, (first_.heads + 2 * first_.kv_heads) * D}, DType::F32).as<float>();
    a.attn = ws.get("stack_attn", {T, first_.heads * D}, DType::BF16).data;
    a.act = ws.get("stack_act", {T, first_.inner}, DType::BF16).data;
    a.part_o = ws.get("stack_part_o", {pieces, group, D}, DType::F32).as<float>();
    a.part_ml = ws.get("stack_part_ml", {pieces, group, 2}, DType::F32).as<float>();
    a.error_flag = ctx.attention_error;
    a.wait_cycles = wait_cycles_;
    const LayersKernels& k = layers_kernels();
    const int status = refuse_next_ ? PH_LAYERS_REFUSED : k.decode_layers(&a, ctx.stream);
    if (status == PH_LAYERS_REFUSED) {
        refused_ = true;                                  // and from now on a launch per operation
        return false;
    }
    QE_LAUNCH(k, status);
    stream.clear();
    return true;
}

void DecodeStack::stall(long long wait_cycles, cudaStream_t stream) {
    refuse_next_ = wait_cycles < 0;
    wait_cycles_ = std::max(wait_cycles, 0ll);
    const int32_t first = wait_cycles_ ? -1 : 0;          // the counter of the first part; a launch leaves zeros
    QE_CUDA(cudaMemcpyAsync(static_cast<int32_t*>(counters_.data()) + 1, &first, 4, cudaMemcpyHostToDevice, stream));
    QE_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace qe
