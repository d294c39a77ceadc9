// All layers of a decode step of a few rows as one launch (csrc/decode_layers.cu): what is fixed for a model and its cache, and
// which steps take it.
//
// Models whose every layer is pre-norm with RMS norms, attention with a norm per head of 128 and half-pair rotation over all
// earlier positions, and a SwiGLU feed-forward, all in bfloat16.  Steps of at most eight requests with one token each.
#pragma once

#include <memory>
#include <vector>

#include "parts.h"

namespace qe {

class QE_API DecodeStack {
public:
    // Null when the layers or the cache entries do not fit.
    static std::unique_ptr<DecodeStack> make(const std::vector<DecodeLayerSpec>& layers, const std::vector<CacheView>& views, cudaStream_t stream);
    // Whether this step goes through the one launch.  The option "decode_stack": "off" keeps a launch per operation, and so does a choice
    // among the kernels that such a step is made of ("decode_kernel", "decode_splits", "row_factor", "norm_ahead"), and a profile.
    bool takes(const StepContext& ctx) const;
    // The part of takes() that a step's lengths decide; a graph is captured for either answer.
    bool short_enough(const std::vector<int>& lengths) const;
    // Every layer over the rows of stream.x, in place; nothing is pending afterwards.  False: the device refused the launch (its CTAs
    // must all be resident) and nothing was done; takes() says no from then on.
    bool run(ResidualStream& stream, StepContext& ctx) const;
    // For tests: the next launch waits for a CTA that never reports, and every wait from now on ends after so many cycles (0: as usual,
    // and nobody is waited for in vain; negative: as if the device refused the next launch).
    void stall(long long wait_cycles, cudaStream_t stream);
private:
    DecodeStack() = default;
    DecodeLayerSpec first_;
    int n_layers_ = 0, group_ = 0, page_size_ = 0, total_rows_ = 0, most_groups_ = 0, num_ctas_ = 0;
    long long page_stride_ = 0, wait_cycles_ = 0;
    bool refuse_next_ = false;
    mutable bool refused_ = false;
    DeviceBuffer layers_, maps_, shares_, counters_;
};

}  // namespace qe
