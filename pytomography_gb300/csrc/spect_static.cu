// Forward projection that allocates nothing: its cross-chunk partial sums, and the rows between
// the two strip kernels, live in fixed file-scope device arrays instead of the plan's scratch.
//
// Who needs it: callers that must not allocate device memory while they run — code on a
// stream whose memory pool forbids further cudaMalloc, host processes whose device memory
// is owned by another framework's allocator, or long-running services that budget every
// allocation up front.  They
// create their plan once at set-up; afterwards this entry point touches only the plan's
// read-only tables, the caller's input and output, and the static arrays below.
//
// Limits and behaviour:
//   * the arrays hold kStaticPartials (16 MiB) and kStaticRows floats (256 MiB: the rows of a
//     group of 16 angles at 128 x 128 x 128); every GPU that loads the library keeps them until
//     the process exits.  (64 MiB, with item lists of their own for groups of 4 angles, took 140
//     us where this takes 105, and made every plan's lists 0.4 ms dearer);
//   * the plan's work items times nx * nz partial sums must fit (at least one item per
//     angle); larger requests are rejected with GB_ERR_SHAPE;
//   * every call shares the arrays and the kernels overwrite every partial they later
//     read (nothing needs to start at zero), so calls that overlap on the GPU (other
//     streams, other threads) race: order them on one stream;
//   * the first call on a device looks the arrays' device addresses up with
//     cudaGetSymbolAddress (with that device current) and caches them; make that first
//     call before any stream capture.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "spect_launch.h"

namespace gb {

static __device__ __align__(256) float g_fwd_static_scratch[kStaticPartials];
static __device__ __align__(256) float g_fwd_static_rows[kStaticRows];
// (a strip plan's largest slot: 128 rows of taps of 22 on both sides, 182 planes, 128 values)
static_assert(kStaticRows >= (size_t)kGroup * 182 * (128 + 2 * 22) * 128, "a group's rows fit");

static std::mutex g_static_mu;
static StaticScratch g_static_ptr[64] = {};

// Device addresses of the static arrays on the current device (looked up once per device).
static gb_status static_scratch(StaticScratch *out) {
    int dev = 0;
    GB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("device ordinal %d out of range", dev);
        return GB_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev].partials) {
        void *p = nullptr, *r = nullptr;
        GB_CUDA(cudaGetSymbolAddress(&r, g_fwd_static_rows));
        GB_CUDA(cudaGetSymbolAddress(&p, g_fwd_static_scratch));
        g_static_ptr[dev] = {static_cast<float *>(p), static_cast<float *>(r)};
    }
    *out = g_static_ptr[dev];
    return GB_OK;
}

}  // namespace gb

using namespace gb;

extern "C" gb_status gb_spect_forward_static(gb_spect_plan *plan, const float *object,
                                             float *proj, int32_t subset, gb_stream_t stream) {
    clear_error();
    GB_CHECK_ARG(plan && object && proj, "null argument");
    int n_sel = 0, n_items = 0;
    size_t need = 0;
    if (!plan_forward_need(plan, subset, &n_sel, &n_items, &need)) {
        set_error("subset %d out of range", subset);
        return GB_ERR_STATE;
    }
    if (need > kStaticPartials) {
        set_error("forward of %d angles (%d work items) needs %zu floats of scratch; the static "
                  "array holds %u",
                  n_sel, n_items, need, (unsigned)kStaticPartials);
        return GB_ERR_SHAPE;
    }
    StaticScratch scratch{};
    gb_status s = static_scratch(&scratch);
    if (s != GB_OK) return s;
    return plan_forward(plan, object, subset, proj, scratch, as_stream(stream));
}
