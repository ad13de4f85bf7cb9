// Host-side launchers of the SPECT kernels (implemented in spect_fwd.cu / spect_bwd.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "gbtomo.h"
#include "spect_kernels.cuh"

// PSF tap-count buckets compiled into the library: a plan's taps are zero-padded
// (centred) to the smallest bucket that holds its widest kernel.
#define GB_FOR_EACH_K(X) X(7) X(11) X(15) X(21) X(25) X(29) X(37) X(45)

namespace gb {

inline int psf_bucket(int k) {
    const int b[] = {7, 11, 15, 21, 25, 29, 37, 45};
    for (int v : b)
        if (k <= v) return v;
    return -1;
}

// Forward PSF kernel: rows per TMA box of its attenuation copy, and the length of its
// sample rows in shared memory for a z slab of zw (rounded to the output block) with
// half-halo hp: a multiple of 32 floats, so every row starts 128-byte aligned.
constexpr int kBoxRows = 8;
__host__ __device__ constexpr int fwd_s_cols(int zw, int hp) { return (zw + 2 * hp + 31) & ~31; }

// tpb: threads per forward CTA, 512 or 768 (one CTA per SM)
size_t fwd_psf_smem_bytes(int K, int N, int Zt, int tpb);
size_t b1_psf_smem_bytes(int K, int N, int Zt);
// Raise the dynamic shared-memory limit of the PSF kernels (done once at plan creation,
// outside any stream capture).
cudaError_t setup_fwd(int K, size_t smem, int tpb);
cudaError_t setup_b1(int K, size_t smem);

// Work items (int4: slot, first plane, end plane, unused) split each angle's planes
// into ranges of about equal work; partial sums are indexed by item.
// tpb: 512 or 768.  Plans of the strip kernels do not come here.
cudaError_t launch_fwd(const SpectDev &g, const float *f, const int *alist, const int4 *items,
                       int n_items, int Zt, int tpb, float *partials, cudaStream_t st);
// ioff[slot] .. ioff[slot+1]: the items of a slot
cudaError_t launch_reduce(int n_slots, const int *ioff, int NZ, const float *partials, float *out,
                          int ratio, const float *gproj, const float *sadd, const int *alist,
                          float *pred, cudaStream_t st);
cudaError_t launch_b1(const SpectDev &g, const float *proj, const int *alist, int n_slots,
                      const int4 *items, int n_items, int Zt, float *W, cudaStream_t st);
// Strip kernels (spect_strip.cu).  strip_configure sets strip, strip_fwd, zg and nzs of a PSF
// plan whose attenuation, if any, comes before the PSF, with N and nz <= 128 and tiles that
// fit `cap` bytes of shared memory; it leaves every other plan alone.
void strip_configure(SpectDev &g, size_t cap);
cudaError_t setup_strip(size_t cap);
// Values of one slot (angle) of the W stack: rows of the back projection, or of the forward.
inline size_t stack_slot(const SpectDev &g) {
    return (size_t)g.Lp * g.nya * (g.strip ? std::max(g.nzs, 32 * ((g.zg + 1) / 2)) : g.nzs);
}
cudaError_t launch_fwd_strip(const SpectDev &g, const float *f, const int *alist,
                             const int4 *items, int n_items, const int4 *yitems, int n_yitems,
                             float *W, float *partials, cudaStream_t st);
cudaError_t launch_b1_strip(const SpectDev &g, const float *proj, const int *alist,
                            const int4 *items, int n_items, float *W, cudaStream_t st);
cudaError_t launch_b2_gather(const SpectDev &g, const float *W, const int *alist, int n_slots,
                             float *out, int mode, const UpdateArgs &u, cudaStream_t st);
// Plans without PSF: B1 and the gather in one kernel.  It takes whole z quads, 16-byte aligned
// projections and blocks whose sample table fits; other calls run B1 and the gather.
bool b2_nopsf_ok(const SpectDev &g, const float *proj, int n_slots);
cudaError_t launch_b2_nopsf(const SpectDev &g, const float *proj, const int *alist, int n_slots,
                            float *out, int mode, const UpdateArgs &u, cudaStream_t st);
cudaError_t launch_b2_adjoint(const SpectDev &g, const float *W, const int *alist, int n_slots,
                              float *out, bool first, cudaStream_t st);
cudaError_t launch_atten(const SpectDev &g, const float *mu, float dx, int n_angles, float *A,
                         cudaStream_t st);
cudaError_t launch_rdp(const float *f, float *grad, int nx, int ny, int nz, const UpdateArgs &u,
                       float beta_scale, cudaStream_t st);
cudaError_t launch_rdp_hvp(const float *f, const float *x, float *out, int nx, int ny, int nz,
                           const UpdateArgs &u, float beta_scale, cudaStream_t st);

// ------------------------------------------------------------------ batches
// Persistent / flat launches over several "entries" (a reconstruction, or one object of a
// batch on a shared plan) at once.  Each entry carries its plan's device description and
// its own buffers; the structures travel as kernel parameters (__grid_constant__), so a
// launch reads no descriptor from global memory and can be recorded in a CUDA graph.
constexpr int kMaxBatch = 32;

struct FwdBatch {
    CUtensorMap tm[kMaxBatch];  // attenuation boxes of each entry (64-byte aligned)
    SpectDev g[kMaxBatch];
    float *W[kMaxBatch];            // strip entries: the rows between the two kernels
    const float *f[kMaxBatch];      // object of each entry
    const int *alist[kMaxBatch];    // the group's angles, per entry
    const int4 *items;              // (slot, first plane, end plane, entry), largest first
    int n_items;
    const int4 *yitems;             // strip entries: items of the second kernel
    int n_yitems;
    int *counter;                   // work-queue position, zeroed before the launch
    float *partials;                // [n_items (strip entries: n_yitems)][nz_max]
    int nz_max;
};

struct ReduceBatch {
    float *out[kMaxBatch];          // [n_sel][N][nz] of each entry
    const float *gproj[kMaxBatch];  // measured projections [n_angles][N][nz] (ratio mode)
    const float *sadd[kMaxBatch];   // additive term, same layout, or null
    const int *alist[kMaxBatch];
    int NZ[kMaxBatch];              // N * nz of each entry
    const int2 *rows;               // (entry, slot) of every output row
    const int *row_off;             // [n_rows + 1] offsets into row_items
    const int *row_items;           // work items of each row in plane order
    const float *partials;
    int nz_max;
    int ratio;                      // 1: out = g / (sum + s + delta)
};

struct B1Batch {
    SpectDev g[kMaxBatch];          // wrange: the entry's own row ranges
    const float *proj[kMaxBatch];   // projection rows of the group's slots
    const int *alist[kMaxBatch];    // the group's angles
    float *W[kMaxBatch];            // [slots][Lp][nya][nz]
    const int4 *items;              // (slot in group, first plane, end plane, entry)
    int n_items;
    int *counter;
};

struct B2Batch {
    SpectDev g[kMaxBatch];
    const float *W[kMaxBatch];
    const int *alist[kMaxBatch];    // the group's angles
    int n_slots[kMaxBatch];
    float *out[kMaxBatch];          // target (write / add) or OSEM object
    const float *nbp[kMaxBatch];    // OSEM: H_m^T 1
    const float *acc[kMaxBatch];    // OSEM: back projection of earlier groups, or null
    int block_off[kMaxBatch + 1];   // first block of each entry (total for unused entries)
    int mode[kMaxBatch];            // gather: B2_WRITE, B2_ADD or B2_OSEM per entry
};

#define GB_DECL_FWD_BATCH(KK)                                                               \
    cudaError_t setup_fwd_psf_batch_##KK();                                                 \
    cudaError_t launch_fwd_psf_batch_##KK(const FwdBatch &p, int grid, cudaStream_t st);
GB_FOR_EACH_K(GB_DECL_FWD_BATCH)
#undef GB_DECL_FWD_BATCH
// Tensor map of a plan's attenuation table for the forward kernel's box copies (a zeroed map
// when the kernel makes none); s_cols is the kernel's S row length.
cudaError_t make_att_tmap(const SpectDev &g, int s_cols, CUtensorMap *out);
cudaError_t setup_b1_batch(int K);
// n entries, of which those with g.strip > 0 have items
cudaError_t launch_fwd_strip_batch(const FwdBatch &p, int n, int grid, cudaStream_t st);
cudaError_t launch_b1_strip_batch(const B1Batch &p, int n, int grid, cudaStream_t st);
cudaError_t launch_b1_batch(int K, const B1Batch &p, int grid, cudaStream_t st);
cudaError_t launch_reduce_batch(const ReduceBatch &p, int n_rows, cudaStream_t st);
cudaError_t launch_b2_gather_batch(const B2Batch &p, int n_blocks, cudaStream_t st);
cudaError_t launch_b2_adjoint_batch(const B2Batch &p, int n_blocks, cudaStream_t st);
// blocks of 256 threads of one entry in the batched gather and adjoint kernels
int b2_gather_blocks(const SpectDev &g);

constexpr int kGroup = 16;  // angles of a plan that share the W stack

// Scratch of gb_spect_forward_static: partial sums, and the strip kernels' rows of a group of
// angles.
struct StaticScratch {
    float *partials, *rows;
};
constexpr size_t kStaticPartials = (size_t)4 << 20, kStaticRows = (size_t)64 << 20;  // floats

// One forward projection of a plan in that scratch (for entry points defined outside
// spect_plan.cu): the work items and partial floats a subset needs (false when the subset is out
// of range), and the projection itself.
bool plan_forward_need(const gb_spect_plan *p, int subset, int *n_sel, int *n_items,
                       size_t *floats);
gb_status plan_forward(gb_spect_plan *p, const float *obj, int subset, float *out,
                       const StaticScratch &fixed, cudaStream_t st);

}  // namespace gb
