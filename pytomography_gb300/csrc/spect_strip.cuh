// Warp-strip building blocks of the PSF projectors: one warp blurs a strip of rows of one
// rotated plane on its own, so the plane loop needs no CTA barrier.
//
// A strip is RS = 8 G consecutive rows (y) of one plane, G = 32 / QL lane groups of QL lanes;
// QL (8, 16 or 32) lanes cover a row's z quads.  The separable blur runs in two passes:
//   y pass  a lane owns 4 z columns x 8 rows and streams the input rows once: every loaded
//           float4 feeds up to 8 output rows (16 packed FMAs per tap);
//   z pass  a lane owns 16 z values x 1 row pair and streams the pair's z line once: every
//           loaded (row, row + 1) pair feeds up to 16 outputs (16 packed FMAs per tap).
// Both passes therefore issue 16 independent f32x2 FMAs per tap against one (y) or half (z)
// 16-byte shared load, so the FMA pipe and not the shared-memory pipe is the limit.
// Between the passes a row pair lies interleaved, (row, row + 1) per z, in the warp's own
// shared buffer: z index zz = z + HB at float2 offset zz + 2 (zz >> 4); the 16-byte gap after
// every 16 values and the pair stride keep the 8 lanes of every quarter warp on different
// banks in the stores of the y pass and in the loads of the z pass.
//
// Taps: a plane whose outermost nonzero tap is at distance h runs the unrolled loops of the
// smallest half width of the ladder that holds h, taps centred and zero padded.
#pragma once
#include <type_traits>

#include "spect_kernels.cuh"

namespace gb {

constexpr int kLadder = 9;
__host__ __device__ constexpr int ladder_half(int l) {
    return l < 7 ? 2 * l + 2 : 4 * l - 10;  // 2, 4, 6, 8, 10, 12, 14, 18, 22
}
// Smallest ladder entry that holds half width h (h <= 22).
__host__ __device__ constexpr int ladder_index(int h) {
    int l = 0;
    while (l < kLadder - 1 && ladder_half(l) < h) l++;
    return l;
}

// Calls f(std::integral_constant<int, 2 h + 1>) for ladder entry l.
template <typename F>
__device__ __forceinline__ void ladder_dispatch(int l, F &&f) {
    switch (l) {
        case 0: f(std::integral_constant<int, 2 * ladder_half(0) + 1>{}); break;
        case 1: f(std::integral_constant<int, 2 * ladder_half(1) + 1>{}); break;
        case 2: f(std::integral_constant<int, 2 * ladder_half(2) + 1>{}); break;
        case 3: f(std::integral_constant<int, 2 * ladder_half(3) + 1>{}); break;
        case 4: f(std::integral_constant<int, 2 * ladder_half(4) + 1>{}); break;
        case 5: f(std::integral_constant<int, 2 * ladder_half(5) + 1>{}); break;
        case 6: f(std::integral_constant<int, 2 * ladder_half(6) + 1>{}); break;
        case 7: f(std::integral_constant<int, 2 * ladder_half(7) + 1>{}); break;
        default: f(std::integral_constant<int, 2 * ladder_half(8) + 1>{}); break;
    }
}

constexpr int kStripTaps = 48;    // floats per tap row in shared memory (45 taps, 16-byte rows)
constexpr int kStripPlanes = 64;  // planes of a work item at most
constexpr int kStripMaxRows = 192;  // rows of a plane at most (N <= 128 and a 22-row halo)

// Halo of the warp buffer in z (a multiple of 4 that holds the ladder's half width).
__host__ __device__ constexpr int strip_hb(int half) { return half <= 14 ? 16 : 24; }

// float2 elements of one row pair in the warp buffer: 4 QL values and the halo, 2 per 16
// values of padding, and a remainder mod 16 that spreads the pairs of a quarter warp.
__host__ __device__ constexpr int strip_pair(int QL, int hb) {
    const int z = 4 * QL + 2 * hb, n = z + 2 * (z / 16) + 2;
    const int rem = QL == 32 ? 0 : QL == 16 ? 8 : 4;
    return (n - rem + 15) / 16 * 16 + rem;
}
__host__ __device__ constexpr int strip_buf(int QL, int hb) {  // float2 per warp
    return 4 * (32 / QL) * strip_pair(QL, hb);
}
__host__ __device__ constexpr int strip_ql(int nz) { return nz > 64 ? 32 : nz > 32 ? 16 : 8; }

// Slabs of 8 quad positions (32 values) of a row in the forward's second kernel.
__host__ __device__ inline int strip_slabs(const SpectDev &g) { return (g.zg + 1) / 2; }

__device__ __forceinline__ int strip_at(int zz) { return zz + 2 * (zz >> 4); }

// y pass: acc[j] += sum_t tap[t] row[j + t] for the lane's 8 rows, rows `stride` floats
// apart from sp on (the first tap's row of output row 0).  CHECK: row i counts only when
// 0 <= i - lo < n; the others are read from `zero`, a row of zeros (an address select: a
// branch here, taken by part of the lanes at a plane's first and last rows, would expose the
// latency of every load).
template <int KK, bool CHECK>
__device__ __forceinline__ void strip_y_pass(const float *__restrict__ sp, int stride,
                                             const float *__restrict__ tap, float2 (&acc)[8][2],
                                             int lo = 0, int n = 0,
                                             const float *__restrict__ zero = nullptr) {
    float w[KK + 3];
#pragma unroll
    for (int i = 0; i < KK + 7; i++) {
        if (i < KK && i % 4 == 0) {
            const float4 t4 = *reinterpret_cast<const float4 *>(tap + i);
            w[i] = t4.x;
            w[i + 1] = t4.y;
            w[i + 2] = t4.z;
            if (i + 3 < KK + 3) w[i + 3] = t4.w;
        }
        const float *p = sp + i * stride;
        if (CHECK) p = (unsigned)(i - lo) < (unsigned)n ? p : zero;
        const float4 v = *reinterpret_cast<const float4 *>(p);
        const float2 va = make_float2(v.x, v.y), vb = make_float2(v.z, v.w);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int t = i - j;
            if (t < 0 || t >= KK) continue;
            const float2 wt = make_float2(w[t], w[t]);
            acc[j][0] = __ffma2_rn(wt, va, acc[j][0]);
            acc[j][1] = __ffma2_rn(wt, vb, acc[j][1]);
        }
    }
}

// z pass: o[j] = sum_t tap[t] pair[j + t] for 16 consecutive z of one row pair; bp points at
// the z group's first value (offset strip_at(16 c) of the pair).
template <int KK, int HB>
__device__ __forceinline__ void strip_z_pass(const float2 *__restrict__ bp,
                                             const float *__restrict__ tap, float2 (&o)[16]) {
    constexpr int REL = HB - KK / 2;  // even: HB and every ladder half width are
    static_assert(REL >= 0 && REL % 2 == 0, "the window starts on a 16-byte boundary");
#pragma unroll
    for (int j = 0; j < 16; j++) o[j] = make_float2(0.f, 0.f);
    float w[KK + 3];
#pragma unroll
    for (int i = 0; i < KK + 15; i += 2) {
        if (i < KK && i % 4 == 0) {
            const float4 t4 = *reinterpret_cast<const float4 *>(tap + i);
            w[i] = t4.x;
            w[i + 1] = t4.y;
            w[i + 2] = t4.z;
            if (i + 3 < KK + 3) w[i + 3] = t4.w;
        }
        const int rel = REL + i;
        const float4 v = *reinterpret_cast<const float4 *>(bp + rel + 2 * (rel >> 4));
        const float2 v0 = make_float2(v.x, v.y), v1 = make_float2(v.z, v.w);
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int t = i - j;
            if (t < 0 || t >= KK) continue;
            o[j] = __ffma2_rn(make_float2(w[t], w[t]), v0, o[j]);
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int t = i + 1 - j;
            if (t < 0 || t >= KK) continue;
            o[j] = __ffma2_rn(make_float2(w[t], w[t]), v1, o[j]);
        }
    }
}

// The z pass of a 1-D PSF: the lane's 16 values as they are (a pass of one tap of 1 and zeros
// would spread an infinity or NaN over the taps' width).
template <int HB>
__device__ __forceinline__ void strip_z_copy(const float2 *__restrict__ bp, float2 (&o)[16]) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
        const int rel = HB + j;
        const float4 v = *reinterpret_cast<const float4 *>(bp + rel + 2 * (rel >> 4));
        o[j] = make_float2(v.x, v.y);
        o[j + 1] = make_float2(v.z, v.w);
    }
}

// Shared bookkeeping of one work item (planes [x0, x1) of one angle, at most kStripPlanes):
// its occupied planes in order and the plane of every strip.
struct StripItem {
    int4 plane[kStripPlanes];  // (first row, last row, first strip, plane * 16 + ladder entry)
    int n_planes, n_strips;
    int next;  // strip counter of the CTA's warps
    int pad;
    unsigned char plane_of[kStripPlanes * kStripMaxRows / 8];  // last: not filled for RS = 0
};
constexpr int kStripItemBytes = (sizeof(StripItem) + 15) / 16 * 16;
constexpr int kPlaneTableBytes = 16 * kStripPlanes + 16;  // without plane_of
constexpr int kStripTapFloats = kStripPlanes * kStripTaps;  // of one direction

// Copies 16 bytes global -> shared without a register; wait with cp_async_wait_all.
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Fills the item's plane table from the plan's (tab: the angle's planes), in strips of RS
// rows (0: no strips).  Called by one warp.
template <int RS>
__device__ __forceinline__ void strip_planes(const int4 *__restrict__ tab, int x0, int x1,
                                             StripItem *it) {
    const int lane = threadIdx.x & 31;
    int4 t[kStripPlanes / 32];
#pragma unroll
    for (int h = 0; h < kStripPlanes / 32; h++) {
        const int xp = x0 + 32 * h + lane;
        t[h] = xp < x1 ? __ldg(tab + xp) : make_int4(0, -1, 0, 0);
    }
    int planes = 0, strips = 0;
#pragma unroll
    for (int h = 0; h < kStripPlanes / 32; h++) {
        const bool hit = t[h].y >= t[h].x;
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        const int at = planes + __popc(hits & ((1u << lane) - 1));
        const int ns = hit && RS ? (t[h].y - t[h].x + RS) / max(RS, 1) : 0;
        int end = ns;  // inclusive scan of the strips
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += v;
        }
        if (hit) {
            const int s0 = strips + end - ns;
            it->plane[at] = make_int4(t[h].x, t[h].y, s0, (x0 + 32 * h + lane) * 16 + t[h].z);
            for (int s = s0; s < s0 + ns; s++) it->plane_of[s] = (unsigned char)at;
        }
        planes += __popc(hits);
        strips += __shfl_sync(0xffffffffu, end, 31);
    }
    if (lane == 0) {
        it->n_planes = planes;
        it->n_strips = strips;
        it->next = 0;
    }
}

// Starts the copies of the taps of planes [x0, x1) (by the whole CTA; cp_async_wait_all and a
// barrier make them visible): 2 kStripTaps floats per plane, y before z, or the y (DIR = 0) or
// z (DIR = 1) taps alone.  Rows are indexed by plane - x0.
template <int DIR = 2>
__device__ __forceinline__ void strip_taps(const SpectDev &g, int ga, int x0, int x1,
                                           float *taps) {
    constexpr int Q = kStripTaps / 4 * (DIR == 2 ? 2 : 1);  // 16-byte pieces per plane
    const float *src = g.staps + ((size_t)g.group[ga] * g.Lp + x0) * 2 * kStripTaps +
                       (DIR == 1 ? kStripTaps : 0);
    for (int i = threadIdx.x; i < (x1 - x0) * Q; i += blockDim.x)
        cp_async16(taps + 4 * i, src + (size_t)(i / Q) * 2 * kStripTaps + 4 * (i % Q));
}

// The next strip of the item for this warp (-1: none left).
__device__ __forceinline__ int strip_next(StripItem *it, int lane) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&it->next, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    return t < it->n_strips ? t : -1;
}

// Brings the A rows of strip s into L2 (a 128-byte line per lane and step): issued one strip
// ahead, so the loads of the strip itself do not wait for DRAM.
template <int RS>
__device__ __forceinline__ void strip_prefetch(const SpectDev &g, const StripItem *it, int s,
                                               const float *__restrict__ A, int lane) {
    const int4 pi = it->plane[it->plane_of[s]];
    const int y0 = pi.x + (s - pi.z) * RS, rows = min(RS, pi.y - y0 + 1);
    const float *p = A + ((size_t)(pi.w >> 4) * g.nya + (y0 - g.ya_lo)) * g.nzs;
    for (int i = 32 * lane; i < rows * g.nzs; i += 1024)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
}

// Stores the lane's 8 rows x 4 columns (first z column zz - HB) as interleaved row pairs.
__device__ __forceinline__ void strip_store_pairs(float2 *__restrict__ buf, int pair0, int stride,
                                                  int zz, const float2 (&acc)[8][2]) {
#pragma unroll
    for (int jp = 0; jp < 4; jp++) {
        float4 *d = reinterpret_cast<float4 *>(buf + (pair0 + jp) * stride + strip_at(zz));
        const float2 a0 = acc[2 * jp][0], a1 = acc[2 * jp][1];
        const float2 b0 = acc[2 * jp + 1][0], b1 = acc[2 * jp + 1][1];
        d[0] = make_float4(a0.x, b0.x, a0.y, b0.y);
        d[1] = make_float4(a1.x, b1.x, a1.y, b1.y);
    }
}

}  // namespace gb
