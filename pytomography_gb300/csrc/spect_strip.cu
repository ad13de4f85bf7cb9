// Strip form of the PSF projectors (spect_strip.cuh) for planes of at most 128 rows and 128 z
// values: attenuation, if any, before the PSF.
//
// Why: the plane-at-a-time kernels (k_fwd_psf, k_b1_psf) run every plane through three passes
// with a CTA barrier after each, 16 warps to an SM, and spend most of their time waiting (FMA
// pipe 30% busy).  Here no warp waits for another while it samples and blurs.  Measured on one
// 12-angle subset of the 128^3, 120-angle workload, FMA pipe busy in brackets:
//   rotated-frame back projection   128 us (26%) -> 60 us (58%)
//   forward                         160 us (30%) -> 60 us (38%) + 37 us (55%), k_fwd_strip
//                                   and k_fwd_ysum; the rows between the two kernels cost
//                                   66 MB of DRAM writes and 113 MB of reads
// and on 9 angles of 101 x 101 x 83 (nz odd: scalar object loads, padded rows) one OSEM
// iteration of 5 subsets went from 1386 to 662 us (its dependent launches included).
// More than 128 z values do not fit the lanes of a row (32 of 4 values); more than 128 rows
// would fit shared memory up to about 190, but k_fwd_ysum has four summing warps of 32 rows and
// its launch bound for them.  Those planes and the PSF-before-attenuation order keep the
// plane-at-a-time kernels (an attenuation inside the blur leaves the back projection no common
// input for the planes of an angle).
#include <algorithm>

#include "spect_launch.h"
#include "spect_strip.cuh"

namespace gb {

// ---------------------------------------------------------------- B1
// W[xp][y][z] = A (.) PSF_xp(P), rows y within 1.5 pixels of the object square.  The
// projection P of the item's angle is the input of every plane, so it is staged once and the
// warps then take strips of any plane independently (no barrier in the loop): y pass from
// the staged P, z pass from the warp's buffer, times A, store.
struct B1StripLayout {  // dynamic shared memory, in floats
    int rows;      // staged rows of P with their zero halo
    int top;       // zero rows above P's row 0
    size_t item, taps, bufs, total;
};
__host__ __device__ inline B1StripLayout b1_strip_layout(const SpectDev &g, int QL, int warps) {
    const int RS = 8 * (32 / QL), hl = ladder_half(ladder_index(g.K / 2));
    B1StripLayout L;
    L.top = g.pad - g.ya_lo + hl;
    L.rows = (g.ya_hi - g.pad) + RS - 1 + hl + L.top;
    L.item = (size_t)L.rows * 4 * QL;
    L.taps = L.item + kStripItemBytes / sizeof(float);
    L.bufs = L.taps + 2 * kStripTapFloats;
    L.total = L.bufs + (size_t)warps * 2 * strip_buf(QL, strip_hb(hl));
    return L;
}

// Four z values from z on (< nz) at p where `ok`, else zeros; vec: one 16-byte load.
__device__ __forceinline__ float4 ld_quad(bool ok, const float *p, int z, int nz, bool vec) {
    if (vec) return ld_data4_if(ok, p);
    return make_float4(ld_data_if(ok, p), ld_data_if(ok && z + 1 < nz, p + 1),
                       ld_data_if(ok && z + 2 < nz, p + 2), ld_data_if(ok && z + 3 < nz, p + 3));
}

// 16-byte load that stays behind the last __syncwarp: hoisted above the z pass, the loads of a
// strip's A would not fit the registers beside its sums.
__device__ __forceinline__ float4 ldg_here(const float *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

template <int QL, int HB, bool Z2>
__device__ __forceinline__ void b1_strip_item(const SpectDev &g, const float *proj,
                                              const int ga, const int x0, const int x1,
                                              float *__restrict__ Ws, float *__restrict__ sm) {
    constexpr int G = 32 / QL, RS = 8 * G, ZG = QL / 4, SC = 4 * QL;
    constexpr int PS = strip_pair(QL, HB);
    const int N = g.N, nz = g.nz, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const B1StripLayout L = b1_strip_layout(g, QL, blockDim.x >> 5);
    StripItem *it = reinterpret_cast<StripItem *>(sm + L.item);
    float *taps = sm + L.taps;
    float2 *buf = reinterpret_cast<float2 *>(sm + L.bufs) + (size_t)warp * strip_buf(QL, HB);
    strip_taps(g, ga, x0, x1, taps);
    for (int i = lane; i < strip_buf(QL, HB) / 2; i += 32)  // the z halo stays zero
        reinterpret_cast<float4 *>(buf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp == 0) strip_planes<RS>(g.planes_bwd + (size_t)ga * g.Lp, x0, x1, it);
    grid_wait();
    const float *P = after_wait(proj);
    // P with its zero halo
    const bool vec = nz % 4 == 0 && ((uintptr_t)P & 15) == 0;
    for (int i = threadIdx.x; i < L.rows * QL; i += blockDim.x) {
        const int r = i / QL - L.top, z = 4 * (i % QL);
        const bool in = (unsigned)r < (unsigned)N && z < nz;
        const float *p = P + (size_t)r * nz + z;
        if (in && vec) {
            cp_async16(sm + 4 * i, p);
            continue;
        }
        *reinterpret_cast<float4 *>(sm + 4 * i) = ld_quad(in, p, z, nz, false);
    }
    cp_async_wait_all();
    __syncthreads();
    const int q = lane % QL, grp = lane / QL;  // y pass: z quad, row group
    const int c = lane % ZG, pr = lane / ZG;   // z pass: z group, row pair
    const float *A = g.att ? g.A + (size_t)ga * g.Lp * g.nya * g.nzs : nullptr;
    for (int s = strip_next(it, lane), sn; s >= 0; s = sn) {
        const int pl = it->plane_of[s];
        const int4 pi = it->plane[pl];
        const int xp = pi.w >> 4;
        const int y0 = pi.x + (s - pi.z) * RS, yl = pi.y;
        sn = strip_next(it, lane);
        if (A && sn >= 0) strip_prefetch<RS>(g, it, sn, A, lane);
        const float *tap = taps + (xp - x0) * 2 * kStripTaps;
        const int y = y0 + 2 * pr;  // the z pass's row pair
        ladder_dispatch(pi.w & 15, [&](auto kk) {
            constexpr int KK = decltype(kk)::value;
            if constexpr (KK / 2 <= HB) {
                {
                    float2 acc[8][2];
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = make_float2(0.f, 0.f);
                    strip_y_pass<KK, false>(
                        sm + (y0 + 8 * grp - g.pad - KK / 2 + L.top) * SC + 4 * q, SC, tap, acc);
                    strip_store_pairs(buf, 4 * grp, PS, 4 * q + HB, acc);
                }
                __syncwarp();
                float2 o[16];
                if constexpr (Z2)
                    strip_z_pass<KK, HB>(buf + pr * PS + 18 * c, tap + kStripTaps, o);
                else
                    strip_z_copy<HB>(buf + pr * PS + 18 * c, o);
                __syncwarp();  // the buffer is free for the next strip
                const size_t off = ((size_t)xp * g.nya + (y - g.ya_lo)) * g.nzs + 4 * c;
                const bool st0 = c < g.zg && y <= yl, st1 = c < g.zg && y + 1 <= yl;
                float4 a[2][4];  // ones without attenuation (the product is then exact)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    a[0][k] = a[1][k] = make_float4(1.f, 1.f, 1.f, 1.f);
                    if (A && st0) a[0][k] = ldg_here(A + off + 4 * k * g.zg);
                    if (A && st1) a[1][k] = ldg_here(A + off + g.nzs + 4 * k * g.zg);
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    float *d = Ws + off + 4 * k * g.zg;
                    if (st0)
                        *reinterpret_cast<float4 *>(d) =
                            mul4(make_float4(o[4 * k].x, o[4 * k + 1].x, o[4 * k + 2].x,
                                             o[4 * k + 3].x), a[0][k]);
                    if (st1)
                        *reinterpret_cast<float4 *>(d + g.nzs) =
                            mul4(make_float4(o[4 * k].y, o[4 * k + 1].y, o[4 * k + 2].y,
                                             o[4 * k + 3].y), a[1][k]);
                }
            }
        });
    }
}

template <int QL, int HB, bool Z2>
__global__ void __launch_bounds__(512, 1)
    k_b1_strip(SpectDev g, const float *proj, const int *__restrict__ alist,
               const int4 *__restrict__ items, float *__restrict__ W) {
    extern __shared__ __align__(128) float sm[];
    grid_release();
    const int4 item = items[blockIdx.x];
    b1_strip_item<QL, HB, Z2>(g, proj + (size_t)item.x * g.N * g.nz, alist[item.x], item.y, item.z,
                          W + (size_t)item.x * g.Lp * g.nya * g.nzs, sm);
}

// Calls f(QL, Z2) (as types) for a batch entry: the lanes of its rows, whether the PSF blurs z.
template <bool ONLY2D, typename F>
__device__ __forceinline__ void strip_dispatch(const SpectDev &g, F &&f) {
    const int ql = strip_ql(g.nz);
    auto both = [&](auto q) {
        if constexpr (ONLY2D)
            f(q, std::true_type{});
        else if (g.psf2d)
            f(q, std::true_type{});
        else
            f(q, std::false_type{});
    };
    if (ql == 32)
        both(std::integral_constant<int, 32>{});
    else if (ql == 16)
        both(std::integral_constant<int, 16>{});
    else
        both(std::integral_constant<int, 8>{});
}

// Persistent batch form: one CTA per SM dequeues the work items of every entry, largest
// first.  The entries share the tap bucket (HB); their row widths and PSF dimensions may differ.
// ONLY2D: every entry's PSF blurs z as well (beside the 1-D forms the kernel is 2% slower).
template <int HB, bool ONLY2D>
__global__ void __launch_bounds__(512, 1) k_b1_strip_batch(const __grid_constant__ B1Batch p) {
    extern __shared__ __align__(128) float sm[];
    __shared__ int s_item;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(p.counter, 1);
        __syncthreads();
        const int i = s_item;
        if (i >= p.n_items) return;
        const int4 item = p.items[i];  // (slot in group, first plane, end plane, entry)
        const int e = item.w, slot = item.x;
        const SpectDev &g = p.g[e];
        const float *P = p.proj[e] + (size_t)slot * g.N * g.nz;
        const int ga = p.alist[e][slot];
        float *W = p.W[e] + (size_t)slot * g.Lp * g.nya * g.nzs;
        strip_dispatch<ONLY2D>(g, [&](auto ql, auto z2) {
            b1_strip_item<decltype(ql)::value, HB, decltype(z2)::value>(g, P, ga, item.y, item.z,
                                                                        W, sm);
        });
    }
}

// ---------------------------------------------------------------- forward
// First kernel: rotated samples times A, blurred along z, into the W stack, here laid out as
// [slot][plane][slab of 8 quad positions][row][32 values], so that the rows of a plane and
// slab are one contiguous piece for the second kernel.  Rows are
// independent, so a warp samples, blurs and stores a strip on its own; the strips of an
// item run over consecutive planes, whose samples share object columns in L1.
struct RowTap {  // bilinear sample of one strip row: north-west corner, inside mask, weights
    int off, mask;
    float nw, ne, sw, se;
    int pad0, pad1;
};

struct FwdStripLayout {  // dynamic shared memory, in floats
    size_t taps, rows, bufs, total;
};
__host__ __device__ inline FwdStripLayout fwd_strip_layout(int QL, int HB, int warps) {
    FwdStripLayout L;
    L.taps = kStripItemBytes / sizeof(float);
    L.rows = L.taps + kStripTapFloats;
    L.bufs = L.rows + (size_t)warps * (256 / QL) * (sizeof(RowTap) / sizeof(float));
    L.total = L.bufs + (size_t)warps * 2 * strip_buf(QL, HB);
    return L;
}

// Rotated samples of four rows at z quad q, times A (Ap: the first row's quad, or null).
__device__ __forceinline__ void gather_rows(const float *f, const SpectDev &g,
                                            const RowTap *rt, int q, bool zin, bool vec,
                                            const float *__restrict__ Ap, float4 (&v)[4]) {
    const int nz = g.nz, step_r = g.N * nz;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int m0 = rt[0].mask, m1 = rt[1].mask, m2 = rt[2].mask, m3 = rt[3].mask;
    if (vec && zin && (m0 & m1 & m2 & m3) == 15) {  // every corner inside the object
        float4 c[4][4], a[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float *p = f + rt[u].off + 4 * q;
            c[u][0] = ld_data4(p);
            c[u][1] = ld_data4(p + nz);
            c[u][2] = ld_data4(p + step_r);
            c[u][3] = ld_data4(p + step_r + nz);
            a[u] = Ap ? __ldg(reinterpret_cast<const float4 *>(Ap + u * g.nzs))
                      : make_float4(1.f, 1.f, 1.f, 1.f);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            Bilin b;
            b.nw = rt[u].nw;
            b.ne = rt[u].ne;
            b.sw = rt[u].sw;
            b.se = rt[u].se;
            v[u] = mul4(make_float4(bilin_combine(b, c[u][0].x, c[u][1].x, c[u][2].x, c[u][3].x),
                                    bilin_combine(b, c[u][0].y, c[u][1].y, c[u][2].y, c[u][3].y),
                                    bilin_combine(b, c[u][0].z, c[u][1].z, c[u][2].z, c[u][3].z),
                                    bilin_combine(b, c[u][0].w, c[u][1].w, c[u][2].w, c[u][3].w)),
                        a[u]);
        }
        return;
    }
    v[0] = v[1] = v[2] = v[3] = zero;
#pragma unroll 1
    for (int u = 0; u < 4; u++) {
        const RowTap t = rt[u];
        const int m = zin ? t.mask : 0;
        const float *p = f + t.off + 4 * q;
        const float4 vnw = ld_quad(m & 1, p, 4 * q, nz, vec);
        const float4 vne = ld_quad(m & 2, p + nz, 4 * q, nz, vec);
        const float4 vsw = ld_quad(m & 4, p + step_r, 4 * q, nz, vec);
        const float4 vse = ld_quad(m & 8, p + step_r + nz, 4 * q, nz, vec);
        const float4 a = Ap && m ? __ldg(reinterpret_cast<const float4 *>(Ap + u * g.nzs)) : zero;
        Bilin b;
        b.nw = t.nw;
        b.ne = t.ne;
        b.sw = t.sw;
        b.se = t.se;
        float4 r = make_float4(bilin_combine(b, vnw.x, vne.x, vsw.x, vse.x),
                               bilin_combine(b, vnw.y, vne.y, vsw.y, vse.y),
                               bilin_combine(b, vnw.z, vne.z, vsw.z, vse.z),
                               bilin_combine(b, vnw.w, vne.w, vsw.w, vse.w));
        if (Ap) r = mul4(r, a);
        // the four results stay in registers: the row's index is not a compile-time constant
        v[0] = u == 0 ? r : v[0];
        v[1] = u == 1 ? r : v[1];
        v[2] = u == 2 ? r : v[2];
        v[3] = u == 3 ? r : v[3];
    }
}

template <int QL, int HB, bool ONLY2D>
__device__ __forceinline__ void fwd_strip_item(const SpectDev &g, const float *obj,
                                               const int ga, const int x0, const int x1,
                                               float *__restrict__ Ws, float *__restrict__ sm) {
    constexpr int G = 32 / QL, RS = 8 * G, ZG = QL / 4, PS = strip_pair(QL, HB);
    const int N = g.N, nz = g.nz, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const FwdStripLayout L = fwd_strip_layout(QL, HB, blockDim.x >> 5);
    StripItem *it = reinterpret_cast<StripItem *>(sm);
    float *taps = sm + L.taps;
    RowTap *rt = reinterpret_cast<RowTap *>(sm + L.rows) + warp * RS;
    float2 *buf = reinterpret_cast<float2 *>(sm + L.bufs) + (size_t)warp * strip_buf(QL, HB);
    strip_taps<1>(g, ga, x0, x1, taps);
    for (int i = lane; i < strip_buf(QL, HB) / 2; i += 32)
        reinterpret_cast<float4 *>(buf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp == 0) strip_planes<RS>(g.planes_fwd + (size_t)ga * g.Lp, x0, x1, it);
    cp_async_wait_all();
    grid_wait();
    const float *f = after_wait(obj);
    __syncthreads();
    float th[6];
#pragma unroll
    for (int k = 0; k < 6; k++) th[k] = g.theta_fwd[6 * ga + k];
    const int q = lane % QL, grp = lane / QL;  // gather: z quad, row group
    const int c = lane % ZG, pr = lane / ZG;   // z pass: z group, row pair
    const bool vec = nz % 4 == 0 && ((uintptr_t)f & 15) == 0;
    const bool zin = 4 * q < nz;
    const float *A = g.att ? g.A + (size_t)ga * g.Lp * g.nya * g.nzs : nullptr;
    const int apos = 4 * ((q & 3) * g.zg + (q >> 2)), ns = strip_slabs(g);
    for (int s = strip_next(it, lane), sn; s >= 0; s = sn) {
        const int pl = it->plane_of[s];
        const int4 pi = it->plane[pl];
        const int xp = pi.w >> 4, y0 = pi.x + (s - pi.z) * RS, yl = pi.y;
        sn = strip_next(it, lane);
        if (A && sn >= 0) strip_prefetch<RS>(g, it, sn, A, lane);
        if (lane < RS) {  // the strip's sample positions, one lane per row
            RowTap t{};
            const int y = y0 + lane;
            if (y <= yl) {
                float ix, iy;
                rot_coords(th, g.lin[xp], g.lin[y], g.half, ix, iy);
                const Bilin b = bilin(ix, iy);
                const int r = b.r0 - g.pad, cc = b.c0 - g.pad;
                const bool r0 = (unsigned)r < (unsigned)N, r1 = (unsigned)(r + 1) < (unsigned)N;
                const bool c0 = (unsigned)cc < (unsigned)N, c1 = (unsigned)(cc + 1) < (unsigned)N;
                t.mask = (r0 && c0 ? 1 : 0) | (r0 && c1 ? 2 : 0) | (r1 && c0 ? 4 : 0) |
                         (r1 && c1 ? 8 : 0);
                t.off = (r * N + cc) * nz;
                t.nw = b.nw;
                t.ne = b.ne;
                t.sw = b.sw;
                t.se = b.se;
            }
            rt[lane] = t;
        }
        __syncwarp();
        const float *Ap = A ? A + ((size_t)xp * g.nya + (y0 - g.ya_lo)) * g.nzs + apos : nullptr;
        // four rows (two pairs) at a time: their loads are all in flight before the first sum
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            float4 v[4];
            const int row = 8 * grp + 4 * h;
            gather_rows(f, g, rt + row, q, zin, vec, Ap ? Ap + row * g.nzs : nullptr, v);
#pragma unroll
            for (int jp = 0; jp < 2; jp++) {
                float4 *d = reinterpret_cast<float4 *>(buf + (4 * grp + 2 * h + jp) * PS +
                                                       strip_at(4 * q + HB));
                const float4 a = v[2 * jp], c2 = v[2 * jp + 1];
                d[0] = make_float4(a.x, c2.x, a.y, c2.y);
                d[1] = make_float4(a.z, c2.z, a.w, c2.w);
            }
        }
        __syncwarp();
        const float *tap = taps + (xp - x0) * kStripTaps;
        const int y = y0 + 2 * pr;
        float *Wp = Ws + ((size_t)xp * ns * g.nya + (y - g.ya_lo)) * 32;
        ladder_dispatch(pi.w & 15, [&](auto kk) {
            constexpr int KK = decltype(kk)::value;
            if constexpr (KK / 2 <= HB) {
                float2 o[16];
                if (ONLY2D || g.psf2d)
                    strip_z_pass<KK, HB>(buf + pr * PS + 18 * c, tap, o);
                else
                    strip_z_copy<HB>(buf + pr * PS + 18 * c, o);
                __syncwarp();  // the buffer is free for the next strip
                if (c < g.zg) {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int pos = k * g.zg + c;
                        float *d = Wp + (size_t)(pos >> 3) * g.nya * 32 + 4 * (pos & 7);
                        if (y <= yl)
                            *reinterpret_cast<float4 *>(d) = make_float4(
                                o[4 * k].x, o[4 * k + 1].x, o[4 * k + 2].x, o[4 * k + 3].x);
                        if (y + 1 <= yl)
                            *reinterpret_cast<float4 *>(d + 32) = make_float4(
                                o[4 * k].y, o[4 * k + 1].y, o[4 * k + 2].y, o[4 * k + 3].y);
                    }
                }
            }
        });
    }
}

template <int QL, int HB, bool ONLY2D>
__global__ void __launch_bounds__(512, 1)
    k_fwd_strip(SpectDev g, const float *f, const int *__restrict__ alist,
                const int4 *__restrict__ items, float *__restrict__ W) {
    extern __shared__ __align__(128) float sm[];
    grid_release();
    const int4 item = items[blockIdx.x];
    fwd_strip_item<QL, HB, ONLY2D>(g, f, alist[item.x], item.y, item.z,
                           W + (size_t)item.x * g.Lp * g.nya * 32 * strip_slabs(g), sm);
}

// ONLY2D: every entry's PSF blurs z as well.
template <int HB, bool ONLY2D>
__global__ void __launch_bounds__(512, 1) k_fwd_strip_batch(const __grid_constant__ FwdBatch p) {
    extern __shared__ __align__(128) float sm[];
    __shared__ int s_item;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(p.counter, 1);
        __syncthreads();
        const int i = s_item;
        if (i >= p.n_items) return;
        const int4 item = p.items[i];  // (slot in group, first plane, end plane, entry)
        const SpectDev &g = p.g[item.w];
        const float *f = p.f[item.w];
        const int ga = p.alist[item.w][item.x];
        float *W = p.W[item.w] + (size_t)item.x * g.Lp * g.nya * 32 * strip_slabs(g);
        switch (strip_ql(g.nz)) {
            case 32: fwd_strip_item<32, HB, ONLY2D>(g, f, ga, item.y, item.z, W, sm); break;
            case 16: fwd_strip_item<16, HB, ONLY2D>(g, f, ga, item.y, item.z, W, sm); break;
            default: fwd_strip_item<8, HB, ONLY2D>(g, f, ga, item.y, item.z, W, sm); break;
        }
    }
}

// Second kernel: blur along y and sum over the planes of an item, for one slab (8 quad
// positions, 32 values of a row).  A warp owns 32 output rows (a lane 8 rows x 1 quad) and
// keeps their sums in registers over all planes.  One more warp brings the rows of a plane and
// slab, a contiguous piece, by one bulk copy into a ring of kYStages planes.  (Issued by one
// of the summing warps, the copies cost that warp 1,300 cycles a plane and held up the
// others.)  Rows outside the plane's range read as zero.
constexpr int kYStages = 2;
constexpr unsigned kDrainPolls = 65536;  // polls (20 us at most) for copies that were issued

struct YsumLayout {  // dynamic shared memory, in floats
    size_t item, taps, zero, total;
};
__host__ __device__ inline YsumLayout ysum_layout(const SpectDev &g) {
    YsumLayout L;
    L.item = (size_t)kYStages * g.nya * 32;
    L.taps = L.item + kPlaneTableBytes / sizeof(float);
    L.zero = L.taps + kStripTapFloats;
    L.total = L.zero + 32;
    return L;
}

// Ws: the slot's W rows; out: the item's partial ray sums [N][nz].  Whole-CTA call of at least
// nw + 1 warps, nw = ceil(N / 32).
__device__ __forceinline__ void ysum_item(const SpectDev &g, const float *Ws,
                                          const int ga, const int x0, const int x1,
                                          const int slab, float *__restrict__ out,
                                          float *__restrict__ sm, unsigned long long *full,
                                          unsigned long long *empty) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (g.N + 31) / 32;
    const YsumLayout L = ysum_layout(g);
    StripItem *it = reinterpret_cast<StripItem *>(sm + L.item);
    float *taps = sm + L.taps;
    if (threadIdx.x == 0)
        for (int s = 0; s < kYStages; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, nw);
        }
    strip_taps<0>(g, ga, x0, x1, taps);
    if (threadIdx.x < 32) sm[L.zero + threadIdx.x] = 0.f;
    if (warp == 0) strip_planes<0>(g.planes_fwd + (size_t)ga * g.Lp, x0, x1, it);
    cp_async_wait_all();
    grid_wait();
    __syncthreads();
    const int np = it->n_planes;
    if (warp >= nw) {
        if (warp > nw || lane != 0) return;
        // A stage is filled again only when every summing warp has left it, and a warp leaves a
        // stage only after its copy has landed: at most one copy per stage is in flight.
        unsigned issued[kYStages] = {};
        for (int n = 0; n < np; n++) {
            // (the test hook leaves the first copy out: the summing warps give up on it)
            if (n == 0 && g.dbg_skip_first_copy) continue;
            const int s = n % kYStages;
            if (n >= kYStages &&
                !mbar_wait_bounded(empty + s, (n / kYStages - 1) & 1, g.wait_polls)) {
                if (g.err) atomicExch(g.err, GB_ERR_WAIT_TIMEOUT);
                break;
            }
            const int4 pi = it->plane[n];
            const unsigned bytes = (unsigned)(pi.y - pi.x + 1) * 128u;
            mbar_arrive_expect_tx(full + s, bytes);
            tma_load_1d(sm + (size_t)s * g.nya * 32,
                        Ws + (((size_t)(pi.w >> 4) * strip_slabs(g) + slab) * g.nya +
                              (pi.x - g.ya_lo)) * 32,
                        bytes, full + s);
#pragma unroll
            for (int k = 0; k < kYStages; k++) issued[k] += k == s;
        }
        // no copy may be in flight when the CTA ends, not even after a wait that gave up: the
        // j-th copy of a stage completes phase j - 1 of its barrier
#pragma unroll
        for (int s = 0; s < kYStages; s++)
            if (issued[s]) mbar_wait_bounded(full + s, (issued[s] - 1) & 1, kDrainPolls);
        return;
    }
    const int q = lane & 7, o0 = 32 * warp + 8 * (lane >> 3);  // quad of the slab, first row
    const float *zero = sm + L.zero + 4 * q;
    float2 acc[8][2];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = make_float2(0.f, 0.f);
    for (int n = 0; n < np; n++) {
        const int s = n % kYStages;
        // A warp that gives up leaves for good, without a result and without releasing the
        // stage: the copying warp then gives up on the stage as well and drains.
        const bool ok = mbar_wait_bounded(full + s, (n / kYStages) & 1, g.wait_polls);
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0 && g.err) atomicExch(g.err, GB_ERR_WAIT_TIMEOUT);
            return;
        }
        const int4 pi = it->plane[n];
        const float *st = sm + (size_t)s * g.nya * 32 + 4 * q;
        const float *tap = taps + ((pi.w >> 4) - x0) * kStripTaps;
        ladder_dispatch(pi.w & 15, [&](auto kk) {
            constexpr int KK = decltype(kk)::value;
            // rows the warp's outputs reach: skip a plane that has none of them
            const int w0 = g.pad + 32 * warp - KK / 2;
            if (w0 > pi.y || w0 + 31 + KK - 1 < pi.x) return;
            const int lo = pi.x - (g.pad + o0 - KK / 2);  // first valid row of the window
            strip_y_pass<KK, true>(st - lo * 32, 32, tap, acc, lo, pi.y - pi.x + 1, zero);
        });
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + s);
    }
    const int pos = 8 * slab + q;
    if (pos >= 4 * g.zg) return;
    const int z = z_of_pos(g, pos), nz = g.nz;
    const bool vec = nz % 4 == 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (o0 + j >= g.N || z >= nz) continue;
        float *d = out + (size_t)(o0 + j) * nz + z;
        if (vec) {
            *reinterpret_cast<float4 *>(d) =
                make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
        } else {
            d[0] = acc[j][0].x;
            if (z + 1 < nz) d[1] = acc[j][0].y;
            if (z + 2 < nz) d[2] = acc[j][1].x;
            if (z + 3 < nz) d[3] = acc[j][1].y;
        }
    }
}

__global__ void __launch_bounds__(160, 4)
    k_fwd_ysum(SpectDev g, const int *__restrict__ alist, const int4 *__restrict__ items,
               const float *W, float *partials) {
    extern __shared__ __align__(128) float sm[];
    __shared__ unsigned long long full[kYStages], empty[kYStages];
    grid_release();
    const int4 item = items[blockIdx.x];
    ysum_item(g, W + (size_t)item.x * g.Lp * g.nya * 32 * strip_slabs(g), alist[item.x], item.y,
              item.z, blockIdx.y, partials + (size_t)blockIdx.x * g.N * g.nz, sm, full, empty);
}

__global__ void __launch_bounds__(160, 4) k_fwd_ysum_batch(const __grid_constant__ FwdBatch p) {
    extern __shared__ __align__(128) float sm[];
    __shared__ unsigned long long full[kYStages], empty[kYStages];
    const int4 item = p.yitems[blockIdx.x];
    const SpectDev &g = p.g[item.w];
    if (blockIdx.y >= strip_slabs(g)) return;
    ysum_item(g, p.W[item.w] + (size_t)item.x * g.Lp * g.nya * 32 * strip_slabs(g),
              p.alist[item.w][item.x], item.y, item.z, blockIdx.y,
              p.partials + (size_t)blockIdx.x * p.nz_max, sm, full, empty);
}

// ---------------------------------------------------------------- host side
static int strip_halo(const SpectDev &g) {
    return strip_hb(ladder_half(ladder_index(g.K / 2)));
}

void strip_configure(SpectDev &g, size_t cap) {
    g.strip = g.strip_fwd = 0;
    if (!g.psf || (g.att && !g.att_first) || g.N > 128 || g.nz > 128) return;
    const int QL = strip_ql(g.nz), HB = strip_halo(g);
    if (ysum_layout(g).total * sizeof(float) > cap) return;
    int b1 = 16, fw = 16;
    while (b1 && b1_strip_layout(g, QL, b1).total * sizeof(float) > cap) b1--;
    while (fw && fwd_strip_layout(QL, HB, fw).total * sizeof(float) > cap) fw--;
    if (b1 < 8 || fw < 8) return;
    g.strip = b1;
    g.strip_fwd = fw;
    g.zg = (g.nz + 15) / 16;
    g.nzs = 16 * g.zg;
}

#define GB_FOR_EACH_STRIP(X) X(32, 16) X(16, 16) X(8, 16) X(32, 24) X(16, 24) X(8, 24)

cudaError_t launch_fwd_strip(const SpectDev &g, const float *f, const int *alist,
                             const int4 *items, int n_items, const int4 *yitems, int n_yitems,
                             float *W, float *partials, cudaStream_t st) {
    const int QL = strip_ql(g.nz), HB = strip_halo(g);
    const size_t smem = fwd_strip_layout(QL, HB, g.strip_fwd).total * sizeof(float);
    cudaError_t e = cudaErrorInvalidValue;
#define GB_CASE(Q, B)                                                                        \
    if (QL == Q && HB == B)                                                                  \
        e = launch_dependent(g.psf2d ? k_fwd_strip<Q, B, true> : k_fwd_strip<Q, B, false>,   \
                             n_items, 32 * g.strip_fwd, smem, st, g, f, alist, items, W);
    GB_FOR_EACH_STRIP(GB_CASE)
#undef GB_CASE
    if (e != cudaSuccess) return e;
    return launch_dependent(k_fwd_ysum, dim3(n_yitems, strip_slabs(g)),
                            32 * ((g.N + 31) / 32 + 1), ysum_layout(g).total * sizeof(float), st, g,
                            alist, yitems, W, partials);
}

cudaError_t launch_b1_strip(const SpectDev &g, const float *proj, const int *alist,
                            const int4 *items, int n_items, float *W, cudaStream_t st) {
    const int QL = strip_ql(g.nz), HB = strip_halo(g), warps = g.strip;
    const size_t smem = b1_strip_layout(g, QL, warps).total * sizeof(float);
#define GB_CASE(Q, B)                                                                        \
    if (QL == Q && HB == B)                                                                  \
        return launch_dependent(g.psf2d ? k_b1_strip<Q, B, true> : k_b1_strip<Q, B, false>,  \
                                n_items, 32 * warps, smem, st, g, proj, alist, items, W);
    GB_FOR_EACH_STRIP(GB_CASE)
#undef GB_CASE
    return cudaErrorInvalidValue;
}

// The strip entries of a batch: those with g.strip > 0 (the others have no item here).
cudaError_t launch_fwd_strip_batch(const FwdBatch &p, int n, int grid, cudaStream_t st) {
    size_t smem = 0, ysmem = 0;
    int slabs = 1, rows = 1, HB = 16, warps = 16;
    bool only2d = true;
    for (int e = 0; e < n; e++)
        if (p.g[e].strip) warps = std::min(warps, p.g[e].strip_fwd);
    for (int e = 0; e < n; e++) {
        const SpectDev &g = p.g[e];
        if (!g.strip) continue;
        HB = strip_halo(g);
        only2d = only2d && g.psf2d;
        smem = std::max(smem, fwd_strip_layout(strip_ql(g.nz), HB, warps).total);
        ysmem = std::max(ysmem, ysum_layout(g).total);
        slabs = std::max(slabs, strip_slabs(g));
        rows = std::max(rows, g.N);
    }
    auto *fn = HB == 16 ? (only2d ? k_fwd_strip_batch<16, true> : k_fwd_strip_batch<16, false>)
                        : (only2d ? k_fwd_strip_batch<24, true> : k_fwd_strip_batch<24, false>);
    fn<<<grid, 32 * warps, smem * sizeof(float), st>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_fwd_ysum_batch<<<dim3(p.n_yitems, slabs), 32 * ((rows + 31) / 32 + 1),
                       ysmem * sizeof(float), st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_b1_strip_batch(const B1Batch &p, int n, int grid, cudaStream_t st) {
    int warps = 16, HB = 16;
    bool only2d = true;
    size_t smem = 0;
    for (int e = 0; e < n; e++)
        if (p.g[e].strip) warps = std::min(warps, p.g[e].strip);
    for (int e = 0; e < n; e++)
        if (p.g[e].strip) {
            smem = std::max(smem, b1_strip_layout(p.g[e], strip_ql(p.g[e].nz), warps).total);
            HB = strip_halo(p.g[e]);
            only2d = only2d && p.g[e].psf2d;
        }
    smem *= sizeof(float);
    auto *fn = HB == 16 ? (only2d ? k_b1_strip_batch<16, true> : k_b1_strip_batch<16, false>)
                        : (only2d ? k_b1_strip_batch<24, true> : k_b1_strip_batch<24, false>);
    fn<<<grid, 32 * warps, smem, st>>>(p);
    return cudaGetLastError();
}

cudaError_t setup_strip(size_t cap) {
    auto raise = [cap](const void *fn) {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    };
    cudaError_t e;
    for (const void *fn :
         {(const void *)k_b1_strip_batch<16, true>, (const void *)k_b1_strip_batch<24, true>,
          (const void *)k_b1_strip_batch<16, false>, (const void *)k_b1_strip_batch<24, false>,
          (const void *)k_fwd_strip_batch<16, true>, (const void *)k_fwd_strip_batch<24, true>,
          (const void *)k_fwd_strip_batch<16, false>, (const void *)k_fwd_strip_batch<24, false>,
          (const void *)k_fwd_ysum, (const void *)k_fwd_ysum_batch})
        if ((e = raise(fn)) != cudaSuccess) return e;
#define GB_CASE(Q, B)                                                        \
    if ((e = raise((const void *)k_b1_strip<Q, B, true>)) != cudaSuccess ||  \
        (e = raise((const void *)k_b1_strip<Q, B, false>)) != cudaSuccess || \
        (e = raise((const void *)k_fwd_strip<Q, B, true>)) != cudaSuccess || \
        (e = raise((const void *)k_fwd_strip<Q, B, false>)) != cudaSuccess)  \
        return e;
    GB_FOR_EACH_STRIP(GB_CASE)
#undef GB_CASE
    return cudaSuccess;
}

}  // namespace gb
