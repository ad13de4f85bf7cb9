// PET sinogram projectors (TOF and non-TOF Joseph, pet_joseph.cuh), the attenuation
// probability sinogram, and listmode -> sinogram binning.
//
// Reference: PETSinogramSystemMatrix (projectors/PET/pet_sinogram_system_matrix.py:12-296):
// the LOR of sinogram element (angle a, radial r, plane p) runs from
// (x1, y1, z1) = (det_xy[a][r][0], plane_z[p][0]) to (x2, y2, z2) = (det_xy[a][r][1],
// plane_z[p][1]) (_get_xyz_sinogram_coordinates, :50-85); subsets are angles i::n
// (:131-144).  TOF sinograms hold every bin of every LOR (bin fastest); one thread traces
// one (LOR, bin) restricted to that bin's TOF window, so the threads of a warp trace the
// bins of the same or neighbouring LORs.  That is the form for few ring pairs or many slices
// (line_pays) and for the rare LORs steeper than 45 degrees; every other LOR takes the line
// kernels (k_sino_fwd_line, k_sino_bwd_line), which use that all ring pairs of a transaxial line
// share its path.  The listmode binning restates
// listmode_to_sinogram / _listmodeTOF_to_sinogramTOF (io/PET/shared.py:175-272).
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "pet_joseph.cuh"

namespace gb {

struct SinoGeom {
    const float *det_xy;   // [A][R][2][2]
    const float *plane_z;  // [P][2]
    int A, R, P;
};

__device__ __forceinline__ void sino_lor(const SinoGeom &sg, int a, int r, int p, float *p0,
                                         float *p1) {
    const float4 xy = *reinterpret_cast<const float4 *>(sg.det_xy + ((size_t)a * sg.R + r) * 4);
    p0[0] = xy.x;
    p0[1] = xy.y;
    p0[2] = sg.plane_z[2 * p];
    p1[0] = xy.z;
    p1[1] = xy.w;
    p1[2] = sg.plane_z[2 * p + 1];
}

// proj [n_sel][R][P](x nb): element q -> (angle slot, r, p[, bin]); angle = first + slot * stride.
// atten: write exp(-sum) (attenuation probability) instead of the sum.
template <bool TOF>
__global__ void __launch_bounds__(256)
    k_sino_fwd(PetDev g, SinoGeom sg, int first, int stride, long long total, int nb,
               const float *__restrict__ img, float *__restrict__ proj, int atten) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const long long lor = TOF ? q / nb : q;
    const int bin = TOF ? (int)(q - lor * nb) : 0;
    const int p = (int)(lor % sg.P);
    const long long t = lor / sg.P;
    const int r = (int)(t % sg.R), slot = (int)(t / sg.R);
    float p0[3], p1[3];
    sino_lor(sg, first + slot * stride, r, p, p0, p1);
    const float v = joseph<false, TOF>(g, p0, p1, nullptr, img, g.tof_tab, bin - g.bin_shift, 0.f);
    proj[q] = atten ? expf(-v) : v;
}

template <bool TOF>
__global__ void __launch_bounds__(256)
    k_sino_bwd(PetDev g, SinoGeom sg, int first, int stride, long long total, int nb,
               const float *__restrict__ proj, float *__restrict__ img) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const float v = proj[q];
    if (v == 0.f) return;
    const long long lor = TOF ? q / nb : q;
    const int bin = TOF ? (int)(q - lor * nb) : 0;
    const int p = (int)(lor % sg.P);
    const long long t = lor / sg.P;
    const int r = (int)(t % sg.R), slot = (int)(t / sg.R);
    float p0[3], p1[3];
    sino_lor(sg, first + slot * stride, r, p, p0, p1);
    joseph<true, TOF>(g, p0, p1, img, nullptr, g.tof_tab, bin - g.bin_shift, v);
}

// ------------------------------------------------------------- line kernels
// The P ring pairs of a transaxial line (angle, radial) cross every plane of the principal
// axis at the same transverse position; only their z differ.  So a CTA takes one line:
//   forward  blends the two neighbouring image columns of every plane into shared memory once
//            and then interpolates each LOR in z alone (2 shared loads a plane instead of 4
//            global ones);
//   back     sums the LORs of the line into one z profile per plane in shared memory and adds
//            each profile to its two columns once.  A thread owns a plane, its profile is a
//            column of the shared array (bank = thread), so the sums need no atomics; the
//            global atomics fall from about 2.5 per LOR and plane to nz / 2 per plane and
//            line.  (Before: at the L2's atomic rate, 3.6e11 16-byte atomics/s.)
// Measured, 15 angles x 301 x 576 elements, 128 x 128 x 48 image, no TOF: back projection
// 1098 -> 204 us, forward 688 -> 242 us; 8 of these angles with 13 TOF bins: 4334 -> 1951 and
// 2974 -> 1240 us.  LORs whose principal axis is z are traced on their own (pet_joseph.cuh).
constexpr int kLineBatch = 64;     // LORs staged at a time by the back projection
constexpr int kLineStage = 96 * 1024;  // bytes of blended columns staged by the forward

struct Line {
    int k;              // principal axis of the line (0 or 1), -1: the end points coincide
    double ekd;         // |d| along it, exact
    float dx, dy, dk, pk;
    float t0, dt;       // plane parameter t(i) = t0 + i dt
    float f0, df;       // transverse coordinate (voxels)
    float vk;
    int i0, i1;         // planes between the end points and inside the image
    int nt, sk, st;     // transverse extent, strides of the principal and transverse axes
};

__device__ __forceinline__ Line sino_line(const PetDev &g, const SinoGeom &sg, int a, int r) {
    const float4 xy = *reinterpret_cast<const float4 *>(sg.det_xy + ((size_t)a * sg.R + r) * 4);
    Line l;
    l.dx = xy.z - xy.x;
    l.dy = xy.w - xy.y;
    const double ex = fabs((double)xy.z - (double)xy.x), ey = fabs((double)xy.w - (double)xy.y);
    l.k = ey > ex ? 1 : (ex > 0.0 ? 0 : -1);
    l.ekd = ey > ex ? ey : ex;
    const bool y = l.k == 1;
    l.dk = y ? l.dy : l.dx;
    l.pk = y ? xy.y : xy.x;
    const float pk1 = y ? xy.w : xy.z, ok = y ? g.org[1] : g.org[0];
    const float pt = y ? xy.x : xy.y, dt = y ? l.dx : l.dy, ot = y ? g.org[0] : g.org[1];
    l.vk = y ? g.vox[1] : g.vox[0];
    const float ivt = 1.f / (y ? g.vox[0] : g.vox[1]);
    const int nk = y ? g.n[1] : g.n[0];
    l.nt = y ? g.n[0] : g.n[1];
    const int nyz = g.n[1] * g.n[2];
    l.sk = y ? g.n[2] : nyz;
    l.st = y ? nyz : g.n[2];
    const float idk = 1.f / l.dk;
    l.t0 = (ok - l.pk) * idk;
    l.dt = l.vk * idk;
    l.f0 = (pt - ot + l.t0 * dt) * ivt;
    l.df = l.dt * dt * ivt;
    l.i0 = max((int)ceilf((fminf(l.pk, pk1) - ok) / l.vk), 0);
    l.i1 = min((int)floorf((fmaxf(l.pk, pk1) - ok) / l.vk), nk - 1);
    if (l.k < 0) l.i1 = l.i0 - 1;
    return l;
}

// z of ring pair p along the line: fz(i) = z0 + i dz in voxels; len, and whether the LOR
// belongs to the line (its principal axis is not z).
struct LineLor {
    float z0, dz, len;
    bool in;
};
__device__ __forceinline__ LineLor line_lor(const PetDev &g, const SinoGeom &sg, const Line &l,
                                            int p) {
    const float za = sg.plane_z[2 * p], zb = sg.plane_z[2 * p + 1], d = zb - za;
    const float ivz = 1.f / g.vox[2];
    LineLor o;
    o.in = l.k >= 0 && !(fabs((double)zb - (double)za) > l.ekd);  // as joseph() decides
    o.len = sqrtf(l.dx * l.dx + l.dy * l.dy + d * d);
    o.z0 = (za - g.org[2] + l.t0 * d) * ivz;
    o.dz = l.dt * d * ivz;
    return o;
}

// TOF weight at distance as (within the window) from the bin centre.
__device__ __forceinline__ float tof_w(const PetDev &g, const float *__restrict__ tab,
                                       float as) {
    const float t = as * g.tof_inv_step;
    const int m = min((int)t, kTofTab);
    return fmaf(t - (float)m, tab[m + 1] - tab[m], tab[m]);
}

// Grid (line = slot R + r, share of the ring pairs).  Elements of the line: proj[line P nb ..].
template <bool TOF>
__global__ void __launch_bounds__(256)
    k_sino_fwd_line(PetDev g, SinoGeom sg, int first, int stride, int nb, int chunk,
                    const float *__restrict__ img, float *__restrict__ proj, int atten) {
    extern __shared__ __align__(16) float sm[];
    const int line = blockIdx.x, a = first + (line / sg.R) * stride, r = line % sg.R;
    const Line l = sino_line(g, sg, a, r);
    const int nz = g.n[2], zs = nz + 2;  // one zero below and above each column
    float *tab = sm + ((size_t)chunk * zs + 3) / 4 * 4;
    if (TOF) copy_tof_table(g, tab);
    const int per = (sg.P + gridDim.y - 1) / gridDim.y;
    const int pa = blockIdx.y * per, pb = min(sg.P, pa + per);
    const int nq = (pb - pa) * nb;  // (ring pair, bin) elements of this CTA
    float *out = proj + ((size_t)line * sg.P + pa) * nb;
    for (int c0 = min(l.i0, l.i1 + 1);; c0 += chunk) {
        const int c1 = min(c0 + chunk, l.i1 + 1);  // planes of this round
        const bool firstc = c0 == min(l.i0, l.i1 + 1), lastc = c1 > l.i1;
        __syncthreads();
        for (int e = threadIdx.x; e < (c1 - c0) * zs; e += blockDim.x) {
            const int i = c0 + e / zs, z = e % zs - 1;
            const float f = fmaf((float)i, l.df, l.f0), fl = floorf(f);
            const int j = (int)fl;
            const float w = f - fl;
            const float *p = img + (size_t)i * l.sk + z;
            float v = 0.f;
            if ((unsigned)z < (unsigned)nz) {
                if ((unsigned)j < (unsigned)l.nt) v = (1.f - w) * __ldg(p + (ptrdiff_t)j * l.st);
                if ((unsigned)(j + 1) < (unsigned)l.nt)
                    v = fmaf(w, __ldg(p + (ptrdiff_t)(j + 1) * l.st), v);
            }
            sm[e] = v;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            const int p = pa + (TOF ? q / nb : q), bin = TOF ? q % nb : 0;
            const LineLor o = line_lor(g, sg, l, p);
            float v = 0.f;
            if (o.in) {
                int i0 = c0, i1 = c1 - 1;
                float s0 = 0.f, ds = 0.f, lim = 0.f, tc = 0.f;
                if (TOF) {
                    tc = (bin - g.bin_shift) * g.bw + g.co;
                    lim = g.nsig * g.sig + g.bw / 2;
                    s0 = (l.t0 - 0.5f) * o.len;
                    ds = l.dt * o.len;
                    // planes inside the window, with one plane of slack
                    const float ia = (tc - lim - s0) / ds, ib = (tc + lim - s0) / ds;
                    i0 = max(i0, (int)floorf(fminf(ia, ib)) - 1);
                    i1 = min(i1, (int)ceilf(fmaxf(ia, ib)) + 1);
                }
                float sum = 0.f;
#pragma unroll 4
                for (int i = i0; i <= i1; i++) {
                    const float fz = fmaf((float)i, o.dz, o.z0), fl = floorf(fz);
                    const int iz = (int)fl + 1;  // row of the lower corner
                    const float w = fz - fl;
                    if ((unsigned)iz <= (unsigned)nz) {
                        const float *c = sm + (size_t)(i - c0) * zs + iz;
                        const float u = fmaf(w, c[1], (1.f - w) * c[0]);
                        if (TOF) {
                            const float as = fabsf(fmaf((float)i, ds, s0) - tc);
                            if (as <= lim) sum = fmaf(u, tof_w(g, tab, as), sum);
                        } else {
                            sum += u;
                        }
                    }
                }
                v = sum * (l.vk * o.len / fabsf(l.dk));
            } else if (firstc) {  // principal axis z: traced on its own
                float p0[3], p1[3];
                sino_lor(sg, a, r, p, p0, p1);
                v = joseph<false, TOF>(g, p0, p1, nullptr, img, g.tof_tab, bin - g.bin_shift, 0.f);
            }
            if (!firstc) v += out[q];
            out[q] = lastc && atten ? expf(-v) : v;
        }
        if (lastc) break;
    }
}

// Grid (line, planes in chunks of blockDim.x, share of the ring pairs).
template <bool TOF>
__global__ void __launch_bounds__(128)
    k_sino_bwd_line(PetDev g, SinoGeom sg, int first, int stride, int nb,
                    const float *__restrict__ proj, float *__restrict__ img) {
    extern __shared__ __align__(16) float sm[];
    const int line = blockIdx.x, a = first + (line / sg.R) * stride, r = line % sg.R;
    const Line l = sino_line(g, sg, a, r);
    const int nz = g.n[2], T = blockDim.x, tid = threadIdx.x;
    const int per = (sg.P + gridDim.z - 1) / gridDim.z;
    const int pa = blockIdx.z * per, pb = min(sg.P, pa + per);
    const float *in = proj + ((size_t)line * sg.P) * nb;
    if (blockIdx.y == 0) {  // LORs whose principal axis is z: traced on their own
        for (int q = tid; q < (pb - pa) * nb; q += T) {
            const int p = pa + (TOF ? q / nb : q), bin = TOF ? q % nb : 0;
            if (line_lor(g, sg, l, p).in) continue;
            const float v = in[(size_t)p * nb + bin];
            float p0[3], p1[3];
            sino_lor(sg, a, r, p, p0, p1);
            if (v != 0.f) joseph<true, TOF>(g, p0, p1, img, nullptr, g.tof_tab, bin - g.bin_shift, v);
        }
    }
    const int b0 = max(l.i0, (int)(blockIdx.y * T));
    if (b0 > l.i1 || b0 >= (int)((blockIdx.y + 1) * T)) return;  // no plane in this chunk
    // profile of plane i: rows -1 .. nz (slices; one guard row below and above), column tid
    float *prof = sm;
    float4 *lor = reinterpret_cast<float4 *>(prof + ((size_t)(nz + 2) * T + 3) / 4 * 4);
    float *vals = reinterpret_cast<float *>(lor + kLineBatch);  // TOF: [kLineBatch][nb]
    float *tab = vals + kLineBatch * nb;
    for (int i = tid; i < (nz + 2) * T; i += T) prof[i] = 0.f;
    if (TOF) copy_tof_table(g, tab);
    const int i = blockIdx.y * T + tid;
    const float f = fmaf((float)i, l.df, l.f0), fl = floorf(f);
    const int j = (int)fl;
    const float wt = f - fl;
    const bool act = i >= l.i0 && i <= l.i1 && j >= -1 && j < l.nt;
    const float lim = g.nsig * g.sig + g.bw / 2, ibw = TOF ? 1.f / g.bw : 0.f;
    for (int p0 = pa; p0 < pb; p0 += kLineBatch) {
        const int n = min(kLineBatch, pb - p0);
        __syncthreads();
        for (int m = tid; m < n; m += T) {
            const LineLor o = line_lor(g, sg, l, p0 + m);
            const float cf = l.vk * o.len / fabsf(l.dk);
            // w: amplitude (no TOF), or the length, 0 where nothing is to add
            float w = 0.f;
            if (o.in) w = TOF ? o.len : cf * in[p0 + m];
            lor[m] = make_float4(o.z0, o.dz, w, cf);
        }
        if (TOF)
            for (int q = tid; q < n * nb; q += T) vals[q] = in[(size_t)p0 * nb + q];
        __syncthreads();
        if (!act) continue;
#pragma unroll 2
        for (int m = 0; m < n; m++) {
            const float4 o = lor[m];
            if (o.z == 0.f) continue;  // the same for the whole CTA
            float v = o.z;
            if (TOF) {
                // the bins whose window holds the plane, with one bin of slack
                const float s = fmaf((float)i, l.dt, l.t0 - 0.5f) * o.z;
                const float c = (s - g.co) * ibw + (float)g.bin_shift, h = lim * ibw;
                const int ba = max(0, (int)floorf(c - h)), bb = min(nb - 1, (int)ceilf(c + h));
                v = 0.f;
                for (int b = ba; b <= bb; b++) {
                    const float as = fabsf(s - ((b - g.bin_shift) * g.bw + g.co));
                    if (as <= lim) v = fmaf(vals[m * nb + b], tof_w(g, tab, as), v);
                }
                v *= o.w;
                if (v == 0.f) continue;
            }
            const float fz = fmaf((float)i, o.y, o.x), fzl = floorf(fz);
            const int iz = (int)fzl + 1;
            if ((unsigned)iz > (unsigned)nz) continue;
            const float wz = fz - fzl;
            float *c = prof + (size_t)iz * T + tid;
            const float a0 = fmaf(v, 1.f - wz, c[0]), a1 = fmaf(v, wz, c[T]);
            c[0] = a0;
            c[T] = a1;
        }
    }
    if (!act) return;
    const bool vec = nz % 4 == 0 && ((uintptr_t)img & 15) == 0;
    for (int u = 0; u < 2; u++) {
        const int jj = j + u;
        const float w = u ? wt : 1.f - wt;
        if ((unsigned)jj >= (unsigned)l.nt) continue;
        float *d = img + (size_t)i * l.sk + (size_t)jj * l.st;
        const float *c = prof + T + tid;
        if (vec) {
            for (int z = 0; z < nz; z += 4) {
                const float4 v = make_float4(w * c[z * T], w * c[(z + 1) * T], w * c[(z + 2) * T],
                                             w * c[(z + 3) * T]);
                if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f)
                    atomicAdd(reinterpret_cast<float4 *>(d + z), v);
            }
        } else {
            for (int z = 0; z < nz; z++) {
                const float v = w * c[z * T];
                if (v != 0.f) atomicAdd(d + z, v);
            }
        }
    }
}

// Listmode -> sinogram.  Per event: within-ring ids w = id % ncpr and rings id / ncpr,
// ordered by decreasing within-ring id (ties keep the event's order; a swap mirrors the
// TOF bin to nb - 1 - bin), sinogram bin (angular, radial) = lor_bins[w_hi][w_lo] and
// plane = plane_idx[ring_hi][ring_lo]; out-of-range bins are dropped.  normalization adds
// half a count at the mirrored pair (lor_bins[w_lo][w_hi], plane_idx[ring_lo][ring_hi]) and
// half at the ordered one.
__global__ void k_lm_to_sino(const int *__restrict__ ev, long long E, int ncol,
                             const float *__restrict__ w, const int *__restrict__ lor_bins,
                             const int *__restrict__ plane_idx, int ncpr, int nr, int A, int R,
                             int P, int nb, int normalization, float *__restrict__ sino) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const int id1 = ev[e * ncol], id2 = ev[e * ncol + 1];
    const int w1 = id1 % ncpr, w2 = id2 % ncpr, r1 = id1 / ncpr, r2 = id2 / ncpr;
    const bool sw = w2 > w1;
    const int wa = sw ? w2 : w1, wb = sw ? w1 : w2, ra = sw ? r2 : r1, rb = sw ? r1 : r2;
    int bin = 0;
    if (nb > 0) {
        bin = ev[e * ncol + 2];
        if (sw) bin = nb - 1 - bin;
        if (bin < 0 || bin >= nb) return;
    }
    const float val = w ? w[e] : 1.f;
    auto put = [&](int x, int y, int rx, int ry, float v) {
        if (x < 0 || x >= ncpr || y < 0 || y >= ncpr || rx < 0 || rx >= nr || ry < 0 || ry >= nr)
            return;
        const int ang = lor_bins[2 * (x * ncpr + y)], rad = lor_bins[2 * (x * ncpr + y) + 1];
        const int pl = plane_idx[rx * nr + ry];
        if (ang < 0 || ang >= A || rad < 0 || rad >= R || pl < 0 || pl >= P) return;
        size_t o = ((size_t)ang * R + rad) * P + pl;
        if (nb > 0) o = o * nb + bin;
        atomicAdd(sino + o, v);
    };
    if (normalization) {
        put(wa, wb, ra, rb, 0.5f * val);
        put(wb, wa, rb, ra, 0.5f * val);
    } else {
        put(wa, wb, ra, rb, val);
    }
}

}  // namespace gb

using namespace gb;

struct gb_pet_sino_plan {
    PetDev dev{};
    SinoGeom geom{};
    float *d_det = nullptr, *d_z = nullptr, *d_tof_tab = nullptr;
    int n_subsets = 1;
    int nb = 0;
};

// Shared memory of the line kernels, raised once per process and device context.
static size_t bwd_line_smem(int nz, int T, int nb, bool tof) {
    return sizeof(float) * (((size_t)(nz + 2) * T + 3) / 4 * 4 + 4 * kLineBatch +
                            (tof ? kLineBatch * nb + kTofTabLen : 0));
}
static int fwd_line_chunk(const PetDev &g) {  // planes staged at a time
    const int nk = std::max(g.n[0], g.n[1]), zs = g.n[2] + 2;
    return std::max(1, std::min(nk, (int)(kLineStage / (sizeof(float) * zs))));
}
static size_t fwd_line_smem(const PetDev &g, bool tof) {
    return sizeof(float) * (((size_t)fwd_line_chunk(g) * (g.n[2] + 2) + 3) / 4 * 4 +
                            (tof ? kTofTabLen : 0));
}
static int bwd_line_threads(const PetDev &g) {
    const int nk = std::max(g.n[0], g.n[1]);
    return nk <= 32 ? 32 : nk <= 64 ? 64 : nk <= 96 ? 96 : 128;
}
// The line kernels' tiles must fit: the back projection's profiles of 128 planes (446 slices
// without TOF, 407 with 13 bins).
static bool line_fits(const PetDev &g, int nb, bool tof) {
    return bwd_line_smem(g.n[2], 128, nb, tof) <= 225 * 1024 && fwd_line_smem(g, tof) <= 225 * 1024;
}
// Planes that the LORs of a line add up, as multiples of the planes of the image.
static double line_work(const PetDev &g, int P, int nb, bool tof) {
    if (!tof) return P;
    const double nk = std::max(g.n[0], g.n[1]);
    const double win = (2.0 * (g.nsig * g.sig) + g.bw) / std::min(g.vox[0], g.vox[1]);
    return (double)P * nb * std::min(win, nk) / nk;
}
// Blocks of an SM by their shared memory (228 KB, 1 KB of it reserved for each).
static int sm_blocks(size_t smem) { return (int)(228 * 1024 / (smem + 1024)); }

// Whether the line kernels pay: they blend (forward) or clear and add (back) nz values per plane
// and line whatever the number P of ring pairs is, and their tiles leave few blocks to an SM
// when nz is large; tracing each LOR costs the same for any nz.  Measured, traced -> line, us
// (4515 lines, 128 x 128 x nz of 4 mm, 13 TOF bins over 650 mm, FWHM 58.5 mm):
//   nz               8            24           48           100            200            380
//   forward    P=16  43 -> 41     43 -> 56     43 -> 85     43 -> 197      43 -> 560      43 -> 996
//              P=64  105 -> 45    106 -> 60    105 -> 88    105 -> 199     106 -> 562     105 -> 1002
//              P=144 197 -> 75    198 -> 86                 199 -> 191     198 -> 499     199 -> 868
//   TOF        P=4   60 -> 55     61 -> 76     64 -> 112    62 -> 247      62 -> 579      62 -> 1076
//              P=16  189 -> 110   189 -> 126   192 -> 150   190 -> 204     190 -> 422     190 -> 754
//              P=64  704 -> 322   705 -> 338   713 -> 363   710 -> 417     709 -> 744     711 -> 1238
//              P=144                                                       1612 -> 1410   1602 -> 2245
//   back       P=1   39 -> 24     40 -> 25     39 -> 28     39 -> 42       40 -> 86       42 -> 213
//              P=16  102 -> 27    100 -> 29    96 -> 31     80 -> 49       95 -> 96       83 -> 236
//              P=144 348 -> 61    386 -> 65                 357 -> 109     350 -> 205     348 -> 449
//   TOF        P=1   49 -> 29     48 -> 35     47 -> 43     33 -> 62       47 -> 168      35 -> 241
//              P=16  214 -> 65    197 -> 76    197 -> 97    174 -> 131     190 -> 357     176 -> 434
//              P=64  683 -> 191   634 -> 218   634 -> 282   639 -> 366     606 -> 1004    647 -> 1133
// A forward of more slices than are staged at once re-reads its sums: 908 -> 946 us at 200 slices
// and P=784 without TOF; with TOF 3635 -> 2676 at 200 slices, 3619 -> 4160 at 380 (P=324).
static bool line_pays(const PetDev &g, int P, int nb, bool tof, bool back) {
    if (!line_fits(g, nb, tof)) return false;
    const int nk = std::max(g.n[0], g.n[1]), nz = g.n[2];
    const double work = line_work(g, P, nb, tof);
    if (back) {
        const int T = bwd_line_threads(g);
        const int warps = sm_blocks(bwd_line_smem(nz, T, nb, tof)) * T / 32;
        return tof ? warps >= (T >= 96 ? 8 : 10) && work >= nz - 70
                   : warps >= 8 && 8 * work >= nz - 64;
    }
    const size_t all = sizeof(float) * nk * ((size_t)nz + 2);
    if (all > (tof ? 165 * 1024 : kLineStage)) return false;
    if (tof && (long long)P * nb < 48) return false;  // (the 16 KB weight table of a block)
    const int blocks = sm_blocks(fwd_line_smem(g, tof));
    const double per_slice = tof ? (blocks >= 3 ? 1.2 : 3.1)
                                 : (blocks >= 7 ? 1.2 : blocks >= 4 ? 1.6 : 4.0);
    return work >= per_slice * (nz + 4);
}
static cudaError_t setup_lines() {
    cudaError_t e;
    int dev = 0, cap = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (const void *fn : {(const void *)k_sino_fwd_line<false>, (const void *)k_sino_fwd_line<true>,
                           (const void *)k_sino_bwd_line<false>, (const void *)k_sino_bwd_line<true>})
        if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, cap)) !=
            cudaSuccess)
            return e;
    return cudaSuccess;
}
// Shares of the ring pairs of a line: enough CTAs for four to an SM.
static int line_split(int lines, int P) {
    return std::max(1, std::min({(4 * device_sm_count() + lines - 1) / lines,
                                 (P + kLineBatch - 1) / kLineBatch, 65535}));
}

// Forward projection of `n` angles (atten: exp(-sum)).
static cudaError_t sino_forward(gb_pet_sino_plan *p, const float *img, float *proj, int first,
                                int stride, int n, bool tof, int atten, cudaStream_t st) {
    const int nb = tof ? p->nb : 1;
    const int lines = n * p->geom.R;
    if (line_pays(p->dev, p->geom.P, nb, tof, false)) {
        const dim3 grid(lines, line_split(lines, p->geom.P));
        const size_t smem = fwd_line_smem(p->dev, tof);
        const int chunk = fwd_line_chunk(p->dev);
        // the block size that leaves the fewest threads without an element
        const int elems = (p->geom.P + (int)grid.y - 1) / (int)grid.y * nb;
        int T = 256;
        for (int t : {224, 192, 160, 128})
            if ((elems + t - 1) / t * t < (elems + T - 1) / T * T) T = t;
        if (tof)
            k_sino_fwd_line<true><<<grid, T, smem, st>>>(p->dev, p->geom, first, stride, nb,
                                                           chunk, img, proj, atten);
        else
            k_sino_fwd_line<false><<<grid, T, smem, st>>>(p->dev, p->geom, first, stride, nb,
                                                            chunk, img, proj, atten);
        return cudaGetLastError();
    }
    const long long total = (long long)lines * p->geom.P * nb;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (tof)
        k_sino_fwd<true><<<blocks, 256, 0, st>>>(p->dev, p->geom, first, stride, total, nb, img,
                                                 proj, atten);
    else
        k_sino_fwd<false><<<blocks, 256, 0, st>>>(p->dev, p->geom, first, stride, total, 1, img,
                                                  proj, atten);
    return cudaGetLastError();
}

static void sino_free(gb_pet_sino_plan *p) {
    if (!p) return;
    dev_free(p->d_det);
    dev_free(p->d_z);
    dev_free(p->d_tof_tab);
    delete p;
}

static void sino_range(const gb_pet_sino_plan *p, int subset, int &first, int &stride, int &n) {
    if (subset < 0) {
        first = 0;
        stride = 1;
        n = p->geom.A;
    } else {
        first = subset;
        stride = p->n_subsets;
        n = p->geom.A > subset ? (p->geom.A - subset + p->n_subsets - 1) / p->n_subsets : 0;
    }
}

extern "C" {

gb_status gb_pet_sino_plan_create(const gb_pet_sino_desc *d, gb_pet_sino_plan **out) {
    clear_error();
    GB_CHECK_ARG(d && out, "null argument");
    *out = nullptr;
    GB_CHECK_ARG(d->nx > 0 && d->ny > 0 && d->nz > 0, "image shape must be positive");
    GB_CHECK_ARG(d->n_angles > 0 && d->n_radial > 0 && d->n_planes > 0,
                 "sinogram shape must be positive");
    GB_CHECK_ARG(d->det_xy && d->plane_z, "sinogram geometry tables missing");
    GB_CHECK_ARG(!d->tof || (d->tof_sigma > 0 && d->tof_bin_width > 0 && d->tof_num_bins > 0),
                 "invalid TOF parameters");
    auto *p = new gb_pet_sino_plan();
    PetDev &g = p->dev;
    g.n[0] = d->nx; g.n[1] = d->ny; g.n[2] = d->nz;
    g.n_vox = d->nx * d->ny * d->nz;
    g.vox[0] = d->vx; g.vox[1] = d->vy; g.vox[2] = d->vz;
    g.org[0] = d->ox; g.org[1] = d->oy; g.org[2] = d->oz;
    g.tof = d->tof;
    g.bw = d->tof_bin_width;
    g.sig = d->tof_sigma;
    g.co = d->tof_center_offset;
    g.nsig = d->tof_n_sigmas;
    g.bin_shift = (d->tof_num_bins - 1) / 2;
    p->nb = d->tof ? d->tof_num_bins : 0;
    p->geom.A = d->n_angles;
    p->geom.R = d->n_radial;
    p->geom.P = d->n_planes;
    const size_t ndet = (size_t)d->n_angles * d->n_radial * 4, nz2 = (size_t)d->n_planes * 2;
    cudaError_t e;
    if ((e = dev_alloc(&p->d_det, ndet * sizeof(float))) != cudaSuccess ||
        (e = cudaMemcpy(p->d_det, d->det_xy, ndet * sizeof(float), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (e = dev_alloc(&p->d_z, nz2 * sizeof(float))) != cudaSuccess ||
        (e = cudaMemcpy(p->d_z, d->plane_z, nz2 * sizeof(float), cudaMemcpyHostToDevice)) !=
            cudaSuccess) {
        set_error("sinogram table upload failed: %s", cudaGetErrorString(e));
        sino_free(p);
        return e == cudaErrorMemoryAllocation ? GB_ERR_OOM : GB_ERR_CUDA;
    }
    p->geom.det_xy = p->d_det;
    p->geom.plane_z = p->d_z;
    if (d->tof) {
        std::vector<float> tab;
        float inv_step = 0.f;
        tof_weight_table(d->tof_bin_width, d->tof_sigma, d->tof_n_sigmas, tab, inv_step);
        if ((e = dev_alloc(&p->d_tof_tab, tab.size() * sizeof(float))) != cudaSuccess ||
            (e = cudaMemcpy(p->d_tof_tab, tab.data(), tab.size() * sizeof(float),
                            cudaMemcpyHostToDevice)) != cudaSuccess) {
            set_error("TOF table upload failed: %s", cudaGetErrorString(e));
            sino_free(p);
            return GB_ERR_CUDA;
        }
        g.tof_tab = p->d_tof_tab;
        g.tof_inv_step = inv_step;
    }
    if ((e = setup_lines()) != cudaSuccess) {
        set_error("shared-memory setup failed: %s", cudaGetErrorString(e));
        sino_free(p);
        return GB_ERR_CUDA;
    }
    *out = p;
    return GB_OK;
}

gb_status gb_pet_sino_plan_destroy(gb_pet_sino_plan *p) {
    clear_error();
    if (p) {
        cudaDeviceSynchronize();
        sino_free(p);
    }
    return GB_OK;
}

gb_status gb_pet_sino_set_subsets(gb_pet_sino_plan *p, int32_t n_subsets) {
    clear_error();
    GB_CHECK_ARG(p && n_subsets >= 1 && n_subsets <= p->geom.A, "n_subsets must be in [1, %d]",
                 p ? p->geom.A : 0);
    p->n_subsets = n_subsets;
    return GB_OK;
}

int32_t gb_pet_sino_subset_size(const gb_pet_sino_plan *p, int32_t subset) {
    if (!p || subset >= p->n_subsets) return -1;
    int first, stride, n;
    sino_range(p, subset, first, stride, n);
    return n;
}

gb_status gb_pet_sino_forward(gb_pet_sino_plan *p, const float *img, float *proj, int32_t subset,
                              int32_t use_tof, gb_stream_t stream) {
    clear_error();
    GB_CHECK_ARG(p && img && proj, "null argument");
    GB_CHECK_ARG(subset < p->n_subsets, "subset out of range");
    int first, stride, n;
    sino_range(p, subset, first, stride, n);
    const bool tof = use_tof && p->nb > 0;
    if (n == 0) return GB_OK;
    GB_CUDA(sino_forward(p, img, proj, first, stride, n, tof, 0, as_stream(stream)));
    return GB_OK;
}

gb_status gb_pet_sino_backward(gb_pet_sino_plan *p, const float *proj, float *img,
                               int32_t subset, int32_t use_tof, gb_stream_t stream) {
    clear_error();
    GB_CHECK_ARG(p && img && proj, "null argument");
    GB_CHECK_ARG(((uintptr_t)img & 15) == 0, "image buffer must be 16-byte aligned");
    GB_CHECK_ARG(subset < p->n_subsets, "subset out of range");
    int first, stride, n;
    sino_range(p, subset, first, stride, n);
    const bool tof = use_tof && p->nb > 0;
    const long long total = (long long)n * p->geom.R * p->geom.P * (tof ? p->nb : 1);
    cudaStream_t st = as_stream(stream);
    GB_CUDA(cudaMemsetAsync(img, 0,
                            (size_t)p->dev.n[0] * p->dev.n[1] * p->dev.n[2] * sizeof(float), st));
    if (total == 0) return GB_OK;
    const int nb = tof ? p->nb : 1;
    if (line_pays(p->dev, p->geom.P, nb, tof, true)) {
        const int nk = std::max(p->dev.n[0], p->dev.n[1]), T = bwd_line_threads(p->dev);
        const int chunks = (nk + T - 1) / T, lines = n * p->geom.R;
        const dim3 grid(lines, chunks, line_split(lines * chunks, p->geom.P));
        const size_t smem = bwd_line_smem(p->dev.n[2], T, nb, tof);
        if (tof)
            k_sino_bwd_line<true><<<grid, T, smem, st>>>(p->dev, p->geom, first, stride, nb, proj,
                                                         img);
        else
            k_sino_bwd_line<false><<<grid, T, smem, st>>>(p->dev, p->geom, first, stride, nb,
                                                          proj, img);
        GB_LAUNCH_CHECK();
        return GB_OK;
    }
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (tof)
        k_sino_bwd<true><<<blocks, 256, 0, st>>>(p->dev, p->geom, first, stride, total, p->nb,
                                                 proj, img);
    else
        k_sino_bwd<false><<<blocks, 256, 0, st>>>(p->dev, p->geom, first, stride, total, 1, proj,
                                                  img);
    GB_LAUNCH_CHECK();
    return GB_OK;
}

gb_status gb_pet_sino_atten(gb_pet_sino_plan *p, const float *mu, float *prob, int32_t subset,
                            gb_stream_t stream) {
    clear_error();
    GB_CHECK_ARG(p && mu && prob, "null argument");
    GB_CHECK_ARG(subset < p->n_subsets, "subset out of range");
    int first, stride, n;
    sino_range(p, subset, first, stride, n);
    if (n == 0) return GB_OK;
    GB_CUDA(sino_forward(p, mu, prob, first, stride, n, false, 1, as_stream(stream)));
    return GB_OK;
}

gb_status gb_pet_lm_to_sino(const int32_t *events, int64_t n_events, int32_t ncol,
                            const float *weights, const int32_t *lor_bins,
                            const int32_t *plane_index, int32_t n_crystals_per_ring,
                            int32_t n_rings, int32_t n_angles, int32_t n_radial,
                            int32_t n_planes, int32_t tof_num_bins, int32_t normalization,
                            float *sino, gb_stream_t stream) {
    clear_error();
    GB_CHECK_ARG(sino && lor_bins && plane_index, "null argument");
    GB_CHECK_ARG(n_events >= 0 && (n_events == 0 || events), "events missing");
    GB_CHECK_ARG(ncol == 2 || ncol == 3, "events need 2 or 3 columns");
    GB_CHECK_ARG(tof_num_bins == 0 || ncol == 3, "TOF binning needs a TOF bin column");
    GB_CHECK_ARG(n_crystals_per_ring > 0 && n_rings > 0 && n_angles > 0 && n_radial > 0 &&
                     n_planes > 0,
                 "sinogram geometry must be positive");
    cudaStream_t st = as_stream(stream);
    const size_t n_out = (size_t)n_angles * n_radial * n_planes * std::max(1, (int)tof_num_bins);
    GB_CUDA(cudaMemsetAsync(sino, 0, n_out * sizeof(float), st));
    if (n_events == 0) return GB_OK;
    k_lm_to_sino<<<(unsigned)((n_events + 255) / 256), 256, 0, st>>>(
        events, n_events, ncol, weights, lor_bins, plane_index, n_crystals_per_ring, n_rings,
        n_angles, n_radial, n_planes, tof_num_bins, normalization, sino);
    GB_LAUNCH_CHECK();
    return GB_OK;
}

}  // extern "C"
