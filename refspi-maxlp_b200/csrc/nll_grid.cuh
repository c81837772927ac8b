// Dense part of the two differentiable likelihoods on the detector's grid
// (adjoint.cu, adjoint_emc.cu).
#pragma once
#include "rspi_common.cuh"

namespace {

constexpr double DG_PI = 3.14159265358979311599796346854;  // the double nearest pi

__device__ __forceinline__ void dg_sincos(float x, float *s, float *c) { sincosf(x, s, c); }
__device__ __forceinline__ void dg_sincos(double x, double *s, double *c) { sincos(x, s, c); }

// Dense part on the detector's grid, q = (x - c, y - c) / size: the sum over
// a ring of pixels of v s_d (|F + r_d|^2 + bg) and its gradients, with the
// reference amplitude r_d from tables (the MaxLP pixel NLL's dense part: v = 1,
// no bg; the slicing NLL's masked sum: v = vscale).  Its phase factors
// into a function of x and one of y, and its form factor depends on the
// radius only, so a CTA that takes DG_TILE pixels of neighbouring radii and
// DG_FRAMES frames at a time needs size + ~200 sines and cosines per frame
// instead of 2 per pixel (26,836 pixels of 185^2 have 2,365 radii).  The
// phases and the form factor's arguments are taken in FP64 and rounded once.
// A thread takes whole orbits of the quarter turn, (x, y), (-y, x), (-x, -y),
// (y, -x) about the centre: one radius, two phases and their conjugates, so
// five table reads and two complex products serve four pixels (one pixel per
// thread was bound by bank conflicts of its three reads: 1.08 ms for the
// value, 1.91 ms with gradients at the size below).  It keeps its pixels'
// gradient sums over all of the CTA's frames and the frames' sums over its
// orbits in FP64, the scale applied once per frame, and the warps transpose
// the latter as they reduce them: 1.5 instructions per pixel instead of 60.
// Bound by the conversions to FP64 (XU pipe 53% busy) and the orbits' chains at
// 128 registers (issue 54%).  Opposite pixels' values meet after they are
// widened, so every term is its pixel's own.
// Measured, value and gradients, against the kernels that take a sine pair per
// pixel: 26,836 pixels x 20,000 frames 1.28 ms (4.4), 24,928 x 5,000 0.31 ms
// (1.17), FP64 with 7,972 x 1,000 0.035 ms (0.10).
constexpr int DG_THREADS = 256;
constexpr int DG_FRAMES = 4;
constexpr long long DG_SMEM = 200 * 1024;   // most of the tables' shared memory
template <typename CT>
constexpr int DG_ORBITS = sizeof(CT) == 4 ? 2 : 1;   // orbits per thread

template <typename CT>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};

__device__ __forceinline__ void phase(double turns, float *s, float *c) {
    sincospif((float)(2. * (turns - rint(turns))), s, c);
}
__device__ __forceinline__ void phase(double turns, double *s, double *c) {
    sincospi(2. * (turns - rint(turns)), s, c);
}

// Sums 16 values over the warp: lane l gets that of value l / 2.
__device__ __forceinline__ double warp_sum16(double (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
        const bool up = (lane & (2 * n)) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(RSPI_FULL_MASK, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(RSPI_FULL_MASK, v[0], 1);
}

template <typename CT, bool GRAD>
__global__ void __launch_bounds__(DG_THREADS, 2)
k_nll_dense_grid(const double *__restrict__ fre, const double *__restrict__ fim, int fstride,
                 double v, double bg_sum, int size,
                 const int4 *__restrict__ order, const int *__restrict__ xy,
                 const int *__restrict__ rad_id, const double *__restrict__ rad_q, int tile_rads,
                 int n_orb, const double *__restrict__ dia, const double *__restrict__ sx,
                 const double *__restrict__ sy, const double *__restrict__ scale,
                 long long n_frames, long long frames_per_cta, bool zero_dia,
                 double *__restrict__ out, double *__restrict__ gfre,
                 double *__restrict__ gfim, double *__restrict__ gdia,
                 double *__restrict__ gsx, double *__restrict__ gsy,
                 double *__restrict__ gscale) {
    using CT2 = typename Pair<CT>::type;
    constexpr int ORB = DG_ORBITS<CT>;
    constexpr int TILE = DG_THREADS * ORB;
    extern __shared__ __align__(16) unsigned char dg_raw[];
    const int half = size / 2 + 1;                      // coordinates 0 .. size / 2
    CT2 *ex = reinterpret_cast<CT2 *>(dg_raw);          // [frame][|x - c|]
    CT2 *ey = ex + DG_FRAMES * half;                    // [frame][|y - c|]
    CT2 *rt = ey + DG_FRAMES * half;                    // [frame][radius]: ff, dff / ddia
    double *qt = reinterpret_cast<double *>(rt + DG_FRAMES * (tile_rads + 1));   // |x - c| / size
    __shared__ double red[DG_THREADS / 32][16];
    __shared__ int s_rad[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int p0 = blockIdx.x * TILE, p1 = min(n_orb, p0 + TILE);
    for (int x = tid; x < half; x += DG_THREADS) qt[x] = (double)x / (double)size;
    if (tid == 0) {
        s_rad[0] = 0x7fffffff;
        s_rad[1] = 0;
    }
    __syncthreads();
    CT f_r[ORB][4], f_i[ORB][4];
    int4 row[ORB];
    int at[ORB], rad[ORB];
    double gr[ORB][4], gi[ORB][4];
    int rlo = 0x7fffffff, rhi = 0;
#pragma unroll
    for (int k = 0; k < ORB; ++k) {
        const int i = p0 + k * DG_THREADS + tid;
        const bool live = i < p1;
        row[k] = live ? order[i] : make_int4(0, 0, 0, 0);
        const int m[4] = {row[k].x, row[k].y, row[k].z, row[k].w};
        at[k] = live ? xy[i] : 0;
        rad[k] = live ? rad_id[i] : -1;
        if (live) {
            rlo = min(rlo, rad[k]);
            rhi = max(rhi, rad[k]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            f_r[k][q] = live ? (CT)fre[(long long)m[q] * fstride] : (CT)0;
            f_i[k][q] = live ? (CT)fim[(long long)m[q] * fstride] : (CT)0;
            gr[k][q] = gi[k][q] = 0.;
        }
    }
    atomicMin(&s_rad[0], rlo);
    atomicMax(&s_rad[1], rhi);
    __syncthreads();
    const int r0 = s_rad[0], n_rad = min(s_rad[1] - r0 + 1, tile_rads);
    const int rstride = tile_rads + 1;                  // the last: no orbit, amplitude 0
#pragma unroll
    for (int k = 0; k < ORB; ++k) rad[k] = rad[k] < 0 ? tile_rads : min(rad[k] - r0, n_rad - 1);
    if (tid < DG_FRAMES) rt[tid * rstride + tile_rads] = CT2{(CT)0, (CT)0};
    double nll = 0.;
    const long long d_end = min(n_frames, ((long long)blockIdx.y + 1) * frames_per_cta);
    for (long long d0 = blockIdx.y * frames_per_cta; d0 < d_end; d0 += DG_FRAMES) {
        const int nf = (int)min((long long)DG_FRAMES, d_end - d0);
        __syncthreads();   // the last frames' tables have been read
        for (int i = tid; i < nf * half; i += DG_THREADS) {
            const int f = i / half, x = i - f * half;
            const double q = qt[x];
            CT s, c;
            phase(q * sx[d0 + f], &s, &c);
            ex[f * half + x] = CT2{c, s};
            phase(q * sy[d0 + f], &s, &c);
            ey[f * half + x] = CT2{c, s};
        }
        for (int i = tid; i < nf * n_rad; i += DG_THREADS) {
            const int f = i / n_rad, j = i - f * n_rad;
            const double pq = DG_PI * rad_q[r0 + j];
            CT x = (CT)(pq * dia[d0 + f]);
            // a frame without a sphere, as the slices take it (kernels.cu:66-67)
            const bool zero = zero_dia && x == (CT)0;
            if (zero) x = (CT)1.e-5;
            CT sn, cs;
            dg_sincos(x, &sn, &cs);
            const CT ix = (CT)1 / x;
            const CT ff = (sn - x * cs) * ix * ix * ix;
            const CT dff = zero ? (CT)0 : sn * ix * ix - (CT)3 * ff * ix;
            rt[f * rstride + j] = CT2{ff, dff * (CT)pq};
        }
        __syncthreads();
        double sum[16];
#pragma unroll
        for (int f = 0; f < DG_FRAMES; ++f) {
            double a64 = 0., d64 = 0., x64 = 0., y64 = 0.;
            if (f < nf) {
                const CT2 *exf = ex + f * half, *eyf = ey + f * half, *rtf = rt + f * rstride;
                const double s2 = 2. * v * scale[d0 + f];
#pragma unroll
                for (int k = 0; k < ORB; ++k) {
                    const int x = at[k] >> 16, y = at[k] & 0xffff;
                    const CT2 ux = exf[x], uy = exf[y], wx = eyf[x], wy = eyf[y];
                    const CT2 a = rtf[rad[k]];
                    // e^{i th} at (x, y) and (-y, x); conjugates at their opposites
                    const CT e0 = ux.x * wy.x - ux.y * wy.y, e1 = ux.x * wy.y + ux.y * wy.x;
                    const CT h0 = uy.x * wx.x + uy.y * wx.y, h1 = uy.x * wx.y - uy.y * wx.x;
                    const CT er = a.x * e0, ei = a.x * e1, hr = a.x * h0, hi = a.x * h1;
                    const CT z0 = f_r[k][0] + er, w0 = f_i[k][0] + ei;
                    const CT z1 = f_r[k][1] + hr, w1 = f_i[k][1] + hi;
                    const CT z2 = f_r[k][2] + er, w2 = f_i[k][2] - ei;
                    const CT z3 = f_r[k][3] + hr, w3 = f_i[k][3] - hi;
                    if (!GRAD) {
                        a64 += ((double)(z0 * z0 + w0 * w0) + (double)(z1 * z1 + w1 * w1)) +
                               ((double)(z2 * z2 + w2 * w2) + (double)(z3 * z3 + w3 * w3));
                    } else {
                        // the values are widened for the gradients anyway
                        auto sq = [](double r, double i, double t) {
                            return fma(r, r, fma(i, i, t));
                        };
                        a64 = sq(z0, w0, sq(z1, w1, sq(z2, w2, sq(z3, w3, a64))));
                        gr[k][0] = fma(s2, (double)z0, gr[k][0]);
                        gi[k][0] = fma(s2, (double)w0, gi[k][0]);
                        gr[k][1] = fma(s2, (double)z1, gr[k][1]);
                        gi[k][1] = fma(s2, (double)w1, gi[k][1]);
                        gr[k][2] = fma(s2, (double)z2, gr[k][2]);
                        gi[k][2] = fma(s2, (double)w2, gi[k][2]);
                        gr[k][3] = fma(s2, (double)z3, gr[k][3]);
                        gi[k][3] = fma(s2, (double)w3, gi[k][3]);
                        // z . e and z . (i e), the pixels widened before they meet
                        const double ap = (double)z0 + (double)z2, bp = (double)w0 - (double)w2;
                        const double aq = (double)z1 + (double)z3, bq = (double)w1 - (double)w3;
                        const double p0 = (double)e0, p1 = (double)e1;
                        const double q0 = (double)h0, q1 = (double)h1;
                        d64 = fma((double)a.y, fma(ap, p0, bp * p1) + fma(aq, q0, bq * q1), d64);
                        const double ff = (double)a.x;
                        const double cp = ff * fma(bp, p0, -ap * p1);
                        const double cq = ff * fma(bq, q0, -aq * q1);
                        x64 = fma((double)x, cp, fma(-(double)y, cq, x64));
                        y64 = fma((double)y, cp, fma((double)x, cq, y64));
                    }
                }
            }
            sum[4 * f] = a64;
            sum[4 * f + 1] = d64;
            sum[4 * f + 2] = x64;
            sum[4 * f + 3] = y64;
        }
        const double w = warp_sum16(sum);
        if ((lane & 1) == 0) red[wid][lane >> 1] = w;
        __syncthreads();
        if (tid < 4 * nf) {
            double t = 0.;
#pragma unroll
            for (int k = 0; k < DG_THREADS / 32; ++k) t += red[k][tid];
            const long long d = d0 + (tid >> 2);
            const double s = v * scale[d];
            const int what = tid & 3;
            if (what == 0) {
                if (blockIdx.x == 0) t += bg_sum;   // once per frame
                nll = fma(s, t, nll);
            }
            if (GRAD) {
                if (what == 0) atomicAdd(&gscale[d], v * t);
                if (what == 1) atomicAdd(&gdia[d], 2. * s * t);
                if (what == 2) atomicAdd(&gsx[d], 4. * DG_PI / (double)size * s * t);
                if (what == 3) atomicAdd(&gsy[d], 4. * DG_PI / (double)size * s * t);
            }
        }
    }
    if (wid == 0) {
        nll = warp_sum(nll);
        if (lane == 0) atomicAdd(out, nll);
    }
    if (GRAD) {
#pragma unroll
        for (int k = 0; k < ORB; ++k) {
            if (p0 + k * DG_THREADS + tid >= p1) continue;
            const int m[4] = {row[k].x, row[k].y, row[k].z, row[k].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                atomicAdd(&gfre[m[q]], gr[k][q]);
                atomicAdd(&gfim[m[q]], gi[k][q]);
            }
        }
    }
}

// The detector grid's tables of the dense part (null order: none).
struct GridTables {
    const int *order, *xy, *rad_id;
    const double *rad_q;
    int tile_rads;
};

int dense_grid_tile(int precision, long long size) {
    // a detector whose phase tables alone leave no room for the radii's
    if (size <= 1 || (precision == 1 ? 16LL : 8LL) * DG_FRAMES * (size + 2) > DG_SMEM / 2)
        return -1;
    return precision == 0 ? DG_THREADS * DG_ORBITS<float>
                          : precision == 1 ? DG_THREADS * DG_ORBITS<double> : -1;
}

// The tables describe whole orbits and fit the CTA's shared memory.
bool grid_tables_ok(int precision, long long size, long long n_pix, const int *order,
                    const int *xy, const int *rad_id, const double *rad_q, int tile_rads) {
    return n_pix <= 0x7fffffffLL && n_pix % 4 == 0 && size <= 0xffff && order && xy && rad_id &&
           rad_q && (reinterpret_cast<uintptr_t>(order) & 15) == 0 && tile_rads >= 1 &&
           tile_rads <= dense_grid_tile(precision, size) &&
           (precision == 1 ? 16LL : 8LL) * DG_FRAMES * (size + 2 + tile_rads + 1) <= DG_SMEM;
}

// out += sum_d v s_d (sum_pixels |F + r_d|^2 + bg_sum); F's parts lie fstride
// doubles apart.  zero_dia: the form factor of diameter 0 is the slices'
// (without: NaN, as the MaxLP pixels' reference amplitude gives).
template <typename CT, bool GRAD>
int launch_dense_grid(const GridTables &g, long long n_pix, int size, const double *fre,
                      const double *fim, int fstride, double v, double bg_sum, bool zero_dia,
                      const double *dia, const double *sx, const double *sy, const double *scale,
                      long long n_frames, double *out, double *gfre, double *gfim, double *gdia,
                      double *gsx, double *gsy, double *gscale, cudaStream_t stream) {
    if (n_pix == 0) return RSPI_OK;
    const size_t smem = sizeof(typename Pair<CT>::type) * DG_FRAMES *
                            (2 * (size_t)(size / 2 + 1) + (size_t)g.tile_rads + 1) +
                        sizeof(double) * (size_t)(size / 2 + 1);
    static RspiSmemOptIn optin;
    if (!rspi_smem_optin((const void *)k_nll_dense_grid<CT, GRAD>, smem, optin))
        return RSPI_ERR_CUDA;
    // about four waves of two CTAs per SM: a CTA's pixel gradients are added
    // to the result once, so fewer frame blocks mean fewer atomics
    const long long n_orb = n_pix / 4, tile = DG_THREADS * DG_ORBITS<CT>;
    const long long tiles = (n_orb + tile - 1) / tile;
    const long long want = max(1LL, 8LL * rspi_sm_count() / tiles);
    long long per = ((n_frames + want - 1) / want + DG_FRAMES - 1) / DG_FRAMES * DG_FRAMES;
    const dim3 grid((unsigned)tiles, (unsigned)((n_frames + per - 1) / per));
    k_nll_dense_grid<CT, GRAD><<<grid, DG_THREADS, smem, stream>>>(
        fre, fim, fstride, v, bg_sum, size, reinterpret_cast<const int4 *>(g.order), g.xy,
        g.rad_id, g.rad_q, g.tile_rads, (int)n_orb, dia, sx, sy, scale, n_frames, per, zero_dia,
        out, gfre, gfim, gdia, gsx, gsy, gscale);
    return RSPI_OK;
}

}  // namespace
