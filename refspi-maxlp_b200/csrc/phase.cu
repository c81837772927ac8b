// Model refinement after the pattern search: error reduction and the
// difference map (maxLP.py:271-298, 342-354), on the device.
//
// The reference transforms with NumPy's centred convention
// fftshift(fftn(ifftshift(x))) and its inverse.  For a line of n values and
// c = n / 2 that is, with j and k counted from the centre,
//     y[k] = sum_j x[j] * exp(s * 2 pi i j k / n),  s = -1 (+1 and a factor
//     1/n for the inverse).
// The lines are transformed directly in FP64: image sides are at most a few
// hundred pixels and any number, often with a large prime factor.  Opposite
// inputs and outputs share their cosines and sines,
//     y[+-k] = x[0] + sum_{j>0} (x[j] + x[-j]) cos(2 pi j k / n)
//                   +- s i (x[j] - x[-j]) sin(2 pi j k / n),
// four real products per (j, k) > 0 for four complex ones, from one n-entry
// table whose index j k mod n is kept exactly in integers.
// The refinement alternates two kernels on lines held in shared memory.  The
// row kernel transforms the rows forward, finishes the step there (the
// difference map's combination, the Fourier projection of the next step) and
// transforms them back; the column kernel transforms the columns back,
// applies the real-space projection and transforms them forward, real values
// between the two.  So a step is two launches instead of five and an image is
// read and written twice instead of ten times.  What bounds it: the shared
// memory's table reads (~10 wavefronts per warp and term) and the launches.
// Measured at 185^2, 15 steps with the support: 0.34 ms on the GPU, 1.04 ms
// with a pass per axis and a thread per output (256 threads, two lines and two
// threads per output pair; one line 0.39, four threads 0.36, four lines 0.52).
//
// Support (maxLP.py:292-298): fconv tapered by expit((mrad - 12) / 2), the
// centred inverse transform, |real part| smoothed by a Gaussian (sigma 3,
// radius 12 = int(4 sigma + 0.5), 'reflect' edges: d c b a | a b c d, axis 0
// then axis 1, the symmetric-kernel order w0 x0 + sum over k = radius..1 of
// wk (x-k + x+k)), then
// thresholded: minvsupp = !(smoothed > 1.2e-4).
#include "rspi_common.cuh"

namespace {

constexpr int MAX_N = 1024;          // longest line a CTA transforms
constexpr int MAX_RADIUS = 64;       // longest Gaussian half-width
constexpr int DFT_THREADS = 256;
constexpr int DFT_SPLIT = 2;         // threads per output pair
constexpr int DFT_LINES = 2;         // lines per CTA: they share the table reads
static_assert(DFT_SPLIT >= DFT_LINES, "a thread of an output pair finishes each line");

// Shared memory of a CTA: the table, and per line its values and results.
__device__ __forceinline__ double2 *dft_lines(double2 *smem, int n, int which) {
    return smem + n * (1 + which * DFT_LINES);
}
size_t dft_smem(long long n) { return sizeof(double2) * (size_t)n * (1 + 2 * DFT_LINES); }

__device__ __forceinline__ void dft_table(double2 *tw, int n) {
    for (int m = threadIdx.x; m < n; m += DFT_THREADS) {
        double s, c;
        sincospi(2.0 * (double)m / (double)n, &s, &c);
        tw[m] = make_double2(c, s);
    }
}

// The centred transform of DFT_LINES lines of n values, in (destroyed) to
// out, both [line][n] in shared memory, times scale.  REAL_IN: the inputs'
// imaginary parts are zero.  REAL_OUT: only the real parts are wanted (the
// imaginary parts are stored as zero).  Ends with a barrier.
template <bool REAL_IN, bool REAL_OUT>
__device__ void dft(const double2 *__restrict__ tw, double2 *in, double2 *out, int n, double sign,
                    double scale) {
    const int c = n / 2, h = (n - 1) / 2;   // pairs (j, -j), j = 1 .. h
    // sums and differences of opposite values in their places
    for (int t = threadIdx.x; t < DFT_LINES * h; t += DFT_THREADS) {
        double2 *x = in + (t / h) * n + c;
        const int j = t % h + 1;
        const double2 p = x[j], q = x[-j];
        x[j] = make_double2(p.x + q.x, p.y + q.y);
        x[-j] = make_double2(p.x - q.x, p.y - q.y);
    }
    __syncthreads();
    const int part = threadIdx.x % DFT_SPLIT;
    const int n_k = n / 2 + 1;              // outputs k = 0 .. c (odd n: c = h)
    for (int k0 = 0; k0 < n_k; k0 += DFT_THREADS / DFT_SPLIT) {
        const int k = k0 + threadIdx.x / DFT_SPLIT;
        double cr[DFT_LINES], ci[DFT_LINES], sr[DFT_LINES], si[DFT_LINES];
#pragma unroll
        for (int l = 0; l < DFT_LINES; ++l) cr[l] = ci[l] = sr[l] = si[l] = 0.;
        if (k < n_k) {
            const int step = (DFT_SPLIT * k) % n;
            int m = ((part + 1) * k) % n;
#pragma unroll 4
            for (int j = part + 1; j <= h; j += DFT_SPLIT) {
                const double2 w = tw[m];
#pragma unroll
                for (int l = 0; l < DFT_LINES; ++l) {
                    const double2 a = in[l * n + c + j], b = in[l * n + c - j];
                    cr[l] = fma(a.x, w.x, cr[l]);
                    if (!REAL_IN) si[l] = fma(b.y, w.y, si[l]);
                    if (!REAL_OUT) {
                        if (!REAL_IN) ci[l] = fma(a.y, w.x, ci[l]);
                        sr[l] = fma(b.x, w.y, sr[l]);
                    }
                }
                m += step;
                if (m >= n) m -= n;
            }
        }
#pragma unroll
        for (int l = 0; l < DFT_LINES; ++l)
#pragma unroll
            for (int o = 1; o < DFT_SPLIT; o <<= 1) {
                cr[l] += __shfl_xor_sync(RSPI_FULL_MASK, cr[l], o);
                ci[l] += __shfl_xor_sync(RSPI_FULL_MASK, ci[l], o);
                sr[l] += __shfl_xor_sync(RSPI_FULL_MASK, sr[l], o);
                si[l] += __shfl_xor_sync(RSPI_FULL_MASK, si[l], o);
            }
        if (k < n_k && part < DFT_LINES) {
#pragma unroll
            for (int l = 0; l < DFT_LINES; ++l) {
                if (l != part) continue;
                const double2 x0 = in[l * n + c];
                double xr = x0.x + cr[l], xi = x0.y + ci[l];
                if (n % 2 == 0) {           // the unpaired j = -c: (-1)^k
                    const double2 e = in[l * n];
                    xr += k & 1 ? -e.x : e.x;
                    xi += k & 1 ? -e.y : e.y;
                }
                const double ur = sign * si[l], ui = sign * sr[l];
                double2 *y = out + l * n + c;
                // k = c of an even n is the output -c, where the sines vanish
                if (n % 2 == 1 || k < c)
                    y[k] = make_double2((xr - ur) * scale, REAL_OUT ? 0. : (xi + ui) * scale);
                if (k > 0) y[-k] = make_double2((xr + ur) * scale, REAL_OUT ? 0. : (xi - ui) * scale);
            }
        }
    }
    __syncthreads();
}

enum Epilogue : int {
    EP_STORE = 0,        // y
    EP_ABS_REAL = 1,     // |re y| into a real array
};

// One pass of the n x n complex image along axis 1 (rows) or 0 (columns).
template <int EP>
__global__ void __launch_bounds__(DFT_THREADS)
k_cdft_lines(const double2 *__restrict__ in, double2 *__restrict__ out, int n, int axis,
             double sign, double scale, double *__restrict__ out_re) {
    extern __shared__ __align__(16) double2 ph_smem[];
    double2 *a = dft_lines(ph_smem, n, 0), *b = dft_lines(ph_smem, n, 1);
    const int l0 = blockIdx.x * DFT_LINES, nl = min(DFT_LINES, n - l0);
    dft_table(ph_smem, n);
    // rows: consecutive threads along the row; columns: across the lines
    auto at = [&](int t, int &l, int &j) {
        l = axis == 1 ? t / n : t % DFT_LINES;
        j = axis == 1 ? t % n : t / DFT_LINES;
        return axis == 1 ? (long long)(l0 + l) * n + j : (long long)j * n + l0 + l;
    };
    for (int t = threadIdx.x; t < DFT_LINES * n; t += DFT_THREADS) {
        int l, j;
        const long long g = at(t, l, j);
        a[l * n + j] = l < nl ? in[g] : make_double2(0., 0.);
    }
    __syncthreads();
    dft<false, EP == EP_ABS_REAL>(ph_smem, a, b, n, sign, scale);
    for (int t = threadIdx.x; t < DFT_LINES * n; t += DFT_THREADS) {
        int l, j;
        const long long g = at(t, l, j);
        if (l >= nl) continue;
        if (EP == EP_STORE)
            out[g] = b[l * n + j];
        else
            out_re[g] = fabs(b[l * n + j].x);
    }
}

// A refinement step's Fourier side, per pixel: STEP_NONE nothing, STEP_ER
// the projection p = proj_fourier(fconv, x), STEP_DM z = 2 p - x.
enum Step : int { STEP_NONE = 0, STEP_ER = 1, STEP_DM = 2, STEP_PLAIN = 3 };

// Rows of the refinement.  prev: the step whose real-space projection comes
// back in t (transformed along the columns): its rows are transformed forward
// to y, and x becomes y (STEP_ER, STEP_PLAIN) or x + y - p (STEP_DM).  next:
// the step that starts from x: its input's rows, transformed back, go to t
// (STEP_PLAIN: x itself).
__global__ void __launch_bounds__(DFT_THREADS)
k_phase_rows(const double2 *__restrict__ fconv, const unsigned char *__restrict__ minvmask,
             const double2 *xin, double2 *xout, double2 *t, int n, int prev, int next) {
    extern __shared__ __align__(16) double2 ph_smem[];
    double2 *a = dft_lines(ph_smem, n, 0), *b = dft_lines(ph_smem, n, 1);
    const int l0 = blockIdx.x * DFT_LINES, nv = min(DFT_LINES, n - l0) * n;
    const long long base = (long long)l0 * n;
    dft_table(ph_smem, n);
    if (prev != STEP_NONE) {
        for (int i = threadIdx.x; i < DFT_LINES * n; i += DFT_THREADS)
            a[i] = i < nv ? t[base + i] : make_double2(0., 0.);
        __syncthreads();
        dft<false, false>(ph_smem, a, b, n, -1., 1.);
    }
    for (int i = threadIdx.x; i < DFT_LINES * n; i += DFT_THREADS) {
        double2 z = make_double2(0., 0.);
        if (i < nv) {
            double2 x = prev == STEP_ER || prev == STEP_PLAIN ? b[i] : xin[base + i];
            const bool known = prev != STEP_PLAIN && next != STEP_PLAIN && minvmask[base + i];
            const double2 f = known ? fconv[base + i] : x;
            if (prev == STEP_DM) {
                const double2 y = b[i];
                x = make_double2(x.x + y.x - f.x, x.y + y.y - f.y);
            }
            if (prev != STEP_NONE) xout[base + i] = x;
            const double2 p = known ? f : x;
            z = next == STEP_DM ? make_double2(2. * p.x - x.x, 2. * p.y - x.y) : p;
        }
        a[i] = z;
    }
    if (next == STEP_NONE) return;
    __syncthreads();
    dft<false, false>(ph_smem, a, b, n, 1., 1. / (double)n);
    for (int i = threadIdx.x; i < nv; i += DFT_THREADS) t[base + i] = b[i];
}

// Columns of the refinement: t's columns transformed back, the real part
// without negatives and without the pixels outside the support, transformed
// forward again.
__global__ void __launch_bounds__(DFT_THREADS)
k_phase_cols(double2 *t, const unsigned char *__restrict__ minvsupp, int n) {
    extern __shared__ __align__(16) double2 ph_smem[];
    double2 *a = dft_lines(ph_smem, n, 0), *b = dft_lines(ph_smem, n, 1);
    const int l0 = blockIdx.x * DFT_LINES, nl = min(DFT_LINES, n - l0);
    dft_table(ph_smem, n);
    for (int i = threadIdx.x; i < DFT_LINES * n; i += DFT_THREADS) {
        const int l = i % DFT_LINES, j = i / DFT_LINES;
        a[l * n + j] = l < nl ? t[(long long)j * n + l0 + l] : make_double2(0., 0.);
    }
    __syncthreads();
    dft<false, true>(ph_smem, a, b, n, 1., 1. / (double)n);
    for (int i = threadIdx.x; i < DFT_LINES * n; i += DFT_THREADS) {
        const int l = i % DFT_LINES, j = i / DFT_LINES;
        const double r = b[l * n + j].x;
        const bool out = l >= nl || minvsupp[(long long)j * n + l0 + l];
        a[l * n + j] = make_double2(r < 0. || out ? 0. : r, 0.);
    }
    __syncthreads();
    dft<true, false>(ph_smem, a, b, n, -1., 1.);
    for (int i = threadIdx.x; i < DFT_LINES * n; i += DFT_THREADS) {
        const int l = i % DFT_LINES, j = i / DFT_LINES;
        if (l < nl) t[(long long)j * n + l0 + l] = b[l * n + j];
    }
}

// proj_fourier(fconv, x): data pixels from fconv.
__global__ void k_proj_fourier(const double2 *__restrict__ fconv,
                               const unsigned char *__restrict__ minvmask,
                               const double2 *__restrict__ x, double2 *__restrict__ p1,
                               long long npix) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < npix; t += stride)
        p1[t] = minvmask[t] ? fconv[t] : x[t];
}

// fconv * expit((mrad - r0) * slope), mrad the integer-centred radius.
__global__ void k_support_taper(const double2 *__restrict__ fconv, int n, double r0,
                                double slope, double2 *__restrict__ out) {
    const long long npix = (long long)n * n;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const int cen = n / 2;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < npix; t += stride) {
        const long long xi = t / n, yi = t - xi * n;
        const double dx = (double)(xi - cen), dy = (double)(yi - cen);
        const double r = sqrt(dx * dx + dy * dy);
        const double e = 1. / (1. + exp(-((r - r0) * slope)));
        const double2 v = fconv[t];
        out[t] = make_double2(v.x * e, v.y * e);
    }
}

// One CTA per line: correlate with the normalised Gaussian of half-width
// `radius` ('reflect' edges); with `thr_out`, minvsupp = !(value > thr).
__global__ void __launch_bounds__(256)
k_gauss_lines(const double *__restrict__ in, double *__restrict__ out, int n, int axis,
              double sigma, int radius, double thr, unsigned char *__restrict__ minvsupp) {
    __shared__ double line[MAX_N];
    __shared__ double w[MAX_RADIUS + 1];
    const int li = blockIdx.x;
    const long long stride = axis == 1 ? 1 : n;
    const long long base = axis == 1 ? (long long)li * n : li;
    for (int j = threadIdx.x; j < n; j += blockDim.x) line[j] = in[base + j * stride];
    if (threadIdx.x == 0) {
        // phi(x) = exp(-x^2 / (2 sigma^2)) / sum over |x| <= radius
        double sum = 0.;
        for (int k = -radius; k <= radius; ++k) sum += exp(-0.5 / (sigma * sigma) * (double)(k * k));
        for (int k = 0; k <= radius; ++k) w[k] = exp(-0.5 / (sigma * sigma) * (double)(k * k)) / sum;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double acc = line[i] * w[0];
        for (int k = radius; k >= 1; --k) {   // outermost pair first
            int lo = i - k, hi = i + k;
            // reflect about the edge: -1 -> 0, n -> n - 1 (radius < n)
            lo = lo < 0 ? -lo - 1 : lo;
            hi = hi >= n ? 2 * n - hi - 1 : hi;
            acc += (line[lo] + line[hi]) * w[k];
        }
        const long long t = base + i * stride;
        if (minvsupp)
            minvsupp[t] = !(acc > thr);
        else
            out[t] = acc;
    }
}

// One pass along `axis`.
template <int EP>
int line_pass(const double2 *in, double2 *out, int n, int axis, double sign, double scale,
              double *out_re, cudaStream_t stream) {
    static RspiSmemOptIn optin;
    if (!rspi_smem_optin((const void *)k_cdft_lines<EP>, dft_smem(n), optin)) return RSPI_ERR_CUDA;
    k_cdft_lines<EP><<<(n + DFT_LINES - 1) / DFT_LINES, DFT_THREADS, dft_smem(n), stream>>>(
        in, out, n, axis, sign, scale, out_re);
    return RSPI_OK;
}

int rows_pass(const double2 *fconv, const unsigned char *minvmask, const double2 *xin,
              double2 *xout, double2 *t, int n, int prev, int next, cudaStream_t stream) {
    static RspiSmemOptIn optin;
    if (!rspi_smem_optin((const void *)k_phase_rows, dft_smem(n), optin)) return RSPI_ERR_CUDA;
    k_phase_rows<<<(n + DFT_LINES - 1) / DFT_LINES, DFT_THREADS, dft_smem(n), stream>>>(
        fconv, minvmask, xin, xout, t, n, prev, next);
    return RSPI_OK;
}

int cols_pass(double2 *t, const unsigned char *minvsupp, int n, cudaStream_t stream) {
    static RspiSmemOptIn optin;
    if (!rspi_smem_optin((const void *)k_phase_cols, dft_smem(n), optin)) return RSPI_ERR_CUDA;
    k_phase_cols<<<(n + DFT_LINES - 1) / DFT_LINES, DFT_THREADS, dft_smem(n), stream>>>(
        t, minvsupp, n);
    return RSPI_OK;
}

bool size_ok(long long n) { return n >= 2 && n <= MAX_N; }

}  // namespace

extern "C" int rspi_cdft2(const double *in, double *out, double *work, long long size,
                          int inverse, cudaStream_t stream) {
    if (!in || !out || !work || !size_ok(size) || (inverse != 0 && inverse != 1))
        return RSPI_ERR_ARG;
    const int n = (int)size;
    const double sign = inverse ? 1. : -1.;
    const double scale = inverse ? 1. / (double)n : 1.;
    double2 *t = reinterpret_cast<double2 *>(work);
    int st = line_pass<EP_STORE>(reinterpret_cast<const double2 *>(in), t, n, 1, sign, scale,
                                 nullptr, stream);
    if (st == RSPI_OK)
        st = line_pass<EP_STORE>(t, reinterpret_cast<double2 *>(out), n, 0, sign, scale, nullptr,
                                 stream);
    if (st != RSPI_OK) return st;
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_phase_support(const double *fconv, long long size, double taper_radius,
                                  double taper_slope, double sigma, int radius, double threshold,
                                  unsigned char *minvsupp, double *work, cudaStream_t stream) {
    if (!fconv || !minvsupp || !work || !size_ok(size) || radius < 0 || radius > MAX_RADIUS ||
        radius >= size || !(sigma > 0.))
        return RSPI_ERR_ARG;
    const int n = (int)size;
    const long long npix = size * size;
    double2 *t1 = reinterpret_cast<double2 *>(work);
    double2 *t2 = t1 + npix;
    double *re = reinterpret_cast<double *>(t2 + npix);
    double *sm = re + npix;
    const double inv_n = 1. / (double)n;
    k_support_taper<<<rspi_blocks(npix, 256), 256, 0, stream>>>(
        reinterpret_cast<const double2 *>(fconv), n, taper_radius, taper_slope, t1);
    int st = line_pass<EP_STORE>(t1, t2, n, 1, 1., inv_n, nullptr, stream);
    if (st == RSPI_OK) st = line_pass<EP_ABS_REAL>(t2, nullptr, n, 0, 1., inv_n, re, stream);
    if (st != RSPI_OK) return st;
    k_gauss_lines<<<n, 256, 0, stream>>>(re, sm, n, 0, sigma, radius, 0., nullptr);
    k_gauss_lines<<<n, 256, 0, stream>>>(sm, nullptr, n, 1, sigma, radius, threshold, minvsupp);
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_phase_refine(const double *fconv, const unsigned char *minvmask,
                                 const unsigned char *minvsupp, double *x, double *work,
                                 long long size, int n_dm, int n_er, cudaStream_t stream) {
    if (!fconv || !minvmask || !minvsupp || !x || !work || !size_ok(size) || n_dm < 0 ||
        n_er < 0)
        return RSPI_ERR_ARG;
    const int n = (int)size, steps = n_dm + n_er;
    const double2 *f = reinterpret_cast<const double2 *>(fconv);
    double2 *xv = reinterpret_cast<double2 *>(x);
    double2 *t = reinterpret_cast<double2 *>(work);
    // steps 0 .. n_dm - 1: x + proj_real(2 p - x) - p with p =
    // proj_fourier(fconv, x); then proj_real(p)
    auto kind = [&](int it) -> int { return it >= steps ? STEP_NONE : it < n_dm ? STEP_DM : STEP_ER; };
    for (int it = 0; it <= steps && steps > 0; ++it) {
        int st = rows_pass(f, minvmask, xv, xv, t, n, it == 0 ? STEP_NONE : kind(it - 1), kind(it),
                           stream);
        if (st == RSPI_OK && it < steps) st = cols_pass(t, minvsupp, n, stream);
        if (st != RSPI_OK) return st;
    }
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_phase_proj_fourier(const double *fconv, const unsigned char *minvmask,
                                       const double *x, double *out, long long size,
                                       cudaStream_t stream) {
    if (!fconv || !minvmask || !x || !out || !size_ok(size)) return RSPI_ERR_ARG;
    const long long npix = size * size;
    k_proj_fourier<<<rspi_blocks(npix, 256), 256, 0, stream>>>(
        reinterpret_cast<const double2 *>(fconv), minvmask, reinterpret_cast<const double2 *>(x),
        reinterpret_cast<double2 *>(out), npix);
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_phase_proj_real(const double *x, const unsigned char *minvsupp, double *out,
                                    double *work, long long size, cudaStream_t stream) {
    if (!x || !minvsupp || !out || !work || !size_ok(size)) return RSPI_ERR_ARG;
    const int n = (int)size;
    const double2 *xv = reinterpret_cast<const double2 *>(x);
    double2 *t = reinterpret_cast<double2 *>(work);
    int st = rows_pass(nullptr, nullptr, xv, nullptr, t, n, STEP_NONE, STEP_PLAIN, stream);
    if (st == RSPI_OK) st = cols_pass(t, minvsupp, n, stream);
    if (st == RSPI_OK)
        st = rows_pass(nullptr, nullptr, xv, reinterpret_cast<double2 *>(out), t, n, STEP_PLAIN,
                       STEP_NONE, stream);
    if (st != RSPI_OK) return st;
    RSPI_RETURN_LAUNCH();
}
