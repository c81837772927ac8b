// Posterior-weighted merge (row a10).
//
// The reference ships, but never launches, merge_all (kernels.cu:139-152: a
// posterior-weighted photon scatter, view[pix] += prob * count) and
// slice_merge (kernels.cu:84-114: the adjoint of the bilinear rotation).
// Composed, they give the standard EMC intensity update per (shift,
// diameter) state s0:
//   num[s0](q) = sum_j R_j^T [ sum_d P[s0,j,d] K_d ](q)
//   den[s0](q) = sum_j w[s0,j] C_j(q),   w[r] = sum_d P[r,d] scale_d,
//   C_j = R_j^T 1 (the coverage of rotation j),  intens = num / den,
// counting only posteriors P >= p_min (P_MIN, emc.py:20).  Posteriors come
// from a (frame, row, log-likelihood) list and the per-frame log-sum-exp.
// FP64 accumulators throughout.
#include "rspi_common.cuh"

namespace {

constexpr int RY = 32;

// pairs (d, r, LL) with exp(LL - logz[d]) >= p_min, from a full FP64 matrix
__global__ void __launch_bounds__(32 * RY)
k_sig_count(const double *__restrict__ ll, long long n_rows, long long n_data,
            const double *__restrict__ logz, double p_min, int *__restrict__ cnt_part,
            int *__restrict__ cnt) {
    __shared__ int sc[RY][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const long long d = (long long)blockIdx.x * 32 + tx;
    int c = 0;
    if (d < n_data) {
        const double lz = logz[d];
        for (long long r = ty; r < n_rows; r += RY)
            if (exp(ll[r * n_data + d] - lz) >= p_min) ++c;
        cnt_part[d * RY + ty] = c;
    }
    sc[ty][tx] = c;
    __syncthreads();
    if (ty == 0 && d < n_data) {
        int tot = 0;
        for (int k = 0; k < RY; ++k) tot += sc[k][tx];
        cnt[d] = tot;
    }
}

__global__ void __launch_bounds__(32 * RY)
k_sig_fill(const double *__restrict__ ll, long long n_rows, long long n_data,
           const double *__restrict__ logz, double p_min, const int *__restrict__ cnt_part,
           const long long *__restrict__ off, long long capacity, int *__restrict__ pd,
           int *__restrict__ pr, double *__restrict__ pll, int *err) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const long long d = (long long)blockIdx.x * 32 + tx;
    if (d >= n_data) return;
    long long pos = off[d];
    for (int k = 0; k < ty; ++k) pos += cnt_part[d * RY + k];
    const double lz = logz[d];
    for (long long r = ty; r < n_rows; r += RY) {
        const double v = ll[r * n_data + d];
        if (exp(v - lz) >= p_min) {
            if (pos < capacity) {
                pd[pos] = (int)d;
                pr[pos] = (int)r;
                pll[pos] = v;
            } else {
                rspi_flag(err, RSPI_ERR_CAPACITY);
            }
            ++pos;
        }
    }
}

// Bilinear footprint of detector pixel (x, y) under rotation (ac, as), the
// geometry of slice_merge (kernels.cu:93-101).  Returns false off-detector.
__device__ __forceinline__ bool footprint(int x, int y, int size, double ac, double as, int &ix,
                                          int &iy, double &fx, double &fy) {
    const int cen = size / 2;
    const double xc = (double)(x - cen), yc = (double)(y - cen);
    const double tx = xadd(xsub(xmul(xc, ac), xmul(yc, as)), (double)cen);
    const double ty = xadd(xadd(xmul(xc, as), xmul(yc, ac)), (double)cen);
    const double fxl = floor(tx), fyl = floor(ty);
    if (fxl < 0. || fxl > size - 2 || fyl < 0. || fyl > size - 2) return false;
    ix = (int)fxl;
    iy = (int)fyl;
    fx = tx - fxl;
    fy = ty - fyl;
    return true;
}

__device__ __forceinline__ void scatter4(double *__restrict__ acc, int size, int ix, int iy,
                                         double fx, double fy, double v) {
    const double cx = 1. - fx, cy = 1. - fy;
    double *a = acc + (long long)ix * size + iy;
    atomicAdd(a, v * cx * cy);
    atomicAdd(a + size, v * fx * cy);
    atomicAdd(a + 1, v * cx * fy);
    atomicAdd(a + size + 1, v * fx * fy);
}

// One warp per significant pair: scatter P * K_d back through rotation j
// into num[s0] and add P * scale_d to w[r].  With row_done only the pairs of
// rows that k_merge_rows left.  A warp tests up to eight pairs at once.
__global__ void __launch_bounds__(256)
k_merge_scatter(const int *__restrict__ pd, const int *__restrict__ pr,
                const double *__restrict__ pll, const long long *__restrict__ total_ptr,
                long long capacity, const double *__restrict__ logz, double p_min,
                const double *__restrict__ scales, const int *__restrict__ ones,
                const int *__restrict__ multi, const long long *__restrict__ ones_accum,
                const long long *__restrict__ multi_accum, const int *__restrict__ place_ones,
                const int *__restrict__ place_multi, const int *__restrict__ count_multi,
                long long num_rot, const double *__restrict__ rot_cs, int size,
                const int *__restrict__ row_done, double *__restrict__ num,
                double *__restrict__ w) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long total = min(*total_ptr, capacity);
    const long long npix = (long long)size * size;
    const int per = (int)max(1LL, min(8LL, (total + nwarp - 1) / nwarp));
    for (long long i0 = warp * per; i0 < total; i0 += nwarp * per) {
        int my_d = 0, my_r = 0;
        double my_p = 0.;
        bool mine = lane < per && i0 + lane < total;
        if (mine) {
            my_r = pr[i0 + lane];
            mine = !row_done || !row_done[my_r];
        }
        if (mine) {
            my_d = pd[i0 + lane];
            my_p = exp(pll[i0 + lane] - logz[my_d]);
            mine = my_p >= p_min;
        }
        for (unsigned left = __ballot_sync(RSPI_FULL_MASK, mine); left; left &= left - 1) {
            const int src = __ffs(left) - 1;
            const int d = __shfl_sync(RSPI_FULL_MASK, my_d, src);
            const int r = __shfl_sync(RSPI_FULL_MASK, my_r, src);
            const double p = __shfl_sync(RSPI_FULL_MASK, my_p, src);
            const long long s0 = r / num_rot, j = r - s0 * num_rot;
            const double ac = rot_cs[2 * j], as = rot_cs[2 * j + 1];
            double *acc = num + s0 * npix;
            if (lane == 0) atomicAdd(&w[r], p * scales[d]);
            const int n_o = ones[d], n_m = multi[d];
            const long long oa = ones_accum[d], ma = multi_accum[d];
            for (int k = lane; k < n_o + n_m; k += 32) {
                int pix;
                double cnt;
                if (k < n_o) {
                    pix = place_ones[oa + k];
                    cnt = 1.;
                } else {
                    pix = place_multi[ma + k - n_o];
                    cnt = (double)count_multi[ma + k - n_o];
                }
                if (pix < 0 || pix >= npix) continue;
                int ix, iy;
                double fx, fy;
                if (footprint(pix / size, pix % size, size, ac, as, ix, iy, fx, fy))
                    scatter4(acc, size, ix, iy, fx, fy, p * cnt);
            }
        }
    }
}

// The pairs of a likelihood row with many photons, a CTA per row.  R_j^T is
// linear, so the row sums P K_d unrotated into the CTA's image (one FP64
// reduction per photon) and then turns that image back (four per populated
// pixel) instead of four per photon.  Rows with fewer than npix / MR_DENSE
// photons are left to k_merge_scatter (row_done 0), which spreads them over
// the GPU: the warps of a CTA would meet in the same pixels of one state.
// Both wait for L2: 30 cycles of 33 between a warp's issues, the atomics at 27%
// of L2's rate.  848,000 pairs of 1,003 frames over 4,500
// rows of 185^2 take 1.88 ms, both kernels (1.95 with every row here, 2.56 with
// one CTA per SM, 3.75 with every photon turned); 101,000 pairs of 1,138
// frames over 4,400 rows of 174^2, three of them dense, 0.73 ms by the scatter
// and 1.07 by row.
constexpr int MR_THREADS = 1024;
constexpr int MR_DENSE = 2;
constexpr int MR_MIN_PAIRS = 16;   // a row's pairs before its photons are counted

__global__ void __launch_bounds__(MR_THREADS, 2)
k_merge_rows(const int *__restrict__ pd, const double *__restrict__ pll,
             const long long *__restrict__ row_off, const int *__restrict__ row_cand,
             long long n_rows, const double *__restrict__ logz, double p_min,
             const double *__restrict__ scales, const int *__restrict__ ones,
             const int *__restrict__ multi, const long long *__restrict__ ones_accum,
             const long long *__restrict__ multi_accum, const int *__restrict__ place_ones,
             const int *__restrict__ place_multi, const int *__restrict__ count_multi,
             long long num_rot, const double *__restrict__ rot_cs, int size,
             double *__restrict__ num, double *__restrict__ w, int *__restrict__ row_done,
             double *__restrict__ images) {
    __shared__ double wsum[MR_THREADS / 32];
    __shared__ unsigned long long n_phot;
    __shared__ int list[MR_THREADS], n_list;
    __shared__ int sig_d[MR_THREADS], n_sig;   // significant pairs of a batch
    __shared__ double sig_p[MR_THREADS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int npix = size * size;
    double *view = images + (long long)blockIdx.x * npix;
    // the CTA's rows r = blockIdx.x + k gridDim.x, tested MR_THREADS at a time
    for (long long base = blockIdx.x; base < n_rows; base += (long long)gridDim.x * MR_THREADS) {
        __syncthreads();   // the previous list's readers are done
        if (threadIdx.x == 0) n_list = 0;
        __syncthreads();
        const long long rt = base + (long long)threadIdx.x * gridDim.x;
        if (rt < n_rows) {
            row_done[rt] = 0;
            if (row_off[rt + 1] - row_off[rt] >= MR_MIN_PAIRS)
                list[atomicAdd(&n_list, 1)] = (int)rt;
        }
        __syncthreads();
        for (int kr = 0; kr < n_list; ++kr) {
            const long long r = list[kr];
            const long long a = row_off[r], b = row_off[r + 1];
            const long long s0 = r / num_rot, j = r - s0 * num_rot;
            const double ac = rot_cs[2 * j], as = rot_cs[2 * j + 1];
            double *acc = num + s0 * npix;
            __syncthreads();   // the previous row's readers are done
            if (threadIdx.x == 0) n_phot = 0;
            __syncthreads();
            // the row's weight and photon entries
            double wp = 0.;
            unsigned np = 0;
            for (long long i = a + threadIdx.x; i < b; i += MR_THREADS) {
                const int pair = row_cand[i], d = pd[pair];
                const double p = exp(pll[pair] - logz[d]);
                if (!(p >= p_min)) continue;
                wp += p * scales[d];
                np += (unsigned)(ones[d] + multi[d]);
            }
            wp = warp_sum(wp);
            np = __reduce_add_sync(RSPI_FULL_MASK, np);
            if (lane == 0) {
                wsum[wid] = wp;
                if (np) atomicAdd(&n_phot, (unsigned long long)np);
            }
            __syncthreads();
            if (n_phot * MR_DENSE < (unsigned long long)npix) continue;
            if (threadIdx.x == 0) {
                double t = 0.;
                for (int k = 0; k < MR_THREADS / 32; ++k) t += wsum[k];
                w[r] = t;
                row_done[r] = 1;
            }
            for (int t = threadIdx.x; t < npix; t += MR_THREADS) __stcg(view + t, 0.);
            __threadfence();
            // a thread tests a pair (most of a row's may be below p_min); the
            // warps share those that are not, several to a pair when they are few
            for (long long i0 = a; i0 < b; i0 += MR_THREADS) {
                __syncthreads();   // the previous batch's readers are done
                if (threadIdx.x == 0) n_sig = 0;
                __syncthreads();
                if (i0 + threadIdx.x < b) {
                    const int pair = row_cand[i0 + threadIdx.x], d = pd[pair];
                    const double p = exp(pll[pair] - logz[d]);
                    if (p >= p_min) {
                        const int k = atomicAdd(&n_sig, 1);
                        sig_d[k] = d;
                        sig_p[k] = p;
                    }
                }
                __syncthreads();
                const int share = n_sig > 0 ? max(1, MR_THREADS / 32 / n_sig) : 1;
                for (int q = wid / share; q < n_sig; q += MR_THREADS / 32 / share) {
                    const int d = sig_d[q];
                    const double p = sig_p[q];
                    const int n_o = ones[d], n_m = multi[d];
                    const long long oa = ones_accum[d], ma = multi_accum[d];
                    for (int k = lane + 32 * (wid % share); k < n_o + n_m; k += 32 * share) {
                        int pix;
                        double cnt;
                        if (k < n_o) {
                            pix = place_ones[oa + k];
                            cnt = 1.;
                        } else {
                            pix = place_multi[ma + k - n_o];
                            cnt = (double)count_multi[ma + k - n_o];
                        }
                        if (pix >= 0 && pix < npix) atomicAdd(view + pix, p * cnt);
                    }
                }
            }
            __threadfence();
            __syncthreads();   // the image is complete (in L2)
            for (int t = threadIdx.x; t < npix; t += MR_THREADS) {
                const double v = __ldcg(view + t);
                if (v == 0.) continue;
                int ix, iy;
                double fx, fy;
                if (footprint(t / size, t % size, size, ac, as, ix, iy, fx, fy))
                    scatter4(acc, size, ix, iy, fx, fy, v);
            }
        }
    }
}

// Coverage C_j = R_j^T 1 of every rotation (independent of the data).
__global__ void k_coverage(long long num_rot, const double *__restrict__ rot_cs, int size,
                           double *__restrict__ cov) {
    const long long npix = (long long)size * size;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < num_rot * npix;
         i += stride) {
        const long long j = i / npix, t = i - j * npix;
        int ix, iy;
        double fx, fy;
        if (footprint((int)(t / size), (int)(t % size), size, rot_cs[2 * j], rot_cs[2 * j + 1],
                      ix, iy, fx, fy))
            scatter4(cov + j * npix, size, ix, iy, fx, fy, 1.);
    }
}

// den[s0][q] = sum_j w[s0*R + j] C_j(q); intens = num / den (0 where den == 0)
__global__ void k_merge_finalize(const double *__restrict__ num, const double *__restrict__ w,
                                 const double *__restrict__ cov, long long n_states0,
                                 long long num_rot, long long npix, double *__restrict__ den,
                                 double *__restrict__ intens) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_states0 * npix;
         i += stride) {
        const long long s0 = i / npix, q = i - s0 * npix;
        double acc = 0.;
        for (long long j = 0; j < num_rot; ++j) {
            const double wj = w[s0 * num_rot + j];
            if (wj != 0.) acc += wj * cov[j * npix + q];
        }
        den[i] = acc;
        intens[i] = acc > 0. ? num[i] / acc : 0.;
    }
}

}  // namespace

extern "C" int rspi_posterior_pairs(const double *ll, long long n_rows, long long n_data,
                                    const double *logz, double p_min, int *cnt_part, int *cnt,
                                    long long *off, long long capacity, int *pair_d, int *pair_r,
                                    double *pair_ll, int *err, cudaStream_t stream) {
    if (!ll || !logz || !cnt_part || !cnt || !off || !pair_d || !pair_r || !pair_ll ||
        n_rows <= 0 || n_data <= 0 || n_rows > 0x7fffffffLL || capacity < 0)
        return RSPI_ERR_ARG;
    const dim3 block(32, RY);
    const unsigned grid = (unsigned)((n_data + 31) / 32);
    k_sig_count<<<grid, block, 0, stream>>>(ll, n_rows, n_data, logz, p_min, cnt_part, cnt);
    const int scan = rspi_scan_i32(cnt, n_data, off, stream);
    if (scan != RSPI_OK) return scan;
    k_sig_fill<<<grid, block, 0, stream>>>(ll, n_rows, n_data, logz, p_min, cnt_part, off,
                                           capacity, pair_d, pair_r, pair_ll, err);
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_merge_coverage(long long num_rot, const double *rot_cs, long long size,
                                   double *cov, cudaStream_t stream) {
    if (num_rot <= 0 || !rot_cs || !cov || size <= 1 || size > 46340) return RSPI_ERR_ARG;
    cudaMemsetAsync(cov, 0, sizeof(double) * num_rot * size * size, stream);
    k_coverage<<<rspi_blocks(num_rot * size * size, 256, 16), 256, 0, stream>>>(
        num_rot, rot_cs, (int)size, cov);
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_merge(const int *pair_d, const int *pair_r, const double *pair_ll,
                          const long long *pair_total, long long capacity, const double *logz,
                          double p_min, const double *scales, const int *ones, const int *multi,
                          const long long *ones_accum, const long long *multi_accum,
                          const int *place_ones, const int *place_multi, const int *count_multi,
                          long long n_states0, long long num_rot, const double *rot_cs,
                          long long size, const double *cov, double *num, double *den,
                          double *w, double *intens, cudaStream_t stream) {
    if (!pair_d || !pair_r || !pair_ll || !pair_total || !logz || !scales || !ones || !multi ||
        !ones_accum || !multi_accum || !rot_cs || !cov || !num || !den || !w || !intens ||
        n_states0 <= 0 || num_rot <= 0 || size <= 1 || size > 46340 || capacity < 0)
        return RSPI_ERR_ARG;
    const long long npix = size * size;
    cudaMemsetAsync(num, 0, sizeof(double) * n_states0 * npix, stream);
    cudaMemsetAsync(w, 0, sizeof(double) * n_states0 * num_rot, stream);
    k_merge_scatter<<<rspi_sm_count() * 8, 256, 0, stream>>>(
        pair_d, pair_r, pair_ll, pair_total, capacity, logz, p_min, scales, ones, multi,
        ones_accum, multi_accum, place_ones, place_multi, count_multi, num_rot, rot_cs,
        (int)size, nullptr, num, w);
    k_merge_finalize<<<rspi_blocks(n_states0 * npix, 256, 16), 256, 0, stream>>>(
        num, w, cov, n_states0, num_rot, npix, den, intens);
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_merge_rows(const int *pair_d, const int *pair_r, const double *pair_ll,
                               const long long *row_off, const int *row_cand, const double *logz,
                               double p_min, const double *scales, const int *ones,
                               const int *multi, const long long *ones_accum,
                               const long long *multi_accum, const int *place_ones,
                               const int *place_multi, const int *count_multi,
                               long long n_states0, long long num_rot, const double *rot_cs,
                               long long size, const double *cov, double *num, double *den,
                               double *w, double *intens, int *row_done, double *images,
                               long long n_images, cudaStream_t stream) {
    if (!pair_d || !pair_r || !pair_ll || !row_off || !row_cand || !logz || !scales || !ones ||
        !multi || !ones_accum || !multi_accum || !rot_cs || !cov || !num || !den || !w ||
        !intens || !row_done || !images || n_images < 1 || n_states0 <= 0 || num_rot <= 0 ||
        size <= 1 || size > 46340)
        return RSPI_ERR_ARG;
    const long long npix = size * size, n_rows = n_states0 * num_rot;
    cudaMemsetAsync(num, 0, sizeof(double) * n_states0 * npix, stream);
    cudaMemsetAsync(w, 0, sizeof(double) * n_rows, stream);
    const unsigned grid = (unsigned)min(min(n_images, n_rows), 0x7fffffffLL);
    k_merge_rows<<<grid, MR_THREADS, 0, stream>>>(
        pair_d, pair_ll, row_off, row_cand, n_rows, logz, p_min, scales, ones, multi, ones_accum,
        multi_accum, place_ones, place_multi, count_multi, num_rot, rot_cs, (int)size, num, w,
        row_done, images);
    k_merge_scatter<<<rspi_sm_count() * 8, 256, 0, stream>>>(
        pair_d, pair_r, pair_ll, row_off + n_rows, 0x7fffffffLL, logz, p_min, scales, ones, multi,
        ones_accum, multi_accum, place_ones, place_multi, count_multi, num_rot, rot_cs, (int)size,
        row_done, num, w);
    k_merge_finalize<<<rspi_blocks(n_states0 * npix, 256, 16), 256, 0, stream>>>(
        num, w, cov, n_states0, num_rot, npix, den, intens);
    RSPI_RETURN_LAUNCH();
}
