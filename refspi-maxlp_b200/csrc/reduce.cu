// Per-frame reduction over states (rows a8, a9): first-index max/argmax
// (emc.py:207-209, prob.max(0) / prob.argmax(0)) and the FP64 log-sum-exp
// that normalises the posterior.  A CTA covers 32 frames (threadIdx.x) and
// splits the state axis over its warps (threadIdx.y); reads of LL[r][d0..d0+31]
// are coalesced.  Each thread keeps an online (max, argmax, sum exp(x-max));
// partial triples merge in a fixed order.
#include <cooperative_groups.h>

#include "rspi_common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int RY = 32;

struct Acc {
    double m;
    double s;
    int i;
};

template <bool LSE>
__device__ __forceinline__ void acc_push(Acc &a, double v, int r) {
    if (a.i < 0) {
        a = Acc{v, 1., r};
        return;
    }
    if (argmax_better(v, r, a.m, a.i)) {
        if (LSE) a.s = isnan(v) || isnan(a.m) ? a.s + 1. : a.s * exp(a.m - v) + 1.;
        a.m = v;
        a.i = r;
    } else if (LSE) {
        a.s += isnan(a.m) ? 1. : exp(v - a.m);
    }
}

__device__ __forceinline__ Acc acc_merge(Acc a, Acc b) {
    if (a.i < 0) return b;
    if (b.i < 0) return a;
    if (argmax_better(b.m, b.i, a.m, a.i)) {
        Acc t = a;
        a = b;
        b = t;
    }
    a.s = a.s + b.s * exp(b.m - a.m);
    return a;
}

// The CTAs of a cluster share a block's rows (rspi_row_ctas): each takes
// consecutive steps of 32 rows, and the first merges their results in order
// (500 frames x 6,750 states in FP64: 0.045 ms instead of 0.108).
template <typename TL, bool LSE>
__global__ void __launch_bounds__(32 * RY, 2)
k_frame_reduce(const TL *__restrict__ ll, long long n_rows, long long n_data,
               double *__restrict__ maxll, int *__restrict__ rmax, double *__restrict__ logz) {
    __shared__ double sm[RY][33];
    __shared__ double ss[RY][33];
    __shared__ int si[RY][33];
    cg::cluster_group cluster = cg::this_cluster();
    const int tx = threadIdx.x, ty = threadIdx.y;
    const long long d = (long long)blockIdx.x * 32 + tx;
    const long long per = ((n_rows + RY - 1) / RY + gridDim.y - 1) / gridDim.y * RY;
    const long long r1 = min(n_rows, (blockIdx.y + 1) * per);
    Acc a{0., 0., -1};
    if (d < n_data) {
        // eight rows' loads in flight per thread, pushed in row order
        long long r = blockIdx.y * per + ty;
        for (; r + 7 * RY < r1; r += 8 * RY) {
            TL v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldg(&ll[(r + u * RY) * n_data + d]);
#pragma unroll
            for (int u = 0; u < 8; ++u) acc_push<LSE>(a, (double)v[u], (int)(r + u * RY));
        }
        for (; r < r1; r += RY) acc_push<LSE>(a, (double)ll[r * n_data + d], (int)r);
    }
    sm[ty][tx] = a.m;
    ss[ty][tx] = a.s;
    si[ty][tx] = a.i;
    __syncthreads();
    if (ty == 0 && d < n_data) {
        Acc b{sm[0][tx], ss[0][tx], si[0][tx]};
        for (int k = 1; k < RY; ++k) b = acc_merge(b, Acc{sm[k][tx], ss[k][tx], si[k][tx]});
        sm[0][tx] = b.m;
        ss[0][tx] = b.s;
        si[0][tx] = b.i;
    }
    cluster.sync();
    if (cluster.block_rank() == 0 && ty == 0 && d < n_data) {
        Acc b{sm[0][tx], ss[0][tx], si[0][tx]};
        for (unsigned k = 1; k < cluster.num_blocks(); ++k)
            b = acc_merge(b, Acc{*cluster.map_shared_rank(&sm[0][tx], k),
                                 *cluster.map_shared_rank(&ss[0][tx], k),
                                 *cluster.map_shared_rank(&si[0][tx], k)});
        if (maxll) maxll[d] = b.m;
        if (rmax) rmax[d] = b.i;
        if (logz) logz[d] = b.m + log(b.s);
    }
    cluster.sync();   // the first CTA has read the others' shared memory
}

}  // namespace

extern "C" int rspi_frame_reduce(const void *ll, int ll_dtype, long long n_rows,
                                 long long n_data, double *maxll, int *rmax, double *logz,
                                 cudaStream_t stream) {
    if (!ll || n_rows <= 0 || n_data <= 0 || n_rows > 0x7fffffffLL) return RSPI_ERR_ARG;
    const dim3 block(32, RY);
    const long long blocks = (n_data + 31) / 32;
    const unsigned n = rspi_row_ctas(blocks, n_rows);
    int st;
    if (ll_dtype == 1 && logz)
        st = rspi_launch_rows(k_frame_reduce<double, true>, blocks, n, block, stream,
                              (const double *)ll, n_rows, n_data, maxll, rmax, logz);
    else if (ll_dtype == 1)
        st = rspi_launch_rows(k_frame_reduce<double, false>, blocks, n, block, stream,
                              (const double *)ll, n_rows, n_data, maxll, rmax, logz);
    else if (ll_dtype == 0 && logz)
        st = rspi_launch_rows(k_frame_reduce<float, true>, blocks, n, block, stream,
                              (const float *)ll, n_rows, n_data, maxll, rmax, logz);
    else if (ll_dtype == 0)
        st = rspi_launch_rows(k_frame_reduce<float, false>, blocks, n, block, stream,
                              (const float *)ll, n_rows, n_data, maxll, rmax, logz);
    else
        return RSPI_ERR_ARG;
    if (st != RSPI_OK) return st;
    RSPI_RETURN_LAUNCH();
}
