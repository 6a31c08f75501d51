// CGLS for the Tikhonov-regularised tomography system A x = B on the device (sm_100a).
//
// Same recurrence as Least_squares::sparse_cgls (src/tomography/least_squares/
// least_squares.cpp:424-496) -- s = B, r = A's, p = r, q = A p, then per iteration
// a = r'r/q'q, x += a p, s -= a q, r = A's, b = r'r/r'r_old, p = r + b p, q = A p --
// with the FP32 matrix in CSR (A) and CSR of the transpose (A', so both
// products are gathers, no atomics), and FP64 for every inner product, the step lengths
// and the row sums.  One cooperative persistent launch runs all iterations; the four
// grid-wide dependencies per iteration are software grid barriers with bounded waits.
// Reductions are deterministic: fixed row-to-thread mapping, fixed-order block and grid
// sums computed identically by every block.
//
// A' has very uneven rows: a model cell is crossed by anything from no ray to thousands
// (config 3: median 3 non-zeros, maximum 3,206; config 5: 778 on average).  Rows longer
// than long_row_limit -- 8 x the mean row length, at least kLongRow -- are listed once per
// call (cgls_long_rows, in row order) and summed with eight accumulators a lane; a warp takes
// one row at a time, long ones first, from its block's share of the rows (spmv_t).  A fixed
// limit of kLongRow made nearly every config-5 row a long one: 2.26 ms per iteration there
// against 1.83 ms with the relative limit and the unrolled gathers (config 3: 0.111 ->
// 0.094 ms).
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "common.cuh"
#include "cgls.cuh"

namespace tomo {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kLongRow = 256;  // A' rows of no more non-zeros are never long ones (long_row_limit)

// Block-wide FP64 sum in a fixed order; result valid in every thread.
__device__ __forceinline__ double block_sum(double v, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < kWarps; i++) t += sh[i];
    return t;
}

// Sum of the per-block partials (same order in every block).
__device__ __forceinline__ double grid_sum(const double *partials, int nb, double *sh)
{
    double v = 0.0;
    if (threadIdx.x < 32) {
        for (int i = threadIdx.x; i < nb; i += 32) v += __ldcg(partials + i);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        if (threadIdx.x == 0) sh[kWarps] = v;
    }
    __syncthreads();
    v = sh[kWarps];
    __syncthreads();
    return v;
}

// Rows of A' longer than this are long ones, summed with eight accumulators a lane (spmv_t;
// t_ptr[M] = the non-zero count).
__device__ __forceinline__ int long_row_limit(const int *t_ptr, int M)
{
    const long long mean8 = 8ll * t_ptr[M] / (M > 0 ? M : 1);
    return mean8 > kLongRow ? (int)mean8 : kLongRow;
}

// One lane's share of a row's product: entries b, b + step, ... of the row, gathers unrolled
// 4 deep.  x is read through L1: it is rewritten only between grid barriers, whose fence
// drops the SM's stale lines (30 iterations, 160,000 rays on 5.8 M non-zeros: 2.94 -> 2.70 ms;
// 160,000 rays of the 401 x 401 x 201 model: 5.71 -> 5.33 ms).
__device__ __forceinline__ double lane_sum(const int *idx, const float *val, const double *x, int b, int e, int step)
{
    double acc = 0.0;
#pragma unroll 4
    for (int k = b; k < e; k += step) acc += (double)__ldg(val + k) * x[__ldg(idx + k)];
    return acc;
}

// y = A x with `G` lanes per row: FP32 matrix values, FP64 vectors and row sums.  Returns this
// thread's share of y'y.
template <int G>
__device__ __forceinline__ double spmv(const int *ptr, const int *idx, const float *val, const double *x, double *y,
                                       int nrows)
{
    const int lane = threadIdx.x & 31;
    const int sub = lane % G;
    const long long gthread = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long groups = (long long)gridDim.x * blockDim.x / G;
    const long long iters = (nrows + groups - 1) / groups;  // warp-uniform trip count
    double local = 0.0;
    for (long long it = 0; it < iters; it++) {
        const long long row = gthread / G + it * groups;
        const bool mine = row < nrows;
        double acc = 0.0;
        if (mine) acc = lane_sum(idx, val, x, __ldg(ptr + row) + sub, __ldg(ptr + row + 1), G);
        for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o, G);
        if (mine && sub == 0) {
            y[row] = acc;
            local += acc * acc;
        }
    }
    return local;
}

// r = A' s.  Returns this thread's share of r'r.
//
// A block's rows are the listed long rows blockIdx, blockIdx + grid, ... and the rows
// w + 8 (blockIdx + grid it) of its warps w.  Rows differ a hundredfold in length, so a fixed
// row per warp left the block waiting for its slowest warp, and a long row summed by the whole
// block (1-12 elements a thread, two block barriers) took 3.3 us of mostly latency, 5 times in
// a row.  Here the warps draw rows from a counter in shared memory, long ones first.  A warp
// sums a long row as the 256 threads of a block would: lane l keeps the eight sums of threads
// l, l + 32, ... (eight gathers in flight) and adds them in that order.  Every row sum, and
// with the shares formed afterwards in row order every partial of r'r, is the number that a
// whole block per long row and a fixed warp per other row give, bit for bit.
// 30 iterations: 160,000 rays, 5.8 M non-zeros on 62,500 cells 2.70 -> 2.13 ms; 10.7 M on
// 269,000 cells 5.33 -> 4.89 ms.
__device__ __forceinline__ double spmv_t(const CglsLaunch &p, const double *x, double *y, double *sh, unsigned *next)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int limit = long_row_limit(p.t_ptr, p.M);
    const int nl = __ldcg(p.n_long);
    const int nlong = nl > (int)blockIdx.x ? (nl - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int step = (int)gridDim.x * kWarps;
    const int iters = (int)(((long long)p.M + step - 1) / step);
    const int total = nlong + iters * kWarps;
    if (threadIdx.x == 0) *next = kWarps;
    __syncthreads();
    for (int item = warp; item < total;) {
        int row = -1, b = 0, e = 0;
        if (item < nlong) {
            row = __ldcg(p.long_rows + blockIdx.x + item * gridDim.x);
            b = __ldg(p.t_ptr + row);
            e = __ldg(p.t_ptr + row + 1);
            double a[kWarps];
#pragma unroll
            for (int w = 0; w < kWarps; w++) a[w] = 0.0;
            for (int k = b + lane; k < e; k += kThreads) {
#pragma unroll
                for (int w = 0; w < kWarps; w++)
                    if (k + 32 * w < e) a[w] += (double)__ldg(p.t_val + k + 32 * w) * x[__ldg(p.t_idx + k + 32 * w)];
            }
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                for (int o = 16; o > 0; o >>= 1) a[w] += __shfl_xor_sync(kFull, a[w], o);
                t += a[w];
            }
            if (lane == 0) y[row] = t;
        } else {
            const long long r = (long long)((item - nlong) / kWarps) * step + blockIdx.x * kWarps + (item - nlong) % kWarps;
            if (r < p.M) {
                row = (int)r;
                b = __ldg(p.t_ptr + row);
                e = __ldg(p.t_ptr + row + 1);
                if (e - b <= limit) {
                    double acc = lane_sum(p.t_idx, p.t_val, x, b + lane, e, 32);
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                    if (lane == 0) y[row] = acc;
                }
            }
        }
        if (lane == 0) item = (int)atomicAdd(next, 1u);
        item = __shfl_sync(kFull, item, 0);
    }
    __syncthreads();
    // the shares: thread 0 the long rows in list order, lane 0 of a warp its other rows in order
    double local = 0.0, first = 0.0;
    if (warp == 0)
        for (int i0 = 0; i0 < nlong; i0 += 32) {
            const int i = i0 + lane;
            const double v = i < nlong ? y[__ldcg(p.long_rows + blockIdx.x + i * gridDim.x)] : 0.0;
            for (int j = 0; j < min(32, nlong - i0); j++) {
                const double t = __shfl_sync(kFull, v, j);
                first += t * t;
            }
        }
    for (int it0 = 0; it0 < iters; it0 += 32) {
        const long long row = blockIdx.x * kWarps + warp + (long long)(it0 + lane) * step;
        const bool mine = it0 + lane < iters && row < p.M &&
                          __ldg(p.t_ptr + row + 1) - __ldg(p.t_ptr + row) <= limit;
        const double v = mine ? y[row] : 0.0;
        const unsigned m = __ballot_sync(kFull, mine);
        for (int j = 0; j < min(32, iters - it0); j++) {
            const double t = __shfl_sync(kFull, v, j);
            if ((m >> j) & 1u) local += t * t;
        }
    }
    return lane == 0 ? first + local : 0.0;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 4) k_cgls(CglsLaunch p)
{
    __shared__ double sh[kWarps + 1];
    __shared__ unsigned next;
    const int nb = gridDim.x;
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nth = (long long)gridDim.x * blockDim.x;
    double *pa = p.partials, *pb = p.partials + nb, *pc = p.partials + 2 * nb;

    // s = B, x = 0
    for (long long i = tid; i < p.N; i += nth) p.s[i] = (double)p.B[i];
    for (long long i = tid; i < p.M; i += nth) p.x[i] = 0.0;
    if (!grid_barrier(p.ctrl, p.spin_limit)) return;
    // r = A' s
    double v = block_sum(spmv_t(p, p.s, p.r, sh, &next), sh);
    if (threadIdx.x == 0) pa[blockIdx.x] = v;
    if (!grid_barrier(p.ctrl, p.spin_limit)) return;
    // p = r, q = A r (= A p)
    for (long long i = tid; i < p.M; i += nth) p.p[i] = p.r[i];
    v = block_sum(spmv<8>(p.a_ptr, p.a_idx, p.a_val, p.r, p.q, p.N), sh);
    if (threadIdx.x == 0) pb[blockIdx.x] = v;
    if (!grid_barrier(p.ctrl, p.spin_limit)) return;
    double rTr = grid_sum(pa, nb, sh);
    double qTq = grid_sum(pb, nb, sh);

    for (int it = 0; it < p.nit; it++) {
        const double a = rTr / qTq;
        double ss = 0.0;
        for (long long i = tid; i < p.M; i += nth) p.x[i] += a * __ldcg(p.p + i);
        for (long long i = tid; i < p.N; i += nth) {
            const double si = __ldcg(p.s + i) - a * __ldcg(p.q + i);
            p.s[i] = si;
            ss += si * si;
        }
        v = block_sum(ss, sh);
        if (threadIdx.x == 0) pc[blockIdx.x] = v;
        if (!grid_barrier(p.ctrl, p.spin_limit)) return;
        if (p.hist) {
            const double sn = grid_sum(pc, nb, sh);
            if (blockIdx.x == 0 && threadIdx.x == 0) p.hist[it] = sqrt(sn);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) p.ctrl[kRounds] = (unsigned)(it + 1);
        // sparse_cgls_gpu's exit test on the r of this iteration (src/utils/cgls/cgls.cu:102)
        if (p.tol > 0.0 && sqrt(rTr) < p.tol) break;
        // r = A' s
        v = block_sum(spmv_t(p, p.s, p.r, sh, &next), sh);
        if (threadIdx.x == 0) pa[blockIdx.x] = v;
        if (!grid_barrier(p.ctrl, p.spin_limit)) return;
        const double rTr_new = grid_sum(pa, nb, sh);
        const double b = rTr_new / rTr;
        rTr = rTr_new;
        for (long long i = tid; i < p.M; i += nth) p.p[i] = __ldcg(p.r + i) + b * __ldcg(p.p + i);
        if (!grid_barrier(p.ctrl, p.spin_limit)) return;
        // q = A p
        v = block_sum(spmv<8>(p.a_ptr, p.a_idx, p.a_val, p.p, p.q, p.N), sh);
        if (threadIdx.x == 0) pb[blockIdx.x] = v;
        if (!grid_barrier(p.ctrl, p.spin_limit)) return;
        qTq = grid_sum(pb, nb, sh);
    }
    // the model update consumes the solution in FP32, as the reference's xdm
    for (long long i = tid; i < p.M; i += nth) p.x32[i] = (float)p.x[i];
}

cudaError_t cgls_grid(int *grid)
{
    int dev = 0, nsm = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cgls, kThreads, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    *grid = nsm * (per_sm < 4 ? per_sm : 4);
    return cudaSuccess;
}

namespace {
struct IsLongRow {
    const int *ptr;
    int M;
    __device__ bool operator()(int r) const { return ptr[r + 1] - ptr[r] > long_row_limit(ptr, M); }
};
}  // namespace

cudaError_t cgls_long_rows(const int *t_ptr, int M, int *rows, int *n_long, void *temp, size_t *temp_bytes,
                           cudaStream_t st)
{
    return cub::DeviceSelect::If(temp, *temp_bytes, thrust::counting_iterator<int>(0), rows, n_long, M,
                                 IsLongRow{t_ptr, M}, st);
}

cudaError_t cgls_run(const CglsLaunch &p, int grid, cudaStream_t st)
{
    CglsLaunch pp = p;
    void *args[] = {&pp};
    return cudaLaunchCooperativeKernel((const void *)k_cgls, dim3(grid), dim3(kThreads), args, 0, st);
}

}  // namespace tomo
