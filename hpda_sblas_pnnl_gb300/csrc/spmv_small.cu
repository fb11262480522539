// y = alpha*A*x + beta*y for small CSR matrices: one launch, no workspace.
//
// Bound: latency.  The tile path (partition, tile kernel, fix-up) is a chain of
// three kernels whose stages hand over through shared memory and barriers;
// a small matrix pays for all of it and fills a few CTAs.  Here a row is one
// chain of four dependent reads (row pointer, column, x, y).  Eight lanes take a
// row (a whole warp's reduction would cost the FP64 pipe five adds per row);
// rows of more than 64 nonzeros are left for the warps, of more than 512 for
// the whole CTA.  A CTA's
// rows are strided over the matrix, so that neighbouring long rows fall to
// different CTAs.  Figures at small_spmv_fits below.
#include "launch.cuh"
#include "ptx.cuh"
#include "sblas_internal.h"

namespace sblas {
namespace {

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;
constexpr int LANES = 8;                   // lanes per row
constexpr int LANE_ROW = 64;               // longest row of these lanes
constexpr int WARP_ROW = 512;              // longest row of a warp

struct SmallArgs {
    int m;
    int nnz;            // entries of val and col
    double alpha, beta;
    const void *val;
    const int *rowptr;
    const int *col;
    const double *x;
    double *y;
    int *status;        // cleared, or null
};

// Adds this lane's nonzeros j, j + stride, ... (U of them, below e) to s.
template <int VK, bool SKIP, int U>
__device__ __forceinline__ double dot_step(const SmallArgs &a, int j, int e, int stride, double s)
{
    int c[U];
    double v[U], x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = j + u * stride;
        c[u] = k < e ? a.col[k] : -1;
        if constexpr (VK == VAL_F64) v[u] = k < e ? static_cast<const double *>(a.val)[k] : 0.0;
        if constexpr (VK == VAL_F32)
            v[u] = k < e ? (double)static_cast<const float *>(a.val)[k] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = c[u] >= 0 ? a.x[c[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (c[u] < 0 || (SKIP && x[u] == 0.0)) continue;
        if constexpr (VK == VAL_PATTERN) s += x[u];
        else s = fma(v[u], x[u], s);
    }
    return s;
}

// One lane's share of the row [b, e), its lanes `stride` apart: steps of U
// nonzeros, the last one only as wide as it has to be (every multiply-add of
// a step occupies the FP64 pipe for ~19 cycles, also where no lane needs it).
template <int VK, bool SKIP, int U>
__device__ __forceinline__ double dot(const SmallArgs &a, int b, int e, int lane, int stride)
{
    double s = 0.0;
    for (; e - b > stride * (U / 2); b += stride * U)
        s = dot_step<VK, SKIP, U>(a, b + lane, e, stride, s);
    if constexpr (U >= 8) {
        if (e - b > stride * (U / 4)) {
            s = dot_step<VK, SKIP, U / 2>(a, b + lane, e, stride, s);
            b += stride * (U / 2);
        }
    }
    for (; e - b > stride; b += 2 * stride) s = dot_step<VK, SKIP, 2>(a, b + lane, e, stride, s);
    if (e > b) s = dot_step<VK, SKIP, 1>(a, b + lane, e, stride, s);
    return s;
}

// `rows` rows per CTA and step, eight lanes each.
template <int VK, bool SKIP>
__global__ void __launch_bounds__(THREADS) small_spmv_kernel(const SmallArgs a, int rows)
{
    __shared__ int nlong;
    __shared__ int long_row[THREADS / LANES];
    __shared__ double part[WARPS];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = tid / LANES, l = tid % LANES;
    const unsigned FULL = 0xffffffffu;
    ptx::griddep_wait();
    if (a.status != nullptr && blockIdx.x == 0 && tid == 0) *a.status = 0;
    auto store = [&](int r, double v) {
        a.y[r] = a.beta != 0.0 ? fma(a.alpha, v, a.beta * a.y[r]) : a.alpha == 1.0 ? v : a.alpha * v;
    };
    for (long long step = 0; step * gridDim.x + blockIdx.x < a.m; step += rows) {
        if (tid == 0) nlong = 0;
        __syncthreads();
        const long long row = (step + g) * gridDim.x + blockIdx.x;
        const bool in = g < rows && row < a.m;
        const int r = (int)row;
        // a row's end past the entries there are is cut off, as the tiles do
        int b = 0, e = 0;
        if (in) {
            b = max(a.rowptr[r], 0);
            e = min(a.rowptr[r + 1], a.nnz);
        }
        const bool mine = in && e - b <= LANE_ROW;
        if (in && !mine && l == 0) long_row[atomicAdd(&nlong, 1)] = r;
        if (__any_sync(FULL, mine)) {
            double s = mine ? dot<VK, SKIP, 4>(a, b, e, l, LANES) : 0.0;
#pragma unroll
            for (int d = LANES / 2; d > 0; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
            if (mine && l == 0) store(r, s);
        }
        __syncthreads();
        const int n = nlong;
        for (int i = 0; i < n; ++i) {   // the list's order does not matter: a row is one sum
            const int q = long_row[i];
            const int qb = max(a.rowptr[q], 0), qe = min(a.rowptr[q + 1], a.nnz);
            if (qe - qb <= WARP_ROW) {
                if (i % WARPS != w) continue;
                double t = dot<VK, SKIP, 8>(a, qb, qe, lane, 32);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(FULL, t, d);
                if (lane == 0) store(q, t);
            } else {   // the same for every thread
                double t = dot<VK, SKIP, 16>(a, qb, qe, tid, THREADS);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(FULL, t, d);
                if (lane == 0) part[w] = t;
                __syncthreads();
                if (tid == 0) {
                    for (int k = 1; k < WARPS; ++k) t += part[k];
                    store(q, t);
                }
                __syncthreads();
            }
        }
        __syncthreads();
    }
}

template <int VK, bool SKIP>
int launch(const SmallArgs &a, cudaStream_t stream)
{
    // rows spread over the SMs first, then up to 32 per CTA
    const int sms = device_num_sms(), cap = 8 * sms;
    int rows = (a.m + sms - 1) / sms;
    rows = rows < 1 ? 1 : rows > THREADS / LANES ? THREADS / LANES : rows;
    const int want = (a.m + rows - 1) / rows;
    SBLAS_CUDA_TRY(launch_pdl(small_spmv_kernel<VK, SKIP>, dim3(want < cap ? want : cap),
                              dim3(THREADS), 0, stream, a, rows));
    return SBLAS_OK;
}

}  // namespace


// The matrices that run here when the shape is left to the library.  Against
// them stands one dense row: an SM does 16K multiply-adds in ~5 us, where the
// tile path spreads them; hence a bound on the mean and on the longest row
// that a matrix of n columns can have.  Measured in a CUDA graph, us per product
// (per-call tile path / analysed tile path / here):
//   power-law   200 rows,   2.4K nonzeros   8.7 /  6.7 / 3.1
//              1500 rows,    18K            8.7 /  7.0 / 5.5
//              3000 rows,    48K            9.2 /  6.7 / 7.2
//              6000 rows,    96K            8.9 /  7.1 / 8.4
//             10000 rows,    52K           13.5 / 11.5 / 7.5
//             25000 rows,   132K           14.5 / 13.6 / 9.9
//             50000 rows,   263K           16.6 / 15.9 / 19.4
//   banded     1500 rows,    18K            8.2 /  6.6 / 2.2
//              6000 rows,    91K            8.9 /  6.8 / 4.0
//   one row of 16K (kept on the tile path)  8.4 /  6.4 / 8.5
bool small_spmv_fits(int m, int n, long long nnz, bool analysed)
{
    const long long longest = nnz < n ? nnz : n;
    if (nnz <= 8192) return true;
    if (longest > 32768 || nnz > 512LL * m) return false;
    return nnz <= (analysed && nnz > 8LL * m ? 32768 : 131072);
}

// Against the row-split kernel (kernel 1), which reads the row pointer and
// writes y in order and waits at no barrier, but walks a long row with the lanes
// of a mean one.  Up to 64 rows per SM, two CTAs, even rows lose half a
// microsecond at most and uneven ones gain up to 400.  us per product, row split
// / here, 8K and 131K nonzeros: rows of about one length, rows drawn towards the
// first, one row of half the nonzeros (16K at most):
//      1216 rows   2.5 / 2.6   3.4 / 3.7     13 / 4.5   45 / 12      59 / 5.3   58 / 12
//      4864        2.8 / 2.5   4.0 / 3.5     27 / 4.4   30 / 9      197 / 5.4   57 / 11
//      9728        2.5 / 2.9   3.8 / 3.7     22 / 4.5   47 / 8      216 / 5.7  111 / 11
//     19456        2.4 / 3.8   3.6 / 4.6     18 / 5.1   73 / 8      194 / 6.4  217 / 12
//     38912        2.5 / 6.2   3.4 / 7.0     15 / 6.7  111 / 8      213 / 7.5  408 / 13
//       400K       5.3 / 44    6.4 / 49
//        10M        90 / 964    91 / 999
// (The tile path, which kernels 2 and 3 would take, at 10M rows: 27000 and 1700.)
bool small_beats_rowsplit(int m, int n, long long nnz)
{
    return m <= 2 * (THREADS / LANES) * device_num_sms() && small_spmv_fits(m, n, nnz, false);
}

int launch_small_spmv(int m, long long nnz, double alpha, const void *val, int val_kind,
                      const int *rowptr, const int *col, const double *x, double beta, double *y,
                      int *status, cudaStream_t stream, bool skip_zero_x)
{
    if (m <= 0) return SBLAS_OK;
    const SmallArgs a{m, (int)nnz, alpha, beta, val, rowptr, col, x, y, status};
    if (skip_zero_x) {
        if (val_kind == VAL_F64) return launch<VAL_F64, true>(a, stream);
        if (val_kind == VAL_PATTERN) return launch<VAL_PATTERN, true>(a, stream);
    } else {
        switch (val_kind) {
        case VAL_F64: return launch<VAL_F64, false>(a, stream);
        case VAL_F32: return launch<VAL_F32, false>(a, stream);
        case VAL_PATTERN: return launch<VAL_PATTERN, false>(a, stream);
        default: break;
        }
    }
    set_error(SBLAS_ERR_ARG, "unknown value kind %d", val_kind);
    return SBLAS_ERR_ARG;
}

int small_spmv_preload_f64()
{
    cudaFuncAttributes fa;
    SBLAS_CUDA_TRY(cudaFuncGetAttributes(&fa, small_spmv_kernel<VAL_F64, false>));
    return SBLAS_OK;
}

}  // namespace sblas
