// Internal declarations shared by the CUDA translation units of
// libsblas_gb300.so.  Nothing here is part of the public C ABI
// (include/sblas_gb300.h and include/spmv_kernel.h are).
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

#include "../../include/sblas_gb300.h"

namespace sblas {

// ---- error state: thread-local status readable through sblas_last_error ----
void set_error(int code, const char *fmt, ...);
void clear_error();
int last_status();

#define SBLAS_CUDA_TRY(expr)                                                          \
    do {                                                                              \
        cudaError_t sblas_e_ = (expr);                                                \
        if (sblas_e_ != cudaSuccess) {                                                \
            ::sblas::set_error(SBLAS_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,      \
                               cudaGetErrorString(sblas_e_), __FILE__, __LINE__);    \
            return SBLAS_ERR_CUDA;                                                    \
        }                                                                             \
    } while (0)

// ---- nnz-tile engine (the load-balanced CSR kernel) ----------------------
// A tile is TILE_THREADS * sigma consecutive nonzeros.  Workspace per call:
//   status[1]             device error flag (bounded waits), first 256 bytes
//   row_part[ntiles + 1]  first owned row of every tile (int32)
//   carry[ntiles]         FP64 partial of the row that continues past the tile
struct TileShape {
    int threads;   // threads per CTA
    int sigma;     // nonzeros per thread
    long long tile() const { return (long long)threads * sigma; }
};

// Shapes compiled into the library (sigma odd: conflict-free shared reads).
int tile_shape_count();
TileShape tile_shape_at(int i);
int tile_shape_index(int sigma);   // -1 if not compiled

size_t tile_workspace_bytes(long long nnz, int sigma);

// Value storage of the matrix:  0 = FP64, 1 = FP32 (widened to FP64, products
// and sums in FP64), 2 = pattern (no value array; every stored entry is 1).
enum ValueKind { VAL_F64 = 0, VAL_F32 = 1, VAL_PATTERN = 2 };

// Launches partition + tile kernel + carry fix-up on `stream`.
// `work` must hold tile_workspace_bytes(nnz, sigma) bytes, 256-byte aligned.
// analysed = true: the partition of `work` was computed by
// launch_tile_analyse for this row pointer and sigma (skipped here).
// auto_shape: the caller gave no shape (small matrices then need no tiles).
// skip_zero_x: nonzeros whose x entry is zero are left out (spMspV), and col
// and val may be longer than rowptr[m]; sigma 11, FP64 or pattern-only.
// reset_status = false keeps the workspace's status word as it is (a call
// made of several launches on one workspace clears it once, at its start).
int launch_tile_spmv(int m, int n, long long nnz, double alpha, const void *val,
                     int val_kind, const int *rowptr, const int *col, const double *x,
                     double beta, double *y, int sigma, void *work, cudaStream_t stream,
                     bool analysed = false, bool reset_status = true, bool skip_zero_x = false,
                     bool auto_shape = false);
// Tiles [t0, t1) of the product (and the fix-up of the rows that end in them)
// after launch_tile_analyse on the same workspace: a caller that receives the
// matrix in pieces runs each as it arrives, in order.  tile_count: the tiles of
// 128 * sigma nonzeros.
int tile_count(long long nnz, int sigma);
int *tile_workspace_part(void *work);   // the partition, tile_count + 1 entries
int launch_tile_range(int m, int n, long long nnz, double alpha, const void *val, int val_kind,
                      const int *rowptr, const int *col, const double *x, double beta, double *y,
                      int sigma, void *work, cudaStream_t stream, int t0, int t1,
                      bool reset_status, bool skip_zero_x = false);
// Status word of a tile workspace (0 = every wait completed), copied to *out
// (host memory that stays until the stream has completed) in stream order.
int tile_workspace_status(void *work, int *out, cudaStream_t stream);
// The sticky per-device word (any tile launch that gave up a wait), read
// after `stream` completes; clear = reset it to 0.
int tile_sticky_status(cudaStream_t stream, bool clear, int *out);
// Bounded-wait limit of the tile kernels (0 = the default, 2 s) and the
// test hook that keeps the producer warp from staging (waits then run out).
// The tile kernel over several matrices in one launch (the batched form
// with one right-hand side): global tiles [0, ntiles), matrix i owning
// tiles [tile0s[i], tile0s[i+1]) and partition entries part[part_off_i ..
// part_off_i + its tiles]; every matrix has at least one tile.  mats: device
// array of descriptors written by fill_multi_mat.
struct MultiTileLaunch {
    const void *mats;
    const int *tile0s;   // [nmat + 1]
    int nmat;
    int ntiles;
    const int *part;
    double *carry;       // [ntiles]
    int *status;
};
int multi_tile_sigma();
size_t multi_tile_count(long long nnz);   // tiles of one matrix (1 when nnz == 0)
size_t multi_mat_bytes();
void fill_multi_mat(void *dst, const void *val, const int *rowptr, const int *col,
                    const double *x, double *y, long long nnz, int m, int tile0, int part_off,
                    double alpha, double beta, int val_kind);
int launch_multi_tile_spmv(const MultiTileLaunch &L, int val_kind, cudaStream_t stream);
// The tile partition of one matrix into part[0 .. ntiles] (nnz > 0).
int launch_tile_partition(int m, long long nnz, const int *rowptr, int sigma, int *part,
                          cudaStream_t stream);
// Configures (under lazy module loading: loads) every kernel of an FP64
// tile SpMV of shape sigma on the current device.
int tile_preload_f64(int sigma);
void set_wait_limit_ns(unsigned long long ns);
void set_test_stall(int on);
int launch_tile_analyse(int m, long long nnz, const int *rowptr, int sigma, void *work,
                        cudaStream_t stream);

// Small matrices (spmv_small.cu): one launch, no workspace.  Callers that
// leave the tile shape to the library take it where small_spmv_fits.
// nnz: entries of val and col (none past them is read).  status: cleared, or
// null.  skip_zero_x as in launch_tile_spmv.
bool small_spmv_fits(int m, int n, long long nnz, bool analysed);
bool small_beats_rowsplit(int m, int n, long long nnz);   // kernel 1
int launch_small_spmv(int m, long long nnz, double alpha, const void *val, int val_kind,
                      const int *rowptr, const int *col, const double *x, double beta, double *y,
                      int *status, cudaStream_t stream, bool skip_zero_x = false);
int small_spmv_preload_f64();

// Row-split kernel (one sub-warp per row; kernel version 1).
int launch_rowsplit_spmv(int m, int n, long long nnz, double alpha, const double *val,
                         const int *rowptr, const int *col, const double *x, double beta,
                         double *y, cudaStream_t stream, bool skip_zero_x = false);

// y[i] = beta * y[i] (beta == 0 writes exact zeros), for m == 0 / nnz == 0.
int launch_scale_y(int m, double beta, double *y, cudaStream_t stream);

// ---- format conversion (setup kernels) ------------------------------------
// Row-sorted COO row indices -> CSR row pointer (atomic-free boundary scan).
// work: a tile workspace of (nnz, sigma) that receives the row pointer's tile
// partition as well (instead of launch_tile_analyse); row arrays for which
// coo_partition_fits (16-byte aligned) only.
bool coo_partition_fits(const int *coo_row);
int launch_coo_rows_to_rowptr(int m, long long nnz, const int *coo_row, int *rowptr,
                              cudaStream_t stream, int sigma = 0, void *work = nullptr);
// CSC -> CSR transpose (stable: columns ascending inside each row).
size_t csc_to_csr_workspace_bytes(int m, int n, long long nnz);
// CSR structure of A -> CSR structure of A^T plus the permutation of values.
size_t csr_transpose_workspace_bytes(int m, int n, long long nnz);
int launch_csr_transpose(int m, int n, long long nnz, const int *rowptr, const int *col,
                         int *t_rowptr, int *t_col, int *perm, void *work, size_t work_bytes,
                         cudaStream_t stream);
int launch_gather_values(long long nnz, int val_kind, const void *src, const int *perm, void *dst,
                         cudaStream_t stream);
// spMspV's x-zero filter: CSR of the nonzeros with x[col] != 0.
size_t csr_filter_x_workspace_bytes(long long nnz);
int launch_csr_filter_x(int m, long long nnz, const int *rowptr, const int *col,
                        const double *val, const double *x, int *orowptr, int *ocol,
                        double *oval, void *work, size_t work_bytes, cudaStream_t stream);
int launch_csc_to_csr(int m, int n, long long nnz, const double *csc_val,
                      const int *csc_colptr, const int *csc_row, double *csr_val,
                      int *csr_rowptr, int *csr_col, void *work, size_t work_bytes,
                      cudaStream_t stream);

// y = alpha*A*x + beta*y with A in CSC (atomic-free, deterministic):
// inspector (row-ordered structure + tile partition into `work`) and executor
// (values into row order + tile kernel).  With values, the inspector is the
// one-shot product's: they are sorted along, and the executor is then called
// with val = nullptr.  Without, it is an analysis reused for many products:
// the permutation and the staging indices that the executor moves each
// product's values through.  work: cscmv_workspace_bytes, 256-byte aligned;
// csc_tile_workspace: the tile workspace inside it (its status word).
size_t cscmv_workspace_bytes(int m, int n, long long nnz);
int launch_csc_analyse(int m, int n, long long nnz, const int *colptr, const int *rowidx,
                       const double *val, void *work, size_t work_bytes, cudaStream_t stream);
int launch_csc_bind_values(int m, int n, long long nnz, const double *val, void *work,
                           size_t work_bytes, cudaStream_t stream);
int launch_cscmv_analysed(int m, int n, long long nnz, double alpha, const double *val,
                          const double *x, double beta, double *y, void *work,
                          size_t work_bytes, cudaStream_t stream);
// keep_analysis: the work of a pattern of up to 2^20 entries holds an analysis afterwards
int launch_cscmv(int m, int n, long long nnz, double alpha, const double *val,
                 const int *colptr, const int *rowidx, const double *x, double beta, double *y,
                 void *work, size_t work_bytes, bool keep_analysis, cudaStream_t stream);
void *csc_tile_workspace(void *work, int m, int n, long long nnz);
// Stable sort of COO entries by keys in [0, key_bound), carrying the other
// index and the value (bucket_sort.cuh passes).  Workspace:
// coo_sort_workspace_bytes.
size_t coo_sort_workspace_bytes(int key_bound, long long nnz);
int launch_coo_sort(int key_bound, long long nnz, const int *keys, const int *other,
                    const double *val, int *keys_out, int *other_out, double *val_out,
                    void *work, size_t work_bytes, cudaStream_t stream);
// out_i[p] = in_i[perm[p]], out_d[p] = in_d[perm[p]] (either output may be null).
int launch_gather(long long nnz, const int *perm, const int *in_i, int *out_i,
                  const double *in_d, double *out_d, cudaStream_t stream);

// ---- per-device resources used by the host (drop-in) entry points --------
constexpr int kPipeChunks = 4;   // chunks of the host-array entry points' copy/compute overlap
struct DeviceContext {
    int device = -1;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t copy_stream = nullptr;   // host -> device copies overlapping the kernels
    cudaEvent_t ev[6] = {};
    // of a chunked host call: copies done (row pointer, each chunk) and kernels
    // done (partition, each chunk)
    cudaEvent_t chunk_ev[kPipeChunks + 1] = {};
    cudaEvent_t run_ev[kPipeChunks + 1] = {};
    int *host_word = nullptr;   // pinned: a launch's status word (made by the first host-array call)
};
// Returns the context of the current device (created on first use, which may be
// inside a stream capture: nothing in it allocates memory).
DeviceContext *device_context();

// Grow-only device scratch buffers owned by the context (slot 0..15).
void *device_scratch(int slot, size_t bytes);

int default_sigma_for(int m, long long nnz);
int csr5_sigma_for(int m, long long nnz);
int device_num_sms();

}  // namespace sblas
