// Stable bucket scatter by one digit of an int key: the step of this library's
// least-significant-digit sorts (own kernels; no library sort).
//
// One pass over n entries in tiles of T = 256 * ITER, digit
// d(e) = (key(e) >> shift) & (nb - 1), nb <= 2048:
//   bucket_hist_kernel    a CTA counts the digits of a chunk of consecutive
//                         tiles in shared memory and writes, before each tile,
//                         the counts so far: prefix[t][d] inside the chunk,
//                         then the chunk's totals
//   bucket_chunks_kernel  the chunk totals scanned over the chunks, per digit,
//                         and the digits' totals
//   bucket_scatter_kernel per tile: stable ranks of its entries (every warp
//                         walks its 32 * ITER entries in order, finding equal
//                         digits by ballots over the digit's bits and counting
//                         in a warp-private shared table), then one array
//                         after another is put into digit order in shared
//                         memory and written out so that consecutive threads
//                         write consecutive positions of one digit's run
// Every table is digit-contiguous, so all its reads and writes are coalesced.
// Entries keep their input order inside every digit (tiles in order, warps in
// order inside a tile, entries in order inside a warp).  Counts are integers
// and positions are computed, not claimed with atomics: every run produces
// the same output.
//
// Bound: latency.  A tile's phases (ranks, runs, keys, values, columns) wait for
// one another, at 24 warps per SM (registers), and no unit is above 60 % of its
// rate; the stores, one request per 128-byte line that a warp's store touches
// (~27 per 32 entries with three arrays in runs of T / nb = 4), are one
// contributor.  20M entries, 1024 digits, keys, columns and values, before the
// prefetches below: 234 us a pass (a coalesced move of the same bytes 119 us,
// their HBM time 94 us).  Two passes of up to 11 bits beat three of 8 all the
// same: 194 us each at 128 digits.  Equal digits by ballots rather than __match_any_sync, which takes a
// warp's distinct values one after another: 312 -> 289 us in a copy of the
// pass; CTAs of 512 threads (twice the warp-private tables): 326 us.
// CSC to CSR, 20M entries, 1M rows, as a call: 890 -> 528 us; one product of a CSC
// matrix with 4.5M entries: 275 -> 155 us.
#pragma once

#include <atomic>
#include <climits>

#include "launch.cuh"
#include "ptx.cuh"
#include "sblas_internal.h"

namespace sblas {
namespace bsort {
// The kernels here are launched behind one another with programmatic stream
// serialisation and read what the kernel before wrote.  Those reads are plain
// loads (no __restrict__, no __ldg): a load marked as reading constant memory
// could be moved ahead of the wait for that kernel.  (None of them lets its
// successor start before its last CTA exits: with early starts the waiting CTAs
// take slots and shared memory from the running ones, 20M entries 608 -> 617
// us, 4.5M 144 -> 148, small sorts the same; taken before the prefetches.)
// internal linkage: every translation unit that includes this header gets its
// own copy of the kernels (no relocatable device code)
namespace {

constexpr int NW = 8;                   // warps per CTA
constexpr int THREADS = NW * 32;
constexpr int MAXB = 2048;              // digit values per pass (11-bit digits)
constexpr int CHUNK_DIGITS = 8;         // digits per CTA of the chunk scan

// Entries per thread of a pass over n entries: 16 (tiles of 4096, about four
// entries per run at 1024 digits), or fewer where that would leave the three
// CTAs that fit on each of the 152 SMs without a tile.
inline int pass_iter(long long n) { return n >= (1LL << 22) ? 16 : n >= (1LL << 19) ? 8 : 4; }

inline long long num_tiles(long long n, int iter)
{
    const long long t = (long long)THREADS * iter;
    return (n + t - 1) / t;
}

constexpr int MAX_CHUNKS = 1024;        // of the digit counts (bucket_chunks_kernel)

// Tiles per chunk of the digit counts: at most MAX_CHUNKS chunks.
inline int chunk_tiles(long long ntiles)
{
    long long c = (ntiles + MAX_CHUNKS - 1) / MAX_CHUNKS;
    return (int)(c < 1 ? 1 : c);
}

__device__ __forceinline__ int digit_of(int key, int shift, int nb)
{
    return (int)(((unsigned)key >> shift) & (unsigned)(nb - 1));
}

// Width of a table row: the digits, or the eight that one thread scans.
__host__ __device__ inline int table_width(int nb) { return nb < 8 ? 8 : nb; }

// Ranks of this warp's entries among the equal digits before them (batch i,
// then lane), counted in the warp's own table.  d[i] < 0: no entry.
template <int ITER>
__device__ __forceinline__ void rank_digits(const int (&d)[ITER], int bits,
                                            unsigned short *mycnt, int lane, int (&rank)[ITER])
{
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
        const bool valid = d[i] >= 0;
        unsigned peers = __ballot_sync(0xffffffffu, valid);
        rank[i] = 0;
        if (peers == 0u) continue;
#pragma unroll
        for (int b = 0; b < 11; ++b)
            if (b < bits) {
                const bool one = (d[i] >> b) & 1;
                const unsigned m = __ballot_sync(0xffffffffu, one);
                peers &= one ? m : ~m;
            }
        const int base = valid ? (int)mycnt[d[i]] : 0;
        rank[i] = base + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0u) mycnt[d[i]] = (unsigned short)(base + __popc(peers));
        __syncwarp();
    }
}

__device__ __forceinline__ uint4 add_u16(uint4 a, uint4 b)
{
    return make_uint4(__vadd2(a.x, b.x), __vadd2(a.y, b.y), __vadd2(a.z, b.z), __vadd2(a.w, b.w));
}
__device__ __forceinline__ int sum_u16(uint4 v)
{
    const unsigned s = (v.x & 0xffffu) + (v.x >> 16) + (v.y & 0xffffu) + (v.y >> 16) +
                       (v.z & 0xffffu) + (v.z >> 16) + (v.w & 0xffffu) + (v.w >> 16);
    return (int)s;
}
// first[j] = at + the counts before the j-th of eight packed counts
__device__ __forceinline__ void starts_u16(uint4 v, int at, int (&first)[8])
{
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        first[2 * j] = at;
        at += (int)(w[j] & 0xffffu);
        first[2 * j + 1] = at;
        at += (int)(w[j] >> 16);
    }
}
__device__ __forceinline__ uint4 pack_u16(const int (&v)[8])
{
    return make_uint4((unsigned)v[0] | ((unsigned)v[1] << 16), (unsigned)v[2] | ((unsigned)v[3] << 16),
                      (unsigned)v[4] | ((unsigned)v[5] << 16), (unsigned)v[6] | ((unsigned)v[7] << 16));
}
// Sum over the warps of the eight counts of digits 8t .. 8t + 7.
template <int WARPS>
__device__ __forceinline__ uint4 count_u16(const unsigned short *wcnt, int width, int t)
{
    uint4 s = make_uint4(0, 0, 0, 0);
#pragma unroll 8
    for (int k = 0; k < WARPS; ++k)
        s = add_u16(s, reinterpret_cast<const uint4 *>(wcnt + k * width)[t]);
    return s;
}
// The warps' counts of digits 8t .. 8t + 7 become running starts from `run`.
template <int WARPS>
__device__ __forceinline__ void warp_starts_u16(unsigned short *wcnt, int width, int t, uint4 run)
{
#pragma unroll 8
    for (int k = 0; k < WARPS; ++k) {
        uint4 *q = reinterpret_cast<uint4 *>(wcnt + k * width) + t;
        const uint4 c = *q;
        *q = run;
        run = add_u16(run, c);
    }
}

// ---- digit counts ----------------------------------------------------------
template <int ITER>
__global__ void __launch_bounds__(THREADS) bucket_hist_kernel(const int *key,
                                                              long long n, int shift, int nb,
                                                              int ntiles, int per_chunk,
                                                              int *prefix,
                                                              int *chunk_sum)
{
    constexpr int T = THREADS * ITER;
    __shared__ int cnt[MAXB];
    const int width = table_width(nb);
    for (int d = threadIdx.x; d < width; d += THREADS) cnt[d] = 0;
    __syncthreads();
    ptx::griddep_wait();
    const int first = blockIdx.x * per_chunk, last = min(first + per_chunk, ntiles);
    for (int t = first; t < last; ++t) {
        const long long e0 = (long long)t * T + threadIdx.x;
        int k[ITER];
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            k[i] = e0 + i * THREADS < n ? *(key + e0 + i * THREADS) : 0;
        int *row = prefix + (long long)t * width;
        for (int d = threadIdx.x; d < width; d += THREADS) row[d] = cnt[d];
        __syncthreads();   // the counts so far are read before this tile's are added
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (e0 + i * THREADS < n) atomicAdd(&cnt[digit_of(k[i], shift, nb)], 1);
        __syncthreads();
    }
    int *sum = chunk_sum + (long long)blockIdx.x * width;
    for (int d = threadIdx.x; d < width; d += THREADS) sum[d] = cnt[d];
}

// Per digit: chunk_sum becomes the exclusive prefix over the chunks, total[d]
// their sum.  A CTA takes eight digits (32 bytes of a row), eight threads a span
// of chunks, all of its counts read at once and kept in registers: there is
// little to do here but wait for memory, so the round trips count.  4.5M
// entries, two passes: 10 us less than with every span read twice, eight counts
// at a time, by 1024-thread CTAs of 32 digits; such CTAs with the counts in
// registers need a whole idle SM each and cost 14 us more.
__global__ void __launch_bounds__(32 * CHUNK_DIGITS) bucket_chunks_kernel(int width, int nchunks,
                                                                          int *chunk_sum,
                                                                          int *total)
{
    constexpr int SPAN = MAX_CHUNKS / 32;
    __shared__ int part[32][CHUNK_DIGITS + 1];
    ptx::griddep_wait();
    const int j = threadIdx.x % CHUNK_DIGITS, g = threadIdx.x / CHUNK_DIGITS;
    const int d = blockIdx.x * CHUNK_DIGITS + j;
    const int per = (nchunks + 31) / 32;      // <= SPAN
    const int c0 = min(g * per, nchunks), c1 = d < width ? min(c0 + per, nchunks) : c0;
    int x[SPAN];
    int s = 0;
#pragma unroll
    for (int i = 0; i < SPAN; ++i) x[i] = c0 + i < c1 ? chunk_sum[(long long)(c0 + i) * width + d] : 0;
#pragma unroll
    for (int i = 0; i < SPAN; ++i) s += x[i];
    part[g][j] = s;
    __syncthreads();
    // warp w scans the 32 spans of digit w of this CTA
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v = part[lane][w];
    const int own = v;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, k);
        if (lane >= k) v += o;
    }
    part[lane][w] = v - own;
    if (lane == 31 && blockIdx.x * CHUNK_DIGITS + w < width)
        total[blockIdx.x * CHUNK_DIGITS + w] = v;
    __syncthreads();
    int p = part[g][j];
#pragma unroll
    for (int i = 0; i < SPAN; ++i) {
        if (c0 + i < c1) chunk_sum[(long long)(c0 + i) * width + d] = p;
        p += x[i];
    }
}

// Exclusive scan over a CTA of THREADS threads of two sums at once.
struct Two {
    int a, b;
};
__device__ __forceinline__ Two block_scan_two(Two v)
{
    __shared__ int wa[NW], wb[NW];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Two in = v;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const int oa = __shfl_up_sync(0xffffffffu, v.a, k);
        const int ob = __shfl_up_sync(0xffffffffu, v.b, k);
        if (lane >= k) {
            v.a += oa;
            v.b += ob;
        }
    }
    if (lane == 31) {
        wa[w] = v.a;
        wb[w] = v.b;
    }
    __syncthreads();
    Two out{v.a - in.a, v.b - in.b};
#pragma unroll
    for (int k = 0; k < NW; ++k)
        if (k < w) {
            out.a += wa[k];
            out.b += wb[k];
        }
    return out;
}

// ---- exclusive scan of int counts (sums < 2^31) ---------------------------
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;   // 4096

// Exclusive scan of the CTA's SCAN_ITEMS values per thread (in registers,
// consecutive per thread); returns this thread's exclusive prefix and the
// CTA total in *total.
__device__ __forceinline__ int block_exclusive_prefix(int thread_sum, int *total)
{
    __shared__ int warp_tot[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v = thread_sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    if (lane == 31) warp_tot[w] = v;
    __syncthreads();
    int wp = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < SCAN_THREADS / 32; ++k) {
        const int t = warp_tot[k];
        wp += (k < w) ? t : 0;
        tot += t;
    }
    __syncthreads();   // warp_tot may be reused by the caller's next call
    *total = tot;
    return wp + v - thread_sum;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_reduce_kernel(const int *__restrict__ in,
                                                                   long long n,
                                                                   int *__restrict__ sums)
{
    const long long base = (long long)blockIdx.x * SCAN_CHUNK;
    int s = 0;
    for (int i = threadIdx.x; i < SCAN_CHUNK; i += SCAN_THREADS)
        if (base + i < n) s += __ldg(in + base + i);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    __shared__ int ws[SCAN_THREADS / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < SCAN_THREADS / 32; ++k) t += ws[k];
        sums[blockIdx.x] = t;
    }
}

// One CTA: exclusive scan of the chunk sums in place (any count).
__global__ void __launch_bounds__(SCAN_THREADS) scan_sums_kernel(int *__restrict__ sums,
                                                                 int nchunks)
{
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < nchunks; b0 += SCAN_CHUNK) {
        int v[SCAN_ITEMS];
        int ts = 0;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const int i = b0 + threadIdx.x * SCAN_ITEMS + k;
            v[k] = i < nchunks ? sums[i] : 0;
            ts += v[k];
        }
        int tot = 0;
        int p = block_exclusive_prefix(ts, &tot) + carry;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const int i = b0 + threadIdx.x * SCAN_ITEMS + k;
            if (i < nchunks) sums[i] = p;
            p += v[k];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
}

// out[i] = sums[chunk] + exclusive prefix of in inside the chunk (in may
// alias out).  If total != nullptr, the last CTA writes the grand total there.
__global__ void __launch_bounds__(SCAN_THREADS) scan_apply_kernel(const int *in, long long n,
                                                                  const int *__restrict__ sums,
                                                                  int *out, int *total)
{
    const long long base = (long long)blockIdx.x * SCAN_CHUNK;
    int v[SCAN_ITEMS];
    int ts = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + threadIdx.x * SCAN_ITEMS + k;
        v[k] = i < n ? in[i] : 0;
        ts += v[k];
    }
    int tot = 0;
    int p = block_exclusive_prefix(ts, &tot) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + threadIdx.x * SCAN_ITEMS + k;
        if (i < n) out[i] = p;
        p += v[k];
    }
    if (total != nullptr && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
        *total = sums[blockIdx.x] + tot;
}

inline size_t scan_tmp_bytes(long long n)
{
    const long long chunks = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    return sizeof(int) * (size_t)(chunks > 0 ? chunks : 1);
}

// Exclusive scan of n ints (out may equal in); tmp: scan_tmp_bytes(n).
// total (device int*, may be null) receives the sum of all n values.
inline int exclusive_scan(const int *in, int *out, long long n, void *tmp, int *total,
                          cudaStream_t stream)
{
    if (n <= 0) {
        if (total) SBLAS_CUDA_TRY(cudaMemsetAsync(total, 0, sizeof(int), stream));
        return SBLAS_OK;
    }
    const long long chunks = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    if (chunks > INT_MAX) {
        set_error(SBLAS_ERR_ARG, "scan of %lld values too large", n);
        return SBLAS_ERR_ARG;
    }
    int *sums = static_cast<int *>(tmp);
    scan_reduce_kernel<<<(unsigned)chunks, SCAN_THREADS, 0, stream>>>(in, n, sums);
    scan_sums_kernel<<<1, SCAN_THREADS, 0, stream>>>(sums, (int)chunks);
    scan_apply_kernel<<<(unsigned)chunks, SCAN_THREADS, 0, stream>>>(in, n, sums, out, total);
    SBLAS_CUDA_TRY(cudaGetLastError());
    return SBLAS_OK;
}

// ---- stable scatter ---------------------------------------------------------
// What a pass moves: the keys and up to two ints and one double per entry.
// An output that is null is not carried; scatter_pass_iter refuses an output
// without its input, so the kernel tests outputs only.
//   SEG   a is not read but is the segment (column of CSC, row of CSR) of the
//         entry in ptr[0 .. nseg]
//   IDX   b is not read but is the entry's own position
//   POS   pos_out[e] receives entry e's output position
struct Arrays {
    const int *key_in = nullptr, *a_in = nullptr, *b_in = nullptr;
    const double *d_in = nullptr;
    const int *ptr = nullptr;
    int nseg = 0;
    int *key_out = nullptr, *a_out = nullptr, *b_out = nullptr;
    double *d_out = nullptr;
    int *pos_out = nullptr;
};

// Shared memory of a scatter CTA: the staging buffer (8 bytes per entry),
// the warps' digit counts and the digits' output offsets.
template <int ITER>
constexpr size_t scatter_smem_bytes(int width)
{
    return size_t(8) * THREADS * ITER + sizeof(unsigned short) * NW * (size_t)width +
           sizeof(int) * (size_t)width;
}

// Segment of every entry of the tile [t0, t0 + cnt), into seg[0 .. cnt): the
// largest s with ptr[s] <= entry.  The first and last segments are found by
// the whole CTA (a 257-way search, three dependent loads for 4M segments),
// each non-empty segment between them marks its first entry, and every warp
// carries the marks forward over its entries (seg doubles as the marks).
template <int ITER>
__device__ __forceinline__ void tile_segments(const int *ptr, int nseg, long long t0,
                                              int cnt, int *seg, int (&out)[ITER])
{
    constexpr int T = THREADS * ITER;
    constexpr int WSPAN = 32 * ITER;
    __shared__ int wlast[NW];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const long long tl = t0 + cnt - 1;
    for (int i = tid; i < T; i += THREADS) seg[i] = -1;
    // segments holding entries t0 and tl: lo + (probes <= the entry) * step
    int lo = 0, hi = nseg, lo2 = 0, hi2 = nseg;
    while (hi - lo > 1 || hi2 - lo2 > 1) {   // the answers are in [lo, hi), [lo2, hi2)
        // rounded up; written so that no step of it leaves 32 bits at 2^31 - 1
        // segments
        const int st = (hi - lo - 1) / (THREADS + 1) + 1;
        const int st2 = (hi2 - lo2 - 1) / (THREADS + 1) + 1;
        const long long p = lo + (long long)(tid + 1) * st, p2 = lo2 + (long long)(tid + 1) * st2;
        const bool le = p < hi && (long long)*(ptr + p) <= t0;
        const bool le2 = p2 < hi2 && (long long)*(ptr + p2) <= tl;
        const int c = __syncthreads_count(le), c2 = __syncthreads_count(le2);
        lo += c * st;
        hi = lo + min(hi - lo, st);
        lo2 += c2 * st2;
        hi2 = lo2 + min(hi2 - lo2, st2);
    }
    __syncthreads();   // seg is cleared
    for (long long s = (long long)lo + 1 + tid; s <= lo2; s += THREADS) {
        const int b = *(ptr + s), e = *(ptr + s + 1);
        if (e > b && b >= t0 && b <= tl) seg[b - t0] = (int)s;
    }
    __syncthreads();
    int carry = -1;
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
        const int v = seg[w * WSPAN + i * 32 + lane];
        const unsigned m = __ballot_sync(0xffffffffu, v >= 0) & (0xffffffffu >> (31 - lane));
        const int got = __shfl_sync(0xffffffffu, v, m ? 31 - __clz(m) : 0);
        out[i] = m ? got : carry;
        carry = __shfl_sync(0xffffffffu, out[i], 31);
    }
    if (lane == 0) wlast[w] = carry;
    __syncthreads();
    int before = lo;
#pragma unroll
    for (int k = 0; k < NW; ++k)
        if (k < w && wlast[k] >= 0) before = wlast[k];
#pragma unroll
    for (int i = 0; i < ITER; ++i) out[i] = out[i] >= 0 ? out[i] : before;
}

// Runs of a tile's digits: thread t takes digits 8t .. 8t + 7.  The warps'
// counts become the slots of their first entries in the tile's digit order,
// gpos[d] + slot is an entry's output position.
__device__ __forceinline__ void tile_runs(unsigned short *wcnt, int *gpos, int width, int per_chunk,
                                          const int *prefix,
                                          const int *chunk_base,
                                          const int *total)
{
    const int t = threadIdx.x;
    const bool own = 8 * t < width;
    uint4 c = make_uint4(0, 0, 0, 0);
    int tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    Two sum{0, 0};
    if (own) {
        c = count_u16<NW>(wcnt, width, t);
        const int4 lo = reinterpret_cast<const int4 *>(total)[2 * t];
        const int4 hi = reinterpret_cast<const int4 *>(total)[2 * t + 1];
        tot[0] = lo.x, tot[1] = lo.y, tot[2] = lo.z, tot[3] = lo.w;
        tot[4] = hi.x, tot[5] = hi.y, tot[6] = hi.z, tot[7] = hi.w;
        sum.a = sum_u16(c);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum.b += tot[j];
    }
    const Two at = block_scan_two(sum);
    if (!own) return;
    int first[8];
    starts_u16(c, at.a, first);
    warp_starts_u16<NW>(wcnt, width, t, pack_u16(first));
    const int4 *row = reinterpret_cast<const int4 *>(prefix + (long long)blockIdx.x * width) + 2 * t;
    const int4 *crow =
        reinterpret_cast<const int4 *>(chunk_base + (long long)(blockIdx.x / per_chunk) * width) +
        2 * t;
    int b = at.b;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int4 r = row[h], c4 = crow[h];
        const int before[4] = {r.x + c4.x, r.y + c4.y, r.z + c4.z, r.w + c4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            gpos[8 * t + 4 * h + j] = b + before[j] - first[4 * h + j];
            b += tot[4 * h + j];
        }
    }
}

template <bool SEG, bool IDX, bool POS, int ITER>
__global__ void __launch_bounds__(THREADS, 3) bucket_scatter_kernel(
    const Arrays op, long long n, int shift, int nb, int bits, int per_chunk,
    const int *prefix, const int *chunk_base,
    const int *total)
{
    constexpr int T = THREADS * ITER;
    constexpr int WSPAN = 32 * ITER;
    extern __shared__ __align__(16) unsigned char bs_smem[];
    const int width = table_width(nb);
    double *buf = reinterpret_cast<double *>(bs_smem);                        // [T]
    int *buf_i = reinterpret_cast<int *>(buf);
    unsigned short *wcnt = reinterpret_cast<unsigned short *>(buf + T);       // [NW][width]
    int *gpos = reinterpret_cast<int *>(wcnt + NW * width);                   // [width]
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const long long t0 = (long long)blockIdx.x * T;
    const int cnt = (int)min((long long)T, n - t0);
    const int mine = w * WSPAN + lane;       // this thread's entries: mine + 32 i
    for (int i = tid; i < NW * width / 8; i += THREADS)
        reinterpret_cast<uint4 *>(wcnt)[i] = make_uint4(0, 0, 0, 0);
    ptx::griddep_wait();
    int key[ITER];
#pragma unroll
    for (int i = 0; i < ITER; ++i)
        key[i] = mine + 32 * i < cnt ? *(op.key_in + t0 + mine + 32 * i) : 0;
    // The arrays that are moved after the keys on their way to L2 from the start,
    // one prefetch per 64 bytes: a tile's phases wait for their loads one after
    // another, and holding the values in registers meanwhile spills (20M
    // entries 594 -> 691 us of device time).  Prefetched: 594 -> 523, 4.5M entries 142 -> 128 (one
    // prefetch per 128 bytes 562 / 137; a tile of the next wave as well 547 / 133).
    constexpr int PF = 64;
    if (op.d_out)
#pragma unroll
        for (int e = tid * (PF / 8); e < T; e += THREADS * (PF / 8))
            if (e < cnt) ptx::prefetch_l2(op.d_in + t0 + e);
    if constexpr (!SEG)
        if (op.a_out)
#pragma unroll
            for (int e = tid * (PF / 4); e < T; e += THREADS * (PF / 4))
                if (e < cnt) ptx::prefetch_l2(op.a_in + t0 + e);
    __syncthreads();
    unsigned short *mycnt = wcnt + w * width;
    int slot[ITER];
    {
        int d[ITER];
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            d[i] = mine + 32 * i < cnt ? digit_of(key[i], shift, nb) : -1;
        rank_digits<ITER>(d, bits, mycnt, lane, slot);
    }
    __syncthreads();
    tile_runs(wcnt, gpos, width, per_chunk, prefix, chunk_base, total);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITER; ++i)
        if (mine + 32 * i < cnt) {
            const int d = digit_of(key[i], shift, nb);
            slot[i] += mycnt[d];
            if constexpr (POS) op.pos_out[t0 + mine + 32 * i] = gpos[d] + slot[i];
            buf_i[slot[i]] = key[i];
        }
    __syncthreads();
    // output position of the tile's j-th entry in digit order, j = tid + THREADS i
    int pos[ITER];
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
        const int j = tid + THREADS * i;
        pos[i] = 0;
        if (j < cnt) {
            const int k = buf_i[j];
            pos[i] = gpos[digit_of(k, shift, nb)] + j;
            if (op.key_out) op.key_out[pos[i]] = k;
        }
    }
    if (op.d_out) {
        double v[ITER];
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            v[i] = mine + 32 * i < cnt ? *(op.d_in + t0 + mine + 32 * i) : 0.0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (mine + 32 * i < cnt) buf[slot[i]] = v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (tid + THREADS * i < cnt) op.d_out[pos[i]] = buf[tid + THREADS * i];
    }
    if (op.a_out) {
        int v[ITER];
        if constexpr (SEG) {
            __syncthreads();
            tile_segments<ITER>(op.ptr, op.nseg, t0, cnt, buf_i, v);
        } else {
#pragma unroll
            for (int i = 0; i < ITER; ++i)
                v[i] = mine + 32 * i < cnt ? *(op.a_in + t0 + mine + 32 * i) : 0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (mine + 32 * i < cnt) buf_i[slot[i]] = v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (tid + THREADS * i < cnt) op.a_out[pos[i]] = buf_i[tid + THREADS * i];
    }
    if (op.b_out) {
        int v[ITER];
#pragma unroll
        for (int i = 0; i < ITER; ++i) {
            const int e = mine + 32 * i;
            v[i] = IDX ? (int)(t0 + e) : e < cnt ? *(op.b_in + t0 + e) : 0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (mine + 32 * i < cnt) buf_i[slot[i]] = v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITER; ++i)
            if (tid + THREADS * i < cnt) op.b_out[pos[i]] = buf_i[tid + THREADS * i];
    }
}

// ---- one pass ----------------------------------------------------------------
// Scratch: prefix [tiles][nb] | chunk bases [chunks][nb] | totals [nb].
struct PassTables {
    int *prefix = nullptr, *chunk_base = nullptr, *total = nullptr;
    long long tiles = 0;
    int per_chunk = 1;
    long long chunks = 0;
    size_t bytes = 0;
};

inline PassTables pass_tables(long long n, int nb, int iter, void *work)
{
    PassTables t;
    t.tiles = num_tiles(n > 0 ? n : 1, iter);
    t.per_chunk = chunk_tiles(t.tiles);
    t.chunks = (t.tiles + t.per_chunk - 1) / t.per_chunk;
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    const size_t row = 4 * (size_t)table_width(nb);
    const size_t p = up(row * (size_t)t.tiles), c = up(row * (size_t)t.chunks);
    unsigned char *w = static_cast<unsigned char *>(work);
    t.prefix = reinterpret_cast<int *>(w);
    t.chunk_base = reinterpret_cast<int *>(w + p);
    t.total = reinterpret_cast<int *>(w + p + c);
    t.bytes = p + c + up(row);
    return t;
}

inline size_t pass_work_bytes(long long n, int nb, int iter) { return pass_tables(n, nb, iter, nullptr).bytes; }
inline size_t pass_work_bytes(long long n, int nb) { return pass_work_bytes(n, nb, pass_iter(n)); }

inline int bits_for(int nb)   // bits of a digit in [0, nb)
{
    int b = 0;
    while ((1 << b) < nb) ++b;
    return b;
}

// Digit counts of a pass (the first two kernels).
template <int ITER>
int count_digits(const int *key, long long n, int shift, int nb, const PassTables &t,
                 cudaStream_t stream)
{
    SBLAS_CUDA_TRY(launch_pdl(bucket_hist_kernel<ITER>, dim3((unsigned)t.chunks), dim3(THREADS), 0,
                              stream, key, n, shift, nb, (int)t.tiles, t.per_chunk, t.prefix,
                              t.chunk_base));
    const int width = table_width(nb);
    SBLAS_CUDA_TRY(launch_pdl(bucket_chunks_kernel,
                              dim3((width + CHUNK_DIGITS - 1) / CHUNK_DIGITS), dim3(32 * CHUNK_DIGITS), 0,
                              stream, width, (int)t.chunks, t.chunk_base, t.total));
    return SBLAS_OK;
}

// A kernel's dynamic shared memory and the largest carveout (these kernels'
// loads stream, nothing they read is reused through L1), set once per device.
template <class K>
int allow_smem(K kfn, size_t bytes, std::atomic<unsigned long long> &done)
{
    int dev = 0;
    SBLAS_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
    if (bit != 0 && (done.load(std::memory_order_acquire) & bit) != 0) return SBLAS_OK;
    SBLAS_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    SBLAS_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        (int)cudaSharedmemCarveoutMaxShared));
    done.fetch_or(bit, std::memory_order_release);
    return SBLAS_OK;
}

template <bool SEG, bool IDX, bool POS, int ITER>
int scatter_pass_iter(const Arrays &op, long long n, int shift, int nb, void *work,
                      cudaStream_t stream)
{
    if (n <= 0) return SBLAS_OK;
    if (nb < 1 || nb > MAXB || (nb & (nb - 1)) != 0) {
        set_error(SBLAS_ERR_ARG, "bucket pass: %d buckets", nb);
        return SBLAS_ERR_ARG;
    }
    if (op.key_in == nullptr || (op.d_out && !op.d_in) || (op.a_out && !(SEG ? op.ptr : op.a_in)) ||
        (op.b_out && !IDX && !op.b_in)) {
        set_error(SBLAS_ERR_ARG, "sort: null device pointer");
        return SBLAS_ERR_ARG;
    }
    const PassTables t = pass_tables(n, nb, ITER, work);
    static_assert(THREADS * ITER <= 65535, "tile offsets are 16-bit");
    int rc = count_digits<ITER>(op.key_in, n, shift, nb, t, stream);
    if (rc != SBLAS_OK) return rc;
    auto kfn = bucket_scatter_kernel<SEG, IDX, POS, ITER>;
    static std::atomic<unsigned long long> configured{0};
    rc = allow_smem(kfn, scatter_smem_bytes<ITER>(MAXB), configured);
    if (rc != SBLAS_OK) return rc;
    SBLAS_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)t.tiles), dim3(THREADS),
                              scatter_smem_bytes<ITER>(table_width(nb)), stream, op, n, shift,
                              nb, bits_for(nb), t.per_chunk, t.prefix, t.chunk_base, t.total));
    return SBLAS_OK;
}

// One stable pass: the entries of `op` scattered by digit
// (key >> shift) & (nb-1).  work: pass_work_bytes(n, nb) bytes.  Stream-ordered.
template <bool SEG, bool IDX>
int scatter_pass(const Arrays &op, long long n, int shift, int nb, void *work,
                 cudaStream_t stream)
{
    switch (pass_iter(n)) {
    case 16: return scatter_pass_iter<SEG, IDX, false, 16>(op, n, shift, nb, work, stream);
    case 8: return scatter_pass_iter<SEG, IDX, false, 8>(op, n, shift, nb, work, stream);
    default: return scatter_pass_iter<SEG, IDX, false, 4>(op, n, shift, nb, work, stream);
    }
}

// Digit widths of a least-significant-digit sort of keys in [0, key_bound):
// as few passes as digits of at most 11 bits allow, equal widths.
struct LsdPlan {
    int passes;
    int width;
};
inline LsdPlan lsd_plan(long long key_bound)
{
    int bits = 1;
    while (bits < 31 && (1LL << bits) < key_bound) ++bits;
    const int passes = (bits + 10) / 11;
    return LsdPlan{passes, (bits + passes - 1) / passes};
}

}  // namespace
}  // namespace bsort
}  // namespace sblas
