// nbl_csr.cu -- the CSR helpers of a pair list on the device: row starts
// (first_neighbours) and triplets of pairs sharing a first atom
// (triplet_list), with the reference's semantics and output order.
//
// first_neighbours (first_neighbours.cc:15-38): seed[k] = first pair of atom
// k; -1 for atoms before the first atom with pairs, nn (the pair count) after
// the last, and an empty row's seed is the next row's start.  One thread per
// pair writes the seeds between its atom and the previous pair's.
//
// triplet_list (triplet_list.cc:15-34): for each row r = [first_i[r],
// first_i[r+1]), every ordered pair (ij, ik), ij != ik, of the row's pairs
// whose distance is below the cutoff (all of them without distances), ij
// major.  With m kept pairs a row has m (m - 1) triplets; triplet
// q = a (m - 1) + c' of the row is (kept[a], kept[c' + (c' >= a)]).  Two
// passes, one warp per row, with one read of the total in between: count m;
// then list the kept pairs (in shared memory up to kRowKeep of them) and write
// the triplets lane-parallel (consecutive lanes, consecutive triplets).  The
// triplets of 5.4 M pairs of a 132,651-atom crystal, from the pair list: 247 us in
// two calls that each counted and scanned, 116 so.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

#include "nbl_b200.h"
#include "nbl_internal.cuh"
#include "nbl_plan.hh"
#include "nbl_sort.cuh"

namespace nbl {
namespace {

constexpr int kCsrThreads = 256;
constexpr int kCsrWarps = kCsrThreads / 32;
constexpr int kMaxKept = 46340;  // m (m - 1) stays below 2^31

// Kept pairs of a row that a warp lists in shared memory.  A longer row is written by
// a CTA, a warp per first pair (no division), from all of its shared memory, or, beyond
// that, from the output: the last pair's partners are the other kept pairs in order, so
// that part of ik is written first and read for the rest.  The call, for rows that keep
// 140 of 150 pairs 800 us (20,000 rows; 960 from a list of their own in device memory,
// 1,000 with 128 here), 400 of 500 620 (2,000 rows; 800, and 1,170 walking the row for
// every kept pair), 500 of 600 1,230 (2,000; 1,140, 1,720), 540 of 700 1,110 (2,000;
// 1,315, 2,220), 1,900 of 2,000 2.1 ms (300; 9.5, 21.4), 2,400 of 2,600 5.0 (300; 15.1,
// 42.9).
constexpr int kRowKeep = 256;

// Bits that the count leaves beside the total.
constexpr int kTripMany = 1;  // a row keeps more than kMaxKept pairs
constexpr int kTripLong = 2;  // a row keeps more than kRowKeep

__global__ void k_seed_init(int64_t n, int32_t v, int32_t *__restrict__ seed) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k <= n) seed[k] = v;
}

// Atom indices outside [0, n) write nothing (the reference leaves that
// undefined).
constexpr int kSeedPairs = 8;  // pairs a thread (loads in flight): 23.4 -> 16.8 us for 5.4 M

__global__ void __launch_bounds__(256)
k_seed_scatter(const int32_t *__restrict__ i, int64_t nn, int64_t n,
               int32_t *__restrict__ seed) {
    const int64_t k0 = (int64_t)blockIdx.x * (256 * kSeedPairs) + threadIdx.x;
    int32_t at[kSeedPairs], before[kSeedPairs];
#pragma unroll
    for (int u = 0; u < kSeedPairs; u++) {
        const int64_t k = k0 + 256 * u;
        at[u] = k < nn ? i[k] : 0;
        before[u] = k > 0 && k < nn ? i[k - 1] : 0;
    }
#pragma unroll
    for (int u = 0; u < kSeedPairs; u++) {
        const int64_t k = k0 + 256 * u;
        if (k >= nn) return;
        const int64_t cur = at[u];
        if (k == 0) {
            if (cur >= 0 && cur <= n) seed[cur] = 0;
        } else {
            const int64_t prev = before[u];
            if (cur != prev) {
                for (int64_t l = std::max<int64_t>(prev + 1, 0); l <= cur && l <= n; l++)
                    seed[l] = (int32_t)k;
            }
        }
        if (k == nn - 1) {
            for (int64_t l = std::max<int64_t>(cur + 1, 0); l <= n; l++) seed[l] = (int32_t)nn;
        }
    }
}

__device__ __forceinline__ bool kept(const double *d, double cutoff, int64_t p) {
    return d == nullptr || d[p] < cutoff;
}

// Triplets m (m - 1) per row.  Rows that start before 0 (the seeds of atoms
// before the first one with pairs) hold none.
__global__ void __launch_bounds__(kCsrThreads)
k_trip_count(const int32_t *__restrict__ first, int64_t nrows, const double *__restrict__ d,
             double cutoff, int32_t *__restrict__ tcount, int *__restrict__ flags) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * kCsrThreads + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCsrThreads) >> 5;
    for (int64_t r = gw; r < nrows; r += nw) {
        const int64_t b = first[r], e = first[r + 1];
        int m = 0;
        if (b >= 0) {
            for (int64_t p0 = b; p0 < e; p0 += 32) {
                const int64_t p = p0 + lane;
                m += __popc(__ballot_sync(0xffffffffu, p < e && kept(d, cutoff, p)));
            }
        }
        if (lane == 0) {
            if (m > kMaxKept) {
                atomicOr(flags, kTripMany);
                m = 0;
            }
            if (m > kRowKeep) atomicOr(flags, kTripLong);
            tcount[r] = m * (m - 1) > 0 ? m * (m - 1) : 0;
        }
    }
}

// (Eight CTAs per SM: with 61 registers instead of 32 the short rows of 5.4 M pairs took
// 39 us, 33 so.)
__global__ void __launch_bounds__(kCsrThreads, 8)
k_trip_fill(const int32_t *__restrict__ first, int64_t nrows, const double *__restrict__ d,
            double cutoff, const int64_t *__restrict__ toff, const int *__restrict__ flags,
            int32_t *__restrict__ ij, int32_t *__restrict__ ik) {
    __shared__ int32_t keep[kCsrWarps][kRowKeep];
    __shared__ int32_t last;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gw = ((int64_t)blockIdx.x * kCsrThreads + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCsrThreads) >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int64_t r = gw; r < nrows; r += nw) {
        const int64_t b = first[r], e = first[r + 1], tb = toff[r];
        const int t = (int)(toff[r + 1] - tb);
        if (b < 0 || t == 0 || t > kRowKeep * (kRowKeep - 1)) continue;  // (below)
        int m = 0;
        __syncwarp();
        for (int64_t p0 = b; p0 < e; p0 += 32) {
            const int64_t p = p0 + lane;
            const bool k = p < e && kept(d, cutoff, p);
            const unsigned bal = __ballot_sync(full, k);
            const int c = m + __popc(bal & lt);
            if (k && c < kRowKeep) keep[warp][c] = (int32_t)p;
            m += __popc(bal);
        }
        __syncwarp();
        const int m1 = m - 1;
        for (int q = lane; q < t; q += 32) {
            const int a = q / m1;
            const int c1 = q - a * m1;
            const int c = c1 + (c1 >= a ? 1 : 0);
            __stcs(ij + tb + q, keep[warp][a]);
            __stcs(ik + tb + q, keep[warp][c]);
        }
    }
    if (!(*flags & kTripLong)) return;
    // --- long rows, one per CTA ---------------------------------------------------
    int32_t *all = &keep[0][0];
    __syncthreads();
    for (int64_t r = blockIdx.x; r < nrows; r += gridDim.x) {
        const int64_t b = first[r], tb = toff[r];
        const int t = (int)(toff[r + 1] - tb);
        if (b < 0 || t <= kRowKeep * (kRowKeep - 1)) continue;  // (the same for all threads)
        const int m1 = (int)__dsqrt_rn((double)t);  // the kept pairs but one: t = m1 (m1 + 1)
        const bool fits = m1 < kCsrWarps * kRowKeep;
        int32_t *list = ik + tb + (t - m1);         // else: the kept pairs but the last
        if (warp == 0) {
            const int64_t e = first[r + 1];
            int m = 0;
            for (int64_t p0 = b; p0 < e; p0 += 32) {
                const int64_t p = p0 + lane;
                const bool k = p < e && kept(d, cutoff, p);
                const unsigned bal = __ballot_sync(full, k);
                const int c = m + __popc(bal & lt);
                if (k && fits && c <= m1) all[c] = (int32_t)p;
                if (k && !fits && c < m1) list[c] = (int32_t)p;
                if (k && c == m1) last = (int32_t)p;
                m += __popc(bal);
            }
        }
        __syncthreads();
        for (int a = warp; a <= m1; a += kCsrWarps) {  // a warp per first pair
            int32_t *oj = ij + tb + (int64_t)a * m1, *ok = ik + tb + (int64_t)a * m1;
            if (fits) {
                const int va = all[a];
                for (int c = lane; c < m1; c += 32) {
                    __stcs(oj + c, va);
                    __stcs(ok + c, all[c + (c >= a ? 1 : 0)]);
                }
            } else {
                const int va = a < m1 ? list[a] : last;
                for (int c = lane; c < m1; c += 32) {
                    const int k = c + (c >= a ? 1 : 0);
                    __stcs(oj + c, va);
                    if (a < m1) __stcs(ok + c, k < m1 ? list[k] : last);
                }
            }
        }
        __syncthreads();
    }
}

// CTAs: one per `rows` rows, at most eight per SM.
int trip_grid(int64_t nrows, int rows, int dev) {
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return (int)std::max<int64_t>(
        1, std::min<int64_t>((nrows + rows - 1) / rows, (int64_t)nsm * 8));
}

}  // namespace
}  // namespace nbl

using namespace nbl;

#define CSR_CUDA(call, where)                                                  \
    do {                                                                       \
        cudaError_t e_ = (call);                                               \
        if (e_ != cudaSuccess) {                                               \
            status = cuda_status(e_, where);                                   \
            goto done;                                                         \
        }                                                                      \
    } while (0)

extern "C" NBL_API nbl_status nbl_first_neighbours(int64_t n, int64_t npairs,
                                                   const int32_t *first, int32_t *seed,
                                                   void *stream) {
    if (n < 0 || npairs < 0 || !seed || (npairs > 0 && !first))
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "bad first_neighbours arguments");
    if (n >= INT32_MAX || npairs >= INT32_MAX)
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "first_neighbours supports < 2^31 rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_seed_init<<<(unsigned)((n + 1 + 255) / 256), 256, 0, st>>>(n, npairs > 0 ? -1 : 0,
                                                                 seed);
    count_launch();
    if (npairs > 0) {
        k_seed_scatter<<<(unsigned)((npairs + 256 * kSeedPairs - 1) / (256 * kSeedPairs)), 256, 0,
                         st>>>(first, npairs, n, seed);
        count_launch();
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? NBL_SUCCESS : cuda_status(e, "first_neighbours");
}

extern "C" NBL_API nbl_status nbl_triplet_count(int64_t nfirst, const int32_t *first_i,
                                                const double *absdist, double cutoff,
                                                int64_t *row_offsets, int64_t *ntriplets,
                                                void *stream) {
    if (!ntriplets || nfirst < 0 || (nfirst > 0 && (!first_i || !row_offsets)))
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "bad triplet_list arguments");
    *ntriplets = 0;
    if (nfirst < 2) return NBL_SUCCESS;
    if (nfirst >= INT32_MAX)
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "triplet_list supports < 2^31 rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    nbl_status status = NBL_SUCCESS;
    const int64_t nrows = nfirst - 1;
    int dev = 0;
    cudaGetDevice(&dev);
    char *scratch = nullptr;
    int64_t host[2] = {0, 0};  // pageable: the copy completes before it returns
    size_t bytes = 0;
    auto add = [&](size_t b) {
        const size_t o = bytes;
        bytes += (b + 255) & ~size_t(255);
        return o;
    };
    const size_t o_t = add(sizeof(int32_t) * nrows);
    const size_t o_s = add(sizeof(int64_t) * scan_scratch_elems(nrows + 1));
    {
        cudaMemPool_t pool = nullptr;
        CSR_CUDA(scratch_pool(dev, &pool), "triplet scratch pool");
        CSR_CUDA(cudaMallocFromPoolAsync((void **)&scratch, bytes, pool, st), "triplet scratch");
        int32_t *tcount = reinterpret_cast<int32_t *>(scratch + o_t);
        // behind the total, so that one copy reads both: the scan's ticket, the flags
        int *word = reinterpret_cast<int *>(row_offsets + nfirst);
        CSR_CUDA(cudaMemsetAsync(word, 0, sizeof(int64_t), st), "memset");
        k_trip_count<<<trip_grid(nrows, kCsrWarps, dev), kCsrThreads, 0, st>>>(first_i, nrows, absdist,
                                                                    cutoff, tcount, word + 1);
        count_launch();
        CSR_CUDA(cudaGetLastError(), "triplet count");
        CSR_CUDA(exclusive_scan_i32_i64(tcount, nrows, row_offsets,
                                        reinterpret_cast<int64_t *>(scratch + o_s), st,
                                        word),
                 "scan");
        CSR_CUDA(cudaMemcpyAsync(host, row_offsets + nrows, 2 * sizeof(int64_t),
                                 cudaMemcpyDeviceToHost, st),
                 "read count");
        CSR_CUDA(cudaStreamSynchronize(st), "triplet count");
        if ((host[1] >> 32) & kTripMany) {
            status = set_error(NBL_ERROR_INVALID_ARGUMENT,
                               "triplet_list: a row keeps more than %d pairs", kMaxKept);
            goto done;
        }
        *ntriplets = host[0];
    }
done:
    if (scratch) cudaFreeAsync(scratch, st);
    return status;
}

extern "C" NBL_API nbl_status nbl_triplet_fill(int64_t nfirst, const int32_t *first_i,
                                               const double *absdist, double cutoff,
                                               const int64_t *row_offsets, int32_t *ij,
                                               int32_t *ik, void *stream) {
    if (nfirst < 0 || (nfirst > 1 && (!first_i || !row_offsets || !ij || !ik)))
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "bad triplet_list arguments");
    if (nfirst < 2) return NBL_SUCCESS;
    int dev = 0;
    cudaGetDevice(&dev);
    k_trip_fill<<<trip_grid(nfirst - 1, 1, dev), kCsrThreads, 0,
                  static_cast<cudaStream_t>(stream)>>>(
        first_i, nfirst - 1, absdist, cutoff, row_offsets,
        reinterpret_cast<const int *>(row_offsets + nfirst) + 1, ij, ik);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? NBL_SUCCESS : cuda_status(e, "triplet fill");
}

extern "C" NBL_API nbl_status nbl_triplet_list(int64_t nfirst, const int32_t *first_i,
                                               const double *absdist, double cutoff,
                                               int32_t *ij, int32_t *ik, int64_t capacity,
                                               int64_t *ntriplets, void *stream) {
    if (!ntriplets || nfirst < 0 || (nfirst > 0 && !first_i))
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "bad triplet_list arguments");
    *ntriplets = 0;
    if (nfirst < 2) return NBL_SUCCESS;
    if (nfirst >= INT32_MAX)
        return set_error(NBL_ERROR_INVALID_ARGUMENT, "triplet_list supports < 2^31 rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    nbl_status status = NBL_SUCCESS;
    int64_t *off = nullptr;
    int dev = 0;
    cudaGetDevice(&dev);
    {
        cudaMemPool_t pool = nullptr;
        CSR_CUDA(scratch_pool(dev, &pool), "triplet scratch pool");
        CSR_CUDA(cudaMallocFromPoolAsync((void **)&off, sizeof(int64_t) * (nfirst + 1), pool, st),
                 "triplet scratch");
        status = nbl_triplet_count(nfirst, first_i, absdist, cutoff, off, ntriplets, stream);
        if (status != NBL_SUCCESS || !ij || !ik || *ntriplets == 0) goto done;
        if (capacity < *ntriplets) {
            status = set_error(NBL_ERROR_CAPACITY, "triplet_list: %lld triplets, capacity %lld",
                               (long long)*ntriplets, (long long)capacity);
            goto done;
        }
        status = nbl_triplet_fill(nfirst, first_i, absdist, cutoff, off, ij, ik, stream);
    }
done:
    if (off) cudaFreeAsync(off, st);
    return status;
}
