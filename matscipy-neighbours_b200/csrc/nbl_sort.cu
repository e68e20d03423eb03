// nbl_sort.cu -- hand-written device exclusive scan and stable LSD radix sort.
//
// Replace the reference's CUB calls (src/libneighbours/device_primitives.cc:
// 31-86: DeviceScan::ExclusiveSum with a temp cudaMalloc and two blocking D2H
// reads per call; DeviceRadixSort::SortPairs).  Here nothing allocates or
// synchronises: all scratch comes from the caller's workspace, so the whole
// pipeline can be captured in a CUDA graph.
//
// Atoms by cell (cell_order): where the cells are numbered densely the binning
// kernel counts them (and each atom's arrival in its cell); a scan gives the
// slices, one kernel drops every atom into its slice in arrival order, and the
// gather ranks an atom among its cell's by index, which restores the ascending
// order.  The ranking reads every atom of a cell for every atom of it, as often as the
// count of an isolated cell does and a 27th of what it does in a bulk; above kRankAtoms
// atoms per cell on average the radix sort takes over (one crowded cell among many
// stays with the ranking: 10,000 atoms there take 0.2 ms of it, the count 1 ms).
// Against two radix passes, init to gather: 13 -> 6 launches, 62 -> 36 us on the
// device for a 200,000-atom gas, 33 -> 20 us for 10,007 atoms.
//
// Scan: three-phase (tile reduce -> recursive scan of tile sums -> tile scan
// with carry-in); no inter-block waiting, so no spin loops at all.
// Sort: as few passes as digits of up to 10 bits allow (a 17-bit dense cell
// key takes two passes of 9 bits); per pass one histogram kernel, one scan of the
// digit-major histogram and one stable scatter kernel.  Stability (needed so
// that the atoms of one cell stay in ascending index order, exactly as the
// reference's counting sort leaves them) comes from ranking keys in index
// order inside each tile with __match_any_sync.
#include <cstdint>

#include <cuda_runtime.h>

#include "nbl_internal.cuh"
#include "nbl_sort.cuh"

namespace nbl {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T &total, T *s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    T incl = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        T w = lane < nwarps ? s_warp[lane] : T(0);
        T wi = warp_incl_scan(w);
        if (lane < nwarps) s_warp[lane] = wi - w;
        if (lane == nwarps - 1) s_warp[32] = wi;
    }
    __syncthreads();
    T r = incl - v + s_warp[warp];
    total = s_warp[32];
    __syncthreads();
    return r;
}

template <typename Tin, typename Tacc>
__global__ void __launch_bounds__(kScanThreads)
k_scan_reduce(const Tin *__restrict__ in, int64_t n, Tacc *__restrict__ sums) {
    __shared__ Tacc s_warp[33];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    Tacc acc = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        int64_t idx = base + (int64_t)it * kScanThreads + threadIdx.x;
        if (idx < n) acc += (Tacc)in[idx];
    }
    Tacc total;
    block_excl_scan<Tacc>(acc, total, s_warp);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// k_scan_reduce and, in the block that finishes last, the exclusive scan of the
// tile sums: two launches a scan instead of three.  (The last block is told by
// a counter, which it clears again; nobody waits.)
template <typename Tin, typename Tacc>
__global__ void __launch_bounds__(kScanThreads)
k_scan_sums(const Tin *__restrict__ in, int64_t n, Tacc *carry, int *ticket) {
    __shared__ Tacc s_warp[33];
    __shared__ int s_last;
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    Tacc acc = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        int64_t idx = base + (int64_t)it * kScanThreads + threadIdx.x;
        if (idx < n) acc += (Tacc)in[idx];
    }
    Tacc total;
    block_excl_scan<Tacc>(acc, total, s_warp);
    if (threadIdx.x == 0) {
        __stcg(carry + blockIdx.x, total);
        __threadfence();
        s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    Tacc run = 0;
    for (int t0 = 0; t0 < (int)gridDim.x; t0 += kScanTile) {
        Tacc v[kScanItems], local = 0;
#pragma unroll
        for (int it = 0; it < kScanItems; it++) {
            const int idx = t0 + (int)threadIdx.x * kScanItems + it;
            v[it] = idx < (int)gridDim.x ? __ldcg(carry + idx) : Tacc(0);
            local += v[it];
        }
        Tacc sum;
        Tacc at = run + block_excl_scan<Tacc>(local, sum, s_warp);
#pragma unroll
        for (int it = 0; it < kScanItems; it++) {
            const int idx = t0 + (int)threadIdx.x * kScanItems + it;
            if (idx < (int)gridDim.x) carry[idx] = at;
            at += v[it];
        }
        run += sum;
    }
    if (threadIdx.x == 0) *ticket = 0;
}

// Cell counts -> cell slices (first, end), one tile (blocked), with the tile's
// carry-in.
__global__ void __launch_bounds__(kScanThreads)
k_cell_slices(const int32_t *__restrict__ count, int64_t n, int2 *__restrict__ table,
              const int32_t *__restrict__ carry) {
    __shared__ int32_t s_warp[33];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int32_t local = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        v[it] = base + it < n ? count[base + it] : 0;
        local += v[it];
    }
    int32_t total;
    int32_t run = block_excl_scan<int32_t>(local, total, s_warp);
    if (carry) run += carry[blockIdx.x];
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        if (base + it < n) table[base + it] = make_int2(run, run + v[it]);
        run += v[it];
    }
}

// Atom t to the slot of its cell that its arrival gave it.
__global__ void __launch_bounds__(256)
k_cell_place(const uint32_t *__restrict__ keys, const int32_t *__restrict__ arrival,
             const int2 *__restrict__ table, int64_t natoms, int32_t *__restrict__ order) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < natoms) order[table[keys[t]].x + arrival[t]] = (int32_t)t;
}

// Exclusive scan of one tile (blocked: thread t owns items t*8 .. t*8+7) with
// an optional carry-in per tile; writes out[n] = grand total when
// `write_total`.
template <typename Tin, typename Tacc>
__global__ void __launch_bounds__(kScanThreads)
k_scan_tile(const Tin *__restrict__ in, int64_t n, Tacc *__restrict__ out,
            const Tacc *__restrict__ carry, int write_total) {
    __shared__ Tacc s_warp[33];
    const int64_t base = (int64_t)blockIdx.x * kScanTile +
                         (int64_t)threadIdx.x * kScanItems;
    Tacc v[kScanItems];
    Tacc local = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        int64_t idx = base + it;
        v[it] = idx < n ? (Tacc)in[idx] : Tacc(0);
        local += v[it];
    }
    Tacc total;
    Tacc run = block_excl_scan<Tacc>(local, total, s_warp);
    const Tacc c = carry ? carry[blockIdx.x] : Tacc(0);
    run += c;
#pragma unroll
    for (int it = 0; it < kScanItems; it++) {
        int64_t idx = base + it;
        if (idx < n) out[idx] = run;
        run += v[it];
    }
    if (write_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
        out[n] = c + total;
}

}  // namespace

int64_t scan_scratch_elems(int64_t n) {
    int64_t total = 0;
    while (n > kScanTile) {
        int64_t tiles = (n + kScanTile - 1) / kScanTile;
        total += 2 * tiles + 1;
        n = tiles;
    }
    return total + 1;
}

template <typename Tin, typename Tacc>
static cudaError_t scan_rec(const Tin *in, int64_t n, Tacc *out, int write_total,
                            Tacc *scratch, cudaStream_t st, int *ticket = nullptr) {
    if (n <= 0) {
        if (write_total) return cudaMemsetAsync(out, 0, sizeof(Tacc), st);
        return cudaSuccess;
    }
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles == 1) {
        k_scan_tile<Tin, Tacc><<<1, kScanThreads, 0, st>>>(in, n, out, nullptr,
                                                          write_total);
        count_launch();
        return cudaGetLastError();
    }
    Tacc *sums = scratch;
    Tacc *carry = scratch + tiles;
    if (ticket != nullptr) {
        k_scan_sums<Tin, Tacc><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, carry, ticket);
        count_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        k_scan_tile<Tin, Tacc><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, out, carry,
                                                                       write_total);
        count_launch();
        return cudaGetLastError();
    }
    k_scan_reduce<Tin, Tacc><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, sums);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = scan_rec<Tacc, Tacc>(sums, tiles, carry, 0, scratch + 2 * tiles + 1, st);
    if (e != cudaSuccess) return e;
    k_scan_tile<Tin, Tacc><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, out, carry,
                                                                   write_total);
    count_launch();
    return cudaGetLastError();
}

cudaError_t exclusive_scan_i32_i64(const int32_t *in, int64_t n, int64_t *out,
                                   int64_t *scratch, cudaStream_t st, int *ticket) {
    return scan_rec<int32_t, int64_t>(in, n, out, 1, scratch, st, ticket);
}

cudaError_t cell_order(const uint32_t *keys, const int32_t *arrival, const int32_t *count,
                       int64_t natoms, int64_t ncells, int32_t *carry, int *ticket, int2 *table,
                       int32_t *order, cudaStream_t st) {
    if (natoms <= 0 || ncells <= 0) return cudaSuccess;
    const int64_t tiles = (ncells + kScanTile - 1) / kScanTile;
    if (tiles > 1) {
        k_scan_sums<int32_t, int32_t>
            <<<(unsigned)tiles, kScanThreads, 0, st>>>(count, ncells, carry, ticket);
        count_launch();
    }
    k_cell_slices<<<(unsigned)tiles, kScanThreads, 0, st>>>(count, ncells, table,
                                                            tiles > 1 ? carry : nullptr);
    count_launch();
    k_cell_place<<<(unsigned)((natoms + 255) / 256), 256, 0, st>>>(keys, arrival, table, natoms,
                                                                   order);
    count_launch();
    return cudaGetLastError();
}

cudaError_t exclusive_scan_i32_i32(const int32_t *in, int64_t n, int32_t *out,
                                   int32_t *scratch, cudaStream_t st) {
    return scan_rec<int32_t, int32_t>(in, n, out, 0, scratch, st);
}

// ---- radix sort -----------------------------------------------------------

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Tiles of 1024 keys: small and mid-sized inputs get enough CTAs to fill the
// GPU (measured on a B200: count phase of 131,072 atoms 0.159 -> 0.146 ms,
// of 16,384 atoms 0.108 -> 0.095 ms against 4096-key tiles; 1M atoms
// unchanged).
constexpr int kSortIters = 4;                                // per warp
constexpr int kSortTile = kSortThreads * kSortIters;         // 1024
constexpr int kDigitMax = 10;                 // bits per pass (at most)
constexpr int kRadix = 1 << kDigitMax;        // bins of the widest pass

// Per-tile digit histogram; `nb` = 1 << digit bits of this pass.
__global__ void __launch_bounds__(kSortThreads)
k_radix_hist(const uint32_t *__restrict__ keys, int64_t n, int shift, int nb,
             int32_t *__restrict__ hist, int ntiles) {
    __shared__ int32_t s_cnt[kRadix];
    for (int d = threadIdx.x; d < nb; d += kSortThreads) s_cnt[d] = 0;
    __syncthreads();
    const uint32_t mask = (uint32_t)nb - 1u;
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int it = 0; it < kSortIters; it++) {
        int64_t idx = base + (int64_t)it * kSortThreads + threadIdx.x;
        if (idx < n) atomicAdd(&s_cnt[(keys[idx] >> shift) & mask], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < nb; d += kSortThreads)
        hist[(int64_t)d * ntiles + blockIdx.x] = s_cnt[d];
}

__global__ void __launch_bounds__(kSortThreads)
k_radix_scatter(const uint32_t *__restrict__ kin, const int32_t *__restrict__ vin,
                uint32_t *__restrict__ kout, int32_t *__restrict__ vout, int64_t n,
                int shift, int nb, const int32_t *__restrict__ hoff, int ntiles) {
    __shared__ int32_t s_wc[kSortWarps][kRadix];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < nb; d += kSortThreads)
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) s_wc[w][d] = 0;
    __syncthreads();
    const uint32_t mask = (uint32_t)nb - 1u;

    const unsigned lt = (1u << lane) - 1u;
    const int64_t wbase = (int64_t)blockIdx.x * kSortTile + (int64_t)warp * (32 * kSortIters);
    uint32_t key[kSortIters];
    int32_t val[kSortIters];
    int32_t rank[kSortIters];
#pragma unroll
    for (int it = 0; it < kSortIters; it++) {
        const int64_t idx = wbase + it * 32 + lane;
        const bool valid = idx < n;
        key[it] = valid ? kin[idx] : 0u;
        val[it] = valid ? vin[idx] : 0;
        // Invalid lanes get a private pseudo-digit so they never match.
        const uint32_t d = valid ? ((key[it] >> shift) & mask) : (kRadix + lane);
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        int r = 0;
        if (valid) r = s_wc[warp][d] + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) s_wc[warp][d] += __popc(peers);
        __syncwarp();
        rank[it] = r;
    }
    __syncthreads();
    // Exclusive prefix over warps, per digit.
    for (int d = threadIdx.x; d < nb; d += kSortThreads) {
        int32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
            int32_t c = s_wc[w][d];
            s_wc[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortIters; it++) {
        const int64_t idx = wbase + it * 32 + lane;
        if (idx < n) {
            const uint32_t d = (key[it] >> shift) & mask;
            const int64_t pos = (int64_t)hoff[(int64_t)d * ntiles + blockIdx.x] +
                                s_wc[warp][d] + rank[it];
            kout[pos] = key[it];
            vout[pos] = val[it];
        }
    }
}

}  // namespace

int64_t radix_hist_elems(int64_t n) {
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    return tiles * kRadix;
}

cudaError_t radix_sort_pairs(uint32_t *keys, int32_t *vals, uint32_t *keys_alt,
                             int32_t *vals_alt, int64_t n, int bits,
                             int32_t *hist, int32_t *hist_scan,
                             int32_t *scan_scratch, cudaStream_t st,
                             bool *result_in_alt) {
    *result_in_alt = false;
    if (n <= 1 || bits <= 0) return cudaSuccess;
    const int ntiles = (int)((n + kSortTile - 1) / kSortTile);
    uint32_t *ka = keys, *kb = keys_alt;
    int32_t *va = vals, *vb = vals_alt;
    // As few passes as digits of at most kDigitMax bits allow, of equal width.
    const int passes = (bits + kDigitMax - 1) / kDigitMax;
    const int digit = (bits + passes - 1) / passes;
    const int nb = 1 << digit;
    for (int shift = 0; shift < bits; shift += digit) {
        k_radix_hist<<<ntiles, kSortThreads, 0, st>>>(ka, n, shift, nb, hist, ntiles);
        count_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        e = exclusive_scan_i32_i32(hist, (int64_t)ntiles * nb, hist_scan, scan_scratch, st);
        if (e != cudaSuccess) return e;
        k_radix_scatter<<<ntiles, kSortThreads, 0, st>>>(ka, va, kb, vb, n, shift, nb,
                                                         hist_scan, ntiles);
        count_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        uint32_t *tk = ka; ka = kb; kb = tk;
        int32_t *tv = va; va = vb; vb = tv;
        *result_in_alt = !*result_in_alt;
    }
    return cudaSuccess;
}

}  // namespace nbl
