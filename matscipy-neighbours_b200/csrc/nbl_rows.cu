// nbl_rows.cu -- the pair passes by rows: the count takes one thread per
// sorted atom and lists its neighbours, the fill takes the output in order.
//
// Count (k_rows_count).  A thread walks its atom's visited cells in the
// reference's z/y/x order and each cell's atoms in ascending order, four
// candidates at a time: an FP32 test against the guard band's outer threshold
// (or, for the plain FP64 precision, the reference's test itself), and for the
// few candidates inside it the decision -- accepted below the inner threshold,
// else the reference's exact FP64 arithmetic.  Each neighbour is appended to
// the atom's list as (sorted atom, visit); the list's length is the row's.
// Neighbouring threads hold atoms of the same or adjacent cells, so a warp's
// candidate loads are broadcasts.
//
// Fill (k_rows_fill).  A warp takes 64 to 512 consecutive output slots, finds the
// rows they belong to, and makes 32 consecutive slots a round: list entry, j's
// record, the exact FP64 D and d, S.  Every store instruction covers whole
// aligned lines of an output array, whatever the rows' lengths.
//
// Why this shape: with a warp per cell (lane = candidate, hits compacted by
// ballots, scans and tables) the passes are made of instructions around the
// pairs, and rows written one by one leave a partial sector at both ends of
// every row in each of five arrays.  Measured, count + fill: 200,000 atoms of a
// slab with per-type cutoffs 85 + 21 us (187 + 120 one thread per atom writing
// its own row), a gas of two neighbours per atom 61 + 20 (73 + 97); the fill
// alone 616 us for the 48 M pairs of a million-atom metal (1,051 from hit words,
// a warp per cell), 4.0 TB/s of output, bound by L1 wavefronts (79 %: position
// gathers, staging) and the loads' latency.
//
// Which count: this one on sparse grids (kSparseAtoms, in nbl_plan.hh, with both
// sides measured) and with plain FP64 tests; k_count_list (nbl_trav_list.cu)
// elsewhere.
//
// Lists: atom i of a system, if its row is in range, owns list_cap 16-byte groups at
// list_base + i * list_cap, the last one a link to a chunk of kListChunk more, whose
// last group links on.  When the chunks run out the row keeps its length, asks for the
// chunks it lacks all the same (a synchronised count is then made once more, with
// that room), and kErrNoList is set; a row that still has no list is written by the
// thread-per-atom fill (nbl_trav_atoms.cu).
#include "nbl_stages.cuh"
#include "nbl_traverse.cuh"

namespace nbl {
namespace {

constexpr int kRowThreads = 128;
// Lanes per atom of a small system, and up to how many atoms (one thread per atom
// leaves most of the chip idle there).  Count with eight lanes / one, us, at 0.5 and 2
// atoms per cell: 2,000 atoms 9 / 26, 10 / 34; 16,000 15 / 27, 18 / 36; 32,000 22 / 29,
// 28 / 38; 48,000 30 / 31, 37 / 41; 64,000 38 / 30, 46 / 43.
constexpr long long kSplitAtoms = 32768;
constexpr int kSplit = 8;
constexpr int kSplitBuf = 16;  // list entries a lane of those buffers

// Appends to a row's list: entries gather in one group's registers and leave
// in one 16-byte store (a store per entry would cost an L1 cycle and a partial
// sector each: 32 lanes write 32 lists).
template <bool WIDE>
struct RowList {
    uint4 q;
    long long wp;  // next group; without a list any more, the groups it holds
    int room;      // groups left before the link; -1: no list any more
    int n;         // row length
    __device__ __forceinline__ void put(const TraverseArgs &a) {
        if (room == 0) {
            const long long next = list_grow(a, wp);
            room = next >= 0 ? kListChunk - 1 : -1;
            wp = next >= 0 ? next : (n - 1) / Entry<WIDE>::kPerGroup;
        }
        if (room > 0) {
            a.list[wp] = q;
            wp++;
            room--;
        }
    }
    __device__ __forceinline__ void push(const TraverseArgs &a, int sj, int v) {
        if constexpr (WIDE) {
            if (n & 1) {
                q.z = (unsigned)sj;
                q.w = (unsigned)v;
            } else {
                q.x = (unsigned)sj;
                q.y = (unsigned)v;
            }
            n++;
            if (!(n & 1)) put(a);
        } else {
            const unsigned e = Entry<false>::make(a.list_shift, sj, v);
            const int k = n & 3;
            if (k == 0) q.x = e;
            if (k == 1) q.y = e;
            if (k == 2) q.z = e;
            n++;
            if (k == 3) {
                q.w = e;
                put(a);
            }
        }
    }
    __device__ __forceinline__ void finish(const TraverseArgs &a) {
        if (n & (Entry<WIDE>::kPerGroup - 1)) put(a);
        if (room < 0) list_lacks(a, n - wp * Entry<WIDE>::kPerGroup, Entry<WIDE>::kPerGroup);
    }
};

// What a thread knows about its atom i while it walks.
struct RowAtom {
    int si;        // sorted index
    int c[3];      // home cell
    int sys;
    double4 p64;
    float4 p32;
    Hot H;
};

// Cell coordinate x of an axis with n cells, folded: the image shift in m;
// false outside an open axis.
__device__ __forceinline__ bool fold_axis(int &x, int n, int periodic, int &m) {
    m = 0;
    if (x < 0 || x >= n) {
        if (!periodic) return false;
        m = (x < 0 && x >= -n) ? -1 : (x >= n && x < 2 * n) ? 1 : floor_div(x, n);
        x -= m * n;
    }
    return true;
}

// Atom A.si's filter record and thresholds; its cell and system are set.
template <bool FP32>
__device__ __forceinline__ void row_thresholds(const TraverseArgs &a, const SysDev &S, RowAtom &A) {
    A.p32 = a.pos32[A.si];
    A.H.lo_rc = A.H.hi_rc = A.H.band = 0.f;
    if (FP32) {
        const double ext = (double)S.n[0] *
                           fmax(fabs(S.bin[0][0]), fmax(fabs(S.bin[0][1]), fabs(S.bin[0][2])));
        const double band =
            guard_band(2.0 * ((double)a.amax[A.sys] + ext) + S.off_max + ext, S.cutoff);
        A.H.lo_rc = __double2float_rd(S.cutoff_sq - band);
        A.H.hi_rc = __double2float_ru(S.cutoff_sq + band);
        A.H.band = __double2float_ru(band);
    }
    A.H.cutoff_sq = S.cutoff_sq;
    A.H.ncut = S.ncutoffs;
    A.H.pt_base = S.pt_base;
}

// A guard-band candidate, decided exactly.
template <int KIND>
__device__ __noinline__ bool row_exact(const TraverseArgs &a, const SysDev &S, int si, int sj,
                                       int v) {
    Hot H;
    H.cutoff_sq = S.cutoff_sq;
    H.ncut = S.ncutoffs;
    H.pt_base = S.pt_base;
    double off[3];
    visit_vector(a, S, v, off);
    return exact_inside<KIND>(H, a, a.pos64[si], a.pos64[sj], off, a.pos32[si].w, a.pos32[sj].w);
}

// The candidates [b, e) (sorted atoms) against atom i, in order: visit v up to
// q1, then v + 1 up to q2, then v + 2.  off: what is added to a candidate's
// unrolled FP32 position to bring it beside atom i's; hit(sj, visit) is called
// for every neighbour.
template <int KIND, bool FP32, typename F>
__device__ __forceinline__ void sweep_range(const TraverseArgs &a, const SysDev &S,
                                            const RowAtom &A, int b, int e, int v, int q1, int q2,
                                            const float off[3], bool self_here, F &&hit) {
    if constexpr (FP32) {
        // candidate minus (atom - offset): the guard band's rounding bound
        const float ax = A.p32.x - off[0], ay = A.p32.y - off[1], az = A.p32.z - off[2];
        for (int s0 = b; s0 < e; s0 += 32) {
            const int n = min(32, e - s0);
            // one bit per candidate inside the outer threshold, and one per
            // candidate surely a neighbour, eight at a time (the array is padded:
            // reading past the range is harmless)
            unsigned near = 0u, sure = 0u;
            const float4 *src = a.pos32 + s0;
            for (int u0 = 0; u0 < n; u0 += 8) {
                unsigned nb = 0u, sb = 0u;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const float4 p = __ldg(src + u0 + u);
                    const float dx = p.x - ax, dy = p.y - ay, dz = p.z - az;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    float lo = A.H.lo_rc, hi = A.H.hi_rc;
                    if (KIND == kCutPerAtom) thresholds<KIND>(A.H, a, A.p32.w, p.w, lo, hi);
                    if (r2 < hi) nb |= 1u << u;
                    if (r2 < lo) sb |= 1u << u;
                }
                near |= nb << u0;
                sure |= sb << u0;
            }
            if (n < 32) near &= (1u << n) - 1u;
            if (self_here && A.si >= s0 && A.si < s0 + 32) near &= ~(1u << (A.si - s0));
            for (; near; near &= near - 1u) {
                const int u = __ffs(near) - 1;
                const int sj = s0 + u;
                const int vj = v + (sj >= q1 ? 1 : 0) + (sj >= q2 ? 1 : 0);
                bool in = (sure >> u) & 1u;
                if (KIND == kCutPerType) {  // the pair's own threshold
                    const float4 p = __ldg(a.pos32 + sj);
                    const float dx = p.x - ax, dy = p.y - ay, dz = p.z - az;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    float lo, hi;
                    thresholds<KIND>(A.H, a, A.p32.w, p.w, lo, hi);
                    in = r2 < lo || (r2 < hi && row_exact<KIND>(a, S, A.si, sj, vj));
                } else if (!in) {
                    in = row_exact<KIND>(a, S, A.si, sj, vj);
                }
                if (in) hit(sj, vj);
            }
        }
    } else {
        int last = -1;
        double o64[3] = {0.0, 0.0, 0.0};
        for (int sj = b; sj < e; sj++) {
            if (self_here && sj == A.si) continue;
            const int vj = v + (sj >= q1 ? 1 : 0) + (sj >= q2 ? 1 : 0);
            if (vj != last) visit_vector(a, S, last = vj, o64);
            const float wj = KIND == kCutPerType ? a.pos32[sj].w : 0.f;
            if (exact_inside<KIND>(A.H, a, A.p64, a.pos64[sj], o64, A.p32.w, wj)) hit(sj, vj);
        }
    }
}

// Atom i against the visited rows [r0, r1) of cells (offsets z, then y; the
// cells of a row by x): the reference's order (neighbour_visit.hh:63-84).  On a
// dense grid that scans one cell each way the three cells of a row are one
// contiguous range of sorted atoms wherever the row does not wrap.
template <int KIND, bool FP32, typename F>
__device__ __forceinline__ void sweep_rows(const TraverseArgs &a, const SysDev &S,
                                           const RowAtom &A, int r0, int r1, F &&hit) {
    const int nx = S.nscan[0], ny = S.nscan[1], nz = S.nscan[2];
    const int wx = 2 * nx + 1, wy = 2 * ny + 1;
    const bool join = a.grid == kGridDense && nx == 1 && A.c[0] > 0 && A.c[0] < S.n[0] - 1;
    const int pieces = join ? 1 : wx;
    for (int r = r0; r < r1; r++) {
        const int d1 = r % wy - ny, d2 = r / wy - nz;
        int c1 = A.c[1] + d1, c2 = A.c[2] + d2, m0, m1, m2;
        if (!fold_axis(c1, S.n[1], S.pbc[1], m1)) continue;
        if (!fold_axis(c2, S.n[2], S.pbc[2], m2)) continue;
        for (int x = 0; x < pieces; x++) {
            int b, e, q1 = INT_MAX, q2 = INT_MAX;
            bool self = d1 == 0 && d2 == 0;
            m0 = 0;
            if (join) {
                const int2 *t = a.table + S.cell_base + A.c[0] +
                                (int64_t)S.n[0] * ((int64_t)c1 + (int64_t)S.n[1] * c2);
                const int2 t0 = t[-1], t1 = t[0], t2 = t[1];
                b = t0.y > t0.x ? t0.x : t1.y > t1.x ? t1.x : t2.x;
                q1 = b + t0.y - t0.x;
                q2 = q1 + t1.y - t1.x;
                e = q2 + t2.y - t2.x;
            } else {
                int c0 = A.c[0] + x - nx;
                if (!fold_axis(c0, S.n[0], S.pbc[0], m0)) continue;
                const int2 sl = cell_lookup(a, S, A.sys, c0, c1, c2);
                b = sl.x;
                e = sl.y;
                self = self && x == nx;
            }
            if (checked_fail(b < 0 || e < b || (long long)e > a.natoms, a.err)) continue;
            float off[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                off[k] = __double2float_rn((double)d2 * S.bin[2][k] + (double)d1 * S.bin[1][k] +
                                           (double)m0 * S.n[0] * S.bin[0][k]);
            sweep_range<KIND, FP32>(a, S, A, b, e, r * wx + x, q1, q2, off, self, hit);
        }
    }
}

// Lanes per atom G (1 or 8): with 8, each lane walks its share of the visited
// rows, and the lists' shares are put behind one another afterwards.
template <int KIND, bool FP32, int G, bool WIDE>
__global__ void __launch_bounds__(kRowThreads)
k_rows_count(const __grid_constant__ TraverseArgs a) {
    using E = Entry<WIDE>;
    __shared__ typename E::T buf[G > 1 ? kSplitBuf : 1][G > 1 ? kRowThreads : 1];
    const unsigned full = 0xffffffffu;
    const long long t = (long long)blockIdx.x * kRowThreads + threadIdx.x;
    const int g = (int)(t % G);
    RowAtom A;
    bool on = t / G < a.natoms;
    A.si = on ? (int)(t / G) : 0;
    A.p64 = a.pos64[A.si];
    const int at = __double2loint(A.p64.w);
    on = on && !checked_fail(at < 0 || at >= a.natoms, a.err) && at >= a.i_lo && at < a.i_hi;
    if (G == 1 && !on) return;
    const int4 hc = a.hcell[A.si];
    A.c[0] = hc.x;
    A.c[1] = hc.y;
    A.c[2] = hc.z;
    A.sys = hc.w;
    const SysDev &S = a.sys[A.sys];
    row_thresholds<FP32>(a, S, A);
    const int rows = on ? (2 * S.nscan[1] + 1) * (2 * S.nscan[2] + 1) : 0;
    RowList<WIDE> L;
    L.q = make_uint4(0u, 0u, 0u, 0u);
    L.wp = S.list_base + (long long)(at - (int)S.atom_base) * S.list_cap;
    L.room = S.list_cap - 1;
    L.n = 0;
    if constexpr (G == 1) {
        sweep_rows<KIND, FP32>(a, S, A, 0, rows, [&](int sj, int v) { L.push(a, sj, v); });
        L.finish(a);
        a.counts[at] = L.n;
    } else {
        typename E::T *dst = reinterpret_cast<typename E::T *>(a.list + L.wp);
        int r0 = rows * g / G, r1 = rows * (g + 1) / G;
        // mode 0: own rows into the buffer; 1: what the buffer did not hold, to
        // its place; 2: a list that chains, by one lane for all rows
        int mode = 0, n = 0, total = 0;
        while (true) {
            sweep_rows<KIND, FP32>(a, S, A, r0, r1, [&](int sj, int v) {
                if (mode == 2) {
                    L.push(a, sj, v);
                } else {
                    if (mode == 0 && n < kSplitBuf) buf[n][threadIdx.x] = E::make(a.list_shift, sj, v);
                    if (mode == 1 && n >= kSplitBuf) dst[n] = E::make(a.list_shift, sj, v);
                    n++;
                }
            });
            if (mode != 0) break;
            int incl = n;
#pragma unroll
            for (int d = 1; d < G; d <<= 1) {
                const int o = __shfl_up_sync(full, incl, d, G);
                if (g >= d) incl += o;
            }
            total = __shfl_sync(full, incl, G - 1, G);
            if (!on) return;
            if (total <= (S.list_cap - 1) * E::kPerGroup) {
                dst += incl - n;
                for (int k = 0; k < min(n, kSplitBuf); k++) dst[k] = buf[k][threadIdx.x];
                if (n <= kSplitBuf) break;
                mode = 1;
                n = 0;
            } else {
                if (g != 0) return;
                mode = 2;
                r0 = 0;
                r1 = rows;
            }
        }
        if (mode == 2) L.finish(a);
        if (g == 0) a.counts[at] = total;
    }
}

// Row of every kRowMark-th output slot.
__global__ void __launch_bounds__(256)
k_row_marks(const int64_t *__restrict__ off, long long n, int32_t *__restrict__ row_of,
            long long row_cap) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const long long e = off[i + 1];
    for (long long c = (off[i] + kRowMark - 1) / kRowMark; c * kRowMark < e && c < row_cap; c++)
        row_of[c] = (int32_t)i;
}

// Last row that starts at or before slot s (off[row] <= s < off[row + 1]): the
// warp cuts the interval into 32 at a time.
__device__ __forceinline__ long long find_row(const int64_t *off, long long n, long long s,
                                              int lane) {
    long long lo = 0, len = n;  // the row lies in [lo, lo + len)
    while (len > 1) {
        const long long part = (len + 31) >> 5, at = lo + part * lane;
        const unsigned m = __ballot_sync(0xffffffffu, part * lane < len && off[at] <= s);
        const int k = 31 - __clz(m);  // (lane 0 holds: off[lo] <= s)
        lo += part * k;
        len = min(part, len - part * k);
    }
    return lo;
}

constexpr int kFillWarps = 8;
// CTAs per SM (48 registers a thread, no spills).  The million-atom metal's fill at
// 3 / 4 / 5 / 6: 755 / 650 / 612 / 703 us; six of them spill and shrink the L1.
constexpr int kFillBlocks = 5;

struct __align__(16) RowWarp {
    double d[96];          // one round's distance vectors
    double2 ia[32];        // rows in hand: atom i's x, y
    double2 ib[32];        // z, atom index and packed image (as bits)
    int4 hc[32];           // home cell and system
    long long list[32];    // first group of the row's list
    int32_t cap[32];       // its entries before the chain
    int32_t edge[32];      // nonzero: visits of the row may cross a periodic face
    int32_t start[32];     // first slot, relative to the chunk
    int32_t si[32];        // sorted index
};

// Entry r of a row's list (first group `base`, `cap` entries before the chain);
// false when the row has no list that far.
template <bool WIDE>
__device__ __forceinline__ bool list_entry(const TraverseArgs &a, long long base, int cap,
                                           long long r, int &sj, int &v) {
    using E = Entry<WIDE>;
    if (!list_reach<WIDE>(a, base, cap, r)) return false;
    E::get(a.list_shift, reinterpret_cast<const typename E::T *>(a.list + base)[r], sj, v);
    return !checked_fail(sj < 0 || sj >= a.natoms, a.err);
}

// Image shift of visit v from home cell hc.
__device__ __forceinline__ void visit_image(const TraverseArgs &a, const SysDev &S, const int4 &hc,
                                            int v, int m[3]) {
    int d[3];
    float unused[3];
    visit_at(a, S, v, d, unused);
    const int c[3] = {hc.x, hc.y, hc.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int x = c[k] + d[k], n = S.n[k];
        m[k] = x < 0 ? (x >= -n ? -1 : floor_div(x, n))
                     : x >= n ? (x < 2 * n ? 1 : floor_div(x, n)) : 0;
    }
}

// S of one pair whose image indices do not pack, from the full records.
__device__ __noinline__ void far_shift(const TraverseArgs &a, const SysDev &S, const int4 &hc,
                                       int si, int sj, int v, int32_t *out) {
    const int4 xi = a.aux[si], xj = a.aux[sj];
    int m[3];
    visit_image(a, S, hc, v, m);
    const int qi[3] = {xi.y, xi.z, xi.w}, qj[3] = {xj.y, xj.z, xj.w};
#pragma unroll
    for (int k = 0; k < 3; k++) __stcs(out + k, qi[k] + (S.pbc[k] ? m[k] - qj[k] : 0));
}

template <bool ALL5, bool WIDE>
__global__ void __launch_bounds__(kFillWarps * 32, kFillBlocks)
k_rows_fill(const __grid_constant__ TraverseArgs a) {
    __shared__ RowWarp smem[kFillWarps];
    __shared__ volatile long long last_chunk[kFillWarps][2];  // (spares registers)
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RowWarp &sm = smem[warp];
    const long long total = a.offsets[a.natoms];
    const long long P = min(total, (long long)a.capacity);
    if (total > a.capacity && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.err, kErrCapacity);
    // Slots a warp takes at a time: a power of two from 64 to 512 that gives a warp
    // about four chunks.  (At 128 / 256 / 512 the fill took 8.6 / 13 / 22 us for 65,000
    // pairs, 19 / 24 / 39 for 400,000, 71 / 72 / 80 for 5.4 M, 660 / 610 / 610 for
    // 48 M, 1,189 / 1,144 / 1,093 for the batch of 4,096 systems.)
    const int step = (int)gridDim.x * kFillWarps;
    int bits = 6;
    while (bits < 9 && (P >> bits) > 4ll * step) bits++;
    const int nchunks = (int)((P + (1 << bits) - 1) >> bits);
    last_chunk[warp][0] = P;
    last_chunk[warp][1] = nchunks;
    __syncwarp();
    for (int ch = (int)blockIdx.x * kFillWarps + warp; ch < (int)last_chunk[warp][1]; ch += step) {
        const long long B0 = (long long)ch << bits;
        const int E = (int)min(1ll << bits, last_chunk[warp][0] - B0);  // slots of the chunk
        int row;
        if ((B0 & (kRowMark - 1)) == 0 && B0 / kRowMark < a.row_cap)
            row = a.row_of[B0 / kRowMark];
        else
            row = (int)find_row(a.offsets, a.natoms, B0, lane);
        int pos = 0;
        while (pos < E && row < a.natoms) {
            // --- the next 32 rows: the non-empty ones, compacted ---------------------
            const int r = row + lane;
            long long o0 = 0, o1 = 0;
            if (r < a.natoms) {
                o0 = a.offsets[r];
                o1 = a.offsets[r + 1];
            }
            const long long wend = __shfl_sync(full, o1, min(31, (int)a.natoms - 1 - row));
            const bool take = o1 > o0 && o0 < B0 + E;
            const unsigned mask = __ballot_sync(full, take);
            const int nrow = __popc(mask);
            __syncwarp();
            if (take) {
                const int k = __popc(mask & lanemask_lt());
                const int s = a.inv[r];
                const double4 p = a.pos64[s];
                const int4 hc = a.hcell[s];
                const SysDev &S = a.sys[hc.w];
                sm.ia[k] = make_double2(p.x, p.y);
                sm.ib[k] = make_double2(p.z, p.w);
                sm.hc[k] = hc;
                sm.list[k] = S.list_base + (r - S.atom_base) * S.list_cap;
                sm.cap[k] = (S.list_cap - 1) * Entry<WIDE>::kPerGroup;
                sm.edge[k] = hc.x < S.nscan[0] || hc.x + S.nscan[0] >= S.n[0] ||
                             hc.y < S.nscan[1] || hc.y + S.nscan[1] >= S.n[1] ||
                             hc.z < S.nscan[2] || hc.z + S.nscan[2] >= S.n[2];
                sm.start[k] = (int)max(o0 - B0, -(1ll << 30));
                sm.si[k] = s;
                // a first row reaching far back: its list position is absolute
                if (o0 - B0 < -(1ll << 30)) atomicOr(a.err, kErrInternal);
            }
            __syncwarp();
            const int lim = (int)min((long long)E, wend - B0);
            for (; pos < lim; pos += 32) {
                // rows that start inside this round mark their first lane
                const int sx = lane < nrow ? sm.start[lane] - pos : 64;
                const unsigned heads =
                    __reduce_or_sync(full, sx > 0 && sx < 32 ? 1u << sx : 0u);
                const int cur = __popc(__ballot_sync(full, sx <= 0)) - 1;
                const int al = cur + __popc(heads & (lanemask_lt() | 1u << lane));
                const bool act = pos + lane < lim;
                long long slot = -1;
                int shift = -1;
                if (act) {
                    slot = B0 + pos + lane;
                    const double2 ia = sm.ia[al], ib = sm.ib[al];
                    int sj, v;
                    if (list_entry<WIDE>(a, sm.list[al], sm.cap[al], pos + lane - sm.start[al],
                                         sj, v)) {
                        const SysDev &S = a.sys[sm.hc[al].w];
                        const int base = (int)S.atom_base;
                        const double4 pj = a.pos64[sj];
                        double off[3];
                        visit_vector(a, S, v, off);
                        const double dx = dadd(dsub(pj.x, ia.x), off[0]);
                        const double dy = dadd(dsub(pj.y, ia.y), off[1]);
                        const double dz = dadd(dsub(pj.z, ib.x), off[2]);
                        if (ALL5 || a.first) __stcs(a.first + slot, __double2loint(ib.y) - base);
                        if (ALL5 || a.second) __stcs(a.second + slot, __double2loint(pj.w) - base);
                        if (ALL5 || a.distvec) {
                            sm.d[3 * lane] = dx;
                            sm.d[3 * lane + 1] = dy;
                            sm.d[3 * lane + 2] = dz;
                        }
                        if (ALL5 || a.absdist) {
                            const double r2 =
                                dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
                            __stcs(a.absdist + slot, __dsqrt_rn(r2));
                        }
                        if (ALL5 || a.shift) {
                            const int qi = __double2hiint(ib.y), qj = __double2hiint(pj.w);
                            int mp = 0;
                            if (sm.edge[al]) {
                                int m[3];
                                visit_image(a, S, sm.hc[al], v, m);
                                mp = pack_image(m[0], m[1], m[2]);
                            }
                            if (qi != kImageWide && qj != kImageWide && mp != kImageWide)
                                shift = qi - qj + mp + kImageBias;
                            else
                                far_shift(a, S, sm.hc[al], sm.si[al], sj, v, a.shift + 3 * slot);
                        }
                    } else {
                        slot = -1;
                    }
                }
                // --- D and S: element 32 q + lane of the round ------------------------
                if (ALL5 || a.distvec || a.shift) {
                    const unsigned good = __ballot_sync(full, slot >= 0);
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        const int el = 32 * q + lane;
                        const int p = (el * 43691) >> 17, c = el - 3 * p;  // el / 3
                        const bool on = (good >> p) & 1u;
                        const long long E0 = 3 * (B0 + pos) + el;
                        if ((ALL5 || a.distvec) && on) __stcs(a.distvec + E0, sm.d[el]);
                        if (ALL5 || a.shift) {
                            const int t = __shfl_sync(full, shift, p);
                            if (on && t >= 0) __stcs(a.shift + E0, ((t >> (10 * c)) & 1023) - 512);
                        }
                    }
                    __syncwarp();
                }
            }
            pos = lim;
            row += 32;
        }
    }
}

// The neighbour matrix: a warp per row, ranks in rounds of 32, the slots past
// the row's end set to zero (so nothing clears the matrix first).  Bound by its
// writes, 28 bytes a slot: 131,072 rows of 64 slots 70 us, 3.3 TB/s (105 from hit
// words, a warp per cell, after 89 of clearing); 74 at four CTAs per SM.
template <bool WIDE>
__global__ void __launch_bounds__(kFillWarps * 32, kFillBlocks)
k_rows_matrix(const __grid_constant__ TraverseArgs a) {
    __shared__ double sd[kFillWarps][96];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long K = a.mat_k;
    const long long step = (long long)gridDim.x * kFillWarps;
    for (long long r = (long long)blockIdx.x * kFillWarps + warp; r < a.natoms; r += step) {
        const long long o0 = a.offsets[r];
        const long long deg = a.offsets[r + 1] - o0;
        const int s = a.inv[r];
        const double4 pi = a.pos64[s];
        const int sys = a.nsys > 1 ? a.hcell[s].w : 0;
        const SysDev &S = a.sys[sys];
        const long long base = S.list_base + (r - S.atom_base) * S.list_cap;
        if (lane == 0) {
            a.mat_count[r] = (int32_t)deg;
            if (deg > K) atomicOr(a.mat_overflow, 1);
        }
        for (long long r0 = 0; r0 < K; r0 += 32) {
            const long long rank = r0 + lane;
            int j = 0;
            double dx = 0.0, dy = 0.0, dz = 0.0;
            if (rank < min(deg, K)) {
                int sj, v;
                if (list_entry<WIDE>(a, base, (S.list_cap - 1) * Entry<WIDE>::kPerGroup, rank, sj,
                                     v)) {
                    const double4 pj = a.pos64[sj];
                    double off[3];
                    visit_vector(a, S, v, off);
                    dx = dadd(dsub(pj.x, pi.x), off[0]);
                    dy = dadd(dsub(pj.y, pi.y), off[1]);
                    dz = dadd(dsub(pj.z, pi.z), off[2]);
                    j = __double2loint(pj.w) - (int)S.atom_base;
                }
            }
            if (rank < K) a.mat_idx[r * K + rank] = j;
            sd[warp][3 * lane] = dx;
            sd[warp][3 * lane + 1] = dy;
            sd[warp][3 * lane + 2] = dz;
            __syncwarp(full);
            const int n3 = 3 * (int)min(32ll, K - r0);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int el = 32 * q + lane;
                if (el < n3) __stcs(a.mat_dist + 3 * (r * K + r0) + el, sd[warp][el]);
            }
            __syncwarp(full);
        }
    }
}

template <bool FP32, int G, bool WIDE>
TravKernel count_kernel(int kind) {
    if (kind == kCutPerAtom) return k_rows_count<kCutPerAtom, FP32, G, WIDE>;
    if (kind == kCutPerType) return k_rows_count<kCutPerType, FP32, G, WIDE>;
    return k_rows_count<kCutScalar, FP32, G, WIDE>;
}

template <bool WIDE>
TravKernel count_kernel(bool fp32, bool split, int kind) {
    if (split) return fp32 ? count_kernel<true, kSplit, WIDE>(kind)
                           : count_kernel<false, kSplit, WIDE>(kind);
    return fp32 ? count_kernel<true, 1, WIDE>(kind) : count_kernel<false, 1, WIDE>(kind);
}

template <bool WIDE>
TravKernel fill_kernel(const TraverseArgs &a) {
    const bool all5 = a.first && a.second && a.distvec && a.absdist && a.shift;
    return a.mat_k > 0 ? k_rows_matrix<WIDE> : all5 ? k_rows_fill<true, WIDE>
                                                    : k_rows_fill<false, WIDE>;
}

}  // namespace

cudaError_t launch_count_rows(bool fp32, int kind, const TraverseArgs &a, cudaStream_t st) {
    if (a.natoms <= 0) return cudaSuccess;
    const bool split = a.natoms <= kSplitAtoms;
    const TravKernel k = a.list_wide ? count_kernel<true>(fp32, split, kind)
                                     : count_kernel<false>(fp32, split, kind);
    const long long threads = a.natoms * (split ? kSplit : 1);
    k<<<(unsigned)((threads + kRowThreads - 1) / kRowThreads), kRowThreads, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_row_marks(const TraverseArgs &a, cudaStream_t st) {
    if (a.natoms <= 0 || a.row_cap <= 0) return cudaSuccess;
    k_row_marks<<<(unsigned)((a.natoms + 255) / 256), 256, 0, st>>>(a.offsets, a.natoms, a.row_of,
                                                                   a.row_cap);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_fill_rows(const TraverseArgs &a, int num_sms, cudaStream_t st) {
    if (a.natoms <= 0) return cudaSuccess;
    const TravKernel k = a.list_wide ? fill_kernel<true>(a) : fill_kernel<false>(a);
    k<<<(unsigned)(num_sms * kFillBlocks), kFillWarps * 32, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace nbl
