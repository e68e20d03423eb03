// nbl_trav_list.cu -- the count pass of dense grids: one warp per work item
// (home cell x tile of up to 32 atoms) counts every atom's neighbours and
// lists them for the row fill (nbl_rows.cu).
//
// The visited cells' atoms are staged in shared memory as FP32 positions in
// the home cell's frame, and lane L takes the L-th block of consecutive
// candidates: it sweeps them against four atoms at a time (packed f32x2) and
// keeps, per atom, one bit per candidate of its block in a register.  Because
// the blocks are consecutive, lane order is list order: no ballots while
// sweeping, one warp scan of the lanes' hits for two atoms, and every hit's
// candidate number goes to its place in a short shared-memory list, from which
// half a warp per atom writes the entries.  A lane's block has an odd length,
// so that the 16-byte candidate loads of a quarter warp fall into different
// banks.
//
// With the candidates dealt out 32 at a time instead (a ballot per atom and
// 32 candidates, hits compacted by population counts) the same pass took 611 us
// on the dense bulk (1,048,576 atoms), bound by the population counts' slow
// pipe; with one thread per atom 674 us, because a warp's atoms lie in three
// cells whose candidates differ.  This form: 492 us there (the two-pass scheme
// that wrote hit words took 371, but its fill 1,051 against 616 us from these
// lists), 25 + 15 us for 10,007 atoms (36 + 36 before).  Bound by the latency of
// staging and list writes at 17 warps per SM, 0.5 instructions a cycle: about 180 us
// staging and set-up, 150 the sweep, 160 the entries.
//
// Where an atom visits many candidates (CULL: more than one full table on average,
// kCullCand) the ones outside the tile's bounding box plus the cutoff never reach the
// table: 1,443 us on 4,096 small periodic systems of about 3,000 candidates per atom
// (2,411 without, at four CTAs per SM).
#include "nbl_traverse.cuh"

namespace nbl {
namespace {

constexpr int kListBlk = 13;              // candidates a lane takes at most (odd)
constexpr int kListCand = 32 * kListBlk;  // candidates staged at a time
constexpr int kListWarps = 4;

template <bool WIDE>
struct __align__(16) ListWarp {
    float4 cand[kListCand];
    typename Entry<WIDE>::T entry[kListCand];  // list entry of each staged candidate
    uint16_t code[kListCand];   // hits of the atoms in hand, in order: staged candidates
    float4 i32[kITile];
    long long lw[kITile];       // entry index of rank 0, as if the current segment began there
    int32_t lim[kITile];        // first rank beyond the segment; -1: no list any more (lw: the
                                // entries it holds)
    int32_t icount[kITile];     // row lengths so far
    int32_t iatom[kITile];
    int32_t isi[kITile];
    int32_t self[kITile];       // staged candidate of each sorted atom of the tile itself
    float off[kSeg][3];
    int32_t bj[kSeg];           // candidate kk of the segment is sorted atom bj + kk
    int32_t pref[kSeg + 1];
};
// CTAs per SM.  (Culling, 4,096 small systems: 1,557 us at 5, 1,615 at 4.)
constexpr int list_blocks(bool wide, bool lj = false) { return wide || lj ? 4 : 5; }
static_assert(list_blocks(false) * (kListWarps * sizeof(ListWarp<false>) + 1024) <= 233472 &&
                  list_blocks(true) * (kListWarps * sizeof(ListWarp<true>) + 1024) <= 233472,
              "the CTAs fit the SM's shared memory");

// Segment batch vb of the item's home cell: one lane per visited offset
// (neighbour_visit.hh:63-84), in the reference's order.
template <bool WIDE>
__device__ __forceinline__ void list_setup(ListWarp<WIDE> &sm, const TraverseArgs &a, const SysDev &S,
                                           const WorkItem &w, int vb, int lane, int &nseg,
                                           int &total, int &zs) {
    const unsigned full = 0xffffffffu;
    nseg = min(kSeg, S.nvisit - vb);
    int len = 0, first = 0;
    bool zero = false;
    if (lane < nseg) {
        int d[3];
        float off[3];
        visit_at(a, S, vb + lane, d, off);
        zero = d[0] == 0 && d[1] == 0 && d[2] == 0;
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            int x = w.c[k] + d[k];
            const int n = S.n[k];
            if (x < 0 || x >= n) {
                if (!S.pbc[k]) ok = false;
                x -= ((x < 0 && x >= -n) ? -1 : (x >= n && x < 2 * n) ? 1 : floor_div(x, n)) * n;
            }
            d[k] = x;
            sm.off[lane][k] = off[k];
        }
        if (ok) {
            int2 sl = cell_lookup(a, S, w.sys, d[0], d[1], d[2]);
            if (checked_fail(sl.x < 0 || sl.y < sl.x || (long long)sl.y > a.natoms, a.err))
                sl = make_int2(0, 0);
            first = sl.x;
            len = sl.y - sl.x;
        }
    }
    int incl = len;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int o = __shfl_up_sync(full, incl, s);
        if (lane >= s) incl += o;
    }
    total = __shfl_sync(full, incl, 31);
    if (lane < nseg) {
        sm.pref[lane] = incl - len;
        sm.bj[lane] = first - (incl - len);
    }
    if (lane == 0) sm.pref[nseg] = total;
    const unsigned zm = __ballot_sync(full, zero);
    zs = zm ? __ffs(zm) - 1 : -1;
    __syncwarp();
}

// Candidates kb .. kb + nk of the batch (short cells: lane = segment) in the
// home cell's frame, and their list entries.
template <bool WIDE>
__device__ __forceinline__ void list_stage(ListWarp<WIDE> &sm, const TraverseArgs &a, int nseg,
                                           int vb, int kb, int nk, int zs, int ib, int lane) {
    using E = Entry<WIDE>;
    __syncwarp();
    sm.self[lane] = zs >= 0 ? ib + lane - sm.bj[zs] - kb : -1;
    if (lane < nseg) {
        const int s0 = max(sm.pref[lane], kb), s1 = min(sm.pref[lane + 1], kb + nk);
        const float ox = sm.off[lane][0], oy = sm.off[lane][1], oz = sm.off[lane][2];
        const float4 *src = a.pos32 + sm.bj[lane];
        const int sj0 = sm.bj[lane];
        float4 p[4];  // four loads in flight before the stores
        for (int kk = s0; kk < s1; kk += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) p[u] = __ldg(src + min(kk + u, s1 - 1));
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (kk + u < s1) {
                    sm.cand[kk + u - kb] =
                        make_float4(p[u].x + ox, p[u].y + oy, p[u].z + oz, p[u].w);
                    sm.entry[kk + u - kb] = E::make(a.list_shift, sj0 + kk + u, vb + lane);
                }
        }
    }
}

// Many candidates: only those inside the outer threshold of the tile's bounding
// box (lo .. hi) are staged, in order, until the table is full; returns how
// many, and the next candidate in kb.  (Lane = candidate, its segment by
// search.)  The box distance is built from the operations of the pair distance,
// each of them monotone, so no pair inside the threshold is lost.
template <bool WIDE>
__device__ __forceinline__ int list_stage_near(ListWarp<WIDE> &sm, const TraverseArgs &a, int nseg,
                                               int total, int vb, int &kb, int zs, int ib,
                                               const float lo[3], const float hi[3], float hi_rc,
                                               int lane) {
    using E = Entry<WIDE>;
    const unsigned full = 0xffffffffu;
    __syncwarp();
    sm.self[lane] = -1;
    __syncwarp();
    const int prefl = lane < nseg ? sm.pref[lane] : INT_MAX;
    int n = 0;
    for (; kb < total && n <= kListCand - 32; kb += 32) {
        const int kk = kb + lane, kc = min(kk, total - 1);
        int seg = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const int v = __shfl_sync(full, prefl, (seg + st) & 31);
            if (seg + st < nseg && v <= kc) seg += st;
        }
        const int sj = sm.bj[seg] + kc;
        float4 p = a.pos32[sj];
        p.x += sm.off[seg][0];
        p.y += sm.off[seg][1];
        p.z += sm.off[seg][2];
        const float dx = fmaxf(fmaxf(p.x - hi[0], lo[0] - p.x), 0.f);
        const float dy = fmaxf(fmaxf(p.y - hi[1], lo[1] - p.y), 0.f);
        const float dz = fmaxf(fmaxf(p.z - hi[2], lo[2] - p.z), 0.f);
        const bool keep = kk < total && fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < hi_rc;
        const unsigned m = __ballot_sync(full, keep);
        if (keep) {
            const int k = n + __popc(m & lanemask_lt());
            sm.cand[k] = p;
            sm.entry[k] = E::make(a.list_shift, sj, vb + seg);
            if (seg == zs && sj - ib >= 0 && sj - ib < kITile) sm.self[sj - ib] = k;
        }
        n += __popc(m);
    }
    return n;
}

// Per-type cutoffs: the squared cutoffs of one atom's type, and minus the one with
// type tj (the widest for a type outside the table; a NaN stays one: neither sign bit
// of the sums it enters is set).  One load a pair in the sweep: a million atoms with
// cutoffs of 5, 3.2 and 3 take 1,500 us, with 5, 5 and 5 1,730; sweeping with the widest
// and testing what that leaves pair by pair 2,030 and 2,110.
struct TypeRow {
    const float *at;
    int n;
};
__device__ __forceinline__ TypeRow type_row(const TraverseArgs &a, const SysDev &S, float w) {
    const int t = __float_as_int(w);
    const bool in = t >= 0 && t < S.ncutoffs;
    return TypeRow{a.pt32 + S.pt_base + (in ? t * S.ncutoffs : 0), in ? S.ncutoffs : 0};
}
__device__ __forceinline__ float type_cut(const TypeRow &row, int tj, float rc2) {
    const float v = (unsigned)tj < (unsigned)row.n ? __ldg(row.at + tj) : rc2;
    return v >= rc2 ? -rc2 : -v;
}

// Staged candidate k against atom il of the tile where the FP32 filter does not
// decide: the reference's exact test.
template <int KIND, bool WIDE>
__device__ __noinline__ bool list_exact(const ListWarp<WIDE> &sm, const TraverseArgs &a,
                                        const SysDev &S, int il, int k) {
    Hot H;
    H.cutoff_sq = S.cutoff_sq;
    H.ncut = S.ncutoffs;
    H.pt_base = S.pt_base;
    const float4 c = sm.cand[k], p = sm.i32[il];
    const int si = sm.isi[il];
    int sj, v;
    Entry<WIDE>::get(a.list_shift, sm.entry[k], sj, v);
    double off[3];
    visit_vector(a, S, v, off);
    return exact_inside<KIND>(H, a, a.pos64[si], a.pos64[sj], off, p.w, c.w);
}

// Appends n hits (code[c0 ..]) of atom il to its list, half a warp per atom (il,
// n, c0 differ by half; n = 0: none).
template <bool WIDE>
__device__ __forceinline__ void list_emit(ListWarp<WIDE> &sm, const TraverseArgs &a, int il, int n,
                                          int c0, int lane) {
    using E = Entry<WIDE>;
    const unsigned full = 0xffffffffu;
    const int l16 = lane & 15;
    const int start = n > 0 ? sm.icount[il] : 0;
    typename E::T *list = reinterpret_cast<typename E::T *>(a.list);
    if (__all_sync(full, n == 0 || start + n <= sm.lim[il])) {
        typename E::T *dst = list + (n > 0 ? sm.lw[il] : 0ll) + start;
        for (int r = l16; r < n; r += 16)
            if (!checked_fail(dst + r < list || dst + r >= list + a.list_cap * E::kPerGroup, a.err))
                dst[r] = sm.entry[sm.code[c0 + r]];
    } else {
        for (int h = 0; h < 32; h += 16) {  // a list that chains: the whole warp, atom by atom
            const int ilh = __shfl_sync(full, il, h), m = __shfl_sync(full, n, h);
            const int first = __shfl_sync(full, start, h), ch = __shfl_sync(full, c0, h);
            for (int done = 0; done < m;) {
                const int at = first + done;
                const int lim = sm.lim[ilh];
                const long long lw = sm.lw[ilh];
                if (lim < 0) break;
                const int take = min(m - done, lim - at);
                __syncwarp();
                if (take <= 0) {
                    if (lane == 0) {
                        const long long next = list_grow(a, (lw + lim) / E::kPerGroup);
                        if (next < 0) {
                            sm.lim[ilh] = -1;
                            sm.lw[ilh] = lim;
                        } else {
                            sm.lw[ilh] = next * E::kPerGroup - lim;
                            sm.lim[ilh] = lim + (kListChunk - 1) * E::kPerGroup;
                        }
                    }
                    __syncwarp();
                    continue;
                }
                for (int r = lane; r < take; r += 32)
                    if (!checked_fail(lw + at + r < 0 || lw + at + r >= a.list_cap * E::kPerGroup,
                                      a.err))
                        list[lw + at + r] = sm.entry[sm.code[ch + done + r]];
                done += take;
            }
        }
    }
    __syncwarp();
    if (n > 0 && l16 == 0) sm.icount[il] = start + n;
    __syncwarp();
}

// Force pass: n hits (code[c0 ..]) of atom il onto its force and energy share,
// half a warp per atom; a fixed order of summation throughout.
template <bool WIDE>
__device__ __forceinline__ void lj_emit(ListWarp<WIDE> &sm, double (*acc)[4], const TraverseArgs &a,
                                        const SysDev &S, int il, int n, int c0, int lane) {
    const unsigned full = 0xffffffffu;
    const int l16 = lane & 15;
    double f[4] = {0.0, 0.0, 0.0, 0.0};
    if (n > 0) {
        const double4 pi = a.pos64[sm.isi[il]];
#pragma unroll 2
        for (int r = l16; r < n; r += 16) {
            int sj, v;
            Entry<WIDE>::get(a.list_shift, sm.entry[sm.code[c0 + r]], sj, v);
            const double4 pj = a.pos64[sj];
            double off[3];
            visit_vector(a, S, v, off);
            const double dx = dadd(dsub(pj.x, pi.x), off[0]);
            const double dy = dadd(dsub(pj.y, pi.y), off[1]);
            const double dz = dadd(dsub(pj.z, pi.z), off[2]);
            const double r2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
            lj_pair(a, dx, dy, dz, r2, f);
        }
    }
    __syncwarp();
    // transposed: lane 4 k of the half ends with the half's sum of f[k]
    const bool up8 = l16 & 8, up4 = l16 & 4;
    double w0 = up8 ? f[2] : f[0], w1 = up8 ? f[3] : f[1];
    w0 += __shfl_xor_sync(full, up8 ? f[0] : f[2], 8);
    w1 += __shfl_xor_sync(full, up8 ? f[1] : f[3], 8);
    double x = up4 ? w1 : w0;
    x += __shfl_xor_sync(full, up4 ? w0 : w1, 4);
    x += __shfl_xor_sync(full, x, 2);
    x += __shfl_xor_sync(full, x, 1);
    if (n > 0 && (l16 & 3) == 0) acc[il][l16 >> 2] += x;
    __syncwarp();
}

// The hits of two atoms of the tile into their lists (LJ: onto their forces).  A lane's word holds its
// block's candidates from the top bit down.
template <bool WIDE, bool LJ>
__device__ __forceinline__ void list_pair(ListWarp<WIDE> &sm, double (*acc)[4],
                                          const TraverseArgs &a, const SysDev &S, unsigned wa,
                                          unsigned wb, int il, int blk, int lane) {
    const unsigned full = 0xffffffffu;
    if (!__any_sync(full, (wa | wb) != 0u)) return;
    const int mine = __popc(wa) | __popc(wb) << 16;
    int incl = mine;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int o = __shfl_up_sync(full, incl, s);
        if (lane >= s) incl += o;
    }
    const int tot = __shfl_sync(full, incl, 31);
    const int na = tot & 0xffff, nb = tot >> 16;
    const int k0 = lane * blk;
    const bool up = lane >= 16;
    if (na + nb <= kListCand) {
        uint16_t *pa = sm.code + ((incl - mine) & 0xffff), *pb = sm.code + na + ((incl - mine) >> 16);
#pragma unroll 4
        for (int t = 0; t < blk; t++) {
            if ((int)wa < 0) *pa++ = (uint16_t)(k0 + t);
            if ((int)wb < 0) *pb++ = (uint16_t)(k0 + t);
            wa <<= 1;
            wb <<= 1;
        }
        __syncwarp();
        if constexpr (LJ)
            lj_emit<WIDE>(sm, acc, a, S, up ? il + 1 : il, up ? nb : na, up ? na : 0, lane);
        else
            list_emit<WIDE>(sm, a, up ? il + 1 : il, up ? nb : na, up ? na : 0, lane);
    } else {  // more than the table holds: one after the other
        for (int h = 0; h < 2; h++) {
            uint16_t *p = sm.code + (h ? (incl - mine) >> 16 : (incl - mine) & 0xffff);
            unsigned w = h ? wb : wa;
            for (int t = 0; t < blk; t++, w <<= 1)
                if ((int)w < 0) *p++ = (uint16_t)(k0 + t);
            __syncwarp();
            if constexpr (LJ)
                lj_emit<WIDE>(sm, acc, a, S, il + h, up ? 0 : h ? nb : na, 0, lane);
            else
                list_emit<WIDE>(sm, a, il + h, up ? 0 : h ? nb : na, 0, lane);
        }
    }
}

// LJ: the pairs go into forces and energies (TraverseArgs::lj_*) instead of lists
// and counts: every hit is evaluated from the code list, half a warp per atom, so
// that the FP64 arithmetic runs with full lanes and the hits' records, consecutive
// in memory for the most part, are gathered together.  (One thread per atom pays
// it for the whole warp at almost every candidate.)  7,483 atoms: 101 -> 24 us,
// 200,001: 249 -> 198, a million: 996 -> 991.
template <int KIND, bool WIDE, bool CULL, bool LJ>
__global__ void __launch_bounds__(kListWarps * 32, list_blocks(WIDE, LJ))
k_count_list(const __grid_constant__ TraverseArgs a) {
    __shared__ double acc_all[LJ ? kListWarps : 1][LJ ? kITile : 1][4];
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    using E = Entry<WIDE>;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ListWarp<WIDE> &sm = reinterpret_cast<ListWarp<WIDE> *>(dyn_smem)[warp];
    double (*acc)[4] = acc_all[LJ ? warp : 0];
    if (LJ) {
        lj_note(a);
        if (a.lj_line > 0.f && lj_sparse(a)) return;
    }
    const int nitems = *a.n_items;
    ItemLoop L(a, (int)blockIdx.x * kListWarps + warp, nitems, lane, false);
    while (L.it < nitems) {
        L.prefetch(a, (int)gridDim.x * kListWarps, nitems, lane, false);
        const SysDev &S = a.sys[L.rec.sys];
        // --- the tile's atoms with rows in [i_lo, i_hi), in order ----------------
        int ni;
        {
            const int nt = item_bad(a, L.rec) ? 0 : L.rec.nt, si = L.rec.ib + lane;
            int at = 0;
            bool in = false;
            if (lane < nt) {
                at = a.aux[si].x;
                in = at >= a.i_lo && at < a.i_hi && !checked_fail(at < 0 || at >= a.natoms, a.err);
            }
            const unsigned im = __ballot_sync(full, in);
            ni = __popc(im);
            sm.i32[lane] = make_float4(kFarAtom, kFarAtom, kFarAtom, 0.f);
            if (LJ) {
#pragma unroll
                for (int k = 0; k < 4; k++) acc[lane][k] = 0.0;
            }
            __syncwarp();
            if (in) {
                const int t = __popc(im & lanemask_lt());
                sm.i32[t] = a.pos32[si];
                sm.isi[t] = si;
                sm.iatom[t] = at;
                sm.icount[t] = 0;
                sm.lw[t] = (S.list_base + (at - S.atom_base) * S.list_cap) * E::kPerGroup;
                sm.lim[t] = (S.list_cap - 1) * E::kPerGroup;
            }
        }
        float lo_rc, hi_rc, band;
        {
            const double b = guard_band(2.0 * (double)a.amax[L.rec.sys] + S.off_max, S.cutoff);
            lo_rc = __double2float_rd(S.cutoff_sq - b);
            hi_rc = __double2float_ru(S.cutoff_sq + b);
            band = __double2float_ru(b);
        }
        const float2 nhi = make_float2(-hi_rc, -hi_rc), nlo = make_float2(-lo_rc, -lo_rc);
        const float2 minus1 = make_float2(-1.f, -1.f);
        const bool sure_ok = KIND != kCutPerAtom || !(*a.err & kNoteWideRadius);
        const float rc2 = __double2float_rn(S.cutoff_sq);
        const float2 pband = make_float2(band, band), nband = make_float2(-band, -band);
        const int nvisit = S.nvisit;
        bool boxed = false;
        float blo[3] = {0.f, 0.f, 0.f}, bhi[3] = {0.f, 0.f, 0.f};
        for (int vb = 0; vb < nvisit && ni > 0; vb += kSeg) {
            int nseg, total, zs;
            list_setup(sm, a, S, L.rec, vb, lane, nseg, total, zs);
            if (CULL && !boxed) {
                boxed = true;
                const float4 p = sm.i32[min(lane, ni - 1)];
                const float c[3] = {p.x, p.y, p.z};
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    blo[k] = bhi[k] = c[k];
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) {
                        blo[k] = fminf(blo[k], __shfl_xor_sync(full, blo[k], d));
                        bhi[k] = fmaxf(bhi[k], __shfl_xor_sync(full, bhi[k], d));
                    }
                }
            }
            for (int kb = 0; kb < total;) {
                int nk;
                if (CULL) {
                    nk = list_stage_near(sm, a, nseg, total, vb, kb, zs, L.rec.ib, blo, bhi, hi_rc,
                                         lane);
                    if (nk == 0) continue;
                } else {
                    nk = min(kListCand, total - kb);
                    list_stage(sm, a, nseg, vb, kb, nk, zs, L.rec.ib, lane);
                    kb += nk;
                }
                const int blk = ((nk + 31) >> 5) | 1;
                for (int k = nk + lane; k < 32 * blk; k += 32)
                    sm.cand[k] = make_float4(kFarCand, kFarCand, kFarCand, 0.f);
                __syncwarp();
                const float4 *mine = sm.cand + lane * blk;
                for (int g0 = 0; g0 < ni; g0 += 4) {
                    const float4 p0 = sm.i32[g0], p1 = sm.i32[g0 + 1], p2 = sm.i32[g0 + 2],
                                 p3 = sm.i32[g0 + 3];
                    const float2 nx0 = make_float2(-p0.x, -p1.x), nx1 = make_float2(-p2.x, -p3.x);
                    const float2 ny0 = make_float2(-p0.y, -p1.y), ny1 = make_float2(-p2.y, -p3.y);
                    const float2 nz0 = make_float2(-p0.z, -p1.z), nz1 = make_float2(-p2.z, -p3.z);
                    const float2 wi0 = make_float2(p0.w, p1.w), wi1 = make_float2(p2.w, p3.w);
                    // one bit per candidate inside the outer threshold, and one per
                    // candidate inside the inner: the sign of r2 - threshold, shifted
                    // in (the comparison and the bit in one ALU operation)
                    unsigned near[4] = {0u, 0u, 0u, 0u}, sure[4] = {0u, 0u, 0u, 0u};
                    TypeRow row[4];
                    if (KIND == kCutPerType) {
                        row[0] = type_row(a, S, p0.w);
                        row[1] = type_row(a, S, p1.w);
                        row[2] = type_row(a, S, p2.w);
                        row[3] = type_row(a, S, p3.w);
                    }
#pragma unroll 2
                    for (int t = 0; t < blk; t++) {
                        const float4 c = mine[t];
                        const float2 x2 = make_float2(c.x, c.x), y2 = make_float2(c.y, c.y),
                                     z2 = make_float2(c.z, c.z);
                        float2 dx = __fadd2_rn(x2, nx0), dy = __fadd2_rn(y2, ny0),
                               dz = __fadd2_rn(z2, nz0);
                        const float2 ra =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        dx = __fadd2_rn(x2, nx1);
                        dy = __fadd2_rn(y2, ny1);
                        dz = __fadd2_rn(z2, nz1);
                        const float2 rb =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        float2 oa, ob, ia, ib;  // r2 - outer, r2 - inner
                        if (KIND == kCutPerAtom) {
                            const float2 w2 = make_float2(c.w, c.w);
                            const float2 sa = __fadd2_rn(w2, wi0), sb = __fadd2_rn(w2, wi1);
                            const float2 qa = __fmul2_rn(sa, sa), qb = __fmul2_rn(sb, sb);
                            // pair cutoffs never exceed the binning cutoff unless a
                            // radius does (then nothing counts as sure, below)
                            const float2 ea = __ffma2_rn(qa, minus1, ra),
                                         eb = __ffma2_rn(qb, minus1, rb);
                            oa = __fadd2_rn(ea, nband);
                            ob = __fadd2_rn(eb, nband);
                            ia = __fadd2_rn(ea, pband);
                            ib = __fadd2_rn(eb, pband);
                        } else if (KIND == kCutPerType) {
                            const int tj = __float_as_int(c.w);
                            const float2 ea = __fadd2_rn(ra, make_float2(type_cut(row[0], tj, rc2),
                                                                         type_cut(row[1], tj, rc2)));
                            const float2 eb = __fadd2_rn(rb, make_float2(type_cut(row[2], tj, rc2),
                                                                         type_cut(row[3], tj, rc2)));
                            oa = __fadd2_rn(ea, nband);
                            ob = __fadd2_rn(eb, nband);
                            ia = __fadd2_rn(ea, pband);
                            ib = __fadd2_rn(eb, pband);
                        } else {
                            oa = __fadd2_rn(ra, nhi);
                            ob = __fadd2_rn(rb, nhi);
                            ia = __fadd2_rn(ra, nlo);
                            ib = __fadd2_rn(rb, nlo);
                        }
                        near[0] = __funnelshift_l(__float_as_uint(oa.x), near[0], 1);
                        near[1] = __funnelshift_l(__float_as_uint(oa.y), near[1], 1);
                        near[2] = __funnelshift_l(__float_as_uint(ob.x), near[2], 1);
                        near[3] = __funnelshift_l(__float_as_uint(ob.y), near[3], 1);
                        sure[0] = __funnelshift_l(__float_as_uint(ia.x), sure[0], 1);
                        sure[1] = __funnelshift_l(__float_as_uint(ia.y), sure[1], 1);
                        sure[2] = __funnelshift_l(__float_as_uint(ib.x), sure[2], 1);
                        sure[3] = __funnelshift_l(__float_as_uint(ib.y), sure[3], 1);
                    }
                    // first candidate of the block at the top bit; an atom is not its
                    // own neighbour
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        near[g] <<= 32 - blk;
                        sure[g] <<= 32 - blk;
                        const int t = g0 + g < ni
                                          ? sm.self[sm.isi[g0 + g] - L.rec.ib] - lane * blk
                                          : -1;
                        if (t >= 0 && t < blk) near[g] &= ~(0x80000000u >> t);
                        sure[g] = sure_ok ? sure[g] & near[g] : 0u;
                    }
                    // what the filter leaves open
                    if (__any_sync(full, near[0] != sure[0] || near[1] != sure[1] ||
                                             near[2] != sure[2] || near[3] != sure[3])) {
#pragma unroll
                        for (int g = 0; g < 4; g++)
                            for (unsigned open = near[g] ^ sure[g]; open; open &= open - 1u) {
                                const unsigned low = open & (0u - open);
                                if (list_exact<KIND, WIDE>(sm, a, S, g0 + g,
                                                           lane * blk + __clz(low)))
                                    sure[g] |= low;
                            }
                        __syncwarp();
                    }
                    list_pair<WIDE, LJ>(sm, acc, a, S, sure[0], sure[1], g0, blk, lane);
                    if (g0 + 2 < ni)
                        list_pair<WIDE, LJ>(sm, acc, a, S, sure[2], sure[3], g0 + 2, blk, lane);
                }
            }
        }
        if (LJ) {
            if (lane < ni) {
                const int64_t at = sm.iatom[lane];
                a.lj_force[3 * at] = acc[lane][0];
                a.lj_force[3 * at + 1] = acc[lane][1];
                a.lj_force[3 * at + 2] = acc[lane][2];
                a.lj_energy[at] = acc[lane][3];
            }
        } else if (lane < ni) {
            a.counts[sm.iatom[lane]] = sm.icount[lane];
            if (sm.lim[lane] < 0) list_lacks(a, sm.icount[lane] - sm.lw[lane], E::kPerGroup);
        }
        __syncwarp();
        L.step();
    }
}

cudaError_t launch(TravKernel k, bool wide, bool lj, const TraverseArgs &a, int num_sms,
                   cudaStream_t st) {
    const int64_t grid =
        std::min<int64_t>((int64_t)num_sms * list_blocks(wide, lj), (a.natoms + 3) / 4);
    return launch_kernel(k, (wide ? sizeof(ListWarp<true>) : sizeof(ListWarp<false>)) * kListWarps,
                         kListWarps, a, (int)grid, st);
}

template <bool WIDE, bool CULL>
TravKernel count_kernel(int kind) {
    return kind == kCutPerAtom   ? k_count_list<kCutPerAtom, WIDE, CULL, false>
           : kind == kCutPerType ? k_count_list<kCutPerType, WIDE, CULL, false>
                                 : k_count_list<kCutScalar, WIDE, CULL, false>;
}

}  // namespace

cudaError_t launch_count_list(int kind, bool cull, const TraverseArgs &a, int num_sms, cudaStream_t st) {
    if (a.natoms <= 0) return cudaSuccess;
    const bool wide = a.list_wide != 0;
    return launch(wide ? (cull ? count_kernel<true, true>(kind) : count_kernel<true, false>(kind))
                       : (cull ? count_kernel<false, true>(kind) : count_kernel<false, false>(kind)),
                  wide, false, a, num_sms, st);
}

cudaError_t launch_lj_list(bool cull, const TraverseArgs &a, int num_sms, cudaStream_t st) {
    if (a.natoms <= 0) return cudaSuccess;
    const bool wide = a.list_wide != 0;
    return launch(wide ? (cull ? k_count_list<kCutScalar, true, true, true>
                               : k_count_list<kCutScalar, true, false, true>)
                       : (cull ? k_count_list<kCutScalar, false, true, true>
                               : k_count_list<kCutScalar, false, false, true>),
                  wide, true, a, num_sms, st);
}

}  // namespace nbl
