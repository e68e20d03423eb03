// nbl_lj.cu -- Lennard-Jones forces and energies straight from the work items:
// candidates, pair test and force in one kernel, with no counts, hit words,
// row offsets or pairs in memory.
//
// One warp per work item (home cell x tile of up to 32 atoms).  The visited
// cells' atoms are staged in shared memory as FP32 positions in the home
// cell's frame and swept against four atoms at a time (packed f32x2, 32
// candidates per ballot); the filter only has to keep every pair of the list,
// because each kept candidate is then decided by the reference's exact FP64
// test.  Two atoms are taken together from there, one per half warp: the
// sweep leaves an atom's hit words in its own 16 lanes, they are listed as
// 16-bit candidate numbers, lane L of the half takes every 16th hit, and its
// partial force and energy stay in registers until one transposed reduction
// per atom (10 shuffles for two atoms).  Every sum has a fixed order, so the
// results are the same bits every run.
//
// What bounds it: instruction issue and the gathers of the hits' FP64
// positions; no HBM traffic to speak of.
#include "nbl_traverse.cuh"

namespace nbl {
namespace {

constexpr int kLjCand = 512;   // candidates staged at a time: 16 chunks, one per lane of a half
constexpr int kLjWarps = 2;
constexpr int kLjBlocks = 8;   // CTAs per SM (registers and shared memory)

struct __align__(16) LjWarp {
    SegSmem sg;
    float x[kLjCand], y[kLjCand], z[kLjCand];
    double4 i64[kITile];
    float4 i32[kITile];
    double acc[kITile][4];      // force and energy share per atom of the tile
    int32_t isi[kITile];
    uint16_t tab[2][kLjCand];   // hits of the two atoms in hand
    uint8_t cseg[kLjCand];
};
static_assert(kLjBlocks * (kLjWarps * sizeof(LjWarp) + 1024) <= 233472,
              "the CTAs fit the SM's shared memory");

// Candidates kb .. kb + nk of the batch into shared memory (home frame), padded
// to whole chunks with far points; cseg gets each one's segment.
__device__ __forceinline__ void lj_stage(LjWarp &sm, const TraverseArgs &a, int nseg, int kb,
                                         int nk, int lane) {
    __syncwarp();
    const int total = sm.sg.pref[nseg];
    if (total > 48 * nseg) {  // long cells: lane = candidate
        int seg = lane < nk ? seg_of(sm.sg, nseg, kb + lane) : 0;
        for (int k = lane; k < nk; k += 32) {
            while (seg + 1 < nseg && sm.sg.pref[seg + 1] <= kb + k) seg++;
            const float4 p = a.pos32[sm.sg.rec[seg].bj + kb + k];
            sm.x[k] = p.x + sm.sg.off32[seg][0];
            sm.y[k] = p.y + sm.sg.off32[seg][1];
            sm.z[k] = p.z + sm.sg.off32[seg][2];
            sm.cseg[k] = (uint8_t)seg;
        }
    } else if (lane < nseg) {  // short cells: lane = segment
        const int s0 = max(sm.sg.pref[lane], kb), s1 = min(sm.sg.pref[lane + 1], kb + nk);
        const float ox = sm.sg.off32[lane][0], oy = sm.sg.off32[lane][1],
                    oz = sm.sg.off32[lane][2];
        const float4 *src = a.pos32 + sm.sg.rec[lane].bj;
#pragma unroll 4
        for (int kk = s0; kk < s1; kk++) {
            const float4 p = src[kk];
            sm.x[kk - kb] = p.x + ox;
            sm.y[kk - kb] = p.y + oy;
            sm.z[kk - kb] = p.z + oz;
            sm.cseg[kk - kb] = (uint8_t)lane;
        }
    }
    const int nkp = (nk + 31) & ~31;
    if (nk + lane < nkp) sm.x[nk + lane] = sm.y[nk + lane] = sm.z[nk + lane] = kFarCand;
    __syncwarp();
}

// Sums of f over the 16 lanes of each half: lane 4 q of the half gets
// component q (every lane of its group of four does).
__device__ __forceinline__ double lj_reduce(const double f[4], int lane) {
    const unsigned full = 0xffffffffu;
    const bool up = (lane & 8) != 0, odd = (lane & 4) != 0;
    double a0 = up ? f[2] : f[0], a1 = up ? f[3] : f[1];
    a0 += __shfl_xor_sync(full, up ? f[0] : f[2], 8);
    a1 += __shfl_xor_sync(full, up ? f[1] : f[3], 8);
    double b = odd ? a1 : a0;
    b += __shfl_xor_sync(full, odd ? a0 : a1, 4);
    b += __shfl_xor_sync(full, b, 2);
    b += __shfl_xor_sync(full, b, 1);
    return b;
}

template <int KIND>
__global__ void __launch_bounds__(kLjWarps * 32, kLjBlocks)
k_lj(const __grid_constant__ TraverseArgs a) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, l16 = lane & 15;
    LjWarp &sm = reinterpret_cast<LjWarp *>(dyn_smem)[warp];
    const int nitems = *a.n_items;
    ItemLoop L(a, (int)blockIdx.x * kLjWarps + warp, nitems, lane, false);
    while (L.it < nitems) {
        L.prefetch(a, (int)gridDim.x * kLjWarps, nitems, lane, false);
        const Home c = load_home<true, false>(a, L.rec);
        const Hot &H = c.H;
        // --- the tile's atoms with rows in [i_lo, i_hi), in order ----------------
        int ni;
        {
            const int nt = item_bad(a, L.rec) ? 0 : L.rec.nt, si = L.rec.ib + lane;
            double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
            bool in = false;
            if (lane < nt) {
                p = a.pos64[si];
                const int ax = __double2loint(p.w);
                in = ax >= a.i_lo && ax < a.i_hi;
            }
            const unsigned im = __ballot_sync(full, in);
            ni = __popc(im);
            if (in) {
                const int t = __popc(im & lanemask_lt());
                sm.i64[t] = p;
                sm.i32[t] = a.pos32[si];
                sm.isi[t] = si;
            }
            if (lane >= ni) sm.i32[lane] = make_float4(kFarAtom, kFarAtom, kFarAtom, 0.f);
            sm.acc[lane][0] = sm.acc[lane][1] = sm.acc[lane][2] = sm.acc[lane][3] = 0.0;
            __syncwarp();
        }
        for (int vb = 0; vb < c.nvisit && ni > 0; vb += kSeg) {
            int nseg, total, zs;
            setup_segments(sm.sg, a, c, vb, lane, nseg, total, zs);
            const int kself0 = (zs >= 0) ? sm.sg.pref[zs] - sm.sg.b[zs] : INT_MIN / 2;
            for (int kb = 0; kb < total; kb += kLjCand) {
                const int nk = min(kLjCand, total - kb);
                const int nck = (nk + 31) >> 5;
                lj_stage(sm, a, nseg, kb, nk, lane);
                for (int g0 = 0; g0 < ni; g0 += 4) {
                    // --- sweep: four atoms, words of atoms g0, g0 + 1 in the two
                    //     halves of w01, of g0 + 2, g0 + 3 in those of w23 ---------
                    const float4 p0 = sm.i32[g0], p1 = sm.i32[g0 + 1], p2 = sm.i32[g0 + 2],
                                 p3 = sm.i32[g0 + 3];
                    const float2 nx0 = make_float2(-p0.x, -p1.x), nx1 = make_float2(-p2.x, -p3.x);
                    const float2 ny0 = make_float2(-p0.y, -p1.y), ny1 = make_float2(-p2.y, -p3.y);
                    const float2 nz0 = make_float2(-p0.z, -p1.z), nz1 = make_float2(-p2.z, -p3.z);
                    unsigned w01 = 0u, w23 = 0u;
                    for (int ch = 0; ch < nck; ch++) {
                        const int k = ch * 32 + lane;
                        const float cx = sm.x[k], cy = sm.y[k], cz = sm.z[k];
                        const float2 x2 = make_float2(cx, cx), y2 = make_float2(cy, cy),
                                     z2 = make_float2(cz, cz);
                        float2 dx = __fadd2_rn(x2, nx0), dy = __fadd2_rn(y2, ny0),
                               dz = __fadd2_rn(z2, nz0);
                        const float2 ra =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        dx = __fadd2_rn(x2, nx1);
                        dy = __fadd2_rn(y2, ny1);
                        dz = __fadd2_rn(z2, nz1);
                        const float2 rb =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        const unsigned m0 = __ballot_sync(full, ra.x < H.hi_rc);
                        const unsigned m1 = __ballot_sync(full, ra.y < H.hi_rc);
                        const unsigned m2 = __ballot_sync(full, rb.x < H.hi_rc);
                        const unsigned m3 = __ballot_sync(full, rb.y < H.hi_rc);
                        if (l16 == ch) {
                            w01 = half ? m1 : m0;
                            w23 = half ? m3 : m2;
                        }
                    }
#pragma unroll 1
                    for (int pr = 0; pr < 2 && g0 + 2 * pr < ni; pr++) {
                        const int il = g0 + 2 * pr + half;
                        const bool row = il < ni;
                        unsigned word = row ? (pr ? w23 : w01) : 0u;
                        if (row) {  // an atom is not its own neighbour
                            const int ks = kself0 + sm.isi[il] - kb;
                            if (ks >= 0 && (ks >> 5) == l16 && ks < nk) word &= ~(1u << (ks & 31));
                        }
                        // --- the hits of each half's atom as a list ---------------
                        const int p = __popc(word);
                        int incl = p;
#pragma unroll
                        for (int s = 1; s < 16; s <<= 1) {
                            const int o = __shfl_up_sync(full, incl, s, 16);
                            if (l16 >= s) incl += o;
                        }
                        const int n = __shfl_sync(full, incl, 15, 16);
                        {
                            uint16_t *t = sm.tab[half] + (incl - p);
                            const int base = l16 * 32;
                            for (; word; word &= word - 1u)
                                *t++ = (uint16_t)(base + __ffs(word) - 1);
                        }
                        __syncwarp();
                        // --- every 16th hit per lane ------------------------------
                        double f[4] = {0.0, 0.0, 0.0, 0.0};
                        const double4 pi = sm.i64[row ? il : 0];
                        for (int r = l16; r < n; r += 16) {
                            const int k = sm.tab[half][r];
                            const SegRec &g = sm.sg.rec[sm.cseg[k]];
                            const int sj = g.bj + kb + k;
                            if (checked_fail(sj < 0 || sj >= a.natoms, a.err)) continue;
                            const double4 pj = a.pos64[sj];
                            const double dx = dadd(dsub(pj.x, pi.x), g.off[0]);
                            const double dy = dadd(dsub(pj.y, pi.y), g.off[1]);
                            const double dz = dadd(dsub(pj.z, pi.z), g.off[2]);
                            const double r2 =
                                dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
                            bool in = r2 < H.cutoff_sq;
                            if (KIND != kCutScalar && in)
                                in = exact_inside<KIND>(
                                    H, a, pi, pj, g.off,
                                    KIND == kCutPerType ? sm.i32[il].w : 0.f,
                                    KIND == kCutPerType ? a.pos32[sj].w : 0.f);
                            if (in) lj_pair(a, dx, dy, dz, r2, f);
                        }
                        const double s = lj_reduce(f, lane);
                        if (row && (lane & 3) == 0) sm.acc[il][l16 >> 2] += s;
                        __syncwarp();
                    }
                }
            }
        }
        if (lane < ni) {
            const long long ax = __double2loint(sm.i64[lane].w);
            if (!checked_fail(ax < 0 || ax >= a.natoms, a.err)) {
                a.lj_force[3 * ax + 0] = sm.acc[lane][0];
                a.lj_force[3 * ax + 1] = sm.acc[lane][1];
                a.lj_force[3 * ax + 2] = sm.acc[lane][2];
                a.lj_energy[ax] = sm.acc[lane][3];
            }
        }
        __syncwarp();
        L.step();
    }
}

TravKernel lj_kernel(int kind) {
    if (kind == kCutPerAtom) return k_lj<kCutPerAtom>;
    if (kind == kCutPerType) return k_lj<kCutPerType>;
    return k_lj<kCutScalar>;
}

}  // namespace

cudaError_t launch_lj_items(int kind, const TraverseArgs &a, int num_sms, cudaStream_t st) {
    const size_t smem = sizeof(LjWarp) * kLjWarps;
    const int64_t grid = std::min<int64_t>((int64_t)num_sms * kLjBlocks,
                                           std::max<int64_t>((a.natoms + 1) / kLjWarps, 1));
    return launch_kernel(lj_kernel(kind), smem, kLjWarps, a, (int)grid, st);
}

}  // namespace nbl
