// brm_midrank.cuh -- mid rows by ranking: a product's place is computed, not sorted.
//
// A row of at most 64 lists (A entries) is done by a group of G warps (short
// rows: several by one warp, brm_rankpack.cuh).  Where
// the merge kernels (brm_midwarp.cuh) sort every product's key, here the
// distinct columns are ranked with a bitmap and a product finds its place
// with population counts:
//
//   1. list table (leaf order) and one bit per list start in product order,
//      so that a product's list is a population count;
//   2. columns of all products into registers (a lane's products are 32
//      apart, so the gathers are coalesced); a bit per column in a bitmap of
//      the row's column range, or, where that is too wide, a summary bit per
//      nonempty 32-column word, whose ranks give the words compact slots;
//   3. the prefix of the words' counts ranks every product's column: u of the
//      row's U distinct columns (the symbolic phase stops here);
//   4. a mask of leaves per column: bit l set when list l holds the column.
//      A column's first leaf has position u; columns of several leaves get a
//      run of positions behind the U for the others, in leaf order (which
//      run does not matter), so a product's position is a population count,
//      whatever order the products are handled in, and columns of one
//      product, most of an irregular row, need nothing more;
//   5. values (coalesced gathers) to their positions;
//   6. the merge tree (BRMerge-SpGEMM/inc/spgemm.h:639-707: leaves a < b of a
//      column meet at the level of their highest differing bit, a lone child
//      passes through): its first two levels from a list of the quads of
//      leaves {4i .. 4i+3} with at least two present, so that every lane that
//      adds has something to add, the few levels above by a lane a column on
//      the way out.
//
// What bounds it: instruction issue (about 3 of 4 slots used).  This part has
// two FP64 lanes an SM (a DADD or DMUL holds the SM's unit for 16 cycles a
// warp), so the merge kernels' partly filled warps of additions cost as much
// as their instructions.  The 27-point stencil on 61x47x53, numeric phase
// (152 k rows, 729 products and 125 columns inside): merge kernel 2.08 ms,
// 16 warp instructions a product; this one 0.85 ms, 8 a product, the FP64
// unit 57 % busy.  Rows of 3..128 products of 512 uneven pairs: 1.84 ->
// 0.91 ms.
//
// Why several warps a row: the loops over a lane's products are unrolled over
// register arrays; one warp a row of 768 products (24 a lane) outgrew the
// instruction cache (3 to 15 stall cycles an instruction, 1.60 ms on the
// same stencil).  Rows of up to 384 products do better with one warp and 12 a
// lane (fewer warps that only pay a row's fixed cost): 0.66 -> 0.56 ms on
// the uneven pairs.
#pragma once

#include <climits>

#include "brm_check.cuh"
#include "brm_common.cuh"
#include "brm_mid.cuh"
#include "brm_midwarp.cuh"
#include "brm_plan.h"

namespace brm {

// Shapes.  G warps a row, NP products a lane: rows of at most F = 32 G NP
// products; WIDE: up to 64 lists (two mask words a column), else 32; the
// row's columns lie in a range below 2^RANGE; at most NFLAT words are a bitmap
// of all its columns.  DENSE: most columns have several products (a run of
// positions each); else those that do are listed and get a run for their
// second and further products, the first product of column u having position
// u.  GROUPS rows a CTA, CTAS on an SM.
template <int BIN_, int NP_, int G_, bool WIDE_, bool DENSE_, int RANGE_, int NFLAT_, int GROUPS_,
          int CTAS_>
struct RankShape {
    static constexpr int BIN = BIN_, NP = NP_, G = G_, RANGE = RANGE_, NFLAT = NFLAT_;
    static constexpr int W = kMwRankCounter + BIN - kBinRank0;  // work counter
    static constexpr bool WIDE = WIDE_, DENSE = DENSE_;
    static constexpr int GROUPS = GROUPS_, CTAS = CTAS_;
    static constexpr int NT = 32 * G;
    static constexpr int THREADS = NT * GROUPS;
    static constexpr int F = 32 * G * NP;
    static constexpr int CLAIM = F <= kRkF1 ? 4 : F <= kRkF2 ? 2 : 1;
    static constexpr int SM_ROWS = GROUPS * CTAS;  // rows of an SM at a time
    static constexpr int KM = WIDE ? 64 : 32;
    static constexpr int MW = WIDE ? 2 : 1;          // mask words a column
    static constexpr int NSUM = 1 << (RANGE - 10);   // summary words of the widest row
    // bytes of a group.  The bitmap words (compact ones, with the summary and
    // its ranks behind them, or all) give way to the values, the words'
    // prefixes to the columns' runs; the quads follow the U columns (a row
    // has at most F - U: each stands for an addition or more)
    static constexpr size_t o_cw = 0;
    static constexpr size_t o_summ = o_cw + 4 * F;
    static constexpr size_t o_srank = o_summ + 4 * NSUM;
    static constexpr size_t end_sum = o_srank + 2 * NSUM;
    static constexpr size_t end_x = end_sum > 8 * F ? mid_a16(end_sum) : 8 * F;
    static constexpr size_t o_mask = end_x > 4 * NFLAT ? end_x : 4 * NFLAT;
    static constexpr size_t o_uc = o_mask + 4 * MW * F;
    static constexpr size_t o_pre = o_uc + 4 * F;
    static constexpr size_t o_av = o_pre + 2 * (NFLAT > F ? NFLAT : F);
    static constexpr size_t o_lofs = o_av + 8 * KM;
    static constexpr size_t o_lleaf = o_lofs + 4 * KM;
    static constexpr size_t o_sb = o_lleaf + KM;
    static constexpr size_t o_gs = o_sb + mid_a16(4 * (F / 32));
    static constexpr size_t per_group = mid_a16(o_gs + 4 * (G + 1) + 16);
    static constexpr size_t bytes = per_group * GROUPS;
    // a quad to join in column i, its first member the column's r-th
    static __device__ __forceinline__ unsigned quad(int sp, int r, int i, unsigned members)
    {
        return (unsigned)(DENSE || r ? sp + r : i) | ((unsigned)(sp + r + 1) << 13) |
               (members << 26);
    }
    static_assert(F <= 8192, "positions are 13 bits");
    static_assert(RANGE <= 20, "columns are 20 bits beside the leaf");
    static_assert(bytes <= 227 * 1024, "shared memory of a CTA");
};

// Exclusive scan over the group of one value a thread; *tot the sum.
template <int G, typename V>
__device__ __forceinline__ V rank_scan(V v, V *gs, int gid, V *tot)
{
    const int lane = threadIdx.x & 31;
    const V inc = warp_incl_scan(v);
    if (G == 1) {
        *tot = __shfl_sync(kFull, inc, 31);
        return inc - v;
    }
    const int w = (threadIdx.x >> 5) % G;
    grp_sync<G>(gid);  // gs may still be read by a previous scan
    if (lane == 31)
        gs[w] = inc;
    grp_sync<G>(gid);
    V off, all;
    if (G <= 4) {
        off = all = 0;
#pragma unroll
        for (int i = 0; i < G; i++) {
            const V x = gs[i];
            off += i < w ? x : 0;
            all += x;
        }
    } else {
        const V x = lane < G ? gs[lane] : V(0);
        const V xi = warp_incl_scan(x);
        off = __shfl_sync(kFull, xi - x, w);
        all = __shfl_sync(kFull, xi, G - 1);
    }
    *tot = all;
    return off + inc - v;
}

// Prefix of the bit counts of words[0, n) into pre (four words a thread);
// returns the total.
template <class S>
__device__ __forceinline__ int rank_words(const unsigned *words, int n, unsigned short *pre,
                                          int *gs, int gid, int t)
{
    int run = 0;
    for (int ib = 0; ib < n; ib += 4 * S::NT) {
        const int i = ib + 4 * t;
        uint4 s = make_uint4(0, 0, 0, 0);
        if (i < n)
            s = *(const uint4 *)&words[i];
        const int c0 = __popc(s.x), c1 = c0 + __popc(s.y), c2 = c1 + __popc(s.z);
        int tot;
        const int ex = run + rank_scan<S::G, int>(c2 + __popc(s.w), gs, gid, &tot);
        if (i < n)
            *(ushort4 *)&pre[i] =
                make_ushort4((unsigned short)ex, (unsigned short)(ex + c0),
                             (unsigned short)(ex + c1), (unsigned short)(ex + c2));
        run += tot;
    }
    return run;
}

// Joins the present members of a quad of the merge tree: members at p0 <= p1
// <= p2 <= p3 (absent ones are not used), bit i of `in` set when member i is
// present; at least one is.
template <typename T>
__device__ __forceinline__ T quad_value(const T *vals, int p0, int p1, int p2, int p3, unsigned in)
{
    const T a = vals[p0], b = vals[p1], c = vals[p2], d = vals[p3];
    T l = (in & 1u) ? a : b;
    if ((in & 3u) == 3u)
        l = vadd(a, b);
    T r = (in & 4u) ? c : d;
    if ((in & 12u) == 12u)
        r = vadd(c, d);
    T v = (in & 3u) ? l : r;
    if ((in & 3u) && (in & 12u))
        v = vadd(l, r);
    return v;
}

// The value of the 16 leaves h (not 0) of a column, the first of them the
// column's i-th; leaf i > 0 of the column lies at s + i, leaf 0 at u (DENSE:
// at s too).
template <typename T, bool DENSE>
__device__ __forceinline__ T sixteen_value(const T *vals, int u, int s, int i, unsigned h)
{
    const unsigned in = ((h & 0xfu) ? 1u : 0u) | ((h & 0xf0u) ? 2u : 0u) |
                        ((h & 0xf00u) ? 4u : 0u) | ((h & 0xf000u) ? 8u : 0u);
    const int p0 = DENSE || i ? s + i : u;
    if ((in & (in - 1u)) == 0u)  // one quad
        return vals[p0];
    const int i1 = i + __popc(h & 0xfu), i2 = i + __popc(h & 0xffu), i3 = i + __popc(h & 0xfffu);
    return quad_value(vals, p0, DENSE || i1 ? s + i1 : u, DENSE || i2 ? s + i2 : u, s + i3, in);
}

// Bits 4i+3 set for the quads of m with at least two members.
__device__ __forceinline__ unsigned quads_to_join(unsigned m)
{
    const unsigned s = m - ((m >> 1) & 0x55555555u);
    return (((s & 0x33333333u) + ((s >> 2) & 0x33333333u)) + 0x66666666u) & 0x88888888u;
}

// What a rank row of f products reports when its B rows are not sorted (not
// valid CSR).  Rows of class 0's length were multiplied in any order before
// there were rank rows: the host then plans them again for the kernels that
// sort (PlanDev::any_order).  Longer ones are refused.
__device__ __forceinline__ int rank_unsorted(int f)
{
    return f <= kRkF0 ? kErrUnsorted : kErrBadInput;
}

// A row whose B rows repeat a column (not valid CSR, but summed all the same
// by the merge kernels: equal leaves meet first): every column by one
// thread, list by list.
template <typename T>
__device__ __noinline__ void rank_row_repeats(const CsrDev B, Counters *cnt, const int *abs,
                                              const int *alen, const T *arow, int k,
                                              const int *ucol, int U, int cmin, int t, int nt,
                                              int *ccol, T *cval)
{
    const int *bcol = B.col;
    const T *bval = (const T *)B.val;
    // (the search below needs sorted lists)
    bool sorted = true;
    int f = 0;
    for (int j = 0; j < k; j++) {
        f += alen[j];
        for (int i = abs[j] + t; i < abs[j] + alen[j] - 1; i += nt)
            sorted &= bcol[i] <= bcol[i + 1];
    }
    if (!sorted)
        atomicOr(&cnt->err, rank_unsorted(f));
    for (int u = t; u < U; u += nt) {
        const int c = cmin + ucol[u];
        ShiftReduce<T, 64> sr;
        sr.n = 0;
        for (int j = 0; j < k; j++) {
            const int s = abs[j], e = s + alen[j];
            for (int i = lower_bound_idx(bcol, s, e, c); i < e && bcol[i] == c; i++) {
                const T v = vmul(arow[j], bval[i]);
                if (sr.n == 0)
                    sr.init(j, v);
                else
                    sr.push(j, v);
            }
        }
        ccol[u] = c;
        cval[u] = sr.n ? sr.finish() : T(0);
    }
}

template <typename T, int MODE, class S>
__global__ void __launch_bounds__(S::THREADS, S::CTAS)
    k_mid_rank(CsrDev A, CsrDev B, PlanDev P, const int *crpt, int *ccol, T *cval)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    constexpr int G = S::G, NT = S::NT, NP = S::NP, MW = S::MW;
    extern __shared__ __align__(16) unsigned char smem[];
    const int gid = threadIdx.x / NT, t = threadIdx.x % NT;
    const int lane = threadIdx.x & 31, w = t >> 5;
    const unsigned ltm = lanemask_lt(), lem = ltm | (1u << lane);
    unsigned char *ws = smem + (size_t)gid * S::per_group;
    unsigned *cw = (unsigned *)(ws + S::o_cw);
    T *vals = (T *)(ws + S::o_cw);
    unsigned *summ = (unsigned *)(ws + S::o_summ);
    unsigned short *srank = (unsigned short *)(ws + S::o_srank);
    unsigned *mask = (unsigned *)(ws + S::o_mask);
    int *ucol = (int *)(ws + S::o_uc);
    unsigned *quads = (unsigned *)(ws + S::o_uc);
    unsigned short *pre = (unsigned short *)(ws + S::o_pre);
    T *av = (T *)(ws + S::o_av);              // A value, B offset by leaf
    int *lofs = (int *)(ws + S::o_lofs);
    unsigned char *lleaf = ws + S::o_lleaf;   // leaf of each nonempty list
    unsigned *sb = (unsigned *)(ws + S::o_sb);
    int *gs = (int *)(ws + S::o_gs);          // scan scratch, then row, F, counts
    int *gm = gs + G + 1;
    const int M = A.M;
    // rows of this class, then of the smaller ones it takes along
    const int b0 = S::BIN - P.rank_span[S::BIN - kBinRank0];
    int n = 0;
    for (int b = b0; b <= S::BIN; b++)
        n += P.cnt->bin_count[b];
    auto row_at = [&](int i) {
        if (i >= n)
            return -1;
        int b = S::BIN;
        for (; i >= P.cnt->bin_count[b]; b--)
            i -= P.cnt->bin_count[b];
        return P.rows[(size_t)b * M + i];
    };
    const int *__restrict__ bcol = B.col;
    const T *__restrict__ bval = (const T *)B.val;
    const T *__restrict__ aval = (const T *)A.val;
    // rows come S::CLAIM at a time from a counter (they differ in length, and one
    // address gives about 1.3 claims a nanosecond); the next one is looked up
    // while the present one is worked on
    const int claim = n >= 32 * S::GROUPS * (int)gridDim.x ? S::CLAIM : 1;
    int *work = &P.cnt->work_mw[S::W];
    int row = -1, nrow = -1, nit = 0;
    if (t == 0) {
        nit = atomicAdd(work, claim);
        nrow = row_at(nit);
    }
    for (;;) {
        if (G > 1) {
            if (t == 0)
                gm[0] = nrow;
            grp_sync<G>(gid);
            row = gm[0];
        } else {
            row = __shfl_sync(kFull, nrow, 0);
        }
        if (row < 0)
            break;
        if (t == 0) {
            nit++;
            if ((nit & (claim - 1)) == 0)
                nit = atomicAdd(work, claim);
        }
        const bool mine = row >= P.r_lo && row < P.r_hi;
        const int a0 = A.rpt[row];
        const int k = A.rpt[row + 1] - a0;
        const int2 cr = P.crange[row];
        const int cmin = cr.x, crng = cr.y - cr.x;
        const int nwords = (crng >> 5) + 1, nsum = (crng >> 10) + 1;
        const bool flat = nwords <= S::NFLAT;
        const bool fits = k <= S::KM && crng >= 0 && nsum <= S::NSUM;
        if (!mine || !fits) {
            if (mine && t == 0)  // the analysis bins prevent this
                atomicOr(&P.cnt->err, kErrWindowOverflow);
            if (t == 0)
                nrow = row_at(nit);
            grp_sync<G>(gid);
            continue;
        }
        // 1. list table by the first warp; the bitmap (or summary) cleared
        {
            uint4 *z = flat ? (uint4 *)cw : (uint4 *)summ;
            const int nz = ((flat ? nwords : nsum) + 3) >> 2;
            for (int i = t; i < nz; i += NT)
                z[i] = make_uint4(0, 0, 0, 0);
        }
        int F = 0;
        if (w == 0) {
            for (int i = lane; i < S::F / 32; i += 32)
                sb[i] = 0;
            __syncwarp();
            int nl = 0;
#pragma unroll
            for (int r = 0; r < S::KM / 32; r++) {
                if (r > 0 && k <= 32 * r)
                    break;
                const int j = 32 * r + lane;
                int len = 0, bs = 0;
                T a = T(0);
                if (j < k) {
                    len = P.alen[a0 + j];
                    bs = P.abs[a0 + j];
                    if (MODE != kMwSymbolic)  // no values in a symbolic call
                        a = aval[a0 + j];
                }
                const int inc = warp_incl_scan(len);
                const int ex = F + inc - len;
                const unsigned ne = __ballot_sync(kFull, len > 0);
                if (len > 0 && ex + len <= S::F) {
                    lofs[j] = bs - ex;
                    av[j] = a;
                    lleaf[nl + __popc(ne & ltm)] = (unsigned char)j;
                    atomicOr(&sb[ex >> 5], 1u << (ex & 31));
                }
                F += __shfl_sync(kFull, inc, 31);
                nl += __popc(ne);
            }
            if (G > 1 && lane == 0) {
                gm[1] = F;
                gm[2] = gm[3] = 0;
            }
        }
        if (t == 0)
            nrow = row_at(nit);
        grp_sync<G>(gid);
        if (G > 1)
            F = gm[1];
        if (F > S::F || F <= 0) {  // the analysis bins prevent this
            if (t == 0)
                atomicOr(&P.cnt->err, kErrWindowOverflow);
            grp_sync<G>(gid);
            continue;
        }
        if (MODE != kMwSymbolic)
            for (int i = t; i < (MW * F + 3) >> 2; i += NT)
                ((uint4 *)mask)[i] = make_uint4(0, 0, 0, 0);
        // 2. this warp's words of 32 products, [w0, w0 + nw).  Lanes beyond
        //    the last product repeat it: everything they mark, place or write
        //    is what its own lane does
        const int nwd = (F + 31) >> 5;
        const int npw = (nwd + G - 1) / G;
        const int w0 = w * npw;
        const int nw = min(npw, nwd - w0);
        int jb = -1;  // lists that start before the word, less one
        if (G > 1) {
            int c = 0;
            for (int i = lane; i < w0 && i < nwd; i += 32)
                c += __popc(sb[i]);
            jb += __reduce_add_sync(kFull, c);
        }
        int c[NP];        // column, from cmin
        unsigned pk[NP];  // leaf << 20 | word slot << 5 | column in the word, then leaf << 20 | u
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int e = min((w0 + u) * 32 + lane, F - 1);
                const unsigned bits = sb[w0 + u];
                const int l = lleaf[jb + __popc(bits & lem)];
                jb += __popc(bits);
                pk[u] = (unsigned)l << 20;
                const int bi = lofs[l] + e;
                c[u] = BRM_IN(P.cnt, bi, B.nnz) ? bcol[bi] : cmin;
            }
        }
        bool bad = false;
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                c[u] -= cmin;
                if ((unsigned)c[u] > (unsigned)crng) {
                    bad = true;  // rows of B that are not sorted
                    c[u] = 0;
                }
                const int x = flat ? c[u] : c[u] >> 5;
                unsigned *q = (flat ? cw : summ) + (x >> 5);
                const unsigned b = 1u << (x & 31);
                pk[u] |= (unsigned)c[u];
                if (!(*q & b))
                    atomicOr(q, b);
            }
        }
        if (bad)
            atomicOr(&P.cnt->err, rank_unsorted(F));
        grp_sync<G>(gid);
        int ncw = nwords;
        if (!flat) {
            // slots of the nonempty words
            ncw = rank_words<S>(summ, nsum, srank, gs, gid, t);
            for (int i = t; i < (ncw + 3) >> 2; i += NT)
                ((uint4 *)cw)[i] = make_uint4(0, 0, 0, 0);
            grp_sync<G>(gid);
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int sw = c[u] >> 10;
                    const unsigned b = 1u << (c[u] & 31);
                    const int ci = srank[sw] + __popc(summ[sw] & ((1u << ((c[u] >> 5) & 31)) - 1u));
                    pk[u] = (pk[u] & 0xfff0001fu) | ((unsigned)ci << 5);
                    if (BRM_IN(P.cnt, ci, S::F) && !(cw[ci] & b))
                        atomicOr(&cw[ci], b);
                }
            }
            grp_sync<G>(gid);
        }
        // 3. distinct columns, and those before each word
        const int U = rank_words<S>(cw, ncw, pre, gs, gid, t);
        if (MODE == kMwSymbolic) {
            if (t == 0)
                P.nnz[row] = U;
            grp_sync<G>(gid);
            continue;
        }
        long long base;
        bool out_in = true;
        if (MODE == kMwPrecise) {
            // a plan that does not match the input must not write past the row
            base = crpt[row];
            out_in = U == crpt[row + 1] - (int)base;
            if (t == 0 && !out_in)
                atomicOr(&P.cnt->err, kErrNnzMismatch);
        } else if (MODE == kMwUpper) {
            base = P.scan_flop[row];
        } else {
            base = P.mw_pre[row];
        }
        if ((MODE == kMwUpper || MODE == kMwScratch) && t == 0)
            P.nnz[row] = U;
        // the row's output must lie inside C (or the scratch): checked build
        if (!out_in || !BRM_IN(P.cnt, base + U - 1, MODE == kMwScratch ? P.mid_cap : P.c_cap)) {
            grp_sync<G>(gid);
            continue;
        }
        const bool nodup = U == F;
        grp_sync<G>(gid);
        // 4. column ranks, columns, and the masks of leaves
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int ci = (int)((pk[u] >> 5) & 0x7fffu);
                const int l = (int)(pk[u] >> 20);
                const int r = pre[ci] + __popc(cw[ci] & ((1u << (pk[u] & 31u)) - 1u));
                pk[u] = ((unsigned)l << 20) | (unsigned)r;
                if (!BRM_IN(P.cnt, r, S::F))
                    continue;
                ucol[r] = c[u];
                if (!nodup)
                    atomicOr(&mask[S::WIDE ? 2 * r + (l >> 5) : r], 1u << (l & 31));
            }
        }
        grp_sync<G>(gid);
        int nq = 0, nm = U;
        unsigned short *mlist = pre + U;  // columns of several leaves (at most F - U)
        if (!nodup) {
            if (!S::DENSE) {
                nm = 0;
                for (int ib = w * 32; ib < U; ib += NT) {
                    const int i = ib + lane;
                    unsigned m0 = 0, m1 = 0;
                    if (i < U) {
                        m0 = mask[MW * i];
                        if (S::WIDE)
                            m1 = mask[MW * i + 1];
                    }
                    const bool multi =
                        (m0 & (m0 - 1u)) || (S::WIDE && m1 && (m0 || (m1 & (m1 - 1u))));
                    const unsigned mb = __ballot_sync(kFull, multi);
                    int o = nm;
                    if (G > 1) {
                        if (mb) {
                            if (lane == 0)
                                o = atomicAdd(&gm[2], __popc(mb));
                            o = __shfl_sync(kFull, o, 0);
                        }
                    } else {
                        nm += __popc(mb);
                    }
                    if (multi && BRM_IN(P.cnt, U + o + __popc(mb & ltm), S::F))
                        mlist[o + __popc(mb & ltm)] = (unsigned short)i;
                }
                grp_sync<G>(gid);
                if (G > 1)
                    nm = gm[2];
            }
            // their runs, and the quads of leaves to join: the first member's
            // position, the second's (DENSE: the next), which are present
            unsigned run = 0;  // positions taken | quads << 16
            for (int ib = w * 32; ib < nm; ib += NT) {
                const int x = ib + lane;
                int i = 0;
                unsigned m0 = 0, m1 = 0, g0 = 0, g1 = 0, cq = 0;
                if (x < nm) {
                    i = S::DENSE ? x : mlist[x];
                    m0 = mask[MW * i];
                    g0 = quads_to_join(m0);
                    if (S::WIDE) {
                        m1 = mask[MW * i + 1];
                        g1 = quads_to_join(m1);
                    }
                    cq = (unsigned)(__popc(m0) + __popc(m1) - (S::DENSE ? 0 : 1)) |
                         ((unsigned)(__popc(g0) + __popc(g1)) << 16);
                }
                const unsigned inc = warp_incl_scan(cq);
                unsigned at;
                if (G > 1) {
                    at = 0;
                    if (lane == 31)
                        at = atomicAdd((unsigned *)&gm[3], inc);
                    at = __shfl_sync(kFull, at, 31);
                } else {
                    at = run;
                    run += __shfl_sync(kFull, inc, 31);
                }
                at += inc - cq;
                if (x < nm) {
                    const int sp = (S::DENSE ? 0 : U - 1) + (int)(at & 0xffffu);
                    int o = U + (int)(at >> 16);
                    pre[i] = (unsigned short)sp;
                    for (; g0; g0 &= g0 - 1u) {
                        const int b = (__ffs(g0) - 1) & ~3;
                        const int r = __popc(m0 & ((1u << b) - 1u));
                        if (BRM_IN(P.cnt, o, S::F))
                            quads[o++] = S::quad(sp, r, i, (m0 >> b) & 15u);
                    }
                    if (S::WIDE)
                        for (; g1; g1 &= g1 - 1u) {
                            const int b = (__ffs(g1) - 1) & ~3;
                            const int r = __popc(m0) + __popc(m1 & ((1u << b) - 1u));
                            if (BRM_IN(P.cnt, o, S::F))
                                quads[o++] = S::quad(sp, r, i, (m1 >> b) & 15u);
                        }
                }
            }
            grp_sync<G>(gid);
            if (G > 1)
                run = (unsigned)gm[3];
            nq = (int)(run >> 16);
            if ((int)(run & 0xffffu) != (S::DENSE ? F : F - U)) {  // a column repeated within a list
                rank_row_repeats<T>(B, P.cnt, P.abs + a0, P.alen + a0, aval + a0, k, ucol, U, cmin,
                                    t, NT, ccol + base, cval + base);
                grp_sync<G>(gid);
                continue;
            }
        }
        // 5. values to their positions
        T v[NP];
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int bi = lofs[pk[u] >> 20] + min((w0 + u) * 32 + lane, F - 1);
                v[u] = BRM_IN(P.cnt, bi, B.nnz) ? bval[bi] : T(0);
            }
        }
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int l = (int)(pk[u] >> 20);
                int p = (int)(pk[u] & 0xffffu);
                if (!nodup) {
                    const unsigned lt = (1u << (l & 31)) - 1u;
                    int i;  // leaves of the column below l
                    if (S::WIDE) {
                        const uint2 m = *(const uint2 *)&mask[2 * p];
                        i = l < 32 ? __popc(m.x & lt) : __popc(m.x) + __popc(m.y & lt);
                    } else {
                        i = __popc(mask[p] & lt);
                    }
                    if (S::DENSE || i)
                        p = pre[p] + i;
                }
                if (BRM_IN(P.cnt, p, S::F))
                    vals[p] = vmul(av[l], v[u]);
            }
        }
        grp_sync<G>(gid);
        // 6. the merge tree: quads of leaves, then what is above them
        if (!nodup) {
            for (int i = t; i < nq; i += NT) {
                const unsigned x = quads[U + i], q = x >> 26;
                const int p = (int)(x & 0x1fffu), o = (int)((x >> 13) & 0x1fffu) - 1;
                const int d1 = (int)(q & 1u), d2 = d1 + (int)((q >> 1) & 1u),
                          d3 = d2 + (int)((q >> 2) & 1u);
                vals[p] = S::DENSE ? quad_value(vals, p, p + d1, p + d2, p + d3, q)
                                   : quad_value(vals, p, d1 ? o + d1 : p, d2 ? o + d2 : p, o + d3, q);
            }
            grp_sync<G>(gid);
            if (S::DENSE || k > 4) {
                for (int x = t; x < nm; x += NT) {
                    const int u = S::DENSE ? x : mlist[x], sp = pre[u];
                    const int p0 = S::DENSE ? sp : u;
                    const unsigned m = mask[MW * u], lo = m & 0xffffu, hi = m >> 16;
                    T r = T(0);
                    if (lo)
                        r = sixteen_value<T, S::DENSE>(vals, p0, sp, 0, lo);
                    if (hi) {
                        const T y = sixteen_value<T, S::DENSE>(vals, p0, sp, __popc(lo), hi);
                        r = lo ? vadd(r, y) : y;
                    }
                    const unsigned m1 = S::WIDE ? mask[MW * u + 1] : 0u;
                    if (S::WIDE && m1) {
                        const unsigned lo1 = m1 & 0xffffu, hi1 = m1 >> 16;
                        const int i = __popc(m);
                        T y = T(0);
                        if (lo1)
                            y = sixteen_value<T, S::DENSE>(vals, p0, sp, i, lo1);
                        if (hi1) {
                            const T z = sixteen_value<T, S::DENSE>(vals, p0, sp, i + __popc(lo1), hi1);
                            y = lo1 ? vadd(y, z) : z;
                        }
                        r = m ? vadd(r, y) : y;
                    }
                    if (S::DENSE) {
                        ccol[base + u] = cmin + ucol[u];
                        cval[base + u] = r;
                    } else {
                        vals[u] = r;
                    }
                }
                grp_sync<G>(gid);
                if (S::DENSE)
                    continue;
            }
        }
        for (int u = t; u < U; u += NT) {
            ccol[base + u] = cmin + ucol[u];
            cval[base + u] = vals[u];
        }
        grp_sync<G>(gid);
    }
    // the last group of the launch clears the counters for the next launch
    // (its own taken items and every other group's are ordered before)
    if (t == 0) {
        __threadfence();
        if (atomicAdd(&P.cnt->done_mw[S::W], 1) == (int)gridDim.x * S::GROUPS - 1) {
            atomicExch(work, 0);
            atomicExch(&P.cnt->done_mw[S::W], 0);
        }
    }
}

// The classes from 1 on (their limits: kRk* in brm_plan.h; class 0:
// brm_rankpack.cuh).  CTAs an SM by shared memory
// or by registers, whichever ends first.  Most columns have several products
// where rows are long and lists many (class 2: stencils, finite elements; of
// distinct columns, 20 lists of 30 products over 2^17 columns, it takes 0.20 ms,
// merged 0.29), few where lists are long and few (power-law graphs).  Rows of 33 to 64 lists are
// both: class 7 holds those of more products than columns in their range, class
// 9 the others.  Numeric phase, as class 7 and as class 9: 64 lists of 20 products
// over 2^17 columns 0.82 and 0.67 ms (merged, before the rank rows: 0.71), 48 of 48
// over 1537 columns 0.54 and 0.54, over 289 columns 0.38 and 0.41.
using Rank1 = RankShape<kBinRank0 + 1, 12, 1, false, false, 19, 384, 4, 6>;
using Rank2 = RankShape<kBinRank0 + 2, 6, 4, false, true, 19, 1536, 1, 10>;
using Rank3 = RankShape<kBinRank0 + 3, 12, 4, false, false, 19, 1536, 1, 7>;
using Rank4 = RankShape<kBinRank0 + 4, 12, 8, false, false, 19, 3072, 1, 4>;
using Rank5 = RankShape<kBinRank0 + 5, 12, 16, false, false, 19, 6144, 1, 2>;
using Rank6 = RankShape<kBinRank0 + 6, 6, 4, true, false, 19, 768, 1, 8>;
using Rank7 = RankShape<kBinRank0 + 7, 12, 8, true, true, 19, 3072, 1, 3>;
using Rank9 = RankShape<kBinRank9, 12, 8, true, false, 19, 3072, 1, 3>;
static_assert(Rank1::F == kRkF1 && Rank2::F == kRkF2 && Rank3::F == kRkF3 &&
                  Rank4::F == kRkF4 && Rank5::F == kRkF5 && Rank6::F == kRkF2 && Rank7::F == kRkF4 &&
                  Rank9::F == kRkF4,
              "the analysis bins by these");
static_assert(Rank1::SM_ROWS == kRkRows[1] && Rank2::SM_ROWS == kRkRows[2] &&
                  Rank3::SM_ROWS == kRkRows[3] && Rank4::SM_ROWS == kRkRows[4] &&
                  Rank5::SM_ROWS == kRkRows[5],
              "plan_rank_spans counts by these");

template <typename T, int MODE, class S>
inline void launch_mid_rank(const CsrDev &A, const CsrDev &B, const PlanDev &P, const int *crpt,
                            int *ccol, T *cval, int num_sms, cudaStream_t s)
{
    if (!plan_live(P, live_bit(S::BIN)) || (P.rank_taken >> (S::BIN - kBinRank0) & 1u))
        return;
    cudaFuncSetAttribute(k_mid_rank<T, MODE, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)S::bytes);
    k_mid_rank<T, MODE, S><<<num_sms * S::CTAS, S::THREADS, S::bytes, s>>>(A, B, P, crpt, ccol,
                                                                            cval);
    count_launch();
}

}  // namespace brm
