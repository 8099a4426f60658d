// brm_rankpack.cuh -- short rank rows, several at a time by one warp.
//
// Rows of at most kRkF0 products and 32 lists take the steps of the rank rows
// (brm_midrank.cuh), but a warp does up to eight of them together: the rows'
// column ranges are laid side by side (row s from summary word soff_s on), so
// that the lists, products and columns of all of them are one sequence, the
// columns in row order, and every step runs over full warps.  Only the list
// table and the output look at single rows.
//
// What bounds it: instruction issue.  A row on its own cost about 770 warp
// instructions for 67 products (512 uneven pairs), half of them fixed, and rows
// of up to 32 products 530 by a bitonic sort, 155 more to count them; together
// they take 560.  Rows of 2 to 128 products of those pairs, counting pass
// included: 1.55 -> 1.34 ms.
#pragma once

#include "brm_midrank.cuh"

namespace brm {

struct PackShape {
    static constexpr int BIN = kBinRank0;
    static constexpr int W = kMwRankCounter;  // work counter
    static constexpr int ROWS = 8;            // rows at a time
    static constexpr int NP = 8;              // products a lane
    static constexpr int F = 32 * NP;
    static constexpr int KM = 64;             // lists
    static constexpr int NSUM = 1 << (kRkRangeBits0 - 10);  // summary words
    static constexpr int WARPS = 8, CTAS = 4;
    // bytes of a warp (as RankShape: the values take the place of the words)
    static constexpr size_t o_cw = 0;
    static constexpr size_t o_summ = o_cw + 4 * F;
    static constexpr size_t o_srank = o_summ + 4 * NSUM;
    static constexpr size_t end_sum = o_srank + 2 * NSUM;
    static constexpr size_t o_mask = end_sum > 8 * F ? end_sum : 8 * F;
    static constexpr size_t o_uc = o_mask + 4 * F;
    static constexpr size_t o_pre = o_uc + 4 * F;
    static constexpr size_t o_tab = o_pre + 2 * F;
    static constexpr size_t o_av = o_tab + 16 * KM;
    static constexpr size_t o_ltab = o_av + 8 * KM;
    static constexpr size_t o_sb = o_ltab + 2 * KM;
    static constexpr size_t per_warp = mid_a16(o_sb + 4 * NP);
    static constexpr size_t bytes = per_warp * WARPS;
    static_assert(o_mask % 16 == 0 && o_tab % 16 == 0, "16-byte accesses");
    static_assert(kRkF0 <= F && kRkNarrowK <= KM, "one row fits");
    static_assert(ROWS * WARPS * CTAS == kRkRows[0], "plan_rank_spans counts by this");
    static_assert(ROWS * kRkF0 < 2048 && ROWS * kRkNarrowK < 512 && ROWS * NSUM < 4096,
                  "packed sums");
};

// Prefix of the bit counts of words[0, n) into pre by a warp, four words a
// lane; returns the total.
__device__ __forceinline__ int pack_words(const unsigned *words, int n, unsigned short *pre)
{
    int run = 0;
    for (int ib = 0; ib < n; ib += 128) {
        const int i = ib + 4 * (threadIdx.x & 31);
        uint4 s = make_uint4(0, 0, 0, 0);
        if (i < n)
            s = *(const uint4 *)&words[i];
        const int c0 = __popc(s.x), c1 = c0 + __popc(s.y), c2 = c1 + __popc(s.z);
        const int c3 = c2 + __popc(s.w);
        const int inc = warp_incl_scan(c3);
        const int ex = run + inc - c3;
        if (i < n)
            *(ushort4 *)&pre[i] =
                make_ushort4((unsigned short)ex, (unsigned short)(ex + c0),
                             (unsigned short)(ex + c1), (unsigned short)(ex + c2));
        run += __shfl_sync(kFull, inc, 31);
    }
    return run;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(32 * PackShape::WARPS, PackShape::CTAS)
    k_mid_pack(CsrDev A, CsrDev B, PlanDev P, const int *crpt, int *ccol, T *cval)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    using S = PackShape;
    constexpr int NP = S::NP;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const unsigned ltm = lanemask_lt(), lem = ltm | (1u << lane);
    unsigned char *ws = smem + (size_t)(threadIdx.x >> 5) * S::per_warp;
    unsigned *cw = (unsigned *)(ws + S::o_cw);
    T *vals = (T *)(ws + S::o_cw);
    unsigned *summ = (unsigned *)(ws + S::o_summ);
    unsigned short *srank = (unsigned short *)(ws + S::o_srank);
    unsigned *mask = (unsigned *)(ws + S::o_mask);
    int *ucol = (int *)(ws + S::o_uc);
    unsigned *quads = (unsigned *)(ws + S::o_uc);
    unsigned short *pre = (unsigned short *)(ws + S::o_pre);
    int4 *tab = (int4 *)(ws + S::o_tab);  // B offset, row's first column, its range, its place
    T *av = (T *)(ws + S::o_av);
    unsigned short *ltab = (unsigned short *)(ws + S::o_ltab);  // list | leaf << 6, nonempty lists
    unsigned *sb = (unsigned *)(ws + S::o_sb);
    const int M = A.M;
    const int n = P.cnt->bin_count[S::BIN];
    const int *rows = P.rows + (size_t)S::BIN * M;
    const int *__restrict__ bcol = B.col;
    const T *__restrict__ bval = (const T *)B.val;
    const T *__restrict__ aval = (const T *)A.val;
    int *work = &P.cnt->work_mw[S::W];
    // rows are taken ROWS at a time, fewer where the grid would run short
    const int nwarps = (int)gridDim.x * S::WARPS;
    const int claim = max(1, min(S::ROWS, n / nwarps));
    int nit = 0;
    if (lane == 0)
        nit = atomicAdd(work, claim);
    for (;;) {
        const int it = __shfl_sync(kFull, nit, 0);
        if (it >= n)
            break;
        if (lane == 0)
            nit = atomicAdd(work, claim);
        const int nr = min(claim, n - it);
        // lane r: row r of the claim
        int row = -1, a0 = 0, k = 0, f = 0, cmin = 0, crng = 0, sw = 0;
        if (lane < nr) {
            row = rows[it + lane];
            a0 = A.rpt[row];
            k = A.rpt[row + 1] - a0;
            f = P.flop[row];
            const int2 cr = P.crange[row];
            cmin = cr.x;
            crng = cr.y - cr.x;
            sw = (crng >> 10) + 1;
            const bool mine = row >= P.r_lo && row < P.r_hi;
            if (!mine || k > kRkNarrowK || f > kRkF0 || f <= 0 || crng < 0 || sw > S::NSUM) {
                if (mine)  // the analysis bins prevent this
                    atomicOr(&P.cnt->err, kErrWindowOverflow);
                row = -1;
                k = f = sw = 0;
            }
        }
        if (MODE == kMwSymbolic) {
            // short rows of few lists whose range takes so many words that two or
            // three would fill a pack: one by one, a product a lane (1.9 M rows of
            // 2 x 8 products over 2^17 columns, symbolic phase 0.99 -> 0.72 ms; 8 x 4
            // 0.58 -> 0.51; over 2^16 columns the pack is as fast)
            const bool alone = row >= 0 && f <= 32 && k <= 8 && sw > 64;
            for (unsigned m = __ballot_sync(kFull, alone); m; m &= m - 1u) {
                const int r = __ffs(m) - 1;
                const int ra0 = __shfl_sync(kFull, a0, r), rk = __shfl_sync(kFull, k, r);
                const int rmin = __shfl_sync(kFull, cmin, r), rrng = __shfl_sync(kFull, crng, r);
                int len = 0, bs = 0;
                if (lane < rk) {
                    len = P.alen[ra0 + lane];
                    bs = P.abs[ra0 + lane];
                }
                int bi = -1, at = 0;
                for (int l = 0; l < rk; l++) {
                    const int n = __shfl_sync(kFull, len, l);
                    const int b = __shfl_sync(kFull, bs, l) - at;
                    bi = lane >= at && lane < at + n ? b + lane : bi;
                    at += n;
                }
                const int c = bi >= 0 && BRM_IN(P.cnt, bi, B.nnz) ? bcol[bi] : INT_MAX;
                if (bi >= 0 && (unsigned)(c - rmin) > (unsigned)rrng)
                    atomicOr(&P.cnt->err, kErrUnsorted);
                const unsigned peers = __match_any_sync(kFull, c);
                const unsigned heads =
                    __ballot_sync(kFull, bi >= 0 && lane == __ffs(peers) - 1);
                if (lane == r)
                    P.nnz[row] = __popc(heads);
            }
            if (alone) {
                row = -1;
                k = f = sw = 0;
            }
        }
        for (int cur = 0; cur < nr;) {
            // the rows [cur, top) that fit together: products, lists, words
            const bool in = lane >= cur && lane < nr;
            const unsigned x =
                in ? (unsigned)f | ((unsigned)k << 11) | ((unsigned)sw << 20) : 0u;
            const unsigned inc = warp_incl_scan(x);
            const bool fit = (inc & 0x7ffu) <= (unsigned)S::F &&
                             ((inc >> 11) & 0x1ffu) <= (unsigned)S::KM &&
                             (inc >> 20) <= (unsigned)S::NSUM;
            const unsigned over = __ballot_sync(kFull, in && !fit);
            const int top = over ? __ffs(over) - 1 : nr;
            const unsigned all = __shfl_sync(kFull, inc, top - 1);
            const int F = (int)(all & 0x7ffu), K = (int)((all >> 11) & 0x1ffu);
            const int nsum = (int)(all >> 20);
            const int kp = (int)(((inc - x) >> 11) & 0x1ffu);  // lists before the lane's row
            const int soff = (int)((inc - x) >> 20);           // words before it
            const bool here = lane >= cur && lane < top && row >= 0;
            const int r0 = cur;
            cur = top;
            if (F == 0)
                continue;
            // 1. list table; summary and masks cleared
            for (int i = lane; i < (nsum + 3) >> 2; i += 32)
                ((uint4 *)summ)[i] = make_uint4(0, 0, 0, 0);
            if (MODE != kMwSymbolic)
                for (int i = lane; i < (F + 3) >> 2; i += 32)
                    ((uint4 *)mask)[i] = make_uint4(0, 0, 0, 0);
            if (lane < NP)
                sb[lane] = 0;
            __syncwarp();
            int nl = 0, fsum = 0;
            for (int q0 = 0; q0 < K; q0 += 32) {
                const int q = q0 + lane;
                int s = r0;
                for (int r = r0 + 1; r < top; r++)
                    s = q >= __shfl_sync(kFull, kp, r) ? r : s;
                const int j = q - __shfl_sync(kFull, kp, s);
                const int ra0 = __shfl_sync(kFull, a0, s);
                const int rmin = __shfl_sync(kFull, cmin, s), rrng = __shfl_sync(kFull, crng, s);
                const int rplace = __shfl_sync(kFull, soff, s) << 10;
                int len = 0, bs = 0;
                T a = T(0);
                if (q < K) {
                    len = P.alen[ra0 + j];
                    bs = P.abs[ra0 + j];
                    if (MODE != kMwSymbolic)  // no values in a symbolic call
                        a = aval[ra0 + j];
                }
                const int linc = warp_incl_scan(len);
                const int ex = fsum + linc - len;
                const unsigned ne = __ballot_sync(kFull, len > 0);
                if (len > 0 && ex + len <= S::F) {
                    tab[q] = make_int4(bs - ex, rmin, rrng, rplace);
                    av[q] = a;
                    ltab[nl + __popc(ne & ltm)] = (unsigned short)(q | (j << 6));
                    atomicOr(&sb[ex >> 5], 1u << (ex & 31));
                }
                fsum += __shfl_sync(kFull, linc, 31);
                nl += __popc(ne);
            }
            __syncwarp();
            if (fsum != F) {  // the analysis prevents this
                if (lane == 0)
                    atomicOr(&P.cnt->err, kErrWindowOverflow);
                __syncwarp();
                continue;
            }
            // 2. columns into registers, summary bits.  Lanes beyond the last
            //    product repeat it: all they mark, place or write is its own
            const int nw = (F + 31) >> 5;
            int jb = -1;
            int c[NP];        // place among the rows' columns
            unsigned pk[NP];  // list << 20 | leaf << 26 | word slot << 5 | column in the word; then
                              // u in the low bits
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int e = min(u * 32 + lane, F - 1);
                    const unsigned bits = sb[u];
                    const unsigned t = ltab[jb + __popc(bits & lem)];
                    jb += __popc(bits);
                    pk[u] = t << 20;
                    const int bi = tab[t & 63u].x + e;
                    c[u] = BRM_IN(P.cnt, bi, B.nnz) ? bcol[bi] : 0;
                }
            }
            bool bad = false;
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int4 t = tab[(pk[u] >> 20) & 63u];
                    int d = c[u] - t.y;
                    if ((unsigned)d > (unsigned)t.z) {
                        bad = true;  // rows of B that are not sorted
                        d = 0;
                    }
                    c[u] = d + t.w;
                    const unsigned b = 1u << ((c[u] >> 5) & 31);
                    if (!(summ[c[u] >> 10] & b))
                        atomicOr(&summ[c[u] >> 10], b);
                }
            }
            if (bad)
                atomicOr(&P.cnt->err, kErrUnsorted);
            __syncwarp();
            // 3. slots of the nonempty words, their bits, columns before each
            const int ncw = pack_words(summ, nsum, srank);
            for (int i = lane; i < (ncw + 3) >> 2; i += 32)
                ((uint4 *)cw)[i] = make_uint4(0, 0, 0, 0);
            __syncwarp();
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int w = c[u] >> 10;
                    const unsigned b = 1u << (c[u] & 31);
                    const int ci = srank[w] + __popc(summ[w] & ((1u << ((c[u] >> 5) & 31)) - 1u));
                    pk[u] |= ((unsigned)ci << 5) | (unsigned)(c[u] & 31);
                    if (BRM_IN(P.cnt, ci, S::F) && !(cw[ci] & b))
                        atomicOr(&cw[ci], b);
                }
            }
            __syncwarp();
            const int U = pack_words(cw, ncw, pre);
            __syncwarp();
            // the lane's row: its columns are [ub, ue)
            int ub = U, ue = U;
            if (lane >= r0 && lane < top && soff < nsum) {
                const int ci = srank[soff];
                ub = ci < ncw ? pre[ci] : U;
            }
            {
                const int nx = __shfl_down_sync(kFull, ub, 1);
                ue = lane + 1 < top ? nx : U;
            }
            if (MODE != kMwPrecise && here)
                P.nnz[row] = ue - ub;
            if (MODE == kMwSymbolic) {
                __syncwarp();
                continue;
            }
            long long base = 0;  // where its columns go, less ub
            bool out_in = here;
            if (here) {
                if (MODE == kMwPrecise) {
                    // a plan that does not match the input must not write past the row
                    base = crpt[row];
                    if (ue - ub != crpt[row + 1] - (int)base) {
                        atomicOr(&P.cnt->err, kErrNnzMismatch);
                        out_in = false;
                    }
                } else {
                    base = MODE == kMwUpper ? P.scan_flop[row] : P.mw_pre[row];
                }
                // checked build: the row's output must lie inside C (or the scratch)
                if (!BRM_IN(P.cnt, base + ue - ub - 1, MODE == kMwScratch ? P.mid_cap : P.c_cap))
                    out_in = false;
                base -= ub;
            }
            const unsigned outm = __ballot_sync(kFull, out_in);
            const int csub = (soff << 10) - cmin;  // place less column
            const bool nodup = U == F;
            // 4. column ranks, places, and the masks of leaves
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int ci = (int)((pk[u] >> 5) & 0x7fffu);
                    const int r = pre[ci] + __popc(cw[ci] & ((1u << (pk[u] & 31u)) - 1u));
                    pk[u] = (pk[u] & 0xfff00000u) | (unsigned)r;
                    if (!BRM_IN(P.cnt, r, S::F))
                        continue;
                    ucol[r] = c[u];
                    if (!nodup)
                        atomicOr(&mask[r], 1u << (pk[u] >> 26));
                }
            }
            __syncwarp();
            int nq = 0, nm = 0;
            unsigned short *mlist = pre + U;  // columns of several leaves (at most F - U)
            bool repeats = false;
            if (!nodup) {
                for (int ib = 0; ib < U; ib += 32) {
                    const int i = ib + lane;
                    const unsigned m = i < U ? mask[i] : 0u;
                    const bool multi = (m & (m - 1u)) != 0u;
                    const unsigned mb = __ballot_sync(kFull, multi);
                    if (multi && BRM_IN(P.cnt, U + nm + __popc(mb & ltm), S::F))
                        mlist[nm + __popc(mb & ltm)] = (unsigned short)i;
                    nm += __popc(mb);
                }
                __syncwarp();
                // their further leaves' positions, and the quads of leaves to
                // join (first member's position, second's, which are present)
                unsigned run = 0;  // positions taken | quads << 16
                for (int ib = 0; ib < nm; ib += 32) {
                    int i = 0;
                    unsigned m = 0, g = 0, cq = 0;
                    if (ib + lane < nm) {
                        i = mlist[ib + lane];
                        m = mask[i];
                        g = quads_to_join(m);
                        cq = (unsigned)(__popc(m) - 1) | ((unsigned)__popc(g) << 16);
                    }
                    const unsigned ci = warp_incl_scan(cq);
                    const unsigned at = run + ci - cq;
                    run += __shfl_sync(kFull, ci, 31);
                    if (ib + lane < nm) {
                        const int sp = U - 1 + (int)(at & 0xffffu);
                        int o = U + (int)(at >> 16);
                        pre[i] = (unsigned short)sp;
                        for (; g; g &= g - 1u) {
                            const int b = (__ffs(g) - 1) & ~3;
                            if (BRM_IN(P.cnt, o, S::F))
                                quads[o++] = Rank1::quad(sp, __popc(m & ((1u << b) - 1u)), i,
                                                         (m >> b) & 15u);
                        }
                    }
                }
                __syncwarp();
                nq = (int)(run >> 16);
                repeats = (int)(run & 0xffffu) != F - U;
            }
            if (repeats) {  // a column repeated within a list: row by row
                for (int r = r0; r < top; r++) {
                    const int rrow = __shfl_sync(kFull, row, r);
                    const int ra0 = __shfl_sync(kFull, a0, r), rk = __shfl_sync(kFull, k, r);
                    const int rub = __shfl_sync(kFull, ub, r), rue = __shfl_sync(kFull, ue, r);
                    const int rsub = __shfl_sync(kFull, csub, r);
                    const long long rb = __shfl_sync(kFull, base, r) + rub;
                    if (rrow >= 0 && (outm >> r & 1u))
                        rank_row_repeats<T>(B, P.cnt, P.abs + ra0, P.alen + ra0, aval + ra0, rk,
                                            ucol + rub, rue - rub, -rsub, lane, 32, ccol + rb,
                                            cval + rb);
                }
                __syncwarp();
                continue;
            }
            // 5. values to their positions
            T v[NP];
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int bi = tab[(pk[u] >> 20) & 63u].x + min(u * 32 + lane, F - 1);
                    v[u] = BRM_IN(P.cnt, bi, B.nnz) ? bval[bi] : T(0);
                }
            }
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    int p = (int)(pk[u] & 0xffffu);
                    if (!nodup) {
                        const int i = __popc(mask[p] & ((1u << (pk[u] >> 26)) - 1u));
                        if (i)
                            p = pre[p] + i;
                    }
                    if (BRM_IN(P.cnt, p, S::F))
                        vals[p] = vmul(av[(pk[u] >> 20) & 63u], v[u]);
                }
            }
            __syncwarp();
            // 6. the merge tree: quads of leaves, then what is above them
            if (!nodup) {
                for (int i = lane; i < nq; i += 32) {
                    const unsigned y = quads[U + i], q = y >> 26;
                    const int p = (int)(y & 0x1fffu), o = (int)((y >> 13) & 0x1fffu) - 1;
                    const int d1 = (int)(q & 1u), d2 = d1 + (int)((q >> 1) & 1u),
                              d3 = d2 + (int)((q >> 2) & 1u);
                    vals[p] = quad_value(vals, p, d1 ? o + d1 : p, d2 ? o + d2 : p, o + d3, q);
                }
                __syncwarp();
                for (int i = lane; i < nm; i += 32) {
                    const int u = mlist[i], sp = pre[u];
                    const unsigned m = mask[u], lo = m & 0xffffu, hi = m >> 16;
                    T r = T(0);
                    if (lo)
                        r = sixteen_value<T, false>(vals, u, sp, 0, lo);
                    if (hi) {
                        const T y = sixteen_value<T, false>(vals, u, sp, __popc(lo), hi);
                        r = lo ? vadd(r, y) : y;
                    }
                    vals[u] = r;
                }
                __syncwarp();
            }
            // the rows' columns, row by row
            for (int r = r0; r < top; r++) {
                if (!(outm >> r & 1u))
                    continue;
                const long long rb = __shfl_sync(kFull, base, r);
                const int rsub = __shfl_sync(kFull, csub, r);
                const int e = __shfl_sync(kFull, ue, r);
                for (int u = __shfl_sync(kFull, ub, r) + lane; u < e; u += 32) {
                    ccol[rb + u] = ucol[u] - rsub;
                    cval[rb + u] = vals[u];
                }
            }
            __syncwarp();
        }
    }
    // the last warp of the launch clears the counters for the next launch
    if (lane == 0) {
        __threadfence();
        if (atomicAdd(&P.cnt->done_mw[S::W], 1) == nwarps - 1) {
            atomicExch(work, 0);
            atomicExch(&P.cnt->done_mw[S::W], 0);
        }
    }
}

template <typename T, int MODE>
inline void launch_mid_pack(const CsrDev &A, const CsrDev &B, const PlanDev &P, const int *crpt,
                            int *ccol, T *cval, int num_sms, cudaStream_t s)
{
    using S = PackShape;
    if (!plan_live(P, live_bit(S::BIN)) || (P.rank_taken & 1u))
        return;
    cudaFuncSetAttribute(k_mid_pack<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)S::bytes);
    k_mid_pack<T, MODE>
        <<<num_sms * S::CTAS, 32 * S::WARPS, S::bytes, s>>>(A, B, P, crpt, ccol, cval);
    count_launch();
}

// The warp rows, the four-warp group rows and the tile rows of one mode, by
// rank or by merging.
// which: kMidGroups (the four-warp groups), kMidWarps (warp and tile rows) or
// both; classes without rows are not launched.
template <typename T, int MODE>
inline void launch_mid_warp(const CsrDev &A, const CsrDev &B, const PlanDev &P, const int *crpt,
                            int *ccol, T *cval, int num_sms, cudaStream_t s,
                            int which = kMidGroups | kMidWarps)
{
    if (which & kMidGroups) {
        if (plan_live(P, live_bit(kBinMidGroup2)))
            launch_mid_group<T, MODE, 5>(A, B, P, crpt, ccol, cval, num_sms, s);
        if (plan_live(P, live_bit(kBinMidGroup)))
            launch_mid_group<T, MODE, 4>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank5>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank7>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank9>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank4>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank3>(A, B, P, crpt, ccol, cval, num_sms, s);
    }
    if (which & kMidWarps) {
        launch_mid_rank<T, MODE, Rank6>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank2>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_rank<T, MODE, Rank1>(A, B, P, crpt, ccol, cval, num_sms, s);
        launch_mid_pack<T, MODE>(A, B, P, crpt, ccol, cval, num_sms, s);
        if (plan_live(P, live_bit(kBinMidWarp)))
            launch_mid_group<T, MODE, 1>(A, B, P, crpt, ccol, cval, num_sms, s);
        if (plan_live(P, live_bit(kBinMidTile2)))
            launch_mid_tile<T, MODE, 8>(A, B, P, crpt, ccol, cval, num_sms, s);
        if (plan_live(P, live_bit(kBinMidTile)))
            launch_mid_tile<T, MODE, 4>(A, B, P, crpt, ccol, cval, num_sms, s);
    }
}

}  // namespace brm
