// brm_seg.cuh -- segmented processing of heavy rows.
//
// A heavy row (more products or lists than a mid-row batch holds) is cut into
// column segments [c_lo, c_hi).  Columns of C are independent, so the merge
// tree of the row restricted to a column range is the same tree with every
// list restricted to that range (BRMerge-SpGEMM/inc/spgemm.h:639-707): the
// leaf index of a product, and therefore the order of its additions, does
// not depend on the cut.  Three steps:
//
//   1. planning (symbolic phase, one CTA per heavy row, longest rows first):
//      a bitmap of the row's columns and a product count per 128-column group
//      over chunks of kPlanBits columns give the row's exact nnz and the cut
//      points: a cut before group g when the running product count crosses a
//      multiple of the cut target (at most kSegCut, a runtime knob) and
//      around groups holding more than kSegCap minus the target (inside such
//      a group the cuts are per column, from 16-bit per-column counts); a
//      segment then holds <= kSegCap products.  Its
//      output offset within the row (distinct columns before c_lo) comes
//      from the same bitmap.
//   2. split table (numeric phase): for every segment boundary and every list
//      of the row, the first list position at or after the boundary column
//      (one block per boundary, one binary search per list).
//   3. segment kernel (numeric phase, one CTA pass per segment): the
//      segment's columns into registers in list-major order; the rank u of
//      every product's column among the segment's distinct columns comes from
//      a bitmap (of all columns, or a summary bit per nonempty 32-column word
//      and the compressed words); a shared counter a column gives a product
//      its turn, its first one position u and the others a run of positions
//      behind the columns, so columns of one product are done when their
//      value is placed.  The others are listed by size: two products by a
//      lane, three or four by a lane in registers (closed forms), up to 8, 16
//      and 32 by that many lanes (leaf order by counting, then the tree),
//      more are put in leaf order by a warp and handed to the column reducer
//      (step 4).  Column u is stored at position u of the row's segment
//      (coalesced).
//   4. column reducer: one warp per long column.
//
// What bounds the segment kernel: latency and issue (three CTAs of eight warps
// an SM, about half of the issue slots).  R-MAT n=2^18, 4.1e7 products in
// 17.9 k segments: 1147 us when every product's column, value, leaf, rank and
// turn were staged in shared memory (111 KB, two CTAs an SM), 915 with the
// columns in registers, 747 with columns of up to 32 products reduced in
// place by groups of lanes (825 since its rows of 3073 to 5888 products are cut
// into segments too, 178 us less elsewhere).  A lane a column instead of a group
// took 979 us with 12 % fewer instructions, the size lists claimed once a warp by
// ballots 883, the next segment's split entries prefetched 831.
#pragma once

#include <climits>

#include "brm_check.cuh"
#include "brm_common.cuh"
#include "brm_mid.cuh"
#include "brm_plan.h"

namespace brm {

constexpr int kPlanThreads = 512;
// Segment cuts are placed at planning-group boundaries (kPlanGroupBits
// columns); a dense group (more than kSegCap - cut products) is a segment of
// its own, and one above kSegCap products gets per-column counts and is cut
// inside (at most kDenseGroups such groups per chunk).
constexpr int kPlanGroupLog2 = 7;
constexpr int kPlanGroupBits = 1 << kPlanGroupLog2;      // 128 columns
constexpr int kPlanGroupWords = kPlanGroupBits / 32;     // 4 bitmap words
static_assert(kPlanGroupWords == 4, "one 16-byte access a group");
constexpr int kPlanGroups = kPlanBits / kPlanGroupBits;  // 2048 per chunk
constexpr int kDenseGroups = 128;  // 16-bit column counts: a count is at most k <= 65535

static_assert(2 * kPlanThreads * 8 / 32 <= kPlanThreads, "the bits of two windows");

struct PlanLayout {
    static constexpr size_t o_bm = 0;
    static constexpr size_t o_hist = o_bm + kPlanWords * 4;
    static constexpr size_t o_gpop = o_hist + kPlanGroups * 4;
    static constexpr size_t o_dix = o_gpop + kPlanGroups * 2;
    static constexpr size_t o_ccnt = o_dix + kPlanGroups * 2;
    static constexpr size_t o_lst = o_ccnt + kDenseGroups * kPlanGroupBits * 2;
    static constexpr size_t o_starts = o_lst + kPlanThreads * 4;  // two windows of starts
    static constexpr size_t o_ws = o_starts + kPlanThreads * 4;
    static constexpr size_t o_misc = o_ws + (kPlanThreads / 32 + 1) * 8;
    static constexpr size_t bytes = o_misc + 64;
};

// Calls f(rc) for every product of the row, rc = column - base; with clip,
// only for the products whose column lies in [lo, chi) (each list is cut by
// binary search).  The lists are taken NT at a time and their products in
// windows of NT * kPlanPer: a bit per list start in product order (starts)
// tells a product its list by a population count, and a warp's loads are
// consecutive within a list.  lst (NT ints, a list's place in B less its first
// product) and starts (two windows of bits) are shared scratch.
constexpr int kPlanPer = 8;
template <int NT, typename Fn>
__device__ __forceinline__ void plan_products(const PlanDev &P, const int *__restrict__ bcol,
                                              int a0, int k, bool clip, int lo, int chi, int base,
                                              int *lst, unsigned *starts, long long *ws, Fn f)
{
    constexpr int W = NT * kPlanPer, NWD = W / 32;  // products and words of a window
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lem = lanemask_lt() | (1u << lane);
    for (int lb = 0; lb < k; lb += NT) {
        const int l = lb + tid;
        int s = 0, len = 0;
        if (l < k) {
            len = P.alen[a0 + l];
            s = P.abs[a0 + l];
            if (clip && len > 0) {
                int e = s + len;
                s = lower_bound_idx(bcol, s, e, lo);
                e = lower_bound_idx(bcol, s, e, chi);
                len = e - s;
            }
        }
        if (tid < 2 * NWD)
            starts[tid] = 0;
        long long tot;
        const long long ex = block_excl_scan<NT, long long>(
            ((long long)(len > 0) << 32) | (long long)len, ws, &tot);
        const int off = (int)(ex & 0xffffffffLL);
        const int n = (int)(tot & 0xffffffffLL);
        if (len > 0)
            lst[(int)(ex >> 32)] = s - off;
        __syncthreads();
        int seen = -1;  // lists that start before the window, less one
        for (long long win = 0; win < n; win += W) {
            unsigned *cur = starts + ((win / W) & 1 ? NWD : 0);
            unsigned *next = starts + ((win / W) & 1 ? 0 : NWD);
            if (len > 0 && off >= win && off < win + W)
                atomicOr(&cur[(off - (int)win) >> 5], 1u << (off & 31));
            __syncthreads();
            int before = 0, all = 0;
            for (int i = lane; i < NWD; i += 32) {
                const int c = __popc(cur[i]);
                all += c;
                before += i < w * kPlanPer ? c : 0;
            }
            int j = seen + __reduce_add_sync(kFull, before);
            seen += __reduce_add_sync(kFull, all);
            const long long e0 = win + w * (32 * kPlanPer);
            int c[kPlanPer];
#pragma unroll
            for (int u = 0; u < kPlanPer; u++) {
                const unsigned bits = cur[w * kPlanPer + u];
                const long long e = e0 + 32 * u + lane;
                c[u] = e < n ? bcol[lst[j + __popc(bits & lem)] + (int)e] : 0;
                j += __popc(bits);
            }
#pragma unroll
            for (int u = 0; u < kPlanPer; u++)
                if (e0 + 32 * u + lane < n)
                    f(c[u] - base);
            if (tid < NWD)
                next[tid] = 0;
            __syncthreads();
        }
    }
}

// Adds h products to a running count kept modulo cut (rem); true when a
// multiple of cut was crossed (a division a group took a third of the planning).
__device__ __forceinline__ bool plan_cross(unsigned &rem, unsigned h, unsigned cut)
{
    rem += h;
    if (rem < cut)
        return false;
    rem -= cut;
    if (rem >= cut)
        rem %= cut;
    return true;
}

// Walks the segment starts of planning group g (chunk-relative) in column
// order and calls f(column_in_group, product_prefix, distinct_prefix) for
// each.  `run` packs (products << 32 | distinct columns) before group g, ph is
// the product count of group g-1 and cross tells whether the running count
// crossed a multiple of `cut` in that group (plan_cross).  A dense group (more than
// dense = kSegCap - cut products) is always cut before and after; it is one
// segment when it holds at most kSegCap products, and inside a larger one a
// new segment starts at a column when the running product count would exceed
// `cut` (a single column above `cut` is a segment of its own).  Any other
// group starts a segment when the group before it crossed a multiple of
// `cut`, so a segment holds less than cut + dense = kSegCap products.
template <typename Fn>
__device__ __forceinline__ void plan_group_starts(int g, unsigned h, unsigned ph,
                                                  unsigned long long run,
                                                  const unsigned short *ccnt, unsigned cut,
                                                  unsigned dense, bool cross, Fn f)
{
    const unsigned pe = (unsigned)(run >> 32);
    const unsigned ue = (unsigned)(run & 0xffffffffu);
    if (h > dense && h <= (unsigned)kSegCap) {
        f(0, pe, ue);
        return;
    }
    if (h > dense) {
        f(0, pe, ue);
        unsigned acc = 0, pp = pe, uu = ue;
        for (int c = 0; c < kPlanGroupBits; c++) {
            const unsigned cc = ccnt[c];
            if (cc == 0)
                continue;
            if (acc > 0 && acc + cc > cut) {
                f(c, pp, uu);
                acc = 0;
            }
            acc += cc;
            pp += cc;
            uu++;  // a column with products is one distinct column
        }
        return;
    }
    if (g == 0 || ph > dense || cross)
        f(0, pe, ue);
}

// ---------------------------------------------------------------------------
// 1. planning
//
// Bound by issue (58 % of the slots at two CTAs an SM, which shared memory
// allows).  R-MAT n=2^18: 293 us with a contiguous share of the products a
// thread and its columns' runs gathered in registers, 226 with windows of
// products a lane apart, 16-byte accesses to the bitmap and no division a
// group; float32 R-MAT n=2^16 420 -> 358.  Four products a lane: 234 and 371;
// 40 registers (three CTAs, were there the shared memory): 246 and 328.
// ---------------------------------------------------------------------------
template <int UNUSED = 0>
__global__ void __launch_bounds__(kPlanThreads, 2) k_heavy_plan(CsrDev A, CsrDev B, PlanDev P)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    constexpr int NT = kPlanThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned *bm = (unsigned *)(smem + PlanLayout::o_bm);
    unsigned *hist = (unsigned *)(smem + PlanLayout::o_hist);
    unsigned short *gpop = (unsigned short *)(smem + PlanLayout::o_gpop);
    unsigned short *dix = (unsigned short *)(smem + PlanLayout::o_dix);
    // per-column product counts of groups above kSegCap products, two 16-bit
    // counters a word
    unsigned *ccnt2 = (unsigned *)(smem + PlanLayout::o_ccnt);
    const unsigned short *ccnt = (const unsigned short *)(smem + PlanLayout::o_ccnt);
    int *lst = (int *)(smem + PlanLayout::o_lst);
    unsigned *starts = (unsigned *)(smem + PlanLayout::o_starts);
    long long *ws = (long long *)(smem + PlanLayout::o_ws);
    int *misc = (int *)(smem + PlanLayout::o_misc);
    const int tid = threadIdx.x;
    const int M = A.M;
    // rows above kHugeFlop products sit at the end of the list; take them first
    const int nhuge = P.cnt->n_huge;
    const int nrows = P.cnt->bin_count[kBinHeavy] + nhuge;
    const int *rows = P.rows + (size_t)kBinHeavy * M;
    const int *__restrict__ bcol = B.col;
    const unsigned cut = (unsigned)P.seg_cut;                // <= kSegMaxCut
    const unsigned dense = (unsigned)(kSegCap - P.seg_cut);  // >= kSegCap / 4
    auto clear_groups = [&](int n) {
        for (int g = tid; g < n; g += NT) {
            hist[g] = 0;
            ((uint4 *)bm)[g] = make_uint4(0, 0, 0, 0);
        }
    };
    clear_groups(kPlanGroups);
    for (;;) {
        if (tid == 0)
            misc[0] = atomicAdd(&P.cnt->work_plan, 1);
        __syncthreads();
        const int item = misc[0];
        __syncthreads();
        if (item >= nrows)
            break;
        const int row = item < nhuge ? rows[M - 1 - item] : rows[item - nhuge];
        const int a0 = A.rpt[row];
        const int k = A.rpt[row + 1] - a0;
        const long long F = P.flop[row];
        const unsigned long long base = P.seg_base[row];
        const unsigned long long bound = seg_bound(F, B.N, P.seg_cut);
        const int2 cr = P.crange[row];  // written by the analysis
        const int mn = cr.x, mx = cr.y;
        if (mx < 0 || mn < 0 || mx >= B.N) {
            if (tid == 0) {
                if (mx >= 0)
                    atomicOr(&P.cnt->err, kErrBadInput);
                P.nnz[row] = 0;
                P.seg_n[row] = 0;
            }
            continue;
        }
        const bool multi = (long long)mx + 1 - mn > kPlanBits;
        long long u_run = 0;
        int nseg = 0;
        bool fail = false;
        for (long long clo = mn; clo <= mx; clo += kPlanBits) {
            const int lo = (int)clo;
            const int chi = (int)min((long long)mx + 1, clo + kPlanBits);
            const int span = chi - lo;
            const int ng = (span + kPlanGroupBits - 1) >> kPlanGroupLog2;
            // bm and hist are zero here: cleared at the start and after every chunk
            if (tid == 0) {
                misc[4] = INT_MAX;  // first group cut per column
                misc[5] = -1;       // last group cut per column
            }
            __syncthreads();
            // pass over the chunk's products: column bitmap and products per
            // group
            bool bad = false;
            plan_products<NT>(P, bcol, a0, k, multi, lo, chi, lo, lst, starts, ws, [&](int rc) {
                if ((unsigned)rc >= (unsigned)span) {
                    bad = true;
                    return;
                }
                const unsigned w = (unsigned)rc >> 5, b = 1u << (rc & 31);
                if (!(bm[w] & b))
                    atomicOr(&bm[w], b);
                atomicAdd(&hist[rc >> kPlanGroupLog2], 1u);
            });
            if (bad)
                atomicOr(&P.cnt->err, kErrBadInput);
            __syncthreads();
            // distinct columns per group, a group a thread (16 bytes apart: a
            // thread's own consecutive groups would meet in two banks)
            for (int g = tid; g < ng; g += NT) {
                const uint4 b = ((const uint4 *)bm)[g];
                gpop[g] = (unsigned short)(__popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w));
            }
            __syncthreads();
            const int gpt = (ng + NT - 1) / NT;
            const int g0 = min(tid * gpt, ng), g1 = min(g0 + gpt, ng);
            // groups above kSegCap products get per-column counts
            int nd_local = 0, dlo = INT_MAX, dhi = -1;
            unsigned long long sp = 0;
            for (int g = g0; g < g1; g++) {
                const unsigned h = hist[g];
                if (h > (unsigned)kSegCap) {
                    nd_local++;
                    dlo = min(dlo, g);
                    dhi = g;
                }
                sp += ((unsigned long long)h << 32) | (unsigned)gpop[g];
            }
            if (nd_local) {
                atomicMin(&misc[4], dlo);
                atomicMax(&misc[5], dhi);
            }
            long long ndt;
            int dx = (int)block_excl_scan<NT, long long>(nd_local, ws, &ndt);
            const int nd = (int)ndt;
            if (nd > kDenseGroups)
                fail = true;  // uniform
            if (!fail && nd > 0) {
                for (int g = g0; g < g1; g++)
                    if (hist[g] > (unsigned)kSegCap)
                        dix[g] = (unsigned short)dx++;
                for (int i = tid; i < nd * kPlanGroupBits / 2; i += NT)
                    ccnt2[i] = 0;
                __syncthreads();
                // only the columns from the first to the last such group
                const int dlo_c = lo + kPlanGroupBits * misc[4];
                const int dhi_c = (int)min((long long)chi,
                                           (long long)lo + (long long)kPlanGroupBits * (misc[5] + 1));
                plan_products<NT>(P, bcol, a0, k, true, dlo_c, dhi_c, lo, lst, starts, ws, [&](int rc) {
                    if ((unsigned)rc < (unsigned)span) {
                        const int g = rc >> kPlanGroupLog2;
                        if (hist[g] > (unsigned)kSegCap) {
                            const int slot = dix[g] * kPlanGroupBits + (rc & (kPlanGroupBits - 1));
                            atomicAdd(&ccnt2[slot >> 1], 1u << (16 * (slot & 1)));
                        }
                    }
                });
                bool big = false;
                for (int i = tid; i < nd * kPlanGroupBits; i += NT)
                    big |= ccnt[i] > kSegCap;
                fail = __syncthreads_or(big) != 0;
            }
            long long tot;
            const unsigned long long ex = (unsigned long long)block_excl_scan<NT, long long>(
                (long long)sp, ws, &tot);
            // count the chunk's segment starts
            int nstart = 0;
            if (!fail) {
                unsigned long long run = ex;
                unsigned ph = (g0 > 0 && g0 < ng) ? hist[g0 - 1] : 0u;
                unsigned rem = ((unsigned)(run >> 32) - ph) % cut;
                for (int g = g0; g < g1; g++) {
                    const unsigned h = hist[g];
                    plan_group_starts(g, h, ph, run,
                                      h > (unsigned)kSegCap ? ccnt + dix[g] * kPlanGroupBits : ccnt, cut,
                                      dense, plan_cross(rem, ph, cut),
                                      [&](int, unsigned, unsigned) { nstart++; });
                    run += ((unsigned long long)h << 32) | (unsigned)gpop[g];
                    ph = h;
                }
            }
            long long stot;
            const int sx = (int)block_excl_scan<NT, long long>(nstart, ws, &stot);
            if ((unsigned long long)(nseg + stot) > bound)
                fail = true;
            const long long u_chunk = u_run;
            u_run += (long long)((unsigned long long)tot & 0xffffffffull);
            if (fail) {
                __syncthreads();
                clear_groups(ng);
                __syncthreads();
                continue;  // keep counting distinct columns; the row takes the spill path
            }
            // write the chunk's segments: c_lo, u_off and the product prefix
            {
                unsigned long long run = ex;
                unsigned ph = (g0 > 0 && g0 < ng) ? hist[g0 - 1] : 0u;
                unsigned rem = ((unsigned)(run >> 32) - ph) % cut;
                int r = sx;
                for (int g = g0; g < g1; g++) {
                    const unsigned h = hist[g];
                    plan_group_starts(g, h, ph, run,
                                      h > (unsigned)kSegCap ? ccnt + dix[g] * kPlanGroupBits : ccnt, cut,
                                      dense, plan_cross(rem, ph, cut),
                                      [&](int c, unsigned pe, unsigned ue) {
                                          if (BRM_IN(P.cnt, base + nseg + r, P.cnt->seg_cap)) {
                                              SegDesc &d = P.seg[base + nseg + r];
                                              d.row = row;
                                              d.c_lo = lo + kPlanGroupBits * g + c;
                                              d.u_off = (int)(u_chunk + (long long)ue);
                                              d.bidx = nseg + r;
                                              d.nprod = (int)pe;  // prefix; a count below
                                          }
                                          r++;
                                      });
                    run += ((unsigned long long)h << 32) | (unsigned)gpop[g];
                    ph = h;
                }
            }
            __syncthreads();  // descriptors of this chunk visible to the block
            clear_groups(ng);
            // c_hi and product count of each segment: read every neighbour
            // first, then write (rounds of NT segments)
            const int ctot_prod = (int)((unsigned long long)tot >> 32);
            for (int i0 = 0; i0 < (int)stot; i0 += NT) {
                const int i = i0 + tid;
                int nc = 0, np = 0;
                if (i < (int)stot) {
                    const bool last = i + 1 == (int)stot;
                    nc = last ? chi : P.seg[base + nseg + i + 1].c_lo;
                    np = (last ? ctot_prod : P.seg[base + nseg + i + 1].nprod) -
                         P.seg[base + nseg + i].nprod;
                }
                __syncthreads();
                if (i < (int)stot) {
                    P.seg[base + nseg + i].c_hi = nc;
                    P.seg[base + nseg + i].nprod = np;
                }
                __syncthreads();
            }
            nseg += (int)stot;
        }
        if (tid == 0) {
            if (fail) {
                // a column denser than a segment holds, or too many cuts:
                // replay the merge for this row in global scratch (spill path)
                P.seg_n[row] = 0;
                P.spill[row] = 1;
                const int idx = atomicAdd(&P.cnt->spill_count, 1);
                P.spill_rows[idx] = row;
                P.spill_off[idx] = atomicAdd(&P.cnt->spill_bytes, spill_row_bytes(F, k));
                misc[1] = 0;
            } else {
                P.seg_n[row] = nseg;
                const unsigned long long tab =
                    atomicAdd(&P.cnt->table_cap, (unsigned long long)(nseg + 1) * (unsigned long long)k);
                misc[2] = (int)(tab & 0xffffffffull);
                misc[3] = (int)(tab >> 32);
                misc[1] = atomicAdd(&P.cnt->n_seg, nseg);
            }
            P.nnz[row] = (int)u_run;
        }
        __syncthreads();
        if (!fail) {
            const long long tab =
                (long long)(((unsigned long long)(unsigned)misc[3] << 32) | (unsigned)misc[2]);
            const int lpos = misc[1];
            for (int i = tid; i < nseg; i += NT) {
                if (BRM_IN(P.cnt, base + i, P.cnt->seg_cap) &&
                    BRM_IN(P.cnt, lpos + i, P.cnt->seg_cap)) {
                    P.seg[base + i].tab = tab;
                    P.seg_list[lpos + i] = (int)(base + i);
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// 2. split table: split[tab + b*k + l] = first position of list l at or after
//    boundary b (b = 0 .. nseg; boundary nseg is the end of the row).  One
//    block per segment computes its boundary's row of the table.
// ---------------------------------------------------------------------------
template <int UNUSED = 0>
__global__ void __launch_bounds__(256) k_split(CsrDev A, CsrDev B, PlanDev P)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    const int i0 = P.seg_range ? P.seg_range[0] : 0;
    const int nsegs = P.seg_range ? P.seg_range[1] : P.cnt->n_seg;
    const int *__restrict__ bcol = B.col;
    for (int it = i0 + blockIdx.x; it < nsegs; it += gridDim.x) {
        const int slot = P.seg_list[it];
        const int row = P.seg[slot].row;
        const int b = P.seg[slot].bidx;
        const int c_lo = P.seg[slot].c_lo;
        const long long tab = P.seg[slot].tab;
        const int nseg = P.seg_n[row];
        const int a0 = A.rpt[row];
        const int k = A.rpt[row + 1] - a0;
        int *t0 = P.split + tab + (long long)b * k;
        if (threadIdx.x == 0) {
            SegRun r;
            r.sp = tab + (long long)b * k;
            r.row = row;
            r.c_lo = c_lo;
            r.c_hi = P.seg[slot].c_hi;
            r.u_off = P.seg[slot].u_off;
            r.nprod = P.seg[slot].nprod;
            r.a0 = a0;
            r.k = k;
            r.next_u = (b + 1 < nseg) ? P.seg[slot + 1].u_off : P.nnz[row];
            P.run[it] = r;
        }
        for (int l = threadIdx.x; l < k; l += blockDim.x) {
            const int s = P.abs[a0 + l];
            const int e = s + P.alen[a0 + l];
            if (BRM_IN(P.cnt, tab + (long long)b * k + l, P.cnt->table_cap))
                t0[l] = (b == 0) ? s : lower_bound_idx(bcol, s, e, c_lo);
            if (b == nseg - 1 && BRM_IN(P.cnt, tab + (long long)(b + 1) * k + l, P.cnt->table_cap))
                t0[k + l] = e;
        }
    }
}

// ---------------------------------------------------------------------------
// 3. segment kernel
// ---------------------------------------------------------------------------
constexpr int kLongMax = kSegCap / kLongMin + 1;
constexpr int kSegPWords = kSegCap / 32;  // words of a bitmap over a segment's products
static_assert(kSegCap % 32 == 0 && kSegPWords <= 96, "p-bitmap prefix: three words per lane");

// Copies a segment record (48 bytes) into shared memory with cp.async.
__device__ __forceinline__ void copy_seg_run(SegRun *dst, const SegRun *src)
{
#pragma unroll
    for (int q = 0; q < 3; q++)
        cp_async16((unsigned char *)dst + 16 * q, (const unsigned char *)src + 16 * q);
}

// n columns of at most W products, W lanes each, warp w of the block's; entry(i)
// is a column (12 bits) and its products less `least`.  Leaf order by counting
// (products are numbered in list order), then the merge tree; the value to
// the column's first position.
template <typename T, int W, typename LeafOf, typename Entry>
__device__ __forceinline__ void seg_columns(int n, int w, T *vals, unsigned short *plist,
                                            const unsigned short *run, const LeafOf &leaf_of,
                                            const Entry &entry, int least)
{
    constexpr int PER = 32 / W;
    const int lane = threadIdx.x & 31, gl = lane & (W - 1), gb = lane & ~(W - 1);
    for (int ib = PER * w; ib < n; ib += PER * (kSegThreads / 32)) {
        const int i = ib + gb / W;
        int u = 0, p = 0, len = 0, x = 0, e = INT_MAX, r = 0;
        T v = T(0);
        if (i < n) {
            const int y = entry(i);
            u = y & 0xfff;
            len = least + (y >> 12);
            p = run[u];
            x = gl ? p + gl : u;
            if (gl < len) {
                e = plist[x];
                v = vals[x];
            }
        }
#pragma unroll
        for (int j = 0; j < W; j++)
            r += __shfl_sync(kFull, e, gb | j) < e;
        __syncwarp();
        if (gl < len) {
            const int y = r ? p + r : u;
            plist[y] = (unsigned short)e;
            vals[y] = v;
        }
        __syncwarp();
        int lf = 0;
        if (gl < len) {
            lf = leaf_of(plist[x]);
            v = vals[x];
        }
        v = group_trie<T, W>(lf, v, len);
        if (gl == 0 && len)
            vals[u] = v;
        __syncwarp();
    }
}

constexpr int kSegNP = kSegCap / kSegThreads;  // products a lane
static_assert(kSegCap % kSegThreads == 0 && kSegCap <= 4096, "12-bit columns, ranks and lists");

template <typename T>
struct SegLayout {
    static constexpr int NW = kSegThreads / 32;
    // bitmap words, with the summary words of a wide segment and their ranks
    // behind them; the values take their place
    static constexpr size_t o_cw = 0;
    static constexpr size_t o_val = 0;
    static constexpr size_t o_summ = o_cw + mid_a16(kSegCap * 4);
    static constexpr size_t o_srank = o_summ + mid_a16(kSumWords * 4);
    static constexpr size_t end_cw = o_srank + mid_a16(kSumWords * 2);
    static constexpr size_t end_val = mid_a16(kSegCap * sizeof(T));
    // list table: B offset less the product offset, then (dead) the order of a
    // long column's products and the warps' bitmaps over the lists
    static constexpr size_t o_lofs = end_cw > end_val ? end_cw : end_val;
    static constexpr size_t o_ord = o_lofs;
    static constexpr size_t o_bmp = o_ord + mid_a16(kSegCap * 2);
    static constexpr size_t o_lleaf = o_lofs + mid_a16(kSegCap * 4);
    static_assert(o_bmp + NW * kSegPWords * 6 <= o_lleaf, "the bitmaps fit in the list table");
    static constexpr size_t o_pre = o_lleaf + mid_a16(kSegCap * 2);   // word prefixes, then runs
    static constexpr size_t o_cnt = o_pre + mid_a16(kSegCap * 2);     // products of each column,
    static constexpr size_t o_list = o_cnt;                           // then products by position
    static constexpr size_t o_ucol = o_cnt + mid_a16(kSegCap * 2);
    // columns of two and of three or four products (from both ends), of five
    // to eight and of nine to sixteen (the same), of up to 32 and of more
    static constexpr int n_a = kSegCap / 2, n_b = kSegCap / 5 + 2, n_c = kSegCap / 17 + 2;
    static constexpr size_t o_lista = o_ucol + mid_a16(kSegCap * 4);
    static constexpr size_t o_listb = o_lista + mid_a16(n_a * 2);
    static constexpr size_t o_listc = o_listb + mid_a16(n_b * 2);
    static constexpr size_t o_llen = o_listc + mid_a16(n_c * 2);  // products of the long ones
    static constexpr size_t o_sb = o_llen + mid_a16(kLongMax * 2);
    static constexpr size_t o_sbp = o_sb + mid_a16(kSegPWords * 4);  // lists before each word of sb
    static constexpr size_t o_ws = o_sbp + mid_a16(kSegPWords * 2);
    static constexpr size_t o_misc = o_ws + mid_a16((NW + 1) * 8);
    static constexpr size_t o_run = o_misc + 64;  // the next segment's record
    static constexpr size_t bytes = o_run + sizeof(SegRun);
};

// Prefix of the bit counts of words[0, n) into pre, a thread's words
// consecutive (a multiple of four, so that threads 16 bytes apart in a phase
// of a load fall on different banks); returns the total.
template <int NT>
__device__ __forceinline__ int seg_word_prefix(const unsigned *words, int n, unsigned short *pre,
                                               int *ws)
{
    constexpr int MAXV = (kSegCap + 4 * NT - 1) / (4 * NT);  // 16-byte loads a thread
    const int vt = (n + 4 * NT - 1) / (4 * NT);
    int cnt[MAXV][4];
    int sum = 0;
#pragma unroll
    for (int q = 0; q < MAXV; q++) {
        const int i = 4 * (threadIdx.x * vt + q);
        uint4 x = make_uint4(0, 0, 0, 0);
        if (q < vt && i < n)
            x = *(const uint4 *)&words[i];
        cnt[q][0] = sum;
        cnt[q][1] = cnt[q][0] + __popc(x.x);
        cnt[q][2] = cnt[q][1] + __popc(x.y);
        cnt[q][3] = cnt[q][2] + __popc(x.z);
        sum = cnt[q][3] + __popc(x.w);
    }
    int tot;
    const int ex = block_excl_scan<NT, int>(sum, ws, &tot);
#pragma unroll
    for (int q = 0; q < MAXV; q++) {
        const int i = 4 * (threadIdx.x * vt + q);
        if (q < vt && i < n)
            *(ushort4 *)&pre[i] = make_ushort4(
                (unsigned short)(ex + cnt[q][0]), (unsigned short)(ex + cnt[q][1]),
                (unsigned short)(ex + cnt[q][2]), (unsigned short)(ex + cnt[q][3]));
    }
    return tot;
}

// Sequential trie of the elements [b, e) of a long column (leaves in
// increasing order, below 2^(D-1)); the elements are loaded GB at a time, so
// a long column does not wait for one load per element.
template <typename T, int D, int GB, typename GetLeaf, typename GetVal>
__device__ __forceinline__ T long_run(const GetLeaf &leaf, const GetVal &val, int b, int e)
{
    RegShiftReduce<T, D> sr;
    sr.init(leaf(b), val(b));
    for (int j0 = b + 1; j0 < e; j0 += GB) {
        int lf[GB];
        T lv[GB];
#pragma unroll
        for (int q = 0; q < GB; q++) {
            if (j0 + q < e) {
                lf[q] = leaf(j0 + q);
                lv[q] = val(j0 + q);
            }
        }
#pragma unroll
        for (int q = 0; q < GB; q++)
            if (j0 + q < e)
                sr.push(lf[q], lv[q]);
    }
    return sr.finish();
}

// A long column (len products in leaf order) reduced by a whole warp.  Its
// leaves (increasing, below 2^bits) are cut into the 32 aligned ranges of 2^s
// leaves, s = bits - 5: every range is one subtree of the merge tree at level
// s, so lane j reduces the products of range j on its own (at most s split
// levels: 12 stack entries suffice for 16-bit leaves), and the subtree values
// are then joined by the trie over their range indices (warp_trie); every
// lane returns the value.  cnt and sv are the warp's 32-entry shared scratch.
template <typename T, typename GetLeaf, typename GetVal>
__device__ __forceinline__ T warp_long_column(const GetLeaf &leaf, const GetVal &val, int len,
                                              int *cnt, T *sv)
{
    const int lane = threadIdx.x & 31;
    const int bits = 32 - __clz(leaf(len - 1) | 1);
    const int s = bits > 5 ? bits - 5 : 0;
    __syncwarp();
    cnt[lane] = 0;
    __syncwarp();
    for (int p = lane; p < len; p += 32)
        atomicAdd(&cnt[leaf(p) >> s], 1);
    __syncwarp();
    const int mc = cnt[lane];
    const int lo = warp_incl_scan(mc) - mc;
    T v = T(0);
    if (mc > 0)
        v = long_run<T, 12, 4>(leaf, val, lo, lo + mc);
    // the nonempty ranges in order, one per lane
    const unsigned hm = __ballot_sync(kFull, mc > 0);
    const int r = __popc(hm & ((1u << lane) - 1u));
    __syncwarp();
    if (mc > 0) {
        sv[r] = v;
        cnt[r] = lane;
    }
    __syncwarp();
    const int nh = __popc(hm);
    const int li = lane < nh ? cnt[lane] : 0;
    const T vi = lane < nh ? sv[lane] : T(0);
    __syncwarp();
    return __shfl_sync(kFull, warp_trie<T>(li, vi, nh), 0);  // the trie's value is in lane 0
}

// What the kernel works on and where it writes: heavy-row segments into C
// (kSegPrecise) or C_bar (kSegUpper); or whole rows of at most kSegCap products
// and 65 to 255 lists (rank class 8), counted (kSegRowSymbolic) or written
// at crpt, at the row's offset in C_bar or in the one-call scratch.
enum SegMode : int {
    kSegPrecise = 0,
    kSegUpper = 1,
    kSegRowSymbolic = 2,
    kSegRowPrecise = 3,
    kSegRowUpper = 4,
    kSegRowScratch = 5,
};

template <typename T, int MODE>
__global__ void __launch_bounds__(kSegThreads, 3 * 256 / kSegThreads)
    k_seg_numeric(CsrDev A, CsrDev B, PlanDev P, const int *crpt, int *ccol, T *cval)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    constexpr int NT = kSegThreads, NP = kSegNP;
    constexpr bool ROWS = MODE >= kSegRowSymbolic;
    using L = SegLayout<T>;
    constexpr int NW = L::NW;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned *cw = (unsigned *)(smem + L::o_cw);
    T *vals = (T *)(smem + L::o_val);
    unsigned *summ = (unsigned *)(smem + L::o_summ);
    unsigned short *srank = (unsigned short *)(smem + L::o_srank);
    int *lofs = (int *)(smem + L::o_lofs);
    unsigned short *ord = (unsigned short *)(smem + L::o_ord);
    unsigned short *lleaf = (unsigned short *)(smem + L::o_lleaf);
    unsigned short *pre = (unsigned short *)(smem + L::o_pre);
    unsigned short *run = pre;
    unsigned *cnt2 = (unsigned *)(smem + L::o_cnt);  // two 16-bit counts a word
    const unsigned short *cnt = (const unsigned short *)(smem + L::o_cnt);
    unsigned short *plist = (unsigned short *)(smem + L::o_list);
    int *ucol = (int *)(smem + L::o_ucol);
    unsigned short *lista = (unsigned short *)(smem + L::o_lista);
    unsigned short *listb = (unsigned short *)(smem + L::o_listb);
    unsigned short *listc = (unsigned short *)(smem + L::o_listc);
    unsigned short *llen = (unsigned short *)(smem + L::o_llen);
    unsigned *sb = (unsigned *)(smem + L::o_sb);
    unsigned short *sbp = (unsigned short *)(smem + L::o_sbp);
    long long *ws = (long long *)(smem + L::o_ws);
    int *wsi = (int *)(smem + L::o_ws);
    int *misc = (int *)(smem + L::o_misc);
    SegRun *srun = (SegRun *)(smem + L::o_run);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned ltm = lanemask_lt(), lem = ltm | (1u << lane);
    const int i0 = !ROWS && P.seg_range ? P.seg_range[0] : 0;
    const int nsegs = ROWS            ? P.cnt->bin_count[kBinSegRow]
                      : P.seg_range ? P.seg_range[1]
                                    : P.cnt->n_seg;
    const int *rows = P.rows + (size_t)kBinSegRow * A.M;
    int *work = ROWS ? &P.cnt->work_mw[kMwRankCounter + kBinSegRow - kBinRank0] : &P.cnt->work_seg;
    const int *__restrict__ bcol = B.col;
    const T *__restrict__ bval = (const T *)B.val;
    const T *__restrict__ aval = (const T *)A.val;
    // leaf of product e (numbered in list order)
    auto leaf_of = [&](int e) -> int {
        return lleaf[sbp[e >> 5] + __popc(sb[e >> 5] & ((2u << (e & 31)) - 1u)) - 1];
    };
    // thread 0 takes the next work item one segment ahead and copies its
    // record into srun (cp.async) while the current segment runs, so a
    // segment starts without a chain of dependent global loads
    int pf = 0;
    bool pf_copied = false;
    if (tid == 0)
        pf = i0 + atomicAdd(work, 1);
    for (;;) {
        if (tid == 0) {
            if (!ROWS) {
                if (!pf_copied && pf < nsegs)
                    copy_seg_run(srun, P.run + pf);
                cp_async_wait_all();
            }
            misc[0] = pf;
        }
        if (tid < kSegPWords)
            sb[tid] = 0;
        if (tid < 8)
            misc[1 + tid] = 0;  // columns of each size, positions, an input error
        __syncthreads();
        const int item = misc[0];
        if (item >= nsegs)
            break;
        SegRun d;
        if (ROWS) {
            d.row = rows[item];
            const int2 cr = P.crange[d.row];
            d.c_lo = cr.x;
            d.c_hi = cr.y + 1;
            d.u_off = 0;
            d.nprod = P.flop[d.row];
            d.a0 = A.rpt[d.row];
            d.k = A.rpt[d.row + 1] - d.a0;
        } else {
            d = *srun;
        }
        if (tid == 0) {
            pf = i0 + atomicAdd(work, 1);  // consumed after the columns are read
            pf_copied = false;
        }
        if (ROWS && (d.row < P.r_lo || d.row >= P.r_hi)) {
            __syncthreads();
            continue;
        }
        const int row = d.row;
        const int a0 = d.a0;
        const int k = d.k;
        const int span = d.c_hi - d.c_lo;
        const int nsum = (span + 1023) >> 10;
        // where each list starts, and ends (rows: how long it is)
        const int *sp0 = ROWS ? P.abs + a0 : P.split + d.sp;
        const int *sp1 = ROWS ? P.alen + a0 : sp0 + k;
        // a segment spanning at most 32 * kSegCap columns ranks its columns
        // with one flat bitmap; wider ones with a summary bit per nonempty
        // word and compressed words
        const int nwf = (span + 31) >> 5;
        const bool flat = nwf <= kSegCap;
        {
            uint4 *z = (uint4 *)(flat ? cw : summ);
            const int nz = ((flat ? nwf : min(nsum, kSumWords)) + 3) >> 2;
            for (int i = tid; i < nz; i += NT)
                z[i] = make_uint4(0, 0, 0, 0);
            for (int i = tid; i < kSegCap / 8; i += NT)
                ((uint4 *)cnt2)[i] = make_uint4(0, 0, 0, 0);
        }
        // 1. nonempty sub-lists of the segment, in leaf order (a thread takes
        //    four consecutive lists per pass), and a bit per list start in
        //    product order: by the first warp where the row has few lists, by
        //    the block for hub rows (thousands of lists, few products of each
        //    in one segment)
        constexpr int LPT = 4;
        int nlists = 0, nprod = 0;
        const bool few = k <= 32 * LPT;
        for (int lb = 0; lb < k && (!few || w == 0); lb += NT * LPT) {
            int st[LPT], len[LPT];
            int ne = 0, psum = 0;
#pragma unroll
            for (int q = 0; q < LPT; q++) {
                const int l = lb + tid * LPT + q;
                st[q] = 0;
                len[q] = 0;
                if (l < k) {
                    st[q] = sp0[l];
                    len[q] = ROWS ? sp1[l] : sp1[l] - st[q];
                }
                ne += len[q] > 0;
                psum += len[q];
            }
            const long long x = ((long long)ne << 32) | (long long)psum;
            long long tot, ex;
            if (few) {
                ex = warp_incl_scan(x);
                tot = __shfl_sync(kFull, ex, 31);
                ex -= x;
            } else {
                ex = block_excl_scan<NT, long long>(x, ws, &tot);
            }
            int li = nlists + (int)(ex >> 32);
            int po = nprod + (int)(ex & 0xffffffffLL);
#pragma unroll
            for (int q = 0; q < LPT; q++) {
                if (len[q] > 0) {
                    if (li < kSegCap && po < kSegCap) {
                        lofs[li] = st[q] - po;
                        lleaf[li] = (unsigned short)(lb + tid * LPT + q);
                        atomicOr(&sb[po >> 5], 1u << (po & 31));
                    }
                    li++;
                    po += len[q];
                }
            }
            nlists += (int)(tot >> 32);
            nprod += (int)(tot & 0xffffffffLL);
        }
        if (few && tid == 0) {
            misc[9] = nlists;
            misc[10] = nprod;
        }
        __syncthreads();
        if (few) {
            nlists = misc[9];
            nprod = misc[10];
        }
        if (nprod > kSegCap || nprod != d.nprod || nsum > kSumWords || span <= 0 || nprod == 0) {
            // (the columns before a chunk's first cut may hold no product)
            if (tid == 0 && (ROWS || nprod != 0 || d.nprod != 0 || d.next_u != d.u_off))
                atomicOr(&P.cnt->err, kErrWindowOverflow);
            __syncthreads();
            continue;
        }
        // 2. this warp's words of 32 products, [w0, w0 + nw): columns into
        //    registers, their bits into the bitmap or the summary.  Lanes
        //    beyond the last product take no part from the counting on
        const int nwd = (nprod + 31) >> 5;
        const int npw = (nwd + NW - 1) / NW;
        const int w0 = w * npw;
        const int nw = min(npw, nwd - w0);
        int jb = -1;  // lists that start before the word, less one
        {
            int x = 0;
            for (int i = lane; i < w0 && i < nwd; i += 32)
                x += __popc(sb[i]);
            jb += __reduce_add_sync(kFull, x);
        }
        int c[NP];        // column, from c_lo; then the product's turn in its column
        unsigned pk[NP];  // list << 17 | word slot << 5 | column in the word; then list << 12 | u
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int e = min((w0 + u) * 32 + lane, nprod - 1);
                const unsigned bits = sb[w0 + u];
                const int j = jb + __popc(bits & lem);
                if (lane == 0)
                    sbp[w0 + u] = (unsigned short)(jb + 1);
                jb += __popc(bits);
                pk[u] = (unsigned)j << 17;
                const int bi = lofs[j] + e;
                c[u] = BRM_IN(P.cnt, bi, B.nnz) ? bcol[bi] : d.c_lo;
            }
        }
        bool bad = false;
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                c[u] -= d.c_lo;
                if ((unsigned)c[u] >= (unsigned)span) {
                    bad = true;  // a column outside the segment: unsorted rows of B
                    c[u] = 0;
                }
                const int x = flat ? c[u] : c[u] >> 5;
                unsigned *q = (flat ? cw : summ) + (x >> 5);
                const unsigned b = 1u << (x & 31);
                if (flat)
                    pk[u] |= (unsigned)c[u];
                if (!(*q & b))
                    atomicOr(q, b);
            }
        }
        if (bad)
            misc[8] = 1;
        __syncthreads();
        // every thread has read this segment's record: copy the next one
        if (!ROWS && tid == 0 && pf < nsegs) {
            copy_seg_run(srun, P.run + pf);
            pf_copied = true;
        }
        if (misc[8]) {  // the plan does not match the input
            if (tid == 0)
                atomicOr(&P.cnt->err, kErrBadInput);
            __syncthreads();
            continue;
        }
        int ncw = nwf;
        if (!flat) {
            // slots of the nonempty words
            ncw = seg_word_prefix<NT>(summ, nsum, srank, wsi);
            for (int i = tid; i < (ncw + 3) >> 2; i += NT)
                ((uint4 *)cw)[i] = make_uint4(0, 0, 0, 0);
            __syncthreads();
#pragma unroll
            for (int u = 0; u < NP; u++) {
                if (u < nw) {
                    const int sw = c[u] >> 10;
                    const unsigned b = 1u << (c[u] & 31);
                    const int ci = srank[sw] + __popc(summ[sw] & ((1u << ((c[u] >> 5) & 31)) - 1u));
                    pk[u] |= ((unsigned)ci << 5) | (unsigned)(c[u] & 31);
                    if (BRM_IN(P.cnt, ci, kSegCap) && !(cw[ci] & b))
                        atomicOr(&cw[ci], b);
                }
            }
            __syncthreads();
        }
        // 3. distinct columns, and those before each word
        const int U = seg_word_prefix<NT>(cw, ncw, pre, wsi);
        const bool nodup = U == nprod;
        if (MODE == kSegRowSymbolic) {
            if (tid == 0)
                P.nnz[row] = U;
            __syncthreads();
            continue;
        }
        // must produce exactly the row's columns, or its share of them
        const long long rbase = MODE == kSegPrecise || MODE == kSegRowPrecise ? (long long)crpt[row]
                                : MODE == kSegRowScratch ? P.mw_pre[row]
                                                         : P.scan_flop[row];
        if ((!ROWS && U != d.next_u - d.u_off) ||
            (MODE == kSegRowPrecise && U != crpt[row + 1] - (int)rbase)) {
            if (tid == 0)
                atomicOr(&P.cnt->err, kErrNnzMismatch);
            __syncthreads();
            continue;
        }
        if ((MODE == kSegRowUpper || MODE == kSegRowScratch) && tid == 0)
            P.nnz[row] = U;
        const long long obase = rbase + d.u_off;
        __syncthreads();
        // 4. column rank of each product and its turn among the column's (in
        //    arbitrary order)
#pragma unroll
        for (int u = 0; u < NP; u++) {
            if (u < nw) {
                const int ci = (int)((pk[u] >> 5) & 0xfffu);
                const int r = pre[ci] + __popc(cw[ci] & ((1u << (pk[u] & 31u)) - 1u));
                pk[u] = ((pk[u] >> 17) << 12) | (unsigned)r;
                if (!BRM_IN(P.cnt, r, kSegCap))
                    continue;
                ucol[r] = c[u];
                c[u] = 0;
                if (!nodup && (w0 + u) * 32 + lane < nprod) {
                    const int sh = 16 * (r & 1);
                    c[u] = (int)((atomicAdd(&cnt2[r >> 1], 1u << sh) >> sh) & 0xffffu);
                }
            }
        }
        __syncthreads();
        // 5. columns of several products: positions for the second and further
        //    ones (column u's i-th at run[u] + i, its first at u), lists by size
        if (!nodup) {
            for (int u = tid; u < U; u += NT) {
                const int n = cnt[u];
                if (n == 1)
                    continue;
                run[u] = (unsigned short)(U - 1 + atomicAdd(&misc[7], n - 1));
                const int cls = n == 2 ? 0 : n <= 4 ? 1 : n <= 8 ? 2 : n <= 16 ? 3 : n < kLongMin ? 4 : 5;
                const int o = atomicAdd(&misc[1 + cls], 1);
                // (the size beside the column's 12 bits)
                if (!BRM_IN(P.cnt, o, cls <= 1 ? L::n_a : cls <= 3 ? L::n_b : L::n_c)) {
                    continue;
                } else if (cls == 0) {
                    lista[o] = (unsigned short)u;
                } else if (cls == 1) {
                    lista[L::n_a - 1 - o] = (unsigned short)(u | ((n - 3) << 12));
                } else if (cls == 2) {
                    listb[o] = (unsigned short)(u | ((n - 5) << 12));
                } else if (cls == 3) {
                    listb[L::n_b - 1 - o] = (unsigned short)(u | ((n - 9) << 12));
                } else if (cls == 4) {
                    listc[o] = (unsigned short)(u | ((n - 17) << 12));
                } else if (o < kLongMax) {
                    listc[L::n_c - 1 - o] = (unsigned short)u;
                    llen[o] = (unsigned short)n;
                }
            }
            __syncthreads();
        }
        const int n2 = misc[1], n34 = misc[2], n8 = misc[3], n16 = misc[4], n32 = misc[5];
        const int nlong = min(misc[6], kLongMax);
        // 6. values to their positions
        {
            constexpr int VB = 4;  // gathers in flight a lane
            static_assert(NP % VB == 0, "whole batches");
#pragma unroll
            for (int ub = 0; ub < NP; ub += VB) {
                if (ub < nw) {
                    T bv[VB], av[VB];
                    int lf[VB];
#pragma unroll
                    for (int q = 0; q < VB; q++) {
                        const int u = ub + q;
                        if (u < nw) {
                            const int j = (int)(pk[u] >> 12);
                            const int bi = lofs[j] + min((w0 + u) * 32 + lane, nprod - 1);
                            lf[q] = lleaf[j];
                            bv[q] = BRM_IN(P.cnt, bi, B.nnz) ? bval[bi] : T(0);
                            av[q] = aval[a0 + lf[q]];
                        }
                    }
#pragma unroll
                    for (int q = 0; q < VB; q++) {
                        const int u = ub + q;
                        if (u < nw && (w0 + u) * 32 + lane < nprod) {
                            int p = (int)(pk[u] & 0xfffu);
                            if (c[u])
                                p = run[p] + c[u];
                            if (!BRM_IN(P.cnt, p, kSegCap))
                                continue;
                            vals[p] = vmul(av[q], bv[q]);
                            plist[p] = (unsigned short)((w0 + u) * 32 + lane);
                        }
                    }
                }
            }
        }
        __syncthreads();
        // 7. columns of several products, each size by its own loop so that
        //    the lanes of a warp run the same code (and starting at another
        //    warp: most sizes fill a few); the value to position u.
        //    Columns with more than 32 products first: one warp each puts them
        //    in leaf order with a bitmap over the products and hands them to
        //    the column reducer through the long-column scratch; of whole rows
        //    (at most 255 lists), and when the scratch is full, its first lane
        //    reduces them
        if (nlong > 0) {
            unsigned *bmp = (unsigned *)(smem + L::o_bmp) + w * kSegPWords;
            unsigned short *wpre =
                (unsigned short *)((unsigned *)(smem + L::o_bmp) + NW * kSegPWords) + w * kSegPWords;
            T *lval = (T *)P.long_val;
            for (int lb = w; lb < nlong; lb += 32 * NW) {
                // the warp's next (up to) 32 columns lb + j * NW: one
                // reservation of long-column scratch covers all of them
                const int lj = lb + lane * NW;
                int lu = 0, ln = 0;
                if (lj < nlong) {
                    lu = listc[L::n_c - 1 - lj];
                    ln = llen[lj];
                }
                const int ncol = __popc(__ballot_sync(kFull, lj < nlong));
                const int lincl = warp_incl_scan(ln);
                unsigned long long rcol = 0, relem = 0;
                if (!ROWS && lane == 31) {
                    rcol = atomicAdd(&P.cnt->long_cols, (unsigned long long)ncol);
                    relem = atomicAdd(&P.cnt->long_elems, (unsigned long long)lincl);
                }
                rcol = __shfl_sync(kFull, rcol, 31);
                relem = __shfl_sync(kFull, relem, 31);
                for (int jc = 0; jc < ncol; jc++) {
                    const int u = __shfl_sync(kFull, lu, jc);
                    const int len = __shfl_sync(kFull, ln, jc);
                    const int rp = run[u];
                    const long long lci = (long long)rcol + jc;
                    const long long leo =
                        (long long)relem + __shfl_sync(kFull, lincl - ln, jc);
                    const bool handoff =
                        !ROWS && lci < P.long_cap_cols && leo + len <= P.long_cap_elems;
                    for (int x = lane; x < nwd; x += 32)
                        bmp[x] = 0;
                    __syncwarp();
                    for (int i = lane; i < len; i += 32) {
                        const int l = plist[i ? rp + i : u];
                        atomicOr(&bmp[l >> 5], 1u << (l & 31));
                    }
                    __syncwarp();
                    {
                        const int x0 = lane * 3;
                        const int c0 = x0 < nwd ? __popc(bmp[x0]) : 0;
                        const int c1 = x0 + 1 < nwd ? __popc(bmp[x0 + 1]) : 0;
                        const int c2 = x0 + 2 < nwd ? __popc(bmp[x0 + 2]) : 0;
                        const int ex = warp_incl_scan(c0 + c1 + c2) - (c0 + c1 + c2);
                        if (x0 < nwd)
                            wpre[x0] = (unsigned short)ex;
                        if (x0 + 1 < nwd)
                            wpre[x0 + 1] = (unsigned short)(ex + c0);
                        if (x0 + 2 < nwd)
                            wpre[x0 + 2] = (unsigned short)(ex + c0 + c1);
                    }
                    __syncwarp();
                    for (int i = lane; i < len; i += 32) {
                        const int x = i ? rp + i : u;
                        const int l = plist[x];
                        const int r = wpre[l >> 5] + __popc(bmp[l >> 5] & ((1u << (l & 31)) - 1u));
                        if (!BRM_IN(P.cnt, r, len)) {
                            continue;
                        } else if (handoff) {
                            P.long_leaf[leo + r] = (unsigned short)leaf_of(l);
                            lval[leo + r] = vals[x];
                        } else {
                            ord[r ? rp + r : u] = (unsigned short)x;
                        }
                    }
                    if (!ROWS && lci < P.long_cap_cols && lane == 0) {
                        LongCol lc;
                        lc.out = obase + u;
                        lc.off = leo;
                        lc.col = d.c_lo + ucol[u];
                        lc.len = handoff ? len : -1;
                        P.long_col[lci] = lc;
                    }
                    __syncwarp();
                    if (handoff)
                        continue;
                    if (lane == 0) {  // (a stack in local memory: registers are short)
                        ShiftReduce<T, 17> sr;
                        sr.init(leaf_of(plist[ord[u]]), vals[ord[u]]);
                        for (int i = 1; i < len; i++)
                            sr.push(leaf_of(plist[ord[rp + i]]), vals[ord[rp + i]]);
                        vals[u] = sr.finish();
                    }
                    __syncwarp();
                }
            }
        }
        if (!nodup) {
            seg_columns<T, 32>(n32, w, vals, plist, run, leaf_of,
                               [&](int i) { return listc[i]; }, 17);
            seg_columns<T, 16>(n16, (w + 5) % NW, vals, plist, run, leaf_of,
                               [&](int i) { return listb[L::n_b - 1 - i]; }, 9);
            seg_columns<T, 8>(n8, (w + 3) % NW, vals, plist, run, leaf_of,
                              [&](int i) { return listb[i]; }, 5);
            for (int i = tid; i < n2; i += NT) {
                const int u = lista[i];
                vals[u] = vadd(vals[u], vals[run[u] + 1]);
            }
            for (int i = (NW - 1 - w) * 32 + lane; i < n34; i += NT) {
                const int x = lista[L::n_a - 1 - i], u = x & 0xfff, p = run[u];
                // sort the (product, value) pairs in registers, then the closed form
                int l0 = plist[u], l1 = plist[p + 1], l2 = plist[p + 2];
                T v0 = vals[u], v1 = vals[p + 1], v2 = vals[p + 2];
                if (!(x >> 12)) {
                    leaf_cas(l0, v0, l1, v1);
                    leaf_cas(l1, v1, l2, v2);
                    leaf_cas(l0, v0, l1, v1);
                    vals[u] = trie3<T>(leaf_of(l0), leaf_of(l1), leaf_of(l2), v0, v1, v2);
                } else {
                    int l3 = plist[p + 3];
                    T v3 = vals[p + 3];
                    leaf_cas(l0, v0, l1, v1);
                    leaf_cas(l2, v2, l3, v3);
                    leaf_cas(l0, v0, l2, v2);
                    leaf_cas(l1, v1, l3, v3);
                    leaf_cas(l1, v1, l2, v2);
                    vals[u] = trie4<T>(leaf_of(l0), leaf_of(l1), leaf_of(l2), leaf_of(l3), v0, v1,
                                       v2, v3);
                }
            }
        }
        __syncthreads();
        // 8. the segment's columns (the column reducer overwrites those handed
        //    to it)
        for (int u = tid; u < U; u += NT) {
            if (BRM_IN(P.cnt, obase + u, MODE == kSegRowScratch ? P.mid_cap : P.c_cap)) {
                ccol[obase + u] = d.c_lo + ucol[u];
                cval[obase + u] = vals[u];
            }
        }
        __syncthreads();
    }
    // whole rows: the last block clears the counter for the next launch
    if (ROWS && tid == 0) {
        int *done = &P.cnt->done_mw[kMwRankCounter + kBinSegRow - kBinRank0];
        __threadfence();
        if (atomicAdd(done, 1) == (int)gridDim.x - 1) {
            atomicExch(work, 0);
            atomicExch(done, 0);
        }
    }
}

template <typename T, int MODE>
inline void launch_seg_kernel(const CsrDev &A, const CsrDev &B, const PlanDev &P, const int *crpt,
                              int *ccol, T *cval, int num_sms, cudaStream_t s)
{
    const size_t ssm = SegLayout<T>::bytes;
    cudaFuncSetAttribute(k_seg_numeric<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)ssm);
    // as many CTAs as fit on every SM (shared memory and registers)
    k_seg_numeric<T, MODE><<<num_sms * (3 * 256 / kSegThreads), kSegThreads, ssm, s>>>(
        A, B, P, crpt, ccol, cval);
    count_launch();
}

// ---------------------------------------------------------------------------
// 4. column reducer: one warp per long column handed over by the segment
//    kernel; its products are in leaf order.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_long_warp(PlanDev P, int *ccol, T *cval)
{
    if (P.cnt->abort)  // a capacity check of a captured pipeline failed
        return;
    __shared__ int s_cnt[4][32];
    __shared__ T s_val[4][32];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long n = min((long long)P.cnt->long_cols, P.long_cap_cols);
    const T *__restrict__ lval = (const T *)P.long_val;
    const unsigned short *__restrict__ lleaf = P.long_leaf;
    for (long long i = (long long)blockIdx.x * 4 + wid; i < n; i += (long long)gridDim.x * 4) {
        const LongCol c = P.long_col[i];
        // (reduced by the segment kernel; checked build: a record outside the
        // scratch or C is skipped)
        if (c.len <= 0 || !BRM_IN(P.cnt, c.off + c.len - 1, P.long_cap_elems) ||
            !BRM_IN(P.cnt, c.out, P.c_cap))
            continue;
        const unsigned short *lf = lleaf + c.off;
        const T *lv = lval + c.off;
        const T r = warp_long_column<T>([&](int j) { return (int)lf[j]; },
                                        [&](int j) { return lv[j]; }, c.len, s_cnt[wid],
                                        s_val[wid]);
        if (lane == 0) {
            ccol[c.out] = c.col;
            cval[c.out] = r;
        }
    }
}

// ---------------------------------------------------------------------------
// 5. segments grouped by row parts: for a numeric phase run part by part
//    (rows [pb[p], pb[p+1]) for p < nparts), the segment list is reordered so
//    every part's segments are contiguous, and ranges[2p], ranges[2p+1] give
//    the part's slice.  cnt (nparts ints) must be zero before the count pass.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int part_of_row(const int *pb, int nparts, int row)
{
    int p = 0;
    while (p + 1 < nparts && row >= pb[p + 1])
        p++;
    return p;
}

template <int UNUSED = 0>
__global__ void __launch_bounds__(256) k_seg_part_count(PlanDev P, const int *pb, int nparts,
                                                        int *cnt)
{
    const int n = P.cnt->n_seg;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&cnt[part_of_row(pb, nparts, P.seg[P.seg_list[i]].row)], 1);
}

template <int UNUSED = 0>
__global__ void __launch_bounds__(256) k_seg_part_scatter(PlanDev P, const int *pb, int nparts,
                                                          const int *cnt, int *fill, int *out,
                                                          int *ranges)
{
    __shared__ int base[kMaxParts + 1];
    if (threadIdx.x == 0) {
        int s = 0;
        for (int p = 0; p < nparts; p++) {
            base[p] = s;
            s += cnt[p];
        }
        base[nparts] = s;
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x < nparts) {
        ranges[2 * threadIdx.x] = base[threadIdx.x];
        ranges[2 * threadIdx.x + 1] = base[threadIdx.x + 1];
    }
    const int n = P.cnt->n_seg;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int slot = P.seg_list[i];
        const int p = part_of_row(pb, nparts, P.seg[slot].row);
        out[base[p] + atomicAdd(&fill[p], 1)] = slot;
    }
}

}  // namespace brm
