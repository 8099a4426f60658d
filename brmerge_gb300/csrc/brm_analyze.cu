// brm_analyze.cu -- row analysis, device scans, Upper compaction, validation.
#include <algorithm>
#include <climits>

#include "brm_check.cuh"
#include "brm_common.cuh"
#include "brm_kernels.h"

namespace brm {

// ---------------------------------------------------------------------------
// Row analysis.  Replaces compute_flop (spgemm.h:31-56) and the flop-balanced
// static row ranges (spgemm.h:496-503): on the GPU the balance comes from
// binning rows by their product count and handing heavy rows out first.
// A group of lanes per row; each block appends its rows to the bin lists with one
// global atomic per bin.
// ---------------------------------------------------------------------------
constexpr int kAnaThreads = 256;
constexpr int kAnaRowsPerGroup = 2;

// Reductions over a group of TW lanes (TW a power of two <= 32, the group
// aligned in the warp); `gm` is the group's lane mask.
template <int TW, typename T>
__device__ __forceinline__ T grp_sum(T v, unsigned gm)
{
#pragma unroll
    for (int o = TW / 2; o > 0; o >>= 1)
        v += __shfl_xor_sync(gm, v, o);
    return v;
}
template <int TW, typename T>
__device__ __forceinline__ T grp_max(T v, unsigned gm)
{
#pragma unroll
    for (int o = TW / 2; o > 0; o >>= 1) {
        const T n = __shfl_xor_sync(gm, v, o);
        v = n > v ? n : v;
    }
    return v;
}
template <int TW, typename T>
__device__ __forceinline__ T grp_min(T v, unsigned gm)
{
#pragma unroll
    for (int o = TW / 2; o > 0; o >>= 1) {
        const T n = __shfl_xor_sync(gm, v, o);
        v = n < v ? n : v;
    }
    return v;
}

// Rows of more than kAnaLongK entries are left, by groups of fewer than 32
// lanes, to the block's whole warps (a second pass in the same launch).
constexpr int kAnaLongK = 96;

// What a block gathers of its rows before it takes places in the global lists.
template <int RPB>
struct AnaBlock {
    int cnt[kNumBins];
    int base[kNumBins];
    int bin[RPB];
    int idx[RPB];
    int flop[RPB];
    int longs[RPB];
    int nlong;
    int max_k;
    unsigned long long mid;
    unsigned long long tot[RPB / 32 + 1][2];  // products and scratch entries of 32 rows, then
                                              // where they start among all rows'
};

// One row by a group of TW lanes (lane gl of it, mask gm): its products, list
// table entries (P.abs, P.alen), class and column range: the first and the
// last column of every list, taken in the same pass (fetched afterwards, by way
// of P.abs and P.alen, they added a round trip to memory: the symbolic phase of
// 3.75 M rows of two lists 1.35 -> 1.17 ms without it and with the block's device
// atomics in one phase; one call on 4096 uneven pairs 32.5 -> 31.4 ms)
template <int TW, int RPB>
__device__ __forceinline__ void analyze_row(const CsrDev &A, const CsrDev &B, const PlanDev &P,
                                            int row, int slot, int gl, unsigned gm,
                                            AnaBlock<RPB> &S)
{
    const int M = A.M, K = B.M;
    int a0 = A.rpt[row];
    int a1 = A.rpt[row + 1];
    long long f = 0;
    int nl = 0, leaf = -1;
    bool bad = false;
    if (a0 < 0 || a1 < a0 || a1 > A.nnz) {  // malformed row pointers: treat the row as empty
        bad = true;
        a0 = a1 = 0;
    }
    constexpr int UN = 4;
    int mn = INT_MAX, mx = -1;
    for (int jb = a0 + gl; jb < a1; jb += UN * TW) {
        int b[UN], bs[UN], be[UN];
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const int j = jb + u * TW;
            b[u] = j < a1 ? A.col[j] : -1;
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const int j = jb + u * TW;
            bs[u] = be[u] = 0;
            if (j < a1) {
                if ((unsigned)b[u] < (unsigned)K) {
                    bs[u] = B.rpt[b[u]];
                    be[u] = B.rpt[b[u] + 1];
                } else {
                    bad = true;
                }
            }
        }
        int c0[UN], c1[UN];
#pragma unroll
        for (int u = 0; u < UN; u++) {
            c0[u] = INT_MAX;
            c1[u] = -1;
            if (be[u] > bs[u]) {
                c0[u] = B.col[bs[u]];
                c1[u] = B.col[be[u] - 1];
            }
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            mn = min(mn, c0[u]);
            mx = max(mx, c1[u]);
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const int j = jb + u * TW;
            if (j < a1) {
                const int len = be[u] - bs[u];
                P.abs[j] = bs[u];
                P.alen[j] = len;
                f += len;
                if (len > 0) {
                    nl++;
                    leaf = max(leaf, j - a0);
                }
            }
        }
    }
    f = grp_sum<TW>(f, gm);
    nl = grp_sum<TW>(nl, gm);
    leaf = grp_max<TW>(leaf, gm);
    bad = (__ballot_sync(gm, bad) & gm) != 0u;
    const bool ovf = f > INT_MAX;
    if (ovf)
        f = INT_MAX;
    // row class (f, nl, a0, a1 are uniform in the group)
    int bin;
    if (f == 0)
        bin = kBinEmpty;
    else if (nl == 1)
        bin = kBinCopy;
    else if (f <= kWarpMaxFlop)
        bin = kBinWarp;
    else if (f <= kMg2F && a1 - a0 <= kMidMaxK)  // unless the column range is too wide
        bin = f <= kMtF    ? kBinMidTile
              : f <= kMt2F ? kBinMidTile2
              : (f <= kMwF && a1 - a0 <= kMwMaxK) ? kBinMidWarp
              : (f <= kMgF && a1 - a0 <= kMwMaxK) ? kBinMidGroup
                           : kBinMidGroup2;
    else if (f <= P.mid_limit && 2 * nl <= P.mid_limit && a1 - a0 <= kMidMaxK)
        bin = kBinBatch;
    else if (a1 - a0 <= kSegMaxK)
        bin = kBinHeavy;  // segmented (brm_seg.cuh)
    else
        bin = kBinMid;    // row CTA / spill path
    if (bin >= kBinWarp && bin != kBinMid) {
        // column range of the row for the segment planning and the mid rows'
        // keys and bitmaps
        mn = grp_min<TW>(mn, gm);
        mx = grp_max<TW>(mx, gm);
        if (gl == 0)
            P.crange[row] = make_int2(mn, mx);
        // rows placed by rank, where their lists and column range allow
        const int rc = rank_class(f, a1 - a0, (long long)mx - mn, M);
        if (rc > 0 || (rc == 0 && !P.any_order))
            bin = kBinRank0 + rc;
        if ((bin == kBinMidWarp && (long long)mx - mn >= (1ll << kMwRangeBits)) ||
            (bin == kBinMidGroup && (long long)mx - mn >= (1ll << kMgRangeBits)) ||
            ((bin == kBinMidTile || bin == kBinMidTile2) &&
             (long long)mx - mn >= (1ll << kMtRangeBits)) ||
            (bin == kBinMidGroup2 && ((long long)mx - mn >= (1ll << kMg2RangeBits) ||
                                      !merge_group2(f, (long long)mx - mn, M, A.nnz))))
            bin = (f <= P.mid_limit && 2 * nl <= P.mid_limit) ? kBinBatch : kBinHeavy;
        if (bin == kBinHeavy && a1 - a0 > kSegMaxK)
            bin = kBinMid;
    }
    if (gl != 0)
        return;
    if (bad)
        atomicOr(&P.cnt->err, kErrBadInput);
    if (ovf)
        atomicOr(&P.cnt->err, kErrOverflow);
    P.flop[row] = (int)f;
    if (bin == kBinHeavy)
        P.seg_base[row] = atomicAdd(&P.cnt->seg_cap, seg_bound(f, B.N, P.seg_cut));
    const int weight = bin == kBinBatch ? max((int)f, 2 * nl) : 0;  // batch weight
    P.mid_flop[row] = weight;
    if (bin == kBinHeavy || bin == kBinMid)
        P.spill[row] = 0;
    // (0 until a kernel has counted the row: one that stops at an error leaves
    // no length of an earlier call behind)
    P.nnz[row] = bin == kBinCopy ? (int)f : 0;
    if (bin == kBinCopy)
        P.copy_leaf[row] = leaf;
    if (bin == kBinHeavy && f > kHugeFlop) {
        // the planning takes these first, so the longest rows do not
        // start last and finish after every other block
        const int h = atomicAdd(&P.cnt->n_huge, 1);
        if (BRM_IN(P.cnt, M - 1 - h, M))
            P.rows[(size_t)kBinHeavy * M + (M - 1 - h)] = row;
        bin = -2;
    }
    S.bin[slot] = bin;
    S.idx[slot] = bin < 0 || bin == kBinEmpty ? 0 : atomicAdd(&S.cnt[bin], 1);
    S.flop[slot] = (int)f;
    if (weight)
        atomicAdd(&S.mid, (unsigned long long)weight);
    atomicMax(&S.max_k, a1 - a0);
}

// A group of TW lanes per row (TW = 8 when rows are short, 32 otherwise),
// kAnaRowsPerGroup rows per group.
template <int TW>
__global__ void __launch_bounds__(kAnaThreads, 6) k_analyze(CsrDev A, CsrDev B, PlanDev P)
{
    constexpr int NW = kAnaThreads / 32;
    constexpr int NGR = kAnaThreads / TW;  // groups per block
    constexpr int RPB = NGR * kAnaRowsPerGroup;
    __shared__ AnaBlock<RPB> S;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gl = threadIdx.x & (TW - 1);    // lane in the group
    const int grp = threadIdx.x / TW;         // group in the block
    const unsigned gm = TW == 32 ? kFull : (((1u << TW) - 1u) << (lane & ~(TW - 1)));
    if (threadIdx.x < kNumBins)
        S.cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        S.nlong = S.max_k = 0;
        S.mid = 0;
    }
    __syncthreads();
    const int M = A.M;
    const int row0 = blockIdx.x * RPB;
    for (int r = 0; r < kAnaRowsPerGroup; r++) {
        const int slot = grp * kAnaRowsPerGroup + r;
        const int row = row0 + slot;
        if (row >= M) {
            if (gl == 0) {
                S.bin[slot] = -1;
                S.flop[slot] = 0;
            }
            continue;
        }
        const int a0 = A.rpt[row], a1 = A.rpt[row + 1];
        if (TW < 32 && a1 - a0 > kAnaLongK && a0 >= 0 && a1 <= A.nnz) {
            if (gl == 0)
                S.longs[atomicAdd(&S.nlong, 1)] = slot;
            continue;
        }
        analyze_row<TW, RPB>(A, B, P, row, slot, gl, gm, S);
    }
    __syncthreads();
    if (TW < 32 && S.nlong) {
        for (int i = w; i < S.nlong; i += NW)
            analyze_row<32, RPB>(A, B, P, row0 + S.longs[i], S.longs[i], lane, kFull, S);
        __syncthreads();
    }
    // the rows' offsets: prefix over the block's slots (64-bit shared atomics
    // a row took longer), then one device atomic a total, and one a bin
    const int slot = threadIdx.x;
    unsigned long long fx = 0, sx = 0, fi = 0, si = 0;
    if (slot < (RPB + 31) / 32 * 32) {
        if (slot < RPB) {
            const int bin = S.bin[slot];
            fx = (unsigned long long)S.flop[slot];
            sx = bin == kBinWarp || bin >= kBinMidWarp ? fx : 0ull;
        }
        fi = warp_incl_scan(fx);
        si = warp_incl_scan(sx);
        if (lane == 31) {
            S.tot[w][0] = fi;
            S.tot[w][1] = si;
        }
    }
    __syncthreads();
    if (threadIdx.x < kNumBins)
        S.base[threadIdx.x] =
            S.cnt[threadIdx.x] ? atomicAdd(&P.cnt->bin_count[threadIdx.x], S.cnt[threadIdx.x]) : 0;
    if (w == 1 && lane < 2) {
        unsigned long long t = 0;
        for (int i = 0; i < (RPB + 31) / 32; i++)
            t += S.tot[i][lane];
        unsigned long long b = t ? atomicAdd(lane ? &P.cnt->mw_total : &P.cnt->total_flop, t) : 0ull;
        for (int i = 0; i < (RPB + 31) / 32; i++) {
            const unsigned long long x = S.tot[i][lane];
            S.tot[i][lane] = b;
            b += x;
        }
    }
    if (threadIdx.x == 64) {
        if (S.mid)
            atomicAdd(&P.cnt->mid_total, S.mid);
        if (S.max_k > 0)
            atomicMax(&P.cnt->max_k, S.max_k);
    }
    __syncthreads();
    if (slot < RPB && S.bin[slot] != -1) {
        const int bin = S.bin[slot], row = row0 + slot;
        if (P.upper)
            P.scan_flop[row] = (long long)(S.tot[w][0] + fi - fx);
        if (bin == kBinWarp || bin >= kBinMidWarp)
            P.mw_pre[row] = (long long)(S.tot[w][1] + si - sx);
        if (bin > kBinEmpty && bin != kBinBatch && BRM_IN(P.cnt, S.base[bin] + S.idx[slot], M))
            P.rows[(size_t)bin * M + S.base[bin] + S.idx[slot]] = row;
    }
}

void launch_analyze(const CsrDev &A, const CsrDev &B, const PlanDev &P, cudaStream_t s)
{
    if (A.M <= 0)
        return;
    constexpr int RPB32 = (kAnaThreads / 32) * kAnaRowsPerGroup;
    // eight lanes a row when rows average at most 32 entries (four loads a lane
    // in flight then cover the row; the 27-point stencil on 128^3 by whole
    // warps: 1.01 ms, by eighths 0.46)
    if ((long long)A.nnz <= 32ll * A.M) {
        constexpr int RPB = (kAnaThreads / 8) * kAnaRowsPerGroup;
        k_analyze<8><<<(A.M + RPB - 1) / RPB, kAnaThreads, 0, s>>>(A, B, P);
    } else {
        k_analyze<32><<<(A.M + RPB32 - 1) / RPB32, kAnaThreads, 0, s>>>(A, B, P);
    }
    count_launch();
}

// ---------------------------------------------------------------------------
// Exclusive scan, out[n] = total, in two launches (tile sums, then every block
// adds up the sums before its tile), or in one where the blocks before a tile
// are few enough for it to add up their items itself.  Replaces
// opt_prefix_sum (spgemm.h:179-187) for crpt.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
// tiles up to which one launch does it: the last block then reads at most
// 28672 items before its own, which takes less than a launch
constexpr int kScanOneLaunch = 8;

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const int *in, int n,
                                                              long long *tile_sums)
{
    __shared__ long long ws[kScanThreads / 32 + 1];
    const long long base = (long long)blockIdx.x * kScanTile;
    long long s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        long long idx = base + (long long)i * kScanThreads + threadIdx.x;
        if (idx < n)
            s += in[idx];
    }
    long long t = block_sum<kScanThreads>(s, ws);
    if (threadIdx.x == 0)
        tile_sums[blockIdx.x] = t;
}

// tile_sums: the tiles' sums, or nullptr to add up the items before the tile.
template <typename OutT>
__global__ void __launch_bounds__(kScanThreads) k_scan_down(const int *in, int n,
                                                            const long long *tile_sums,
                                                            OutT *out, Counters *cnt)
{
    __shared__ long long ws[kScanThreads / 32 + 1];
    const long long base = (long long)blockIdx.x * kScanTile;
    long long before = 0;
    if (tile_sums) {
        for (int i = threadIdx.x; i < (int)blockIdx.x; i += kScanThreads)
            before += tile_sums[i];
    } else {
#pragma unroll 8
        for (long long i = threadIdx.x; i < base; i += kScanThreads)
            before += in[i];
    }
    // blocked arrangement: thread t owns items [t*I, t*I+I) of the tile
    long long v[kScanItems];
    long long s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        long long idx = base + (long long)threadIdx.x * kScanItems + i;
        v[i] = idx < n ? in[idx] : 0;
        s += v[i];
    }
    before = block_sum<kScanThreads>(before, ws);
    __syncthreads();
    long long tot;
    long long ex = block_excl_scan<kScanThreads>(s, ws, &tot);
    long long run = before + ex;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        long long idx = base + (long long)threadIdx.x * kScanItems + i;
        if (idx < n) {
            if (sizeof(OutT) == 4 && run > INT_MAX) {
                if (cnt)
                    atomicOr(&cnt->err, kErrOverflow);
                out[idx] = (OutT)INT_MAX;
            } else {
                out[idx] = (OutT)run;
            }
        }
        run += v[i];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        long long total = before + tot;
        if (cnt)
            cnt->cnnz = total;
        if (sizeof(OutT) == 4 && total > INT_MAX) {
            if (cnt)
                atomicOr(&cnt->err, kErrOverflow);
            out[n] = (OutT)INT_MAX;
        } else {
            out[n] = (OutT)total;
        }
    }
}

size_t scan_tmp_bytes(int n)
{
    size_t tiles = (size_t)(n + kScanTile - 1) / kScanTile;
    return (tiles + 2) * sizeof(long long);
}

template <typename OutT>
static void scan_impl(const int *in, OutT *out, int n, Counters *cnt, void *tmp, cudaStream_t s)
{
    long long *ts = (long long *)tmp;
    int tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles == 0)
        tiles = 1;
    if (tiles <= kScanOneLaunch) {
        ts = nullptr;
    } else {
        k_scan_reduce<<<tiles, kScanThreads, 0, s>>>(in, n, ts);
        count_launch();
    }
    k_scan_down<OutT><<<tiles, kScanThreads, 0, s>>>(in, n, ts, out, cnt);
    count_launch();
}

void launch_scan_i32(const int *in, int *out, int n, Counters *cnt, void *tmp, cudaStream_t s)
{
    scan_impl<int>(in, out, n, cnt, tmp, s);
}

void launch_scan_i64(const int *in, long long *out, int n, void *tmp, cudaStream_t s)
{
    scan_impl<long long>(in, out, n, nullptr, tmp, s);
}

// ---------------------------------------------------------------------------
// Upper compaction (spgemm.h:429-444): C_bar -> C, in tiles of kCompactTile
// entries of C whatever the rows (a warp per row left the longest row of a
// power-law product, 2e5 entries, to one warp: the whole Upper call on R-MAT
// n=2^18 4.23 -> 3.06 ms).  A
// block finds the tile's first row by a 256-way search, marks where the rows
// start, and a maximum scan gives every entry its row.
// ---------------------------------------------------------------------------
constexpr int kCompactThreads = 256;
constexpr int kCompactPer = 16;
constexpr int kCompactTile = kCompactThreads * kCompactPer;

template <typename T>
__global__ void __launch_bounds__(kCompactThreads)
    k_compact(int M, const long long *scan_flop, const int *__restrict__ bar_col,
              const T *__restrict__ bar_val, const int *crpt, int *ccol, T *cval, Counters *cnt)
{
    __shared__ int s_row[kCompactTile];  // row of each entry, less the tile's first
    __shared__ int s_warp[kCompactThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int nnz = crpt[M];
    const int ntiles = nnz / kCompactTile + (nnz % kCompactTile != 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int q0 = tile * kCompactTile;
        const int len = min(kCompactTile, nnz - q0);
        // last row that starts at or before q0: lo keeps crpt[lo] <= q0
        int lo = 0, n = M;  // candidates lo .. lo + n - 1
        while (n > 1) {
            const int step = (n + kCompactThreads - 1) / kCompactThreads;
            const bool ok = tid * step < n && crpt[lo + tid * step] <= q0;
            const int c = __syncthreads_count(ok);  // ok holds for a prefix of the threads
            lo += (c - 1) * step;
            n = min(step, n - (c - 1) * step);
        }
        const int r0 = lo;
        for (int i = tid; i < kCompactTile; i += kCompactThreads)
            s_row[i] = 0;
        __syncthreads();
        for (int r = r0 + tid; r < M; r += kCompactThreads) {
            const int s = crpt[r];
            if (s >= q0 + len)
                break;
            if (crpt[r + 1] > s)  // one nonempty row starts at each entry
                s_row[max(s - q0, 0)] = r - r0;
        }
        __syncthreads();
        // running maximum: a thread's kCompactPer consecutive entries, then
        // the warps' (the tile's first row, marked 0, is below every other)
        int m[kCompactPer];
#pragma unroll
        for (int i = 0; i < kCompactPer; i++)
            m[i] = max(s_row[tid * kCompactPer + i], i ? m[i - 1] : 0);
        int top = m[kCompactPer - 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(kFull, top, o);
            if (lane >= o)
                top = max(top, x);
        }
        if (lane == 31)
            s_warp[w] = top;
        int before = __shfl_up_sync(kFull, top, 1);
        __syncthreads();
        if (lane == 0)
            before = 0;
        for (int i = 0; i < w; i++)
            before = max(before, s_warp[i]);
#pragma unroll
        for (int i = 0; i < kCompactPer; i++)
            s_row[tid * kCompactPer + i] = max(m[i], before);
        __syncthreads();
#pragma unroll 4
        for (int i = 0; i < kCompactPer; i++) {
            const int q = tid + i * kCompactThreads;
            if (q < len) {
                const int r = r0 + s_row[q];
                const long long src = scan_flop[r] + (q0 + q - crpt[r]);
                // checked build: an entry outside C_bar is skipped
                if (BRM_IN(cnt, src, (long long)cnt->total_flop)) {
                    ccol[q0 + q] = bar_col[src];
                    cval[q0 + q] = bar_val[src];
                }
            }
        }
        __syncthreads();
    }
}

void launch_compact(int dtype, const PlanDev &P, int nnz, const int *bar_col, const void *bar_val,
                    const int *crpt, int *ccol, void *cval, cudaStream_t s)
{
    if (P.M <= 0 || nnz <= 0)
        return;
    const int grid = std::min(nnz / kCompactTile + 1, 1 << 16);
    if (dtype == 0)
        k_compact<double><<<grid, kCompactThreads, 0, s>>>(P.M, P.scan_flop, bar_col,
                                                           (const double *)bar_val, crpt, ccol,
                                                           (double *)cval, P.cnt);
    else
        k_compact<float><<<grid, kCompactThreads, 0, s>>>(P.M, P.scan_flop, bar_col,
                                                          (const float *)bar_val, crpt, ccol,
                                                          (float *)cval, P.cnt);
    count_launch();
}

// ---------------------------------------------------------------------------
// CSR validation (the invariants the reference's reader enforces,
// CSR.cpp:454-477): rpt[0] == 0, rpt non-decreasing, rpt[M] == nnz, columns in
// [0, ncols) and strictly increasing within each row.  One warp per row;
// *bad_row receives the smallest offending row (atomicMin), -1 if none was
// seen (the host initialises it to INT_MAX).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_validate(CsrDev X, int ncols, int *bad_row)
{
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    if (gw == 0 && lane == 0) {
        if (X.rpt[0] != 0)
            atomicMin(bad_row, 0);
        if (X.rpt[X.M] != X.nnz)
            atomicMin(bad_row, X.M > 0 ? X.M - 1 : 0);
    }
    for (int row = gw; row < X.M; row += nw) {
        const int s = X.rpt[row], e = X.rpt[row + 1];
        bool bad = (s > e) || (s < 0) || (e > X.nnz);
        if (!bad) {
            for (int j = s + lane; j < e; j += 32) {
                int c = X.col[j];
                if ((unsigned)c >= (unsigned)ncols)
                    bad = true;
                else if (j + 1 < e && X.col[j + 1] <= c)
                    bad = true;
            }
        }
        if (__any_sync(kFull, bad) && lane == 0)
            atomicMin(bad_row, row);
    }
}

void launch_validate(const CsrDev &X, int ncols, int *bad_row, cudaStream_t s)
{
    int grid = (X.M + 7) / 8;
    if (grid < 1)
        grid = 1;
    if (grid > 65535 * 4)
        grid = 65535 * 4;
    k_validate<<<grid, 256, 0, s>>>(X, ncols, bad_row);
    count_launch();
}

}  // namespace brm

namespace brm {

__global__ void k_pipe_admit(PlanDev P, int M, PipeCaps caps, int stage)
{
    Counters *c = P.cnt;
    bool bad;
    if (stage == 0)
        bad = (long long)c->total_flop > caps.products || (long long)c->seg_cap > caps.seg_slots ||
              (long long)(c->mw_total + c->mid_total) > caps.products + caps.nnz_a;
    else
        bad = (long long)c->table_cap > caps.table || (long long)c->spill_bytes > caps.spill_bytes;
    if (bad) {
        c->abort = 1;
        atomicOr(&c->err, kErrCapacity);
    }
}

void launch_pipe_admit(const PlanDev &P, int M, const PipeCaps &caps, int stage, cudaStream_t s)
{
    k_pipe_admit<<<1, 1, 0, s>>>(P, M, caps, stage);
    count_launch();
}

}  // namespace brm

// SM version of the device code this library runs on the current device.
extern "C" int brm_device_code_version(int *sm)
{
    if (!sm)
        return BRM_ERR_INVALID_VALUE;
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, brm::k_scan_reduce);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return e == cudaErrorNoDevice ? BRM_ERR_NO_DEVICE : BRM_ERR_CUDA;
    }
    *sm = fa.binaryVersion;
    return BRM_SUCCESS;
}
