// brm_plan.h -- data shared between the host orchestration and the kernels.
//
// A plan is the device state that the symbolic phase leaves for the numeric
// phase (the reference keeps the same state in local arrays between its
// symbolic and numeric loops, BRMerge-SpGEMM/inc/spgemm.h:476-578).
#pragma once

#include <cstdint>

#include <vector_types.h>

namespace brm {

// Tuning constants of the row kernels.
constexpr int kRowThreads = 512;            // threads of a row CTA
constexpr int kCap = 6144;                  // products staged in shared memory per window
constexpr int kLMax = 4096;                 // lists (A-row entries) kept in shared memory
constexpr int kChunkWords = 4096;           // bitmap words per column chunk
constexpr int kChunkBits = kChunkWords * 32;  // columns per chunk (131072)
constexpr int kWarpMaxFlop = 32;            // rows up to this many products go to warp kernels
constexpr int kHeavyFlop = 4 * kCap;        // rows above this are scheduled first
constexpr int kRadixBits = 7;

// Batched mid-row kernels: rows with more than kWarpMaxFlop products, weight
// w = max(products, 2 * nonempty lists) <= kMidFlop and at most kMidMaxK A
// entries are packed, in row order, into batches (a batch starts where the
// row-order prefix of w crosses a multiple of kMidFlop, so a batch holds at
// most kMidCap products and kMidMaxLists nonempty lists).
constexpr int kMidThreads = 256;
constexpr int kMidCap = 4096;
constexpr int kMidFlop = kMidCap / 2;
constexpr int kMidMaxLists = kMidCap / 2;
constexpr int kMidMaxK = 255;
constexpr int kMidMaxRows = kMidCap / (kWarpMaxFlop + 1) + 2;

// Merged mid rows, where the rank rows below do not take them.  Warp mid rows:
// more than kWarpMaxFlop and at most kMwF products, at most
// kMwMaxK A entries, columns within a range below 2^kMwRangeBits; one warp
// each.  Group rows: up to kMgF products and kMwMaxK A entries, range below
// 2^kMgRangeBits, four warps each; longer group rows (up to kMg2F products,
// kMidMaxK A entries) in their own class.  All take precedence over the
// batched mid rows and over the segmented heavy rows.  Holding the first two
// classes to 64 lists keeps their merge-tree stacks at seven levels and
// their kernels within 80 registers without spills.  Rows of more than kMgF
// products are merged only where merge_group2 says so; in R-MAT n=2^18 they
// are cut (merged they took 178 us, the whole call 2.24 -> 2.18 ms without).
constexpr int kMwF = 768;
constexpr int kMwMaxK = 64;
constexpr int kMwRangeBits = 22;
constexpr int kMtF = 64;          // tile rows: at most 64 products, half a warp each
constexpr int kMt2F = 128;        // second tile class: at most 128 products
constexpr int kMtRangeBits = 25;
constexpr int kMgF = 3072;
constexpr int kMgRangeBits = 20;
constexpr int kMg2F = 5888;       // second group class (two groups a CTA fit 2 CTAs an SM)
constexpr int kMg2RangeBits = 19;
// Rank rows (brm_midrank.cuh): rows of at most 64 lists whose products are
// placed by population counts instead of sorted; they take precedence over the
// tile, warp and group rows above, which keep the wide ranges (one level of
// summary words outgrows a row's shared memory there).  Class 8 takes the rows
// of 65 to 255 lists through the segment kernel, a row a segment.
// R-MAT n=2^18: rows of 769..3072 products 0.35 -> 0.28 ms.
// The most products of a row of each class:
constexpr int kRkF0 = 128;
constexpr int kRkF1 = 384;
constexpr int kRkF2 = 768;
constexpr int kRkF3 = 1536;
constexpr int kRkF4 = 3072;
constexpr int kRkF5 = 6144;
constexpr int kRkNarrowK = 32;      // lists of the rows with one mask word a column
constexpr int kRkMaxK = 64;
constexpr int kRkF8 = 3072;         // class 8: more lists, by a segment's kernel
constexpr int kRkSegMaxK = 255;
constexpr int kRkRangeBits0 = 18;   // column range, class 0
constexpr int kRkPackBits = 17;     // two rows of class 0 share a pack below
constexpr int kRkRangeBits8 = 18;   // class 8
constexpr int kRkRangeBits = 19;    // the others
// Rows of each narrow class that one SM works on at a time (class 0: eight a warp).
constexpr int kRkRows[6] = {256, 24, 10, 7, 4, 2};
// A row of class 0 with a pack to itself pays all of the pack's fixed cost.
// Numeric phase, 2^18 columns, 30 M products, packed and by the kernels that
// sort: rows of 2 x 8 products 2.14 and 1.30 ms, 4 x 12 0.84 and 0.61, 8 x 8 0.64
// and 0.50; 4 x 24 0.50 and 0.60, 16 x 7 0.51 and 0.63, 30 x 1 1.29 and 2.40, 16 x 2
// 1.15 and 1.27.  So it takes more than kMtF products or, of at most 32 (a warp that
// walks the lists one by one otherwise), 16 lists.  A matrix of few rows keeps
// them all in the pack: launches of two more classes cost more than it does
// (numeric phase, 5000 rows of up to 10 entries over 150,000 columns 60 us packed
// and 72 split up, 40,000 of up to 12 127 and 105).
constexpr int kRkAloneRows = 16384;
__host__ __device__ inline bool rank_alone(long long f, int k, int rows)
{
    return f > kMtF || (f <= 32 && k >= 16) || rows < kRkAloneRows;
}
// Classes 7 and 9 are told apart where there are rows enough for both (1000 rows of
// up to 46 entries over 1000 columns: numeric phase 94 us in one class, 112 in two;
// 5000 of up to 58 over 5000: 209 and 193).
constexpr int kRkSplitRows = 4096;
// The class of a row of f products, k lists and columns within `range` of the
// first, in a matrix of `rows` rows; -1 where it has none.
__host__ __device__ inline int rank_class(long long f, int k, long long range, int rows)
{
    if (f <= 0 || f > kRkF5 || range < 0 || range >= (1ll << kRkRangeBits))
        return -1;
    if (k <= kRkNarrowK) {
        if (f <= kRkF0)
            return range < (1ll << (rank_alone(f, k, rows) ? kRkRangeBits0 : kRkPackBits)) ? 0 : -1;
        return f <= kRkF1 ? 1 : f <= kRkF2 ? 2 : f <= kRkF3 ? 3 : f <= kRkF4 ? 4 : 5;
    }
    if (k <= kRkMaxK)
        return f <= kRkF0 ? -1 : f <= kRkF2 ? 6 : f > kRkF4 ? -1 : f <= range && rows >= kRkSplitRows ? 9 : 7;
    return f > kRkF0 && f <= kRkF8 && k <= kRkSegMaxK && range < (1ll << kRkRangeBits8) ? 8 : -1;
}
// Rows of more than kMgF and at most kMg2F products that no rank class takes
// (33 to 255 lists): merged by a group where columns are shared by several
// products, else cut into segments, which pay by the column of several
// products.  The column range tells them apart: A * A, matrices of k entries a
// row spread over a band, one call, merged against segments:
//   57 x 57 products  range 457: 1.13 ms, 1.52   1141: 1.10, 1.07   3421: 1.11, 0.88
//   76 x 76           range 913: 1.09, 1.34      1521: 1.08, 1.26   2433: 1.07, 0.95
//   100 x 35          range 401: 1.11, 1.50      1201: 1.09, 1.05
// But a group's thread merges ceil(f / 128) products, and where that is 32 its
// reads meet in one bank (57 % slower): those are cut whatever their range.
// A group takes about 120 us for a row, so a few such rows among others are cut too:
// R-MAT n=1500, 8 entries a row, numeric phase 0.15 and 0.27 ms.  Merged are those of
// matrices of many rows or of rows that long on average (kMg2MeanK entries: 1143 rows of
// 100 x 35 products, numeric phase 0.19 ms merged, 0.23 cut).
// Rows that reach into a second planning chunk pay for the planning of both, which
// up to kMg2WideF products costs more than it saves where it is not reused: 40 x 90
// products over 2^19 columns, merged against segments: symbolic 0.48, 0.62, one call
// 1.05, 1.13, Upper 1.10, 1.34 (numeric phase alone 0.83, 0.49).
constexpr int kMg2Share = 3;
constexpr int kMg2WideF = 31 * 128;
constexpr int kMg2Rows = 2048;
constexpr int kMg2MeanK = 32;
__host__ __device__ inline bool merge_group2(long long f, long long range, int rows, int nnz)
{
    return f <= kMgF ||
           ((rows >= kMg2Rows || nnz > (long long)kMg2MeanK * rows) &&
            ((f >= kMg2Share * (range + 1) && (f + 127) / 128 != 32) ||
             (f <= kMg2WideF && range >= (1ll << kRkRangeBits8))));
}
// Subsets of the mid-row kernels (they can run on different streams).
constexpr int kMidGroups = 1;     // the batched mid rows and the four-warp group rows
constexpr int kMidWarps = 2;      // the warp and tile rows

// Segmented heavy rows: a row that is not a mid row is cut, at 32-column word
// (or, inside very dense words, column) boundaries, into column segments of at
// most kSegCap products within one planning chunk of kPlanBits columns.  The
// planning pass records, for every segment boundary and every list of the
// row, where the list crosses the boundary (the split table), so each segment
// is an independent unit of work.
#ifndef BRM_SEG_THREADS
#define BRM_SEG_THREADS 256
#endif
#ifndef BRM_SEG_CAP
#define BRM_SEG_CAP 3072
#endif
constexpr int kSegThreads = BRM_SEG_THREADS;
constexpr int kSegCap = BRM_SEG_CAP;
static_assert(kRkF8 <= kSegCap, "rank rows of class 8 are a segment's size");
// Target products between cuts (a runtime knob, brm_tuning.seg_cut): the
// default and the largest accepted.  Segments average about the target, so a
// larger one means fewer segments (less fixed work per product in the
// segment kernel, a smaller split table) but more dense planning groups
// (above kSegCap - target products), whose columns are counted one by one.
// R-MAT n=2^18 C = A*A one-call Precise: 1536 -> 2.33 ms, 2048 -> 2.21,
// 2304 -> 2.16, 2560 -> 2.18, 2688 -> 2.24; float32 R-MAT n=2^16: 3.31, 3.08,
// 3.24, 3.30, 3.65 (same output).
constexpr int kSegCut = kSegCap * 3 / 4;
constexpr int kSegMaxCut = kSegCap * 7 / 8;
constexpr int kSegMaxK = 65535;           // leaf index stored in 16 bits
constexpr int kLongMin = 33;              // products of a column handed to the column reducer
constexpr int kHugeFlop = 16 * kSegCap;   // heavy rows planned first (longest first)
constexpr int kMaxParts = 16;             // row parts of a numeric phase run part by part
constexpr int kPlanWordsLog2 = 13;
constexpr int kPlanWords = 1 << kPlanWordsLog2;  // bitmap words per planning chunk
constexpr int kPlanBits = kPlanWords * 32;       // 2^18 columns
constexpr int kSumWords = kPlanBits / 1024;      // summary words of a segment bitmap

// Device error bits, OR-ed into Counters::err and read back by the host.
enum DevErr : int {
    kErrNone = 0,
    kErrWindowOverflow = 1,  // a numeric window exceeded its shared-memory capacity
    kErrNnzMismatch = 2,     // numeric row length differs from the symbolic count
    kErrSpillCapacity = 4,   // spill scratch smaller than a spill row needs
    kErrOverflow = 8,        // an int32 quantity overflowed
    kErrBadInput = 16,       // an index out of range seen by a kernel
    kErrCapacity = 32,       // a batch exceeded a captured pipeline's capacities
    kErrChecked = 64,        // a bounds check of the checked build failed (brm_check.cuh)
    kErrUnsorted = 128,      // a short row of unsorted B rows, for the kernels that sort
};

// Row classes assigned by the analysis kernel.
enum RowBin : int {
    kBinEmpty = 0,  // no products: nnz 0
    kBinCopy = 1,   // exactly one nonempty list: C row = a * B row
    kBinWarp = 2,   // <= kWarpMaxFlop products, >= 2 nonempty lists
    kBinHeavy = 3,  // row CTA, scheduled first
    kBinMid = 4,    // row CTA
    kBinBatch = 5,  // batched mid-row kernels (no row list: row-order batches)
    kBinMidWarp = 6,  // one warp per row (brm_midwarp.cuh)
    kBinMidGroup = 7, // four warps per row (brm_midwarp.cuh)
    kBinMidTile = 8,  // half a warp per row, products sorted in registers (brm_midwarp.cuh)
    kBinMidTile2 = 9, // the same with twice the products
    kBinMidGroup2 = 10,  // four warps per row, longer rows (brm_midwarp.cuh)
    kBinRank0 = 11,      // rank rows, classes 0 .. 7 (brm_midrank.cuh)
    kBinSegRow = 19,     // rank rows of more than 64 lists, class 8 (brm_seg.cuh)
    kBinRank9 = 20,      // rank rows, class 9 (brm_midrank.cuh)
    kNumBins = 21,
};

constexpr int kRankClasses = kNumBins - kBinRank0;
// work counters of the mid-row kernels: the merge shapes, then the rank classes
constexpr int kMwRankCounter = 3;
constexpr int kMwCounters = kMwRankCounter + kRankClasses;

// Device counters (one struct in device memory, zeroed per phase).
struct Counters {
    int bin_count[kNumBins];
    int spill_count;
    int work_sym;      // dynamic row counter of the symbolic row kernel
    int max_k;         // longest A row
    // err, then the counters of the numeric phase: cleared by one memset, with
    // or without err
    int err;           // OR of DevErr bits
    int work_num;      // dynamic row counter of the numeric row kernel
    int work_bnum;     // dynamic batch counter, numeric
    int work_seg;      // dynamic segment counter, numeric
    // long columns of the segment kernel handed to the column reducers:
    // columns and elements reserved so far (two counters, so neither can
    // overflow into the other however many columns a call has)
    unsigned long long long_cols;
    unsigned long long long_elems;
    unsigned long long total_flop;
    unsigned long long mw_total;   // products of the warp, tile, merge and rank rows
    unsigned long long mid_total;  // weights of the batched mid rows
    unsigned long long spill_bytes;  // scratch reserved for spill rows
    long long cnnz;    // total nnz of C (int64 before the int32 check)
    int n_batch;       // number of mid-row batches
    int work_bsym;     // dynamic batch counter, symbolic
    unsigned long long seg_cap;    // descriptor slots reserved by the analysis
    unsigned long long table_cap;  // split-table entries reserved by the planning
    int n_seg;         // segments written by the planning
    int work_plan;     // dynamic row counter of the heavy-row planning
    int n_huge;        // heavy rows above kHugeFlop products (listed from the end)
    // set by the capacity checks of a captured batch pipeline when the batch
    // does not fit its buffers; every kernel that writes at data-dependent
    // offsets then returns at once (the call reports BRM_ERR_CAPACITY)
    int abort;
    // first failed bounds check of the checked build: source line, index, bound
    int chk_line;
    long long chk_idx;
    long long chk_bound;
    // dynamic row counters of the warp / four-warp mid-row kernels (one per
    // shape) and the groups of a launch that have finished; the last group
    // of a launch sets both back to zero, so every launch starts from zero
    // whatever phase or pipeline runs it
    int work_mw[kMwCounters];
    int done_mw[kMwCounters];
};

// Descriptor slots reserved for a heavy row with F products and the cut
// target `cut`: the cut rule makes at most F / cut cuts at product
// thresholds (plus one per chunk), 2 per dense group (a group with more than
// dense = kSegCap - cut products; at most F / dense of them) and at most
// 2 h / cut + 1 inside a dense group of h products, plus one chunk start per
// kPlanBits columns: at most 3 F / cut + 3 F / dense <= 6 F / min(cut, dense)
// and the chunk terms.
__host__ __device__ inline unsigned long long seg_bound(long long F, int N, int cut)
{
    const int m = cut < kSegCap - cut ? cut : kSegCap - cut;
    return 6ull * (unsigned long long)((F + m - 1) / m) +
           2ull * ((unsigned)N / (unsigned)kPlanBits) + 8ull;
}

// Runtime policy knobs of the row classes (chosen by brm_autotune or
// brm_set_tuning; every capacity stays compile-time): the heavy-row cut
// target seg_cut in [kMinSegCut, kSegMaxCut] (segments hold at most kSegCap
// products whatever the target) and the mid-row weight limit mid_flop in
// [kMinMidFlop, kMidFlop] (batches hold at most 2 * mid_flop <= kMidCap).
// The results do not depend on them: only where rows and segments are cut.
constexpr int kMinSegCut = 256;
constexpr int kMinMidFlop = 128;

// One column segment of a heavy row.
struct SegDesc {
    int row;
    int c_lo;       // first column of the segment
    int c_hi;       // one past the last column
    int u_off;      // distinct columns of the row before c_lo
    int bidx;       // boundary index of c_lo in the row's split table
    int nprod;      // products in the segment
    long long tab;  // split-table offset of the row (boundary-major, k entries each)
};

// A segment as the segment kernel reads it: one 48-byte record per entry of
// the segment list (in list order), written by k_split, so that a segment
// needs a single dependent load after the work counter (and the next one is
// copied into shared memory while the current segment runs).
struct __align__(16) SegRun {
    long long sp;  // split-table offset of the segment's first boundary row (tab + bidx * k)
    int row;
    int c_lo;
    int c_hi;
    int u_off;     // distinct columns of the row before c_lo
    int nprod;
    int a0;        // A row start and length
    int k;
    int next_u;    // distinct columns of the row before the next segment (or its nnz)
};
static_assert(sizeof(SegRun) == 48, "three 16-byte copies");

// A column of a heavy-row segment with many products, handed from the
// segment kernel to the column reducer: its products' leaves and values in
// leaf order at [off, off + len) of the long-column scratch, and the output
// position.  len < 0: the segment kernel reduced the column itself.
struct LongCol {
    long long out;  // index into (ccol, cval)
    long long off;  // first element in the scratch
    int col;        // column of C
    int len;
};

// Device arrays of a plan (all sized for M rows unless noted).
struct PlanDev {
    int M;
    int *flop;        // [M] products per row
    int *nnz;         // [M] symbolic row length (Upper: numeric row length)
    int *rows;        // [kNumBins * M] row lists, bin b at rows + b*M
    int *copy_leaf;   // [M] leaf of the single nonempty list (copy rows)
    unsigned char *spill;  // [M] 1 if the row takes the spill path
    int *spill_rows;  // [M] spill row list
    unsigned long long *spill_off;  // [M] scratch byte offset per spill list entry
    long long *scan_flop;  // [M] offset of each row in C_bar (Upper)
    int *abs;              // [nnz(A)] start of B row acol[j] (list start of A entry j)
    int *alen;             // [nnz(A)] length of B row acol[j] (0 if acol[j] is out of range)
    int *mid_flop;         // [M] products of batched mid rows, 0 for other rows
    long long *mid_pre;    // [M+1] exclusive scan of mid_flop
    long long *mw_pre;     // [M] offset of each warp, tile, merge or rank row in the one-call
                           // scratch (the batched mid rows lie behind them, at
                           // Counters::mw_total + mid_pre)
    int *batch_start;      // [M+1] first row of each mid batch
    unsigned long long *seg_base;  // [M] first descriptor slot of each heavy row
    int *seg_n;            // [M] segments of each heavy row (0: not segmented)
    int2 *crange;          // [M] smallest and largest column of each heavy row (x > y: none)
    SegDesc *seg;          // [Counters::seg_cap] segment descriptors (numbered per row)
    int *seg_list;         // [Counters::seg_cap] descriptor slot of every written segment
    SegRun *run;           // [Counters::seg_cap] records of the segment list (numeric phase)
    int *split;            // [Counters::table_cap] split table (numeric phase)
    LongCol *long_col;     // [long_cap_cols] long-column descriptors (numeric phase)
    unsigned short *long_leaf;  // [long_cap_elems] leaves of the long columns' products
    void *long_val;        // [long_cap_elems] their values (the value type)
    long long long_cap_cols;
    long long long_cap_elems;
    // numeric launches may cover only rows [r_lo, r_hi) (a part of C copied
    // back while the next part computes); seg_range (device, 2 ints), when
    // set, is the part's range of seg_list
    int r_lo;
    int r_hi;
    const int *seg_range;
    // policy knobs (see kMinSegCut): heavy-row cut target, mid-row weight limit
    int seg_cut;
    int mid_limit;
    int upper;  // the analysis writes scan_flop
    int any_order;  // no rows of rank class 0 (a plan made again after kErrUnsorted)
    // entries of the arrays the numeric kernels write (C, or C_bar for
    // Upper) and of the one-call mid-row scratch; the bounds of the checked
    // build
    long long c_cap;
    long long mid_cap;
    Counters *cnt;
    // host side only: the launches the plan needs (kLive* bits); all ones
    // when the host does not know the class counts (a captured pipeline);
    // rank_span[c]: rank classes below c whose few rows c's launch takes along,
    // rank_taken their bits
    unsigned live;
    int rank_span[kRankClasses];
    unsigned rank_taken;
};

// Launch mask of a plan (PlanDev::live): bit b set when row class b (RowBin)
// has rows, kLiveSegs when heavy rows were cut into segments.  The launchers
// skip the kernels of empty classes, which for small products are most of
// the launches of a call.
constexpr unsigned kLiveSegs = 1u << 30;
constexpr unsigned kLiveAll = 0xffffffffu;
constexpr unsigned live_bit(int bin) { return 1u << bin; }
// rows of the one-call scratch
constexpr unsigned kLiveMidRows = live_bit(kBinWarp) | live_bit(kBinBatch) | live_bit(kBinMidWarp) |
                                  live_bit(kBinMidGroup) | live_bit(kBinMidTile) |
                                  live_bit(kBinMidTile2) | live_bit(kBinMidGroup2) |
                                  (live_bit(kNumBins) - live_bit(kBinRank0));
constexpr unsigned kLiveGroups = live_bit(kBinBatch) | live_bit(kBinMidGroup) |
                                 live_bit(kBinMidGroup2) | live_bit(kBinRank0 + 3) |
                                 live_bit(kBinRank0 + 4) | live_bit(kBinRank0 + 5) |
                                 live_bit(kBinRank0 + 7) | live_bit(kBinSegRow) |
                                 live_bit(kBinRank9);  // kMidGroups
inline bool plan_live(const PlanDev &P, unsigned bits) { return (P.live & bits) != 0; }

// Capacities of a captured batch pipeline: every buffer sized by a count the
// planning computes on the device is grown to these once, and admission
// kernels compare each batch's counts with them (Counters::abort).
struct PipeCaps {
    long long rows;         // rows of the stacked A (and of C)
    long long nnz_a;        // entries of the stacked A
    long long b_rows;       // rows of the stacked B
    long long nnz_b;        // entries of the stacked B
    long long cols;         // columns of the stacked B
    long long products;     // intermediate products (bounds nnz(C); with nnz_a the mid-row scratch)
    long long seg_slots;    // heavy-row segment descriptors
    long long table;        // split-table entries
    long long spill_bytes;  // spill scratch
};

struct CsrDev {
    int M, N, nnz;
    const int *rpt;
    const int *col;
    const void *val;
};

}  // namespace brm
