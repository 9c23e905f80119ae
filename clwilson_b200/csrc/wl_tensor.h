// wl_tensor.h -- column products on the tensor cores: what the engine hands
// over and what the kernels of wl_tensor.cu share with their planner.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

#include "wl_internal.h"

namespace wl {

// One bucket's columns [c0, c1) of the resident table: every row r in
// [row_begin, row_begin + nrows) gets prod q^{v_q(T!)} over them.
struct TensorTask {
    uint64_t T;
    uint64_t c0, c1;
    uint32_t row_begin, nrows;
    int L;
    uint32_t q_max;      // bound on its largest column
    uint32_t id = 0;     // the caller's place in its list (tensor_products sets it)
};

// Geometry of the tensor-core product (see wl_tensor.cu).
constexpr uint32_t TN_K = 512;          // bytes of a group product: 128 limbs of 32 bits
constexpr uint32_t TN_KB = TN_K / 128;  // 128-byte blocks of it
constexpr uint32_t TN_M = 128;          // groups per tile (tensor memory lanes)
constexpr uint32_t TN_N = 256;          // row digits per tile: TN_N / (4L) rows
constexpr uint32_t TN_GMAX = 512;       // columns per group at most
constexpr uint32_t TN_COLS_PER_BLOCK = 4096;   // columns per CTA of the digit sort
constexpr uint32_t TN_SCATTER = 2;      // CTAs of the write-out per CTA of the count
constexpr uint32_t TN_WMAX = 9;         // bits of a digit at most
constexpr uint32_t TN_LABELS = 4096;    // digit labels of a task at most
constexpr uint32_t TN_DIGITS = 32;      // digits per block of the window products
constexpr uint32_t TN_SEG = 64;         // slots per segment of the label fold
__host__ __device__ constexpr uint32_t tn_rows(int L) { return TN_N / (4u * (uint32_t)L); }

// Where the rows live: their moduli, the accumulators to multiply into, and a
// word that a kernel sets when one of its waits runs out (after wl_ctx::wait_ns).
struct TensorTarget {
    const RowMod* mods;
    uint4* acc;
    uint32_t* err;
};

// Device descriptor of a task.
struct TensorDesc {
    uint64_t T;
    uint64_t part0;      // first element of its lane-run products (slot-major, rows_pad apart)
    uint64_t seg_part0;  // first element of its segment products
    uint64_t win0;       // first element of its window products (a row of them per window and digit block)
    uint32_t c0, c1;
    uint32_t q_max;      // no column is above it
    uint32_t row_begin, nrows, rows_pad;   // rows_pad: whole row tiles
    uint32_t w, nwin;    // digit width and count
    uint32_t lab0;       // first label (nwin << w of them)
    uint32_t lab_seg0;   // first entry of its table of label segments (one longer than the labels)
    uint32_t blk0;       // first CTA of the digit sort
    uint32_t ct0;        // first row-constant tile
    uint32_t fold_blk0, row_blk0;   // first CTA of the segment fold / per-row kernels
    uint32_t seg0, nseg;
    uint32_t list0;      // first list entry
    uint32_t long0, nlong, short0, nshort;   // its lane runs of both lengths: first, padded count
};
// What a task takes, from its digit counts.
struct TensorSize { uint32_t entries, longs, shorts, slots, segs; };
// Groups per lane run: a label's groups go in runs of 32, the rest in runs of
// 4, so that a label wastes about two groups however many it has.
constexpr uint32_t TN_LONG = 32, TN_SHORT = 4;
// A section of a task: 128-lane blocks of lane runs of the same length.
struct TensorSec {
    uint32_t task;
    uint32_t tn;         // groups per lane run
    uint32_t mt0;        // first group tile
    uint32_t run0;       // first lane run
    uint32_t reduce;     // products of lanes with the same slot are multiplied before they are written
    uint32_t g;          // tails: integers per group
};
// A lane run: tn consecutive groups of one label's list, one after another in
// one lane of the accumulator.  Group t covers list[start + t*g .. +g), cut at
// end.  Its product goes to `slot` of the task (RUN_NONE: nowhere).
struct LaneRun { uint32_t start, end, g, slot; };
constexpr uint32_t RUN_NONE = 0xFFFFFFFFu;
// Consecutive slots of one label, for the label fold.
struct FoldSeg { uint32_t slot0, n; };
// The consecutive-integer tails of a bucket's rows, T+1 .. Tp per row: groups of
// `g` integers, group j the integers T + 1 + j g .., shared by all rows; a row
// takes the first (Tp - T) / g of them here and the rest, fewer than g, one by one.
struct TensorTail { uint64_t T; uint32_t row_begin, nrows, L; };
// The largest integer a group may hold: a lane's share of a group's integers stays
// below 2^160 up to 44 bits.
constexpr uint64_t TAIL_MAX = 1ull << 44;
constexpr uint32_t TAIL_SLOTS = 4;     // products per row: one from each warp quarter
// One CTA's work: 128-lane blocks [cb0, cb0 + ncb) of a section against row tile `tile` of its task.
struct TensorItem { uint32_t sec, tile, cb0, ncb; };

void launch_tensor_count(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const uint32_t* cols, uint32_t* counts,
                         cudaStream_t st);
// the tasks' sizes, from the counts
void launch_tensor_size(const TensorDesc* d, uint32_t ntask, const uint32_t* counts, TensorSize* size, cudaStream_t st);
// their list places (cursor), lane runs, label segments
void launch_tensor_layout(const TensorDesc* d, uint32_t ntask, const uint32_t* counts, uint32_t* cursor, LaneRun* runs,
                          FoldSeg* segs, uint32_t* lab_seg, cudaStream_t st);
void launch_tensor_scatter(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const uint32_t* cols,
                           uint32_t* cursor, uint32_t* list, cudaStream_t st);
// the group products of nmt group tiles, in the tiles' shared-memory image
void launch_tensor_build(const TensorSec* sec, uint32_t nsec, uint32_t nmt, const LaneRun* lr, const uint32_t* list,
                         uint8_t* w, cudaStream_t st);
// ones: R mod n of every row of every tile
void launch_tensor_consts(int L, const TensorDesc* d, uint32_t ntask, uint32_t ntiles, const RowMod* mods, uint8_t* consts,
                          uint4* ones, cudaStream_t st);
int launch_tensor_gemm(int L, uint32_t nitems, const TensorDesc* d, const TensorSec* sec, const TensorItem* items,
                       const LaneRun* lr, const RowMod* mods,
                       const uint8_t* w, const uint8_t* consts, const uint4* ones, void* part, uint32_t* err,
                       uint64_t wait_ns, cudaStream_t st);
// tails: group products, the matrix product with each row's own number of groups
// (items: cb0 = 0, ncb = group tiles), and the rest of each row's integers with
// the product into acc
void launch_tensor_tail_build(const TensorDesc* d, const TensorSec* sec, uint32_t nsec, uint32_t nmt, uint8_t* w,
                              cudaStream_t st);
int launch_tensor_tail_gemm(int L, uint32_t nitems, const TensorDesc* d, const TensorSec* sec, const TensorItem* items,
                            const RowInfo* info, const RowMod* mods, const uint8_t* w, const uint8_t* consts,
                            const uint4* ones, void* part, uint32_t* err, uint64_t wait_ns, cudaStream_t st);
void launch_tensor_tail_rows(int L, const TensorDesc* d, const TensorSec* sec, uint32_t ntask, uint32_t nblocks,
                             const RowInfo* info, const RowMod* mods, const uint4* ones, const void* part, uint4* acc,
                             cudaStream_t st);
void launch_tensor_fold(int L, const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const FoldSeg* segs,
                        const RowMod* mods, const void* part, void* seg_part, cudaStream_t st);
void launch_tensor_combine(int L, const TensorDesc* d, uint32_t ntask, uint32_t nblocks, uint32_t max_blocks,
                           const uint32_t* lab_seg, const RowMod* mods, const uint4* ones, const void* seg_part,
                           void* win, uint4* acc, cudaStream_t st);

}  // namespace wl
