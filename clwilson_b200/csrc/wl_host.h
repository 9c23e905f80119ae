// wl_host.h -- host-side internals shared by the engine (wl_engine.cu) and the
// serving session (wl_serve.cu): device buffers, error macros, the context.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include <cuda_runtime.h>

#include "wilson.h"
#include "wl_internal.h"
#include "wl_tensor.h"

// A growable device buffer.
struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    bool inner = false;    // lies in another buffer (TensorBufs::block): not freed by itself
};
inline void release(DevBuf& b) {
    if (b.p && !b.inner) cudaFree(b.p);
    b = DevBuf();
}

inline int ensure(DevBuf& b, size_t bytes) {
    if (bytes <= b.cap && b.p) return 0;
    release(b);
    size_t nb = std::max<size_t>(bytes, 256);
    if (cudaMalloc(&b.p, nb) != cudaSuccess) {
        cudaGetLastError();
        return WL_ERR_NOMEM;
    }
    b.cap = nb;
    return 0;
}

template <class T> inline T* as(DevBuf& b) { return reinterpret_cast<T*>(b.p); }

// Rows per thread of the prefix-fold sweep for a bucket of nrows rows, given
// the tuned choice (1, 2 or 4): one row below 512 rows, at most two below 1,024.
inline int sparse_rpt_for(int tuned, uint32_t nrows) {
    if (nrows < 512) return 1;
    if (tuned == 4 && nrows < 1024) return 2;
    return tuned;
}

// Row tiles of a bucket's n rows for the sweep kernels (256-thread CTAs).
// Full tiles of 256 * rpt rows (one split per CTA), then tiles of 256 rows,
// then the last rows in one tile whose group width is the rest rounded up to
// a power of two (at least min_tps) up to 32 rows and to a multiple of 32
// above: several splits share a CTA when the width is below 256, and few
// lanes carry no row (a power-of-two width for the rest would leave up to
// half of them empty).
// same_groups: every tile of the bucket runs the same number of splits per
// CTA -- the dense sweep stages a CTA's columns in chunks shared by its
// groups, and the power of two that a split's product drops depends on the
// chunk length, so all rows of a split must see the same chunks.  Then a
// bucket of 256 * rpt rows or more keeps full tiles, one split per CTA, and
// its last rows go in one tile of the rest's width that also runs one split
// per CTA (groups = 1; the CTA's threads past it idle); a smaller bucket is
// one tile.
struct RowTile {
    uint32_t row0, tps;
    int rpt;
    uint32_t groups = 0;     // splits per CTA; 0: 256 / tps
};
inline uint32_t group_width(uint32_t lanes, uint32_t min_tps) {
    return lanes <= 32 ? std::max(lanes, min_tps) : (lanes + 31) / 32 * 32;
}
inline void row_tiles(uint32_t n, int rpt, uint32_t min_tps, std::vector<RowTile>& out, bool same_groups = false) {
    out.clear();
    uint32_t r0 = 0;
    const uint32_t full = 256u * (uint32_t)rpt;
    while (n - r0 >= full) { out.push_back({ r0, 256u, rpt }); r0 += full; }
    if (same_groups && r0 > 0) {
        const uint32_t rest = n - r0;
        if (rest) out.push_back({ r0, group_width((rest + rpt - 1) / rpt, min_tps), rpt, 1u });
        return;
    }
    while (n - r0 >= 256u) { out.push_back({ r0, 256u, 1 }); r0 += 256u; }
    const uint32_t rest = n - r0;
    if (!rest) return;
    out.push_back({ r0, group_width(rest, min_tps), 1 });
}
// Splits one item of the tile runs.
inline uint32_t tile_groups(const RowTile& t) { return t.groups ? t.groups : 256u / t.tps; }
// The sweep items of one tile: one per split for full-width tiles, else one
// per tile_groups consecutive splits.
template <class Push>
inline void tile_items(const RowTile& t, uint32_t s_begin, uint32_t s_end, Push push) {
    const uint32_t per = tile_groups(t);
    const uint32_t code = t.groups ? (t.tps | (t.groups << 16)) : t.tps;
    for (uint32_t s = s_begin; s < s_end; s += per) push(t.row0, s, code);
}

// Limb width of residues mod p^2 for primes up to pmax_incl.
inline int limb_width(uint64_t pmax_incl) {
    if (pmax_incl < (1ull << 31)) return 2;
    if (pmax_incl < (1ull << 47)) return 3;
    return 4;
}

#define CK(x)                                                        \
    do {                                                             \
        cudaError_t e_ = (x);                                        \
        if (e_ != cudaSuccess) {                                     \
            fprintf(stderr, "wilson: CUDA error %s at %s:%d\n",      \
                    cudaGetErrorString(e_), __FILE__, __LINE__);     \
            return WL_ERR_CUDA;                                      \
        }                                                            \
    } while (0)

#define RC(x)                      \
    do {                           \
        int r_ = (x);              \
        if (r_) return r_;         \
    } while (0)

// Workspace of the tensor-core column products (wl_tensor_host.cu).
struct TensorBufs {
    cudaMemPool_t pool = nullptr;   // serving: grow from this pool, in the order of `st` (ensure_step's reason)
    cudaStream_t st = nullptr;
    DevBuf block;          // one allocation that holds all of them while they are small
    DevBuf desc, counts, cursor, lab_seg, runs, segs, tables, list, w, consts, ones, part, seg, win;
};

constexpr uint64_t WAIT_NS = 4000000000ull;

struct wl_ctx {
    int device = 0;
    int sms = 148;
    int cell_variant = 1;   // formulation of the sweep's cell step (see wl_kernels.cu cellv)
    wl_tuning tune = {};     // sweep kernel choices per limb width (wl_autotune)
    cudaStream_t st = nullptr;
    cudaStream_t st2 = nullptr;   // dense sweep, overlapped with the sparse sweep
    cudaEvent_t ev[8] = {};
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaEvent_t big0 = nullptr, big1 = nullptr;
    cudaEvent_t rows_ready = nullptr;   // row tables uploaded and k_setup_rows done (main stream)
    double ms_big = 0;
    DevBuf base;            // odd primes < 65536 (sieving primes of the column sieve)
    uint32_t nbase = 0;
    std::vector<uint32_t> small;   // the same on the host
    DevBuf cols;            // column cache: all primes < col_limit, ascending, u32
    uint64_t ncols = 0, col_limit = 0;
    DevBuf gprod, gk;       // exact products of its aligned groups of COL_GROUP columns
    uint64_t ngroups = 0;   // 0 until a prefix-fold sweep asks for them (col_groups)
    DevBuf bitmap, segcount, offsets;
    DevBuf tp, keys, counts, buckets, rowinfo, rowmod, items, part, ipart, defs, rowout, dsplit;
    // columns above 2^32
    cudaStream_t st3 = nullptr;
    DevBuf bbitmap, bsegcount, boffsets, boffs, wcols, wbuckets, witems, wpart, wdefs, bacc, bdef, wkeys, wcounts;
    DevBuf uacc, udef;   // columns below 2^32: per-row product of all splits, per-bucket deficit
    DevBuf prod;         // wl_rows_product: moduli, partial products, products
    DevBuf windesc, seglo;   // test-prime windows of all ranges, their segment starts
    uint32_t launches = 0;
    uint64_t h2d = 0, d2h = 0;
    double ms_sieve = 0;
    uint64_t sieve_ints = 0, sieve_bytes = 0;
    uint64_t tensor_macs = 0;   // of the current call
    std::atomic<uint64_t> wait_ns{ WAIT_NS };   // limit of a wait inside the tensor-core products' kernels
    DevBuf work;         // dense sweep work counters: column cells, window cells, products; then the
                         // tensor-core product's error word
    TensorBufs tb;
    bool tensor = true;  // false: every bucket and tail takes the sweeps (WL_TENSOR=0 in the environment when
                         // the context is opened; while the sweeps' kernels are timed for tuning)
};

// Every prime below `limit` (<= 2^32) in the context's resident column table.
// After an error there may be no table (col_limit = 0).
int ensure_columns(wl_ctx* c, uint64_t limit);
// The column groups of the resident table for the prefix-fold sweep, built on
// the main stream when first asked for after the table was; none (every column
// one cell) when there is no memory for them or with WL_COL_GROUPS=0 in the
// environment, for comparisons.
wl::ColGroups col_groups(wl_ctx* c);

// A range's window of test primes and its classes.
struct RangeState {
    uint64_t pmin, pmax, lo0;
    uint32_t nseg;
    uint64_t word_off, seg_off;
    uint64_t tp_off = 0, ntp = 0;
    uint64_t T[3] = { 0, 0, 0 };
    uint64_t per_class[3] = { 0, 0, 0 };
};

// Test primes of each range, ascending (deterministic Miller-Rabin on the
// device); with allow_empty a range without primes is not an error.
int gen_test_primes(wl_ctx* c, const wl_range* ranges, size_t nr, std::vector<RangeState>& rs,
                    std::vector<uint64_t>& tps, bool allow_empty = false);
// Frees the tensor-core products' workspace.
void tensor_release(wl_ctx* c);
// Workspace the tensor-core products may take for about `entries` list entries
// and `rows` rows; 0: too little memory, the sweeps run instead.
size_t tensor_budget(wl_ctx* c, double entries, double rows);
// Modelled times (ms) of the tensor-core product and of the sweeps for a bucket
// of nrows rows over nsparse + ndense columns from index c0 on; returns its list
// entries.
double tensor_times(uint32_t nrows, int L, uint64_t T, uint64_t c0, uint64_t nsparse, uint64_t ndense, double* tensor,
                    double* sweeps);
// Multiplies each task's columns into its rows' accumulators, on the main
// stream (it waits once for the stream).  done: the first column of each task that
// is not multiplied in, which after WL_ERR_NOMEM may lie anywhere in the task.
int tensor_products(wl_ctx* c, std::vector<wl::TensorTask> tasks, const wl::TensorTarget& to, size_t budget,
                    std::vector<uint64_t>* done = nullptr);
// Multiplies the rows' consecutive-integer tails T+1 .. Tp into their
// accumulators, on the main stream; c->rowinfo holds the rows ri.
int tensor_tails(wl_ctx* c, const std::vector<wl::TensorTail>& tails, const std::vector<wl::RowInfo>& ri,
                 const wl::TensorTarget& to);
// results.txt value of one row (cl_wilson.cpp:872-898): 1 if it is a result line.
int result_of(const wl_row& r, int32_t* value);
