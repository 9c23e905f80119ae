// wl_tensor_host.cu -- plans the tensor-core column products (wl_tensor.cu):
// cuts the buckets into tasks that fit the workspace, reads back what each takes
// (the digits are counted and laid out in lane runs on the device) and launches
// the kernels.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "wilson.h"
#include "wl_host.h"
#include "wl_internal.h"
#include "wl_tensor.h"

using namespace wl;

namespace {

int bit_length(uint64_t v) {
    int b = 0;
    while (v) { v >>= 1; ++b; }
    return b;
}

// p_n (the column of index n - 1) lies between n ln n and n (ln n + ln ln n) for n >= 6.
uint64_t column_at_least(uint64_t idx) {
    const double n = (double)idx + 1;
    return idx < 6 ? 2 : (uint64_t)(n * std::log(n));
}
uint64_t column_at_most(uint64_t idx) {
    const double n = (double)idx + 1;
    return idx < 6 ? 13 : (uint64_t)(n * (std::log(n) + std::log(std::log(n)))) + 1;
}

// Digit width by the number of columns.  A wide digit means fewer list entries
// per column (one per nonzero digit of the exponent) but more labels, each of
// which pads its last run by about 2.5 groups of 140 columns.  With exponents of
// 30 to 40 bits (the dense regime) w = 9 saves half an entry per column over
// w = 8 and costs 4 x 256 labels, which 600,000 columns repay; where most
// exponents are below 256 (full searches) more than 8 bits save nothing.
uint32_t digit_width(uint64_t ncols, uint64_t T, uint64_t q_mid) {
    if (ncols >= 600000) return T / q_mid > 65535 ? 9 : 8;
    return ncols >= 280000 ? 8 : ncols >= 100000 ? 7 : ncols >= 30000 ? 6 : 5;
}

uint64_t middle_column(const TensorTask& t) { return std::max<uint64_t>(2, column_at_least(t.c0 + (t.c1 - t.c0) / 2)); }

double entries_per_column(const TensorTask& t, uint32_t w) {
    return std::max(1.0, std::ceil((double)bit_length(t.T / middle_column(t)) / w));
}

// Digit width and windows of a task: v_q(T!) <= T / (q - 1) <= T / (q0 - 1).
void task_digits(const TensorTask& t, uint32_t* w, uint32_t* nwin) {
    const uint64_t q0 = column_at_least(t.c0);
    const int bits = std::max(1, bit_length(t.T / (q0 > 2 ? q0 - 1 : 1)));
    *w = digit_width(t.c1 - t.c0, t.T, middle_column(t));
    *nwin = (uint32_t)(bits + (int)*w - 1) / *w;
    while (((uint64_t)*nwin << *w) > TN_LABELS) {
        --*w;
        *nwin = (uint32_t)(bits + (int)*w - 1) / *w;
    }
}

uint32_t row_tiles_of(uint32_t nrows, int L) { return (nrows + tn_rows(L) - 1) / tn_rows(L); }

// A buffer that must grow grows by half, so that calls and steps of slowly rising
// size do not free and allocate each time.
int grow(TensorBufs& tb, DevBuf& b, size_t bytes) {
    if (bytes <= b.cap && b.p) return 0;
    const size_t want = std::max(bytes, b.cap + b.cap / 2);
    if (!tb.pool) return ensure(b, want) ? ensure(b, bytes) : 0;
    if (b.p && !b.inner) cudaFreeAsync(b.p, tb.st);
    b = DevBuf();
    for (size_t n : { want, bytes }) {
        if (cudaMallocFromPoolAsync(&b.p, n, tb.pool, tb.st) == cudaSuccess) {
            b.cap = n;
            return 0;
        }
        cudaGetLastError();
        b.p = nullptr;
    }
    return WL_ERR_NOMEM;
}

// The workspace of a small call in one allocation: a dozen of them would be most
// of a small search's first call (each some 0.1 ms).
int first_block(TensorBufs& tb) {
    if (tb.block.p) return 0;
    struct Part { DevBuf* b; size_t bytes; };
    const Part parts[] = { { &tb.w, 4u << 20 },       { &tb.consts, 2u << 20 },   { &tb.list, 1u << 20 },
                           { &tb.part, 1u << 20 },    { &tb.seg, 256u << 10 },    { &tb.win, 256u << 10 },
                           { &tb.runs, 128u << 10 },  { &tb.counts, 64u << 10 },  { &tb.cursor, 64u << 10 },
                           { &tb.lab_seg, 64u << 10 }, { &tb.segs, 64u << 10 },   { &tb.tables, 64u << 10 },
                           { &tb.ones, 64u << 10 },   { &tb.desc, 16u << 10 } };
    size_t total = 0;
    for (const Part& p : parts) total += p.bytes;
    RC(ensure(tb.block, total));
    uint8_t* at = as<uint8_t>(tb.block);
    for (const Part& p : parts) {
        if (!p.b->p) {
            p.b->p = at;
            p.b->cap = p.bytes;
            p.b->inner = true;
        }
        at += p.bytes;
    }
    return 0;
}

// Shares of the workspace: list entries (4 bytes each), group tiles (64 KB each;
// where tasks are many and small, most of them padding), and the bytes of the
// lane-run products and of the row constants.  Buckets are cut into pieces and
// rows into slabs so that a task keeps within them, and a chunk takes as many
// tasks as keep within them together: with the folded products, which are never
// more than the lane runs', a chunk holds about 1.2 GB at most.  Buffers that grew by
// half may be half as large again.
struct Limits {
    double entries, tiles, part, consts;
};
constexpr uint32_t WAVE_TASKS = 1024;      // tasks counted in one launch

// Tables of one chunk, uploaded together.
struct Tables {
    std::vector<uint8_t> bytes;
    template <class T> size_t add(const std::vector<T>& v) {
        const size_t at = (bytes.size() + 255) & ~size_t(255);
        bytes.resize(at + v.size() * sizeof(T) + 16);
        if (!v.empty()) memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
};

class Products {
public:
    Products(wl_ctx* c, const TensorTarget& to, size_t budget) : c(c), tb(c->tb), to(to) {
        lim.entries = std::min<double>((double)budget / 2 / 9.0, (double)(1u << 25));
        lim.tiles = std::min<double>((double)budget * 3 / 8, 402e6) / (double)(TN_M * TN_K);
        lim.part = std::min<double>((double)budget / 4, 256e6);
        lim.consts = std::min<double>((double)budget / 4, 128e6);
    }
    std::vector<uint64_t>* done = nullptr;   // see tensor_products
    void add(const TensorTask& whole);
    int run();

private:
    wl_ctx* c;
    TensorBufs& tb;
    TensorTarget to;
    Limits lim;
    std::vector<TensorTask> tasks;
    // the current wave
    std::vector<TensorDesc> desc;
    std::vector<TensorSize> size;

    int wave(size_t t0, size_t t1);
    int chunk(const TensorTask* t, size_t i0, size_t i1);
    uint32_t slab_rows(const TensorTask& t, const TensorSize& z) const;
};

uint32_t tiles_of_runs(uint32_t runs, uint32_t tn) { return (runs + TN_M - 1) / TN_M * tn; }
uint32_t group_tiles(const TensorSize& z) { return tiles_of_runs(z.longs, TN_LONG) + tiles_of_runs(z.shorts, TN_SHORT); }

void Products::add(const TensorTask& whole) {
    if (whole.c1 <= whole.c0 || !whole.nrows) return;
    // pieces of columns whose list and group products fit
    uint64_t step = whole.c1 - whole.c0;
    for (int it = 0; it < 40 && step > 65536; ++it) {
        TensorTask t = whole;
        t.c0 = std::max(whole.c0, whole.c1 - step);
        if ((double)step * entries_per_column(t, digit_width(step, t.T, middle_column(t))) <= lim.entries) break;
        step = (step + 1) / 2;
    }
    for (uint64_t a = whole.c0; a < whole.c1; a += step) {
        TensorTask t = whole;
        t.c0 = a;
        t.c1 = std::min(whole.c1, a + step);
        t.q_max = (uint32_t)std::min<uint64_t>(whole.q_max, column_at_most(t.c1 - 1));
        tasks.push_back(t);
    }
}

int Products::run() {
    for (size_t t0 = 0; t0 < tasks.size(); t0 += WAVE_TASKS) RC(wave(t0, std::min(tasks.size(), t0 + WAVE_TASKS)));
    return 0;
}

// Rows of a task that go together: its lane-run products and row constants within their shares.
uint32_t Products::slab_rows(const TensorTask& t, const TensorSize& z) const {
    const uint32_t rt = tn_rows(t.L);
    const double esz = t.L == 2 ? 8 : 16;
    const double tiles = std::min(lim.part / ((double)std::max<uint32_t>(z.slots, 1) * rt * esz),
                                  lim.consts / (double)(TN_N * TN_K));
    return std::max<uint32_t>(1, (uint32_t)std::min(tiles, 1e6)) * rt;
}

// Counts the digits of tasks [t0, t1) (one launch, one wait for their sizes), then runs them in chunks.
int Products::wave(size_t t0, size_t t1) {
    cudaStream_t st = c->st;
    RC(first_block(tb));
    const uint32_t nt = (uint32_t)(t1 - t0);
    desc.assign(nt, TensorDesc());
    size.assign(nt, TensorSize());
    uint32_t nlab = 0, nblk = 0;
    for (uint32_t i = 0; i < nt; ++i) {
        const TensorTask& t = tasks[t0 + i];
        TensorDesc& d = desc[i];
        memset(&d, 0, sizeof(d));
        d.T = t.T;
        d.c0 = (uint32_t)t.c0;
        d.c1 = (uint32_t)t.c1;
        d.q_max = t.q_max;
        task_digits(t, &d.w, &d.nwin);
        d.lab0 = nlab;
        d.lab_seg0 = nlab + i;
        nlab += d.nwin << d.w;
        d.blk0 = nblk;
        nblk += (d.c1 - d.c0 + TN_COLS_PER_BLOCK - 1) / TN_COLS_PER_BLOCK;
    }
    const size_t size_at = ((size_t)nt * sizeof(TensorDesc) + 255) & ~size_t(255);
    RC(grow(tb, tb.desc, size_at + nt * sizeof(TensorSize)));
    RC(grow(tb, tb.counts, (size_t)nlab * 4 + 16));
    RC(grow(tb, tb.cursor, (size_t)nlab * 4 + 16));
    RC(grow(tb, tb.lab_seg, (size_t)(nlab + nt) * 4 + 16));
    TensorSize* dsize = (TensorSize*)(as<uint8_t>(tb.desc) + size_at);
    CK(cudaMemcpyAsync(tb.desc.p, desc.data(), nt * sizeof(TensorDesc), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(tb.counts.p, 0, (size_t)nlab * 4, st));
    launch_tensor_count(as<TensorDesc>(tb.desc), nt, nblk, as<uint32_t>(c->cols), as<uint32_t>(tb.counts), st);
    launch_tensor_size(as<TensorDesc>(tb.desc), nt, as<uint32_t>(tb.counts), dsize, st);
    CK(cudaMemcpyAsync(size.data(), dsize, nt * sizeof(TensorSize), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    CK(cudaGetLastError());
    c->launches += 2;
    c->h2d += nt * sizeof(TensorDesc);
    c->d2h += nt * sizeof(TensorSize);
    // chunks of consecutive tasks of one limb width, and the largest sizes they need
    std::vector<std::pair<size_t, size_t>> chunks;
    uint64_t list = 0, w = 0, part = 0, consts = 0, runs = 0, segs = 0;
    for (size_t i = 0; i < nt;) {
        size_t j = i;
        double e = 0, p = 0, k = 0;
        uint64_t mt = 0, nr = 0, ns = 0;
        for (; j < nt && tasks[t0 + j].L == tasks[t0 + i].L; ++j) {
            const TensorTask& t = tasks[t0 + j];
            const TensorSize& z = size[j];
            // two pieces of one bucket multiply into the same rows: never in one chunk
            // (pieces are neighbours; their entries may fall short of what cut them)
            if (j > i && t.row_begin == tasks[t0 + j - 1].row_begin) break;
            const uint32_t rows = std::min(t.nrows, slab_rows(t, z)), tiles = row_tiles_of(rows, t.L);
            const double pe = (double)z.slots * tiles * tn_rows(t.L) * (t.L == 2 ? 8 : 16);
            const double ke = (double)tiles * TN_N * TN_K;
            const bool whole = rows >= t.nrows;     // a task in several slabs goes alone
            if (j > i && (!whole || e + (double)z.entries > lim.entries || (double)(mt + group_tiles(z)) > lim.tiles ||
                          p + pe > lim.part || k + ke > lim.consts))
                break;
            e += (double)z.entries;
            p += pe;
            k += ke;
            mt += group_tiles(z);
            nr += z.longs + z.shorts + 2 * TN_M;
            ns += z.segs;
            if (!whole) { ++j; break; }
        }
        chunks.push_back({ i, j });
        list = std::max(list, (uint64_t)e);
        w = std::max(w, mt * TN_M * TN_K);
        part = std::max(part, (uint64_t)p);
        consts = std::max(consts, (uint64_t)k);
        runs = std::max(runs, nr);
        segs = std::max(segs, ns);
        i = j;
    }
    RC(grow(tb, tb.list, list * 4 + 16));
    RC(grow(tb, tb.w, w + 16));
    RC(grow(tb, tb.part, part + 16));
    RC(grow(tb, tb.consts, consts + 16));
    RC(grow(tb, tb.runs, runs * sizeof(LaneRun) + 16));
    RC(grow(tb, tb.segs, segs * sizeof(FoldSeg) + 16));
    for (auto& x : chunks) RC(chunk(tasks.data() + t0, x.first, x.second));
    return 0;
}

// Tasks [i0, i1) of the wave: their lists and group products once, then per
// slab of rows the constants, the matrix product and the label folds.  The first
// slab is the largest, so that an allocation fails before any row is multiplied.
int Products::chunk(const TensorTask* ts, size_t i0, size_t i1) {
    cudaStream_t st = c->st;
    const int L = ts[i0].L;
    const uint32_t rt = tn_rows(L), nt = (uint32_t)(i1 - i0);
    const size_t esz = L == 2 ? 8 : 16;
    std::vector<TensorDesc> dc(desc.begin() + i0, desc.begin() + i1);
    std::vector<TensorSec> secs;
    uint32_t nmt = 0, nblk = 0, max_blocks = 0, list = 0, nrun = 0, nseg = 0;
    for (uint32_t i = 0; i < nt; ++i) {
        TensorDesc& d = dc[i];
        const TensorSize& z = size[i0 + i];
        max_blocks = std::max(max_blocks, (d.nwin << d.w) / TN_DIGITS);
        d.blk0 = nblk;
        nblk += (d.c1 - d.c0 + TN_COLS_PER_BLOCK - 1) / TN_COLS_PER_BLOCK;
        d.list0 = list;
        list += z.entries;
        d.seg0 = nseg;
        d.nseg = z.segs;
        nseg += z.segs;
        d.nlong = (z.longs + TN_M - 1) / TN_M * TN_M;
        d.nshort = (z.shorts + TN_M - 1) / TN_M * TN_M;
        d.long0 = nrun;
        d.short0 = nrun + d.nlong;
        nrun += d.nlong + d.nshort;
        if (d.nlong) secs.push_back({ i, TN_LONG, nmt, d.long0, 1, 0 });
        nmt += d.nlong / TN_M * TN_LONG;
        if (d.nshort) secs.push_back({ i, TN_SHORT, nmt, d.short0, 0, 0 });
        nmt += d.nshort / TN_M * TN_SHORT;
    }
    if (!nmt) return 0;
    const uint32_t slab = nt > 1 ? 0xFFFFFFFFu : slab_rows(ts[i0], size[i0]);
    bool first = true;
    for (uint64_t r0 = 0; first || r0 < ts[i0].nrows; r0 += slab) {
        uint32_t ntile = 0, row_blk = 0, fold_blk = 0;
        uint64_t part = 0, seg = 0, win = 0, units = 0;
        for (uint32_t i = 0; i < nt; ++i) {
            TensorDesc& d = dc[i];
            const TensorTask& t = ts[i0 + i];
            d.row_begin = t.row_begin + (uint32_t)r0;
            d.nrows = (uint32_t)std::min<uint64_t>(slab, t.nrows - r0);
            const uint32_t tiles = row_tiles_of(d.nrows, L);
            d.rows_pad = tiles * rt;
            d.ct0 = ntile;
            ntile += tiles;
            d.row_blk0 = row_blk;
            row_blk += (d.nrows + 127) / 128;
            d.fold_blk0 = fold_blk;
            fold_blk += d.nseg * ((d.rows_pad + 127) / 128);
            d.part0 = part;
            part += (uint64_t)size[i0 + i].slots * d.rows_pad;
            d.seg_part0 = seg;
            seg += (uint64_t)d.nseg * d.rows_pad;
            d.win0 = win;
            win += (uint64_t)((d.nwin << d.w) / TN_DIGITS) * d.rows_pad;
            units += (uint64_t)group_tiles(size[i0 + i]) * tiles;
        }
        c->tensor_macs += units * TN_M * TN_N * TN_K;
        // items of 32 to 256 group tiles, about eight per SM where the work allows:
        // shorter ones would show the 128 KB of constants that each brings in
        const uint64_t per_item = std::min<uint64_t>(256, std::max<uint64_t>(32, units / ((uint64_t)c->sms * 8)));
        std::vector<TensorItem> items;
        for (uint32_t s = 0; s < secs.size(); ++s) {
            const TensorSec& x = secs[s];
            const TensorDesc& d = dc[x.task];
            const uint32_t tiles = d.rows_pad / rt, ncb = (x.tn == TN_LONG ? d.nlong : d.nshort) / TN_M;
            const uint32_t step = (uint32_t)std::max<uint64_t>(1, per_item / x.tn);
            // row tiles inside: CTAs that run together read the same group tiles from L2
            for (uint32_t cb = 0; cb < ncb; cb += step)
                for (uint32_t r = 0; r < tiles; ++r) items.push_back({ s, r, cb, std::min(step, ncb - cb) });
        }
        Tables tab;
        const size_t o_desc = tab.add(dc), o_sec = tab.add(secs), o_item = tab.add(items);
        RC(grow(tb, tb.ones, (size_t)ntile * rt * 16 + 16));
        RC(grow(tb, tb.tables, tab.bytes.size()));
        RC(grow(tb, tb.seg, seg * esz + 16));
        RC(grow(tb, tb.win, win * esz + 16));
        RC(grow(tb, tb.part, part * esz + 16));
        CK(cudaMemcpyAsync(tb.tables.p, tab.bytes.data(), tab.bytes.size(), cudaMemcpyHostToDevice, st));
        c->h2d += tab.bytes.size();
        uint8_t* base = as<uint8_t>(tb.tables);
        const TensorDesc* dd = (const TensorDesc*)(base + o_desc);
        const TensorSec* ds = (const TensorSec*)(base + o_sec);
        const LaneRun* dr = as<LaneRun>(tb.runs);
        const RowMod* mods = to.mods;
        if (first) {
            launch_tensor_layout(dd, nt, as<uint32_t>(tb.counts), as<uint32_t>(tb.cursor), as<LaneRun>(tb.runs),
                                 as<FoldSeg>(tb.segs), as<uint32_t>(tb.lab_seg), st);
            launch_tensor_scatter(dd, nt, nblk, as<uint32_t>(c->cols), as<uint32_t>(tb.cursor), as<uint32_t>(tb.list), st);
            launch_tensor_build(ds, (uint32_t)secs.size(), nmt, dr, as<uint32_t>(tb.list), as<uint8_t>(tb.w), st);
            c->launches += 3;
        }
        launch_tensor_consts(L, dd, nt, ntile, mods, as<uint8_t>(tb.consts), as<uint4>(tb.ones), st);
        if (launch_tensor_gemm(L, (uint32_t)items.size(), dd, ds, (const TensorItem*)(base + o_item), dr, mods,
                               as<uint8_t>(tb.w), as<uint8_t>(tb.consts), as<uint4>(tb.ones), tb.part.p,
                               to.err, c->wait_ns, st))
            return WL_ERR_CUDA;
        launch_tensor_fold(L, dd, nt, fold_blk, as<FoldSeg>(tb.segs), mods, tb.part.p, tb.seg.p, st);
        launch_tensor_combine(L, dd, nt, row_blk, max_blocks, as<uint32_t>(tb.lab_seg), mods, as<uint4>(tb.ones),
                              tb.seg.p, tb.win.p, to.acc, st);
        CK(cudaGetLastError());
        c->launches += 5;
        first = false;
        if (nt > 1) break;
    }
    if (done)
        for (size_t i = i0; i < i1; ++i) (*done)[ts[i].id] = ts[i].c1;
    return 0;
}

}  // namespace

void tensor_release(wl_ctx* c) {
    TensorBufs& tb = c->tb;
    DevBuf* all[] = { &tb.w, &tb.consts, &tb.list, &tb.part, &tb.seg, &tb.win, &tb.runs, &tb.counts, &tb.cursor,
                      &tb.lab_seg, &tb.segs, &tb.tables, &tb.ones, &tb.desc };
    for (DevBuf* b : all) {
        if (b->p && !b->inner && tb.pool) {
            cudaFreeAsync(b->p, tb.st);
            *b = DevBuf();
        } else {
            release(*b);
        }
    }
    release(tb.block);
}

// The least free memory the tensor-core path takes on, and the most workspace it plans for.
static constexpr size_t TENSOR_MIN_BUDGET = 1ull << 30, TENSOR_MAX_BUDGET = 2ull << 30;

size_t tensor_budget(wl_ctx* c, double entries, double rows) {
    // lists, group products, constants and products of a small call, several
    // times over: the query of the free memory would cost it a sixth of its time
    if (16.0 * entries + 16384.0 * rows <= 192e6) return TENSOR_MIN_BUDGET;
    const TensorBufs& b = c->tb;
    const size_t held = b.list.cap + b.w.cap + b.consts.cap + b.part.cap + b.seg.cap + b.win.cap;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { cudaGetLastError(); free_b = 8ull << 30; }
    const size_t budget = std::min(TENSOR_MAX_BUDGET, (free_b + held) / 2);
    return budget < TENSOR_MIN_BUDGET ? 0 : budget;
}

// Times in picoseconds, measured on B200.  A list entry costs the digit sort and
// its share of a group product, and each 256-column tile of rows its share of
// the matrix product; the sweeps cost a cell per row and column, in the dense
// regime about eight, and more where a bucket has few rows (several splits to a
// CTA, short chunks: 2.6 ps a cell at 5 to 10 rows of 3 limbs).
//   entry: 36 (3.1 ms for 8.7e7 entries at 4 limbs); per row tile: 0.8 (17.0 ms
//   for 2.2e10 at 2 limbs)
//   cell: 0.68 / 1.0 / 1.35; dense column: 8 / 11 / 14.6 (L = 2 / 3 / 4)
double tensor_times(uint32_t nrows, int L, uint64_t T, uint64_t c0, uint64_t nsparse, uint64_t ndense, double* tensor,
                    double* sweeps) {
    static const double cell[3] = { 0.68, 1.0, 1.35 }, dense[3] = { 8.0, 11.0, 14.6 };
    const uint64_t ncols = nsparse + ndense;
    *tensor = *sweeps = 0;
    if (!ncols || !nrows) return 0;
    TensorTask t = {};
    t.T = T;
    t.c0 = c0;
    t.c1 = c0 + ncols;
    uint32_t w, nwin;
    task_digits(t, &w, &nwin);
    const double entries = (double)ncols * entries_per_column(t, w) + 150.0 * (double)(1u << w);
    *tensor = entries * (36.0 + 0.8 * row_tiles_of(nrows, L)) * 1e-9;
    *sweeps = ((double)nrows + 16.0) * (cell[L - 2] * (double)nsparse + dense[L - 2] * (double)ndense) * 1e-9;
    return entries;
}

int tensor_products(wl_ctx* c, std::vector<TensorTask> tasks, const TensorTarget& to, size_t budget,
                    std::vector<uint64_t>* done) {
    if (done) done->resize(tasks.size());
    for (uint32_t i = 0; i < tasks.size(); ++i) {
        tasks[i].id = i;
        if (done) (*done)[i] = tasks[i].c0;
    }
    std::stable_sort(tasks.begin(), tasks.end(), [](const TensorTask& a, const TensorTask& b) { return a.L < b.L; });
    Products p(c, to, budget);
    p.done = done;
    for (const TensorTask& t : tasks) p.add(t);
    return p.run();
}

// The tails of buckets, a slab of rows at a time: TAIL_TILES row tiles (128 MB of
// constants) with the groups that the slab's last row needs.  Rows are in ascending
// p, so ascending Tp, and a row tile needs whole group tiles only up to its last
// row's end.  One launch takes slabs of one limb width, of several tails where they
// are small, that keep within TAIL_TILES and 128 MB of groups together.
int tensor_tails(wl_ctx* c, const std::vector<TensorTail>& tails, const std::vector<RowInfo>& ri, const TensorTarget& to) {
    constexpr uint32_t TAIL_TILES = 1024, TAIL_GROUP_TILES = 2048;
    cudaStream_t st = c->st;
    TensorBufs& tb = c->tb;
    RC(first_block(tb));
    std::vector<TensorTail> slabs;
    for (const TensorTail& t : tails) {
        const uint32_t step = TAIL_TILES * tn_rows((int)t.L);
        for (uint32_t r0 = 0; r0 < t.nrows; r0 += step)
            slabs.push_back({ t.T, t.row_begin + r0, std::min(step, t.nrows - r0), t.L });
    }
    for (size_t i0 = 0; i0 < slabs.size();) {
        const int L = (int)slabs[i0].L;
        const uint32_t rt = tn_rows(L);
        std::vector<TensorDesc> dc;
        std::vector<TensorSec> secs;
        std::vector<TensorItem> items;
        uint32_t ntile = 0, nmt = 0, row_blk = 0;
        uint64_t part = 0;
        size_t i1 = i0;
        for (; i1 < slabs.size() && (int)slabs[i1].L == L; ++i1) {
            const TensorTail& t = slabs[i1];
            const uint64_t last = ri[t.row_begin + t.nrows - 1].Tp;
            const double k = 511.99 / std::log2((double)last + 2.0);
            const uint32_t g = 8 * (uint32_t)std::min<double>(k, (double)TN_GMAX / 8), tiles = row_tiles_of(t.nrows, L);
            const uint64_t mts = ((last - t.T) / g + TN_M - 1) / TN_M;
            if (i1 > i0 && (ntile + tiles > TAIL_TILES || nmt + mts > TAIL_GROUP_TILES)) break;
            TensorDesc d;
            memset(&d, 0, sizeof(d));
            d.T = t.T;
            d.row_begin = t.row_begin;
            d.nrows = t.nrows;
            d.rows_pad = tiles * rt;
            d.ct0 = ntile;
            d.row_blk0 = row_blk;
            d.part0 = part;
            const uint32_t s = (uint32_t)secs.size();
            secs.push_back({ s, 0, nmt, 0, 1, g });
            for (uint32_t r = 0; r < tiles; ++r) {
                const uint32_t lr = std::min(t.nrows, (r + 1) * rt) - 1;
                const uint64_t need = (ri[t.row_begin + lr].Tp - t.T) / g;
                if (need) items.push_back({ s, r, 0, (uint32_t)((need + TN_M - 1) / TN_M) });
            }
            dc.push_back(d);
            ntile += tiles;
            nmt += (uint32_t)mts;
            row_blk += (t.nrows + 127) / 128;
            part += (uint64_t)TAIL_SLOTS * d.rows_pad;
        }
        // the longest tails first
        std::stable_sort(items.begin(), items.end(),
                         [](const TensorItem& a, const TensorItem& b) { return a.ncb > b.ncb; });
        Tables tab;
        const size_t o_desc = tab.add(dc), o_sec = tab.add(secs), o_item = tab.add(items);
        RC(grow(tb, tb.tables, tab.bytes.size()));
        RC(grow(tb, tb.consts, (size_t)ntile * TN_N * TN_K + 16));
        RC(grow(tb, tb.ones, (size_t)ntile * rt * 16 + 16));
        RC(grow(tb, tb.part, part * (L == 2 ? 8 : 16) + 16));
        RC(grow(tb, tb.w, (size_t)nmt * TN_M * TN_K + 16));
        CK(cudaMemcpyAsync(tb.tables.p, tab.bytes.data(), tab.bytes.size(), cudaMemcpyHostToDevice, st));
        c->h2d += tab.bytes.size();
        uint8_t* base = as<uint8_t>(tb.tables);
        const TensorDesc* dd = (const TensorDesc*)(base + o_desc);
        const TensorSec* ds = (const TensorSec*)(base + o_sec);
        const uint32_t nt = (uint32_t)dc.size();
        launch_tensor_consts(L, dd, nt, ntile, to.mods, as<uint8_t>(tb.consts), as<uint4>(tb.ones), st);
        if (nmt) launch_tensor_tail_build(dd, ds, nt, nmt, as<uint8_t>(tb.w), st);
        if (!items.empty() &&
            launch_tensor_tail_gemm(L, (uint32_t)items.size(), dd, ds, (const TensorItem*)(base + o_item),
                                    as<RowInfo>(c->rowinfo), to.mods, as<uint8_t>(tb.w), as<uint8_t>(tb.consts),
                                    as<uint4>(tb.ones), tb.part.p, to.err, c->wait_ns, st))
            return WL_ERR_CUDA;
        launch_tensor_tail_rows(L, dd, ds, nt, row_blk, as<RowInfo>(c->rowinfo), to.mods, as<uint4>(tb.ones), tb.part.p,
                                to.acc, st);
        CK(cudaGetLastError());
        c->launches += 4;
        for (const TensorItem& it : items) c->tensor_macs += (uint64_t)it.ncb * TN_M * TN_N * TN_K;
        i0 = i1;
    }
    return 0;
}
