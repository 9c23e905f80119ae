// wl_tensor_host.cu -- plans the tensor-core column products (wl_tensor.cu):
// cuts the buckets into tasks that fit the workspace, reads the digit counts
// back, lays the labels out in lane runs and launches the kernels.
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

// Groups per lane run: a label's groups go in runs of 32, the rest in runs of
// 4, so that a label wastes about two groups however many it has.
constexpr uint32_t TN_LONG = 32, TN_SHORT = 4;

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

// Columns of a group of which none is above q: an eighth of them stays below 2^512
// (k_tensor_build), so the group below 2^4096.
uint32_t group_columns(uint64_t q) {
    const double k = 511.99 / std::log2((double)std::max<uint64_t>(q, 2) + 1.0);
    return 8 * (uint32_t)std::min<double>(k, (double)TN_GMAX / 8);
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

// What a task takes, from its digit counts.
struct TaskSize {
    uint64_t entries = 0, mt_long = 0, mt_short = 0, slots = 0;
};

// Shares of the workspace: group lists and products together, lane-run
// products, row constants.  Tasks are cut so that a chunk keeps within them.
struct Limits {
    double entries, part, consts;
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
    Products(wl_ctx* c, size_t budget) : c(c), tb(c->tb) {
        lim.entries = std::min<double>((double)budget / 2 / 9.0, (double)(1u << 25));
        lim.part = std::min<double>((double)budget / 4, 256e6);
        lim.consts = std::min<double>((double)budget / 4, 128e6);
    }
    void add(const TensorTask& whole);
    int run();

private:
    wl_ctx* c;
    TensorBufs& tb;
    Limits lim;
    std::vector<TensorTask> tasks;
    // the current wave
    std::vector<TensorDesc> desc;
    std::vector<uint32_t> cnt;
    std::vector<TaskSize> size;

    int wave(size_t t0, size_t t1);
    TaskSize measure(const TensorTask& t, const TensorDesc& d) const;
    int chunk(const TensorTask* t, size_t i0, size_t i1);
    uint32_t slab_rows(const TensorTask& t, const TaskSize& z) const;
};

// Columns of label l of task t have v_q(T!) >= d 2^(wj), so q <= T / (d 2^(wj)) + 1.
// `all` is group_columns(t.q_max), which most labels have.
uint32_t label_columns(const TensorTask& t, const TensorDesc& d, uint32_t l, uint32_t all) {
    const uint32_t dg = l & ((1u << d.w) - 1), j = l >> d.w;
    const uint64_t q = (t.T >> (d.w * j)) / dg + 1;
    return q >= t.q_max ? all : group_columns(q);
}
// Long and short runs of a label with n list entries in groups of g.
void label_runs(uint32_t n, uint32_t g, uint32_t* longs, uint32_t* shorts) {
    const uint32_t ng = (n + g - 1) / g;
    *longs = ng / TN_LONG;
    *shorts = (ng % TN_LONG + TN_SHORT - 1) / TN_SHORT;
    if (*shorts * TN_SHORT >= TN_LONG) {
        ++*longs;
        *shorts = 0;
    }
}

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

TaskSize Products::measure(const TensorTask& t, const TensorDesc& d) const {
    TaskSize z;
    uint64_t longs = 0, shorts = 0, labels = 0;
    const uint32_t all = group_columns(t.q_max);
    for (uint32_t l = 0; l < (d.nwin << d.w); ++l) {
        const uint32_t n = cnt[d.lab0 + l];
        if (!n) continue;
        uint32_t a, b;
        label_runs(n, label_columns(t, d, l, all), &a, &b);
        z.entries += n;
        longs += a;
        shorts += b;
        labels += a > 0;
    }
    z.mt_long = (longs + TN_M - 1) / TN_M * TN_LONG;
    z.mt_short = (shorts + TN_M - 1) / TN_M * TN_SHORT;
    z.slots = shorts + labels + (longs + 31) / 32;
    return z;
}

// Rows of a task that go together: its lane-run products and row constants within their shares.
uint32_t Products::slab_rows(const TensorTask& t, const TaskSize& z) const {
    const uint32_t rt = tn_rows(t.L);
    const double esz = t.L == 2 ? 8 : 16;
    const double tiles = std::min(lim.part / ((double)std::max<uint64_t>(z.slots, 1) * rt * esz),
                                  lim.consts / (double)(TN_N * TN_K));
    return std::max<uint32_t>(1, (uint32_t)std::min(tiles, 1e6)) * rt;
}

// Counts the digits of tasks [t0, t1) (one launch, one wait), then runs them in chunks.
int Products::wave(size_t t0, size_t t1) {
    cudaStream_t st = c->st;
    const uint32_t nt = (uint32_t)(t1 - t0);
    desc.assign(nt, TensorDesc());
    size.assign(nt, TaskSize());
    uint32_t nlab = 0, nblk = 0;
    for (uint32_t i = 0; i < nt; ++i) {
        const TensorTask& t = tasks[t0 + i];
        TensorDesc& d = desc[i];
        memset(&d, 0, sizeof(d));
        d.T = t.T;
        d.c0 = (uint32_t)t.c0;
        d.c1 = (uint32_t)t.c1;
        task_digits(t, &d.w, &d.nwin);
        d.lab0 = nlab;
        nlab += d.nwin << d.w;
        d.blk0 = nblk;
        nblk += (d.c1 - d.c0 + TN_COLS_PER_BLOCK - 1) / TN_COLS_PER_BLOCK;
    }
    RC(ensure(tb.desc, nt * sizeof(TensorDesc)));
    RC(ensure(tb.counts, (size_t)nlab * 4 + 16));
    CK(cudaMemcpyAsync(tb.desc.p, desc.data(), nt * sizeof(TensorDesc), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(tb.counts.p, 0, (size_t)nlab * 4, st));
    launch_tensor_count(as<TensorDesc>(tb.desc), nt, nblk, as<uint32_t>(c->cols), as<uint32_t>(tb.counts), st);
    cnt.assign(nlab, 0);
    CK(cudaMemcpyAsync(cnt.data(), tb.counts.p, (size_t)nlab * 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    CK(cudaGetLastError());
    c->launches++;
    c->h2d += nt * sizeof(TensorDesc);
    c->d2h += (size_t)nlab * 4;
    // chunks of consecutive tasks of one limb width, and the largest sizes they need
    std::vector<std::pair<size_t, size_t>> chunks;
    uint64_t list = 0, w = 0, part = 0, consts = 0;
    for (size_t i = 0; i < nt;) {
        size_t j = i;
        double e = 0, p = 0, k = 0;
        uint64_t mt = 0;
        for (; j < nt && tasks[t0 + j].L == tasks[t0 + i].L; ++j) {
            const TensorTask& t = tasks[t0 + j];
            const TaskSize z = size[j] = measure(t, desc[j]);
            const uint32_t rows = std::min(t.nrows, slab_rows(t, z)), tiles = row_tiles_of(rows, t.L);
            const double pe = (double)z.slots * tiles * tn_rows(t.L) * (t.L == 2 ? 8 : 16);
            const double ke = (double)tiles * TN_N * TN_K;
            const bool whole = rows >= t.nrows;     // a task in several slabs goes alone
            if (j > i && (!whole || e + (double)z.entries > lim.entries || p + pe > lim.part || k + ke > lim.consts)) break;
            e += (double)z.entries;
            p += pe;
            k += ke;
            mt += z.mt_long + z.mt_short;
            if (!whole) { ++j; break; }
        }
        chunks.push_back({ i, j });
        list = std::max(list, (uint64_t)e);
        w = std::max(w, mt * TN_M * TN_K);
        part = std::max(part, (uint64_t)p);
        consts = std::max(consts, (uint64_t)k);
        i = j;
    }
    RC(ensure(tb.list, list * 4 + 16));
    RC(ensure(tb.w, w + 16));
    RC(ensure(tb.part, part + 16));
    RC(ensure(tb.consts, consts + 16));
    for (auto& x : chunks) RC(chunk(tasks.data() + t0, x.first, x.second));
    return 0;
}

// Tasks [i0, i1) of the wave: their lists and group products once, then per
// slab of rows the constants, the matrix product and the label folds.
int Products::chunk(const TensorTask* ts, size_t i0, size_t i1) {
    cudaStream_t st = c->st;
    const int L = ts[i0].L;
    const uint32_t rt = tn_rows(L), nt = (uint32_t)(i1 - i0);
    const size_t esz = L == 2 ? 8 : 16;
    std::vector<TensorDesc> dc(desc.begin() + i0, desc.begin() + i1);
    std::vector<TensorSec> secs;
    std::vector<LaneRun> runs;
    std::vector<FoldSeg> segs;
    std::vector<uint32_t> lab_seg, cursor;
    uint64_t entries = 0;
    uint32_t nmt = 0, nlab = 0, nblk = 0, max_blocks = 0;
    std::vector<uint32_t> sec_of(2 * nt, 0xFFFFFFFFu), nslot(nt, 0);
    for (uint32_t i = 0; i < nt; ++i) {
        TensorDesc& d = dc[i];
        const TensorTask& t = ts[i0 + i];
        const uint32_t from = d.lab0, labels = d.nwin << d.w;
        const TaskSize& z = size[i0 + i];
        max_blocks = std::max(max_blocks, (d.nwin << d.w) / TN_DIGITS);
        d.lab0 = nlab;
        d.blk0 = nblk;
        d.seg0 = (uint32_t)segs.size();
        nlab += labels;
        nblk += (d.c1 - d.c0 + TN_COLS_PER_BLOCK - 1) / TN_COLS_PER_BLOCK;
        uint32_t slots = 0;
        const uint32_t all = group_columns(t.q_max);
        // the runs of both sections side by side: long ones first
        const uint32_t long0 = (uint32_t)runs.size(), nlong = (uint32_t)(z.mt_long / TN_LONG * TN_M);
        const uint32_t short0 = long0 + nlong, nshort = (uint32_t)(z.mt_short / TN_SHORT * TN_M);
        runs.resize(short0 + nshort, LaneRun{ 0, 0, 1, RUN_NONE });
        uint32_t il = long0, is = short0;
        for (uint32_t l = 0; l < labels; ++l) {
            lab_seg.push_back((uint32_t)segs.size() - d.seg0);
            cursor.push_back((uint32_t)entries);
            const uint32_t n = cnt[from + l];
            if (!n) continue;
            const uint32_t g = label_columns(t, d, l, all);
            uint32_t a, b;
            label_runs(n, g, &a, &b);
            const uint32_t s0 = slots;
            uint64_t at = entries;
            const uint32_t end = (uint32_t)(entries + n);
            for (uint32_t k = 0; k < a; ++k) {
                // one slot per warp that the label's long runs touch
                if (k && (il - long0) % 32 == 0) ++slots;
                runs[il++] = { (uint32_t)std::min<uint64_t>(at, end), end, g, slots };
                at += (uint64_t)g * TN_LONG;
            }
            if (a) ++slots;
            for (uint32_t k = 0; k < b; ++k) {
                runs[is++] = { (uint32_t)std::min<uint64_t>(at, end), end, g, slots++ };
                at += (uint64_t)g * TN_SHORT;
            }
            for (uint32_t k = s0; k < slots; k += TN_SEG) segs.push_back({ k, std::min(TN_SEG, slots - k) });
            entries += n;
        }
        lab_seg.push_back((uint32_t)segs.size() - d.seg0);
        d.nseg = (uint32_t)segs.size() - d.seg0;
        nslot[i] = slots;
        if (nlong) {
            sec_of[2 * i] = (uint32_t)secs.size();
            secs.push_back({ i, TN_LONG, nmt, long0, 1, 0 });
            nmt += (uint32_t)z.mt_long;
        }
        if (nshort) {
            sec_of[2 * i + 1] = (uint32_t)secs.size();
            secs.push_back({ i, TN_SHORT, nmt, short0, 0, 0 });
            nmt += (uint32_t)z.mt_short;
        }
    }
    if (!nmt) return 0;
    const uint32_t slab = std::max<uint32_t>(rt, nt > 1 ? 0xFFFFFFFFu : slab_rows(ts[i0], size[i0]));
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
            part += (uint64_t)nslot[i] * d.rows_pad;
            d.seg_part0 = seg;
            seg += (uint64_t)d.nseg * d.rows_pad;
            d.win0 = win;
            win += (uint64_t)((d.nwin << d.w) / TN_DIGITS) * d.rows_pad;
            units += (size[i0 + i].mt_long + size[i0 + i].mt_short) * tiles;
        }
        // items of 32 to 256 group tiles, about eight per SM where the work allows:
        // shorter ones would show the 128 KB of constants that each brings in
        const uint64_t per_item = std::min<uint64_t>(256, std::max<uint64_t>(32, units / ((uint64_t)c->sms * 8)));
        std::vector<TensorItem> items;
        for (uint32_t i = 0; i < nt; ++i)
            for (uint32_t k = 0; k < 2; ++k) {
                const uint32_t s = sec_of[2 * i + k];
                if (s == 0xFFFFFFFFu) continue;
                const uint32_t tn = secs[s].tn, tiles = dc[i].rows_pad / rt;
                const uint32_t ncb = (uint32_t)((k ? size[i0 + i].mt_short : size[i0 + i].mt_long) / tn);
                const uint32_t step = (uint32_t)std::max<uint64_t>(1, per_item / tn);
                // row tiles inside: CTAs that run together read the same group tiles from L2
                for (uint32_t cb = 0; cb < ncb; cb += step)
                    for (uint32_t r = 0; r < tiles; ++r) items.push_back({ s, r, cb, std::min(step, ncb - cb) });
            }
        Tables tab;
        const size_t o_desc = tab.add(dc), o_item = tab.add(items), o_sec = tab.add(secs), o_run = tab.add(runs),
                     o_seg = tab.add(segs), o_lab = tab.add(lab_seg), o_cur = tab.add(cursor);
        RC(ensure(tb.tables, tab.bytes.size()));
        RC(ensure(tb.seg, seg * esz + 16));
        RC(ensure(tb.win, win * esz + 16));
        RC(ensure(tb.part, part * esz + 16));
        CK(cudaMemcpyAsync(tb.tables.p, tab.bytes.data(), tab.bytes.size(), cudaMemcpyHostToDevice, st));
        c->h2d += tab.bytes.size();
        uint8_t* base = as<uint8_t>(tb.tables);
        const TensorDesc* dd = (const TensorDesc*)(base + o_desc);
        const TensorSec* ds = (const TensorSec*)(base + o_sec);
        const LaneRun* dr = (const LaneRun*)(base + o_run);
        const RowMod* mods = as<RowMod>(c->rowmod);
        if (first) {
            launch_tensor_scatter(dd, nt, nblk, as<uint32_t>(c->cols), (uint32_t*)(base + o_cur), as<uint32_t>(tb.list), st);
            launch_tensor_build(ds, (uint32_t)secs.size(), nmt, dr, as<uint32_t>(tb.list), as<uint8_t>(tb.w), st);
            c->launches += 2;
        }
        launch_tensor_consts(L, dd, nt, ntile, mods, as<uint8_t>(tb.consts), as<uint4>(tb.ones), st);
        if (launch_tensor_gemm(L, (uint32_t)items.size(), dd, ds, (const TensorItem*)(base + o_item), dr, mods,
                               as<uint8_t>(tb.w), as<uint8_t>(tb.consts), as<uint4>(tb.ones), tb.part.p,
                               as<uint32_t>(c->work) + 6, st))
            return WL_ERR_CUDA;
        launch_tensor_fold(L, dd, nt, fold_blk, (const FoldSeg*)(base + o_seg), mods, tb.part.p, tb.seg.p, st);
        launch_tensor_combine(L, dd, nt, row_blk, max_blocks, (const uint32_t*)(base + o_lab), mods, as<uint4>(tb.ones),
                              tb.seg.p, tb.win.p, as<uint4>(c->uacc), st);
        CK(cudaGetLastError());
        c->launches += 5;
        first = false;
        if (nt > 1) break;
    }
    return 0;
}

}  // namespace

// The least free memory the tensor-core path takes on, and the most workspace it plans for.
static constexpr size_t TENSOR_MIN_BUDGET = 1ull << 30, TENSOR_MAX_BUDGET = 2ull << 30;

size_t tensor_budget(wl_ctx* c, size_t free_bytes) {
    const TensorBufs& b = c->tb;
    const size_t held = b.list.cap + b.w.cap + b.consts.cap + b.part.cap + b.seg.cap + b.win.cap;
    const size_t budget = std::min(TENSOR_MAX_BUDGET, (free_bytes + held) / 2);
    return budget < TENSOR_MIN_BUDGET ? 0 : budget;
}

// Times in picoseconds, measured on B200.  A list entry costs the digit sort and
// its share of a group product, and each 256-column tile of rows its share of
// the matrix product; the sweeps cost a cell per row and column, in the dense
// regime about eight.
//   entry: 45 (4.3 ms for 9.6e7 entries at 4 limbs); per row tile: 0.8 (17.0 ms
//   for 2.2e10 at 2 limbs)
//   cell: 0.68 / 1.0 / 1.35; dense column: 8 / 11 / 14.6 (L = 2 / 3 / 4)
double tensor_saves(uint32_t nrows, int L, uint64_t T, uint64_t c0, uint64_t nsparse, uint64_t ndense) {
    static const double cell[3] = { 0.68, 1.0, 1.35 }, dense[3] = { 8.0, 11.0, 14.6 };
    const uint64_t ncols = nsparse + ndense;
    if (!ncols || !nrows) return 0;
    TensorTask t = {};
    t.T = T;
    t.c0 = c0;
    t.c1 = c0 + ncols;
    uint32_t w, nwin;
    task_digits(t, &w, &nwin);
    const double entries = (double)ncols * entries_per_column(t, w) + 150.0 * (double)(1u << w);
    const double here = entries * (45.0 + 0.8 * row_tiles_of(nrows, L));
    const double sweeps = (double)nrows * (cell[L - 2] * (double)nsparse + dense[L - 2] * (double)ndense);
    return (sweeps - here) * 1e-9;
}

int tensor_products(wl_ctx* c, std::vector<TensorTask> tasks, uint32_t nrows_total, size_t budget) {
    std::stable_sort(tasks.begin(), tasks.end(), [](const TensorTask& a, const TensorTask& b) { return a.L < b.L; });
    RC(ensure(c->tb.ones, (size_t)nrows_total * 16 + 16));
    Products p(c, budget);
    for (const TensorTask& t : tasks) p.add(t);
    return p.run();
}
