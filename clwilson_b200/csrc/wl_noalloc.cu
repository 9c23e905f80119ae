// wl_noalloc.cu -- the column product of one class without any device allocation.
//
// wl_column_product_noalloc() runs the same kernels as the engine's capped
// sweep (k_setup_rows, k_sweep_dense, k_sweep, k_finish) for caller-owned input and output
// buffers, with every intermediate (row constants, split partial products,
// split deficits, launch descriptors) in one fixed, file-scope device array.
// It is for callers that cannot allocate device memory while they run: hosts
// that reserve all device memory in their own pool at start-up and forbid
// cudaMalloc afterwards (cudaMalloc/cudaFree synchronise the device and fail
// once the pool holds the memory), and real-time paths that must not take the
// driver's allocation lock.
//
// The scratch array is allocated by the CUDA runtime when the library is
// loaded, on every GPU that loads it, and held until the process exits.
//
// The input contract is checked on the device, since the inputs live there:
// a row whose prime is even, below 5 or not below p_bound, and every row when
// the columns are not ascending primes in [2, T], get s0 = s1 = UINT64_MAX.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "wilson.h"
#include "wl_internal.h"

namespace {

constexpr uint32_t NA_MAX_ROWS = WL_NOALLOC_MAX_ROWS;
constexpr uint32_t NA_MAX_PARTIALS = WL_NOALLOC_MAX_PARTIALS;   // splits x rows
constexpr uint32_t NA_MAX_SPLITS = 1024;
constexpr uint32_t NA_MAX_ITEMS = (NA_MAX_ROWS / 256) * NA_MAX_SPLITS + NA_MAX_SPLITS;

// byte offsets of the scratch regions (each 256-byte aligned)
constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t OFF_BUCKET = 0;
constexpr size_t OFF_ITEMS = align256(OFF_BUCKET + sizeof(wl::Bucket));
constexpr size_t OFF_INFO = align256(OFF_ITEMS + sizeof(wl::SweepItem) * NA_MAX_ITEMS);
constexpr size_t OFF_MODS = align256(OFF_INFO + sizeof(wl::RowInfo) * NA_MAX_ROWS);
constexpr size_t OFF_OUT = align256(OFF_MODS + sizeof(wl::RowMod) * NA_MAX_ROWS);
constexpr size_t OFF_DEFS = align256(OFF_OUT + sizeof(wl::RowOut) * NA_MAX_ROWS);
constexpr size_t OFF_FLAG = align256(OFF_DEFS + sizeof(wl::Deficit) * NA_MAX_SPLITS);
constexpr size_t OFF_PART = align256(OFF_FLAG + sizeof(uint32_t));
constexpr size_t SCRATCH_BYTES = align256(OFF_PART + 16ull * NA_MAX_PARTIALS);
constexpr uint32_t BAD_ROW = 0xFFFFFFFFu;   // RowInfo.type of a row whose prime breaks the contract
static_assert(SCRATCH_BYTES <= WL_NOALLOC_SCRATCH_BYTES, "scratch layout exceeds the stated size");

}  // namespace

// The scratch itself: shared by every call on a device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[WL_NOALLOC_SCRATCH_BYTES];

namespace {

// The column-contract flag starts at zero in every call (the array keeps the
// previous call's contents).
__global__ void k_noalloc_clear() {
    *reinterpret_cast<uint32_t*>(g_noalloc_scratch + OFF_FLAG) = 0;
}

// One sweep's items: `tiles` row tiles of its splits from split0 on,
// 256 / tps splits to an item when the rows fit one narrow tile.
struct ItemPlan {
    uint32_t tps, split0, tiles, nitems;
};

__device__ wl::SweepItem plan_item(const ItemPlan& p, uint32_t i) {
    wl::SweepItem it;
    it.bucket = 0;
    it.tps = p.tps;
    if (p.tps == 256) {
        // all row tiles of a split before the next: the first splits fold most often and start first
        it.row0 = (i % p.tiles) * 256;
        it.split0 = p.split0 + i / p.tiles;
    } else {
        it.row0 = 0;
        it.split0 = p.split0 + i * (256 / p.tps);
    }
    return it;
}

// Fill the sweep descriptors (the dense sweep's, then the prefix-fold sweep's)
// and the row records from the caller's primes (so that no host-to-device copy
// is needed either), and check the inputs: each prime odd in [5, p_bound), the
// columns ascending in [2, T].
__global__ void k_noalloc_prep(const uint64_t* __restrict__ primes, uint32_t nrows, uint64_t p_bound, uint64_t T,
                               const uint32_t* __restrict__ cols, uint32_t ncols, ItemPlan dense, ItemPlan sparse) {
    unsigned char* base = g_noalloc_scratch;
    wl::SweepItem* items = reinterpret_cast<wl::SweepItem*>(base + OFF_ITEMS);
    wl::RowInfo* info = reinterpret_cast<wl::RowInfo*>(base + OFF_INFO);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nthreads = gridDim.x * blockDim.x;
    bool cols_ok = true;
    for (uint32_t j = i; j < ncols; j += nthreads) {
        const uint32_t q = cols[j];
        cols_ok &= q >= 2u && (uint64_t)q <= T && (j == 0 || cols[j - 1] < q);
    }
    if (!cols_ok) *reinterpret_cast<uint32_t*>(base + OFF_FLAG) = 1u;
    if (i < dense.nitems) items[i] = plan_item(dense, i);
    else if (i < dense.nitems + sparse.nitems) items[i] = plan_item(sparse, i - dense.nitems);
    if (i < nrows) {
        wl::RowInfo r;
        r.p = primes[i];
        r.Tp = T;
        r.bucket = 0;
        r.it_begin = 0;
        r.it_count = 0;
        const bool ok = (r.p & 1) && r.p >= 5 && r.p < p_bound;
        r.type = ok ? 0u : BAD_ROW;
        info[i] = r;
    }
}

// The bucket, once the columns are checked: columns up to qd take the dense
// splits (all of them when there is no other split).  With bad columns it has
// none, so that the sweeps read nothing that breaks their contract.  One warp;
// the count of columns <= qd by 32-ary search.
__global__ void k_noalloc_bucket(uint32_t nrows, uint64_t T, const uint32_t* __restrict__ cols, uint32_t ncols,
                                 uint32_t qd, uint32_t ndense, uint32_t nsparse, uint32_t L) {
    const uint32_t lane = threadIdx.x;
    if (*reinterpret_cast<const uint32_t*>(g_noalloc_scratch + OFF_FLAG)) ncols = 0;
    uint32_t lo = 0, hi = ncols;          // columns [0, lo) are <= qd, [hi, ncols) are not
    if (nsparse == 0) lo = hi;
    if (ndense == 0) hi = lo;
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t at = (uint64_t)lo + (uint64_t)lane * step;
        const uint32_t n = __popc(__ballot_sync(0xffffffffu, at < hi && cols[at < hi ? at : lo] <= qd));
        if (n == 0) { hi = lo; break; }   // cols[lo] > qd
        const uint32_t last = lo + (n - 1) * step;   // <= qd; the next probe is not
        hi = min(hi, last + step);
        lo = last + 1;
    }
    if (lane == 0) {
        wl::Bucket b;
        b.T = T;
        b.part_base = 0;
        b.ncols = ncols;
        b.row_begin = 0;
        b.nrows = nrows;
        b.nsplit = ndense + nsparse;
        b.def_base = 0;
        b.L = L;
        b.type = 0;
        b.range = 0;
        b.cdense = lo;
        b.ndense = ndense;
        b.dstart = 0;
        b.cbase = 0;
        *reinterpret_cast<wl::Bucket*>(g_noalloc_scratch + OFF_BUCKET) = b;
    }
}

__global__ void k_noalloc_out(uint32_t nrows, uint64_t* __restrict__ s0s1) {
    const wl::RowOut* out = reinterpret_cast<const wl::RowOut*>(g_noalloc_scratch + OFF_OUT);
    const wl::RowInfo* info = reinterpret_cast<const wl::RowInfo*>(g_noalloc_scratch + OFF_INFO);
    const bool cols_bad = *reinterpret_cast<const uint32_t*>(g_noalloc_scratch + OFF_FLAG) != 0;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nrows) {
        const bool bad = cols_bad || info[i].type == BAD_ROW;
        s0s1[2 * i] = bad ? ~0ull : out[i].s0;
        s0s1[2 * i + 1] = bad ? ~0ull : out[i].s1;
    }
}

// device address of the scratch array, resolved once per device; the first
// call on a device takes the mutex, later ones only read the atomic
constexpr int NA_MAX_DEVICES = 64;
std::atomic<unsigned char*> g_scratch_addr[NA_MAX_DEVICES];
int g_sms[NA_MAX_DEVICES] = {};
std::mutex g_resolve_mutex;

int resolve_scratch(int dev, unsigned char** base, int* sms) {
    unsigned char* b = g_scratch_addr[dev].load(std::memory_order_acquire);
    if (!b) {
        std::lock_guard<std::mutex> lock(g_resolve_mutex);
        b = g_scratch_addr[dev].load(std::memory_order_relaxed);
        if (!b) {
            void* ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) {
                cudaGetLastError();
                return WL_ERR_CUDA;
            }
            int n = 0;
            if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
                cudaGetLastError();
                n = 148;
            }
            g_sms[dev] = n;
            b = static_cast<unsigned char*>(ptr);
            g_scratch_addr[dev].store(b, std::memory_order_release);
        }
    }
    *base = b;
    *sms = g_sms[dev];
    return 0;
}

}  // namespace

extern "C" int wl_column_product_noalloc(const uint64_t* primes, uint32_t nrows, uint64_t p_bound, uint64_t T,
                                         const uint32_t* cols, uint32_t ncols, uint64_t* s0s1, void* stream) {
    if (!primes || !s0s1 || nrows == 0 || T == 0 || p_bound > WL_MAXP + 1 || p_bound < 6) return WL_ERR_ARG;
    if (ncols > 0 && !cols) return WL_ERR_ARG;
    if (nrows > NA_MAX_ROWS) return WL_ERR_TOO_LARGE;
    // an error left by the caller's earlier CUDA work stays the caller's: report it, launch nothing
    if (cudaPeekAtLastError() != cudaSuccess) return WL_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NA_MAX_DEVICES) return WL_ERR_CUDA;
    unsigned char* base = nullptr;
    int sms = 0;
    if (resolve_scratch(dev, &base, &sms)) return WL_ERR_CUDA;
    const int L = p_bound - 1 < (1ull << 31) ? 2 : (p_bound - 1 < (1ull << 47) ? 3 : 4);

    // split the columns so that about 2 x (SMs x 2048) threads work, each
    // split at least 2048 columns long, within the scratch limits
    uint32_t nsplit = 1;
    if (ncols > 0) {
        const uint64_t want = ((uint64_t)sms * 4096 + nrows - 1) / nrows;
        uint64_t s = want;
        s = s < ncols / 2048 ? s : ncols / 2048;
        s = s < NA_MAX_SPLITS ? s : NA_MAX_SPLITS;
        s = s < NA_MAX_PARTIALS / nrows ? s : NA_MAX_PARTIALS / nrows;
        nsplit = s > 0 ? (uint32_t)s : 1;
    }
    if ((uint64_t)nsplit * nrows > NA_MAX_PARTIALS) return WL_ERR_TOO_LARGE;
    // Columns up to qd, where the exponent changes at most columns, take the dense
    // sweep: an exponentiation at each of them would make the first of equal
    // prefix-fold splits several times as long as the rest (2,000 rows, T = 1e8,
    // 1.08e6 columns: 5.65 ms of sweep, most of it one split).  qd lies a factor
    // of two above the engine's line, since these few splits are the whole launch.
    // The splits are shared out by cells (about six to a dense column); the count
    // of columns below qd that this goes by is an estimate, and any share is right.
    const double Td = (double)T, qx = 2.0 * std::sqrt(Td * std::log(std::sqrt(Td) + 3.0)) + 16.0;
    const uint32_t qd = qx < 4294967295.0 ? (uint32_t)qx : 0xFFFFFFFFu;
    const double nd = std::min((double)ncols, 1.2551 * qx / std::log(qx)), ns = (double)ncols - nd;
    uint32_t sd = 0;
    if (ncols > 0) {
        sd = (uint32_t)(nsplit * 6.0 * nd / (6.0 * nd + ns) + 0.5);
        sd = std::max<uint32_t>(sd, 1);
        if (ns <= 0) sd = nsplit;
        else if (sd >= nsplit) sd = nsplit > 1 ? nsplit - 1 : 0;
        // the prefix-fold sweep in whole waves of four CTAs per SM (a split and row
        // tile each), the splits left over to the dense sweep, which runs before it
        // and would otherwise leave most of the SMs idle
        const uint32_t tiles = (nrows + 255) / 256, slots = 4 * (uint32_t)sms, ss = nsplit - sd;
        if (nrows >= 256 && sd && ss * tiles >= slots) {
            const uint32_t whole = ss * tiles / slots * slots / tiles;
            sd = std::max(sd, std::min(nsplit - whole, (uint32_t)(nd / 128.0)));
            nsplit = sd + whole;
        }
    }
    auto plan = [&](uint32_t split0, uint32_t n, uint32_t min_tps) {
        ItemPlan p = { 256, split0, (nrows + 255) / 256, 0 };
        if (n == 0) return p;
        if (nrows >= 256) {
            p.nitems = p.tiles * n;
        } else {
            p.tps = min_tps;
            while (p.tps < nrows) p.tps <<= 1;
            const uint32_t per = 256 / p.tps;
            p.nitems = (n + per - 1) / per;
        }
        return p;
    };
    const ItemPlan dense = plan(0, sd, 8), sparse = plan(sd, nsplit - sd, 1);
    const uint32_t nitems = dense.nitems + sparse.nitems;
    if (nitems > NA_MAX_ITEMS) return WL_ERR_TOO_LARGE;

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // enough threads for the items and rows, and for the check of the columns to be short
    const uint32_t prep_threads = std::max(std::max(nitems, nrows), std::min(ncols / 8, (uint32_t)sms * 1024u));
    // each launch's own error is checked right after it
    k_noalloc_clear<<<1, 1, 0, st>>>();
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    k_noalloc_prep<<<(prep_threads + 255) / 256, 256, 0, st>>>(primes, nrows, p_bound, T, cols, ncols, dense, sparse);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    k_noalloc_bucket<<<1, 32, 0, st>>>(nrows, T, cols, ncols, qd, sd, nsplit - sd, (uint32_t)L);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    wl::Bucket* bk = reinterpret_cast<wl::Bucket*>(base + OFF_BUCKET);
    wl::SweepItem* items = reinterpret_cast<wl::SweepItem*>(base + OFF_ITEMS);
    wl::RowInfo* info = reinterpret_cast<wl::RowInfo*>(base + OFF_INFO);
    wl::RowMod* mods = reinterpret_cast<wl::RowMod*>(base + OFF_MODS);
    wl::RowOut* out = reinterpret_cast<wl::RowOut*>(base + OFF_OUT);
    wl::Deficit* defs = reinterpret_cast<wl::Deficit*>(base + OFF_DEFS);
    uint4* part = reinterpret_cast<uint4*>(base + OFF_PART);
    wl::launch_setup_rows(info, nrows, mods, st);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    wl::launch_sweep_dense(L, 1, dense.nitems, bk, items, mods, cols, nullptr, part, defs, st, wl::DENSE_SMEM_W3, 8);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    wl::launch_sweep(1, L, 1, sparse.nitems, bk, items + dense.nitems, mods, cols, part, defs, st);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    wl::launch_finish(L, bk, info, mods, part, defs, 1, nullptr, 0, nrows, 0, out, st);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    k_noalloc_out<<<(nrows + 255) / 256, 256, 0, st>>>(nrows, s0s1);
    if (cudaGetLastError() != cudaSuccess) return WL_ERR_CUDA;
    return 0;
}
