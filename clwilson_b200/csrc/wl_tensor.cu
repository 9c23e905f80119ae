// wl_tensor.cu -- column products on the 5th-generation tensor cores.
//
// The sweep's work is, for every row modulus n = p^2 of a bucket and every
// column q, one multiplication by q^{e}, e = v_q(T!).  One row and column at a
// time that is 2L+1 32-bit multiplies (k_sweep), which the integer pipe
// bounds.  Here the multiplications by whole groups of columns become an
// integer matrix product:
//
//   * W, the exact product of a group of columns (up to 512 bytes), is the
//     same for every row.  Its residue modulo n is a contraction:
//         W mod n = sum_k W_k * (256^k mod n)        (W_k: bytes of W),
//     and with the constants 256^k mod n split into bytes as well, an
//     unsigned 8-bit matrix product with 32-bit accumulators:
//         D[g][r, i] = sum_k W[g][k] * byte_i(256^k mod n_r)  <= 512 * 255^2 < 2^25,
//     exact in int32.  tcgen05.mma kind::i8 runs it: groups are the M side
//     (128 tensor-memory lanes), the 4L bytes of each row's residue the N
//     side (256 columns hold 256 / (4L) rows), k the contraction.
//   * The epilogue reads a row's 4L digits of one group in one thread, forms
//     V = sum_i D_i 256^i (L+1 limbs) and multiplies the thread's running
//     product by it with L+1 Montgomery limb steps.  A group of 140 or so
//     columns so costs a row the multiplies of L+1 cells.
//   * Exponents: the columns are sorted by the base-2^w digits of e (label
//     (j, d): digit j is d).  One lane multiplies groups of one label only, so
//         prod q^e = prod_j ( prod_d A_{j,d}^d )^{2^(w j)},
//     A_{j,d} the product over the label, with the powers taken once per row.
//
// The constants carry a factor 2^(32(L+1)) that the limb steps take out again,
// and running products are in Montgomery form (R = 2^(32L)) throughout, so no
// power of two has to be restored: a row's result is exact.
//
// Both operands lie in global memory as the shared-memory image that the
// matrix instruction reads (K-major rows of 128 bytes, 128-byte swizzle), so
// that plain bulk copies of whole blocks bring them in.
#include "wl_tensor.h"
#include "wl_arith.cuh"

namespace wl {

// ---------------------------------------------------------------------------
// Digit sort: the columns of a task by the labels of their exponents.
// ---------------------------------------------------------------------------

template <class D>
__device__ __forceinline__ uint32_t task_of_block(const D* __restrict__ d, uint32_t nt, uint32_t b, uint32_t D::*first) {
    uint32_t lo = 0, hi = nt - 1;         // the last task with first <= b
    while (lo < hi) {
        const uint32_t m = (lo + hi + 1) >> 1;
        if (d[m].*first <= b) lo = m; else hi = m - 1;
    }
    return lo;
}

// Adds 1 to h[label] for every lane with label != 0, returning the value
// before (the lane's slot).  Neighbouring columns mostly share their exponent
// in the sparse regime, so a warp with one label adds once.
__device__ __forceinline__ uint32_t warp_count(uint32_t* h, uint32_t label, bool on) {
    const uint32_t act = __ballot_sync(0xffffffffu, on);
    if (!act) return 0;
    const int src = __ffs(act) - 1;
    const uint32_t first = __shfl_sync(0xffffffffu, label, src);
    if (__all_sync(0xffffffffu, !on || label == first)) {
        uint32_t base = 0;
        const uint32_t lane = threadIdx.x & 31;
        if ((int)lane == src) base = atomicAdd(&h[first], (uint32_t)__popc(act));
        base = __shfl_sync(0xffffffffu, base, src);
        return base + __popc(act & ((1u << lane) - 1u));
    }
    return on ? atomicAdd(&h[label], 1u) : 0u;
}

__global__ void __launch_bounds__(256)
k_tensor_count(const TensorDesc* __restrict__ desc, uint32_t ntask, const uint32_t* __restrict__ cols,
               uint32_t* __restrict__ counts) {
    __shared__ uint32_t h[TN_LABELS];
    const TensorDesc d = desc[task_of_block(desc, ntask, blockIdx.x, &TensorDesc::blk0)];
    const uint32_t nlab = d.nwin << d.w, mask = (1u << d.w) - 1;
    for (uint32_t i = threadIdx.x; i < nlab; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint32_t b0 = d.c0 + (blockIdx.x - d.blk0) * TN_COLS_PER_BLOCK;
    const uint32_t b1 = min(d.c1, b0 + TN_COLS_PER_BLOCK);
    // four columns at a time, so that their loads and divisions overlap
    for (uint32_t k = b0 + threadIdx.x; k - threadIdx.x < b1; k += 4 * 256) {
        uint64_t e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = k + 256 * i < b1 ? legendre(d.T, cols[k + 256 * i]) : 0;
        for (uint32_t j = 0; j < d.nwin; ++j) {
            if (!__any_sync(0xffffffffu, (e[0] | e[1] | e[2] | e[3]) != 0)) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t dg = (uint32_t)e[i] & mask;
                warp_count(h, (j << d.w) | dg, dg != 0);
                e[i] >>= d.w;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nlab; i += blockDim.x)
        if (h[i]) atomicAdd(&counts[d.lab0 + i], h[i]);
}

// cursor[label] starts at the label's place in `list`.  The order inside a
// label depends on the order of the CTAs; its product does not.  One digit at a
// time: a column's slot among the CTA's columns of its label is counted once and
// stays in a register until the CTA has its place in the list (counting again
// for the write-out cost a third of the kernel: 0.58 ms for 5e7 columns).
__global__ void __launch_bounds__(256)
k_tensor_scatter(const TensorDesc* __restrict__ desc, uint32_t ntask, const uint32_t* __restrict__ cols,
                 uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
    constexpr int PER = TN_COLS_PER_BLOCK / TN_SCATTER / 256;
    __shared__ uint32_t h[1u << TN_WMAX];
    const TensorDesc d = desc[task_of_block(desc, ntask, blockIdx.x / TN_SCATTER, &TensorDesc::blk0)];
    const uint32_t nd = 1u << d.w, mask = nd - 1;
    const uint32_t b0 = d.c0 + (blockIdx.x - d.blk0 * TN_SCATTER) * (256 * PER) + threadIdx.x;
    const uint32_t b1 = d.c1;
    uint64_t e[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) e[k] = b0 + 256 * k < b1 ? legendre(d.T, cols[b0 + 256 * k]) : 0;
    for (uint32_t j = 0; j < d.nwin; ++j) {
        uint64_t any = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) any |= e[k];
        if (!__syncthreads_or(any != 0)) break;            // no digit left
        for (uint32_t i = threadIdx.x; i < nd; i += 256) h[i] = 0;
        __syncthreads();
        uint32_t rank[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const uint32_t dg = (uint32_t)e[k] & mask;
            rank[k] = warp_count(h, dg, dg != 0);
        }
        __syncthreads();
        uint32_t* cur = cursor + d.lab0 + (j << d.w);
        for (uint32_t i = threadIdx.x; i < nd; i += 256)
            if (h[i]) h[i] = atomicAdd(&cur[i], h[i]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const uint32_t dg = (uint32_t)e[k] & mask;
            if (dg) list[h[dg] + rank[k]] = cols[b0 + 256 * k];
            e[k] >>= d.w;
        }
    }
}

// ---------------------------------------------------------------------------
// Layout: labels -> places in the list, lane runs, slots and segments.  One CTA
// per task scans its labels 256 at a time; planned here rather than on the host
// because a batch has hundreds of tasks of thousands of labels each (192 tasks:
// 80 ms of host time, most of the call).
// ---------------------------------------------------------------------------

// Columns of a group of which none is above q: an eighth of them stays below 2^512
// (k_tensor_build), so the group below 2^4096.
__device__ __forceinline__ uint32_t group_columns(uint64_t q) {
    const double k = 511.99 / log2((double)(q < 2 ? 2 : q) + 1.0);
    return 8 * (uint32_t)fmin(k, (double)(TN_GMAX / 8));
}

struct LabelPlan { uint32_t n, g, longs, shorts; };

// Columns of label (j, d) have v_q(T!) >= d 2^(wj), so q <= T / (d 2^(wj)) + 1.
__device__ __forceinline__ LabelPlan plan_label(const TensorDesc& d, uint32_t l, uint32_t n, uint32_t g_all) {
    LabelPlan p = { n, g_all, 0, 0 };
    if (!n) return p;
    const uint32_t dg = l & ((1u << d.w) - 1), j = l >> d.w;
    const uint64_t q = (d.T >> (d.w * j)) / dg + 1;
    if (q < d.q_max) p.g = group_columns(q);
    const uint32_t ng = (n + p.g - 1) / p.g;
    p.longs = ng / TN_LONG;
    p.shorts = (ng % TN_LONG + TN_SHORT - 1) / TN_SHORT;
    if (p.shorts * TN_SHORT >= TN_LONG) { ++p.longs; p.shorts = 0; }
    return p;
}

// Exclusive prefix sum of v over the CTA's 256 threads, *total its sum.
__device__ __forceinline__ uint32_t cta_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t ws[8];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += x;
    }
    __syncthreads();
    if (lane == 31) ws[wid] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        before += i < wid ? ws[i] : 0u;
        all += ws[i];
    }
    *total = all;
    return before + incl - v;
}

// FILL = 0: sizes only.  FILL = 1: the tables too.
template <int FILL>
__global__ void __launch_bounds__(256)
k_tensor_layout(const TensorDesc* __restrict__ desc, const uint32_t* __restrict__ counts, TensorSize* __restrict__ size,
                uint32_t* __restrict__ cursor, LaneRun* __restrict__ runs, FoldSeg* __restrict__ segs,
                uint32_t* __restrict__ lab_seg) {
    const TensorDesc d = desc[blockIdx.x];
    const uint32_t labels = d.nwin << d.w, g_all = group_columns(d.q_max);
    uint32_t entries = 0, longs = 0, shorts = 0, slots = 0, nseg = 0;
    for (uint32_t l0 = 0; l0 < labels; l0 += 256) {
        const uint32_t l = l0 + threadIdx.x;
        const LabelPlan p = plan_label(d, l, l < labels ? counts[d.lab0 + l] : 0u, g_all);
        uint32_t t_n, t_long, t_short, t_slot, t_seg;
        const uint32_t at = entries + cta_scan(p.n, &t_n);
        const uint32_t lo = longs + cta_scan(p.longs, &t_long), sh = shorts + cta_scan(p.shorts, &t_short);
        // one slot per warp that the label's long runs touch, one per short run
        const uint32_t nslot = p.shorts + (p.longs ? (lo + p.longs - 1) / 32 - lo / 32 + 1 : 0u);
        const uint32_t sl = slots + cta_scan(nslot, &t_slot);
        const uint32_t sg = nseg + cta_scan((nslot + TN_SEG - 1) / TN_SEG, &t_seg);
        if (FILL && l < labels) {
            const uint32_t start = d.list0 + at, end = start + p.n;
            cursor[d.lab0 + l] = start;
            lab_seg[d.lab_seg0 + l] = sg;
            for (uint32_t k = 0; k < p.longs; ++k)
                runs[d.long0 + lo + k] = { start + k * p.g * TN_LONG, end, p.g, sl + (lo + k) / 32 - lo / 32 };
            const uint32_t s0 = sl + nslot - p.shorts, c0 = start + p.longs * p.g * TN_LONG;
            for (uint32_t k = 0; k < p.shorts; ++k)
                runs[d.short0 + sh + k] = { c0 + k * p.g * TN_SHORT, end, p.g, s0 + k };
            for (uint32_t k = 0; k < nslot; k += TN_SEG)
                segs[d.seg0 + sg + k / TN_SEG] = { sl + k, min(TN_SEG, nslot - k) };
        }
        entries += t_n;
        longs += t_long;
        shorts += t_short;
        slots += t_slot;
        nseg += t_seg;
    }
    if (FILL) {
        if (threadIdx.x == 0) lab_seg[d.lab_seg0 + labels] = nseg;
        // the last tiles' lanes without a run: groups of no column
        for (uint32_t k = longs + threadIdx.x; k < d.nlong; k += 256) runs[d.long0 + k] = { 0, 0, 1, RUN_NONE };
        for (uint32_t k = shorts + threadIdx.x; k < d.nshort; k += 256) runs[d.short0 + k] = { 0, 0, 1, RUN_NONE };
    } else if (threadIdx.x == 0) {
        size[blockIdx.x] = { entries, longs, shorts, slots, nseg };
    }
}

// ---------------------------------------------------------------------------
// Group products: one warp multiplies up to g columns into 128 limbs.  Each
// lane multiplies its share of the columns serially (5 limbs), then five levels
// of pairwise products in shared memory bring 32 shares to one number.  The
// columns are dealt out so that an eighth of them (four lanes) stays below
// 2^512, so a lane holds at most 160 bits, a pair 288 and from there on every
// operand fits its power of two.
//
// Bound by the multiply pipe (fmaheavy 87% busy in a form that gave each lane
// four columns of the schoolbook product, half of whose terms were zero).  The
// three upper levels, nine tenths of the work, therefore cut the square of
// partial products into one block per lane (4 x 8, 8 x 8, 8 x 16 limbs): each
// lane multiplies its block out in registers with no term wasted, and the
// blocks are added up afterwards, four limbs per lane.
// ---------------------------------------------------------------------------

constexpr uint32_t TB_WARPS = 8;
constexpr uint32_t TB_X = 160;          // words of the operands: 32 shares of 5 limbs
constexpr uint32_t TB_P = 32 * 28;      // words of the partial products

// Four limbs of a lane, whose carry (and the lower lanes') goes up to the next
// lane of the same product (lp lanes each); returns what leaves the top lane.
// At most lp rounds, almost always one or two.
__device__ __forceinline__ uint32_t carry_up(uint32_t (&out)[4], uint32_t carry, uint32_t li, uint32_t lp) {
    uint32_t add = 0;
    for (uint32_t round = 0; round < lp; ++round) {
        uint32_t in = __shfl_up_sync(0xffffffffu, carry, 1);
        if (li == lp - 1) add += carry;
        if (li == 0) in = 0;
        if (!__any_sync(0xffffffffu, in != 0)) break;
        uint64_t z = in;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            z += out[i];
            out[i] = (uint32_t)z;
            z >>= 32;
        }
        carry = (uint32_t)z;
    }
    return add;
}

// Products of operands of NL + 1 limbs (the last one short), 2 lp = NL lanes to
// a product, four columns of the schoolbook product per lane.
template <int NL>
__device__ __forceinline__ void build_low(const uint32_t* x, uint32_t* c0, uint32_t* c1, uint32_t* c2, uint32_t lane,
                                          uint32_t (&out)[4], uint32_t* top_limb) {
    constexpr uint32_t lp = NL / 2;
    const uint32_t pr = lane / lp, li = lane % lp;
    const uint32_t* a = x + pr * 2 * (NL + 1);
    const uint32_t* b = a + NL + 1;
    const int col = 4 * (int)li;
    uint32_t lo[4] = { 0, 0, 0, 0 };
    uint64_t hi[4] = { 0, 0, 0, 0 };
    auto bat = [&](int i) -> uint32_t { return (unsigned)i <= (unsigned)NL ? b[i] : 0u; };   // zero outside
    uint32_t w0 = bat(col), w1 = bat(col + 1), w2 = bat(col + 2), w3 = bat(col + 3);
#pragma unroll
    for (int k = 0; k <= NL; ++k) {
        const uint32_t av = a[k];
        uint64_t p;
        p = (uint64_t)av * w0 + lo[0]; lo[0] = (uint32_t)p; hi[0] += p >> 32;
        p = (uint64_t)av * w1 + lo[1]; lo[1] = (uint32_t)p; hi[1] += p >> 32;
        p = (uint64_t)av * w2 + lo[2]; lo[2] = (uint32_t)p; hi[2] += p >> 32;
        p = (uint64_t)av * w3 + lo[3]; lo[3] = (uint32_t)p; hi[3] += p >> 32;
        w3 = w2; w2 = w1; w1 = w0;
        w0 = bat(col - k - 1);
    }
    const uint32_t top = a[NL] * b[NL];      // column 2 NL: its high half and all above are zero
    __syncwarp();
    const uint32_t cb0 = pr * (2 * NL + 3);  // two zeros, then the product's columns
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t at = cb0 + 2 + col + i;
        c0[at] = lo[i];
        c1[at] = (uint32_t)hi[i];
        c2[at] = (uint32_t)(hi[i] >> 32);
    }
    if (li == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { c1[cb0 + i] = 0; c2[cb0 + i] = 0; }
        c0[cb0 + 2 + 2 * NL] = top;
    }
    __syncwarp();
    // limb c = lo(c) + mid(c - 1) + high(c - 2) and the carry
    uint64_t s = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t at = cb0 + 2 + col + i;
        s += (uint64_t)c0[at] + c1[at - 1] + c2[at - 2];
        out[i] = (uint32_t)s;
        s >>= 32;
    }
    const uint32_t add = carry_up(out, (uint32_t)s, li, lp);
    const uint32_t at = cb0 + 2 + 2 * NL;
    *top_limb = c0[at] + c1[at - 1] + c2[at - 2] + add;   // the product's last lane
}

// Products of operands of NL limbs, NL / 2 lanes to a product, one block of
// BA x BB limbs per lane.  x: the operands one after another; the lane's four
// limbs of its product come back in out.
template <int NL, int BA, int BB>
__device__ __forceinline__ void build_high(const uint32_t* x, uint32_t* part, uint32_t lane, uint32_t (&out)[4]) {
    constexpr uint32_t lp = NL / 2, NA = NL / BA, NBB = NL / BB, ST = BA + BB + 4;   // stride without bank conflicts
    static_assert(NA * NBB == lp, "one block per lane");
    const uint32_t pr = lane / lp, li = lane % lp;
    const uint32_t ia = li % NA, jb = li / NA;
    uint32_t a[BA], b[BB], t[BA + BB];
    {
        const uint4* pa = reinterpret_cast<const uint4*>(x + pr * 2 * NL + ia * BA);
        const uint4* pb = reinterpret_cast<const uint4*>(x + pr * 2 * NL + NL + jb * BB);
#pragma unroll
        for (int i = 0; i < BA / 4; ++i) {
            const uint4 v = pa[i];
            a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < BB / 4; ++i) {
            const uint4 v = pb[i];
            b[4 * i] = v.x; b[4 * i + 1] = v.y; b[4 * i + 2] = v.z; b[4 * i + 3] = v.w;
        }
    }
#pragma unroll
    for (int i = 0; i < BA; ++i) {
        uint32_t carry = 0;
#pragma unroll
        for (int j = 0; j < BB; ++j) {
            const uint64_t p = (uint64_t)a[i] * b[j] + (i ? t[i + j] : 0u) + carry;
            t[i + j] = (uint32_t)p;
            carry = (uint32_t)(p >> 32);
        }
        t[i + BB] = carry;
    }
    {
        uint4* pt = reinterpret_cast<uint4*>(part + lane * ST);
#pragma unroll
        for (int i = 0; i < (BA + BB) / 4; ++i) pt[i] = make_uint4(t[4 * i], t[4 * i + 1], t[4 * i + 2], t[4 * i + 3]);
    }
    __syncwarp();
    // limbs 4 li .. 4 li + 3: quad li - ia qa - jb qb of every block that reaches there
    constexpr int qa = BA / 4, qb = BB / 4, reach = (qa + qb + qa - 1) / qa;
    uint32_t carry = 0;
    out[0] = out[1] = out[2] = out[3] = 0;
#pragma unroll
    for (int j = 0; j < (int)NBB; ++j) {
        const int rel = (int)li - j * qb;
        const int i0 = rel >= 0 ? rel / qa : -1;
#pragma unroll
        for (int k = 0; k < reach; ++k) {
            const int i = i0 - k;
            if (i < 0 || i >= (int)NA || rel - i * qa >= qa + qb) continue;
            const uint4 v = *reinterpret_cast<const uint4*>(part + (pr * lp + j * NA + i) * ST + 4 * (rel - i * qa));
            asm("add.cc.u32 %0, %0, %5;\n\t"
                "addc.cc.u32 %1, %1, %6;\n\t"
                "addc.cc.u32 %2, %2, %7;\n\t"
                "addc.cc.u32 %3, %3, %8;\n\t"
                "addc.u32 %4, %4, 0;"
                : "+r"(out[0]), "+r"(out[1]), "+r"(out[2]), "+r"(out[3]), "+r"(carry)
                : "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
        }
    }
    carry_up(out, carry, li, lp);
}

// The place of a lane's four limbs of group m of group tile mt: limbs 4 lane ..
// 4 lane + 3 are bytes 16 lane .. of the group, chunk lane % 8 of block lane / 8
// (128-byte swizzle: chunk ^ (row % 8)).
__device__ __forceinline__ uint4* group_place(uint8_t* w, uint32_t mt, uint32_t m, uint32_t lane) {
    const uint32_t kb = lane >> 3, ch = lane & 7;
    return reinterpret_cast<uint4*>(w + (((uint64_t)mt * TN_KB + kb) * TN_M + m) * 128 + ((ch ^ (m & 7)) << 4));
}

// The lane's part [k0, k1) of a group's n numbers: a quarter of its eighth.
__device__ __forceinline__ void share_of(uint32_t n, uint32_t lane, uint32_t* k0, uint32_t* k1) {
    const uint32_t e = lane >> 2, q0 = n * e / 8, nq = n * (e + 1) / 8 - q0;
    *k0 = q0 + nq * (lane & 3) / 4;
    *k1 = q0 + nq * ((lane & 3) + 1) / 4;
}

__device__ __forceinline__ void share_times(uint32_t (&a)[5], uint32_t q) {
    uint64_t carry = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const uint64_t v = (uint64_t)a[i] * q + carry;
        a[i] = (uint32_t)v;
        carry = v >> 32;
    }
}

// The product of the warp's 32 shares; the lane's four limbs come back in out.
__device__ __forceinline__ void build_tree(const uint32_t (&a)[5], uint32_t* x, uint32_t* p, uint32_t lane, uint32_t (&out)[4]) {
#pragma unroll
    for (int i = 0; i < 5; ++i) x[lane * 5 + i] = a[i];
    __syncwarp();
    uint32_t top;
    build_low<4>(x, p, p + 176, p + 352, lane, out, &top);     // 5 x 5 limbs -> 9
    {
        const uint32_t ob = (lane >> 1) * 9, li = lane & 1;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[ob + 4 * li + i] = out[i];
        if (li == 1) x[ob + 8] = top;
    }
    __syncwarp();
    build_low<8>(x, p, p + 176, p + 352, lane, out, &top);     // 9 x 9 limbs -> 16 (the 17th is zero)
    uint4* xv = reinterpret_cast<uint4*>(x) + lane;
    *xv = make_uint4(out[0], out[1], out[2], out[3]);
    __syncwarp();
    build_high<16, 4, 8>(x, p, lane, out);
    *xv = make_uint4(out[0], out[1], out[2], out[3]);
    __syncwarp();
    build_high<32, 8, 8>(x, p, lane, out);
    *xv = make_uint4(out[0], out[1], out[2], out[3]);
    __syncwarp();
    build_high<64, 8, 16>(x, p, lane, out);
}

__global__ void __launch_bounds__(TB_WARPS * 32)
k_tensor_build(const TensorSec* __restrict__ secs, uint32_t nsec, const LaneRun* __restrict__ lr,
               const uint32_t* __restrict__ list, uint8_t* __restrict__ w) {
    __shared__ __align__(16) uint32_t sx[TB_WARPS][TB_X];
    __shared__ __align__(16) uint32_t sp[TB_WARPS][TB_P];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr uint32_t PER_TILE = TN_M / TB_WARPS;      // CTAs per group tile
    const uint32_t mt = blockIdx.x / PER_TILE;
    const uint32_t m = (blockIdx.x % PER_TILE) * TB_WARPS + wid;      // lane of the tile
    const TensorSec sec = secs[task_of_block(secs, nsec, mt, &TensorSec::mt0)];
    const uint32_t local = mt - sec.mt0, cb = local / sec.tn, t = local % sec.tn;
    const LaneRun run = lr[sec.run0 + cb * TN_M + m];
    const uint64_t beg = (uint64_t)run.start + (uint64_t)t * run.g;
    const uint32_t n = beg < run.end ? (uint32_t)min((uint64_t)run.g, run.end - beg) : 0u;
    uint4* dst = group_place(w, mt, m, lane);
    if (n == 0) {                                      // no column: the product is 1
        *dst = make_uint4(lane == 0 ? 1u : 0u, 0u, 0u, 0u);
        return;
    }
    uint32_t a[5] = { 1, 0, 0, 0, 0 }, k0, k1, out[4];
    share_of(n, lane, &k0, &k1);
    for (uint32_t k = k0; k < k1; ++k) share_times(a, list[beg + k]);
    build_tree(a, sx[wid], sp[wid], lane, out);
    *dst = make_uint4(out[0], out[1], out[2], out[3]);
}

// Groups of consecutive integers: group j = 128 tile + m of a bucket's tail holds
// T + 1 + j g .. T + (j + 1) g.
__global__ void __launch_bounds__(TB_WARPS * 32)
k_tensor_tail_build(const TensorDesc* __restrict__ desc, const TensorSec* __restrict__ secs, uint32_t nsec,
                    uint8_t* __restrict__ w) {
    __shared__ __align__(16) uint32_t sx[TB_WARPS][TB_X];
    __shared__ __align__(16) uint32_t sp[TB_WARPS][TB_P];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr uint32_t PER_TILE = TN_M / TB_WARPS;
    const uint32_t mt = blockIdx.x / PER_TILE;
    const uint32_t m = (blockIdx.x % PER_TILE) * TB_WARPS + wid;
    const TensorSec sec = secs[task_of_block(secs, nsec, mt, &TensorSec::mt0)];
    const uint64_t first = desc[sec.task].T + 1 + ((uint64_t)(mt - sec.mt0) * TN_M + m) * sec.g;
    uint32_t a[5] = { 1, 0, 0, 0, 0 }, k0, k1, out[4];
    share_of(sec.g, lane, &k0, &k1);
    for (uint32_t k = k0; k < k1; ++k) {
        const uint64_t N = first + k;
        const uint32_t hi = (uint32_t)(N >> 32);
        if (hi == 0) {
            share_times(a, (uint32_t)N);
        } else {                                       // a lo + (a hi) 2^32
            uint32_t b[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) b[i] = a[i];
            share_times(a, (uint32_t)N);
            share_times(b, hi);
            uint64_t c = 0;
#pragma unroll
            for (int i = 1; i < 5; ++i) {
                c += (uint64_t)a[i] + b[i - 1];
                a[i] = (uint32_t)c;
                c >>= 32;
            }
        }
    }
    build_tree(a, sx[wid], sp[wid], lane, out);
    *group_place(w, mt, m, lane) = make_uint4(out[0], out[1], out[2], out[3]);
}

// ---------------------------------------------------------------------------
// Row constants: bytes of 2^(8k + 32(L+1)) mod n for k < 512, in row tiles of
// TN_N digit columns.  One thread per (row, 16 values of k).
// ---------------------------------------------------------------------------

template <int L>
__global__ void __launch_bounds__(256)
k_tensor_consts(const TensorDesc* __restrict__ desc, uint32_t ntask, const RowMod* __restrict__ mods,
                uint8_t* __restrict__ consts, uint4* __restrict__ ones) {
    constexpr uint32_t RT = TN_N / (4 * L);
    constexpr uint32_t SEGS = TN_K / 16;          // threads per row
    constexpr uint32_t PER_CTA = 256 / SEGS;      // rows per CTA
    constexpr uint32_t CTAS = (RT + PER_CTA - 1) / PER_CTA;
    const uint32_t tile = blockIdx.x / CTAS;
    const uint32_t r = (blockIdx.x % CTAS) * PER_CTA + threadIdx.x / SEGS;   // row of the tile
    const uint32_t sg = threadIdx.x % SEGS;
    if (r >= RT) return;
    const TensorDesc& d = desc[task_of_block(desc, ntask, tile, &TensorDesc::ct0)];
    const uint32_t rl = (tile - d.ct0) * RT + r;
    const bool live = rl < d.nrows;
    uint32_t b[4 * L][4];                          // byte i of the 16 values, packed
#pragma unroll
    for (int i = 0; i < 4 * L; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) b[i][k] = 0;
    if (live) {
        const uint32_t row = d.row_begin + rl;
        const RowMod md = mods[row];
        uint32_t n[L];
#pragma unroll
        for (int k = 0; k < L; ++k) n[k] = md.n[k];
        const Res<L> one = mont_one<L>(n);         // R mod n
        if (sg == 0)
            ones[tile * RT + r] = make_uint4(one.w[0], one.w[1], L > 2 ? one.w[2 < L ? 2 : 0] : 0, L > 3 ? one.w[3 < L ? 3 : 0] : 0);
        Res<L> m256 = one;                         // 256 R mod n
        for (int k = 0; k < 8; ++k) dbl_mod<L>(m256, n);
        // 2^(128 sg + 32) R = 2^(8 (16 sg) + 32 (L + 1)) mod n
        const uint32_t e = 128u * sg + 32u;
        Res<L> c = one;
        for (int bit = 31 - __clz(e); bit >= 0; --bit) {
            c = mont_mul<L>(c, c, n, md.ninv);
            if ((e >> bit) & 1) { reduce_full<L>(c, n); dbl_mod<L>(c, n); }
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            reduce_full<L>(c, n);
#pragma unroll
            for (int i = 0; i < 4 * L; ++i)
                b[i][k >> 2] |= ((c.w[i >> 2] >> (8 * (i & 3))) & 255u) << (8 * (k & 3));
            if (k < 15) c = mont_mul<L>(c, m256, n, md.ninv);
        }
    }
    const uint32_t kb = sg >> 3, ch = sg & 7;
#pragma unroll
    for (int i = 0; i < 4 * L; ++i) {
        const uint32_t col = r * 4 * L + i;
        uint8_t* dst = consts + (((uint64_t)tile * TN_KB + kb) * TN_N + col) * 128 + ((ch ^ (col & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(b[i][0], b[i][1], b[i][2], b[i][3]);
    }
}

// ---------------------------------------------------------------------------
// The matrix product with the running products in its epilogue.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Waits for the phase, for about limit_ns at most (a step of a wait is bounded
// by the hardware); false when the limit was reached.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try(bar, parity)) return true;
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (uint32_t k = 0; k < (1u << 28); ++k) {
        if (mbar_try(bar, parity)) return true;
        if ((k & 255u) == 255u) {
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t - t0 > limit_ns) break;
        }
    }
    return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// What a CTA has in flight when one of its waits has run out ends before its
// shared and tensor memory go: these waits have a limit of their own.
constexpr uint64_t TG_DRAIN_NS = 4000000000ull;
// Shared-memory descriptor of a K-major operand block: rows of 128 bytes, 128-byte
// swizzle, groups of eight rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t (&v)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
// The wait takes the loaded registers through it, so that no use moves above it.
template <int L>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[L][4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < L; ++j)
        asm volatile("" : "+r"(v[j][0]), "+r"(v[j][1]), "+r"(v[j][2]), "+r"(v[j][3]));
}

constexpr uint32_t TG_STAGES = 5;                     // 16 KB stages of group tiles
constexpr uint32_t TG_EPI_WARPS = 16, TG_WG = TG_EPI_WARPS / 4;
constexpr uint32_t TG_THREADS = (TG_EPI_WARPS + 2) * 32;
constexpr uint32_t TG_A_BYTES = TN_M * 128;           // one block of a group tile
constexpr uint32_t TG_B_BYTES = TN_N * 128;           // one block of a row tile
constexpr uint32_t TG_SMEM = TN_KB * TG_B_BYTES + TG_STAGES * TG_A_BYTES + 1024 /* alignment */ + 256 /* barriers */;
// kind::i8 instruction descriptor: S32 accumulators, unsigned 8-bit A and B, both K-major
constexpr uint32_t TG_IDESC = (2u << 4) | ((TN_N >> 3) << 17) | ((TN_M >> 4) << 24);

// running product *= V 2^(-32(L+1)), V = sum_i D_i 256^i of the group's digits.
// One reduction step brings V (below 2^18 n) to L limbs below 2n first, so that
// L limb steps remain: 2L^2 + L wide multiplies.  The digits are put together
// with shifts and adds, which run beside the multiplies on the ALU.
template <int L>
__device__ __forceinline__ void fold_digits(Res<L>& P, const uint32_t (&D)[L][4], const uint32_t* n, uint32_t ninv) {
    uint32_t v[L + 1];
    uint32_t c = 0;
#pragma unroll
    for (int j = 0; j < L; ++j) {
        // c + D0 + D1 2^8 + D2 2^16 + D3 2^24: c < 2^19, the rest below 2^49
        const uint32_t a = D[j][0] + c;
        asm("{\n\t.reg .u32 s1, h1, s2, h2, s3, h3;\n\t"
            "shl.b32 s1, %3, 8;\n\t"
            "shr.u32 h1, %3, 24;\n\t"
            "shl.b32 s2, %4, 16;\n\t"
            "shr.u32 h2, %4, 16;\n\t"
            "shl.b32 s3, %5, 24;\n\t"
            "shr.u32 h3, %5, 8;\n\t"
            "add.cc.u32 s1, s1, %2;\n\t"
            "addc.u32 h1, h1, h2;\n\t"
            "add.cc.u32 s1, s1, s2;\n\t"
            "addc.u32 h1, h1, h3;\n\t"
            "add.cc.u32 %0, s1, s3;\n\t"
            "addc.u32 %1, h1, 0;\n\t}"
            : "=r"(v[j]), "=r"(c) : "r"(a), "r"(D[j][1]), "r"(D[j][2]), "r"(D[j][3]));
    }
    v[L] = c;
    // (V + m n) / 2^32
    uint32_t y[L];
    const uint32_t m = v[0] * ninv;
    uint64_t A = (uint64_t)m * n[0] + v[0];
#pragma unroll
    for (int k = 1; k < L; ++k) {
        A = (uint64_t)m * n[k] + v[k] + (A >> 32);
        y[k - 1] = (uint32_t)A;
    }
    y[L - 1] = v[L] + (uint32_t)(A >> 32);
    uint32_t t[L];
#pragma unroll
    for (int k = 0; k < L; ++k) t[k] = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) limb_step<L>(t, P, y[k], n, ninv);
#pragma unroll
    for (int k = 0; k < L; ++k) P.w[k] = t[k];
}

template <int L> struct PartOf { typedef uint4 T; };
template <> struct PartOf<2> { typedef uint2 T; };
template <int L> __device__ __forceinline__ typename PartOf<L>::T part_pack(const Res<L>& r);
template <> __device__ __forceinline__ uint2 part_pack<2>(const Res<2>& r) { return make_uint2(r.w[0], r.w[1]); }
template <> __device__ __forceinline__ uint4 part_pack<3>(const Res<3>& r) { return make_uint4(r.w[0], r.w[1], r.w[2], 0); }
template <> __device__ __forceinline__ uint4 part_pack<4>(const Res<4>& r) { return make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]); }
__device__ __forceinline__ void part_unpack(const uint2& v, Res<2>& r) { r.w[0] = v.x; r.w[1] = v.y; }
__device__ __forceinline__ void part_unpack(const uint4& v, Res<3>& r) { r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; }
__device__ __forceinline__ void part_unpack(const uint4& v, Res<4>& r) { r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w; }
template <int L>
__device__ __forceinline__ Res<L> res_of(const uint4& v) {
    Res<L> r;
    r.w[0] = v.x; r.w[1] = v.y;
    if (L > 2) r.w[2 < L ? 2 : 0] = v.z;
    if (L > 3) r.w[3 < L ? 3 : 0] = v.w;
    return r;
}

// One CTA per item, one CTA per SM.  Warps 0-15 are the epilogue (four
// warpgroups, each a quarter of the tile's rows), warp 16 brings the operand
// blocks in, warp 17 issues the matrix instructions.  The row constants (128 KB) stay
// for the item; group tiles stream through 16 KB stages; the accumulator is
// double-buffered (2 x 256 tensor-memory columns), so that the epilogue of one
// tile runs beside the next tile's product.
//
// TAIL = 1: the groups are those of a bucket's consecutive-integer tail, lane
// after lane, and a row leaves out those past its own end (info); an item is a
// row tile with the group tiles that some row of it needs, and each warp writes
// one product per row.
template <int L, int TAIL>
__global__ void __launch_bounds__(TG_THREADS, 1)
k_tensor_gemm(const TensorDesc* __restrict__ desc, const TensorSec* __restrict__ secs,
              const TensorItem* __restrict__ items, const LaneRun* __restrict__ lr, const RowInfo* __restrict__ info,
              const RowMod* __restrict__ mods,
              const uint8_t* __restrict__ w, const uint8_t* __restrict__ consts, const uint4* __restrict__ ones,
              typename PartOf<L>::T* __restrict__ part, uint32_t* __restrict__ err, uint64_t wait_ns) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t sB = base, sA = base + TN_KB * TG_B_BYTES;
    const uint32_t bars = sA + TG_STAGES * TG_A_BYTES;
    const uint32_t bFull = bars, bEmpty = bars + 8 * TG_STAGES, bConst = bEmpty + 8 * TG_STAGES;
    const uint32_t bAccFull = bConst + 8, bAccEmpty = bAccFull + 16, bLast = bAccEmpty + 16, sTmem = bLast + 8;
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TensorItem it = items[blockIdx.x];
    const TensorSec sec = secs[it.sec];
    const TensorDesc& d = desc[sec.task];
    const uint32_t tn = TAIL ? it.ncb : sec.tn, ncb = TAIL ? 1 : it.ncb, ntiles = ncb * tn;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < TG_STAGES; ++s) { mbar_init(bFull + 8 * s, 1); mbar_init(bEmpty + 8 * s, 1); }
        mbar_init(bConst, 1);
        mbar_init(bLast, 1);
        for (uint32_t s = 0; s < 2; ++s) { mbar_init(bAccFull + 8 * s, 1); mbar_init(bAccEmpty + 8 * s, TG_EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (wid == TG_EPI_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(sTmem));
    bool ok = wait_ns != 0;       // with a limit of 0 no wait is waited for

    if (wid == TG_EPI_WARPS) {
        if (lane == 0) {
            const uint8_t* cs = consts + (uint64_t)(d.ct0 + it.tile) * TN_KB * TG_B_BYTES;
            mbar_expect(bConst, TN_KB * TG_B_BYTES);
            for (uint32_t k = 0; k < TN_KB; ++k) bulk_load(sB + k * TG_B_BYTES, cs + k * TG_B_BYTES, TG_B_BYTES, bConst);
            const uint8_t* src = w + (uint64_t)(sec.mt0 + it.cb0 * tn) * TN_KB * TG_A_BYTES;
            const uint32_t nblk = ntiles * TN_KB;
            uint32_t s = 0, ph = 0, issued = 0;
            for (; ok && issued < nblk; ++issued) {
                ok = mbar_wait(bEmpty + 8 * s, ph ^ 1, wait_ns);
                if (!ok) break;
                mbar_expect(bFull + 8 * s, TG_A_BYTES);
                bulk_load(sA + s * TG_A_BYTES, src + (uint64_t)issued * TG_A_BYTES, TG_A_BYTES, bFull + 8 * s);
                if (++s == TG_STAGES) { s = 0; ph ^= 1; }
            }
            // the copies in flight end before the shared memory goes, whoever gave up
            ok &= mbar_wait(bConst, 0, TG_DRAIN_NS);
            for (uint32_t k = issued > TG_STAGES ? issued - TG_STAGES : 0; k < issued; ++k)
                ok &= mbar_wait(bFull + 8 * (k % TG_STAGES), (k / TG_STAGES) & 1, TG_DRAIN_NS);
        }
    } else if (wid == TG_EPI_WARPS + 1) {
        if (lane == 0) {
            ok = ok && mbar_wait(bConst, 0, wait_ns);
            uint32_t s = 0, ph = 0;
            bool issued = false;
            for (uint32_t t = 0; t < ntiles && ok; ++t) {
                const uint32_t buf = t & 1;
                ok = mbar_wait(bAccEmpty + 8 * buf, ((t >> 1) & 1) ^ 1, wait_ns);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (uint32_t kb = 0; kb < TN_KB; ++kb) {
                    ok = mbar_wait(bFull + 8 * s, ph, wait_ns);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = smem_desc(sA + s * TG_A_BYTES), db = smem_desc(sB + kb * TG_B_BYTES);
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)       // 32 bytes of K each
                        mma_i8(tmem + buf * TN_N, da + 2 * k, db + 2 * k, TG_IDESC, (kb | k) != 0);
                    mma_commit(bEmpty + 8 * s);
                    issued = true;
                    if (++s == TG_STAGES) { s = 0; ph ^= 1; }
                }
                if (ok) mma_commit(bAccFull + 8 * buf);
            }
            // the matrix instructions end before the tensor memory goes (the epilogue,
            // which waits for the last tile, may have given up)
            if (issued) {
                mma_commit(bLast);
                ok &= mbar_wait(bLast, 0, TG_DRAIN_NS);
            }
        }
    } else {
        // rows of this warpgroup: a quarter of the tile's
        constexpr uint32_t RT = TN_N / (4 * L), RH = (RT + TG_WG - 1) / TG_WG;
        const uint32_t wg = wid >> 2, quarter = wid & 3;
        const uint32_t r0 = min(wg * RH, RT);
        uint32_t n[RH][L], ninv[RH];
        Res<L> P[RH];
        const uint32_t row0 = d.row_begin + it.tile * RT + r0;   // the thread's first row
        const uint32_t left = d.nrows - min(d.nrows, it.tile * RT + r0);
        const uint32_t live = min(left, min(RH, RT - r0));
#pragma unroll
        for (uint32_t r = 0; r < RH; ++r) {
            const RowMod m = mods[r < live ? row0 + r : d.row_begin];
#pragma unroll
            for (int k = 0; k < L; ++k) n[r][k] = m.n[k];
            ninv[r] = m.ninv;
        }
        uint32_t ends[TAIL ? RH : 1];              // groups of each row
        if (TAIL) {
#pragma unroll
            for (uint32_t r = 0; r < RH; ++r)
                ends[TAIL ? r : 0] = r < live ? (uint32_t)((info[row0 + r].Tp - d.T) / sec.g) : 0u;
        }
        const uint32_t taddr = tmem + (quarter << 21) + r0 * 4 * L;
        uint32_t t = 0;
        for (uint32_t cb = it.cb0; cb < it.cb0 + ncb && ok; ++cb) {
#pragma unroll
            for (uint32_t r = 0; r < RH; ++r) P[r] = res_of<L>(ones[(d.ct0 + it.tile) * RT + (r < live ? r0 + r : 0)]);
            for (uint32_t k = 0; k < tn; ++k, ++t) {
                const uint32_t buf = t & 1;
                ok = mbar_wait(bAccFull + 8 * buf, (t >> 1) & 1, wait_ns);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = taddr + buf * TN_N;
                uint32_t D[2][L][4];
#pragma unroll
                for (int j = 0; j < L; ++j) tmem_ld4(D[0][j], ta + 4 * j);
#pragma unroll
                for (uint32_t r = 0; r < RH; ++r) {
                    tmem_wait_ld<L>(D[r & 1]);
                    if (r + 1 < RH) {
                        // the last warpgroup may have fewer rows: it then reads one it has twice
                        const uint32_t nr = (r0 + r + 1 < RT) ? r + 1 : 0;
#pragma unroll
                        for (int j = 0; j < L; ++j) tmem_ld4(D[(r + 1) & 1][j], ta + nr * 4 * L + 4 * j);
                    }
                    if (TAIL) {
                        Res<L> Q = P[r];
                        fold_digits<L>(Q, D[r & 1], n[r], ninv[r]);
                        const bool take = k * TN_M + quarter * 32 + lane < ends[TAIL ? r : 0];
#pragma unroll
                        for (int j = 0; j < L; ++j) P[r].w[j] = take ? Q.w[j] : P[r].w[j];
                    } else {
                        fold_digits<L>(P[r], D[r & 1], n[r], ninv[r]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bAccEmpty + 8 * buf);
            }
            if (!ok) break;
            const uint32_t slot = TAIL ? quarter : lr[sec.run0 + cb * TN_M + quarter * 32 + lane].slot;
            bool write = slot != RUN_NONE;
            if (TAIL || sec.reduce) {
                // lanes of one label lie side by side: the first of them collects
                // their product (segmented reduction over the warp)
#pragma unroll 1
                for (uint32_t off = 1; off < 32; off <<= 1) {
                    const uint32_t other = __shfl_down_sync(0xffffffffu, slot, off);
                    const bool same = lane + off < 32 && other == slot;
#pragma unroll
                    for (uint32_t r = 0; r < RH; ++r) {
                        Res<L> y;
#pragma unroll
                        for (int k = 0; k < L; ++k) y.w[k] = __shfl_down_sync(0xffffffffu, P[r].w[k], off);
                        const Res<L> z = mont_mul<L>(P[r], y, n[r], ninv[r]);
#pragma unroll
                        for (int k = 0; k < L; ++k) P[r].w[k] = same ? z.w[k] : P[r].w[k];
                    }
                }
                const uint32_t before = __shfl_up_sync(0xffffffffu, slot, 1);
                write = write && (lane == 0 || before != slot);
            }
            const uint64_t at = d.part0 + (uint64_t)slot * d.rows_pad + it.tile * RT + r0;
            if (write) {
#pragma unroll
                for (uint32_t r = 0; r < RH; ++r)
                    if (r < live) part[at + r] = part_pack<L>(P[r]);
            }
        }
    }
    if (!ok) atomicOr(err, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == TG_EPI_WARPS + 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ---------------------------------------------------------------------------
// Labels: slot products -> segments of 64 slots -> windows -> rows.
// ---------------------------------------------------------------------------

constexpr uint32_t TF_THREADS = 128;

// A *= P^d, d >= 1
template <int L>
__device__ __forceinline__ void fold_pow_small(Res<L>& A, const Res<L>& P, uint32_t d, const uint32_t* n, uint32_t ninv) {
    Res<L> Y = P;
    for (int b = 30 - __clz(d); b >= 0; --b) {
        Y = mont_mul<L>(Y, Y, n, ninv);
        if ((d >> b) & 1) Y = mont_mul<L>(Y, P, n, ninv);
    }
    A = mont_mul<L>(A, Y, n, ninv);
}

// One thread per (row, segment): rows are the fast index.  CTAs of a task:
// nseg x ceil(rows_pad / 128), rows inside.
template <int L>
__global__ void __launch_bounds__(TF_THREADS)
k_tensor_fold(const TensorDesc* __restrict__ desc, uint32_t ntask, const FoldSeg* __restrict__ segs,
              const RowMod* __restrict__ mods, const typename PartOf<L>::T* __restrict__ part,
              typename PartOf<L>::T* __restrict__ seg_part) {
    const TensorDesc& d = desc[task_of_block(desc, ntask, blockIdx.x, &TensorDesc::fold_blk0)];
    const uint32_t per = (d.rows_pad + TF_THREADS - 1) / TF_THREADS;
    const uint32_t b = blockIdx.x - d.fold_blk0;
    const uint32_t sg = b / per, r = (b % per) * TF_THREADS + threadIdx.x;
    if (r >= d.nrows) return;
    const FoldSeg fs = segs[d.seg0 + sg];
    const RowMod m = mods[d.row_begin + r];
    uint32_t n[L];
#pragma unroll
    for (int k = 0; k < L; ++k) n[k] = m.n[k];
    const typename PartOf<L>::T* p = part + d.part0 + (uint64_t)fs.slot0 * d.rows_pad + r;
    Res<L> X;
    part_unpack(p[0], X);
    for (uint32_t k = 1; k < fs.n; ++k) {
        Res<L> y;
        part_unpack(p[(uint64_t)k * d.rows_pad], y);
        X = mont_mul<L>(X, y, n, m.ninv);
    }
    seg_part[d.seg_part0 + (uint64_t)sg * d.rows_pad + r] = part_pack<L>(X);
}

// One thread per (row, window j, block b of 32 digits): prod A_{j,d}^d over the
// block's digits d = 32 b + o, as prod A^o (running products from the top digit
// down) times (prod A)^(32 b).  Blocks keep the serial chain at about 80 products.
// lab_seg[lab_seg0 + l] .. lab_seg[lab_seg0 + l + 1]: segments of label l (task-relative).
template <int L>
__global__ void __launch_bounds__(TF_THREADS)
k_tensor_windows(const TensorDesc* __restrict__ desc, uint32_t ntask, const uint32_t* __restrict__ lab_seg,
                 const RowMod* __restrict__ mods, const uint4* __restrict__ ones,
                 const typename PartOf<L>::T* __restrict__ seg_part, typename PartOf<L>::T* __restrict__ win) {
    const TensorDesc& d = desc[task_of_block(desc, ntask, blockIdx.x, &TensorDesc::row_blk0)];
    const uint32_t nb = (1u << d.w) / TN_DIGITS, j = blockIdx.y / nb, b = blockIdx.y % nb;
    const uint32_t r = (blockIdx.x - d.row_blk0) * TF_THREADS + threadIdx.x;
    if (j >= d.nwin || r >= d.nrows) return;
    const uint32_t row = d.row_begin + r;
    const RowMod m = mods[row];
    uint32_t n[L];
#pragma unroll
    for (int k = 0; k < L; ++k) n[k] = m.n[k];
    Res<L> S = res_of<L>(ones[d.ct0 * tn_rows(L) + r]), R = S;
    const uint32_t* ls = lab_seg + d.lab_seg0 + (j << d.w) + b * TN_DIGITS;
    bool any = false;
    for (int o = TN_DIGITS - 1; o >= 0; --o) {
        for (uint32_t s = ls[o]; s < ls[o + 1]; ++s) {
            Res<L> y;
            part_unpack(seg_part[d.seg_part0 + (uint64_t)s * d.rows_pad + r], y);
            S = any ? mont_mul<L>(S, y, n, m.ninv) : y;
            any = true;
        }
        if (any && o) R = mont_mul<L>(R, S, n, m.ninv);
    }
    if (any && b) fold_pow_small<L>(R, S, b * TN_DIGITS, n, m.ninv);
    win[d.win0 + ((uint64_t)j * nb + b) * d.rows_pad + r] = part_pack<L>(R);
}

// acc[row] *= prod_j (window j)^(2^(w j)), windows from the top (Horner)
template <int L>
__global__ void __launch_bounds__(TF_THREADS)
k_tensor_rows(const TensorDesc* __restrict__ desc, uint32_t ntask, const RowMod* __restrict__ mods,
              const typename PartOf<L>::T* __restrict__ win, uint4* __restrict__ acc) {
    const TensorDesc& d = desc[task_of_block(desc, ntask, blockIdx.x, &TensorDesc::row_blk0)];
    const uint32_t r = (blockIdx.x - d.row_blk0) * TF_THREADS + threadIdx.x;
    if (r >= d.nrows) return;
    const uint32_t row = d.row_begin + r;
    const RowMod m = mods[row];
    uint32_t n[L];
#pragma unroll
    for (int k = 0; k < L; ++k) n[k] = m.n[k];
    const uint32_t nb = (1u << d.w) / TN_DIGITS;
    const typename PartOf<L>::T* p = win + d.win0 + r;
    Res<L> X;
    for (int j = (int)d.nwin - 1; j >= 0; --j) {
        const bool top = j == (int)d.nwin - 1;
        for (uint32_t k = 0; k < d.w && !top; ++k) X = mont_mul<L>(X, X, n, m.ninv);
        for (uint32_t b = 0; b < nb; ++b) {
            Res<L> y;
            part_unpack(p[((uint64_t)j * nb + b) * d.rows_pad], y);
            X = top && b == 0 ? y : mont_mul<L>(X, y, n, m.ninv);
        }
    }
    // acc * (X R) / R: the product itself, with no power of two left over
    const Res<L> A = mont_mul<L>(res_of<L>(acc[row]), X, n, m.ninv);
    acc[row] = make_uint4(A.w[0], A.w[1], L > 2 ? A.w[2 < L ? 2 : 0] : 0, L > 3 ? A.w[3 < L ? 3 : 0] : 0);
}

// The rest of a row's tail, fewer than g integers after its last whole group, one
// cell each; then acc *= that, the four products of the groups, and the power of
// two that the cells took out.
template <int L>
__global__ void __launch_bounds__(TF_THREADS)
k_tensor_tail_rows(const TensorDesc* __restrict__ desc, const TensorSec* __restrict__ secs, uint32_t ntask,
                   const RowInfo* __restrict__ info, const RowMod* __restrict__ mods, const uint4* __restrict__ ones,
                   const typename PartOf<L>::T* __restrict__ part, uint4* __restrict__ acc) {
    const uint32_t ti = task_of_block(desc, ntask, blockIdx.x, &TensorDesc::row_blk0);
    const TensorDesc& d = desc[ti];
    const uint32_t r = (blockIdx.x - d.row_blk0) * TF_THREADS + threadIdx.x;
    if (r >= d.nrows) return;
    const uint32_t row = d.row_begin + r;
    const RowMod m = mods[row];
    uint32_t n[L];
#pragma unroll
    for (int k = 0; k < L; ++k) n[k] = m.n[k];
    const uint64_t Tp = info[row].Tp, len = Tp - d.T, g = secs[ti].g, whole = len / g * g;
    const Res<L> one = res_of<L>(ones[d.ct0 * tn_rows(L) + r]);
    Res<L> X = one;
    uint32_t bits = 0;
    for (uint64_t N = d.T + whole + 1; N <= Tp; ++N) {
        if (N < 0x80000000ull) {
            cell_w<L>(X, (uint32_t)N, n, m.ninv);
            bits += 32;
        } else {
            cell64<L>(X, N, n, m.ninv);
            bits += 64;
        }
    }
    Res<L> two = one;
    dbl_mod<L>(two, n);
    X = mont_mul<L>(X, mont_pow<L>(two, (u128)bits, one, n, m.ninv), n, m.ninv);
    if (whole) {
#pragma unroll 1
        for (uint32_t k = 0; k < TAIL_SLOTS; ++k) {
            Res<L> y;
            part_unpack(part[d.part0 + (uint64_t)k * d.rows_pad + r], y);
            X = mont_mul<L>(X, y, n, m.ninv);
        }
    }
    const Res<L> A = mont_mul<L>(res_of<L>(acc[row]), X, n, m.ninv);
    acc[row] = make_uint4(A.w[0], A.w[1], L > 2 ? A.w[2 < L ? 2 : 0] : 0, L > 3 ? A.w[3 < L ? 3 : 0] : 0);
}

// ---------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------

void launch_tensor_count(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const uint32_t* cols, uint32_t* counts,
                         cudaStream_t st) {
    k_tensor_count<<<nblocks, 256, 0, st>>>(d, ntask, cols, counts);
}
void launch_tensor_size(const TensorDesc* d, uint32_t ntask, const uint32_t* counts, TensorSize* size, cudaStream_t st) {
    k_tensor_layout<0><<<ntask, 256, 0, st>>>(d, counts, size, nullptr, nullptr, nullptr, nullptr);
}
void launch_tensor_layout(const TensorDesc* d, uint32_t ntask, const uint32_t* counts, uint32_t* cursor, LaneRun* runs,
                          FoldSeg* segs, uint32_t* lab_seg, cudaStream_t st) {
    k_tensor_layout<1><<<ntask, 256, 0, st>>>(d, counts, nullptr, cursor, runs, segs, lab_seg);
}
void launch_tensor_scatter(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const uint32_t* cols,
                           uint32_t* cursor, uint32_t* list, cudaStream_t st) {
    k_tensor_scatter<<<nblocks * TN_SCATTER, 256, 0, st>>>(d, ntask, cols, cursor, list);
}
void launch_tensor_build(const TensorSec* sec, uint32_t nsec, uint32_t nmt, const LaneRun* lr, const uint32_t* list,
                         uint8_t* w, cudaStream_t st) {
    k_tensor_build<<<nmt * (TN_M / TB_WARPS), TB_WARPS * 32, 0, st>>>(sec, nsec, lr, list, w);
}
template <int L>
static void consts_l(const TensorDesc* d, uint32_t ntask, uint32_t ntiles, const RowMod* mods, uint8_t* consts, uint4* ones,
                     cudaStream_t st) {
    constexpr uint32_t per = 256 / (TN_K / 16), ctas = (TN_N / (4 * L) + per - 1) / per;
    k_tensor_consts<L><<<ntiles * ctas, 256, 0, st>>>(d, ntask, mods, consts, ones);
}
void launch_tensor_consts(int L, const TensorDesc* d, uint32_t ntask, uint32_t ntiles, const RowMod* mods, uint8_t* consts,
                          uint4* ones, cudaStream_t st) {
    if (L == 2) consts_l<2>(d, ntask, ntiles, mods, consts, ones, st);
    else if (L == 3) consts_l<3>(d, ntask, ntiles, mods, consts, ones, st);
    else consts_l<4>(d, ntask, ntiles, mods, consts, ones, st);
}
template <int L, int TAIL>
static int gemm_l(uint32_t nitems, const TensorDesc* d, const TensorSec* sec, const TensorItem* items, const LaneRun* lr,
                  const RowInfo* info, const RowMod* mods, const uint8_t* w, const uint8_t* consts, const uint4* ones,
                  void* part, uint32_t* err, uint64_t wait_ns, cudaStream_t st) {
    if (cudaFuncSetAttribute(k_tensor_gemm<L, TAIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TG_SMEM) !=
        cudaSuccess)
        return -1;
    k_tensor_gemm<L, TAIL><<<nitems, TG_THREADS, TG_SMEM, st>>>(d, sec, items, lr, info, mods, w, consts, ones,
                                                                (typename PartOf<L>::T*)part, err, wait_ns);
    return 0;
}
int launch_tensor_gemm(int L, uint32_t nitems, const TensorDesc* d, const TensorSec* sec, const TensorItem* items,
                       const LaneRun* lr, const RowMod* mods, const uint8_t* w, const uint8_t* consts,
                       const uint4* ones, void* part, uint32_t* err, uint64_t wait_ns, cudaStream_t st) {
    if (L == 2) return gemm_l<2, 0>(nitems, d, sec, items, lr, nullptr, mods, w, consts, ones, part, err, wait_ns, st);
    if (L == 3) return gemm_l<3, 0>(nitems, d, sec, items, lr, nullptr, mods, w, consts, ones, part, err, wait_ns, st);
    return gemm_l<4, 0>(nitems, d, sec, items, lr, nullptr, mods, w, consts, ones, part, err, wait_ns, st);
}
void launch_tensor_tail_build(const TensorDesc* d, const TensorSec* sec, uint32_t nsec, uint32_t nmt, uint8_t* w,
                              cudaStream_t st) {
    k_tensor_tail_build<<<nmt * (TN_M / TB_WARPS), TB_WARPS * 32, 0, st>>>(d, sec, nsec, w);
}
int launch_tensor_tail_gemm(int L, uint32_t nitems, const TensorDesc* d, const TensorSec* sec, const TensorItem* items,
                            const RowInfo* info, const RowMod* mods, const uint8_t* w, const uint8_t* consts,
                            const uint4* ones, void* part, uint32_t* err, uint64_t wait_ns, cudaStream_t st) {
    if (L == 2) return gemm_l<2, 1>(nitems, d, sec, items, nullptr, info, mods, w, consts, ones, part, err, wait_ns, st);
    if (L == 3) return gemm_l<3, 1>(nitems, d, sec, items, nullptr, info, mods, w, consts, ones, part, err, wait_ns, st);
    return gemm_l<4, 1>(nitems, d, sec, items, nullptr, info, mods, w, consts, ones, part, err, wait_ns, st);
}
template <int L>
static void tail_rows_l(const TensorDesc* d, const TensorSec* sec, uint32_t ntask, uint32_t nblocks, const RowInfo* info,
                        const RowMod* mods, const uint4* ones, const void* part, uint4* acc, cudaStream_t st) {
    k_tensor_tail_rows<L><<<nblocks, TF_THREADS, 0, st>>>(d, sec, ntask, info, mods, ones,
                                                          (const typename PartOf<L>::T*)part, acc);
}
void launch_tensor_tail_rows(int L, const TensorDesc* d, const TensorSec* sec, uint32_t ntask, uint32_t nblocks,
                             const RowInfo* info, const RowMod* mods, const uint4* ones, const void* part, uint4* acc,
                             cudaStream_t st) {
    if (L == 2) tail_rows_l<2>(d, sec, ntask, nblocks, info, mods, ones, part, acc, st);
    else if (L == 3) tail_rows_l<3>(d, sec, ntask, nblocks, info, mods, ones, part, acc, st);
    else tail_rows_l<4>(d, sec, ntask, nblocks, info, mods, ones, part, acc, st);
}
template <int L>
static void fold_l(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const FoldSeg* segs, const RowMod* mods,
                   const void* part, void* seg_part, cudaStream_t st) {
    typedef typename PartOf<L>::T T;
    k_tensor_fold<L><<<nblocks, TF_THREADS, 0, st>>>(d, ntask, segs, mods, (const T*)part, (T*)seg_part);
}
void launch_tensor_fold(int L, const TensorDesc* d, uint32_t ntask, uint32_t nblocks, const FoldSeg* segs,
                        const RowMod* mods, const void* part, void* seg_part, cudaStream_t st) {
    if (L == 2) fold_l<2>(d, ntask, nblocks, segs, mods, part, seg_part, st);
    else if (L == 3) fold_l<3>(d, ntask, nblocks, segs, mods, part, seg_part, st);
    else fold_l<4>(d, ntask, nblocks, segs, mods, part, seg_part, st);
}
template <int L>
static void combine_l(const TensorDesc* d, uint32_t ntask, uint32_t nblocks, uint32_t max_blocks, const uint32_t* lab_seg,
                      const RowMod* mods, const uint4* ones, const void* seg_part, void* win, uint4* acc, cudaStream_t st) {
    typedef typename PartOf<L>::T T;
    k_tensor_windows<L><<<dim3(nblocks, max_blocks), TF_THREADS, 0, st>>>(d, ntask, lab_seg, mods, ones, (const T*)seg_part,
                                                                       (T*)win);
    k_tensor_rows<L><<<nblocks, TF_THREADS, 0, st>>>(d, ntask, mods, (const T*)win, acc);
}
void launch_tensor_combine(int L, const TensorDesc* d, uint32_t ntask, uint32_t nblocks, uint32_t max_blocks,
                           const uint32_t* lab_seg, const RowMod* mods, const uint4* ones, const void* seg_part,
                           void* win, uint4* acc, cudaStream_t st) {
    if (L == 2) combine_l<2>(d, ntask, nblocks, max_blocks, lab_seg, mods, ones, seg_part, win, acc, st);
    else if (L == 3) combine_l<3>(d, ntask, nblocks, max_blocks, lab_seg, mods, ones, seg_part, win, acc, st);
    else combine_l<4>(d, ntask, nblocks, max_blocks, lab_seg, mods, ones, seg_part, win, acc, st);
}

}  // namespace wl
