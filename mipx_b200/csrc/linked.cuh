// Linked restart cycle: the N PDHG iterations between two checks as one launch
// without a barrier between its steps.
//
// An LP whose matrix stays in the chip's caches spends its iteration on what
// lies between the two step kernels, not on their work: launch gaps, and a
// chain of L2 latencies for a matrix that every launch starts again with an
// empty L1.  Here one cooperative grid keeps its rows and columns for the whole
// cycle -- a warp reads the same slices every iteration, from L1 -- and a step's
// results travel as cells, a value with the number of the iteration that made
// it.  A gather loads the cell and, if its number is not yet the wanted one,
// loads it again: no flag, no fence, no grid-wide wait, and a row starts as soon
// as its own entries are there.
//
// What bounds it: the way through L2 (590 cycles from store to load on one die,
// 1,000 across, twice per iteration), the sum of a row in entry order (12 cycles
// per entry), and L1's tag stage, which takes one of a warp's 32 scattered cells
// per clock -- so a slice's rows are spread over several warps with 2-8 lanes
// per row.  Counters at 2,000 x 5,000: L1 busy 50 % of the cycle, L2 32 %, DRAM
// 0.03 %, loads waited for in 4 of 10 issue slots.  Measured (B200, FP64, us per iteration, the steps alone, launches ->
// linked): 400 x 1,000 7.2 -> 2.5, 2,000 x 5,000 8.0 -> 3.0, 6,000 x 15,000
// 8.7 -> 3.9, 20,000 x 50,000 10.3 -> 8.4.  (Before that: one 8-16 CTA cluster
// with the vectors copied to every SM through distributed shared memory, 6.0 at
// 2,000 x 5,000: a copy arrives at 12-22 bytes per clock and SM.)
//
// Why no cell is overwritten too early: x_j is read by the rows i with an entry
// in column j, and column j's next value needs y_i of the same rows i, each of
// which its owner publishes after its own reads (its value depends on them).
// Entries of value 0 (padding among them) are not waited for and add nothing.  The
// step kernels add 0 x[c] for theirs: the same bits while x is finite.
// Why it always ends: a warp runs its columns' step k, then its rows' step k,
// and waits only for cells of strictly earlier half-steps; every block is
// resident (cooperative launch).  Should a block be kept from running all the
// same, waits end after LinkWait::polls loads, set the error word and leave, and
// a launch that finds it set does nothing.
//
// Every row is summed in the order of the per-step kernels (sellDot, rowDotU +
// groupSum) and updated by the same expressions.  Which LPs it runs: link_plan.hpp.
#pragma once

#include "kernels.cuh"

namespace pdlpx {

constexpr int kLinkPolls = 1 << 22;  // ~2 s of L2 round trips
inline int linkPolls(int option) { return option > 0 ? option : kLinkPolls; }

// How the waits of a launch end when what they wait for does not come.
struct LinkWait {
    int* err;   // error word, set by the first wait that runs out
    int polls;  // loads of a cell until then
};
__device__ __forceinline__ bool linkFailed(const LinkWait& w) { return *reinterpret_cast<volatile int*>(w.err) != 0; }

constexpr int kLinkU = 4;  // cells per lane per round
// Sleep between polls (ns) beside CSR rows: their LPs have few rows or columns that
// everything gathers, and warps polling the same few lines of L2 hold up the
// stores to them.  Transportation 97 x 131 3.80 -> 3.30 us per iteration, 150 x 150
// 5.71 -> 4.72 (B200); LPs without such rows lose 0-4 % by it.
constexpr int kLinkNap = 80;

// Device time of the last cycle: all of it (globaltimer), and the SM clocks that
// a row's warp waited for and summed new x (the primal half-steps) and a
// column's warp new y (the dual half-steps).
struct LinkTime {
    unsigned long long ns;
    long long primal_clk, dual_clk;
    int iters;
    int pad;
};

// ---- cells ---------------------------------------------------------------------
// One 8-byte word per 32 bits of value, each with the number beside it, so every
// word says by itself whether it is the wanted one.
template <class X>
struct LinkCell;
template <>
struct __align__(16) LinkCell<double> {
    unsigned long long w[2];  // low, high half of the value | number << 32
};
template <>
struct __align__(8) LinkCell<float> {
    unsigned long long w[1];
};
__device__ __forceinline__ unsigned long long linkWord(unsigned v, unsigned tag) {
    unsigned long long w;
    asm("mov.b64 %0, {%1, %2};" : "=l"(w) : "r"(v), "r"(tag));
    return w;
}
__device__ __forceinline__ unsigned linkTag(unsigned long long w) { return static_cast<unsigned>(w >> 32); }
__device__ __forceinline__ void linkStore(LinkCell<double>* c, double v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(c),
                 "l"(linkWord(static_cast<unsigned>(__double2loint(v)), tag)),
                 "l"(linkWord(static_cast<unsigned>(__double2hiint(v)), tag))
                 : "memory");
}
__device__ __forceinline__ void linkStore(LinkCell<float>* c, float v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(c), "l"(linkWord(__float_as_uint(v), tag)) : "memory");
}
// A cell in registers, loaded again unless it is the wanted one (predicated, so
// that the loads of a round stay in flight together).  A load's elements are the
// 64-bit words that linkStore writes: only within an element is a value sure to
// come with its own number -- the elements of a vector load are accesses of their
// own, in no given order.
template <class X>
struct LinkReg;
template <>
struct LinkReg<double> {
    unsigned long long w0, w1;
    __device__ __forceinline__ void set(unsigned tag) { w0 = w1 = linkWord(0u, tag); }
    __device__ __forceinline__ void load(const LinkCell<double>* c, unsigned tag) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, %5;\n\tsetp.ne.or.u32 p, %4, %5, p;\n\t"
            "@p ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n\t}"
            : "+l"(w0), "+l"(w1)
            : "l"(c), "r"(linkTag(w0)), "r"(linkTag(w1)), "r"(tag)
            : "memory");
    }
    __device__ __forceinline__ bool ready(unsigned tag) const { return linkTag(w0) == tag && linkTag(w1) == tag; }
    __device__ __forceinline__ double value() const {
        return __hiloint2double(static_cast<int>(static_cast<unsigned>(w1)), static_cast<int>(static_cast<unsigned>(w0)));
    }
};
template <>
struct LinkReg<float> {
    unsigned long long w0;
    __device__ __forceinline__ void set(unsigned tag) { w0 = linkWord(0u, tag); }
    __device__ __forceinline__ void load(const LinkCell<float>* c, unsigned tag) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, %3;\n\t"
            "@p ld.relaxed.gpu.global.b64 %0, [%1];\n\t}"
            : "+l"(w0)
            : "l"(c), "r"(linkTag(w0)), "r"(tag)
            : "memory");
    }
    __device__ __forceinline__ bool ready(unsigned tag) const { return linkTag(w0) == tag; }
    __device__ __forceinline__ float value() const { return __uint_as_float(static_cast<unsigned>(w0)); }
};

// The cells x[c[u]] of iteration `tag`, loaded until all of the warp's are
// there; entries with value 0 are not waited for and give 0.  The warp polls
// together: with lanes that leave the loop one by one the same kernel took 5-10
// times as long.  NAP: nanoseconds of sleep between polls.  False when the wait
// ran out.
template <int U, int NAP, class V, class X>
__device__ __forceinline__ bool linkGather(const LinkCell<X>* __restrict__ x, const int (&c)[U], const V (&v)[U],
                                           unsigned tag, X (&g)[U], const LinkWait& wait) {
    LinkReg<X> r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u].set(v[u] == V(0) ? tag : ~tag);
    for (int polls = 0;;) {
#pragma unroll
        for (int u = 0; u < U; ++u) r[u].load(x + c[u], tag);
        bool ready = true;
#pragma unroll
        for (int u = 0; u < U; ++u) ready = ready && r[u].ready(tag);
        if (__all_sync(0xffffffffu, ready)) break;
        if constexpr (NAP > 0) __nanosleep(NAP);
        if ((++polls & 1023) == 0 || polls >= wait.polls) {
            const bool out = polls >= wait.polls || linkFailed(wait);
            if (__any_sync(0xffffffffu, out)) {
                atomicExch(wait.err, 1);
                return false;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) g[u] = r[u].value();
    return true;
}

// One slice's rows with L lanes each (32 / L rows per warp): a lane gathers
// every L-th entry of row r of the slice, and the entries go into the sum one by
// one in sellDot's order, handed round by shuffles.
template <int L, int NAP = 0, class V, class X>
__device__ __forceinline__ double linkSellDot(const int* __restrict__ idx, const V* __restrict__ val, int2 h, int r,
                                              int lane, const LinkCell<X>* x, unsigned tag, const LinkWait& wait, bool& ok) {
    const int q = lane % L;
    const int* ip = idx + h.x + r;
    const V* vp = val + h.x + r;
    double acc = 0.0;
    for (int k0 = 0; k0 < h.y; k0 += L * kLinkU) {
        int c[kLinkU];
        V v[kLinkU];
        X g[kLinkU];
#pragma unroll
        for (int u = 0; u < kLinkU; ++u) {
            const int k = k0 + u * L + q;
            const bool in = k < h.y;
            c[u] = in ? __ldg(ip + k * kSlice) : 0;
            v[u] = in ? __ldg(vp + k * kSlice) : V(0);
        }
        ok = linkGather<kLinkU, NAP>(x, c, v, tag, g, wait) && ok;
#pragma unroll
        for (int u = 0; u < kLinkU; ++u) {
            if (k0 + u * L >= h.y) break;  // the same in every lane
            if constexpr (L == 1) {
                acc += static_cast<double>(v[u]) * static_cast<double>(g[u]);
            } else {
#pragma unroll
                for (int w = 0; w < L; ++w)
                    acc += static_cast<double>(__shfl_sync(0xffffffffu, v[u], w, L)) *
                           static_cast<double>(__shfl_sync(0xffffffffu, g[u], w, L));
            }
        }
    }
    return acc;
}

// rowDotU<G, U> + groupSum<G> with a warp standing in for the G lanes (G <= 32:
// 32 / G rows per warp at once; above, G / 32 virtual warps one after another,
// added in warp order).  Every lane of a row's group returns its sum.
template <int U, class V, class X>
__device__ __forceinline__ double linkLaneSum(int b, int e, int first, int G, const int* __restrict__ idx,
                                              const V* __restrict__ val, const LinkCell<X>* x, unsigned tag, const LinkWait& wait,
                                              bool& ok) {
    double s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = 0.0;
    // eight cells in flight: two of rowDotU's rounds of four, or one of eight
    constexpr int W = 8;
    const int rounds = __reduce_max_sync(0xffffffffu, (e - b + W * G - 1) / (W * G));
    for (int k0 = b + first, q = 0; q < rounds; ++q, k0 += W * G) {
        int c[W];
        V v[W];
        X g[W];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const int k = k0 + u * G;
            const bool in = k < e;
            c[u] = in ? __ldg(idx + k) : 0;
            v[u] = in ? __ldg(val + k) : V(0);
        }
        ok = linkGather<W, kLinkNap>(x, c, v, tag, g, wait) && ok;
#pragma unroll
        for (int u = 0; u < W; ++u) s[u % U] += static_cast<double>(v[u]) * static_cast<double>(g[u]);
    }
    double t = s[0];
#pragma unroll
    for (int u = 1; u < U; ++u) t += s[u];
    return t;
}
template <class V, class X>
__device__ __forceinline__ double linkRowDot(int b, int e, int lane, int G, int U, const int* __restrict__ idx,
                                             const V* __restrict__ val, const LinkCell<X>* x, unsigned tag, const LinkWait& wait,
                                             bool& ok) {
    double t = 0.0;
    const int vw = G <= 32 ? 1 : G / 32;
    for (int w = 0; w < vw; ++w) {
        const int first = G <= 32 ? lane % G : w * 32 + lane;
        double s = U == 8 ? linkLaneSum<8>(b, e, first, G, idx, val, x, tag, wait, ok)
                          : linkLaneSum<4>(b, e, first, G, idx, val, x, tag, wait, ok);
        for (int off = min(G, 32) / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        t = w == 0 ? s : t + s;
    }
    return t;
}

// One matrix side: its long rows [0, nl) as CSR, the rest sliced ELL (lanes 0)
// or CSR.  A unit is one warp's work: a long row, 32 / L rows of a slice, or
// the CSR rows of one warp.
template <class T>
struct LinkSide {
    const int2* hdr;
    const int* idx;
    const T* val;
    const int* ptr;
    const int* cidx;
    const T* cval;
    int rows, nl;
    int lanes, unroll;    // CSR rows past nl: lanes per row, sums per lane (rowDotU)
    int llanes, lunroll;  // long rows
    int units;            // linkUnits with the kernel's lanes per sliced-ELL row
};
inline int linkUnits(int rows, int nl, int lanes, int sub) {
    const int per = lanes == 0 ? kSlice / sub : (lanes < 32 ? 32 / lanes : 1);
    return nl + (rows - nl + per - 1) / per;
}

template <class T>
struct LinkArgs {
    IterArgs<T> it;
    LinkSide<T> P, D;  // columns (A^T), rows (A)
    LinkCell<T>*x, *y;
    LinkWait wait;
    LinkTime* time;
};

// Sum of this lane's row of unit u (L lanes per sliced-ELL row).
template <int L, bool CSR, class T, class X>
__device__ __forceinline__ double linkUnitDot(const LinkSide<T>& a, int u, int lane, const LinkCell<X>* x, unsigned tag,
                                              const LinkWait& wait, bool& ok) {
    if (!CSR || (u >= a.nl && a.lanes == 0)) {
        const int v = u - a.nl;
        return linkSellDot<L, CSR ? kLinkNap : 0>(a.idx, a.val, __ldg(a.hdr + v / L), v % L * (32 / L) + lane / L, lane, x, tag, wait, ok);
    }
    const bool lng = u < a.nl;
    const int G = lng ? a.llanes : a.lanes, W = lng ? a.lunroll : a.unroll;
    const int per = lng || G >= 32 ? 1 : 32 / G;
    const int r = lng ? u : a.nl + (u - a.nl) * per + (per > 1 ? lane / G : 0);
    const bool in = r < a.rows;
    const int b = in ? __ldg(a.ptr + r) : 0, e = in ? __ldg(a.ptr + r + 1) : 0;
    return linkRowDot(b, e, lane, G, W, a.cidx, a.cval, x, tag, wait, ok);
}
// The row this lane updates of unit u (-1: none).
template <int L, bool CSR, class T>
__device__ __forceinline__ int linkUnitRow(const LinkSide<T>& a, int u, int lane) {
    if (CSR && u < a.nl) return lane == 0 ? u : -1;
    const int G = !CSR || a.lanes == 0 ? L : min(a.lanes, 32);
    const int r = a.nl + (u - a.nl) * (32 / G) + lane / G;
    return r < a.rows && lane % G == 0 ? r : -1;
}

// LP, LD: lanes per sliced-ELL row of the columns / rows; CSR: some rows are CSR
// (else both sides are sliced ELL throughout).
template <int LP, int LD, bool CSR, class T>
__device__ __forceinline__ void linkedCycle(const LinkArgs<T>& a) {
    const IterArgs<T>& p = a.it;
    const DevState* st = p.st;
    const bool failed = linkFailed(a.wait);
    if (st->done || st->prec != precTag<T>() || failed) return;
    const int cur = st->phase == 0 ? st->total : st->polish_count;
    const int lim = st->phase == 0 ? p.max_iter : p.polish_max_iter;
    const int iters = min(p.N, lim - cur);
    if (iters <= 0) return;
    const double step = st->step, pw = st->pw;
    const int inner = st->inner;
    // numbers go on from cycle to cycle, so no cell of an earlier cycle has a
    // wanted one (the cells are cleared when a solve starts)
    const unsigned base = static_cast<unsigned>(st->checks) * static_cast<unsigned>(p.N + 1) + 1u;

    const int lane = static_cast<int>(threadIdx.x) & 31;
    // neighbouring units on different blocks
    const int wid = static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) * (static_cast<int>(threadIdx.x) >> 5);
    const int nw = static_cast<int>(gridDim.x) * (static_cast<int>(blockDim.x) >> 5);
    const int uP = a.P.units, uD = a.D.units;
    // the rows' units follow the columns', so that they fall on other warps
    const int firstD = ((wid - uP) % nw + nw) % nw;

    for (int u = firstD; u < uD; u += nw) {
        const int i = linkUnitRow<LD, CSR>(a.D, u, lane);
        if (i < 0) continue;
        if constexpr (sizeof(T) == 4)
            linkStore(a.y + i, p.yg[i], base);
        else
            linkStore(a.y + i, p.yc[i], base);
    }
    unsigned long long t0 = 0;
    long long clk = 0, dclk = 0, pclk = 0;
    const bool dclock = wid == 0 && lane == 0, pclock = firstD == 0 && lane == 0;
    if (dclock) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    bool ok = true;
    for (int it = 1; it <= iters; ++it) {
        const bool last = it == iters;
        const int k = inner + it;
        const unsigned tag = base + static_cast<unsigned>(it);
        const double lam = static_cast<double>(k) / static_cast<double>(k + 1);
        if (dclock) clk = clock64();
        for (int u = wid; u < uP; u += nw) {
            // everything the step needs beside the sum, before the wait for y
            const int j = linkUnitRow<LP, CSR>(a.P, u, lane);
            ColPack<T> q{};
            double xcd = 0.0, xi = 0.0, tau = 0.0;
            if (j >= 0) {
                q = p.cp[j];
                xcd = p.xc[j];
                xi = static_cast<double>(p.xi[j]);
                tau = step * static_cast<double>(q.tau) / pw;
            }
            const double s = linkUnitDot<LP, CSR>(a.P, u, lane, a.y, tag - 1u, a.wait, ok);
            if (dclock && u == 0) dclk += clock64() - clk;
            if (j < 0) continue;
            double xh, xr;
            const double xn = primalValues<T>(q, xcd, xi, s, tau, lam, xh, xr);
            linkStore(a.x + j, static_cast<T>(xr), tag);
            p.xc[j] = xn;
            if (last) p.xh[j] = static_cast<T>(xh);
        }
        __syncwarp();
        if (pclock) clk = clock64();
        for (int u = firstD; u < uD; u += nw) {
            const int i = linkUnitRow<LD, CSR>(a.D, u, lane);
            RowPack<T> q{};
            double ycd = 0.0, yi = 0.0;
            if (i >= 0) {
                q = p.rp[i];
                ycd = p.yc[i];
                yi = static_cast<double>(p.yi[i]);
            }
            const double s = linkUnitDot<LD, CSR>(a.D, u, lane, a.x, tag, a.wait, ok);
            if (pclock && u == 0) pclk += clock64() - clk;
            if (i < 0) continue;
            double py;
            const double yn = dualValues<T>(q, ycd, yi, s, step, pw, lam, py);
            linkStore(a.y + i, static_cast<T>(yn), tag);
            p.yc[i] = yn;
            if constexpr (sizeof(T) == 4) {
                if (last) p.yg[i] = static_cast<float>(yn);
            }
            if (last) p.yh[i] = static_cast<T>(py);
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, !ok)) return;
    }
    if (dclock) {
        unsigned long long t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        a.time->ns = t1 - t0;
        a.time->dual_clk = dclk;
        a.time->iters = iters;
    }
    if (pclock) a.time->primal_clk = pclk;
}

}  // namespace pdlpx
