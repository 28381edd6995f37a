// Restart cycle of a tiny LP in one block: every warp owns one 32-row slice of one
// side, whose entries, constants and current iterates it keeps in registers for
// the whole cycle; y and x_refl lie in shared memory between two barriers.
//
// What bounds it is one chain per iteration: a gather from shared memory (29
// cycles), a row's multiply-adds in entry order (12 each), the update and a
// barrier, on each side.  Spread over the SMs, the linked cycle pays two ways
// through L2 instead.  Measured (B200, us per iteration with checks every 2,000,
// FP32 values, launches -> this): 20 x 40 5.8 -> 0.8, 60 x 150 6.2 -> 1.0 (linked
// 2.1), 90 x 250 7.0 -> 1.2 (linked 2.3); FP64 5.4 -> 0.7, 5.6 -> 0.9, 6.4 -> 1.1.
//
// Sums and updates are those of the step kernels, in their order: the same bits.
#pragma once

#include "linked.cuh"

namespace pdlpx {

constexpr int kTinyWarps = 12;   // slices of both sides; 168 registers per thread
constexpr int kTinyShort = 16;   // most entries of a row on one side ...
constexpr int kTinyLong = 40;    // ... and on the other

__device__ __forceinline__ void tinyBarrier(int threads) {
    // the roles' loops meet at it from different places
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// This lane's row of slice h, in registers; places are 16-bit.
template <int MAX, class T>
struct TinyRow {
    unsigned c[MAX / 2];
    T v[MAX];
    int len;
    __device__ __forceinline__ void load(const int* __restrict__ idx, const T* __restrict__ val, int2 h, int lane) {
        len = h.y;
#pragma unroll
        for (int u = 0; u < MAX; ++u) {
            const bool in = u < len;
            const unsigned k = in ? static_cast<unsigned>(__ldg(idx + h.x + u * kSlice + lane)) : 0u;
            if (u % 2 == 0)
                c[u / 2] = k;
            else
                c[u / 2] |= k << 16;
            v[u] = in ? __ldg(val + h.x + u * kSlice + lane) : T(0);
        }
    }
    // sellDot's order and rounding (entries past the slice's end up to a multiple
    // of four add 0 x[0], as there); the next four entries are gathered while four
    // are added
    __device__ __forceinline__ double dot(const T* x) const {
        constexpr int U = 4;
        T g[2][U];
        auto fetch = [&](int k) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = k * U + u;
                g[k & 1][u] = x[(c[e / 2] >> (16 * (e & 1))) & 0xffffu];
            }
        };
        double acc = 0.0;
        fetch(0);
#pragma unroll
        for (int k = 0; k < MAX / U; ++k) {
            if (k * U >= len) break;  // the same in every lane
            if (k + 1 < MAX / U) fetch(k + 1);
#pragma unroll
            for (int u = 0; u < U; ++u)
                acc = __fma_rn(static_cast<double>(v[k * U + u]), static_cast<double>(g[k & 1][u]), acc);
        }
        return acc;
    }
};

// MP / MD: most entries of a column / row.
template <int MP, int MD, class T>
__global__ void __launch_bounds__(32 * kTinyWarps, 1) tinySteps(LinkArgs<T> a) {
    const IterArgs<T>& p = a.it;
    const DevState* st = p.st;
    if (st->done || st->prec != precTag<T>()) return;
    const int cur = st->phase == 0 ? st->total : st->polish_count;
    const int lim = st->phase == 0 ? p.max_iter : p.polish_max_iter;
    const int iters = min(p.N, lim - cur);
    if (iters <= 0) return;
    const double step = st->step, pw = st->pw;
    const int inner = st->inner;
    __shared__ T xs[kTinyWarps * kSlice], ys[kTinyWarps * kSlice];
    const int threads = static_cast<int>(blockDim.x);
    const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
    const int n = a.P.rows, m = a.D.rows;
    const int sp = (n + kSlice - 1) / kSlice;
    for (int i = static_cast<int>(threadIdx.x); i < m; i += threads) {
        if constexpr (sizeof(T) == 4)
            ys[i] = p.yg[i];
        else
            ys[i] = p.yc[i];
    }
    auto lambda = [&](int it) {
        const int k = inner + it;
        return static_cast<double>(k) / static_cast<double>(k + 1);
    };
    if (warp < sp) {
        const int j = warp * kSlice + lane;
        const bool own = j < n;
        TinyRow<MP, T> row;
        row.load(a.P.idx, a.P.val, __ldg(a.P.hdr + warp), lane);
        ColPack<T> q{};
        double xc = 0.0, xi = 0.0, tau = 0.0;
        if (own) {
            q = p.cp[j];
            xc = p.xc[j];
            xi = static_cast<double>(p.xi[j]);
            tau = step * static_cast<double>(q.tau) / pw;
        }
        unsigned long long t0 = 0;
        long long clk = 0, pclk = 0, dclk = 0;
        const bool clock = threadIdx.x == 0;
        if (clock) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        tinyBarrier(threads);  // y is there
        double lam = lambda(1);
        for (int it = 1; it <= iters; ++it) {
            if (clock) clk = clock64();
            const double s = row.dot(ys);
            double xh, xr;
            xc = primalValues<T>(q, xc, xi, s, tau, lam, xh, xr);
            if (own) xs[j] = static_cast<T>(xr);
            tinyBarrier(threads);
            if (clock) {
                const long long c = clock64();
                pclk += c - clk;
                clk = c;
            }
            if (own && it == iters) {
                p.xh[j] = static_cast<T>(xh);
                p.xc[j] = xc;
            }
            lam = lambda(it + 1);  // while the rows are summed
            tinyBarrier(threads);
            if (clock) dclk += clock64() - clk;
        }
        if (clock) {
            unsigned long long t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            *a.time = LinkTime{t1 - t0, pclk, dclk, iters, 0};
        }
    } else {
        const int i = (warp - sp) * kSlice + lane;
        const bool own = i < m;
        TinyRow<MD, T> row;
        row.load(a.D.idx, a.D.val, __ldg(a.D.hdr + (warp - sp)), lane);
        RowPack<T> q{};
        double yc = 0.0, yi = 0.0;
        if (own) {
            q = p.rp[i];
            yc = p.yc[i];
            yi = static_cast<double>(p.yi[i]);
        }
        tinyBarrier(threads);
        for (int it = 1; it <= iters; ++it) {
            const double lam = lambda(it);
            tinyBarrier(threads);
            const double s = row.dot(xs);
            double py;
            yc = dualValues<T>(q, yc, yi, s, step, pw, lam, py);
            if (own) {
                ys[i] = static_cast<T>(yc);
                if (it == iters) {
                    p.yh[i] = static_cast<T>(py);
                    p.yc[i] = yc;
                    if constexpr (sizeof(T) == 4) p.yg[i] = static_cast<float>(yc);
                }
            }
            tinyBarrier(threads);
        }
    }
}

}  // namespace pdlpx
