// Which LPs' steps the linked restart cycle (linked.cuh) runs.  Host only.
//
// The linked cycle and the step launches give the same bits, so the choice is one
// of speed alone.  Measured on B200 (us per iteration with the check, launches ->
// linked, 190 random, transportation and power-law LPs):
//  * Sliced ELL on both sides: 1.2-3.4 times as fast up to 150k entries (400 x
//    1,000 7.9 -> 3.3, 2,000 x 5,000 9.0 -> 4.3, 42k x 40k of 120k 7.3 -> 6.2), but
//    57k x 32k rows 6.8 -> 6.9.  Up to 600k it depends on the LP: 30k x 51k of 308k
//    10.3 -> 6.4, 6k x 29k of 322k 13.9 -> 20.1, 25k x 29k of 630k 14.7 -> 14.1.
//  * Long rows beside sliced ELL (power law), a warp each: up to 50k entries and
//    rows of 512 14.4 -> 9.4 and better; beyond 1,756 x 8,375 of 83k 18.0 -> 11.9,
//    but 4,203 x 6,843 of 65k 13.6 -> 14.2 and every LP of 420k or more slower.
//  * A CSR side.  Every row of it gathers the same few values, and the warps polling
//    their lines of L2 hold up the stores to them: what decides is the loads per
//    line (crowd).  Up to 1,000, with one round of loads per row and one unit per
//    warp, transportation 70 x 70 5.2 -> 3.0, 97 x 131 4.4 -> 3.4, 70 x 300 6.4 ->
//    4.0; 150 x 150 (1,200) 5.5 -> 5.1, 200 x 200 (1,600) 5.5 -> 6.8, 300 x 100
//    between 0.9 and 1.1 times as fast from run to run.  Both sides crowded, 398 x
//    318 dense 5.8 -> 10.7; 143 x 7,113 (4,400) 7.3 -> 15.0; more than two units per
//    warp, 35,834 x 488 6.6 -> 16.9; long rows besides, power law 12-15 -> 16-28.
//    Above that crowd it pays only where the launches walk long sliced-ELL columns,
//    97 x 1,752 dense 12.6 -> 7.9.
// Between the sure cases and the hopeless ones the engine tries both (kTry): a cycle
// of each, then the faster one.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>

namespace pdlpx {

struct LinkSideShape {
    int rows = 0;
    int nl = 0;        // long rows among them, in CSR
    int lanes = 0;     // of the others: 0 sliced ELL, else CSR lanes per row
    int longest = 0;   // entries of the longest of the others
    int units = 0;     // linkUnits
};
struct LinkShape {
    std::int64_t nnz = 0;
    int longest = 0;   // entries of the longest of the long rows
    int warps = 0;     // of the grid
    LinkSideShape P, D;  // columns, rows
};

constexpr std::int64_t kLinkEntries = 600000;  // no LP beyond
// Rows and columns likewise: their cells would take 16 bytes each for nothing, since
// no LP of more than kLinkUnits units per warp gained (6.4 units 6.8 -> 6.9, 4.3 units
// 14.7 -> 14.1).
constexpr std::int64_t kLinkRows = 1000000;
constexpr int kLinkUnits = 12;
inline bool linkRoom(std::int64_t nnz, std::int64_t m, std::int64_t n) { return nnz <= kLinkEntries && m + n <= kLinkRows; }

enum class LinkRule { kNever, kTry, kAlways };

// Rounds of eight loads per lane that a warp takes for a CSR row (linkRowDot).
inline int linkRounds(int longest, int lanes) {
    return std::max(1, lanes / 32) * ((longest + 8 * lanes - 1) / (8 * lanes));
}

inline LinkRule linkRule(const LinkShape& s) {
    const bool csr = s.P.lanes > 0 || s.D.lanes > 0, longs = s.P.nl > 0 || s.D.nl > 0;
    if (s.longest > 1000 || s.P.units + s.D.units > static_cast<std::int64_t>(kLinkUnits) * s.warps) return LinkRule::kNever;
    if (!csr && !longs) {
        if (s.nnz <= 150000 && s.P.rows + s.D.rows <= 60000) return LinkRule::kAlways;
        return s.nnz <= kLinkEntries ? LinkRule::kTry : LinkRule::kNever;
    }
    if (!csr) {
        if (s.nnz <= 50000 && s.longest <= 512) return LinkRule::kAlways;
        return s.nnz <= 350000 ? LinkRule::kTry : LinkRule::kNever;
    }
    if (longs || s.nnz > 90000) return LinkRule::kNever;
    int rounds = 1, serial = 0, per_warp = 1;
    for (const LinkSideShape* a : {&s.P, &s.D}) {
        if (a->lanes > 0)
            rounds = std::max(rounds, linkRounds(a->longest, a->lanes));
        else
            serial = std::max(serial, a->longest);
        per_warp = std::max(per_warp, (a->units + s.warps - 1) / std::max(1, s.warps));
    }
    // loads of x (by the rows) and of y (by the columns) per line of eight cells
    const std::int64_t x = 8 * s.nnz / std::max(1, s.P.rows), y = 8 * s.nnz / std::max(1, s.D.rows);
    if (x + y <= 1000 && rounds == 1 && per_warp == 1 && s.nnz <= 50000) return LinkRule::kAlways;
    if (per_warp > 2 || rounds > 8 || std::min(x, y) > 500) return LinkRule::kNever;
    return x + y <= 2500 || serial >= 32 ? LinkRule::kTry : LinkRule::kNever;
}

// Share of a device that a solve's linked grid takes from the other solves on it.  As
// many grids run side by side as one SM holds blocks of them; further ones wait, while
// step launches of many solves overlap.  So a device takes grids up to that number,
// twice as many where the linked cycle is twice as fast as the launches to begin
// with; beyond, cycles run by launches (the same bits, so every cycle may choose).
// Measured on B200 (us per iteration of all solves, 1, 2, 4, 8 solver threads):
//   2,000 x 5,000 (two blocks per SM)  linked 3.4 2.1 2.0 2.1   launches 8.6 4.6 2.4 1.3
//   6,000 x 15,000 (one)               linked 4.0 4.0 3.9 3.9   launches 9.3 5.0 2.7 1.7
//   20,000 x 50,000 (one)              linked 8.5 8.3 8.3 8.3   launches 11.5 7.2 5.2 3.8
//   transportation 97 x 131 (one)      linked 3.3 3.1 3.1 3.2   launches 5.5 3.0 1.6 0.9
//   power law 2,000 x 8,000 (one)      linked 8.9 9.4 9.0 8.9   launches 15.7 8.2 4.3 2.3
//   400 x 1,000 (eight)                linked 2.6 1.4 0.8 0.5   launches 7.3 3.9 2.1 1.1
constexpr int kLinkFull = 1024;
inline int linkShareOf(int blocks_per_sm, bool twice) {
    return std::max(1, kLinkFull / (std::max(1, blocks_per_sm) * (twice ? 2 : 1)));
}
// At 1.5 units per warp of a full grid or fewer, both sides sliced ELL.
inline bool linkTwice(std::int64_t units, int sms) { return 2 * units <= 3 * static_cast<std::int64_t>(sms) * 16; }

inline std::atomic<int> g_link_share[64];  // by device
class LinkShare {
public:
    LinkShare(int device, int share) : device_(device) { set(share); }
    ~LinkShare() { set(0); }
    LinkShare(const LinkShare&) = delete;
    LinkShare& operator=(const LinkShare&) = delete;
    // this solve's grid now takes `share`
    void set(int share) {
        if (device_ < 0 || device_ >= 64) return;
        g_link_share[device_].fetch_add(share - share_, std::memory_order_relaxed);
        share_ = share;
    }
    bool fits() const {
        return share_ > 0 && g_link_share[device_].load(std::memory_order_relaxed) <= std::max(kLinkFull, share_);
    }

private:
    int device_, share_ = 0;
};

// A pack of sliced-ELL LPs: lanes per column (twice as many per row) of its linked
// cycle, 0 where the step launches run.  units4, units2: units of the live LPs with 4
// lanes per column (8 per row), with 2; warps: the most the grid has.  What decides is
// the units a warp walks one after another.  Measured on B200 (us per iteration in
// FP64, launches -> linked): 300 LPs of 50 x 125 (278k entries, 1.8 units per warp)
// 13.7 -> 7.9, 2 of 15,000 x 40,000 (640k, 3.7) 17.9 -> 15.1, but 3 (960k, 5.5) 19.4
// -> 20.8, 100 of 1,000 x 300 (741k, 6.1) 14.6 -> 18.4, 20 of 5,000 x 20,000 with one
// or two entries per column (600k, 15.8) 18.8 -> 30.4, 6 and 20 of 20,000 x 5,000
// (120k, 7.1 and 400k, 23.8) 11.1 -> 12.3 and 14.7 -> 37.9.  Batches, whose live LPs
// become fewer: 64 LPs (2.1M entries, ms per call) 274 by launches, 242-248 linked
// from 4.5 or 5.5 units per warp on, 257 from 3.5 on; 24 LPs in FP64 181 -> 121.
inline int linkPackLanes(std::int64_t nnz, std::int64_t units4, std::int64_t units2, std::int64_t warps) {
    const int lanes = units4 <= 3 * warps ? 4 : 2;
    const std::int64_t units = lanes == 4 ? units4 : units2;
    return units > 0 && 2 * units <= 9 * warps && nnz <= 1000000 ? lanes : 0;
}

}  // namespace pdlpx
