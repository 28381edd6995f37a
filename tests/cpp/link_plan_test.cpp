// linkRule (csrc/link_plan.hpp) on LPs whose steps were timed by launches and linked:
// "never" where the launches are faster by 20 % or more, "always" where the linked
// cycle is, "try" between.  Sizes and units are those of a device with 148 SMs.
#include <cstdio>
#include <memory>
#include <vector>

#include "link_plan.hpp"

using namespace pdlpx;

static int bad = 0;
static int units(int rows, int nl, int lanes, int sub) {
    const int per = lanes == 0 ? 32 / sub : (lanes < 32 ? 32 / lanes : 1);
    return nl + (rows - nl + per - 1) / per;
}
// lanes 0: sliced ELL; lp, ld: lanes per sliced-ELL column, row
static void expect(LinkRule want, const char* name, long long nnz, int m, int n, int lanesP, int lanesD, int longP,
                   int longD, int lp, int ld, int nlP = 0, int nlD = 0, int longest = 0) {
    LinkShape s;
    s.nnz = nnz;
    s.longest = longest;
    s.P = LinkSideShape{n, nlP, lanesP, longP, units(n, nlP, lanesP, lp)};
    s.D = LinkSideShape{m, nlD, lanesD, longD, units(m, nlD, lanesD, ld)};
    const int most = lanesP || lanesD || nlP || nlD ? 8 : 16, all = s.P.units + s.D.units, sms = 148;
    const int warps = (all + sms - 1) / sms;
    s.warps = sms * (warps < most ? warps : most);
    const LinkRule got = linkRule(s);
    if (got == want) return;
    std::printf("FAIL %s: %d instead of %d\n", name, static_cast<int>(got), static_cast<int>(want));
    ++bad;
}

// `count` LPs of m x n with `nnz` entries each, all live
static void pack(int want, const char* name, long long count, int m, int n, long long nnz) {
    const long long u4 = count * ((n + 7) / 8 + (m + 3) / 4), u2 = count * ((n + 15) / 16 + (m + 7) / 8);
    const int got = linkPackLanes(count * nnz, u4, u2, 148 * 16);
    if (got == want) return;
    std::printf("FAIL pack %s: %d instead of %d\n", name, got, want);
    ++bad;
}

// How many solves of one kind, one after another, find room.
static int fitting(int share) {
    std::vector<std::unique_ptr<LinkShare>> all;
    for (int k = 0; k < 40; ++k) {
        all.push_back(std::make_unique<LinkShare>(3, share));
        if (!all.back()->fits()) return k;
    }
    return 40;
}
static void shares(int want, int got) {
    if (want == got) return;
    std::printf("FAIL %d solves instead of %d\n", got, want);
    ++bad;
}

int main() {
    shares(1, fitting(linkShareOf(1, false)));  // grids that fill the SMs, as CSR ones do
    shares(2, fitting(linkShareOf(1, true)));
    shares(4, fitting(linkShareOf(2, true)));
    shares(8, fitting(linkShareOf(8, false)));
    shares(0, fitting(0));  // no grid
    {
        LinkShare a(3, linkShareOf(1, false)), b(3, linkShareOf(1, false));
        if (a.fits() || b.fits()) std::printf("FAIL two full grids\n"), ++bad;
        b.set(0);  // runs by launches from now on
        if (!a.fits()) std::printf("FAIL alone again\n"), ++bad;
        LinkShare c(4, linkShareOf(1, false)), d(-1, 5), e(64, 5);
        if (!c.fits() || d.fits() || e.fits()) std::printf("FAIL other devices\n"), ++bad;
    }
    shares(1, fitting(kLinkFull + 1));
    if (!linkTwice(3552, 148) || linkTwice(3553, 148)) std::printf("FAIL units\n"), ++bad;
    pack(0, "no LP", 0, 50, 125, 930);
    pack(4, "12 of 1,000 x 2,500", 12, 1000, 2500, 20000);
    pack(2, "300 of 50 x 125", 300, 50, 125, 930);
    pack(0, "800 of 50 x 125", 800, 50, 125, 930);
    pack(2, "2 of 15,000 x 40,000", 2, 15000, 40000, 320000);
    pack(0, "3 of 15,000 x 40,000", 3, 15000, 40000, 320000);
    pack(0, "100 of 1,000 x 300", 100, 1000, 300, 7410);
    pack(0, "20 of 5,000 x 20,000", 20, 5000, 20000, 30000);
    pack(0, "6 of 20,000 x 5,000", 6, 20000, 5000, 19900);
    pack(0, "entries", 1, 1000, 1000, 1000001);
    const auto never = LinkRule::kNever, maybe = LinkRule::kTry, always = LinkRule::kAlways;
    // sliced ELL on both sides
    expect(always, "400 x 1,000", 8000, 400, 1000, 0, 0, 12, 35, 4, 8);
    expect(always, "2,000 x 5,000", 40000, 2000, 5000, 0, 0, 12, 37, 4, 8);
    expect(always, "42,395 x 17,000", 120000, 42395, 17000, 0, 0, 12, 20, 4, 8);
    expect(maybe, "56,694 x 32,108", 80000, 56694, 32108, 0, 0, 3, 9, 1, 8);
    expect(maybe, "5,798 x 29,377", 322000, 5798, 29377, 0, 0, 15, 84, 2, 4);
    expect(maybe, "30,000 x 75,000", 600000, 30000, 75000, 0, 0, 12, 37, 2, 4);
    expect(never, "one entry more", 600001, 30000, 75000, 0, 0, 12, 37, 2, 4);
    expect(maybe, "100,000 x 100,000", 551506, 100000, 100000, 0, 0, 10, 18, 2, 4);
    expect(never, "200,000 x 100,000", 400000, 200000, 100000, 0, 0, 8, 8, 4, 8);
    if (!linkRoom(600000, 500000, 500000) || linkRoom(600000, 500001, 500000) || linkRoom(600001, 1, 1))
        std::printf("FAIL room\n"), ++bad;
    // long columns or rows beside it
    expect(always, "power law 3,039 x 4,575", 45000, 3039, 4575, 0, 0, 64, 30, 4, 8, 101, 0, 289);
    expect(maybe, "power law 4,203 x 6,843", 65000, 4203, 6843, 0, 0, 64, 32, 4, 8, 134, 0, 360);
    expect(maybe, "transportation 10 x 1,000", 20000, 1010, 10000, 0, 0, 2, 10, 1, 8, 0, 10, 1000);
    expect(never, "rows of 1,001", 20000, 1010, 10000, 0, 0, 2, 10, 1, 8, 0, 10, 1001);
    expect(never, "power law 9,677 x 43,549", 426000, 9677, 43549, 0, 0, 70, 72, 4, 8, 694, 0, 900);
    // a CSR side
    expect(always, "transportation 97 x 131", 25414, 228, 12707, 0, 32, 2, 131, 1, 8);
    expect(always, "transportation 70 x 300", 42000, 370, 21000, 0, 32, 2, 300 - 44, 1, 8);
    expect(maybe, "transportation 150 x 150", 45000, 300, 22500, 0, 64, 2, 150, 1, 8);
    expect(maybe, "transportation 200 x 210", 84000, 410, 42000, 0, 64, 2, 210, 1, 8);
    expect(never, "transportation 300 x 200", 120000, 500, 60000, 0, 64, 2, 300, 1, 8);
    expect(always, "57 x 119 dense", 4298, 57, 119, 0, 32, 44, 84, 4, 8);
    expect(maybe, "97 x 1,752 dense", 88420, 97, 1752, 0, 64, 60, 966, 4, 8);
    expect(never, "398 x 318 dense", 38108, 398, 318, 32, 32, 156, 120, 4, 8);
    expect(never, "143 x 7,113", 78921, 143, 7113, 0, 64, 13, 621, 4, 8);
    expect(never, "66 x 6,656", 44313, 66, 6656, 0, 64, 9, 732, 4, 8);
    expect(never, "35,834 x 488", 78432, 35834, 488, 64, 0, 218, 10, 4, 8);
    expect(never, "44,082 x 93", 9249, 44082, 93, 32, 0, 139, 4, 4, 8);
    expect(never, "power law 1,175 x 8,124", 77000, 1175, 8124, 0, 32, 70, 92, 4, 8, 155, 0, 311);
    // uniformly long rows: none is split off as a long one, a warp sums each
    expect(never, "8 x 10,000 dense", 80000, 8, 10000, 0, 256, 8, 10000, 4, 8);
    return bad != 0;
}
