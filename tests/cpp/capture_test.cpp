// captured() and residentAtOnce() (csrc/capture.hpp) with the device calls faked.
#include <cstdio>
#include <string>

#include "capture.hpp"

static int bad = 0;
static void same(const std::string& got, const std::string& want) {
    if (got == want) return;
    std::printf("FAIL: %s instead of %s\n", got.c_str(), want.c_str());
    ++bad;
}

// the calls that were made, then the result
static std::string run(int begin, int launches, int end) {
    std::string log;
    const int e = pdlpx::captured<int>([&] { log += 'b'; return begin; }, [&] { log += 'l'; return launches; },
                                       [&] { log += 'e'; return end; });
    return log + std::to_string(e);
}

int main() {
    same(run(0, 0, 0), "ble0");
    same(run(7, 0, 0), "b7");
    same(run(0, 7, 0), "ble7");  // a refused launch: the capture ends, the error stays
    same(run(0, 7, 9), "ble7");
    same(run(0, 0, 9), "ble9");
    // no cooperative launches, no room, the last block that fits, one more, no grid
    same(pdlpx::residentAtOnce(0, 2, 148, 1) ? "1" : "0", "0");
    same(pdlpx::residentAtOnce(1, 0, 148, 1) ? "1" : "0", "0");
    same(pdlpx::residentAtOnce(1, 1, 148, 148) ? "1" : "0", "1");
    same(pdlpx::residentAtOnce(1, 1, 147, 148) ? "1" : "0", "0");
    same(pdlpx::residentAtOnce(1, 1, 148, 0) ? "1" : "0", "0");
    return bad != 0;
}
