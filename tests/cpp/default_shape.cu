// The default launch shape against the load of the device: what one scene alone
// takes, what it takes among many, and the count of contexts kept by threads.
#include <cstdio>
#include <thread>
#include <vector>

#include "launch_shape.h"

using namespace lgb;

static int failed = 0;
static void expect(bool ok, const char* what, int n) {
    if (!ok) std::printf("%s, %d particles\n", what, n), failed = 1;
}

int main() {
    const int sms = 152, wave = wave_particles(sms);
    const Tuning t{128, 2, 128, 8, 1, 1};
    DeviceLoad d;
    auto is_crowded = [&](int contexts, long long particles, bool cells = false) {
        d.add(contexts, particles);
        const bool c = crowded(d, cells, sms);
        d.add(-contexts, -particles);
        return c;
    };
    expect(!is_crowded(1, 100 * wave), "one context is a crowd", 100 * wave);
    expect(!is_crowded(4, 100 * wave), "four contexts are a crowd", 100 * wave);
    expect(!is_crowded(500, 2 * wave), "two waves are a crowd", 2 * wave);
    expect(is_crowded(5, 2 * wave + 1), "five contexts are no crowd", 2 * wave + 1);
    expect(!is_crowded(500, wave / 2, true), "half a wave is a crowd", wave / 2);
    expect(is_crowded(5, wave / 2 + 1, true), "five mixed contexts are no crowd", wave / 2 + 1);
    expect(is_crowded(512, 7546040), "512 contexts are no crowd", 7546040);

    for (int n : {1000, 8000, 11000, 11001, 20000, 20001, wave, wave + 1, 300000})
        for (int format : {LUSTRINE_LISTS_COLUMN, LUSTRINE_LISTS_COMPACT, LUSTRINE_LISTS_COMPACT_WIDE})
            for (int hashed : {0, 1})
                for (int cells : {0, 1}) {
                    if (format != LUSTRINE_LISTS_COLUMN && cells) continue;
                    auto shape = [&](bool crowd) { return default_shape(t, format, n, n, hashed, cells, crowd, sms); };
                    const Tuning alone = shape(false), among = shape(true);
                    expect(among.list_block == 128, "four lanes in a crowd", n);
                    expect(among.unroll <= 2, "more than two gathers in a crowd", n);
                    expect(format == LUSTRINE_LISTS_COMPACT_WIDE || among.xsph_unroll <= 4, "XSPH gathers in a crowd", n);
                    const int group = format == LUSTRINE_LISTS_COMPACT ? 11000
                                      : format == LUSTRINE_LISTS_COLUMN && !cells ? 20000 : 0;
                    expect((alone.list_block == 256) == (!hashed && n <= group), "lanes alone", n);
                    for (const Tuning& q : {alone, among})
                        expect(q.block == 128 && q.ppt == 1 && q.lists == 1 && q.unroll >= 1, "other fields", n);
                }

    std::vector<std::thread> threads;  // counts of threads that come and go add up
    for (int k = 0; k < 8; k++)
        threads.emplace_back([&] {
            for (int r = 0; r < 100000; r++) d.add(1, 1000), d.add(-1, -1000);
            d.add(1, 50000);
        });
    for (auto& q : threads) q.join();
    expect(d.contexts == 8 && d.particles == 400000 && crowded(d, false, sms), "contexts counted", 400000);
    return failed;
}
