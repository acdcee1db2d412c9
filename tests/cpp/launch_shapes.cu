// The launches of the PBF list build and passes for every launch shape, taken
// from the launchers over a CUDA runtime that only records them
// (launch_shapes_runtime.cpp).  One line each: pass, particles, lists (column,
// the records' kind, or scene-frame column), shape, blocks, threads, kernel.
#include <cstdio>

#include "pbf_kernels.h"

struct Launch {
    const void* kernel;
    unsigned grid, block;
    int count;
};
extern "C" Launch g_launch;

using namespace lgb;

int main() {
    static uint4 rec[1];
    const char* kinds[] = {"column", "16", "24", "32", "frame"};
    for (int kind = 0; kind < 5; kind++)
        for (int n : {10000, 11001, 20001, 1 << 20})
            for (int list_block : {64, 128, 256})
                for (int block : {64, 128, 256})
                    for (int unroll : {1, 2, 4, 8}) {
                        StepParams p{};
                        CellPack cp{};
                        p.n = n;
                        p.max_nbrs = 64;
                        const bool compact = kind >= 1 && kind <= 3;
                        p.rec = p.rec2 = compact ? rec : nullptr;
                        p.wide = compact ? kind - 1 : 0;
                        p.frame = kind == 4;
                        const bool mixed = p.frame != 0;
                        const Tuning tu{block, unroll, list_block, unroll, 1, 1};
                        auto row = [&](const char* pass) {
                            std::printf("%s %d %s %d %d %d %u %u %p %d\n", pass, n, kinds[kind], list_block, block, unroll,
                                        g_launch.grid, g_launch.block, g_launch.kernel, g_launch.count);
                            g_launch.count = 0;
                        };
                        launch_lists_lambda(mixed, tu, p, cp, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                            nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
                        row("lists");
                        launch_lambda(mixed, tu, p, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
                        row("lambda");
                        launch_delta(mixed, tu, p, cp, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                     nullptr, nullptr);
                        row("delta");
                        launch_xsph(mixed, tu, p, cp, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                    nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
                        row("xsph");
                    }
    return 0;
}
