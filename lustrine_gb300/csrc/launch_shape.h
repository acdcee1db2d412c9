// launch_shape.h -- the launch shape of a context that has none set (host).
#pragma once

#include <atomic>

#include "lustrine_gb300.h"
#include "pbf_kernels.h"

namespace lgb {

// The contexts alive on a device and the particles they hold.
struct DeviceLoad {
    std::atomic<int> contexts{0};
    std::atomic<long long> particles{0};
    void add(int c, long long n) {
        contexts.fetch_add(c, std::memory_order_relaxed);
        particles.fetch_add(n, std::memory_order_relaxed);
    }
};

// More gathers in flight shorten a particle's chain of dependent loads but take
// registers (U = 4: 56, nine blocks of 128 per SM), so they pay while all
// particles still fit the GPU at once.
constexpr int wave_particles(int sms) { return sms * 9 * 128; }

// Whether a context's steps are likely to share the GPU with more of others' than
// fits it: more than a few contexts are alive, which a program steps together
// (up to four: one scene and copies of it, stepped in turn), with more than two
// waves of particles, half a wave where the positions are per-cell mixed (64
// registers).  What shortens a chain then costs the others instructions and
// registers.  Measured, us a step of k contexts of some n particles, shape alone /
// in a crowd:
//     k, n          16-bit        on voxels    voxels, per-cell mixed
//     64, 2,000     207 / 214     217 / 224    234 / 234
//     32, 8,000     132 / 138     148 / 147    182 / 169
//     128, 8,000    404 / 404     444 / 429    539 / 515
//     8, 16,000     75 / 75       89 / 85      102 / 97
//     128, 16,000   517 / 504     730 / 581    886 / 785
//     32, 40,000    301 / 291     385 / 348    507 / 436
// 512 contexts of 1,024 to 65,536 particles (7.5 M) 1.81 ms / 1.69, with the shape
// alone for those up to 4,000 1.75; 96 of 2,000 to 20,000 on voxels 343 us / 329.
constexpr int CROWD_CONTEXTS = 4;
inline bool crowded(const DeviceLoad& d, bool cells, int sms) {
    const long long room = cells ? wave_particles(sms) / 2 : 2LL * wave_particles(sms);
    return d.contexts.load(std::memory_order_relaxed) > CROWD_CONTEXTS &&
           d.particles.load(std::memory_order_relaxed) > room;
}

// The default shape by list format, size and load, from t's remaining fields (the
// results are the same bits in every shape).  cells: per-cell mixed positions.
// Measured, us per step at the fixed shape (2 gathers, 8 in XSPH) and at this
// rule's, one context, 4 iterations:
//   column lists, fp32 with static particles: 77,000 63.7 / 58.8, 150,000
//     87.7 / 74.3, 262,144 99.6 / 94.8, 500,000 155 / 153
//   column lists, per-cell mixed: 150,000 94.8 / 88.0 with 4 and 4 (2 and 2:
//     93.7), 300,000 128 / 126 with 2 and 2 (4 and 4: 132), 3 M hashed 1141 / 1119
//   16-bit records: 10,000 37.1 / 35.5, 37 scenes of 157,443 73.4 / 69.9;
//     200 scenes of 3.0 M 573 / 545 with 1 and 4 (4 and 4: 576)
//   24-bit records: 200,000 62.1 (2 and 2: 63.2), 600,000 162.5 / 161.8,
//     2 M 497 / 492 (4 and 4: 522)
//   32-bit records: 18 M (with a fourth of the upload) 4,183 / 3,873 with 1 and 1
//     in blocks of 256 (4 and 4: 4,254)
constexpr int XSPH_WIDE_MAX = 250000;
inline Tuning default_shape(Tuning t, int format, int n, int cap, bool hashed, bool cells, bool crowd, int sms) {
    const bool small = n <= wave_particles(sms);
    if (!crowd && n <= lists_group_max(hashed, format == LUSTRINE_LISTS_COMPACT,
                                       format == LUSTRINE_LISTS_COMPACT_WIDE, cells))
        t.list_block = LISTS_GROUP_BLOCK;
    if (format == LUSTRINE_LISTS_COMPACT_WIDE && cap >= COMPACT_MAX_N) {
        t.block = 256;
        t.unroll = t.xsph_unroll = 1;
    } else if (format == LUSTRINE_LISTS_COMPACT_WIDE) {
        t.xsph_unroll = n <= XSPH_WIDE_MAX ? 8 : 2;
    } else if (format == LUSTRINE_LISTS_COMPACT) {
        t.unroll = !small ? 1 : (crowd ? 2 : 4);
        t.xsph_unroll = 4;
    } else {
        t.unroll = t.xsph_unroll = crowd || (cells && !small) ? 2 : 4;
    }
    return t;
}

}  // namespace lgb
