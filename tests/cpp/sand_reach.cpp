// contact_reach2 over diameters: zero, subnormal, ordinary, huge, infinite,
// negative and NaN, against its definition.
#include "sand_reach.h"

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

static int check(float d) {
    const float r = lgb::contact_reach2(d);
    bool ok;
    if (std::isnan(d))
        ok = std::isnan(r);
    else if (d < 0.0f)
        ok = r < 0.0f;
    else
        ok = std::sqrt(r) <= d && (std::isinf(r) || std::sqrt(std::nextafter(r, INFINITY)) > d);
    if (!ok) std::printf("diameter %g: %g\n", d, r);
    return !ok;
}

int main() {
    int bad = 0;
    for (float d : {0.0f, -0.0f, 1.0f, 1e-45f, 1e-30f, 3e-23f, 1.2e-19f, 1.1e-19f, 1e19f, 1.8446742e19f, 1.8446744e19f, 1e30f,
                    3.4028235e38f, INFINITY, -1.0f, -1e-45f, -1e30f, -INFINITY, NAN})
        bad |= check(d);
    for (uint32_t b = 0; b < 0xFFFFFFFFu - 40009u; b += 40009u) {  // through every float's exponent, both signs
        float d;
        std::memcpy(&d, &b, 4);
        bad |= check(d);
    }
    return bad;
}
