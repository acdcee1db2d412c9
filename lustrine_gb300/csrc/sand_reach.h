// sand_reach.h -- the sand contacts' distance test without a square root (host).
#pragma once

#include <cmath>

namespace lgb {

// The largest d2 whose float square root rounds to at most diameter (the
// rounded root is monotonic: sqrt(d2) > diameter exactly when d2 > this);
// negative where no root does (a negative diameter: no contacts), NaN for NaN
// (a comparison with it is never true, as with the diameter itself).
inline float contact_reach2(float diameter) {
    if (diameter < 0.0f) return -1.0f;
    float r = diameter * diameter;  // within a few floats of it, or at the range's end
    while (std::sqrt(r) > diameter) r = std::nextafter(r, 0.0f);  // ends at 0
    while (std::isfinite(r) && std::sqrt(std::nextafter(r, INFINITY)) <= diameter) r = std::nextafter(r, INFINITY);
    return r;
}

}  // namespace lgb
