// fast_root.h -- where the pair sums may share one approximate reciprocal square root
// (pbf_sums.cuh: root_and_spiky).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../include/fluid_gb300.h"
#include "fgb_device.cuh"

namespace fgb {

// The mantissas m for which 1 / (1 + m 2^-23) lies within 2^-43 (relative) of the
// midpoint of two floats: there a reciprocal known to 2^-43 may round either way.
// Found by going through all 2^23 of them; tests/test_fast_root.py does so again.
static constexpr uint32_t kNearTieReciprocals[] = {
    0x00f686, 0x0164b0, 0x05018f, 0x06908f, 0x069913, 0x07cc45, 0x09bcb0, 0x0ae8f1, 0x0c1284, 0x0efa43, 0x109909, 0x10ce81,
    0x12abab, 0x14f105, 0x16dbcf, 0x186799, 0x19791b, 0x1beaaf, 0x2013d1, 0x20ddd1, 0x224cf7, 0x26449f, 0x276b84, 0x2aaaac,
    0x2b27b2, 0x2b8be1, 0x2d1367, 0x2d1c3e, 0x2d8f69, 0x2e4f88, 0x317931, 0x31f990, 0x384a93, 0x4100c1, 0x423dc3, 0x466730,
    0x4698d0, 0x4cccd0, 0x4f7d05, 0x4fba38, 0x50ac19, 0x50dd0d, 0x525d25, 0x543d43, 0x5c23dd, 0x5e86a9, 0x5e9bd0, 0x605475,
    0x61368b, 0x625473, 0x6401c8, 0x658fd0, 0x6c7ec7, 0x6e4bc5, 0x700ff1, 0x702a3b, 0x70ff0f, 0x7c3237, 0x7c62e2, 0x7e01ff,
    0x7f44fe, 0x7ffffb, 0x7ffffd, 0x7fffff,
};

inline float bits_to_float(uint32_t u) {
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
}

// Whether pbf_sums.cuh's root_and_spiky<true> gives the IEEE root and quotient for every
// pair of this solver: r = sqrt(r2) is exact over the whole range (checked on the device
// for every float), and (h - r)^2 / r is by Markstein's theorem wherever the reciprocal
// of r is correctly rounded.  For the r whose reciprocal may not be, both roundings (and
// the floats beside them) are put through the same steps here.  The range of h keeps
// every intermediate value of the sums in the normal range; the ref profile also divides
// by rho0 and corr_ref, whose reciprocals are correctly rounded, so only a divisor with
// an all-ones mantissa is left out, as the theorem does.
inline bool fast_root_exact(const Phys &ph) {
    if (!(ph.h >= 0x1p-7f && ph.h <= 0x1p7f) || ph.corr_n != 4.f) return false;
    for (float c : {ph.rho0, ph.corr_ref}) {
        uint32_t u;
        memcpy(&u, &c, sizeof u);
        if (!(c >= 0x1p-20f && c <= 0x1p30f) || (u & 0x7fffffu) == 0x7fffffu) {
            if (ph.profile == FGB_PROFILE_REF) return false;
        }
    }
    for (int e = -27; e <= 7; ++e)
        for (uint32_t m : kNearTieReciprocals) {
            const float r = bits_to_float(((uint32_t)(e + 127) << 23) | m);
            if (r < kKernelEpsilon || r > ph.h) continue;
            const float hr = ph.h - r, a = hr * hr, near = 1.f / r;
            for (float y : {near, std::nextafter(near, 0.f), std::nextafter(near, INFINITY)}) {
                const float w = a * y;
                if (std::fma(std::fma(-r, w, a), y, w) != a / r) return false;
            }
        }
    return true;
}

}  // namespace fgb
