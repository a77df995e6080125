// fvm_colortable.h -- the colour tables, computed by the compiler: one object
// for the host entry and for the image kernel's device copy.
#pragma once
#include <algorithm>

#include "../../include/fvm_b200.h"
#include "fvm_kernels.cuh"

namespace fvm {

// The five 256-entry tables, t = i/255, in the reference generators'
// expressions: jet (piecewise linear, :672-716), hot (:719-734), and the
// polynomial plasma (:737-754), inferno (:757-779) and viridis (:782-799).
constexpr ColormapLUT colormap_lut(int cmap) {
    ColormapLUT L{};
    for (int i = 0; i < 256; i++) {
        const float t = i / 255.0f;
        float r = 0.0f, g = 0.0f, b = 0.0f;
        switch (cmap) {
        case FVM_CMAP_JET:
            if (t < 0.125f) {
                r = 0.0f, g = 0.0f, b = 0.5f + 4.0f * t;
            } else if (t < 0.375f) {
                r = 0.0f, g = 4.0f * (t - 0.125f), b = 1.0f;
            } else if (t < 0.625f) {
                r = 4.0f * (t - 0.375f), g = 1.0f, b = 1.0f - 4.0f * (t - 0.375f);
            } else if (t < 0.875f) {
                r = 1.0f, g = 1.0f - 4.0f * (t - 0.625f), b = 0.0f;
            } else {
                r = 1.0f - 4.0f * (t - 0.875f), g = 0.0f, b = 0.0f;
            }
            break;
        case FVM_CMAP_HOT:
            r = std::min(1.0f, t * 2.5f);
            g = std::max(0.0f, std::min(1.0f, (t - 0.4f) * 2.5f));
            b = std::max(0.0f, (t - 0.8f) * 5.0f);
            break;
        case FVM_CMAP_PLASMA:
            r = 0.050383f + t * (2.028462f + t * (-1.312035f + t * 0.233106f));
            g = 0.029803f + t * (0.192182f + t * (1.429032f + t * (-1.651143f + t * 0.500000f)));
            b = 0.527975f + t * (1.573141f + t * (-2.481592f + t * 0.880392f));
            r = std::clamp(r, 0.0f, 1.0f), g = std::clamp(g, 0.0f, 1.0f), b = std::clamp(b, 0.0f, 1.0f);
            break;
        case FVM_CMAP_INFERNO:
            r = std::clamp(1.5f * t, 0.0f, 1.0f);
            g = std::clamp(2.0f * (t - 0.25f), 0.0f, 1.0f);
            b = std::clamp(0.6f - 1.2f * t, 0.0f, 0.6f);
            break;
        default:  // FVM_CMAP_VIRIDIS
            r = 0.267004f + t * (0.003991f + t * (0.494266f + t * 0.234652f));
            g = 0.004874f + t * (1.014627f + t * (-0.531556f + t * 0.512042f));
            b = 0.329415f + t * (1.423671f + t * (-2.252694f + t * 0.499477f));
            r = std::clamp(r, 0.0f, 1.0f), g = std::clamp(g, 0.0f, 1.0f), b = std::clamp(b, 0.0f, 1.0f);
            break;
        }
        L.rgb[3 * i] = r;
        L.rgb[3 * i + 1] = g;
        L.rgb[3 * i + 2] = b;
    }
    return L;
}

}  // namespace fvm
