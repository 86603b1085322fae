// kron.cuh -- ellipses and boxes of the AUTO / Kron photometry,
// src/cuda/cudaanalyse.cu:318-440.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace sx {

#define SX_RINT(x) (int)(floor(x + 0.5))

__device__ __forceinline__ void kron_box(int w, int h, double mx, double my, float dxlim, float dylim, KronGeo &g) {
    g.flags = 0;
    if ((g.xmin = SX_RINT(mx - dxlim)) < 0) {
        g.xmin = 0;
        g.flags |= SX_OBJ_APERT_PB;
    }
    if ((g.xmax = SX_RINT(mx + dxlim) + 1) > w) {
        g.xmax = w;
        g.flags |= SX_OBJ_APERT_PB;
    }
    if ((g.ymin = SX_RINT(my - dylim)) < 0) {
        g.ymin = 0;
        g.flags |= SX_OBJ_APERT_PB;
    }
    if ((g.ymax = SX_RINT(my + dylim) + 1) > h) {
        g.ymax = h;
        g.flags |= SX_OBJ_APERT_PB;
    }
}

// ellipse of scale `scale` (6 sigma in pass 1, the Kron factor in pass 2) and
// its box; false when it is the (empty) minimum aperture
__device__ __forceinline__ bool kron_geo(int w, int h, double mx, double my, float a, float b, float cxx, float cyy,
                                         float cxy, double scale, float klim2, KronGeo &g) {
    const double autoaper = 0.0;
    float dxlim, dylim;
    const bool ell = scale * sqrtf(a * b) > autoaper / 2.0;
    if (ell) {
        g.cx2 = cxx;
        g.cy2 = cyy;
        g.cxy = cxy;
        dxlim = g.cx2 - g.cxy * g.cxy / (4.0 * g.cy2);
        dxlim = dxlim > 0.0 ? scale / sqrtf(dxlim) : 0.0;
        dylim = g.cy2 - g.cxy * g.cxy / (4.0 * g.cx2);
        dylim = dylim > 0.0 ? scale / sqrtf(dylim) : 0.0;
        g.klim2 = klim2;
    } else {
        g.cx2 = g.cy2 = 1.0;
        g.cxy = 0.0;
        dxlim = dylim = autoaper / 2.0;
        g.klim2 = dxlim * dxlim;
    }
    kron_box(w, h, mx, my, dxlim, dylim, g);
    return ell;
}

__device__ __forceinline__ int kron_npix(const KronGeo &g) { return (g.xmax - g.xmin) * (g.ymax - g.ymin); }

}  // namespace sx
