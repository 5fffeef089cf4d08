// Device helpers of the site-by-site sum (sites.cuh) that more than one
// translation unit uses.
#pragma once

#include "pair.cuh"
#include "sites.cuh"

namespace vext {

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// x mod n for any x.
__device__ __forceinline__ int wrap(int x, int n) {
    x %= n;
    return x < 0 ? x + n : x;
}

// Energy and gradient sums of pose (director o, center gi gj gk) over the lists of
// its two sites in FP64, with the correctly rounded reciprocal; partial over the
// lanes.  Few poses come here: 64 us more than with two Newton steps in the
// 47^3 x 50 skewed field's 7.4 ms.
__device__ __forceinline__ void site_pose_fp64(const SiteView &v, int o, int gi, int gj, int gk,
                                               int lane, double &e, double (&g)[6]) {
    e = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) g[k] = 0.0;
    for (int s = 0; s < 2; ++s) {
        const int4 fl = v.floor[2 * o + s];
        const double *f = v.shift + 3 * (2 * o + s);
        const int vi = wrap(gi + fl.x, v.S), vj = wrap(gj + fl.y, v.S), vk = wrap(gk + fl.z, v.S);
        const RegionInfo &r = v.regs[((vi / v.bi) * v.nrj + vj / v.bj) * v.nrk + vk / v.bk];
        double px, py, pz;
        frac_to_cart(v.H, (vi - r.i0 + f[0] - 0.5 * v.bi) / v.S,
                     (vj - r.j0 + f[1] - 0.5 * v.bj) / v.S, (vk - r.k0 + f[2] - 0.5 * v.bk) / v.S,
                     px, py, pz);
        double gs[3] = {0, 0, 0};
        for (int k = lane; k < r.n_total; k += 32) {
            const float4 h = v.hi[r.off + k], l = v.lo[r.off + k];
            const double dx = px - ((double)h.x + (double)l.x),
                         dy = py - ((double)h.y + (double)l.y),
                         dz = pz - ((double)h.z + (double)l.z);
            const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
            if (d2 >= v.rc2) continue;
            const int t = __float_as_int(h.w);
            const double c12 = v.td[4 * t], c6 = v.td[4 * t + 1], fl2 = v.td[4 * t + 3];
            const double s2 = d2 < fl2 ? fl2 : d2;
            const double i2 = __drcp_rn(s2);
            const double i6 = i2 * i2 * i2;
            e += c12 * i6 * i6 - c6 * i6 + v.td[4 * t + 2];
            if (d2 >= fl2) {
                const double de = 2.0 * (-6.0 * c12 * i6 * i6 + 3.0 * c6 * i6) * i2;
                gs[0] += de * dx;
                gs[1] += de * dy;
                gs[2] += de * dz;
            }
        }
        const double off = s ? v.off1 : v.off0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            g[k] += gs[k];
            g[3 + k] += off * gs[k];
        }
    }
}

}  // namespace vext
