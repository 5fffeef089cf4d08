// Warp-level evaluation of one pose over its bin list, shared by the pose
// batches (posebatch.cu) and the String update (string.cu).
#pragma once

#include "pair.cuh"

namespace vext {

// This lane's far entries begin + lane + stride i < end of one pose, the two
// sites in the two lanes of the packed FP32x2 instructions (pose.cu's far loop):
// d = x - r_s, n1 = hardware reciprocal of d2, n3 = n1^3, e = n3 (c12 n3 - c6),
// fp = (n1 n3)(c6 - 2 c12 n3), dE/dsite += -6 fp d.  MASK = false for inner
// entries (within the cutoff of every pose of the bin: no mask, the shift
// summed once per entry into shift_sum).  FP32 partials are flushed into the
// FP64 sums every 16 entries.  MASK: a site whose FP32 d2 lies within
// kBorderTol of rc^2 -- where the FP32 test might decide the pair unlike the
// FP64 one -- leaves the FP32 sums and takes the pair in FP64
// (fp64_border_pair, from the hi + lo position and the FP64 site sd).
// LOADS: entries a lane loads together (long lists only: a short one would
// mostly load its last entry again).
template <bool MASK, int LOADS>
__device__ __forceinline__ void far_lane_sums(const PoseBatchSys &y, long long base, int begin,
                                              int end, int lane, int stride, float2 nsx,
                                              float2 nsy, float2 nsz, const double (&sd)[2][3],
                                              double (&v)[7], double &shift_sum) {
    const int mine = end - begin > lane ? (end - begin - lane + stride - 1) / stride : 0;
#pragma unroll 1
    for (int i0 = 0; i0 < mine; i0 += 16) {
        float2 fe = make_float2(0.f, 0.f), gx = fe, gy = fe, gz = fe;
        float fs = 0.f;
        const int i1 = min(i0 + 16, mine);
        auto add = [&](long long k, const float4 &h, const float4 &tp) {
            const float2 dx = __fadd2_rn(make_float2(h.x, h.x), nsx),
                         dy = __fadd2_rn(make_float2(h.y, h.y), nsy),
                         dz = __fadd2_rn(make_float2(h.z, h.z), nsz);
            const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            float r0, r1;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d2.x));
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d2.y));
            const float2 n1 = make_float2(r0, r1);
            float2 n3 = __fmul2_rn(__fmul2_rn(n1, n1), n1);
            if (MASK) {
                float2 m = make_float2(set_lt(d2.x, y.rc2f), set_lt(d2.y, y.rc2f));
                const float2 x = __fadd2_rn(d2, make_float2(-y.rc2f, -y.rc2f));
                const bool b0 = fabsf(x.x) < kBorderTol, b1 = fabsf(x.y) < kBorderTol;
                if (b0 || b1) {   // rare
                    const float4 l = y.lo[k];
                    const double ax = (double)h.x + (double)l.x, ay = (double)h.y + (double)l.y,
                                 az = (double)h.z + (double)l.z;
                    const int ty = __float_as_int(h.w);
                    if (b0) {
                        m.x = 0.f;
                        fp64_border_pair(sd[0][0], sd[0][1], sd[0][2], ax, ay, az, y.td, ty, y.rc2,
                                         v[0], v + 1);
                    }
                    if (b1) {
                        m.y = 0.f;
                        fp64_border_pair(sd[1][0], sd[1][1], sd[1][2], ax, ay, az, y.td, ty, y.rc2,
                                         v[0], v + 4);
                    }
                }
                n3 = __fmul2_rn(n3, m);
                fe = __ffma2_rn(m, make_float2(tp.z, tp.z), fe);
            } else {
                fs += tp.z;
            }
            fe = __ffma2_rn(n3, __ffma2_rn(make_float2(tp.x, tp.x), n3, make_float2(-tp.y, -tp.y)),
                            fe);
            const float2 fp =
                __fmul2_rn(__fmul2_rn(n1, n3),
                           __ffma2_rn(make_float2(-2.f * tp.x, -2.f * tp.x), n3,
                                      make_float2(tp.y, tp.y)));
            gx = __ffma2_rn(fp, dx, gx);
            gy = __ffma2_rn(fp, dy, gy);
            gz = __ffma2_rn(fp, dz, gz);
        };
        auto entry = [&](int i) { return base + begin + lane + (long long)stride * i; };
        if constexpr (LOADS == 1) {
            for (int i = i0; i < i1; ++i) {
                const float4 h = y.hi[entry(i)];
                add(entry(i), h, y.tf[__float_as_int(h.w)]);   // (c12, c6, shift, floor2)
            }
        } else {
            // LOADS entries in flight together (each is a chain of list, table
            // and arithmetic latencies), summed in order
#pragma unroll 1
            for (int j0 = i0; j0 < i1; j0 += LOADS) {
                float4 hv[LOADS], tv[LOADS];
#pragma unroll
                for (int j = 0; j < LOADS; ++j) hv[j] = y.hi[entry(min(j0 + j, i1 - 1))];
#pragma unroll
                for (int j = 0; j < LOADS; ++j) tv[j] = y.tf[__float_as_int(hv[j].w)];
#pragma unroll
                for (int j = 0; j < LOADS; ++j)
                    if (j0 + j < i1) add(entry(j0 + j), hv[j], tv[j]);
            }
        }
        v[0] += (double)fe.x + (double)fe.y;
        if (!MASK) shift_sum += (double)fs;
        v[1] -= 6.0 * (double)gx.x;
        v[2] -= 6.0 * (double)gy.x;
        v[3] -= 6.0 * (double)gz.x;
        v[4] -= 6.0 * (double)gx.y;
        v[5] -= 6.0 * (double)gy.y;
        v[6] -= 6.0 * (double)gz.y;
    }
}

// Sums of one pose over its bin list: v = (E, dE/dsite0 [3], dE/dsite1 [3]),
// partial over the entries lane, lane + stride, ... (reduced by the caller).  FAR64 evaluates every entry in FP64
// (the FP64 mode, whose entries are all near, with the correctly rounded
// reciprocal; the re-evaluation of flagged poses, IEEE = false, with the
// hardware seed + two Newton steps, within an ulp or two of it); otherwise
// near entries in FP64 with the hardware reciprocal seed + one Newton step
// (relative error <= 2^-46) and far entries in packed FP32.
template <bool FAR64, int LOADS, bool IEEE = FAR64>
__device__ __forceinline__ void pose_sums(const PoseBatchSys &y, const RegionInfo &r,
                                          const double (&sd)[2][3], int lane, int stride,
                                          double (&v)[7]) {
    constexpr int NEAR = LOADS > 1 ? LOADS / 2 : 1;
    const int end = FAR64 ? r.n_total : r.n_near;
    auto add = [&](const float4 &h, const float4 &l) {
        const double x = (double)h.x + (double)l.x, yy = (double)h.y + (double)l.y,
                     z = (double)h.z + (double)l.z;
        const int t = __float_as_int(h.w);
        const double c12 = y.td[4 * t], c6 = y.td[4 * t + 1], shift = y.td[4 * t + 2],
                     fl = y.td[4 * t + 3];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double dx = sd[s][0] - x, dy = sd[s][1] - yy, dz = sd[s][2] - z;
            const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
            if (d2 >= y.rc2) continue;
            const double s2 = d2 < fl ? fl : d2;
            const double i2 = IEEE ? 1.0 / s2 : FAR64 ? rcp64_nr<2>(s2) : rcp64_nr<1>(s2);
            const double i6 = i2 * i2 * i2;
            v[0] += fma(i6, fma(c12, i6, -c6), shift);
            if (d2 > fl) {
                // dE/dsite = 2 dE/d(d2) (site - x),  dE/d(d2) = i2 i6 (3 c6 - 6 c12 i6)
                const double w = i2 * i6 * fma(-12.0 * c12, i6, 6.0 * c6);
                v[1 + 3 * s] = fma(w, dx, v[1 + 3 * s]);
                v[2 + 3 * s] = fma(w, dy, v[2 + 3 * s]);
                v[3 + 3 * s] = fma(w, dz, v[3 + 3 * s]);
            }
        }
    };
    if constexpr (LOADS == 1) {
        for (int e = lane; e < end; e += stride) add(y.hi[r.off + e], y.lo[r.off + e]);
    } else {
#pragma unroll 1
        for (int e0 = lane; e0 < end; e0 += NEAR * stride) {
            float4 hv[NEAR], lv[NEAR];
#pragma unroll
            for (int j = 0; j < NEAR; ++j) {
                const int e = min(e0 + j * stride, end - 1);
                hv[j] = y.hi[r.off + e];
                lv[j] = y.lo[r.off + e];
            }
#pragma unroll
            for (int j = 0; j < NEAR; ++j)
                if (e0 + j * stride < end) add(hv[j], lv[j]);
        }
    }
    if (FAR64) return;
    // far entries lie beyond r_split of every site: no contact floor
    const float2 nsx = make_float2(-(float)sd[0][0], -(float)sd[1][0]),
                 nsy = make_float2(-(float)sd[0][1], -(float)sd[1][1]),
                 nsz = make_float2(-(float)sd[0][2], -(float)sd[1][2]);
    double shift_sum = 0.0;
    far_lane_sums<false, LOADS>(y, r.off, r.n_near, r.n_near + r.n_inner, lane, stride, nsx, nsy, nsz,
                         sd, v, shift_sum);
    far_lane_sums<true, LOADS>(y, r.off, r.n_near + r.n_inner, r.n_total, lane, stride, nsx, nsy, nsz,
                        sd, v, shift_sum);
    v[0] += 2.0 * shift_sum;
}

__device__ __forceinline__ void warp_reduce7(double (&v)[7]) {
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
}


// A pose: normalised quaternion (w, x, y, z), its norm, valid input.
struct PosePoint {
    double q[4], norm;
    bool ok;
};

// Energy and site forces v = (E, dE/dsite0, dE/dsite1) of one pose by W warps
// (W = 1, 2, 4, 8 consecutive warps of a 256-thread CTA share the pose; every
// warp of the CTA calls this together and gets its pose's whole sums).  part:
// shared memory [8][7].  MIXED = false: the FP64 mode (every entry near).
template <bool MIXED, int LOADS>
__device__ __forceinline__ void pose_eval(const PoseBatchSys &y, const double *q,
                                          const double *center, int W, int warp, int lane,
                                          double (*part)[7], double band_lo, double band_hi,
                                          int *status, PosePoint &pt, double (&v)[7]) {
    const int sub = warp % W;
    const double nq = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    bool ok = isfinite(nq) && nq > 0;
    const double qw = ok ? q[0] / nq : 1.0, qx = ok ? q[1] / nq : 0.0,
                 qy = ok ? q[2] / nq : 0.0, qz = ok ? q[3] / nq : 0.0;
    const double u[3] = {1.0 - 2.0 * (qy * qy + qz * qz), 2.0 * (qx * qy + qw * qz),
                         2.0 * (qx * qz - qw * qy)};
    const double c0 = center[0], c1 = center[1], c2 = center[2];
    double f[3];
    int b[3];
    const int nb[3] = {y.nb0, y.nb1, y.nb2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double w = c0 * y.Hinv.m[k] + c1 * y.Hinv.m[3 + k] + c2 * y.Hinv.m[6 + k];
        ok = ok && isfinite(w);
        w = isfinite(w) ? w - floor(w) : 0.0;
        if (w >= 1.0) w = 0.0;
        f[k] = w;
        b[k] = min(nb[k] - 1, (int)(w * nb[k]));
    }
    if (!ok && lane == 0) atomicExch(status, DEV_BAD_INPUT);
    pt.q[0] = qw;
    pt.q[1] = qx;
    pt.q[2] = qy;
    pt.q[3] = qz;
    pt.norm = nq;
    pt.ok = ok;
    const RegionInfo r = y.regs[(b[0] * y.nb1 + b[1]) * y.nb2 + b[2]];
    double cx, cy, cz;
    frac_to_cart(y.H, f[0] - r.of[0], f[1] - r.of[1], f[2] - r.of[2], cx, cy, cz);
    double sd[2][3];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double off = s ? y.off1 : y.off0;
        sd[s][0] = cx + off * u[0];
        sd[s][1] = cy + off * u[1];
        sd[s][2] = cz + off * u[2];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) v[k] = 0.0;
    pose_sums<!MIXED, LOADS>(y, r, sd, lane + 32 * sub, 32 * W, v);
    warp_reduce7(v);
    if (W > 1) {   // (W is a launch argument: uniform over the CTA)
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < 7; ++k) part[warp][k] = v[k];
        __syncthreads();
        const int w0 = warp - sub;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            double t = part[w0][k];
            for (int j = 1; j < W; ++j) t += part[w0 + j][k];
            v[k] = t;
        }
        __syncthreads();
    }
    // the refinement band: the pose again in FP64, by all of its warps
    // (uniform over them: each holds the pose's v[0])
    if (MIXED) {
        const bool again = v[0] > band_lo && v[0] < band_hi;
        if (again) {
#pragma unroll
            for (int k = 0; k < 7; ++k) v[k] = 0.0;
            pose_sums<true, LOADS, false>(y, r, sd, lane + 32 * sub, 32 * W, v);
            warp_reduce7(v);
        }
        if (W > 1) {   // every warp of the CTA passes both barriers
            if (again && lane == 0)
#pragma unroll
                for (int k = 0; k < 7; ++k) part[warp][k] = v[k];
            __syncthreads();
            if (again) {
                const int w0 = warp - sub;
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    double t = part[w0][k];
                    for (int j = 1; j < W; ++j) t += part[w0 + j][k];
                    v[k] = t;
                }
            }
            __syncthreads();
        }
    }
}

}  // namespace vext
