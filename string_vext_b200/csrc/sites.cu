// The site-by-site field sum (sites.cuh): plan, warp-per-cluster kernel, and
// the forward sum of a pose's two sites.  The forward + adjoint poses are put
// together in batch.cu, beside the other batch kernels' outputs.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pair.cuh"
#include "sitepose.cuh"

namespace vext {

// ---------------------------------------------------------------- kernel

struct SiteArgs {
    SiteView v;
    double *value;            // SiteScratch::value
    int near_in;              // near pairs provably inside the cutoff
    int region0;              // first region
};

constexpr int kSiteWarps = 2;     // clusters per CTA
constexpr int kFarQueue = 32;     // entries a far queue gathers before they are taken
constexpr int kNearQueue = 8;

// FP64 pairs reach this far (A) beyond r_split.  Lists about regions of poses
// hold every pair within r_split in FP64 and most within another 0.5-1.5 A
// (site offset and region radius); without them the FP32 errors would grow: of
// 24 fields of a dense and a sparse cell the mean rms error at E <= 0 is 2.2e-5
// and 7.0e-6 K pose by pose with 8-center regions, 1.6e-5 and 5.8e-6 K with
// 16-center ones, 2.3e-5 and 6.7e-6 K here without the margin, 1.6e-5 and 3.3e-6
// K with it (60^3 x 64 layered adjoint 13.94 -> 14.66 ms).
constexpr double kNearMargin = 0.9;

// Entries waiting in shared memory, per warp: FP32 ones as the operand pairs
// of the packed instructions.
struct SiteQueue {
    float4 xy[kFarQueue + 32], zc[kFarQueue + 32];       // inside: (x,x,y,y), (z,z,c12,c12)
    float4 sxy[kFarQueue + 32], szc[kFarQueue + 32];     // shell
    float4 scs[kFarQueue + 32];                          // (-c6, limit, shift, index)
    double2 near[kNearQueue + 32][4];                    // (x,y), (z,c12), (c6,shift), (floor2,
                                                         // test: 1)
    float2 c6[kFarQueue + 32];                           // inside: (-c6,-c6)
};

// A lane's two sites.
struct SitePoint {
    double p[2][3];
    float2 nx, ny, nz;        // minus the positions
};
struct SiteSum {
    double e[2], g[2][3];     // g: the gradient is -6 g
};
struct SitePartial {
    float2 e, gx, gy, gz;
};

// One far entry (a, b: queue entry; c6: minus the coefficient), both sites of
// the lane.  MASK: added where d2 < limit, or, with a limit above rc2f, taken
// off where d2 >= limit; near_rc collects the least |d2 - rc2f|.
template <bool ADJ, bool MASK>
__device__ __forceinline__ void site_pair(float4 a, float4 b, float2 mc6, float shift,
                                          const SitePoint &t, float limit, float rc2f,
                                          SitePartial &s, float &near_rc) {
    const float2 dx = __fadd2_rn(make_float2(a.x, a.y), t.nx),
                 dy = __fadd2_rn(make_float2(a.z, a.w), t.ny),
                 dz = __fadd2_rn(make_float2(b.x, b.y), t.nz);
    const float2 c12 = make_float2(b.z, b.w);
    const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    float r0, r1;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d2.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d2.y));
    const float2 n1 = make_float2(r0, r1);
    float2 n3 = __fmul2_rn(__fmul2_rn(n1, n1), n1);
    // e = n3 (c12 n3 - c6), dE/dd2 = -3 n1 n3 (2 c12 n3 - c6)
    const float2 w = __fmul2_rn(c12, n3);
    const float2 x = __fadd2_rn(w, mc6);
    if (MASK) {
        const float all = limit > rc2f ? -1.f : 0.f;
        const float2 m = __fadd2_rn(make_float2(set_lt(d2.x, limit), set_lt(d2.y, limit)),
                                    make_float2(all, all));
        near_rc = fminf(near_rc, fminf(fabsf(d2.x - rc2f), fabsf(d2.y - rc2f)));
        n3 = __fmul2_rn(n3, m);
        s.e = __ffma2_rn(m, make_float2(shift, shift), s.e);
    }
    s.e = __ffma2_rn(n3, x, s.e);
    if (ADJ) {
        const float2 f = __fmul2_rn(__fmul2_rn(n1, n3), __fadd2_rn(w, x));
        s.gx = __ffma2_rn(f, dx, s.gx);
        s.gy = __ffma2_rn(f, dy, s.gy);
        s.gz = __ffma2_rn(f, dz, s.gz);
    }
}

template <bool ADJ>
__device__ __forceinline__ void add_energy(SitePartial &s, SiteSum &sum) {
    sum.e[0] += (double)s.e.x;
    sum.e[1] += (double)s.e.y;
    s.e = make_float2(0.f, 0.f);
}

// d in site_pair is entry - site, in site_near site - entry: g changes sign.
template <bool ADJ>
__device__ __forceinline__ void add_gradient(const SitePartial &s, SiteSum &sum) {
    if (!ADJ) return;
    sum.g[0][0] -= (double)s.gx.x;
    sum.g[1][0] -= (double)s.gx.y;
    sum.g[0][1] -= (double)s.gy.x;
    sum.g[1][1] -= (double)s.gy.y;
    sum.g[0][2] -= (double)s.gz.x;
    sum.g[1][2] -= (double)s.gz.y;
}

// One near entry in FP64, both sites.  TEST: with the cutoff test and the
// contact floor.
template <bool ADJ, bool TEST>
__device__ __forceinline__ void site_near(const double2 *n, const SitePoint &t, double rc2,
                                          SiteSum &sum) {
    const double2 a = n[0], b = n[1], c = n[2];
    const double fl = TEST ? n[3].x : 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const double dx = t.p[h][0] - a.x, dy = t.p[h][1] - a.y, dz = t.p[h][2] - b.x;
        const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
        const double s2 = TEST ? fmax(d2, fl) : d2;
        const double i2 = rcp64_nr<1>(s2);
        const double i6 = i2 * i2 * i2;
        const double w = b.y * i6, x = w - c.x;
        double en = fma(i6, x, c.y);
        if (TEST) en = d2 < rc2 ? en : 0.0;
        sum.e[h] += en;
        if (ADJ) {
            double f = (i2 * i6) * (x + w);
            if (TEST) f = d2 < fl || d2 >= rc2 ? 0.0 : f;
            sum.g[h][0] = fma(f, dx, sum.g[h][0]);
            sum.g[h][1] = fma(f, dy, sum.g[h][1]);
            sum.g[h][2] = fma(f, dz, sum.g[h][2]);
        }
    }
}

template <bool ADJ>
__device__ __forceinline__ void take_near(const SiteQueue &q, int n, const SitePoint &t,
                                          double rc2, SiteSum &sum) {
    int j = 0;
#pragma unroll 1
    for (; j + 1 < n; j += 2) {
        if (q.near[j][3].y + q.near[j + 1][3].y == 0.0) {
            // two entries side by side: their chains are long
            site_near<ADJ, false>(q.near[j], t, rc2, sum);
            site_near<ADJ, false>(q.near[j + 1], t, rc2, sum);
        } else {
            site_near<ADJ, true>(q.near[j], t, rc2, sum);
            site_near<ADJ, true>(q.near[j + 1], t, rc2, sum);
        }
    }
    if (j < n) site_near<ADJ, true>(q.near[j], t, rc2, sum);
}

template <bool ADJ>
__device__ __forceinline__ void take_inside(const SiteQueue &q, int n, const SitePoint &t,
                                            SiteSum &sum) {
    SitePartial s;
    s.e = s.gx = s.gy = s.gz = make_float2(0.f, 0.f);
    float unused = 0.f;
    int j = 0;
    // energy partials over 8 entries (kExpandFlush)
#pragma unroll 1
    for (; j + 8 <= n; j += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            site_pair<ADJ, false>(q.xy[j + k], q.zc[j + k], q.c6[j + k], 0.f, t, 0.f, 0.f, s,
                                  unused);
        add_energy<ADJ>(s, sum);
    }
#pragma unroll 1
    for (; j < n; ++j)
        site_pair<ADJ, false>(q.xy[j], q.zc[j], q.c6[j], 0.f, t, 0.f, 0.f, s, unused);
    add_energy<ADJ>(s, sum);
    add_gradient<ADJ>(s, sum);
}

// Entries of the cutoff shell; those in the expansion have a limit above rc^2
// and are taken off where they lie outside.  Pairs whose FP32 d2 lies within
// kBorderTol of rc^2 stay out of the FP32 sums and are decided and added in
// FP64 (rare: the queue is gone through again for them).
template <bool ADJ>
__device__ __forceinline__ void take_shell(const SiteQueue &q, int n, const SitePoint &t,
                                           const SiteView &v, long long off, SiteSum &sum) {
    SitePartial s;
    s.e = s.gx = s.gy = s.gz = make_float2(0.f, 0.f);
    float near_rc = 1.f;
    int j = 0;
#pragma unroll 1
    for (; j + 4 <= n; j += 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 c = q.scs[j + k];
            site_pair<ADJ, true>(q.sxy[j + k], q.szc[j + k], make_float2(c.x, c.x), c.z, t, c.y,
                                 v.rc2f, s, near_rc);
        }
        if ((j & 12) == 12) add_energy<ADJ>(s, sum);   // partials over 16, as pose by pose
    }
#pragma unroll 1
    for (; j < n; ++j) {
        const float4 c = q.scs[j];
        site_pair<ADJ, true>(q.sxy[j], q.szc[j], make_float2(c.x, c.x), c.z, t, c.y, v.rc2f, s,
                             near_rc);
    }
    add_energy<ADJ>(s, sum);
    add_gradient<ADJ>(s, sum);
    const float lo = v.rc2f - kBorderTol, hi = v.rc2f + kBorderTol;
    if (near_rc <= fmaxf(v.rc2f - lo, hi - v.rc2f)) {
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            const float4 a = q.sxy[k], b = q.szc[k], c = q.scs[k];
            const float2 dx = __fadd2_rn(make_float2(a.x, a.y), t.nx),
                         dy = __fadd2_rn(make_float2(a.z, a.w), t.ny),
                         dz = __fadd2_rn(make_float2(b.x, b.y), t.nz);
            const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            const double taken = c.y > v.rc2f ? 1.0 : 0.0;   // by the expansion
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float d = h ? d2.y : d2.x;
                if (d < lo || d >= hi) continue;   // the FP32 sums decided it
                const int at = __float_as_int(c.w);
                const float4 hh = v.hi[off + at], l = v.lo[off + at];
                const double *td = v.td + 4 * __float_as_int(hh.w);
                const double x = t.p[h][0] - ((double)hh.x + (double)l.x),
                             y = t.p[h][1] - ((double)hh.y + (double)l.y),
                             z = t.p[h][2] - ((double)hh.z + (double)l.z);
                const double r2 = fma(x, x, fma(y, y, z * z));
                const double wt = (r2 < v.rc2 ? 1.0 : 0.0) - taken;
                const double i2 = rcp64_nr<2>(r2);
                const double i6 = i2 * i2 * i2, w = td[0] * i6;
                sum.e[h] += wt * fma(i6, w - td[1], td[2]);
                const double f = wt * (i2 * i6) * (2.0 * w - td[1]);
                sum.g[h][0] = fma(f, x, sum.g[h][0]);
                sum.g[h][1] = fma(f, y, sum.g[h][1]);
                sum.g[h][2] = fma(f, z, sum.g[h][2]);
            }
        }
    }
}

// A warp takes one cluster of one region through the entries that the region's
// expansion leaves: every lane classifies one entry of a group of 32 by its
// distance from the cluster's middle (nearer than r_split + kNearMargin +
// radius: FP64; inside rc - radius: FP32 without a test; up to rc + radius:
// FP32 with the cutoff test; beyond: nothing) and queues it; once a queue is
// full all lanes take its entries, two sites each.  No barrier, no staging: the
// entries come from L1/L2, the warps are independent.
//
// The expansion holds all entries within rc of the region's origin, also those
// in its shell: a cluster takes off the few that lie outside for its sites,
// instead of adding the many that lie inside (in all: layered adjoint 12.5 ->
// 11.2 ms; up to rc - 0.4 radius of the region 11.5, to rc + 0.3 radius 11.5).
//
// 60^3 x 64 layered forward + adjoint: 8.8 of 11.2 ms (pose by pose, on lists
// about regions of poses, 18.1 in all), about 1.3 of it classification and 3.6
// near entries.  Bound by the latency of the FP64 and FP32 chains at 16 warps
// per SM (issue slots 58 %, FP64 pipe 39 %, FMA pipe 29 % busy; 20 warps with
// spills are slower, forward 20 beat 24 by 1-2 %).  Hence eight inside entries,
// four shell entries and two near ones side by side (half as many: 2 % slower,
// one near entry: 3 %), taken from full queues: straight from each group of 32
// the sums took 0.8 ms more.  Two warps a CTA leave fewer idle than four at odd
// cluster counts (47^3 x 50 skewed field 1 %).
template <bool ADJ>
__global__ void __launch_bounds__(32 * kSiteWarps, (ADJ ? 16 : 20) / kSiteWarps)
    site_cluster_kernel(SiteArgs g) {
    __shared__ SiteQueue queue[kSiteWarps];
    const SiteView &v = g.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (v.n_clusters + kSiteWarps - 1) / kSiteWarps;
    const int region = g.region0 + blockIdx.x / per, k = blockIdx.x % per * kSiteWarps + warp;
    if (k >= v.n_clusters) return;
    SiteQueue &q = queue[warp];
    const RegionInfo &r = v.regs[region];
    const float4 mid = v.cluster[k];
    const int s0 = k * kClusterSites + lane;   // and s0 + 32
    SitePoint t;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 3; ++i) t.p[h][i] = v.pos[3 * (s0 + 32 * h) + i];
    t.nx = make_float2(-(float)t.p[0][0], -(float)t.p[1][0]);
    t.ny = make_float2(-(float)t.p[0][1], -(float)t.p[1][1]);
    t.nz = make_float2(-(float)t.p[0][2], -(float)t.p[1][2]);
    // class radii; 1e-4 A covers the FP32 distances
    const float rn = (float)(v.r_split + kNearMargin) + mid.w + 1e-4f,
                ri = fmaxf(v.rc - mid.w - 1e-4f, 0.f), ro = v.rc + mid.w + 1e-4f;
    const float rn2 = rn * rn, ri2 = ri * ri, ro2 = ro * ro;
    const float rf = (float)v.floor_out + mid.w + 1e-4f;
    const float rf2 = g.near_in ? rf * rf : 1e30f;   // near entries nearer: tested
    SiteSum sum;
    sum.e[0] = sum.e[1] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) sum.g[0][i] = sum.g[1][i] = 0.0;
    double shift_in = 0.0;   // entries inside the cutoff of every site
    const long long off = r.off;
    const int near_end = v.poly ? r.n_near + r.n_mid : r.n_total;
    const int far_from = v.poly ? r.n_near + r.n_inner : r.n_total, total = r.n_total;
    // shell entries that the expansion holds
    const int taken_from = v.poly ? far_from : 0, taken_to = v.poly ? far_from + r.n_shella : 0;
    int n_near = 0, n_in = 0, n_shell = 0;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        const int end = part ? total : near_end;
        int base = part ? far_from : 0;
        float4 next = base + lane < end ? v.hi[off + base + lane] : make_float4(0, 0, 0, 0);
#pragma unroll 1
        for (; base < end; base += 32) {
            const float4 h = next;
            const bool mine = base + lane < end;
            if (base + 32 + lane < end) next = v.hi[off + base + 32 + lane];
            const float cx = h.x - mid.x, cy = h.y - mid.y, cz = h.z - mid.z;
            const float d2c = fmaf(cx, cx, fmaf(cy, cy, cz * cz));
            const bool taken = base + lane >= taken_from && base + lane < taken_to;
            const bool near = mine && !taken && d2c < rn2;
            const bool in = mine && !near && !taken && d2c < ri2;
            const bool shell = mine && !near && d2c >= ri2 && (taken || d2c < ro2);
            const unsigned mn = __ballot_sync(0xffffffffu, near),
                           mi = __ballot_sync(0xffffffffu, in),
                           ms = __ballot_sync(0xffffffffu, shell), below = (1u << lane) - 1;
            if (in || shell) {
                const float4 tp = v.tf[__float_as_int(h.w)];   // (c12, c6, shift, -)
                if (in) {
                    const int at = n_in + __popc(mi & below);
                    q.xy[at] = make_float4(h.x, h.x, h.y, h.y);
                    q.zc[at] = make_float4(h.z, h.z, tp.x, tp.x);
                    q.c6[at] = make_float2(-tp.y, -tp.y);
                    shift_in += (double)tp.z;
                } else {
                    const int at = n_shell + __popc(ms & below);
                    q.sxy[at] = make_float4(h.x, h.x, h.y, h.y);
                    q.szc[at] = make_float4(h.z, h.z, tp.x, tp.x);
                    q.scs[at] =
                        make_float4(-tp.y, taken ? v.rc2f + kBorderTol : v.rc2f - kBorderTol, tp.z,
                                    __int_as_float(base + lane));
                }
            } else if (near) {
                const float4 l = v.lo[off + base + lane];
                const double *td = v.td + 4 * __float_as_int(h.w);
                double2 *n = q.near[n_near + __popc(mn & below)];
                n[0] = make_double2((double)h.x + (double)l.x, (double)h.y + (double)l.y);
                n[1] = make_double2((double)h.z + (double)l.z, td[0]);
                n[2] = make_double2(td[1], td[2]);
                n[3] = make_double2(td[3], d2c < rf2 ? 1.0 : 0.0);
            }
            n_near += __popc(mn);
            n_in += __popc(mi);
            n_shell += __popc(ms);
            const bool last = part == 1 ? base + 32 >= end : base + 32 >= end && far_from >= total;
            const bool do_near = n_near >= kNearQueue || last, do_in = n_in >= kFarQueue || last,
                       do_shell = n_shell >= kFarQueue || last;
            if (!(do_near || do_in || do_shell)) continue;
            __syncwarp();
            if (do_near) {
                take_near<ADJ>(q, n_near, t, v.rc2, sum);
                n_near = 0;
            }
            if (do_in) {
                take_inside<ADJ>(q, n_in, t, sum);
                n_in = 0;
            }
            if (do_shell) {
                take_shell<ADJ>(q, n_shell, t, v, off, sum);
                n_shell = 0;
            }
            __syncwarp();
        }
    }
    shift_in = warp_total(shift_in);
    // ---- outputs
    const long long S3 = (long long)v.S * v.S * v.S;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int s = s0 + 32 * h;
        const int4 m0 = v.meta[2 * s], m1 = v.meta[2 * s + 1];
        const int vi = r.i0 + m0.y, vj = r.j0 + m0.z, vk = r.k0 + m0.w;
        if (m0.x < 0 || vi >= v.S || vj >= v.S || vk >= v.S) continue;
        double e = sum.e[h] + shift_in;
        double gr[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) gr[i] = -6.0 * sum.g[h][i];
        if (v.poly) {
            const double *pp = v.poly + (size_t)region * kTaylorPolyPad;
            const double px = t.p[h][0], py = t.p[h][1], pz = t.p[h][2];
            const size_t at = (size_t)region * v.n_sites + s;
            if (ADJ) {
                double pg[3];
                e += taylor_poly_grad(pp, px, py, pz, pg);
                const float4 w = reinterpret_cast<const float4 *>(v.eval)[at];
                e += (double)w.x;
                gr[0] += pg[0] + (double)w.y;
                gr[1] += pg[1] + (double)w.z;
                gr[2] += pg[2] + (double)w.w;
            } else {
                e += taylor_poly(pp, px, py, pz);
                e += (double)v.eval[at];
            }
        }
        const int ci = wrap(vi + m1.x, v.S), cj = wrap(vj + m1.y, v.S), ck = wrap(vk + m1.z, v.S);
        const long long c = ((long long)ci * v.S + cj) * v.S + ck;
        if (ADJ) {
            double2 *out = reinterpret_cast<double2 *>(g.value + 4 * (m0.x * S3 + c));
            out[0] = make_double2(e, gr[0]);
            out[1] = make_double2(gr[1], gr[2]);
        } else {
            g.value[m0.x * S3 + c] = e;
        }
    }
}

__global__ void site_energy_kernel(const double *value, long long S3, int O, double *e64) {
    const long long n = S3 * O;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const long long o = i / S3, c = i - o * S3;
        e64[i] = value[2 * o * S3 + c] + value[(2 * o + 1) * S3 + c];
    }
}

// ---------------------------------------------------------------- plan

// Radius of a cluster (A) up to which poses are summed site by site: the
// region's by the cube root of its share of the 16 n_axes sites.  The finer the
// grid, the more is gained (18.1 -> 11.2 ms at 0.25 A); four uneven frameworks at
// 35^3 x 64 with clusters of 0.4-1.4 A, forward + adjoint: none by sites 19.6 ms,
// up to 0.8 A 16.4, up to 1 A or all 16.75.
constexpr double kSiteRadius = 0.8;

// Images within rc of a site from which on the sum site by site pays: its values
// pass through memory once more (0.5 ms forward, 0.8 forward + adjoint at 60^3 x
// 64), its clusters win on the pairs.  Pose by pose against site by site, forward
// and forward + adjoint, at 60^3 x 64 in a 30 A cell: 70 images 1.36 / 1.93 and
// 2.39 / 2.98 ms, 140 images 2.45 / 2.29 and 3.66 / 3.48, 280 images 3.71 / 3.37 and
// 7.40 / 4.83; at 42^3 x 43 in 20 and 28 A cells the ratio is 0.83-0.89 and 1.02-1.04
// with 70 images, 1.20-1.28 and 1.20-1.31 with 140.
constexpr double kSiteImages = 110;

// Bytes of scratch beyond which a field is summed pose by pose.
constexpr long long kSiteScratch = 8LL << 30;

// Blocks of `n` voxels of the smallest half diagonal.
static double site_block(const Mat3 &H, int size, int n, int &bi, int &bj, int &bk) {
    double best = 1e300;
    for (int a = 1; a <= n; ++a)
        for (int b = 1; a * b <= n; ++b) {
            if (n % (a * b)) continue;
            const int c = n / (a * b);
            if (a > size || b > size || c > size) continue;
            const double r = block_radius(H, size, a + 1, b + 1, c + 1);
            if (r < best - 1e-12) {
                best = r;
                bi = a;
                bj = b;
                bk = c;
            }
        }
    return best;
}

struct SiteLayout {
    int bi = 0, bj = 0, bk = 0;
    std::vector<double> pos, shift;           // [n_sites][3], [2 O][3]
    std::vector<int> meta, floor;             // [n_sites][8], [2 O][4]
    std::vector<float> cluster;               // [n_clusters][4]
};

// Split sites [first, last) of `order` at multiples of the cluster size across
// their longest extent until single clusters are left.
static void split_sites(const std::vector<double> &pos, std::vector<int> &order, int first,
                        int last) {
    const int n = last - first;
    if (n <= kClusterSites) return;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int k = first; k < last; ++k)
        for (int d = 0; d < 3; ++d) {
            lo[d] = std::min(lo[d], pos[3 * (size_t)order[k] + d]);
            hi[d] = std::max(hi[d], pos[3 * (size_t)order[k] + d]);
        }
    int d = 0;
    for (int k = 1; k < 3; ++k)
        if (hi[k] - lo[k] > hi[d] - lo[d]) d = k;
    const int clusters = (n + kClusterSites - 1) / kClusterSites;
    const int half = first + (clusters + 1) / 2 * kClusterSites;
    std::nth_element(order.begin() + first, order.begin() + half, order.begin() + last,
                     [&](int a, int b) {
                         const double x = pos[3 * (size_t)a + d], y = pos[3 * (size_t)b + d];
                         return x < y || (x == y && a < b);
                     });
    split_sites(pos, order, first, half);
    split_sites(pos, order, half, last);
}

static void site_layout(const System &sys, const RegionSet &rs, int n_axes, const double *axes,
                        SiteLayout &l) {
    const int size = rs.size;
    l.bi = rs.bi;
    l.bj = rs.bj;
    l.bk = rs.bk;
    const int per = l.bi * l.bj * l.bk, n = 2 * n_axes * per;
    std::vector<double> pos(3 * (size_t)n);
    std::vector<int> meta(8 * (size_t)n);
    l.shift.resize(6 * (size_t)n_axes);
    l.floor.assign(8 * (size_t)n_axes, 0);
    int at = 0;
    for (int o = 0; o < n_axes; ++o)
        for (int s = 0; s < 2; ++s) {
            const double off = sys.offsets[s];
            const double *u = axes + 3 * o;
            double f[3];
            int fl[3];
            for (int k = 0; k < 3; ++k) {
                const double d = off * (u[0] * sys.Hinv.m[k] + u[1] * sys.Hinv.m[3 + k] +
                                        u[2] * sys.Hinv.m[6 + k]);
                const double x = 0.5 + size * d;
                fl[k] = (int)std::floor(x);
                f[k] = x - std::floor(x);
                l.shift[3 * (size_t)(2 * o + s) + k] = f[k];
                l.floor[4 * (size_t)(2 * o + s) + k] = fl[k];
            }
            for (int a = 0; a < l.bi; ++a)
                for (int b = 0; b < l.bj; ++b)
                    for (int c = 0; c < l.bk; ++c) {
                        frac_to_cart(sys.H, (a + f[0] - 0.5 * l.bi) / size,
                                     (b + f[1] - 0.5 * l.bj) / size, (c + f[2] - 0.5 * l.bk) / size,
                                     pos[3 * (size_t)at], pos[3 * (size_t)at + 1],
                                     pos[3 * (size_t)at + 2]);
                        const int m[8] = {2 * o + s, a, b, c, -fl[0], -fl[1], -fl[2], 0};
                        std::copy(m, m + 8, &meta[8 * (size_t)at]);
                        ++at;
                    }
        }
    std::vector<int> order(n);
    for (int k = 0; k < n; ++k) order[k] = k;
    split_sites(pos, order, 0, n);
    const int clusters = (n + kClusterSites - 1) / kClusterSites, padded = clusters * kClusterSites;
    l.pos.resize(3 * (size_t)padded);
    l.meta.resize(8 * (size_t)padded);
    l.cluster.resize(4 * (size_t)clusters);
    for (int k = 0; k < padded; ++k) {
        // the last cluster's idle places repeat its first site, unwritten
        const int from = k < n ? order[k] : order[(clusters - 1) * kClusterSites];
        std::copy(&pos[3 * (size_t)from], &pos[3 * (size_t)from] + 3, &l.pos[3 * (size_t)k]);
        std::copy(&meta[8 * (size_t)from], &meta[8 * (size_t)from] + 8, &l.meta[8 * (size_t)k]);
        if (k >= n) l.meta[8 * (size_t)k] = -1;
    }
    for (int k = 0; k < clusters; ++k) {
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, r = 0;
        for (int i = k * kClusterSites; i < (k + 1) * kClusterSites; ++i)
            for (int d = 0; d < 3; ++d) {
                lo[d] = std::min(lo[d], l.pos[3 * (size_t)i + d]);
                hi[d] = std::max(hi[d], l.pos[3 * (size_t)i + d]);
            }
        for (int i = k * kClusterSites; i < (k + 1) * kClusterSites; ++i) {
            double d2 = 0;
            for (int d = 0; d < 3; ++d) {
                const double x = l.pos[3 * (size_t)i + d] - (float)(0.5 * (lo[d] + hi[d]));
                d2 += x * x;
            }
            r = std::max(r, std::sqrt(d2));
        }
        for (int d = 0; d < 3; ++d) l.cluster[4 * (size_t)k + d] = (float)(0.5 * (lo[d] + hi[d]));
        l.cluster[4 * (size_t)k + 3] = (float)(r * (1 + 1e-6));
    }
}

bool sites_worthwhile(const System &sys, int size, int n_axes, const Options &o, bool adjoint) {
    // pinned kernels and region sizes keep the sum pose by pose
    if (o.variant || o.batch_shape || o.cb || o.mode != VEXT_MODE_MIXED) return false;
    // fewer than four clusters a region; a plan of more than 0.25 GB
    if (size < 8 || n_axes < 16 || n_axes > 1024) return false;
    const long long S3 = (long long)size * size * size;
    const double *h = sys.H.m;
    const double volume = h[0] * (h[4] * h[8] - h[5] * h[7]) - h[1] * (h[3] * h[8] - h[5] * h[6]) +
                          h[2] * (h[3] * h[7] - h[4] * h[6]);
    if (4.18879 * sys.cutoff * sys.cutoff * sys.cutoff * sys.n_atoms < kSiteImages * volume)
        return false;
    // scratch: V (and its gradient) at every site, and the expansions' part of it
    if (S3 * n_axes * 2 * (adjoint ? 48 : 12) > kSiteScratch) return false;
    int bi = 0, bj = 0, bk = 0;
    const double radius = site_block(sys.H, size, 8, bi, bj, bk);
    return radius * std::cbrt(4.0 / n_axes) < kSiteRadius &&
           o.r_split + kNearMargin + 2 * radius < sys.cutoff;
}

int get_site_regions(System *sys, int size, int block, double r_split, RegionSet **out,
                     cudaStream_t stream) {
    int bi = 0, bj = 0, bk = 0;
    const double radius = site_block(sys->H, size, block, bi, bj, bk) + 1e-9;
    return get_block_regions(sys, size, bi, bj, bk, radius, 0.0, true, true, r_split, out,
                             stream);
}

int site_plan_build(const System &sys, const RegionSet &rs, int n_axes, const double *axes,
                    bool adjoint, SitePlan &plan, cudaStream_t stream) {
    SiteLayout l;
    site_layout(sys, rs, n_axes, axes, l);
    size_t bytes = 0;
    auto place = [&bytes](size_t n) {
        const size_t at = bytes;
        bytes = (bytes + n + 255) & ~(size_t)255;
        return at;
    };
    const size_t at_pos = place(sizeof(double) * l.pos.size()),
                 at_meta = place(sizeof(int) * l.meta.size()),
                 at_cluster = place(sizeof(float) * l.cluster.size()),
                 at_shift = place(sizeof(double) * l.shift.size()),
                 at_floor = place(sizeof(int) * l.floor.size());
    std::vector<char> up(bytes, 0);
    std::memcpy(&up[at_pos], l.pos.data(), sizeof(double) * l.pos.size());
    std::memcpy(&up[at_meta], l.meta.data(), sizeof(int) * l.meta.size());
    std::memcpy(&up[at_cluster], l.cluster.data(), sizeof(float) * l.cluster.size());
    std::memcpy(&up[at_shift], l.shift.data(), sizeof(double) * l.shift.size());
    std::memcpy(&up[at_floor], l.floor.data(), sizeof(int) * l.floor.size());
    char *base = static_cast<char *>(plan.arena);
    VEXT_TRY(ensure_capacity(base, plan.arena_cap, bytes));
    plan.arena = base;
    // in stream order: calls before this one may still read the old plan
    VEXT_CUDA(cudaMemcpyAsync(base, up.data(), bytes, cudaMemcpyHostToDevice, stream));
    SiteView &v = plan.view;
    v.H = sys.H;
    v.rc2 = sys.cutoff * sys.cutoff;
    v.rc2f = (float)v.rc2;
    v.rc = (float)sys.cutoff;
    v.off0 = sys.offsets[0];
    v.off1 = sys.offsets[1];
    v.r_split = rs.r_split;
    double fl = 0.0;
    for (int t = 0; t < sys.n_types; ++t) fl = std::max(fl, sys.h_td[4 * t + 3]);
    v.floor_out = std::sqrt(fl);
    v.S = rs.size;
    v.O = n_axes;
    v.regs = rs.d_info;
    v.hi = rs.d_hi;
    v.lo = rs.d_lo;
    v.tf = sys.d_tf;
    v.td = sys.d_td;
    v.n_regions = rs.n_regions;
    v.bi = rs.bi;
    v.bj = rs.bj;
    v.bk = rs.bk;
    v.nrj = rs.n_rj;
    v.nrk = rs.n_rk;
    v.n_clusters = (int)(l.cluster.size() / 4);
    v.n_sites = v.n_clusters * kClusterSites;
    v.pos = reinterpret_cast<const double *>(base + at_pos);
    v.meta = reinterpret_cast<const int4 *>(base + at_meta);
    v.cluster = reinterpret_cast<const float4 *>(base + at_cluster);
    v.shift = reinterpret_cast<const double *>(base + at_shift);
    v.floor = reinterpret_cast<const int4 *>(base + at_floor);
    v.poly = nullptr;
    v.eval = nullptr;
    // an expansion costs about 1,000 operations an entry and 140 an output (the
    // 28,800 regions of the 60^3 x 64 layered field: 1.83 and 0.44 ms); it takes 12
    // (forward 9) off every (site, entry) pair
    const double n = (double)rs.n_taylor / std::max(rs.n_regions, 1);
    if (taylor_allowed(sys, rs) && n * v.n_sites * (adjoint ? 12.0 : 9.0) >
                                       n * 1000.0 + v.n_sites * (adjoint ? 4 : 1) * 140.0) {
        VEXT_TRY(taylor_prepare_sites(sys, rs, v.n_sites, v.pos, adjoint, plan.expansion, stream));
        v.poly = plan.expansion.poly;
    }
    plan.rs = &rs;
    plan.reach_lo = plan.reach_hi = 0;
    for (int k = 0; k < 2 * n_axes; ++k) {
        plan.reach_lo = std::max(plan.reach_lo, -l.floor[4 * (size_t)k]);
        plan.reach_hi = std::max(plan.reach_hi, l.floor[4 * (size_t)k]);
    }
    return 0;
}

// Scratch from which on it has to leave as much again free: the sum pose by pose
// needs none of it, and what the rest of the call and the program allocate later
// should still fit.  (Not less: cudaMemGetInfo takes 70 us, and calls that make
// and drop a system would pay it each time.)
constexpr size_t kSiteScratchCareful = 1u << 30;

int site_scratch_reserve(const SitePlan &plan, bool adjoint, SiteScratch &s) {
    const SiteView &v = plan.view;
    const size_t S3 = (size_t)v.S * v.S * v.S, words = adjoint ? 4 : 1,
                 value = 2 * v.O * S3 * words,
                 sums = v.poly ? taylor_workspace_sites(*plan.rs) : 0,
                 eval = v.poly ? (size_t)v.n_regions * v.n_sites * words : 0;
    const size_t more = (value > s.value_cap ? 8 * value : 0) +
                        (sums > s.sums_cap ? 4 * sums : 0) + (eval > s.eval_cap ? 4 * eval : 0);
    if (more >= kSiteScratchCareful) {
        size_t free = 0, total = 0;
        VEXT_CUDA(cudaMemGetInfo(&free, &total));
        if (2 * more > free)
            return fail(VEXT_ERR_MEMORY, "%zu bytes of scratch, %zu free", more, free);
    }
    VEXT_TRY(ensure_capacity(s.value, s.value_cap, value));
    if (v.poly) {
        VEXT_TRY(ensure_capacity(s.sums, s.sums_cap, sums));
        VEXT_TRY(ensure_capacity(s.eval, s.eval_cap, eval));
    }
    return 0;
}

SiteView site_view(const SitePlan &plan) {
    SiteView v = plan.view;
    v.regs = plan.rs->d_info;
    v.hi = plan.rs->d_hi;
    v.lo = plan.rs->d_lo;
    return v;
}

int site_enqueue(const System &sys, const SitePlan &plan, bool adjoint,
                 const SiteScratch &scratch, int plane0, int plane1, int *status,
                 cudaStream_t stream) {
    SiteArgs g;
    g.v = site_view(plan);
    g.v.eval = scratch.eval;
    g.value = scratch.value;
    g.near_in = plan.rs->r_split + kNearMargin + 2.0 * plan.rs->taylor_radius + 1e-3 < sys.cutoff;
    const SiteView &v = g.v;
    if (plane1 <= plane0) return 0;
    if (v.poly && plane0 == 0)
        VEXT_TRY(taylor_enqueue_sites(sys, *plan.rs, v.n_sites, plan.expansion, scratch.sums,
                                      scratch.eval, status, stream));
    const int per_plane = v.nrj * v.nrk;
    g.region0 = plane0 * per_plane;
    const unsigned blocks =
        (unsigned)((plane1 - plane0) * per_plane) * ((v.n_clusters + kSiteWarps - 1) / kSiteWarps);
    if (adjoint) site_cluster_kernel<true><<<blocks, 32 * kSiteWarps, 0, stream>>>(g);
    else site_cluster_kernel<false><<<blocks, 32 * kSiteWarps, 0, stream>>>(g);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

int site_energies(const SitePlan &plan, const SiteScratch &scratch, double *e64,
                  cudaStream_t stream) {
    const SiteView &v = plan.view;
    site_energy_kernel<<<1184, 256, 0, stream>>>(scratch.value, (long long)v.S * v.S * v.S, v.O,
                                                 e64);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

void site_field_free(SiteField *f) {
    if (!f) return;
    f->plan.release();
    f->scratch.release();
    delete f;
}

}  // namespace vext
