// Forward + adjoint of many pose sets of different systems in ONE launch:
// the String paths of a batch of frameworks x guests (each path a few dozen
// images), evaluated every iteration.
//
// One to eight warps per pose (more for small batches).  The pose's center is
// wrapped into its system's cell and binned (the bin lists of system.cu, built
// at creation); the lanes stride over the bin's list: near entries in FP64
// from hi + lo with the contact floor, far entries in packed FP32x2 (the two
// sites in the two lanes; reciprocal of d^2 per pair, cubed) with per-lane
// FP32 partials flushed into FP64 every 16 entries.  The seven sums (E,
// dE/dsite for both sites) are reduced over the warp, then over the pose's
// warps in shared memory; a pose whose energy falls in the refinement band is
// recomputed entirely in FP64 by its warps.  Shell pairs whose FP32 d2 lies
// within kBorderTol of the cutoff (where the FP32 and FP64 cutoff tests may
// disagree) are taken in FP64 on the spot.  Outputs as
// vext_pose_energy_grad: E, dE/dcenter, tangent dE/dq, dE/du.  Pair term and
// forces as in pose.cu.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "poseeval.cuh"

namespace vext {

struct PoseBatchArgs {
    const PoseBatchSys *sys;
    const long long *offsets;   // [n_systems + 1]: poses of system k
    int n_systems;
    long long n;
    const double *centers, *quats;
    double *energy, *gc, *gq, *gu;
    double band_lo, band_hi;
    int *status;
    int wpp;                    // warps per pose (set at launch)
};

// a.wpp warps (1, 2, 4 or 8) share a pose, its lanes striding over the bin
// list together, so that small batches (a String path) still fill the GPU;
// the warps' sums are added in shared memory in a fixed order.  MIXED = false:
// the FP64 mode (every entry near, evaluated as in refinement).
template <bool MIXED, int LOADS>
__global__ void __launch_bounds__(256, 2) pose_batch_kernel(PoseBatchArgs a) {
    __shared__ double part[8][7];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = a.wpp, per_cta = 8 / W, sub = warp % W;
    const long long groups = (a.n + per_cta - 1) / per_cta;
    for (long long grp = blockIdx.x; grp < groups; grp += gridDim.x) {   // uniform per CTA
        const long long p0 = grp * per_cta + warp / W;
        const bool live = p0 < a.n;
        const long long p = live ? p0 : a.n - 1;   // idle warps repeat the last pose, unwritten
        // system of pose p: offsets[k] <= p < offsets[k + 1]
        int lo = 0, hi = a.n_systems - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.offsets[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        const PoseBatchSys &y = a.sys[lo];
        PosePoint pt;
        double v[7];
        pose_eval<MIXED, LOADS>(y, a.quats + 4 * p, a.centers + 3 * p, W, warp, lane, part, a.band_lo,
                         a.band_hi, a.status, pt, v);
        if (sub != 0) continue;
        if (live && lane == 0) {
            if (a.energy) a.energy[p] = v[0];
            double gu[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (a.gc) a.gc[3 * p + k] = v[1 + k] + v[4 + k];
                gu[k] = y.off0 * v[1 + k] + y.off1 * v[4 + k];
                if (a.gu) a.gu[3 * p + k] = gu[k];
            }
            if (a.gq) {
                const double qw = pt.q[0], qx = pt.q[1], qy = pt.q[2], qz = pt.q[3];
                // dE/dq = J(q)^T dE/du, projected on the tangent space of |q| = 1
                double g[4];
                g[0] = 2 * qz * gu[1] - 2 * qy * gu[2];
                g[1] = 2 * qy * gu[1] + 2 * qz * gu[2];
                g[2] = -4 * qy * gu[0] + 2 * qx * gu[1] - 2 * qw * gu[2];
                g[3] = -4 * qz * gu[0] + 2 * qw * gu[1] + 2 * qx * gu[2];
                const double dot = g[0] * qw + g[1] * qx + g[2] * qy + g[3] * qz;
                const double inv = pt.ok ? 1.0 / pt.norm : 0.0;
                a.gq[4 * p + 0] = (g[0] - dot * qw) * inv;
                a.gq[4 * p + 1] = (g[1] - dot * qx) * inv;
                a.gq[4 * p + 2] = (g[2] - dot * qy) * inv;
                a.gq[4 * p + 3] = (g[3] - dot * qz) * inv;
            }
        }
    }
}

constexpr long long kWarps = 148 * 16;   // resident warps the launches aim at

// Warps per pose: the smallest power of two up to 8 that gives about kWarps warps,
// so small batches spread each pose's list over several warps.
int warps_per_pose(long long n) {
    int w = 1;
    while (w < 8 && n * (2 * w) <= kWarps) w *= 2;
    return w;
}

// Lists from this mean length on are worth loading ahead.
constexpr double kLongList = 512;

// mean_list: entries of a bin list, over the batch's poses; max_list: the mean
// of the system with the longest.  Long lists load several entries at a time.
// A pose of the densest system takes as long as max_list entries, all poses
// together at least as long as `load` entries a warp: with one warp per pose the
// former is a tail where it is well above the latter (of uneven lists, 1.5 times
// the mean and more), and two warps per pose halve it, but pay twice for what a
// pose costs beside its entries.  One and two warps, by max_list and load: 8,480
// and 3,870 102 and 75 us (6,174 String poses of 12 frameworks), 3,540 and 1,280
// 39.6 and 37.0, 1,760 and 360 18.6 and 16.5; 1,300 and 380 16.5 and 20.0, 1,800
// and 490 19.3 and 22.6, 1,890 and 2,460 35.6 and 44.0, 1,170 and 1,200 24.9 and 35.1.
static int pose_batch_launch(PoseBatchArgs a, bool mixed, double mean_list, double max_list,
                             cudaStream_t st) {
    a.wpp = warps_per_pose(a.n);
    const bool long_lists = mean_list >= kLongList && a.wpp <= 2;
    const double load = (double)a.n * mean_list / kWarps;
    if (long_lists && max_list >= 1.5 * mean_list && max_list >= 1.6 * load + 1100.0) a.wpp = 2;
    const long long groups = (a.n + 8 / a.wpp - 1) / (8 / a.wpp);
    const int blocks = (int)std::min<long long>(groups, kWarps);
    auto kernel = mixed ? long_lists ? pose_batch_kernel<true, 4> : pose_batch_kernel<true, 1>
                        : long_lists ? pose_batch_kernel<false, 4> : pose_batch_kernel<false, 1>;
    kernel<<<blocks, 256, 0, st>>>(a);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

PoseBatchSys pose_describe(const System *sys, const RegionSet *rs) {
    PoseBatchSys y;
    std::memset(&y, 0, sizeof y);   // padding too: descriptors are compared bytewise
    y.H = sys->H;
    y.Hinv = sys->Hinv;
    y.rc2 = sys->cutoff * sys->cutoff;
    y.rc2f = (float)y.rc2;
    y.off0 = sys->offsets[0];
    y.off1 = sys->offsets[1];
    y.nb0 = rs->nb[0];
    y.nb1 = rs->nb[1];
    y.nb2 = rs->nb[2];
    y.regs = rs->d_info;
    y.hi = rs->d_hi;
    y.lo = rs->d_lo;
    y.td = sys->d_td;
    y.tf = sys->d_tf;
    return y;
}

int pose_upload_desc(System *sys, const RegionSet *rs, const PoseBatchSys **out) {
    // The descriptor is uploaded synchronously on first use and whenever the
    // bin lists moved (compared with the host copy of the last upload); inside
    // a stream capture it is therefore already in place.
    const PoseBatchSys y = pose_describe(sys, rs);
    const bool upload =
        !sys->d_pose_desc || std::memcmp(&sys->h_pose_desc, &y, sizeof y) != 0;
    if (!sys->d_pose_desc) {
        VEXT_CUDA(device_malloc(&sys->d_pose_desc, sizeof(PoseBatchSys)));
        VEXT_CUDA(device_malloc(&sys->d_pose_offsets, 2 * sizeof(long long)));
        const long long off[2] = {0, 0};   // one system: the kernel never reads them
        VEXT_CUDA(cudaMemcpy(sys->d_pose_offsets, off, sizeof off, cudaMemcpyHostToDevice));
    }
    if (upload) {
        VEXT_CUDA(cudaMemcpy(sys->d_pose_desc, &y, sizeof y, cudaMemcpyHostToDevice));
        std::memcpy(&sys->h_pose_desc, &y, sizeof y);
    }
    *out = sys->d_pose_desc;
    return 0;
}

int pose_warp_enqueue(System *sys, const RegionSet *rs, int n, const double *centers,
                      const double *quats, const Options &o, double *energy, double *gc,
                      double *gq, double *gu, cudaStream_t st) {
    const PoseBatchSys *d_sys = nullptr;
    VEXT_TRY(pose_upload_desc(sys, rs, &d_sys));
    PoseBatchArgs a;
    a.sys = d_sys;
    a.offsets = sys->d_pose_offsets;
    a.n_systems = 1;
    a.n = n;
    a.centers = centers;
    a.quats = quats;
    a.energy = energy;
    a.gc = gc;
    a.gq = gq;
    a.gu = gu;
    const bool band = o.mode == VEXT_MODE_MIXED && o.band_hi > o.band_lo;
    a.band_lo = band ? o.band_lo : 0.0;
    a.band_hi = band ? o.band_hi : 0.0;
    a.status = sys->d_status;
    const double list = (double)rs->n_entries / std::max(rs->n_regions, 1);
    return pose_batch_launch(a, o.mode == VEXT_MODE_MIXED, list, list, st);
}

}  // namespace vext

using namespace vext;

struct vext_pose_batch_s {
    std::vector<vext_system> systems;
    long long n = 0;
    int n_systems = 0;
    double mean_list = 0, max_list = 0;   // entries of a bin list (pose_batch_launch)
    Options opt;
    PoseBatchSys *d_sys = nullptr;
    long long *d_offsets = nullptr;
    int *d_status = nullptr;
    ~vext_pose_batch_s() {
        device_free(d_sys);
        device_free(d_offsets);
        device_free(d_status);
    }
};

extern "C" int vext_pose_batch_create(int n_systems, const vext_system *systems,
                                      const int64_t *pose_offsets, const vext_options *opt,
                                      vext_pose_batch *out) {
    if (!out || n_systems < 1 || !systems || !pose_offsets)
        return fail(VEXT_ERR_ARGUMENT, "bad pose batch arguments");
    *out = nullptr;
    if (pose_offsets[0] != 0) return fail(VEXT_ERR_ARGUMENT, "pose_offsets[0] must be 0");
    for (int k = 0; k < n_systems; ++k) {
        if (!systems[k]) return fail(VEXT_ERR_ARGUMENT, "null system %d", k);
        if (pose_offsets[k + 1] < pose_offsets[k])
            return fail(VEXT_ERR_ARGUMENT, "pose_offsets must not decrease");
    }
    auto *b = new vext_pose_batch_s();
    std::unique_ptr<vext_pose_batch_s> guard(b);
    b->systems.assign(systems, systems + n_systems);
    b->n_systems = n_systems;
    b->n = pose_offsets[n_systems];
    b->opt = resolve_options(opt);
    if (b->opt.mode != VEXT_MODE_MIXED && b->opt.mode != VEXT_MODE_FP64)
        return fail(VEXT_ERR_ARGUMENT, "unknown precision mode %d", b->opt.mode);
    const double r_split = b->opt.mode == VEXT_MODE_FP64 ? 1e30 : b->opt.r_split;
    int dev = 0;
    VEXT_CUDA(cudaGetDevice(&dev));
    std::vector<PoseBatchSys> hs(n_systems);
    for (int k = 0; k < n_systems; ++k) {
        System *sys = &systems[k]->sys;
        if (sys->device != dev)
            return fail(VEXT_ERR_ARGUMENT, "system %d lives on another device", k);
        std::lock_guard<std::mutex> lock(sys->lock);
        RegionSet *rs = nullptr;
        VEXT_TRY(get_bin_regions(sys, r_split, &rs, sys->stream));
        hs[k] = pose_describe(sys, rs);
        const double list = (double)rs->n_entries / std::max(rs->n_regions, 1);
        b->mean_list += (double)(pose_offsets[k + 1] - pose_offsets[k]) / std::max(b->n, 1LL) * list;
        if (pose_offsets[k + 1] > pose_offsets[k]) b->max_list = std::max(b->max_list, list);
    }
    std::vector<long long> offs(pose_offsets, pose_offsets + n_systems + 1);
    VEXT_CUDA(device_malloc(&b->d_sys, sizeof(PoseBatchSys) * n_systems));
    VEXT_CUDA(cudaMemcpy(b->d_sys, hs.data(), sizeof(PoseBatchSys) * n_systems,
                         cudaMemcpyHostToDevice));
    VEXT_CUDA(device_malloc(&b->d_offsets, sizeof(long long) * (n_systems + 1)));
    VEXT_CUDA(cudaMemcpy(b->d_offsets, offs.data(), sizeof(long long) * (n_systems + 1),
                         cudaMemcpyHostToDevice));
    VEXT_CUDA(device_malloc(&b->d_status, sizeof(int)));
    VEXT_CUDA(cudaMemset(b->d_status, 0, sizeof(int)));
    *out = guard.release();
    return 0;
}

extern "C" int vext_pose_batch_run(vext_pose_batch b, const double *centers, const double *quats,
                                   double *energy, double *grad_center, double *grad_quat,
                                   double *grad_director, void *stream) {
    if (!b) return fail(VEXT_ERR_ARGUMENT, "null pose batch");
    if (b->n == 0) return 0;
    if (!centers || !quats) return fail(VEXT_ERR_ARGUMENT, "centers and quaternions required");
    PoseBatchArgs a;
    a.sys = b->d_sys;
    a.offsets = b->d_offsets;
    a.n_systems = b->n_systems;
    a.n = b->n;
    a.centers = centers;
    a.quats = quats;
    a.energy = energy;
    a.gc = grad_center;
    a.gq = grad_quat;
    a.gu = grad_director;
    const bool band = b->opt.mode == VEXT_MODE_MIXED && b->opt.band_hi > b->opt.band_lo;
    a.band_lo = band ? b->opt.band_lo : 0.0;
    a.band_hi = band ? b->opt.band_hi : 0.0;
    a.status = b->d_status;
    return pose_batch_launch(a, b->opt.mode == VEXT_MODE_MIXED, b->mean_list, b->max_list,
                             (cudaStream_t)stream);
}

extern "C" int vext_pose_batch_status(vext_pose_batch b) {
    if (!b) return fail(VEXT_ERR_ARGUMENT, "null pose batch");
    int h = 0;
    VEXT_CUDA(cudaDeviceSynchronize());
    VEXT_CUDA(cudaMemcpy(&h, b->d_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        VEXT_CUDA(cudaMemset(b->d_status, 0, sizeof(int)));
        if (h == DEV_BAD_INPUT) return fail(VEXT_ERR_ARGUMENT, "non-finite pose center or zero quaternion");
        return fail(VEXT_ERR_TIMEOUT, "device status %d", h);
    }
    return 0;
}

extern "C" int vext_pose_batch_destroy(vext_pose_batch b) {
    delete b;
    return 0;
}
