// Systems (framework + guest resident on the device) and their region lists.
//
// The pair coefficients follow the reference's ReusePotential
// (src/string_vext/neighbor.py:21-28) in FP64: sigma = (sigma_f + sigma_g)/2,
// eps = sqrt(eps_f eps_g), c12 = 4 eps sigma^12, c6 = 4 eps sigma^6,
// shift = -4 eps ((sigma/rc)^12 - (sigma/rc)^6), floor2 = (0.1 sigma)^2.
//
// Image enumeration (replacing TriclinicSitePotential's fixed reach box and
// kd-tree, physics.py:43-57): for a region with fractional origin f_o and
// radius rho, every (atom j, lattice shift n) whose image lies within
// R = rc + max|offset| + rho of the origin is listed.  Along axis k the
// fractional extent of a ball of radius R is R |Hinv[:,k]|, so n_k runs over
// [ceil(-d_k - R e_k), floor(-d_k + R e_k)] with d = f_j - f_o; the exact
// distance test is done in FP64 on (d + n) @ H.  No minimum image is used.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

#include "internal.cuh"
#include "sites.cuh"

namespace vext {

// ------------------------------------------------------------ error state

static thread_local std::string g_error;

void set_error(const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_error = buf;
}

int fail(int code, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_error = buf;
    return code;
}

Options resolve_options(const vext_options *opt) {
    vext_options d;
    vext_default_options(&d);
    if (!opt) opt = &d;
    Options o;
    o.mode = opt->mode;
    // Far pairs skip the contact floor, so r_split must exceed every floor
    // distance 0.1 sigma: it is clamped to at least 1 A.
    o.r_split = opt->r_split > 0 ? std::max(opt->r_split, 1.0) : kDefaultRSplit;
    o.band_lo = opt->band_lo;
    o.band_hi = opt->band_hi;
    o.cb = opt->centers_per_region;
    o.variant = opt->variant;
    o.batch_shape = opt->batch_shape;
    return o;
}

// ------------------------------------------------------------ block shapes

double block_radius(const Mat3 &H, int size, int ni, int nj, int nk) {
    // Centers of one block span (n-1)/S along each fractional axis; the
    // farthest center from the block's mean is a corner of that box.
    const double ha = 0.5 * (ni - 1) / size, hb = 0.5 * (nj - 1) / size,
                 hc = 0.5 * (nk - 1) / size;
    double best = 0;
    for (int s = 0; s < 8; ++s) {
        double x, y, z;
        frac_to_cart(H, (s & 1 ? ha : -ha), (s & 2 ? hb : -hb), (s & 4 ? hc : -hc), x, y, z);
        best = std::max(best, std::sqrt(x * x + y * y + z * z));
    }
    return best;
}

void choose_block_shape(const Mat3 &H, int size, int cb, int &bi, int &bj, int &bk) {
    double best = 1e300;
    bi = bj = 1;
    bk = std::min(cb, size);
    for (int a = 1; a <= cb; ++a)
        for (int b = 1; a * b <= cb; ++b) {
            if (cb % (a * b)) continue;
            const int c = cb / (a * b);
            if (a > size || b > size || c > size) continue;
            const double r = block_radius(H, size, a, b, c);
            if (r < best - 1e-12) {
                best = r;
                bi = a;
                bj = b;
                bk = c;
            }
        }
}

// ------------------------------------------------------------ list build

struct BuildArgs {
    Mat3 H;
    double einv[3];
    const double *frac;
    const int *type;
    int n_atoms;
    double r_list0;   // rc + max|offset| (+ margin)
    double r_near0;   // r_split + max|offset| (+ margin)
    double r_inner0;  // cutoff - max|offset| (- margin): inner entries lie within r_inner0 - rho
    double r_outer0;  // cutoff + 1e-3 A: outer shell entries lie beyond r_outer0 + rho
    double r_taylor;  // inner entries beyond it belong to the local expansion
    double r_tfar;    // and those beyond this one need fewer of its degrees
    double r_shella0; // shell entries within r_shella0 - rho: the nearer of two symmetric sites
                      // is inside the cutoff for every pose (0: none are set apart)
};

// Class boundaries (squared distance from the origin) of one region, in
// increasing order: near | mid | taylor | taylor far | shell a | shell | outer
// is the order of the classes and of the entries (an eighth one, always empty,
// for the scans in pairs).
constexpr int kClasses = 8;
struct ClassRadii {
    double rl, at[kClasses - 1];
    __device__ ClassRadii(const BuildArgs &a, const RegionInfo &r) {
        rl = a.r_list0 + r.rho;
        const double rn = a.r_near0 + r.rho, ri = fmax(a.r_inner0 - r.rho, 0.0),
                     ra = fmax(a.r_shella0 - r.rho, 0.0), ro = a.r_outer0 + r.rho;
        at[0] = rn * rn;
        at[3] = fmax(ri * ri, at[0]);
        at[1] = fmin(fmax(a.r_taylor * a.r_taylor, at[0]), at[3]);
        at[2] = fmin(fmax(a.r_tfar * a.r_tfar, at[1]), at[3]);
        at[4] = fmax(ra * ra, at[3]);
        at[5] = fmax(ro * ro, at[4]);
        at[6] = 1e300;
    }
};
// A thread's counts: all classes, or those of lists without an expansion (pose
// bins), whose other ones are empty.  Either way 4 KB per region of a list build.
struct ClassCounts {
    int n[kClasses];
    __device__ void put(const int (&from)[kClasses]) {
#pragma unroll
        for (int i = 0; i < kClasses; ++i) n[i] = from[i];
    }
    __device__ void get(int (&to)[kClasses]) const {
#pragma unroll
        for (int i = 0; i < kClasses; ++i) to[i] = n[i];
    }
};
struct BinCounts {
    int n[4];   // near, mid, shell, outer
    __device__ void put(const int (&from)[kClasses]) {
        n[0] = from[0];
        n[1] = from[1];
        n[2] = from[5];
        n[3] = from[6];
    }
    __device__ void get(int (&to)[kClasses]) const {
        to[0] = n[0];
        to[1] = n[1];
        to[2] = to[3] = to[4] = to[7] = 0;
        to[5] = n[2];
        to[6] = n[3];
    }
};

// Visit every candidate image of atom j for a region; f(dist2, rel) per image.
template <typename F>
__device__ __forceinline__ void for_each_image(const BuildArgs &a, const RegionInfo &r, int j,
                                               double rl, F &&f) {
    const double d0 = a.frac[3 * j] - r.of[0];
    const double d1 = a.frac[3 * j + 1] - r.of[1];
    const double d2 = a.frac[3 * j + 2] - r.of[2];
    const double e0 = __dmul_rn(rl, a.einv[0]), e1 = __dmul_rn(rl, a.einv[1]),
                 e2 = __dmul_rn(rl, a.einv[2]);
    const int lo0 = (int)ceil(__dsub_rn(-d0, e0)), hi0 = (int)floor(__dadd_rn(-d0, e0));
    const int lo1 = (int)ceil(__dsub_rn(-d1, e1)), hi1 = (int)floor(__dadd_rn(-d1, e1));
    const int lo2 = (int)ceil(__dsub_rn(-d2, e2)), hi2 = (int)floor(__dadd_rn(-d2, e2));
    const double rl2 = rl * rl;
    for (int n0 = lo0; n0 <= hi0; ++n0)
        for (int n1 = lo1; n1 <= hi1; ++n1)
            for (int n2 = lo2; n2 <= hi2; ++n2) {
                // explicit FMAs: the count and fill kernels must take
                // bit-identical decisions for every candidate
                const double u = d0 + n0, v = d1 + n1, w = d2 + n2;
                const double x = fma(u, a.H.m[0], fma(v, a.H.m[3], __dmul_rn(w, a.H.m[6])));
                const double y = fma(u, a.H.m[1], fma(v, a.H.m[4], __dmul_rn(w, a.H.m[7])));
                const double z = fma(u, a.H.m[2], fma(v, a.H.m[5], __dmul_rn(w, a.H.m[8])));
                const double q = fma(x, x, fma(y, y, __dmul_rn(z, z)));
                if (q < rl2) f(q, x, y, z);
            }
}

template <int NT>
__device__ __forceinline__ void block_scan2(int a, int b, int &pa, int &pb, int &ta, int &tb,
                                            int *sh) {
    // Exclusive scan of two ints over the block (NT threads, NT <= 1024).
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ya = __shfl_up_sync(0xffffffffu, xa, o);
        const int yb = __shfl_up_sync(0xffffffffu, xb, o);
        if (lane >= o) {
            xa += ya;
            xb += yb;
        }
    }
    if (lane == 31) {
        sh[warp] = xa;
        sh[32 + warp] = xb;
    }
    __syncthreads();
    if (warp == 0) {
        int va = lane < NT / 32 ? sh[lane] : 0, vb = lane < NT / 32 ? sh[32 + lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(0xffffffffu, va, o);
            const int yb = __shfl_up_sync(0xffffffffu, vb, o);
            if (lane >= o) {
                va += ya;
                vb += yb;
            }
        }
        sh[64 + lane] = va;   // inclusive warp prefixes
        sh[96 + lane] = vb;
    }
    __syncthreads();
    const int wa = warp ? sh[64 + warp - 1] : 0, wb = warp ? sh[96 + warp - 1] : 0;
    pa = wa + xa - a;
    pb = wb + xb - b;
    ta = sh[64 + NT / 32 - 1];
    tb = sh[96 + NT / 32 - 1];
    __syncthreads();
}

// Threads per region of the list builds: field lists take 128 (fewer idle
// threads in the last round of atoms, half the counts to hand over), pose bins
// 256.
constexpr int kBuildThreads = 256, kFieldBuildThreads = 128;

// Per region: the entries of each class, and per thread (atoms j = tid, tid +
// NT, ...) its counts per class for the fill.
template <int NT, typename Counts>
__global__ void __launch_bounds__(NT)
    region_count_kernel(BuildArgs a, RegionInfo *regs, int n_regions, Counts *counts) {
    const int region = blockIdx.x;
    if (region >= n_regions) return;
    const RegionInfo r = regs[region];
    const ClassRadii cls(a, r);
    int from[kClasses] = {0, 0, 0, 0, 0, 0, 0, 0};   // entries at or beyond each boundary
    for (int j = threadIdx.x; j < a.n_atoms; j += NT)
        for_each_image(a, r, j, cls.rl, [&](double q, double, double, double) {
            ++from[0];
#pragma unroll
            for (int i = 1; i < kClasses; ++i) from[i] += q >= cls.at[i - 1];
        });
    int c[kClasses];
#pragma unroll
    for (int i = 0; i < kClasses; ++i) c[i] = from[i] - (i + 1 < kClasses ? from[i + 1] : 0);
    counts[(long long)region * NT + threadIdx.x].put(c);
    __shared__ int sh[128];
    int p, q, t[kClasses];
#pragma unroll
    for (int i = 0; i < kClasses; i += 2)
        block_scan2<NT>(c[i], c[i + 1], p, q, t[i], t[i + 1], sh);
    if (threadIdx.x == 0) {
        RegionInfo &w = regs[region];
        w.n_near = t[0];
        w.n_mid = t[1];
        w.n_inner = t[1] + t[2] + t[3];
        w.n_tnear = t[2];
        w.n_shella = t[4];
        w.n_outer = t[6];
        w.n_total = t[0] + t[1] + t[2] + t[3] + t[4] + t[5] + t[6];
    }
}

// Entry order inside each class: thread-major (thread t's atoms t, t + NT,
// ... in turn, each atom's images in enumeration order), so a thread's slots
// follow from a block scan of the per-thread counts that region_count_kernel
// stored and the candidates are enumerated once here.
template <int NT, typename Counts>
__global__ void __launch_bounds__(NT, 512 / NT)
    region_fill_kernel(BuildArgs a, const RegionInfo *regs, int n_regions,
                       const Counts *counts, float4 *hi, float4 *lo, int *status) {
    const int region = blockIdx.x;
    if (region >= n_regions) return;
    const RegionInfo r = regs[region];
    const ClassRadii cls(a, r);
    __shared__ int sh[128];
    int c[kClasses];
    counts[(long long)region * NT + threadIdx.x].get(c);
    // this thread's next slot and end per class (indexed by unrolled loops
    // only: a runtime index would put them in local memory)
    int w[kClasses], end[kClasses], t[kClasses];
#pragma unroll
    for (int i = 0; i < kClasses; i += 2)
        block_scan2<NT>(c[i], c[i + 1], w[i], w[i + 1], t[i], t[i + 1], sh);
    if (threadIdx.x == 0 &&
        (t[0] != r.n_near || t[1] != r.n_mid || t[2] != r.n_tnear ||
         t[1] + t[2] + t[3] != r.n_inner || t[4] != r.n_shella || t[6] != r.n_outer ||
         t[0] + t[1] + t[2] + t[3] + t[4] + t[5] + t[6] != r.n_total))
        atomicExch(status, DEV_BAD_LIST);
    int base = 0;
#pragma unroll
    for (int i = 0; i < kClasses; ++i) {
        w[i] += base;
        end[i] = w[i] + c[i];
        base += t[i];
    }
    for (int j = threadIdx.x; j < a.n_atoms; j += NT) {
        const int ty = a.type[j];
        for_each_image(a, r, j, cls.rl, [&](double q, double x, double y, double z) {
            int k = 0;
#pragma unroll
            for (int i = 1; i < kClasses; ++i) k += q >= cls.at[i - 1];
            int slot = 0, lim = 0;
#pragma unroll
            for (int i = 0; i < kClasses; ++i)
                if (k == i) {
                    slot = w[i]++;
                    lim = end[i];
                }
            if (slot >= lim) {
                atomicExch(status, DEV_BAD_LIST);
                return;
            }
            const float hx = (float)x, hy = (float)y, hz = (float)z;
            hi[r.off + slot] = make_float4(hx, hy, hz, __int_as_float(ty));
            lo[r.off + slot] = make_float4((float)(x - hx), (float)(y - hy), (float)(z - hz), 0.f);
        });
    }
    bool full = true;
#pragma unroll
    for (int i = 0; i < kClasses; ++i) full = full && w[i] == end[i];
    if (!full) atomicExch(status, DEV_BAD_LIST);
}

// ------------------------------------------------------------ region sets

RegionSet::~RegionSet() {
    device_free(d_info);
    device_free(d_hi);
    device_free(d_lo);
}

// Per-device scratch of the per-(region, thread) class counts that the count
// pass hands to the fill pass; one list build at a time uses it (the lock is
// held until the build's kernels have finished).  It belongs to the context
// it was allocated in: after a device reset (a new context, told apart by
// its unique id) the old array is gone and a new one is allocated.
namespace {
struct BuildScratch {
    std::mutex lock;
    unsigned char *ptr = nullptr;
    size_t cap = 0;
    unsigned long long ctx_id = 0;
};
BuildScratch &build_scratch(int device) {
    static BuildScratch scratch[64];
    return scratch[device & 63];
}
// Waits for the stream before the scratch lock is released, also on the
// early error returns of build_lists.
struct StreamDrain {
    cudaStream_t stream;
    ~StreamDrain() { cudaStreamSynchronize(stream); }
};
}  // namespace

void release_build_scratch(int device) {
    BuildScratch &scratch = build_scratch(device);
    std::lock_guard<std::mutex> guard(scratch.lock);
    if (scratch.ptr && current_context_id() == scratch.ctx_id) device_free(scratch.ptr);
    scratch.ptr = nullptr;
    scratch.cap = 0;
}

static int build_lists(System *sys, RegionSet *rs, cudaStream_t stream) {
    BuildScratch &scratch = build_scratch(sys->device);
    std::lock_guard<std::mutex> scratch_guard(scratch.lock);
    StreamDrain drain{stream};
    BuildArgs a;
    a.H = sys->H;
    for (int k = 0; k < 3; ++k) a.einv[k] = sys->einv[k];
    a.frac = sys->d_frac;
    a.type = sys->d_type;
    a.n_atoms = sys->n_atoms;
    // 1e-6 A margins keep every pair within rc (resp. r_split) listed despite
    // FP64 rounding of the distances (~1e-14 A).
    const double offset = rs->sites ? 0.0 : sys->max_offset;
    a.r_list0 = sys->cutoff + offset + 1e-6;
    a.r_near0 = rs->r_split + offset + 1e-6;
    a.r_inner0 = sys->cutoff - offset - 1e-6;
    a.r_outer0 = sys->cutoff + 1e-3;
    // field lists set the entries of the local expansion apart, and those near
    // shell entries whose nearer site is always inside: |d0|^2 + o^2 < rc^2
    // for every center (|d0| the entry's distance from it)
    a.r_taylor = rs->d_taylor;
    a.r_tfar = rs->d_tfar;
    const double ra2 = sys->cutoff * sys->cutoff - sys->max_offset * sys->max_offset;
    a.r_shella0 = rs->d_taylor < sys->cutoff && ra2 > 0 ? std::sqrt(ra2) - 1e-3 : 0.0;
    // (site lists: those within rc; a cluster takes the ones outside off again)
    if (rs->sites && rs->d_taylor < sys->cutoff) a.r_shella0 = sys->cutoff + rs->taylor_radius;
    const int n = rs->n_regions;
    if (!rs->d_info) VEXT_CUDA(device_malloc(&rs->d_info, sizeof(RegionInfo) * n));
    VEXT_CUDA(cudaMemcpyAsync(rs->d_info, rs->h_info.data(), sizeof(RegionInfo) * n,
                              cudaMemcpyHostToDevice, stream));
    cudaEvent_t e0 = sys->ev[3], e1 = sys->ev[4];
    VEXT_CUDA(cudaEventRecord(e0, stream));
    const unsigned long long ctx = current_context_id();
    if (scratch.ptr && ctx != 0 && scratch.ctx_id != 0 && ctx != scratch.ctx_id) {
        // allocated in a context that has since been reset: it went with that
        // context; allocate anew
        scratch.ptr = nullptr;
        scratch.cap = 0;
    }
    const bool field = rs->size > 0;
    VEXT_TRY(ensure_capacity(scratch.ptr, scratch.cap,
                             (size_t)n * (field ? kFieldBuildThreads * sizeof(ClassCounts)
                                                : kBuildThreads * sizeof(BinCounts))));
    scratch.ctx_id = ctx;
    ClassCounts *field_counts = reinterpret_cast<ClassCounts *>(scratch.ptr);
    BinCounts *bin_counts = reinterpret_cast<BinCounts *>(scratch.ptr);
    if (field)
        region_count_kernel<kFieldBuildThreads>
            <<<n, kFieldBuildThreads, 0, stream>>>(a, rs->d_info, n, field_counts);
    else
        region_count_kernel<kBuildThreads>
            <<<n, kBuildThreads, 0, stream>>>(a, rs->d_info, n, bin_counts);
    VEXT_CUDA(cudaGetLastError());
    VEXT_CUDA(cudaMemcpyAsync(rs->h_info.data(), rs->d_info, sizeof(RegionInfo) * n,
                              cudaMemcpyDeviceToHost, stream));
    VEXT_CUDA(cudaStreamSynchronize(stream));
    long long off = 0, near = 0, outer = 0, taylor = 0;
    for (auto &r : rs->h_info) {
        r.off = off;
        off += r.n_total;
        near += r.n_near;
        outer += r.n_outer;
        taylor += r.n_inner - r.n_mid;
    }
    rs->n_entries = off;
    rs->n_near = near;
    rs->n_outer = outer;
    rs->n_taylor = taylor;
    VEXT_CUDA(cudaMemcpyAsync(rs->d_info, rs->h_info.data(), sizeof(RegionInfo) * n,
                              cudaMemcpyHostToDevice, stream));
    if (off > rs->capacity || !rs->d_hi) {
        device_free(rs->d_hi);
        device_free(rs->d_lo);
        rs->d_hi = rs->d_lo = nullptr;
        rs->capacity = 0;
        VEXT_CUDA(device_malloc(&rs->d_hi, sizeof(float4) * std::max<long long>(off, 1)));
        VEXT_CUDA(device_malloc(&rs->d_lo, sizeof(float4) * std::max<long long>(off, 1)));
        rs->capacity = std::max<long long>(off, 1);
    }
    if (field)
        region_fill_kernel<kFieldBuildThreads><<<n, kFieldBuildThreads, 0, stream>>>(
            a, rs->d_info, n, field_counts, rs->d_hi, rs->d_lo, sys->d_status);
    else
        region_fill_kernel<kBuildThreads><<<n, kBuildThreads, 0, stream>>>(
            a, rs->d_info, n, bin_counts, rs->d_hi, rs->d_lo, sys->d_status);
    VEXT_CUDA(cudaGetLastError());
    VEXT_CUDA(cudaEventRecord(e1, stream));
    VEXT_CUDA(cudaEventSynchronize(e1));
    VEXT_CUDA(cudaEventElapsedTime(&rs->build_ms, e0, e1));
    sys->list_timed = true;
    rs->stale = false;
    return check_status(sys, stream);
}

static double det3(const Mat3 &m) {
    const double *h = m.m;
    return h[0] * (h[4] * h[8] - h[5] * h[7]) - h[1] * (h[3] * h[8] - h[5] * h[6]) +
           h[2] * (h[3] * h[7] - h[4] * h[6]);
}

// Where a region's local expansion starts, for sites within `radius` of its origin
// (taylor_start goes through all types some 24 times: called once per list set).
static double expansion_start(const System &sys, double radius, double r_split) {
    return std::max(taylor_start(sys, radius), r_split + radius);
}

// Entries per region that it is expected to hold; 0: none.
static double expansion_entries(const System &sys, double radius, double start) {
    const double inner = sys.cutoff - radius;
    if (!(start < inner)) return 0.0;
    return 4.18879 * (inner * inner * inner - start * start * start) * sys.n_atoms *
           std::fabs(det3(sys.Hinv));
}

int get_field_regions(System *sys, int size, int cb, double r_split, int expand_axes,
                      bool adjoint, RegionSet **out, cudaStream_t stream) {
    int bi, bj, bk;
    choose_block_shape(sys->H, size, cb, bi, bj, bk);
    const double rho = block_radius(sys->H, size, bi, bj, bk) + 1e-9;
    bool expand = false;
    if (expand_axes > 0 && r_split < 1e29) {
        const auto key = std::make_tuple(size, cb, r_split);
        auto known = sys->expansion_entries.find(key);
        if (known == sys->expansion_entries.end()) {
            const double radius = rho + sys->max_offset;
            known = sys->expansion_entries
                        .emplace(key, expansion_entries(*sys, radius,
                                                        expansion_start(*sys, radius, r_split)))
                        .first;
        }
        expand = known->second >= kTaylorMinEntriesPoses &&
                 taylor_pays(known->second, (double)expand_axes * bi * bj * bk, adjoint);
    }
    VEXT_TRY(get_block_regions(sys, size, bi, bj, bk, rho, sys->max_offset, false, expand, r_split,
                               out, stream));
    if (!expand || taylor_worthwhile(*sys, **out, expand_axes, adjoint)) return 0;
    // fewer entries than expected: plain lists, also in the calls to come
    RegionSet *rs = *out;
    sys->expansion_entries[std::make_tuple(size, cb, r_split)] =
        (double)rs->n_taylor / rs->n_regions;
    if (rs->use.use_count() == 1 && sys->field_plan_set != rs) {
        sys->sets.erase(std::find(sys->sets.begin(), sys->sets.end(), rs));
        delete rs;
    }
    return get_block_regions(sys, size, bi, bj, bk, rho, sys->max_offset, false, false, r_split,
                             out, stream);
}

// Lists of blocks of bi x bj x bk grid centers (sites: voxels) for sites within
// rho + offset of a block's middle.
int get_block_regions(System *sys, int size, int bi, int bj, int bk, double rho, double offset,
                      bool sites, bool expand, double r_split, RegionSet **out,
                      cudaStream_t stream) {
    for (RegionSet *rs : sys->sets)
        if (rs->size == size && rs->bi == bi && rs->bj == bj && rs->bk == bk &&
            rs->sites == sites && rs->expand == expand && rs->r_split == r_split) {
            if (rs->stale) {
                for (auto &r : rs->h_info)
                    r.n_near = r.n_total = r.n_inner = r.n_outer = r.n_mid = r.n_tnear =
                        r.n_shella = 0;
                VEXT_TRY(build_lists(sys, rs, stream));
            }
            *out = rs;
            return 0;
        }
    RegionSet *rs = new RegionSet();
    rs->size = size;
    rs->r_split = r_split;
    rs->sites = sites;
    rs->expand = expand;
    rs->bi = bi;
    rs->bj = bj;
    rs->bk = bk;
    rs->n_ri = (size + rs->bi - 1) / rs->bi;
    rs->n_rj = (size + rs->bj - 1) / rs->bj;
    rs->n_rk = (size + rs->bk - 1) / rs->bk;
    rs->n_regions = rs->n_ri * rs->n_rj * rs->n_rk;
    rs->h_info.resize(rs->n_regions);
    int idx = 0;
    for (int I = 0; I < rs->n_ri; ++I)
        for (int J = 0; J < rs->n_rj; ++J)
            for (int K = 0; K < rs->n_rk; ++K) {
                RegionInfo &r = rs->h_info[idx++];
                std::memset(&r, 0, sizeof r);
                r.i0 = I * rs->bi;
                r.j0 = J * rs->bj;
                r.k0 = K * rs->bk;
                r.ni = std::min(rs->bi, size - r.i0);
                r.nj = std::min(rs->bj, size - r.j0);
                r.nk = std::min(rs->bk, size - r.k0);
                // origin = mean of a whole block's centers ((i + .5)/S ...), also
                // where the grid's edge cuts the block: the centers sit at the
                // same places relative to it in every region
                r.of[0] = (r.i0 + 0.5 * rs->bi) / size;
                r.of[1] = (r.j0 + 0.5 * rs->bj) / size;
                r.of[2] = (r.k0 + 0.5 * rs->bk) / size;
                r.rho = rho;
            }
    rs->taylor_radius = offset + rho;
    const double start = expand ? expansion_start(*sys, rs->taylor_radius, r_split) : 1e30;
    if (expansion_entries(*sys, rs->taylor_radius, start) >= kTaylorMinEntries) {
        rs->d_taylor = start;
        rs->d_tfar = std::max(rs->d_taylor,
                              taylor_start(*sys, rs->taylor_radius, kTaylorFarOrder));
    }
    // without expansions a cut block's origin is the mean of its own centers:
    // shorter lists (21^3 and 35^3 grids 2-3 % faster)
    if (!sites && !expand)
        for (RegionInfo &r : rs->h_info) {
            r.of[0] = (r.i0 + 0.5 * r.ni) / size;
            r.of[1] = (r.j0 + 0.5 * r.nj) / size;
            r.of[2] = (r.k0 + 0.5 * r.nk) / size;
            r.rho = block_radius(sys->H, size, r.ni, r.nj, r.nk) + 1e-9;
        }
    int rc = build_lists(sys, rs, stream);
    if (rc) {
        delete rs;
        return rc;
    }
    sys->sets.push_back(rs);
    *out = rs;
    return 0;
}

// Width (A, between lattice planes) of the pose bins.

void drop_idle_site_lists(System *sys) {
    auto idle = [sys](const RegionSet *rs) {
        return rs->sites && rs->use.use_count() == 1 &&
               !(sys->site_field && sys->site_field->plan.rs == rs);
    };
    for (RegionSet *&rs : sys->sets)
        if (idle(rs)) {
            delete rs;
            rs = nullptr;
        }
    sys->sets.erase(std::remove(sys->sets.begin(), sys->sets.end(), nullptr), sys->sets.end());
}

int get_bin_regions(System *sys, double r_split, RegionSet **out, cudaStream_t stream,
                    double bin_width) {
    for (RegionSet *rs : sys->sets)
        if (rs->size == 0 && rs->r_split == r_split && rs->bin_width == bin_width) {
            if (rs->stale) {
                for (auto &r : rs->h_info)
                    r.n_near = r.n_total = r.n_inner = r.n_outer = r.n_mid = r.n_tnear =
                        r.n_shella = 0;
                VEXT_TRY(build_lists(sys, rs, stream));
            }
            *out = rs;
            return 0;
        }
    RegionSet *rs = new RegionSet();
    rs->r_split = r_split;
    rs->bin_width = bin_width;
    // Bins about bin_width wide between lattice planes.
    for (int k = 0; k < 3; ++k)
        rs->nb[k] = std::max(1, (int)std::ceil((1.0 / sys->einv[k]) / bin_width));
    rs->n_ri = rs->nb[0];
    rs->n_rj = rs->nb[1];
    rs->n_rk = rs->nb[2];
    rs->n_regions = rs->nb[0] * rs->nb[1] * rs->nb[2];
    rs->h_info.resize(rs->n_regions);
    int idx = 0;
    for (int I = 0; I < rs->nb[0]; ++I)
        for (int J = 0; J < rs->nb[1]; ++J)
            for (int K = 0; K < rs->nb[2]; ++K) {
                RegionInfo &r = rs->h_info[idx++];
                std::memset(&r, 0, sizeof r);
                r.of[0] = (I + 0.5) / rs->nb[0];
                r.of[1] = (J + 0.5) / rs->nb[1];
                r.of[2] = (K + 0.5) / rs->nb[2];
                // half-diagonal of the bin parallelepiped (any wrapped center
                // in the bin, boundaries included)
                double best = 0;
                for (int s = 0; s < 8; ++s) {
                    double x, y, z;
                    frac_to_cart(sys->H, (s & 1 ? 0.5 : -0.5) / rs->nb[0],
                                 (s & 2 ? 0.5 : -0.5) / rs->nb[1], (s & 4 ? 0.5 : -0.5) / rs->nb[2],
                                 x, y, z);
                    best = std::max(best, std::sqrt(x * x + y * y + z * z));
                }
                r.rho = best + 1e-9;
            }
    int rc = build_lists(sys, rs, stream);
    if (rc) {
        delete rs;
        return rc;
    }
    sys->sets.push_back(rs);
    *out = rs;
    return 0;
}

int check_status(System *sys, cudaStream_t stream) {
    int h = 0;
    VEXT_CUDA(cudaMemcpyAsync(&h, sys->d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    VEXT_CUDA(cudaStreamSynchronize(stream));
    if (h == DEV_OK) return 0;
    VEXT_CUDA(cudaMemsetAsync(sys->d_status, 0, sizeof(int), stream));
    VEXT_CUDA(cudaStreamSynchronize(stream));
    if (h == DEV_TIMEOUT) return fail(VEXT_ERR_TIMEOUT, "a device wait gave up (status %d)", h);
    return fail(VEXT_ERR_CUDA, "device list build inconsistency (status %d)", h);
}

void System::drop_adjoint_batch() {
    if (adj_batch) vext_batch_destroy(adj_batch);
    adj_batch = nullptr;
    adj_size = 0;
    adj_axes.clear();
    if (slab_batch) vext_batch_destroy(slab_batch);
    slab_batch = nullptr;
    slab_axes.clear();
    drop_host_parts();
}

void System::drop_host_parts() {
    for (vext_batch b : host_parts) vext_batch_destroy(b);
    for (cudaEvent_t e : host_part_done) cudaEventDestroy(e);
    host_parts.clear();
    host_part_done.clear();
    host_size = 0;
    host_axes.clear();
}

System::~System() {
    FreeTogether together;
    drop_adjoint_batch();   // it points into the region sets
    for (RegionSet *rs : sets) delete rs;
    device_free(d_g32);
    field_plan.release();
    site_field_free(site_field);
    device_free(d_sums);
    device_free(d_base);
    device_free(d_e64);
    device_free(d_refine);
    device_free(d_axes);
    device_free(d_f32);
    device_free(d_small);
    device_free(d_e64T);
    device_free(d_flags);
    device_free(d_pose_scratch);
    device_free(d_pose_io);
    device_free(d_pose_desc);
    device_free(d_pose_offsets);
    for (auto &e : ev)
        if (e) cudaEventDestroy(e);
    if (aux) cudaStreamDestroy(aux);
    if (stream) cudaStreamDestroy(stream);
}

}  // namespace vext

using namespace vext;

extern "C" void vext_default_options(vext_options *opt) {
    std::memset(opt, 0, sizeof *opt);
    opt->mode = VEXT_MODE_MIXED;
    opt->r_split = kDefaultRSplit;
    opt->band_lo = -1e-2;
    opt->band_hi = 100.0;
    opt->centers_per_region = 0;
}

extern "C" const char *vext_last_error(void) { return g_error.c_str(); }

extern "C" const char *vext_version(void) { return "vext_b200 0.1.0 (sm_100a)"; }

extern "C" int vext_system_create(const vext_system_desc *d, vext_system *out) {
    if (!d || !out) return fail(VEXT_ERR_ARGUMENT, "null argument");
    *out = nullptr;
    if (d->n_atoms < 1 || !d->frac || !d->sigma || !d->epsilon)
        return fail(VEXT_ERR_ARGUMENT, "at least one framework atom with sigma/epsilon required");
    if (!(d->cutoff > 0) || !std::isfinite(d->cutoff))
        return fail(VEXT_ERR_ARGUMENT, "positive finite cutoff required");
    if (!(d->guest_sigma > 0) || !(d->guest_epsilon > 0))
        return fail(VEXT_ERR_ARGUMENT, "positive guest sigma/epsilon required");
    if (!std::isfinite(d->offsets[0]) || !std::isfinite(d->offsets[1]))
        return fail(VEXT_ERR_ARGUMENT, "finite site offsets required");
    const double *h = d->cell;
    for (int k = 0; k < 9; ++k)
        if (!std::isfinite(h[k])) return fail(VEXT_ERR_ARGUMENT, "non-finite cell");
    const double det = h[0] * (h[4] * h[8] - h[5] * h[7]) - h[1] * (h[3] * h[8] - h[5] * h[6]) +
                       h[2] * (h[3] * h[7] - h[4] * h[6]);
    if (!(det > 0)) return fail(VEXT_ERR_ARGUMENT, "cell determinant must be positive");
    for (int i = 0; i < d->n_atoms; ++i) {
        for (int k = 0; k < 3; ++k)
            if (!std::isfinite(d->frac[3 * i + k]))
                return fail(VEXT_ERR_ARGUMENT, "non-finite fractional coordinate (atom %d)", i);
        if (!(d->sigma[i] > 0) || !(d->epsilon[i] > 0) || !std::isfinite(d->sigma[i]) ||
            !std::isfinite(d->epsilon[i]))
            return fail(VEXT_ERR_ARGUMENT, "invalid framework LJ parameters (atom %d)", i);
    }
    auto *handle = new vext_system_s();
    System &s = handle->sys;
    cudaGetDevice(&s.device);
    std::memcpy(s.H.m, h, sizeof s.H.m);
    // inverse via the adjugate
    const double *m = h;
    double inv[9] = {(m[4] * m[8] - m[5] * m[7]) / det, (m[2] * m[7] - m[1] * m[8]) / det,
                     (m[1] * m[5] - m[2] * m[4]) / det, (m[5] * m[6] - m[3] * m[8]) / det,
                     (m[0] * m[8] - m[2] * m[6]) / det, (m[2] * m[3] - m[0] * m[5]) / det,
                     (m[3] * m[7] - m[4] * m[6]) / det, (m[1] * m[6] - m[0] * m[7]) / det,
                     (m[0] * m[4] - m[1] * m[3]) / det};
    std::memcpy(s.Hinv.m, inv, sizeof inv);
    for (int k = 0; k < 3; ++k)
        s.einv[k] = std::sqrt(inv[k] * inv[k] + inv[3 + k] * inv[3 + k] + inv[6 + k] * inv[6 + k]);
    s.n_atoms = d->n_atoms;
    s.guest_sigma = d->guest_sigma;
    s.guest_epsilon = d->guest_epsilon;
    s.offsets[0] = d->offsets[0];
    s.offsets[1] = d->offsets[1];
    s.max_offset = std::max(std::fabs(d->offsets[0]), std::fabs(d->offsets[1]));
    s.cutoff = d->cutoff;
    s.temperature = d->temperature;
    // distinct (sigma, epsilon) pairs -> type ids, in order of first appearance
    std::map<std::pair<double, double>, int> ids;
    std::vector<int> type(d->n_atoms);
    std::vector<double> frac(3 * (size_t)d->n_atoms);
    for (int i = 0; i < d->n_atoms; ++i) {
        auto key = std::make_pair(d->sigma[i], d->epsilon[i]);
        auto it = ids.find(key);
        if (it == ids.end()) it = ids.emplace(key, (int)ids.size()).first;
        type[i] = it->second;
        for (int k = 0; k < 3; ++k) {
            const double f = d->frac[3 * i + k];
            double w = f - std::floor(f);   // numpy.mod(f, 1) for finite f
            if (w >= 1.0) w = 0.0;
            frac[3 * i + k] = w;
        }
    }
    s.n_types = (int)ids.size();
    {
        uint64_t hsh = 1469598103934665603ull;
        auto mix = [&hsh](const void *p, size_t n) {
            const unsigned char *c = static_cast<const unsigned char *>(p);
            for (size_t i = 0; i < n; ++i) hsh = (hsh ^ c[i]) * 1099511628211ull;
        };
        mix(h, 9 * sizeof(double));
        mix(&d->cutoff, sizeof(double));
        mix(&s.n_atoms, sizeof(int));
        mix(frac.data(), frac.size() * sizeof(double));
        mix(type.data(), type.size() * sizeof(int));
        std::vector<std::pair<double, double>> by_id(ids.size());
        for (auto &kv : ids) by_id[kv.second] = kv.first;
        mix(by_id.data(), by_id.size() * sizeof(by_id[0]));
        s.frame_hash = hsh;
    }
    if (s.n_types > kMaxTypes) {
        delete handle;
        return fail(VEXT_ERR_CAPACITY, "%d distinct framework (sigma, epsilon) pairs; limit %d",
                    (int)ids.size(), kMaxTypes);
    }
    std::vector<float4> tf(s.n_types);
    s.h_td.assign(4 * (size_t)s.n_types, 0.0);
    for (auto &kv : ids) {
        const int t = kv.second;
        const double ms = (kv.first.first + d->guest_sigma) / 2;
        const double me = std::sqrt(kv.first.second * d->guest_epsilon);
        const double s6 = std::pow(ms, 6);
        const double c12 = 4 * me * (s6 * s6);
        const double c6 = 4 * me * s6;
        const double cut6 = std::pow(ms / d->cutoff, 6);
        const double shift = -4 * me * (cut6 * cut6 - cut6);
        const double floor2 = (.1 * ms) * (.1 * ms);
        s.h_td[4 * t + 0] = c12;
        s.h_td[4 * t + 1] = c6;
        s.h_td[4 * t + 2] = shift;
        s.h_td[4 * t + 3] = floor2;
        tf[t] = make_float4((float)c12, (float)c6, (float)shift, (float)floor2);
    }
    cudaError_t err = cudaSuccess;
    auto chk = [&](cudaError_t e) {
        if (e != cudaSuccess && err == cudaSuccess) err = e;
    };
    chk(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
    chk(cudaStreamCreateWithFlags(&s.aux, cudaStreamNonBlocking));
    for (auto &e : s.ev) chk(cudaEventCreate(&e));
    // one allocation and one upload
    size_t bytes = 0;
    auto place = [&bytes](size_t n) {
        const size_t at = bytes;
        bytes = (bytes + n + 255) & ~(size_t)255;
        return at;
    };
    const size_t at_frac = place(sizeof(double) * frac.size()),
                 at_type = place(sizeof(int) * type.size()),
                 at_tf = place(sizeof(float4) * tf.size()),
                 at_td = place(sizeof(double) * s.h_td.size()), at_status = place(sizeof(int));
    chk(device_malloc(&s.d_base, bytes));
    if (err == cudaSuccess) {
        std::vector<char> up(bytes, 0);
        std::memcpy(&up[at_frac], frac.data(), sizeof(double) * frac.size());
        std::memcpy(&up[at_type], type.data(), sizeof(int) * type.size());
        std::memcpy(&up[at_tf], tf.data(), sizeof(float4) * tf.size());
        std::memcpy(&up[at_td], s.h_td.data(), sizeof(double) * s.h_td.size());
        char *base = static_cast<char *>(s.d_base);
        s.d_frac = reinterpret_cast<double *>(base + at_frac);
        s.d_type = reinterpret_cast<int *>(base + at_type);
        s.d_tf = reinterpret_cast<float4 *>(base + at_tf);
        s.d_td = reinterpret_cast<double *>(base + at_td);
        s.d_status = reinterpret_cast<int *>(base + at_status);
        chk(cudaMemcpy(base, up.data(), bytes, cudaMemcpyHostToDevice));
    }
    if (err != cudaSuccess) {
        delete handle;
        return fail(VEXT_ERR_CUDA, "system upload failed: %s", cudaGetErrorString(err));
    }
    *out = handle;
    return 0;
}

extern "C" int vext_system_invalidate(vext_system h) {
    if (!h) return fail(VEXT_ERR_ARGUMENT, "null system");
    std::lock_guard<std::mutex> guard(h->sys.lock);
    for (RegionSet *rs : h->sys.sets) rs->stale = true;
    h->sys.no_sites_from = h->sys.no_expansions_from = 1LL << 62;
    h->sys.drop_adjoint_batch();
    return 0;
}

extern "C" int vext_last_timings(vext_system h, double *list_ms, double *near_ms,
                                 double *far_ms, double *epilogue_ms) {
    if (!h) return fail(VEXT_ERR_ARGUMENT, "null system");
    System &s = h->sys;
    std::lock_guard<std::mutex> guard(s.lock);
    float a = 0, b = 0, c = 0, d = 0;
    if (s.list_timed) {
        VEXT_CUDA(cudaEventSynchronize(s.ev[4]));
        VEXT_CUDA(cudaEventElapsedTime(&a, s.ev[3], s.ev[4]));
    }
    if (s.timed) {
        VEXT_CUDA(cudaEventSynchronize(s.ev[2]));
        if (s.split_timed) {
            VEXT_CUDA(cudaEventElapsedTime(&b, s.ev[0], s.ev[5]));
            VEXT_CUDA(cudaEventElapsedTime(&c, s.ev[5], s.ev[1]));
        } else {
            VEXT_CUDA(cudaEventElapsedTime(&b, s.ev[0], s.ev[1]));
        }
        VEXT_CUDA(cudaEventElapsedTime(&d, s.ev[1], s.ev[2]));
    }
    if (list_ms) *list_ms = s.list_timed ? a : 0.0;
    if (near_ms) *near_ms = b;
    if (far_ms) *far_ms = c;
    if (epilogue_ms) *epilogue_ms = d;
    s.list_timed = false;
    return 0;
}

extern "C" int vext_system_destroy(vext_system sys) {
    if (!sys) return 0;
    int dev = 0;
    cudaGetDevice(&dev);
    const int own = sys->sys.device;
    if (dev != own) cudaSetDevice(own);
    delete sys;
    if (dev != own) cudaSetDevice(dev);
    return 0;
}
