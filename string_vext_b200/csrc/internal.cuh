// Internal structures shared by the vext_b200 translation units.
//
// Data layout in HBM (per system = framework + guest):
//   frac   double [n_atoms][3]   wrapped fractional coordinates
//   type   int    [n_atoms]      index into the pair-parameter tables
//   tf     float4 [n_types]      (c12, c6, shift, floor2) in FP32
//   td     double [n_types][4]   the same in FP64 (reference arithmetic)
// Per region set (one grid size + block shape, or the pose bins):
//   info   RegionInfo [n_regions]
//   hi     float4 [entries]  (x, y, z) of an image relative to the region
//                            origin rounded to FP32; w = type id (int bits)
//   lo     float4 [entries]  residual (x - hi.x, ...) so hi + lo is the FP64
//                            relative position to ~1e-14 A
// Each region's entries are contiguous (info.off), "near" entries first:
// entries closer to the origin than r_split + max|offset| + rho are near,
// so every (site, image) pair nearer than r_split has a near entry.  Then
// the far inner entries, then the shell, whose last n_outer entries lie
// beyond rc + rho + 1e-3 A of the origin.
#pragma once

#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "common.cuh"

namespace vext {

// Device memory (memory.cu).  Allocations come from a pool per device that
// keeps up to kPoolKeep bytes of what was freed; device_free waits for the
// device first, as cudaFree does (a block whose wait is refused, during a stream
// capture, is kept for the next free).
cudaError_t device_malloc_bytes(void **p, size_t bytes);
template <typename T>
cudaError_t device_malloc(T **p, size_t bytes) {
    return device_malloc_bytes(reinterpret_cast<void **>(p), bytes);
}
void device_free(void *p);

// While one is alive on a thread, its device_free calls wait together, when the
// last one goes.
struct FreeTogether {
    FreeTogether();
    ~FreeTogether();
};

// Free the list builds' scratch on a device (system.cu).
void release_build_scratch(int device);

// Copy finished device memory to host memory, through page-locked staging by
// several threads when `dst` is pageable and large; *finite (when given, FP32
// data) is cleared if a value is not finite.
int copy_to_host(void *dst, const void *src, size_t bytes, bool *finite = nullptr);

// Whether a call that failed so may succeed with less device memory.
inline bool memory_failure(int code) { return code == VEXT_ERR_MEMORY || code == VEXT_ERR_CUDA; }

// Unique id of the calling thread's current context (0 when unavailable).
unsigned long long current_context_id();

constexpr int kMaxTypes = 1024;     // distinct framework (sigma, epsilon) pairs
constexpr double kDefaultRSplit = 5.0;

struct alignas(16) RegionInfo {
    double of[3];       // origin, fractional
    double rho;         // max distance (A) from the origin to any pose center
    long long off;      // first entry
    int n_near;         // near entries
    int n_total;        // all entries
    int i0, j0, k0;     // first grid center (field regions)
    int ni, nj, nk;     // grid centers per axis (field regions)
    int n_inner;        // far entries within the cutoff of every site of every pose of the
                        // region (they follow the near entries; the shell ones come last)
    int n_outer;        // the last shell entries: beyond rc + rho + 1e-3 A of the origin,
                        // hence beyond rc of every pose center of the region
    int n_mid;          // the first of the inner entries: too near the origin for its local
                        // expansion (taylor.cuh), which covers the rest
    int n_shella;       // the first of the shell entries: so near that a symmetric director's
                        // site on the entry's side is inside the cutoff for every pose (site
                        // lists: within the cutoff of the origin)
    int n_tnear;        // the first of the expansion's entries: the others need fewer degrees
    int pad[1];
};
static_assert(sizeof(RegionInfo) % 16 == 0, "RegionInfo must stay 16-byte aligned");

struct RegionSet {
    // key
    int size = 0, bi = 0, bj = 0, bk = 0;   // field regions (size > 0) or bins (size == 0)
    int nb[3] = {0, 0, 0};                  // bins per axis (pose regions)
    double bin_width = 0;                   // target bin width (A, pose regions)
    double r_split = 0;
    bool sites = false;                     // regions of voxels: lists about single sites
    bool expand = false;                    // classes for local expansions (taylor.cuh)
    // data
    int n_regions = 0;
    int n_ri = 0, n_rj = 0, n_rk = 0;       // regions per axis
    long long n_entries = 0, n_near = 0, n_outer = 0;
    long long n_taylor = 0;                 // inner entries of the expansions (taylor.cuh)
    double d_taylor = 1e30;                 // their smallest distance from the origin
    double d_tfar = 1e30;                   // from here on kTaylorFarOrder degrees do
    double taylor_radius = 0;               // every site of a region lies this near its origin
    RegionInfo *d_info = nullptr;
    float4 *d_hi = nullptr, *d_lo = nullptr;
    std::shared_ptr<int> use = std::make_shared<int>(0);   // batches on it hold a copy
    std::vector<RegionInfo> h_info;
    long long capacity = 0;                 // allocated entries (hi and lo)
    bool stale = false;                     // rebuild before the next use
    float build_ms = 0;
    ~RegionSet();
};

// One system's local expansions in a field or batch (taylor.cuh): the
// evaluation matrix and the per-region polynomials (null poly: the system's
// inner pairs are summed directly).
struct TaylorPlan {
    double *poly = nullptr;     // [n_regions][kTaylorPolyPad]
    float *matrix = nullptr;    // [kTaylorPad][rows]
    size_t poly_cap = 0, matrix_cap = 0;
    int rows = 0;               // outputs of a region's poses, padded to the tile
    int outs = 0;               // outputs per pose: 1 (energy) or 7
    void release() {
        device_free(poly);
        device_free(matrix);
        poly = nullptr;
        matrix = nullptr;
        poly_cap = matrix_cap = 0;
    }
};

// One system's view for the warp-per-pose kernel (posebatch.cu).
struct PoseBatchSys {
    Mat3 H, Hinv;
    double rc2;
    float rc2f;
    double off0, off1;
    int nb0, nb1, nb2;
    const RegionInfo *regs;
    const float4 *hi, *lo;
    const double *td;   // (c12, c6, shift, floor2) per type
    const float4 *tf;
};

struct SiteField;
void site_field_free(SiteField *f);

struct System {
    int device = 0;
    Mat3 H, Hinv;
    double einv[3];        // |column k of Hinv| = 1 / lattice-plane spacing
    int n_atoms = 0, n_types = 0;
    double guest_sigma = 0, guest_epsilon = 0, offsets[2] = {0, 0}, cutoff = 0, temperature = 0;
    double max_offset = 0;
    // FNV-1a hash of the framework as the region lists see it (cell, cutoff,
    // wrapped fractional coordinates, type ids and the framework (sigma,
    // epsilon) of every type): systems with equal hashes differ only in the
    // guest, so one region-list set serves them all when it is built for the
    // largest site offset among them
    uint64_t frame_hash = 0;
    void *d_base = nullptr;    // one allocation holding the five arrays below
    double *d_frac = nullptr;
    int *d_type = nullptr;
    float4 *d_tf = nullptr;
    double *d_td = nullptr;
    int *d_status = nullptr;   // device status word
    std::vector<double> h_td;  // n_types x 4
    std::vector<RegionSet *> sets;
    // expected expansion entries per region of field lists: (size, cb, r_split)
    std::map<std::tuple<int, int, double>, double> expansion_entries;
    bool outputs_finite = true;    // float32 outputs of the last vext_field call
    // scratch of the field path
    double *d_e64 = nullptr;
    size_t e64_cap = 0;
    int *d_refine = nullptr;   // [0] = count, then pose indices
    size_t refine_cap = 0;
    double *d_axes = nullptr;
    size_t axes_cap = 0;
    float *d_f32 = nullptr;        // host-output staging of the float32 field
    size_t f32_cap = 0;
    float *d_small = nullptr;      // marginal, 2 x site, grid
    size_t small_cap = 0;
    double *d_e64T = nullptr;      // [S^3][O] FP64 output staging
    size_t e64T_cap = 0;
    int *d_flags = nullptr;        // [0] non-finite count
    size_t flags_cap = 0;
    // local expansions of the field path: plan of the last (lists, directors)
    TaylorPlan field_plan;
    const RegionSet *field_plan_set = nullptr;
    std::vector<double> field_plan_axes;
    float *d_sums = nullptr;
    size_t sums_cap = 0;
    // site-by-site sums of the field path (sites.cuh)
    SiteField *site_field = nullptr;
    // poses from which on the field path does without site-by-site sums and
    // without expansions, because their scratch could not be had
    long long no_sites_from = 1LL << 62, no_expansions_from = 1LL << 62;
    // scratch of the pose path
    void *d_pose_scratch = nullptr;
    size_t pose_scratch_cap = 0;
    double *d_pose_io = nullptr;     // host-pointer entry staging
    size_t pose_io_cap = 0;
    PoseBatchSys *d_pose_desc = nullptr;   // warp-per-pose path: device copy of h_pose_desc
    PoseBatchSys h_pose_desc;
    long long *d_pose_offsets = nullptr;
    cudaStream_t stream = nullptr;   // private stream for host-pointer entries
    cudaStream_t aux = nullptr;      // second stream: copy-back beside pair work
    cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    bool timed = false;              // ev[0..2] hold the last field call's kernel/epilogue
    bool list_timed = false;         // ev[3..4] hold the last list build
    bool split_timed = false;        // ev[5] separates the near and far kernels
    // cached one-system forward + adjoint batch (vext_field_adjoint_device and
    // vext_field_adjoint into page-locked buffers), keyed by grid size,
    // directors, options and the FP64 energy output; its float32 outputs are
    // retargeted per call
    vext_batch adj_batch = nullptr;
    int adj_size = 0;
    std::vector<double> adj_axes;
    double adj_key[4] = {0, 0, 0, 0};   // r_split, band_lo, band_hi, variant
    bool adj_device = false;            // outputs in device memory
    double *adj_energy64 = nullptr;
    float *d_g32 = nullptr;          // host-output staging of the float32 gradient
    size_t g32_cap = 0;
    // the host entry's batches (vext_field_adjoint): one per block of
    // directors, each writing its contiguous slice of d_f32 / d_g32, so the copy
    // of one block overlaps the next block's pair work
    std::vector<vext_batch> host_parts;
    std::vector<cudaEvent_t> host_part_done;
    int host_size = 0;
    std::vector<double> host_axes;
    double host_key[4] = {0, 0, 0, 0};
    float *host_e = nullptr, *host_g = nullptr;
    // the same entry into page-locked buffers: one batch over all directors,
    // its poses slab by slab along the slowest grid axis (batch_run_slab)
    vext_batch slab_batch = nullptr;
    int slab_size = 0, slab_count = 0;
    std::vector<double> slab_axes;
    double slab_key[4] = {0, 0, 0, 0};
    std::mutex lock;
    void drop_adjoint_batch();   // both caches (they point into the region sets)
    void drop_host_parts();
    ~System();
};

// Batches (batch.cu); lock_systems = false when the caller holds the locks.
int batch_build(int n_systems, const vext_system *systems, int size, int n_axes,
                const double *axes, const vext_options *opt, float *const *outputs,
                float *const *gradients, double *const *outputs_f64, bool lock_systems,
                vext_batch *out, int rule_axes, int slabs);
int batch_replay(vext_batch b, cudaStream_t stream);
int batch_run_slab(vext_batch b, int k, cudaStream_t stream, int *plane0, int *plane1);
int batch_slab_status(vext_batch b);
int batch_retarget(vext_batch b, int k, float *out, float *grad, cudaStream_t stream);
bool device_memory(const void *p);   // device or managed, not host memory

// Region sets (system.cu)
// expand_axes: directors of a call that sums by local expansions where they pay
// (adjoint: forward + adjoint); 0: lists without classes for them.
int get_field_regions(System *sys, int size, int cb, double r_split, int expand_axes,
                      bool adjoint, RegionSet **out, cudaStream_t stream);
int get_block_regions(System *sys, int size, int bi, int bj, int bk, double rho, double offset,
                      bool sites, bool expand, double r_split, RegionSet **out,
                      cudaStream_t stream);
// Delete the lists for single sites that neither a batch nor the field path's
// plan uses (under the system's lock).
void drop_idle_site_lists(System *sys);
constexpr double kBinWidth = 0.75;  // pose-bin width between lattice planes (A)
int get_bin_regions(System *sys, double r_split, RegionSet **out, cudaStream_t stream,
                    double bin_width = kBinWidth);
void choose_block_shape(const Mat3 &H, int size, int cb, int &bi, int &bj, int &bk);
double block_radius(const Mat3 &H, int size, int ni, int nj, int nk);

// Device buffer growth helper
template <typename T>
int ensure_capacity(T *&ptr, size_t &cap, size_t need) {
    if (need <= cap && ptr) return 0;
    if (ptr) device_free(ptr);
    ptr = nullptr;
    cap = 0;
    size_t n = need < 1 ? 1 : need;
    cudaError_t err = device_malloc((void **)&ptr, n * sizeof(T));
    if (err != cudaSuccess)
        return fail(VEXT_ERR_MEMORY, "device allocation of %zu bytes failed: %s", n * sizeof(T),
                    cudaGetErrorString(err));
    cap = n;
    return 0;
}

int check_status(System *sys, cudaStream_t stream);  // reads and clears the status word


struct Options {
    int mode;
    double r_split;
    double band_lo, band_hi;
    int cb;
    int variant;
    int batch_shape;   // 0 = autotune, else 1 + kernel-table index
};
Options resolve_options(const vext_options *opt);

// |d0|^2 (entry - grid center) beyond which no site of a pose lies inside any
// type's contact floor: a site is at least |d0| - max|o| from the entry, so
// beyond sqrt(max floor2) + max|o| (with a relative margin far above FP64
// rounding) every pair skips the floor test without changing a bit.
inline double floor_clear_radius2(const System &sys) {
    double fl = 0.0;
    for (int t = 0; t < sys.n_types; ++t) fl = std::max(fl, sys.h_td[4 * t + 3]);
    const double rf =
        (std::sqrt(fl) + std::max(std::fabs(sys.offsets[0]), std::fabs(sys.offsets[1]))) *
            (1.0 + 1e-9) + 1e-9;
    return rf * rf;
}

// Far entries per FP32 energy partial in the unmasked pass over inner entries:
// kFlush, or kExpandFlush of those too near for an expansion (RegionInfo::n_mid).
// A partial's rounding grows with its sum, and these lie next to one another in the
// lists: mean rms error at E <= 0 of six slab frameworks 1.95e-5 K with partials over
// 16, 1.73e-5 over 8, 1.67e-5 over 4 (60^3 x 64 layered forward + adjoint 17.70, 17.64
// and 17.81 ms), 1.70e-5 where all pairs are summed in the lists' plain order.
constexpr int kFlush = 16, kExpandFlush = 4;

// Directors per work item of a batch with these options (32 or 64; its
// regions hold 512 / that many grid centers).
int batch_item_directors(const Options &o, bool adjoint);

// Pose pipeline (pose.cu): enqueue without host synchronisation, then check.
int pose_enqueue(System *sys, int n, const double *centers, const double *quats,
                 const Options &o, double *energy, double *gc, double *gq, double *gu,
                 cudaStream_t st);
int pose_status(System *sys, cudaStream_t st);

// Warp-per-pose evaluation of n poses of one system on its bin lists `rs`
// (small batches, where the binned pipeline's per-bin CTAs would idle).
int pose_warp_enqueue(System *sys, const RegionSet *rs, int n, const double *centers,
                      const double *quats, const Options &o, double *energy, double *gc,
                      double *gq, double *gu, cudaStream_t st);

// One system's view of its bin lists for the pose kernels.
PoseBatchSys pose_describe(const System *sys, const RegionSet *rs);
int warps_per_pose(long long n);
// Its device copy, uploaded when it changed.
int pose_upload_desc(System *sys, const RegionSet *rs, const PoseBatchSys **out);

// Field kernel launcher (field.cu): computes E64 [O][S^3] for all regions.
int launch_field(System *sys, const RegionSet *rs, int n_axes, const double *axes_host,
                 const double *d_axes, double *d_e64, int cb, int variant, cudaStream_t stream,
                 bool *expanded);

}  // namespace vext

struct vext_system_s {
    vext::System sys;
};
