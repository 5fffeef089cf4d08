// Fields summed site by site.
//
// The two-site energy of a pose is V(c + o_0 u) + V(c + o_1 u), with V the
// potential of one site.  On a fine grid the sites of different poses lie
// close together: site s of director j sits at a shift of o_s u_j from its
// center, so in units of the grid it lands at the same place of every voxel.
// A region is here a block of 8 or 16 voxels; the 2 O sites that fall into each
// (O directors, two sites) have the same places relative to the
// region's origin in every region.  They are split once into clusters of 64
// neighbours, and a warp evaluates V and its gradient at one cluster: what
// counts for its lists is the cluster's radius (0.2-0.5 A) instead of the
// site offset plus the region radius (0.9-1.6 A), so far fewer images need
// FP64 or a cutoff test.  Images far from the region's origin act through its
// local expansion (taylor.cuh).  A pose then adds its two sites.
#pragma once

#include "taylor.cuh"

namespace vext {

constexpr int kClusterSites = 64;

// One system's sites on one grid for one set of directors, as the kernels see
// them.
struct SiteView {
    Mat3 H;
    double rc2, off0, off1, r_split;
    float rc, rc2f;
    double floor_out;           // site-atom distance beyond which no contact floor applies
    int S, O;
    const RegionInfo *regs;     // regions of voxels
    const float4 *hi, *lo;
    const float4 *tf;
    const double *td;
    int n_regions, bi, bj, bk, nrj, nrk;
    int n_clusters, n_sites;    // sites padded to whole clusters
    const double *pos;          // [n_sites][3] relative to the region origin
    const int4 *meta;           // [n_sites][2]: (2 o + s or -1, a_i, a_j, a_k), (d_i, d_j, d_k, 0):
                                // voxel a of the block; the center is voxel + d (mod S)
    const float4 *cluster;      // [n_clusters]: middle, radius
    const double *shift;        // [2 O][3]: place within the voxel, in voxels
    const int4 *floor;          // [2 O]: voxel of the site = center + floor (mod S)
    const double *poly;         // local expansions, or null: inner entries are summed directly
    const float *eval;          // their higher degrees at the sites: [n_regions][n_sites] x (1 or 4)
};

struct SitePlan {
    const RegionSet *rs = nullptr;   // null: the system is summed pose by pose
    SiteView view;
    void *arena = nullptr;           // the view's own arrays
    size_t arena_cap = 0;
    int reach_lo = 0, reach_hi = 0;  // a center's sites lie at most this many voxel planes
                                     // before and after its own (slowest axis)
    TaylorPlan expansion;            // matrix and polynomials (poly null: none)
    void release() {
        device_free(arena);
        arena = nullptr;
        arena_cap = 0;
        expansion.release();
        rs = nullptr;
    }
};

// Device buffers that one system at a time works in.
struct SiteScratch {
    float *sums = nullptr, *eval = nullptr;
    double *value = nullptr;   // [2 O][S^3] x (1 or 4): V, and its gradient
    size_t sums_cap = 0, eval_cap = 0, value_cap = 0;
    void release() {
        device_free(sums);
        device_free(eval);
        device_free(value);
        sums = eval = nullptr;
        value = nullptr;
        sums_cap = eval_cap = value_cap = 0;
    }
};

// The field path's plan, kept for its last (lists, directors).
struct SiteField {
    SitePlan plan;
    SiteScratch scratch;
    std::vector<double> axes;
};

// Whether the site-by-site sum is expected to be the faster one (the rule is
// explained at its definition).
bool sites_worthwhile(const System &sys, int size, int n_axes, const Options &o, bool adjoint);

// Lists of the voxel regions of a system (cached like the other region sets).
int get_site_regions(System *sys, int size, int block, double r_split, RegionSet **out,
                     cudaStream_t stream);
// Voxels of a region: 8 in batches; a field call that builds its lists pays
// twice the list work and memory for them (the 60^3 x 64 layered calculate_vext
// 28.4 ms with 8, 16.0 with 16).  The sums with 8 and 16: layered adjoint 11.2 and
// 11.6 ms, uneven batch adjoint 16.4 and 20.0; 47^3 x 50 skewed field 7.67 and 7.48.
constexpr int kBatchVoxels = 8, kFieldVoxels = 16;

int site_plan_build(const System &sys, const RegionSet &rs, int n_axes, const double *axes,
                    bool adjoint, SitePlan &plan, cudaStream_t stream);

int site_scratch_reserve(const SitePlan &plan, bool adjoint, SiteScratch &scratch);

// V (and its gradient) into scratch.value at the sites of region planes
// [plane0, plane1) along the slowest axis (with plane 0: all the expansions).
int site_enqueue(const System &sys, const SitePlan &plan, bool adjoint,
                 const SiteScratch &scratch, int plane0, int plane1, int *status,
                 cudaStream_t stream);

// The view with the lists where they stand now (a rebuild may have moved them).
SiteView site_view(const SitePlan &plan);

// Forward: pose energies [O][S^3] of the last site_enqueue.
int site_energies(const SitePlan &plan, const SiteScratch &scratch, double *e64,
                  cudaStream_t stream);

}  // namespace vext
