// Local expansion of the far inner pairs of a region about its origin.
//
// Images farther than a radius d_T from the origin O of a region (a block of
// grid centers) act on its sites, all within R of O, as a smooth potential.
// With x the image and s the site relative to O,
//   |x - s|^(-2 lam) = sum_n C_n^lam(cos g) |s|^n / |x|^(n + 2 lam),
//   C_n^lam = sum_k beta^lam_{n,k} P_{n-2k}    (Gegenbauer in Legendre),
// and the addition theorem of the real solid harmonics R_lm give
//   sum_x c12 |x-s|^-12 - c6 |x-s|^-6 = sum_{l,m,k} |s|^{2k} R_lm(s) A_klm,
//   A_klm = sum_x (c12 beta^6_{l+2k,k} |x|^{-2(l+k)-12}
//                  - c6 beta^3_{l+2k,k} |x|^{-2(l+k)-6}) R_lm(x)
// truncated at degree l + 2k <= kTaylorOrder.  The terms of degree 0 to 3
// are kept apart as an FP64 polynomial (taylor_poly); the rest, at most a
// few tenths of a kelvin per pose, are FP32 sums in units of R.
#pragma once

#include <utility>

#include "internal.cuh"

namespace vext {

constexpr int kTaylorOrder = 12;
constexpr int kTaylorFarOrder = 8;   // degrees that entries from RegionSet::d_tfar on need
constexpr int kTaylorLow = 4;        // degrees below this: the FP64 polynomial
constexpr int kTaylorPoly = 20;      // its coefficients
constexpr int kTaylorPolyPad = 24;   // doubles per region

// Expected entries per region below which site lists are built without a class
// for the expansion (they gain from about 40), and lists for poses without one
// whatever the directors (taylor_pays).
constexpr double kTaylorMinEntries = 40, kTaylorMinEntriesPoses = 120;

// Columns |m| of the expansion that one warp sums (balanced: 66-76 sums).
constexpr int kTaylorRoles = 6;
__host__ __device__ constexpr int role_column(int r, int i) {
    constexpr int at[kTaylorRoles][3] = {{1, -1, -1}, {2, 11, -1}, {3, 9, 12},
                                         {0, 6, -1},  {4, 7, -1},  {5, 8, 10}};
    return at[r][i];
}

// (l, k) pairs of column m with degree kTaylorLow..kTaylorOrder before (l0, k0).
__host__ __device__ constexpr int column_pos(int m, int l0, int k0) {
    int c = 0;
    for (int l = m; l <= kTaylorOrder; ++l)
        for (int k = 0; l + 2 * k <= kTaylorOrder; ++k) {
            if (l == l0 && k == k0) return c;
            if (l + 2 * k >= kTaylorLow) ++c;
        }
    return c;
}
__host__ __device__ constexpr int column_sums(int m) {
    return m < 0 ? 0 : column_pos(m, -1, -1) * (m ? 2 : 1);
}
__host__ __device__ constexpr int role_sums(int r) {
    return column_sums(role_column(r, 0)) + column_sums(role_column(r, 1)) +
           column_sums(role_column(r, 2));
}
__host__ __device__ constexpr int role_start(int r) {
    int c = 0;
    for (int q = 0; q < r; ++q) c += role_sums(q);
    return c;
}
constexpr int kTaylorSums = role_start(kTaylorRoles);          // 435
constexpr int kTaylorPad = (kTaylorSums + 15) / 16 * 16;       // row length of the sums

// beta^lam_{n,k}: C_n^lam = sum_k beta^lam_{n,k} P_{n-2k}.
__host__ __device__ constexpr double gegenbauer_legendre(int n, int k, double lam) {
    double v = 2.0 * (n - 2 * k) + 1.0;
    for (int i = 0; i < n - k; ++i) v *= (lam + i) / (1.5 + i);
    for (int i = 0; i < k; ++i) v *= (lam - 0.5 + i) / (i + 1.0);
    return v;
}
__host__ __device__ constexpr double sqrt_newton(double x) {
    if (x <= 0) return 0.0;
    double r = x > 1 ? x : 1.0;
    for (int i = 0; i < 60; ++i) r = 0.5 * (r + x / r);
    return r;
}

template <int B, int E, typename F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (B < E) {
        f(std::integral_constant<int, B>{});
        static_for<B + 1, E>(f);
    }
}

// The degree 0-3 polynomial of a region at s (Angstrom, FP64) and its
// gradient: p = (1, x, y, z, xx, xy, xz, yy, yz, zz, xxx, xxy, xxz, xyy,
// xyz, xzz, yyy, yyz, yzz, zzz).
__device__ __forceinline__ double taylor_poly(const double *p, double x, double y, double z) {
    const double qx = fma(p[10], x, fma(p[11], y, fma(p[12], z, p[4])));
    const double qy = fma(p[13], y, fma(p[14], z, p[5]));
    const double qz = fma(p[15], z, p[6]);
    const double lx = fma(x, qx, fma(y, qy, fma(z, qz, p[1])));
    const double ry = fma(p[16], y, fma(p[17], z, p[7]));
    const double rz = fma(p[18], z, p[8]);
    const double ly = fma(y, ry, fma(z, rz, p[2]));
    const double lz = fma(z, fma(p[19], z, p[9]), p[3]);
    return fma(x, lx, fma(y, ly, fma(z, lz, p[0])));
}

__device__ __forceinline__ double taylor_poly_grad(const double *p, double x, double y, double z,
                                                   double (&g)[3]) {
    const double x2 = 2.0 * x, y2 = 2.0 * y, z2 = 2.0 * z;
    g[0] = p[1] + x2 * (p[4] + p[11] * y + p[12] * z + 1.5 * p[10] * x) +
           y * (p[5] + p[13] * y + p[14] * z) + z * (p[6] + p[15] * z);
    g[1] = p[2] + y2 * (p[7] + p[13] * x + p[17] * z + 1.5 * p[16] * y) +
           x * (p[5] + p[11] * x + p[14] * z) + z * (p[8] + p[18] * z);
    g[2] = p[3] + z2 * (p[9] + p[15] * x + p[18] * y + 1.5 * p[19] * z) +
           x * (p[6] + p[12] * x + p[14] * y) + y * (p[8] + p[17] * y);
    return taylor_poly(p, x, y, z);
}

// The polynomial at both sites of a pose.
__device__ __forceinline__ double taylor_pair(const double *p, double cx, double cy, double cz,
                                              double off0, double off1, double ux, double uy,
                                              double uz) {
    return taylor_poly(p, cx + off0 * ux, cy + off0 * uy, cz + off0 * uz) +
           taylor_poly(p, cx + off1 * ux, cy + off1 * uy, cz + off1 * uz);
}

// ---------------------------------------------------------------- host side

// Smallest distance from the origin at which the truncation error of an
// expansion of this order is within tolerance for sites within `radius`
// (system.cu builds the lists with it); a value beyond the cutoff when there is
// none.
double taylor_start(const System &sys, double radius, int order = kTaylorOrder);

// Whether summing the inner pairs of `rs` by expansion is the faster way for
// `n_axes` directors (the rule is explained at its definition), and allowed
// for this system's pair coefficients.
bool taylor_worthwhile(const System &sys, const RegionSet &rs, int n_axes, bool adjoint);
// The rule itself, for `entries` per region and `poses` of a region.
bool taylor_pays(double entries, double poses, bool adjoint);

// Build the evaluation matrix of a (system, region shape, directors) triple.
int taylor_prepare(const System &sys, const RegionSet &rs, int n_axes, const double *d_axes,
                   bool adjoint, TaylorPlan &plan, cudaStream_t stream);

// The same for single sites: `d_sites` [n_sites][3] relative to a region's
// origin (sites.cuh), outputs value (and gradient) per site.
int taylor_prepare_sites(const System &sys, const RegionSet &rs, int n_sites,
                         const double *d_sites, bool adjoint, TaylorPlan &plan,
                         cudaStream_t stream);
int taylor_enqueue_sites(const System &sys, const RegionSet &rs, int n_sites,
                         const TaylorPlan &plan, float *sums, float *out, int *status,
                         cudaStream_t stream);
size_t taylor_workspace_sites(const RegionSet &rs);   // floats of `sums`

// Whether a pair's truncation error stays within tolerance for `sys` on lists
// that another guest of the same framework may have built.
bool taylor_allowed(const System &sys, const RegionSet &rs);

// Floats of the per-region sums taylor_enqueue needs as workspace.
inline size_t taylor_workspace(const RegionSet &rs) { return (size_t)rs.n_regions * kTaylorPad; }

// Sum the expansions of every region (with the near shell entries when
// `symmetric`) and evaluate degrees >= kTaylorLow at every pose: the energies
// into e32 or e64 ([O][S^3]), the gradients (dE/dc, tangent dE/du) into g32
// ([O][S^3][6], adjoint plans).
int taylor_enqueue(const System &sys, const RegionSet &rs, int n_axes, const TaylorPlan &plan,
                   bool symmetric, float *sums, float *const *e32, double *e64,
                   float *const *g32, cudaStream_t stream);

}  // namespace vext
