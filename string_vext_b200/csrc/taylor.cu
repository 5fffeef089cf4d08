// Sums and evaluation of the local expansions (taylor.cuh).
//
//   taylor_sums_kernel  one CTA per region: A_klm over its expansion entries
//                       (FP32, one warp per group of columns |m|, a lane per
//                       entry) and the degree 0-3 polynomial (FP64, a warp)
//   taylor_eval_kernel  the poses of a full block sit at the same places
//                       relative to the origin in every region of a system,
//                       so values and gradients at all poses are one matrix
//                       product: [outputs of a region x sums] . [sums x
//                       regions], register-tiled packed FP32; single sites
//                       take taylor_mma_kernel (taylormma.cu) instead
//   taylor_matrix_kernel  that matrix: solid harmonics and their gradients
//                       at the poses' sites, in FP64, rounded once
//
// Replaces, for far entries inside the cutoff of every site, the pair loop
// over all poses: per entry about 1,500 FMA instead of 12.5 per (site, entry)
// pair of a region's 1,024 sites.
#include <algorithm>
#include <cmath>
#include <vector>

#include "pair.cuh"
#include "taylor.cuh"
#include "taylormma.cuh"

namespace vext {

struct SumArgs {
    const RegionInfo *regs;
    int n_regions;
    const float4 *hi, *lo;
    const float4 *tf;
    const double *td;
    float inv_r;          // 1 / unit length
    int symmetric;        // near shell entries (RegionInfo::n_shella) belong to the expansion
    int rest;             // inner entries outside the expansion are all summed in FP32
    int far;              // entries after the first n_tnear lie beyond RegionSet::d_tfar
    float *sums;          // [n_regions][kTaylorPad]; split: the operand of taylor_mma_kernel
    int split;
    double *poly;         // [n_regions][kTaylorPolyPad]
};

// Column M of one entry: acc += W_kl Q_lM (C_M, S_M), degrees >= kTaylorLow.
// Q: Schmidt semi-normalised solid-harmonic factors (r^l P_l^M / (x^2 +
// y^2)^{M/2}); a[j] = c6 r^-6 u^j, b[j] = c12 r^-12 u^j with u = R^2 / r^2.
template <int M, int AT, int ORDER>
__device__ __forceinline__ void column_add(float z, float r2, const float *cm, const float *sm,
                                           const float (&a)[ORDER + 1],
                                           const float (&b)[ORDER + 1], float *acc) {
    // normalised Q_MM: N_M = (2 - d_M0) / (2M)! and (2M - 1)!!
    constexpr double qmm = [] {
        double v = 1.0;
        for (int m = 2; m <= M; ++m) v *= sqrt_newton((2.0 * m - 1.0) / (2.0 * m));
        return v;
    }();
    float q0 = 0.f, q1 = 0.f;
    static_for<M, ORDER + 1>([&](auto L) {
        constexpr int l = decltype(L)::value;
        float q;
        if constexpr (l == M) {
            q = (float)qmm;
        } else if constexpr (l == M + 1) {
            constexpr float f = (float)((2.0 * l - 1.0) / sqrt_newton((double)l * l - M * M));
            q = f * z * q1;
        } else {
            constexpr double nrm = 1.0 / sqrt_newton((double)l * l - M * M);
            constexpr float f = (float)((2.0 * l - 1.0) * nrm);
            constexpr float g = (float)(-sqrt_newton((l - 1.0) * (l - 1.0) - M * M) * nrm);
            q = fmaf(f * z, q1, g * r2 * q0);
        }
        q0 = q1;
        q1 = q;
        static_for<0, (ORDER - l) / 2 + 1>([&](auto K) {
            constexpr int k = decltype(K)::value;
            if constexpr (l + 2 * k >= kTaylorLow) {
                constexpr float b6 = (float)gegenbauer_legendre(l + 2 * k, k, 6.0);
                constexpr float b3 = (float)-gegenbauer_legendre(l + 2 * k, k, 3.0);
                constexpr int at = AT + column_pos(M, l, k) * (M ? 2 : 1);
                const float w = fmaf(b6, b[l + k], b3 * a[l + k]) * q;
                if constexpr (M == 0) {
                    acc[at] += w;
                } else {
                    acc[at] = fmaf(w, cm[M], acc[at]);
                    acc[at + 1] = fmaf(w, sm[M], acc[at + 1]);
                }
            }
        });
    });
}

// 32 sums held by each lane -> lane i holds the warp total of sum i.
__device__ __forceinline__ float transpose_sum(float *v, int lane) {
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = up ? v[i] : v[i + h];
            const float keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    return v[0];
}

// The sums of one role over entries [first, n), up to degree ORDER.
template <int ROLE, int ORDER>
__device__ __forceinline__ void role_entries(const SumArgs &s, const float4 *hi, int first, int n,
                                             int lane, float *acc) {
    constexpr int m0 = role_column(ROLE, 0), m1 = role_column(ROLE, 1),
                  m2 = role_column(ROLE, 2);
    constexpr int c0 = m0 <= ORDER ? m0 : 0, c1 = m1 <= ORDER && m1 > 0 ? m1 : 0,
                  c2 = m2 <= ORDER && m2 > 0 ? m2 : 0;
    constexpr int mtop = c0 > c1 ? (c0 > c2 ? c0 : c2) : (c1 > c2 ? c1 : c2);
    float4 next = first + lane < n ? hi[first + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int e = first + lane; e < n; e += 32) {
        const float4 h = next;
        const float4 tp = s.tf[__float_as_int(h.w)];   // (c12, c6, -, -)
        if (e + 32 < n) next = hi[e + 32];
        const float x = h.x * s.inv_r, y = h.y * s.inv_r, z = h.z * s.inv_r;
        const float r2 = fmaf(x, x, fmaf(y, y, z * z));
        const float u = __frcp_rn(r2);
        const float d2 = fmaf(h.x, h.x, fmaf(h.y, h.y, h.z * h.z));
        const float i2 = __frcp_rn(d2);
        const float i6 = i2 * i2 * i2;
        float a[ORDER + 1], b[ORDER + 1];
        a[0] = tp.y * i6;
        b[0] = tp.x * i6 * i6;
#pragma unroll
        for (int j = 1; j <= ORDER; ++j) {
            a[j] = a[j - 1] * u;
            b[j] = b[j - 1] * u;
        }
        float cm[mtop + 1], sm[mtop + 1];
        cm[0] = 1.f;
        sm[0] = 0.f;
#pragma unroll
        for (int m = 1; m <= mtop; ++m) {
            cm[m] = fmaf(x, cm[m - 1], -y * sm[m - 1]);
            sm[m] = fmaf(x, sm[m - 1], y * cm[m - 1]);
        }
        if constexpr (m0 <= ORDER) column_add<m0, 0, ORDER>(z, r2, cm, sm, a, b, acc);
        if constexpr (m1 >= 0 && m1 <= ORDER)
            column_add<m1, column_sums(m0), ORDER>(z, r2, cm, sm, a, b, acc);
        if constexpr (m2 >= 0 && m2 <= ORDER)
            column_add<m2, column_sums(m0) + column_sums(m1), ORDER>(z, r2, cm, sm, a, b, acc);
    }
}

// n entries, the first `n_full` of which need every degree.  The others, four
// fifths of a fine grid's, take a third of the sums: 2.17 -> 1.55 ms for the
// 28,800 regions of the 60^3 x 64 layered field (1.83 with the shell entries that
// the expansion has held since; the whole field 14.67 -> 14.08
// ms; with order 7, which starts farther out, 14.21, with 9 14.20).
template <int ROLE>
__device__ __forceinline__ void role_sum(const SumArgs &s, const float4 *hi, int n_full, int n,
                                         int lane, int region, float *out) {
    constexpr int N = role_sums(ROLE), NP = (N + 31) / 32 * 32;
    float acc[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[i] = 0.f;
    role_entries<ROLE, kTaylorOrder>(s, hi, 0, n_full, lane, acc);
    role_entries<ROLE, kTaylorFarOrder>(s, hi, n_full, n, lane, acc);
#pragma unroll
    for (int g = 0; g < NP / 32; ++g) {
        const float t = transpose_sum(acc + 32 * g, lane);
        const int i = role_start(ROLE) + 32 * g + lane;
        if (32 * g + lane >= N) continue;
        if (s.split) mma_store_split<kMmaN>(s.sums, region, kMmaOrder.at[i], t);
        else out[i] = t;
    }
}

// Degrees 0-3 in FP64: with phi(q) = c12 q^-6 - c6 q^-3 + shift at q = |x|^2
// and s.x the only direction-dependent term, phi(|x|^2 - 2 x.s + s^2) to
// third degree in s.  Entries [-n_rest, 0) are not in the expansion but summed in
// FP32 with coefficients rounded to it: what the rounding took off them is added
// here.  (Summed pair by pair the errors of c6 and shift partly cancel over all
// entries; an expansion leaves those of the nearest ones alone.  Mean rms error at
// E <= 0 of six slab frameworks: pair by pair 1.70e-5 K, by expansion 1.67e-5, with
// the correction 1.49e-5.)
__device__ __forceinline__ void poly_sum(const SumArgs &s, const float4 *hi, const float4 *lo,
                                         int n_rest, int n, int lane, double *out) {
    double v[24];   // f0, f1, f1 x (3), f2 x (3), f2 xx (6), f3 xxx (10)
#pragma unroll
    for (int i = 0; i < 24; ++i) v[i] = 0.0;
#pragma unroll 1
    for (int e = lane - n_rest; e < n; e += 32) {
        const float4 h = hi[e], l = lo[e];
        const double x = (double)h.x + (double)l.x, y = (double)h.y + (double)l.y,
                     z = (double)h.z + (double)l.z;
        const int t = __float_as_int(h.w);
        double c12 = s.td[4 * t], c6 = s.td[4 * t + 1], shift = s.td[4 * t + 2];
        if (e < 0) {
            const float4 r = s.tf[t];
            c12 -= (double)r.x;
            c6 -= (double)r.y;
            shift -= (double)r.z;
        }
        const double i2 = rcp64_nr<2>(fma(x, x, fma(y, y, z * z)));
        const double i6 = i2 * i2 * i2, b = c12 * i6 * i6, a = c6 * i6;
        const double i4 = i2 * i2;
        const double f1 = i2 * fma(-6.0, b, 3.0 * a), f2 = i4 * fma(42.0, b, -12.0 * a),
                     f3 = i6 * fma(-336.0, b, 60.0 * a);
        v[0] += b - a + shift;
        v[1] += f1;
        v[2] = fma(f1, x, v[2]);
        v[3] = fma(f1, y, v[3]);
        v[4] = fma(f1, z, v[4]);
        const double gx = f2 * x, gy = f2 * y, gz = f2 * z;
        v[5] += gx;
        v[6] += gy;
        v[7] += gz;
        v[8] = fma(gx, x, v[8]);
        v[9] = fma(gx, y, v[9]);
        v[10] = fma(gx, z, v[10]);
        v[11] = fma(gy, y, v[11]);
        v[12] = fma(gy, z, v[12]);
        v[13] = fma(gz, z, v[13]);
        const double hxx = f3 * x * x, hxy = f3 * x * y, hyy = f3 * y * y, hzz = f3 * z * z;
        v[14] = fma(hxx, x, v[14]);
        v[15] = fma(hxx, y, v[15]);
        v[16] = fma(hxx, z, v[16]);
        v[17] = fma(hyy, x, v[17]);
        v[18] = fma(hxy, z, v[18]);
        v[19] = fma(hzz, x, v[19]);
        v[20] = fma(hyy, y, v[20]);
        v[21] = fma(hyy, z, v[21]);
        v[22] = fma(hzz, y, v[22]);
        v[23] = fma(hzz, z, v[23]);
    }
#pragma unroll
    for (int i = 0; i < 24; ++i)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    if (lane == 0) {
        const double k3 = -4.0 / 3.0;
        out[0] = v[0];
        for (int k = 0; k < 3; ++k) out[1 + k] = -2.0 * v[2 + k];
        out[4] = v[1] + 2.0 * v[8];
        out[5] = 4.0 * v[9];
        out[6] = 4.0 * v[10];
        out[7] = v[1] + 2.0 * v[11];
        out[8] = 4.0 * v[12];
        out[9] = v[1] + 2.0 * v[13];
        // -2 s^2 (f2 x . s) - 4/3 (f3 xxx . sss)
        out[10] = fma(k3, v[14], -2.0 * v[5]);
        out[11] = fma(-4.0, v[15], -2.0 * v[6]);
        out[12] = fma(-4.0, v[16], -2.0 * v[7]);
        out[13] = fma(-4.0, v[17], -2.0 * v[5]);
        out[14] = -8.0 * v[18];
        out[15] = fma(-4.0, v[19], -2.0 * v[5]);
        out[16] = fma(k3, v[20], -2.0 * v[6]);
        out[17] = fma(-4.0, v[21], -2.0 * v[7]);
        out[18] = fma(-4.0, v[22], -2.0 * v[6]);
        out[19] = fma(k3, v[23], -2.0 * v[7]);
    }
}

constexpr int kSumWarps = 4;         // regions per CTA
constexpr int kSumChunk = 2048;      // regions whose roles run one after another

// One warp sums one group of columns (blockIdx-derived role; the last one is
// the FP64 polynomial) of one region.  All CTAs in flight run the same role,
// but for the change-overs: seven roles side by side in a CTA, 40 KB of
// unrolled code between them, spent most of their time waiting for
// instructions (3.8 ms for the 28,800 regions of the 60^3 x 64 layered field).
// A chunk's entries stay in L2 from role to role.
__global__ void __launch_bounds__(32 * kSumWarps, 4) taylor_sums_kernel(SumArgs s) {
    const int lane = threadIdx.x & 31;
    constexpr int per_role = kSumChunk / kSumWarps, per_chunk = per_role * (kTaylorRoles + 1);
    const int chunk = blockIdx.x / per_chunk, rest = blockIdx.x % per_chunk;
    const int role = rest / per_role;
    const int region = chunk * kSumChunk + rest % per_role * kSumWarps + (threadIdx.x >> 5);
    if (region >= s.n_regions) return;
    const RegionInfo &r = s.regs[region];
    const long long first = r.off + r.n_near + r.n_mid;
    const int n = r.n_inner - r.n_mid + (s.symmetric ? r.n_shella : 0);
    const int n_full = s.far ? r.n_tnear : n;
    const float4 *hi = s.hi + first;
    float *out = s.sums + (size_t)region * kTaylorPad;
    switch (role) {
    case 0: role_sum<0>(s, hi, n_full, n, lane, region, out); break;
    case 1: role_sum<1>(s, hi, n_full, n, lane, region, out); break;
    case 2: role_sum<2>(s, hi, n_full, n, lane, region, out); break;
    case 3: role_sum<3>(s, hi, n_full, n, lane, region, out); break;
    case 4: role_sum<4>(s, hi, n_full, n, lane, region, out); break;
    case 5: role_sum<5>(s, hi, n_full, n, lane, region, out); break;
    default:
        if (lane < kTaylorPad - kTaylorSums) {
            if (s.split) mma_store_split<kMmaN>(s.sums, region, lane, 0.f);
            else out[kTaylorSums + lane] = 0.f;
        }
        poly_sum(s, hi, s.lo + first, s.rest ? r.n_mid : 0, n, lane,
                 s.poly + (size_t)region * kTaylorPolyPad);
    }
}

// ---------------------------------------------------------------- matrix

struct SumIndex {   // sum -> (l, k, m, 0 cosine / 1 sine)
    uchar4 at[kTaylorSums];
};

static const SumIndex &sum_index() {
    static const SumIndex index = [] {
        SumIndex x{};
        for (int r = 0; r < kTaylorRoles; ++r) {
            int base = role_start(r);
            for (int c = 0; c < 3; ++c) {
                const int m = role_column(r, c);
                if (m < 0) continue;
                for (int l = m; l <= kTaylorOrder; ++l)
                    for (int k = 0; l + 2 * k <= kTaylorOrder; ++k) {
                        if (l + 2 * k < kTaylorLow) continue;
                        const int at = base + column_pos(m, l, k) * (m ? 2 : 1);
                        for (int cs = 0; cs < (m ? 2 : 1); ++cs)
                            x.at[at + cs] = make_uchar4(l, k, m, cs);
                    }
                base += column_sums(m);
            }
        }
        return x;
    }();
    return index;
}

struct MatrixArgs {
    Mat3 H;
    int S, bi, bj, bk;       // grid size, block shape
    int poses, rows;         // poses of a region, padded row length
    const double *axes;
    double off0, off1, inv_r;
    int outs;                // 1 (energy) or 7; sites: 1 or 4
    const double *sites;     // [poses][3]: single sites instead of poses
    float *matrix;
};

// Value and gradient of |s|^{2k} Q_lm(s) {C_m, S_m}(s).
__device__ __forceinline__ void solid_term(int l, int k, int m, int cs, double x, double y,
                                           double z, double &val, double (&g)[3]) {
    const double r2 = x * x + y * y + z * z;
    // q, dq/dz at fixed r^2, dq/d(r^2)
    double q1 = 1.0, q1z = 0.0, q1r = 0.0, q0 = 0.0, q0z = 0.0, q0r = 0.0;
    for (int i = 2; i <= m; ++i) q1 *= sqrt((2.0 * i - 1.0) / (2.0 * i));
    for (int i = m + 1; i <= l; ++i) {
        const double nrm = 1.0 / sqrt((double)(i * i - m * m));
        const double f = (2.0 * i - 1.0) * nrm,
                     h = i > m + 1 ? sqrt((double)((i - 1) * (i - 1) - m * m)) * nrm : 0.0;
        const double q = f * z * q1 - h * r2 * q0;
        const double qz = f * (q1 + z * q1z) - h * r2 * q0z;
        const double qr = f * z * q1r - h * (q0 + r2 * q0r);
        q0 = q1;
        q0z = q1z;
        q0r = q1r;
        q1 = q;
        q1z = qz;
        q1r = qr;
    }
    double c = 1.0, s = 0.0, cp = 0.0, sp = 0.0;   // (x + iy)^m and ^(m - 1)
    for (int i = 0; i < m; ++i) {
        cp = c;
        sp = s;
        c = x * cp - y * sp;
        s = x * sp + y * cp;
    }
    const double t = cs ? s : c, tx = m * (cs ? sp : cp), ty = m * (cs ? cp : -sp);
    double p = 1.0, pr = 0.0;   // r2^k and its derivative
    for (int i = 0; i < k; ++i) {
        pr = pr * r2 + p;
        p *= r2;
    }
    val = p * q1 * t;
    const double rad = 2.0 * (pr * q1 + p * q1r) * t;
    g[0] = rad * x + p * q1 * tx;
    g[1] = rad * y + p * q1 * ty;
    g[2] = rad * z + p * q1z * t;
}

__global__ void __launch_bounds__(128) taylor_matrix_kernel(MatrixArgs a, SumIndex index) {
    const int pose = blockIdx.x * blockDim.x + threadIdx.x;
    if (pose >= a.poses) return;
    const uchar4 w = index.at[blockIdx.y];
    float *row = a.matrix + (size_t)blockIdx.y * a.rows;
    if (a.sites) {   // the other operand of taylor_mma_kernel
        double v, g[3];
        const double *p = a.sites + 3 * pose;
        solid_term(w.x, w.y, w.z, w.w, p[0] * a.inv_r, p[1] * a.inv_r, p[2] * a.inv_r, v, g);
        const int k = kMmaOrder.at[blockIdx.y];
        mma_store_split<kMmaM>(a.matrix, pose * a.outs, k, (float)v);
        for (int d = 0; d < 3 && a.outs == 4; ++d)
            mma_store_split<kMmaM>(a.matrix, pose * 4 + 1 + d, k, (float)(g[d] * a.inv_r));
        return;
    }
    const int cb = a.bi * a.bj * a.bk, o = pose / cb, c = pose % cb;
    const int ck = c % a.bk, cj = (c / a.bk) % a.bj, ci = c / (a.bk * a.bj);
    double cx, cy, cz;
    frac_to_cart(a.H, (ci + 0.5 - 0.5 * a.bi) / a.S, (cj + 0.5 - 0.5 * a.bj) / a.S,
                 (ck + 0.5 - 0.5 * a.bk) / a.S, cx, cy, cz);
    const double u[3] = {a.axes[3 * o], a.axes[3 * o + 1], a.axes[3 * o + 2]};
    double out[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int s = 0; s < 2; ++s) {
        const double off = s ? a.off1 : a.off0;
        double v, g[3];
        solid_term(w.x, w.y, w.z, w.w, (cx + off * u[0]) * a.inv_r, (cy + off * u[1]) * a.inv_r,
                   (cz + off * u[2]) * a.inv_r, v, g);
        out[0] += v;
        for (int k = 0; k < 3; ++k) {
            out[1 + k] += g[k] * a.inv_r;
            out[4 + k] += off * g[k] * a.inv_r;
        }
    }
    if (a.outs == 1) {
        row[pose] = (float)out[0];
        return;
    }
    const double wu = out[4] * u[0] + out[5] * u[1] + out[6] * u[2];
    for (int k = 0; k < 3; ++k) out[4 + k] -= wu * u[k];
    for (int k = 0; k < 7; ++k) row[(pose >> 1) * 14 + 2 * k + (pose & 1)] = (float)out[k];
}

// ---------------------------------------------------------------- evaluation

struct EvalArgs {
    const float *matrix;     // [kTaylorPad][rows]
    const float *sums;       // [n_regions][kTaylorPad]
    int rows, tiles;         // padded row length, tiles of rows
    int poses, n_regions;
    const RegionInfo *regs;
    int S, O, bi, bj, bk;
    float *const *e32;       // device words holding the output pointers
    float *const *g32;
    double *e64;
};

constexpr int kEvalK = 16;
// rows per thread
__host__ __device__ constexpr int eval_rows(int outs) { return outs == 1 ? 16 : 14; }
__host__ __device__ constexpr int eval_tile(int outs) { return 16 * eval_rows(outs); }

// Tile: eval_tile rows (32 poses x 7 outputs, or 256 poses) x NT / 16 CT
// regions; a thread holds 14 or 16 rows (packed in pairs: two poses) x CT
// regions.  Bound by the FMA pipe.  28,800 regions: energy and gradient
// 1.99 ms as 128 threads x 8 regions (256 x 4: 2.12; 6 regions at 3 CTAs/SM:
// 2.09; unpacked FMA: 2.07); 14,400 regions of 16 centers, energy alone: 0.46
// ms as 256 x 4 (128 x 8: 0.53).
template <int OUTS, int NT, int CT>
__global__ void __launch_bounds__(NT, 2) taylor_eval_kernel(EvalArgs a) {
    constexpr int RT = eval_rows(OUTS), RP = RT / 2, TILE = eval_tile(OUTS);
    constexpr int COLS = NT / 16 * CT;   // regions per tile
    __shared__ __align__(16) float ms[2][kEvalK][TILE];
    __shared__ __align__(16) float2 ss[2][kEvalK][COLS];
    // warps 4 (rows) x NT / 128 (regions), lanes 4 x 8: one wavefront per
    // shared-memory load
    const int tid = threadIdx.x, rg = (tid >> 5 & 3) * 4 + (tid >> 3 & 3),
              cg = (tid >> 7) * 8 + (tid & 7);
    // one grid dimension for both: 65,535 region tiles would be 4.2 M regions
    const int row0 = (int)(blockIdx.x % a.tiles) * TILE,
              reg0 = (int)(blockIdx.x / a.tiles) * COLS;
    float2 acc[RP][CT];
#pragma unroll
    for (int i = 0; i < RP; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) acc[i][j] = make_float2(0.f, 0.f);
    constexpr int SV = COLS * kEvalK / 4, SL = (SV + NT - 1) / NT;   // float4 of sums, per thread
    float4 hold[SL];
    auto load_m = [&](int buf, int k0) {
#pragma unroll
        for (int i = 0; i < (kEvalK * TILE / 4 + NT - 1) / NT; ++i) {
            const int v = tid + i * NT, k = v / (TILE / 4), c = v % (TILE / 4) * 4;
            if (k >= kEvalK) break;
            const uint32_t dst = smem_addr(&ms[buf][k][c]);
            const float *src = a.matrix + (size_t)(k0 + k) * a.rows + row0 + c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
        }
        asm volatile("cp.async.commit_group;");
    };
    auto load_s = [&](int k0) {
#pragma unroll
        for (int i = 0; i < SL; ++i) {
            const int v = min(tid + i * NT, SV - 1);
            const int r = min(reg0 + (v >> 2), a.n_regions - 1);
            hold[i] = *reinterpret_cast<const float4 *>(a.sums + (size_t)r * kTaylorPad + k0 +
                                                        (v & 3) * 4);
        }
    };
    auto store_s = [&](int buf) {
#pragma unroll
        for (int i = 0; i < SL; ++i) {
            const int v = tid + i * NT, c = v >> 2, k = (v & 3) * 4;
            if (v >= SV) break;
            ss[buf][k][c] = make_float2(hold[i].x, hold[i].x);
            ss[buf][k + 1][c] = make_float2(hold[i].y, hold[i].y);
            ss[buf][k + 2][c] = make_float2(hold[i].z, hold[i].z);
            ss[buf][k + 3][c] = make_float2(hold[i].w, hold[i].w);
        }
    };
    // one k of operands ahead of the FMAs that use them
    float2 m[2][RP], v[2][CT];
    auto fetch = [&](int buf, int k, float2 (&mk)[RP], float2 (&vk)[CT]) {
#pragma unroll
        for (int i = 0; i < RP; ++i)
            mk[i] = *reinterpret_cast<const float2 *>(&ms[buf][k][rg * RT + 2 * i]);
#pragma unroll
        for (int j = 0; j < CT / 2; ++j) {
            const float4 q =
                *reinterpret_cast<const float4 *>(&ss[buf][k][NT / 8 * j + 2 * cg]);
            vk[2 * j] = make_float2(q.x, q.y);
            vk[2 * j + 1] = make_float2(q.z, q.w);
        }
    };
    load_m(0, 0);
    load_s(0);
    store_s(0);
    for (int k0 = 0, buf = 0; k0 < kTaylorPad; k0 += kEvalK, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;");
        __syncthreads();
        const bool more = k0 + kEvalK < kTaylorPad;
        if (more) {
            load_m(buf ^ 1, k0 + kEvalK);
            load_s(k0 + kEvalK);
        }
        fetch(buf, 0, m[0], v[0]);
#pragma unroll
        for (int k = 0; k < kEvalK; ++k) {
            if (k + 1 < kEvalK) fetch(buf, k + 1, m[(k + 1) & 1], v[(k + 1) & 1]);
#pragma unroll
            for (int i = 0; i < RP; ++i)
#pragma unroll
                for (int j = 0; j < CT; ++j)
                    acc[i][j] = __ffma2_rn(m[k & 1][i], v[k & 1][j], acc[i][j]);
        }
        if (more) store_s(buf ^ 1);
    }
    const int cb = a.bi * a.bj * a.bk;
    const long long S3 = (long long)a.S * a.S * a.S;
    float *e32 = a.e32 ? *a.e32 : nullptr, *g32 = OUTS == 7 ? *a.g32 : nullptr;
#pragma unroll
    for (int j = 0; j < CT; ++j) {
        const int reg = reg0 + NT / 8 * (j >> 1) + 2 * cg + (j & 1);
        if (reg >= a.n_regions) continue;
        const RegionInfo &r = a.regs[reg];
        const int i0 = r.i0, j0 = r.j0, kk0 = r.k0;
        auto place = [&](int pose, long long &idx) {
            if (pose >= a.poses) return false;
            const int o = pose / cb, c = pose % cb;
            const int gk = kk0 + c % a.bk, gj = j0 + (c / a.bk) % a.bj,
                      gi = i0 + c / (a.bk * a.bj);
            if (gi >= a.S || gj >= a.S || gk >= a.S) return false;
            idx = o * S3 + ((long long)gi * a.S + gj) * a.S + gk;
            return true;
        };
        if constexpr (OUTS == 1) {
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                long long idx;
                if (!place(row0 + rg * RT + i, idx)) continue;
                const float v = i & 1 ? acc[i / 2][j].y : acc[i / 2][j].x;
                if (a.e64) a.e64[idx] = (double)v;
                else e32[idx] = v;
            }
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                long long idx;
                if (!place((row0 / 14 + rg) * 2 + h, idx)) continue;
                auto get = [&](int i) { return h ? acc[i][j].y : acc[i][j].x; };
                e32[idx] = get(0);
                float2 *g = reinterpret_cast<float2 *>(g32 + 6 * idx);
                g[0] = make_float2(get(1), get(2));
                g[1] = make_float2(get(3), get(4));
                g[2] = make_float2(get(5), get(6));
            }
        }
    }
}

// ---------------------------------------------------------------- host side

// Truncation error in K/A of one pair at distance d, sites within `radius`
// (the gradient of the omitted degrees towards the entry, where all the
// Gegenbauer polynomials add up).
static double truncation(double c12, double c6, double radius, double d, int order) {
    const double ratio = radius / d;
    const double p6 = std::pow(d, -6.0);
    double g6 = 1.0, g3 = 1.0, t = 1.0, sum = 0.0;   // C_n^6(1), C_n^3(1), ratio^n
    for (int n = 1; n <= order + 30; ++n) {
        g6 *= (n + 11.0) / n;
        g3 *= (n + 5.0) / n;
        t *= ratio;
        if (n > order) sum += std::fabs(c12 * p6 * p6 * g6 - c6 * p6 * g3) * t * n / radius;
    }
    return sum;
}

// Allowed truncation error of a pair at d_T.  It falls as d^-20 and faster,
// so few entries come near it; the FP32 sums it replaces are off by 1e-6
// K/A and more.
constexpr double kTruncation = 3e-6;

static double worst_truncation(const System &sys, double radius, double d,
                               int order = kTaylorOrder) {
    double worst = 0.0;
    for (int t = 0; t < sys.n_types; ++t)
        worst = std::max(worst, truncation(sys.h_td[4 * t], sys.h_td[4 * t + 1], radius, d, order));
    return worst;
}

double taylor_start(const System &sys, double radius, int order) {
    double lo = 2.0 * radius, hi = sys.cutoff;
    if (!(lo < hi) || worst_truncation(sys, radius, hi, order) > kTruncation) return 1e30;
    for (int i = 0; i < 24; ++i) {
        const double mid = 0.5 * (lo + hi);
        (worst_truncation(sys, radius, mid, order) > kTruncation ? lo : hi) = mid;
    }
    return hi;
}

bool taylor_allowed(const System &sys, const RegionSet &rs) {
    if (!(rs.d_taylor < sys.cutoff) || rs.n_regions < 1) return false;
    // another guest of the same framework on shared lists: its own bound
    return worst_truncation(sys, rs.taylor_radius, rs.d_taylor) <= 1.05 * kTruncation &&
           (rs.d_tfar >= sys.cutoff ||
            worst_truncation(sys, rs.taylor_radius, rs.d_tfar, kTaylorFarOrder) <=
                1.05 * kTruncation);
}

// Bytes of the evaluation matrix beyond which a field does without expansions:
// 10,700 directors on 8-center regions, forward + adjoint.  It grows with the
// directors alone (2 M directors on a 4^3 grid: 190 GB).
constexpr double kTaylorMatrix = 1 << 30;

bool taylor_pays(double n, double poses, bool adjoint) {
    if (poses * (adjoint ? 7.0 : 1.0) * kTaylorPad * sizeof(float) > kTaylorMatrix) return false;
    const double direct = n * poses * 2.0 * (adjoint ? 19.0 : 9.3);
    const double taylor = n * 2100.0 + poses * (adjoint ? 7.0 : 1.0) * 580.0;
    return direct > taylor;
}

bool taylor_worthwhile(const System &sys, const RegionSet &rs, int n_axes, bool adjoint) {
    return taylor_allowed(sys, rs) &&
           taylor_pays((double)rs.n_taylor / rs.n_regions,
                       (double)n_axes * rs.bi * rs.bj * rs.bk, adjoint);
}

static int prepare(const System &sys, const RegionSet &rs, int poses, const double *d_axes,
                   const double *d_sites, int outs, TaylorPlan &plan, cudaStream_t stream) {
    const int rows_used = d_sites || outs == 1 ? poses * outs : (poses + 1) / 2 * 14;
    const int tile = d_sites ? kMmaM : eval_tile(outs);
    const int rows = (rows_used + tile - 1) / tile * tile;
    const size_t words = (size_t)kTaylorPad * rows * (d_sites ? 2 : 1);
    VEXT_TRY(ensure_capacity(plan.matrix, plan.matrix_cap, words));
    VEXT_TRY(ensure_capacity(plan.poly, plan.poly_cap, (size_t)rs.n_regions * kTaylorPolyPad));
    plan.rows = rows;
    plan.outs = outs;
    VEXT_CUDA(cudaMemsetAsync(plan.matrix, 0, sizeof(float) * words, stream));
    MatrixArgs a;
    a.H = sys.H;
    a.S = rs.size;
    a.bi = rs.bi;
    a.bj = rs.bj;
    a.bk = rs.bk;
    a.poses = poses;
    a.rows = rows;
    a.axes = d_axes;
    a.off0 = sys.offsets[0];
    a.off1 = sys.offsets[1];
    a.inv_r = 1.0 / rs.taylor_radius;
    a.outs = outs;
    a.sites = d_sites;
    a.matrix = plan.matrix;
    taylor_matrix_kernel<<<dim3((poses + 127) / 128, kTaylorSums), 128, 0, stream>>>(a,
                                                                                   sum_index());
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

int taylor_prepare(const System &sys, const RegionSet &rs, int n_axes, const double *d_axes,
                   bool adjoint, TaylorPlan &plan, cudaStream_t stream) {
    return prepare(sys, rs, n_axes * rs.bi * rs.bj * rs.bk, d_axes, nullptr, adjoint ? 7 : 1, plan,
                   stream);
}

int taylor_prepare_sites(const System &sys, const RegionSet &rs, int n_sites,
                         const double *d_sites, bool adjoint, TaylorPlan &plan,
                         cudaStream_t stream) {
    return prepare(sys, rs, n_sites, nullptr, d_sites, adjoint ? 4 : 1, plan, stream);
}

static int sum_expansions(const System &sys, const RegionSet &rs, const TaylorPlan &plan,
                          bool symmetric, bool split, float *sums, cudaStream_t stream) {
    SumArgs s;
    s.regs = rs.d_info;
    s.n_regions = rs.n_regions;
    s.hi = rs.d_hi;
    s.lo = rs.d_lo;
    s.tf = sys.d_tf;
    s.td = sys.d_td;
    s.inv_r = (float)(1.0 / rs.taylor_radius);
    s.symmetric = symmetric;
    s.rest = !rs.sites;   // (site lists: clusters take some of them in FP64)
    s.far = rs.d_tfar < sys.cutoff - rs.taylor_radius;   // the inner entries' bound
    s.sums = sums;
    s.split = split;
    s.poly = plan.poly;
    const int chunks = (rs.n_regions + kSumChunk - 1) / kSumChunk;
    taylor_sums_kernel<<<chunks * (kSumChunk / kSumWarps) * (kTaylorRoles + 1), 32 * kSumWarps, 0,
                         stream>>>(s);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

int taylor_enqueue(const System &sys, const RegionSet &rs, int n_axes, const TaylorPlan &plan,
                   bool symmetric, float *sums, float *const *e32, double *e64,
                   float *const *g32, cudaStream_t stream) {
    VEXT_TRY(sum_expansions(sys, rs, plan, symmetric, false, sums, stream));
    EvalArgs a;
    a.matrix = plan.matrix;
    a.sums = sums;
    a.rows = plan.rows;
    a.poses = n_axes * rs.bi * rs.bj * rs.bk;
    a.n_regions = rs.n_regions;
    a.regs = rs.d_info;
    a.S = rs.size;
    a.O = n_axes;
    a.bi = rs.bi;
    a.bj = rs.bj;
    a.bk = rs.bk;
    a.e32 = e32;
    a.g32 = g32;
    a.e64 = e64;
    a.tiles = plan.rows / eval_tile(plan.outs);
    const unsigned blocks = (unsigned)a.tiles * ((rs.n_regions + 63) / 64);
    if (plan.outs == 7)
        taylor_eval_kernel<7, 128, 8><<<blocks, 128, 0, stream>>>(a);
    else
        taylor_eval_kernel<1, 256, 4><<<blocks, 256, 0, stream>>>(a);
    VEXT_CUDA(cudaGetLastError());
    return 0;
}

int taylor_enqueue_sites(const System &sys, const RegionSet &rs, int n_sites,
                         const TaylorPlan &plan, float *sums, float *out, int *status,
                         cudaStream_t stream) {
    VEXT_TRY(sum_expansions(sys, rs, plan, true, true, sums, stream));
    return taylor_mma(plan.matrix, plan.rows / kMmaM, sums, rs.n_regions, n_sites * plan.outs, out,
                      status, stream);
}

}  // namespace vext
