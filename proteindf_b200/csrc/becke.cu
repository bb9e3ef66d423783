// Becke partition weights on the device (K7).
//
// For point r owned by atom A (DfGenerateGrid::calcMultiCenterWeight_Becke,
// src/libpdf/DfGenerateGrid.cpp:1811-1876, Ps_uij :2043-2086):
//   P_m(r) = prod_{n != m} s(nu_mn),  s(nu) = (1 - f(f(f(nu)))) / 2,  f(x) = x (3 - x^2) / 2
//   mu_mn  = (|r - R_m| - |r - R_n|) / |R_m - R_n|
//   nu_mn  = mu_mn + a_mn (1 - mu_mn^2), a = u / (u^2 - 1), u = (R_m - R_n)/(R_m + R_n),
//            a clamped to [-1/2, 1/2] (atomic size adjustment, Becke radii)
//   w(r)   = w_single(r) * P_A(r) / sum_m P_m(r).
// Partner atoms n with atomic number <= 0 (dummy atoms, `ghost`) are left out of
// every product, as Ps_uij does (:2056); a dummy atom m still has its own P_m.
// One thread per point; the atoms (coordinates and radius) are staged in
// shared memory once per CTA. All arithmetic is FP64, and this file is compiled
// without fused multiply-adds, so that every operation rounds once in the order
// written: the weights then equal the CPU restatement's (plain IEEE operations in
// the same order) bit for bit, and the weight screen keeps the same points.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "pdfxc_internal.cuh"

namespace pdfxc {

namespace {

__device__ __forceinline__ double becke_s(double nu) {
#pragma unroll
    for (int k = 0; k < 3; ++k) nu = 0.5 * nu * (3.0 - nu * nu);
    return 0.5 * (1.0 - nu);
}

__global__ void __launch_bounds__(128) k_becke(const double* __restrict__ atom_xyz, const double* __restrict__ brad,
                                               const int* __restrict__ ghost, int natom, int size_adjust,
                                               int64_t npts, const double* __restrict__ xyz,
                                               const int* __restrict__ owner, const double* __restrict__ w_single,
                                               double* __restrict__ w_out) {
    extern __shared__ double4 atoms[];  // x, y, z, radius (negative: a dummy partner, left out)
    for (int a = threadIdx.x; a < natom; a += blockDim.x)
        atoms[a] = make_double4(atom_xyz[3 * a], atom_xyz[3 * a + 1], atom_xyz[3 * a + 2],
                                ghost && ghost[a] ? -1.0 : brad[a]);
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npts; i += (int64_t)gridDim.x * blockDim.x) {
        const double rx = xyz[3 * i], ry = xyz[3 * i + 1], rz = xyz[3 * i + 2];
        const int own = owner[i];
        double tot = 0.0, pown = 0.0;
        for (int m = 0; m < natom; ++m) {
            const double4 A = atoms[m];
            const double rm = sqrt((rx - A.x) * (rx - A.x) + (ry - A.y) * (ry - A.y) + (rz - A.z) * (rz - A.z));
            double p = 1.0;
            for (int n = 0; n < natom && p != 0.0; ++n) {
                if (n == m) continue;
                const double4 B = atoms[n];
                if (B.w < 0.0) continue;
                const double Am = A.w < 0.0 ? brad[m] : A.w;
                const double rn = sqrt((rx - B.x) * (rx - B.x) + (ry - B.y) * (ry - B.y) + (rz - B.z) * (rz - B.z));
                const double Rmn = sqrt((A.x - B.x) * (A.x - B.x) + (A.y - B.y) * (A.y - B.y) + (A.z - B.z) * (A.z - B.z));
                double u = (rm - rn) * (1.0 / Rmn);
                if (size_adjust) {
                    const double au = (Am - B.w) / (Am + B.w);
                    double a = au / (au * au - 1.0);
                    a = a < -0.5 ? -0.5 : (a > 0.5 ? 0.5 : a);
                    u = u + a * (1.0 - u * u);
                }
                p *= becke_s(u);
            }
            tot += p;
            if (m == own) pown = p;
        }
        w_out[i] = w_single[i] * (pown / tot);
    }
}

// Pair constants of atoms m and n: inv = 1/|R_m - R_n|, adj = a_mn (0 without size adjustment).
// A dummy partner n (ghost[n] != 0) gets inv = 0 and adj = -1: then nu = -1 and its factor
// s = (1 - f3(-1)) / 2 is exactly 1 (f(-1) = -1 in IEEE arithmetic), the same as leaving it out.
__device__ __forceinline__ void becke_pair(const double* __restrict__ atom_xyz, const double* __restrict__ brad,
                                           const int* __restrict__ ghost, int size_adjust, int m, int n, double& inv,
                                           double& adj) {
    inv = adj = 0.0;
    if (m == n) return;
    if (ghost && ghost[n]) {
        adj = -1.0;
        return;
    }
    const double dx = atom_xyz[3 * m] - atom_xyz[3 * n], dy = atom_xyz[3 * m + 1] - atom_xyz[3 * n + 1],
                 dz = atom_xyz[3 * m + 2] - atom_xyz[3 * n + 2];
    inv = 1.0 / sqrt(dx * dx + dy * dy + dz * dz);
    if (size_adjust) {
        const double au = (brad[m] - brad[n]) / (brad[m] + brad[n]);
        const double a = au / (au * au - 1.0);
        adj = a < -0.5 ? -0.5 : (a > 0.5 ? 0.5 : a);
    }
}

// The pair table: inv[m*n_atom + n], adj[m*n_atom + n].
__global__ void k_becke_pairs(const double* __restrict__ atom_xyz, const double* __restrict__ brad,
                              const int* __restrict__ ghost, int natom, int size_adjust, double* inv, double* adj) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < natom * natom; e += gridDim.x * blockDim.x)
        becke_pair(atom_xyz, brad, ghost, size_adjust, e / natom, e % natom, inv[e], adj[e]);
}

// The tables of k_becke_near, one CTA per atom m: (inv, adj) of its row in FP64 and in FP32, whether
// any of them is not finite (two atoms in one place, radii of zero), and its kNearList nearest atoms by
// distance, itself first (ties by index), or all of them where there are no more.
constexpr int kNearList = 16;
__global__ void __launch_bounds__(128) k_becke_near_tables(const double* __restrict__ atom_xyz,
                                                           const double* __restrict__ brad,
                                                           const int* __restrict__ ghost, int natom, int size_adjust,
                                                           double2* __restrict__ pair, float2* __restrict__ pairf,
                                                           int* __restrict__ near, int* __restrict__ odd) {
    extern __shared__ double nd[];  // [natom] squared distance to m
    __shared__ double bd[128];
    __shared__ int bi[128];
    const int m = blockIdx.x, t = threadIdx.x;
    bool wild = false;
    for (int n = t; n < natom; n += blockDim.x) {
        double inv, adj;
        becke_pair(atom_xyz, brad, ghost, size_adjust, m, n, inv, adj);
        pair[(size_t)m * natom + n] = make_double2(inv, adj);
        pairf[(size_t)m * natom + n] = make_float2((float)inv, (float)adj);
        wild = wild || !isfinite((float)inv) || !isfinite((float)adj);
        const double dx = atom_xyz[3 * m] - atom_xyz[3 * n], dy = atom_xyz[3 * m + 1] - atom_xyz[3 * n + 1],
                     dz = atom_xyz[3 * m + 2] - atom_xyz[3 * n + 2];
        nd[n] = n == m ? -1.0 : dx * dx + dy * dy + dz * dz;
    }
    wild = __syncthreads_or(wild);
    if (t == 0) odd[m] = wild ? 1 : 0;
    if (natom <= kNearList) {  // every atom: ranking them costs more (16 atoms, 2,000 points: call 109 -> 93 us)
        if (t < natom) near[m * kNearList + t] = t;
        return;
    }
    for (int k = 0; k < kNearList; ++k) {
        __syncthreads();
        double d = 1e300;
        int b = natom;
        for (int n = t; n < natom; n += blockDim.x)
            if (nd[n] < d) d = nd[n], b = n;
        bd[t] = d, bi[t] = b;
        __syncthreads();
        for (int s = 64; s > 0; s >>= 1) {
            if (t < s && (bd[t + s] < bd[t] || (bd[t + s] == bd[t] && bi[t + s] < bi[t])))
                bd[t] = bd[t + s], bi[t] = bi[t + s];
            __syncthreads();
        }
        if (t == 0) {
            const int w = bi[0] < natom ? bi[0] : m;  // only NaN coordinates leave none
            near[m * kNearList + k] = w;
            nd[w] = 1e301;
        }
    }
}

// The weights of k_becke at a fraction of its work, bit for bit the same. Far from most atoms m the
// product P_m is so small against sum_m P_m that its exact value cannot change any rounding of the
// sum. A CTA takes 32 points:
//   1. the distances |r - R_n| (FP64, and an FP32 copy), each point's nearest atom c and an FP32
//      estimate of P_c;
//   2. the filter, a warp per m with a lane per point: an FP32 upper bound of P_m from the factors of
//      c's nearest atoms alone (every factor is at most 1 and carries a margin for the FP32 rounding);
//      m is dropped when the bound falls below `share` = 2^-80 of P_c. Nothing is dropped where a pair constant of
//      the molecule is not finite: P_m may then be a NaN, which the sum has to show;
//   3. P_m of the kept (m, point) pairs (about 10 of 100 atoms), packed over the CTA's threads in the
//      order of m, with the operations and the order of k_becke;
//   4. per point the sum over m in ascending order, twice: with every dropped P_m at its lower and at
//      its upper bound. FP64 addition is monotone, so when both sums agree to the bit they are the sum
//      of all P_m; when they do not (a rounding boundary inside the interval, n_dropped 2^-78 P_c wide:
//      2^-71.5 with 90 atoms dropped, 2^-69 with 470) the point is summed over all atoms.
// Bound by the issue of the FP32 filter and the FP64 pipe in step 3. Seeded chains on USER 75 x 302
// grids, ncu (this form / one point per thread up to 48 atoms, a warp per point above): 30 atoms 0.56 /
// 0.94 ms, 43 atoms 1.14 / 3.58, 100 atoms 8.7 / 39.
constexpr int kNearPts = 32, kNearCap = 1024;

// P_m at the point whose distances are r[n * kNearPts]: the factors in ascending partner order, up
// to a product of zero. Four factors are formed ahead of the products.
__device__ __forceinline__ double becke_product(const double* r, const double2* __restrict__ pm, int m, int natom) {
    const double rm = r[m * kNearPts];
    auto factor = [&](int n) {
        const double2 c = __ldg(pm + n);
        double u = (rm - r[n * kNearPts]) * c.x;
        u = u + c.y * (1.0 - u * u);
        return becke_s(u);
    };
    double p = 1.0;
    int n = 0;
    for (; n + 4 <= natom && p != 0.0; n += 4) {
        double s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] = n + k == m ? 1.0 : factor(n + k);
        const double q = (((p * s[0]) * s[1]) * s[2]) * s[3];
        if (fabs(q) > 0.0) {
            p = q;
        } else {  // a zero (or a NaN that may follow one): factor by factor, up to the zero
            for (int k = 0; k < 4 && p != 0.0; ++k) p *= s[k];
        }
    }
    for (; n < natom && p != 0.0; ++n)
        if (n != m) p *= factor(n);
    return p;
}

// FP32 factor s(nu_mn) and a bound of its rounding error: |d mu| <= 1.8e-7 (r_m + r_n) / R_mn, at most
// 3.4 times that in s, and 1e-6 for the polynomial. That holds while mu stays near [-1, 1]: from a margin of
// 0.25 on the polynomial may be anything. max(s, 0) + margin still bounds the factor from above there (up
// to a margin of 1 the cubics map what lies beyond 1 back into [-1, 1], and above it the sum is past 1); s
// alone says nothing.
__device__ __forceinline__ float becke_s32(float rm, float rn, float2 c, float& margin) {
    const float u = (rm - rn) * c.x;
    float nu = fmaf(c.y, fmaf(-u, u, 1.0f), u);
#pragma unroll
    for (int k = 0; k < 3; ++k) nu *= fmaf(-0.5f, nu * nu, 1.5f);
    margin = fmaf((rm + rn) * c.x, 8e-7f, 1e-6f);
    return fmaf(-0.5f, nu, 0.5f);
}

template <int kNearW>
__global__ void __launch_bounds__(32 * kNearW) k_becke_near(const double* __restrict__ atom_xyz, int natom,
                                                             const double2* __restrict__ pair,
                                                             const float2* __restrict__ pairf,
                                                             const int* __restrict__ near,
                                                             const int* __restrict__ odd, int64_t npts,
                                                             const double* __restrict__ xyz,
                                                             const int* __restrict__ owner,
                                                             const double* __restrict__ w_single,
                                                             double* __restrict__ w_out, float share) {
    extern __shared__ double sm[];
    double* rr = sm;                                               // [natom][32]: |r - R_n|
    double* pe = rr + (size_t)natom * kNearPts;                    // [kNearCap]: P_m of the kept pairs
    float* rf = reinterpret_cast<float*>(pe + kNearCap);           // [natom][32]: FP32 copy of rr
    uint32_t* mask = reinterpret_cast<uint32_t*>(rf + (size_t)natom * kNearPts);  // [natom]: points that keep m
    int* off = reinterpret_cast<int*>(mask + natom);               // [natom + 1]: pairs before m
    __shared__ float s_min[kNearW][kNearPts], s_prod[kNearW][kNearPts];
    __shared__ int s_arg[kNearW][kNearPts], s_c[kNearPts], s_end;
    constexpr unsigned kAll = 0xffffffffu;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int nlist = min(kNearList, natom);
    bool wild = false;
    for (int m = t; m < natom; m += 32 * kNearW) wild = wild || odd[m] != 0;
    const bool keep_all = __syncthreads_or(wild);
    for (int64_t i0 = blockIdx.x * (int64_t)kNearPts; i0 < npts; i0 += (int64_t)gridDim.x * kNearPts) {
        const int64_t i = i0 + lane;
        const bool live = i < npts;
        const int own = live ? owner[i] : -1;
        // 1. distances (lane = point), the nearest atom
        const double rx = live ? xyz[3 * i] : 0.0, ry = live ? xyz[3 * i + 1] : 0.0, rz = live ? xyz[3 * i + 2] : 0.0;
        float best = 3e38f;
        int arg = 0;
        for (int m = warp; m < natom; m += kNearW) {
            const double ax = atom_xyz[3 * m] - rx, ay = atom_xyz[3 * m + 1] - ry, az = atom_xyz[3 * m + 2] - rz;
            const double d = sqrt(ax * ax + ay * ay + az * az);
            rr[m * kNearPts + lane] = d;
            rf[m * kNearPts + lane] = (float)d;
            if ((float)d < best) best = (float)d, arg = m;
        }
        s_min[warp][lane] = best, s_arg[warp][lane] = arg;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < kNearW; ++w)
                if (s_min[w][lane] < best) best = s_min[w][lane], arg = s_arg[w][lane];
            s_c[lane] = arg;
        }
        __syncthreads();
        const int c = s_c[lane];
        {  // P_c in FP32, its factors divided over the warps
            const float rc = rf[c * kNearPts + lane];
            float p = 1.0f;
            for (int n = warp; n < natom; n += kNearW) {
                float e;
                const float s = becke_s32(rc, rf[n * kNearPts + lane], __ldg(pairf + (size_t)c * natom + n), e);
                p *= n == c ? 1.0f : (e <= 0.25f ? s : 0.0f);
            }
            s_prod[warp][lane] = p;
        }
        __syncthreads();
        // the drop threshold: share P_c, and nothing dropped where P_c is near the end of the FP32 range or a
        // point is so far away that FP32 does not tell the distances apart (from 1e5 to 1e6 bohr on)
        float pc = 1.0f;
#pragma unroll
        for (int w = 0; w < kNearW; ++w) pc *= s_prod[w][lane];
        const float thr = pc > 1e-10f && !keep_all ? pc * share : 0.0f;
        // 2. the filter: c's nearest atoms and their distances in registers, four factors at a time
        int nn[kNearList];
        float rn[kNearList];
#pragma unroll
        for (int k = 0; k < kNearList; ++k) {
            nn[k] = __ldg(near + c * kNearList + min(k, nlist - 1));
            rn[k] = rf[nn[k] * kNearPts + lane];
        }
        for (int m = warp; m < natom; m += kNearW) {
            const float rm = rf[m * kNearPts + lane];
            const float2* pm = pairf + (size_t)m * natom;
            float p = 1.0f;
            bool drop = !live;
#pragma unroll
            for (int k0 = 0; k0 < kNearList; k0 += 4) {
                float2 pc4[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) pc4[k] = __ldg(pm + nn[k0 + k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float e;
                    const float s = becke_s32(rm, rn[k0 + k], pc4[k], e);
                    // (a list shorter than kNearList repeats its last atom: not a factor twice)
                    p *= nn[k0 + k] != m && k0 + k < nlist ? fmaxf(s, 0.0f) + e : 1.0f;
                }
                drop = drop || p < thr;
                if (__all_sync(kAll, drop)) break;
            }
            const unsigned keep = __ballot_sync(kAll, live && (!drop || m == own));
            if (lane == 0) mask[m] = keep;
        }
        __syncthreads();
        if (warp == 0) {  // pairs before each m
            int run = 0;
            for (int m0 = 0; m0 < natom; m0 += 32) {
                const int v = m0 + lane < natom ? __popc(mask[m0 + lane]) : 0;
                int x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kAll, x, o);
                    if (lane >= o) x += y;
                }
                if (m0 + lane < natom) off[m0 + lane] = run + x - v;
                run += __shfl_sync(kAll, x, 31);
            }
            if (lane == 0) off[natom] = run;
        }
        __syncthreads();
        // 3. and 4., in runs of whole atoms of at most kNearCap kept pairs
        const double bound = 2.0 * (double)thr;
        double lo = 0.0, hi = 0.0, pown = 0.0;
        for (int ms = 0; ms < natom;) {
            if (t == 0) {
                int me = natom;
                if (off[natom] - off[ms] > kNearCap) {  // the last atom end within the capacity
                    int a = ms + 1, b = natom;
                    while (b - a > 1) {
                        const int mid = (a + b) / 2;
                        if (off[mid] - off[ms] <= kNearCap) a = mid;
                        else b = mid;
                    }
                    me = a;
                }
                s_end = me;
            }
            __syncthreads();
            const int me = s_end, e0 = off[ms], ne = off[me] - e0;
            for (int e = t; e < ne; e += 32 * kNearW) {
                int a = ms, b = me;  // the atom of pair e0 + e: the last m with off[m] <= e0 + e
                while (b - a > 1) {
                    const int mid = (a + b) / 2;
                    if (off[mid] <= e0 + e) a = mid;
                    else b = mid;
                }
                unsigned bits = mask[a];
                for (int k = e0 + e - off[a]; k > 0; --k) bits &= bits - 1;
                pe[e] = becke_product(rr + __ffs(bits) - 1, pair + (size_t)a * natom, a, natom);
            }
            __syncthreads();
            if (warp == 0 && live) {
                for (int m = ms; m < me; ++m) {
                    const unsigned bits = mask[m];
                    if (bits >> lane & 1) {
                        const double p = pe[off[m] - e0 + __popc(bits & ((1u << lane) - 1))];
                        lo += p, hi += p;
                        if (m == own) pown = p;
                    } else {
                        lo -= bound, hi += bound;
                    }
                }
            }
            __syncthreads();
            ms = me;
        }
        if (warp == 0 && live) {
            if (!(lo == hi)) {
                lo = 0.0;
                for (int m = 0; m < natom; ++m) {
                    const double p = becke_product(rr + lane, pair + (size_t)m * natom, m, natom);
                    lo += p;
                    if (m == own) pown = p;
                }
            }
            w_out[i] = w_single[i] * (pown / lo);
        }
        __syncthreads();  // the shared rows are rewritten for the next points
    }
}

// Stratmann-Scuseria partition (DfGenerateGrid::calcMultiCenterWeight_SS,
// src/libpdf/DfGenerateGrid.cpp:1878-1956): s = (1 - g(mu))/2 with g the
// piecewise polynomial of a = 0.64, no size adjustment. s is exactly 0 for
// mu >= a and exactly 1 for mu <= -a (the polynomial is -1 / +1 at z = -1 / +1),
// which bounds the atoms that matter at a point (k_ss); 1/R_mn from the pair table.
__device__ __forceinline__ double ss_s(double u) {
    constexpr double a = 0.64;
    double g;
    if (u < -a) {
        g = -1.0;
    } else if (u > a) {
        g = 1.0;
    } else {
        const double z = u / a, z2 = z * z, z3 = z2 * z, z5 = z2 * z3;
        g = (1.0 / 16.0) * (35.0 * z - 35.0 * z3 + 21.0 * z5 - 5.0 * z5 * z2);
    }
    return 0.5 * (1.0 - g);
}

// One thread per point. For a point r owned by atom A at distance d, an atom m can have
// P_m = prod_n s(mu_mn) != 0 only if |A - m| < 2 d / (1 - a) (otherwise mu_mA >= a, s = 0), and
// a factor s(mu_mn) can differ from 1 only if |m - n| < 2 |r - m| / (1 - a) (otherwise
// mu_mn <= -a, s = 1): both bounds from |r - n| >= |m - n| - |r - m|, and s is exactly 0 / 1 at
// +-a. So the candidates m are A and A's neighbours up to 2 d / (1 - a), and the factors of P_m
// come from m's neighbours up to 2 |r - m| / (1 - a), each list sorted by distance; the
// skipped factors are exactly 1 and the skipped terms exactly 0. Points deep inside their
// owner's cell see no candidate and no factor (w = w_single). nbr_idx / nbr_dist: per atom the
// other atoms in ascending distance (natom - 1 entries).
__global__ void __launch_bounds__(128) k_ss(const double* __restrict__ atom_xyz, int natom,
                                            const double* __restrict__ inv, const int* __restrict__ nbr_idx,
                                            const double* __restrict__ nbr_dist, int64_t npts,
                                            const double* __restrict__ xyz, const int* __restrict__ owner,
                                            const double* __restrict__ w_single, double* __restrict__ w_out) {
    constexpr double kReach = 2.0 / (1.0 - 0.64);
    const int nn = natom - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npts; i += (int64_t)gridDim.x * blockDim.x) {
        const double rx = xyz[3 * i], ry = xyz[3 * i + 1], rz = xyz[3 * i + 2];
        const int own = owner[i];
        auto dist = [&](int a) {
            const double dx = rx - atom_xyz[3 * a], dy = ry - atom_xyz[3 * a + 1], dz = rz - atom_xyz[3 * a + 2];
            return sqrt(dx * dx + dy * dy + dz * dz);
        };
        const double lim_own = kReach * dist(own);
        double tot = 0.0, pown = 0.0;
        for (int k = -1; k < nn; ++k) {
            int m = own;
            if (k >= 0) {
                if (nbr_dist[(size_t)own * nn + k] >= lim_own) break;
                m = nbr_idx[(size_t)own * nn + k];
            }
            const double rm = dist(m), lim_m = kReach * rm;
            const double* im = inv + (size_t)m * natom;
            const int* ni = nbr_idx + (size_t)m * nn;
            const double* nd = nbr_dist + (size_t)m * nn;
            double p = 1.0;
            for (int j = 0; j < nn && p != 0.0; ++j) {
                if (nd[j] >= lim_m) break;
                const int n = ni[j];
                p *= ss_s((rm - dist(n)) * __ldg(im + n));
            }
            tot += p;
            if (m == own) pown = p;
        }
        w_out[i] = w_single[i] * (pown / tot);
    }
}

}  // namespace

void launch_ss(const double* atom_xyz, int natom, double* inv, double* adj, const int* nbr_idx,
               const double* nbr_dist, int64_t npts, const double* xyz, const int* owner, const double* w_single,
               double* w_out, bool tables, cudaStream_t s) {
    if (tables)
        k_becke_pairs<<<(natom * natom + 255) / 256, 256, 0, s>>>(atom_xyz, atom_xyz, nullptr, natom, 0, inv, adj);
    const int threads = 128;
    int64_t blocks = (npts + threads - 1) / threads;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    k_ss<<<(unsigned)blocks, threads, 0, s>>>(atom_xyz, natom, inv, nbr_idx, nbr_dist, npts, xyz, owner, w_single,
                                              w_out);
}

void launch_becke_pairs(const double* atom_xyz, const double* brad, int natom, int size_adjust, double* inv,
                        double* adj, cudaStream_t s) {
    k_becke_pairs<<<(natom * natom + 255) / 256, 256, 0, s>>>(atom_xyz, brad, nullptr, natom, size_adjust, inv, adj);
}

// The weights of k_becke with the pair constants from the table (one multiply per pair instead of
// two square roots and a division) and a warp per point: lane l forms P_m for m = l, l + 32, ...
// with the factors in ascending partner order, and lane 0 sums the P_m in ascending m, the
// operations and order of k_becke. The pair constants are read from the transposed table
// (invT[n][m] = inv[m][n], adjT[n][m] = adj[m][n]), so that the lanes' loads for one partner n
// are consecutive; per warp, the point's distances and the P_m sit in shared memory, 16 bytes
// per atom.
constexpr int BECKE_WW = 8;  // warps per CTA
__global__ void __launch_bounds__(32 * BECKE_WW) k_becke_warp(const double* __restrict__ atom_xyz, int natom,
                                                              const double* __restrict__ invT,
                                                              const double* __restrict__ adjT, int64_t npts,
                                                              const double* __restrict__ xyz,
                                                              const int* __restrict__ owner,
                                                              const double* __restrict__ w_single,
                                                              double* __restrict__ w_out) {
    extern __shared__ double smw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* rr = smw + (size_t)warp * 2 * natom;  // [natom]: |r - R_m|
    double* ps = rr + natom;                      // [natom]: P_m(r)
    for (int64_t i = blockIdx.x * (int64_t)BECKE_WW + warp; i < npts; i += (int64_t)gridDim.x * BECKE_WW) {
        const double rx = xyz[3 * i], ry = xyz[3 * i + 1], rz = xyz[3 * i + 2];
        for (int m = lane; m < natom; m += 32) {
            const double ax = atom_xyz[3 * m] - rx, ay = atom_xyz[3 * m + 1] - ry, az = atom_xyz[3 * m + 2] - rz;
            rr[m] = sqrt(ax * ax + ay * ay + az * az);
        }
        __syncwarp();
        for (int m = lane; m < natom; m += 32) {
            const double rm = rr[m];
            double p = 1.0;
            for (int n = 0; n < natom && p != 0.0; ++n) {
                if (n == m) continue;
                double u = (rm - rr[n]) * __ldg(invT + (size_t)n * natom + m);
                u = u + __ldg(adjT + (size_t)n * natom + m) * (1.0 - u * u);
                p *= becke_s(u);
            }
            ps[m] = p;
        }
        __syncwarp();
        if (lane == 0) {
            double tot = 0.0;
            for (int m = 0; m < natom; ++m) tot += ps[m];
            w_out[i] = w_single[i] * (ps[owner[i]] / tot);
        }
        __syncwarp();  // rr and ps are rewritten for the next point
    }
}

__global__ void k_transpose_n2(const double* __restrict__ a, double* __restrict__ at, int n) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e / n), c = (int)(e % n);
        at[(int64_t)c * n + r] = a[e];
    }
}

// Above this many atoms (32 points' distances and lists past 200 KiB of shared memory) the warp form. The
// near form is the faster one up to there; host call, near / warp form: 200 atoms, 0.32 M points 8.7 / 29.9 ms;
// 450 atoms, 0.72 M points 75 / 361.
size_t becke_near_max_atoms() { return 480; }

// Warps per CTA: at 100 atoms eight warps share what shared memory lets four CTAs hold (12.6 -> 8.7 ms with
// the lists in registers); few atoms leave eight warps too little each (30 atoms:
// 0.56 ms with four, 0.61 with eight; 43 atoms 1.14 with four).
constexpr int kNearSmall = 48;

size_t becke_near_table_bytes(int natom) {
    return (size_t)natom * natom * (sizeof(double2) + sizeof(float2)) + sizeof(int) * (kNearList + 1) * (size_t)natom;
}

static size_t becke_near_smem(int natom) {
    return (size_t)natom * kNearPts * (sizeof(double) + sizeof(float)) + sizeof(double) * kNearCap +
           sizeof(int) * (2 * (size_t)natom + 1);
}

void launch_becke_near(const double* atom_xyz, const double* brad, const int* ghost, int natom, int size_adjust,
                       void* tab, int64_t npts, const double* xyz, const int* owner, const double* w_single,
                       double* w_out, bool tables, cudaStream_t s) {
    const size_t n2 = (size_t)natom * natom;
    double2* pair = static_cast<double2*>(tab);
    float2* pairf = reinterpret_cast<float2*>(pair + n2);
    int* near = reinterpret_cast<int*>(pairf + n2);
    int* odd = near + kNearList * (size_t)natom;
    if (tables)
        k_becke_near_tables<<<natom, 128, sizeof(double) * natom, s>>>(atom_xyz, brad, ghost, natom, size_adjust, pair,
                                                                       pairf, near, odd);
    const size_t smem = becke_near_smem(natom);
    // the limit belongs to the function in the whole process: the largest size, whatever this call's (calls
    // on other threads would lower one another's; so in every launcher whose size varies)
    const int limit = (int)becke_near_smem((int)becke_near_max_atoms());
    // The weights do not depend on the share, only how many atoms are dropped and how often a point is summed
    // again; a looser one from the environment (PDFXC_BECKE_SHARE) lets the tests reach the second sum.
    const char* env = std::getenv("PDFXC_BECKE_SHARE");
    const float share = env ? (float)std::atof(env) : 0x1p-80f;
    int64_t blocks = (npts + kNearPts - 1) / kNearPts;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    if (natom <= kNearSmall) {
        cudaFuncSetAttribute(k_becke_near<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
        k_becke_near<4><<<(unsigned)blocks, 128, smem, s>>>(atom_xyz, natom, pair, pairf, near, odd, npts, xyz, owner,
                                                            w_single, w_out, share);
    } else {
        cudaFuncSetAttribute(k_becke_near<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
        k_becke_near<8><<<(unsigned)blocks, 256, smem, s>>>(atom_xyz, natom, pair, pairf, near, odd, npts, xyz, owner,
                                                            w_single, w_out, share);
    }
}

size_t becke_warp_max_atoms() { return (200u * 1024u) / (2 * sizeof(double) * BECKE_WW); }

// tab: 4 n_atom^2 doubles (the pair table, then its transpose)
void launch_becke_warp(const double* atom_xyz, const double* brad, const int* ghost, int natom, int size_adjust,
                       double* tab, int64_t npts, const double* xyz, const int* owner, const double* w_single,
                       double* w_out, bool tables, cudaStream_t s) {
    const size_t n2 = (size_t)natom * natom;
    double *inv = tab, *adj = tab + n2, *invT = tab + 2 * n2, *adjT = tab + 3 * n2;
    if (tables) {
        k_becke_pairs<<<(unsigned)((n2 + 255) / 256), 256, 0, s>>>(atom_xyz, brad, ghost, natom, size_adjust, inv, adj);
        const unsigned tb = (unsigned)std::min<size_t>((n2 + 255) / 256, 148 * 8);
        k_transpose_n2<<<tb, 256, 0, s>>>(inv, invT, natom);
        k_transpose_n2<<<tb, 256, 0, s>>>(adj, adjT, natom);
    }
    int64_t blocks = (npts + BECKE_WW - 1) / BECKE_WW;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    const size_t smem = 2 * sizeof(double) * BECKE_WW * natom;
    cudaFuncSetAttribute(k_becke_warp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(2 * sizeof(double) * BECKE_WW * becke_warp_max_atoms()));
    k_becke_warp<<<(unsigned)blocks, 32 * BECKE_WW, smem, s>>>(atom_xyz, natom, invT, adjT, npts, xyz, owner, w_single,
                                                               w_out);
}

void launch_becke(const double* atom_xyz, const double* brad, const int* ghost, int natom, int size_adjust,
                  int64_t npts, const double* xyz, const int* owner, const double* w_single, double* w_out,
                  cudaStream_t s) {
    const int threads = 128;
    int64_t blocks = (npts + threads - 1) / threads;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    const size_t smem = sizeof(double4) * natom;
    cudaFuncSetAttribute(k_becke, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(double4) * becke_max_atoms()));
    k_becke<<<(unsigned)blocks, threads, smem, s>>>(atom_xyz, brad, ghost, natom, size_adjust, npts, xyz, owner,
                                                    w_single, w_out);
}

size_t becke_max_atoms() { return (220u * 1024u) / sizeof(double4); }

}  // namespace pdfxc
