// XC nuclear gradient on the device (FP64): DfCalcGridX::energyGradient /
// energyGradient_part (src/libpdf/DfCalcGridX.cpp:1073-1415).
//
// AO-centre term, per block of 128 points with its screened AO list: with X = P_sub phi, the
// coefficients a = 0.5 w vrho and c = w (2 vgAA + vgAB) grad rho_A, and Z = a phi + c . grad phi, the
// contribution of AO i on atom B is
//   G_i = 2 a grad phi_i X_i + sum_k c_k (grad d_k phi_i X_i + grad phi_i Y_ki),  Y_k = P_sub d_k phi,
// and sum_k c_k Y_k = P_sub (c . grad phi) = P_sub Z - a X =: Y - a X, so one contraction of Z, which the
// adjoint needs anyway, stands for the three of the derivatives, and
//   G_i = grad phi_i (a X_i + Y_i) + (grad grad phi_i c) X_i,
// formed from the shells' radial sums (no plane of derivatives is stored; the reference evaluates
// getAOs / getDAOs / getD2AOs, :667-863);
// grad[B] -= 4 G_i (the reference's -2 w, doubled for the closed shell), grad[owner] += 4 G_i (the grid
// moves with its atom).
// Grid-weight term, per point with coefficient c = w_single f (f the energy density):
//                the derivative of the Becke partition omega_A = P_A / sum_i P_i with
//                respect to every nucleus (Johnson, Gill and Pople, J. Chem. Phys. 98,
//                5612 (1993), appendix B), written from the partition function; the
//                reference's own version of this term evaluates to zero (its JGP_t,
//                src/libpdf/DfGenerateGrid.cpp:2357-2372, returns 0 unless |mu| > 1).
#include <cuda_runtime.h>

#include "ao.cuh"
#include "pdfxc_internal.cuh"

namespace pdfxc {

namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// grad[3 * atom + k] += scale * (sum over the warp of v[k]); every lane calls it with the same atom.
__device__ __forceinline__ void warp_add3(double* grad, int atom, double scale, double vx, double vy, double vz) {
    const double sx = warp_sum(vx), sy = warp_sum(vy), sz = warp_sum(vz);
    if ((threadIdx.x & 31) == 0 && (sx != 0.0 || sy != 0.0 || sz != 0.0)) {
        atomicAdd(&grad[3 * atom], scale * sx);
        atomicAdd(&grad[3 * atom + 1], scale * sy);
        atomicAdd(&grad[3 * atom + 2], scale * sz);
    }
}

// grad[3 * own + k] += scale * v[k], lanes with the same owner summed first (a warp's
// points usually share one or two owners).
__device__ __forceinline__ void warp_add3_by_owner(double* grad, int own, double scale, double vx, double vy,
                                                   double vz) {
    const int lane = threadIdx.x & 31;
    unsigned todo = 0xffffffffu;
    while (todo) {
        const int src = __ffs(todo) - 1;
        const int o = __shfl_sync(0xffffffffu, own, src);
        const bool mine = own == o;
        todo &= ~__ballot_sync(0xffffffffu, mine);
        const double sx = warp_sum(mine ? vx : 0.0), sy = warp_sum(mine ? vy : 0.0), sz = warp_sum(mine ? vz : 0.0);
        if (lane == src && (sx != 0.0 || sy != 0.0 || sz != 0.0)) {
            atomicAdd(&grad[3 * o], scale * sx);
            atomicAdd(&grad[3 * o + 1], scale * sy);
            atomicAdd(&grad[3 * o + 2], scale * sz);
        }
    }
}

// One CTA per block, 256 threads: the point is threadIdx.x % 128, the halves of the CTA take the
// first and the second half of the block's shells (runs of one atom's shells stay together but for
// one). Reads X, Y and the radial sums once; 16 warps per SM (its registers) do not cover the latency
// (L1 prefetches of the shells ahead changed nothing). 30-atom PBE chain, 477k points: 0.52 ms (0.97 with
// the atomics on one copy of the gradient), for 3.0 ms of the stored second derivatives (1.2) and the pass
// over 14 planes (1.8), and three contractions less.
template <bool GGA>
__global__ void __launch_bounds__(256, 2) k_grad_atoms(BasisView bas, GridView g, const int* __restrict__ owner,
                                                       int natom, int blk0, const double* __restrict__ coef,
                                                       const char* ws, double* grad) {
    __shared__ double s_xyz[3][128];
    __shared__ int s_row[128], s_l[128], s_at[128];
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    grad += (size_t)6 * natom * (blk % GRAD_COPIES);
    const int p = threadIdx.x & (BLOCK_PTS - 1), half = threadIdx.x >> 7;
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    const double* base = reinterpret_cast<const double*>(ws + m.ws) + p;
    const double* X = base + GRAD_X * plane;
    const double* Y = base + GRAD_Y * plane;
    const double* S0p = base + (GGA ? 4 : 3) * plane;
    const double* S1p = S0p + (size_t)m.nsh * BLOCK_PTS;
    const double* S2p = S1p + (size_t)m.nsh * BLOCK_PTS;
    const size_t gp = (size_t)blk * BLOCK_PTS + p;
    const double px = g.px[gp], py = g.py[gp], pz = g.pz[gp];
    const double a = coef[gp * 4], cx = coef[gp * 4 + 1], cy = coef[gp * 4 + 2], cz = coef[gp * 4 + 3];
    double tx = 0.0, ty = 0.0, tz = 0.0;  // all shells of this thread
    for (int i0 = 0; i0 < m.nsh; i0 += 128) {
        const int kn = min(128, m.nsh - i0);
        __syncthreads();
        for (int k = threadIdx.x; k < kn; k += 256) {
            const int sh = g.blk_shells[m.sh0 + i0 + k], at = bas.sh_atom[sh];
            s_row[k] = g.blk_shell_row[m.sh0 + i0 + k], s_l[k] = bas.sh_l[sh], s_at[k] = at;
#pragma unroll
            for (int c = 0; c < 3; ++c) s_xyz[c][k] = bas.atom_xyz[3 * at + c];
        }
        __syncthreads();
        const int k1 = half ? kn : (kn + 1) / 2;
        int k = half ? (kn + 1) / 2 : 0;
        while (k < k1) {
            const int at = s_at[k];  // uniform over a warp
            const double x = px - s_xyz[0][k], y = py - s_xyz[1][k], z = pz - s_xyz[2][k];
            double ax = 0.0, ay = 0.0, az = 0.0, unused = 0.0;
            for (; k < k1 && s_at[k] == at; ++k) {
                const int L = s_l[k], row0 = s_row[k];
                const size_t o = (size_t)(i0 + k) * BLOCK_PTS;
                const double S0 = S0p[o], S1 = S1p[o];
                double xv[5], u[5];
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    xv[c] = c < 2 * L + 1 ? X[(size_t)(row0 + c) * BLOCK_PTS] : 0.0;
                    if (GGA) u[c] = c < 2 * L + 1 ? fma(a, xv[c], Y[(size_t)(row0 + c) * BLOCK_PTS]) : 0.0;
                    else u[c] = 2.0 * a * xv[c];
                }
                shell_rho<true>(L, x, y, z, S0, S1, u, unused, ax, ay, az);
                if (GGA) shell_hess(L, x, y, z, S0, S1, S2p[o], xv, cx, cy, cz, ax, ay, az);
            }
            warp_add3(grad, at, -4.0, ax, ay, az);
            tx += ax, ty += ay, tz += az;
        }
    }
    warp_add3_by_owner(grad, owner[gp], 4.0, tx, ty, tz);
}

__device__ __forceinline__ void becke_poly(double nu, double& p1, double& p2, double& p3) {
    p1 = 0.5 * nu * (3.0 - nu * nu);
    p2 = 0.5 * p1 * (3.0 - p1 * p1);
    p3 = 0.5 * p2 * (3.0 - p2 * p2);
}

// Grid-weight term. 32 points per CTA (a lane each), the atoms divided over its four warps; shared
// memory holds each point's atom distances and partition products, [natom][32] each. Pair constants
// (1/R_ij and the size adjustment a_ij) come from the table k_becke_pairs writes.
// For B != owner A and every other atom i, one evaluation of nu_iB gives
// s_iB = (1 - f3)/2, s_Bi = (1 + f3)/2 (nu_Bi = -nu_iB), s'(nu_iB) = s'(nu_Bi) and
// grad_B mu_iB = -grad_B mu_Bi, so that
//   grad_B Z += s' dnu grad_B mu_iB (P_i / s_iB - P_B / s_Bi),
//   grad_B P_A = s'(nu_AB) dnu grad_B mu_AB P_A / s_AB,
// where P_i / s_iB is the product of P_i's other factors (taken as 0 when s_iB has
// underflowed: the term is then below 1e-250).
// A pair of atoms whose P_i and P_B both lie below 2^-80 Z at all of the CTA's points is left out: at
// that size s' / s is at most 2e4 (s ~ (1 - nu)^8), so its terms are below 1e-19 of the others. The
// points of a CTA are neighbours, so most pairs of a larger molecule go.
// Bound by the FP64 pipe. 30-atom chain, 477k points: 1.88 ms (a thread per point, every pair: 4.09).
//
// ROWS_IN_DRAM: the two [natom] rows of every point live in a scratch array in device memory
// ([2][natom][32 gridDim.x], a warp's accesses coalesced) instead of shared memory; the form for
// systems whose rows do not fit shared memory. The live atoms (a list and a flag per atom) follow in
// shared memory.
constexpr int GW_T = 32, GW_W = 4;
template <bool ROWS_IN_DRAM>
__global__ void __launch_bounds__(GW_T* GW_W) k_grad_weight(
    const double* __restrict__ atom_xyz, int natom, const double* __restrict__ inv, const double* __restrict__ adj,
    int64_t nslots, const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const int* __restrict__ owner, const double* __restrict__ wsingle, const double* __restrict__ fdens, double* grad,
    double* __restrict__ scratch) {
    extern __shared__ double sm[];
    __shared__ double s_z[GW_W][GW_T];
    __shared__ int s_n;
    constexpr unsigned kAll = 0xffffffffu;
    const size_t stride = ROWS_IN_DRAM ? (size_t)gridDim.x * GW_T : (size_t)GW_T;
    double* rr = ROWS_IN_DRAM ? scratch + (size_t)blockIdx.x * GW_T : sm;  // [natom][stride]
    double* Pm = rr + (size_t)natom * stride;                               // [natom][stride]
    int* list = reinterpret_cast<int*>(sm + (ROWS_IN_DRAM ? 0 : 2 * (size_t)natom * GW_T));  // [natom] live atoms
    int* live_at = list + natom;                                                              // [natom] 0 or 1
    const int t = threadIdx.x & 31, warp = threadIdx.x >> 5;
    grad += (size_t)6 * natom * (blockIdx.x % GRAD_COPIES);
    constexpr double kTiny = 1e-250;
    for (int64_t i0 = blockIdx.x * (int64_t)GW_T; i0 < nslots; i0 += (int64_t)gridDim.x * GW_T) {
        const int64_t i = i0 + t;
        const bool live = i < nslots;
        const double c = live ? wsingle[i] * fdens[i] : 0.0;
        if (!__any_sync(kAll, c != 0.0)) continue;  // the same points in every warp: uniform over the CTA
        const double rx = live ? px[i] : 0.0, ry = live ? py[i] : 0.0, rz = live ? pz[i] : 0.0;
        const int A = live ? owner[i] : 0;
        for (int m = warp; m < natom; m += GW_W) {
            const double ax = __ldg(atom_xyz + 3 * m) - rx, ay = __ldg(atom_xyz + 3 * m + 1) - ry,
                         az = __ldg(atom_xyz + 3 * m + 2) - rz;
            rr[m * stride + t] = sqrt(ax * ax + ay * ay + az * az);
        }
        __syncthreads();
        // partition products
        double z4 = 0.0;
        for (int m = warp; m < natom; m += GW_W) {
            const double rm = rr[m * stride + t];
            const double *im = inv + (size_t)m * natom, *am = adj + (size_t)m * natom;
            double p = 1.0;
            for (int n = 0; n < natom; ++n) {
                if (n == m) continue;
                const double mu = (rm - rr[n * stride + t]) * __ldg(im + n);
                double p1, p2, p3;
                becke_poly(mu + __ldg(am + n) * (1.0 - mu * mu), p1, p2, p3);
                p *= 0.5 * (1.0 - p3);
            }
            Pm[m * stride + t] = p;
            z4 += p;
        }
        s_z[warp][t] = z4;
        __syncthreads();
        const double Z = (s_z[0][t] + s_z[1][t]) + (s_z[2][t] + s_z[3][t]);
        const bool act = c != 0.0 && Z > 0.0;
        const double invZ = act ? 1.0 / Z : 0.0;
        for (int m = warp; m < natom; m += GW_W) {  // an atom is live where any point needs its P
            const bool need = __any_sync(kAll, act && !(Pm[m * stride + t] < 8.271806125530277e-25 * Z));
            if (t == 0) live_at[m] = need ? 1 : 0;
        }
        __syncthreads();
        if (warp == 0) {
            int n = 0;
            for (int m0 = 0; m0 < natom; m0 += 32) {
                const bool f = m0 + t < natom && live_at[m0 + t];
                const unsigned bits = __ballot_sync(kAll, f);
                if (f) list[n + __popc(bits & ((1u << t) - 1))] = m0 + t;
                n += __popc(bits);
            }
            if (t == 0) s_n = n;
        }
        __syncthreads();
        const int nlive = s_n;
        const double PA = Pm[A * stride + t];
        const double omega = PA * invZ;
        double Tx = 0.0, Ty = 0.0, Tz = 0.0;
        for (int B = warp; B < natom; B += GW_W) {
            const bool all = live_at[B] != 0;  // against every atom, or against the live ones
            const int nn = all ? natom : nlive;
            double dx = 0.0, dy = 0.0, dz = 0.0;
            if (act && B != A) {
                const double RBx = __ldg(atom_xyz + 3 * B), RBy = __ldg(atom_xyz + 3 * B + 1),
                             RBz = __ldg(atom_xyz + 3 * B + 2);
                const double rB = rr[B * stride + t];
                const double irB = 1.0 / rB;
                const double ux = (RBx - rx) * irB, uy = (RBy - ry) * irB, uz = (RBz - rz) * irB;
                const double PB = Pm[B * stride + t];
                // sum over n of h (u + mu e), h = -f / R_nB, e the unit vector from n to B: the u terms
                // in one sum, the e terms by component
                double hs = 0.0, ex = 0.0, ey = 0.0, ez = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
                for (int j = 0; j < nn; ++j) {
                    const int n = all ? j : list[j];
                    if (n == B) continue;
                    const double iR = __ldg(inv + (size_t)n * natom + B);
                    const double a = __ldg(adj + (size_t)n * natom + B);
                    const double mu = (rr[n * stride + t] - rB) * iR;
                    const double nu = mu + a * (1.0 - mu * mu);
                    double p1, p2, p3;
                    becke_poly(nu, p1, p2, p3);
                    const double s_nB = 0.5 * (1.0 - p3), s_Bn = 0.5 * (1.0 + p3);
                    const double k = -(27.0 / 16.0) * (1.0 - p2 * p2) * (1.0 - p1 * p1) * (1.0 - nu * nu) *
                                     (1.0 - 2.0 * a * mu);
                    // P_n / s_nB and P_B / s_Bn with one division (s_nB + s_Bn = 1: their product
                    // underflows only where a quotient is dropped anyway)
                    const bool okn = s_nB > kTiny, okb = s_Bn > kTiny;
                    const double is = 1.0 / ((okn ? s_nB : 1.0) * (okb ? s_Bn : 1.0));
                    const double rn = okn ? Pm[n * stride + t] * (okb ? s_Bn : 1.0) * is : 0.0;
                    const double rb = okb ? PB * (okn ? s_nB : 1.0) * is : 0.0;
                    const double h = -k * (rn - rb) * iR, q = h * mu * iR;
                    const double ox = RBx - __ldg(atom_xyz + 3 * n), oy = RBy - __ldg(atom_xyz + 3 * n + 1),
                                 oz = RBz - __ldg(atom_xyz + 3 * n + 2);
                    hs += h;
                    ex = fma(q, ox, ex), ey = fma(q, oy, ey), ez = fma(q, oz, ez);
                    if (n == A) {
                        const double ha = -k * rn * iR, qa = ha * mu * iR;
                        gx = ha * ux + qa * ox, gy = ha * uy + qa * oy, gz = ha * uz + qa * oz;
                    }
                }
                dx = c * (gx - omega * (hs * ux + ex)) * invZ;
                dy = c * (gy - omega * (hs * uy + ey)) * invZ;
                dz = c * (gz - omega * (hs * uz + ez)) * invZ;
            }
            warp_add3(grad, B, 1.0, dx, dy, dz);
            Tx += dx, Ty += dy, Tz += dz;
        }
        warp_add3_by_owner(grad, A, -1.0, Tx, Ty, Tz);
        __syncthreads();  // the rows and lists are rewritten by the next tile of points
    }
}

}  // namespace

void launch_grad_atoms(const BasisView& b, const GridView& g, const int* owner, int natom, int blk0, int nblk, bool gga,
                       const double* coef, const char* ws, double* grad, cudaStream_t s) {
    if (gga)
        k_grad_atoms<true><<<nblk, 256, 0, s>>>(b, g, owner, natom, blk0, coef, ws, grad);
    else
        k_grad_atoms<false><<<nblk, 256, 0, s>>>(b, g, owner, natom, blk0, coef, ws, grad);
}

// Shared memory per CTA: 520 bytes per atom (two rows of 32 doubles, a list entry and a flag); beyond
// 400 atoms the rows live in device memory (grad_weight_scratch_doubles of scratch).
int grad_weight_max_atoms() { return (int)((200u * 1024u) / (2 * sizeof(double) * GW_T)); }

namespace {
constexpr int kWeightDramCtas = 148 * 4;
// Limits of the dynamic shared memory (the functions' for the whole process, so not by this call's size): the
// most atoms of the shared form; for the other an SM's 227 KiB less the kernel's own 1040 bytes
constexpr int kWeightSmem = 400 * (2 * (int)sizeof(double) * GW_T + 2 * (int)sizeof(int));
constexpr int kWeightListSmem = 227 * 1024 - 1040;
}

size_t grad_weight_scratch_doubles(int natom) { return (size_t)2 * natom * kWeightDramCtas * GW_T; }

void launch_grad_weight(const double* atom_xyz, int natom, const double* inv, const double* adj, int64_t nslots,
                        const double* px, const double* py, const double* pz, const int* owner, const double* wsingle,
                        const double* fdens, double* grad, double* scratch, cudaStream_t s) {
    const size_t lists = 2 * sizeof(int) * (size_t)natom;
    int64_t blocks = (nslots + GW_T - 1) / GW_T;
    if (scratch) {
        if (blocks > kWeightDramCtas) blocks = kWeightDramCtas;
        cudaFuncSetAttribute(k_grad_weight<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWeightListSmem);
        k_grad_weight<true><<<(unsigned)blocks, GW_T * GW_W, lists, s>>>(atom_xyz, natom, inv, adj, nslots, px, py, pz,
                                                                        owner, wsingle, fdens, grad, scratch);
    } else {
        const size_t smem = 2 * sizeof(double) * GW_T * (size_t)natom + lists;
        if (blocks > 148 * 32) blocks = 148 * 32;
        cudaFuncSetAttribute(k_grad_weight<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWeightSmem);
        k_grad_weight<false><<<(unsigned)blocks, GW_T * GW_W, smem, s>>>(atom_xyz, natom, inv, adj, nslots, px, py, pz,
                                                                         owner, wsingle, fdens, grad, nullptr);
    }
}

}  // namespace pdfxc
