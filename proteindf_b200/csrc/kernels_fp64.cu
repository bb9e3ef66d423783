// FP64 drop-in kernels of the XC build.
//
// Per block of up to 128 grid points with its screened AO list (nb AOs), one build runs
//   ao_eval      phi[mu][p] and, for a GGA, the shells' radial sums (DfCalcGridX.cpp:667-769)
//   gemm_x       X = P_sub * phi, P_sub = P_A[aos, aos]; an LDA's epilogue sums rho per tile of rows
//   rho_rad      rho_A(p) = sum_mu phi X, grad rho_A = 2 sum_mu grad phi X (:865-931) (GGA)
//   functional   the functional, Exc and electron-count partials, and the
//                per-point Vxc coefficients (:2056-2193, :2455-2500)
//   z_rad        Z[nu][p] = 0.5 w vrho phi + c . grad phi, c = w (2 vgAA + vgAB) grad rho_A (GGA)
//   gemm_v       Vacc[aos, aos] += phi * Z^T (an LDA scales phi by 0.5 w vrho instead)
//   finish       V = Vacc + Vacc^T, FP64 block sums of Exc and the electron count
// V = phi Z^T + Z phi^T reproduces the reference's element formula
// V_ij += w vrho phi_i phi_j + phi_i (c . grad phi_j) + phi_j (c . grad phi_i).
// The open shell runs the same kernels with two densities and two Z planes. The no-allocation build,
// the density at points and the adjoint store X (rho_functional, gradient.cu).
#include <cuda_runtime.h>

#include "ao.cuh"
#include "functional.cuh"
#include "pdfxc_internal.cuh"

namespace pdfxc {

namespace {

// One CTA per block, 256 threads: the point is threadIdx.x % 128, the two
// halves of the CTA take alternate shells. Stores are coalesced along points.
// Per shell the contraction is summed once (shell_radial), then every component
// is formed from the radial sums (ao_from_radial).
template <bool GGA>
__global__ void __launch_bounds__(256) k_ao_eval(BasisView bas, GridView g, int blk0, char* ws) {
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    const int p = threadIdx.x & (BLOCK_PTS - 1);
    const int half = threadIdx.x >> 7;
    double* phi = reinterpret_cast<double*>(ws + m.ws);
    double* dphi = phi + (size_t)m.nbp * BLOCK_PTS;
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    const int gp = blk * BLOCK_PTS + p;
    const double rx = g.px[gp], ry = g.py[gp], rz = g.pz[gp];
    for (int i = half; i < m.nsh; i += 2) {
        const int s = g.blk_shells[m.sh0 + i];
        const int row0 = g.blk_shell_row[m.sh0 + i];
        const int a = bas.sh_atom[s];
        const double x = rx - bas.atom_xyz[3 * a], y = ry - bas.atom_xyz[3 * a + 1],
                     z = rz - bas.atom_xyz[3 * a + 2];
        const int L = bas.sh_l[s], n = 2 * L + 1;
        double S0, S1;
        shell_radial<GGA>(bas, s, x * x + y * y + z * z, S0, S1);
        for (int c = 0; c < n; ++c) {
            double v, gx, gy, gz;
            ao_from_radial<GGA>(L * L + c, x, y, z, S0, S1, v, gx, gy, gz);
            const size_t o = (size_t)(row0 + c) * BLOCK_PTS + p;
            phi[o] = v;
            if (GGA) {
                dphi[o] = gx;
                dphi[plane + o] = gy;
                dphi[2 * plane + o] = gz;
            }
        }
    }
    // zero the padding rows
    for (int r = m.nb + half; r < m.nbp; r += 2) {
        const size_t o = (size_t)r * BLOCK_PTS + p;
        phi[o] = 0.0;
        if (GGA) dphi[o] = dphi[plane + o] = dphi[2 * plane + o] = 0.0;
    }
}

// FP64 tensor-core MMA: D(8x8) += A(8x4, row-major) B(4x8, col-major), FP64 in and out.
// Per thread (g = lane / 4, t = lane % 4): a = A[g][t], b = B[t][g], d = {D[g][2t], D[g][2t+1]}.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Asynchronous copies global -> shared; with ok = false the destination is zero-filled and nothing is read.
__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(ok ? 8 : 0));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(ok ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The FP64 contractions cover a block's nb AOs with T = ceil(nb / 64) tiles per dimension, tile i
// taking an equal share of the 16-row pairs of DMMA rows, cut at the last row of eight: nb rounded up
// to 8, not to 64, is what the tensor pipe works for. (On the benchmark's 100-atom chain nb averages 218,
// 221 rounded up to 8 and 250 rounded up to 64: 21 % off the sum of nb^2.) r8, n8: first row of eight and
// their number (at most 8).
__device__ __forceinline__ void fp64_tile(int nb, int T, int i, int& r8, int& n8) {
    const int pairs = (nb + 15) / 16;
    r8 = 2 * (i * pairs / T);
    n8 = min((nb + 7) / 8, 2 * ((i + 1) * pairs / T)) - r8;
}

// X[m][p] = sum_k P[aos[m]][aos[k]] phi[k][p]: CTA tile up to 64 rows x 128 points, K step 16 in a
// ring of three shared-memory stages filled by asynchronous copies (one barrier per step), 8 warps
// of all the tile's rows x 16 points (up to 8 x 2 DMMA tiles), so that a trimmed tile shortens every
// warp alike. Bound by the FP64 tensor pipe. Planes are [nbp][128] arrays of the block's workspace:
// source plane src0, destination plane dst0 (the adjoint: phi -> X, and Z -> P_sub Z).
// MODE (bits): X_STORE writes X. X_PHI (LDA) reduces it: the tile goes to shared memory and each thread
// sums rho for its point and half of the tile's rows; the tile's sums go to row 4 tile of plane sum0
// (nb >= 1 AOs give ceil(nb / 64) tiles and at least 8 rows). An LDA build needs the sums only, which
// saves X's round trip through HBM and the pass over phi and X: (H2O)8 SVWN, with the symmetric Vxc
// contraction below, 0.83 -> 0.64 ms. The same for a GGA (grad rho from the radial sums in the epilogue)
// was slower, 21.5 -> 22.7 ms at 100 atoms: with two CTAs per SM the radial sums' latency is not hidden,
// and k_rho_rad, a pass of its own, streams them.
// Rows of phi at nb and beyond are not read. Row strides of 20 and 132 doubles keep the fragment
// loads free of bank conflicts (4 g + t and g + 4 t distinct modulo 16).
constexpr int GX_BM = 64, GX_BK = 16, GX_S = 3, GX_AS = GX_BK + 4, GX_BS = BLOCK_PTS + 4;
constexpr int GX_STAGE = GX_BM * GX_AS + GX_BK * GX_BS;  // doubles
constexpr int GX_SMEM = GX_S * GX_STAGE * 8;
constexpr int GX_XS = BLOCK_PTS + 8;  // row of the X tile in shared memory: its 16-byte stores conflict-free
static_assert(GX_BM * GX_XS <= GX_S * GX_STAGE, "the X tile reuses the stages");
enum { X_STORE = 1, X_PHI = 2 };

// one K step (kn of its 16 columns, in fours) of a warp's MC x 2 DMMA tiles
template <int MC>
__device__ __forceinline__ void gx_step(const double* As, const double* Bs, int kn, double (&acc)[8][2][2]) {
    auto four = [&](int kk) {
        double a[MC], b[2];
#pragma unroll
        for (int i = 0; i < MC; ++i) a[i] = As[i * 8 * GX_AS + kk];
#pragma unroll
        for (int j = 0; j < 2; ++j) b[j] = Bs[kk * GX_BS + j * 8];
#pragma unroll
        for (int i = 0; i < MC; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    };
    if (kn >= GX_BK) {
#pragma unroll
        for (int kk = 0; kk < GX_BK; kk += 4) four(kk);
    } else {
#pragma unroll 1
        for (int kk = 0; kk < kn; kk += 4) four(kk);
    }
}

template <int MODE>
__global__ void __launch_bounds__(256, 2) k_gemm_x(GridView g, const double* __restrict__ P, int nao,
                                                int blk0, char* ws, int src0, int dst0, int sum0, int64_t t0) {
    extern __shared__ __align__(16) double gx_sm[];
    int blk, ti;
    if (g.xtiles) {  // one CTA per tile of the list
        const int2 it = g.xtiles[t0 + blockIdx.x];
        blk = it.x, ti = it.y;
    } else {
        blk = blk0 + blockIdx.y, ti = blockIdx.x;
    }
    const BlockMeta m = g.meta[blk];
    const int T = (m.nb + 63) / 64;
    if (ti >= T) return;
    int r8, mc;
    fp64_tile(m.nb, T, ti, r8, mc);
    const int m0 = r8 * 8;
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    const double* phi = reinterpret_cast<const double*>(ws + m.ws) + (size_t)src0 * plane;
    double* X = reinterpret_cast<double*>(ws + m.ws) + (size_t)dst0 * plane;
    const int* aos = g.blk_aos + m.ao0;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int gq = lane >> 2, tq = lane & 3;
    // this thread's share of a stage: A column t % 16 of rows t / 16 + 16 q (gathered from P), B
    // the 16-byte piece t % 64 of phi rows t / 64 + 4 q
    const double* prow[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = (t >> 4) + 16 * q;
        prow[q] = r < 8 * mc && m0 + r < m.nb ? P + (size_t)aos[m0 + r] * nao : nullptr;
    }
    const int nk = (m.nb + GX_BK - 1) / GX_BK;
    int next = (t & 15) < m.nb ? aos[t & 15] : -1;  // the AO of this thread's A column, a step ahead of its use
    auto issue = [&](int kt) {
        double* st = gx_sm + (kt % GX_S) * GX_STAGE;
        const int col = next, k = (kt + 1) * GX_BK + (t & 15);
        next = k < m.nb ? aos[k] : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool ok = col >= 0 && prow[q];
            cp_async8(st + ((t >> 4) + 16 * q) * GX_AS + (t & 15), ok ? prow[q] + col : P, ok);
        }
        double* bs = st + GX_BM * GX_AS;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = (t >> 6) + 4 * q, kr = kt * GX_BK + r;
            const bool ok = kr < m.nb;
            cp_async16(bs + r * GX_BS + 2 * (t & 63), phi + (ok ? (size_t)kr * BLOCK_PTS + 2 * (t & 63) : 0), ok);
        }
    };
    double acc[8][2][2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int k = 0; k < GX_S - 1; ++k) {
        if (k < nk) issue(k);
        cp_async_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<GX_S - 2>();
        __syncthreads();  // stage kt has landed for every thread, and stage kt - 1 is consumed
        if (kt + GX_S - 1 < nk) issue(kt + GX_S - 1);
        cp_async_commit();
        const double* st = gx_sm + (kt % GX_S) * GX_STAGE;
        const double* As = st + gq * GX_AS + tq;
        const double* Bs = st + GX_BM * GX_AS + tq * GX_BS + warp * 16 + gq;
        const int kn = m.nb - kt * GX_BK;
        switch (mc) {  // uniform over the CTA
            case 8: gx_step<8>(As, Bs, kn, acc); break;
            case 7: gx_step<7>(As, Bs, kn, acc); break;
            case 6: gx_step<6>(As, Bs, kn, acc); break;
            case 5: gx_step<5>(As, Bs, kn, acc); break;
            case 4: gx_step<4>(As, Bs, kn, acc); break;
            case 3: gx_step<3>(As, Bs, kn, acc); break;
            case 2: gx_step<2>(As, Bs, kn, acc); break;
            default: gx_step<1>(As, Bs, kn, acc);
        }
    }
    if (MODE & X_STORE) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < mc)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    *reinterpret_cast<double2*>(X + (size_t)(m0 + i * 8 + gq) * BLOCK_PTS + warp * 16 + j * 8 + 2 * tq) =
                        make_double2(acc[i][j][0], acc[i][j][1]);
    }
    if (MODE == X_STORE) return;
    __syncthreads();  // the last stage is consumed (no copies are in flight)
    double* Xs = gx_sm;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (i < mc)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                *reinterpret_cast<double2*>(Xs + (i * 8 + gq) * GX_XS + warp * 16 + j * 8 + 2 * tq) =
                    make_double2(acc[i][j][0], acc[i][j][1]);
    __syncthreads();
    const int p = t & (BLOCK_PTS - 1), half = t >> 7;
    const int rows = min(8 * mc, m.nb - m0), mid = (rows + 1) / 2;
    double sum = 0.0;
    for (int r = half ? mid : 0; r < (half ? rows : mid); ++r)
        sum = fma(phi[(size_t)(m0 + r) * BLOCK_PTS + p], Xs[r * GX_XS + p], sum);
    __syncthreads();  // the X tile is read
    if (half) gx_sm[p] = sum;
    __syncthreads();
    if (!half) {
        double* sums = reinterpret_cast<double*>(ws + m.ws) + sum0 * plane;
        sums[(size_t)4 * ti * BLOCK_PTS + p] = sum + gx_sm[p];
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One CTA (128 threads, one per point) per block.
template <bool GGA>
__global__ void __launch_bounds__(BLOCK_PTS) k_rho_functional(GridView g, int blk0, int fn, int incremental,
                                                              double rho_cut, char* ws, double* rho_store,
                                                              double* coef, double* blk_sum) {
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    const int p = threadIdx.x;
    const int nplanes = GGA ? 4 : 1;
    const double* phi = reinterpret_cast<const double*>(ws + m.ws);
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    const double* X = phi + nplanes * plane;
    double rho = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    for (int r = 0; r < m.nb; ++r) {
        const size_t o = (size_t)r * BLOCK_PTS + p;
        const double x = X[o];
        rho = fma(phi[o], x, rho);
        if (GGA) {
            gx = fma(phi[plane + o], x, gx);
            gy = fma(phi[2 * plane + o], x, gy);
            gz = fma(phi[3 * plane + o], x, gz);
        }
    }
    gx *= 2.0, gy *= 2.0, gz *= 2.0;
    const size_t gp = (size_t)blk * BLOCK_PTS + p;
    double* rs = rho_store + gp * 4;
    if (incremental) {
        rho += rs[0];
        gx += rs[1], gy += rs[2], gz += rs[3];
    }
    rs[0] = rho, rs[1] = gx, rs[2] = gy, rs[3] = gz;
    const double w = g.pw[gp];
    double e = 0.0, a = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
    if (w != 0.0 && rho > rho_cut) {
        const double gam = gx * gx + gy * gy + gz * gz;
        const XcOut o = eval_functional(fn, rho, rho, gam, gam, gam);
        e = w * o.f;
        a = 0.5 * w * o.va;
        if (GGA) {
            const double cc = w * (2.0 * o.vgaa + o.vgab);
            cx = cc * gx, cy = cc * gy, cz = cc * gz;
        }
    }
    double* cf = coef + gp * 4;
    cf[0] = a, cf[1] = cx, cf[2] = cy, cf[3] = cz;
    // Z[nu][p] = 0.5 w vrho phi + c . grad phi, written over X (no longer needed), all nbp rows
    double* Z = const_cast<double*>(X);
    for (int r = 0; r < m.nbp; ++r) {
        const size_t o = (size_t)r * BLOCK_PTS + p;
        double z = a * phi[o];
        if (GGA) z += cx * phi[plane + o] + cy * phi[2 * plane + o] + cz * phi[3 * plane + o];
        Z[o] = z;
    }
    // block sums in FP64 (deterministic order)
    __shared__ double red[2][BLOCK_PTS / 32];
    double se = warp_sum(e), sn = warp_sum(w * rho);
    if ((p & 31) == 0) red[0][p >> 5] = se, red[1][p >> 5] = sn;
    __syncthreads();
    if (p == 0) {
        double E = 0.0, N = 0.0;
        for (int i = 0; i < BLOCK_PTS / 32; ++i) E += red[0][i], N += red[1][i];
        blk_sum[2 * blk] = E;
        blk_sum[2 * blk + 1] = N;
    }
}

// Builds without stored AO gradients. Layout of a block (doubles): phi [nbp][128], one plane per
// spin [nbp][128] (X, then Z), then, for a GGA, the radial sums S0 [nsh][128] and S1 [nsh][128].
// k_ao_eval_rad writes phi and the radial sums; everything that needs grad phi forms it from them
// (ao.cuh). The shells (rows, angular momenta, atoms, primitives) are staged in shared memory, 64 at a
// time. (k_ao_eval above, with stored gradients, serves the no-allocation build alone.)
// NR: the radial sums stored, 0 (an LDA: phi only), 2, or 3 with S2 = sum_k c_k a_k^2 e^{-a_k r^2}
// ([nsh][128] after S1, for second derivatives).
template <int NR>
__global__ void __launch_bounds__(256) k_ao_eval_rad(BasisView bas, GridView g, int blk0, char* ws, int rad0) {
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    const int p = threadIdx.x & (BLOCK_PTS - 1);
    const int half = threadIdx.x >> 7;
    double* phi = reinterpret_cast<double*>(ws + m.ws);
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    double* S0p = phi + rad0 * plane;
    double* S1p = S0p + (size_t)m.nsh * BLOCK_PTS;
    const int gp = blk * BLOCK_PTS + p;
    const double rx = g.px[gp], ry = g.py[gp], rz = g.pz[gp];
    __shared__ ShellRec recs[64];  // the block's shells, 64 at a time
    for (int i0 = 0; i0 < m.nsh; i0 += 64) {
        __syncthreads();
        for (int k = threadIdx.x; k < 64 && i0 + k < m.nsh; k += blockDim.x)
            stage_shell(bas, g.blk_shells[m.sh0 + i0 + k], g.blk_shell_row[m.sh0 + i0 + k], recs[k]);
        __syncthreads();
        for (int i = i0 + half; i < min(i0 + 64, m.nsh); i += 2) {
            const ShellRec& r = recs[i - i0];
            const double x = rx - r.ax, y = ry - r.ay, z = rz - r.az;
            const int L = r.lq, n = 2 * L + 1;
            double S0, S1 = 0.0, S2 = 0.0;
            if (NR == 3) shell_radial2_staged(bas, r, x * x + y * y + z * z, S0, S1, S2);
            else shell_radial_staged<NR != 0>(bas, r, x * x + y * y + z * z, S0, S1);
            if (NR >= 2) S0p[(size_t)i * BLOCK_PTS + p] = S0, S1p[(size_t)i * BLOCK_PTS + p] = S1;
            if (NR == 3) S1p[(size_t)(m.nsh + i) * BLOCK_PTS + p] = S2;
            for (int c = 0; c < n; ++c) {
                double v, gx, gy, gz;
                ao_from_radial<false>(L * L + c, x, y, z, S0, S1, v, gx, gy, gz);
                phi[(size_t)(r.row0 + c) * BLOCK_PTS + p] = v;
            }
        }
    }
}

struct ShellStage {
    double ax[128], ay[128], az[128];
    int row0[128], lq[128];
};

__device__ __forceinline__ void stage_shells(const BasisView& bas, const GridView& g, const BlockMeta& m, int i0,
                                             ShellStage& st) {
    for (int k = threadIdx.x; k < 128 && i0 + k < m.nsh; k += blockDim.x) {
        const int s = g.blk_shells[m.sh0 + i0 + k];
        const int a = bas.sh_atom[s];
        st.ax[k] = bas.atom_xyz[3 * a], st.ay[k] = bas.atom_xyz[3 * a + 1], st.az[k] = bas.atom_xyz[3 * a + 2];
        st.row0[k] = g.blk_shell_row[m.sh0 + i0 + k];
        st.lq[k] = bas.sh_l[s];
    }
}

// Prefetch into L1 of the line holding p (no wait, no register).
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// The passes over the radial sums: 256 threads per block, the point is threadIdx.x % 128, the two
// halves of the CTA take alternate shells. Bound by HBM; what a thread itself can keep in flight (one
// shell's loads) is a third of what the bandwidth needs at 24 warps per SM, so the lines of the shell
// kRadAhead shells on are prefetched into L1.
constexpr int kRadAhead = 8;

// rho and sum grad phi X per point of one spin (X in plane xplane, sums to acc_a) or both (xplane + 1,
// acc_b; one pass over the radial sums). 100-atom ULTRA_FINE build: 2.8 ms (128 threads per block, no
// prefetch: 3.0).
template <int NS>
__global__ void __launch_bounds__(256, 3) k_rho_rad(BasisView bas, GridView g, int blk0, const char* ws, int xplane,
                                                    int rad0, double* acc_a, double* acc_b) {
    __shared__ ShellStage st;
    __shared__ double s_half[NS][4][BLOCK_PTS];
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    const int p = threadIdx.x & (BLOCK_PTS - 1), half = threadIdx.x >> 7;
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    const double* X = reinterpret_cast<const double*>(ws + m.ws) + xplane * plane + p;
    const double* S0p = reinterpret_cast<const double*>(ws + m.ws) + rad0 * plane + p;
    const double* S1p = S0p + (size_t)m.nsh * BLOCK_PTS;
    const size_t gp = (size_t)blk * BLOCK_PTS + p;
    const double px = g.px[gp], py = g.py[gp], pz = g.pz[gp];
    double sum[NS][4];
#pragma unroll
    for (int s = 0; s < NS; ++s) sum[s][0] = sum[s][1] = sum[s][2] = sum[s][3] = 0.0;
    for (int i0 = 0; i0 < m.nsh; i0 += 128) {
        __syncthreads();
        stage_shells(bas, g, m, i0, st);
        __syncthreads();
        const int kn = min(128, m.nsh - i0);
        for (int k = half; k < kn; k += 2) {
            if (k + kRadAhead < kn) {
                const int ka = k + kRadAhead, na = 2 * st.lq[ka] + 1;
                prefetch_l1(S0p + (size_t)(i0 + ka) * BLOCK_PTS);
                prefetch_l1(S1p + (size_t)(i0 + ka) * BLOCK_PTS);
                for (int c = 0; c < na; ++c)
#pragma unroll
                    for (int s = 0; s < NS; ++s) prefetch_l1(X + s * plane + (size_t)(st.row0[ka] + c) * BLOCK_PTS);
            }
            const int L = st.lq[k], row0 = st.row0[k];
            const double S0 = S0p[(size_t)(i0 + k) * BLOCK_PTS], S1 = S1p[(size_t)(i0 + k) * BLOCK_PTS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                double xv[5];
#pragma unroll
                for (int c = 0; c < 5; ++c) xv[c] = c < 2 * L + 1 ? X[s * plane + (size_t)(row0 + c) * BLOCK_PTS] : 0.0;
                shell_rho<true>(L, px - st.ax[k], py - st.ay[k], pz - st.az[k], S0, S1, xv, sum[s][0], sum[s][1],
                                sum[s][2], sum[s][3]);
            }
        }
    }
    if (half)
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int k = 0; k < 4; ++k) s_half[s][k][p] = sum[s][k];
    __syncthreads();
    if (!half)
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int k = 0; k < 4; ++k) (s ? acc_b : acc_a)[gp * 4 + k] = sum[s][k] + s_half[s][k][p];
}

// Z[nu][p] = 0.5 w vrho phi + c . grad phi for one spin (plane zplane, over X) or both (zplane + 1).
// 100-atom ULTRA_FINE build: 2.35 ms (128 threads per block, no prefetch: 3.55).
template <int NS>
__global__ void __launch_bounds__(256, 3) k_z_rad(BasisView bas, GridView g, int blk0, const double* coef_a,
                                                  const double* coef_b, char* ws, int zplane, int rad0) {
    __shared__ ShellStage st;
    const int blk = blk0 + blockIdx.x;
    const BlockMeta m = g.meta[blk];
    const int p = threadIdx.x & (BLOCK_PTS - 1), half = threadIdx.x >> 7;
    const size_t plane = (size_t)m.nbp * BLOCK_PTS;
    double* Z = reinterpret_cast<double*>(ws + m.ws) + zplane * plane + p;
    const double* S0p = reinterpret_cast<const double*>(ws + m.ws) + rad0 * plane + p;
    const double* S1p = S0p + (size_t)m.nsh * BLOCK_PTS;
    const size_t gp = (size_t)blk * BLOCK_PTS + p;
    const double px = g.px[gp], py = g.py[gp], pz = g.pz[gp];
    double cf[NS][4];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int k = 0; k < 4; ++k) cf[s][k] = (s ? coef_b : coef_a)[gp * 4 + k];
    for (int i0 = 0; i0 < m.nsh; i0 += 128) {
        __syncthreads();
        stage_shells(bas, g, m, i0, st);
        __syncthreads();
        const int kn = min(128, m.nsh - i0);
        for (int k = half; k < kn; k += 2) {
            if (k + kRadAhead < kn) {
                prefetch_l1(S0p + (size_t)(i0 + k + kRadAhead) * BLOCK_PTS);
                prefetch_l1(S1p + (size_t)(i0 + k + kRadAhead) * BLOCK_PTS);
            }
            const int L = st.lq[k], row0 = st.row0[k];
            const double S0 = S0p[(size_t)(i0 + k) * BLOCK_PTS], S1 = S1p[(size_t)(i0 + k) * BLOCK_PTS];
            const double x = px - st.ax[k], y = py - st.ay[k], z = pz - st.az[k];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                double zc[5];
                shell_z(L, x, y, z, S0, S1, cf[s][0], cf[s][1], cf[s][2], cf[s][3], zc);
#pragma unroll
                for (int c = 0; c < 5; ++c)
                    if (c < 2 * L + 1) Z[s * plane + (size_t)(row0 + c) * BLOCK_PTS] = zc[c];
            }
        }
    }
}

// Vacc[aos[m]][aos[n]] += sum_p phi[m][p] Z[n][p]: CTA tile up to 64 x 64 AOs (fp64_tile in both
// dimensions), K = 128 points in steps of 16 through two shared-memory stages, 4 warps as 2 x 2 of up
// to 4 x 4 DMMA tiles. Bound by the FP64 tensor pipe; two stages and 128 registers let four CTAs share
// an SM, which hide one another's first loads and atomics (three CTAs of three stages: a 100-atom build
// 21.8 ms against 20.9; a persistent form with the ring running on across tiles was slower still). A tile of
// an odd number of rows of eight gives its first warps more work, and a warp stays on its quarter of the
// SM, so the warps' places in the tile rotate with the CTA. Rows at nb and beyond are not read.
// LDA: Z = a phi with a = 0.5 w vrho per point, so there is no Z plane: B is phi again, scaled by a as
// its fragments are loaded, and phi diag(a) phi^T is symmetric: only the tiles tm <= tn are computed
// (the list ltiles), those off the diagonal counted twice (the finish adds Vacc^T).
constexpr int GV_B = 64, GV_BK = 16, GV_S = 2, GV_AS = GV_BK + 4;
constexpr int GV_STAGE = 2 * GV_B * GV_AS;  // doubles: A [m][k], B [n][k]
constexpr int GV_SMEM = GV_S * GV_STAGE * 8;

template <bool LDA, int MI, int NJ>
__device__ __forceinline__ void gv_step(const double* As, const double* Bs, const double* av, double (&acc)[4][4][2]) {
#pragma unroll
    for (int kk = 0; kk < GV_BK; kk += 4) {
        double a[MI], b[NJ];
#pragma unroll
        for (int i = 0; i < MI; ++i) a[i] = As[i * 8 * GV_AS + kk];
#pragma unroll
        for (int j = 0; j < NJ; ++j) b[j] = LDA ? av[kk] * Bs[j * 8 * GV_AS + kk] : Bs[j * 8 * GV_AS + kk];
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
}
template <bool LDA, int MI>
__device__ __forceinline__ void gv_step_n(int nj, const double* As, const double* Bs, const double* av,
                                          double (&acc)[4][4][2]) {
    switch (nj) {
        case 4: gv_step<LDA, MI, 4>(As, Bs, av, acc); break;
        case 3: gv_step<LDA, MI, 3>(As, Bs, av, acc); break;
        case 2: gv_step<LDA, MI, 2>(As, Bs, av, acc); break;
        case 1: gv_step<LDA, MI, 1>(As, Bs, av, acc); break;
        default: break;
    }
}

template <bool LDA>
__global__ void __launch_bounds__(128, 4) k_gemm_v(GridView g, int blk0, char* ws, int zplane, const double* coef,
                                                double* Vacc, int nao, int tiles, int64_t t0) {
    extern __shared__ __align__(16) double gv_sm[];
    __shared__ double s_a[LDA ? BLOCK_PTS : 1];
    int blk, tm, tn;
    if (LDA || g.vtiles) {  // one CTA per tile of the list
        const int2 it = (LDA ? g.ltiles : g.vtiles)[t0 + blockIdx.x];
        blk = it.x, tm = it.y >> 16, tn = it.y & 0xFFFF;
    } else {
        blk = blk0 + blockIdx.y, tm = blockIdx.x / tiles, tn = blockIdx.x % tiles;
    }
    const BlockMeta m = g.meta[blk];
    const int T = (m.nb + 63) / 64;
    if (tm >= T || tn >= T) return;
    int mr8, mc, nr8, nc;
    fp64_tile(m.nb, T, tm, mr8, mc);
    fp64_tile(m.nb, T, tn, nr8, nc);
    const int m0 = mr8 * 8, n0 = nr8 * 8;
    const double* phi = reinterpret_cast<const double*>(ws + m.ws);
    const double* Z = LDA ? phi : phi + (size_t)zplane * m.nbp * BLOCK_PTS;
    const int* aos = g.blk_aos + m.ao0;
    const int t = threadIdx.x, lane = t & 31, warp = ((t >> 5) + blockIdx.x) & 3;
    // a (read after the first barrier of the loop), doubled for a tile that stands for its mirror too
    if (LDA) s_a[t] = coef[4 * ((size_t)blk * BLOCK_PTS + t)] * (tm == tn ? 1.0 : 2.0);
    const int gq = lane >> 2, tq = lane & 3;
    const int wm8 = (warp >> 1) * ((mc + 1) >> 1), wn8 = (warp & 1) * ((nc + 1) >> 1);  // the warp's first rows of eight
    const int mi = warp >> 1 ? mc >> 1 : (mc + 1) >> 1, nj = warp & 1 ? nc >> 1 : (nc + 1) >> 1;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto issue = [&](int kt) {  // thread: the 16-byte piece t % 8 of rows t / 8 + 16 q of both operands
        double* st = gv_sm + (kt % GV_S) * GV_STAGE;
        const int c = 2 * (t & 7);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = (t >> 3) + 16 * q;
            const bool oka = r < 8 * mc && m0 + r < m.nb, okb = r < 8 * nc && n0 + r < m.nb;
            cp_async16(st + r * GV_AS + c, phi + (oka ? (size_t)(m0 + r) * BLOCK_PTS + kt * GV_BK + c : 0), oka);
            cp_async16(st + (GV_B + r) * GV_AS + c, Z + (okb ? (size_t)(n0 + r) * BLOCK_PTS + kt * GV_BK + c : 0), okb);
        }
    };
    constexpr int nk = BLOCK_PTS / GV_BK;
#pragma unroll
    for (int k = 0; k < GV_S - 1; ++k) {
        issue(k);
        cp_async_commit();
    }
#pragma unroll 1
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<GV_S - 2>();
        __syncthreads();  // stage kt has landed for every thread, and stage kt - 1 is consumed
        if (kt + GV_S - 1 < nk) issue(kt + GV_S - 1);
        cp_async_commit();
        const double* st = gv_sm + (kt % GV_S) * GV_STAGE;
        const double* As = st + (wm8 * 8 + gq) * GV_AS + tq;
        const double* Bs = st + (GV_B + wn8 * 8 + gq) * GV_AS + tq;
        const double* av = s_a + (LDA ? kt * GV_BK + tq : 0);
        switch (mi) {  // uniform over the warp
            case 4: gv_step_n<LDA, 4>(nj, As, Bs, av, acc); break;
            case 3: gv_step_n<LDA, 3>(nj, As, Bs, av, acc); break;
            case 2: gv_step_n<LDA, 2>(nj, As, Bs, av, acc); break;
            case 1: gv_step_n<LDA, 1>(nj, As, Bs, av, acc); break;
            default: break;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = m0 + (wm8 + i) * 8 + gq;
        if (i >= mi || r >= m.nb) continue;
        const size_t rowoff = (size_t)aos[r] * nao;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = n0 + (wn8 + j) * 8 + 2 * tq;
            if (j >= nj) continue;
            if (c < m.nb) atomicAdd(&Vacc[rowoff + aos[c]], acc[i][j][0]);
            if (c + 1 < m.nb) atomicAdd(&Vacc[rowoff + aos[c + 1]], acc[i][j][1]);
        }
    }
}

__global__ void k_symmetrize(const double* __restrict__ Vacc, double* V, int nao) {
    const int64_t n2 = (int64_t)nao * nao;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n2; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / nao), j = (int)(e % nao);
        V[e] = Vacc[e] + Vacc[(int64_t)j * nao + i];
    }
}

// Deterministic FP64 sum of the per-block partials: one CTA, fixed order.
__global__ void k_block_sums(const double* __restrict__ blk_sum, int nblk, double* out) {
    __shared__ double se[256], sn[256];
    double e = 0.0, n = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) e += blk_sum[2 * b], n += blk_sum[2 * b + 1];
    se[threadIdx.x] = e, sn[threadIdx.x] = n;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) se[threadIdx.x] += se[threadIdx.x + s], sn[threadIdx.x] += sn[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = se[0], out[1] = sn[0];
}

// Per-segment (per-molecule of a batch) FP64 sums of the block partials: one CTA per
// segment, blocks [seg_blk[i], seg_blk[i+1]), the same fixed order as k_block_sums.
__global__ void k_segment_sums(const double* __restrict__ blk_sum, const int* __restrict__ seg_blk, double* out) {
    __shared__ double se[256], sn[256];
    const int b0 = seg_blk[blockIdx.x], b1 = seg_blk[blockIdx.x + 1];
    double e = 0.0, n = 0.0;
    for (int b = b0 + threadIdx.x; b < b1; b += blockDim.x) e += blk_sum[2 * b], n += blk_sum[2 * b + 1];
    se[threadIdx.x] = e, sn[threadIdx.x] = n;
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) se[threadIdx.x] += se[threadIdx.x + st], sn[threadIdx.x] += sn[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[2 * blockIdx.x] = se[0], out[2 * blockIdx.x + 1] = sn[0];
}

}  // namespace

void launch_segment_sums(const double* blk_sum, const int* seg_blk, int nseg, double* out, cudaStream_t s) {
    k_segment_sums<<<nseg, 256, 0, s>>>(blk_sum, seg_blk, out);
}

void launch_ao_eval(const BasisView& b, const GridView& g, int blk0, int nblk, bool gga, char* ws,
                    int /*max_nsh*/, cudaStream_t s) {
    if (gga)
        k_ao_eval<true><<<nblk, 256, 0, s>>>(b, g, blk0, ws);
    else
        k_ao_eval<false><<<nblk, 256, 0, s>>>(b, g, blk0, ws);
}

void launch_gemm_x(const GridView& g, const double* P, int nao, int blk0, int nblk, int max_nbp,
                          int nplanes, char* ws, cudaStream_t s) {
    // X follows the phi planes (1 for LDA, 4 with gradients)
    launch_gemm_x_plane(g, P, nao, blk0, nblk, max_nbp, 0, nplanes, ws, s);
}

template <int MODE>
static void run_gemm_x(const GridView& g, const double* P, int nao, int blk0, int nblk, int max_nbp, int src0, int dst0,
                       int sum0, char* ws, cudaStream_t s) {
    cudaFuncSetAttribute(k_gemm_x<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, GX_SMEM);
    if (g.xtiles && g.h_xtile0) {
        const int64_t t0 = g.h_xtile0[blk0], n = g.h_xtile0[blk0 + nblk] - t0;
        if (n > 0) k_gemm_x<MODE><<<(unsigned)n, 256, GX_SMEM, s>>>(g, P, nao, blk0, ws, src0, dst0, sum0, t0);
        return;
    }
    dim3 grid((max_nbp + GX_BM - 1) / GX_BM, nblk);
    k_gemm_x<MODE><<<grid, 256, GX_SMEM, s>>>(g, P, nao, blk0, ws, src0, dst0, sum0, 0);
}

void launch_gemm_x_plane(const GridView& g, const double* P, int nao, int blk0, int nblk, int max_nbp, int src, int dst,
                         char* ws, cudaStream_t s) {
    run_gemm_x<X_STORE>(g, P, nao, blk0, nblk, max_nbp, src, dst, 0, ws, s);
}

void launch_gemm_x_lda(const GridView& g, const double* P, int nao, int blk0, int nblk, int xplane, int sum0, char* ws,
                       cudaStream_t s) {
    if (xplane >= 0) run_gemm_x<X_PHI | X_STORE>(g, P, nao, blk0, nblk, 0, 0, xplane, sum0, ws, s);
    else run_gemm_x<X_PHI>(g, P, nao, blk0, nblk, 0, 0, 0, sum0, ws, s);
}

void launch_rho_rad(const BasisView& b, const GridView& g, int blk0, int nblk, int xplane, int rad0, const char* ws,
                    double* acc_a, double* acc_b, cudaStream_t s) {
    if (acc_b)
        k_rho_rad<2><<<nblk, 256, 0, s>>>(b, g, blk0, ws, xplane, rad0, acc_a, acc_b);
    else
        k_rho_rad<1><<<nblk, 256, 0, s>>>(b, g, blk0, ws, xplane, rad0, acc_a, nullptr);
}

void launch_ao_eval_rad(const BasisView& b, const GridView& g, int blk0, int nblk, int rad0, int nrad, char* ws,
                        cudaStream_t s) {
    if (nrad == 0) k_ao_eval_rad<0><<<nblk, 256, 0, s>>>(b, g, blk0, ws, rad0);
    else if (nrad == 2) k_ao_eval_rad<2><<<nblk, 256, 0, s>>>(b, g, blk0, ws, rad0);
    else k_ao_eval_rad<3><<<nblk, 256, 0, s>>>(b, g, blk0, ws, rad0);
}

void launch_z_rad(const BasisView& b, const GridView& g, int blk0, int nblk, const double* coef_a, const double* coef_b,
                  int zplane, int rad0, char* ws, cudaStream_t s) {
    if (coef_b)
        k_z_rad<2><<<nblk, 256, 0, s>>>(b, g, blk0, coef_a, coef_b, ws, zplane, rad0);
    else
        k_z_rad<1><<<nblk, 256, 0, s>>>(b, g, blk0, coef_a, nullptr, ws, zplane, rad0);
}

void launch_rho_functional(const GridView& g, int blk0, int nblk, int fn, bool incremental, double rho_cut,
                           char* ws, double* rho, double* coef, double* blk_sum, cudaStream_t s) {
    if (functional_is_gga(fn))
        k_rho_functional<true><<<nblk, BLOCK_PTS, 0, s>>>(g, blk0, fn, incremental, rho_cut, ws, rho, coef, blk_sum);
    else
        k_rho_functional<false><<<nblk, BLOCK_PTS, 0, s>>>(g, blk0, fn, incremental, rho_cut, ws, rho, coef, blk_sum);
}

void launch_gemm_v(const GridView& g, int blk0, int nblk, int max_nbp, bool gga, const double* coef, char* ws,
                   double* Vacc, int nao, cudaStream_t s) {
    (void)coef;
    launch_gemm_v_plane(g, blk0, nblk, max_nbp, gga ? 4 : 1, ws, Vacc, nao, s);
}

void launch_gemm_v_plane(const GridView& g, int blk0, int nblk, int max_nbp, int zplane, char* ws, double* Vacc,
                         int nao, cudaStream_t s) {
    const int tiles = (max_nbp + GV_B - 1) / GV_B;
    cudaFuncSetAttribute(k_gemm_v<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GV_SMEM);
    if (g.vtiles && g.h_vtile0) {
        const int64_t t0 = g.h_vtile0[blk0], n = g.h_vtile0[blk0 + nblk] - t0;
        if (n > 0)
            k_gemm_v<false><<<(unsigned)n, 128, GV_SMEM, s>>>(g, blk0, ws, zplane, nullptr, Vacc, nao, tiles, t0);
        return;
    }
    dim3 grid(tiles * tiles, nblk);
    k_gemm_v<false><<<grid, 128, GV_SMEM, s>>>(g, blk0, ws, zplane, nullptr, Vacc, nao, tiles, 0);
}

void launch_gemm_v_lda(const GridView& g, int blk0, int nblk, const double* coef, char* ws, double* Vacc, int nao,
                       cudaStream_t s) {
    cudaFuncSetAttribute(k_gemm_v<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GV_SMEM);
    const int64_t t0 = g.h_ltile0[blk0], n = g.h_ltile0[blk0 + nblk] - t0;
    if (n > 0) k_gemm_v<true><<<(unsigned)n, 128, GV_SMEM, s>>>(g, blk0, ws, 0, coef, Vacc, nao, 0, t0);
}

void launch_block_sums(const double* blk_sum, int nblk, double* scalars, cudaStream_t s) {
    k_block_sums<<<1, 256, 0, s>>>(blk_sum, nblk, scalars);
}

// dV = V - Vprev (or V with no previous iteration), then Vprev = V: the XC part of
// DfFockMatrix::setXC_DIRECT (src/libpdf/DfFockMatrix.h:711-721) on the device.
__global__ void k_fock_delta(const double* __restrict__ V, double* Vprev, double* __restrict__ dV, size_t n,
                             int has_prev) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = V[i];
        dV[i] = has_prev ? v - Vprev[i] : v;
        Vprev[i] = v;
    }
}

void launch_fock_delta(const double* V, double* Vprev, double* dV, size_t n, bool has_prev, cudaStream_t s) {
    k_fock_delta<<<148 * 8, 256, 0, s>>>(V, Vprev, dV, n, has_prev ? 1 : 0);
}

// The upper triangle of a symmetric n x n matrix packed row by row: (i, j >= i) at
// i n - i (i - 1) / 2 + (j - i). One CTA per row; the reads and writes along j are coalesced.
__global__ void k_pack_upper(const double* __restrict__ V, int n, double* __restrict__ packed) {
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int64_t o = (int64_t)i * n - (int64_t)i * (i - 1) / 2 - i;
        for (int j = i + threadIdx.x; j < n; j += blockDim.x) packed[o + j] = V[(int64_t)i * n + j];
    }
}

// Both triangles from the packed upper triangle, in 32 x 32 tiles: a tile on or above the
// diagonal copies packed rows; a tile below it reads its mirror tile's packed rows (coalesced)
// into shared memory and writes the transpose.
__global__ void k_unpack_upper(const double* __restrict__ packed, int n, double* __restrict__ V) {
    __shared__ double t[32][33];
    const int nt = (n + 31) / 32;
    for (int64_t tile = blockIdx.x; tile < (int64_t)nt * nt; tile += gridDim.x) {
        const int ti = (int)(tile / nt), tj = (int)(tile % nt);
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
        if (ti <= tj) {
            for (int r = ty; r < 32; r += 8) {
                const int i = ti * 32 + r, j = tj * 32 + tx;
                if (i < n && j < n) {
                    const int a = min(i, j), b = max(i, j);
                    V[(int64_t)i * n + j] = packed[(int64_t)a * n - (int64_t)a * (a - 1) / 2 + (b - a)];
                }
            }
        } else {
            // rows tj*32.. of the mirror tile (row index < column index: the packed upper part)
            for (int r = ty; r < 32; r += 8) {
                const int a = tj * 32 + r, b = ti * 32 + tx;
                if (a < n && b < n) t[r][tx] = packed[(int64_t)a * n - (int64_t)a * (a - 1) / 2 + (b - a)];
            }
            __syncthreads();
            for (int r = ty; r < 32; r += 8) {
                const int i = ti * 32 + r, j = tj * 32 + tx;
                if (i < n && j < n) V[(int64_t)i * n + j] = t[tx][r];
            }
            __syncthreads();
        }
    }
}

void launch_pack_upper(const double* V, int n, double* packed, cudaStream_t s) {
    k_pack_upper<<<148 * 8, 256, 0, s>>>(V, n, packed);
}

void launch_unpack_upper(const double* packed, int n, double* V, cudaStream_t s) {
    k_unpack_upper<<<148 * 8, 256, 0, s>>>(packed, n, V);
}

void launch_finish(const double* Vacc, double* V, int nao, const double* blk_sum, int nblk, double* scalars,
                   cudaStream_t s) {
    k_symmetrize<<<148 * 8, 256, 0, s>>>(Vacc, V, nao);
    k_block_sums<<<1, 256, 0, s>>>(blk_sum, nblk, scalars);
}

}  // namespace pdfxc
