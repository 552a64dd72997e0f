// msod_mixed_diffu.cu -- mixed-precision hex GLL diffusion residual on the tensor cores.
//
// Same residuals as full_diffusion_ijk (elem_diffu.f90:10-197; formulas in
// msod_diffu.cu) from FP32 fields, with the 1-D contractions on the tensor
// cores as FP16 (or BF16) hi + lo split products (FP32 accumulation) and the
// energy-flux assembly and the nodal scatter-add in FP64 (FP64 outputs).
//
// Per element (one block of one warp per tile, persistent over elements):
//   1. gather rho, T, u, mu_fluid, mu_e, mu_sgs, He, gpvol of the thread's two points;
//   2. gradient stage: rho, T, u_1..3 are shifted by their value at lattice
//      node (0,0,0) (the derivative annihilates constants), scaled by a power
//      of two per element and field, split into hi + lo half planes; per
//      direction, two accumulating mma.sync.m16n8k16 per two fields and 8 lines
//      (A = [f_hi | f_lo], B = [D_hi^T ; D_hi^T] then [D_lo^T ; 0]) give the
//      15 iso-parametric derivatives per point;
//   3. point pass: physical gradients, stress tau, tau.u and the contravariant
//      fluxes gpvol He(:,d)^T X of X = grad rho, tau.u, grad T, tau rows
//      (18 per point), plus nu_e and kappa_e per output node
//      (elem_diffu.f90:143-146); each flux is shifted by its value X_ref at
//      lattice node (0,0,0), scaled per element and flux, and split into half
//      planes;
//   4. weak divergence: per direction, the transposed 1-D operator
//      (B = [D_hi ; D_hi] then [D_lo ; 0], indexed (input, output)) on the six
//      shifted fluxes of that direction, plus X_ref times the operator's
//      column sum (evaluated in FP64 once per block); six sums per point
//      accumulated over the directions in shared memory;
//   5. Rmass += nu_e sum(grad rho), Rmom_m += sum(tau_m), and in FP64
//      Rener += sum(tau.u) + kappa_e sum(grad T); red.global.add.f64.
// Shared-memory half planes use the swizzled layout of msod_mma.cuh.
// porder 1..7.  One tile per warp, as in msod_mixed.cu; a thread's two points stay in
// its registers from the gather to the point pass.  Two tiles per warp in blocks of
// four warps / one tile per warp / now, FP16: porder 7 24^3 0.851 / 0.706 / 0.635 ms,
// 6 32^3 1.555 / 1.444 / 1.311, 5 40^3 1.996 / 1.776 / 1.742, 4 48^3 2.164 / 2.114 /
// 2.182, 3 48^3 1.620 / 1.530 / 1.533, 2 64^3 3.508 / 2.434 / 2.736, 1 64^3 3.377 /
// 1.718 / 1.741.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "msod_device.cuh"
#include "msod_kernels.h"
#include "msod_mma.cuh"

namespace msod {
namespace {

constexpr int kNG = 5;   // differentiated node fields: rho, T, u_1..3
constexpr int kNX = 6;   // flux vectors: grad rho, tau.u, grad T, tau rows 1..3
constexpr int kNFX = 3 * kNX;

constexpr int kFx0 = 8;  // scale of the first flux, behind the node fields'
enum { X_GRHO = 0, X_TAUU, X_GT, X_TAU0, X_TAU1, X_TAU2 };

template <int P, bool BF16>
struct MixedDiffuGeom {
    static constexpr int Q = P + 1, N = Q * Q * Q, W = (Q + 1) / 2, NP = node_plane<Q>();
    static constexpr int NT = 32 * Q;        // one warp per tile (k-plane or j-plane) of lines
    static constexpr int NTASK = Q * Q * W;  // task: points (2w, 2w+1) of one i-row
    static_assert(NTASK <= NT, "one task per thread");
    static constexpr int BITS = BF16 ? 8 : 11;
    static constexpr int PB = plane_bytes<Q>();  // bytes of one field half
    static constexpr size_t half_bytes = (size_t)2 * kNFX * PB;
    static constexpr size_t smem = half_bytes + (size_t)(3 * kNG + 2) * NP * sizeof(float) +
                                   (size_t)2 * NP * sizeof(int) + (3 * 32 + 8) * sizeof(float);
    // Blocks per SM that shared memory allows, as long as a thread keeps kMixedRegs registers.
    static constexpr int MINB = mixed_blocks(smem, NT, kMixedRegs);
};

template <int P, bool BF16, bool NUE>
__global__ void __launch_bounds__(32 * (P + 1), MixedDiffuGeom<P, BF16>::MINB)
    diffu_mixed_kernel(int nelem, int npoin, const int *__restrict__ connec, const float *__restrict__ He,
                       const float *__restrict__ gpvol, const int *__restrict__ inv,
                       const float *__restrict__ dlxigp_ip, float Cp, float Pr,
                       const float *__restrict__ rho, const float *__restrict__ u, const float *__restrict__ Tem,
                       const float *__restrict__ mu_fluid, const float *__restrict__ mu_e,
                       const float *__restrict__ mu_sgs, const float *__restrict__ nu_elem,
                       double *__restrict__ Rmass, double *__restrict__ Rmom, double *__restrict__ Rener)
{
    using G = MixedDiffuGeom<P, BF16>;
    constexpr int Q = G::Q, N = G::N, W = G::W, NTASK = G::NTASK, NT = G::NT, NP = G::NP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *sHalf = smem_raw;                                  // [2*kNFX][G::PB]
    float *sG = reinterpret_cast<float *>(sHalf + G::half_bytes);     // [15][NP] iso-derivatives; then [6][NP] sums
    float *sNK = sG + 3 * kNG * NP;                                    // [2][NP] nu_e, kappa_e
    int *sNode = reinterpret_cast<int *>(sNK + 2 * NP);                // [NP], positions node_at
    int *sPerm = sNode + NP;                                           // gmsh node
    float *sScale = reinterpret_cast<float *>(sPerm + NP);            // [32]: 0..4 node fields, kFx0.. fluxes
    float *sInv = sScale + 32;
    unsigned *sMax = reinterpret_cast<unsigned *>(sInv);
    float *sRef = sInv + 32;  // [kNFX] flux values at lattice node (0,0,0)
    float *sRefG = sRef + 32;  // [kNG] node fields there

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;
    for (int i = tid; i < N; i += NT) sPerm[node_at<Q>(i / (Q * Q), i / Q % Q, i % Q)] = table_node<Q>(inv, i);
    if (Q < 8) {  // rows and points beyond Q are never written and stay zero
        uint4 *z = reinterpret_cast<uint4 *>(sHalf);
        for (int i = tid; i < (int)(G::half_bytes / 16); i += NT) z[i] = make_uint4(0, 0, 0, 0);
    }
    // B fragments per direction.  Gradient: B[k][n] = D[n][k]; divergence:
    // B[k][n] = D[k][n] (k input point, n output point); hi and lo halves.
    unsigned Bgh[3], Bgl[3], Bdh[3], Bdl[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int c0 = 2 * tq, c1 = c0 + 1;
        auto D = [&](int r, int c) { return table_D<Q>(inv, dlxigp_ip, d, r, c); };
        split_pair<BF16>((g < Q && c0 < Q) ? D(g, c0) : 0.0f, (g < Q && c1 < Q) ? D(g, c1) : 0.0f,
                         Bgh[d], Bgl[d]);
        split_pair<BF16>((g < Q && c0 < Q) ? D(c0, g) : 0.0f, (g < Q && c1 < Q) ? D(c1, g) : 0.0f,
                         Bdh[d], Bdl[d]);
    }
    // Column sums of the divergence operator at the thread's output points 2t, 2t+1.
    float colsum[3][2];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int a = 2 * tq + h;
            double cs = 0.0;
            if (a < Q)
                for (int c = 0; c < Q; ++c) cs += (double)table_D<Q>(inv, dlxigp_ip, d, c, a);
            colsum[d][h] = (float)cs;
        }
    // ldmatrix matrix m of the A operand is (hi f, hi f+1, lo f, lo f+1), row r8
    // of tile w = warp; a field that stands alone is loaded twice.
    const int m = lane >> 3, r8 = lane & 7;
    const int alone = (m & 1) * 2 * G::PB, plane_off = alone + (m >> 1) * G::PB;
    // The thread's task of the split and the point pass: points (2w, 2w+1) of i-row `row`.
    const bool valid = tid < NTASK;
    const int row = valid ? tid / W : 0, w = valid ? tid - row * W : 0;
    const int row_off = row_pos(row / Q, row % Q) * kRowB + 4 * w;
    const bool two = valid && 2 * w + 1 < Q;
    const int l0 = node_at<Q>(row / Q, row % Q, 2 * w);
    const int a0 = table_node<Q>(inv, row * Q + 2 * w), a1 = table_node<Q>(inv, row * Q + 2 * w + (two ? 1 : 0));
    // Node ids, loaded an element ahead (the grid has nelem blocks at most).
    int id[2] = {ldg_once(connec + (size_t)a0 * nelem + blockIdx.x), ldg_once(connec + (size_t)a1 * nelem + blockIdx.x)};
    const size_t np = (size_t)npoin;
    const float twoThirds = 2.0f / 3.0f;

#pragma unroll 1
    for (int e = blockIdx.x; e < nelem; e += gridDim.x) {
        const float nue = NUE ? ldg(nu_elem + e) : 0.0f;
        // The thread's two points: node fields, viscosities, He and gpvol, kept in registers.
        float fld[2][kNG], muf[2], mue[2], mus[2], hv[2][9], gv[2];
        int node[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int a = h ? a1 : a0, v = id[h] - 1;
            const bool ok = (h ? two : valid) && (unsigned)v < (unsigned)npoin;
            const size_t p = ok ? v : 0;
            node[h] = ok ? v : -1;
            fld[h][0] = ok ? ldg_once(rho + p) : 1.0f;  // 1 at a missing node keeps nu_e = mu_e / rho finite
            fld[h][1] = ok ? ldg_once(Tem + p) : 0.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c) fld[h][2 + c] = ok ? ldg_once(u + c * np + p) : 0.0f;
            muf[h] = ok ? ldg_once(mu_fluid + p) : 0.0f;
            mue[h] = NUE ? nue : ldg(mu_e + (size_t)a * nelem + e);
            mus[h] = ldg(mu_sgs + (size_t)a * nelem + e);
            const size_t base = (size_t)e * N + a;
#pragma unroll
            for (int j = 0; j < 9; ++j) hv[h][j] = ldg(He + base * 9 + j);
            gv[h] = ldg(gpvol + base);
        }
        {
            const int en = e + (int)gridDim.x < nelem ? e + (int)gridDim.x : e;
            id[0] = ldg_once(connec + (size_t)a0 * nelem + en);
            id[1] = ldg_once(connec + (size_t)a1 * nelem + en);
        }
        __syncthreads();  // the previous element is done with every shared array
        if (tid < 32) sMax[tid] = 0u;
        if (valid) sNode[l0] = node[0];
        if (two) sNode[l0 + 1] = node[1];
        if (tid == 0)  // task 0, first point: lattice node (0,0,0)
#pragma unroll
            for (int f = 0; f < kNG; ++f) sRefG[f] = fld[0][f];
        __syncthreads();

        // ---- gradient stage: split rho, T, u_1..3 (shifted by node (0,0,0)) ----
        {
            float v[kNG][2];
#pragma unroll
            for (int f = 0; f < kNG; ++f) {
                const float ref = sRefG[f];
                v[f][0] = valid ? __fsub_rn(fld[0][f], ref) : 0.0f;
                v[f][1] = two ? __fsub_rn(fld[1][f], ref) : 0.0f;
                const float mx = fmaxf(0.0f, fmaxf(fabsf(v[f][0]), fabsf(v[f][1])));
                const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
                if (lane == 0) atomicMax(&sMax[f], mb);
            }
            __syncthreads();
            if (tid < kNG) scale_from_max(sMax[tid], G::BITS, sScale[tid], sInv[tid]);
            __syncthreads();
            if (valid) {
#pragma unroll
                for (int f = 0; f < kNG; ++f) {
                    const float s = sScale[f];
                    unsigned hi, lo;
                    split_scaled<BF16>(__fmul_rn(v[f][0], s), __fmul_rn(v[f][1], s), hi, lo);
                    *reinterpret_cast<unsigned *>(sHalf + (2 * f) * G::PB + row_off) = hi;
                    *reinterpret_cast<unsigned *>(sHalf + (2 * f + 1) * G::PB + row_off) = lo;
                }
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            const unsigned bh = d == 0 ? Bgh[0] : (d == 1 ? Bgh[1] : Bgh[2]);
            const unsigned bl = d == 0 ? Bgl[0] : (d == 1 ? Bgl[1] : Bgl[2]);
            const unsigned char *rowp = sHalf + plane_off + operand_row<Q>(d, warp, r8);
            int lat[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) lat[s] = pass_point<Q>(d, s, g, tq, warp);
#pragma unroll
            for (int f = 0; f < kNG; f += 2) {
                const unsigned char *src = rowp + 2 * f * G::PB - (f + 1 < kNG ? 0 : alone);
                unsigned a[4];
                if (d == 0)
                    ldsm_x4(a, src);
                else
                    ldsm_x4_t(a, src);
                float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma_acc<BF16>(c, a, bh, bh);
                mma_acc<BF16>(c, a, bl, 0u);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (f + k >= kNG) break;
                    const float inv = sInv[f + k];
#pragma unroll
                    for (int s = 0; s < 2; ++s)
                        if (lat[s] >= 0) sG[(d * kNG + f + k) * NP + lat[s]] = c[2 * k + s] * inv;
                }
            }
        }
        __syncthreads();

        // ---- point pass: stress, fluxes, nu_e, kappa_e; flux maxima ----
        {
            float fl[2][kNFX];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool live = h ? two : valid;
                const int l = live ? l0 + h : 0;
                float gi[3][kNG];
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int f = 0; f < kNG; ++f) gi[d][f] = sG[(d * kNG + f) * NP + l];
                const float r = fld[h][0], me = NUE ? r * mue[h] : mue[h], ms = mus[h];
                const float(&uu)[5] = fld[h];  // u at 2..4
                const float(&Hm)[9] = hv[h];  // Hm[j*3+i] = He(i, j)
                float gR[3], gT[3], gU[3][3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    gR[i] = Hm[i] * gi[0][0] + Hm[3 + i] * gi[1][0] + Hm[6 + i] * gi[2][0];
                    gT[i] = Hm[i] * gi[0][1] + Hm[3 + i] * gi[1][1] + Hm[6 + i] * gi[2][1];
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        gU[i][j] = Hm[j] * gi[0][2 + i] + Hm[3 + j] * gi[1][2 + i] + Hm[6 + j] * gi[2][2 + i];
                }
                const float mu_fgp = muf[h] + r * ms;
                const float mu_tot = mu_fgp + me;
                const float divU = gU[0][0] + gU[1][1] + gU[2][2];
                float tau[3][3], tauU[3];
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) tau[i][j] = mu_tot * (gU[i][j] + gU[j][i]);
#pragma unroll
                for (int i = 0; i < 3; ++i) tau[i][i] -= mu_fgp * twoThirds * divU;
#pragma unroll
                for (int i = 0; i < 3; ++i) tauU[i] = tau[i][0] * uu[2] + tau[i][1] * uu[3] + tau[i][2] * uu[4];
                const float *Xv[kNX] = {gR, tauU, gT, tau[0], tau[1], tau[2]};
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int x = 0; x < kNX; ++x) {
                        const float val =
                            live ? gv[h] * (Hm[d * 3] * Xv[x][0] + Hm[d * 3 + 1] * Xv[x][1] +
                                                Hm[d * 3 + 2] * Xv[x][2])
                                 : 0.0f;
                        fl[h][d * kNX + x] = val;
                    }
                if (live) {
                    sNK[l] = me / r;
                    sNK[NP + l] = muf[h] * Cp / Pr + me * Cp / Pr + Cp * r * ms / 0.9f;
                }
            }
            if (tid == 0)  // task 0, first point: lattice node (0,0,0)
#pragma unroll
                for (int x = 0; x < kNFX; ++x) sRef[x] = fl[0][x];
            __syncthreads();
#pragma unroll
            for (int x = 0; x < kNFX; ++x) {
                fl[0][x] = valid ? __fsub_rn(fl[0][x], sRef[x]) : 0.0f;
                fl[1][x] = two ? __fsub_rn(fl[1][x], sRef[x]) : 0.0f;
                const float mx = fmaxf(0.0f, fmaxf(fabsf(fl[0][x]), fabsf(fl[1][x])));
                const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
                if (lane == 0) atomicMax(&sMax[kFx0 + x], mb);
            }
            __syncthreads();
            if (tid >= kFx0 && tid < kFx0 + kNFX) scale_from_max(sMax[tid], G::BITS, sScale[tid], sInv[tid]);
            __syncthreads();
            if (valid) {
#pragma unroll
                for (int x = 0; x < kNFX; ++x) {
                    const float s = sScale[kFx0 + x];
                    unsigned hi, lo;
                    split_scaled<BF16>(__fmul_rn(fl[0][x], s), __fmul_rn(fl[1][x], s), hi, lo);
                    *reinterpret_cast<unsigned *>(sHalf + (2 * x) * G::PB + row_off) = hi;
                    *reinterpret_cast<unsigned *>(sHalf + (2 * x + 1) * G::PB + row_off) = lo;
                }
            }
        }
        __syncthreads();

        // ---- weak divergence: six sums per point over the three directions ----
        float *sAcc = sG;  // the iso-derivatives are consumed
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            const unsigned bh = d == 0 ? Bdh[0] : (d == 1 ? Bdh[1] : Bdh[2]);
            const unsigned bl = d == 0 ? Bdl[0] : (d == 1 ? Bdl[1] : Bdl[2]);
            const unsigned char *rowp = sHalf + plane_off + operand_row<Q>(d, warp, r8);
            int lat[2];
            float acc[2][kNX];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                lat[s] = pass_point<Q>(d, s, g, tq, warp);
#pragma unroll
                for (int x = 0; x < kNX; ++x) acc[s][x] = (d == 0 || lat[s] < 0) ? 0.0f : sAcc[x * NP + lat[s]];
            }
#pragma unroll
            for (int x = 0; x < kNX; x += 2) {
                const unsigned char *src = rowp + 2 * (d * kNX + x) * G::PB;
                unsigned a[4];
                if (d == 0)
                    ldsm_x4(a, src);
                else
                    ldsm_x4_t(a, src);
                float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma_acc<BF16>(c, a, bh, bh);
                mma_acc<BF16>(c, a, bl, 0u);
                const float cs0 = d == 0 ? colsum[0][0] : (d == 1 ? colsum[1][0] : colsum[2][0]);
                const float cs1 = d == 0 ? colsum[0][1] : (d == 1 ? colsum[1][1] : colsum[2][1]);
                const float2 inv2 = *reinterpret_cast<const float2 *>(sInv + kFx0 + d * kNX + x);
                const float2 ref2 = *reinterpret_cast<const float2 *>(sRef + d * kNX + x);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float inv = k ? inv2.y : inv2.x, ref = k ? ref2.y : ref2.x;
#pragma unroll
                    for (int s = 0; s < 2; ++s)
                        acc[s][x + k] = fmaf(c[2 * k + s], inv, fmaf(ref, s ? cs1 : cs0, acc[s][x + k]));
                }
            }
            if (d < 2) {
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    if (lat[s] >= 0)
#pragma unroll
                        for (int x = 0; x < kNX; ++x) sAcc[x * NP + lat[s]] = acc[s][x];
                __syncthreads();
            } else {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (lat[s] < 0) continue;
                    const int node = sNode[lat[s]];
                    if (node < 0) continue;
                    red_add(Rmass + node, f2d(sNK[lat[s]] * acc[s][X_GRHO]));
#pragma unroll
                    for (int i = 0; i < 3; ++i) red_add(Rmom + (size_t)i * npoin + node, f2d(acc[s][X_TAU0 + i]));
                    // energy-flux assembly in FP64
                    red_add(Rener + node, fma(f2d(sNK[NP + lat[s]]), f2d(acc[s][X_GT]), f2d(acc[s][X_TAUU])));
                }
            }
        }
    }  // elements
}

template <int P, bool BF16, bool NUE>
cudaError_t launch_pbn(const MixedDiffuArgs &a, cudaStream_t st)
{
    using G = MixedDiffuGeom<P, BF16>;
    static_assert(G::smem <= 227 * 1024, "shared memory budget");
    auto kern = diffu_mixed_kernel<P, BF16, NUE>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem);
    if (err != cudaSuccess) return err;
    if (a.nelem == 0) return cudaSuccess;
    const int grid = persistent_grid(kern, G::NT, G::smem, a.nelem);
    if (grid < 1) return cudaErrorInvalidConfiguration;
    // Not launched over the zeroing kernel: blocks that start beside it are spread
    // unevenly over the SMs for all of the kernel (porder-4 48^3 convection 2.83 against 2.68 ms).
    kern<<<grid, G::NT, G::smem, st>>>(a.nelem, a.npoin, a.connec, a.He, a.gpvol,
                        a.invAtoIJK, a.dlxigp_ip, a.Cp, a.Pr, a.rho, a.u, a.Tem, a.mu_fluid, a.mu_e, a.mu_sgs,
                        a.nu_elem, a.Rmass, a.Rmom, a.Rener);
    return cudaGetLastError();
}

template <int P>
cudaError_t launch_p(const MixedDiffuArgs &a, int precision, cudaStream_t st)
{
    const bool bf = precision == MSOD_PREC_BF16, nue = a.nu_elem != nullptr;
    if (bf) return nue ? launch_pbn<P, true, true>(a, st) : launch_pbn<P, true, false>(a, st);
    return nue ? launch_pbn<P, false, true>(a, st) : launch_pbn<P, false, false>(a, st);
}

}  // namespace

cudaError_t launch_diffu_mixed(int porder, int precision, const MixedDiffuArgs &a, cudaStream_t st)
{
    switch (porder) {
    case 1: return launch_p<1>(a, precision, st);
    case 2: return launch_p<2>(a, precision, st);
    case 3: return launch_p<3>(a, precision, st);
    case 4: return launch_p<4>(a, precision, st);
    case 5: return launch_p<5>(a, precision, st);
    case 6: return launch_p<6>(a, precision, st);
    case 7: return launch_p<7>(a, precision, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace msod
