// msod_mixed.cu -- mixed-precision hex GLL convection residual on the tensor cores.
//
// Same residuals as full_convec_ijk (elem_convec.f90:198-431, Rener per
// :674-832; formulas in msod_convec.cu) from FP32 fields, with:
//   * the 1-D derivative contractions of the 31 differentiated nodal products
//     on the tensor cores as FP16 (or BF16) hi + lo split products with FP32
//     accumulation;
//   * the nodal scatter-add and the final energy-flux assembly in FP64 (the
//     outputs are FP64 arrays).
//
// Splitting.  Each field f of an element is shifted by its value at the
// element's lattice node (0,0,0) -- the derivative operator annihilates
// constants, so derivatives are unchanged while the split only has to carry
// the field's variation over the element -- and scaled by a power of two s_f
// chosen per element and field so that max |s_f (f - f_ref)| lies in
// [2^(B-1), 2^B) with B = 11 (FP16) or 8 (BF16).  hi = rint(v) is then an
// integer of at most B bits (exact in the half format) and lo = v - hi lies
// in [-1/2, 1/2].  The derivative matrix is split by plain rounding,
// D = D_hi + D_lo.  Products, shifts and scalings use explicit roundings, so
// a field that is constant over the element splits into exact zeros.
//
// Contraction.  Per (two fields, direction, tile of 8 lines) two accumulating
// mma.sync.m16n8k16:
//   A (16x16) = [f_hi | f_lo]          rows: line of the first / second field,
//                                      cols: input point (hi | lo)
//   B1 (16x8) = [D_hi^T ; D_hi^T]      rows: input point (hi | lo), cols: output point
//   B2 (16x8) = [D_lo^T ; 0]
// C = f_hi D_hi^T + f_lo D_hi^T + f_hi D_lo^T (the dropped f_lo D_lo^T is
// below 2^-21 of the product).  Lines shorter than 8 points are zero padded.
//
// Shared-memory layout of one field half: 64 rows of 16 bytes (8 halves along
// i), row (k, j) stored at position 8k + (j xor k).  ldmatrix reads the A
// operand of xi lines directly (rows = lines) and of eta / zeta lines
// transposed (rows = input points); the xor swizzle keeps the eight rows of
// every ldmatrix phase on distinct banks in all three directions.
//
// Accumulation.  As in the FP32 kernel, each direction pass adds the
// contribution of its iso-parametric derivatives, through the He column of
// that direction and the point's own nodal values, to seven per-point
// accumulators in shared memory; the last pass assembles the energy residual
// in FP64 and scatter-adds all residuals with red.global.add.f64.
// porder 1..7; persistent blocks of one warp per tile (Q warps), one element at
// a time.  The kernel waits on its phases' loads, so residency pays: two fields
// of one tile per contraction instead of one field of two tiles halves a
// thread's state (two points instead of four) and leaves no warp without a tile.
// A thread gathers the two points that it splits, with the node ids loaded an
// element ahead, and the positions in shared memory (node_at) keep the passes'
// nodal reads off each other's banks (a third of the L1 pipe's cycles before).
// FP16, two tiles per warp in blocks of four warps / one tile per warp / now:
// porder 7 24^3 0.907 / 0.815 / 0.677 ms, 6 32^3 1.842 / 1.424 / 1.343, 5 40^3
// 2.354 / 2.052 / 1.925, 4 48^3 4.918 / 2.692 / 2.644, 3 48^3 2.647 / 1.867 / 1.821,
// 2 64^3 5.990 / 3.180 / 3.347, 1 64^3 5.532 / 2.139 / 2.156.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "msod_device.cuh"
#include "msod_kernels.h"
#include "msod_mma.cuh"

namespace msod {
namespace {

constexpr int kNF = 31;       // differentiated products
enum { B_RHO = 0, B_H, B_U0, B_U1, B_U2, B_Q0, B_Q1, B_Q2, NBASE };
enum { A_M = 0, A_MOM0, A_MOM1, A_MOM2, A_E, A_DIVU, A_DIVQ, NACC };

// Field numbering: 0 rho, 1 p, 2-4 u_i, 5-7 q_i, 8-16 q_i u_j (i major),
// 17-22 u_i u_j (i <= j: 00 01 02 11 12 22), 23 H, 24 rho H, 25-27 rho H u_i,
// 28-30 H u_i, with H = E + |u|^2 / 2.
struct Nodal {
    float r, p, u[3], q[3], H, rH;
};

// The point's nodal values as the passes use them (all but p).
__device__ __forceinline__ Nodal nodal_from(const float *sBase, int np, int l)
{
    Nodal n;
    n.r = sBase[B_RHO * np + l];
    n.H = sBase[B_H * np + l];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        n.u[c] = sBase[(B_U0 + c) * np + l];
        n.q[c] = sBase[(B_Q0 + c) * np + l];
    }
    n.rH = __fmul_rn(n.r, n.H);
    return n;
}

__host__ __device__ constexpr int sym_i(int m) { return m < 3 ? 0 : (m < 5 ? 1 : 2); }
__host__ __device__ constexpr int sym_j(int m) { return m < 3 ? m : (m < 5 ? m - 2 : 2); }

__device__ __forceinline__ float field(int f, const Nodal &n)
{
    if (f == 0) return n.r;
    if (f == 1) return n.p;
    if (f < 5) return n.u[f - 2];
    if (f < 8) return n.q[f - 5];
    if (f < 17) return __fmul_rn(n.q[(f - 8) / 3], n.u[(f - 8) % 3]);
    if (f < 23) return __fmul_rn(n.u[sym_i(f - 17)], n.u[sym_j(f - 17)]);
    if (f == 23) return n.H;
    if (f == 24) return n.rH;
    if (f < 28) return __fmul_rn(n.rH, n.u[f - 25]);
    return __fmul_rn(n.H, n.u[f - 28]);
}

// Per-point coefficients of one direction pass.
struct PointCoef {
    float rho, H, u[3], h[3], cu, cq;
};

// Adds field f's iso-derivative dv (this pass's direction) to the point's
// accumulators: the rules of the FP32 kernel, field by field.
__device__ __forceinline__ void apply_field(int f, float dv, const PointCoef &c, float (&acc)[NACC])
{
    const float h4 = 0.25f;
    if (f == 0) {
        const float t = c.cu * dv;
        acc[A_M] = fmaf(0.5f, t, acc[A_M]);
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[A_MOM0 + i] = fmaf(h4 * c.u[i], t, acc[A_MOM0 + i]);
        acc[A_E] = fmaf(h4 * c.H, t, acc[A_E]);
    } else if (f == 1) {
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[A_MOM0 + i] = fmaf(c.h[i], dv, acc[A_MOM0 + i]);
    } else if (f < 5) {
        acc[A_DIVU] = fmaf(c.h[f - 2], dv, acc[A_DIVU]);
        acc[A_MOM0 + f - 2] = fmaf(h4 * c.cq, dv, acc[A_MOM0 + f - 2]);
    } else if (f < 8) {
        acc[A_DIVQ] = fmaf(c.h[f - 5], dv, acc[A_DIVQ]);
        acc[A_MOM0 + f - 5] = fmaf(h4 * c.cu, dv, acc[A_MOM0 + f - 5]);
    } else if (f < 17) {
        const int i = (f - 8) / 3, j = (f - 8) % 3;
        acc[A_MOM0 + i] = fmaf(h4 * c.h[j], dv, acc[A_MOM0 + i]);
    } else if (f < 23) {
        const int i = sym_i(f - 17), j = sym_j(f - 17);
        const float rd = h4 * c.rho * dv;
        acc[A_MOM0 + i] = fmaf(c.h[j], rd, acc[A_MOM0 + i]);
        if (i != j) acc[A_MOM0 + j] = fmaf(c.h[i], rd, acc[A_MOM0 + j]);
    } else if (f == 23) {
        acc[A_E] = fmaf(h4 * c.cq, dv, acc[A_E]);
    } else if (f == 24) {
        acc[A_E] = fmaf(h4 * c.cu, dv, acc[A_E]);
    } else if (f < 28) {
        acc[A_E] = fmaf(h4 * c.h[f - 25], dv, acc[A_E]);
    } else {
        acc[A_E] = fmaf(h4 * c.rho * c.h[f - 28], dv, acc[A_E]);
    }
}

template <int P, bool BF16>
struct MixedGeom {
    static constexpr int Q = P + 1, N = Q * Q * Q, W = (Q + 1) / 2, NP = node_plane<Q>();
    static constexpr int NT = 32 * Q;        // one warp per tile (k-plane or j-plane) of lines
    static constexpr int NTASK = Q * Q * W;  // task: points (2w, 2w+1) of one i-row
    static_assert(NTASK <= NT, "one task per thread");
    static constexpr int BITS = BF16 ? 8 : 11;
    static constexpr int PB = plane_bytes<Q>();  // bytes of one field half
    static constexpr size_t half_bytes = (size_t)2 * kNF * PB;
    static constexpr size_t smem = half_bytes + (size_t)(NBASE + NACC) * NP * sizeof(float) +
                                   (size_t)2 * NP * sizeof(int) + (2 * 32 + 4) * sizeof(float);
    // Blocks per SM that shared memory allows, as long as a thread keeps kMixedRegs registers.
    static constexpr int MINB = mixed_blocks(smem, NT, kMixedRegs);
};

template <int P, bool BF16>
__global__ void __launch_bounds__(32 * (P + 1), MixedGeom<P, BF16>::MINB)
    convec_mixed_kernel(int nelem, int npoin, const int *__restrict__ connec, const float *__restrict__ He,
                        const float *__restrict__ gpvol, const int *__restrict__ inv,
                        const float *__restrict__ dlxigp_ip,
                        const float *__restrict__ u, const float *__restrict__ q, const float *__restrict__ rho,
                        const float *__restrict__ pr, const float *__restrict__ E, double *__restrict__ Rmass,
                        double *__restrict__ Rmom, double *__restrict__ Rener)
{
    using G = MixedGeom<P, BF16>;
    constexpr int Q = G::Q, N = G::N, W = G::W, NTASK = G::NTASK, NT = G::NT, NP = G::NP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *sHalf = smem_raw;                                  // [2*kNF][G::PB]: hi, lo of each field
    float *sBase = reinterpret_cast<float *>(sHalf + G::half_bytes);  // [NBASE][NP], positions node_at
    float *sAcc = sBase + NBASE * NP;                                  // [NACC][NP]
    int *sNode = reinterpret_cast<int *>(sAcc + NACC * NP);            // [NP]
    int *sPerm = sNode + NP;                                           // gmsh node
    float *sScale = reinterpret_cast<float *>(sPerm + NP);            // [32] s_f
    float *sInv = sScale + 32;                                         // [32] 1 / s_f (max bits first)
    float *sRefP = sInv + 32;                                          // p at lattice node (0,0,0)
    unsigned *sMax = reinterpret_cast<unsigned *>(sInv);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Once per block: tables, the zero padding of the half planes (rows and
    // points beyond Q are never written), the B fragments.
    for (int i = tid; i < N; i += NT) sPerm[node_at<Q>(i / (Q * Q), i / Q % Q, i % Q)] = table_node<Q>(inv, i);
    if (Q < 8) {
        uint4 *z = reinterpret_cast<uint4 *>(sHalf);
        for (int i = tid; i < (int)(G::half_bytes / 16); i += NT) z[i] = make_uint4(0, 0, 0, 0);
    }
    // B fragments per direction: col lane/4 (output point), rows 2t, 2t+1 (input point).
    unsigned Bh[3], Bl[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int r = lane >> 2, c0 = 2 * (lane & 3), c1 = c0 + 1;
        const float d0 = (r < Q && c0 < Q) ? table_D<Q>(inv, dlxigp_ip, d, r, c0) : 0.0f;
        const float d1 = (r < Q && c1 < Q) ? table_D<Q>(inv, dlxigp_ip, d, r, c1) : 0.0f;
        split_pair<BF16>(d0, d1, Bh[d], Bl[d]);
    }
    const size_t np = (size_t)npoin;
    // The thread's task: points (2w, 2w+1) of i-row (rk, rj), which it gathers and
    // splits.  The node ids are loaded an element ahead.
    const bool valid = tid < NTASK;
    const int row = valid ? tid / W : 0, w = valid ? tid - row * W : 0;
    const bool two = valid && 2 * w + 1 < Q;
    const int rk = row / Q, rj = row - rk * Q;
    const int l0 = node_at<Q>(rk, rj, 2 * w), l1 = l0 + 1;
    const int off = row_pos(rk, rj) * kRowB + 4 * w;
    const int a0 = table_node<Q>(inv, row * Q + 2 * w), a1 = table_node<Q>(inv, row * Q + 2 * w + (two ? 1 : 0));
    auto node_id = [&](int a, int el) { return ldg_once(connec + (size_t)a * nelem + el); };
    int id0 = node_id(a0, blockIdx.x), id1 = node_id(a1, blockIdx.x);  // the grid has nelem blocks at most
#pragma unroll 1
    for (int e = blockIdx.x; e < nelem; e += gridDim.x) {
    Nodal n0, n1;
    {
        auto gather = [&](int v, Nodal &n, bool own) {
            const bool ok = own && (unsigned)v < (unsigned)npoin;  // a missing node reads as zeros
            const size_t p = ok ? v : 0;
            n.r = ok ? ldg_once(rho + p) : 0.0f;
            n.p = ok ? ldg_once(pr + p) : 0.0f;
            n.H = ok ? ldg_once(E + p) : 0.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                n.u[c] = ok ? ldg_once(u + c * np + p) : 0.0f;
                n.q[c] = ok ? ldg_once(q + c * np + p) : 0.0f;
            }
            return ok ? v : -1;
        };
        auto store = [&](int pos, int node, Nodal &n, bool own) {
            const float k2 = __fmaf_rn(n.u[0], n.u[0], __fmaf_rn(n.u[1], n.u[1], __fmul_rn(n.u[2], n.u[2])));
            n.H = __fmaf_rn(0.5f, k2, n.H);
            n.rH = __fmul_rn(n.r, n.H);
            if (!own) return;
            sNode[pos] = node;
            sBase[B_RHO * NP + pos] = n.r;
            sBase[B_H * NP + pos] = n.H;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sBase[(B_U0 + c) * NP + pos] = n.u[c];
                sBase[(B_Q0 + c) * NP + pos] = n.q[c];
            }
        };
        const int v0 = gather(id0 - 1, n0, valid), v1 = gather(id1 - 1, n1, two);
        const int en = e + (int)gridDim.x < nelem ? e + (int)gridDim.x : e;
        id0 = node_id(a0, en);
        id1 = node_id(a1, en);
        __syncthreads();  // the previous element's passes are done with every shared array
        if (tid < 32) sMax[tid] = 0u;
        store(l0, v0, n0, valid);
        store(l1, v1, n1, two);
        if (tid == 0) *sRefP = n0.p;
    }
    __syncthreads();

    // He columns of the first direction pass, in flight during the split.
    const int g = lane >> 2, tq = lane & 3;
    float hcur[2][3];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int l = pass_point<Q>(0, s, g, tq, warp);
        const float *hp = He + ((size_t)e * N + sPerm[l < 0 ? 0 : l]) * 9;
#pragma unroll
        for (int c = 0; c < 3; ++c) hcur[s][c] = ldg(hp + c);
    }

    // Shifted products of the thread's task (two points) in registers, their
    // per-field maxima over the element (non-negative floats order like their
    // bit patterns), then the split into the half planes.
    float v[kNF][2];
    {
        Nodal nref = nodal_from(sBase, NP, 0);
        nref.p = *sRefP;
#pragma unroll
        for (int f = 0; f < kNF; ++f) {
            const float fr = field(f, nref);
            v[f][0] = valid ? __fsub_rn(field(f, n0), fr) : 0.0f;
            v[f][1] = two ? __fsub_rn(field(f, n1), fr) : 0.0f;
            const float mx = fmaxf(0.0f, fmaxf(fabsf(v[f][0]), fabsf(v[f][1])));
            const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
            if (lane == 0) atomicMax(&sMax[f], mb);
        }
    }
    __syncthreads();
    if (tid < kNF) {
        // s_f = 2^(B-1-ex) for a maximum in [2^ex, 2^(ex+1)); ex clamped so s_f and 1/s_f are normal.
        int ex = (int)((sMax[tid] >> 23) & 0xFF) - 127;
        ex = min(max(ex, -100), 127);
        sScale[tid] = __int_as_float((127 + G::BITS - 1 - ex) << 23);
        sInv[tid] = __int_as_float((127 + ex - (G::BITS - 1)) << 23);
    }
    __syncthreads();
    if (valid) {
        float4 sc;
#pragma unroll
        for (int f = 0; f < kNF; ++f) {
            if (f % 4 == 0) sc = *reinterpret_cast<const float4 *>(sScale + f);
            const float s = f % 4 == 0 ? sc.x : (f % 4 == 1 ? sc.y : (f % 4 == 2 ? sc.z : sc.w));
            unsigned hi, lo;
            split_scaled<BF16>(__fmul_rn(v[f][0], s), __fmul_rn(v[f][1], s), hi, lo);
            *reinterpret_cast<unsigned *>(sHalf + (2 * f) * G::PB + off) = hi;
            *reinterpret_cast<unsigned *>(sHalf + (2 * f + 1) * G::PB + off) = lo;
        }
    }
    __syncthreads();

    // Warp w takes tile w (a k-plane for xi / eta lines, a j-plane for zeta
    // lines) of two fields f, f+1 at a time; ldmatrix matrix m of the A operand is
    // (hi f, hi f+1, lo f, lo f+1), row r8.  The last field stands alone: its rows
    // twice, the second result unused.
    const int m = lane >> 3, r8 = lane & 7;
    const int alone = (m & 1) * 2 * G::PB, plane_off = alone + (m >> 1) * G::PB;
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        const unsigned bh = d == 0 ? Bh[0] : (d == 1 ? Bh[1] : Bh[2]);
        const unsigned bl = d == 0 ? Bl[0] : (d == 1 ? Bl[1] : Bl[2]);
        // The thread's points: output points 2t and 2t+1 of line g of the tile.
        int lat[2];
        bool live[2];
        PointCoef cf[2];
        float acc[2][NACC], gp[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int lp = pass_point<Q>(d, s, g, tq, warp);
            live[s] = lp >= 0;
            const int l = live[s] ? lp : 0;
            lat[s] = l;
            const Nodal n = nodal_from(sBase, NP, l);
            cf[s].rho = n.r;
            cf[s].H = n.H;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                cf[s].u[c] = n.u[c];
                cf[s].h[c] = hcur[s][c];
            }
            cf[s].cu = n.u[0] * cf[s].h[0] + n.u[1] * cf[s].h[1] + n.u[2] * cf[s].h[2];
            cf[s].cq = n.q[0] * cf[s].h[0] + n.q[1] * cf[s].h[1] + n.q[2] * cf[s].h[2];
#pragma unroll
            for (int k = 0; k < NACC; ++k) acc[s][k] = (d == 0 || !live[s]) ? 0.0f : sAcc[k * NP + l];
        }
        // Loads in flight during the contractions: the next pass's He columns,
        // or gpvol for the last pass's scatter.
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (d < 2) {
                const int l = pass_point<Q>(d + 1, s, g, tq, warp);
                const float *hp = He + ((size_t)e * N + sPerm[l < 0 ? 0 : l]) * 9 + (d + 1) * 3;
#pragma unroll
                for (int c = 0; c < 3; ++c) hcur[s][c] = ldg(hp + c);
                gp[s] = 0.0f;
            } else {
                gp[s] = ldg(gpvol + (size_t)e * N + sPerm[lat[s]]);
            }
        }
        const unsigned char *rowp = sHalf + plane_off + operand_row<Q>(d, warp, r8);
#pragma unroll
        for (int f = 0; f < kNF; f += 2) {
            const unsigned char *src = rowp + 2 * f * G::PB - (f + 1 < kNF ? 0 : alone);
            unsigned a[4];
            if (d == 0)
                ldsm_x4(a, src);
            else
                ldsm_x4_t(a, src);
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_acc<BF16>(c, a, bh, bh);
            mma_acc<BF16>(c, a, bl, 0u);
            const float2 inv2 = *reinterpret_cast<const float2 *>(sInv + f);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (f + k >= kNF) break;
                const float inv = k ? inv2.y : inv2.x;
#pragma unroll
                for (int s = 0; s < 2; ++s) apply_field(f + k, c[2 * k + s] * inv, cf[s], acc[s]);
            }
        }
        if (d < 2) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (live[s])
#pragma unroll
                    for (int k = 0; k < NACC; ++k) sAcc[k * NP + lat[s]] = acc[s][k];
            __syncthreads();
        } else {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (!live[s]) continue;
                const int node = sNode[lat[s]];
                if (node < 0) continue;
                const Nodal n = nodal_from(sBase, NP, lat[s]);
                const float divU = acc[s][A_DIVU], divQ = acc[s][A_DIVQ];
                const float rm = acc[s][A_M] + 0.5f * (divQ + n.r * divU);
                red_add(Rmass + node, f2d(gp[s] * rm));
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float rmom = acc[s][A_MOM0 + i] + 0.25f * (n.u[i] * divQ + n.q[i] * divU);
                    red_add(Rmom + (size_t)i * npoin + node, f2d(gp[s] * rmom));
                }
                // energy-flux assembly in FP64
                const double t = fma(f2d(n.H), f2d(divQ), f2d(n.rH) * f2d(divU));
                red_add(Rener + node, f2d(gp[s]) * fma(0.25, t, f2d(acc[s][A_E])));
            }
        }
    }
    }  // elements
}

template <int P, bool BF16>
cudaError_t launch_mixed_pb(const MixedConvecArgs &a, cudaStream_t st)
{
    using G = MixedGeom<P, BF16>;
    static_assert(G::smem <= 227 * 1024, "shared memory budget");
    auto kern = convec_mixed_kernel<P, BF16>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem);
    if (err != cudaSuccess) return err;
    if (a.nelem == 0) return cudaSuccess;
    const int grid = persistent_grid(kern, G::NT, G::smem, a.nelem);
    if (grid < 1) return cudaErrorInvalidConfiguration;
    // Not launched over the zeroing kernel: blocks that start beside it are spread
    // unevenly over the SMs for all of the kernel (porder-4 48^3 convection 2.83 against 2.68 ms).
    kern<<<grid, G::NT, G::smem, st>>>(a.nelem, a.npoin, a.connec, a.He, a.gpvol,
                        a.invAtoIJK, a.dlxigp_ip, a.u, a.q, a.rho, a.pr, a.E, a.Rmass, a.Rmom, a.Rener);
    return cudaGetLastError();
}

template <int P>
cudaError_t launch_mixed_p(const MixedConvecArgs &a, int precision, cudaStream_t st)
{
    return precision == MSOD_PREC_BF16 ? launch_mixed_pb<P, true>(a, st) : launch_mixed_pb<P, false>(a, st);
}

}  // namespace

cudaError_t launch_convec_mixed(int porder, int precision, const MixedConvecArgs &a, cudaStream_t st)
{
    switch (porder) {
    case 1: return launch_mixed_p<1>(a, precision, st);
    case 2: return launch_mixed_p<2>(a, precision, st);
    case 3: return launch_mixed_p<3>(a, precision, st);
    case 4: return launch_mixed_p<4>(a, precision, st);
    case 5: return launch_mixed_p<5>(a, precision, st);
    case 6: return launch_mixed_p<6>(a, precision, st);
    case 7: return launch_mixed_p<7>(a, precision, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace msod
