// msod_convec.cu -- plain (FP32 / FP64) hex GLL convection residual.
//
// Computes what full_convec_ijk computes (elem_convec.f90:198-431; Rener as
// defined by full_convec_ijk_split, elem_convec.f90:674-832):
//
//   Rmass  += gpvol [ 1/2 (div q + rho div u) + 1/2 u.grad rho ]
//   Rmom_i += gpvol [ 1/4 (div F_i + u_i div q + q_i div u + rho div Fuu_i) + d_i p
//                     + 1/4 sum_j (u_i u_j d_j rho + q_j d_j u_i + u_j d_j q_i) ]
//   Rener  += gpvol [ 1/4 (div(rho H u) + H div q + rho H div u + rho div(H u))
//                     + 1/4 sum_i (q_i d_i H + u_i d_i(rho H) + H u_i d_i rho) ]
//
// with F = q (x) u, Fuu = u (x) u, k = |u|^2/2 and H = E + k (the reference's
// separate E and k terms, elem_convec.f90:810-817, are linear in them).
//
// Pairwise form.  Along a line of direction d, with D its 1-D derivative matrix,
// h = He(:,d) at the output point r, and for a point s of the line
// U_s = h.u_s, Q_s = h.q_s, direction d's share of the bracket above at r is
//
//   4 mom_i = sum_s D_rs [ u_i,r (U_r rho_s + Q_s) + u_i,s (Q_r + rho_r U_s)
//                        + q_i,s (U_r + U_s) + q_i,r U_s + 4 h_i p_s ]
//   4 ener  = the same with u_i -> H, q_i -> rho H and without p
//   2 mass  = sum_s D_rs [ U_r rho_s + Q_s + rho_r U_s ]
//
// (the metric is taken at r in every term, as the reference does, so nothing
// else of the metric enters).  Writing every value at s as the value at r plus
// a difference turns it into, with t = h.(u_s - u_r),
//
//   4 mom_i = sum_s D_rs [ (u_i,s - u_i,r)(Q_r + rho_r U_r + rho_r t) + (q_i,s - q_i,r)(2 U_r + t) ]
//             + u_i,r S + 2 q_i,r div u + 4 h_i dp      (S = U_r drho + h.dq + rho_r div u)
//   2 mass  = S
//
// with drho, dp, dq, div u the sums of D_rs times the differences, plus the row
// sum of D (zero but for the table's rounding) times the bracket at s = r.
// The 31 products of the bracket's own form, each differentiated in three
// directions, become 12 multiply-adds per pair of points beside the ten
// differences and six linear sums; no product field is formed; and since only
// differences are summed, the constant part of every field, which a derivative
// cancels, no longer leaves its rounding behind (momentum residual against 64
// bits on 64^3 smooth fields: 8e-8 instead of 6e-6 relative).
//
// Design (one group of NE elements per block, one thread per GLL line,
// msod_group.cuh):
//   * one thread issues the bulk copies of the group's He and gpvol spans;
//     meanwhile each thread gathers the points of its zeta line through connec,
//     forms H and rho H once per point and stores the records (u, H), (q, rho H)
//     and (rho, p) of its points to the shared-memory lattice;
//   * three passes (zeta, xi, eta) evaluate the pairwise form along the lines of
//     a direction, point after point of the line: the line's records sit in
//     registers (the zeta pass has them from the gather), the derivative matrix's
//     rows come from shared memory, and the five sums of a point (momentum,
//     energy, mass) pass from one direction's thread to the next through
//     shared memory;
//   * the last pass applies gpvol and scatter-adds with red.global.add.
#include <cuda_runtime.h>

#include "msod_group.cuh"

namespace msod {
namespace {

// Elements per block, threads per line, blocks per SM that the register budget
// allows for, and the form of the passes, measured per porder (FP32, ms).  The
// comparisons stand as they were made; a call takes now: porder 1 128^3 0.281, 2
// 100^3 0.520, 3 80^3 0.658, 4 64^3 0.942, 5 51^3 1.130, 6 40^3 1.054, 7 32^3 0.767, 8
// 26^3 0.903.
// Whole warps of lines count most (5 x 25 lines at porder 4: 125 of 128
// threads), then what is left of the L1 beside the blocks' shared memory, where
// the gathers' lines are in flight: three blocks of 64 KB stay within a 196 KB
// carveout.  On 64^3 porder-4 hexes 5 elements take 0.944 (1.044 before the
// pitch search, where 4, with 100 of 128 threads, took 1.15, 6 1.17, 8 1.13, 9
// 1.10).  A fourth block per SM (12 bytes per point less through kSlots, 128
// registers) gains nothing: 1.04.
template <typename real, int P>
constexpr int convec_ne()
{
    constexpr int nf[9] = {0, 32, 14, 8, 5, 4, 2, 2, 2}, nd[9] = {0, 32, 14, 8, 5, 3, 2, 1, 1};
    return sizeof(real) == 4 ? nf[P] : nd[P];
}
// Two threads share a line where one would spill (porder 8; FP64 from 7 up).
// At lower porders they lose what the second load of the line costs (porder 4
// 1.30, porder 3 1.01 against 0.71 on 80^3).
template <typename real, int P>
constexpr int convec_s()
{
    return P >= (sizeof(real) == 4 ? 8 : 7) ? 2 : 1;
}
template <typename real, int P>
constexpr int convec_minb()
{
    constexpr int nb[9] = {0, 1, 4, 4, 3, 2, 2, 1, 1};
    return sizeof(real) == 4 ? nb[P] : 1;
}
// All points of a line at once (the pairs' differences shared) or one point
// after the other (fewer registers): porder 3 0.711 / 0.738, 4 0.944 / 1.05, 6
// 1.052 / 1.149 (40^3), but 2 0.565 / 0.557 (100^3), 5 1.169 / 1.143 (51^3) and 7
// 0.855 / 0.786 (32^3), where the sums of all points no longer fit beside the
// line.
template <typename real, int P>
constexpr bool convec_all_points()
{
    return sizeof(real) == 4 && (P == 1 || P == 3 || P == 4 || P == 6);
}
// The three directions as one copy of the pass with run-time strides (porders
// 6 to 8, whose unrolled passes overrun the instruction cache: porder 6 1.052 /
// 1.148) or unrolled (porder 4 0.944 / 1.05, porder 3 0.711 / 0.911).
template <int P>
constexpr bool convec_rolled()
{
    return P >= 6;
}
// Sums kept in the spent part of the He records (ConvecShared::kSlots): 2, mass and
// energy and the node, where it makes room for another block (porder 7: 0.786 / 0.860;
// porder 5 1.143 / 1.155); 1, mass and node, at porder 3, where it makes room for 60
// instead of 28 KB of L1 beside four blocks (12 M element points, numbered along x
// 0.248 / 0.257, nodes in random order 1.61 / 2.37, elements in random order 0.75 / 1.01);
// elsewhere the records' bank conflicts cost more than the room gives.
template <typename real, int P>
constexpr int convec_slots()
{
    return sizeof(real) == 8 ? 0 : (P == 5 || P == 7 ? 2 : (P == 3 ? 1 : 0));
}
// Blocks of closely numbered elements gather through the L1 (group_close): on 12 M
// element points in elements with nodes of their own, past it / through it, ms: porder 1
// 0.345 / 0.299, 2 0.425 / 0.329, 3 0.576 / 0.402; on a mesh numbered along x it costs
// nothing there.  From porder 4 up it would gain as much (4 0.541 / 0.424), but costs up to 1 %
// on the mesh numbered along x.
template <typename real, int P>
constexpr bool convec_close()
{
    return sizeof(real) == 4 && P <= 3;
}
// Shared memory that an SM should keep for the blocks (percent, -1: as many blocks as
// fit).  Porder 1 would take seven blocks in 228 KB and leave 28 KB of L1, where the cache
// lines of the gathers in flight no longer fit: six in 196 KB take 0.203 instead of 0.187
// ms on a mesh numbered along x, but 0.557 instead of 0.880 with nodes in random order and
// 0.574 instead of 1.025 with elements in random order (12 M element points).
template <typename real, int P>
constexpr int convec_carveout()
{
    return sizeof(real) == 4 && P == 1 ? 80 : -1;
}
template <typename real, int P>
using ConvecGeom = GroupGeom<real, P, convec_ne<real, P>(), convec_s<real, P>()>;

// Shared memory of a block.
template <class G>
struct ConvecShared {
    using real = typename G::real;
    static constexpr size_t kW = G::HEB + G::GPB + 16;
    static constexpr size_t kV = kW + G::NREC * sizeof(Four<real>);
    static constexpr size_t kA = kV + G::NREC * sizeof(Four<real>);
    static constexpr int kSlots = convec_slots<real, G::P>();
    static constexpr size_t kZ = kA + (kSlots == 2 ? G::NPR * sizeof(Two<real>) : G::NREC * sizeof(Four<real>));
    static constexpr size_t kM = kZ + G::NSC * sizeof(real);
    static constexpr size_t kNode = kM + (kSlots == 1 ? 0 : G::NSC * sizeof(real));
    static constexpr size_t kTab = (kNode + (kSlots ? 0 : G::NSC * sizeof(int)) + 15) / 16 * 16;
    static constexpr size_t kBytes = kTab + GroupTables<G, true>::kBytes;
    unsigned char *base;
    int el;  // the thread's element
    __device__ __forceinline__ unsigned long long *bar() const
    {
        return reinterpret_cast<unsigned long long *>(base + G::HEB + G::GPB);
    }
    __device__ __forceinline__ Four<real> *W() const { return reinterpret_cast<Four<real> *>(base + kW); }  // u, H
    __device__ __forceinline__ Four<real> *V() const { return reinterpret_cast<Four<real> *>(base + kV); }  // q, p
    __device__ __forceinline__ Four<real> *A() const { return reinterpret_cast<Four<real> *>(base + kA); }  // 4 mom, 4 ener
    __device__ __forceinline__ real *Z() const { return reinterpret_cast<real *>(base + kZ) + el * G::SK; }  // rho
    __device__ __forceinline__ real *M() const { return reinterpret_cast<real *>(base + kM) + el * G::SK; }  // 2 mass
    __device__ __forceinline__ int *node() const { return reinterpret_cast<int *>(base + kNode) + el * G::SK; }
    __device__ __forceinline__ Two<real> *A2() const { return reinterpret_cast<Two<real> *>(base + kA) + el * G::HK; }
    // The sums of a point (record o, its He record at he) between the passes.
    // kSlots: the zeta column of a point's He record is read in the zeta pass
    // only, by the thread that owns the point's zeta line; from then on it holds
    // the mass sum, the energy sum (2) and the point's node.
    __device__ __forceinline__ void put(int o, real *he, const Two<real> &a, const Two<real> &b, real m) const
    {
        if constexpr (kSlots == 2) {
            A2()[o] = a;
            M()[o] = b.x;
            he[6] = b.y;
            he[7] = m;
        } else {
            Four<real> p;
            p.a = a;
            p.b = b;
            A()[o] = p;
            (kSlots ? he[7] : M()[o]) = m;
        }
    }
    __device__ __forceinline__ void add(int o, const real *he, Two<real> &a, Two<real> &b, real &m) const
    {
        if constexpr (kSlots == 2) {
            a = add2(a, A2()[o]);
            b = add2(b, two(M()[o], he[6]));
            m += he[7];
        } else {
            const Four<real> p = A()[o];
            a = add2(a, p.a);
            b = add2(b, p.b);
            m += kSlots ? he[7] : M()[o];
        }
    }
    __device__ __forceinline__ int node_at(int o, const real *he) const
    {
        if constexpr (kSlots != 0)
            return __float_as_int(he[8]);
        else
            return node()[o];
    }
    __device__ __forceinline__ GroupTables<G, true> tab() const { return GroupTables<G, true>{base + kTab}; }
};

// The records of one line.
template <class G>
struct ConvecLine {
    Four<typename G::real> w[G::Q], v[G::Q];  // (u, H), (q, rho H)
    Two<typename G::real> z[G::Q];            // (rho, p)
    __device__ __forceinline__ void set(int s, const Four<typename G::real> &uH, const Four<typename G::real> &qp,
                                        typename G::real rho)
    {
        w[s] = uH;
        v[s].a = qp.a;
        v[s].b = two(qp.b.x, rho * uH.b.y);
        z[s] = two(rho, qp.b.y);
    }
};

// One direction of a pass: the line's record and lattice strides, and where its
// coefficients lie.
template <class G>
struct ConvecDir {
    int dir, base, step, lat, lstep;
    bool first, last;
    __device__ __forceinline__ ConvecDir(const GroupThread<G> &t, int ip)
    {
        dir = ip == 0 ? 2 : ip - 1;
        first = ip == 0;
        last = ip == 2;
        step = dir == 0 ? 1 : (dir == 1 ? G::RP : G::PP);
        lstep = dir == 0 ? 1 : (dir == 1 ? G::Q : G::L);
        base = t.rec0(dir);
        lat = t.lat0(dir);
    }
};
template <class G>
__device__ __forceinline__ void convec_finish(const ConvecDir<G> &d, const ConvecShared<G> &sm,
                                              const GroupMetric<G> &gm, int el, int o, int pt, int node0,
                                              Two<typename G::real> a, Two<typename G::real> b, typename G::real m,
                                              int npoin, typename G::real *__restrict__ Rmass,
                                              typename G::real *__restrict__ Rmom,
                                              typename G::real *__restrict__ Rener)
{
    using real = typename G::real;
    real *he = gm.he(el, pt);
    if (!d.first) sm.add(o, he, a, b, m);
    if (!d.last) {
        sm.put(o, he, a, b, m);
        if constexpr (ConvecShared<G>::kSlots != 0)
            if (d.first) he[8] = __int_as_float(node0);
    } else {
        const int node = sm.node_at(o, he);
        if (node >= 0) {
            const real g = *gm.vol(el, pt), g4 = (real)0.25 * g;
            red_add(Rmass + node, (real)0.5 * g * m);
            red_add(Rmom + node, g4 * a.x);
            red_add(Rmom + (size_t)npoin + node, g4 * a.y);
            red_add(Rmom + 2 * (size_t)npoin + node, g4 * b.x);
            red_add(Rener + node, g4 * b.y);
        }
    }
}

// Points R0 .. R0+R-1 of a line, one after the other.
template <class G, int SEG>
__device__ __forceinline__ void convec_points(const ConvecLine<G> &ln, const GroupThread<G> &t, const ConvecDir<G> &d,
                                              const ConvecShared<G> &sm, const GroupRows<G, true> &tab, const GroupMetric<G> &gm,
                                              const int (&id)[G::R], int npoin,
                                              typename G::real *__restrict__ Rmass,
                                              typename G::real *__restrict__ Rmom,
                                              typename G::real *__restrict__ Rener)
{
    using real = typename G::real;
    using R2 = Two<real>;
    constexpr int Q = G::Q, R0 = SEG * G::R, R1 = R0 + G::R < Q ? R0 + G::R : Q;
    constexpr real k2 = (real)2, k3 = (real)3, k4 = (real)4;
#pragma unroll
    for (int r = R0; r < R1; ++r) {
        const int pt = tab.node(d.lat + r * d.lstep);
        const real *hp = gm.he(t.el, pt) + d.dir * 3;
        const real h0 = hp[0], h1 = hp[1], h2 = hp[2];
        const Four<real> wr = ln.w[r], vr = ln.v[r];
        const real rr = ln.z[r].x;
        const real U = fma(wr.b.x, h2, fma(wr.a.y, h1, wr.a.x * h0));
        const real Qc = fma(vr.b.x, h2, fma(vr.a.y, h1, vr.a.x * h0));
        const real X0 = U + U, Y0 = fma(rr, U, Qc);
        R2 A = two((real)0, (real)0), B = A, dz = A, dq = A;  // momentum 1-2; momentum 3, energy; drho, dp; dq 1-2
        real dq3 = (real)0, divu = (real)0, Dr[Q];
        tab.row(Dr, d.dir, r);
#pragma unroll
        for (int s = 0; s < Q; ++s) {
            if (s == r) continue;
            const real D = Dr[s];
            const R2 D2 = two(D, D);
            const R2 wa = sub2(ln.w[s].a, wr.a), wb = sub2(ln.w[s].b, wr.b);
            const R2 va = sub2(ln.v[s].a, vr.a), vb = sub2(ln.v[s].b, vr.b);
            const R2 dzs = sub2(ln.z[s], ln.z[r]);
            const real tt = fma(wb.x, h2, fma(wa.y, h1, wa.x * h0));
            const real X = D * (X0 + tt), Y = D * fma(rr, tt, Y0);
            A = fma2(va, two(X, X), fma2(wa, two(Y, Y), A));
            B = fma2(vb, two(X, X), fma2(wb, two(Y, Y), B));
            dz = fma2(D2, dzs, dz);
            dq = fma2(D2, va, dq);
            dq3 = fma(D, vb.x, dq3);
            divu = fma(D, tt, divu);
        }
        const real sg = tab.sum(d.dir, r);
        const real divq = fma(dq3, h2, fma(dq.y, h1, dq.x * h0));
        const real S = fma(rr, divu, fma(U, dz.x, divq));
        const real cw = fma(k2 * sg, Y0, S), cv = fma(k3 * sg, U, k2 * divu);
        const real dp = k4 * fma(sg, ln.z[r].y, dz.y);
        A = fma2(wr.a, two(cw, cw), fma2(vr.a, two(cv, cv), A));
        B = fma2(wr.b, two(cw, cw), fma2(vr.b, two(cv, cv), B));
        A = fma2(two(h0, h1), two(dp, dp), A);
        B.x = fma(h2, dp, B.x);
        convec_finish<G>(d, sm, gm, t.el, d.base + r * d.step, pt, id[r - R0], A, B, fma(sg, fma(rr, U, Y0), S), npoin, Rmass, Rmom,
                         Rener);
    }
}

// All points of a line at once: the differences of a pair of points serve both
// of its rows.
template <class G>
__device__ __forceinline__ void convec_pairs(const ConvecLine<G> &ln, const GroupThread<G> &t, const ConvecDir<G> &d,
                                             const ConvecShared<G> &sm, const GroupRows<G, true> &tab, const GroupMetric<G> &gm,
                                              const int (&id)[G::R], int npoin,
                                             typename G::real *__restrict__ Rmass, typename G::real *__restrict__ Rmom,
                                             typename G::real *__restrict__ Rener)
{
    using real = typename G::real;
    using R2 = Two<real>;
    constexpr int Q = G::Q;
    constexpr real k2 = (real)2, k3 = (real)3, k4 = (real)4;
    const R2 zero = two((real)0, (real)0);
    int pt[Q];
    real h[Q][3], U[Q], Y0[Q], dq3[Q], divu[Q];
    R2 A[Q], B[Q], dz[Q], dq[Q];
#pragma unroll
    for (int r = 0; r < Q; ++r) pt[r] = tab.node(d.lat + r * d.lstep);
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        const real *hp = gm.he(t.el, pt[r]) + d.dir * 3;
        h[r][0] = hp[0];
        h[r][1] = hp[1];
        h[r][2] = hp[2];
    }
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        U[r] = fma(ln.w[r].b.x, h[r][2], fma(ln.w[r].a.y, h[r][1], ln.w[r].a.x * h[r][0]));
        Y0[r] = fma(ln.z[r].x, U[r], fma(ln.v[r].b.x, h[r][2], fma(ln.v[r].a.y, h[r][1], ln.v[r].a.x * h[r][0])));
        A[r] = B[r] = dz[r] = dq[r] = zero;
        dq3[r] = divu[r] = (real)0;
    }
#pragma unroll
    for (int r = 0; r < Q - 1; ++r) {
        real Dr[Q], Dc[Q];  // row and column r
        tab.row(Dr, d.dir, r);
        tab.col(Dc, d.dir, r);
#pragma unroll
        for (int s = r + 1; s < Q; ++s) {
            const R2 wa = sub2(ln.w[s].a, ln.w[r].a), wb = sub2(ln.w[s].b, ln.w[r].b);
            const R2 va = sub2(ln.v[s].a, ln.v[r].a), vb = sub2(ln.v[s].b, ln.v[r].b);
            const R2 zz = sub2(ln.z[s], ln.z[r]);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                // Row m, its partner's values minus its own = sign * the differences.
                const int m = side ? s : r;
                const real D = side ? -Dc[s] : Dr[s];
                const real tt = fma(wb.x, h[m][2], fma(wa.y, h[m][1], wa.x * h[m][0]));
                const real x0 = U[m] + U[m];
                const real X = D * (side ? x0 - tt : x0 + tt), Y = D * fma(side ? -ln.z[m].x : ln.z[m].x, tt, Y0[m]);
                A[m] = fma2(va, two(X, X), fma2(wa, two(Y, Y), A[m]));
                B[m] = fma2(vb, two(X, X), fma2(wb, two(Y, Y), B[m]));
                dz[m] = fma2(two(D, D), zz, dz[m]);
                dq[m] = fma2(two(D, D), va, dq[m]);
                dq3[m] = fma(D, vb.x, dq3[m]);
                divu[m] = fma(D, tt, divu[m]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        const real rr = ln.z[r].x, Ur = U[r];
        const real sg = tab.sum(d.dir, r);
        const real divq = fma(dq3[r], h[r][2], fma(dq[r].y, h[r][1], dq[r].x * h[r][0]));
        const real S = fma(rr, divu[r], fma(Ur, dz[r].x, divq));
        const real cw = fma(k2 * sg, Y0[r], S), cv = fma(k3 * sg, Ur, k2 * divu[r]);
        const real dp = k4 * fma(sg, ln.z[r].y, dz[r].y);
        R2 a = fma2(ln.w[r].a, two(cw, cw), fma2(ln.v[r].a, two(cv, cv), A[r]));
        R2 b = fma2(ln.w[r].b, two(cw, cw), fma2(ln.v[r].b, two(cv, cv), B[r]));
        a = fma2(two(h[r][0], h[r][1]), two(dp, dp), a);
        b.x = fma(h[r][2], dp, b.x);
        convec_finish<G>(d, sm, gm, t.el, d.base + r * d.step, pt[r], id[r], a, b, fma(sg, fma(rr, Ur, Y0[r]), S), npoin, Rmass,
                         Rmom, Rener);
    }
}

template <class G>
__device__ __forceinline__ void convec_pass(ConvecLine<G> &ln, const GroupThread<G> &t, int ip,
                                            const ConvecShared<G> &sm, const GroupRows<G, true> &tab, const GroupMetric<G> &gm,
                                              const int (&id)[G::R], int npoin,
                                            typename G::real *__restrict__ Rmass,
                                            typename G::real *__restrict__ Rmom,
                                            typename G::real *__restrict__ Rener)
{
    if (!t.active) return;
    const ConvecDir<G> d(t, ip);
    if (!d.first || G::S > 1) {
#pragma unroll
        for (int s = 0; s < G::Q; ++s) {
            const int o = d.base + s * d.step;
            ln.set(s, sm.W()[o], sm.V()[o], sm.Z()[o]);
        }
    }
    if constexpr (G::S == 1 && convec_all_points<typename G::real, G::P>()) {
        convec_pairs<G>(ln, t, d, sm, tab, gm, id, npoin, Rmass, Rmom, Rener);
    } else if constexpr (G::S == 1) {
        convec_points<G, 0>(ln, t, d, sm, tab, gm, id, npoin, Rmass, Rmom, Rener);
    } else {
        if (t.seg == 0)
            convec_points<G, 0>(ln, t, d, sm, tab, gm, id, npoin, Rmass, Rmom, Rener);
        else
            convec_points<G, 1>(ln, t, d, sm, tab, gm, id, npoin, Rmass, Rmom, Rener);
    }
}

template <class G, int MINB>
__global__ void __launch_bounds__(G::NT, MINB)
    convec_kernel(int nelem, int npoin, const int *__restrict__ connec,
                  const typename G::real *__restrict__ He, const typename G::real *__restrict__ gpvol,
                  const typename G::real *__restrict__ u, const typename G::real *__restrict__ q,
                  const typename G::real *__restrict__ rho, const typename G::real *__restrict__ pr,
                  const typename G::real *__restrict__ E, const int *__restrict__ inv,
                  const typename G::real *__restrict__ dlxigp_ip, const TableScratch *__restrict__ tabs,
                  typename G::real *__restrict__ Rmass, typename G::real *__restrict__ Rmom,
                  typename G::real *__restrict__ Rener)
{
    using real = typename G::real;
    constexpr int Q = G::Q, N = G::N, R = G::R;
    static_assert(G::S <= 2, "one or two segments per line");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    const GroupThread<G> t(tid);
    const ConvecShared<G> sm{smem_raw, t.el};
    const int r0 = t.seg * R;
    const int e0 = blockIdx.x * G::NE;
    const GroupMetric<G> gm(smem_raw, smem_raw + G::HEB, sm.bar(), He, gpvol, e0, nelem, tid);
    ConvecLine<G> ln;
    int id[R];  // the nodes of the thread's points of its zeta line (-1: none)
    {
        const int e = e0 + t.el;
        const size_t np = (size_t)npoin;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const bool ok = t.active && e < nelem && (R * G::S == Q || r0 + k < Q);
            const int row = ok ? GroupTables<G, true>::node(inv, t.template lat<2>(r0 + k)) : 0;
            const int v = ok ? ldg_once(connec + (size_t)row * nelem + e) - 1 : -1;
            id[k] = (unsigned)v < (unsigned)npoin ? v : -1;
        }
        sm.tab().build(inv, dlxigp_ip, tid);
        real f[R][9];
        auto gather = [&](auto load) {
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const bool ok = id[k] >= 0;  // a missing node reads as zeros
                const size_t p = ok ? (size_t)id[k] : 0;
                f[k][0] = ok ? load(u + p) : (real)0;
                f[k][1] = ok ? load(u + np + p) : (real)0;
                f[k][2] = ok ? load(u + 2 * np + p) : (real)0;
                f[k][3] = ok ? load(E + p) : (real)0;
                f[k][4] = ok ? load(q + p) : (real)0;
                f[k][5] = ok ? load(q + np + p) : (real)0;
                f[k][6] = ok ? load(q + 2 * np + p) : (real)0;
                f[k][7] = ok ? load(rho + p) : (real)0;
                f[k][8] = ok ? load(pr + p) : (real)0;
            }
        };
        if (convec_close<real, G::P>() && group_close<G>(id))
            gather([](const real *x) { return ldg(x); });
        else
            gather([](const real *x) { return ldg_once(x); });
        const int base = t.rec0(2);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const real H = f[k][3] + (real)0.5 * fma(f[k][2], f[k][2], fma(f[k][1], f[k][1], f[k][0] * f[k][0]));
            Four<real> w, v;
            w.a = two(f[k][0], f[k][1]);
            w.b = two(f[k][2], H);
            v.a = two(f[k][4], f[k][5]);
            v.b = two(f[k][6], f[k][8]);
            if (t.active && (R * G::S == Q || r0 + k < Q)) {
                const int o = base + (r0 + k) * G::template step<2>();
                sm.W()[o] = w;
                sm.V()[o] = v;
                sm.Z()[o] = f[k][7];
                if constexpr (ConvecShared<G>::kSlots == 0) sm.node()[o] = id[k];
            }
            if (G::S == 1) ln.set(k, w, v, f[k][7]);
        }
    }
    __syncthreads();
    // Bounded wait for the bulk copies; a wait that ran out is reported and
    // nothing is assembled (every thread learns it at the barrier below).
    const GroupRows<G, true> tab(sm.tab());
    const bool ok = gm.wait(sm.bar());
    auto pass = [&](int ip) {
        if (ip == 2) grid_dependency_wait();  // the residuals are zeroed
        convec_pass<G>(ln, t, ip, sm, tab, gm, id, npoin, Rmass, Rmom, Rener);
        if (ip < 2 && __syncthreads_or(!ok)) {
            if (tid == 0) report_wait_fault(tabs);
            grid_dependency_wait();  // the kernel never ends ahead of the zeroing
            return false;
        }
        return true;
    };
    if constexpr (convec_rolled<G::P>()) {
#pragma unroll 1
        for (int ip = 0; ip < 3; ++ip)
            if (!pass(ip)) return;
    } else {
#pragma unroll
        for (int ip = 0; ip < 3; ++ip)
            if (!pass(ip)) return;
    }
}

template <typename real, int P>
cudaError_t launch_convec_p(const ConvecArgs<real> &a, const TableScratch *tabs, cudaStream_t st)
{
    using G = ConvecGeom<real, P>;
    constexpr size_t smem = ConvecShared<G>::kBytes;
    static_assert(smem <= 227 * 1024, "shared memory budget");
    if (!tabs) return cudaErrorInvalidValue;
    auto kern = convec_kernel<G, convec_minb<real, P>()>;
    static std::atomic<unsigned long long> allowed{0};
    const cudaError_t err = allow_smem(allowed, kern, smem, convec_carveout<real, P>());
    if (err != cudaSuccess) return err;
    const unsigned ngroups = (unsigned)((a.nelem + G::NE - 1) / G::NE);
    return launch_after(kern, ngroups, G::NT, smem, st, a.nelem, a.npoin, a.connec, a.He, a.gpvol, a.u, a.q, a.rho,
                        a.pr, a.E, a.invAtoIJK, a.dlxigp_ip, tabs, a.Rmass, a.Rmom, a.Rener);
}

}  // namespace

template <typename real>
cudaError_t launch_convec_plain(int porder, const ConvecArgs<real> &a, const TableScratch *tabs, cudaStream_t st)
{
    switch (porder) {
    case 1: return launch_convec_p<real, 1>(a, tabs, st);
    case 2: return launch_convec_p<real, 2>(a, tabs, st);
    case 3: return launch_convec_p<real, 3>(a, tabs, st);
    case 4: return launch_convec_p<real, 4>(a, tabs, st);
    case 5: return launch_convec_p<real, 5>(a, tabs, st);
    case 6: return launch_convec_p<real, 6>(a, tabs, st);
    case 7: return launch_convec_p<real, 7>(a, tabs, st);
    case 8: return launch_convec_p<real, 8>(a, tabs, st);
    default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_convec_plain<float>(int, const ConvecArgs<float> &, const TableScratch *, cudaStream_t);
template cudaError_t launch_convec_plain<double>(int, const ConvecArgs<double> &, const TableScratch *, cudaStream_t);

}  // namespace msod
