// msod_diffu.cu -- plain FP32 hex GLL diffusion residual (FP64: msod_diffu64.cu).
//
// Computes what full_diffusion_ijk computes (elem_diffu.f90:10-197):
//   pass 1 (per point b): grad rho, grad T, grad u; mu_f = mu_fluid + rho mu_sgs;
//     tau = (mu_f + mu_e)(grad u + grad u^T) - 2/3 mu_f div u I;  tauU = tau u
//   pass 2 (per output node a):
//     Rmass += nu_e(a)   sum_{d,b} w_d(a,b) . grad rho(b)
//     Rener +=           sum_{d,b} w_d(a,b) . (tauU(b) + kappa_e(a) grad T(b))
//     Rmom_m +=          sum_{d,b} w_d(a,b) . tau_m(b)
//   with w_d(a,b)_i = He(i,d,b) gpvol(b) dlxigp_ip(b,d,iso_d(a)) over the
//   points b of a's d-line, nu_e(a) = mu_e/rho and
//   kappa_e(a) = mu_fluid Cp/Pr + mu_e Cp/Pr + Cp rho mu_sgs / 0.9 evaluated at
//   the output node (elem_diffu.f90:143-146).
//
// Design (one group of NE elements per block, one thread per GLL line,
// msod_group.cuh):
//   0. bulk copies bring the group's He and gpvol; each thread gathers the
//      points of its zeta line (node fields through connec, mu_e and mu_sgs in
//      the element layout) and keeps them in registers; rho, T and u go to the
//      shared-memory lattice as records;
//   1. xi and eta passes store the iso-parametric derivatives of the five
//      fields;
//   2. zeta stage, at the points of the thread's zeta line: zeta derivatives
//      from the line's registers, physical gradients and stress, and the
//      contravariant fluxes gpvol He(:,d)^T X of the six vectors X = grad rho,
//      tauU, grad T, tau rows 1..3; the xi and eta fluxes go to shared memory
//      (over the derivatives), the zeta divergence stays in registers;
//   3. xi and eta passes apply the transposed 1-D derivative matrix to their
//      fluxes, in place;
//   4. the thread of the zeta line adds the three divergences of its points,
//      forms the residuals and scatter-adds them with red.global.add.
// The viscosities, nu_e, kappa_e and the node ids never leave the registers of
// the zeta line's thread.  The 1-D derivative matrices come from shared memory or,
// on large meshes, from the constant bank (diffu_const_points).
#include <cuda_runtime.h>

#include "msod_group.cuh"

namespace msod {
namespace {

// 1-D derivative matrices of the current call, per porder (large meshes: copied
// from the per-call table area by prepare_diffu_plain, ahead of the zeroing).
__constant__ float c_Df[MSOD_MAX_PORDER + 1][kTableDMax];

// The matrices' rows: shared-memory tables of the block, or (CONSTD) operands
// from the constant bank.
template <class G, bool CONSTD>
struct DiffuRows {
    GroupRows<G, false> tab;
    __device__ __forceinline__ explicit DiffuRows(const GroupTables<G, false> &t) : tab(t) {}
    __device__ __forceinline__ void row(typename G::real (&v)[G::Q], int dir, int r) const { tab.row(v, dir, r); }
};
template <class G>
struct DiffuRows<G, true> {
    __device__ __forceinline__ explicit DiffuRows(const GroupTables<G, false> &) {}
    __device__ __forceinline__ void row(typename G::real (&v)[G::Q], int dir, int r) const
    {
#pragma unroll
        for (int c = 0; c < G::Q; ++c) v[c] = c_Df[G::P][(dir * G::Q + r) * G::Q + c];
    }
};

// Viscosity source of the diffusion kernel: the mu_e array, or one value per
// element (mu_e(e, a) = rho(a) nu_elem(e)).
enum { VISC_MU_E = 0, VISC_NU_ELEM = 1 };

// Elements per block and blocks per SM that the register budget allows for.  The
// comparisons stand as they were made; a call takes now (ms): porder 1 128^3 0.326,
// 2 100^3 0.592, 3 80^3 0.743, 4 64^3 0.946, 5 51^3 0.933, 6 40^3 0.874, 7 32^3 0.665, 8
// 26^3 0.691.
// Whole warps of lines (5 x 25 lines at porder 4: 125 of 128 threads) count
// most, then the L1 that the blocks' shared memory leaves for the gathers'
// lines in flight (porder 5: three blocks of 65.6 KB, within a 196 KB carveout,
// 1.00 ms on 51^3; of 67.7 KB, beyond it, 1.37).  ms: porder 4 (64^3) 5 elements at three blocks 1.030, at four (128
// registers, spills) 1.077; before the divisions left the point work, 8
// elements at two blocks took 1.302, 9 1.284, 4 at four 1.236, where 5 took
// 1.152.  Porder 5 (51^3) 3 elements at three 0.996, 4 at two 1.053; 6 (40^3) 3
// 1.094, 2 at two 1.156; 7 (32^3) 2 at two 0.853; 8 (26^3) 1 0.717; 3 (80^3) 8 at
// the compiler's choice 0.779, at four 0.795; 2 (100^3) 16 at four 0.619, at the
// compiler's choice 0.717.
template <int P>
constexpr int diffu_ne()
{
    constexpr int n[9] = {0, 32, 16, 8, 5, 3, 3, 2, 1};
    return n[P];
}
template <int P>
constexpr int diffu_minb()
{
    constexpr int n[9] = {0, 1, 4, 1, 3, 3, 1, 2, 1};
    return n[P];
}
// Where a few KB less let the blocks of an SM fit in 196 KB, which leaves 60 KB of L1
// instead of 28: the eta derivative of u3 is written over u3 (a barrier more), and at
// porders 3 and 7 the points' gpvol come straight from global memory.  On 12 M element
// points, staged / so, ms: porder 6 0.588 / 0.461 (gpvol too 0.480), 7 0.594 / 0.480, 3
// 0.284 / 0.276; with elements in random order 0.938 / 0.726, 0.824 / 0.662, 0.802 / 0.644.
template <int P>
constexpr bool diffu_over()
{
    return P == 3 || P == 6 || P == 7;
}
template <int P>
constexpr bool diffu_gpvol_staged()
{
    return P != 3 && P != 7;
}
// Blocks of closely numbered elements gather through the L1 (group_close).  On 12 M
// element points in elements with nodes of their own, past it / through it, ms: porder 3
// 0.473 / 0.410, 4 0.523 / 0.420, 6 0.835 / 0.533 (with the smaller shared memory); on a
// mesh numbered along x the rule costs nothing there (3 0.281 / 0.276, 4 0.364 / 0.349),
// at the others it costs 1-6 % (7 0.480 / 0.489) and the former line form, for which
// lanes ran along an element's lattice, was not faster (5 0.580, 7 0.785, 8 0.973).
template <int P>
constexpr bool diffu_close()
{
    return P == 3 || P == 4 || P == 6;
}
template <int P>
using DiffuGeom = GroupGeom<float, P, diffu_ne<P>(), 1, P == 1, diffu_gpvol_staged<P>()>;

// Element points from which the kernel takes its matrices from the constant
// bank.  That saves it registers and shared-memory loads, and at porders 5 and 6
// the L1 that the tables' shared memory costs (ms, bank / shared memory: porder
// 5 51^3 0.996 / 1.327, 6 40^3 1.094 / 1.405, 4 64^3 1.030 / 1.046, 3 80^3 0.779 /
// 0.854, 2 100^3 0.619 / 0.680, 1 128^3 0.392 / 0.425, 7 32^3 0.853 / 0.882, 8 26^3
// 0.717 / 0.754), but costs the call the table kernel and a copy to the bank,
// ~6 us: the lines below are where the two meet.
template <int P>
constexpr long long diffu_const_points()
{
    return P == 5 || P == 6 ? 500000 : (P == 4 ? 12000000 : 3000000);
}

// Shared memory of a block.  X1 and X3 hold the xi and eta derivatives of
// (rho, T, u1, u2), then the fluxes (and divergences) of grad rho, tauU, grad T
// and tau_1; X2 holds the node fields (rho, T, u1, u2), then (Y1, Y3, eight bytes
// each) the fluxes of tau_2, tau_3: as halves of 16-byte records, which each direction
// reads and writes alone, they took twice the wavefronts (porder 4 64^3 0.951 / 0.925
// ms, 5 51^3 0.904 / 0.886, 7 32^3 0.791 / 0.770).  Not at porder 3, whose rows of four
// conflict as pairs too (80^3 0.718 / 0.733).  kOver: the eta derivative of u3 takes u3's
// place (each eta line's thread reads its u3 first; the xi lines are done with it).
template <class G>
struct DiffuShared {
    using real = typename G::real;
    static constexpr bool kPairs = G::P != 3;
    static constexpr size_t k1 = G::HEB + G::GPB + 16;
    static constexpr size_t k2 = k1 + G::NREC * sizeof(Four<real>);
    static constexpr size_t k3 = k2 + G::NPR * sizeof(Four<real>);
    static constexpr size_t kU = k3 + G::NREC * sizeof(Four<real>);
    static constexpr size_t kE1 = kU + G::NSC * sizeof(real);
    static constexpr bool kOver = diffu_over<G::P>();
    static constexpr size_t kE3 = kOver ? kU : kE1 + G::NSC * sizeof(real);
    static constexpr size_t kTab = ((kOver ? kE1 : kE3) + G::NSC * sizeof(real) + 15) / 16 * 16;
    static constexpr size_t bytes(bool constd) { return kTab + (constd ? 0 : GroupTables<G, false>::kBytes); }
    unsigned char *base;
    int el;  // the thread's element
    __device__ __forceinline__ unsigned long long *bar() const
    {
        return reinterpret_cast<unsigned long long *>(base + G::HEB + G::GPB);
    }
    __device__ __forceinline__ GroupTables<G, false> tab() const { return GroupTables<G, false>{base + kTab}; }
    __device__ __forceinline__ Four<real> *X1() const { return reinterpret_cast<Four<real> *>(base + k1); }
    __device__ __forceinline__ Four<real> *X2() const { return reinterpret_cast<Four<real> *>(base + k2); }
    __device__ __forceinline__ Four<real> *X3() const { return reinterpret_cast<Four<real> *>(base + k3); }
    // The flux pair (tau_2, tau_3) of record o along xi and eta.
    __device__ __forceinline__ Two<real> *Y1() const { return reinterpret_cast<Two<real> *>(base + k2) + el * G::HK; }
    __device__ __forceinline__ Two<real> *Y3() const { return Y1() + G::NPR; }
    template <int DIR>
    __device__ __forceinline__ Two<real> &pair(int o) const
    {
        if constexpr (kPairs)
            return (DIR == 0 ? Y1() : Y3())[o];
        else
            return DIR == 0 ? X2()[o].a : X2()[o].b;
    }
    __device__ __forceinline__ void put_pairs(int o, const Two<real> &xi, const Two<real> &eta) const
    {
        if constexpr (kPairs) {
            Y1()[o] = xi;
            Y3()[o] = eta;
        } else {
            Four<real> s;
            s.a = xi;
            s.b = eta;
            X2()[o] = s;
        }
    }
    __device__ __forceinline__ Four<real> pairs(int o) const
    {
        if constexpr (kPairs) {
            Four<real> s;
            s.a = Y1()[o];
            s.b = Y3()[o];
            return s;
        } else {
            return X2()[o];
        }
    }
    __device__ __forceinline__ real *U3() const { return reinterpret_cast<real *>(base + kU) + el * G::SK; }   // u3
    __device__ __forceinline__ real *E1() const { return reinterpret_cast<real *>(base + kE1) + el * G::SK; }  // its xi derivative
    __device__ __forceinline__ real *E3() const { return reinterpret_cast<real *>(base + kE3) + el * G::SK; }  // its eta derivative
};

// Derivatives of the five fields along the thread's line in direction DIR.
template <class G, int DIR, bool CONSTD>
__device__ __forceinline__ void diffu_grad(const GroupThread<G> &t, const DiffuShared<G> &sm, const DiffuRows<G, CONSTD> &tab)
{
    using real = typename G::real;
    using R2 = Two<real>;
    constexpr int Q = G::Q;
    const int base = t.rec0(DIR);
    Four<real> f[Q];
    real u3[Q];
#pragma unroll
    for (int c = 0; c < Q; ++c) {
        f[c] = sm.X2()[base + c * G::template step<DIR>()];
        u3[c] = sm.U3()[base + c * G::template step<DIR>()];
    }
    real D[Q][Q];  // all rows before the first store: no load waits behind one
#pragma unroll
    for (int r = 0; r < Q; ++r) tab.row(D[r], DIR, r);
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        Four<real> g;
        g.a = g.b = two((real)0, (real)0);
        real g3 = (real)0;
#pragma unroll
        for (int c = 0; c < Q; ++c) {
            g.a = fma2(two(D[r][c], D[r][c]), f[c].a, g.a);
            g.b = fma2(two(D[r][c], D[r][c]), f[c].b, g.b);
            g3 = fma(D[r][c], u3[c], g3);
        }
        const int o = base + r * G::template step<DIR>();
        (DIR == 0 ? sm.X1() : sm.X3())[o] = g;
        (DIR == 0 ? sm.E1() : sm.E3())[o] = g3;
    }
}

// Weak divergence of the thread's line in direction DIR, in place.
template <class G, int DIR, bool CONSTD>
__device__ __forceinline__ void diffu_div(const GroupThread<G> &t, const DiffuShared<G> &sm, const DiffuRows<G, CONSTD> &tab)
{
    using real = typename G::real;
    using R2 = Two<real>;
    constexpr int Q = G::Q;
    const int base = t.rec0(DIR);
    Four<real> *X = DIR == 0 ? sm.X1() : sm.X3();
    Four<real> f[Q];
    R2 f2[Q];
#pragma unroll
    for (int c = 0; c < Q; ++c) {
        const int o = base + c * G::template step<DIR>();
        f[c] = X[o];
        f2[c] = sm.template pair<DIR>(o);
    }
    real D[Q][Q];
#pragma unroll
    for (int c = 0; c < Q; ++c) tab.row(D[c], DIR, c);
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        Four<real> s;
        R2 s2 = two((real)0, (real)0);
        s.a = s.b = s2;
#pragma unroll
        for (int c = 0; c < Q; ++c) {
            const R2 Dc = two(D[c][r], D[c][r]);
            s.a = fma2(Dc, f[c].a, s.a);
            s.b = fma2(Dc, f[c].b, s.b);
            s2 = fma2(Dc, f2[c], s2);
        }
        const int o = base + r * G::template step<DIR>();
        X[o] = s;
        sm.template pair<DIR>(o) = s2;
    }
}

template <class G, int VISC, int MINB, bool CONSTD>
__global__ void __launch_bounds__(G::NT, MINB)
    diffu_kernel(int nelem, int npoin, const int *__restrict__ connec, const typename G::real *__restrict__ He,
                 const typename G::real *__restrict__ gpvol, const int *__restrict__ inv,
                 const typename G::real *__restrict__ dlxigp_ip, const TableScratch *__restrict__ tabs,
                 typename G::real Cp, typename G::real Pr, const typename G::real *__restrict__ rho,
                 const typename G::real *__restrict__ u, const typename G::real *__restrict__ Tem,
                 const typename G::real *__restrict__ mu_fluid, const typename G::real *__restrict__ mu_e,
                 const typename G::real *__restrict__ mu_sgs, const typename G::real *__restrict__ nu_elem,
                 typename G::real *__restrict__ Rmass, typename G::real *__restrict__ Rmom,
                 typename G::real *__restrict__ Rener)
{
    using real = typename G::real;
    using R2 = Two<real>;
    constexpr int Q = G::Q;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, e0 = blockIdx.x * G::NE;
    const GroupThread<G> t(tid);
    const DiffuShared<G> sm{smem_raw, t.el};
    const GroupMetric<G> gm(smem_raw, smem_raw + G::HEB, sm.bar(), He, gpvol, e0, nelem, tid);
    const int e = e0 + t.el, base = t.rec0(2);
    const bool in = t.active && e < nelem;
    const size_t np = (size_t)npoin;

    // The points of the thread's zeta line (a missing node reads as zeros).
    int id[Q], pt[Q];
    R2 rT[Q], u12[Q];
    real u3[Q], muf[Q], ms[Q], me[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) pt[k] = GroupTables<G, false>::node(inv, t.template lat<2>(k));
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const int v = in ? ldg_once(connec + (size_t)pt[k] * nelem + e) - 1 : -1;
        id[k] = (unsigned)v < (unsigned)npoin ? v : -1;
    }
    if (!CONSTD) sm.tab().build(inv, dlxigp_ip, tid);
    real gvr[G::GPSTAGED ? 1 : Q];
    if constexpr (!G::GPSTAGED)
#pragma unroll
        for (int k = 0; k < Q; ++k) gvr[k] = in ? ldg_once(gpvol + (size_t)e * G::N + pt[k]) : (real)0;
    // mu_sgs and mu_e ahead of the node fields, or between them: as measured (porder 4
    // 0.349 against 0.370 ms, 3 0.286 / 0.301; but 5 0.414 / 0.394, 8 0.599 / 0.576).
    constexpr bool kEarly = G::P == 3 || G::P == 4;
    if constexpr (kEarly)
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const size_t i = in ? (size_t)pt[k] * nelem + e : 0;
            ms[k] = in ? ldg_once(mu_sgs + i) : (real)0;
            me[k] = (VISC == VISC_MU_E && in) ? ldg_once(mu_e + i) : (real)0;
        }
    auto gather = [&](auto load) {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const bool ok = id[k] >= 0;
            const size_t p = ok ? (size_t)id[k] : 0, i = in ? (size_t)pt[k] * nelem + e : 0;
            rT[k] = two(ok ? load(rho + p) : (real)0, ok ? load(Tem + p) : (real)0);
            u12[k] = two(ok ? load(u + p) : (real)0, ok ? load(u + np + p) : (real)0);
            u3[k] = ok ? load(u + 2 * np + p) : (real)0;
            muf[k] = ok ? load(mu_fluid + p) : (real)0;
            if constexpr (!kEarly) {
                ms[k] = in ? ldg_once(mu_sgs + i) : (real)0;
                me[k] = (VISC == VISC_MU_E && in) ? ldg_once(mu_e + i) : (real)0;
            }
        }
    };
    if (diffu_close<G::P>() && group_close<G>(id))
        gather([](const real *x) { return ldg(x); });
    else
        gather([](const real *x) { return ldg_once(x); });
    if (VISC == VISC_NU_ELEM) {
        const real nu = in ? ldg(nu_elem + e) : (real)0;
#pragma unroll
        for (int k = 0; k < Q; ++k) me[k] = rT[k].x * nu;
    }
    if (t.active)
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            Four<real> f;
            f.a = rT[k];
            f.b = u12[k];
            sm.X2()[base + k * G::template step<2>()] = f;
            sm.U3()[base + k * G::template step<2>()] = u3[k];
        }
    __syncthreads();
    const DiffuRows<G, CONSTD> tab(sm.tab());
    if (t.active) diffu_grad<G, 0, CONSTD>(t, sm, tab);
    if constexpr (DiffuShared<G>::kOver) __syncthreads();
    if (t.active) diffu_grad<G, 1, CONSTD>(t, sm, tab);
    // Bounded wait for the bulk copies; a wait that ran out is reported and
    // nothing is assembled.
    const bool ok = gm.wait(sm.bar());
    if (__syncthreads_or(!ok)) {
        if (tid == 0) report_wait_fault(tabs);
        grid_dependency_wait();  // the kernel never ends ahead of the zeroing
        return;
    }
    // Zeta stage: acc[r][0..2] = the zeta divergence at point r of the fluxes of
    // (grad rho, tauU), (grad T, tau_1), (tau_2, tau_3).
    const real CpPr = Cp / Pr, Cp09 = Cp / (real)0.9;
    R2 acc[Q][3];
    real nu[Q], kap[Q];
#pragma unroll
    for (int r = 0; r < Q; ++r) acc[r][0] = acc[r][1] = acc[r][2] = two((real)0, (real)0);
    if (t.active) {
        real Dn[Q];
        tab.row(Dn, 2, 0);
#pragma unroll
        for (int c = 0; c < Q; ++c) {
            const int o = base + c * G::template step<2>();
            real Dr[Q], H[9];
#pragma unroll
            for (int j = 0; j < Q; ++j) Dr[j] = Dn[j];
            const real *hp = gm.he(t.el, pt[c]);
#pragma unroll
            for (int j = 0; j < 9; ++j) H[j] = hp[j];
            real gv;
            if constexpr (G::GPSTAGED)
                gv = *gm.vol(t.el, pt[c]);
            else
                gv = gvr[c];
            const Four<real> gx = sm.X1()[o], ge = sm.X3()[o];
            R2 za = two((real)0, (real)0), zb = za;
            real z3 = (real)0;
            if (c + 1 < Q) tab.row(Dn, 2, c + 1);  // before this point's stores
#pragma unroll
            for (int j = 0; j < Q; ++j) {
                const real D = Dr[j];
                za = fma2(two(D, D), rT[j], za);
                zb = fma2(two(D, D), u12[j], zb);
                z3 = fma(D, u3[j], z3);
            }
            const R2 xa = gx.a, xb = gx.b, ea = ge.a, eb = ge.b;
            const real x3 = sm.E1()[o], e3 = sm.E3()[o];
            // Physical gradients: (grad rho, grad T)_i and (grad u1, grad u2)_i as pairs.
            R2 gRT[3], gU[3];
            real gU3[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const R2 h0 = two(H[i], H[i]), h1 = two(H[3 + i], H[3 + i]), h2 = two(H[6 + i], H[6 + i]);
                gRT[i] = fma2(h2, za, fma2(h1, ea, mul2(h0, xa)));
                gU[i] = fma2(h2, zb, fma2(h1, eb, mul2(h0, xb)));
                gU3[i] = fma(H[6 + i], z3, fma(H[3 + i], e3, H[i] * x3));
            }
            const real r = rT[c].x;
            const real mf = muf[c] + r * ms[c], mt = mf + me[c];
            const real cut = mf * ((real)2 / (real)3) * (gU[0].x + gU[1].y + gU3[2]);
            const real t00 = mt * (gU[0].x + gU[0].x) - cut, t11 = mt * (gU[1].y + gU[1].y) - cut,
                       t22 = mt * (gU3[2] + gU3[2]) - cut;
            const real t01 = mt * (gU[1].x + gU[0].y), t02 = mt * (gU[2].x + gU3[0]), t12 = mt * (gU[2].y + gU3[1]);
            const real v0 = u12[c].x, v1 = u12[c].y, v2 = u3[c];
            const real q0 = fma(t02, v2, fma(t01, v1, t00 * v0)), q1 = fma(t12, v2, fma(t11, v1, t01 * v0)),
                       q2 = fma(t22, v2, fma(t12, v1, t02 * v0));
            // The six vectors as pairs: (grad rho, tauU), (grad T, tau_1), (tau_2, tau_3).
            const R2 v[3][3] = {{two(gRT[0].x, q0), two(gRT[1].x, q1), two(gRT[2].x, q2)},
                                {two(gRT[0].y, t00), two(gRT[1].y, t01), two(gRT[2].y, t02)},
                                {two(t01, t02), two(t11, t12), two(t12, t22)}};
            R2 F[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const real w0 = gv * H[d * 3], w1 = gv * H[d * 3 + 1], w2 = gv * H[d * 3 + 2];
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    F[d][x] = fma2(two(w2, w2), v[x][2], fma2(two(w1, w1), v[x][1], mul2(two(w0, w0), v[x][0])));
            }
            Four<real> s;
            s.a = F[0][0];
            s.b = F[0][1];
            sm.X1()[o] = s;
            s.a = F[1][0];
            s.b = F[1][1];
            sm.X3()[o] = s;
            sm.put_pairs(o, F[0][2], F[1][2]);
#pragma unroll
            for (int rr = 0; rr < Q; ++rr) {
                const real D = Dr[rr];
#pragma unroll
                for (int x = 0; x < 3; ++x) acc[rr][x] = fma2(two(D, D), F[2][x], acc[rr][x]);
            }
            nu[c] = me[c] / r;
            kap[c] = fma(muf[c] + me[c], CpPr, Cp09 * (r * ms[c]));
        }
    }
    __syncthreads();
    if (t.active) {
        diffu_div<G, 0, CONSTD>(t, sm, tab);
        diffu_div<G, 1, CONSTD>(t, sm, tab);
    }
    grid_dependency_wait();  // the residuals are zeroed
    __syncthreads();
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (id[k] < 0) continue;
        const int o = base + k * G::template step<2>();
        const Four<real> x1 = sm.X1()[o], x2 = sm.pairs(o), x3 = sm.X3()[o];
        const R2 s0 = add2(add2(acc[k][0], x1.a), x3.a), s1 = add2(add2(acc[k][1], x1.b), x3.b),
                 s2 = add2(add2(acc[k][2], x2.a), x2.b);
        red_add(Rmass + id[k], nu[k] * s0.x);
        red_add(Rener + id[k], fma(kap[k], s1.x, s0.y));
        red_add(Rmom + id[k], s1.y);
        red_add(Rmom + np + id[k], s2.x);
        red_add(Rmom + 2 * np + id[k], s2.y);
    }
}

// Whether the call reads its matrices from the constant bank.
template <int P>
bool diffu_const(const DiffuArgs<float> &a)
{
    return (long long)a.nelem * DiffuGeom<P>::N >= diffu_const_points<P>();
}

template <int P>
cudaError_t prepare_diffu_p(const DiffuArgs<float> &a, TableScratch *tabs, cudaStream_t st)
{
    if (!diffu_const<P>(a)) return cudaSuccess;
    const cudaError_t err = launch_table_prep(P, a, tabs, st);
    if (err != cudaSuccess) return err;
    constexpr size_t row = sizeof(float) * kTableDMax;
    return cudaMemcpyToSymbolAsync(c_Df, tabs->Df, sizeof(float) * 3 * (P + 1) * (P + 1), row * P,
                                   cudaMemcpyDeviceToDevice, st);
}

template <int P, int VISC, bool CONSTD>
cudaError_t launch_diffu_pc(const DiffuArgs<float> &a, const TableScratch *tabs, cudaStream_t st)
{
    using G = DiffuGeom<P>;
    constexpr size_t smem = DiffuShared<G>::bytes(CONSTD);
    static_assert(smem <= 227 * 1024, "shared memory budget");
    auto kern = diffu_kernel<G, VISC, diffu_minb<P>(), CONSTD>;
    static std::atomic<unsigned long long> allowed{0};
    const cudaError_t err = allow_smem(allowed, kern, smem);
    if (err != cudaSuccess) return err;
    const unsigned grid = (unsigned)((a.nelem + G::NE - 1) / G::NE);
    return launch_after(kern, grid, G::NT, smem, st, a.nelem, a.npoin, a.connec, a.He, a.gpvol, a.invAtoIJK,
                        a.dlxigp_ip, tabs, a.Cp, a.Pr, a.rho, a.u, a.Tem, a.mu_fluid, a.mu_e, a.mu_sgs, a.nu_elem,
                        a.Rmass, a.Rmom, a.Rener);
}
template <int P, int VISC>
cudaError_t launch_diffu_pn(const DiffuArgs<float> &a, const TableScratch *tabs, cudaStream_t st)
{
    return diffu_const<P>(a) ? launch_diffu_pc<P, VISC, true>(a, tabs, st)
                             : launch_diffu_pc<P, VISC, false>(a, tabs, st);
}

template <int P>
cudaError_t launch_diffu_p(const DiffuArgs<float> &a, const TableScratch *tabs, cudaStream_t st)
{
    return a.nu_elem ? launch_diffu_pn<P, VISC_NU_ELEM>(a, tabs, st) : launch_diffu_pn<P, VISC_MU_E>(a, tabs, st);
}

}  // namespace

template <>
cudaError_t prepare_diffu_plain<float>(int porder, const DiffuArgs<float> &a, TableScratch *tabs, cudaStream_t st)
{
    switch (porder) {
    case 1: return prepare_diffu_p<1>(a, tabs, st);
    case 2: return prepare_diffu_p<2>(a, tabs, st);
    case 3: return prepare_diffu_p<3>(a, tabs, st);
    case 4: return prepare_diffu_p<4>(a, tabs, st);
    case 5: return prepare_diffu_p<5>(a, tabs, st);
    case 6: return prepare_diffu_p<6>(a, tabs, st);
    case 7: return prepare_diffu_p<7>(a, tabs, st);
    case 8: return prepare_diffu_p<8>(a, tabs, st);
    default: return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_diffu_plain<float>(int porder, const DiffuArgs<float> &a, const TableScratch *tabs, cudaStream_t st)
{
    switch (porder) {
    case 1: return launch_diffu_p<1>(a, tabs, st);
    case 2: return launch_diffu_p<2>(a, tabs, st);
    case 3: return launch_diffu_p<3>(a, tabs, st);
    case 4: return launch_diffu_p<4>(a, tabs, st);
    case 5: return launch_diffu_p<5>(a, tabs, st);
    case 6: return launch_diffu_p<6>(a, tabs, st);
    case 7: return launch_diffu_p<7>(a, tabs, st);
    case 8: return launch_diffu_p<8>(a, tabs, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace msod
