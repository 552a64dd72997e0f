// msod_visc.cu -- plain entropy-viscosity estimator for mu_e and the element
// features of the learned estimator.
//
// The reference consumes mu_e (elem_diffu.f90:19, mu_e(nelem,ngaus)) but
// contains no estimator; its numerical parameters name one
// (mod_numerical_params.f90:22-28: ce = 0.1, cmax = 0.5, cglob = 1,
// flag_normalise_entropy = 1).  This file writes the entropy-viscosity method
// of Guermond, Pasquetti & Popov (J. Comput. Phys. 230 (2011) 4248-4267) for
// one snapshot of the fields:
//   entropy      eta = rho/(gamma-1) * log(p / rho^gamma)
//   residual     R = div(eta u) - eta div u - u . grad eta      (per GLL point)
//                (the entropy equation's residual with the time derivative
//                replaced by its steady balance -eta div u - u.grad eta; R
//                vanishes where the discrete entropy flux is resolved and grows
//                across under-resolved fronts)
//   normalise    n_eta = || eta - mean(eta) ||_inf over the mesh (cglob = 1)
//   per element  h = (sum_g gpvol)^(1/3) / porder,
//                nu_max = cmax h max_e(|u| + c),  c = sqrt(gamma p / rho),
//                nu_E   = ce h^2 max_e |R| / n_eta,
//                nu     = min(nu_max, nu_E)
//   output       mu_e(e, a) = rho(a) nu(e)   in the reference's mu_e layout.
#include <cuda_runtime.h>

#include "msod_group.cuh"

namespace msod {

namespace {

// ---------------------------------------------------------------------------
// Entropy statistics over the nodes: sum, min and max of eta.
// ---------------------------------------------------------------------------
// Three kernels in a row, each started while the one ahead still runs: the
// statistics load and form eta before they wait for the initial values, the
// estimator and the features gather before they wait for the norm.
__global__ void entropy_stats_init(EntropyStats *st, int *count)
{
    grid_dependents_launch();
    st->sum = 0.0;
    st->kmin = f2key(3.0e38f);
    st->kmax = f2key(-3.0e38f);
    st->done = 0u;
    if (count) *count = 0;
}

// p is given directly (pr) or as rho * Rgas * T (Tem with Rgas > 0).
__global__ void entropy_stats_kernel(int npoin, const float *__restrict__ rho, const float *__restrict__ p_or_T,
                                     float Rgas, float gamma, EntropyStats *st)
{
    grid_dependents_launch();
    float s = 0.0f, mn = 3.0e38f, mx = -3.0e38f;
    auto add = [&](float r, float q) {
        const float p = Rgas > 0.0f ? r * Rgas * q : q;
        const float eta = r / (gamma - 1.0f) * (logf(p) - gamma * logf(r));
        s += eta;
        mn = fminf(mn, eta);
        mx = fmaxf(mx, eta);
    };
    // Four grid strides per trip, every load issued before the arithmetic
    // (eight loads in flight per thread instead of two).
    const int G = gridDim.x * blockDim.x;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (; i < npoin - 3 * G; i += 4 * G) {
        float r[4], q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r[k] = ldg(rho + i + k * G);
            q[k] = ldg(p_or_T + i + k * G);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) add(r[k], q[k]);
    }
    for (; i < npoin; i += G) add(ldg(rho + i), ldg(p_or_T + i));
    // Warp, then block reduction: one set of global atomics per block (the
    // atomics on these three words serialise in L2).
    double sd = (double)s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sd += __shfl_xor_sync(0xffffffffu, sd, o);
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    __shared__ double bs[32];
    __shared__ float bmn[32], bmx[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) {
        bs[warp] = sd;
        bmn[warp] = mn;
        bmx[warp] = mx;
    }
    __syncthreads();
    if (warp == 0) {
        sd = lane < nw ? bs[lane] : 0.0;
        mn = lane < nw ? bmn[lane] : 3.0e38f;
        mx = lane < nw ? bmx[lane] : -3.0e38f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sd += __shfl_xor_sync(0xffffffffu, sd, o);
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (lane == 0) {
            grid_dependency_wait();  // the initial values
            atomicAdd(&st->sum, sd);
            atomicMin(&st->kmin, f2key(mn));
            atomicMax(&st->kmax, f2key(mx));
            __threadfence();
            // The last block forms the norm, once for the mesh: an FP64 division per
            // element costs the features a third of their time on this GPU.
            if (atomicAdd(&st->done, 1u) == gridDim.x - 1) {
                __threadfence();
                const volatile EntropyStats *v = st;
                const double mean = v->sum / (double)npoin;
                const double lo = (double)key2f(v->kmin), hi = (double)key2f(v->kmax);
                const float norm = (float)fmax(hi - mean, mean - lo);
                st->norm = norm > 0.0f ? norm : 1.0f;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Plain estimator: one group of NE elements per block, one thread per line
// (msod_group.cuh).
//
//   * each thread gathers its zeta line, forms eta and |u| + c once per point and
//     stores the records (u, eta); each of the three passes loads a line's
//     records, forms eta u and applies the derivative matrix to (u, eta, eta u);
//   * the xi and eta passes add their shares in shared memory; maxima per element
//     by integer atomics on the floats' bits, the volume as a sum of line sums in
//     a fixed order;
//   * He and gpvol come by bulk copy.  In list mode (the per-element fallback)
//     the group's elements are scattered, and both are read in place.
// Bound by the gathers' latency and the L1 / shared-memory pipe.  Estimator with
// its statistics, before / now: porder 4 64^3 0.923 / 0.548 ms, 5 51^3 0.901 /
// 0.532, 7 32^3 0.772 / 0.374, 2 100^3 0.707 / 0.341, 1 128^3 0.533 / 0.203.
// The line arithmetic is operation for operation the one that the shipped
// networks were trained against: on smooth shock fields R is near its rounding
// floor, and the product-rule defect formed from differences of nodal values
// (as the convection forms its terms, no faster here) moves the fallback's
// viscosity by 3e-4.
// ---------------------------------------------------------------------------
// Elements per block (ms, estimator with the statistics, with that other line
// arithmetic, which takes as long): porder 4 (64^3) 8 0.597,
// 4 0.640, 5 0.647, 10 0.756; 5 (51^3) 4 0.605, 7 0.629, 8 0.672, 3 0.696; 6 (40^3) 3
// 0.549, 4 0.553, 2 0.616; 7 (32^3) 3 0.438, 2 0.476, 4 0.561; 3 (80^3) 8 0.491, 4
// 0.609; 2 (100^3) 16 0.356, 14 0.373; 1 (128^3) 32 0.251, 16 0.264.  Without He in
// shared memory the list's blocks are held by their registers, and few groups
// share the SMs: porder 4, learned viscosity on 48^3 hexes (8 % of the elements in
// the list) 218.9 us with 8 elements, 214.4 with 5, 212.2 with 5 in six blocks per
// SM; their He spans prefetched into L2 216.2.  A bound on the registers gains
// nothing without a list.
template <int P, bool LIST>
struct ViscGroup {
    static constexpr int ne[8] = {0, 32, 16, 8, 8, 4, 3, 3}, nl[8] = {0, 32, 16, 8, 5, 4, 3, 3};
    // R in the spent zeta columns of He (each read in the zeta pass only, by the thread
    // that owns the point's zeta line) and gpvol read in place.
    static constexpr bool SLIM = !LIST && P == 5;
    using G = GroupGeom<float, P, LIST ? nl[P] : ne[P], 1, (P <= 2), !SLIM>;
    // Blocks per SM that the registers are held to (0: the compiler's choice).
    static constexpr int MINB = LIST && P == 4 ? 6 : 0;
    // Shared memory that an SM should keep for the blocks (percent, -1: as many blocks
    // as fit).  Beyond 196 KB 28 KB of L1 are left, too few for the cache lines of the
    // gathers in flight: one block less takes, ms, porder 1 0.148 instead of 0.146 on a
    // mesh numbered along x and 0.22 instead of 0.34 with nodes in random order, 3 0.185 /
    // 0.172 and 0.48 / 0.89 (12 M element points).  At porder 5 SLIM makes the four
    // blocks fit: 0.230 against 0.245 and 0.70 against 1.20 (a block less: 0.248, 0.59).
    static constexpr int CARVEOUT = LIST ? -1 : (P == 1 || P == 3 ? 80 : -1);
};

template <class G, bool LIST>
struct ViscShared {
    static constexpr size_t kHe = LIST ? 0 : G::HEB + G::GPB + 16;
    static constexpr size_t kR = kHe + G::NREC * sizeof(Four<float>);
    static constexpr bool kSlots = !LIST && !G::GPSTAGED;
    static constexpr size_t kV = kR + (kSlots ? 0 : G::NSC * sizeof(float));
    static constexpr size_t kEl = kV + (size_t)G::NE * G::L * sizeof(float);  // per element: max speed, max |R|, nu
    static constexpr size_t kTab = (kEl + 3 * (size_t)G::NE * sizeof(float) + 15) / 16 * 16;
    static constexpr size_t kBytes = kTab + GroupTables<G, false>::kBytes;
    unsigned char *base;
    int el;  // the thread's element
    __device__ __forceinline__ unsigned long long *bar() const
    {
        return reinterpret_cast<unsigned long long *>(base + G::HEB + G::GPB);
    }
    __device__ __forceinline__ Four<float> *W() const { return reinterpret_cast<Four<float> *>(base + kHe); }  // u, eta
    __device__ __forceinline__ float *R() const { return reinterpret_cast<float *>(base + kR) + el * G::SK; }
    __device__ __forceinline__ float *vol() const { return reinterpret_cast<float *>(base + kV); }  // line sums
    __device__ __forceinline__ int *speed() const { return reinterpret_cast<int *>(base + kEl); }
    __device__ __forceinline__ unsigned *res() const { return reinterpret_cast<unsigned *>(speed() + G::NE); }
    __device__ __forceinline__ float *nu() const { return reinterpret_cast<float *>(res() + G::NE); }
    __device__ __forceinline__ GroupTables<G, false> tab() const { return GroupTables<G, false>{base + kTab}; }
};

// Direction DIR's share of R at the line's points.
template <class G, int DIR, class HeAt>
__device__ __forceinline__ void visc_line(const Four<float> (&w)[G::Q], const GroupThread<G> &t,
                                          const GroupRows<G, false> &tab, const HeAt &he,
                                          const int (&pt)[G::Q], float (&R)[G::Q])
{
    constexpr int Q = G::Q;
    float2 e12[Q];  // eta u_1, eta u_2
    float e3[Q];
#pragma unroll
    for (int c = 0; c < Q; ++c) {
        e12[c] = mul2(w[c].a, two(w[c].b.y, w[c].b.y));
        e3[c] = w[c].b.y * w[c].b.x;
    }
#pragma unroll
    for (int r = 0; r < Q; ++r) {
        const float *hp = he(pt[r]) + DIR * 3;
        const float h0 = hp[0], h1 = hp[1], h2 = hp[2];
        float D[Q], de3 = 0.0f;
        float2 du = two(0.0f, 0.0f), dw = du, de = du;  // D.(u_1, u_2), D.(u_3, eta), D.(eta u_1, eta u_2)
        tab.row(D, DIR, r);
#pragma unroll
        for (int c = 0; c < Q; ++c) {
            const float2 DD = two(D[c], D[c]);
            du = fma2(DD, w[c].a, du);
            dw = fma2(DD, w[c].b, dw);
            de = fma2(DD, e12[c], de);
            de3 = fmaf(D[c], e3[c], de3);
        }
        const float div_eu = fmaf(h2, de3, fmaf(h1, de.y, h0 * de.x)), div_u = fmaf(h2, dw.x, fmaf(h1, du.y, h0 * du.x));
        const float U = w[r].a.x * h0 + w[r].a.y * h1 + w[r].b.x * h2;
        R[r] = div_eu - w[r].b.y * div_u - U * dw.y;
    }
}
template <class G, int DIR>
__device__ __forceinline__ void visc_load(Four<float> (&w)[G::Q], const GroupThread<G> &t, const Four<float> *W)
{
    const int base = t.rec0(DIR);
#pragma unroll
    for (int s = 0; s < G::Q; ++s) w[s] = W[base + s * G::template step<DIR>()];
}

template <class G, bool LIST, int MINB>
__global__ void __launch_bounds__(G::NT, MINB)
    entropy_visc_kernel(int nelem, int npoin, const int *__restrict__ connec, const float *__restrict__ He,
                        const float *__restrict__ gpvol, const int *__restrict__ inv,
                        const float *__restrict__ dlxigp_ip, const float *__restrict__ rho,
                        const float *__restrict__ u, const float *__restrict__ p_or_T, float Rgas, float gamma,
                        float ce, float cmax, int normalise, const EntropyStats *st,
                        const int *__restrict__ list, const int *__restrict__ count, float *__restrict__ mu_e,
                        float *__restrict__ nu_out, float *__restrict__ numax_out)
{
    constexpr int Q = G::Q, N = G::N, NE = G::NE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    const GroupThread<G> t(tid);
    const ViscShared<G, LIST> sm{smem_raw, t.el};
    // The block's elements: e0 .. e0+NE-1 (one group per block), or in list mode
    // the entries e0 .. of the compacted list, the blocks striding over the
    // list's groups; -1 beyond the end.
    const int nwork = LIST ? ldg(count) : nelem;
    bool first = true;
    for (int gb = blockIdx.x; gb * NE < nwork; gb += gridDim.x) {
        const int e0 = gb * NE;
        const GroupMetric<G> gm = [&]() {
            if constexpr (LIST)
                return GroupMetric<G>();
            else
                return GroupMetric<G>(smem_raw, smem_raw + G::HEB, sm.bar(), He, gpvol, e0, nelem, tid);
        }();
        auto element = [&](int el) { return e0 + el < nwork ? (LIST ? ldg(list + e0 + el) : e0 + el) : -1; };
        const int e = t.active ? element(t.el) : -1;
        auto he = [&](int a) -> const float * {
            if constexpr (LIST)
                return He + ((size_t)(e < 0 ? 0 : e) * N + a) * 9;
            else
                return gm.he(t.el, a);
        };
        // R of the point with record o and gmsh node a.
        auto Rat = [&](int o, int a) -> float & {
            if constexpr (ViscShared<G, LIST>::kSlots)
                return gm.he(t.el, a)[6];
            else
                return sm.R()[o];
        };
        int pt[Q], id[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) pt[k] = GroupTables<G, false>::node(inv, t.template lat<2>(k));
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const int v = e >= 0 ? ldg_once(connec + (size_t)pt[k] * nelem + e) - 1 : -1;
            id[k] = (unsigned)v < (unsigned)npoin ? v : -1;
        }
        if (first) sm.tab().build(inv, dlxigp_ip, tid);
        if (tid < NE) {
            sm.speed()[tid] = 0;
            sm.res()[tid] = 0u;
        }
        Four<float> w[Q];
        float rh[Q], spd = 0.0f, vol = 0.0f;
        {
            const size_t np = (size_t)npoin;
            float f[Q][5];
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                const bool ok = id[k] >= 0;
                const size_t p = ok ? (size_t)id[k] : 0;
                f[k][0] = ok ? ldg_once(rho + p) : 1.0f;
                f[k][1] = ok ? ldg_once(p_or_T + p) : 1.0f;
#pragma unroll
                for (int c = 0; c < 3; ++c) f[k][2 + c] = ok ? ldg_once(u + c * np + p) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                const float r = f[k][0], p = (Rgas > 0.0f && id[k] >= 0) ? r * Rgas * f[k][1] : f[k][1];
                const float s = sqrtf(f[k][2] * f[k][2] + f[k][3] * f[k][3] + f[k][4] * f[k][4]) + sqrtf(gamma * p / r);
                spd = __uint_as_float(max(__float_as_uint(spd), __float_as_uint(s)));  // as their bits: NaN counts
                rh[k] = r;
                w[k].a = two(f[k][2], f[k][3]);
                w[k].b = two(f[k][4], r / (gamma - 1.0f) * (logf(p) - gamma * logf(r)));
            }
            const int base = t.rec0(2);
            if (t.active)
#pragma unroll
                for (int k = 0; k < Q; ++k) sm.W()[base + k * G::template step<2>()] = w[k];
        }
        __syncthreads();
        first = false;
        const GroupRows<G, false> tab(sm.tab());
        // A bounded wait that ran out leaves the group's viscosity NaN.
        const bool ok = LIST || gm.wait(sm.bar());
        float R[Q];
        int lp[Q];
        if (t.active) {
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if constexpr (LIST || !G::GPSTAGED)
                    vol += e >= 0 ? ldg(gpvol + (size_t)e * N + pt[k]) : 0.0f;
                else
                    vol += *gm.vol(t.el, pt[k]);
            }
            sm.vol()[(t.q1 * Q + t.q0) * NE + t.el] = ok ? vol : __int_as_float(0x7fffffff);
            if (e >= 0) atomicMax(reinterpret_cast<unsigned *>(sm.speed()) + t.el, __float_as_uint(spd));
            visc_line<G, 2>(w, t, tab, he, pt, R);
            const int base = t.rec0(2);
#pragma unroll
            for (int k = 0; k < Q; ++k) Rat(base + k * G::template step<2>(), pt[k]) = R[k];
        }
        __syncthreads();
        if (t.active) {
            visc_load<G, 0>(w, t, sm.W());
#pragma unroll
            for (int k = 0; k < Q; ++k) lp[k] = GroupTables<G, false>::node(inv, t.template lat<0>(k));
            visc_line<G, 0>(w, t, tab, he, lp, R);
            const int base = t.rec0(0);
#pragma unroll
            for (int k = 0; k < Q; ++k) Rat(base + k, lp[k]) += R[k];
        }
        __syncthreads();
        if (t.active) {
            visc_load<G, 1>(w, t, sm.W());
#pragma unroll
            for (int k = 0; k < Q; ++k) lp[k] = GroupTables<G, false>::node(inv, t.template lat<1>(k));
            visc_line<G, 1>(w, t, tab, he, lp, R);
            const int base = t.rec0(1);
            unsigned mx = 0u;
#pragma unroll
            for (int k = 0; k < Q; ++k)
                mx = max(mx, __float_as_uint(fabsf(Rat(base + k * G::template step<1>(), lp[k]) + R[k])));
            if (e >= 0) atomicMax(sm.res() + t.el, mx);
        }
        __syncthreads();
        if (tid < NE) {
            const int ee = element(tid);
            // Waits for the statistics in any case: the kernel never ends ahead of them.
            const float norm = entropy_norm(&st->norm), neta = normalise ? norm : 1.0f;
            float v = 0.0f;
            for (int l = 0; l < G::L; ++l) v += sm.vol()[l * NE + tid];
            const float h = cbrtf(v) / (float)(Q - 1);
            const float numax = cmax * h * __int_as_float(sm.speed()[tid]);
            const float nuE = ce * h * h * __uint_as_float(sm.res()[tid]) / neta;
            const float nu = fminf(numax, nuE);
            sm.nu()[tid] = nu;
            if (ee >= 0) {
                if (nu_out) nu_out[ee] = nu;
                if (numax_out && !LIST) numax_out[ee] = numax;
            }
        }
        __syncthreads();
        if constexpr (LIST) continue;
        if (mu_e && e >= 0) {
            const float nu = sm.nu()[t.el];
#pragma unroll
            for (int k = 0; k < Q; ++k) mu_e[(size_t)pt[k] * nelem + e] = rh[k] * nu;
        }
        break;  // one group per block outside list mode
    }
}

template <int P, bool LIST>
cudaError_t visc_pl(const ViscArgs &a, cudaStream_t st)
{
    using G = typename ViscGroup<P, LIST>::G;
    constexpr size_t smem = ViscShared<G, LIST>::kBytes;
    static_assert(smem <= 227 * 1024, "shared memory budget");
    auto kern = entropy_visc_kernel<G, LIST, ViscGroup<P, LIST>::MINB>;
    static std::atomic<unsigned long long> allowed{0};
    const cudaError_t err = allow_smem(allowed, kern, smem, ViscGroup<P, LIST>::CARVEOUT);
    if (err != cudaSuccess) return err;
    // List mode: resident blocks stride over the list (its length is known on
    // the device only); otherwise one group per block.
    const int ngroups = (a.nelem + G::NE - 1) / G::NE;
    const unsigned grid = (unsigned)(LIST ? persistent_grid(kern, G::NT, smem, ngroups) : ngroups);
    if (grid == 0) return cudaErrorInvalidConfiguration;
    if constexpr (!LIST)
        return launch_after(kern, grid, G::NT, smem, st, a.nelem, a.npoin, a.connec, a.He, a.gpvol, a.invAtoIJK,
                            a.dlxigp_ip, a.rho, a.u, a.p_or_T, a.Rgas, a.gamma, a.ce, a.cmax, a.normalise, a.stats,
                            a.list, a.count, a.mu_e, a.nu, a.numax);
    kern<<<grid, G::NT, smem, st>>>(a.nelem, a.npoin, a.connec, a.He, a.gpvol, a.invAtoIJK, a.dlxigp_ip, a.rho, a.u,
                                    a.p_or_T, a.Rgas, a.gamma, a.ce, a.cmax, a.normalise, a.stats, a.list, a.count,
                                    a.mu_e, a.nu, a.numax);
    return cudaGetLastError();
}
template <int P>
cudaError_t visc_p(const ViscArgs &a, cudaStream_t st)
{
    return a.list ? visc_pl<P, true>(a, st) : visc_pl<P, false>(a, st);
}

}  // namespace

cudaError_t launch_entropy_stats(int npoin, const float *rho, const float *p_or_T, float Rgas, float gamma,
                                 EntropyStats *st, int *count, cudaStream_t s)
{
    entropy_stats_init<<<1, 1, 0, s>>>(st, count);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int blocks = (npoin + 255) / 256;
    if (blocks > 8 * sms) blocks = 8 * sms;
    return launch_after(entropy_stats_kernel, (unsigned)blocks, 256, 0, s, npoin, rho, p_or_T, Rgas, gamma, st);
}

cudaError_t launch_entropy_visc(int porder, const ViscArgs &a, cudaStream_t st)
{
    switch (porder) {
    case 1: return visc_p<1>(a, st);
    case 2: return visc_p<2>(a, st);
    case 3: return visc_p<3>(a, st);
    case 4: return visc_p<4>(a, st);
    case 5: return visc_p<5>(a, st);
    case 6: return visc_p<6>(a, st);
    case 7: return visc_p<7>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace msod
