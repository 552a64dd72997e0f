// msod_diffu64.cu -- FP64 hex GLL diffusion residual (formulas in msod_diffu.cu).
//
// Bound by FP64 issue: two multiply-adds a clock and SM, 64 cycles for a warp's
// instruction on a scheduler, so shared-memory traffic and residency hardly count, and
// what counts is that no lane idles and nothing spills.  A thread therefore takes whole
// points instead of lines (the line form of msod_diffu.cu carries 16 numbers per point
// of its line, 256 registers of doubles at porder 7: 5 KB of spills a thread; and at
// porder 8 81 of its 96 threads work): it sums the three directions' derivatives of its
// points from shared memory, forms the fluxes there, and after one barrier sums their
// divergences.  us per call, line form / points: 10^6 element points, porder 4 616 / 596,
// 5 810 / 704, 6 930 / 732, 7 772 / 675, 8 1019 / 812; 10^5 points, 4 87 / 73, 5 155 /
// 91, 6 196 / 117, 7 176 / 119, 8 193 / 95.
#include <cuda_runtime.h>

#include "msod_device.cuh"
#include "msod_kernels.h"

namespace msod {
namespace {

// NE elements a block, PP points a thread: blocks of 6 to 12 warps that leave few
// lanes idle (porder 1 to 8: 256, 189, 256, 250, 216, 343, 512, 729 points).
template <int P>
struct Diffu64Geom {
    static constexpr int Q = P + 1, L = Q * Q, N = Q * Q * Q;
    static constexpr int NE = P >= 5 ? 1 : (P == 4 ? 2 : (P == 3 ? 4 : (P == 2 ? 7 : 32)));
    static constexpr int NPT = NE * N, PP = P >= 7 ? 2 : 1;
    static constexpr int NT = ((NPT + PP - 1) / PP + 31) / 32 * 32;
    static constexpr int MINB = P == 7 ? 2 : 1;  // blocks per SM that the registers are held to
    // Node fields, fluxes (direction d, vector x at 6 d + x) and derivative matrices.
    static constexpr size_t smem = ((size_t)(5 + 18) * NPT + 3 * L) * sizeof(double);
};

enum { D_RHO = 0, D_T, D_U, D_FIELDS = 5 };                                   // node fields
enum { X_GRHO = 0, X_TAUU, X_GT, X_TAU, X_VECTORS = 6 };                      // vectors of the weak divergence

template <int P>
__global__ void __launch_bounds__(Diffu64Geom<P>::NT, Diffu64Geom<P>::MINB)
    diffu64_kernel(int nelem, int npoin, const int *__restrict__ connec, const double *__restrict__ He,
                   const double *__restrict__ gpvol, const int *__restrict__ inv,
                   const double *__restrict__ dlxigp_ip, double Cp, double Pr, const double *__restrict__ rho,
                   const double *__restrict__ u, const double *__restrict__ Tem,
                   const double *__restrict__ mu_fluid, const double *__restrict__ mu_e,
                   const double *__restrict__ mu_sgs, double *__restrict__ Rmass, double *__restrict__ Rmom,
                   double *__restrict__ Rener)
{
    using G = Diffu64Geom<P>;
    constexpr int Q = G::Q, L = G::L, N = G::N, NPT = G::NPT, PP = G::PP, NT = G::NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sF = reinterpret_cast<double *>(smem_raw);  // [D_FIELDS][NPT]
    double *sX = sF + D_FIELDS * NPT;                    // [3][X_VECTORS][NPT]
    double *sD = sX + 3 * X_VECTORS * NPT;               // [3][Q][Q]
    const int tid = threadIdx.x, e0 = blockIdx.x * G::NE;
    const size_t np = (size_t)npoin;
    // Indices are clamped: malformed tables give wrong numbers, never an access out of bounds.
    auto gmsh = [&](int l) { return min(max(ldg(inv + l) - 1, 0), N - 1); };
    for (int i = tid; i < 3 * L; i += NT) {
        const int d = i / L, r = (i / Q) % Q, c = i % Q;
        sD[i] = ldg(dlxigp_ip + (size_t)(c * 3 + d) * N + gmsh(d == 0 ? r : (d == 1 ? r * Q : r * L)));
    }
    // The thread's points (a missing node reads as zeros).
    int id[PP];
    bool in[PP];
    double r[PP], v[PP][3], muf[PP], ms[PP], me[PP], H[PP][9], gv[PP];
#pragma unroll
    for (int k = 0; k < PP; ++k) {
        const int i = tid + k * NT, el = i / N, e = e0 + el;
        in[k] = i < NPT && e < nelem;
        const int a = in[k] ? gmsh(i - el * N) : 0;
        const size_t row = (size_t)a * nelem + (in[k] ? e : 0), pt = (size_t)(in[k] ? e : 0) * N + a;
        const int n = in[k] ? ldg(connec + row) - 1 : -1;
        id[k] = (unsigned)n < (unsigned)npoin ? n : -1;
        const bool ok = id[k] >= 0;
        const size_t p = ok ? (size_t)id[k] : 0;
        r[k] = ok ? ldg(rho + p) : 0.0;
        const double T = ok ? ldg(Tem + p) : 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[k][c] = ok ? ldg(u + c * np + p) : 0.0;
        muf[k] = ok ? ldg(mu_fluid + p) : 0.0;
        ms[k] = ldg(mu_sgs + row);
        me[k] = ldg(mu_e + row);
#pragma unroll
        for (int j = 0; j < 9; ++j) H[k][j] = ldg(He + pt * 9 + j);
        gv[k] = ldg(gpvol + pt);
        if (i < NPT) {
            sF[D_RHO * NPT + i] = r[k];
            sF[D_T * NPT + i] = T;
#pragma unroll
            for (int c = 0; c < 3; ++c) sF[(D_U + c) * NPT + i] = v[k][c];
        }
    }
    __syncthreads();
    // Gradients, stress and fluxes gpvol He(:, d)^T X at the thread's points.
#pragma unroll
    for (int k = 0; k < PP; ++k) {
        if (!in[k]) continue;
        const int i = tid + k * NT, l = i % N;
        const int at[3] = {l % Q, l / Q % Q, l / L}, step[3] = {1, Q, L};
        double g[D_FIELDS][3];  // physical gradients
#pragma unroll
        for (int f = 0; f < D_FIELDS; ++f) g[f][0] = g[f][1] = g[f][2] = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double *row = sD + d * L + at[d] * Q, *line = sF + i - at[d] * step[d];
            double s[D_FIELDS] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int c = 0; c < Q; ++c)
#pragma unroll
                for (int f = 0; f < D_FIELDS; ++f) s[f] = fma(row[c], line[f * NPT + c * step[d]], s[f]);
#pragma unroll
            for (int f = 0; f < D_FIELDS; ++f)
#pragma unroll
                for (int j = 0; j < 3; ++j) g[f][j] = fma(H[k][3 * d + j], s[f], g[f][j]);
        }
        const double mf = muf[k] + r[k] * ms[k], mt = mf + me[k];
        const double cut = mf * (2.0 / 3.0) * (g[D_U][0] + g[D_U + 1][1] + g[D_U + 2][2]);
        double X[X_VECTORS][3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            X[X_GRHO][m] = g[D_RHO][m];
            X[X_GT][m] = g[D_T][m];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                X[X_TAU + m][j] = m > j ? X[X_TAU + j][m] : mt * (g[D_U + m][j] + g[D_U + j][m]) - (m == j ? cut : 0.0);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m)
            X[X_TAUU][m] = fma(X[X_TAU + m][2], v[k][2], fma(X[X_TAU + m][1], v[k][1], X[X_TAU + m][0] * v[k][0]));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double w0 = gv[k] * H[k][3 * d], w1 = gv[k] * H[k][3 * d + 1], w2 = gv[k] * H[k][3 * d + 2];
#pragma unroll
            for (int x = 0; x < X_VECTORS; ++x)
                sX[(d * X_VECTORS + x) * NPT + i] = fma(w2, X[x][2], fma(w1, X[x][1], w0 * X[x][0]));
        }
    }
    __syncthreads();
    // Weak divergences: the transposed matrices.
    double s[PP][X_VECTORS];
#pragma unroll
    for (int k = 0; k < PP; ++k) {
        if (!in[k]) continue;
        const int i = tid + k * NT, l = i % N;
        const int at[3] = {l % Q, l / Q % Q, l / L}, step[3] = {1, Q, L};
#pragma unroll
        for (int x = 0; x < X_VECTORS; ++x) s[k][x] = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double *col = sD + d * L + at[d], *line = sX + d * X_VECTORS * NPT + i - at[d] * step[d];
#pragma unroll
            for (int c = 0; c < Q; ++c)
#pragma unroll
                for (int x = 0; x < X_VECTORS; ++x) s[k][x] = fma(col[c * Q], line[x * NPT + c * step[d]], s[k][x]);
        }
    }
    grid_dependency_wait();  // the residuals are zeroed
#pragma unroll
    for (int k = 0; k < PP; ++k) {
        if (id[k] < 0) continue;
        const double kappa = fma(muf[k] + me[k], Cp / Pr, Cp / 0.9 * (r[k] * ms[k]));
        red_add(Rmass + id[k], me[k] / r[k] * s[k][X_GRHO]);
        red_add(Rener + id[k], fma(kappa, s[k][X_GT], s[k][X_TAUU]));
#pragma unroll
        for (int m = 0; m < 3; ++m) red_add(Rmom + m * np + id[k], s[k][X_TAU + m]);
    }
}

template <int P>
cudaError_t launch_diffu64(const DiffuArgs<double> &a, cudaStream_t st)
{
    using G = Diffu64Geom<P>;
    static_assert(G::smem <= 227 * 1024, "shared memory budget");
    if (a.nu_elem) return cudaErrorInvalidValue;  // FP32 only
    auto kern = diffu64_kernel<P>;
    static std::atomic<unsigned long long> allowed{0};
    const cudaError_t err = allow_smem(allowed, kern, G::smem);
    if (err != cudaSuccess) return err;
    const unsigned grid = (unsigned)((a.nelem + G::NE - 1) / G::NE);
    return launch_after(kern, grid, G::NT, G::smem, st, a.nelem, a.npoin, a.connec, a.He, a.gpvol, a.invAtoIJK,
                        a.dlxigp_ip, a.Cp, a.Pr, a.rho, a.u, a.Tem, a.mu_fluid, a.mu_e, a.mu_sgs, a.Rmass, a.Rmom,
                        a.Rener);
}

}  // namespace

template <>
cudaError_t prepare_diffu_plain<double>(int, const DiffuArgs<double> &, TableScratch *, cudaStream_t)
{
    return cudaSuccess;
}

template <>
cudaError_t launch_diffu_plain<double>(int porder, const DiffuArgs<double> &a, const TableScratch *, cudaStream_t st)
{
    switch (porder) {
    case 1: return launch_diffu64<1>(a, st);
    case 2: return launch_diffu64<2>(a, st);
    case 3: return launch_diffu64<3>(a, st);
    case 4: return launch_diffu64<4>(a, st);
    case 5: return launch_diffu64<5>(a, st);
    case 6: return launch_diffu64<6>(a, st);
    case 7: return launch_diffu64<7>(a, st);
    case 8: return launch_diffu64<8>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace msod
