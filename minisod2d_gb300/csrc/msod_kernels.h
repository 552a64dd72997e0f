// msod_kernels.h -- launcher interfaces between the C-ABI layer and the kernels.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "msod.h"

namespace msod {

// A porder's library-owned device area: the 1-D derivative matrices D[d][r][c] on
// their way to the constant bank (written by table_prep_kernel, msod_tables.cu).
constexpr int kTableDMax = 3 * (MSOD_MAX_PORDER + 1) * (MSOD_MAX_PORDER + 1);
struct TableScratch {
    float Df[kTableDMax];
    // Set (sticky, zero at allocation) by a kernel whose bounded wait for a
    // bulk copy into shared memory ran out; the kernel then skipped its work.
    // Checked mode reads and clears it after each call.
    int wait_fault;
};

// Records a bounded wait that ran out (see TableScratch::wait_fault).
__device__ __forceinline__ void report_wait_fault(const TableScratch *t)
{
    atomicOr(const_cast<int *>(&t->wait_fault), 1);
}
template <typename real>
struct ElementArgs {
    int nelem, npoin;
    const int *connec;
    const real *He, *gpvol, *dlxigp_ip;
    const int *invAtoIJK;
};

template <typename real>
struct ConvecArgs : ElementArgs<real> {
    const real *u, *q, *rho, *pr, *E;
    real *Rmass, *Rmom, *Rener;
};

struct MlpNorm;

template <typename real>
struct DiffuArgs : ElementArgs<real> {
    real Cp, Pr;
    const real *rho, *u, *Tem, *mu_fluid, *mu_e, *mu_sgs;
    const real *nu_elem;  // if set: mu_e(e, a) = rho(a) * nu_elem[e] and mu_e is not read
    real *Rmass, *Rmom, *Rener;
};

// Zeroes up to six residual arrays (one launch).  The kernels below that follow
// it on the stream with launch_after start while it still runs and wait for it
// before their first reduction.
struct ZeroSpans {
    void *p[6];
    size_t bytes[6];
    int n = 0;
    void add(void *ptr, size_t b)
    {
        p[n] = ptr;
        bytes[n++] = b;
    }
};
cudaError_t launch_zero(const ZeroSpans &z, cudaStream_t st);

// Allows kern `smem` bytes of dynamic shared memory on the current device, once
// per device and kernel (done: one bit per device, owned by the kernel's launcher),
// and asks for `carveout` percent of an SM's memory for its blocks (-1: no wish).
template <typename Kernel>
inline cudaError_t allow_smem(std::atomic<unsigned long long> &done, Kernel kern, size_t smem, int carveout = -1)
{
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess && carveout >= 0)
        err = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
    if (err == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return err;
}

// Launches kern so that its blocks may start before the kernel ahead of it on
// the stream has finished (programmatic dependent launch); kern calls
// grid_dependency_wait() before it touches what that kernel writes.  Only right
// behind a kernel: what kern reads earlier has to be complete before that kernel
// starts, which a copy queued in between is not.
template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                                A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// D of one call (one block, stream-ordered before the kernel).
cudaError_t launch_table_prep(int porder, const ElementArgs<float> &a, TableScratch *scratch, cudaStream_t st);

// Plain kernels (outputs zeroed by launch_zero just before, or earlier on the
// stream; tabs: where a bounded wait that ran out is recorded).
template <typename real>
cudaError_t launch_convec_plain(int porder, const ConvecArgs<real> &a, const TableScratch *tabs, cudaStream_t st);
// Diffusion: prepare_diffu_plain first, ahead of the kernel that launch_diffu_plain's
// follows on the stream (the zeroing, or the convection behind it): the matrices of a
// call that reads them from the constant bank are then complete when that kernel starts.
template <typename real>
cudaError_t prepare_diffu_plain(int porder, const DiffuArgs<real> &a, TableScratch *tabs, cudaStream_t st);
template <typename real>
cudaError_t launch_diffu_plain(int porder, const DiffuArgs<real> &a, const TableScratch *tabs, cudaStream_t st);
template <>
cudaError_t prepare_diffu_plain<float>(int porder, const DiffuArgs<float> &a, TableScratch *tabs, cudaStream_t st);
template <>
cudaError_t launch_diffu_plain<float>(int porder, const DiffuArgs<float> &a, const TableScratch *tabs, cudaStream_t st);
template <>  // msod_diffu64.cu
cudaError_t prepare_diffu_plain<double>(int porder, const DiffuArgs<double> &a, TableScratch *tabs, cudaStream_t st);
template <>
cudaError_t launch_diffu_plain<double>(int porder, const DiffuArgs<double> &a, const TableScratch *tabs,
                                       cudaStream_t st);
// Mixed-precision convection: FP32 fields, FP64 residuals (zeroed by
// launch_zero just before).  precision: MSOD_PREC_FP16 or MSOD_PREC_BF16.
struct MixedConvecArgs : ElementArgs<float> {
    const float *u, *q, *rho, *pr, *E;
    double *Rmass, *Rmom, *Rener;
};
cudaError_t launch_convec_mixed(int porder, int precision, const MixedConvecArgs &a, cudaStream_t st);

// Mixed-precision diffusion: FP32 fields, FP64 residuals (zeroed by
// launch_zero just before).  nu_elem set: mu_e(e, a) = rho(a) nu_elem[e] and
// mu_e is not read.
struct MixedDiffuArgs : ElementArgs<float> {
    float Cp, Pr;
    const float *rho, *u, *Tem, *mu_fluid, *mu_e, *mu_sgs, *nu_elem;
    double *Rmass, *Rmom, *Rener;
};
cudaError_t launch_diffu_mixed(int porder, int precision, const MixedDiffuArgs &a, cudaStream_t st);

// ---------------------------------------------------------------------------
// Entropy viscosity and the learned estimator
// ---------------------------------------------------------------------------
struct EntropyStats {
    double sum;  // sum of eta over the nodes
    int kmin;    // order-preserving int keys of min / max eta
    int kmax;
    unsigned done;  // blocks that have added their share
    float norm;     // || eta - mean(eta) ||_inf (1 if it vanishes)
};

constexpr int kMlpIn = 12, kMlpH = 32;
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kMlpH * kMlpIn;
constexpr int kOffW2 = kOffB1 + kMlpH;
constexpr int kOffB2 = kOffW2 + kMlpH * kMlpH;
constexpr int kOffW3 = kOffB2 + kMlpH;
constexpr int kOffB3 = kOffW3 + kMlpH;
constexpr int kMlpParams = kOffB3 + 1;  // 1505
static_assert(kMlpParams == MSOD_MLP_NPARAMS, "parameter count");

struct MlpNorm {
    float mean[kMlpIn], inv_std[kMlpIn], fmin[kMlpIn], fmax[kMlpIn];
};

// Linear tetrahedra (fem_convec, fem_diffu): 4 nodes, 4 Gauss points; tables
// Ngp(4,4), dNgp(3,4,4) are device arrays in the reference's layouts.
template <typename real>
struct TetConvecArgs {
    int nelem, npoin;
    const int *connec;
    const real *Ngp, *dNgp, *He, *gpvol;
    const real *u, *q, *rho, *pr, *E;
    real *Rmass, *Rmom, *Rener;
};
template <typename real>
struct TetDiffuArgs {
    int nelem, npoin;
    const int *connec;
    const real *Ngp, *dNgp, *He, *gpvol;
    real Cp, Pr;
    const real *rho, *u, *Tem, *mu_fluid, *mu_e, *mu_sgs;
    real *Rmass, *Rmom, *Rener;
};
template <typename real>
cudaError_t launch_fem_convec(const TetConvecArgs<real> &a, cudaStream_t st);
template <typename real>
cudaError_t launch_fem_diffu(const TetDiffuArgs<real> &a, cudaStream_t st);
// Range check of count connec entries against 1..npoin (sets bit 8 of flags).
cudaError_t launch_check_connec(long long count, int npoin, const int *connec, int *flags, cudaStream_t st);
// Jacobian of elements with n nodes = n points (elem_jacobian / tet_jacobian).
template <typename real>
cudaError_t launch_jacobian_nodes(int n, int nelem, int npoin, const int *connec, const real *coord,
                                  const real *dNgp, const real *wgp, real *gpvol, real *He, cudaStream_t st);

struct ViscArgs {
    int nelem, npoin;
    const int *connec;
    const float *He, *gpvol, *dlxigp_ip;
    const int *invAtoIJK;
    const float *rho, *u, *p_or_T;
    float Rgas, gamma, ce, cmax;
    int normalise;
    const EntropyStats *stats;
    // If set: process only the elements list[0 .. *count) (the compacted list
    // of flagged elements written by launch_mlp_predict), write nu only.
    const int *list, *count;
    float *mu_e, *nu, *numax;
};

struct FeatureArgs {
    int nelem, npoin;
    const int *connec;
    const float *He, *gpvol;
    const float *dlxigp_ip;
    const int *invAtoIJK;
    const float *rho, *u, *p_or_T;
    float Rgas, gamma, cmax;
    const EntropyStats *stats;
    float *feat, *numax;
};

// count, if given, is set to zero ahead of the kernels that follow.  launch_features
// and launch_entropy_visc without a list come right behind it on the stream.
cudaError_t launch_entropy_stats(int npoin, const float *rho, const float *p_or_T, float Rgas, float gamma,
                                 EntropyStats *st, int *count, cudaStream_t s);
cudaError_t launch_entropy_visc(int porder, const ViscArgs &a, cudaStream_t st);
cudaError_t launch_features(int porder, const FeatureArgs &a, cudaStream_t st);
// y = 10^-s, nu = y numax (if nu), flag = 1 outside the training range (if
// flag); with list: list[0 .. *count) = the flagged elements (any order).
cudaError_t launch_mlp_predict(int nelem, const float *feat, const __half *wh, const MlpNorm *nm, const float *numax,
                               float *y, float *nu, int *flag, int *list, int *count, cudaStream_t st);
cudaError_t launch_mlp_norm(int n, const float *feat, MlpNorm *nm, cudaStream_t st);
cudaError_t launch_mlp_grad(int n, const float *feat, const float *target, const float *weight, const int *idx,
                            int batch, uint32_t seed,
                            int step, const float *master, const MlpNorm *nm, float *grad, float *loss, cudaStream_t st);
cudaError_t launch_mlp_adam(float *master, float *m, float *v, float *grad, __half *wh, float lr, int t,
                            cudaStream_t st);
cudaError_t launch_mlp_to_half(const float *master, __half *wh, cudaStream_t st);

// Setup kernels.
template <typename real>
cudaError_t launch_elem_jacobian(int porder, int nelem, int npoin, const int *connec, const real *coord,
                                 const real *dNgp, const real *wgp, real *gpvol, real *He, cudaStream_t st);

// Validation: accumulates failure bits into *flags (device int).
cudaError_t launch_check_tables(int porder, int nelem, int npoin, const int *connec, const float *dlxigp_ip,
                                const int *invAtoIJK, const int *AtoI, const int *AtoJ, const int *AtoK,
                                int *flags, cudaStream_t st);

}  // namespace msod
