// msod_tables.cu -- the derivative matrices of the constant-bank diffusion, and the
// zeroing of the residuals.
//
// table_prep_kernel, one block, reads the caller's dlxigp_ip / invAtoIJK (device
// arrays in the reference's layouts) and writes, into a small library-owned
// device area that is then copied to the constant bank,
//   D[d][r][c] = dlxigp_ip(g, d, c) for a point g whose 1-D index in
//            direction d is r: the 1-D derivative matrix the reference
//            replicates per point (elem_hex.f90:43-44, mod_maths.f90:274-281).
// Every other kernel reads its tables from the caller's arrays itself.
// Indices are clamped, so malformed tables give wrong numbers (reported by
// msod_check_element_tables), never out-of-bounds accesses.
#include <cuda_runtime.h>

#include "msod_device.cuh"
#include "msod_kernels.h"

namespace msod {
namespace {

__global__ void table_prep_kernel(int Q, const int *__restrict__ invAtoIJK, const float *__restrict__ dlxigp_ip,
                                  float *__restrict__ D)
{
    const int N = Q * Q * Q;
    for (int i = threadIdx.x; i < 3 * Q * Q; i += blockDim.x) {
        const int d = i / (Q * Q), r = (i / Q) % Q, c = i % Q;
        const int l = d == 0 ? r : (d == 1 ? r * Q : r * Q * Q);
        const int a = min(max(invAtoIJK[l] - 1, 0), N - 1);
        D[i] = dlxigp_ip[(size_t)(c * 3 + d) * N + a];
    }
}

// Each block zeroes one 16 KB piece of one array (four 16-byte stores a
// thread); the ends of an array that are not 16-byte aligned go to its first
// block.
constexpr size_t kZeroPiece = 16384;
struct ZeroPlan {
    ZeroSpans z;
    unsigned first[7];  // first block of each array
};
__global__ void __launch_bounds__(256) zero_kernel(ZeroPlan pl)
{
    grid_dependents_launch();  // the residual kernel may start (it waits before its first reduction)
    int k = 0;
    while (k + 1 < pl.z.n && blockIdx.x >= pl.first[k + 1]) ++k;
    const unsigned piece = blockIdx.x - pl.first[k];
    const size_t a = reinterpret_cast<size_t>(pl.z.p[k]), e = a + pl.z.bytes[k];
    size_t a16 = (a + 15) & ~(size_t)15, e16 = e & ~(size_t)15;
    if (a16 > e16) a16 = e16 = e;  // no aligned 16 bytes: words only
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const size_t i0 = a16 + piece * kZeroPiece + 16 * threadIdx.x;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (i0 + 4096 * j < e16) *reinterpret_cast<float4 *>(i0 + 4096 * j) = zero;
    if (piece == 0 && threadIdx.x < 8) {
        const size_t h = a + 4 * threadIdx.x, t = e16 + 4 * threadIdx.x;
        if (h < a16) *reinterpret_cast<float *>(h) = 0.0f;
        if (t < e) *reinterpret_cast<float *>(t) = 0.0f;
    }
}

}  // namespace

cudaError_t launch_zero(const ZeroSpans &z, cudaStream_t st)
{
    ZeroPlan pl;
    pl.z = z;
    unsigned n = 0;
    for (int k = 0; k < z.n; ++k) {
        pl.first[k] = n;
        n += (unsigned)((z.bytes[k] + kZeroPiece) / kZeroPiece);
    }
    zero_kernel<<<n, 256, 0, st>>>(pl);
    return cudaGetLastError();
}

cudaError_t launch_table_prep(int porder, const ElementArgs<float> &a, TableScratch *scratch, cudaStream_t st)
{
    table_prep_kernel<<<1, 256, 0, st>>>(porder + 1, a.invAtoIJK, a.dlxigp_ip, scratch->Df);
    return cudaGetLastError();
}

}  // namespace msod
