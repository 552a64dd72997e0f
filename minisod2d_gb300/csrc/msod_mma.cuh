// msod_mma.cuh -- helpers of the mixed-precision (tensor-core) kernels:
// hi + lo half splits, ldmatrix / mma.sync wrappers, the swizzled layout of
// one field's half plane, float -> double on the integer pipe.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace msod {

// Registers a thread keeps at least when blocks are added to an SM.  Measured
// (ms, convection / diffusion FP16, porder 4 48^3): 112 2.830 / 2.483, 96 2.692 /
// 2.114, 80 2.687 / 2.121; porder 5 40^3 diffusion 1.775, 1.776, 1.926; porder 2
// 64^3 3.417 / 2.788, 3.180 / 2.434, 3.122 / 2.490; porders 6 and 7 are alike (two
// blocks by shared memory).
constexpr int kMixedRegs = 96;
// Blocks of `threads` threads and `smem` bytes that an SM holds when every
// thread has `regs` registers at least (each of the four schedulers has 512 for
// each lane of its warps).
constexpr int mixed_blocks(size_t smem, int threads, int regs)
{
    int b = (int)((size_t)228 * 1024 / (smem + 1024));
    while (b > 1 && 512 / ((b * threads / 32 + 3) / 4) < regs) --b;
    return b < 1 ? 1 : b;
}

constexpr int kRowB = 16;  // bytes per half-plane row: 8 halves along i

// One field half of an element: 8 rows per k-plane of the element, 8 Q rows.
// Measured against 8 x 8-row planes for every order (48^3 hexes): porder-5
// convection 5.24 -> 4.04 ms and porder-4 diffusion 2.78 -> 2.27 ms (more
// blocks per SM), the other kernels unchanged (0 selects the full planes).
#ifndef MIXED_TRIM_PLANES
#define MIXED_TRIM_PLANES 1
#endif
template <int Q>
constexpr int plane_bytes()
{
    return (MIXED_TRIM_PLANES ? 8 * Q : 64) * kRowB;
}

// gmsh node of lattice point l = (K Q + J) Q + I, and the 1-D derivative matrices
// D(d, r, c) = dlxigp_ip(g, d, c) at a point g whose 1-D index in direction d is r,
// read once per block (clamped: malformed tables give wrong numbers, never an
// access out of bounds).
template <int Q>
__device__ __forceinline__ int table_node(const int *__restrict__ inv, int l)
{
    return min(max(__ldg(inv + l) - 1, 0), Q * Q * Q - 1);
}
template <int Q>
__device__ __forceinline__ float table_D(const int *__restrict__ inv, const float *__restrict__ dlx, int d, int r, int c)
{
    return __ldg(dlx + (size_t)(c * 3 + d) * Q * Q * Q + table_node<Q>(inv, d == 0 ? r : (d == 1 ? r * Q : r * Q * Q)));
}

// Shared-memory position of lattice point (K, J, I) in a plane of node_plane<Q>()
// words, I contiguous.  The passes read two points of each of up to eight lines
// per thread quad (lines along I for xi, else along J or K): k-planes a few words
// further apart, and for Q = 8 an exclusive-or of the rows, keep those reads on
// distinct banks.
template <int Q>
constexpr int node_pitch()
{
    return Q == 4 ? 20 : (Q == 5 ? 28 : (Q == 7 ? 52 : Q * Q));
}
template <int Q>
constexpr int node_plane()
{
    return (Q * node_pitch<Q>() + 3) / 4 * 4;
}
template <int Q>
__device__ __forceinline__ int node_at(int K, int J, int I)
{
    if (Q == 8) return K * 64 + (((J >> 1 | (J & 1) << 2) ^ (K >> 1)) << 3) + I;
    return K * node_pitch<Q>() + J * Q + I;
}

// Position of slot s of a pass (output point 2t + s along direction d of line g
// of tile o); -1 when padded.
template <int Q>
__device__ __forceinline__ int pass_point(int d, int s, int g, int tq, int o)
{
    const int pt = 2 * tq + s;
    const int I = d == 0 ? pt : g;
    const int J = d == 0 ? g : (d == 1 ? pt : o);
    const int K = d == 2 ? pt : o;
    return g < Q && pt < Q ? node_at<Q>(K, J, I) : -1;
}

// Row (k, j) of a half plane sits at position 8k + (j xor k): the eight rows
// of every ldmatrix phase fall on distinct banks for xi, eta and zeta lines.
__device__ __forceinline__ int row_pos(int k, int j) { return 8 * k + (j ^ k); }

// Byte offset in a half plane of row r8 of the A operand of direction d, tile w:
// for xi and eta lines row j = r8 of k-plane w, for zeta lines row j = w of k-plane
// r8.  There is no k-plane beyond Q: those zeta rows, which meet zero coefficients,
// are the rows beyond Q of k-plane w, which nothing writes after they are zeroed.
// They must be zero, not only finite elsewhere: a row of another field, or one that
// an earlier element left behind, can hold an infinity or a NaN, and zero times that
// is a NaN.  Same banks as row_pos(r8, w): the eight rows of a phase stay distinct.
template <int Q>
__device__ __forceinline__ int operand_row(int d, int w, int r8)
{
    return (d == 2 && r8 < Q ? row_pos(r8, w) : row_pos(w, r8)) * kRowB;
}

template <bool BF16>
__device__ __forceinline__ unsigned pack2(float a, float b)
{
    if (BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const unsigned *>(&h);
    }
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const unsigned *>(&h);
}

// Split of a pair of derivative-matrix entries into hi and lo halves.
template <bool BF16>
__device__ __forceinline__ void split_pair(float a, float b, unsigned &hi, unsigned &lo)
{
    hi = pack2<BF16>(a, b);
    float2 f;
    if (BF16)
        f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&hi));
    else
        f = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    lo = pack2<BF16>(a - f.x, b - f.y);
}

__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], const void *row)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], const void *row)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// d = A B + d (m16n8k16, FP32 accumulate).
template <bool BF16>
__device__ __forceinline__ void mma_acc(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    if (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
                     "{%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
                     "{%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// float -> double by re-biasing the IEEE exponent on the integer pipe (FP64
// arithmetic is scarce on this GPU); zeros, subnormals, infinities and NaNs
// take the FP64 conversion.
__device__ __forceinline__ double f2d(float x)
{
    const unsigned b = __float_as_uint(x);
    const unsigned ex = (b >> 23) & 0xFFu;
    if (ex == 0u || ex == 0xFFu) return (double)x;
    const unsigned long long bits = ((unsigned long long)(b >> 31) << 63) |
                                    ((unsigned long long)(ex + (1023u - 127u)) << 52) |
                                    ((unsigned long long)(b & 0x7FFFFFu) << 29);
    return __longlong_as_double((long long)bits);
}

// A scaled pair -> packed hi halves (rint: exact small integers) and lo halves
// (the remainders, |lo| <= 1/2).
template <bool BF16>
__device__ __forceinline__ void split_scaled(float a, float b, unsigned &hi, unsigned &lo)
{
    const float M = 12582912.0f;  // 1.5 * 2^23: adding and subtracting it rounds to an integer
    const float ha = __fsub_rn(__fadd_rn(a, M), M), hb = __fsub_rn(__fadd_rn(b, M), M);
    hi = pack2<BF16>(ha, hb);
    lo = pack2<BF16>(__fsub_rn(a, ha), __fsub_rn(b, hb));
}

// Power-of-two scale s = 2^(bits-1-ex) of a field whose maximum magnitude
// (bit pattern of a non-negative float) lies in [2^ex, 2^(ex+1)), and 1/s;
// ex is clamped so both stay normal.
__device__ __forceinline__ void scale_from_max(unsigned maxbits, int bits, float &s, float &inv)
{
    int ex = (int)((maxbits >> 23) & 0xFFu) - 127;
    ex = min(max(ex, -100), 127);
    s = __int_as_float((127 + bits - 1 - ex) << 23);
    inv = __int_as_float((127 + ex - (bits - 1)) << 23);
}

}  // namespace msod
