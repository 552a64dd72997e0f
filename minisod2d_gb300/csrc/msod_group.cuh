// msod_group.cuh -- element groups for the line-parallel hex kernels: the
// thread-to-line map, the shared-memory lattice of vector records, the bulk
// staging of He and gpvol, and pairwise (f32x2) arithmetic.
//
// What bounds these kernels is the L1 / shared-memory pipe (the wavefronts of
// every load, store and reduction of an SM) beside FP32 issue, so the layout
// is chosen by wavefronts per element point:
//   * a block takes NE consecutive elements, and the lanes of a warp run along
//     the elements first.  connec, mu_e and mu_sgs are element-fastest, and on
//     meshes numbered along x the same local node of consecutive elements, for
//     neighbouring local nodes, fills whole sectors: a gather or reduction of
//     a node field touches 1-3 cache lines per warp, where lanes that run over
//     one element's lattice touch seven or eight.  At porders 1 and 2, whose
//     warps hold only a line or two of each element, they run along xi ahead of
//     the elements, so that the nodes of an xi line, neighbours in most
//     numberings, share sectors whatever the order of the elements (12 M element
//     points, porder 1, elements first / xi first: convection 0.221 / 0.187 ms,
//     elements in random order 1.57 / 1.03);
//   * on other numberings the gathers touch more lines (elements with nodes of their own,
//     porder 4: twelve), and what counts is that the lines in flight fit in the
//     L1 beside the blocks' shared memory (group_close, and the choices by the L1's size in
//     the kernels);
//   * He and gpvol of a group are contiguous (He(3,3,ngaus,nelem)): one bulk
//     copy each brings them to shared memory.  Read by the line threads from
//     global memory, a point's three He values cost one L1 tag lookup per lane
//     and value (9 x ~28 cycles per warp and point), from shared memory ~2
//     wavefronts each;
//   * node fields are stored as 16-byte records, so a point takes three loads.
//     With lanes along elements the records of an 8-lane phase differ by
//     multiples of the element stride ES: ES is padded so that they, and the
//     lines beside them, fall on distinct banks.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "msod_device.cuh"
#include "msod_kernels.h"

namespace msod {
namespace {

// ---- pairs ---------------------------------------------------------------
template <typename real>
struct Pair;
template <>
struct Pair<float> {
    using T = float2;
};
template <>
struct Pair<double> {
    using T = double2;
};
template <typename real>
using Two = typename Pair<real>::T;

__device__ __forceinline__ float2 two(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 two(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c)
{
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    return __fadd2_rn(a, make_float2(-b.x, -b.y));
}
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// Four reals of one shared-memory record.
template <typename real>
struct alignas(16) Four {
    Two<real> a, b;
};

// ---- geometry ------------------------------------------------------------
// Pitches of the record lattice, by porder and elements per block, searched for
// the fewest wavefronts of the 16- and 4-byte accesses of the three directions'
// line passes (lanes along elements, then lines) at little padding.  An access
// of 16 bytes per lane takes four wavefronts per warp without conflicts; with
// rows and planes packed (5, 25, 125) the xi lines of porder 4 take 7.75, with
// the xi lines run through along K first 4.0.
struct GroupPitch {
    int row, plane, elem;
    bool swap;
};
constexpr GroupPitch group_pitch(int P, int NE, bool ifirst)
{
    if (ifirst && P == 2) return {3, 9, 27, true};
    switch (P * 100 + NE) {
    case 132: return {2, 5, 10, true};
    case 308: return {4, 16, 67, false};
    case 405: return {5, 25, 125, true};
    case 409: return {5, 25, 129, true};
    case 503: return {6, 36, 219, false};
    case 504: return {6, 37, 222, true};
    case 507: return {6, 38, 231, false};
    case 602: return {7, 49, 348, false};
    case 603: return {7, 49, 347, true};
    case 604: return {7, 49, 346, false};
    case 701: return {8, 67, 533, true};
    case 702: return {8, 65, 524, true};
    case 703: return {8, 65, 523, true};
    case 802: return {9, 81, 732, false};
    case 803: return {9, 81, 731, true};
    default: break;
    }
    const int Q = P + 1, RP = Q % 2 ? Q : Q + 1;
    return {RP, Q * RP, Q * Q * RP, false};
}

// Arrays of 4-byte (8-byte) numbers per record are kept at a pitch per element of
// that many numbers more than the records', which are placed for 16-byte
// accesses: fewest conflicts over the three directions (wavefronts per warp and
// direction without / with: 4-byte porder 5, 4 elements 3.0 / 1.3, 6, 2 elements 2.0
// / 1.5, 7 2.0 / 1.3, 8 1.8 / 1.3, 2, 16 elements (elements
// first) 1.8 / 1.0; 8-byte 5 3.6 / 2.0, 7 4.0 / 2.0).  Without / with, ms: convection porder 7 32^3 0.781 / 0.767, 6 40^3 1.060 /
// 1.053, 5 51^3 1.130 / 1.128; diffusion 7 0.770 / 0.763, 2 100^3 0.564 / 0.558;
// estimator 2 0.375 / 0.349.  Groups that are not listed gain nothing (porder 4, 5
// elements: 2.3 / 2.0) or lose (the estimator at porder 6, 3 elements, 0.484 / 0.491).
constexpr int group_pad4(int P, int NE, bool ifirst)
{
    switch (P * 100 + NE) {
    case 216: return ifirst ? 0 : 3;
    case 504: return 10;
    case 602: return 20;
    case 702: return 4;
    case 802: return 20;
    default: return 0;
    }
}
constexpr int group_pad8(int P, int NE)
{
    switch (P * 100 + NE) {
    case 504: return 6;
    case 702: return 12;
    default: return 0;
    }
}

// Q points per line, L lines per direction, N points per element, NE elements
// per block, S threads per line (each owns R consecutive points; the split is
// by warp, so that a warp's code and coefficients are uniform).  IFIRST: lanes
// along xi ahead of the elements.  GPSTAGED: gpvol in shared memory too.
template <typename real_t, int P_, int NE_, int S_ = 1, bool IF_ = (P_ <= 2), bool GP_ = true>
struct GroupGeom {
    using real = real_t;
    static constexpr int P = P_, NE = NE_, S = S_;
    static constexpr int Q = P + 1, L = Q * Q, N = Q * Q * Q;
    static constexpr int R = (Q + S - 1) / S;
    // Record of point (I, J, K) of element el: I + RP J + PP K + ES el.
    static constexpr GroupPitch PITCH = group_pitch(P, NE, IF_);
    static constexpr int RP = PITCH.row, PP = PITCH.plane, ES = PITCH.elem;
    static constexpr bool SWAP = PITCH.swap;
    static constexpr int NREC = (NE - 1) * ES + P * (1 + RP + PP) + 1;
    static constexpr bool IFIRST = IF_;
    // Numbers per array of scalars (pairs) and their element pitch beyond ES.
    static constexpr int SK = sizeof(real) == 4 ? group_pad4(P, NE, IF_) : 0, NSC = NREC + NE * SK;
    static constexpr int HK = sizeof(real) == 4 ? group_pad8(P, NE) : 0, NPR = NREC + NE * HK;
    static constexpr int LT = ((NE * L + 31) / 32) * 32;  // threads of one segment
    static constexpr int NT = S * LT;
    // Pitch of an element's He and gpvol in shared memory.  Where an element's
    // He is a multiple of all banks (porders 3 and 7: 64 x 9 and 512 x 9 words)
    // it is copied by itself, to a pitch of 16 bytes more, so that the elements
    // of a warp do not fall on one bank; other groups are copied as one span.
    static constexpr bool STAGED = sizeof(real) == 4;  // FP64: read in place (bound by FP64 issue, short of shared memory)
    static constexpr bool SPLIT = STAGED && N >= 64 && (9 * N) % 32 == 0;
    static constexpr int BANKS = 128 / (int)sizeof(real), OFF = 16 / (int)sizeof(real);
    static constexpr int pitch(int n) { return SPLIT ? n + (BANKS + OFF - n % BANKS) % BANKS : n; }
    static constexpr int HEP = pitch(9 * N), GPP = pitch(N);
    // Spans of the group with up to 12 bytes of shift (SpanPlan).
    static constexpr size_t span(int p, int n) { return (((size_t)(NE - 1) * p + n) * sizeof(real) + 12 + 15) / 16 * 16; }
    static constexpr size_t HEB = STAGED ? span(HEP, 9 * N) : 0;
    static constexpr bool GPSTAGED = STAGED && GP_;
    static constexpr size_t GPB = GPSTAGED ? span(GPP, N) : 0;
    template <int DIR>
    static constexpr int step()
    {
        return DIR == 0 ? 1 : (DIR == 1 ? RP : PP);
    }
};

// The thread's element and its line (q0, q1) of each direction: the line
// through (J, K) = (q0, q1) along xi (swapped where SWAP), (I, K) along eta,
// (I, J) along zeta.
template <class G>
struct GroupThread {
    int el, q0, q1, seg;
    bool active;
    __device__ __forceinline__ GroupThread(int tid)
    {
        seg = G::S == 1 ? 0 : tid / G::LT;
        const int t = tid - seg * G::LT;
        active = t < G::NE * G::L;
        if constexpr (G::IFIRST) {
            const int row = active ? t / G::Q : 0;
            q0 = active ? t - row * G::Q : 0;
            q1 = row / G::NE;
            el = row - q1 * G::NE;
        } else {
            const int line = active ? t / G::NE : 0;
            el = active ? t - line * G::NE : 0;
            q1 = line / G::Q;
            q0 = line - q1 * G::Q;
        }
    }
    // Record of the line's first point and its lattice index (K Q + J) Q + I.
    __device__ __forceinline__ int rec0(int dir) const
    {
        const bool sw = dir == 0 && G::SWAP;
        const int a = dir == 0 ? G::RP : 1, b = dir == 2 ? G::RP : G::PP;
        return el * G::ES + (sw ? q1 * a + q0 * b : q0 * a + q1 * b);
    }
    __device__ __forceinline__ int lat0(int dir) const
    {
        const bool sw = dir == 0 && G::SWAP;
        const int a = dir == 0 ? G::Q : 1, b = dir == 2 ? G::Q : G::L;
        return sw ? q1 * a + q0 * b : q0 * a + q1 * b;
    }
    // Lattice index of point r of the line.
    template <int DIR>
    __device__ __forceinline__ int lat(int r) const
    {
        return lat0(DIR) + r * (DIR == 0 ? 1 : (DIR == 1 ? G::Q : G::L));
    }
};

// Whether the warp's elements number their nodes closely (within an element's number
// of nodes along zeta), as a mesh of elements with nodes of their own does.  The lines of
// such an element share few cache lines, which one warp load after the other comes back
// to: they are then gathered through the L1, others past it (ldg_once).
template <class G>
__device__ __forceinline__ bool group_close(const int (&id)[G::R])
{
    static_assert(G::R > 1, "two points of a line");
    return __all_sync(0xffffffffu, abs(id[1] - id[0]) < G::N);
}

// Bulk copies of a group's He and gpvol spans into shared memory (one
// mbarrier phase), a span per lane of the first warp; the unaligned ends, if
// any, by plain loads.
template <class G>
struct GroupMetric {
    using real = typename G::real;
    // He(i, dir, a) of element el at He[el HEP + 9 a + 3 dir + i], gpvol(a) at gp[el GPP + a].
    real *He;
    const real *gp;
    int last;  // the group's last element
    __device__ __forceinline__ GroupMetric() : He(nullptr), gp(nullptr), last(0) {}
    __device__ __forceinline__ real *he(int el, int a) const
    {
        return He + (G::STAGED ? el : min(el, last)) * G::HEP + a * 9;
    }
    __device__ __forceinline__ const real *vol(int el, int a) const
    {
        return gp + (G::GPSTAGED ? el * G::GPP : min(el, last) * G::N) + a;
    }
    // Bounded wait for the bulk copies (false: the limit ran out).
    __device__ __forceinline__ bool wait(unsigned long long *bar) const { return G::STAGED ? mbar_wait(bar, 0) : true; }
    __device__ __forceinline__ GroupMetric(unsigned char *heb, unsigned char *gpb, unsigned long long *bar,
                                           const real *gHe, const real *ggp, int e0, int nelem, int tid)
    {
        last = min(G::NE, nelem - e0) - 1;
        if constexpr (!G::STAGED) {
            He = const_cast<real *>(gHe) + (size_t)e0 * G::N * 9;
            gp = ggp + (size_t)e0 * G::N;
            return;
        }
        constexpr int SPANS = G::SPLIT ? G::NE : 1;
        static_assert(SPANS <= 32, "one lane of the first warp per span");
        char *hs = reinterpret_cast<char *>(heb), *gs = reinterpret_cast<char *>(gpb);
        const int ne = min(G::NE, nelem - e0), spans = G::SPLIT ? ne : 1;
        const size_t n = (size_t)(G::SPLIT ? 1 : ne) * G::N;
        const unsigned hsh = (unsigned)(reinterpret_cast<size_t>(gHe + (size_t)e0 * G::N * 9) & 15);
        const unsigned gsh = (unsigned)(reinterpret_cast<size_t>(ggp + (size_t)e0 * G::N) & 15);
        if (tid < 32) {
            const int k = tid < spans ? tid : 0;  // the lane's span (the spans are alike modulo 16 bytes)
            const size_t off = ((size_t)e0 + k) * G::N;
            const SpanPlan ph(gHe + off * 9, n * 9 * sizeof(real)), pg(ggp + off, n * sizeof(real));
            if (tid == 0) {
                mbar_init(bar, 1);
                mbar_arrive_expect_tx(bar, (unsigned)spans * (ph.bulk + (G::GPSTAGED ? pg.bulk : 0u)));
            }
            __syncwarp();
            if (tid < spans) {
                ph.issue(hs + (size_t)k * G::HEP * sizeof(real), bar);
                if (G::GPSTAGED) pg.issue(gs + (size_t)k * G::GPP * sizeof(real), bar);
            }
            if (ph.head + ph.tail + pg.head + pg.tail != 0)
                for (int s = 0; s < spans; ++s) {
                    const size_t o = ((size_t)e0 + s) * G::N;
                    const SpanPlan qh(gHe + o * 9, n * 9 * sizeof(real)), qg(ggp + o, n * sizeof(real));
                    if (tid >= 8 && tid < 14) qh.plain(hs + (size_t)s * G::HEP * sizeof(real), tid - 8);
                    if (G::GPSTAGED && tid >= 16 && tid < 22) qg.plain(gs + (size_t)s * G::GPP * sizeof(real), tid - 16);
                }
        }
        He = reinterpret_cast<real *>(hs + hsh);
        gp = G::GPSTAGED ? reinterpret_cast<const real *>(gs + gsh) : ggp + (size_t)e0 * G::N;
    }
};

// The element tables of a call in shared memory, built by each block from the
// caller's arrays while its first loads are in flight: gmsh node of a lattice
// point, the directions' 1-D derivative matrices and their transposes (rows
// padded for vector loads), and their row sums.  dlxigp_ip(g, d, c) depends on g
// through its 1-D index in direction d only (elem_hex.f90:43-44).  Indices are
// clamped, so malformed tables give wrong numbers (reported by
// msod_check_element_tables), never accesses out of bounds.  A block spends two
// dependent loads of a few lanes on it, hidden behind the gather; the table
// kernel and the copy to the constant bank that this replaces were two
// launches per call (porder-4 convection on 16^3 hexes 43 -> 20 us with the
// zeroing in one launch; on 64^3 0.950 ms with the coefficients from shared
// memory, 0.944 from the constant bank).
// FULL: transposes, row sums and the node permutation too (the diffusion reads
// each matrix whole and needs none of them).
template <class G, bool FULL>
struct GroupTables {
    using real = typename G::real;
    static constexpr int Q = G::Q, N = G::N;
    static constexpr int ROW = (Q + 3) / 4 * 4;  // pitch of a row
    static constexpr size_t kD = (size_t)(FULL ? 6 : 3) * Q * ROW * sizeof(real);
    // Permutation entries of two bytes where the block's shared memory is short of 128 (the
    // porder-3 convection); elsewhere they cost up to 1.6 % (porder 7 32^3).
    using Node = std::conditional_t<G::P == 3, unsigned short, int>;
    static constexpr size_t kBytes = kD + (FULL ? (size_t)(3 * Q) * sizeof(real) + (size_t)N * sizeof(Node) : 0);
    unsigned char *base;  // 16-byte aligned
    __device__ __forceinline__ real *D(int dir, int r) const { return reinterpret_cast<real *>(base) + (dir * Q + r) * ROW; }
    __device__ __forceinline__ real *Dt(int dir, int c) const { return D(3 + dir, c); }
    __device__ __forceinline__ real *sums() const { return reinterpret_cast<real *>(base + kD); }  // [dir Q + r]
    __device__ __forceinline__ Node *perm() const { return reinterpret_cast<Node *>(sums() + 3 * Q); }
    static __device__ __forceinline__ int node(const int *inv, int l) { return min(max(ldg(inv + l) - 1, 0), N - 1); }
    // All threads call it; complete after the next barrier.
    __device__ __forceinline__ void build(const int *__restrict__ inv, const real *__restrict__ dlx, int tid) const
    {
        if (FULL)
            for (int i = tid; i < N; i += G::NT) perm()[i] = (Node)node(inv, i);
        const int i = tid - (G::NT - 32);  // the last warp: one row per lane
        if (i >= 0 && i < 3 * Q) {
            const int d = i / Q, r = i - d * Q;
            const int a = node(inv, d == 0 ? r : (d == 1 ? r * Q : r * Q * Q));
            real v[Q];
#pragma unroll
            for (int c = 0; c < Q; ++c) v[c] = ldg(dlx + (size_t)(c * 3 + d) * N + a);
            double sum = 0.0;
#pragma unroll
            for (int c = 0; c < Q; ++c) {
                D(d, r)[c] = v[c];
                if (FULL) {
                    Dt(d, c)[r] = v[c];
                    sum += (double)v[c];
                }
            }
            if (FULL) sums()[i] = (real)sum;
        }
    }
};

// Loads of shared memory that no thread writes any more: plain functions of the
// address to the compiler, which may move them across the stores of the sums
// and fluxes (it cannot tell them apart from other shared memory) and so hide
// their latency.  The address comes from after_barrier, which keeps them below
// the barrier that completed the data.
__device__ __forceinline__ unsigned after_barrier(const void *p)
{
    unsigned a;
    asm volatile("mov.u32 %0, %1;" : "=r"(a) : "r"(smem_u32(p)) : "memory");
    return a;
}
__device__ __forceinline__ void lds(int &v, unsigned a) { asm("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a)); }
__device__ __forceinline__ void lds_u16(int &v, unsigned a) { asm("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a)); }
__device__ __forceinline__ void lds(float &v, unsigned a) { asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void lds(double &v, unsigned a) { asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); }
__device__ __forceinline__ void lds(Four<float> &v, unsigned a)
{
    asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.b.x), "=f"(v.b.y) : "r"(a));
}
__device__ __forceinline__ void lds(Four<double> &v, unsigned a)
{
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.a.x), "=d"(v.a.y) : "r"(a));
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.b.x), "=d"(v.b.y) : "r"(a + 16));
}

// The tables as the passes read them (after the barrier that follows build).
template <class G, bool FULL>
struct GroupRows {
    using real = typename G::real;
    using T = GroupTables<G, FULL>;
    unsigned base;
    __device__ __forceinline__ explicit GroupRows(const T &t) : base(after_barrier(t.base)) {}
    __device__ __forceinline__ void load(real (&v)[G::Q], int row) const
    {
        constexpr int Q = G::Q;
#pragma unroll
        for (int c = 0; c < Q; c += 4) {
            Four<real> f;
            lds(f, base + (unsigned)((row * T::ROW + c) * sizeof(real)));
            v[c] = f.a.x;
            if (c + 1 < Q) v[c + 1 < Q ? c + 1 : 0] = f.a.y;
            if (c + 2 < Q) v[c + 2 < Q ? c + 2 : 0] = f.b.x;
            if (c + 3 < Q) v[c + 3 < Q ? c + 3 : 0] = f.b.y;
        }
    }
    // Row r, column c of direction dir's matrix; its row sums; lattice -> gmsh node.
    __device__ __forceinline__ void row(real (&v)[G::Q], int dir, int r) const { load(v, dir * G::Q + r); }
    __device__ __forceinline__ void col(real (&v)[G::Q], int dir, int c) const { load(v, (3 + dir) * G::Q + c); }
    __device__ __forceinline__ real sum(int dir, int r) const
    {
        real v;
        lds(v, base + (unsigned)(T::kD + (dir * G::Q + r) * sizeof(real)));
        return v;
    }
    __device__ __forceinline__ int node(int l) const
    {
        int v;
        const unsigned at = base + (unsigned)(T::kD + 3 * G::Q * sizeof(real) + l * sizeof(typename T::Node));
        if constexpr (sizeof(typename T::Node) == 2)
            lds_u16(v, at);
        else
            lds(v, at);
        return v;
    }
};

}  // namespace
}  // namespace msod
