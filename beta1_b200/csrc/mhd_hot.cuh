// Launch arguments and point addressing of the hot stencil kernels.
//
// A hot kernel receives the blocks it covers by value (kernel parameters, in
// the constant bank), and finds its point without touching global memory:
//
// * block of the CTA: blockIdx.y, or for flattened launches over uneven
//   blocks a binary search of the blocks' first CTAs;
// * (i, j, k) of the thread: 32-bit multiply-shift quotients with the
//   multipliers of the block's extents formed on the host (a 64-bit integer
//   division costs about 70 instructions, and a point needs four);
// * field planes: every plane of a block has the same stride, so plane q of
//   the pool is at p0 + q vol, q a compile-time number; neighbours are 32-bit
//   offsets from the thread's own point (+-si, +-sj, +-1).
//
// The kernels before read the CTA table, then the block's view, then one
// pointer per field from global memory: three dependent loads before the
// first field value, and two registers per field pointer.
#pragma once

#include "mhd_layout.cuh"

#include <vector>

namespace mhd
{

// first plane of field f in a block's pool range (a constant where f is one)
__host__ __device__ constexpr int plane_of(int f)
{
    int q = 0;
#define MHD_PLANE(id, name, loc, nc, ng) \
    if (f > F_##id)                      \
        q += nc;
    MHD_FIELD_LIST(MHD_PLANE)
#undef MHD_PLANE
    return q;
}
constexpr int kPoolPlanes = plane_of(NFIELD);
// planes of the mixed form's FP32 range: face geometry, face states, weights
constexpr int kPlane32Q = G32_N, kPlane32W = G32_N + Q32_N;

// quotient of a non-negative 31-bit number by a fixed divisor: (t mul) >> shift
struct FastDiv
{
    uint32_t mul, shift;
};
// mul = floor(2^(31 + l) / d) + 1 with l = ceil(log2 d): exact for t < 2^31
inline FastDiv fast_div(uint32_t d)
{
    uint32_t l = 0;
    while ((uint64_t(1) << l) < d)
        ++l;
    return FastDiv{uint32_t((uint64_t(1) << (31 + l)) / d + 1), 31 + l};
}
__host__ __device__ inline uint32_t fast_quot(uint32_t t, FastDiv f)
{
    return uint32_t((uint64_t(t) * f.mul) >> f.shift);
}

struct HotBlock
{
    double *p0;         // plane 0 of the block
    float *p32;         // plane 0 of its FP32 range (mixed form; null otherwise)
    double *rk;         // SSP-RK2 start-of-step state (null otherwise)
    const double *qref; // its run's reference state of the mixed flux
    uint32_t vol;       // points per plane
    uint32_t si, sj;    // strides of i and j
    uint32_t o;         // offset of the point (0, 0, 0)
    int ni, nj, nk;
    int run, blk;
    int poles;          // 1: a Pole at j = 0, 2: at j = n_j
    int cta0[3];        // flattened launches: first CTA per kind, within this launch
    // quotients by n_k + e and n_j + e: e = 0 (KIND_CELL0), 2 (KIND_CELL1), 1 (KIND_STAG)
    FastDiv dk[3], dj[3];
};

template <int NB> struct HotArgs
{
    int n;    // blocks
    int flat; // one grid row of every block's CTAs
    HotBlock v[NB];
};
// capacities of a launch: a context of few blocks passes little, a batch is
// split into launches of at most kHotMax blocks
constexpr int kHotFew = 8, kHotMax = 64;
static_assert(sizeof(HotArgs<kHotMax>) <= 16384, "kernel parameters");

// The blocks of a context in launches of at most kHotMax: per launch its
// arguments (few: the same blocks in the small form, when they fit) and the
// CTAs per kind (flattened: all; else of the largest block), of 256 threads.
struct HotChunk
{
    HotArgs<kHotMax> args;
    HotArgs<kHotFew> few;
    uint32_t ctas[3];
    int64_t padded; // points of the largest block with all its ghost layers
};
struct HotGrid
{
    std::vector<HotChunk> chunks;
    int G = 4;
};

#ifdef __CUDACC__

// Programmatic dependent launch: a kernel launched with the attribute may start
// while the kernel before it drains; what it does before pdl_wait() must read
// nothing an earlier kernel writes.  Every kernel of the step waits, so a
// kernel that has finished implies all before it have.
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// block of the calling CTA and the thread's index among the block's threads
template <int KIND, class A> __device__ __forceinline__ const HotBlock &hot_block(const A &a, uint32_t &t)
{
    uint32_t cta = blockIdx.x;
    int bi = int(blockIdx.y);
    if (a.flat)
    {
        int lo = 0, hi = a.n;
        while (hi - lo > 1)
        {
            const int mid = (lo + hi) >> 1;
            if (uint32_t(a.v[mid].cta0[KIND]) <= cta)
                lo = mid;
            else
                hi = mid;
        }
        bi = lo;
        cta -= uint32_t(a.v[lo].cta0[KIND]);
    }
    t = cta * blockDim.x + threadIdx.x;
    return a.v[bi];
}

// point t of a kind's box (k fastest) and its offset p within a plane
template <int KIND>
__device__ __forceinline__ bool hot_point(const HotBlock &b, uint32_t t, int &i, int &j, int &k, uint32_t &p)
{
    constexpr int lo = KIND == KIND_CELL1 ? -1 : 0;
    constexpr int e = KIND == KIND_CELL1 ? 2 : KIND == KIND_STAG ? 1 : 0;
    const uint32_t q = fast_quot(t, b.dk[KIND]);
    const int kk = int(t - q * uint32_t(b.nk + e));
    const int ii = int(fast_quot(q, b.dj[KIND]));
    const int jj = int(q) - ii * (b.nj + e);
    i = ii + lo;
    j = jj + lo;
    k = kk + lo;
    p = b.o + uint32_t(i) * b.si + uint32_t(j) * b.sj + uint32_t(k);
    return ii < b.ni + e;
}

// staggered point t of the block, or of the box rng[6 blk] (lo[3], hi[3])
// when a region table is given
__device__ __forceinline__ bool hot_stagger(const HotBlock &b, const int *rng, uint32_t t, int &i, int &j, int &k,
                                            uint32_t &p)
{
    if (!rng)
        return hot_point<KIND_STAG>(b, t, i, j, k, p);
    const int *r = rng + 6 * b.blk;
    const uint32_t n2 = uint32_t(r[5] - r[2]), n1 = uint32_t(r[4] - r[1]), n0 = uint32_t(r[3] - r[0]);
    if (n0 == 0 || n1 == 0 || n2 == 0 || t >= n0 * n1 * n2)
        return false;
    const uint32_t q = t / n2;
    k = r[2] + int(t - q * n2);
    const uint32_t ii = q / n1;
    j = r[1] + int(q - ii * n1);
    i = r[0] + int(ii);
    p = b.o + uint32_t(i) * b.si + uint32_t(j) * b.sj + uint32_t(k);
    return true;
}

// plane q of the block at the thread's point
__device__ __forceinline__ double *hot_plane(const HotBlock &b, uint32_t p, int q)
{
    return b.p0 + (uint64_t(b.vol) * uint32_t(q) + p);
}
// component m of field f at the thread's point
__device__ __forceinline__ double *hot_at(const HotBlock &b, uint32_t p, int f, int m = 0)
{
    return hot_plane(b, p, plane_of(f) + m);
}
__device__ __forceinline__ float *hot_plane32(const HotBlock &b, uint32_t p, int q)
{
    return b.p32 + (uint64_t(b.vol) * uint32_t(q) + p);
}

// L2 prefetch of what a later CTA of the launch reads: the CTA kAhead CTAs on
// (x fastest, then y), its points' range of each listed plane, one bulk
// prefetch per plane by one lane.  planes: pool planes, or ~q for plane q of
// the FP32 range.  For the flux passes, whose 80 to 124 registers leave 16 to
// 24 warps per SM to hide DRAM latency: FP64 84 -> 71 us on 0.76 M cells, mixed
// 221 -> 199 us on 2.27 M.  37 to 148 CTAs ahead are the same, 296 and more
// slower.  The passes with more warps or a weight stream got slower (PV 96 ->
// 110 us, B_cell 50 -> 52) and do not use it.
constexpr uint32_t kAhead = 74;
template <int KIND, int N, class A>
__device__ __forceinline__ void hot_prefetch(const A &a, const int16_t (&planes)[N])
{
    static_assert(N <= 32, "one warp");
    if (threadIdx.x >= N)
        return;
    uint32_t cta = blockIdx.x + kAhead;
    int bi = int(blockIdx.y);
    if (a.flat)
    {
        if (cta >= gridDim.x)
            return;
        int lo = 0, hi = a.n;
        while (hi - lo > 1)
        {
            const int mid = (lo + hi) >> 1;
            if (uint32_t(a.v[mid].cta0[KIND]) <= cta)
                lo = mid;
            else
                hi = mid;
        }
        bi = lo;
        cta -= uint32_t(a.v[lo].cta0[KIND]);
    }
    else if (cta >= gridDim.x)
    {
        cta -= gridDim.x;
        if (++bi >= a.n || cta >= gridDim.x)
            return;
    }
    const HotBlock &b = a.v[bi];
    int i, j, k;
    uint32_t p0, p1;
    if (!hot_point<KIND>(b, cta * blockDim.x, i, j, k, p0))
        return;
    if (!hot_point<KIND>(b, cta * blockDim.x + blockDim.x - 1, i, j, k, p1))
        p1 = p0 + blockDim.x < b.vol ? p0 + blockDim.x : b.vol - 1;
    const int q = planes[threadIdx.x];
    const char *at;
    uint32_t bytes;
    if (q >= 0)
    {
        p0 &= ~1u;
        at = reinterpret_cast<const char *>(b.p0 + (uint64_t(b.vol) * uint32_t(q) + p0));
        bytes = (p1 - p0 + 2) / 2 * 16;
    }
    else
    {
        p0 &= ~3u;
        at = reinterpret_cast<const char *>(b.p32 + (uint64_t(b.vol) * uint32_t(~q) + p0));
        bytes = (p1 - p0 + 4) / 4 * 16;
    }
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(bytes) : "memory");
}

// inner cell
__device__ __forceinline__ bool hot_inner(const HotBlock &b, int i, int j, int k)
{
    return uint32_t(i) < uint32_t(b.ni) && uint32_t(j) < uint32_t(b.nj) && uint32_t(k) < uint32_t(b.nk);
}
// is the staggered point (i, j, k) >= 0 an inner face / edge of axis a
__device__ __forceinline__ bool hot_face(const HotBlock &b, int a, int i, int j, int k)
{
    return i < b.ni + (a == 0) && j < b.nj + (a == 1) && k < b.nk + (a == 2);
}
__device__ __forceinline__ bool hot_edge(const HotBlock &b, int a, int i, int j, int k)
{
    return i < b.ni + (a != 0) && j < b.nj + (a != 1) && k < b.nk + (a != 2);
}
#endif

} // namespace mhd
