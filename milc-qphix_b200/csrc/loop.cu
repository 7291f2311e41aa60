// Resident solver loop: the iterations of one solver phase (a CG pass between
// restarts, a mixed-precision run between reliable updates, a multi-shift
// pass) in ONE cooperative launch.
//
// The launch-per-kernel form of an iteration (dslash.cu, blas.cu) is bound by
// launches and by each kernel's ramp on small and medium lattices: at 8^4 in
// FP64 an iteration of four kernels inside the CUDA-graph while loop took
// 30 us, although its 19 MB of links come from L2.  Here every block stays
// resident and the phases of an iteration are separated by grid barriers:
//   1  tmp = D p          | barrier
//   2  ttt = D tmp + m4 p, p.ttt        | barrier with sum, scalar step
//   3  r += a ttt, |r|^2                | barrier with sum, scalar step
//   4  x += a p, p = r + b p (or the shifts' updates) | barrier
// The scalar steps are the functors of solver_steps.cuh on a copy of the
// SolverState in shared memory: every block sums the same partials in the
// same order, so all copies stay identical and no scalar is read back from
// another block.  Block 0 stores its copy at the end.
//
// Barrier: one counter, added to with release by one thread per block and
// polled with acquire by that thread; 2.5 k cycles at 148 blocks, and 3.7 k
// with a sum (every block reads all partials).  Publishing {value, epoch}
// words per block and polling all of them, without atomics, took 6.5 k: 148
// blocks polling 148 words load the L2 more than one hot word does.  Every
// wait is bounded (wait_limit() polls); a block whose wait runs out stores the
// failure word and returns, and so do the others, whose next wait then cannot
// end.
//
// Dslash: a group of PARTS * SG threads owns SG consecutive sites; part k of
// the group (SG threads) applies one direction's links of one hop (8 parts) or
// both hops (4), and the parts' sums are combined through shared memory.
// Against one thread per site the chain of eight dependent load stages becomes
// one or two, and a lattice of 2048 sites occupies 16 thousand threads.  SG =
// 32 keeps every link load 512 contiguous bytes per warp (with 4 or 8 lanes
// per site, 128- or 64-byte runs, the same phase ran at 24 and 16 B per clock
// and SM); smaller groups only spread lattices that would leave SMs idle.
//
// us per iteration of the kernels in the graph loop / here (one B200, m =
// 0.02, reliable updates included): FP64 8^4 30.0 / 10.0, 12^3x24 39.0 /
// 21.2, 16^3x32 69.4 / 59.4, 24^3x48 276 / 263; FP32 25.6 / 9.5, 29.9 /
// 15.2, 45.5 / 31.2, 143.5 / 130.0; FP32 with 12-real Naik links 27.9 / 11.9,
// 33.1 / 18.7, 47.3 / 34.9, 133.2 / 127.4; 16-bit links 27.6 / 12.0, 32.5 /
// 18.4, 42.7 / 30.5, 104.6 / 99.8.  At 8^4 the barriers are half of the
// iteration; at 24^3x48 (12-real) the loop runs at 5.6 TB/s of DRAM with 32 %
// of the issue slots used, waiting for loads and at the groups' barriers.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <stdexcept>
#include <string>

#include "device_common.cuh"
#include "solver_steps.cuh"

namespace qb {

namespace {

constexpr int kLoopMaxBlocks = 256;         // partial sums per buffer

// most threads of a block: 64 registers each for FP32 sums, 128 for FP64
// eight_parts: largest lattice (sites per parity) whose Dslash is split into
// eight parts a site instead of four.  Eight make the chain of loads one stage
// long, four halve the instructions spent on indices and on the combination.
// The lines are where a lattice fills one round (FP32: 148 SMs x 4 groups x 32
// sites = 18944) and three rounds (FP64: 148 x 2 x 32 = 9472 each) of
// eight-part groups; between whole rounds either form can be ahead, by 8 % at
// most.  us per iteration with eight / four (four phases, 10368, 18432, 20736,
// 24576 and 30720 sites): FP64 16.6 / 15.4, 17.7 / 17.3, 21.2 / 23.3, 21.4 /
// 23.0, 26.2 / 25.5; FP32 12.5 / 13.5, 14.9 / 15.1, 18.0 / 16.4, 19.2 / 17.9,
// 18.9 / 17.2; 12-real 16.9 / 17.1, 18.6 / 17.5, 21.6 / 18.1, 21.9 / 18.9, 23.6
// / 21.5; 16-bit vectors 17.6 / 16.9, 18.7 / 17.6, 22.8 / 18.5, 23.3 / 19.7,
// 25.2 / 22.3.  4096 sites: FP64 11.7 / 12.7, FP32 11.4 / 12.6; 24^3x48: 16-bit
// links 109.5 / 101.3, FP64 271 / 265.  (The eight-part 12- and 13-real forms
// spill about 90 bytes a thread, the mirrored 13-real one 52.)
template <typename SV> struct LoopThreads {
    static constexpr int value = 1024, eight_parts = 18944;
};
template <> struct LoopThreads<double> {
    static constexpr int value = 512, eight_parts = 28416;
};

// j / n for 0 <= j < 2^31 by a multiplication: m = ceil(2^(31+s) / n) with
// 2^s >= n, so m n <= 2^(31+s) + 2^s and the quotient is exact
struct FastDiv {
    unsigned m;
    int s;  // (shift after the high word)
    __device__ __forceinline__ int div(int j) const { return (int)(__umulhi((unsigned)j, m) >> s); }
};

template <typename SV, typename SL>
struct LoopArgs {
    Geom g;
    LinkView<SL> links[2];  // by output parity
    int parity;             // parity of p, ttt, r, x
    VecView<SV> p, tmp, ttt, r;
    VecView<SV> p2;         // second buffer of the direction (k_small_loop)
    void *x;                // CG: the solution (FP32 under 16-bit vectors)
    double m4, delta2;
    SolverState *st;
    unsigned *counter;      // barrier arrivals
    double *partials;       // [2 parities of the epoch][block]
    int *err;
    unsigned polls;         // poll limit of a barrier wait
    int sg, lg_sg;          // sites of a group (4..32) and its logarithm
    int groups;             // groups of a block
    FastDiv dx, dy, dz;     // by Nxh, Ny, Nz
    // multi-shift
    int n;
    VecBlock *xs, *ps;
    float2 *hist;
    MsHistEntry *hist_s;
};

// ------------------------------------------------------------------ barrier --
__device__ __forceinline__ void arrive_release(unsigned *c)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
}
__device__ __forceinline__ unsigned load_acquire(const unsigned *c)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
    return v;
}

struct LoopShared {
    SolverState st;
    double w[32];
    int fail;
};

struct LoopBarrier {
    unsigned *counter;
    double *partials;
    unsigned polls;
    unsigned epoch;
};

// Grid barrier; writes made before by any thread of the grid are visible to
// every thread after.  False when the wait ran out.
__device__ __forceinline__ bool grid_wait(LoopShared &sh, LoopBarrier &b)
{
    ++b.epoch;
    __syncthreads();
    if (threadIdx.x == 0) {
        arrive_release(b.counter);
        const unsigned target = b.epoch * gridDim.x;  // modulo 2^32, as the counter
        unsigned k = 0;
        while (k < b.polls && (int)(load_acquire(b.counter) - target) < 0) ++k;
        if (k >= b.polls) sh.fail = 1;
    }
    __syncthreads();
    return sh.fail == 0;
}

// Grid barrier that also adds `v` over all threads of the grid in a fixed
// order: every block sums the same partials the same way, so all get the same
// total.  The partials are double-buffered by epoch parity: a block writes
// epoch e + 2 only after barrier e + 1, which every block enters after it
// has read epoch e.
__device__ __forceinline__ bool grid_sum(double v, double &total, LoopShared &sh, LoopBarrier &b)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5, nb = gridDim.x;
    double *part = b.partials + ((b.epoch + 1) & 1u) * kLoopMaxBlocks;
    v = warp_sum(v);
    if (lane == 0) sh.w[w] = v;
    __syncthreads();
    if (w == 0) {
        double s = lane < nw ? sh.w[lane] : 0.0;
        s = warp_sum(s);
        if (lane == 0) part[blockIdx.x] = s;
    }
    if (!grid_wait(sh, b)) return false;
    double s = 0.0;
    if (32 * w < nb) {
        for (int i = tid; i < nb; i += blockDim.x) s += __ldcg(part + i);
        s = warp_sum(s);
    }
    if (lane == 0) sh.w[w] = s;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < nw && 32 * k < nb; ++k) t += sh.w[k];
    total = t;
    return true;
}

// ------------------------------------------------------------------- Dslash --
// Links are read once per iteration and site: past L1.  (Marking them
// evict-first in L2 where they do not fit did not make the vectors stay:
// 24^3x48 133.9 against 130.6 us per iteration, 12-real.)
#define QB_LD_LINK(TYPE, VEC, REGS, ...)                                                             \
    __device__ __forceinline__ TYPE ld_link(const TYPE *p)                                           \
    {                                                                                                \
        TYPE v;                                                                                      \
        asm volatile("ld.global.nc.L1::no_allocate." VEC " " REGS ";" : __VA_ARGS__ : "l"(p));      \
        return v;                                                                                    \
    }
QB_LD_LINK(float4, "v4.f32", "{%0, %1, %2, %3}, [%4]", "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w))
QB_LD_LINK(int4, "v4.s32", "{%0, %1, %2, %3}, [%4]", "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w))
QB_LD_LINK(double2, "v2.f64", "{%0, %1}, [%2]", "=d"(v.x), "=d"(v.y))
QB_LD_LINK(float2, "v2.f32", "{%0, %1}, [%2]", "=f"(v.x), "=f"(v.y))
#undef QB_LD_LINK

// Loads of vectors that this kernel writes: not through the non-coherent
// path (the barrier's fence makes the other blocks' stores visible).
__device__ __forceinline__ void ld_vec(const VecView<double> &f, int j, double v[6])
{
    const double2 a = f.p[j], b = f.p[f.vh + j], c = f.p[2 * f.vh + j];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}
__device__ __forceinline__ void ld_vec(const VecView<float> &f, int j, float v[6])
{
    const float2 a = f.p[j], b = f.p[f.vh + j], c = f.p[2 * f.vh + j];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}
__device__ __forceinline__ void ld_vec(const VecView<__half> &f, int j, float v[6])
{
    VecView<__half>::unpack(f.p[j], v);
}

// The Dslash input r + b p of a direction that is not stored yet (`first`: p
// itself)
template <typename SV>
struct SumIn {
    VecView<SV> p, r;
    SV b;
    bool first;
    __device__ __forceinline__ SV at(SV pv, SV rv) const { return first ? pv : fma_(b, pv, rv); }
};
template <typename SV>
__device__ __forceinline__ void ld_vec(const SumIn<SV> &f, int j, SV v[6])
{
    SV q[6];
    ld_vec(f.p, j, v);
    ld_vec(f.r, j, q);
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = f.at(v[k], q[k]);
}

// What a thread of part (direction d, hop 1 + 2h) keeps for all its sites
struct PartGeom {
    int n, str;  // extent and stride of d
    bool x;
};

// block indices of the forward and backward neighbour 1 + 2h hops away
// (geometry.cuh neighbor(); x in checkerboard units: xh + xodd + {0, -1, 1,
// -2}; |offset| <= extent, so one wrap is enough)
__device__ __forceinline__ void part_neighbors(const PartGeom &q, const SiteCoords &s, int d, int h, int j, int &f,
                                               int &b)
{
    const int c = d == 0 ? s.xh : d == 1 ? s.y : d == 2 ? s.z : s.t;
    f = c + (q.x ? s.xodd + h : 1 + 2 * h);
    b = c + (q.x ? s.xodd - 1 - h : -1 - 2 * h);
    f -= f >= q.n ? q.n : 0;
    b += b < 0 ? q.n : 0;
    f = j + (f - c) * q.str;
    b = j + (b - c) * q.str;
}

// acc = U_f psi(f) - U_b^dag psi(b) for the pair (direction d, fat or Naik h)
// of site j.  lk: the links of the output parity, lo: of the other.  Mirrored: the
// backward link is read as the forward link of its own site b (lo), where
// the caller's backward links are exactly those (LinkSet::mirrored).
template <bool MIR, typename In>
__device__ __forceinline__ void part_dslash(const LinkView<double> &lk, const LinkView<double> &lo,
                                            const In &in, int d, int h, int j, int f, int b,
                                            double acc[6])
{
    double vf[6], vb[6], u[18], w[18];
    const double2 *c = lk.p + (size_t)(36 * d + 18 * h) * lk.vh + j;
    const double2 *cb = MIR ? lo.p + (size_t)(36 * d + 18 * h) * lk.vh + b : c + (size_t)9 * lk.vh;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const double2 z = ld_link(c + (size_t)e * lk.vh);
        u[2 * e] = z.x; u[2 * e + 1] = z.y;
    }
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const double2 z = ld_link(cb + (size_t)e * lk.vh);
        w[2 * e] = z.x; w[2 * e + 1] = z.y;
    }
    ld_vec(in, f, vf);
    ld_vec(in, b, vb);
    mv_add_fma(acc, u, vf);
    mv_adj_sub_fma(acc, w, vb);
}

template <bool MIR, typename In, typename SL>
__device__ __forceinline__ void part_dslash(const LinkView<SL> &lk, const LinkView<SL> &lo, const In &in,
                                            int d, int h, int j, int f, int b, float acc[6])
{
    float vf[6], vb[6], u[36];
    const size_t vh = lk.vh;
    if constexpr (std::is_same<SL, __half>::value) {
        // words 18h .. 18h+17 of the direction's 36 (two 16-bit values each)
        // are the pair's two matrices: chunks 0-4 (fat) or 4-8 (Naik)
        int4 raw[MIR ? 6 : 5];
        const int4 *c = lk.p + (size_t)(9 * d + 4 * h) * vh + j;
#pragma unroll
        for (int k = 0; k < (MIR ? 3 : 5); ++k) raw[k] = ld_link(c + k * vh);
        if constexpr (MIR) {
            const int4 *cb = lo.p + (size_t)(9 * d + 4 * h) * vh + b;
#pragma unroll
            for (int k = 0; k < 3; ++k) raw[3 + k] = ld_link(cb + k * vh);
        }
        ld_vec(in, f, vf);
        ld_vec(in, b, vb);
        const unsigned *w = reinterpret_cast<const unsigned *>(raw);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const float2 z = fx16x2(h ? w[2 + k] : w[k]);
            u[2 * k] = z.x;
            u[2 * k + 1] = z.y;
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int o = MIR ? 12 : 9;
            const float2 z = fx16x2(h ? w[o + 2 + k] : w[o + k]);
            u[18 + 2 * k] = z.x;
            u[18 + 2 * k + 1] = z.y;
        }
    } else {
        constexpr bool RN = !std::is_same<SL, float>::value;
        const size_t chunk = (size_t)(d * (RN ? kReconChunks : 18) + 9 * h) * vh;
        const float4 *c = lk.p + chunk + j;
        if (RN && h) {
            if constexpr (RN) {
                float4 cn[6];
                const float4 *cb = MIR ? lo.p + chunk + b : c + 3 * vh;
#pragma unroll
                for (int k = 0; k < 3; ++k) cn[k] = ld_link(c + k * vh);
#pragma unroll
                for (int k = 0; k < 3; ++k) cn[3 + k] = ld_link(cb + k * vh);
                unsigned bits = lk.fetch_aux(j);
                float4 lam = lk.fetch_lam(d, j);
                if constexpr (MIR) {
                    // the backward link's sign bit (ratio) is its own site's forward one
                    const unsigned bb = (lo.fetch_aux(b) >> (2 * d)) & 1u;
                    bits = (bits & ~(2u << (2 * d))) | (bb << (2 * d + 1));
                    if constexpr (LinkView<SL>::has_lam) {
                        const float4 lb = lo.fetch_lam(d, b);
                        lam.z = lb.x;
                        lam.w = lb.y;
                    }
                }
                ld_vec(in, f, vf);
                ld_vec(in, b, vb);
                lk.naik_from(cn, d, bits, lam, u, u + 18);
            }
        } else {
            float4 cf[9];
            if constexpr (MIR) {
                const float4 *cb = lo.p + chunk + b;
                float2 e8, b8;
#pragma unroll
                for (int k = 0; k < 4; ++k) cf[k] = ld_link(c + k * vh);
                e8 = ld_link(reinterpret_cast<const float2 *>(c + 4 * vh));
#pragma unroll
                for (int k = 0; k < 4; ++k) cf[5 + k] = ld_link(cb + k * vh);
                b8 = ld_link(reinterpret_cast<const float2 *>(cb + 4 * vh));
                ld_vec(in, f, vf);
                ld_vec(in, b, vb);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    u[4 * k] = cf[k].x; u[4 * k + 1] = cf[k].y; u[4 * k + 2] = cf[k].z; u[4 * k + 3] = cf[k].w;
                    u[18 + 4 * k] = cf[5 + k].x; u[18 + 4 * k + 1] = cf[5 + k].y;
                    u[18 + 4 * k + 2] = cf[5 + k].z; u[18 + 4 * k + 3] = cf[5 + k].w;
                }
                u[16] = e8.x; u[17] = e8.y;
                u[34] = b8.x; u[35] = b8.y;
            } else {
#pragma unroll
                for (int k = 0; k < 9; ++k) cf[k] = ld_link(c + k * vh);
                ld_vec(in, f, vf);
                ld_vec(in, b, vb);
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    u[4 * k] = cf[k].x; u[4 * k + 1] = cf[k].y; u[4 * k + 2] = cf[k].z; u[4 * k + 3] = cf[k].w;
                }
            }
        }
    }
    mv_add_fma(acc, u, vf);
    mv_adj_sub_fma(acc, u + 18, vb);
    if constexpr (std::is_same<SL, __half>::value) {
        const float sc = h ? lk.scale_long : lk.scale_fat;
#pragma unroll
        for (int i = 0; i < 6; ++i) acc[i] *= sc;
    }
}

// barrier over the threads of one group (warps of the block)
__device__ __forceinline__ void group_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// One thread's place in its group: site i of the group's sg, part (d, h) of 8
// or part d of 4 (both hops)
struct GroupPlace {
    int grp, gthreads, t, i, part, d, h;
    PartGeom q;
};

template <int PARTS, typename SV, typename SL>
__device__ __forceinline__ GroupPlace group_place(const LoopArgs<SV, SL> &a)
{
    GroupPlace p;
    p.gthreads = PARTS * a.sg;
    p.grp = threadIdx.x / p.gthreads;
    p.t = threadIdx.x - p.grp * p.gthreads;
    p.i = p.t & (a.sg - 1);
    p.part = p.t >> a.lg_sg;
    p.d = p.part & 3;
    p.h = p.part >> 2;
    const Geom &g = a.g;
    p.q.x = p.d == 0;
    p.q.n = p.q.x ? g.nxh : p.d == 1 ? g.ny : p.d == 2 ? g.nz : g.nt;
    p.q.str = p.q.x ? 1 : p.d == 1 ? g.sy : p.d == 2 ? g.sz : g.st;
    return p;
}

// One tile: out = D in (+ m4 p, with the products p.out added to dot; `own`
// gives component c of p at site j) at the group's sites j0 .. j0 + sg - 1 of
// parity cb.  `buf`: 6 reals per thread of
// the group; the caller alternates two of them, so a thread that reaches the
// next tile's barrier has read the buffer of the tile before.
template <int PARTS, bool MDAGM, bool MIR, typename SV, typename SL, typename In, typename A, typename Own>
__device__ __forceinline__ void tile_dslash(const LoopArgs<SV, SL> &a, const GroupPlace &p, int j0, int cb,
                                            const In &in, const VecView<SV> &out, A *buf, double &dot, Own own)
{
    const int j = j0 + p.i, vh = a.g.vh, sg = a.sg, part = p.part;
    SiteCoords s;
    {
        int r = a.dx.div(j);
        s.xh = j - r * a.g.nxh;
        int r2 = a.dy.div(r);
        s.y = r - r2 * a.g.ny;
        s.t = a.dz.div(r2);
        s.z = r2 - s.t * a.g.nz;
        s.xodd = (s.y + s.z + s.t + cb) & 1;
    }
    int f, b;
    A acc[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = A(0);
    if constexpr (PARTS == 8) {
        part_neighbors(p.q, s, p.d, p.h, j, f, b);
        part_dslash<MIR>(a.links[cb], a.links[1 - cb], in, p.d, p.h, j, f, b, acc);
    } else {
        A naik[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) naik[k] = A(0);
        part_neighbors(p.q, s, p.d, 0, j, f, b);
        part_dslash<MIR>(a.links[cb], a.links[1 - cb], in, p.d, 0, j, f, b, acc);
        part_neighbors(p.q, s, p.d, 1, j, f, b);
        part_dslash<MIR>(a.links[cb], a.links[1 - cb], in, p.d, 1, j, f, b, naik);
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] += naik[k];
    }
    cx_t<A> pv;
    if constexpr (MDAGM && !std::is_same<SV, __half>::value)
        if (part < 3) pv = own(part, j);
#pragma unroll
    for (int k = 0; k < 6; ++k) buf[(part * 6 + k) * sg + p.i] = acc[k];
    group_sync(1 + p.grp, p.gthreads);
    if constexpr (std::is_same<SV, __half>::value) {
        if (part == 0) {
#pragma unroll
            for (int k = 0; k < 6; ++k)
#pragma unroll
                for (int q = 1; q < PARTS; ++q) acc[k] += buf[(q * 6 + k) * sg + p.i];
            if constexpr (MDAGM) {
                A pj[6];
                ld_vec(a.p, j, pj);
                const A m = (A)a.m4;
#pragma unroll
                for (int k = 0; k < 6; ++k) acc[k] = acc[k] + m * pj[k];
                out.store(j, acc);  // acc now holds the stored (rounded) value
#pragma unroll
                for (int k = 0; k < 6; ++k) dot += (double)(pj[k] * acc[k]);
            } else {
                out.store(j, acc);
            }
        }
    } else if (part < 3) {  // part c stores component c
        cx_t<A> z;
        z.x = z.y = A(0);
#pragma unroll
        for (int q = 0; q < PARTS; ++q) {
            z.x += buf[(q * 6 + 2 * part) * sg + p.i];
            z.y += buf[(q * 6 + 2 * part + 1) * sg + p.i];
        }
        if constexpr (MDAGM) {
            const A m = (A)a.m4;
            z.x = z.x + m * pv.x;
            z.y = z.y + m * pv.y;
            dot += (double)(pv.x * z.x);
            dot += (double)(pv.y * z.y);
        }
        out.p[part * vh + j] = z;
    }
}

// out = D in (+ m4 p) over the lattice, the groups striding over the tiles
template <int PARTS, bool MDAGM, bool MIR, typename SV, typename SL, typename In, typename A, typename Own>
__device__ __forceinline__ void phase_dslash(const LoopArgs<SV, SL> &a, const GroupPlace &p, int cb, const In &in,
                                             const VecView<SV> &out, A *comb, double &dot, Own own)
{
    if (p.grp >= a.groups) return;
    const int per = a.groups * a.sg;
    unsigned k = 0;
    for (int j0 = blockIdx.x * per + p.grp * a.sg; j0 < a.g.vh; j0 += gridDim.x * per, ++k)
        tile_dslash<PARTS, MDAGM, MIR>(a, p, j0, cb, in, out, comb + ((size_t)p.grp * 2 + (k & 1)) * 6 * p.gthreads, dot,
                                       own);
}

// 16-byte words of the flat element-wise phases
template <typename R> struct FlatWord;
template <> struct FlatWord<float> {
    using type = float4;
    static constexpr int n = 4;
    static __device__ __forceinline__ void get(const float4 &w, float v[4]) { v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w; }
    static __device__ __forceinline__ float4 make(const float v[4]) { return make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct FlatWord<double> {
    using type = double2;
    static constexpr int n = 2;
    static __device__ __forceinline__ void get(const double2 &w, double v[2]) { v[0] = w.x; v[1] = w.y; }
    static __device__ __forceinline__ double2 make(const double v[2]) { return make_double2(v[0], v[1]); }
};

// phase_residual and phase_direction handle two words of every vector per
// thread at a time, all loads first: one at a time they ran at the latency of a
// load per 16 bytes and thread.  (The shifts' phases, and k_small_loop, where a
// thread has one word or none, take one.)

// r += s ttt: |r|^2 of this thread's share
template <typename SV>
__device__ __forceinline__ double phase_residual(int vh, SV s, const VecView<SV> &r, const VecView<SV> &ttt)
{
    using F = FlatWord<SV>;
    using W = typename F::type;
    const int n = 6 * vh / F::n, step = gridDim.x * blockDim.x;
    W *rp = reinterpret_cast<W *>(r.p);
    const W *tp = reinterpret_cast<const W *>(ttt.p);
    double sum = 0.0;
    auto word = [&](const W &rw, const W &tw) {
        SV rv[F::n], tv[F::n];
        F::get(rw, rv);
        F::get(tw, tv);
#pragma unroll
        for (int e = 0; e < F::n; ++e) {
            rv[e] = rv[e] + s * tv[e];
            sum += (double)(rv[e] * rv[e]);
        }
        return F::make(rv);
    };
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + step < n; i += 2 * step) {
        const W r0 = rp[i], r1 = rp[i + step], t0 = tp[i], t1 = tp[i + step];
        rp[i] = word(r0, t0);
        rp[i + step] = word(r1, t1);
    }
    if (i < n) rp[i] = word(rp[i], tp[i]);
    return sum;
}

// x += s p, then (when `dir`; the iteration that ends a run before it leaves
// p) p = r + b p.  x is updated here, where p is read anyway, and not beside
// r: one read of p less per iteration.
template <typename SV>
__device__ __forceinline__ void phase_direction(int vh, SV s, SV b, bool dir, SV *x, const VecView<SV> &p,
                                                const VecView<SV> &r)
{
    using F = FlatWord<SV>;
    using W = typename F::type;
    const int n = 6 * vh / F::n, step = gridDim.x * blockDim.x;
    W *xp = reinterpret_cast<W *>(x), *pp = reinterpret_cast<W *>(p.p);
    const W *rp = reinterpret_cast<const W *>(r.p);
    auto word = [&](int i, const W &xw, const W &pw, const W &rw) {
        SV xv[F::n], pv[F::n], rv[F::n];
        F::get(xw, xv);
        F::get(pw, pv);
        F::get(rw, rv);
#pragma unroll
        for (int e = 0; e < F::n; ++e) {
            xv[e] = xv[e] + s * pv[e];
            pv[e] = rv[e] + b * pv[e];
        }
        xp[i] = F::make(xv);
        if (dir) pp[i] = F::make(pv);
    };
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + step < n; i += 2 * step) {
        const W x0 = xp[i], x1 = xp[i + step], p0 = pp[i], p1 = pp[i + step], r0 = rp[i], r1 = rp[i + step];
        word(i, x0, p0, r0);
        word(i + step, x1, p1, r1);
    }
    if (i < n) word(i, xp[i], pp[i], rp[i]);
}

// x_k += beta_k p_k, p_k = zeta_k r + alpha_k p_k for every active shift
// (k_ms_update's arithmetic)
template <typename SV>
__device__ __forceinline__ void phase_shifts(int vh, const SolverState &S, VecBlock *xs, VecBlock *ps,
                                             const VecView<SV> &r)
{
    using F = FlatWord<SV>;
    using W = typename F::type;
    const int n = 6 * vh / F::n, step = gridDim.x * blockDim.x;
    const int nn = S.num_now, it = S.iteration;
    const bool conv = S.converged != 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        SV rv[F::n];
        if (!conv) F::get(reinterpret_cast<const W *>(r.p)[i], rv);
        for (int k = 0; k < nn; ++k) {
            const int sd = S.shift_done_at[k];
            if (sd < it) continue;
            W *pk = static_cast<W *>(ps[k].data) + i, *xk = static_cast<W *>(xs[k].data) + i;
            SV pv[F::n], xv[F::n];
            F::get(*pk, pv);
            F::get(*xk, xv);
            const SV bk = (SV)S.beta_i[k];
#pragma unroll
            for (int e = 0; e < F::n; ++e) xv[e] = xv[e] + bk * pv[e];
            *xk = F::make(xv);
            if (!conv && sd != it) {
                const SV ak = (SV)S.alpha[k];
                const double zk = S.zeta_ip1[k];
#pragma unroll
                for (int e = 0; e < F::n; ++e) {
                    const SV tt = (SV)((double)rv[e] * zk);
                    pv[e] = tt + ak * pv[e];
                }
                *pk = F::make(pv);
            }
        }
    }
}

// the deferred form (k_ms_defer's arithmetic): r (phase_defer) and the shifts'
// scalars (defer_scalars) into the iteration's slot, p_low = z r + a p_low
__device__ __forceinline__ void defer_scalars(const SolverState &S, int slot, MsHistEntry *hs, int n)
{
    const int it = S.iteration, nn = S.num_now;
    const bool conv = S.converged != 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        MsHistEntry e;
        e.b = S.beta_i[k];
        e.a = S.alpha[k];
        e.z = S.zeta_ip1[k];
        const int sd = S.shift_done_at[k];
        e.upd = k >= nn || sd < it ? 0 : (1 | (!conv && sd != it ? 2 : 0));
        hs[(size_t)slot * n + k] = e;
    }
}

__device__ __forceinline__ void phase_defer(int vh, SolverState &S, const VecView<float> &p, const VecView<float> &r,
                                            float2 *hist, MsHistEntry *hs, int n)
{
    const int slot = S.iteration - S.ms_seg_start - 1, jl = S.j_low;
    const bool conv = S.converged != 0;
    if (blockIdx.x == 0) defer_scalars(S, slot, hs, n);
    const int n4 = 6 * vh / 4, step = gridDim.x * blockDim.x;
    float4 *h = reinterpret_cast<float4 *>(hist + (size_t)slot * 3 * vh);
    const float ak = (float)S.alpha[jl];
    const double zk = S.zeta_ip1[jl];
    using F = FlatWord<float>;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += step) {
        const float4 w = reinterpret_cast<const float4 *>(r.p)[i];
        h[i] = w;
        if (conv) continue;
        float rv[4], pv[4];
        F::get(w, rv);
        F::get(reinterpret_cast<const float4 *>(p.p)[i], pv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float tt = (float)((double)rv[e] * zk);
            pv[e] = tt + ak * pv[e];
        }
        reinterpret_cast<float4 *>(p.p)[i] = F::make(pv);
    }
}

__device__ __forceinline__ void load_state(SolverState &to, const SolverState *from)
{
    const int nw = sizeof(SolverState) / sizeof(int);
    const int *src = reinterpret_cast<const int *>(from);
    int *dst = reinterpret_cast<int *>(&to);
    for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = src[i];
}

template <typename SV, typename SL, int MODE, bool MIR, int PARTS>
__global__ void __launch_bounds__(LoopThreads<SV>::value, 1) k_solver_loop(const LoopArgs<SV, SL> a)
{
    using A = typename Acc<SV>::type;
    __shared__ LoopShared sh;
    extern __shared__ __align__(16) unsigned char dyn[];
    A *comb = reinterpret_cast<A *>(dyn);
    SolverState &S = sh.st;
    {
        load_state(sh.st, a.st);
        if (threadIdx.x == 0) sh.fail = 0;
    }
    __syncthreads();
    const int vh = a.g.vh, par = a.parity;
    const bool warp0 = threadIdx.x < 32;
    constexpr bool kMs = MODE == kLoopMs || MODE == kLoopMsDefer;
    LoopBarrier bar{a.counter, a.partials, a.polls, 0};
    const GroupPlace place = group_place<PARTS>(a);
    bool ok = true;
    for (;;) {
        double v = 0.0, tot;
        const auto own = [&](int c, int j) {
            if constexpr (std::is_same<SV, __half>::value) return cx_t<A>();
            else return a.p.p[c * vh + j];
        };
        phase_dslash<PARTS, false, MIR>(a, place, 1 - par, a.p, a.tmp, comb, v, [] (int, int) { return cx_t<A>(); });
        if (!(ok = grid_wait(sh, bar))) break;
        phase_dslash<PARTS, true, MIR>(a, place, par, a.tmp, a.ttt, comb, v, own);
        if (!(ok = grid_sum(v, tot, sh, bar))) break;
        if (warp0) FinMdagm{&S, kMs ? 1 : 0}(&tot, (int)threadIdx.x);
        __syncthreads();
        const double step = kMs ? S.beta_i[S.j_low] : S.a;
        if constexpr (std::is_same<SV, __half>::value) {
            // 16-bit records: one thread per site; x is FP32
            const VecView<float> x{static_cast<float2 *>(a.x), vh};
            const A s = (A)step;
            v = 0.0;
            for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < vh; j += gridDim.x * blockDim.x) {
                A xv[6], pv[6], rv[6], tv[6];
                ld_vec(x, j, xv);
                ld_vec(a.p, j, pv);
                ld_vec(a.r, j, rv);
                ld_vec(a.ttt, j, tv);
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    xv[i] = xv[i] + s * pv[i];
                    rv[i] = rv[i] + s * tv[i];
                }
                x.store(j, xv);
                a.r.store(j, rv);
#pragma unroll
                for (int i = 0; i < 6; ++i) v += (double)(rv[i] * rv[i]);
            }
        } else {
            v = phase_residual<SV>(vh, (SV)step, a.r, a.ttt);
        }
        if (!(ok = grid_sum(v, tot, sh, bar))) break;
        if constexpr (MODE == kLoopCg) {
            if (threadIdx.x == 0) FinCgUpdate{&S, 0, false, 1.0}(&tot);
        } else if constexpr (MODE == kLoopMx) {
            if (threadIdx.x == 0) FinMx{&S, 0, a.delta2}(&tot);
        } else {
            if (warp0) FinMsResidual{&S, 0}(&tot, (int)threadIdx.x);
        }
        __syncthreads();
        if constexpr (MODE == kLoopMs) {
            if constexpr (!std::is_same<SV, __half>::value) phase_shifts<SV>(vh, S, a.xs, a.ps, a.r);
        } else if constexpr (MODE == kLoopMsDefer) {
            if constexpr (std::is_same<SV, float>::value) {
                const int slot = S.iteration - S.ms_seg_start - 1;
                if (slot < 0 || slot >= S.ms_seg_cap) {  // uniform over the grid
                    if (threadIdx.x == 0) {
                        S.error = 3;
                        S.stop_at = 0;
                    }
                    __syncthreads();
                } else {
                    phase_defer(vh, S, a.p, a.r, a.hist, a.hist_s, a.n);
                }
            }
        } else if constexpr (std::is_same<SV, __half>::value) {
            const A b = (A)S.b;
            for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < vh && !S.skip_axpy; j += gridDim.x * blockDim.x) {
                A rv[6], pv[6];
                ld_vec(a.r, j, rv);
                ld_vec(a.p, j, pv);
#pragma unroll
                for (int i = 0; i < 6; ++i) pv[i] = rv[i] + b * pv[i];
                a.p.store(j, pv);
            }
        } else {
            phase_direction<SV>(vh, (SV)step, (SV)S.b, !S.skip_axpy, static_cast<SV *>(a.x), a.p, a.r);
        }
        if (S.stop_at != INT_MAX) break;
        if (!(ok = grid_wait(sh, bar))) break;
    }
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(a.err, kErrLoopWait);
        return;
    }
    if (blockIdx.x == 0) {
        __syncthreads();
        load_state(*a.st, &sh.st);
    }
}

// The loop of a lattice whose sites all fit the grid at once, bound by its
// barriers: three per iteration instead of four.  The direction p = r + b p is
// not stored by a phase of its own; the first half of M^dag M forms it at the
// neighbours it gathers, the second half at its own sites, storing it in the
// other of two buffers (every use has the same operands, hence the same
// bits):
//   1  tmp = D (r + b p)                          | barrier
//   2  p' = r + b p, ttt = D tmp + m4 p', p'.ttt  | barrier with sum
//   3  r += a ttt, x += a p', |r|^2 (multi-shift: r into its slot) | barrier with sum
// Twice the gathered bytes in phase 1, but no barrier and no pass for the
// direction.  us per iteration with four phases / three: 8^4 FP64 11.4 / 10.0,
// FP32 11.4 / 9.5, 12-real 13.4 / 11.9.
template <typename SV> struct SmallThreads { static constexpr int value = 512; };
template <> struct SmallThreads<double> { static constexpr int value = 256; };

template <typename SV, typename SL, int MODE>
__global__ void __launch_bounds__(SmallThreads<SV>::value, 1) k_small_loop(const LoopArgs<SV, SL> a)
{
    using F = FlatWord<SV>;
    using W = typename F::type;
    __shared__ LoopShared sh;
    extern __shared__ __align__(16) unsigned char dyn[];
    SV *comb = reinterpret_cast<SV *>(dyn);
    SolverState &S = sh.st;
    load_state(sh.st, a.st);
    if (threadIdx.x == 0) sh.fail = 0;
    __syncthreads();
    const int vh = a.g.vh, par = a.parity;
    const bool warp0 = threadIdx.x < 32;
    constexpr bool kMs = MODE == kLoopMsDefer;
    LoopBarrier bar{a.counter, a.partials, a.polls, 0};
    const GroupPlace place = group_place<8>(a);
    const int n = 6 * vh / F::n, flat0 = blockIdx.x * blockDim.x + threadIdx.x, flat_step = gridDim.x * blockDim.x;
    VecView<SV> cur = a.p, other = a.p2;
    bool ok = true, first = true;
    SV b = SV(0);
    for (;;) {
        double v = 0.0, tot;
        const SumIn<SV> in{cur, a.r, b, first};
        phase_dslash<8, false, false>(a, place, 1 - par, in, a.tmp, comb, v, [](int, int) { return cx_t<SV>(); });
        if (!(ok = grid_wait(sh, bar))) break;
        phase_dslash<8, true, false>(a, place, par, a.tmp, a.ttt, comb, v, [&](int c, int j) {
            cx_t<SV> z = in.p.p[c * vh + j];
            const cx_t<SV> q = in.r.p[c * vh + j];
            z.x = in.at(z.x, q.x);
            z.y = in.at(z.y, q.y);
            other.p[c * vh + j] = z;
            return z;
        });
        if (!(ok = grid_sum(v, tot, sh, bar))) break;
        const VecView<SV> keep = cur;
        cur = other;
        other = keep;
        first = false;
        if (warp0) FinMdagm{&S, kMs ? 1 : 0}(&tot, (int)threadIdx.x);
        __syncthreads();
        const SV s = (SV)(kMs ? S.beta_i[S.j_low] : S.a);
        const int slot = kMs ? S.iteration - S.ms_seg_start - 1 : 0;
        const bool slot_ok = !kMs || (slot >= 0 && slot < S.ms_seg_cap);
        W *h = kMs && slot_ok ? reinterpret_cast<W *>(a.hist + (size_t)slot * 3 * vh) : nullptr;
        v = 0.0;
        for (int i = flat0; i < n; i += flat_step) {
            SV rv[F::n], tv[F::n];
            F::get(reinterpret_cast<const W *>(a.r.p)[i], rv);
            F::get(reinterpret_cast<const W *>(a.ttt.p)[i], tv);
            if constexpr (!kMs) {
                SV xv[F::n], pv[F::n];
                F::get(static_cast<const W *>(a.x)[i], xv);
                F::get(reinterpret_cast<const W *>(cur.p)[i], pv);
#pragma unroll
                for (int e = 0; e < F::n; ++e) xv[e] = xv[e] + s * pv[e];
                static_cast<W *>(a.x)[i] = F::make(xv);
            }
#pragma unroll
            for (int e = 0; e < F::n; ++e) {
                rv[e] = rv[e] + s * tv[e];
                v += (double)(rv[e] * rv[e]);
            }
            const W w = F::make(rv);
            reinterpret_cast<W *>(a.r.p)[i] = w;
            if (h) h[i] = w;
        }
        if (!(ok = grid_sum(v, tot, sh, bar))) break;
        if constexpr (MODE == kLoopCg) {
            if (threadIdx.x == 0) FinCgUpdate{&S, 0, false, 1.0}(&tot);
        } else if constexpr (MODE == kLoopMx) {
            if (threadIdx.x == 0) FinMx{&S, 0, a.delta2}(&tot);
        } else {
            if (warp0) FinMsResidual{&S, 0}(&tot, (int)threadIdx.x);
        }
        __syncthreads();
        if constexpr (kMs) {
            if (!slot_ok) {  // uniform over the grid
                if (threadIdx.x == 0) {
                    S.error = 3;
                    S.stop_at = 0;
                }
                __syncthreads();
            } else if (blockIdx.x == 0) {
                defer_scalars(S, slot, a.hist_s, a.n);
            }
        }
        b = (SV)(kMs ? S.alpha[S.j_low] : S.b);
        if (S.stop_at != INT_MAX) break;
    }
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(a.err, kErrLoopWait);
        return;
    }
    // the direction as the four-phase loop leaves it, in the caller's buffer
    // (all reads of the last phases are behind the last barrier)
    const bool dir = kMs ? S.converged == 0 : S.skip_axpy == 0;
    for (int i = flat0; i < n; i += flat_step) {
        SV pv[F::n], rv[F::n];
        F::get(reinterpret_cast<const W *>(cur.p)[i], pv);
        F::get(reinterpret_cast<const W *>(a.r.p)[i], rv);
#pragma unroll
        for (int e = 0; e < F::n; ++e) pv[e] = dir ? fma_(b, pv[e], rv[e]) : pv[e];
        reinterpret_cast<W *>(a.p.p)[i] = F::make(pv);
    }
    if (blockIdx.x == 0) load_state(*a.st, &sh.st);
}

void check(cudaError_t e, const char *what)
{
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// bytes of the links of one site of a parity block
template <typename SL> constexpr size_t kLinkBytes = 72 * sizeof(cx_t<SL>) * 2;
template <> constexpr size_t kLinkBytes<__half> = 576;
template <> constexpr size_t kLinkBytes<Recon12> = (size_t)kReconChunks * 64;
template <> constexpr size_t kLinkBytes<Recon13> = (size_t)kReconChunks * 64;

// the links of both parities that the loop reads as mirrored (loop_wants_mirrored)
constexpr size_t kMirroredMin = (size_t)64 << 20, kMirroredMax = (size_t)152 << 20;

constexpr int kLoopMaxSites16 = 500000;

int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        check(cudaGetDevice(&dev), "cudaGetDevice");
        check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
        sms = std::min(sms, kLoopMaxBlocks);
    }
    return sms;
}

FastDiv fast_div(int n)
{
    int s = 0;
    while ((1LL << s) < n) ++s;
    FastDiv d;
    d.m = (unsigned)(((1ULL << (31 + s)) + n - 1) / n);
    d.s = s - 1;
    return d;
}

// one block per SM, groups of 32 sites; a lattice with fewer groups than SMs
// takes smaller ones (vh is a multiple of 128).  False when the blocks cannot
// all be resident (a process with a share of the SMs).
template <typename SV, typename SL, typename K>
bool launch_kernel(LoopArgs<SV, SL> &a, K kernel, int parts, int max_threads, const Launch &L)
{
    using A = typename Acc<SV>::type;
    const int vh = L.g->vh, sms = sm_count();
    a.sg = 32;
    a.lg_sg = 5;
    while (a.sg > 4 && vh / a.sg < sms) {
        a.sg >>= 1;
        --a.lg_sg;
    }
    const int ngroups = vh / a.sg, gthreads = parts * a.sg;
    a.groups = std::min(max_threads / gthreads, (ngroups + sms - 1) / sms);
    a.groups = std::min(a.groups, 8);  // one hardware barrier each
    const int nb = std::min(sms, (ngroups + a.groups - 1) / a.groups);
    // every block has a thread per partial sum
    const int threads = std::max(a.groups * gthreads, std::min(256, (nb + 31) / 32 * 32));
    const size_t smem = (size_t)a.groups * gthreads * 12 * sizeof(A);
    a.dx = fast_div(L.g->nxh);
    a.dy = fast_div(L.g->ny);
    a.dz = fast_div(L.g->nz);
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(max_threads * 12 * sizeof(A))),
          "solver loop: shared memory");
    check(cudaMemsetAsync(a.counter, 0, sizeof(unsigned), L.stream), "solver loop: memset");
    L.arm();
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(nb), dim3(threads),
                                                      args, smem, L.stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        (void)cudaGetLastError();  // not sticky
        return false;
    }
    check(e, "solver loop: launch");
    return true;
}

template <typename SV, typename SL, int MODE, bool MIR, int PARTS>
bool launch_form(LoopArgs<SV, SL> &a, const Launch &L)
{
    return launch_kernel<SV, SL>(a, k_solver_loop<SV, SL, MODE, MIR, PARTS>, PARTS, LoopThreads<SV>::value, L);
}

template <typename SV, typename SL, int MODE>
bool launch(const LoopRun &q, const Launch &L)
{
    const int vh = L.g->vh;
    LoopArgs<SV, SL> a;
    a.g = *L.g;
    for (int cb = 0; cb < 2; ++cb) a.links[cb] = link_view<SL>(*q.links, cb, vh);
    a.parity = q.parity;
    a.p = view<SV>(q.p, vh);
    a.tmp = view<SV>(q.tmp, vh);
    a.ttt = view<SV>(q.ttt, vh);
    a.r = view<SV>(q.r, vh);
    a.x = q.x.data;
    a.m4 = q.m4;
    a.delta2 = q.delta2;
    a.st = q.st;
    a.counter = static_cast<unsigned *>(q.slots);
    a.partials = static_cast<double *>(q.slots) + 4;
    a.err = L.err;
    a.polls = wait_limit();
    a.n = q.n;
    a.xs = q.xs;
    a.ps = q.ps;
    a.hist = static_cast<float2 *>(q.hist.data);
    a.hist_s = q.hist_s;
    if constexpr (MODE != kLoopMs && !std::is_same<SV, __half>::value) {
        if (q.p2.data && vh <= sm_count() * (SmallThreads<SV>::value / 8)) {
            a.p2 = view<SV>(q.p2, vh);
            return launch_kernel<SV, SL>(a, k_small_loop<SV, SL, MODE>, 8, SmallThreads<SV>::value, L);
        }
    }
    const bool eight = vh <= LoopThreads<SV>::eight_parts;
    if (q.links->mirrored == 1 && loop_wants_mirrored(*q.links, vh)) {
        // (only FP64 links are large enough for it on a lattice of eight parts)
        if constexpr (2 * kLinkBytes<SL> * LoopThreads<SV>::eight_parts >= kMirroredMin)
            if (eight) return launch_form<SV, SL, MODE, true, 8>(a, L);
        return launch_form<SV, SL, MODE, true, 4>(a, L);
    }
    return eight ? launch_form<SV, SL, MODE, false, 8>(a, L) : launch_form<SV, SL, MODE, false, 4>(a, L);
}

}  // namespace

size_t solver_loop_slot_bytes() { return (4 + 2 * kLoopMaxBlocks) * sizeof(double); }

// Reading each link once, in its own site's block (LinkSet::mirrored),
// touches 0.5 to 0.67 of the link bytes of an iteration, but the backward
// links are then gathers.  It pays where it lets the links stay in the 126 MB
// L2 from one iteration to the next, us per iteration with / without:
// 96 MB (12^3x24 FP64) 22.2 / 27.3; 151 MB (16^3x32 FP32) 31.9 / 37.4; 132 MB
// (12-real) 36.7 / 38.8; 48 MB (12^3x24 FP32) 15.9 / 16.2; 184 MB (20^3x40
// 16-bit) 69.3 / 63.0; 302 MB (16^3x32 FP64) 60.4 / 60.9.
bool loop_wants_mirrored(const LinkSet &ls, int vh)
{
    const size_t site = ls.recon ? kLinkBytes<Recon12> : ls.prec == Prec::Double ? kLinkBytes<double>
                                                      : ls.prec == Prec::Single ? kLinkBytes<float>
                                                                                : kLinkBytes<__half>;
    const size_t bytes = 2 * site * vh;
    return bytes >= kMirroredMin && bytes <= kMirroredMax;
}

bool solver_loop_wants_p2(Prec pv, const Launch &L)
{
    return pv == Prec::Double   ? L.g->vh <= sm_count() * (SmallThreads<double>::value / 8)
           : pv == Prec::Single ? L.g->vh <= sm_count() * (SmallThreads<float>::value / 8)
                                : false;
}

bool solver_loop_run(Prec pv, const LoopRun &q, const Launch &L)
{
    // QPHIX_B200_LOOP=0: the phases' kernels one by one (for comparison)
    const char *e = std::getenv("QPHIX_B200_LOOP");
    if (L.halo || dslash_variant_forced() || (e && e[0] == '0')) return false;
    const LinkSet &ls = *q.links;
    // On large lattices the one-thread-per-site Dslash kernels stream the
    // 16-bit links better than the loop's, and their launches no longer count.
    // us per iteration of the kernels / the loop, FP32 vectors: 24^3x48 (0.33 M
    // sites) 110.0 / 103.7, 32^3x32 (0.52 M) 163.1 / 158.4, 32^3x48 (0.79 M)
    // 231.7 / 236.1, 32^3x64 (1.05 M) 298.3 / 314.3; 16-bit vectors 111.4 /
    // 105.9, 160.0 / 155.7, 228.7 / 228.5, 295.5 / 303.5.  With the other
    // storages the loop is the faster one or equal: 32^3x64 FP64 847 / 823,
    // FP32 435 / 415, 12-real 435 / 421; 40^3x64 (2.05 M) 1618 / 1594, 835 /
    // 811, 817 / 816.
    if (ls.prec == Prec::Half && L.g->vh > kLoopMaxSites16) return false;
    // Updating every shift's two vectors is a stream of its own, which the
    // kernel's full occupancy moves faster than the loop's one block per SM, the
    // more so the more shifts there are.  us per iteration of the kernels / the
    // loop with 2, 4, 8 and 12 shifts: FP64 20^3x40 (0.16 M sites) 160 / 139,
    // 173 / 157, 204 / 190, 232 / 219; 24^3x32 (0.22 M) 204 / 191, 224 / 214,
    // 255 / 252, 285 / 289; 24^3x48 (0.33 M) 294 / 282, 319 / 311, 365 / 368,
    // 409 / 425.  FP32 24^3x48 158 / 142, 171 / 159, 199 / 186, 226 / 210;
    // 32^3x32 (0.52 M) 240 / 224, 266 / 245, 302 / 282, 335 / 317: the FP32 line
    // is below where the two would cross.
    if (q.mode == kLoopMs && L.g->vh > (pv == Prec::Double ? 200000 : 400000)) return false;
    if (pv == Prec::Double && ls.prec == Prec::Double) {
        if (q.mode == kLoopCg) return launch<double, double, kLoopCg>(q, L);
        if (q.mode == kLoopMs) return launch<double, double, kLoopMs>(q, L);
    } else if (pv == Prec::Single && ls.recon == 1) {
        if (q.mode == kLoopMx) return launch<float, Recon12, kLoopMx>(q, L);
        if (q.mode == kLoopMsDefer) return launch<float, Recon12, kLoopMsDefer>(q, L);
    } else if (pv == Prec::Single && ls.recon == 2) {
        if (q.mode == kLoopMx) return launch<float, Recon13, kLoopMx>(q, L);
        if (q.mode == kLoopMsDefer) return launch<float, Recon13, kLoopMsDefer>(q, L);
    } else if (pv == Prec::Single && ls.prec == Prec::Single) {
        if (q.mode == kLoopCg) return launch<float, float, kLoopCg>(q, L);
        if (q.mode == kLoopMx) return launch<float, float, kLoopMx>(q, L);
        if (q.mode == kLoopMs) return launch<float, float, kLoopMs>(q, L);
        return launch<float, float, kLoopMsDefer>(q, L);
    } else if (pv == Prec::Single && ls.prec == Prec::Half) {
        if (q.mode == kLoopMx) return launch<float, __half, kLoopMx>(q, L);
        if (q.mode == kLoopMsDefer) return launch<float, __half, kLoopMsDefer>(q, L);
    } else if (pv == Prec::Half && ls.prec == Prec::Half) {
        if (q.mode == kLoopMx) return launch<__half, __half, kLoopMx>(q, L);
    }
    return false;
}

// ------------------------------------------------------------ mirrored links --
namespace {

// *flag = 1 when a backward matrix differs in any bit from the forward one of
// its own site (one thread per site of a parity block, direction and hop)
template <typename R>
__global__ void __launch_bounds__(kBlock) k_links_mirrored(const cx_t<R> *own, const cx_t<R> *other, Geom g, int cb,
                                                           int *flag)
{
    constexpr int K = 16 / sizeof(cx_t<R>);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = i % g.vh, q = i / g.vh;  // q = 2 d + h
    if (q >= 8) return;
    const int d = q >> 1, h = q & 1;
    const int b = neighbor(g, decode(g, cb, j), 8 * h + 2 * d);
    bool same = true;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const cx_t<R> x = own[link_cx_index(K, d, 18 * h + 9 + e, j, g.vh)];
        const cx_t<R> y = other[link_cx_index(K, d, 18 * h + e, b, g.vh)];
        if constexpr (sizeof(R) == 8)
            same = same && __double_as_longlong(x.x) == __double_as_longlong(y.x) &&
                   __double_as_longlong(x.y) == __double_as_longlong(y.y);
        else
            same = same && __float_as_int(x.x) == __float_as_int(y.x) && __float_as_int(x.y) == __float_as_int(y.y);
    }
    if (!same) *flag = 1;
}

}  // namespace

bool links_mirrored(const LinkSet &ls, const Launch &L, int *d_flag)
{
    const Geom &g = *L.g;
    check(cudaMemsetAsync(d_flag, 0, sizeof(int), L.stream), "links_mirrored");
    const unsigned grid = (unsigned)(((long long)g.vh * 8 + kBlock - 1) / kBlock);
    for (int cb = 0; cb < 2; ++cb) {
        if (ls.prec == Prec::Double)
            k_links_mirrored<double><<<grid, kBlock, 0, L.stream>>>(static_cast<const double2 *>(ls.blk[cb]),
                                                                    static_cast<const double2 *>(ls.blk[1 - cb]), g,
                                                                    cb, d_flag);
        else
            k_links_mirrored<float><<<grid, kBlock, 0, L.stream>>>(static_cast<const float2 *>(ls.blk[cb]),
                                                                   static_cast<const float2 *>(ls.blk[1 - cb]), g, cb,
                                                                   d_flag);
    }
    int f = 1;
    check(cudaMemcpyAsync(&f, d_flag, sizeof(int), cudaMemcpyDeviceToHost, L.stream), "links_mirrored");
    check(cudaStreamSynchronize(L.stream), "links_mirrored");
    return f == 0;
}

}  // namespace qb
