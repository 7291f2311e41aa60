// Symanzik one-loop gauge force: QPHIX_{F3,D3}_symanzik_1loop_gauge_force
// and the gauge-field / momentum objects it works on
// (QPHIX_*_create_G_from_raw, _create_F_from_raw, extract, destroy).
//
// Reference: gauge_force_imp.cpp:136-199 passes the gauge field, the
// momenta, coeffs->plaquette / rectangle / parallelogram and eps to per-site
// bodies (gforce_imp_body, update_mg_body) that live in the unvendored
// milc-qphix-codegen; the host layout code (create_G_from_raw,
// create_F_from_raw, qphix_f3.cpp:160-470) fixes the raw formats: 72 reals
// per site, the four forward links (or the four momenta, full 3x3
// anti-Hermitian matrices) of the site, even sites first.  The arithmetic
// is the one-loop Symanzik force as MILC defines it (imp_gauge_force; eps
// carries beta/3):
//
//   A_mu(x) <- A_mu(x) + eps TA( U_mu(x) sum_loops c_loop S_loop(x, mu) ),
//   TA(M) = (M - M^dag)/2 - tr(M - M^dag)/6,
//
// over the 6 plaquettes, 18 1x2 rectangles and 24 six-link parallelograms
// through each link, S_loop the product of the loop's other links from
// x + mu back to x; it is the derivative of S = -1/3 sum c Re tr U_loop
// (restated independently in oracle/gauge_force_oracle.py, which the tests
// also check against finite differences of that action).  As in the
// reference, one call updates the links of one checkerboard: the objects'
// parity, EVENODD meaning EVEN (qphix_f3.cpp:178-179, 347-348).
//
// One thread owns one link (site of the parity, direction mu).  The 48
// staples are not walked one by one: with A = the step (nu, s) from x + mu,
// C = the step (-rho, -r) into x and W the steps between, the plaquettes,
// the rectangles that end with a rho step and all parallelograms are
//   sum_{rho r} ( sum_{nu s} A W ) C,
// so the products that end in the same step are summed before the last
// multiplication (gf_program): 134 products of 3x3 matrices and 182 link
// loads per link instead of 181 and 229.  The links come from L1/L2 (every
// link is read by ~150 threads).  FP64 for D3, FP32 for F3.
#include <cstring>
#include <type_traits>

#include "context.h"
#include "device_common.cuh"

namespace qb {

namespace {

// One entry of the evaluation of a link's staple sum: a link U (its adjoint
// when the path passes it backwards) and what is done with it.
//   kStart  M = U
//   kMul    M = M U
//   kMix    M = c1 M + c0 U
//   kFold   S = S + X U; X = 0
// and, when `add` is 1 + t, then X = X + c_t M (c_0 plaquette, c_1
// rectangle, c_2 parallelogram coefficient), when it is 4, X = X + M.  The
// link's site is x plus a displacement of -2..2 along each axis, kept in the
// entry, so that a thread only adds up the block indices of its own wrapped
// coordinates.
enum GfOp : unsigned { kStart = 0, kMul = 1, kMix = 2, kFold = 3 };
// bits: 0-1 op, 2-3 axis of U, 4 adjoint, 5-7 add, 8 parity of the
// displacement, 9 + 3a .. 11 + 3a displacement along a plus 2
struct GfEntry {
    static constexpr unsigned make(GfOp op, int axis, bool adj, int add, const int disp[4])
    {
        unsigned e = (unsigned)op | (unsigned)axis << 2 | (unsigned)adj << 4 | (unsigned)add << 5;
        e |= (unsigned)((disp[0] + disp[1] + disp[2] + disp[3]) & 1) << 8;
        for (int a = 0; a < 4; ++a) e |= (unsigned)(disp[a] + 2) << (9 + 3 * a);
        return e;
    }
};
constexpr int kGfProgram = 184;  // entries of the longest program
// by which coefficients are non-zero (bit t: c_t) and direction
struct GfPrograms {
    unsigned entry[8][4][kGfProgram];
    int length[8][4];
};

// Appends the program of direction mu to p; terms with a zero coefficient are
// left out.  (Evaluated by the compiler; a program longer than kGfProgram
// does not compile.)
constexpr void gf_program(GfPrograms &p, int mask, int mu)
{
    const bool c0 = mask & 1, c1 = mask & 2, c2 = mask & 4;
    int pos[4] = {0, 0, 0, 0};
    // one step of a path from the current position (kStart and kMix: from x + mu)
    auto add = [&](GfOp op, int axis, int sign, int coef = 0) {
        if (op == kStart || op == kMix)
            for (int d = 0; d < 4; ++d) pos[d] = d == mu;
        if (sign < 0) --pos[axis];
        p.entry[mask][mu][p.length[mask][mu]++] = GfEntry::make(op, axis, sign < 0, coef, pos);
        if (sign > 0) ++pos[axis];
    };
    if (!mask) return;
    for (int rho = 0; rho < 4; ++rho) {
        if (rho == mu) continue;
        for (int r = 1; r >= -1; r -= 2) {
            if (c2)
                for (int nu = 0; nu < 4; ++nu) {
                    if (nu == mu || nu == rho) continue;
                    for (int s = 1; s >= -1; s -= 2) {  // parallelogram [nu s, rho r, -mu, -nu s, -rho r]
                        add(kStart, nu, s);
                        add(kMul, rho, r);
                        add(kMul, mu, -1);
                        add(kMul, nu, -s, 3);
                    }
                }
            if (c1) {
                // rectangle [rho r, rho r, -mu, -rho r, -rho r]
                add(kStart, rho, r);
                add(kMul, rho, r);
                add(kMul, mu, -1);
                add(kMul, rho, -r, 2);
                // rectangle [mu, rho r, -mu, -mu, -rho r] and the plaquette
                // [rho r, -mu, -rho r], whose last two steps are the same
                add(kStart, mu, 1);
                add(kMul, rho, r);
                add(kMul, mu, -1);
                if (c0) {
                    add(kMix, rho, r);
                    add(kMul, mu, -1, 4);  // (the weights are in M)
                } else {
                    add(kMul, mu, -1, 2);
                }
            } else if (c0) {
                add(kStart, rho, r);
                add(kMul, mu, -1, 1);
            }
            add(kFold, rho, -r);
        }
    }
    if (c1) {  // rectangles [nu s, -mu, -mu, -nu s, mu]
        for (int nu = 0; nu < 4; ++nu) {
            if (nu == mu) continue;
            for (int s = 1; s >= -1; s -= 2) {
                add(kStart, nu, s);
                add(kMul, mu, -1);
                add(kMul, mu, -1);
                add(kMul, nu, -s, 2);
            }
        }
        add(kFold, mu, 1);
    }
}

constexpr GfPrograms gf_programs()
{
    GfPrograms p{};
    for (int mask = 0; mask < 8; ++mask)
        for (int mu = 0; mu < 4; ++mu) gf_program(p, mask, mu);
    return p;
}

// Part of the module's image, so that it is there whenever the kernel is.  (A
// copy to a symbol at the first call runs on the default stream, which the
// library's non-blocking stream does not wait for: a kernel that reads the
// length before it lands adds no staple at all.)
constexpr GfPrograms kGfPrograms = gf_programs();
__constant__ GfPrograms c_gf = kGfPrograms;

// One row of a product of 3x3 complex matrices (row-major reals u[6 r + 2 c] +
// i u[6 r + 2 c + 1]): t = (a_0, a_1, a_2) b or b^dag, as chains of fused
// multiply-adds: two per pair of real products, where re += ar * br - ai * bi
// compiles to three instructions.
template <bool ADJ, typename R>
__device__ __forceinline__ void mm_row(const R a[6], const R b[18], R t[6])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        R re = R(0), im = R(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const R ar = a[2 * j], ai = a[2 * j + 1];
            const R br = ADJ ? b[6 * k + 2 * j] : b[6 * j + 2 * k];
            const R bi = ADJ ? b[6 * k + 2 * j + 1] : b[6 * j + 2 * k + 1];  // (conjugated below)
            re = j == 0 ? ar * br : fma_(ar, br, re);
            im = j == 0 ? ai * br : fma_(ai, br, im);
            re = ADJ ? fma_(ai, bi, re) : fma_(-ai, bi, re);
            im = ADJ ? fma_(-ar, bi, im) : fma_(ar, bi, im);
        }
        t[2 * k] = re;
        t[2 * k + 1] = im;
    }
}

// a = a b or a b^dag (a row of the product needs only that row of a)
template <bool ADJ, typename R>
__device__ __forceinline__ void mm_inplace(R a[18], const R b[18])
{
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        R t[6];
        mm_row<ADJ>(a + 6 * r, b, t);
#pragma unroll
        for (int i = 0; i < 6; ++i) a[6 * r + i] = t[i];
    }
}

template <typename R>
struct GaugeView {
    const cx_t<R> *b[2];
    Geom g;
};

// One thread per link (direction-major: a warp's threads share the program
// and gather consecutive sites).  What bounds it at 12 warps per SM is the
// instruction issue and the latency of the gathers, so
//  * the next entry's link is loaded before the product with the current one
//    (two links, M and X in registers; the loop is unrolled by two so that no
//    link is copied);
//  * the block indices of the wrapped coordinates x - 2 .. x + 2 along each
//    axis are computed once into shared memory;
//  * adjoints are taken in the product, by a branch the whole warp takes;
//  * the staple sum S, used seven times per link, is in shared memory, and in
//    FP64 so is X, used 37 times (24^3x48, one checkerboard: 3.48 ms against
//    3.76 ms with X in registers at three blocks per SM both, 4.80 ms at four
//    blocks with spills; FP32 2.17 ms with X in registers at five blocks,
//    2.25 ms with X in shared memory at six).
constexpr int kGfThreads = 128;
template <typename R> constexpr bool kGfSharedX = std::is_same<R, double>::value;
template <typename R> struct GfMinBlocks { static constexpr int value = 5; };
template <> struct GfMinBlocks<double> { static constexpr int value = 3; };

template <typename R>
struct GfShared {
    R acc[18][kGfThreads];  // S
    R x[kGfSharedX<R> ? 18 : 1][kGfThreads];  // X
    int idx[4][5][kGfThreads];  // by axis and displacement + 2
};

template <typename R>
__device__ __forceinline__ void gf_load(const GaugeView<R> &U, const GfShared<R> &sh, int cb, unsigned e, R u[18])
{
    const int tid = threadIdx.x, vh = U.g.vh;
    const int j = sh.idx[0][(e >> 9) & 7][tid] + sh.idx[1][(e >> 12) & 7][tid] + sh.idx[2][(e >> 15) & 7][tid] +
                  sh.idx[3][(e >> 18) & 7][tid];
    const cx_t<R> *p = U.b[(cb ^ (e >> 8)) & 1] + (size_t)((e >> 2) & 3) * 9 * vh + j;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const cx_t<R> z = __ldg(p + (size_t)k * vh);
        u[2 * k] = z.x;
        u[2 * k + 1] = z.y;
    }
}

template <bool ADJ, typename R>
__device__ __forceinline__ void gf_apply(GfShared<R> &sh, unsigned op, const R u[18], R M[18], R X[18], R c0, R c1)
{
    if (op == kMul) {
        mm_inplace<ADJ>(M, u);
    } else if (op == kFold) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            R a[6], t[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                if constexpr (kGfSharedX<R>) {
                    a[k] = sh.x[6 * r + k][threadIdx.x];
                    sh.x[6 * r + k][threadIdx.x] = R(0);
                } else {
                    a[k] = X[6 * r + k];
                    X[6 * r + k] = R(0);
                }
            }
            mm_row<ADJ>(a, u, t);
#pragma unroll
            for (int k = 0; k < 6; ++k) sh.acc[6 * r + k][threadIdx.x] += t[k];
        }
    } else {
        const bool mix = op == kMix;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const R x = ADJ ? u[6 * k + 2 * r] : u[6 * r + 2 * k];
                const R y = ADJ ? -u[6 * k + 2 * r + 1] : u[6 * r + 2 * k + 1];
                M[6 * r + 2 * k] = mix ? fma_(c1, M[6 * r + 2 * k], c0 * x) : x;
                M[6 * r + 2 * k + 1] = mix ? fma_(c1, M[6 * r + 2 * k + 1], c0 * y) : y;
            }
    }
}

template <typename R>
__global__ void __launch_bounds__(kGfThreads, GfMinBlocks<R>::value)
k_gauge_force(GaugeView<R> U, cx_t<R> *mom, int cb, R eps, R c0, R c1, R c2, int mask)
{
    static_assert(sizeof(GfShared<R>) <= 48 * 1024, "static shared memory");
    __shared__ GfShared<R> sh;
    const Geom &g = U.g;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x, tid = threadIdx.x;
    if (idx >= 4 * g.vh) return;
    const int mu = idx / g.vh, j = idx - mu * g.vh;
    {
        const SiteCoords s = decode(g, cb, j);
        const int x = 2 * s.xh + s.xodd;
#pragma unroll
        for (int o = -2; o <= 2; ++o) {  // (every extent is at least 4)
            sh.idx[0][o + 2][tid] = wrap(x + o, g.nx) >> 1;
            sh.idx[1][o + 2][tid] = wrap(s.y + o, g.ny) * g.sy;
            sh.idx[2][o + 2][tid] = wrap(s.z + o, g.nz) * g.sz;
            sh.idx[3][o + 2][tid] = wrap(s.t + o, g.nt) * g.st;
        }
    }
    R M[18], X[18], ua[18], ub[18];
#pragma unroll
    for (int i = 0; i < 18; ++i) {
        M[i] = R(0);
        sh.acc[i][tid] = R(0);
        if constexpr (kGfSharedX<R>) sh.x[i][tid] = R(0);
        else X[i] = R(0);
    }
    const unsigned *prog = c_gf.entry[mask][mu];
    const int n = c_gf.length[mask][mu];
    auto apply = [&](unsigned e, const R u[18]) {
        if (e & 16u) gf_apply<true>(sh, e & 3u, u, M, X, c0, c1);
        else gf_apply<false>(sh, e & 3u, u, M, X, c0, c1);
        const unsigned add = (e >> 5) & 7u;
        if (add) {
            const R c = add == 1 ? c0 : add == 2 ? c1 : add == 3 ? c2 : R(1);
#pragma unroll
            for (int k = 0; k < 18; ++k) {
                if constexpr (kGfSharedX<R>) sh.x[k][tid] = fma_(c, M[k], sh.x[k][tid]);
                else X[k] = fma_(c, M[k], X[k]);
            }
        }
    };
    if (n) gf_load(U, sh, cb, prog[0], ua);
#pragma unroll 1
    for (int i = 0; i < n; i += 2) {
        if (i + 1 < n) gf_load(U, sh, cb, prog[i + 1], ub);
        apply(prog[i], ua);
        if (i + 1 < n) {
            if (i + 2 < n) gf_load(U, sh, cb, prog[i + 2], ua);
            apply(prog[i + 1], ub);
        }
    }
#pragma unroll
    for (int i = 0; i < 18; ++i) ua[i] = sh.acc[i][tid];
    {
        const cx_t<R> *p = U.b[cb] + (size_t)mu * 9 * g.vh + j;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const cx_t<R> z = __ldg(p + (size_t)k * g.vh);
            M[2 * k] = z.x;
            M[2 * k + 1] = z.y;
        }
    }
    mm_inplace<false>(M, ua);  // W = U S
    // TA(W) = (W - W^dag)/2 - tr(W - W^dag)/6
    const R tr = (M[1] + M[9] + M[17]) * (R(1) / R(3));  // imaginary part of tr(W - W^dag)/2 / 3
    cx_t<R> *m = mom + (size_t)mu * 9 * g.vh + j;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            R fr = R(0.5) * (M[6 * r + 2 * q] - M[6 * q + 2 * r]);
            R fi = R(0.5) * (M[6 * r + 2 * q + 1] + M[6 * q + 2 * r + 1]);
            if (r == q) fi -= tr;
            cx_t<R> z = m[(size_t)(3 * r + q) * g.vh];
            z.x += eps * fr;
            z.y += eps * fi;
            m[(size_t)(3 * r + q) * g.vh] = z;
        }
}

// raw (72 reals per site, site cb*vh + j) <-> blocks [dir][9][vh] of the
// parities in mask (bit cb)
template <typename D, typename RAW>
__global__ void k_gf_from_raw(D *b0, D *b1, const RAW *raw, int vh, int mask)
{
    const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (idx >= (size_t)2 * vh * 36) return;
    const int e = idx % 9, d = (idx / 9) % 4;
    const size_t s = idx / 36;
    const int cb = s >= (size_t)vh;
    if (!((mask >> cb) & 1)) return;
    const int j = (int)(s - (size_t)cb * vh);
    D z;
    z.x = raw[2 * idx];
    z.y = raw[2 * idx + 1];
    (cb ? b1 : b0)[((size_t)d * 9 + e) * vh + j] = z;
}

template <typename S, typename RAW>
__global__ void k_gf_to_raw(RAW *raw, const S *b0, const S *b1, int vh, int mask)
{
    const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (idx >= (size_t)2 * vh * 36) return;
    const int e = idx % 9, d = (idx / 9) % 4;
    const size_t s = idx / 36;
    const int cb = s >= (size_t)vh;
    if (!((mask >> cb) & 1)) return;
    const int j = (int)(s - (size_t)cb * vh);
    const S z = (cb ? b1 : b0)[((size_t)d * 9 + e) * vh + j];
    raw[2 * idx] = (RAW)z.x;
    raw[2 * idx + 1] = (RAW)z.y;
}

template <typename R> struct GfApi;
template <> struct GfApi<float> {
    using G = QPHIX_F3_GaugeField;
    using F = QPHIX_F3_Force;
};
template <> struct GfApi<double> {
    using G = QPHIX_D3_GaugeField;
    using F = QPHIX_D3_Force;
};

int parity_mask(QPHIX_evenodd_t eo) { return ((eo & QPHIX_EVEN) ? 1 : 0) | ((eo & QPHIX_ODD) ? 2 : 0); }

template <typename F>
QPHIX_status_t gf_guarded(F f)
{
    try {
        f();
        ctx().last_error.clear();
        return QPHIX_SUCCESS;
    } catch (const Error &e) {
        ctx().last_error = e.what();
        return e.status;
    } catch (const std::exception &e) {
        ctx().last_error = e.what();
        return QPHIX_FAIL;
    }
}

void require(bool ok, const char *msg)
{
    if (!ok) throw Error(msg);
}

// both parity blocks of a field, raw -> device, parities of `mask`
template <typename R>
void upload_blocks(void *blk[2], const R *raw, int mask)
{
    Context &c = ctx();
    const int vh = c.g.vh;
    const size_t bytes = (size_t)36 * vh * sizeof(cx_t<R>);
    for (int cb = 0; cb < 2; ++cb) {
        blk[cb] = dev_alloc(bytes);
        QB_CUDA(cudaMemsetAsync(blk[cb], 0, bytes, c.stream));
    }
    const size_t nraw = (size_t)2 * vh * 72;
    R *stage = static_cast<R *>(dev_alloc(nraw * sizeof(R)));
    QB_CUDA(cudaMemsetAsync(stage, 0, nraw * sizeof(R), c.stream));
    if (mask & 1) h2d_copy(stage, raw, nraw / 2 * sizeof(R));
    if (mask & 2) h2d_copy(stage + nraw / 2, raw + nraw / 2, nraw / 2 * sizeof(R));
    const int grid = (int)(((size_t)2 * vh * 36 + kBlock - 1) / kBlock);
    k_gf_from_raw<cx_t<R>, R><<<grid, kBlock, 0, c.stream>>>(static_cast<cx_t<R> *>(blk[0]),
                                                             static_cast<cx_t<R> *>(blk[1]), stage, vh, mask);
    dev_free(stage);
    sync_check();
    QB_CUDA(cudaGetLastError());
}

template <typename R>
void download_blocks(R *raw, void *const blk[2], int mask)
{
    Context &c = ctx();
    const int vh = c.g.vh;
    const size_t nraw = (size_t)2 * vh * 72;
    R *stage = static_cast<R *>(dev_alloc(nraw * sizeof(R)));
    const int grid = (int)(((size_t)2 * vh * 36 + kBlock - 1) / kBlock);
    k_gf_to_raw<cx_t<R>, R><<<grid, kBlock, 0, c.stream>>>(stage, static_cast<const cx_t<R> *>(blk[0]),
                                                           static_cast<const cx_t<R> *>(blk[1]), vh, mask);
    if (mask & 1) d2h_copy(raw, stage, nraw / 2 * sizeof(R));
    if (mask & 2) d2h_copy(raw + nraw / 2, stage + nraw / 2, nraw / 2 * sizeof(R));
    dev_free(stage);
    sync_check();
    QB_CUDA(cudaGetLastError());
}

template <typename H>
void free_blocks(H *h)
{
    for (auto &b : h->blk) {
        dev_free(b);
        b = nullptr;
    }
}

void check_evenodd(QPHIX_evenodd_t eo, const char *who)
{
    if (eo != QPHIX_EVEN && eo != QPHIX_ODD && eo != QPHIX_EVENODD) throw Error(std::string(who) + ": bad evenodd");
}

void check_single_rank(const char *who)
{
    const Context &c = ctx();
    if (c.halo.on && c.halo.nranks > 1) throw Error(std::string(who) + ": not available with several ranks");
}

template <typename R>
typename GfApi<R>::G *create_G(R *raw, QPHIX_evenodd_t evenodd)
{
    using G = typename GfApi<R>::G;
    G *h = nullptr;
    const QPHIX_status_t st = gf_guarded([&] {
        require(ctx().initialized, "create_G_from_raw: QPhiX library used before QPHIX_init");
        require(raw != nullptr, "create_G_from_raw: NULL source");
        check_evenodd(evenodd, "create_G_from_raw");
        check_single_rank("create_G_from_raw");
        h = new G();
        h->parity = evenodd == QPHIX_EVENODD ? QPHIX_EVEN : evenodd;
        h->compress12 = 0;
        // the staples reach links of both parities: the reference reads the
        // whole raw field whatever evenodd says (qphix_f3.cpp:184)
        upload_blocks<R>(h->blk, raw, 3);
        h->geo = h->blk[0];
    });
    if (st != QPHIX_SUCCESS && h) {
        free_blocks(h);
        delete h;
        h = nullptr;
    }
    return h;
}

template <typename R>
void extract_G(R *dest, typename GfApi<R>::G *h, QPHIX_evenodd_t evenodd)
{
    gf_guarded([&] {
        require(ctx().initialized, "extract_G_to_raw: QPhiX library used before QPHIX_init");
        require(dest && h, "extract_G_to_raw: NULL argument");
        check_evenodd(evenodd, "extract_G_to_raw");
        download_blocks<R>(dest, h->blk, parity_mask(evenodd));
    });
}

template <typename R>
typename GfApi<R>::F *create_F(R *raw, QPHIX_evenodd_t evenodd)
{
    using F = typename GfApi<R>::F;
    F *h = nullptr;
    const QPHIX_status_t st = gf_guarded([&] {
        require(ctx().initialized, "create_F_from_raw: QPhiX library used before QPHIX_init");
        require(raw != nullptr, "create_F_from_raw: NULL source");
        check_evenodd(evenodd, "create_F_from_raw");
        check_single_rank("create_F_from_raw");
        h = new F();
        h->parity = evenodd == QPHIX_EVENODD ? QPHIX_EVEN : evenodd;
        upload_blocks<R>(h->blk, raw, parity_mask(evenodd));
        h->heo = h->blk[0];
        h->htmp = h->blk[1];
    });
    if (st != QPHIX_SUCCESS && h) {
        free_blocks(h);
        delete h;
        h = nullptr;
    }
    return h;
}

template <typename R>
void extract_F(R *dest, typename GfApi<R>::F *h, QPHIX_evenodd_t evenodd)
{
    gf_guarded([&] {
        require(ctx().initialized, "extract_F_to_raw: QPhiX library used before QPHIX_init");
        require(dest && h, "extract_F_to_raw: NULL argument");
        check_evenodd(evenodd, "extract_F_to_raw");
        download_blocks<R>(dest, h->blk, parity_mask(evenodd));
    });
}

template <typename H>
void destroy(H *h)
{
    if (!h) return;
    gf_guarded([&] {
        free_blocks(h);
        if (ctx().initialized) sync_check();
    });
    delete h;
}

// flops of one link's force, loop by loop: 2 (plaquette) or 4 (six-link
// loops) 3x3 complex products per staple (198 flops each), its weighted sum
// (36), U times the sum (198), TA and the update (54)
double flops_per_link(const QPHIX_gauge_coeffs_t &co)
{
    double f = 198 + 54;
    if (co.plaquette != 0.0) f += 6 * (198.0 * 2 + 36);
    if (co.rectangle != 0.0) f += 18 * (198.0 * 4 + 36);
    if (co.parallelogram != 0.0) f += 24 * (198.0 * 4 + 36);
    return f;
}

template <typename R>
void gauge_force(QPHIX_info_t *info, typename GfApi<R>::G *G, typename GfApi<R>::F *F,
                 QPHIX_gauge_coeffs_t *coeffs, R eps)
{
    Context &c = ctx();
    QPHIX_status_t s = gf_guarded([&] {
        require(c.initialized, "symanzik_1loop_gauge_force: QPhiX library used before QPHIX_init");
        require(info && G && F && coeffs, "symanzik_1loop_gauge_force: NULL argument");
        // gauge_force_imp.cpp:142
        require(F->parity == G->parity, "symanzik_1loop_gauge_force: force and gauge field parities differ");
        check_single_rank("symanzik_1loop_gauge_force");
        info->final_sec = wall_seconds();
        const int cb = G->parity == QPHIX_EVEN ? 0 : 1;
        GaugeView<R> U;
        U.b[0] = static_cast<const cx_t<R> *>(G->blk[0]);
        U.b[1] = static_cast<const cx_t<R> *>(G->blk[1]);
        U.g = c.g;
        QB_CUDA(cudaEventRecord(c.ev_solve[0], c.stream));
        const int grid = (4 * c.g.vh + kGfThreads - 1) / kGfThreads;
        const R co[3] = {(R)coeffs->plaquette, (R)coeffs->rectangle, (R)coeffs->parallelogram};
        const int mask = (co[0] != R(0) ? 1 : 0) | (co[1] != R(0) ? 2 : 0) | (co[2] != R(0) ? 4 : 0);
        k_gauge_force<R><<<grid, kGfThreads, 0, c.stream>>>(U, static_cast<cx_t<R> *>(F->blk[cb]), cb, eps, co[0],
                                                            co[1], co[2], mask);
        QB_CUDA(cudaGetLastError());
        QB_CUDA(cudaEventRecord(c.ev_solve[1], c.stream));
        sync_check();
        float ms = 0.f;
        QB_CUDA(cudaEventElapsedTime(&ms, c.ev_solve[0], c.ev_solve[1]));
        c.stats = Stats{};
        c.stats.solve_ms = ms;
        info->final_sec = wall_seconds() - info->final_sec;
        info->final_flop = flops_per_link(*coeffs) * 4.0 * c.g.vh;
        info->status = QPHIX_SUCCESS;
    });
    if (s != QPHIX_SUCCESS && info) info->status = s;
}

}  // namespace
}  // namespace qb

using namespace qb;

#pragma GCC visibility push(default)
extern "C" {

QPHIX_F3_GaugeField *QPHIX_F3_create_G_from_raw(QPHIX_F_Real *raw, QPHIX_evenodd_t eo) { return create_G<float>(raw, eo); }
void QPHIX_F3_extract_G_to_raw(QPHIX_F_Real *dest, QPHIX_F3_GaugeField *G, QPHIX_evenodd_t eo) { extract_G<float>(dest, G, eo); }
void QPHIX_F3_destroy_G(QPHIX_F3_GaugeField *G) { destroy(G); }
QPHIX_F3_Force *QPHIX_F3_create_F_from_raw(QPHIX_F_Real *raw, QPHIX_evenodd_t eo) { return create_F<float>(raw, eo); }
void QPHIX_F3_extract_F_to_raw(QPHIX_F_Real *dest, QPHIX_F3_Force *F, QPHIX_evenodd_t eo) { extract_F<float>(dest, F, eo); }
void QPHIX_F3_destroy_F(QPHIX_F3_Force *F) { destroy(F); }
void QPHIX_F3_symanzik_1loop_gauge_force(QPHIX_info_t *info, QPHIX_F3_GaugeField *G, QPHIX_F3_Force *F,
                                         QPHIX_gauge_coeffs_t *coeffs, QPHIX_F_Real eps)
{
    gauge_force<float>(info, G, F, coeffs, eps);
}

QPHIX_D3_GaugeField *QPHIX_D3_create_G_from_raw(QPHIX_D_Real *raw, QPHIX_evenodd_t eo) { return create_G<double>(raw, eo); }
void QPHIX_D3_extract_G_to_raw(QPHIX_D_Real *dest, QPHIX_D3_GaugeField *G, QPHIX_evenodd_t eo) { extract_G<double>(dest, G, eo); }
void QPHIX_D3_destroy_G(QPHIX_D3_GaugeField *G) { destroy(G); }
QPHIX_D3_Force *QPHIX_D3_create_F_from_raw(QPHIX_D_Real *raw, QPHIX_evenodd_t eo) { return create_F<double>(raw, eo); }
void QPHIX_D3_extract_F_to_raw(QPHIX_D_Real *dest, QPHIX_D3_Force *F, QPHIX_evenodd_t eo) { extract_F<double>(dest, F, eo); }
void QPHIX_D3_destroy_F(QPHIX_D3_Force *F) { destroy(F); }
void QPHIX_D3_symanzik_1loop_gauge_force(QPHIX_info_t *info, QPHIX_D3_GaugeField *G, QPHIX_D3_Force *F,
                                         QPHIX_gauge_coeffs_t *coeffs, QPHIX_D_Real eps)
{
    gauge_force<double>(info, G, F, coeffs, eps);
}

}  // extern "C"
#pragma GCC visibility pop
