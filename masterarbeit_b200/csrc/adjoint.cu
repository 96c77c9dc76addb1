// adjoint.cu -- vector-Jacobian product of N APE_all steps followed by the clover charge.
//
// Forward map (the reference's qtop flow, LGT_Code/main_qtop/qtop.c:76-91):
//   U_{k+1} = Proj(U_k + alpha S[U_k])   (smearing_APE_all, LGT_Code/modules/obs/smearing.c:74-105)
//   Q = sum_x q(x) / (32 pi^2)           (topologicalCharge, LGT_Code/modules/obs/topologicalcharge.c:164-199)
// The reference has no derivative code; this file is new.
//
// Conventions.  A link is a quaternion in R^4 with the inner product <a, b> = (1/2) Re tr(a b^dag),
// the 4-vector dot product.  For a product P = a b: dP/da contracts as  p b^dag,  dP/db as  a^dag p.
// G_k denotes dQ/dU_k in that sense.  The output for a link U of U_0 is the su(2) gradient under
// U -> exp(eps X) U with X = i x.sigma, i.e. g = vec(G_0 U^dag) (three coefficients).
//
// Passes.
//  1. Forward with sqrt(N) checkpointing: U_0 and every c-th level are kept (c = ckpt or ceil(sqrt N)).
//  2. G_N = dQ/dU_N: the charge kernel leaves F-bar = dQ/dF per site and plane; the gradient with
//     respect to every 1-, 2- and 3-link line is gathered from the loops it is an edge of
//     (k_line_gradient), and a link's from the lines it is part of (k_line_chain).
//  3. Per segment, recompute its levels from the checkpoint; per level, backwards:
//     v-bar = (G_{k+1} - u' <u', G_{k+1}>) / |v|, the Jacobian of u' = v/|v| (k_ape_vbar), then
//     G_k = v-bar + alpha * (the 18 staple terms in which a link appears) (k_ape_gather).
#include <algorithm>
#include <cmath>
#include <vector>

#include "ape.cuh"
#include "internal.cuh"

using namespace su2g;

namespace {

// ----------------------------------------------------------- dQ / dU_N ---

// a b for a pure quaternion a (a.c0 is not read), and for a pure b.
template <typename R>
__device__ __forceinline__ Q<R> q_pure_mul(const Q<R>& a, const Q<R>& b)
{
    return q_make<R>(-a.c1 * b.c1 - a.c2 * b.c2 - a.c3 * b.c3, a.c1 * b.c0 - a.c2 * b.c3 + a.c3 * b.c2,
                     a.c1 * b.c3 + a.c2 * b.c0 - a.c3 * b.c1, -a.c1 * b.c2 + a.c2 * b.c1 + a.c3 * b.c0);
}
template <typename R>
__device__ __forceinline__ Q<R> q_mul_pure(const Q<R>& a, const Q<R>& b)
{
    return q_make<R>(-a.c1 * b.c1 - a.c2 * b.c2 - a.c3 * b.c3, a.c0 * b.c1 - a.c2 * b.c3 + a.c3 * b.c2,
                     a.c0 * b.c2 + a.c1 * b.c3 - a.c3 * b.c1, a.c0 * b.c3 - a.c1 * b.c2 + a.c2 * b.c1);
}

// The plane of directions (d, v) among clover_plane's six, and whether d is its first direction.
__host__ __device__ constexpr int plane_of(int d, int v)
{
    for (int p = 0; p < 6; ++p)
        if ((clover_plane_a(p) == d && clover_plane_b(p) == v) || (clover_plane_a(p) == v && clover_plane_b(p) == d)) return p;
    return -1;
}
__host__ __device__ constexpr bool plane_first(int d, int v) { return clover_plane_a(plane_of(d, v)) == d; }

// Gradient of Q with respect to the e-link line L = L^e_D(x), all lines independent.  L is an edge of
// the e x e loop above it in each plane (D, v) and of the one below, and each loop enters F at its four
// corners.  With F-bar = dQ/dF (pure) and the path x -> x+v -> x+v+D -> x+D of lines B, A, B' (each e
// links) around the loop above, those four terms are the path with F-bar inserted at each corner:
//   F(x) M + M F(x+D) + [B F(x+v)] [A B'^dag] + [B A] [F(x+v+D) B'^dag],  M = B A B'^dag;
// the loop below runs the other way round and enters with the opposite sign, as does every loop of a
// plane whose first direction is v.  The charge's gradient after n smearing steps is what little of these terms varies slowly
// over the lattice, so that their rounding decides its accuracy.  Each term is therefore rounded at its own size and loops above
// and below are subtracted term by term: rms against 80-bit
// arithmetic after ten steps at 8x6x8x10 1.80e-14, where B [F(x+v) A + A F(x+v+D)] B'^dag with sums folded into multiply-adds has
// 2.11e-14 and a walk over every leaf 1.77e-14 (without smearing 4.2e-16, 4.3e-16 and 6.2e-16), for one product more a loop: a VJP
// of ten FP64 steps at 16x12x16x20 on B200 654 -> 664 us.
template <typename R, int D>
__device__ __forceinline__ Q<R> line_gradient(const FieldCA<R>& L, const R* fbar, const Geom& g,
                                              const Site& s, int par, int h, int e)
{
    const int q1 = par ^ (e & 1);   // parity one segment away
    const int upD = shift_by(g, D, s.c[D], e);
    const auto F = [&](int p, int pr, int n) {
        return ldq_ca(fbar, (size_t)p * g.V + (unsigned)(pr * g.Vh + (int)((unsigned)n >> 1)));
    };
    Q<R> acc = q_zero<R>();
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        if (v == D) continue;
        const int p = plane_of(D, v);
        const int up = s.n + shift_by(g, v, s.c[v], e), dn = s.n + shift_by(g, v, s.c[v], -e);
        const Q<R> A = L.ld(D, q1, up), B = L.ldh(v, par, h), B2 = L.ld(v, q1, s.n + upD);
        const Q<R> a = L.ld(D, q1, dn), b = q_dag(L.ld(v, q1, dn)), b2 = L.ld(v, par, dn + upD);
        const Q<R> BA = q_mul(B, A), ba = q_mul(b, a);
        const Q<R> M = q_sub(q_mul_nd(BA, B2), q_mul(ba, b2));
        Q<R> N = q_sub(q_mul(q_mul_pure(B, F(p, q1, up)), q_mul_nd(A, B2)), q_mul(q_mul_pure(b, F(p, q1, dn)), q_mul(a, b2)));
        N = q_add(N, q_sub(q_mul(BA, q_pure_mul(F(p, par, up + upD), q_dag(B2))), q_mul(ba, q_pure_mul(F(p, par, dn + upD), b2))));
        N = q_add(N, q_add(q_pure_mul(F(p, par, s.n), M), q_mul_pure(M, F(p, q1, s.n + upD))));
        acc = plane_first(D, v) ? q_add(acc, N) : q_sub(acc, N);
    }
    return acc;
}

// Line gradients T_e of all sites, directions D and sizes e, one per thread: CTA b takes (D, e) number
// b mod 12 of site block b / 12 (parities paired per warp), so that the twelve share their loads in L2.
// A gather: every result is written once, no atomics, and the sums run in a fixed order.  It replaced a
// walk over every leaf that added each link's term with an atomic (1728 products and 576 atomics a site;
// here 36 line gradients of about 17 products and 36 loads each): a whole VJP of five steps without the
// gradient's copy at 24^4 on B200 1580 -> 825 us (FP32) and 5290 -> 1510 us (FP64), at 8^4 605 -> 200 us
// (FP64).  Four CTAs per SM (FP64) and six (FP32): a VJP of ten steps, us, unbounded (104 registers in FP64) and with 3, 4, 5, 6:
// FP64 16x12x16x20 571, 561, 560, 561, 562; 24^4 2446, 2423, 2396, 2415, 2415; 32^4 7658, 7585, 7462, 7475, 7512; FP32 402, 404, 401, 392,
// 389; 1318, 1316, 1319, 1283, 1268; 4111, 4109, 4110, 3995, 3945; 8^4 all within 2 %.  FP64 at 32^4: 54 % of the FP64 pipe, L1 and
// L2 at 42 %; FP32: 64 % of the issue slots, waiting for instructions most.
constexpr int kLineBlock = 128;

template <typename R>
__global__ void __launch_bounds__(kLineBlock, sizeof(R) == 4 ? 6 : 4) k_line_gradient(Field<R> U, Field<R> L2, Field<R> L3, Field<R> T1, Field<R> T2,
                                                              Field<R> T3, Geom g, const R* fbar)
{
    pdl_trigger();
    const int job = blockIdx.x % 12, D = job & 3, e = 1 + (job >> 2);
    Site s{};
    int par, h;
    const bool valid = site_warp_pair(g, blockIdx.x / 12, threadIdx.x, blockDim.x, s, par, h);
    pdl_wait(h, s.n);
    if (!valid) return;
    FieldCA<R> L;
    Field<R> T;
    L.Vh = T.Vh = g.Vh;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        L.p[d] = e == 1 ? U.p[d] : (e == 2 ? L2.p[d] : L3.p[d]);
        T.p[d] = e == 1 ? T1.p[d] : (e == 2 ? T2.p[d] : T3.p[d]);
    }
    const R k4 = e == 1 ? R(1.5 * 0.25) : (e == 2 ? R(-0.15 * 0.25) : R(0.25 / 90.0));
    switch (D) {
        case 0: T.sth(0, par, h, q_scale(line_gradient<R, 0>(L, fbar, g, s, par, h, e), k4)); break;
        case 1: T.sth(1, par, h, q_scale(line_gradient<R, 1>(L, fbar, g, s, par, h, e), k4)); break;
        case 2: T.sth(2, par, h, q_scale(line_gradient<R, 2>(L, fbar, g, s, par, h, e), k4)); break;
        default: T.sth(3, par, h, q_scale(line_gradient<R, 3>(L, fbar, g, s, par, h, e), k4)); break;
    }
}

// dQ/dU_D(x) from the line gradients: U = U_D(x) is the first link of its lines at x, the second of
// those at x - D and the third of L^3 at x - 2D,
//   T1(x) + [T2(x) + U(x-D)^dag T3(x-D)] U(x+D)^dag + U(x-D)^dag T2(x-D)
//   + T3(x) L2(x+D)^dag + L2(x-2D)^dag T3(x-2D).
template <typename R>
__global__ void __launch_bounds__(kBlock) k_line_chain(Field<R> Unc, Field<R> L2nc, Field<R> T1nc, Field<R> T2nc, Field<R> T3nc,
                                                       Field<R> G, Geom g)
{
    pdl_trigger();
    Site s{};
    int par, h;
    const bool valid = site_warp_pair(g, blockIdx.x, threadIdx.x, blockDim.x, s, par, h);
    pdl_wait(h, s.n);
    if (!valid) return;
    const FieldCA<R> U = field_ca(Unc), L2 = field_ca(L2nc), T1 = field_ca(T1nc), T2 = field_ca(T2nc), T3 = field_ca(T3nc);
    const int q = par ^ 1;
#pragma unroll
    for (int D = 0; D < 4; ++D) {
        const int up = s.n + up_off_rt(g, s.c, D), dn = s.n + dn_off_rt(g, s.c, D), dn2 = s.n + shift_by(g, D, s.c[D], -2);
        const Q<R> um = U.ld(D, q, dn);
        Q<R> a = T1.ldh(D, par, h);
        a = q_mul_nd_add(a, q_mul_dn_add(T2.ldh(D, par, h), um, T3.ld(D, q, dn)), U.ld(D, q, up));
        a = q_mul_dn_add(a, um, T2.ld(D, q, dn));
        a = q_mul_nd_add(a, T3.ldh(D, par, h), L2.ld(D, q, up));
        a = q_mul_dn_add(a, L2.ld(D, par, dn2), T3.ld(D, par, dn2));
        G.sth(D, par, h, a);
    }
}

// ------------------------------------------------------ one APE step back ---

// 128-thread CTAs for both kernels; per SM four (FP32) and three (FP64) for v-bar, five and four for the
// gather, whose loads otherwise all run ahead (202 registers in FP64).  A VJP of five steps at 24^4, us:
// FP64 1552 -> 1361, FP32 785 -> 740 against two 256-thread CTAs for v-bar and no bound for the gather.
// One shape serves all grids: a VJP of ten steps, us, with 2, 3, 4 and 6 CTAs for v-bar: FP64 8^4 236, 235, 240, 256;
// 16x12x16x20 566, 562, 563, 638; 24^4 2559, 2454, 2460, 2688; 32^4 8161, 7794, 7695, 8381; FP32 16x12x16x20 390, 387, 381, 398,
// 32^4 4249, 4263, 4186, 4148; with 3, 4, 5, 6 for the gather: FP64 8^4 228, 237, 238, 237; 16x12x16x20 560, 563, 563, 587; 24^4 2525,
// 2442, 2469, 2503; 32^4 8088, 7760, 7744, 7845; FP32 all within 2 %.
constexpr int kSmearAdjBlock = 128;

// v-bar(x, mu) = (Gn - u' <u', Gn>) / |v|,  v = U + alpha S,  u' = v / |v|  (all four directions).
// The staple sums are the forward step's own (ape_staples), so v is exactly the forward's
// pre-projection link.
template <typename R>
__global__ void __launch_bounds__(kSmearAdjBlock, sizeof(R) == 4 ? 4 : 3) k_ape_vbar(Field<R> U, Field<R> Gnc, Field<R> Vbar, Geom g, R alpha)
{
    pdl_trigger();
    Site s{};
    int par, h;
    const bool valid = site_warp_pair(g, blockIdx.x, threadIdx.x, blockDim.x, s, par, h);
    pdl_wait(h, s.n);
    if (!valid) return;
    const FieldCA<R> Gn = field_ca(Gnc);
    ape_staples<R, SU2G_APE_ALL>(field_ca(U), g, s, par, h, [&](int mu, const Q<R>& u, const Q<R>& S) {
        const Q<R> v = q_axpy(alpha, S, u);
        const R inv = rsqrt_r(q_norm2(v));
        const Q<R> up = q_scale(v, inv);
        const Q<R> gn = Gn.ldh(mu, par, h);
        Vbar.sth(mu, par, h, q_scale(q_axpy(-q_dot(up, gn), up, gn), inv));
    });
}

// G_k(y, l) = vbar(y, l) + alpha * sum of the 18 staple terms containing U_l(y) (derivation in the
// file header's conventions; smearing.c:42-71 for the staples):
//  for mu != l:  vbar(y,mu) U_l(y+mu) U_mu(y+l)^dag          (first factor of the upper staple of (y, mu))
//                vbar(y-mu,mu)^dag U_l(y-mu) U_mu(y-mu+l)    (third factor, upper staple of (y-mu, mu))
//                U_mu(y) U_l(y+mu) vbar(y+l,mu)^dag          (first factor, lower staple of (y+l, mu))
//                U_mu(y-mu)^dag U_l(y-mu) vbar(y+l-mu,mu)    (third factor, lower staple of (y+l-mu, mu))
//  for nu != l:  U_nu(y-nu)^dag vbar(y-nu,l) U_nu(y-nu+l)    (middle, upper staple of (y-nu, l))
//                U_nu(y) vbar(y+nu,l) U_nu(y+l)^dag          (middle, lower staple of (y+nu, l))
template <typename R, int L>
__device__ __forceinline__ void gather_link(const FieldCA<R>& U, const FieldCA<R>& Vb, const Field<R>& G, const Geom& g,
                                            const Site& s, int par, int h, R alpha)
{
    const int q = par ^ 1;
    const int dl = up_off<L>(g, s);
    Q<R> acc = q_zero<R>();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        if (m == L) continue;
        const int ym = s.n + dn_off_rt(g, s.c, m);   // y - m
        const int yp = s.n + up_off_rt(g, s.c, m);   // y + m
        const int yl = s.n + dl;                     // y + l
        const int yml = ym + dl;                     // y - m + l
        // The six terms with a common plane share factors: with A = U_m(y), X = U_l(y+m),
        // Xv = vbar(y+m, l), B = U_m(y+l), Vm = vbar(y, m), Vn = vbar(y+l, m)
        //   Vm X B^dag + A Xv B^dag + A X Vn^dag = (Vm X + A Xv) B^dag + (A X) Vn^dag,
        // and with C = U_m(y-m), Y = U_l(y-m), Yv = vbar(y-m, l), D = U_m(y-m+l),
        // Wm = vbar(y-m, m), Wd = vbar(y-m+l, m)
        //   Wm^dag Y D + C^dag Yv D + C^dag Y Wd = (Wm^dag Y + C^dag Yv) D + (C^dag Y) Wd:
        // 10 products and 12 loads instead of 12 and 18.
        {
            const Q<R> A = U.ld(m, par, s.n), X = U.ld(L, q, yp), Xv = Vb.ld(L, q, yp);
            const Q<R> B = U.ld(m, q, yl), Vm = Vb.ld(m, par, s.n), Vn = Vb.ld(m, q, yl);
            const Q<R> AX = q_mul(A, X);
            acc = q_add(acc, q_mul_nd(q_add(q_mul(Vm, X), q_mul(A, Xv)), B));
            acc = q_add(acc, q_mul_nd(AX, Vn));
        }
        {
            const Q<R> C = U.ld(m, q, ym), Y = U.ld(L, q, ym), Yv = Vb.ld(L, q, ym);
            const Q<R> D = U.ld(m, par, yml), Wm = Vb.ld(m, q, ym), Wd = Vb.ld(m, par, yml);
            acc = q_add(acc, q_mul(q_add(q_mul_dn(Wm, Y), q_mul_dn(C, Yv)), D));
            acc = q_add(acc, q_mul(q_mul_dn(C, Y), Wd));
        }
    }
    G.sth(L, par, h, q_axpy(alpha, acc, Vb.ldh(L, par, h)));
}

// One link per thread, blockIdx.y = its direction.  Warp 2k takes parity 0 and warp 2k+1 parity 1
// of the same 32 half-volume indices (site_warp_pair): every warp reads consecutive links of one
// parity array, and both parities of a region are loaded by the same SM.
template <typename R>
__global__ void __launch_bounds__(kSmearAdjBlock, sizeof(R) == 4 ? 5 : 4) k_ape_gather(Field<R> Unc, Field<R> Vbnc, Field<R> G, Geom g, R alpha)
{
    pdl_trigger();
    Site s{};
    int par, h;
    const bool valid = site_warp_pair(g, blockIdx.x, threadIdx.x, blockDim.x, s, par, h);
    pdl_wait(h, s.n);
    if (!valid) return;
    const FieldCA<R> U = field_ca(Unc), Vb = field_ca(Vbnc);
    switch (blockIdx.y) {
        case 0: gather_link<R, 0>(U, Vb, G, g, s, par, h, alpha); break;
        case 1: gather_link<R, 1>(U, Vb, G, g, s, par, h, alpha); break;
        case 2: gather_link<R, 2>(U, Vb, G, g, s, par, h, alpha); break;
        default: gather_link<R, 3>(U, Vb, G, g, s, par, h, alpha); break;
    }
}

// su(2) gradient g = vec(G U^dag) per link, written in the reference's site-major order [n][mu][3].
template <typename R>
__global__ void __launch_bounds__(kBlock) k_grad_out(Field<R> Gnc, Field<R> Unc, Geom g, double* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int par, h = i >> 1;
    Site s = site_lex(g, i, par);
    pdl_wait(h, s.n);
    if (i >= g.V) return;
    const FieldCA<R> G = field_ca(Gnc), U = field_ca(Unc);
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        const Q<R> v = q_mul_nd(G.ldh(mu, par, h), U.ldh(mu, par, h));
        double* o = out + ((size_t)s.n * 4 + mu) * 3;
        o[0] = (double)v.c1;
        o[1] = (double)v.c2;
        o[2] = (double)v.c3;
    }
}

// ------------------------------------------------------------- driver ---

struct FieldBuf {
    void* base = nullptr;
    void* dirs[4] = {nullptr, nullptr, nullptr, nullptr};
};

// Scratch of one VJP from the handle's own stream-ordered pool.  The pool keeps its memory between
// calls (release threshold: unlimited), so repeated calls do not map gigabytes of pages again; the
// memory goes back when the handle is destroyed.
int ensure_pool(su2g_lattice* h)
{
    if (h->pool) return SU2G_OK;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = h->device;
    int rc = check_cuda(h, cudaMemPoolCreate(&h->pool, &props), "creating the scratch pool");
    if (rc) return rc;
    uint64_t keep = ~0ull;
    return check_cuda(h, cudaMemPoolSetAttribute(h->pool, cudaMemPoolAttrReleaseThreshold, &keep),
                      "configuring the scratch pool");
}

struct Arena {
    su2g_lattice* h;
    std::vector<void*> ptrs;
    int rc = SU2G_OK;
    explicit Arena(su2g_lattice* hh) : h(hh) { rc = ensure_pool(hh); }
    void* get(size_t bytes)
    {
        if (rc) return nullptr;
        void* p = nullptr;
        cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, h->pool, h->stream);
        if (e != cudaSuccess) {
            rc = check_cuda(h, e, "allocating adjoint buffers");
            return nullptr;
        }
        ptrs.push_back(p);
        return p;
    }
    FieldBuf field()
    {
        FieldBuf f;
        const size_t dir_bytes = 2ull * h->g.Vh * h->link_bytes;
        f.base = get(4 * dir_bytes);
        if (f.base)
            for (int mu = 0; mu < 4; ++mu) f.dirs[mu] = (char*)f.base + mu * dir_bytes;
        return f;
    }
    ~Arena()
    {
        for (void* p : ptrs) cudaFreeAsync(p, h->stream);
    }
};

template <typename R>
int vjp_t(su2g_lattice* h, int n_ape, double alpha, int c, double* q_out, double* grad_host)
{
    const Geom& g = h->g;
    const int nseg = n_ape > 0 ? (n_ape + c - 1) / c : 1;
    const int grid = (int)((g.V + kBlock - 1) / kBlock);
    const size_t dir_bytes = 2ull * g.Vh * h->link_bytes;
    Arena ar(h);
    std::vector<FieldBuf> ck(nseg), lev(std::max(c - 1, 0));
    for (auto& f : ck) f = ar.field();
    for (auto& f : lev) f = ar.field();
    FieldBuf tmp[2] = {ar.field(), ar.field()};
    FieldBuf G[2] = {ar.field(), ar.field()};
    FieldBuf Vb = ar.field();
    R* fbar = (R*)ar.get((size_t)6 * g.V * 4 * sizeof(R));
    double* gout = grad_host ? (double*)ar.get((size_t)g.V * 12 * sizeof(double)) : nullptr;
    if (ar.rc) return ar.rc;
    int rc = SU2G_OK;
    // U_0: the handle's field (directions may live in either of its allocations)
    for (int mu = 0; mu < 4; ++mu)
        if ((rc = check_cuda(h, cudaMemcpyAsync(ck[0].dirs[mu], h->dirp[mu], dir_bytes, cudaMemcpyDeviceToDevice,
                                                h->stream), "copying U_0")))
            return rc;
    // forward: keep U_{j c}; the other levels go through two scratch fields
    void* const* cur = ck[0].dirs;
    for (int k = 0; k < n_ape; ++k) {
        void* const* dst = ((k + 1) % c == 0 && (k + 1) / c < nseg) ? ck[(k + 1) / c].dirs : tmp[k & 1].dirs;
        if ((rc = ape_step(h, cur, dst, SU2G_APE_ALL, alpha))) return rc;
        cur = dst;
    }
    // Q, and F-bar = dQ/dF as it goes
    if ((rc = ensure_lines(h)) || (rc = qtop_enqueue(h, cur, 0, fbar))) return rc;
    // G_N = dQ/dU_N; the line gradients go into fields that are free until the smearing is reversed:
    // v-bar's, the other gradient's and the forward scratch that does not hold U_N
    void *l2[4], *l3[4];
    line_dirs(h, l2, l3);
    const Field<R> UN = make_field<R>(cur, g.Vh), L2 = make_field<R>(l2, g.Vh), L3 = make_field<R>(l3, g.Vh);
    const Field<R> T1 = make_field<R>(Vb.dirs, g.Vh), T2 = make_field<R>(G[1].dirs, g.Vh),
                   T3 = make_field<R>(tmp[n_ape & 1].dirs, g.Vh);
    const int lblocks = (int)((g.V + kLineBlock - 1) / kLineBlock);
    launch_begin(h, SU2G_K_OTHER);
    launch_pdl(k_line_gradient<R>, 12 * lblocks, kLineBlock, h->stream, UN, L2, L3, T1, T2, T3, g, fbar);
    launch_pdl(k_line_chain<R>, grid, kBlock, h->stream, UN, L2, T1, T2, T3, make_field<R>(G[0].dirs, g.Vh), g);
    if ((rc = launch_end(h, SU2G_K_OTHER, "charge adjoint kernels"))) return rc;
    // backwards through the smearing, one checkpoint segment at a time
    int gi = 0;
    for (int j = nseg - 1; j >= 0; --j) {
        const int k0 = j * c, m = std::min(c, n_ape - k0);
        std::vector<void* const*> L(m > 0 ? m : 1);
        L[0] = ck[j].dirs;
        for (int i = 1; i < m; ++i) {
            if ((rc = ape_step(h, L[i - 1], lev[i - 1].dirs, SU2G_APE_ALL, alpha))) return rc;
            L[i] = lev[i - 1].dirs;
        }
        for (int i = m - 1; i >= 0; --i) {
            Field<R> Uk = make_field<R>(L[i], g.Vh);
            Field<R> Gn = make_field<R>(G[gi].dirs, g.Vh), Gk = make_field<R>(G[gi ^ 1].dirs, g.Vh);
            Field<R> Vbf = make_field<R>(Vb.dirs, g.Vh);
            launch_begin(h, SU2G_K_OTHER);
            const int blocks = (g.V + kSmearAdjBlock - 1) / kSmearAdjBlock;
            launch_pdl(k_ape_vbar<R>, blocks, kSmearAdjBlock, h->stream, Uk, Gn, Vbf, g, (R)alpha);
            launch_pdl(k_ape_gather<R>, dim3(blocks, 4), kSmearAdjBlock, h->stream, Uk, Vbf, Gk, g, (R)alpha);
            if ((rc = launch_end(h, SU2G_K_OTHER, "smearing adjoint kernels"))) return rc;
            gi ^= 1;
        }
    }
    if (grad_host) {
        launch_begin(h, SU2G_K_OTHER);
        launch_pdl(k_grad_out<R>, grid, kBlock, h->stream, make_field<R>(G[gi].dirs, g.Vh), make_field<R>(ck[0].dirs, g.Vh), g,
                   gout);
        if ((rc = launch_end(h, SU2G_K_OTHER, "gradient output"))) return rc;
        if ((rc = check_cuda(h, cudaMemcpyAsync(grad_host, gout, (size_t)g.V * 12 * sizeof(double),
                                                cudaMemcpyDeviceToHost, h->stream), "copying the gradient")))
            return rc;
    }
    if ((rc = fetch_results(h, 0, 2))) return rc;
    if (q_out) *q_out = h->h_out[0];
    return SU2G_OK;
}

int segment_length(int n_ape, int ckpt)
{
    if (ckpt > 0) return std::min(ckpt, std::max(n_ape, 1));
    int c = (int)std::ceil(std::sqrt((double)std::max(n_ape, 1)));
    return std::max(c, 1);
}

// One step along su(2) coefficients x (per site and direction, the layout of the VJP's gradient):
// U_mu(n) <- exp(eps X) U_mu(n), X = i x.sigma, exp(eps X) = (cos(eps|x|), sin(eps|x|) x/|x|), for
// the sites [n0, n0 + count) whose coefficients are in `xs` (12 doubles per site).
template <typename R>
__global__ void __launch_bounds__(kBlock) k_tangent_step(const double* __restrict__ xs, Field<R> U, Geom g, int n0,
                                                         int count, double eps)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int n = n0 + i;
        int par;
        const Site s = site_lex(g, n, par);
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) {
            const double* x = xs + (size_t)i * 12 + 3 * mu;
            const double nx = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
            double sn, cs;
            sincos(eps * nx, &sn, &cs);
            const double f = nx > 0.0 ? sn / nx : 0.0;
            const Q<R> E = q_make<R>((R)cs, (R)(f * x[0]), (R)(f * x[1]), (R)(f * x[2]));
            U.sth(mu, par, n >> 1, q_mul(E, U.ld(mu, par, s.n)));
        }
    }
}

}  // namespace

extern "C" int su2g_ape_qtop_vjp(su2g_lattice* h, int32_t n_ape, double alpha, int32_t ckpt, double* q, double* grad)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_ape_qtop_vjp: null handle");
    if (n_ape < 0 || ckpt < 0 || !std::isfinite(alpha))
        return set_error(h, SU2G_EINVAL, "su2g_ape_qtop_vjp: bad argument (n_ape=%d, ckpt=%d)", n_ape, ckpt);
    cudaSetDevice(h->device);
    const int c = segment_length(n_ape, ckpt);
    return h->prec == SU2G_FP32 ? vjp_t<float>(h, n_ape, alpha, c, q, grad) : vjp_t<double>(h, n_ape, alpha, c, q, grad);
}

extern "C" int su2g_vjp_plan(const su2g_lattice* h, int32_t n_ape, int32_t ckpt, int32_t* levels_stored,
                             int64_t* device_bytes)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_vjp_plan: null handle");
    if (n_ape < 0 || ckpt < 0) return set_error(nullptr, SU2G_EINVAL, "su2g_vjp_plan: bad argument");
    const int c = segment_length(n_ape, ckpt);
    const int nseg = n_ape > 0 ? (n_ape + c - 1) / c : 1;
    const int levels = nseg + std::max(c - 1, 0);   // checkpoints + one recomputed segment
    const int64_t field = 4ll * h->g.V * (int64_t)h->link_bytes;
    if (levels_stored) *levels_stored = levels;
    // levels + 2 forward scratch + 2 gradients + v-bar + F-bar (6 quaternions per site) + output staging
    if (device_bytes)
        *device_bytes = (int64_t)(levels + 5) * field + 6ll * h->g.V * (int64_t)h->link_bytes + 96ll * h->g.V;
    return SU2G_OK;
}

extern "C" int su2g_tangent_step(su2g_lattice* h, const double* x, double eps)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_tangent_step: null handle");
    if (!x || !std::isfinite(eps)) return set_error(h, SU2G_EINVAL, "su2g_tangent_step: bad argument");
    cudaSetDevice(h->device);
    int rc = ensure_aos(h);   // the coefficients stream through the transfer staging, 12 of its 16 doubles a site
    if (rc) return rc;
    for (size_t n0 = 0; n0 < (size_t)h->g.V; n0 += h->aos_sites) {
        const int cnt = (int)std::min(h->aos_sites, (size_t)h->g.V - n0);
        rc = check_cuda(h, cudaMemcpyAsync(h->d_aos, x + n0 * 12, (size_t)cnt * 12 * sizeof(double),
                                           cudaMemcpyHostToDevice, h->stream),
                        "uploading tangent coefficients");
        if (rc) return rc;
        const int grid = grid_for(h, cnt, 8);
        launch_begin(h, SU2G_K_OTHER);
        if (h->prec == SU2G_FP32)
            k_tangent_step<float><<<grid, kBlock, 0, h->stream>>>(h->d_aos, make_field<float>(h->dirp, h->g.Vh), h->g,
                                                                 (int)n0, cnt, eps);
        else
            k_tangent_step<double><<<grid, kBlock, 0, h->stream>>>(h->d_aos, make_field<double>(h->dirp, h->g.Vh), h->g,
                                                                  (int)n0, cnt, eps);
        if ((rc = launch_end(h, SU2G_K_OTHER, "tangent step"))) return rc;
    }
    return check_cuda(h, cudaStreamSynchronize(h->stream), "tangent step");
}
