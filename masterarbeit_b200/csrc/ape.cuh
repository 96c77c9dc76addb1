// ape.cuh -- the APE staple sums of one site, shared by the smearing step and its adjoint.
// Reference: staples_smearing / smearing_APE_all, _spatial, _temporal
// (LGT_Code/modules/obs/smearing.c:42-168).
#pragma once
#include "internal.cuh"

namespace su2g {

__host__ __device__ constexpr bool ape_updates(int mode, int mu)
{
    return mode == SU2G_APE_ALL ? true : (mode == SU2G_APE_SPATIAL ? mu != 0 : mu == 0);
}
// Is nu a staple direction for link mu?  staples_smearing(n, dir, dt) skips kk == dir and kk == dt
// with dt = dir (all), 0 (spatial, temporal)  (smearing.c:51, :89, :122, :155).
__host__ __device__ constexpr bool ape_staple(int mode, int mu, int nu)
{
    return nu != mu && (mode == SU2G_APE_ALL ? true : nu != 0);
}

// Staple sums S_mu(x) of the links the mode updates, and the links u_mu(x) they need, with the
// staples of smearing.c:42-71:
//   S_mu(x) = sum_nu U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu).
// The middle product P = U_mu(x+nu) U_nu(x+mu)^dag of the forward staple of mu in plane nu is
// also the dagger of the middle product of the forward staple of nu in plane mu, so each plane's
// P is formed once.  emit(mu, u_mu, S_mu) is called for each updated link when its sum is complete.
//
// The backward staples of all four links go plane by plane: U_nu(x-nu) is read once for its three links, and a plane's
// loads (7) do not wait for a link's end.  Against link by link, where one link's state at a time is live but
// U_nu(x-nu) stays in registers or is read again: FP64 24^4 30.2 -> 28.4 us a step, 48^4 512 -> 487; FP32 24^4 16.2 -> 15.3,
// 40x30x36x34 72 -> 64, 48^4 250 -> 235.  The spatial and temporal steps have no more than two links a plane and
// keep the order by links (spatial by planes: FP64 0 to 2 %, FP32 spills at eight CTAs per SM); so does the FP32 step on
// fields of large time slices (PLANES false, k_ape).
//
// FOLD: a staple's last product is added up within its multiply-adds (rounded at the size of the growing sum);
// else it is rounded by itself and then added, which is the more accurate (FP64, ten steps against 80-bit arithmetic,
// rms: all 1.82e-16 and 1.47e-16, spatial 1.49e-16 and 1.31e-16).
template <bool FOLD, typename R>
__device__ __forceinline__ Q<R> staple_add(const Q<R>& S, const Q<R>& a, const Q<R>& b)
{
    return FOLD ? q_mul_add(S, a, b) : q_add(S, q_mul(a, b));
}
template <typename R, int MODE, bool PLANES = true, bool FOLD = true, typename F, typename Emit>
__device__ __forceinline__ void ape_staples(const F& in, const Geom& g, const Site& s, int par, int h, Emit&& emit)
{
    const int q = par ^ 1;
    int xp[4], xm[4];
    Q<R> u[4], S[4];
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        xp[mu] = s.n + up_off_rt(g, s.c, mu);
        xm[mu] = s.n + dn_off_rt(g, s.c, mu);
        S[mu] = q_zero<R>();
        bool need = ape_updates(MODE, mu);
#pragma unroll
        for (int nu = 0; nu < 4; ++nu) need = need || (ape_updates(MODE, nu) && ape_staple(MODE, nu, mu));
        if (need) u[mu] = in.ldh(mu, par, h);
    }
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
#pragma unroll
        for (int nu = mu + 1; nu < 4; ++nu) {
            const bool a = ape_updates(MODE, mu) && ape_staple(MODE, mu, nu);
            const bool b = ape_updates(MODE, nu) && ape_staple(MODE, nu, mu);
            if (!a && !b) continue;
            const Q<R> P = q_mul_nd(in.ld(mu, q, xp[nu]), in.ld(nu, q, xp[mu]));
            if (a) S[mu] = staple_add<FOLD>(S[mu], u[nu], P);   // U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag
            if (b) S[nu] = FOLD ? q_mul_nd_add(S[nu], u[mu], P) : q_add(S[nu], q_mul_nd(u[mu], P));   // U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag
        }
    if (MODE == SU2G_APE_ALL && PLANES) {   // plane by plane
#pragma unroll
        for (int nu = 0; nu < 4; ++nu) {
            const Q<R> a = in.ld(nu, q, xm[nu]);   // U_nu(x-nu), of all three links
#pragma unroll
            for (int mu = 0; mu < 4; ++mu) {
                if (mu == nu) continue;
                const Q<R> b = in.ld(mu, q, xm[nu]);                      // U_mu(x-nu)
                const Q<R> c = in.ld(nu, par, xm[nu] + (xp[mu] - s.n));   // U_nu(x-nu+mu)
                S[mu] = staple_add<FOLD>(S[mu], q_mul_dn(a, b), c);
            }
        }
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) emit(mu, u[mu], S[mu]);
        return;
    }
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        if (!ape_updates(MODE, mu)) continue;
        const int dmu = xp[mu] - s.n;
#pragma unroll
        for (int nu = 0; nu < 4; ++nu) {
            if (!ape_staple(MODE, mu, nu)) continue;
            const Q<R> a = in.ld(nu, q, xm[nu]);          // U_nu(x-nu)
            const Q<R> b = in.ld(mu, q, xm[nu]);          // U_mu(x-nu)
            const Q<R> c = in.ld(nu, par, xm[nu] + dmu);  // U_nu(x-nu+mu)
            S[mu] = staple_add<FOLD>(S[mu], q_mul_dn(a, b), c);
        }
        emit(mu, u[mu], S[mu]);
    }
}

}  // namespace su2g
