// kpmath.cuh -- the Kennedy-Pendleton sampler's division by beta, and the FP64 logarithm, squared cosine and
// sine/cosine pair of its uniforms u = (w + 1/2) / 2^32 of a 32-bit random word.
//
// The general library functions spend most of their instructions on arguments that cannot occur here
// (negative, zero, denormal, infinite, any size) and fetch each coefficient with two moves.  These use what
// is known of u: 33 significant bits, inside (0, 1), a multiple of the period known to the integer word.
//  - log: the table-driven method of P. T. P. Tang (ACM TOMS 16(4), 1990).  u = 2^E m with m in [1, 2), and for each
//    of 128 intervals of m a number c near 1/m (near 1/(2m') for m' = m/2 above 1.375), so that r = m c - 1 is exact
//    and |r| <= 2^-8: log u = E ln 2 - log c + log1p(r).  ln 2 and -log c are split into a multiple of 2^-47 and a rest
//    of 20 bits.  u having 33 bits, the high parts and r add up without rounding, also where they cancel (u near 1,
//    with c = 1/2 in the last interval); what remains, r^2 (-1/2 + r/3 - ...) and the rests, is small against
//    the sum: one rounding in all.
//  - cosines and sines: the angle is reduced exactly in integers, then near-minimax polynomials (Chebyshev
//    fits in 60 digits) behind an exact first term, of which pi is held in two parts.
// tests/golden/make_kpmath.py computes the constants.  Against 80-bit arithmetic, largest (rms) error in ulp: log 0.52 (0.289),
// cos^2 2.5 (0.55), sine 1.02 (0.30), cosine 1.02 (0.30); CUDA's log 0.54 (0.289), the square of its cospi 3.38 (0.78), its sincospi 1.48 (0.36).
// (ARM Optimized Routines' and musl's log, MIT licence, follow the same method: a table of 128 pairs c, -log c, and one
// multiply-add for r.)  Twenty FP64 heatbath sweeps at beta = 3.09 on B200, with the library functions and with these: 8^4 465, 387
// us; 24^4 1.91, 1.65 ms; 48^4 26.1, 23.9 ms.
#pragma once
#include <cmath>
#include <cstdint>

namespace su2g {

// What the sampler takes for beta: FP32 beta itself, FP64 its reciprocal as hi + lo, so that a product with
// it is as accurate as the division it stands for (two multiply-adds a link instead).  lo is 0 where the
// reciprocal is 0 or infinite.
template <typename R>
struct KpBeta;
template <>
struct KpBeta<float> {
    float beta;
};
template <>
struct KpBeta<double> {
    double hi, lo;
};
template <typename R>
inline KpBeta<R> kp_beta(double beta);
template <>
inline KpBeta<float> kp_beta<float>(double beta)
{
    return {(float)beta};
}
template <>
inline KpBeta<double> kp_beta<double>(double beta)
{
    const double hi = 1.0 / beta;
    return {hi, std::isfinite(beta) && std::isfinite(hi) ? std::fma(-beta, hi, 1.0) / beta : 0.0};
}
// x / beta
__device__ __forceinline__ float kp_over_beta(float x, const KpBeta<float>& b) { return __fdividef(x, b.beta); }
__device__ __forceinline__ double kp_over_beta(double x, const KpBeta<double>& b) { return fma(x, b.hi, x * b.lo); }

// (2^52 + w) as a double: a 32-bit word enters FP64 arithmetic without a conversion instruction
__device__ __forceinline__ double kp_magic(uint32_t w) { return __hiloint2double(0x43300000, (int)w); }

// {-log c to a multiple of 2^-47, c}; the low word of c is 0, and the high word of the rest of -log c stands in its place
static __device__ const double2 kKpLog[128] = {
    {0x1.fefeaa2b10000p-9, 0x1.fe0203cebc04ap-1}, {0x1.7db6f5f8c7000p-7, 0x1.fa120bcc89efep-1},
    {0x1.3ceba4346e000p-6, 0x1.f63103cdf4f01p-1}, {0x1.b9f8727b12800p-6, 0x1.f25f8bcb204cfp-1},
    {0x1.1b0d90923d800p-5, 0x1.ee9c83ce8fc2dp-1}, {0x1.58a63afc8f400p-5, 0x1.eae803cda9193p-1},
    {0x1.95caf8ecad400p-5, 0x1.e7418bce0465fp-1}, {0x1.d27848adba800p-5, 0x1.e3a90bccb7a42p-1},
    {0x1.075993598e400p-4, 0x1.e01e03cee2603p-1}, {0x1.254062f0a9400p-4, 0x1.dca003cb6fe51p-1},
    {0x1.42eef3ea6f200p-4, 0x1.d92f03cb043f9p-1}, {0x1.6063a29392200p-4, 0x1.d5cb0bcbc7313p-1},
    {0x1.7da58ed7cc600p-4, 0x1.d2730bcb39d29p-1}, {0x1.9ab33c6209c00p-4, 0x1.cf2703ce99affp-1},
    {0x1.b78b2abb1d400p-4, 0x1.cbe703ce81f6ap-1}, {0x1.d4305166d2000p-4, 0x1.c8b283cc2ad0bp-1},
    {0x1.f0a1400130000p-4, 0x1.c5898bcb1bd74p-1}, {0x1.0670872caf900p-3, 0x1.c26b8bcd6f031p-1},
    {0x1.1479784688700p-3, 0x1.bf580bce4de3fp-1}, {0x1.22663190aeb00p-3, 0x1.bc500bcda45d7p-1},
    {0x1.303ce98e4c800p-3, 0x1.b95203cc2fb62p-1}, {0x1.3dfd030ed7c00p-3, 0x1.b65e03cea75dap-1},
    {0x1.4ba38539a5800p-3, 0x1.b3748bcdb52ebp-1}, {0x1.59347f9990500p-3, 0x1.b09483ce27953p-1},
    {0x1.66acfa272b300p-3, 0x1.adbe8bcb6421cp-1}, {0x1.740eb7540ee00p-3, 0x1.aaf20bccb431dp-1},
    {0x1.815b881439a00p-3, 0x1.a82e8bcc12c48p-1}, {0x1.8e92dde888600p-3, 0x1.a57403ce02ac0p-1},
    {0x1.9bb428e7e9500p-3, 0x1.a2c28bce62812p-1}, {0x1.a8bed7c882f00p-3, 0x1.a01a03ce630bap-1},
    {0x1.b5b4d1e8fca00p-3, 0x1.9d7a0bccb91f0p-1}, {0x1.c2958f58d0500p-3, 0x1.9ae283cd2480dp-1},
    {0x1.cf6308e09dc00p-3, 0x1.985303ceb1216p-1}, {0x1.dc1cc00acd900p-3, 0x1.95cb8bcce8c3fp-1},
    {0x1.e8bfab2aa9500p-3, 0x1.934c8bcef064cp-1}, {0x1.f5505964b9200p-3, 0x1.90d50bcdc7cbcp-1},
    {0x1.00e72a5ada180p-2, 0x1.8e650bcdb340dp-1}, {0x1.071b47fcd7700p-2, 0x1.8bfd03cd51be1p-1},
    {0x1.0d46dd79ac400p-2, 0x1.899c0bcea6f98p-1}, {0x1.136865293a980p-2, 0x1.874283ce12f6cp-1},
    {0x1.1980f2dd42b80p-2, 0x1.84f00bcd09886p-1}, {0x1.1f904ee48db80p-2, 0x1.82a48bcdb6f60p-1},
    {0x1.2596410df9600p-2, 0x1.806003cecf82fp-1}, {0x1.2b9290ab90480p-2, 0x1.7e228bcc2d42ep-1},
    {0x1.3187b6954fb00p-2, 0x1.7beb0bce9795ap-1}, {0x1.3772cf2c02e80p-2, 0x1.79ba8bca83e3ep-1},
    {0x1.3d54fd5c1f700p-2, 0x1.779083ce0c39bp-1}, {0x1.432f6ba055a80p-2, 0x1.756c8bcc482c4p-1},
    {0x1.49008a0401300p-2, 0x1.734f0bce399e6p-1}, {0x1.4ec9862600500p-2, 0x1.713783cedd7afp-1},
    {0x1.548a303add280p-2, 0x1.6f2603ca67e64p-1}, {0x1.5a42580f50580p-2, 0x1.6d1a83ce9ccb4p-1},
    {0x1.5ff3360a7a500p-2, 0x1.6b1483cd5c8fbp-1}, {0x1.659b34303eb80p-2, 0x1.691483cb2068dp-1},
    {0x1.6b3b8e2359e80p-2, 0x1.671a0bce13b6fp-1}, {0x1.70d4182789600p-2, 0x1.65250bca1533bp-1},
    {0x1.7664a6239f700p-2, 0x1.633583c88033bp-1}, {0x1.7bedc5237b580p-2, 0x1.614b43ce40f02p-1},
    {0x1.816f4b5a0d580p-2, 0x1.5f664bceae524p-1}, {0x1.86e90ea330c80p-2, 0x1.5d8683cd209fbp-1},
    {0x1.8c5ba1058bf00p-2, 0x1.5babcbcc9efd7p-1}, {0x1.91c6dab45ea80p-2, 0x1.59d60bce13a21p-1},
    {0x1.9729d51139800p-2, 0x1.58058bce2cd76p-1}, {0x1.9c86a32dc0980p-2, 0x1.563983cea4dcfp-1},
    {0x1.a1dc61cd5fb00p-2, 0x1.54724bca0c0afp-1}, {0x1.a72a2966be200p-2, 0x1.52b00bcd5e983p-1},
    {0x1.ac7155a58c800p-2, 0x1.50f243cd88b38p-1}, {0x1.b1b1c2ebe0380p-2, 0x1.4f390bcdc9711p-1},
    {0x1.b6eb4d53cf480p-2, 0x1.4d8443cd61d47p-1}, {0x1.bc1dd0b0dc580p-2, 0x1.4bd403cc4832bp-1},
    {0x1.c149ef115f200p-2, 0x1.4a2803ce35666p-1}, {0x1.c66f86bff8900p-2, 0x1.48804bcd7973ep-1},
    {0x1.cb8dad44dba00p-2, 0x1.46dd03cd1f9bap-1}, {0x1.d0a699e726500p-2, 0x1.453d8bcd9d64ap-1},
    {0x1.d5b7d0ae2d380p-2, 0x1.43a283ce2e557p-1}, {0x1.dac38e62c7400p-2, 0x1.420b43cd0a413p-1},
    {0x1.dfc81d106f280p-2, 0x1.40784bce92054p-1}, {0x1.e4c6f48688280p-2, 0x1.3ee90bce9e9bcp-1},
    {0x1.e9bff75989500p-2, 0x1.3d5d83cebb391p-1}, {0x1.eeb238640ed00p-2, 0x1.3bd603cd435f6p-1},
    {0x1.f39e674811f80p-2, 0x1.3a524bcdbb2fep-1}, {0x1.f88465efebc80p-2, 0x1.38d24bce8aa66p-1},
    {0x1.fd64e88f61600p-2, 0x1.3755c3ce32524p-1}, {0x1.011f801261c80p-1, 0x1.35dd0bce1e98dp-1},
    {0x1.038a1b7ce8240p-1, 0x1.34678bce3c20ap-1}, {0x1.05f1649264f40p-1, 0x1.32f5cbce1b516p-1},
    {0x1.0855b704b49c0p-1, 0x1.318783ce75bfap-1}, {0x1.0ab7706ce1540p-1, 0x1.301c8bced3fadp-1},
    {0x1.0d1617cb9ec00p-1, 0x1.2eb503cebdf7dp-1}, {0x1.0f720b89b7780p-1, 0x1.2d50cbcc9d27ap-1},
    {0x1.11cbabf87e940p-1, 0x1.2bef8bcdd7bc4p-1}, {0x1.1422121244140p-1, 0x1.2a91cbceacd54p-1},
    {0x1.16759d7abc600p-1, 0x1.293743cd88374p-1}, {0x1.18c6afbf5f500p-1, 0x1.27dfcbce3b6bcp-1},
    {0x1.1b153d17da5c0p-1, 0x1.268b43cd65fbep-1}, {0x1.1d6139a678b40p-1, 0x1.2539cbc96c6cap-1},
    {0x1.1faa293870b40p-1, 0x1.23eb83ced0c04p-1}, {0x1.21f0dfc65cf00p-1, 0x1.22a00bce41d7ap-1},
    {0x1.2434e17485580p-1, 0x1.21578bce31c5cp-1}, {0x1.2676221343100p-1, 0x1.20120bce032d5p-1},
    {0x1.28b5079f60840p-1, 0x1.1ecf4bccc43f0p-1}, {0x1.2af1874265a00p-1, 0x1.1d8f4bcb50fe0p-1},
    {0x1.2d2b22d2eea00p-1, 0x1.1c524bcc05320p-1}, {0x1.2f62b55509780p-1, 0x1.1b17cbce1926bp-1},
    {0x1.3197c0fa80e80p-1, 0x1.19e00bce5e1f2p-1}, {0x1.33ca3aa328d00p-1, 0x1.18ab03ce8c82cp-1},
    {0x1.35fa171d39f40p-1, 0x1.1778cbcdf826ep-1}, {0x1.382836a589100p-1, 0x1.1648cbcd5fe50p-1},
    {0x1.3a53a467ee2c0p-1, 0x1.151b8bcc5c447p-1}, {0x1.3c7c54ff74f00p-1, 0x1.13f10bce6396ep-1},
    {0x1.3ea32b76b3240p-1, 0x1.12c8c3cdf8798p-1}, {0x1.40c7a7880dd00p-1, 0x1.11a303cda453dp-1},
    {0x1.42e9bf1df81c0p-1, 0x1.107fcbce09353p-1}, {0x1.4509e0d33f2c0p-1, 0x1.0f5ec3ce29497p-1},
    {0x1.472711733d280p-1, 0x1.0e4083cc8bc3bp-1}, {0x1.4942b27a2fdc0p-1, 0x1.0d244bce444b7p-1},
    {0x1.4b5bc8156e5c0p-1, 0x1.0c0a8bcbb9173p-1}, {0x1.4d72c2a3a0180p-1, 0x1.0af303cc11c6ep-1},
    {0x1.4f879935028c0p-1, 0x1.09ddcbcd27472p-1}, {0x1.519a42cba3580p-1, 0x1.08cac3ceca6c8p-1},
    {0x1.53aab65b9a600p-1, 0x1.07ba03cd95465p-1}, {0x1.55b9678b43340p-1, 0x1.06ab43ca7f181p-1},
    {0x1.57c5543370e80p-1, 0x1.059f0bcd6f7e6p-1}, {0x1.59cfeadfb1a40p-1, 0x1.049483ceefaf2p-1},
    {0x1.5bd7aa8e73600p-1, 0x1.038c83ce41a9fp-1}, {0x1.5dde04b14a880p-1, 0x1.02864bcea4822p-1},
    {0x1.5fe1f46d189c0p-1, 0x1.018243cdd9abep-1}, {0x1.62e42fefa3a00p-1, 0x1.00000bce0ca87p-1},
};
// (sin(2 pi y) / y - 2 pi) / y^2 and (cos(2 pi y) - 1) / y^2 as polynomials in y^2, highest power first; 2 pi and ln 2 in
// two parts
static __constant__ const double kKpSin2Pi[6] = {
    0x1.e4a9d9166f052p+1, -0x1.e3027dea82bd7p+3, 0x1.50783208843ebp+5, -0x1.32d2cce500387p+6,
    0x1.466bc6775a476p+6, -0x1.4abbce625be52p+5};
static __constant__ const double kKpCos2Pi[7] = {
    -0x1.b2f3eb054afcdp+0, 0x1.f9ce245cada0bp+2, -0x1.a6d1eef479be1p+4, 0x1.e1f5068688d5bp+5,
    -0x1.55d3c7e3cb241p+6, 0x1.03c1f081b5ac0p+6, -0x1.3bd3cc9be45dep+4};
static __constant__ const double kKp2Pi[2] = {
    0x1.921fb54442d18p+2, 0x1.1a62633145c07p-52};
static __constant__ const double kKpLn2[2] = {
    0x1.62e42fefa3a00p-1, -0x1.0ca8700000000p-49};
// log1p(r) = r + r^2 (-1/2 + r/3 - r^2/4 + ...), highest power first; the reduction's constants
static __constant__ const double kKpLog1p[6] = {1.0 / 7, -1.0 / 6, 1.0 / 5, -1.0 / 4, 1.0 / 3, -1.0 / 2};
static __constant__ const double kKpMisc[4] = {0x1p-32,                         // 2^-32
                                               -(0x1p20 - 0x1p-33),             // u = magic 2^-32 + this
                                               -(0x1p52 + 1023.0),              // E from the biased exponent
                                               -(0x1p19 + 0x1p-3)};             // (2V + 1) 2^-33 - 1/8

template <int N>
__device__ __forceinline__ double kp_poly(const double (&c)[N], double x)
{
    double p = c[0];
#pragma unroll
    for (int i = 1; i < N; ++i) p = fma(p, x, c[i]);
    return p;
}

// log((w + 1/2) / 2^32)
__device__ __forceinline__ double kp_log_word(uint32_t w)
{
    const double u = fma(kp_magic(w), kKpMisc[0], kKpMisc[1]);
    const int hi = __double2hiint(u);
    const double2 e = __ldg(&kKpLog[(hi >> 13) & 127]);
    const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(u));
    const double E = kp_magic((uint32_t)hi >> 20) + kKpMisc[2];
    const double r = fma(m, __hiloint2double(__double2hiint(e.y), 0), -1.0);
    const double s = fma(E, kKpLn2[0], e.x) + r;
    const double rest = fma(E, kKpLn2[1], __hiloint2double(__double2loint(e.y), 0));
    return s + fma(r * r, kp_poly(kKpLog1p, r), rest);
}

// y = V 2^-33 - 1/8 for V < 2^31, and sin(2 pi y) for |y| <= 1/8
__device__ __forceinline__ double kp_eighth(uint32_t V) { return fma(kp_magic(V), 0.5 * kKpMisc[0], kKpMisc[3]); }
__device__ __forceinline__ double kp_sin2pi(double y, double z)
{
    return fma(y, kKp2Pi[0], y * fma(z, kp_poly(kKpSin2Pi, z), kKp2Pi[1]));
}

// cos^2(2 pi u) = cos^2(pi f), f = 2u mod 1 = q / 2 + 2y: 1 - sin^2(2 pi y) or, with q = 1, sin^2(2 pi y)
__device__ __forceinline__ double kp_cos2pi_sq_word(uint32_t w)
{
    const uint32_t v = ((w << 1) | 1u) + 0x40000000u;
    const double y = kp_eighth(v & 0x7fffffffu);
    const double s = kp_sin2pi(y, y * y);
    return v >> 31 ? s * s : fma(-s, s, 1.0);
}

// sin and cos of 2 pi u: u = q / 4 + y, |y| <= 1/8
__device__ __forceinline__ void kp_sincos2pi_word(uint32_t w, double* sn, double* cs)
{
    const uint32_t v = w + 0x20000000u;             // (u + 1/8) 2^32 - 1/2
    const int q = (int)(v >> 30);
    // y = (V - 2^29 + 1/2) 2^-32 with V = v mod 2^30
    const double y = kp_eighth(((v << 1) | 1u) & 0x7fffffffu);
    const double z = y * y;
    const double s = kp_sin2pi(y, z);
    const double c = fma(z, kp_poly(kKpCos2Pi, z), 1.0);
    const double a = q & 1 ? c : s, b = q & 1 ? s : c;
    // quadrants 0..3: (s, c), (c, -s), (-s, -c), (-c, s)
    *sn = q & 2 ? -a : a;
    *cs = (q + 1) & 2 ? -b : b;
}

}  // namespace su2g
