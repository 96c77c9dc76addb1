// kpmath.cuh -- the Kennedy-Pendleton sampler's division by beta, and the FP64 logarithm, squared cosine and
// sine/cosine pair of its uniforms u = (w + 1/2) / 2^32 of a 32-bit random word.
//
// The general library functions spend most of their instructions on arguments that cannot occur here
// (negative, zero, denormal, infinite, any size) and fetch each coefficient with two moves.  These use what
// is known of u: 33 significant bits, inside (0, 1), a multiple of the period known to the integer word.
//  - log: the table-driven method of P. T. P. Tang (ACM TOMS 16(4), 1990): u = 2^k z, z in [0.6875, 1.375), and
//    for the 128 intervals of z a number c near 1/z of at most 20 bits, so that r = z c - 1, |r| <= 2^-8, is
//    exact; log u = k ln 2 - log c + log1p(r).  Each c is the one near 1/z whose -log c lies closest to a double
//    (S. Gal and B. Bachelis, ACM TOMS 17(1), 1991).  The interval that ends at 1 has c = 1, so that the
//    relative error stays small where log u goes to 0.
//  - cosines and sines: the angle is reduced exactly in integers, then near-minimax polynomials (Chebyshev
//    fits computed from sin and cos in 60 digits) of relative error below 2^-57.
// Against 80-bit arithmetic over 8 x 10^7 words, largest error in ulp of the value: log 1.2, cos^2 5.3, sine and
// cosine 1.5.  On B200, with beta entering as its reciprocal (KpBeta): FP64 heatbath pass at
// 24^4 16.4 -> 14.6 us, at 24x14x18x22 9.0 -> 8.5 us, at 48^4 164 -> 156 us.
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

// {c, -log c} of the 128 intervals
static __device__ const double2 kKpLog[128] = {
    {1.4502067565917969, -0x1.7ca08898e64d2p-2}, {1.4419288635253906, -0x1.76c3e885f17cfp-2},
    {1.4343223571777344, -0x1.715960c817972p-2}, {1.4258003234863281, -0x1.6b3f33e2b02bdp-2},
    {1.41802978515625, -0x1.65a69fc3f12c0p-2}, {1.4107627868652344, -0x1.6063c1b8afb98p-2},
    {1.4025306701660156, -0x1.5a659b7d1e595p-2}, {1.3950920104980469, -0x1.54f39037b15e4p-2},
    {1.3872871398925781, -0x1.4f34e02c01e5ap-2}, {1.3801841735839844, -0x1.49f33d6f44c54p-2},
    {1.3729400634765625, -0x1.448fb6909c9eep-2}, {1.3653755187988281, -0x1.3ee75fb3e33dbp-2},
    {1.3582916259765625, -0x1.3993c49cc4cd5p-2}, {1.350830078125, -0x1.33efc101dbbe0p-2},
    {1.3437347412109375, -0x1.2e8b31a10e158p-2}, {1.3368949890136719, -0x1.295172127b308p-2},
    {1.3297004699707031, -0x1.23cae78619eefp-2}, {1.3233489990234375, -0x1.1ee3be1a0284dp-2},
    {1.3161773681640625, -0x1.19533db820b23p-2}, {1.3090553283691406, -0x1.13c4e332ffc4cp-2},
    {1.3029670715332031, -0x1.0efed7fc7ceb4p-2}, {1.2958183288574219, -0x1.095ca0bb97224p-2},
    {1.2894248962402344, -0x1.044c091120f28p-2}, {1.2833824157714844, -0x1.fef9630155f0cp-3},
    {1.2768211364746094, -0x1.f47a18330c2c5p-3}, {1.2702713012695312, -0x1.e9f1ae45ceed5p-3},
    {1.2639427185058594, -0x1.dfb71ca827b96p-3}, {1.2576179504394531, -0x1.d570fd4018959p-3},
    {1.2520599365234375, -0x1.cc5ec66cdb6fbp-3}, {1.2457847595214844, -0x1.c2147f9d5871ep-3},
    {1.2397956848144531, -0x1.b835ebb85f26cp-3}, {1.2334251403808594, -0x1.ada8fbbafedf6p-3},
    {1.2275810241699219, -0x1.a3eef0afbc70cp-3}, {1.2221565246582031, -0x1.9add0e14ed73bp-3},
    {1.21588134765625, -0x1.9052284cabe92p-3}, {1.2107124328613281, -0x1.8798920a69aa3p-3},
    {1.2050895690917969, -0x1.7e0ff7fcacbecp-3}, {1.1992111206054688, -0x1.740c396fab86bp-3},
    {1.1935920715332031, -0x1.6a6dd6014cd2ep-3}, {1.188018798828125, -0x1.60d807b59f4a8p-3},
    {1.1825904846191406, -0x1.5776f496caa4fp-3}, {1.176849365234375, -0x1.4d7f7f51bbae8p-3},
    {1.1714096069335938, -0x1.440275997007ap-3}, {1.166107177734375, -0x1.3ab7dcdcf9065p-3},
    {1.1610221862792969, -0x1.31c49fcc05d7cp-3}, {1.15570068359375, -0x1.285c0b9973d71p-3},
    {1.1509628295898438, -0x1.1ff2483876a40p-3}, {1.1457481384277344, -0x1.16a57b6dd8366p-3},
    {1.1400947570800781, -0x1.0c841f6e4dc07p-3}, {1.1354179382324219, -0x1.0419004335043p-3},
    {1.1304817199707031, -0x1.f65963da2ee6ep-4}, {1.1252937316894531, -0x1.e38234d93723dp-4},
    {1.1201095581054688, -0x1.d0984e51dcc00p-4}, {1.1158103942871094, -0x1.c0d7f4cd0c220p-4},
    {1.110260009765625, -0x1.ac6b0012d1e89p-4}, {1.1059036254882812, -0x1.9c508e42cbebfp-4},
    {1.1014747619628906, -0x1.8be0d7ff20ac5p-4}, {1.0964164733886719, -0x1.79066407d9b51p-4},
    {1.0919265747070312, -0x1.683795f940f59p-4}, {1.0871505737304688, -0x1.56432323e85e7p-4},
    {1.0828628540039062, -0x1.461360f35a9bep-4}, {1.0774879455566406, -0x1.31b1b2628c91ep-4},
    {1.0729827880859375, -0x1.20883bd4a3b93p-4}, {1.0685272216796875, -0x1.0f7cf37882ff2p-4},
    {1.0643119812011719, -0x1.fe9878a6e75c6p-5}, {1.05999755859375, -0x1.dd51ed50e7d06p-5},
    {1.0559005737304688, -0x1.bd988afbb5ad5p-5}, {1.0512657165527344, -0x1.998ede2f593b3p-5},
    {1.0467453002929688, -0x1.7641b91e166c5p-5}, {1.0431671142578125, -0x1.5a348dcd50af0p-5},
    {1.0385856628417969, -0x1.3625db229ea13p-5}, {1.0343246459960938, -0x1.14782629590ddp-5},
    {1.0303916931152344, -0x1.ea855411dbf76p-6}, {1.0258941650390625, -0x1.a2d9a7d3876cap-6},
    {1.0222129821777344, -0x1.67f44d9b53c4bp-6}, {1.0175971984863281, -0x1.1dce1cc1a93c7p-6},
    {1.0137252807617188, -0x1.beb104f246eaap-7}, {1.0097122192382812, -0x1.3cb6e7fc7f2b1p-7},
    {1.0059928894042969, -0x1.8793ec7ad9f61p-8}, {1, 0x0.0p+0},
    {0.99642562866210938, 0x1.d556dc2bfda86p-9}, {0.98861312866210938, 0x1.7744003ec2851p-7},
    {0.98088455200195312, 0x1.3c38352c1d0dep-6}, {0.9734039306640625, 0x1.b9a642b46b063p-6},
    {0.96609115600585938, 0x1.1a99a1645e9d5p-5}, {0.95890426635742188, 0x1.57c4f611fa4d8p-5},
    {0.95203018188476562, 0x1.92b4eec1c40dap-5}, {0.945037841796875, 0x1.cf18a60b4e0eap-5},
    {0.93750762939453125, 0x1.085102d3a1a1ep-4}, {0.93073272705078125, 0x1.26060fc20b950p-4},
    {0.92376708984375, 0x1.44cb27ba4a028p-4}, {0.91715621948242188, 0x1.623630ed51834p-4},
    {0.91082000732421875, 0x1.7e9b761cf51c7p-4}, {0.9047393798828125, 0x1.9a0b37ddc9bdap-4},
    {0.89813613891601562, 0x1.b80c50b979cc8p-4}, {0.89179611206054688, 0x1.d5108f7d2fcdfp-4},
    {0.88550186157226562, 0x1.f21398953a975p-4}, {0.8793487548828125, 0x1.0751a5756c753p-3},
    {0.87409210205078125, 0x1.1399306f4c2a2p-3}, {0.8675689697265625, 0x1.22f07e2f08204p-3},
    {0.86231231689453125, 0x1.2f62d9392efa9p-3}, {0.85604476928710938, 0x1.3e5372eae45b7p-3},
    {0.85037994384765625, 0x1.4bec6c8698c86p-3}, {0.84471893310546875, 0x1.599a4c2d3db99p-3},
    {0.83951950073242188, 0x1.663f6113eb4d8p-3}, {0.83394622802734375, 0x1.73e38bcd17bf3p-3},
    {0.82857894897460938, 0x1.811cc50e68c9bp-3}, {0.82295989990234375, 0x1.8f0c5d87d3411p-3},
    {0.8179931640625, 0x1.9b7223f1f3117p-3}, {0.81297683715820312, 0x1.a80b39a8726bfp-3},
    {0.80736541748046875, 0x1.b63a92424780ap-3}, {0.80272293090820312, 0x1.c20a042ab67cap-3},
    {0.79777145385742188, 0x1.ceb6063607fe1p-3}, {0.79251480102539062, 0x1.dc40145d0e170p-3},
    {0.78776931762695312, 0x1.e88ce3ced8b8ep-3}, {0.78264999389648438, 0x1.f5e718eb4e6d2p-3},
    {0.77817153930664062, 0x1.00d3e38761adcp-2}, {0.773590087890625, 0x1.06dfcfba8ec49p-2},
    {0.7683868408203125, 0x1.0dc8f9c27f0abp-2}, {0.7642669677734375, 0x1.134a4c9ac6f2ap-2},
    {0.75931930541992188, 0x1.19f0ddfe40a82p-2}, {0.75508880615234375, 0x1.1fa97835c6c8dp-2},
    {0.75066375732421875, 0x1.25ae3b5756306p-2}, {0.74670028686523438, 0x1.2b1a01d229dd8p-2},
    {0.74186325073242188, 0x1.31c1ab41daa3ep-2}, {0.73740005493164062, 0x1.37ef8ad1479e4p-2},
    {0.7339324951171875, 0x1.3cc328be81a4fp-2}, {0.7297515869140625, 0x1.429cc1105fe19p-2},
};
// sin(pi y) / y, sin(2 pi y) / y and cos(2 pi y) as polynomials in y^2, highest power first
static __constant__ const double kKpSinPi[9] = {
    0x1.9d462020fcc78p-21, -0x1.6f7acdb8f6580p-16, 0x1.e8f3675ee37ddp-12, -0x1.e3074dfaf87afp-8,
    0x1.5078348551854p-4, -0x1.32d2cce627c86p-1, 0x1.466bc6775aa7dp+1, -0x1.4abbce625be52p+2,
    0x1.921fb54442d18p+1};
static __constant__ const double kKpSin2Pi[7] = {
    0x1.e3f38399551bfp+1, -0x1.e30071afc3e59p+3, 0x1.50782fda12d96p+5, -0x1.32d2cce2e5b19p+6,
    0x1.466bc677587f8p+6, -0x1.4abbce625be41p+5, 0x1.921fb54442d18p+2};
static __constant__ const double kKpCos2Pi[8] = {
    -0x1.b264ba152378ap+0, 0x1.f9cc41140bb60p+2, -0x1.a6d1ec7906c20p+4, 0x1.e1f5068355e15p+5,
    -0x1.55d3c7e3c90f8p+6, 0x1.03c1f081b5aacp+6, -0x1.3bd3cc9be45dep+4, 0x1.0000000000000p+0};
// log1p(r) = r + r^2 (-1/2 + r/3 - r^2/4 + ...), highest power first; ln 2; the reduction's constants
static __constant__ const double kKpLog1p[6] = {1.0 / 7, -1.0 / 6, 1.0 / 5, -1.0 / 4, 1.0 / 3, -1.0 / 2};
static __constant__ const double kKpMisc[6] = {0x1.62e42fefa39efp-1,            // ln 2
                                               0x1p-32,                         // 2^-32
                                               -(0x1p20 - 0x1p-33),             // u = magic 2^-32 + this
                                               -(0x1p20 + 0.5),                 // the same, minus 1/2
                                               -(0x1p52 + 0x1p31),              // signed word from its offset form
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
    const double u = fma(kp_magic(w), kKpMisc[1], kKpMisc[2]);
    const int hi = __double2hiint(u), t = hi - 0x3fe60000;
    const double2 e = __ldg(&kKpLog[(t >> 13) & 127]);
    const double z = __hiloint2double(hi - (t & (int)0xfff00000), __double2loint(u));
    // k = t >> 20 in [-33, 0]
    const double k = kp_magic((uint32_t)(t >> 20) ^ 0x80000000u) + kKpMisc[4];
    const double r = fma(z, e.x, -1.0);
    const double q = fma(r * r, kp_poly(kKpLog1p, r), r);
    return fma(k, kKpMisc[0], e.y + q);
}

// cos^2(2 pi u): of period 1/2 in u, so with y = 1/2 - (2u mod 1) in (-1/2, 1/2) it is sin^2(pi y)
__device__ __forceinline__ double kp_cos2pi_sq_word(uint32_t w)
{
    const double y = fma(kp_magic(0u - ((w << 1) | 1u)), kKpMisc[1], kKpMisc[3]);
    const double s = y * kp_poly(kKpSinPi, y * y);
    return s * s;
}

// sin and cos of 2 pi u: u = q / 4 + y, |y| <= 1/8
__device__ __forceinline__ void kp_sincos2pi_word(uint32_t w, double* sn, double* cs)
{
    const uint32_t v = w + 0x20000000u;             // (u + 1/8) 2^32 - 1/2
    const int q = (int)(v >> 30);
    // y = (V - 2^29 + 1/2) 2^-32 with V = v mod 2^30
    const double y = fma(kp_magic(((v << 1) | 1u) & 0x7fffffffu), 0.5 * kKpMisc[1], kKpMisc[5]);
    const double z = y * y;
    const double s = y * kp_poly(kKpSin2Pi, z), c = kp_poly(kKpCos2Pi, z);
    const double a = q & 1 ? c : s, b = q & 1 ? s : c;
    // quadrants 0..3: (s, c), (c, -s), (-s, -c), (-c, s)
    *sn = q & 2 ? -a : a;
    *cs = (q + 1) & 2 ? -b : b;
}

}  // namespace su2g
