// The sampler functions of kpmath.cuh compiled for the host (the same operations in the same order; fma is exact on
// both), against 80-bit arithmetic.  Prints one "name max_ulp rms_ulp" line per function (test_sampler_math.py).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#define __device__
#define __constant__
#define __forceinline__ inline
struct double2 {
    double x, y;
};
static inline float __fdividef(float x, float y) { return x / y; }
static inline double __hiloint2double(int h, int l)
{
    const uint64_t v = ((uint64_t)(uint32_t)h << 32) | (uint32_t)l;
    double d;
    memcpy(&d, &v, 8);
    return d;
}
static inline uint64_t bits(double d)
{
    uint64_t v;
    memcpy(&v, &d, 8);
    return v;
}
static inline int __double2hiint(double d) { return (int)(bits(d) >> 32); }
static inline int __double2loint(double d) { return (int)(uint32_t)bits(d); }
template <class T>
static inline T __ldg(const T* p) { return *p; }
#include "kpmath.cuh"
using namespace su2g;

struct Err {
    long double max = 0, sq = 0;
    long n = 0;
    void add(double got, long double want)
    {
        int e;
        std::frexp((double)want, &e);
        const long double u = std::fabs(got - want) / std::ldexp(1.0L, e - 53);
        max = u > max ? u : max;
        sq += u * u;
        ++n;
    }
    void print(const char* name) const { std::printf("%s %.4Lf %.4Lf\n", name, max, std::sqrt(sq / n)); }
};

int main()
{
    std::mt19937_64 gen(1);
    Err over;
    for (int i = 0; i < 2000000; ++i) {
        const double beta = std::exp2(-6.0 + 12.0 * (gen() >> 11) * 0x1p-53), x = std::exp2(-3.0 + 12.0 * (gen() >> 11) * 0x1p-53);
        over.add(kp_over_beta(x, kp_beta<double>(beta)), (long double)x / beta);
    }
    over.print("over_beta");
    const double inf = INFINITY;
    const bool limits = kp_over_beta(0.5, kp_beta<double>(inf)) == 0.0 && kp_over_beta(0.5, kp_beta<double>(0.0)) == inf &&
                        kp_over_beta(0.5, kp_beta<double>(1e-320)) == inf && kp_over_beta(0.5, kp_beta<double>(-2.0)) == -0.25;
    std::printf("limits %d 0\n", limits);

    // The words: both ends, the ends of the logarithm's intervals, the quadrants' and octants' borders, and any others.
    Err lg, c2, sn, cs;
    const long double pi2 = 6.283185307179586476925286766559005768394L;
    const auto word = [&](uint32_t w) {
        const long double u = (w + 0.5L) / 4294967296.0L, q = std::round(u * 4), y = u - q / 4;
        const long double s = std::sin(pi2 * y), c = std::cos(pi2 * y);
        const int Q = (int)q & 3;
        const long double S = Q == 0 ? s : Q == 1 ? c : Q == 2 ? -s : -c, C = Q == 0 ? c : Q == 1 ? -s : Q == 2 ? -c : s;
        double a, b;
        kp_sincos2pi_word(w, &a, &b);
        lg.add(kp_log_word(w), std::log(u));
        c2.add(kp_cos2pi_sq_word(w), C * C);
        sn.add(a, S);
        cs.add(b, C);
    };
    for (uint32_t i = 0; i < 32; ++i)
        for (uint32_t d = 0; d < 20000; ++d) {
            word((i << 27) + d);   // i = 0: the smallest words
            word((i << 27) - d);   // i = 0: the largest
        }
    for (int e = 0; e < 32; ++e)
        for (uint64_t j = 128; j <= 256; ++j) {
            const uint64_t edge = j << 32 >> (8 + e);
            for (int d = -8; d <= 8; ++d) word((uint32_t)(edge + d));
        }
    for (int i = 0; i < 3000000; ++i) word((uint32_t)gen());
    lg.print("log");
    c2.print("cos2");
    sn.print("sin");
    cs.print("cos");
    return 0;
}
