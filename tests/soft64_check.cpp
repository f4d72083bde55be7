// Host build of csrc/soft64.cuh against the machine's own FP64: every quotient
// and root bit for bit, sines and cosines against long double.  argv: a family
// of operands and a count.  The approximations of the FP32 unit are off by up
// to one unit (reciprocal) and two (reciprocal square root) at random.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

static std::mt19937_64 rng(7);
static float off(float r, int n)
{
    uint32_t b;
    memcpy(&b, &r, 4);
    b += (uint32_t)n;
    memcpy(&r, &b, 4);
    return r;
}
namespace tp {
namespace sd {
inline float rcp_approx(float x) { return off((float)(1.0 / (double)x), x == 2.0f || x == 1.0f ? 0 : (int)(rng() % 3) - 1); }
inline float rsqrt_approx(float x) { return off((float)(1.0 / std::sqrt((double)x)), (int)(rng() % 5) - 2); }
}  // namespace sd
}  // namespace tp
#define TP_SOFT64_HOST_APPROX
#include "soft64.cuh"
using namespace tp::sd;

static double operand(int family)
{
    uint64_t m = rng() & 0xfffffffffffffull;
    switch (family) {
    case 1: m &= 0xffull << 44; break;                       // few leading bits
    case 2: m = ~(m & 0xff) & 0xfffffffffffffull; break;     // just below a power of two
    case 3: m &= 0xff; break;                                // just above one
    case 4: m = m & 1 ? 0xfffffffffffffull : 0; break;
    default: break;
    }
    // exponents over the whole window and a little past it
    return value((rng() & 1) << 63 | (uint64_t)(1023 - 460 + rng() % 920) << 52 | m);
}

static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }

int main(int argc, char** argv)
{
    const int family = atoi(argv[1]);
    const long n = atol(argv[2]);
    long bad = 0;
    double worst = 0.0;
    for (long i = 0; i < n; i++) {
        const double a = operand(family), b = operand((int)(rng() % 5));
        double c = a;
        if (i % 16 == 0) c = value((bits(a) & ~0xfffffffffffffull) | ((bits(b) + rng() % 5 - 2) & 0xfffffffffffffull));
        const double p = a * b, s = std::fabs(a), q = value(bits(s * s) + rng() % 3 - 1);
        bad += !same(div(c, b), c / b) + !same(div(p, b), p / b) + !same(sqrt_rn(s), std::sqrt(s)) +
               !same(sqrt_rn(q), std::sqrt(q));
        // angles over the reduced range, near multiples of a quarter turn, and small
        const double u = (double)(rng() >> 11) * 0x1p-53;
        double x = i % 3 == 0 ? std::ldexp(0.5 + u / 2, -11 + (int)(rng() % 21))
                 : i % 3 == 1 ? (double)(rng() % 40) * 0.78539816339744831 + std::ldexp(u - 0.5, -(int)(rng() % 22)) : 6.3 * u;
        if (rng() & 1) x = -x;
        double sn, cs;
        sin_cos(x, sn, cs);
        const long double rs = sinl((long double)x), rc = cosl((long double)x);
        auto ulps = [](double v, long double r) {
            const double d = std::fabs((double)r);
            return (double)(std::fabs((long double)v - r) / (std::nextafter(d, INFINITY) - d));
        };
        worst = std::fmax(worst, std::fmax(ulps(sn, rs), ulps(cs, rc)));
    }
    const double sp[] = {0.0, -0.0, 1.0, -1.0, 3.0, INFINITY, -INFINITY, NAN, 5e-324, 1e-310, 1e308, 1e-200, 1e200, 0x1p-12, 1024.0};
    for (double a : sp) {
        for (double b : sp) bad += !same(div(a, b), a / b);
        double sn, cs;
        sin_cos(a, sn, cs);
        bad += !same(sqrt_rn(a), std::sqrt(a)) + !(std::fabs(a) < INFINITY ? std::fabs(sn - std::sin(a)) < 1e-15 : sn != sn);
    }
    printf("%ld wrong, %.4f units\n", bad, worst);
    // half a unit of the rounding, 2^-6.5 of one before it
    return bad != 0 || !(worst < 0.512);
}
