// Host build of lean64's fixed-point functions against long double libm:
// prints `<name> <largest error>` (units of 2^-57, or ulp of a double result),
// and `round_by_one <mismatches>`.  Built and run by tests/test_fixed_point_host.py.
#include <cmath>
#include <cstdio>
#include <random>

#define LEAN64_FN __host__ __device__ __forceinline__
#define LEAN64_HOST_TABLES
#include "../noa_gb300/csrc/lean64.cuh"

using namespace lean64;

static double ulp_error(double v, long double ref) {
    int e;
    std::frexp((double)ref, &e);
    return (double)(fabsl((long double)v - ref) / std::ldexp(1.0, e - 53));
}

static double unit_error(long long v, long double ref) { return (double)fabsl((long double)v - ref * 0x1p57L); }

int main() {
    std::mt19937_64 gen(7);
    std::uniform_real_distribution<double> uni(0, 1);
    const char *names[] = {"log", "log3p", "log_of", "exp", "exp_to", "ratio"};
    double worst[6] = {};
    long mismatches = 0;
    const auto take = [&](int k, double v) { worst[k] = v <= worst[k] ? worst[k] : v; };
    const auto round_check = [&](double x) {
        volatile double y = 1. - x;
        volatile double z = 1. - y;
        mismatches += z != round_by_one(x);
    };
    for (int i = 0; i < 500000; i++) {
        const double x = std::exp((2 * uni(gen) - 1) * 40);
        take(0, unit_error(lean_log_fx(x), logl(x)));
        take(1, unit_error(lean_log3p_fx(x), logl(3 + (long double)x)));
        const long long v = (long long)std::ldexp(std::exp((2 * uni(gen) - 1) * 20 - 16), 57) + 1;
        take(2, unit_error(log_of_fx(v), logl((long double)v) - 57 * logl(2.L)));
        const long long a = (long long)std::ldexp(2 * uni(gen) - 1, 57) * 63;
        take(3, ulp_error(lean_exp_fx(a), expl((long double)a * 0x1p-57L)));
        const long long b = (long long)std::ldexp(uni(gen) * 4.15 - uni(gen) * (i & 1) * 40, 57);
        take(4, unit_error(exp_to_fx(b), expl((long double)b * 0x1p-57L)));
        const unsigned long long n = (gen() >> 2) >> (gen() % 20) | 1, d = ((gen() >> 2) | 1ull << 50) >> (gen() % 8);
        take(5, ulp_error(ratio_fx(n, d), (long double)n / (long double)d));
        round_check(std::exp(-45 * uni(gen)));
    }
    for (int k = -60; k <= 0; k++)
        for (int m = 0; m < 4096; m++)
            round_check(std::ldexp(1 + m / 4096., k - 1));
    round_check(1.);
    round_check(0x1.fffffffffffffp-1);
    for (int k = 0; k < 6; k++)
        std::printf("%s %.4f\n", names[k], worst[k]);
    std::printf("round_by_one %ld\n", mismatches);
}
