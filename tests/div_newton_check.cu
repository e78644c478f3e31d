// Host check of div_newton (astrosimgpu_b200/csrc/asg_device.cuh) against the
// IEEE division, run by tests/test_div_newton.py: `div_newton_check CASES SEED`
// prints one line per operand class, "name cases mismatches".
//
// The seed of the reciprocal is the hardware's on the GPU; here it is 1/b off
// by any relative error up to the stated bound, with and without the
// hardware's truncation to the upper 32 bits.  The host fma rounds once, as
// the GPU's does.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "asg_device.cuh"

namespace {

std::uint64_t g_seed, g_count;

std::uint64_t bits() { return asg::mix64(g_seed, 0, g_count++); }
double unit() { return asg::unit53(bits()); }

double from_bits(std::uint64_t u) {
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
}

// significand (53-bit integer, top bit set) times 2^(e - 52)
double make(std::uint64_t sig, int e) { return std::ldexp(static_cast<double>(sig), e - 52); }

double seed_of(double b) {
    const double y = 1.0 / b * (1.0 + (2.0 * unit() - 1.0) * 0x1p-19);
    if (bits() & 1) return y;
    std::uint64_t u;
    const double t = 1.0 / b * (1.0 + (2.0 * unit() - 1.0) * 0x1p-20);
    std::memcpy(&u, &t, sizeof u);
    return from_bits(u & 0xFFFFFFFF00000000ull);
}

struct Class {
    const char* name;
    long long cases = 0, bad = 0;
    void check(double a, double b) {
        if (asg::div_newton_excluded(b)) return;
        ++cases;
        const double got = asg::div_newton(a, b, seed_of(b)), want = a / b;
        if (std::memcmp(&got, &want, sizeof got) != 0) {
            if (bad++ < 3) std::fprintf(stderr, "%s: %a / %a: got %a, want %a\n", name, a, b, got, want);
        }
    }
    void print() const { std::printf("%s %lld %lld\n", name, cases, bad); }
};

constexpr std::uint64_t kTop = 1ull << 52;

// Inverse of an odd B modulo 2^64 (Newton).
std::uint64_t inverse(std::uint64_t B) {
    std::uint64_t x = B;
    for (int i = 0; i < 6; ++i) x *= 2 - B * x;
    return x;
}

}  // namespace

int main(int argc, char** argv) {
    const long long n = argc > 1 ? std::atoll(argv[1]) : 1000000;
    g_seed = argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1;
    Class random{"random"}, wide{"wide"}, edge{"edge"}, mid{"midpoint"}, model{"model"};
    for (long long i = 0; i < n; ++i) {
        random.check(make(kTop | (bits() >> 12), 0), make(kTop | (bits() >> 12), 0));
        wide.check(make(kTop | (bits() >> 12), static_cast<int>(bits() % 801) - 400),
                   make(kTop | (bits() >> 12), static_cast<int>(bits() % 801) - 400));
        // divisors next to the excluded ones, next to 1, and with few bits set
        std::uint64_t B = kTop | (bits() >> 12);
        switch (i % 3) {
            case 0: B = 2 * kTop - (1ull << 32) - 1 - (bits() >> (30 + bits() % 34)); break;
            case 1: B = kTop + (bits() >> (20 + bits() % 44)); break;
            default: B = kTop | (1ull << (bits() % 52)) | (bits() & 3);
        }
        edge.check(make(kTop | (bits() >> 12), 0), make(B, 0));
        // quotients next to a midpoint of two doubles: M B = A 2^j + d with a
        // 54-bit odd M and |d| <= 4
        B = (i & 1 ? B : (kTop | (bits() >> 12))) | 1;
        const int j = 53 + static_cast<int>(bits() & 1);
        const std::uint64_t mask = (1ull << j) - 1;
        long long d = 1 + static_cast<long long>(bits() & 3);
        if (bits() & 1) d = -d;
        std::uint64_t M = (static_cast<std::uint64_t>(d) * inverse(B)) & mask;
        if (M < (1ull << 53)) M += 1ull << 53;
        const unsigned __int128 P = static_cast<unsigned __int128>(M) * B -
                                    static_cast<unsigned __int128>(static_cast<__int128>(d));
        const std::uint64_t A = static_cast<std::uint64_t>(P >> j);
        if ((M & 1) && M < (1ull << 54) && (P & mask) == 0 && A >= kTop && A < 2 * kTop)
            mid.check(make(A, 0), make(B, 0));
        // the astrocyte's divisions
        const double x = std::ldexp(unit(), -static_cast<int>(bits() % 12)) + 0x1p-60;
        model.check(x, x + 0.13);
        model.check(x, x + 0.08234);
        model.check(0.0009 * x * x, 0.01 + x * x);
        model.check(0.0002098 * (x + 0.13), x + 0.9434);
    }
    for (const Class* c : {&random, &wide, &edge, &mid, &model}) c->print();
    return 0;
}
