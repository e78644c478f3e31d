// On the GPU: the hardware's reciprocal seed and div_newton with it
// (astrosimgpu_b200/csrc/asg_device.cuh), run by tests/test_div_newton_gpu.py.
// Prints the largest |1 - b y| over every upper word of divisors in [1, 2) and
// their neighbours in the lower word, also scaled by powers of two, and the
// divisions that differ from the IEEE quotient: "max_error cases mismatches".
#include <cstdint>
#include <cstdio>

#include "asg_device.cuh"

namespace {

constexpr unsigned kFractions = 1u << 20;  // of a divisor's upper word
constexpr int kLows = 4, kScales = 9;

__global__ void check(double* worst, unsigned long long* counts) {
    double w = 0.0;
    unsigned long long cases = 0, bad = 0;
    for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < kFractions;
         f += gridDim.x * blockDim.x) {
        for (int l = 0; l < kLows; ++l) {
            const unsigned long long r = asg::mix64(7, f, l);
            const unsigned lows[kLows] = {0u, 0xFFFFFFFFu, 0x80000000u, static_cast<unsigned>(r)};
            for (int s = 0; s < kScales; ++s) {
                const int e = (s - kScales / 2) * 98;  // 2^-392 .. 2^392
                const unsigned hi = (static_cast<unsigned>(1023 + e) << 20) | f;
                const double b = __hiloint2double(static_cast<int>(hi), static_cast<int>(lows[l]));
                const double y = asg::rcp_seed(b);
                w = fmax(w, fabs(fma(-b, y, 1.0)));
                if (asg::div_newton_excluded(b)) continue;
                // a random numerator of about the divisor's size
                const double a = ldexp(1.0 + asg::unit53(r ^ (0x9E3779B97F4A7C15ull * (s + 1))), e / 2);
                ++cases;
                bad += asg::div_newton(a, b, y) != a / b;
            }
        }
    }
    atomicMax(reinterpret_cast<unsigned long long*>(worst),
              static_cast<unsigned long long>(__double_as_longlong(w)));  // w >= 0
    atomicAdd(counts, cases);
    atomicAdd(counts + 1, bad);
}

}  // namespace

int main() {
    double* w;
    unsigned long long* c;
    if (cudaMallocManaged(&w, sizeof *w) != cudaSuccess ||
        cudaMallocManaged(&c, 2 * sizeof *c) != cudaSuccess)
        return 1;
    *w = 0.0;
    c[0] = c[1] = 0;
    check<<<512, 128>>>(w, c);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    std::printf("%.17g %llu %llu\n", *w, c[0], c[1]);
    return 0;
}
