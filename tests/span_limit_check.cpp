// Prints span_that_fits and most_spikes (astrosimgpu_b200/csrc/asg_span.hpp)
// for the cases on standard input: want neurons edges substeps ref_steps count_bits.
#include <cstdio>

#include "asg_span.hpp"

int main() {
    int want, substeps, ref, bits;
    unsigned long long n, e;
    while (std::scanf("%d %llu %llu %d %d %d", &want, &n, &e, &substeps, &ref, &bits) == 6) {
        std::printf("%d", asg::span_that_fits(want, n, e, substeps, ref, bits));
        for (int L = 1; L <= want; ++L)
            std::printf(" %lld", static_cast<long long>(asg::most_spikes(L, substeps, ref)));
        std::printf("\n");
    }
}
