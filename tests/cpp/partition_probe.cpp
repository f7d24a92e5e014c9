// Prints fftcheb_partition's answer for every line of sizes on stdin.
#include "../../rsatb_b200/csrc/fftcheb_partition.cuh"

#include <cstdio>

int main() {
    using namespace rsatb_b200;
    unsigned long long workspace, fixed, cplx;
    long long brows;
    int b, samples, moments, bastin, sections, max_ctas = 296;
    unsigned long long part;
    while (std::scanf("%llu %llu %lld %d %d %d %llu %d %llu %d", &workspace, &fixed, &brows, &b,
                      &samples, &moments, &cplx, &bastin, &part, &sections) == 10) {
        const FftchebSizes s{size_t(workspace), size_t(fixed), brows, b, samples, moments,
                             size_t(cplx), bastin != 0, size_t(part), max_ctas, sections};
        FftchebPartition p{};
        const int fit = int(fftcheb_partition(s, &p));
        std::printf("%d %lld %d %lld %zu %d\n", fit, (long long)p.sec_brows, p.n_sections,
                    (long long)p.chunk_rows, p.e_bytes, p.ctas);
    }
}
