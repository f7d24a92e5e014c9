// Prints dmma_any_wanted for every line "W b complex double rows row_blocks" on stdin (148 SMs).
#include "../../rsatb_b200/csrc/dmma_any_rule.cuh"

#include <cstdio>

int main() {
    int W, b, cm, dbl, deg;
    long long rows;
    while (std::scanf("%d %d %d %d %lld %d", &W, &b, &cm, &dbl, &rows, &deg) == 6)
        std::printf("%d\n", rsatb_b200::step_detail::dmma_any_wanted(W, b, cm != 0, dbl != 0, rows, deg,
                                                                     148) ? 1 : 0);
}
