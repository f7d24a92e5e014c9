// The rule that sends a step to the any-shape tensor-core kernel.  Host only.
#pragma once

#include <cstdint>

namespace rsatb_b200 {
namespace step_detail {

// Where the any-shape tensor-core kernel is the default.  It gives every block row
// a warp, however many the others would use: ahead while an SM has few block rows
// (per_sm) and where the others lose their wide loads (W no multiple of 4) or have
// no specialisation (blocks of 4, 6, 7); behind once the others' threads fill the
// SMs, the more the emptier its 8 x 8 tiles are (blocks of 2, 3).  Blocks of 8 at
// W = 8, 16, 32, 64, 128, 256 in FP64 (W <= 16 in FP32) stay with the tiled kernel
// before it, equal or faster.  Measured at 17 blocks a row, per term of a
// propagation, time of the others / time of this kernel, at 4,096 | 16,384 |
// 32,768 block rows (per_sm 27, 110, 221) and 8,192 where the line lies there:
//   FP64    b = 2 W = 8 1.4 | 0.8 | 0.5 (8,192: 1.1), 31 1.3 | 1.3 | 1.3
//           b = 3 W = 4 2.6 | 1.4 | 0.9, 16 2.0 | 1.3 | 1.3
//           b = 4 W = 4 3.2 | 1.5 | 1.3    b = 7 W = 16 5.3 | 3.1 | 3.6
//           b = 5 W = 8 2.0 | 1.4 | 1.1, 6 2.0 | 1.3 | 0.75, 16 1.05 (8,192: 0.9),
//           32 0.9, 57 1.3 | 1.2 | 1.3     b = 8 W = 24 1.7 | 2.4 | 2.5
//   complex b = 2 W = 8 1.6 | 0.8 | 0.5 (8,192: 1.1)    b = 3 W = 4 2.6 | 1.1 | 0.8
//           b = 5 W = 12 1.4 | 0.8 | 0.9 (8,192: 1.2), 8 1.2 | 0.7 | 0.6 (8,192: 1.0),
//           32 0.97, 48 1.3 | 1.2 | 1.1    b = 8 W = 12 1.7 | 2.0 | 1.9, 32 1.1 | 0.9
//   FP32    b = 2 W = 8 1.4 | 0.7 | 0.5, 24 1.1 (8,192: 0.8)    b = 3 W = 4 2.4 | 1.2 | 0.8
//           b = 4 W = 4 2.8 | 1.4 | 0.9, 8 3.3 | 1.9 | 1.2
//           b = 5 W = 8 1.3 | 0.9 | 0.8 (8,192: 1.0), 16 1.0, 24 1.0 (1,024: 1.5)
//           b = 8 W = 24 1.4 | 1.3 | 1.3, 57 1.2 | 1.1, 48 0.9, 2 3.8 | 1.8 | 1.0
//   complex b = 2 W = 8 1.4 | 0.7 | 0.5    b = 3 W = 8 2.3 | 1.0 | 0.6
//           b = 4 W = 4 3.1 | 1.2 | 1.0    b = 5 W = 12 1.2 | 0.7 | 0.5 (8,192: 0.8)
//           b = 8 W = 6 3.1 | 1.1 | 0.6, 12 1.3 | 0.9 (8,192: 0.8), 16 0.9 (1,024: 2.0)
// Rows of few blocks (sparse: 5 a row measured, FP64 unless said) leave more of the
// time to the epilogue and the dots, where a warp per block row does worse: b = 2
// W = 8 0.9 | 0.8, b = 3 W = 4 1.3 | 0.8, b = 4 W = 4 1.7 | 1.0, 24 1.3 | 0.9,
// b = 5 W = 4 1.2 | 0.9, 57 0.7 | 0.6, b = 7 W = 16 2.6 | 1.8, FP32 b = 8 W = 24
// 1.0 | 0.9, 57 0.8 | 0.7, complex b = 2 W = 16 1.2, 48 0.85, b = 5 W = 48 1.1, 62 0.9.
inline bool dmma_any_wanted(int W, int b, bool cm, bool dbl, int64_t rows, double row_blocks,
                            int sm_count) {
    const int64_t per_sm = rows / sm_count;
    const bool sparse = row_blocks < 10.0;
    const bool own = b == 4 || b == 6 || b == 7;  // the others run any size in one kernel
    if (dbl && !cm) {
        const bool odd = W % 4 != 0;
        if (b == 8) return true;
        if (own)
            return (W < 32 || odd) && !(b == 4 && sparse && per_sm > 56 && W >= 16 && !odd);
        if (b == 5) {
            if (sparse) return per_sm <= 56 && W < 31 && W != 16;
            return per_sm <= 112 ? W < 16 || (W < 32 && W % 16 != 0) || W % 2 != 0
                                 : W > 24 && W % 2 != 0;
        }
        if (b == 3) {
            if (sparse) return per_sm <= 56 && W < 24;
            return per_sm <= 112 ? W < 32 || odd : W > 8 && (W < 24 || odd);
        }
        if (sparse) return false;
        return per_sm <= 56 ? W < 24 || odd : W > 24 && W % 2 != 0;
    }
    if (dbl) {
        if (W > 48 && W % 8 == 0) return false;
        if (own) return true;
        if (b == 8) return per_sm <= 32 || W < 8 || (W & (W - 1)) != 0;
        if (b == 5) {
            if (sparse) return per_sm <= 32 && W <= 48 && W != 32 && W != 16;
            return per_sm <= 32 ? W != 32 : W > 32;
        }
        if (b == 3) return per_sm <= 112 || W >= 8;
        return per_sm <= 56 && !(sparse && W >= 48);
    }
    if (!cm) {
        if (b == 8) {
            if (sparse) return W < 24 && (per_sm <= 56 || W < 4);
            return W < 32 ? per_sm <= 224 || W > 2 : W < 64 && W % 4 != 0;
        }
        if (b == 4) {
            if (sparse) return W <= 24 && per_sm <= 56;
            return W <= 24 && (per_sm <= 112 || W >= 8);
        }
        if (own) return W <= 24;
        if (b == 3) return sparse ? W < 24 && per_sm <= 56 : W <= 24 && per_sm <= 112;
        return per_sm <= 56 && W <= (per_sm <= 8 && !sparse ? 24 : b == 5 ? 8 : sparse ? 8 : 16);
    }
    if (b == 4 && sparse) return W <= 16 && per_sm <= 56;
    if (own) return W <= 16 && (per_sm <= 224 || W >= 8);
    if (b == 3) return W <= 16 && per_sm <= (sparse ? 56 : 112);
    if (b == 8) return per_sm <= 56 && W <= (per_sm <= 8 ? 16 : per_sm <= 32 ? 12 : 6);
    if (b == 5) return per_sm <= 56 && W <= (per_sm <= 32 ? 16 : 6);
    return W <= 16 && per_sm <= 32;
}

}  // namespace step_detail
}  // namespace rsatb_b200
