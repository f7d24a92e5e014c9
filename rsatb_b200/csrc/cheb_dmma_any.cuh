// Fused Chebyshev step on the FP64 tensor cores for the shapes cheb_dmma.cuh
// has no tiling for: any block size b = 2 to 8, any panel width, real and
// complex block values, FP64 panels and FP32 panels widened on load.
//
// mma.sync m8n8k4 f64 tiles, one block row (and up to 8 NG panel columns) per
// warp.  The contraction index runs over the whole block row, k' = (block,
// column of the block), in steps of 4, so blocks of 5 waste no K lanes: lane
// fc of a step takes k' = 4 s + fc, whatever block that falls in.  Output rows
// beyond b and columns beyond the panel are zero lanes.
//
// A complex block (CM) is the real 2b x 2b block [[Ar, -Ai], [Ai, Ar]] over
// (column, re | im) against the panel's (re, im) rows: M = 2b, K = 2b per
// block and N the complex columns; the (re, im) rows of an output sit in lanes
// 4 apart and are brought together by one shuffle for the epilogue.
//
// U steps are loaded together, unmasked but in a row's last group.  Bound by
// latency at narrow panels (one warp per block row, the loads of U steps in
// flight): 12.6 us for 118,784 blocks of 8 at W <= 8 (61 MB of values), 8.6 us
// for 69,632 blocks of 5; by the FP64 tensor pipe (26.6 TF/s measured for this
// tile) at wide ones.  With the lane's offsets formed at every step and masked
// loads these took 22.8 and 12.6 us, complex blocks of 5 at 6 columns 45 us
// (now 16.8).  Against the kernels it replaces: dmma_any_rule.cuh.
#pragma once

#include "cheb_dmma.cuh"

#include <type_traits>

namespace rsatb_b200 {

constexpr int kDmmaAnyWarps = 4;

// Steps loaded together.  For a compile-time block size U steps are a whole
// number of blocks (KB contraction rows each), so a lane's place inside its
// blocks is the same in every group and its offsets are formed once; B = 0
// (any size) carries the place along.
template <int B, int NG, bool CM>
constexpr int dmma_any_u() {
    return B == 5 ? 5 : B == 8 ? (NG == 1 ? 8 : 4) : NG == 1 ? 8 : NG <= 4 ? 4 : 2;
}

template <typename VT>
__device__ __forceinline__ void load_pair(const VT* p, VT& e, VT& o) {
    if constexpr (sizeof(VT) == 8) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p));
        e = t.x;
        o = t.y;
    } else {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        e = t.x;
        o = t.y;
    }
}

// PAIR (real blocks, even widths, NG even): groups 2p and 2p + 1 take the even
// and the odd columns of a 16-column span, so one 2-value load feeds both.
template <typename VT, int B, int NG, int MT, bool CM, bool CV, bool PAIR>
__global__ void __launch_bounds__(kDmmaAnyWarps * 32, CM ? (NG == 1 ? 5 : NG <= 3 ? 4 : 2)
                                          : NG <= 2 ? (B == 8 ? 7 : 6) : NG <= 4 ? 4 : 3)
    cheb_step_dmma_any(StepArgs a, int n_chunks) {
    static_assert(!CM || CV, "a complex matrix needs a complex panel");
    static_assert(!PAIR || (!CM && NG % 2 == 0), "pairs of column groups");
    constexpr int U = dmma_any_u<B, NG, CM>();
    constexpr int KBC = B ? (CM ? 2 * B : B) : 1;  // KB when known
    static_assert(B == 0 || 4 * U % KBC == 0, "a group is whole blocks");
    extern __shared__ double asm_dots[];  // per warp: dots d0, d1 per real column
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fr = lane >> 2, fc = lane & 3;
    const int b = B ? B : a.block_size, W = a.W;
    const int KB = B ? KBC : CM ? 2 * b : b;  // contraction rows (and output rows) per block
    const int NC = CM ? W / 2 : W;        // tile columns
    const int64_t bb = int64_t(b) * b * (CM ? 2 : 1);
    const VT* __restrict__ vals = static_cast<const VT*>(a.vals);
    const VT* __restrict__ in = static_cast<const VT*>(a.in);
    const int ndots = a.dot_mode == DOT_DOUBLING ? 2 : (a.dot_mode == DOT_PLAIN ? 1 : 0);
    double* dots = asm_dots + warp * 2 * W;
    if (ndots)
        for (int c = lane; c < 2 * W; c += 32) dots[c] = 0.0;
    __syncwarp();

    // This lane's offsets.  Rows beyond KB and columns beyond NC read a valid
    // neighbour instead: an output element depends only on its own row of A and
    // its own column of B, and those outputs are dropped.  For complex blocks
    // the part (re | im) of k' is fc's parity and that of the output row fr's:
    // Ar where they agree, +-Ai where they differ.
    int aoff[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int r = min(8 * m + fr, KB - 1);
        aoff[m] = CM ? (r >> 1) * b * 2 + ((r ^ fc) & 1) : r * b;
    }
    const bool neg = CM && (fc & 1) && !(fr & 1);
    // Known block size: step u of a group sits dk[u] blocks on, at column cu[u].
    int dk[U], ao[U], xo[U];
    if constexpr (B != 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = 4 * u + fc;
            dk[u] = k / KBC;
            const int cu = k - dk[u] * KBC;
            ao[u] = dk[u] * int(bb) + (CM ? (cu & ~1) : cu);
            xo[u] = (CM ? cu >> 1 : cu) * W;
        }
    }

    const int64_t items = a.n_block_rows * n_chunks;
    for (int64_t it = int64_t(blockIdx.x) * kDmmaAnyWarps + warp; it < items;
         it += int64_t(gridDim.x) * kDmmaAnyWarps) {
        const int64_t i = it / n_chunks;
        const int col0 = int(it - i * n_chunks) * 8 * NG;
        const int k0 = __ldg(a.row_ptr + i), k1 = __ldg(a.row_ptr + i + 1);
        int boff[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if constexpr (PAIR)
                boff[g] = min(col0 + 8 * (g & ~1) + 2 * fr, NC - 2) + (g & 1);
            else
                boff[g] = CM ? 2 * min(col0 + 8 * g + fr, NC - 1) + (fc & 1)
                             : min(col0 + 8 * g + fr, NC - 1);
        }
        double acc[NG][MT][2];
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[g][m][0] = acc[g][m][1] = 0.0;
        // This lane's k' = (kk, c); a known block size keeps kk at the group's
        // first block.
        int kk = B ? k0 : k0 + fc / KB, c = B ? 0 : fc % KB;
        const int64_t KT = int64_t(k1 - k0) * KB;
        auto group = [&](auto tail) {
            constexpr bool TAIL = decltype(tail)::value;
            VT ar[U][MT], br[U][NG];
            bool valid[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const VT* blk;
                const VT* xr;
                if constexpr (B != 0) {
                    valid[u] = !TAIL || kk + dk[u] < k1;
                    const int back = TAIL && !valid[u] ? kk + dk[u] - (k1 - 1) : 0;
                    const int64_t j = __ldg(a.col_ind + kk + dk[u] - back);
                    blk = vals + kk * bb + ao[u] - back * bb;
                    xr = in + j * (int64_t(b) * W) + xo[u];
                } else {
                    valid[u] = !TAIL || kk < k1;
                    const int kc = TAIL ? min(kk, k1 - 1) : kk;
                    const int64_t j = __ldg(a.col_ind + kc);
                    blk = vals + int64_t(kc) * bb + (CM ? (c & ~1) : c);
                    xr = in + (j * b + (CM ? c >> 1 : c)) * W;
                    c += 4;
                    // KB >= 2: at most two blocks further
                    const int q = (c >= KB) + (c >= 2 * KB);
                    c -= q * KB;
                    kk += q;
                }
#pragma unroll
                for (int m = 0; m < MT; ++m) ar[u][m] = __ldg(blk + aoff[m]);
#pragma unroll
                for (int g = 0; g < NG; g += PAIR ? 2 : 1) {
                    if constexpr (PAIR)
                        load_pair<VT>(xr + boff[g], br[u][g], br[u][g + 1]);
                    else
                        br[u][g] = __ldg(xr + boff[g]);
                }
            }
            if constexpr (B != 0) kk += 4 * U / KBC;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                double af[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const double v = neg ? -double(ar[u][m]) : double(ar[u][m]);
                    af[m] = valid[u] ? v : 0.0;
                }
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    const double bv = valid[u] ? double(br[u][g]) : 0.0;
#pragma unroll
                    for (int m = 0; m < MT; ++m) dmma_884(acc[g][m], af[m], bv);
                }
            }
        };
        int64_t s = 0;
        for (; s + 4 * U <= KT; s += 4 * U) group(std::false_type());
        if (s < KT) group(std::true_type());
        // Epilogue: lane holds output row fr (of tile m), columns 2 fc + {0, 1}
        // of group g, or (PAIR) 4 fc + {0, 1, 2, 3} of a pair's span.  The panel
        // values of two groups are read before either is finished.
        constexpr int GE = MT == 2 || NG % 2 ? 1 : 2;
        static_assert(NG % GE == 0, "whole batches");
        const bool even = CV || (W & 1) == 0;
#pragma unroll
        for (int gb = 0; gb < NG; gb += GE) {
            VT px[GE][MT][2], pp[GE][MT][2], pq[GE][MT][2], p0[GE][MT][2];
            // First real column of this lane's pair of values in group g, tile m,
            // and its row; false where it holds none.
            const auto place = [&](int g, int m, int64_t& row, int& col) {
                if constexpr (CM) {
                    const int r = 4 * m + (fr >> 1);
                    const int n = col0 + 8 * g + 2 * fc + (fr & 1);
                    row = i * b + r;
                    col = 2 * n;
                    return r < b && n < NC;
                } else {
                    row = i * b + fr;
                    col = PAIR ? col0 + 8 * (g & ~1) + 4 * fc + 2 * (g & 1)
                               : col0 + 8 * g + 2 * fc;
                    return fr < b && col < W;
                }
            };
            if (even) {
#pragma unroll
                for (int e = 0; e < GE; ++e)
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        int64_t row;
                        int col;
                        if (!place(gb + e, m, row, col)) continue;
                        const int64_t off = row * W + col;
                        if (a.x) load_vals<VT, 2>(static_cast<const VT*>(a.x) + off, px[e][m]);
                        if (a.p) load_vals<VT, 2>(static_cast<const VT*>(a.p) + off, pp[e][m]);
                        if (a.q) load_vals<VT, 2>(static_cast<const VT*>(a.q) + off, pq[e][m]);
                        if (ndots == 1)
                            load_vals<VT, 2>(static_cast<const VT*>(a.psi0) + off, p0[e][m]);
                    }
            }
#pragma unroll
            for (int e = 0; e < GE; ++e) {
                const int g = gb + e;
                double e0[2] = {0, 0}, e1[2] = {0, 0};
                int col = 0;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    int64_t row;
                    const bool mine = place(g, m, row, col);
                    VT out[2];
                    if constexpr (CM) {
                        // Even rows are real parts, odd rows imaginary: an even
                        // lane row finishes complex column 2 fc, its partner 2 fc + 1.
                        const int odd = fr & 1;
                        const double own = odd ? acc[g][m][1] : acc[g][m][0];
                        const double send = odd ? acc[g][m][0] : acc[g][m][1];
                        const double got = __shfl_xor_sync(0xffffffffu, send, 4);
                        out[0] = VT(odd ? got : own);
                        out[1] = VT(odd ? own : got);
                    } else if constexpr (PAIR) {
                        out[0] = VT(acc[g & ~1][0][g & 1]);
                        out[1] = VT(acc[g | 1][0][g & 1]);
                    } else {
                        out[0] = VT(acc[g][0][0]);
                        out[1] = VT(acc[g][0][1]);
                    }
                    if (!mine) continue;
                    if (even) {
                        // A null x still counts as read (finish_row looks at a.x).
                        finish_row<VT, 2, CV>(a, row, col / 2, out, e0, e1, px[e][m], pp[e][m],
                                              pq[e][m], p0[e][m]);
                    } else if constexpr (!CV) {  // odd width: one column at a time
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            const VT o1[1] = {out[v]};
                            double f0[1] = {0}, f1[1] = {0};
                            if (col + v < W) finish_row<VT, 1, false>(a, row, col + v, o1, f0, f1);
                            e0[v] = f0[0];
                            e1[v] = f1[0];
                        }
                    }
                }
                if (ndots) {
                    // The rows of a column sit fr apart (complex: fr of one parity).
#pragma unroll
                    for (int o = CM ? 8 : 4; o < 32; o <<= 1)
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            e0[v] += __shfl_xor_sync(0xffffffffu, e0[v], o);
                            if (ndots == 2) e1[v] += __shfl_xor_sync(0xffffffffu, e1[v], o);
                        }
                    if (fr < (CM ? 2 : 1))
#pragma unroll
                        for (int v = 0; v < 2; ++v)
                            if (col + v < W) {
                                dots[col + v] += e0[v];
                                dots[W + col + v] += e1[v];
                            }
                }
            }
        }
        __syncwarp();
    }
    if (ndots) {
        __syncthreads();
        double* mine = a.partials + size_t(blockIdx.x) * ndots * W;
        for (int idx = threadIdx.x; idx < ndots * W; idx += blockDim.x) {
            const int d = idx / W, col = idx - d * W;
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kDmmaAnyWarps; ++w) s += asm_dots[w * 2 * W + d * W + col];
            mine[idx] = s;
        }
        // Two levels and sixteen loads at every size: the kernel's main loop is
        // scheduled 15 % slower with the other form behind it (blocks of 5, complex,
        // 4,096 rows, 6 columns 20.8 against 24.3 us).
        finish_partials<16, 0>(a, ndots);
    }
}

}  // namespace rsatb_b200
