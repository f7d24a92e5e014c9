// Fused BSR SpMM + Chebyshev step + FP64 column dots.
//
// One launch computes, for every row of the N x W output panel,
//
//     y = s2 * (((s_in * (A in)) - c * x) * s_out) + g_p * p [+ g_q * q]
//
// which covers BlockSpMat::mult_dense (s_in = alpha, no x, no p), the
// rescaled operator of Chebyshev::apply_form (rsatb/calc/cheby.hpp:555-591:
// y = A x; y -= c x; y *= 1/hw) and the recurrence t2 = 2 Op~ t1 - t0
// (rsatb/calc/dos.hpp:169-170), and accumulates in FP64 the per-column dots
// the KPM loop takes right after each step (dos.hpp:156-162):
//
//     DOT_DOUBLING   <y|x>, <y|y>      (the doubled recurrence)
//     DOT_PLAIN      <psi0|y>          (the plain recurrence)
//
// with <a|b> = sum_i conj(a_i) b_i per column.
//
// Layout: the panel is row-major with W real values per row (W = R for a
// real multivector, 2R for a complex one, (re, im) interleaved).  A thread
// owns V consecutive values of one block row; L = W / V threads share a
// block row and the CTA holds a whole number of such groups, so a
// grid-stride loop keeps each thread on the same columns and its dot partial sums stay in
// registers until one CTA-level reduction at the end.  The CTA partials go
// to global memory and the last CTA to finish sums them in CTA order, so the
// dots are deterministic for a given launch shape.
#pragma once

#include "common.cuh"

namespace rsatb_b200 {

enum DotMode { DOT_NONE = 0, DOT_DOUBLING = 1, DOT_PLAIN = 2 };

struct StepArgs {
    int64_t n_block_rows;
    const int32_t* row_ptr;
    const int32_t* col_ind;
    const void* vals;
    int block_size;    // runtime block size (generic kernel)
    int W;             // real values per row
    const void* in;    // SpMM operand
    const void* x;     // -c*x term and <y|x> partner (null: none)
    const void* p;     // recurrence predecessor (null: none)
    const void* psi0;  // DOT_PLAIN partner
    const void* q;     // optional extra term g_q * q (null: none)
    void* y;
    double s_in, c, s_out, s2, g_p, g_q;
    int imag;          // A = i * vals (real values, complex panel)
    int dot_mode;
    double* partials;  // [gridDim.x][ndots][W]
    double* dots_out;  // [ndots][W]
    unsigned* counter;
    unsigned* fault;   // set non-zero by a kernel whose bounded wait gave up (null: none)
    void* ax;          // optional sum over the recurrence, ax += (ax_re + i ax_im) y, by the
                       // kernels that take it (step_takes_ax); null: none
    double ax_re, ax_im;
    int ax_init;       // ax starts here as (ax0_re + i ax0_im) x instead of its contents
    double ax0_re, ax0_im;
    int wait_check;    // non-zero: the bulk-copy kernel only runs a wait that cannot
                       // complete (a 5 ms limit), to check the fault report
};

// Loads of V consecutive values.  CG = false: the read-only data path
// (__ldg), for data no thread of the launch writes; CG = true: L2-coherent
// loads (__ldcg), for data written earlier in the same launch.
template <typename T, bool CG>
__device__ __forceinline__ T ld_path(const T* p) {
    if constexpr (CG) return __ldcg(p);
    else return __ldg(p);
}

template <typename VT, int V, bool CG = false>
__device__ __forceinline__ void load_vals(const VT* __restrict__ p, VT (&o)[V]) {
    if constexpr (sizeof(VT) == 8 && V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
            const double2 t = ld_path<double2, CG>(reinterpret_cast<const double2*>(p) + i);
            o[2 * i] = t.x;
            o[2 * i + 1] = t.y;
        }
    } else if constexpr (sizeof(VT) == 4 && V % 4 == 0) {
#pragma unroll
        for (int i = 0; i < V / 4; ++i) {
            const float4 t = ld_path<float4, CG>(reinterpret_cast<const float4*>(p) + i);
            o[4 * i] = t.x;
            o[4 * i + 1] = t.y;
            o[4 * i + 2] = t.z;
            o[4 * i + 3] = t.w;
        }
    } else if constexpr (sizeof(VT) == 4 && V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
            const float2 t = ld_path<float2, CG>(reinterpret_cast<const float2*>(p) + i);
            o[2 * i] = t.x;
            o[2 * i + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) o[i] = ld_path<VT, CG>(p + i);
    }
}

template <typename VT, int V>
__device__ __forceinline__ void store_vals(VT* __restrict__ p, const VT (&o)[V]) {
    if constexpr (sizeof(VT) == 8 && V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            reinterpret_cast<double2*>(p)[i] = make_double2(o[2 * i], o[2 * i + 1]);
    } else if constexpr (sizeof(VT) == 4 && V % 4 == 0) {
#pragma unroll
        for (int i = 0; i < V / 4; ++i)
            reinterpret_cast<float4*>(p)[i] =
                make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
    } else if constexpr (sizeof(VT) == 4 && V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            reinterpret_cast<float2*>(p)[i] = make_float2(o[2 * i], o[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) p[i] = o[i];
    }
}

// (d0, d1) += a * (b0, b1): one packed FP32 FMA (fma.rn.f32x2, sm_100),
// each lane an IEEE fused multiply-add, so the results equal two fmaf.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a, float b0, float b1) {
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %2};\n\t"
        "mov.b64 rb, {%3, %4};\n\t"
        "mov.b64 rd, {%0, %1};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rd;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "+f"(d0), "+f"(d1)
        : "f"(a), "f"(b0), "f"(b1));
}

// acc[v] += a * x[v] for v < V; FP32 with V even as packed pairs.
template <typename VT, int V>
__device__ __forceinline__ void fma_row(VT (&acc)[V], VT a, const VT (&x)[V]) {
    if constexpr (sizeof(VT) == 4 && V % 2 == 0) {
#pragma unroll
        for (int v = 0; v < V; v += 2) fma2(acc[v], acc[v + 1], a, x[v], x[v + 1]);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = fma(a, x[v], acc[v]);
    }
}

// ax += c y for V values of one row in FP64, rounded once a term as the separate
// launch rounds (the start c0 x too); a real panel takes Re(c).
template <typename VT, int V, bool CV>
__device__ __forceinline__ void add_ax(const StepArgs& a, int64_t off, const VT (&xv)[V],
                                       const VT (&yv)[V]) {
    VT* o = static_cast<VT*>(a.ax) + off;
    VT s[V];
    const auto mul = [](double re, double im, const VT (&z)[V], int v) {
        if constexpr (CV)
            return v & 1 ? re * double(z[v]) + im * double(z[v - 1])
                         : re * double(z[v]) - im * double(z[v + 1]);
        else
            return re * double(z[v]);
    };
    if (a.ax_init) {
#pragma unroll
        for (int v = 0; v < V; ++v) s[v] = VT(mul(a.ax0_re, a.ax0_im, xv, v));
    } else {
        load_vals<VT, V, true>(o, s);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) s[v] = VT(double(s[v]) + mul(a.ax_re, a.ax_im, yv, v));
    store_vals<VT, V>(o, s);
}

// Epilogue for one output row: rescale, recurrence, store, dots.  CG: the
// x, p, q and psi0 panels are read through L2 (written earlier in the same
// launch).  px, pp, pq, p0: the x, p, q and psi0 values where the caller has read
// them already (so that their latency runs beside other work: the branches here
// keep the loads of one row's groups from overlapping).
template <typename VT, int V, bool CV, bool CG = false, bool AX = false>
__device__ __forceinline__ void finish_row(const StepArgs& a, int64_t row, int g,
                                           const VT (&acc)[V], double (&d0)[V],
                                           double (&d1)[V], const VT* px = nullptr,
                                           const VT* pp = nullptr, const VT* pq = nullptr,
                                           const VT* p0 = nullptr) {
    const int64_t off = row * a.W + int64_t(g) * V;
    double t[V];
#pragma unroll
    for (int v = 0; v < V; ++v) t[v] = double(acc[v]);
    if (CV && a.imag) {
        // (i * W) applied: (re, im) -> (-im, re)
#pragma unroll
        for (int v = 0; v < V; v += 2) {
            const double re = t[v];
            t[v] = -t[v + 1];
            t[v + 1] = re;
        }
    }
    VT xv[V];
    if (px) {
#pragma unroll
        for (int v = 0; v < V; ++v) xv[v] = px[v];
    } else if (a.x) {
        load_vals<VT, V, CG>(static_cast<const VT*>(a.x) + off, xv);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v) xv[v] = VT(0);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        double u = t[v] * a.s_in;
        if (a.x) u = fma(-a.c, double(xv[v]), u);
        t[v] = u * a.s_out;
    }
    if (a.p) {
        VT pv[V];
        if (pp) {
#pragma unroll
            for (int v = 0; v < V; ++v) pv[v] = pp[v];
        } else {
            load_vals<VT, V, CG>(static_cast<const VT*>(a.p) + off, pv);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] = fma(a.s2, t[v], a.g_p * double(pv[v]));
    } else if (a.s2 != 1.0) {
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] *= a.s2;
    }
    if (a.q) {
        VT qv[V];
        if (pq) {
#pragma unroll
            for (int v = 0; v < V; ++v) qv[v] = pq[v];
        } else {
            load_vals<VT, V, CG>(static_cast<const VT*>(a.q) + off, qv);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] = fma(a.g_q, double(qv[v]), t[v]);
    }
    VT yv[V];
#pragma unroll
    for (int v = 0; v < V; ++v) yv[v] = VT(t[v]);
    store_vals<VT, V>(static_cast<VT*>(a.y) + off, yv);
    if constexpr (AX) {
        if (a.ax) add_ax<VT, V, CV>(a, off, xv, yv);
    }

    if (a.dot_mode == DOT_DOUBLING) {
        // <y|x> and <y|y>, from the stored (rounded) y.
        if constexpr (CV) {
#pragma unroll
            for (int v = 0; v < V; v += 2) {
                const double yr = double(yv[v]), yi = double(yv[v + 1]);
                const double xr = double(xv[v]), xi = double(xv[v + 1]);
                d0[v] += yr * xr + yi * xi;
                d0[v + 1] += yr * xi - yi * xr;
                d1[v] += yr * yr + yi * yi;
            }
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const double yr = double(yv[v]);
                d0[v] += yr * double(xv[v]);
                d1[v] += yr * yr;
            }
        }
    } else if (a.dot_mode == DOT_PLAIN) {
        VT qv[V];
        if (p0) {
#pragma unroll
            for (int v = 0; v < V; ++v) qv[v] = p0[v];
        } else {
            load_vals<VT, V, CG>(static_cast<const VT*>(a.psi0) + off, qv);
        }
        if constexpr (CV) {
#pragma unroll
            for (int v = 0; v < V; v += 2) {
                const double qr = double(qv[v]), qi = double(qv[v + 1]);
                const double yr = double(yv[v]), yi = double(yv[v + 1]);
                d0[v] += qr * yr + qi * yi;
                d0[v + 1] += qr * yi - qi * yr;
            }
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) d0[v] += double(qv[v]) * double(yv[v]);
        }
    }
}

// dst[o] = sum of n partial vectors of O values at P, P + step, ... (elements):
// T = blockDim / O threads share an output where there are more threads than
// outputs, their sums combined in part order; otherwise each thread takes whole
// outputs.  NL loads in flight per thread (sixteen cost most kernels registers and
// with them CTAs per SM); a fixed order.  dst may be the first vector.  All the
// CTA's threads (at most 256) call it.
template <int NL = 8>
__device__ __forceinline__ void sum_partials(const double* P, int n, size_t step, int O,
                                             double* dst) {
    __shared__ double comb[256];
    const int nt = blockDim.x;
    const int T = max(1, nt / O);  // threads per output
    const int part = T > 1 ? threadIdx.x / O : 0;
    for (int o = T > 1 ? threadIdx.x % O : threadIdx.x; o < O; o += T > 1 ? O : nt) {
        double sum = 0.0;
        if (part < T)
            for (int b = part; b < n; b += NL * T) {
                double v[NL];
#pragma unroll
                for (int u = 0; u < NL; ++u)
                    v[u] = b + u * T < n ? __ldcg(P + size_t(b + u * T) * step + o) : 0.0;
#pragma unroll
                for (int h = NL / 2; h > 0; h >>= 1)
#pragma unroll
                    for (int u = 0; u < h; ++u) v[u] += v[u + h];
                sum += v[0];
            }
        if (T > 1)
            comb[threadIdx.x] = sum;
        else
            dst[o] = sum;
    }
    if (T > 1) {
        __syncthreads();
        if (threadIdx.x < O) {
            double t = 0.0;
            for (int q = 0; q < T; ++q) t += comb[q * O + threadIdx.x];
            dst[threadIdx.x] = t;
        }
    }
}

// After every CTA wrote its partial dots: the last CTA to arrive (ticket
// counters) sums them over the CTAs.  In two levels where a thread of that CTA
// would have more than two rounds of loads (kOneLevel): the last of every 32 CTAs
// sums its group's partials in place of the group's first, the last of those sums
// the groups.  The sums sit on the step's critical path as a chain of L2 round
// trips: at 1,024 CTAs of 24 outputs the step takes 34 us with one level, 24 with
// both (17 without dots); FP64 blocks of 8 at W = 32 58.9 -> 47.7, W = 16 38.0 ->
// 30.0; but at 128 CTAs of 16 outputs 8.7 us with one level and 10.4 with two.  The
// order is fixed for a given grid: deterministic dots.  Resets the counters for the
// next launch.  Needs blockDim.x <= 256.
constexpr int kGroupCtas = 32;
constexpr int kOneLevel = 16;       // values a thread sums alone at most
constexpr int kGroupCounter0 = 8;   // the groups' counters: counter[8 + group]
constexpr int kMaxGroups = 48;      // the fault word lies beyond them
template <int NL = 8, int ONE = kOneLevel>
__device__ __forceinline__ void finish_partials(const StepArgs& a, int ndots) {
    __threadfence();
    __syncthreads();
    __shared__ unsigned ticket;
    const int O = ndots * a.W;
    const int G = int(gridDim.x);
    int n = G;
    size_t step = O;
    const int groups = (G + kGroupCtas - 1) / kGroupCtas;
    if ((ONE ? G * O > ONE * int(blockDim.x) : groups > 1) && groups <= kMaxGroups) {
        const int group = blockIdx.x / kGroupCtas;
        const int size = min(kGroupCtas, G - group * kGroupCtas);
        unsigned* gc = a.counter + kGroupCounter0 + group;
        if (threadIdx.x == 0) ticket = atomicAdd(gc, 1u);
        __syncthreads();
        if (ticket != unsigned(size - 1)) return;
        __threadfence();
        if (threadIdx.x == 0) *gc = 0u;
        double* P = a.partials + size_t(group) * kGroupCtas * O;
        sum_partials<NL>(P, size, O, O, P);
        n = groups;
        step = size_t(kGroupCtas) * O;
        __threadfence();
        __syncthreads();
    }
    if (threadIdx.x == 0) ticket = atomicAdd(a.counter, 1u);
    __syncthreads();
    if (ticket != unsigned(n - 1)) return;
    __threadfence();
    sum_partials<NL>(a.partials, n, step, O, a.dots_out);
    if (threadIdx.x == 0) *a.counter = 0u;  // ready for the next launch
}

// CTA reduction of the per-thread dot partials, then the last-CTA
// reduction over CTAs.  Deterministic: fixed summation order throughout.
template <int V>
__device__ __forceinline__ void reduce_dots(const StepArgs& a, int L, const double (&d0)[V],
                                            const double (&d1)[V]) {
    extern __shared__ double red[];  // [ndots][blockDim.x][V]
    const int ndots = (a.dot_mode == DOT_DOUBLING) ? 2 : 1;
    const int nt = blockDim.x;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        red[threadIdx.x * V + v] = d0[v];
        if (ndots == 2) red[(nt + threadIdx.x) * V + v] = d1[v];
    }
    __syncthreads();
    const int W = a.W;
    double* mine = a.partials + size_t(blockIdx.x) * ndots * W;
    for (int idx = threadIdx.x; idx < ndots * W; idx += nt) {
        const int d = idx / W, w = idx - d * W;
        const int g = w / V, v = w - g * V;
        double s = 0.0;
        for (int t = g; t < nt; t += L) s += red[(d * nt + t) * V + v];
        mine[idx] = s;
    }
    finish_partials(a, ndots);
}

// CTAs per SM that the register kernel is compiled for (0: the compiler's choice).
// Without it a few registers more or less, from any code after the main loop, move
// the occupancy: scalar rows at 33 nonzeros and FP32 blocks of 8 went from 219 to
// 357 us and from 102 to 153 us an application that way.
template <typename VT, int B, int V, int AX>
constexpr int step_min_ctas() {
    constexpr bool d = sizeof(VT) == 8;
    if (AX == 2) return 3;
    if (B == 1) return V == 1 ? (d ? 6 : 5) : V == 2 ? 5 : V == 4 ? (d ? 4 : 0) : d ? 3 : 4;
    if (B == 5) return V == 1 ? 5 : V == 2 ? 4 : V == 4 ? (d ? 2 : 3) : d ? 1 : 2;
    return V == 1 ? 4 : V == 2 ? (d ? 2 : 3) : V == 4 ? (d ? 1 : 2) : 1;
}

// Compile-time block size B.  MT: real component type of the matrix values;
// CM: complex matrix values; CV: complex panel; AX (scalar rows): 1 adds into
// StepArgs::ax, 2 reads x, p and four nonzeros ahead too.
template <typename VT, typename MT, int B, int V, bool CM, bool CV, int AX = 0>
__global__ void __launch_bounds__(256, step_min_ctas<VT, B, V, AX>())
    cheb_step_kernel(StepArgs a) {
    static_assert(!AX || B == 1, "the sum is added at scalar rows");
    static_assert(!CM || CV, "a complex matrix needs a complex panel");
    static_assert(!CV || V % 2 == 0, "complex panels need (re, im) pairs per thread");
    const int L = a.W / V;
    const int g = threadIdx.x % L;
    const int64_t total = a.n_block_rows * L;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    const MT* __restrict__ vals = static_cast<const MT*>(a.vals);
    const VT* __restrict__ in = static_cast<const VT*>(a.in);
    constexpr int BB = B * B * (CM ? 2 : 1);

    double d0[V], d1[V];
#pragma unroll
    for (int v = 0; v < V; ++v) d0[v] = d1[v] = 0.0;

    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total; t += stride) {
        const int64_t i = t / L;
        VT acc[B][V];
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
            for (int v = 0; v < V; ++v) acc[r][v] = VT(0);
        const int k0 = __ldg(a.row_ptr + i), k1 = __ldg(a.row_ptr + i + 1);
        if constexpr (AX == 2) {
            // x and p first, then four nonzeros in flight.
            const int64_t off = i * a.W + int64_t(g) * V;
            VT xv[V], pv[V];
#pragma unroll
            for (int v = 0; v < V; ++v) xv[v] = pv[v] = VT(0);
            if (a.x) load_vals<VT, V>(static_cast<const VT*>(a.x) + off, xv);
            if (a.p) load_vals<VT, V>(static_cast<const VT*>(a.p) + off, pv);
            const VT* X = in + int64_t(g) * V;
            int k = k0;
            for (; k + 4 <= k1; k += 4) {
                int j[4];
                MT w[4];
                VT xb[4][V];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    j[u] = __ldg(a.col_ind + k + u);
                    w[u] = __ldg(vals + k + u);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) load_vals<VT, V>(X + int64_t(j[u]) * a.W, xb[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) fma_row<VT, V>(acc[0], VT(w[u]), xb[u]);
            }
            if (k < k1) {  // one to three left: clamped loads, guarded sums
                int j[3];
                MT w[3];
                VT xb[3][V];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const int kc = min(k + u, k1 - 1);
                    j[u] = __ldg(a.col_ind + kc);
                    w[u] = __ldg(vals + kc);
                }
#pragma unroll
                for (int u = 0; u < 3; ++u) load_vals<VT, V>(X + int64_t(j[u]) * a.W, xb[u]);
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (k + u < k1) fma_row<VT, V>(acc[0], VT(w[u]), xb[u]);
            }
            finish_row<VT, V, CV, false, true>(a, i, g, acc[0], d0, d1, xv, pv);
            continue;
        }
        for (int k = k0; k < k1; ++k) {
            const int64_t j = __ldg(a.col_ind + k);
            // X_j: B rows x V values of this thread's columns.
            VT xb[B][V];
#pragma unroll
            for (int c = 0; c < B; ++c)
                load_vals<VT, V>(in + (j * B + c) * a.W + int64_t(g) * V, xb[c]);
            const MT* blk = vals + int64_t(k) * BB;
            constexpr int RW = B * (CM ? 2 : 1);  // values per block row
#pragma unroll
            for (int r = 0; r < B; ++r) {
                MT arow[RW];
                load_vals<MT, RW>(blk + r * RW, arow);
#pragma unroll
                for (int c = 0; c < B; ++c) {
                    if constexpr (CM) {
                        const VT ar = VT(arow[2 * c]);
                        const VT ai = VT(arow[2 * c + 1]);
#pragma unroll
                        for (int v = 0; v < V; v += 2) {
                            acc[r][v] = fma(ar, xb[c][v], acc[r][v]);
                            acc[r][v] = fma(-ai, xb[c][v + 1], acc[r][v]);
                            acc[r][v + 1] = fma(ar, xb[c][v + 1], acc[r][v + 1]);
                            acc[r][v + 1] = fma(ai, xb[c][v], acc[r][v + 1]);
                        }
                    } else {
                        fma_row<VT, V>(acc[r], VT(arow[c]), xb[c]);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < B; ++r)
            finish_row<VT, V, CV, false, AX != 0>(a, i * B + r, g, acc[r], d0, d1);
    }
    if (a.dot_mode != DOT_NONE) reduce_dots<V>(a, L, d0, d1);
}

// Whether a step on A adds into StepArgs::ax: the register kernel of scalar
// rows does (its default), where the separate launch that reads the step's
// output back was a third of a term (us a term in two launches and in one: 80,000
// rows of 4 nonzeros, 4 FP64 complex columns 12.7, 10.3; 64 99.8, 83; 300,000 rows
// of 33, 32 FP32 complex columns 268, 260).
bool step_takes_ax(const rsatb_bsr_matrix* A);

// Runtime block size (b <= 16): the fallback for block sizes without a
// specialisation.  Same arithmetic, rows of the block handled one at a time.
template <typename VT, typename MT, int V, bool CM, bool CV>
__global__ void __launch_bounds__(256, sizeof(VT) == 8 && !CV ? 4 : 5)
    cheb_step_kernel_any_b(StepArgs a) {
    const int L = a.W / V;
    const int g = threadIdx.x % L;
    const int B = a.block_size;
    const int64_t total = a.n_block_rows * L;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    const MT* __restrict__ vals = static_cast<const MT*>(a.vals);
    const VT* __restrict__ in = static_cast<const VT*>(a.in);
    const int BB = B * B * (CM ? 2 : 1);

    double d0[V], d1[V];
#pragma unroll
    for (int v = 0; v < V; ++v) d0[v] = d1[v] = 0.0;

    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total; t += stride) {
        const int64_t i = t / L;
        const int k0 = __ldg(a.row_ptr + i), k1 = __ldg(a.row_ptr + i + 1);
        for (int r = 0; r < B; ++r) {
            VT acc[V];
#pragma unroll
            for (int v = 0; v < V; ++v) acc[v] = VT(0);
            for (int k = k0; k < k1; ++k) {
                const int64_t j = __ldg(a.col_ind + k);
                const MT* blk = vals + int64_t(k) * BB;
                for (int c = 0; c < B; ++c) {
                    VT xv[V];
                    load_vals<VT, V>(in + (j * B + c) * a.W + int64_t(g) * V, xv);
                    if constexpr (CM) {
                        const VT ar = VT(__ldg(blk + 2 * (r * B + c)));
                        const VT ai = VT(__ldg(blk + 2 * (r * B + c) + 1));
#pragma unroll
                        for (int v = 0; v < V; v += 2) {
                            acc[v] = fma(ar, xv[v], acc[v]);
                            acc[v] = fma(-ai, xv[v + 1], acc[v]);
                            acc[v + 1] = fma(ar, xv[v + 1], acc[v + 1]);
                            acc[v + 1] = fma(ai, xv[v], acc[v + 1]);
                        }
                    } else {
                        const VT av = VT(__ldg(blk + r * B + c));
#pragma unroll
                        for (int v = 0; v < V; ++v) acc[v] = fma(av, xv[v], acc[v]);
                    }
                }
            }
            finish_row<VT, V, CV>(a, i * B + r, g, acc, d0, d1);
        }
    }
    if (a.dot_mode != DOT_NONE) reduce_dots<V>(a, L, d0, d1);
}

// Per-column <a|b> over n_rows rows (mu_0 = <psi|psi>), same reduction.
template <typename VT, int V, bool CV>
__global__ void __launch_bounds__(256) coldot_kernel(StepArgs a) {
    const int L = a.W / V;
    const int g = threadIdx.x % L;
    const int64_t total = a.n_block_rows * L;  // here: scalar rows
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    double d0[V], d1[V];
#pragma unroll
    for (int v = 0; v < V; ++v) d0[v] = d1[v] = 0.0;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total; t += stride) {
        const int64_t row = t / L;
        const int64_t off = row * a.W + int64_t(g) * V;
        VT av[V], bv[V];
        load_vals<VT, V>(static_cast<const VT*>(a.x) + off, av);
        load_vals<VT, V>(static_cast<const VT*>(a.in) + off, bv);
        if constexpr (CV) {
#pragma unroll
            for (int v = 0; v < V; v += 2) {
                const double ar = double(av[v]), ai = double(av[v + 1]);
                const double br = double(bv[v]), bi = double(bv[v + 1]);
                d0[v] += ar * br + ai * bi;
                d0[v + 1] += ar * bi - ai * br;
            }
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) d0[v] += double(av[v]) * double(bv[v]);
        }
    }
    reduce_dots<V>(a, L, d0, d1);
}

// Launch entries for one fused step, defined per precision in
// cheb_step_f64.cu / cheb_step_f32.cu.
int launch_cheb_step_f64(rsatb_context* ctx, const rsatb_bsr_matrix* A, int vec_dtype,
                         StepArgs args);
int launch_cheb_step_f32(rsatb_context* ctx, const rsatb_bsr_matrix* A, int vec_dtype,
                         StepArgs args);
int launch_coldot_f64(rsatb_context* ctx, int vec_dtype, int64_t n_rows, StepArgs args);
int launch_coldot_f32(rsatb_context* ctx, int vec_dtype, int64_t n_rows, StepArgs args);

}  // namespace rsatb_b200
