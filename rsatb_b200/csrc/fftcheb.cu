// FFT-Chebyshev Kubo-Greenwood transport on the device: the
// dc_spectrum_fftcheb / accumulate_fftcheb_block path of
// rsatb/calc/fftcheb_transport.hpp:270-660, Greenwood and Bastin formulations.
//
// Per sample block (all R samples at once) and per section of rows:
//   left chain   l_m = T_m(Op~) psi,          stored as J_a l_m for a = x, y, z
//   right chains r_m^a = T_m(Op~) J_a psi,    stored as they are
// with J_a = -(1 / 2 hw) V_a (current, rsatb/calc/ac.hpp:35-60, through
// Chebyshev::apply_dual, cheby.hpp:249-291), then per row, axis and sample
// the DCT-III of (g_m / pi) x_m (fft.hpp:125-154) for both chains and the
// contraction K_k += sum conj(L3_k) R3_k / max(1e-14, 1 - eps_k^2)
// (fftcheb_transport.hpp:481-495).
//
// B200 layout (the reference's per-row FFTW layout is not kept):
// * scalar rows with velocities on H's pattern: all four chains in one panel
//   and one launch per moment (moment_kernel); otherwise the three right chains
//   are one N x 3R panel ([row][axis][sample]), so a moment is one wide fused
//   step for them, one narrow one for l, three current SpMMs and a store copy;
// * the stores are moment-major, S[m][axis][row][sample], so every moment's
//   rows land with coalesced writes;
// * the DCT-III of a chunk of rows is a strided batched inverse M-point
//   FFT (cuFFT, sequences interleaved: stride = batch) of dct3_input_kernel's
//   sequences, built and read back with coalesced accesses;
// * the contraction gives each energy k to one CTA per chunk: no atomics,
//   the same summation order on every run;
// * at M = 256, 512, 1024 and 2048 (Greenwood) the row stage is one
//   hand-written kernel after a coalesced gather: transform and contraction
//   without a transform buffer's round trips (greenwood_fused_kernel).
#include "cheb_kernels.cuh"
#include "fftcheb_partition.cuh"

#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <type_traits>
#include <vector>

namespace rsatb_b200 {

int run_step(rsatb_context* ctx, const rsatb_bsr_matrix* A, int vdt, const StepArgs& a);
void kpm_kernel_weights(int kernel, int n, double* g);

namespace {

#define RSATB_CUFFT_TRY(call)                                                              \
    do {                                                                                   \
        cufftResult r_ = (call);                                                           \
        if (r_ != CUFFT_SUCCESS)                                                           \
            return set_error(RSATB_CUDA_ERROR, "%s failed (cufftResult %d)", #call, int(r_)); \
    } while (0)

// Right-chain panel from the three J_a psi buffers: P[row][a][s] = J[a][row][s].
template <typename T>
__global__ void pack_axes_kernel(int64_t n_rows, int R, const T* j0, const T* j1, const T* j2,
                                 T* panel) {
    const int64_t total = n_rows * 3 * R;  // complex entries
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int s = int(e % R);
        const int a = int((e / R) % 3);
        const int64_t row = e / (3 * int64_t(R));
        const T* src = a == 0 ? j0 : (a == 1 ? j1 : j2);
        panel[2 * e] = src[2 * (row * R + s)];
        panel[2 * e + 1] = src[2 * (row * R + s) + 1];
    }
}

// Rows [row0, row0 + rows) of the right panel into store slot m:
// S[m][a][row][s] (complex entries), slot size 3 * rows * R.
template <typename T>
__global__ void store_right_kernel(int64_t row0, int64_t rows, int R, const T* panel, T* slot) {
    const int64_t total = rows * 3 * R;
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
         e += int64_t(gridDim.x) * blockDim.x) {
        // e indexes the destination: a-major
        const int s = int(e % R);
        const int64_t row = (e / R) % rows;
        const int a = int(e / (rows * R));
        const int64_t src = ((row0 + row) * 3 + a) * R + s;
        slot[2 * e] = panel[2 * src];
        slot[2 * e + 1] = panel[2 * src + 1];
    }
}

// The same copy in 16-byte units: the R samples of one (row, axis) are one
// contiguous run in both layouts, of 2 R sizeof(T) / 16 units (R even for
// FP32; every run, slot and panel then starts on a 16-byte boundary).
template <typename T>
__global__ void store_right_vec_kernel(int64_t row0, int64_t rows, int R, const T* panel,
                                       T* slot) {
    const int upr = int(2 * R * sizeof(T) / 16);  // units per run
    const int64_t total = rows * 3 * upr;
    const float4* src = reinterpret_cast<const float4*>(panel);
    float4* dst = reinterpret_cast<float4*>(slot);
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int u = int(e % upr);
        const int64_t run = e / upr;  // destination run a * rows + row
        const int64_t row = run % rows;
        const int a = int(run / rows);
        dst[e] = src[((row0 + row) * 3 + a) * upr + u];
    }
}

// ---------------------------------------------------------------------------
// One moment of both chains in one launch, for scalar rows whose H, Vx, Vy and
// Vz share a pattern (H real, V_a = i W_a): the route of the orthogonal form
// of pz operators at a real k-point.
//
// The chains live in one panel of 4 W1 reals per row, [row][l, r^x, r^y,
// r^z][sample], so a nonzero pulls one contiguous run of its neighbour's row,
// and the four matrices' values sit together ({h, w_x, w_y, w_z} per nonzero,
// one vector load).  A launch reads moment m (cur) and
//   writes the currents J_a l_m of the section's rows to the left store,
//   copies the section's r^a_m to the right store,
//   replaces moment m - 1 (prev) by moment m + 1 of every row:
//     y = 2 (Op cur - c cur) / hw - prev   (without the 2 and prev at m = 0),
// the arithmetic of finish_row (products and sums over the nonzeros in the
// vectors' precision and in pattern order, rescale and recurrence in FP64), so
// its results equal those of the separate launches.
//
// A thread owns V consecutive reals of one row (16 bytes where the sample
// count allows, always whole complex values of one chain); C = 4 W1 / V
// threads share a row.  A CTA's rows are consecutive, so its nonzeros' values
// and indices are one contiguous run, staged in shared memory: read per thread
// they were a serial chain of first touches (110 us per moment against 75.8 at
// 47,632 rows of 33 nonzeros, 16 FP32 samples), and only the gathered rows are
// left to wait for.  Bound by the latency of those (512 bytes per nonzero, 55 %
// L1 hits at 11,908 rows), 32 warps x 4 loads per SM.  The six launches this replaces (left
// step, right step, three currents, store copy) took 141 us; 11,536 rows x 5
// FP64 samples: 18.7 us against 51.
template <typename T>
struct MomentArgs {
    int64_t n_rows, row0, row1;  // all rows; the section's rows [row0, row1)
    const int32_t* row_ptr;
    const int32_t* col_ind;
    const T* wgt;                // 4 values per nonzero
    const T* cur;
    T* prev;
    T* sl;                       // this moment's slots of the left and right store
    T* sr;
    int W1;                      // reals per row and chain (2 R)
    int C;                       // threads per row
    int cap;                     // nonzeros staged per pass
    int advance;                 // form moment m + 1
    double c, inv_hw, s2, g_p;   // g_p == 0: no predecessor
    double cscale;               // -1 / (2 hw)
};

// Evict-first stores: a moment's store rows are next read by the row stage,
// after every other moment.
template <typename T, int V>
__device__ __forceinline__ void store_stream(T* p, const T (&o)[V]) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            __stcs(reinterpret_cast<double2*>(p) + i, make_double2(o[2 * i], o[2 * i + 1]));
    } else if constexpr (V % 4 == 0) {
#pragma unroll
        for (int i = 0; i < V / 4; ++i)
            __stcs(reinterpret_cast<float4*>(p) + i,
                   make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]));
    } else {
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            __stcs(reinterpret_cast<float2*>(p) + i, make_float2(o[2 * i], o[2 * i + 1]));
    }
}

constexpr int kMomentCap = 640;

template <typename T> struct Vec4;
template <> struct Vec4<float> {
    static __device__ __forceinline__ void load(const float* p, float (&w)[4]) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
    }
};
template <> struct Vec4<double> {
    static __device__ __forceinline__ void load(const double* p, double (&w)[4]) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p));
        const double2 u = __ldg(reinterpret_cast<const double2*>(p) + 1);
        w[0] = t.x; w[1] = t.y; w[2] = u.x; w[3] = u.y;
    }
};

template <typename T, int V, int U, int MINB>
__global__ void __launch_bounds__(256, MINB) moment_kernel(MomentArgs<T> a) {
    extern __shared__ __align__(16) unsigned char msm_raw[];
    T* sw = reinterpret_cast<T*>(msm_raw);                        // [cap][4]
    int32_t* sj = reinterpret_cast<int32_t*>(sw + 4 * a.cap);     // [cap]
    const int C = a.C;
    const int lr = threadIdx.x / C, ch = threadIdx.x - lr * C;
    const int64_t i0 = int64_t(blockIdx.x) * (blockDim.x / C);
    const int64_t i = i0 + lr;
    const bool live = i < a.n_rows;
    const bool left = ch < C / 4;
    const bool in_sec = live && i >= a.row0 && i < a.row1;
    const bool cur_ax = left && in_sec;  // this thread forms currents
    const int PW = 4 * a.W1;
    const T* X = a.cur + ch * V;
    T acc[V], cx[3][V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = cx[0][v] = cx[1][v] = cx[2][v] = T(0);
    const int64_t i1 = min(i0 + blockDim.x / C, a.n_rows);
    const int kb = __ldg(a.row_ptr + i0), ke = __ldg(a.row_ptr + i1);
    const int k0 = live ? __ldg(a.row_ptr + i) : ke;
    const int k1 = live ? __ldg(a.row_ptr + i + 1) : ke;
    // The CTA's nonzeros (consecutive in the pattern) come to shared memory in
    // passes of cap, coalesced; one pass unless a row is longer than cap.
    for (int base = kb; base < ke; base += a.cap) {
        const int m = min(a.cap, ke - base);
        if (base != kb) __syncthreads();
        for (int t = threadIdx.x; t < m; t += blockDim.x) {
            T w[4];
            Vec4<T>::load(a.wgt + 4 * (int64_t(base) + t), w);
            sj[t] = __ldg(a.col_ind + base + t);
            store_vals<T, 4>(sw + 4 * t, w);
        }
        __syncthreads();
        int k = max(k0, base) - base;
        const int kn = min(k1, base + m) - base;
        for (; k + U <= kn; k += U) {
            T x[U][V];
#pragma unroll
            for (int u = 0; u < U; ++u) load_vals<T, V>(X + int64_t(sj[k + u]) * PW, x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const T* w = sw + 4 * (k + u);
                fma_row<T, V>(acc, w[0], x[u]);
                if (cur_ax) {
#pragma unroll
                    for (int q = 0; q < 3; ++q) fma_row<T, V>(cx[q], w[q + 1], x[u]);
                }
            }
        }
        if (k < kn) {  // the last, short group: clamped loads, guarded sums
            T x[U][V];
#pragma unroll
            for (int u = 0; u < U; ++u)
                load_vals<T, V>(X + int64_t(sj[min(k + u, kn - 1)]) * PW, x[u]);
#pragma unroll
            for (int u = 0; u < U - 1; ++u)
                if (k + u < kn) {
                    const T* w = sw + 4 * (k + u);
                    fma_row<T, V>(acc, w[0], x[u]);
                    if (cur_ax) {
#pragma unroll
                        for (int q = 0; q < 3; ++q) fma_row<T, V>(cx[q], w[q + 1], x[u]);
                    }
                }
        }
    }
    if (!live) return;
    T xv[V];
    load_vals<T, V>(X + i * PW, xv);
    if (in_sec) {
        const int64_t rows = a.row1 - a.row0;
        if (left) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                T o[V];
#pragma unroll
                for (int v = 0; v < V; v += 2) {  // i times the real sums
                    o[v] = T(-double(cx[q][v + 1]) * a.cscale);
                    o[v + 1] = T(double(cx[q][v]) * a.cscale);
                }
                store_stream<T, V>(a.sl + (q * rows + (i - a.row0)) * a.W1 + ch * V, o);
            }
        } else {
            const int q = ch / (C / 4) - 1, e = (ch - (q + 1) * (C / 4)) * V;
            store_stream<T, V>(a.sr + (q * rows + (i - a.row0)) * a.W1 + e, xv);
        }
    }
    if (!a.advance) return;
    T* P = a.prev + i * PW + ch * V;
    T y[V];
    if (a.g_p != 0.0) {
#pragma unroll
        for (int v = 0; v < V; ++v) y[v] = P[v];
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        double t = fma(-a.c, double(xv[v]), double(acc[v])) * a.inv_hw;
        if (a.g_p != 0.0) t = fma(a.s2, t, a.g_p * double(y[v]));
        y[v] = T(t);
    }
    store_vals<T, V>(P, y);
}

// The start of the panel: l_0 = psi, r^a_0 = J_a psi; one thread per (row, sample).
template <typename T>
__global__ void moment_init_kernel(int64_t n_rows, int R, const int32_t* row_ptr,
                                   const int32_t* col_ind, const T* wgt, const T* psi,
                                   double cscale, T* panel) {
    const int64_t total = n_rows * R;
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = e / R;
        const int s = int(e - i * R);
        T cx[3][2] = {{0, 0}, {0, 0}, {0, 0}};
        for (int k = __ldg(row_ptr + i), k1 = __ldg(row_ptr + i + 1); k < k1; ++k) {
            T w[4], x[2];
            load_vals<T, 2>(psi + 2 * (int64_t(__ldg(col_ind + k)) * R + s), x);
            Vec4<T>::load(wgt + 4 * int64_t(k), w);
#pragma unroll
            for (int q = 0; q < 3; ++q) fma_row<T, 2>(cx[q], w[q + 1], x);
        }
        T* out = panel + i * 8 * R + 2 * s;
        out[0] = psi[2 * e];
        out[1] = psi[2 * e + 1];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            out[2 * (q + 1) * R] = T(-double(cx[q][1]) * cscale);
            out[2 * (q + 1) * R + 1] = T(double(cx[q][0]) * cscale);
        }
    }
}

// {h, w_x, w_y, w_z} per nonzero.
template <typename T>
__global__ void pack_weights_kernel(int64_t nnz, const T* h, const T* wx, const T* wy,
                                    const T* wz, T* wgt) {
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < nnz;
         e += int64_t(gridDim.x) * blockDim.x) {
        const T v[4] = {h[e], wx[e], wy[e], wz[e]};
        store_vals<T, 4>(wgt + 4 * e, v);
    }
}

// *differs becomes non-zero when a velocity's pattern is not H's (the caller then
// keeps the separate launches).
__global__ void compare_patterns_kernel(int64_t n_rows, int64_t nnz, const int32_t* rp,
                                        const int32_t* ci, const int32_t* rpx,
                                        const int32_t* cix, const int32_t* rpy,
                                        const int32_t* ciy, const int32_t* rpz,
                                        const int32_t* ciz, int* differs) {
    bool bad = false;
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < nnz;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int32_t j = ci[e];
        bad |= cix[e] != j || ciy[e] != j || ciz[e] != j;
    }
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e <= n_rows;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int32_t r = rp[e];
        bad |= rpx[e] != r || rpy[e] != r || rpz[e] != r;
    }
    if (bad) *differs = 1;
}

// Input of the M-point transform that gives the DCT-III of fft.hpp:125-154
//   y_k = w_0 x_0 + 2 sum_{m >= 1} w_m x_m cos(pi m (k + 1/2) / M)
// for a chunk of sequences: sequence q (0 <= q < nq, q = (a * chunk_rows + row)
// * R + s, rows offset row_off inside the section) of store S (slot stride
// slot_elems complex entries, section rows sec_rows) weighted by w_m.
//   F_0 = w_0 x_0,  F_m = e^{i pi m / 2M} (w_m x_m - i w_{M-m} x_{M-m}),
// whose inverse DFT v_p = sum_m F_m e^{2 pi i m p / M} holds y in the order of
// dct3_energy (Makhoul, IEEE Trans. ASSP 28, 27, 1980; linear in x, so complex
// x is two real transforms at once): half the points and half the buffer of
// the even extension's 2M-point transform.  One thread reads x_m and x_{M-m}
// and writes F_m and F_{M-m}; blockIdx.y is m <= M / 2.
__host__ __device__ inline int dct3_energy(int M, int p) {
    return p < (M + 1) / 2 ? 2 * p : 2 * (M - 1 - p) + 1;
}

template <typename T>
__global__ void dct3_input_kernel(int M, int64_t nq, int chunk_rows, int R, int64_t sec_rows,
                                  int64_t row_off, int64_t slot_elems, const T* S,
                                  const double* w, double2* F) {
    const int m = blockIdx.y, mm = M - m;
    double c, sn;
    sincospi(double(m) / (2.0 * double(M)), &sn, &c);
    const double wm = w[m], wr = m ? w[mm] : 0.0;
    for (int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; q < nq;
         q += int64_t(gridDim.x) * blockDim.x) {
        const int s = int(q % R);
        const int64_t row = (q / R) % chunk_rows;
        const int a = int(q / (int64_t(chunk_rows) * R));
        const int64_t src = (a * sec_rows + row_off + row) * R + s;
        const T* p = S + 2 * (int64_t(m) * slot_elems + src);
        const double xr = wm * double(p[0]), xi = wm * double(p[1]);
        if (m == 0) {
            F[q] = make_double2(xr, xi);
            continue;
        }
        const T* pr = S + 2 * (int64_t(mm) * slot_elems + src);
        const double zr = wr * double(pr[0]), zi = wr * double(pr[1]);
        // x - i z, times (c + i sn)
        const double ar = xr + zi, ai = xi - zr;
        F[int64_t(m) * nq + q] = make_double2(ar * c - ai * sn, ar * sn + ai * c);
        if (mm != m) {
            // z - i x, times e^{i pi (M - m) / 2M} = sn + i c
            const double br = zr + xi, bi = zi - xr;
            F[int64_t(mm) * nq + q] = make_double2(br * sn - bi * c, br * c + bi * sn);
        }
    }
}

// Bastin phi1 / phi2 inputs (fftcheb_transport.hpp:453-461, fft.hpp:156-174):
// the weighted moments w[m] S_m (complex w) in the first M points of a
// 2M-point sequence, zeros in the last M; [point][sequence], the sequences in
// dct3_input_kernel's order.
template <typename T>
__global__ void pad_kernel(int M, int64_t nq, int chunk_rows, int R, int64_t sec_rows,
                           int64_t row_off, int64_t slot_elems, const T* S, const double2* w,
                           double2* E) {
    const int m = blockIdx.y;
    const double2 wm = w[m];
    for (int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; q < nq;
         q += int64_t(gridDim.x) * blockDim.x) {
        const int s = int(q % R);
        const int64_t row = (q / R) % chunk_rows;
        const int a = int(q / (int64_t(chunk_rows) * R));
        const int64_t src = int64_t(m) * slot_elems + (a * sec_rows + row_off + row) * R + s;
        const double xr = double(S[2 * src]), xi = double(S[2 * src + 1]);
        E[int64_t(m) * nq + q] = make_double2(wm.x * xr - wm.y * xi, wm.x * xi + wm.y * xr);
        E[int64_t(M + m) * nq + q] = make_double2(0.0, 0.0);
    }
}

// Bastin kernel accumulation (fftcheb_transport.hpp:496-519), phi3 (the DCT-III)
// taken from phi1's transform: its angles are theta_k = pi (k + 1/2) / M and
// theta_{2M-1-k} = 2 pi - theta_k, so phi3_k = (phi1_k + phi1_{2M-1-k}) / 2.
// For energy k
// (one CTA) and every component (a, b), a <= b,
//   K[k][ab] += sum over rows, samples of
//     eps_k (conj(L3_a) R1_b + conj(L1_a) R3_b)
//     + i sqrt(1 - eps_k^2) (conj(L2_a) R3_b - conj(L3_a) R2_b),
// summed per thread, then in a fixed tree order (deterministic).
__global__ void __launch_bounds__(256) bastin_contract_kernel(int M, int64_t nq, int64_t per_axis,
                                                              const double2* L1, const double2* R1,
                                                              const double2* L2, const double2* R2,
                                                              double* K) {
    const int k = blockIdx.x;
    const double th = M_PI * (double(k) + 0.5) / double(M);
    const double eps = cos(th), root = sin(th);
    __shared__ double red[12][256];
    double acc[6][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}};
    const int64_t o = int64_t(k) * nq, o2 = int64_t(2 * M - 1 - k) * nq;
    const auto half_sum = [](double2 x, double2 y) {
        return make_double2(0.5 * (x.x + y.x), 0.5 * (x.y + y.y));
    };
    // conj(x) y, accumulated into (re, im)
    auto cmac = [](double (&d)[2], double2 x, double2 y, double f_re, double f_im) {
        const double re = x.x * y.x + x.y * y.y, im = x.x * y.y - x.y * y.x;
        d[0] += f_re * re - f_im * im;
        d[1] += f_re * im + f_im * re;
    };
    for (int64_t q = threadIdx.x; q < per_axis; q += blockDim.x) {
        int comp = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double2 l1 = L1[o + a * per_axis + q], l2 = L2[o + a * per_axis + q];
            const double2 l3 = half_sum(l1, L1[o2 + a * per_axis + q]);
#pragma unroll
            for (int b = a; b < 3; ++b, ++comp) {
                const double2 r1 = R1[o + b * per_axis + q], r2 = R2[o + b * per_axis + q];
                const double2 r3 = half_sum(r1, R1[o2 + b * per_axis + q]);
                cmac(acc[comp], l3, r1, eps, 0.0);
                cmac(acc[comp], l1, r3, eps, 0.0);
                cmac(acc[comp], l2, r3, 0.0, root);
                cmac(acc[comp], l3, r2, 0.0, -root);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        red[2 * c][threadIdx.x] = acc[c][0];
        red[2 * c + 1][threadIdx.x] = acc[c][1];
    }
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int c = 0; c < 12; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 12) K[int64_t(k) * 12 + threadIdx.x] += red[threadIdx.x][0];
}

// K[k][a] += sum over the chunk's (row, s) of conj(L3[k][q]) R3[k][q] /
// max(1e-14, 1 - eps_k^2): one CTA per transform output p (energy
// dct3_energy(M, p)), fixed order.
__global__ void __launch_bounds__(256) greenwood_contract_kernel(int M, int64_t nq,
                                                                 int64_t per_axis,
                                                                 const double2* L3,
                                                                 const double2* R3,
                                                                 double* K) {
    const int k = dct3_energy(M, blockIdx.x);
    const double eps = cos(M_PI * (double(k) + 0.5) / double(M));
    const double wden = 1.0 - eps * eps;
    const double inv = 1.0 / (wden > 1e-14 ? wden : 1e-14);
    __shared__ double red[3][2][256];
    double acc[3][2] = {{0, 0}, {0, 0}, {0, 0}};
    const double2* l = L3 + int64_t(blockIdx.x) * nq;
    const double2* r = R3 + int64_t(blockIdx.x) * nq;
    for (int a = 0; a < 3; ++a)
        for (int64_t q = threadIdx.x; q < per_axis; q += blockDim.x) {
            const double2 x = l[a * per_axis + q], y = r[a * per_axis + q];
            acc[a][0] += x.x * y.x + x.y * y.y;
            acc[a][1] += x.x * y.y - x.y * y.x;
        }
    for (int a = 0; a < 3; ++a) {
        red[a][0][threadIdx.x] = acc[a][0];
        red[a][1][threadIdx.x] = acc[a][1];
    }
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int a = 0; a < 3; ++a) {
                red[a][0][threadIdx.x] += red[a][0][threadIdx.x + w];
                red[a][1][threadIdx.x] += red[a][1][threadIdx.x + w];
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int a = 0; a < 3; ++a) {
            // components xx, yy, zz of the 6-component tensor (xx xy xz yy yz zz)
            const int comp = a == 0 ? 0 : (a == 1 ? 3 : 5);
            K[2 * (int64_t(k) * 6 + comp)] += red[a][0][0] * inv;
            K[2 * (int64_t(k) * 6 + comp) + 1] += red[a][1][0] * inv;
        }
}

// ---------------------------------------------------------------------------
// Fused Greenwood row stage for M = 256, 512, 1024 and 2048: the DCT-III as the
// M-point transform of dct3_input_kernel's sequence and the contraction in one
// kernel, so no transform input or output goes through HBM.  The transform
// runs in FP64, but for FP32 vectors at M = 2048 in FP32; the products
// conj(L3) R3 and their sums are FP64 in both.
//
// M = 16 x 16 x r (n = n0 + r n1 + 16 r n2, k = k0 + 16 k1 + 256 k2, n0, k2 < r,
// w = e^{2 pi i / M}); 16 r threads hold a sequence, 16 values each:
//   pass A  thread n' = n0 + r n1: 16-point DFT over n2 -> k0, times w^{n' k0}
//   pass B  thread (n0, k0): 16-point DFT over n1 -> k1, times w^{16 n0 k1}
//   pass C  thread's 16 / r pairs (k1, k0): r-point DFT over n0 -> k2
// exchanged through shared memory.  Strides between A and B: 17 r entries per
// k0 (16 r written by consecutive lanes, read r at a time at a step of r);
// between B and C: 16 r + 1 per k1 (written by consecutive lanes, read at a
// stride of 1 modulo the banks).  Pass A forms
//   F_n = ph_n x_n + conj(ph_{M-n}) x_{M-n},  F_0 = ph_0 x_0,
//   ph_m = w_m e^{i pi m / 2M},
// as it loads.  A CTA of 256 threads holds 8 / r pairs of a left and a right
// sequence side by side; after pass C the two swap halves of their outputs, so
// each thread accumulates conj(L3_k) R3_k for 8 energies in FP64 over the CTA's
// pairs (a fixed grid-stride order); fused_reduce_kernel sums the partials in a
// fixed order, so results do not depend on timing.
//
// Half the points of the even extension's 2M: half the work, in registers for
// two CTAs per SM.  8,192 pairs of 2048 moments: FP32 119 us against 176 with the
// extended transform.  At 512 and 1024 moments it replaces cuFFT's two passes
// over HBM per side.  Bound by shared memory and issue.
//
// The store is moment-major (each moment's rows written coalesced by the
// recurrence), so one sequence is M values 8 or 16 bytes apiece at a stride
// of the slot size; gather_sequences_kernel first turns a chunk of consecutive
// sequences into sequence-major rows with a tiled transpose (both sides
// coalesced), from which pass A reads contiguous values.
constexpr int kFusedThreads = 256;

// r for a moment count the fused stage serves, else 0.
inline int fused_radix(int M) {
    return M == 256 || M == 512 || M == 1024 || M == 2048 ? M / 256 : 0;
}
// Exchange entries of one sequence; pairs of sequences per CTA; partial sums.
__host__ __device__ constexpr int fused_xch(int r) { return 16 * (16 * r + r); }
__host__ __device__ constexpr int fused_pairs(int r) { return 8 / r; }
// Tables: w^j (j < M / 4), ph (M), and pass B's w^{16 n0 k1} at n0 * 17 + k1.
__host__ __device__ constexpr int fused_tab(int r) { return 64 * r + 256 * r + 17 * r; }
// Shared memory: exchange, tables.
template <typename C>
size_t fused_smem(int r) {
    return size_t(2 * fused_pairs(r) * fused_xch(r) + fused_tab(r)) * sizeof(C);
}

// Complex arithmetic on float2 (FP32 transform) and double2 (FP64 transform).
template <typename C> struct Cx;
template <> struct Cx<float2> {
    using S = float;
    __device__ static float2 make(float x, float y) { return make_float2(x, y); }
};
template <> struct Cx<double2> {
    using S = double;
    __device__ static double2 make(double x, double y) { return make_double2(x, y); }
};
template <typename C>
__device__ __forceinline__ C c_add(C a, C b) {
    return Cx<C>::make(a.x + b.x, a.y + b.y);
}
template <typename C>
__device__ __forceinline__ C c_sub(C a, C b) {
    return Cx<C>::make(a.x - b.x, a.y - b.y);
}
template <typename C>
__device__ __forceinline__ C c_mul(C a, C b) {
    return Cx<C>::make(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C>
__device__ __forceinline__ C c_mul_i(C a) {
    return Cx<C>::make(-a.y, a.x);
}

// out[k] = sum_j in[j] i^{jk}, k = 0..3, in place.
template <typename C>
__device__ __forceinline__ void dft4_inv(C& a0, C& a1, C& a2, C& a3) {
    const C s02 = c_add(a0, a2), d02 = c_sub(a0, a2);
    const C s13 = c_add(a1, a3), d13 = c_mul_i(c_sub(a1, a3));
    a0 = c_add(s02, s13);
    a2 = c_sub(s02, s13);
    a1 = c_add(d02, d13);
    a3 = c_sub(d02, d13);
}

// 16-point DFT with the + sign, in place, as 4 x 4: j = j0 + 4 j1,
// k = c + 4 r.  Output k sits at v[4 (k % 4) + k / 4] (dft16_at).
template <typename C>
__device__ __forceinline__ void dft16_inv(C (&v)[16]) {
    using S = typename Cx<C>::S;
    constexpr S c8 = S(0.92387953251128674);  // cos(pi / 8)
    constexpr S s8 = S(0.38268343236508978);  // sin(pi / 8)
    constexpr S r2 = S(0.70710678118654752);  // cos(pi / 4)
#pragma unroll
    for (int j0 = 0; j0 < 4; ++j0) dft4_inv(v[j0], v[j0 + 4], v[j0 + 8], v[j0 + 12]);
    // v[j0 + 4 c] *= e^{2 pi i j0 c / 16}
    v[1 + 4] = c_mul(v[1 + 4], Cx<C>::make(c8, s8));     // 1
    v[2 + 4] = c_mul(v[2 + 4], Cx<C>::make(r2, r2));     // 2
    v[3 + 4] = c_mul(v[3 + 4], Cx<C>::make(s8, c8));     // 3
    v[1 + 8] = c_mul(v[1 + 8], Cx<C>::make(r2, r2));     // 2
    v[2 + 8] = c_mul_i(v[2 + 8]);                        // 4
    v[3 + 8] = c_mul(v[3 + 8], Cx<C>::make(-r2, r2));    // 6
    v[1 + 12] = c_mul(v[1 + 12], Cx<C>::make(s8, c8));   // 3
    v[2 + 12] = c_mul(v[2 + 12], Cx<C>::make(-r2, r2));  // 6
    v[3 + 12] = c_mul(v[3 + 12], Cx<C>::make(-c8, -s8)); // 9
#pragma unroll
    for (int c = 0; c < 4; ++c) dft4_inv(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}
__device__ __forceinline__ int dft16_at(int k) { return 4 * (k & 3) + (k >> 2); }

// r-point DFT with the + sign, r <= 16, natural order out.
template <typename C, int r>
__device__ __forceinline__ void dft_r_inv(C (&v)[r]) {
    if constexpr (r == 2) {
        const C t = c_sub(v[0], v[1]);
        v[0] = c_add(v[0], v[1]);
        v[1] = t;
    } else if constexpr (r == 4) {
        dft4_inv(v[0], v[1], v[2], v[3]);
    } else if constexpr (r == 8) {
        using S = typename Cx<C>::S;
        constexpr S r2 = S(0.70710678118654752);  // cos(pi / 4)
        C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft4_inv(e[0], e[1], e[2], e[3]);
        dft4_inv(o[0], o[1], o[2], o[3]);
        o[1] = c_mul(o[1], Cx<C>::make(r2, r2));
        o[2] = c_mul_i(o[2]);
        o[3] = c_mul(o[3], Cx<C>::make(-r2, r2));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = c_add(e[k], o[k]);
            v[k + 4] = c_sub(e[k], o[k]);
        }
    }
}

// w^n = e^{2 pi i n / M} from the quarter table q[j] = w^j, j < M / 4.
template <typename C, int M>
__device__ __forceinline__ C twiddle(const C* q, int n) {
    const C b = q[n & (M / 4 - 1)];
    switch ((n / (M / 4)) & 3) {
        case 0: return b;
        case 1: return Cx<C>::make(-b.y, b.x);
        case 2: return Cx<C>::make(-b.x, -b.y);
        default: return Cx<C>::make(b.y, -b.x);
    }
}

// The powers b^k, k = 0..15, of a twiddle b as b4^(k / 4) b^(k % 4), from b
// and b4 = b^4 (two reads of the quarter table, whose strided lanes would
// otherwise conflict on the shared-memory banks sixteen at a time): at most
// four roundings more than a table entry.
template <typename C>
struct Pow16 {
    C lo[4], hi[4];
    __device__ __forceinline__ Pow16(C b, C b4) {
        lo[0] = hi[0] = Cx<C>::make(1, 0);
        lo[1] = b;
        lo[2] = c_mul(b, b);
        lo[3] = c_mul(lo[2], b);
        hi[1] = b4;
        hi[2] = c_mul(b4, b4);
        hi[3] = c_mul(hi[2], b4);
    }
    __device__ __forceinline__ C operator()(int k) const {
        if (k < 4) return lo[k];
        if ((k & 3) == 0) return hi[k >> 2];
        return c_mul(hi[k >> 2], lo[k & 3]);
    }
};

// Element e of a store as the transform's complex type.
template <typename C>
__device__ __forceinline__ C load_c(const float* S, int64_t e) {
    const float2 f = __ldg(reinterpret_cast<const float2*>(S) + e);
    return Cx<C>::make(typename Cx<C>::S(f.x), typename Cx<C>::S(f.y));
}
template <typename C>
__device__ __forceinline__ C load_c(const double* S, int64_t e) {
    const double2 f = __ldg(reinterpret_cast<const double2*>(S) + e);
    return Cx<C>::make(typename Cx<C>::S(f.x), typename Cx<C>::S(f.y));
}

// The 16 outputs of thread t of a sequence whose element m is S[m]: out[j r +
// k2] is p = k0 + 16 k1 + 256 k2 for the pair 16 k0 + k1 = t + 16 r j.  All the
// CTA's threads run it together (xch: this sequence's exchange buffer).
template <typename C, int r, typename T>
__device__ __forceinline__ void fused_transform(const T* S, int t, const C* qtw, const C* ph,
                                                const C* wb, C* xch, C (&out)[16]) {
    constexpr int M = 256 * r, TPS = 16 * r;
    C v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int n = t + TPS * j;
        C f = c_mul(ph[n], load_c<C>(S, n));
        if (n != 0) {
            const C p = ph[M - n];
            f = c_add(f, c_mul(Cx<C>::make(p.x, -p.y), load_c<C>(S, M - n)));
        }
        v[j] = f;
    }
    dft16_inv(v);
    {
        const Pow16<C> tw(twiddle<C, M>(qtw, t), twiddle<C, M>(qtw, 4 * t));  // w^{n' k0}
#pragma unroll
        for (int k0 = 0; k0 < 16; ++k0) xch[k0 * 17 * r + t] = c_mul(v[dft16_at(k0)], tw(k0));
    }
    __syncthreads();
    const int n0 = t % r, kb0 = t / r;
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = xch[kb0 * 17 * r + n0 + r * n1];
    dft16_inv(v);
    __syncthreads();
    if constexpr (r > 1) {
        // Read, not formed as powers: a pass-B factor multiplies 16 r outputs of the
        // sequence alike, so its rounding adds up in the sums of products (FP32, 2048
        // moments, 16 samples of 47,632 rows: sigma off by 1.50e-7 with powers).
        xch[t] = v[dft16_at(0)];
#pragma unroll
        for (int k1 = 1; k1 < 16; ++k1)
            xch[k1 * (16 * r + 1) + t] = c_mul(v[dft16_at(k1)], wb[n0 * 17 + k1]);
    } else {
#pragma unroll
        for (int k1 = 0; k1 < 16; ++k1) xch[k1 * (16 * r + 1) + t] = v[dft16_at(k1)];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16 / r; ++j) {
        const int pi = t + TPS * j, k1 = pi & 15, k0 = pi >> 4;
        C u[r];
#pragma unroll
        for (int q = 0; q < r; ++q) u[q] = xch[k1 * (16 * r + 1) + k0 * r + q];
        dft_r_inv<C, r>(u);
#pragma unroll
        for (int q = 0; q < r; ++q) out[j * r + q] = u[q];
    }
    __syncthreads();  // xch is rewritten
}

// The tables of the transform (fused_tab): w^j, ph_m and pass B's factors.
__global__ void fused_tables_kernel(int M, const double* w, double2* tab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s, c;
    if (i < M / 4) {
        sincospi(2.0 * double(i) / double(M), &s, &c);
        tab[i] = make_double2(c, s);
    } else if (i < M / 4 + M) {
        const int m = i - M / 4;
        sincospi(double(m) / (2.0 * double(M)), &s, &c);  // e^{i pi m / 2M}
        tab[i] = make_double2(w[m] * c, w[m] * s);
    } else if (i < fused_tab(M / 256)) {
        const int e = i - (M / 4 + M);  // w^{16 n0 k1} = e^{2 pi i n0 k1 / 16 r}
        sincospi(double((e / 17) * (e % 17)) / (8.0 * double(M / 256)), &s, &c);
        tab[i] = make_double2(c, s);
    }
}

// Tq[side][i][m] = S_side[m * slot + q0 + i] for i < nqc (complex entries, M a
// multiple of 32): 32 x 32 tiles through shared memory, blockIdx.z the side
// (left, right).
template <typename T>
__global__ void __launch_bounds__(256) gather_sequences_kernel(int M, int64_t q0, int64_t nqc,
                                                               int64_t slot, const T* SL,
                                                               const T* SR, T* Tq) {
    using C = typename std::conditional<std::is_same<T, float>::value, float2, double2>::type;
    __shared__ C tile[32][33];
    const C* S = reinterpret_cast<const C*>(blockIdx.z ? SR : SL);
    C* out = reinterpret_cast<C*>(Tq) + int64_t(blockIdx.z) * nqc * M;
    const int64_t i0 = int64_t(blockIdx.x) * 32;
    const int m0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int m = m0 + ty + 8 * r;
        if (i0 + tx < nqc) tile[ty + 8 * r][tx] = S[int64_t(m) * slot + q0 + i0 + tx];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t i = i0 + ty + 8 * r;
        if (i < nqc) out[i * M + m0 + tx] = tile[tx][ty + 8 * r];
    }
}

// Gathered sequences i < nqc of one chunk (Tq, left then right), transform in
// the precision of C; partial[cta][pair][p] += sum over the pair's sequences of
// conj(L3) R3, the products and the sums in FP64.
template <typename T, typename C, int r>
__global__ void __launch_bounds__(kFusedThreads, 2)
    greenwood_fused_kernel(int64_t nqc, const T* Tq, const double2* tab, double2* partial) {
    constexpr int M = 256 * r, TPS = 16 * r, P = fused_pairs(r);
    extern __shared__ __align__(16) unsigned char fsm_raw[];
    C* xch0 = reinterpret_cast<C*>(fsm_raw);
    C* qtw = xch0 + 2 * P * fused_xch(r);
    C* ph = qtw + M / 4;
    C* wb = ph + M;
    for (int j = threadIdx.x; j < fused_tab(r); j += blockDim.x)
        qtw[j] = Cx<C>::make(typename Cx<C>::S(tab[j].x), typename Cx<C>::S(tab[j].y));
    __syncthreads();
    const int seq = threadIdx.x / TPS, t = threadIdx.x - seq * TPS;
    const int side = seq & 1, pair = seq >> 1;  // left and right side by side
    C* mine = xch0 + seq * fused_xch(r);
    C* other = xch0 + (seq ^ 1) * fused_xch(r);
    double2 acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = make_double2(0.0, 0.0);
    const int64_t step = int64_t(gridDim.x) * P;
    // The same number of rounds for every pair of a CTA (barriers inside);
    // pairs past the end transform the last sequence and add nothing.
    for (int64_t i0 = int64_t(blockIdx.x) * P; i0 < nqc; i0 += step) {
        const int64_t i = i0 + pair;
        const bool live = i < nqc;
        C out[16];
        fused_transform<C, r>(Tq + 2 * (side * nqc + (live ? i : nqc - 1)) * M, t, qtw, ph, wb,
                              mine, out);
        // The left thread gives its outputs 8.. and takes the right's 0..7.
#pragma unroll
        for (int j = 0; j < 8; ++j)
            mine[j * TPS + t] = Cx<C>::make(side ? out[j].x : out[j + 8].x,
                                            side ? out[j].y : out[j + 8].y);
        __syncthreads();
        if (live) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const C o = other[j * TPS + t];
                const double lx = side ? o.x : out[j].x, ly = side ? o.y : out[j].y;
                const double rx = side ? out[j + 8].x : o.x, ry = side ? out[j + 8].y : o.y;
                acc[j].x += lx * rx + ly * ry;  // conj(L3) R3
                acc[j].y += lx * ry - ly * rx;
            }
        }
        __syncthreads();
    }
    double2* p = partial + (int64_t(blockIdx.x) * P + pair) * M;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int o = side ? j + 8 : j;
        const int pi = t + TPS * (o / r), e = (pi >> 4) + 16 * (pi & 15) + 256 * (o % r);
        p[e] = make_double2(p[e].x + acc[j].x, p[e].y + acc[j].y);
    }
}

// K[k][comp] += sum over the n_part partials / max(1e-14, 1 - eps_k^2), one CTA
// per transform output, a fixed order.
__global__ void __launch_bounds__(128) fused_reduce_kernel(int M, int n_part,
                                                           const double2* partial, int comp,
                                                           double* K) {
    __shared__ double2 red[128];
    double re = 0.0, im = 0.0;
    for (int c = threadIdx.x; c < n_part; c += blockDim.x) {
        const double2 p = partial[int64_t(c) * M + blockIdx.x];
        re += p.x;
        im += p.y;
    }
    red[threadIdx.x] = make_double2(re, im);
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[threadIdx.x].x += red[threadIdx.x + w].x;
            red[threadIdx.x].y += red[threadIdx.x + w].y;
        }
        __syncthreads();
    }
    if (threadIdx.x) return;
    const int k = dct3_energy(M, blockIdx.x);
    const double eps = cos(M_PI * (double(k) + 0.5) / double(M));
    const double wden = 1.0 - eps * eps;
    const double inv = 1.0 / (wden > 1e-14 ? wden : 1e-14);
    K[2 * (int64_t(k) * 6 + comp)] += red[0].x * inv;
    K[2 * (int64_t(k) * 6 + comp) + 1] += red[0].y * inv;
}

// One chunk of the fused stage, for the transform's type and radix.
template <typename T, typename C, int r>
int fused_launch(rsatb_context* ctx, int grid, int64_t n, const T* Tq, const double2* tab,
                 double2* partial) {
    RSATB_CUDA_TRY(cudaFuncSetAttribute(greenwood_fused_kernel<T, C, r>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(fused_smem<C>(r))));
    greenwood_fused_kernel<T, C, r>
        <<<grid, kFusedThreads, fused_smem<C>(r), ctx->stream>>>(n, Tq, tab, partial);
    RSATB_LAUNCH_CHECK(ctx);
    return RSATB_SUCCESS;
}

template <typename T, typename C>
int fused_launch_r(rsatb_context* ctx, int r, int grid, int64_t n, const T* Tq,
                   const double2* tab, double2* partial) {
    switch (r) {
        case 1: return fused_launch<T, C, 1>(ctx, grid, n, Tq, tab, partial);
        case 2: return fused_launch<T, C, 2>(ctx, grid, n, Tq, tab, partial);
        case 4: return fused_launch<T, C, 4>(ctx, grid, n, Tq, tab, partial);
        default: return fused_launch<T, C, 8>(ctx, grid, n, Tq, tab, partial);
    }
}

// The fused row stage serves Greenwood at fused_radix's moment counts unless
// RSATB_FFTCHEB_FUSED=0.
bool fused_enabled() {
    const char* s = std::getenv("RSATB_FFTCHEB_FUSED");
    return !(s && s[0] == '0');
}

// RSATB_FFTCHEB_FP64=1: the FP64 transform for FP32 vectors too.
bool fused_fp64_forced() {
    const char* s = std::getenv("RSATB_FFTCHEB_FP64");
    return s && s[0] == '1';
}

// Owning device buffer released on scope exit.
struct DevBuf {
    void* p = nullptr;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    int alloc(size_t bytes) {
        if (bytes == 0) bytes = 16;
        RSATB_CUDA_TRY(cudaMalloc(&p, bytes));
        return RSATB_SUCCESS;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
    }
    template <typename T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

// The context's workspace pool, made at its first use: it keeps what calls give
// back, up to a sixteenth of the device's memory, for the next one.  Memory it
// keeps stays the process's: the driver takes it back for a cudaMalloc or
// cuMemCreate that would fail otherwise, whoever calls it.
constexpr size_t kKeepWorkShare = 16;

int work_pool(rsatb_context* ctx) {
    if (ctx->work_pool) return RSATB_SUCCESS;
    size_t free_b = 0, total_b = 0;
    RSATB_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = ctx->device;
    cudaMemPool_t pool = nullptr;
    RSATB_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = total_b / kKeepWorkShare;
    const cudaError_t e =
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) cudaMemPoolDestroy(pool);
    RSATB_CUDA_TRY(e);
    ctx->work_pool = pool;
    ctx->work_keep = keep;
    return RSATB_SUCCESS;
}

// Bytes the pool holds that no call uses.
int kept_work(rsatb_context* ctx, size_t* bytes) {
    uint64_t held = 0, used = 0;
    *bytes = 0;
    if (!ctx->work_pool) return RSATB_SUCCESS;
    RSATB_CUDA_TRY(
        cudaMemPoolGetAttribute(ctx->work_pool, cudaMemPoolAttrReservedMemCurrent, &held));
    RSATB_CUDA_TRY(cudaMemPoolGetAttribute(ctx->work_pool, cudaMemPoolAttrUsedMemCurrent, &used));
    *bytes = size_t(held - used);
    return RSATB_SUCCESS;
}

// Device memory of one call: every buffer is a piece of one block, an allocation
// released at the end, or the pool's for a context that calls again: from the
// second call in a row of one size on, up to what the pool keeps.  (The block from
// cudaMalloc and its cudaFree take 10 ms at 11 GB, 0.8 ms at 0.3 GB; out of the
// pool microseconds, but 65 and 5 ms where the pool maps it anew, so a single
// call, or calls of ever other sizes, do not go there.)
class Arena {
  public:
    ~Arena() {
        if (!base_) return;
        if (pooled_) {
            cudaFreeAsync(base_, stream_);
            cudaStreamSynchronize(stream_);  // seen as free from here on
        } else {
            cudaFree(base_);
        }
    }
    size_t reserve(size_t bytes) {
        const size_t at = total_;
        total_ += (std::max<size_t>(bytes, 16) + 255) & ~size_t(255);
        return at;
    }
    int commit(rsatb_context* ctx) {
        RSATB_TRY(work_pool(ctx));
        size_t kept = 0;
        RSATB_TRY(kept_work(ctx, &kept));
        const bool pooled = total_ <= ctx->work_keep && (kept || total_ == ctx->work_last);
        ctx->work_last = total_;
        // A kept block too small for this call is not held beside the new one.
        if (kept && (!pooled || kept < total_)) {
            RSATB_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
            RSATB_CUDA_TRY(cudaMemPoolTrimTo(ctx->work_pool, 0));
        }
        void* p = nullptr;
        if (pooled)
            RSATB_CUDA_TRY(cudaMallocFromPoolAsync(&p, total_, ctx->work_pool, ctx->stream));
        else
            RSATB_CUDA_TRY(cudaMalloc(&p, total_));
        pooled_ = pooled;
        stream_ = ctx->stream;
        base_ = static_cast<char*>(p);
        return RSATB_SUCCESS;
    }
    template <typename T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(base_ + offset);
    }

  private:
    size_t total_ = 0;
    char* base_ = nullptr;
    bool pooled_ = false;
    cudaStream_t stream_ = nullptr;
};

// The context's inverse Z2Z plan of `batch` interleaved sequences of n points
// (stride batch), made at its first use; *work is its work area's size.
int fft_plan(rsatb_context* ctx, int n, int64_t batch, cufftHandle* out, size_t* work) {
    for (auto& f : ctx->fft)
        if (f.batch == batch && f.n == n) {
            *out = f.handle;
            *work = f.work;
            return RSATB_SUCCESS;
        }
    auto& f = ctx->fft[ctx->fft_next];
    ctx->fft_next ^= 1;
    if (f.batch) {
        f.batch = 0;
        cufftDestroy(f.handle);
    }
    cufftHandle h = 0;
    RSATB_CUFFT_TRY(cufftCreate(&h));
    size_t w = 0;
    int nn = n;
    cufftResult r = cufftSetAutoAllocation(h, 0);
    if (r == CUFFT_SUCCESS)
        r = cufftMakePlanMany(h, 1, &nn, &nn, int(batch), 1, &nn, int(batch), 1, CUFFT_Z2Z,
                              int(batch), &w);
    if (r != CUFFT_SUCCESS) {
        cufftDestroy(h);
        return set_error(RSATB_CUDA_ERROR, "cufftMakePlanMany failed (cufftResult %d)", int(r));
    }
    f.handle = h;
    f.n = n;
    f.batch = batch;
    f.work = w;
    *out = h;
    *work = w;
    return RSATB_SUCCESS;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

StepArgs plain_args(int W) {
    StepArgs a{};
    a.W = W;
    a.s_in = 1.0;
    a.s_out = 1.0;
    a.s2 = 1.0;
    a.dot_mode = DOT_NONE;
    return a;
}

// Matrix restricted to block rows [b0, b1): row_ptr keeps absolute block
// indices, so values, column indices and the input panel are unchanged and
// output row i of the launch is block row b0 + i.
rsatb_bsr_matrix row_view(const rsatb_bsr_matrix* A, int b0, int b1) {
    rsatb_bsr_matrix v = *A;
    v.row_ptr = A->row_ptr + b0;
    v.n_block_rows = b1 - b0;
    return v;
}

struct Ctx {
    rsatb_context* ctx;
    const rsatb_cheb_op* op;
    bool sandwich;
    int vdt;
};

// out = s2 * (Op in - c in) / hw + g_p * prev (Chebyshev::apply_form and the
// recurrence axpby), W real values per row; u, w: sandwich scratch.
int op_step(const Ctx& c, int W, const void* in, const void* prev, void* out, void* u, void* w,
            double s2, double g_p) {
    StepArgs last = plain_args(W);
    last.x = in;
    last.p = prev;
    last.y = out;
    last.c = c.op->center;
    last.s_out = 1.0 / c.op->half_width;
    last.s2 = s2;
    last.g_p = g_p;
    if (!c.sandwich) {
        last.in = in;
        return run_step(c.ctx, c.op->H, c.vdt, last);
    }
    StepArgs a = plain_args(W);
    a.in = in;
    a.y = u;
    RSATB_TRY(run_step(c.ctx, c.op->Z, c.vdt, a));
    a.in = u;
    a.y = w;
    RSATB_TRY(run_step(c.ctx, c.op->H, c.vdt, a));
    last.in = w;
    return run_step(c.ctx, c.op->ZH, c.vdt, last);
}

// J_a x = -(1 / 2 hw) * (dressed V_a) x on block rows [b0, b1), written
// compactly to out (rows b0.. of the result at out[0..]).  Sandwich: Z^H V Z.
int current_rows(const Ctx& c, const rsatb_bsr_matrix* V, int W, const void* x, void* out,
                 int b0, int b1, void* u, void* w) {
    const double scale = -1.0 / (2.0 * c.op->half_width);
    StepArgs a = plain_args(W);
    if (!c.sandwich) {
        const rsatb_bsr_matrix view = row_view(V, b0, b1);
        a.in = x;
        a.y = out;
        a.s_in = scale;
        return run_step(c.ctx, &view, c.vdt, a);
    }
    a.in = x;
    a.y = u;
    RSATB_TRY(run_step(c.ctx, c.op->Z, c.vdt, a));
    a.in = u;
    a.y = w;
    RSATB_TRY(run_step(c.ctx, V, c.vdt, a));
    const rsatb_bsr_matrix view = row_view(c.op->ZH, b0, b1);
    a.in = w;
    a.y = out;
    a.s_in = scale;
    return run_step(c.ctx, &view, c.vdt, a);
}

unsigned grid_for(int64_t n, int sm) {
    int64_t g = (n + 255) / 256;
    if (g > int64_t(sm) * 16) g = int64_t(sm) * 16;
    return unsigned(g < 1 ? 1 : g);
}

// RSATB_FFTCHEB_MOMENT=0: the separate launches of a moment.
bool moment_enabled() {
    const char* s = std::getenv("RSATB_FFTCHEB_MOMENT");
    return !(s && s[0] == '0');
}

// Threads per row of moment_kernel: 16 bytes each where the samples allow it
// (FP32: an even sample count; FP64: one complex value).
template <typename T>
int moment_threads_per_row(int R) {
    const int v = sizeof(T) == 4 && R % 2 == 0 ? 4 : 2;
    return 8 * R / v;
}

// Orthogonal form, scalar rows, a real H and imaginary-unit velocities with
// as many nonzeros as H; the patterns themselves are compared on the device.
bool moment_matrices_ok(const Ctx& c, const rsatb_bsr_matrix* const* V, int R) {
    const rsatb_bsr_matrix* H = c.op->H;
    const auto real = [](const rsatb_bsr_matrix* A) { return !dtype_is_complex(A->dtype); };
    if (c.sandwich || H->block_size != 1 || !real(H) || (H->flags & RSATB_BSR_IMAGINARY_UNIT))
        return false;
    if (8 * R / (H->dtype == RSATB_F32 && R % 2 == 0 ? 4 : 2) > 256) return false;
    for (int a = 0; a < 3; ++a)
        if (!real(V[a]) || !(V[a]->flags & RSATB_BSR_IMAGINARY_UNIT) ||
            V[a]->nnz_blocks != H->nnz_blocks)
            return false;
    return true;
}

template <typename T>
int fftcheb_impl(const Ctx& c, const rsatb_bsr_matrix* const* V, const T* psi, int R, int M,
                 int formulation, double prefactor, int sections, size_t workspace, int kernel,
                 double* sigma_out, double* energy_out, rsatb_fftcheb_stats* stats) {
    const bool bastin = formulation == 1;
    rsatb_context* ctx = c.ctx;
    cudaStream_t st = ctx->stream;
    const int b = c.op->H->block_size;
    const int nb = c.op->H->n_block_rows;
    const int64_t N = int64_t(nb) * b;
    const int W1 = 2 * R, W3 = 6 * R;  // real values per row: left, right panel
    const size_t cplx = 2 * sizeof(T);

    const size_t fixed = size_t(N) * cplx * (3 * R /*rinit*/ + 3 * 3 * R /*r*/ + 3 * R /*l*/ +
                                      3 * R /*J psi*/ + (c.sandwich ? 2 * 3 * R : 0));
    if (workspace == 0) {
        size_t free_b = 0, total_b = 0, kept = 0;
        RSATB_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
        RSATB_TRY(kept_work(ctx, &kept));  // this call takes it or gives it back
        workspace = (free_b + kept) / 10 * 8;
    }
    // One launch per moment (moment_kernel) where the four matrices allow it
    // and its buffers (two panels, the start, the packed values) are no larger
    // than the separate launches' or small in the workspace, and a section still
    // fits beside them; RSATB_FFTCHEB_MOMENT=0 keeps the separate launches.
    const int radix = bastin ? 0 : fused_radix(M);
    const bool fused = radix && fused_enabled();
    const size_t part_bytes = fused ? fused_pairs(radix) * size_t(M) * sizeof(double2) : 0;
    FftchebSizes sizes{workspace, fixed,      nb, b, R, M, cplx, bastin,
                       part_bytes, ctx->sm_count * 2, sections};
    FftchebPartition part{};
    const int64_t nnz = c.op->H->nnz_blocks;
    const size_t fixed_m =
        size_t(N) * cplx * 3 * 4 * R + 4 * size_t(nnz) * sizeof(T) + sizeof(int) + 256;
    bool one_launch = moment_enabled() && moment_matrices_ok(c, V, R) &&
                      fixed_m <= std::max(fixed, workspace / 8);
    if (one_launch) {
        sizes.fixed = fixed_m;
        one_launch = fftcheb_partition(sizes, &part) == FftchebFit::kFits;
        sizes.fixed = fixed;
    }
    if (one_launch) {
        void* sc = nullptr;
        RSATB_TRY(ctx_scratch(ctx, sizeof(int), &sc));
        int* d_differs = static_cast<int*>(sc);
        RSATB_CUDA_TRY(cudaMemsetAsync(d_differs, 0, sizeof(int), st));
        const rsatb_bsr_matrix* H = c.op->H;
        compare_patterns_kernel<<<grid_for(std::max<int64_t>(nnz, N + 1), ctx->sm_count), 256, 0,
                                  st>>>(N, nnz, H->row_ptr, H->col_ind, V[0]->row_ptr,
                                        V[0]->col_ind, V[1]->row_ptr, V[1]->col_ind,
                                        V[2]->row_ptr, V[2]->col_ind, d_differs);
        RSATB_LAUNCH_CHECK(ctx);
        int differs = 0;
        RSATB_CUDA_TRY(cudaMemcpyAsync(&differs, d_differs, sizeof(int), cudaMemcpyDeviceToHost,
                                       st));
        RSATB_CUDA_TRY(cudaStreamSynchronize(st));
        if (differs)
            one_launch = false;
        else
            sizes.fixed = fixed_m;
    }
    switch (fftcheb_partition(sizes, &part)) {
        case FftchebFit::kNoSection:
            return set_error(
                RSATB_OUT_OF_MEMORY,
                "workspace of %zu bytes holds no section (needs %zu + %zu per block row)",
                workspace, sizes.fixed, fftcheb_store_per_brow(sizes));
        case FftchebFit::kNoRow:
            return set_error(RSATB_OUT_OF_MEMORY,
                             "workspace too small for one block row of stores");
        case FftchebFit::kFits: break;
    }
    const int64_t sec_brows = part.sec_brows, chunk_rows = part.chunk_rows;
    const int n_sections = part.n_sections;

    // Buffers.
    Arena mem;
    const size_t panel = size_t(N) * 8 * R;  // reals of one moment_kernel panel
    const size_t v1 = size_t(N) * R * cplx;  // bytes of one N x R panel
    const int64_t sec_rows_max = sec_brows * b;
    const int64_t slot = 3 * sec_rows_max * R;  // complex entries per moment slot
    const int64_t nq_max = 3 * chunk_rows * R;
    const size_t e_bytes = part.e_bytes;
    const size_t oPan = one_launch ? mem.reserve(2 * panel * sizeof(T)) : 0;
    const size_t oInit = one_launch ? mem.reserve(panel * sizeof(T)) : 0;
    const size_t oWgt = one_launch ? mem.reserve(4 * size_t(nnz) * sizeof(T)) : 0;
    const size_t oJ = one_launch ? 0 : mem.reserve(3 * v1);
    const size_t oRinit = one_launch ? 0 : mem.reserve(3 * v1);
    const size_t oR = one_launch ? 0 : mem.reserve(9 * v1);
    const size_t oL = one_launch ? 0 : mem.reserve(3 * v1);
    const size_t oU = c.sandwich ? mem.reserve(3 * v1) : 0;
    const size_t oW = c.sandwich ? mem.reserve(3 * v1) : 0;
    const size_t oS = mem.reserve(2 * size_t(M) * slot * cplx);
    const size_t oE = mem.reserve(e_bytes);
    const size_t oK = mem.reserve(size_t(M) * 12 * sizeof(double));
    const size_t oWts = mem.reserve(size_t(M) * sizeof(double));
    const size_t oPw = bastin ? mem.reserve(2 * size_t(M) * sizeof(double2)) : 0;
    // Fused row stage: up to two CTAs per SM, partial sums per CTA, pair of sequences
    // and energy; chunks of fused_qc sequences gathered into the transform
    // buffer (sequence-major, both sides).  FP32 vectors take the FP32
    // transform at M = 2048 (FP64 products and sums) unless
    // RSATB_FFTCHEB_FP64=1; every other case the FP64 one.
    const bool fused32 = fused && M == 2048 && std::is_same<T, float>::value &&
                         !fused_fp64_forced();
    const int fused_grid = part.ctas;
    const int n_part = fused ? fused_grid * fused_pairs(radix) : 0;
    const size_t oPart = fused ? mem.reserve(size_t(n_part) * M * sizeof(double2)) : 0;
    const size_t oTab = fused ? mem.reserve(size_t(fused_tab(radix)) * sizeof(double2)) : 0;
    // cuFFT's work area, for the chunk sizes of a full section.
    const int fft_n = bastin ? 2 * M : M;
    size_t fft_work = 0;
    if (!fused) {
        cufftHandle h = 0;
        for (const int64_t r : {sec_rows_max % chunk_rows, chunk_rows}) {
            size_t w = 0;
            if (r) RSATB_TRY(fft_plan(ctx, fft_n, 3 * r * R, &h, &w));
            fft_work = std::max(fft_work, w);
        }
    }
    const size_t oFft = mem.reserve(fft_work);
    DevBuf extra_work;  // a last, shorter section's plan may want more
    RSATB_TRY(mem.commit(ctx));
    void* const u_scr = c.sandwich ? mem.at<void>(oU) : nullptr;
    void* const w_scr = c.sandwich ? mem.at<void>(oW) : nullptr;
    T* const pan0 = mem.at<T>(oPan);
    T* const start = mem.at<T>(oInit);
    double* const d_wts = mem.at<double>(oWts);
    double2* const d_pw = mem.at<double2>(oPw);
    double2* const d_part = mem.at<double2>(oPart);
    double2* const d_tab = mem.at<double2>(oTab);
    T* J[3];
    for (int a = 0; a < 3; ++a) J[a] = mem.at<T>(oJ) + size_t(a) * N * 2 * R;
    T* rinit = mem.at<T>(oRinit);
    T* r[3];
    T* l[3];
    for (int i = 0; i < 3; ++i) {
        r[i] = mem.at<T>(oR) + size_t(i) * N * 6 * R;
        l[i] = mem.at<T>(oL) + size_t(i) * N * 2 * R;
    }
    T* SL = mem.at<T>(oS);
    T* SR = SL + 2 * size_t(M) * slot;
    double2* EL = mem.at<double2>(oE);
    double2* ER = EL + size_t(M) * nq_max;
    // Bastin: phi1 and phi2 of both sides.
    double2* EL1 = EL;
    double2* ER1 = EL1 + 2 * size_t(M) * nq_max;
    double2* EL2 = ER1 + 2 * size_t(M) * nq_max;
    double2* ER2 = EL2 + 2 * size_t(M) * nq_max;
    double* K = mem.at<double>(oK);

    std::vector<double> g(M), wts(M);
    kpm_kernel_weights(kernel, M, g.data());
    for (int m = 0; m < M; ++m) wts[m] = g[m] / M_PI;  // phi3_weight (fftcheb_transport.hpp)
    RSATB_CUDA_TRY(cudaMemcpyAsync(d_wts, wts.data(), M * sizeof(double),
                                   cudaMemcpyHostToDevice, st));
    // Bastin phase weights (fftcheb_transport.hpp:302-310): phase_weight[m] =
    // 2 g_m / (pi (1 + [m == 0])) e^{i pi m / 2M}, phase_weight_m = m times it.
    std::vector<double2> pw;
    if (bastin) {
        pw.resize(2 * size_t(M));
        for (int m = 0; m < M; ++m) {
            const double coeff = 2.0 * g[m] / (M_PI * (1.0 + (m == 0 ? 1.0 : 0.0)));
            const double th = M_PI * double(m) / (2.0 * double(M));
            pw[m] = make_double2(coeff * std::cos(th), coeff * std::sin(th));
            pw[M + m] = make_double2(pw[m].x * double(m), pw[m].y * double(m));
        }
        RSATB_CUDA_TRY(cudaMemcpyAsync(d_pw, pw.data(), pw.size() * sizeof(double2),
                                       cudaMemcpyHostToDevice, st));
    }
    RSATB_CUDA_TRY(cudaMemsetAsync(K, 0, size_t(M) * 12 * sizeof(double), st));

    int64_t fused_qc = std::max<int64_t>(
        1, std::min<int64_t>(8192, int64_t(e_bytes / (2 * size_t(M) * cplx))));
    if (const char* cap = std::getenv("RSATB_FFTCHEB_CHUNK")) {  // smaller chunks (tests)
        const int64_t c = std::atoll(cap);
        if (c > 0 && c < fused_qc) fused_qc = c;
    }
    if (fused) {
        fused_tables_kernel<<<(fused_tab(radix) + 255) / 256, 256, 0, st>>>(M, d_wts, d_tab);
        RSATB_LAUNCH_CHECK(ctx);
    }

    cudaEvent_t ev0, ev1;
    RSATB_CUDA_TRY(cudaEventCreate(&ev0));
    RSATB_CUDA_TRY(cudaEventCreate(&ev1));
    struct EvG {
        cudaEvent_t a, b;
        ~EvG() {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
        }
    } evg{ev0, ev1};
    float rec_ms = 0.f, dct_ms = 0.f;

    // J_a psi and the right-chain start.
    MomentArgs<T> ma{};
    int m_threads = 0;
    size_t m_smem = 0;
    if (one_launch) {
        ma.n_rows = N;
        ma.row_ptr = c.op->H->row_ptr;
        ma.col_ind = c.op->H->col_ind;
        const rsatb_bsr_matrix* H = c.op->H;
        T* const wgt = mem.at<T>(oWgt);
        pack_weights_kernel<T><<<grid_for(nnz, ctx->sm_count), 256, 0, st>>>(
            nnz, static_cast<const T*>(H->values), static_cast<const T*>(V[0]->values),
            static_cast<const T*>(V[1]->values), static_cast<const T*>(V[2]->values), wgt);
        RSATB_LAUNCH_CHECK(ctx);
        ma.wgt = wgt;
        ma.W1 = W1;
        ma.C = moment_threads_per_row<T>(R);
        ma.c = c.op->center;
        ma.inv_hw = 1.0 / c.op->half_width;
        ma.cscale = -1.0 / (2.0 * c.op->half_width);
        // Rows per CTA: up to 256 threads, and as many average rows as fit one
        // pass of kMomentCap nonzeros; a CTA with longer ones takes more passes.
        // (By the longest row, one long row made every CTA a single row: 100,000
        // rows of 9 nonzeros and one of 1,009, 4 FP64 samples 237 us a moment, now
        // 103; the separate launches 1,177.)
        const int longest = std::max(1, c.op->H->max_row_blocks);
        const int average = int(std::max<int64_t>(1, (nnz + N - 1) / std::max<int64_t>(N, 1)));
        int rpc = std::min(256 / ma.C, kMomentCap / average);
        if (rpc < 1) rpc = 1;
        m_threads = rpc * ma.C;
        ma.cap = int(std::min<int64_t>(kMomentCap, int64_t(rpc) * longest));
        m_smem = size_t(ma.cap) * (4 * sizeof(T) + sizeof(int32_t));
        moment_init_kernel<T><<<grid_for(N * R, ctx->sm_count), 256, 0, st>>>(
            N, R, ma.row_ptr, ma.col_ind, ma.wgt, psi, ma.cscale, start);
        RSATB_LAUNCH_CHECK(ctx);
    } else {
        for (int a = 0; a < 3; ++a)
            RSATB_TRY(current_rows(c, V[a], W1, psi, J[a], 0, nb, u_scr, w_scr));
        pack_axes_kernel<T><<<grid_for(N * 3 * R, ctx->sm_count), 256, 0, st>>>(N, R, J[0], J[1],
                                                                               J[2], rinit);
        RSATB_LAUNCH_CHECK(ctx);
    }

    int64_t chunks = 0;
    for (int sec = 0; sec < n_sections; ++sec) {
        const int sb0 = int(sec * sec_brows);
        const int sb1 = int(std::min<int64_t>(nb, sb0 + sec_brows));
        const int64_t rows0 = int64_t(sb0) * b;
        const int64_t rows = int64_t(sb1 - sb0) * b;
        const int64_t sslot = 3 * rows * R;  // this section's slot size
        RSATB_CUDA_TRY(cudaEventRecord(ev0, st));
        if (one_launch) {
            // Moment 0 is read from its own buffer, moment 1 formed in panel 0,
            // then the panels alternate (panel 1 takes moment 2 over a copy of
            // moment 0, its predecessor).
            T* pan[2] = {pan0, pan0 + panel};
            if (M > 1)
                RSATB_CUDA_TRY(cudaMemcpyAsync(pan[1], start, panel * sizeof(T),
                                               cudaMemcpyDeviceToDevice, st));
            const int rpc = m_threads / ma.C;
            const unsigned grid = unsigned((N + rpc - 1) / rpc);
            ma.row0 = rows0;
            ma.row1 = rows0 + rows;
            for (int m = 0; m < M; ++m) {
                ma.cur = m == 0 ? start : pan[(m + 1) & 1];
                ma.prev = pan[m & 1];
                ma.sl = SL + 2 * size_t(m) * sslot;
                ma.sr = SR + 2 * size_t(m) * sslot;
                ma.advance = m + 1 < M;
                ma.s2 = m == 0 ? 1.0 : 2.0;
                ma.g_p = m == 0 ? 0.0 : -1.0;
                // Resident CTAs against loads in flight (us per moment, 47,632
                // rows, 16 FP32 samples): 4 CTAs x 4 loads 75.8, 3 x 4 86.9,
                // 3 x 8 84.2, 5 x 2 90.0.
                if constexpr (sizeof(T) == 4) {
                    if (R % 2 == 0)
                        moment_kernel<T, 4, 4, 4><<<grid, m_threads, m_smem, st>>>(ma);
                    else
                        moment_kernel<T, 2, 4, 5><<<grid, m_threads, m_smem, st>>>(ma);
                } else {
                    moment_kernel<T, 2, 4, 4><<<grid, m_threads, m_smem, st>>>(ma);
                }
                RSATB_LAUNCH_CHECK(ctx);
            }
        } else {
            RSATB_CUDA_TRY(cudaMemcpyAsync(r[0], rinit, size_t(N) * 3 * R * cplx,
                                           cudaMemcpyDeviceToDevice, st));
            const T* lp = psi;       // l_{m-1}
            const T* lc = nullptr;   // l_m
            int ri_prev = 0, ri_cur = -1;
            int li = 0;
            for (int m = 0; m < M; ++m) {
                const T* lm;  // l_m
                int rm;       // index of r_m
                if (m == 0) {
                    lm = psi;
                    rm = 0;
                } else if (m == 1) {
                    T* lo = l[li];
                    li = (li + 1) % 3;
                    RSATB_TRY(op_step(c, W1, lp, nullptr, lo, u_scr, w_scr, 1.0, 0.0));
                    RSATB_TRY(op_step(c, W3, r[ri_prev], nullptr, r[1], u_scr, w_scr, 1.0, 0.0));
                    lc = lo;
                    ri_cur = 1;
                    lm = lc;
                    rm = 1;
                } else {
                    T* lo = l[li];
                    li = (li + 1) % 3;
                    const int rn = 3 - ri_prev - ri_cur;
                    RSATB_TRY(op_step(c, W1, lc, lp, lo, u_scr, w_scr, 2.0, -1.0));
                    RSATB_TRY(op_step(c, W3, r[ri_cur], r[ri_prev], r[rn], u_scr, w_scr, 2.0, -1.0));
                    lp = lc;
                    lc = lo;
                    ri_prev = ri_cur;
                    ri_cur = rn;
                    lm = lc;
                    rm = rn;
                }
                T* sl = SL + 2 * size_t(m) * sslot;
                for (int a = 0; a < 3; ++a)
                    RSATB_TRY(current_rows(c, V[a], W1, lm, sl + 2 * size_t(a) * rows * R, sb0, sb1,
                                           u_scr, w_scr));
                if (sizeof(T) == 8 || R % 2 == 0)
                    store_right_vec_kernel<T>
                        <<<grid_for(sslot * 2 * int64_t(sizeof(T)) / 16, ctx->sm_count), 256, 0, st>>>(
                            rows0, rows, R, r[rm], SR + 2 * size_t(m) * sslot);
                else
                    store_right_kernel<T><<<grid_for(sslot, ctx->sm_count), 256, 0, st>>>(
                        rows0, rows, R, r[rm], SR + 2 * size_t(m) * sslot);
                RSATB_LAUNCH_CHECK(ctx);
            }
        }
        RSATB_CUDA_TRY(cudaEventRecord(ev1, st));
        RSATB_CUDA_TRY(cudaEventSynchronize(ev1));
        float t = 0.f;
        cudaEventElapsedTime(&t, ev0, ev1);
        rec_ms += t;

        // Row stage: fused (Greenwood, fused_radix), else in chunks of rows
        // through the transform input, cuFFT and the contraction.
        RSATB_CUDA_TRY(cudaEventRecord(ev0, st));
        if (fused) {
            const int64_t per_axis = rows * R;
            T* Tq = reinterpret_cast<T*>(EL);
            for (int a = 0; a < 3; ++a) {
                RSATB_CUDA_TRY(
                    cudaMemsetAsync(d_part, 0, size_t(n_part) * M * sizeof(double2), st));
                for (int64_t i0 = 0; i0 < per_axis; i0 += fused_qc) {
                    const int64_t n = std::min<int64_t>(fused_qc, per_axis - i0);
                    const dim3 gg(unsigned((n + 31) / 32), M / 32, 2);
                    gather_sequences_kernel<T><<<gg, 256, 0, st>>>(
                        M, int64_t(a) * per_axis + i0, n, sslot, SL, SR, Tq);
                    RSATB_LAUNCH_CHECK(ctx);
                    bool done = false;
                    if constexpr (std::is_same<T, float>::value) {
                        if (fused32) {
                            RSATB_TRY((fused_launch<T, float2, 8>(ctx, fused_grid, n, Tq,
                                                                  d_tab,
                                                                  d_part)));
                            done = true;
                        }
                    }
                    if (!done)
                        RSATB_TRY((fused_launch_r<T, double2>(ctx, radix, fused_grid, n, Tq,
                                                              d_tab,
                                                              d_part)));
                    ++chunks;
                }
                fused_reduce_kernel<<<M, 128, 0, st>>>(
                    M, n_part, d_part, a == 0 ? 0 : (a == 1 ? 3 : 5), K);
                RSATB_LAUNCH_CHECK(ctx);
            }
        }
        for (int64_t c0 = 0; !fused && c0 < rows; c0 += chunk_rows) {
            const int64_t cr = std::min<int64_t>(chunk_rows, rows - c0);
            const int64_t nq = 3 * cr * R;
            cufftHandle plan = 0;
            size_t wneed = 0;
            RSATB_TRY(fft_plan(ctx, fft_n, nq, &plan, &wneed));
            void* area = mem.at<void>(oFft);
            if (wneed > fft_work) {
                RSATB_CUDA_TRY(cudaStreamSynchronize(st));
                extra_work.release();
                RSATB_TRY(extra_work.alloc(wneed));
                area = extra_work.p;
            }
            RSATB_CUFFT_TRY(cufftSetStream(plan, st));
            RSATB_CUFFT_TRY(cufftSetWorkArea(plan, area));
            const unsigned gx = std::min(64u, grid_for(nq, ctx->sm_count));
            if (!bastin) {
                const dim3 grid(gx, M / 2 + 1);
                const T* src[2] = {SL, SR};
                double2* dst[2] = {EL, ER};
                for (int t = 0; t < 2; ++t) {
                    dct3_input_kernel<T><<<grid, 256, 0, st>>>(M, nq, int(cr), R, rows, c0, sslot,
                                                               src[t], d_wts, dst[t]);
                    RSATB_LAUNCH_CHECK(ctx);
                    RSATB_CUFFT_TRY(cufftExecZ2Z(plan,
                                                 reinterpret_cast<cufftDoubleComplex*>(dst[t]),
                                                 reinterpret_cast<cufftDoubleComplex*>(dst[t]),
                                                 CUFFT_INVERSE));
                }
                greenwood_contract_kernel<<<M, 256, 0, st>>>(M, nq, cr * R, EL, ER, K);
                RSATB_LAUNCH_CHECK(ctx);
            } else {
                const dim3 grid(gx, M);
                const double2* w1 = d_pw;
                const double2* w2 = w1 + M;
                double2* dst[4] = {EL1, ER1, EL2, ER2};
                const T* src[4] = {SL, SR, SL, SR};
                const double2* wt[4] = {w1, w1, w2, w2};
                for (int t = 0; t < 4; ++t) {
                    pad_kernel<T><<<grid, 256, 0, st>>>(M, nq, int(cr), R, rows, c0, sslot,
                                                        src[t], wt[t], dst[t]);
                    RSATB_LAUNCH_CHECK(ctx);
                    RSATB_CUFFT_TRY(cufftExecZ2Z(plan, reinterpret_cast<cufftDoubleComplex*>(dst[t]),
                                                 reinterpret_cast<cufftDoubleComplex*>(dst[t]),
                                                 CUFFT_INVERSE));
                }
                bastin_contract_kernel<<<M, 256, 0, st>>>(M, nq, cr * R, EL1, ER1, EL2, ER2, K);
                RSATB_LAUNCH_CHECK(ctx);
            }
            ++chunks;
        }
        RSATB_CUDA_TRY(cudaEventRecord(ev1, st));
        RSATB_CUDA_TRY(cudaEventSynchronize(ev1));
        cudaEventElapsedTime(&t, ev0, ev1);
        dct_ms += t;
    }

    std::vector<double> Kh(size_t(M) * 12);
    RSATB_CUDA_TRY(cudaMemcpyAsync(Kh.data(), K, Kh.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, st));
    RSATB_CUDA_TRY(cudaStreamSynchronize(st));
    RSATB_TRY(ctx_check_fault(ctx));
    // Sample average and the ascending energy grid of
    // fftcheb_transport.hpp:602-659: E_k = c + hw cos(pi (M - 1 - k + 1/2) / M).
    for (int k = 0; k < M; ++k) {
        const int src = M - 1 - k;
        energy_out[k] = c.op->center +
                        c.op->half_width * std::cos(M_PI * (double(src) + 0.5) / double(M));
        if (!bastin)
            for (int comp = 0; comp < 6; ++comp)
                sigma_out[k * 6 + comp] = prefactor * Kh[2 * (size_t(src) * 6 + comp)] / double(R);
    }
    if (bastin) {
        // sigma(mu, T = 0): cumulative trapezoid of Re(i zeta(eps)) over the
        // ascending Chebyshev grid (fftcheb_transport.hpp:635-659), zeta the
        // sample-averaged kernel.
        double running[6] = {0, 0, 0, 0, 0, 0}, prev[6] = {0, 0, 0, 0, 0, 0};
        double eps_prev = 0.0;
        for (int k = 0; k < M; ++k) {
            const int src = M - 1 - k;
            const double eps = std::cos(M_PI * (double(src) + 0.5) / double(M));
            for (int comp = 0; comp < 6; ++comp) {
                const double integrand = -Kh[2 * (size_t(src) * 6 + comp) + 1] / double(R);
                if (k > 0) running[comp] += 0.5 * (prev[comp] + integrand) * (eps - eps_prev);
                sigma_out[k * 6 + comp] = prefactor * running[comp];
                prev[comp] = integrand;
            }
            eps_prev = eps;
        }
    }
    if (stats) {
        stats->sections = n_sections;
        stats->fft_chunks = chunks;
        stats->recurrence_ms = rec_ms;
        stats->transform_ms = dct_ms;
        stats->store_bytes = 2 * size_t(M) * slot * cplx;
    }
    return RSATB_SUCCESS;
}

// ------------------------------------------------------------ QE route
//
// Quasi-eigenstate Greenwood (dc_spectrum_qe, fftcheb_transport.hpp:
// 662-884): the same bilinear form as the fftcheb Greenwood route,
// sigma(e_j) = sum_{m,m'} w_m(j) w_m'(j) <L_m|R_m'> / max(1e-14, 1 - e_j^2),
// w_m(j) = (m ? 2 : 1) g_m / pi T_m(e_j), evaluated at a window of nodes j
// only.  The weights are real, so it factors as <P_j|Q_j> with the left and
// right quasi-eigenstates P_j = sum_m w_m(j) L_m and Q_j = sum_m w_m(j) R_m:
// each pass adds a batch of QE_BATCH consecutive moment panels into all the
// node vectors in one launch (each node vector read and written once per
// batch, FP64 whatever the panel precision), and one fixed-order dot per
// (node, axis) finishes.  No row store and no transform.

constexpr int kQeBatch = 8;

template <typename T>
struct QePanels {
    const T* p[3 * kQeBatch];  // right: one [row][axis][sample] panel per
                               // moment; left: three [row][sample] per moment
};

// Q[j][a][row][s] += sum_b w[b][j] X_b(a, row, s) for the nb moments of a
// batch; one thread per (a, row, s).
template <typename T, bool RIGHT>
__global__ void qe_accumulate(int64_t n_rows, int R, int nb, int NE, QePanels<T> X,
                              const double* __restrict__ w, double2* __restrict__ Q) {
    const int64_t n_el = 3 * n_rows * R;
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < n_el;
         e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t s = e % R;
        const int64_t t = e / R;
        const int64_t row = t % n_rows;
        const int a = int(t / n_rows);
        double xr[kQeBatch], xi[kQeBatch];
#pragma unroll
        for (int b = 0; b < kQeBatch; ++b) {
            xr[b] = xi[b] = 0.0;
            if (b < nb) {
                const T* src = RIGHT ? X.p[b] + 2 * ((row * 3 + a) * R + s)
                                     : X.p[3 * b + a] + 2 * (row * R + s);
                xr[b] = double(src[0]);
                xi[b] = double(src[1]);
            }
        }
        for (int j = 0; j < NE; ++j) {
            double2 q = Q[int64_t(j) * n_el + e];
#pragma unroll
            for (int b = 0; b < kQeBatch; ++b) {
                if (b < nb) {
                    const double wb = __ldg(w + b * NE + j);
                    q.x = fma(wb, xr[b], q.x);
                    q.y = fma(wb, xi[b], q.y);
                }
            }
            Q[int64_t(j) * n_el + e] = q;
        }
    }
}

// D[j][a] = sum_{row, s} conj(P[j][a][row][s]) Q[j][a][row][s]: one CTA per
// (node, axis), fixed-order tree reduction.
__global__ void __launch_bounds__(256) qe_node_dots(int64_t per_axis, const double2* P,
                                                    const double2* Q, double* D) {
    __shared__ double red[2][256];
    const int64_t base = int64_t(blockIdx.x) * per_axis;
    double ar = 0.0, ai = 0.0;
    for (int64_t q = threadIdx.x; q < per_axis; q += blockDim.x) {
        const double2 x = P[base + q], y = Q[base + q];
        ar += x.x * y.x + x.y * y.y;
        ai += x.x * y.y - x.y * y.x;
    }
    red[0][threadIdx.x] = ar;
    red[1][threadIdx.x] = ai;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[0][threadIdx.x] += red[0][threadIdx.x + w];
            red[1][threadIdx.x] += red[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        D[2 * blockIdx.x] = red[0][0];
        D[2 * blockIdx.x + 1] = red[1][0];
    }
}

template <typename T>
int qe_impl(const Ctx& c, const rsatb_bsr_matrix* const* V, const T* psi, int R, int M,
            const std::vector<int>& nodes, double prefactor, int kernel, double* sigma_out,
            double* energy_out) {
    rsatb_context* ctx = c.ctx;
    cudaStream_t st = ctx->stream;
    const int b = c.op->H->block_size;
    const int nbr = c.op->H->n_block_rows;
    const int64_t N = int64_t(nbr) * b;
    const int W1 = 2 * R, W3 = 6 * R;
    const size_t cplx = 2 * sizeof(T);
    const int NE = int(nodes.size());
    const int RB = kQeBatch + 2;  // right ring: the batch plus the recurrence's predecessors

    std::vector<double> g(M);
    kpm_kernel_weights(kernel, M, g.data());
    // weights w[m][j] and the node energies (src = M - 1 - ascending index)
    std::vector<double> wts(size_t(M) * NE), denom(NE);
    for (int j = 0; j < NE; ++j) {
        const int src = M - 1 - nodes[j];
        const double th = M_PI * (double(src) + 0.5) / double(M);
        const double e = std::cos(th);
        denom[j] = std::max(1e-14, 1.0 - e * e);
        for (int m = 0; m < M; ++m)
            wts[size_t(m) * NE + j] = (m == 0 ? 1.0 : 2.0) * g[m] / M_PI * std::cos(double(m) * th);
    }
    DevBuf bW, bJ, bR, bL, bLA, bU, bWs, bQ, bP, bD;
    RSATB_TRY(bW.alloc(wts.size() * sizeof(double)));
    RSATB_CUDA_TRY(cudaMemcpyAsync(bW.p, wts.data(), wts.size() * sizeof(double),
                                   cudaMemcpyHostToDevice, st));
    RSATB_TRY(bJ.alloc(size_t(N) * 3 * R * cplx));
    RSATB_TRY(bR.alloc(size_t(RB) * N * 3 * R * cplx));
    RSATB_TRY(bL.alloc(size_t(3) * N * R * cplx));
    RSATB_TRY(bLA.alloc(size_t(kQeBatch) * 3 * N * R * cplx));
    if (c.sandwich) {
        RSATB_TRY(bU.alloc(size_t(N) * 3 * R * cplx));
        RSATB_TRY(bWs.alloc(size_t(N) * 3 * R * cplx));
    }
    const int64_t n_el = 3 * N * R;
    RSATB_TRY(bQ.alloc(size_t(NE) * n_el * sizeof(double2)));
    RSATB_TRY(bP.alloc(size_t(NE) * n_el * sizeof(double2)));
    RSATB_TRY(bD.alloc(size_t(NE) * 3 * sizeof(double2)));
    RSATB_CUDA_TRY(cudaMemsetAsync(bQ.p, 0, size_t(NE) * n_el * sizeof(double2), st));
    RSATB_CUDA_TRY(cudaMemsetAsync(bP.p, 0, size_t(NE) * n_el * sizeof(double2), st));
    T* J[3];
    for (int a = 0; a < 3; ++a) J[a] = bJ.as<T>() + size_t(a) * N * 2 * R;
    auto rslot = [&](int m) { return bR.as<T>() + size_t(m % RB) * N * 6 * R; };
    T* l[3];
    for (int i = 0; i < 3; ++i) l[i] = bL.as<T>() + size_t(i) * N * 2 * R;
    auto laslot = [&](int bidx, int a) {
        return bLA.as<T>() + (size_t(bidx) * 3 + a) * N * 2 * R;
    };
    const unsigned grid = grid_for(n_el, ctx->sm_count);
    auto flush = [&](bool right, int m_last, int nb) -> int {
        QePanels<T> X{};
        const int m0 = m_last - nb + 1;
        for (int q = 0; q < nb; ++q) {
            if (right) {
                X.p[q] = rslot(m0 + q);
            } else {
                for (int a = 0; a < 3; ++a) X.p[3 * q + a] = laslot((m0 + q) % kQeBatch, a);
            }
        }
        const double* w = bW.as<double>() + size_t(m0) * NE;
        double2* dst = right ? bQ.as<double2>() : bP.as<double2>();
        if (right)
            qe_accumulate<T, true><<<grid, 256, 0, st>>>(N, R, nb, NE, X, w, dst);
        else
            qe_accumulate<T, false><<<grid, 256, 0, st>>>(N, R, nb, NE, X, w, dst);
        RSATB_LAUNCH_CHECK(ctx);
        return RSATB_SUCCESS;
    };

    // Right pass: R_0 = (J_a psi) packed [row][axis][sample], R_m by the
    // recurrence on the N x 3R panel.
    for (int a = 0; a < 3; ++a)
        RSATB_TRY(current_rows(c, V[a], W1, psi, J[a], 0, nbr, bU.p, bWs.p));
    pack_axes_kernel<T><<<grid_for(N * 3 * R, ctx->sm_count), 256, 0, st>>>(N, R, J[0], J[1],
                                                                           J[2], rslot(0));
    RSATB_LAUNCH_CHECK(ctx);
    for (int m = 0; m < M; ++m) {
        if (m == 1)
            RSATB_TRY(op_step(c, W3, rslot(0), nullptr, rslot(1), bU.p, bWs.p, 1.0, 0.0));
        else if (m >= 2)
            RSATB_TRY(op_step(c, W3, rslot(m - 1), rslot(m - 2), rslot(m), bU.p, bWs.p, 2.0,
                              -1.0));
        if ((m + 1) % kQeBatch == 0 || m == M - 1)
            RSATB_TRY(flush(true, m, m % kQeBatch + 1));
    }
    // Left pass: L_m = J_a T_m(Op) psi (J_a^H = J_a: V_a and the sandwich's
    // Z^H V_a Z are Hermitian).
    const T* lp = nullptr;
    const T* lc = psi;
    int li = 0;
    for (int m = 0; m < M; ++m) {
        if (m >= 1) {
            T* lo = l[li];
            li = (li + 1) % 3;
            if (m == 1) RSATB_TRY(op_step(c, W1, lc, nullptr, lo, bU.p, bWs.p, 1.0, 0.0));
            else RSATB_TRY(op_step(c, W1, lc, lp, lo, bU.p, bWs.p, 2.0, -1.0));
            lp = lc;
            lc = lo;
        }
        for (int a = 0; a < 3; ++a)
            RSATB_TRY(current_rows(c, V[a], W1, lc, laslot(m % kQeBatch, a), 0, nbr, bU.p,
                                   bWs.p));
        if ((m + 1) % kQeBatch == 0 || m == M - 1)
            RSATB_TRY(flush(false, m, m % kQeBatch + 1));
    }
    qe_node_dots<<<unsigned(NE * 3), 256, 0, st>>>(N * R, bP.as<double2>(), bQ.as<double2>(),
                                                  bD.as<double>());
    RSATB_LAUNCH_CHECK(ctx);
    std::vector<double> D(size_t(NE) * 6);
    RSATB_CUDA_TRY(cudaMemcpyAsync(D.data(), bD.p, D.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, st));
    RSATB_CUDA_TRY(cudaStreamSynchronize(st));
    RSATB_TRY(ctx_check_fault(ctx));
    // Ascending energies (fftcheb_transport.hpp:940-954); sigma zero outside
    // the node window, Re of the sample-averaged kernel inside.
    for (int k = 0; k < M; ++k) {
        const int src = M - 1 - k;
        energy_out[k] = c.op->center +
                        c.op->half_width * std::cos(M_PI * (double(src) + 0.5) / double(M));
    }
    std::fill(sigma_out, sigma_out + size_t(M) * 6, 0.0);
    for (int j = 0; j < NE; ++j)
        for (int a = 0; a < 3; ++a) {
            const int comp = a == 0 ? 0 : (a == 1 ? 3 : 5);
            sigma_out[size_t(nodes[j]) * 6 + comp] =
                prefactor * D[2 * (size_t(j) * 3 + a)] / denom[j] / double(R);
        }
    return RSATB_SUCCESS;
}

}  // namespace
}  // namespace rsatb_b200

using namespace rsatb_b200;

extern "C" int rsatb_dc_spectrum_fftcheb(rsatb_ctx_t ctx, const rsatb_cheb_op* op, rsatb_bsr_t Vx,
                                         rsatb_bsr_t Vy, rsatb_bsr_t Vz, const void* psi,
                                         int n_vectors, rsatb_dtype vec_dtype, int n_moments,
                                         int formulation, double prefactor,
                                         int partition_sections, size_t max_workspace_bytes,
                                         int kernel, double* sigma_out, double* energy_out,
                                         rsatb_fftcheb_stats* stats) {
    clear_error();
    RSATB_TRY(check_ctx(ctx));
    if (!op || !psi || !sigma_out || !energy_out)
        return set_error(RSATB_INVALID_ARGUMENT, "null argument");
    if (op->form != RSATB_FORM_ORTHOGONAL && op->form != RSATB_FORM_SANDWICH)
        return set_error(RSATB_NOT_SUPPORTED, "operator form %d is not available on the device",
                         op->form);
    const bool sandwich = op->form == RSATB_FORM_SANDWICH;
    const rsatb_bsr_matrix* mats[6] = {op->H, sandwich ? op->Z : op->H,
                                       sandwich ? op->ZH : op->H, Vx, Vy, Vz};
    const char* names[6] = {"H", "Z", "ZH", "Vx", "Vy", "Vz"};
    for (int i = 0; i < 6; ++i) {
        RSATB_TRY(check_bsr(mats[i], names[i]));
        if (mats[i]->n_block_rows != op->H->n_block_rows ||
            mats[i]->n_block_cols != op->H->n_block_rows ||
            mats[i]->block_size != op->H->block_size)
            return set_error(RSATB_INVALID_ARGUMENT, "%s does not match H's shape", names[i]);
        if (dtype_is_double(mats[i]->dtype) != dtype_is_double(vec_dtype))
            return set_error(RSATB_INVALID_ARGUMENT, "%s precision differs from the vectors'",
                             names[i]);
    }
    if (!dtype_is_complex(vec_dtype))
        return set_error(RSATB_INVALID_ARGUMENT, "transport needs complex sample vectors");
    if (!(op->half_width > 0.0))
        return set_error(RSATB_INVALID_ARGUMENT, "half_width must be positive");
    if (n_vectors <= 0 || n_moments <= 0)
        return set_error(RSATB_INVALID_ARGUMENT, "n_vectors and n_moments must be positive");
    if (6 * n_vectors > 1536)
        return set_error(RSATB_NOT_SUPPORTED, "%d samples exceed one block (256 at most)",
                         n_vectors);
    if (formulation != 0 && formulation != 1)
        return set_error(RSATB_INVALID_ARGUMENT,
                         "formulation %d: 0 (Greenwood) or 1 (Bastin)", formulation);
    if (!aligned16(psi)) return set_error(RSATB_INVALID_ARGUMENT, "psi must be 16-byte aligned");
    if (stats) *stats = rsatb_fftcheb_stats{};
    const rsatb_bsr_matrix* V[3] = {Vx, Vy, Vz};
    Ctx c{ctx, op, sandwich, int(vec_dtype)};
    if (dtype_is_double(vec_dtype))
        return fftcheb_impl<double>(c, V, static_cast<const double*>(psi), n_vectors, n_moments,
                                    formulation, prefactor, partition_sections,
                                    max_workspace_bytes, kernel, sigma_out, energy_out, stats);
    return fftcheb_impl<float>(c, V, static_cast<const float*>(psi), n_vectors, n_moments,
                               formulation, prefactor, partition_sections, max_workspace_bytes,
                               kernel, sigma_out, energy_out, stats);
}

extern "C" int rsatb_dc_spectrum_qe(rsatb_ctx_t ctx, const rsatb_cheb_op* op, rsatb_bsr_t Vx,
                                    rsatb_bsr_t Vy, rsatb_bsr_t Vz, const void* psi,
                                    int n_vectors, rsatb_dtype vec_dtype, int n_moments,
                                    double prefactor, int kernel, const int32_t* nodes,
                                    int n_nodes, double* sigma_out, double* energy_out) {
    clear_error();
    RSATB_TRY(check_ctx(ctx));
    if (!op || !psi || !sigma_out || !energy_out || (n_nodes > 0 && !nodes))
        return set_error(RSATB_INVALID_ARGUMENT, "null argument");
    if (op->form != RSATB_FORM_ORTHOGONAL && op->form != RSATB_FORM_SANDWICH)
        return set_error(RSATB_NOT_SUPPORTED, "operator form %d is not available on the device",
                         op->form);
    const bool sandwich = op->form == RSATB_FORM_SANDWICH;
    const rsatb_bsr_matrix* mats[6] = {op->H, sandwich ? op->Z : op->H,
                                       sandwich ? op->ZH : op->H, Vx, Vy, Vz};
    const char* names[6] = {"H", "Z", "ZH", "Vx", "Vy", "Vz"};
    for (int i = 0; i < 6; ++i) {
        RSATB_TRY(check_bsr(mats[i], names[i]));
        if (mats[i]->n_block_rows != op->H->n_block_rows ||
            mats[i]->n_block_cols != op->H->n_block_rows ||
            mats[i]->block_size != op->H->block_size)
            return set_error(RSATB_INVALID_ARGUMENT, "%s does not match H's shape", names[i]);
        if (dtype_is_double(mats[i]->dtype) != dtype_is_double(vec_dtype))
            return set_error(RSATB_INVALID_ARGUMENT, "%s precision differs from the vectors'",
                             names[i]);
    }
    if (!dtype_is_complex(vec_dtype))
        return set_error(RSATB_INVALID_ARGUMENT, "transport needs complex sample vectors");
    if (!(op->half_width > 0.0))
        return set_error(RSATB_INVALID_ARGUMENT, "half_width must be positive");
    if (n_vectors <= 0 || n_moments <= 0)
        return set_error(RSATB_INVALID_ARGUMENT, "n_vectors and n_moments must be positive");
    if (6 * n_vectors > 1536)
        return set_error(RSATB_NOT_SUPPORTED, "%d samples exceed one block (256 at most)",
                         n_vectors);
    if (!aligned16(psi)) return set_error(RSATB_INVALID_ARGUMENT, "psi must be 16-byte aligned");
    // The node window: ascending output-grid indices, sorted and unique;
    // empty means every node (dc_spectrum_qe's nodes_ascending).
    std::vector<int> nd;
    if (n_nodes <= 0) {
        nd.resize(n_moments);
        for (int k = 0; k < n_moments; ++k) nd[k] = k;
    } else {
        nd.assign(nodes, nodes + n_nodes);
        std::sort(nd.begin(), nd.end());
        nd.erase(std::unique(nd.begin(), nd.end()), nd.end());
        if (nd.front() < 0 || nd.back() >= n_moments)
            return set_error(RSATB_INVALID_ARGUMENT, "dc_spectrum_qe: node index out of range");
    }
    const rsatb_bsr_matrix* V[3] = {Vx, Vy, Vz};
    Ctx c{ctx, op, sandwich, int(vec_dtype)};
    if (dtype_is_double(vec_dtype))
        return qe_impl<double>(c, V, static_cast<const double*>(psi), n_vectors, n_moments, nd,
                               prefactor, kernel, sigma_out, energy_out);
    return qe_impl<float>(c, V, static_cast<const float*>(psi), n_vectors, n_moments, nd,
                          prefactor, kernel, sigma_out, energy_out);
}
