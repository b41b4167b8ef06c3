// tm_kernels.cuh -- the search kernels for one batch of orientations.
//
// Data flow per orientation (o) of a batch, T = template box, X x Y = padded
// micrograph, XP = row pitch of half-spectra in complex values (X/2+1 rounded
// up to a multiple of the pass-B column chunk):
//
//   k_slice_colfft   Fourier slice of the 3-D template (trilinear, Hermitian
//                    mirror; image.cpp:2450-2607, 2899-3020) x (-1)^(i+j)
//                    (SwapRealSpaceQuadrants) x projection filter, then the
//                    inverse FFT along y of each of the T/2+1 columns
//   k_row_c2r        inverse c2r FFT of each row -> real T x T projection,
//                    plus per-row sums for the edge mean and variance
//   k_norm           per-orientation edge mean e and 1/sigma
//                    (match_template.cpp:1060-1068)
//   k_pass_a         (p - e)/sigma, placed at the origin of an X-wide row and
//                    forward FFT along x using only its T non-zero samples
//                    (X/T twiddled T-point FFTs) -> A[o][row][kx]
//   k_pass_b         per column kx: pruned forward FFT along y of the T rows
//                    of A, multiply by the prepared micrograph spectrum
//                    I'[ky][kx] (whitened spectrum x conj(placement phase) / N,
//                    DC zero), inverse FFT along y -> C[o][y][kx]
//   k_pass_c         per row y: c2r FFT along x of C[o][y][:] and, in
//                    registers, the MIP / argmax / sum / sum-of-squares /
//                    histogram update of match_template.cpp:1102-1149 over the
//                    batch; per-pixel state is read and written once per batch
//
// The placement of the projection at (X/2 - T/2, Y/2 - T/2)
// (ClipIntoLargerRealSpace2D, image.cpp:8398-8465), the forward-FFT scaling
// 1/N and the zeroed central pixel are folded into I' once per micrograph.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <float.h>
#include <type_traits>
#include "tm_fft.cuh"
#include "tm_ptx.cuh"

namespace tmk {

using tmfft::cmul;
using tmfft::cmul_conj;
using tmfft::Twiddles;

__host__ __device__ constexpr int round_up16(int v) { return (v + 15) / 16 * 16; }
// region stride >= len whose value mod 16 equals `rem` (bank skew between regions)
__host__ __device__ constexpr int skewed(int len, int rem) { return round_up16(len) + rem; }

// Length of the pruned forward transform of T non-zero samples inside an
// N-point transform: the smallest L >= T that divides N and that the radix-V
// plan can split.  The N-point spectrum is then N/L twiddled L-point
// transforms of the zero-padded samples.
__host__ __device__ constexpr int prune_len(int T, int N, int V) {
    for (int L = T; L <= N; L++)
        if (N % L == 0 && tmfft::plannable(L, V)) return L;
    return -1;
}
// values per thread of the column transforms: 16 for powers of two, 18 for
// heights with a factor 3
__host__ __device__ constexpr int col_radix(int Y) { return Y % 3 == 0 ? 18 : 16; }

// Layout of the FP32 correlation spectra C between passes B and C of a height Y: tiles of
// c_tile_rows(Y) rows x 4 columns, C[o][y / R][kx / 4][y % R][kx % 4].  A column pass writes 4
// columns of every row of one orientation: in this layout whole tiles of 256 bytes (128
// where 8 does not divide the height) instead of 32-byte pieces of rows 16 KB apart, which the
// memory takes at 5.5 instead of 2.7-3.0 TB/s (a store-only kernel, 2.15 GB, 4096 x 4096).  The
// row pass gathers a row's 32-byte pieces by tensor-map copies; the blocks on the R rows
// of a tile read it at about the same time, through the L2 (4.8-5.5 TB/s in a load-only
// kernel, against 7.2 for whole rows; it needs 2.8).
__host__ __device__ constexpr int c_tile_rows(int Y) { return Y % 8 == 0 ? 8 : Y % 4 == 0 ? 4 : Y % 2 == 0 ? 2 : 1; }
__host__ __device__ inline size_t c_index_rt(int Y, int o, int y, int kx, int XP) {
    const int R = c_tile_rows(Y);
    return (((size_t)o * (Y / R) + y / R) * (XP / 4) + kx / 4) * (4 * R) + (y % R) * 4 + kx % 4;
}
template <int Y>
__host__ __device__ constexpr size_t c_index(int o, int y, int kx, int XP) {
    constexpr int R = c_tile_rows(Y);
    static_assert(R >= 4, "compiled heights are whole tiles of at least 4 rows");
    return (((size_t)o * (Y / R) + y / R) * (XP / 4) + kx / 4) * (4 * R) + (y % R) * 4 + kx % 4;
}
// A row of C in the row pass's shared memory: its XP / 4 column groups arrive in c_row_boxes(XP)
// copies of c_row_box(XP) groups (at most 256, a multiple of 4 for 128-byte aligned pieces)
__host__ __device__ constexpr int c_row_boxes(int XP) { return (XP / 4 + 255) / 256; }
__host__ __device__ constexpr int c_row_box(int XP) {
    return ((XP / 4 + c_row_boxes(XP) - 1) / c_row_boxes(XP) + 3) / 4 * 4;
}
__host__ __device__ constexpr int c_row_len(int XP) { return 4 * c_row_boxes(XP) * c_row_box(XP); }   // float2

struct BatchArgs {
    int nb;                       // orientations in this batch
    int orient0;                  // index of the batch's first orientation within the plane
    long long gidx0;              // global orientation index of the batch's first orientation
    const float* rot;             // plane rotation table: 6 floats per orientation (m00 m01 m10 m11 m20 m21)
    const float2* tmpl;           // T*T*(T/2+1) template spectrum
    const float* filter;          // T*(T/2+1) projection filter
    float2* S;                    // nb * T * (T/2+1)
    float* P;                     // nb * T * T
    double* rowstat;              // nb * T * 4
    float2* norm;                 // nb: (edge mean, 1/sigma)
    float2* A;                    // nb * T * XP
    float2* C;                    // nb * Y * XP, tiled (c_index); the FP16 form's own layout
    const float2* Ip;             // Y * XP prepared micrograph spectrum
    float* mip;                   // Y * X
    int* best;                    // Y * X
    int* best_parts;              // best of a divided batch's parts 1, 2, ...: kPassCParts - 1 planes of Y * X (or null)
    double* sum;                  // Y * X
    double* sumsq;                // Y * X
    unsigned long long* hist;     // hist_bins
    float hist_min, hist_inv_step;
    int hist_bins;
    int* err;                     // device error flag (a bounded wait ran out)
    int half_scale_exp;           // FP16 form: the correlation spectra are stored times 2^half_scale_exp
    int tc_iexp, tc_zexp;         // FP16 column pass: I' held times 2^tc_iexp, stage-1 operand Z times 2^tc_zexp
    long long norm_pixels;        // pixel count of the projection variance (0: X*Y, the box;
                                  // a window of a larger micrograph passes the micrograph's)
    int XP;                       // row pitch (complex values) of A, C and Ip: X/2+1 rounded
                                  // up to a multiple of the pass-B column chunk
    Twiddles tw;                  // x axis (passes A and C): every length divides X
    Twiddles twy;                 // y axis (pass B): every length divides Y
    Twiddles twt;                 // template box (slice and projection kernels): lengths divide T
};

// --------------------------------------------------------------------------------------
// Trilinear Fourier interpolation with the reference's bounds and Hermitian rules
// (Image::ReturnLinearInterpolatedFourier, image.cpp:2899-3020), even T.
//
// N samples at once, without branches: a sample with x < 0 is the conjugate of the one at
// the mirrored indices, and a sample outside the box is zero, so that all 8 N loads are
// independent and in flight together.  (One sample at a time, with a branch for the mirrored
// ones, a block waited for memory once per sample: 24-29 us for a slice of 32 to 128.)
template <int T, int N>
__device__ __forceinline__ void interp3(const float2* __restrict__ vol, const float (&x)[N], const float (&y)[N],
                                        const float (&z)[N], float2 (&out)[N]) {
    constexpr int TP = T / 2 + 1;
    const int lb = -(T / 2), ub = T / 2 - 1;
    float2 v[N][2][2][2];
    bool neg[N], in[N];
    int i0[N], j0[N], k0[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
        neg[n] = !(x[n] >= 0.f);
        i0[n] = (int)floorf(x[n]);
        j0[n] = (int)floorf(y[n]);
        k0[n] = (int)floorf(z[n]);
        in[n] = (neg[n] ? i0[n] >= -(T / 2) : i0[n] + 1 <= T / 2) && j0[n] >= lb && j0[n] + 1 <= ub && k0[n] >= lb && k0[n] + 1 <= ub;
        const int px = neg[n] ? -i0[n] : i0[n], step = neg[n] ? -1 : 1;
#pragma unroll
        for (int dk = 0; dk < 2; dk++) {
            const int kk = neg[n] ? -(k0[n] + dk) : k0[n] + dk;
            const int pz = kk >= 0 ? kk : T + kk;
#pragma unroll
            for (int dj = 0; dj < 2; dj++) {
                const int jj = neg[n] ? -(j0[n] + dj) : j0[n] + dj;
                const int py = jj >= 0 ? jj : T + jj;
                const float2* at = vol + (in[n] ? (pz * T + py) * TP + px : 0);
                v[n][dk][dj][0] = __ldg(at);
                v[n][dk][dj][1] = __ldg(at + (in[n] ? step : 0));
            }
        }
    }
#pragma unroll
    for (int n = 0; n < N; n++) {
        float2 acc = make_float2(0.f, 0.f);
        const float wx1 = x[n] - (float)i0[n], wx0 = 1.f - wx1;
#pragma unroll
        for (int dk = 0; dk < 2; dk++) {
            const float wz = 1.f - fabsf(z[n] - (float)(k0[n] + dk));
#pragma unroll
            for (int dj = 0; dj < 2; dj++) {
                const float w = wz * (1.f - fabsf(y[n] - (float)(j0[n] + dj)));
                const float2 a = v[n][dk][dj][0], b = v[n][dk][dj][1];
                acc.x = fmaf(a.x, w * wx0, acc.x);
                acc.y = fmaf(a.y, w * wx0, acc.y);
                acc.x = fmaf(b.x, w * wx1, acc.x);
                acc.y = fmaf(b.y, w * wx1, acc.y);
            }
        }
        out[n] = in[n] ? make_float2(acc.x, neg[n] ? -acc.y : acc.y) : make_float2(0.f, 0.f);
    }
}

// --------------------------------------------------------------------------------------
// k_slice_colfft: block = CB columns x (T/V) threads (column fastest);
// grid = (ceil((T/2+1)/CB), nb)
template <int T>
struct SliceCol {
    static constexpr int V = T % 3 == 0 ? 24 : 16;   // values per thread
    static constexpr int PT = T / V;                 // threads per column
    static constexpr int RS = skewed(tmfft::padded_len(T), 1);
    static constexpr int CB = (16 * RS * 8 <= 48 * 1024) ? 16 : (8 * RS * 8 <= 48 * 1024) ? 8 : 4;   // columns per block
    static constexpr int NT = CB * PT;
};

template <int T>
__global__ void __launch_bounds__(SliceCol<T>::NT)
k_slice_colfft(BatchArgs a) {
    using SC = SliceCol<T>;
    constexpr int TP = T / 2 + 1;
    constexpr int PT = SC::PT, V = SC::V, CB = SC::CB, RS = SC::RS;
    __shared__ float2 sm[CB * RS];
    const int il = threadIdx.x % CB, tp = threadIdx.x / CB;
    const int i = blockIdx.x * CB + il;
    const int o = blockIdx.y;
    const bool valid = i <= T / 2;
    const float* m = a.rot + 6 * (size_t)(a.orient0 + o);
    const float m00 = __ldg(m), m01 = __ldg(m + 1), m10 = __ldg(m + 2), m11 = __ldg(m + 3), m20 = __ldg(m + 4), m21 = __ldg(m + 5);
    float2 v[V];
    constexpr int N = 4;   // samples interpolated together
#pragma unroll
    for (int r0 = 0; r0 < V; r0 += N) {
        float cx[N], cy[N], cz[N], f[N];
        float2 val[N];
#pragma unroll
        for (int n = 0; n < N; n++) {
            const int y = tp + PT * (r0 + n);
            const int j = y < T / 2 ? y : y - T;
            // column 0: j > 0 and j = -T/2 interpolate at (0, j); other j < 0 mirror (0, -j)
            const int jj = (i > 0 || j > 0 || j == -(T / 2)) ? j : -j;
            // RotateCoords (matrix.h:32-37) in float without fused multiply-add,
            // so that samples on the box boundary are kept or dropped exactly
            // as the reference does
            const float fx = (float)i, fy = (float)jj;
            cx[n] = __fadd_rn(__fmul_rn(m00, fx), __fmul_rn(m01, fy));
            cy[n] = __fadd_rn(__fmul_rn(m10, fx), __fmul_rn(m11, fy));
            cz[n] = __fadd_rn(__fmul_rn(m20, fx), __fmul_rn(m21, fy));
            f[n] = valid ? __ldg(a.filter + (size_t)y * TP + i) : 0.f;
        }
        interp3<T, N>(a.tmpl, cx, cy, cz, val);
#pragma unroll
        for (int n = 0; n < N; n++) {
            const int y = tp + PT * (r0 + n);
            const int j = y < T / 2 ? y : y - T;
            if (i == 0 && j < 0 && j != -(T / 2)) val[n].y = -val[n].y;
            if (!valid || (i == 0 && j == 0)) val[n] = make_float2(0.f, 0.f);
            const float fs = (i + j) & 1 ? -f[n] : f[n];
            v[r0 + n] = make_float2(__fmul_rn(val[n].x, fs), __fmul_rn(val[n].y, fs));   // (not fused into the transform)
        }
    }
    tmfft::fft<T, V, +1>(v, tp, sm + il * RS, a.twt, [] __device__() { __syncthreads(); });
    if (valid) {
        float2* out = a.S + (size_t)o * T * TP;
#pragma unroll
        for (int r = 0; r < V; r++) out[(size_t)(tp + PT * r) * TP + i] = v[r];
    }
}

// --------------------------------------------------------------------------------------
// k_row_c2r: each row of T/2+1 complex -> T reals via a T/2-point inverse FFT
// (even/odd packing; imaginary parts of the DC and Nyquist terms ignored as in
// FFTW's c2r).  block = ROWS rows x PH threads; grid = (T/ROWS, nb).
template <int T>
struct RowC2R {
    static constexpr int H = T / 2;
    static constexpr int V = H % 3 == 0 ? 24 : 16;              // values per thread
    static constexpr int PH = H / V;                            // threads per row
    static constexpr int RS = skewed(tmfft::padded_len(H), PH % 16);
    static constexpr int ROWS0 = (256 / PH) < T ? (256 / PH) : T;
    static constexpr int ROWS = (ROWS0 * RS * 8 <= 48 * 1024) ? ROWS0 : ROWS0 / 2;   // rows per block
    static constexpr int NT = ROWS * PH;
    static_assert(32 % PH == 0 || PH % 32 == 0, "row reductions use warp shuffles");
};

template <int T>
__global__ void __launch_bounds__(RowC2R<T>::NT)
k_row_c2r(BatchArgs a) {
    using RC = RowC2R<T>;
    constexpr int TP = T / 2 + 1, H = RC::H, PH = RC::PH, ROWS = RC::ROWS, V = RC::V;
    constexpr int RS = RC::RS;
    __shared__ float2 sm[ROWS * RS];
    const int t = threadIdx.x % PH, rl = threadIdx.x / PH;
    const int y = blockIdx.x * ROWS + rl;
    const int o = blockIdx.y;
    const float2* Hrow = a.S + ((size_t)o * T + y) * TP;
    float2 v[V];
#pragma unroll
    for (int r = 0; r < V; r++) {
        const int k = t + PH * r;
        float2 hk = Hrow[k];
        float2 hm = Hrow[H - k];
        if (k == 0) { hk.y = 0.f; hm.y = 0.f; }
        const float2 e = make_float2(hk.x + hm.x, hk.y - hm.y);
        const float2 d = make_float2(hk.x - hm.x, hk.y + hm.y);
        const float2 od = cmul(d, a.twt.template w<+1>(k, T));
        v[r] = make_float2(e.x - od.y, e.y + od.x);
    }
    tmfft::fft<H, V, +1>(v, t, sm + rl * RS, a.twt, [] __device__() { __syncthreads(); });
    float* prow = a.P + ((size_t)o * T + y) * T;
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int r = 0; r < V; r++) {
        const int mm = t + PH * r;
        reinterpret_cast<float2*>(prow)[mm] = v[r];
        s += v[r].x + v[r].y;
        q = fmaf(v[r].x, v[r].x, fmaf(v[r].y, v[r].y, q));
    }
    double ds = s, dq = q;
#pragma unroll
    for (int off = PH / 2; off > 0; off >>= 1) {
        ds += __shfl_xor_sync(0xffffffffu, ds, off);
        dq += __shfl_xor_sync(0xffffffffu, dq, off);
    }
    // edge sum: full first and last rows, else the first and last pixel
    float e0 = 0.f, e1 = 0.f;
    if (t == 0) e0 = v[0].x;                                   // pixel 0 = z[0].x
    if (t == (H - 1) % PH) e1 = v[(H - 1) / PH].y;            // pixel T-1 = z[H-1].y
    float ee = e0 + e1;
#pragma unroll
    for (int off = PH / 2; off > 0; off >>= 1) ee += __shfl_xor_sync(0xffffffffu, ee, off);
    const double edge = (y == 0 || y == T - 1) ? ds : (double)ee;
    if (t == 0) {
        double* st = a.rowstat + ((size_t)o * T + y) * 4;
        st[0] = ds;
        st[1] = dq;
        st[2] = edge;
        st[3] = 0.0;
    }
}

// --------------------------------------------------------------------------------------
// k_norm: one warp per orientation.  e = edge mean (ReturnAverageOfRealValuesOnEdges,
// image.cpp:5907-5945); variance as match_template.cpp:1066-1067 with the
// mean of squares and the mean of the edge-subtracted projection.
template <int T>
__global__ void __launch_bounds__(256)
k_norm(BatchArgs a, long long n_image) {
    const int lane = threadIdx.x & 31;
    const int o = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (o >= a.nb) return;
    double s = 0, q = 0, e = 0;
    for (int y = lane; y < T; y += 32) {
        const double* st = a.rowstat + ((size_t)o * T + y) * 4;
        s += st[0];
        q += st[1];
        e += st[2];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
        e += __shfl_xor_sync(0xffffffffu, e, off);
    }
    if (lane == 0) {
        const double n = (double)T * T;
        const float edge_mean = (float)(e / (double)(4 * T - 4));
        const double em = edge_mean;
        const double s1 = s - n * em;                 // sum of (p - e)
        const double s2 = q - 2.0 * em * s + n * em * em;  // sum of (p - e)^2
        const double ratio = n / (double)n_image;
        const double var = (s2 / n) * ratio - ((s1 / n) * ratio) * ((s1 / n) * ratio);
        a.norm[o] = make_float2(edge_mean, (float)(1.0 / sqrt(var)));
    }
}

// --------------------------------------------------------------------------------------
// k_pass_a: one block per (row, orientation); X/16 threads, thread j = s + MX*t'.
// The T samples are the first T of an LA-point zero-padded input (LA = T when T
// divides X).
template <int T, int X>
__global__ void __launch_bounds__(X / 16)
k_pass_a(BatchArgs a) {
    const int XP = a.XP;
    constexpr int LA = prune_len(T, X, 16);
    constexpr int MX = X / LA, PT = LA / 16;
    constexpr int RS = skewed(tmfft::padded_len(LA), 1);
    static_assert(LA > 0, "no pruned row transform for this template and width");
    __shared__ float2 sm[MX * RS];
    __shared__ float q[T];
    const int j = threadIdx.x;
    const int s = j % MX, tp = j / MX;
    const int row = blockIdx.x, o = blockIdx.y;
    const float2 nrm = a.norm[o];
    const float* prow = a.P + ((size_t)o * T + row) * T;
    for (int m = j; m < T; m += X / 16) q[m] = (prow[m] - nrm.x) * nrm.y;
    __syncthreads();
    float2 v[16];
    const float2 w0 = a.tw.template w<-1>(s * tp, X);
    const float2 w1 = a.tw.template w<-1>(s * PT, X);
    float2 w = w0;
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int n = tp + PT * r;
        const float qv = (LA == T || n < T) ? q[n] : 0.f;
        v[r] = make_float2(qv * w.x, qv * w.y);
        w = cmul(w, w1);
    }
    tmfft::fft<LA, 16, -1>(v, tp, sm + s * RS, a.tw, [] __device__() { __syncthreads(); });
    float2* out = a.A + ((size_t)o * T + row) * XP;
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int kx = j + (X / 16) * r;
        if (kx <= X / 2) out[kx] = v[r];
    }
}

// --------------------------------------------------------------------------------------
// Work items of the column passes: (column group, orientation).  A block owns
// whole column groups, every orientation of a group in turn (its micrograph
// values stay in TMEM), and the blocks take adjacent groups in rounds: block b
// has groups b, b + nblk, b + 2 nblk, ...  All blocks then read the same rows of A and of I',
// 32 bytes of each, and write adjacent tiles at about the same time, so that the memory
// sees whole lines.
// Groups left over after the whole rounds are split by orientation ranges, each block
// on one group, or, where that makes the longest block's list shorter, their items are shared out evenly, in
// runs of consecutive orientations that can cross from one group to the next (257
// groups on 148 blocks, 33 orientations: 0.60 -> 0.53 ms, 39 blocks idled in the last round; 132 groups on 592 blocks,
// 96 orientations: 0.186 -> 0.175).
struct ColSchedule {
    int nb, nblk, b, rounds, tail, n;   // tail: this block's first item of the groups left over
    __host__ __device__ ColSchedule(int ngroups, int nbatch, int blk, int nblocks) : nb(nbatch), nblk(nblocks), b(blk) {
        rounds = ngroups / nblk;
        const int rem = ngroups % nblk;
        const int parts = rem ? min(nb, nblk / rem) : 1;
        const int left = rem * nb, each = left / nblk, more = left - each * nblk;
        int end = 0;
        tail = 0;
        if ((nb + parts - 1) / parts > each + (more > 0)) {
            tail = b * each + min(b, more);
            end = tail + each + (b < more);
        } else if (b < rem * parts) {
            const int p = b / rem;
            tail = b % rem * nb + p * nb / parts;
            end = b % rem * nb + (p + 1) * nb / parts;
        }
        n = rounds * nb + end - tail;
    }
    // most items a block gets
    __host__ __device__ static int max_items(int ngroups, int nbatch, int nblocks) {
        return (ngroups + nblocks - 1) / nblocks * nbatch;
    }
    // (group, orientation) of the block's idx-th item.  k_pass_b keeps the schedule
    // in shared memory (its fields cost no registers across the item loop);
    // k_pass_b_rg expands it into a list of items there.
    __host__ __device__ void locate(int idx, int& g, int& o) const { place(nb, nblk, b, rounds, tail, idx, g, o); }
    // the same from the block's shared-memory copy, read afresh on every call
    __device__ static void locate(const volatile ColSchedule* s, int idx, int& g, int& o) {
        place(s->nb, s->nblk, s->b, s->rounds, s->tail, idx, g, o);
    }

private:
    __host__ __device__ static void place(int nb, int nblk, int b, int rounds, int tail, int idx, int& g, int& o) {
        if (idx < rounds * nb) {
            g = (idx / nb) * nblk + b;
            o = idx % nb;
        } else {
            const int i = tail + idx - rounds * nb;
            g = rounds * nblk + i / nb;
            o = i % nb;
        }
    }
};
static_assert(sizeof(ColSchedule) <= 48, "the schedule sits in the last 48 bytes of a column pass's shared memory");

// --------------------------------------------------------------------------------------
// k_pass_b: persistent; block = W columns x P / 2 threads (thread = cp + W/2 j, P = Y/V),
// two adjacent columns per thread (tmfft::Pair); work item = (group of W columns,
// orientation), orientation fastest.  Each thread parks the V values of the prepared
// micrograph spectrum I' of its two columns in tensor memory (TMEM, 4V columns of its lane)
// for all orientations of the group, which leaves shared memory to the exchange buffer, 16
// bytes per element and column pair.  Blocks are padded to whole warps (tcgen05 loads
// are whole-warp operations); the padding lanes repeat the last thread's work without storing it.
// The rows of A for the next item stream in with cp.async while the current item is
// transformed.  Twiddles come from tables of the stages' bases in shared memory (from the
// L2, all warps of a block waited for them at each stage).
// What bounds it: the FP32 pipe (44 % busy at 256 x 3888; one item's loads, butterflies and stores take turns
// at the block's barriers), then its writes of C.  One column per thread -> this, 32
// orientations of 4096 columns: 256 x 3888 1.52 -> 1.46 ms, 384 x 5832 3.36 -> 2.39; 33 of 2048 columns: 256 x 2916 0.70
// -> 0.53, 256 x 2592 0.85 -> 0.70; 96 of 1024: 64 x 1024 0.21 -> 0.17; 96 of 512: 256 x 512 0.073 -> 0.059; the
// smallest lose a little (96 of 256: 32 x 256 0.023 -> 0.025).  (At 5832, both pairs of a thread one after the other, without spills but
// with 11 warps: 2.73 ms.)
// The forward transform along y is pruned: MY = Y/L twiddled L-point transforms
// of the T rows of A zero-padded to L (L = T for power-of-two heights).
template <int T, int Y>
struct PassB {
    static constexpr int V = col_radix(Y);                          // values per thread: the column radix
    static constexpr int P = Y / V;                                 // threads per column pair
    static constexpr int W = P <= 16 ? 8 : 4;                       // columns per item: one tile of C, or two (at least two warps)
    static constexpr int WP = W / 2;
    static constexpr int NA = WP * P;                               // threads with columns of their own
    static constexpr int NT = (NA + 31) / 32 * 32;
    static constexpr int L = prune_len(T, Y, V);                    // pruned forward length
    static constexpr int MY = Y / L, PT = L / V;
    // Spare elements: one per V in the inverse transform (Stockham strides of V and its powers).  In
    // the forward transforms 8 lanes hold 8 / WP neighbouring threads, of different regions at the
    // same element where there are as many regions, for which an odd distance of the regions is enough.
    static constexpr int D = V, DF = MY * WP >= 8 ? 0 : V;
    static constexpr int RST = (tmfft::pad_at<DF>(L) + 3) / 4 * 4 + (MY == 2 ? 2 : MY == 3 ? 3 : 1);
    static constexpr int CS = (MY * RST > tmfft::pad_at<D>(Y)) ? MY * RST : tmfft::pad_at<D>(Y);
    static constexpr size_t EXCH = sizeof(float4) * WP * CS;
    static constexpr size_t ASZ = sizeof(float4) * T * WP;          // one A staging buffer
    // the transforms' stage tables, then the pruned forward's factors w0, w1 per butterfly
    static constexpr int FTAB = tmfft::stage_table_len<L, V>(), TAB = FTAB + tmfft::stage_table_len<Y, V>();
    static constexpr size_t TABS = (sizeof(float2) * TAB + 15) / 16 * 16 + sizeof(float4) * P;
    static constexpr int ABUFS = (EXCH + TABS + 2 * ASZ + 64 <= 232448) ? 2 : 1;
    static constexpr size_t SMEM = EXCH + ABUFS * ASZ + TABS + 64;  // + TMEM address slot, schedule
    // TMEM: 4V columns per thread; the warps of one lane quadrant sit side by side
    static constexpr int TCOLS = 4 * V;
    static constexpr uint32_t TMEM_COLS = [] {
        const int need = (NT / 32 + 3) / 4 * TCOLS;
        uint32_t n = 32;
        while ((int)n < need) n *= 2;
        return n;
    }();
    // resident blocks per SM: 128 registers per thread, shared memory, TMEM
    static constexpr int BPS = [] {
        int n = 512 / NT;
        if (n * (SMEM + 1024) > 233472) n = (int)(233472 / (SMEM + 1024));
        if (n * (int)TMEM_COLS > 512) n = 512 / (int)TMEM_COLS;
        return n < 1 ? 1 : n;
    }();
    // the addresses of radix-18 exchanges are worked out for each item where registers are few: kept
    // over the items they spill (256 x 3888, 32 orientations: 1.55 ms, 1.46 so; where they fit, a few percent
    // are lost)
    static constexpr bool ADDRESSES_ANEW = V == 18 && NT * BPS > 384;
    static_assert(L > 0 && Y % V == 0 && P % PT == 0, "no pruned plan for this template and height");
    static_assert(NT <= 1024 && SMEM <= 232448, "pass B block exceeds the per-block limits");
    static_assert(TMEM_COLS <= 512, "pass B TMEM layout exceeds 512 columns");
    static_assert(V == 16 || V == 18, "TMEM load sequence covers 16 or 18 values");
};

// RB = 0: FP32 complex, tiled (c_index).  RB > 0 (the FP16 form): C in FP16
// complex times 2^half_scale_exp, rows interleaved in blocks of RB,
// C16[o][y / RB][kx][y % RB], so that a warp's stores (16 consecutive rows of a
// column) fill whole 32-byte sectors and the tensor-core row pass reads a
// block of RB rows with one bulk copy.
template <int T, int Y, int RB = 0>
__global__ void __launch_bounds__(PassB<T, Y>::NT, PassB<T, Y>::BPS)
k_pass_b(BatchArgs a, int ngroups) {
    using PB = PassB<T, Y>;
    using tmfft::Pair;
    constexpr int W = PB::W, WP = PB::WP, MY = PB::MY, PT = PB::PT, NT = PB::NT, V = PB::V, P = PB::P, L = PB::L;
    const int XP = a.XP;
    extern __shared__ __align__(128) unsigned char smem_b[];
    float4* exch = reinterpret_cast<float4*>(smem_b);
    float4* abuf = reinterpret_cast<float4*>(smem_b + PB::EXCH);
    float4* w01 = reinterpret_cast<float4*>(smem_b + PB::EXCH + PB::ABUFS * PB::ASZ);
    float2* tab = reinterpret_cast<float2*>(w01 + P);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_b + PB::SMEM - 64);
    volatile ColSchedule* sch = reinterpret_cast<volatile ColSchedule*>(smem_b + PB::SMEM - 48);
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const bool act = PB::NA == NT || tid < PB::NA;
    const int cp = tid % WP, j0 = act ? tid / WP : P - 1;   // column pair, butterfly
    auto sync = [] { __syncthreads(); };
    if (tid == 0) {
        const ColSchedule cs(ngroups, a.nb, blockIdx.x, gridDim.x);
        sch->nb = cs.nb; sch->nblk = cs.nblk; sch->b = cs.b; sch->rounds = cs.rounds;
        sch->tail = cs.tail; sch->n = cs.n;
    }
    __syncthreads();
    const int n_items = sch->n;
    if (n_items == 0) return;
    if (warp == 0) {
        tmptx::tmem_alloc(tmem_slot, PB::TMEM_COLS);
        tmptx::tmem_relinquish();
    }
    tmfft::fill_stage_table<L, V>(tab, a.twy, tid, NT);
    tmfft::fill_stage_table<Y, V>(tab + PB::FTAB, a.twy, tid, NT);
    for (int i = tid; i < P; i += NT) {
        // twiddles of the pruned forward, W_Y^(s * (tp + PT*r)) = w0 * w1^r
        const float2 w0 = a.twy.template w<-1>((i % MY) * (i / MY), Y), w1 = a.twy.template w<-1>((i % MY) * PT, Y);
        w01[i] = make_float4(w0.x, w0.y, w1.x, w1.y);
    }
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    const uint32_t tmem = *tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(PB::TCOLS * (warp >> 2));
    // the item's T rows of A into dst[row][column pair]
    auto issue_rows = [&](int it, float4* dst) {
        int grp, oo;
        ColSchedule::locate(sch, it, grp, oo);
        const float2* src = a.A + (size_t)oo * T * XP + grp * W;
        for (int e = tid; e < T * WP; e += NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tmptx::smem_u32(dst + e)),
                         "l"(src + (size_t)(e / WP) * XP + 2 * (e % WP))
                         : "memory");
    };
    if (PB::ABUFS == 2) {
        issue_rows(0, abuf);
        tmptx::cp_async_commit();
    }
    float4* const colbuf = exch + cp;
    int cur_group = -1;
#pragma unroll 1
    for (int it = 0; it < n_items; it++) {
        const float4* acur = abuf + (PB::ABUFS == 2 ? (it & 1) : 0) * (T * WP) + cp;
        float4* anext = abuf + (PB::ABUFS == 2 ? ((it + 1) & 1) : 0) * (T * WP);
        int group, o;
        ColSchedule::locate(sch, it, group, o);
        const int kx = group * W + 2 * cp;
        int j = j0;
        if constexpr (PB::ADDRESSES_ANEW) asm volatile("" : "+r"(j));
        const int s = j % MY, tp = j / MY;   // residue of the pruned forward, its butterfly
        float4* const fwdbuf = colbuf + s * PB::RST * WP;
        // The buffer the next rows go into was last read at the start of the
        // previous item's forward transform, whose barriers every thread has
        // passed; the exchange buffer is guarded by the transforms' own barriers.
        // With a single staging buffer the rows are reloaded in place, after a barrier.
        if (PB::ABUFS == 1) sync();
        if (PB::ABUFS == 2) {
            if (it + 1 < n_items) issue_rows(it + 1, anext);
            tmptx::cp_async_commit();
            tmptx::cp_async_wait<1>();
        } else {
            issue_rows(it, anext);
            tmptx::cp_async_commit();
            tmptx::cp_async_wait<0>();
        }
        sync();  // this item's rows of A are visible to every thread
        if (group != cur_group) {
            // the V I' values of each of this thread's columns, k = j + P r, as column pairs of
            // the real and the imaginary parts
            const float2* Ig = a.Ip + (size_t)j * XP + kx;
            auto fetch = [&](float* f, int r) {
                const float4 iv = __ldg(reinterpret_cast<const float4*>(Ig + (size_t)P * r * XP));
                f[0] = iv.x;
                f[1] = iv.z;
                f[2] = iv.y;
                f[3] = iv.w;
            };
#pragma unroll 1
            for (int h = 0; h < 4; h++) {
                float ib[16];
#pragma unroll
                for (int r = 0; r < 4; r++) fetch(ib + 4 * r, 4 * h + r);
                tmptx::tmem_st16(tmem + 16 * h, ib);
            }
            if constexpr (V == 18) {
                float ib[8];
                fetch(ib, 16);
                fetch(ib + 4, 17);
                tmptx::tmem_st8(tmem + 64, ib);
            }
            tmptx::tmem_wait_st();
            cur_group = group;
        }
        Pair v[V];
        {
            const float4 ww = w01[j];
            float2 w = make_float2(ww.x, ww.y);
            const float2 w1 = make_float2(ww.z, ww.w);
#pragma unroll
            for (int r = 0; r < V; r++) {
                const int n = tp + PT * r;   // rows n >= T of the L-point input are zero
                const bool in = L == T || n < T;
                const float4 f = acur[(in ? n : 0) * WP];
                const Pair x = tmfft::pmul({make_float2(f.x, f.z), make_float2(f.y, f.w)}, w);
                v[r] = in ? x : Pair{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                w = cmul(w, w1);
            }
        }
        // every thread passed the item barrier since the buffer was last read
        tmfft::pfft<L, V, -1, WP, PB::DF, false>(v, tp, fwdbuf, tab, act, sync);
        // thread (s, tp) holds F[k], k = s + MY*(tp + PT*r) = j + P*r
        {
            float iv[16], iw[16];
            auto mul = [&](int r, const float* f) {
                v[r] = tmfft::pmul_conj(make_float2(f[0], f[1]), make_float2(f[2], f[3]), v[r]);
            };
            tmptx::tmem_ld16(tmem, iv);
            tmptx::tmem_wait_ld16(iv);
            tmptx::tmem_ld16(tmem + 16, iw);   // in flight while the first values are multiplied
#pragma unroll
            for (int r = 0; r < 4; r++) mul(r, iv + 4 * r);
            tmptx::tmem_wait_ld16(iw);
            tmptx::tmem_ld16(tmem + 32, iv);
#pragma unroll
            for (int r = 0; r < 4; r++) mul(4 + r, iw + 4 * r);
            tmptx::tmem_wait_ld16(iv);
            tmptx::tmem_ld16(tmem + 48, iw);
#pragma unroll
            for (int r = 0; r < 4; r++) mul(8 + r, iv + 4 * r);
            tmptx::tmem_wait_ld16(iw);
            if constexpr (V == 18) tmptx::tmem_ld8(tmem + 64, iv);
#pragma unroll
            for (int r = 0; r < 4; r++) mul(12 + r, iw + 4 * r);
            if constexpr (V == 18) {
                tmptx::tmem_wait_ld16(iv);
                mul(16, iv);
                mul(17, iv + 4);
            }
        }
        tmfft::pfft<Y, V, +1, WP, PB::D>(v, j, colbuf, tab + PB::FTAB, act, sync);
        if (!act) continue;
        if constexpr (RB > 0) {
            static_assert(Y % RB == 0 && (P % RB == 0), "a thread's rows sit at one position of their blocks");
            // row j + P r sits in block j / RB + r P / RB at position j % RB (RB divides P)
            const float sc = __int_as_float((127 + a.half_scale_exp) << 23);   // 2^e
            __half2* Co = reinterpret_cast<__half2*>(a.C) + (size_t)o * Y * XP + ((size_t)(j / RB) * XP + kx) * RB + (j % RB);
#pragma unroll
            for (int r = 0; r < V; r++) {   // streaming stores, as the FP32 output
                const __half2 h0 = __floats2half2_rn(v[r].re.x * sc, v[r].im.x * sc);
                const __half2 h1 = __floats2half2_rn(v[r].re.y * sc, v[r].im.y * sc);
                __stcs(reinterpret_cast<unsigned int*>(Co + (size_t)r * P * XP), *reinterpret_cast<const unsigned int*>(&h0));
                __stcs(reinterpret_cast<unsigned int*>(Co + (size_t)r * P * XP + RB), *reinterpret_cast<const unsigned int*>(&h1));
            }
        } else {
            // Rows that a whole number of tiles lies between are that many rows of XP apart: the
            // rows of even r from the first's place, those of odd r from the second's
            static_assert(2 * P % c_tile_rows(Y) == 0, "every second row of a thread sits at one position of its tile");
            float2* const C0 = a.C + c_index<Y>(o, j, kx, XP);
            float2* const C1 = P % c_tile_rows(Y) == 0 ? C0 + (size_t)P * XP : a.C + c_index<Y>(o, j + P, kx, XP);
#pragma unroll
            for (int r = 0; r < V; r++)   // streaming; a warp writes whole tiles
                __stcs(reinterpret_cast<float4*>((r % 2 ? C1 : C0) + (size_t)(r / 2) * 2 * P * XP),
                       make_float4(v[r].re.x, v[r].im.x, v[r].re.y, v[r].im.y));
        }
    }
    tmptx::cp_async_wait<0>();
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    if (warp == 0) tmptx::tmem_dealloc(*tmem_slot, PB::TMEM_COLS);
}

// --------------------------------------------------------------------------------------
// k_pass_b_rg: the column pass of 4096-high micrographs with 256-row pruned
// transforms (T = 256), arranged so that two of its three exchanges stay
// inside a warp.  Write the column spectrum index k = s + 16 k1 + 256 k2 and
// the output row m = m' + 256 M (s, k1, k2, M in 0..15, m' in 0..255).  Both
// transforms split by the residue s = k mod 16:
//   F[s + 16 k'] = sum_{n<256} (a[n] W4096^(-n s)) W256^(-n k')
//   y[m' + 256 M] = sum_s (W4096^(m' s) G_s[m']) W16^(M s),
//   G_s[m'] = sum_{k'} Z[s + 16 k'] W256^(m' k'),   Z = I' conj(F)
// (W_N^e = exp(2 pi i e / N)).  A residue's 256 values live in the 16 lanes of
// one half-warp from the forward 256-point transform through the multiply by
// I' to G_s: each 256-point transform is 16 x 16 with one transpose through
// the warp's own shared memory (__syncwarp only).  One block-wide exchange
// then gathers the 16 residues of each output row m' for the last 16-point
// DFT.  Per item (4 columns of one orientation) that is two block barriers
// instead of the six of k_pass_b's Stockham stages.
//
// Two adjacent columns go through a thread side by side (tmfft::Pair): additions and the
// constants of the 16-point transforms take one instruction for both, the twiddles are
// fetched once, and shared memory is accessed 16 bytes at a time.
//
// Roles: residue phases -- warp s holds residue s, lane 2 q + cp the columns 2 cp and 2 cp + 1
// of line q; final phase -- thread 2 m' + cp holds row m' of those columns.  The block buffer is
// blk[s][m'][cp], 16 bytes each: every phase accesses 128 adjacent bytes per 8 lanes.  In the
// final phase a thread puts its 16 output rows m' + 256 M back where it read its 16 residues, so
// that the buffer becomes the item's 512 tiles of C, [M][m'][cp], and two tensor-map stores
// write it to memory while the next item's residue phases run (with stores from the
// threads, all of which reach them together, the pass took 3.85 ms per 128 orientations against 2.93 with
// the stores left out).  A warp's transposes have buffers of their own, of 8 bytes per element
// for want of shared memory: the real parts of the column pairs go first, then the imaginary parts.
struct PassBRg {
    static constexpr int T = 256, Y = 4096, W = 4, NT = 512;
    static constexpr int RS = 17;                       // row stride of a transpose buffer (float2)
    static constexpr int SCR = 16 * RS + 8;             // one column pair's, == 8 (mod 16)
    static constexpr size_t EXCH = sizeof(float4) * 16 * 256 * 2;
    static constexpr size_t SCRS = sizeof(float2) * 16 * 2 * SCR;
    static constexpr size_t ASZ = sizeof(float4) * 2 * T;   // A staging: [row][column pair]
    static constexpr int ABUFS = 2;                     // rows of A prefetched one item ahead
    static constexpr int MAX_ITEMS = 2048;              // a block's item list (group << 16 | orientation)
    static constexpr size_t LIST = sizeof(int) * MAX_ITEMS;
    static constexpr size_t SMEM = EXCH + SCRS + ABUFS * ASZ + LIST + 64;
    // 4 warps per lane quadrant x 64 columns of I' (columns 0-255), 32 of the twiddles
    // W4096^(-(q + 16 r) s) (256-383) and 32 of the powers W256^(-q r) (384-511)
    static constexpr uint32_t TMEM_COLS = 512;
    static_assert(SMEM <= 232448, "pass B block exceeds shared memory");
};

__global__ void __launch_bounds__(PassBRg::NT, 1)
k_pass_b_rg(BatchArgs a, const __grid_constant__ CUtensorMap cmap, int ngroups) {
    using PB = PassBRg;
    using tmfft::Pair;
    constexpr int T = PB::T, Y = PB::Y, RS = PB::RS;
    extern __shared__ __align__(128) unsigned char smem_b[];
    float4* const blk = reinterpret_cast<float4*>(smem_b);
    float4* const abuf = reinterpret_cast<float4*>(smem_b + PB::EXCH + PB::SCRS);
    int* const items = reinterpret_cast<int*>(smem_b + PB::EXCH + PB::SCRS + PB::ABUFS * PB::ASZ);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_b + PB::EXCH + PB::SCRS + PB::ABUFS * PB::ASZ + PB::LIST);
    const int tid = threadIdx.x;
    // this block's items (the launcher checks that they fit the list)
    int n_items;
    {
        const ColSchedule sch(ngroups, a.nb, blockIdx.x, gridDim.x);
        n_items = sch.n;
        for (int i = tid; i < sch.n; i += PB::NT) {
            int g, o;
            sch.locate(i, g, o);
            items[i] = (g << 16) | o;
        }
    }
    if (n_items == 0) return;
    if ((tid >> 5) == 0) {
        tmptx::tmem_alloc(tmem_slot, PB::TMEM_COLS);
        tmptx::tmem_relinquish();
    }
    // the item's 256 rows of A into the staging buffer (thread: row tid / 2, column pair
    // tid % 2); items are (column group, orientation), orientation fastest
    const float2* const Asrc = a.A + (size_t)(tid >> 1) * a.XP + 2 * (tid & 1);
    const uint32_t adst = tmptx::smem_u32(abuf + tid);
    auto issue_rows = [&](int grp, int oo, int buf) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(adst + buf * (uint32_t)(PB::ASZ)),
                     "l"(Asrc + (size_t)oo * T * a.XP + grp * 4)
                     : "memory");
    };
    tmptx::tmem_fence_before_sync();
    __syncthreads();   // the item list, the TMEM address
    tmptx::tmem_fence_after_sync();
    issue_rows(items[0] >> 16, items[0] & 0xffff, 0);
    tmptx::cp_async_commit();
    const int s = tid >> 5, q = (tid >> 1) & 15, cp = tid & 1;   // residue, line, column pair
    const uint32_t tmem = *tmem_slot + ((uint32_t)(32 * (s & 3)) << 16);
    const uint32_t tmi = tmem + 64 * (s >> 2);         // this thread's I' values
    const uint32_t tmw = tmem + 256 + 32 * (s >> 2);   // W4096^(-(q + 16 r) s), r = 0..15
    const uint32_t tmq = tmem + 384 + 32 * (s >> 2);   // W256^(-q r) by the product tree, r = 0..15
    {
        float2 one[16];
#pragma unroll
        for (int r = 0; r < 16; r++) one[r] = make_float2(1.f, 0.f);
        tmfft::apply_twiddles<16>(one, a.twy.template w<-1>(16 * q, Y));   // 1 w^r = w^r
        float wb[16];
        // in the order of the transforms' groups of four: r = g, g + 4, g + 8, g + 12 for g = 0..3
#pragma unroll
        for (int h = 0; h < 2; h++) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = 2 * h + i / 4 + 4 * (i % 4);
                const float2 w = a.twy.template w<-1>((q + 16 * r) * s, Y);
                wb[2 * i] = w.x;
                wb[2 * i + 1] = w.y;
            }
            tmptx::tmem_st16(tmw + 16 * h, wb);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = 2 * h + i / 4 + 4 * (i % 4);
                wb[2 * i] = one[r].x;
                wb[2 * i + 1] = one[r].y;
            }
            tmptx::tmem_st16(tmq + 16 * h, wb);
        }
        tmptx::tmem_wait_st();
    }
    tmptx::cp_async_wait<0>();
    __syncthreads();   // the first item's rows
    int cur_group = -1;
    auto put = [](float4* at, Pair p) { *at = make_float4(p.re.x, p.re.y, p.im.x, p.im.y); };
    auto get = [](const float4* at) {
        const float4 f = *at;
        return Pair{make_float2(f.x, f.y), make_float2(f.z, f.w)};
    };
#pragma unroll 1
    for (int it = 0; it < n_items; it++) {
        const int group = items[it] >> 16, o = items[it] & 0xffff;
        {
            // rows of item it + 1 into the buffer that item it - 1 used
            if (it + 1 < n_items) issue_rows(items[it + 1] >> 16, items[it + 1] & 0xffff, (it + 1) & 1);
            tmptx::cp_async_commit();
        }
        if (group != cur_group) {
            // this thread's 16 I' values of two columns, k = s + 16 q + 256 r, as column pairs of
            // the real and the imaginary parts
            const float4* Ig = reinterpret_cast<const float4*>(a.Ip + (size_t)(s + 16 * q) * a.XP + group * 4 + 2 * cp);
#pragma unroll 1
            for (int h = 0; h < 4; h++) {
                float ib[16];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float4 iv = __ldg(Ig + (size_t)(128 * (h + 4 * r)) * a.XP);
                    ib[4 * r] = iv.x;
                    ib[4 * r + 1] = iv.z;
                    ib[4 * r + 2] = iv.y;
                    ib[4 * r + 3] = iv.w;
                }
                tmptx::tmem_st16(tmi + 16 * h, ib);
            }
            tmptx::tmem_wait_st();
            cur_group = group;
        }
        // this column pair's transpose buffer: 16 x 16 real or imaginary parts
        float2* const scr = reinterpret_cast<float2*>(smem_b + PB::EXCH) + (2 * s + cp) * PB::SCR;
        // Each 16-point transform goes by groups of four, with the group's loads before its first
        // level and its factors and stores after its second, so that the FP32 pipe and shared
        // memory are busy at the same time (in phases over all 16 values they took turns, all
        // warps being in the same phase: 4.09 ms per 128 orientations).  The factors come from
        // TMEM a group ahead, into the halves of wb in turn.
        Pair v[16];
        float wb[16];
        auto first = [&](uint32_t col) {
            tmptx::tmem_ld8(col, wb);
            tmptx::tmem_ld8(col + 8, wb + 8);
        };
        auto arrived = [&] { tmptx::tmem_wait_ld8x2(wb, wb + 8); };
        auto next = [&](uint32_t col, int g) {
            if (g < 2) tmptx::tmem_ld8(col + 16 + 8 * g, wb + 8 * (g & 1));
        };
        auto factor = [&](int g, int k) { return make_float2(wb[8 * (g & 1) + 2 * k], wb[8 * (g & 1) + 2 * k + 1]); };
        auto mul_by_conj = [](Pair z, float2 w) {
            const float2 x = cmul_conj(make_float2(z.re.x, z.im.x), w), y = cmul_conj(make_float2(z.re.y, z.im.y), w);
            return Pair{make_float2(x.x, y.x), make_float2(x.y, y.y)};
        };
        // forward: b[n] = a[n] W4096^(-n s) for n = q + 16 r, 16-point DFT over r (-> k1), W256^(-q k1)
        {
            const float4* ac = abuf + (it & 1) * (2 * T) + (tid & 31);
            first(tmw);
            tmfft::sfor<4>([&](auto gc) {
                constexpr int g = decltype(gc)::value;
                arrived();
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const float4 f = ac[32 * (g + 4 * k)];
                    v[g + 4 * k] = tmfft::pmul({make_float2(f.x, f.z), make_float2(f.y, f.w)}, factor(g, k));
                }
                next(tmw, g);
                tmfft::pdft4<-1>(v[g], v[4 + g], v[8 + g], v[12 + g]);
            });
        }
        first(tmq);
        tmfft::pdft16_mid<-1>(v);
        tmfft::sfor<4>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            tmfft::pdft4<-1, g == 2>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            arrived();
#pragma unroll
            for (int k = 0; k < 4; k++) {   // row n1 = q, column k1 = g + 4 k
                if (g + k > 0) v[4 * g + k] = tmfft::pmul(v[4 * g + k], factor(g, k));
                scr[RS * q + g + 4 * k] = v[4 * g + k].re;
            }
            next(tmq, g);
        });
        {
            float2 im[16];   // X[r] of the transform just done
#pragma unroll
            for (int r = 0; r < 16; r++) im[r] = v[4 * (r % 4) + r / 4].im;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 16; r++) v[r].re = scr[RS * r + q];   // lane k1 = q holds n1 = r
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 16; r++) scr[RS * q + r] = im[r];
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 4; g++) {
#pragma unroll
            for (int k = 0; k < 4; k++) v[g + 4 * k].im = scr[RS * (g + 4 * k) + q];
            tmfft::pdft4<-1>(v[g], v[4 + g], v[8 + g], v[12 + g]);
        }
        __syncwarp();
        first(tmi);
        tmfft::pdft16_mid<-1>(v);
        // -> k2: F[s + 16 q + 256 r]; Z = I' conj(F); inverse: level 1 of the 16-point DFT over k2 (-> m1)
        tmfft::sfor<4>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            tmfft::pdft4<-1, g == 2>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            arrived();
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[4 * g + k] = tmfft::pmul_conj(make_float2(wb[4 * k], wb[4 * k + 1]), make_float2(wb[4 * k + 2], wb[4 * k + 3]), v[4 * g + k]);
            if constexpr (g < 3) first(tmi + 16 * (g + 1));
            else first(tmq);
            tmfft::pdft4<+1>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        });
        tmfft::pdft16_mid<+1>(v);
        // W256^(m1 q), transpose
        tmfft::sfor<4>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            tmfft::pdft4<+1, g == 2>(v[g], v[4 + g], v[8 + g], v[12 + g]);
            arrived();
#pragma unroll
            for (int k = 0; k < 4; k++) {   // row k1 = q, column m1 = g + 4 k
                if (g + k > 0) v[g + 4 * k] = tmfft::pmul(v[g + 4 * k], tmfft::conjf2(factor(g, k)));
                scr[RS * q + g + 4 * k] = v[g + 4 * k].re;
            }
            next(tmq, g);
        });
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 16; r++) v[r].re = scr[RS * r + q];   // lane m1 = q holds k1 = r
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 16; r++) scr[RS * q + r] = v[r].im;
        __syncwarp();
        // 16-point DFT over k1 (-> m2), then W4096^(s (m1 + 16 m2))
#pragma unroll
        for (int g = 0; g < 4; g++) {
#pragma unroll
            for (int k = 0; k < 4; k++) v[g + 4 * k].im = scr[RS * (g + 4 * k) + q];
            tmfft::pdft4<+1>(v[g], v[4 + g], v[8 + g], v[12 + g]);
        }
        first(tmw);
        tmfft::pdft16_mid<+1>(v);
        tmfft::sfor<4>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            tmfft::pdft4<+1, g == 2>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            arrived();
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * g + k] = mul_by_conj(v[4 * g + k], factor(g, k));
            next(tmw, g);
        });
        // the previous item's stores have read the block buffer
        if (tid == 0) tmptx::bulk_wait_read();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; i++) put(blk + (s * 256 + q + 16 * (i / 4 + 4 * (i % 4))) * 2 + cp, v[i]);   // G_s[m' = q + 16 r]
        tmptx::cp_async_wait<0>();   // the next item's rows (issued at the top of this item)
        __syncthreads();
        // final phase: row m' = tid / 2 of column pair tid % 2; 16-point DFT over the residues (-> M)
#pragma unroll
        for (int g = 0; g < 4; g++) {
#pragma unroll
            for (int k = 0; k < 4; k++) v[g + 4 * k] = get(blk + 512 * (g + 4 * k) + tid);
            tmfft::pdft4<+1>(v[g], v[4 + g], v[8 + g], v[12 + g]);
        }
        tmfft::pdft16_mid<+1>(v);
        tmfft::sfor<4>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            tmfft::pdft4<+1, g == 2>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const Pair z = v[4 * g + k];
                blk[512 * (g + 4 * k) + tid] = make_float4(z.re.x, z.im.x, z.re.y, z.im.y);
            }
        });
        // the item's tiles are complete once every warp has come here; only warp 0 waits for that
        tmptx::fence_proxy_async_smem();
        if (s == 0) {
            asm volatile("bar.sync 1, 512;" ::: "memory");
            if (tid == 0) {
                tmptx::tensor3_s2g(&cmap, 0, group, o * (Y / 8), blk);
                tmptx::tensor3_s2g(&cmap, 0, group, o * (Y / 8) + 256, blk + 4096);
                tmptx::bulk_commit();
            }
        } else {
            asm volatile("bar.arrive 1, 512;" ::: "memory");
        }
    }
    if (tid == 0) tmptx::bulk_wait_all();
    tmptx::cp_async_wait<0>();
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    if ((tid >> 5) == 0) tmptx::tmem_dealloc(*tmem_slot, PB::TMEM_COLS);
}

// --------------------------------------------------------------------------------------
// Copies of a block's shared-memory histogram: lane l counts into copy
// l % n, bin b of copy c at word b * n + c, so that lanes of one warp whose
// values fall in the same bin (the bins near zero take most of them) rarely
// update the same word or bank.  n is the largest power of two up to
// max_copies whose copies fit in 32 KB.
__host__ __device__ inline int hist_copies(int bins, int max_copies) {
    int n = max_copies;
    while (n > 1 && (long long)bins * n * 4 > 32768) n >>= 1;
    return n;
}

// --------------------------------------------------------------------------------------
// k_pass_c: the row pass.  Each row's c2r is an H = X/2-point inverse transform of the
// even/odd packing (8 complex values = 16 pixels per thread, P = X/16 threads per
// row); two orientations go through it side by side (tmfft::Pair), so that the
// additions of both take one instruction, the twiddles are fetched once, the shared-memory
// accesses are 16 bytes wide, and a thread ends with the two values of a pixel next to
// each other: one three-way maximum and one two-wide multiply-add of the histogram.
//
// The transform is the Stockham plan 8, 8, ... of tmfft::fft.  Its butterflies b of stages
// 1, 2, ... fall into 8 groups j = b mod 8 that exchange nothing after the first exchange, so
// group j is put in G = P/8 adjacent lanes (lane l has b = 8 l + j): one exchange over the
// whole row hands group j its P values, every later one stays in the group's part of the
// exchange buffer (__syncwarp only).  That buffer is double, so a pair of orientations
// costs one block barrier instead of twelve, and the warps may run almost a whole pair apart.
// A block has max(1, 128 / P) rows, so that it is made of whole warps in every lane
// quadrant, and goes through the image in steps of the grid (all blocks resident): twiddles
// and histogram are set up once, and the rows of C of the next pair -- the next rows' first
// pair after the last -- arrive by tensor-map copies while a pair is transformed.
//
// The per-pixel sum and sum of squares stay in the thread's TMEM columns 0-63 over the
// batch and go from there to the FP64 running sums.  Below 2048 pixels they are FP64
// sums of every value (EXACT).  From 2048 on they are plain FP32 sums over at most 8
// orientations in registers, added (Kahan) every 8 orientations into compensated FP32 sums.
// Columns 64-127 hold the thread's twiddle multipliers.  The best orientation is written to memory when a pixel's
// maximum changes (the n-th orientation changes it with probability 1/n) and never read.
//
// Small images have too few rows for the chip (512 x 512: 128 blocks of four rows, one or none per SM, each
// waiting for its own latencies: 206 us for 256 orientations): PARTS blocks of a cluster then share a group of
// rows, each with a part of the batch.  Every part starts from the maxima so far and
// keeps its own best orientations; at the end each block merges a share of the pixels over the parts' shared
// memory, in the order of the orientations (a later part has to exceed the earlier ones).
// 512 x 512, 256 orientations: 206 -> 126 us (101 at the rate of 4096 x 4096); 256 x 256, 32 on one block per eight rows
// 35 us, 128 on eight 34.
constexpr int kPassCParts = 8;
template <int X>
struct PassC {
    static constexpr int H = X / 2;
    using PL = tmfft::Plan<H, 8>;
    static constexpr int P = H / 8;                 // threads per row
    static constexpr int G = P / 8;                 // lanes per group
    static constexpr int S = P + P / 8;             // pairs of a group's part of the exchange buffer (one spare per 8)
    static constexpr int ROWS = P >= 128 ? 1 : 128 / P;
    static constexpr int NT = P * ROWS;             // 128 threads (256 at X = 4096)
    static constexpr int EXL = 8 * S;               // exchange buffer of a row
    // Widths whose sums take every value by itself: plain FP32 sums over 8 orientations have 2.7 times the
    // error of sums compensated at each (128 orientations of unit noise: 6.2e-7 against 2.3e-7,
    // emulated), FP64 has none to speak of.  The conversions share their unit with those of the histogram: 512
    // orientations at 1024 x 1024 0.81 ms with plain sums, 0.87 so (0.97 with two-term FP32 sums of
    // each value); 512 x 512 0.287 and 0.278; 256 x 256 0.143 both
    static constexpr bool EXACT = X < 2048;
    // 512 threads per SM at 128 registers: every block has its 128 TMEM columns per warp
    static constexpr int MIN_BLOCKS = 512 / NT;
    static constexpr int WCOLS = 128;
    static constexpr uint32_t TMEM_COLS = WCOLS * ((NT / 32 + 3) / 4);   // warps of a lane quadrant side by side
    static_assert(PL::radix(0) == 8 && PL::radix(1) == 8 && (PL::stages == 3 || PL::stages == 4) && G <= 32, "pass C widths");
    // blocks that share a group of rows of an image of height Y: as many as are resident together
    static int parts(int Y, int resident) {
        int n = 1;
        while (n < kPassCParts && Y / ROWS * 2 * n <= resident) n *= 2;
        return n;
    }
    // dynamic shared memory for a row pitch XP and `bins` histogram bins (one word for values outside)
    static size_t smem_bytes(int XP, int bins) {
        return 128 + sizeof(float2) * (size_t)ROWS * 2 * c_row_len(XP) + sizeof(float4) * 2 * (size_t)ROWS * EXL + 4 * ((size_t)bins + 1);
    }
    // blocks resident per SM (228 KB, 1 KB of it the system's per block): MIN_BLOCKS up to about 860 bins,
    // one fewer above to 2048 pixels, where a grid of MIN_BLOCKS leaves the last blocks to a second wave
    // (with 1024 bins: 2048 x 2916, 128 orientations 1.35 ms, 1.18 so; 512 x 512, 512 orientations 0.377 in
    // four parts, 0.369 in the two that are resident)
    static int resident(int XP, int bins) {
        const int n = (int)(233472 / (smem_bytes(XP, bins) + 1024));
        return n < MIN_BLOCKS ? n : MIN_BLOCKS;
    }
};

// the larger of three values; a NaN never wins
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// a double in two TMEM columns
__device__ __forceinline__ double f64_of(float lo, float hi) { return __hiloint2double(__float_as_int(hi), __float_as_int(lo)); }
__device__ __forceinline__ void f64_to(double d, float& lo, float& hi) {
    lo = __int_as_float(__double2loint(d));
    hi = __int_as_float(__double2hiint(d));
}

// Twiddle multipliers of stage s of the row pass's transform in lane l of group j, in 16 TMEM
// columns: butterfly u's powers w^1 .. w^(RS-1) at float pairs u (RS - 1) + r - 1.  At
// widths from 2048 each power is a table entry, below the product tree of
// tmfft::apply_twiddles.
template <int X>
struct PassCTw {
    using PC = PassC<X>;
    using PL = typename PC::PL;
    template <int s>
    __device__ static void fill(uint32_t col, int l, int j, const tmfft::Twiddles& tw) {
        constexpr int RS = PL::radix(s), Ns = PL::ns(s), H = PC::H;
        float g[16];
#pragma unroll
        for (int i = 0; i < 16; i++) g[i] = 0.f;
#pragma unroll
        for (int u = 0; u < 8 / RS; u++) {
            const int jm = (8 * (l + PC::G * u) + j) % Ns;
            float2 p[8];
            if constexpr (X >= 2048) {
#pragma unroll
                for (int r = 1; r < RS; r++) p[r] = tw.template w<+1>(jm * (H / (Ns * RS)) * r, H);
            } else {
                p[1] = tw.template w<+1>(jm * (H / (Ns * RS)), H);
                if constexpr (RS > 2) { p[2] = cmul(p[1], p[1]); p[3] = cmul(p[2], p[1]); }
                if constexpr (RS > 4) {
                    p[4] = cmul(p[2], p[2]);
                    p[5] = cmul(p[4], p[1]);
                    p[6] = cmul(p[4], p[2]);
                    p[7] = cmul(p[4], p[3]);
                }
            }
#pragma unroll
            for (int r = 1; r < RS; r++) {
                g[2 * (u * (RS - 1) + r - 1)] = p[r].x;
                g[2 * (u * (RS - 1) + r - 1) + 1] = p[r].y;
            }
        }
        tmptx::tmem_st16(col, g);
    }
    // the stage's butterflies on v (tb: its multipliers, loaded before)
    template <int s>
    __device__ static __forceinline__ void stage(tmfft::Pair (&v)[8], float (&tb)[16]) {
        constexpr int RS = PL::radix(s), NU = 8 / RS;
        tmptx::tmem_wait_ld16(tb);
#pragma unroll
        for (int u = 0; u < NU; u++) {
            tmfft::Pair e[RS];
            e[0] = v[u];
#pragma unroll
            for (int r = 1; r < RS; r++) {
                const int i = u * (RS - 1) + r - 1;
                e[r] = tmfft::pmul(v[u + r * NU], make_float2(tb[2 * i], tb[2 * i + 1]));
            }
            tmfft::pdft<RS, +1>(e);
#pragma unroll
            for (int r = 0; r < RS; r++) v[u + r * NU] = e[r];
        }
    }
};

// DIVIDED: the `parts` blocks of a cluster share a group of rows (a group per cluster).
template <int X, bool DIVIDED = false>
__global__ void __launch_bounds__(PassC<X>::NT, PassC<X>::MIN_BLOCKS)
k_pass_c(BatchArgs a, const __grid_constant__ CUtensorMap cmap, int Y, int parts) {
    using PC = PassC<X>;
    using PL = typename PC::PL;
    using TW = PassCTw<X>;
    constexpr int P = PC::P, G = PC::G, S = PC::S, NT = PC::NT, ROWS = PC::ROWS, EXL = PC::EXL;
    constexpr uint32_t kWaitLimit = 1u << 24;
    const int LR = c_row_len(a.XP);   // float2 of a row in shared memory
    // dynamic shared memory: mbarrier, TMEM slot | row pair | exchange 0 | exchange 1 | histogram
    extern __shared__ __align__(128) unsigned char smem_c[];
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_c);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_c + 64);
    float2* const rows = reinterpret_cast<float2*>(smem_c + 128);
    float4* const exch = reinterpret_cast<float4*>(rows + ROWS * 2 * LR);
    unsigned int* const shist = reinterpret_cast<unsigned int*>(exch + 2 * ROWS * EXL);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int t = tid % P, rl = tid / P;
    const int l = t % G, j = t / G;   // lane and group of the stages after the first
    const int nblocks = Y / ROWS;
    // this block's rows and pairs of orientations
    int part = 0, rb0 = blockIdx.x, i0 = 0, npairs = (a.nb + 1) >> 1;   // pairs i0 .. npairs - 1
    if constexpr (DIVIDED) {
        part = (int)blockIdx.x % parts;
        rb0 = (int)blockIdx.x / parts;
        i0 = part * npairs / parts;
        npairs = (part + 1) * npairs / parts;
    }
    auto best = [&]() -> int* {
        if constexpr (DIVIDED) return part == 0 ? a.best : a.best_parts + (size_t)(part - 1) * Y * X;
        else return a.best;
    };
    if (tid == 0) tmptx::mbar_init(mbar, 1);
    if (warp == 0) {
        tmptx::tmem_alloc(tmem_slot, PC::TMEM_COLS);
        tmptx::tmem_relinquish();
    }
    for (int b = tid; b <= a.hist_bins; b += NT) shist[b] = 0u;
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    // this thread's TMEM columns (lane quadrant warp % 4)
    const uint32_t tcomp = *tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(PC::WCOLS * (warp >> 2));
    // rows rb ROWS .. of orientations 2 i and 2 i + 1 (the last of an odd batch twice), each
    // as its column groups' pieces of the tiles (groups beyond the pitch arrive as zeros)
    // (called by warp 0: a lane issues one box)
    const int tile_rows = c_tile_rows(Y), boxes = c_row_boxes(a.XP), box = c_row_box(a.XP);
    auto issue_pair = [&](int rb, int i) {
        if (tid == 0) tmptx::mbar_arrive_expect_tx(mbar, (uint32_t)(2 * ROWS * LR) * (uint32_t)sizeof(float2));
        __syncwarp();
        for (int e = tid; e < 2 * ROWS * boxes; e += 32) {
            const int k = e / (2 * ROWS), hr = e % (2 * ROWS);   // box; orientation and row
            const int o = 2 * i + hr / ROWS, y = rb * ROWS + hr % ROWS;
            tmptx::tensor5_g2s(rows + hr * LR + 4 * k * box, &cmap, 0, y % tile_rows, k * box, y / tile_rows,
                               o < a.nb ? o : 2 * i, mbar);
        }
    };
    if (warp == 0 && npairs > i0 && rb0 < nblocks) issue_pair(rb0, i0);
    {
        // the packing's multipliers W_X^k, k = t + P r (columns 64-79), and those of stages 1, 2, 3
        float z[16];
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const float2 w = a.tw.template w<+1>(t + P * r, X);
            z[2 * r] = w.x;
            z[2 * r + 1] = w.y;
        }
        tmptx::tmem_st16(tcomp + 64, z);
        TW::template fill<1>(tcomp + 80, l, j, a.tw);
        TW::template fill<2>(tcomp + 96, l, j, a.tw);
        if constexpr (PL::stages == 4) TW::template fill<3>(tcomp + 112, l, j, a.tw);
        tmptx::tmem_wait_st();
    }
    // value v[r] holds the pixels own + 2 P r (real parts) and the next (imaginary parts)
    const int own = rl * X + 16 * l + 2 * j;
    // histogram bin int((v - min) / step) as one multiply-add: (v - min) / step = v / step + hoff
    const float hoff = -a.hist_min * a.hist_inv_step;
    const float2 hinv2 = make_float2(a.hist_inv_step, a.hist_inv_step), hoff2 = make_float2(hoff, hoff);
    const unsigned int nbins = (unsigned int)a.hist_bins;
    bool timed_out = false, stop = false;
    uint32_t n = 0;   // pairs done: parity of the barrier's phase and of the exchange buffer
    for (int rb = rb0; rb < nblocks && !stop; rb += gridDim.x) {   // (DIVIDED: leaves after the first)
    const size_t pix0 = (size_t)rb * ROWS * X;
    float mip[16];
    float fs[PC::EXACT ? 1 : 16], pq[PC::EXACT ? 1 : 16];   // plain sums over at most 8 orientations
#pragma unroll
    for (int r = 0; r < 16; r++) mip[r] = a.mip[pix0 + own + 2 * P * (r / 2) + r % 2];
#pragma unroll
    for (int r = 0; r < (PC::EXACT ? 1 : 16); r++) fs[r] = pq[r] = 0.f;
    {
        float z[16];
#pragma unroll
        for (int i = 0; i < 16; i++) z[i] = 0.f;
        tmptx::tmem_st16(tcomp, z);
        tmptx::tmem_st16(tcomp + 16, z);
        tmptx::tmem_st16(tcomp + 32, z);
        tmptx::tmem_st16(tcomp + 48, z);
        tmptx::tmem_wait_st();
    }
    for (int i = i0; i < npairs; i++, n++) {
        float4* const ex = exch + (n & 1) * (ROWS * EXL) + rl * EXL;
        float tb[16];
        tmptx::tmem_ld16(tcomp + 64, tb);
        if (!tmptx::mbar_wait_bounded(mbar, n & 1, kWaitLimit)) {
            timed_out = true;
            atomicExch(a.err, 1);
        }
        tmfft::Pair v[8];
        tmptx::tmem_wait_ld16(tb);
        {
            const float2* c = rows + rl * LR + t;
            const float2* d = rows + rl * LR + (P - t);
#pragma unroll
            for (int r = 0; r < 8; r++) {   // k = t + P r and H - k
                const float2 w = make_float2(tb[2 * r], tb[2 * r + 1]);
                float2 z[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float2 hk = c[h * ROWS * LR + P * r], hm = d[h * ROWS * LR + P * (7 - r)];
                    if (r == 0 && t == 0) hk.y = hm.y = 0.f;   // as FFTW's c2r
                    const float2 e = make_float2(hk.x + hm.x, hk.y - hm.y);
                    const float2 df = make_float2(hk.x - hm.x, hk.y + hm.y);
                    const float2 od = cmul(df, w);
                    z[h] = make_float2(e.x - od.y, e.y + od.x);
                }
                v[r] = {make_float2(z[0].x, z[1].x), make_float2(z[0].y, z[1].y)};
            }
        }
        auto put = [](float4* at, tmfft::Pair p) { *at = make_float4(p.re.x, p.re.y, p.im.x, p.im.y); };
        auto get = [](const float4* at) {
            const float4 f = *at;
            return tmfft::Pair{make_float2(f.x, f.y), make_float2(f.z, f.w)};
        };
        tmfft::pdft<8, +1>(v);
#pragma unroll
        for (int r = 0; r < 8; r++) put(ex + S * r + t, v[r]);
        tmptx::tmem_ld16(tcomp + 80, tb);
        if (__syncthreads_or(timed_out)) {   // every thread learns whether a wait ran out
            stop = true;
            break;
        }
        // every thread has read its row values: the next pair's rows may arrive
        if (warp == 0) {
            if (i + 1 < npairs) issue_pair(rb, i + 1);
            else if (!DIVIDED && rb + (int)gridDim.x < nblocks) issue_pair(rb + gridDim.x, 0);
        }
        float4* const eg = ex + S * j;
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = get(eg + l + G * r);
        TW::template stage<1>(v, tb);
        tmptx::tmem_ld16(tcomp + 96, tb);
        auto pad = [](int e) { return e + (e >> 3); };
        __syncwarp();   // the group's values are read
#pragma unroll
        for (int r = 0; r < 8; r++) put(eg + 9 * l + r, v[r]);   // pad(8 l + r)
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = get(eg + pad(l + G * r));
        TW::template stage<2>(v, tb);
        if constexpr (PL::stages == 4) {
            tmptx::tmem_ld16(tcomp + 112, tb);
            __syncwarp();
            const int at = 72 * (l >> 3) + (l & 7);
#pragma unroll
            for (int r = 0; r < 8; r++) put(eg + at + 9 * r, v[r]);   // pad(64 (l / 8) + l % 8 + 8 r)
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] = get(eg + pad(l + G * r));
            TW::template stage<3>(v, tb);
        }
        // values of orientations 2 i and 2 i + 1 at the thread's pixel r
        auto val = [&](int r) { return r % 2 ? v[r / 2].im : v[r / 2].re; };
        const int g = (int)a.gidx0 + 2 * i;
        const bool two = 2 * i + 1 < a.nb;   // else the second repeats the first
#pragma unroll
        for (int r0 = 0; r0 < 16; r0 += 4) {
            // strict >, first orientation first: the new maximum is v.x, else v.y, else the old one
            float m[4];
            bool changed = false;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                m[k] = fmax3(mip[r0 + k], val(r0 + k).x, val(r0 + k).y);
                changed = changed || m[k] > mip[r0 + k];
            }
            if (changed) {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (m[k] > mip[r0 + k]) best()[pix0 + own + 2 * P * ((r0 + k) / 2) + k % 2] = val(r0 + k).x == m[k] ? g : g + 1;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) mip[r0 + k] = m[k];
        }
        auto count = [&](float b) {
            const unsigned int bin = (unsigned int)__float2int_rz(b);
            atomicAdd(&shist[bin < nbins ? bin : nbins], 1u);
        };
        // the sums and the histogram, compiled for a pair and for the single last one of an odd batch (a branch at
        // each pixel cost the EXACT form 4 %)
        auto add = [&](auto pair) {
            constexpr bool both = decltype(pair)::value;
            auto bins = [&](int r) {
                const float2 p = val(r);
                if constexpr (both) {
                    const float2 b = tmfft::fma2(p, hinv2, hoff2);
                    count(b.x);
                    count(b.y);
                } else {
                    count(fmaf(p.x, a.hist_inv_step, hoff));
                }
            };
            if constexpr (PC::EXACT) {
                // FP64 sums of pixel r in columns 2 r (sum) and 32 + 2 r (sum of squares), 4 pixels at a
                // time, whose bins are counted while the sums arrive
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    float sm[8], sq[8];
                    tmptx::tmem_ld8(tcomp + 8 * h, sm);
                    tmptx::tmem_ld8(tcomp + 32 + 8 * h, sq);
#pragma unroll
                    for (int k = 0; k < 4; k++) bins(4 * h + k);
                    tmptx::tmem_wait_ld8x2(sm, sq);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 p = val(4 * h + k);
                        double ds = f64_of(sm[2 * k], sm[2 * k + 1]), dq = f64_of(sq[2 * k], sq[2 * k + 1]);
                        const double x = p.x;
                        ds += x;
                        dq = fma(x, x, dq);
                        if constexpr (both) {
                            const double y = p.y;
                            ds += y;
                            dq = fma(y, y, dq);
                        }
                        f64_to(ds, sm[2 * k], sm[2 * k + 1]);
                        f64_to(dq, sq[2 * k], sq[2 * k + 1]);
                    }
                    tmptx::tmem_st8(tcomp + 8 * h, sm);
                    tmptx::tmem_st8(tcomp + 32 + 8 * h, sq);
                }
                tmptx::tmem_wait_st();
            } else {
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    const float2 p = val(r);
                    fs[r] += p.x;
                    pq[r] = fmaf(p.x, p.x, pq[r]);
                    if constexpr (both) {
                        fs[r] += p.y;
                        pq[r] = fmaf(p.y, p.y, pq[r]);
                    }
                    bins(r);
                }
            }
        };
        if (two) add(std::true_type{});
        else add(std::false_type{});
        if (!PC::EXACT && (((i - i0) & 3) == 3 || i == npairs - 1)) {
            // Kahan: the compensation holds what the last addition added beyond its input
#pragma unroll
            for (int sweep = 0; sweep < 4; sweep++) {   // 8 pixels of one sum at a time
                float* part = ((sweep >> 1) ? pq : fs) + 8 * (sweep & 1);
                const uint32_t col = tcomp + 32 * (sweep >> 1) + 8 * (sweep & 1);
                float sm[8], cm[8];   // sum, compensation
                tmptx::tmem_ld8(col, sm);
                tmptx::tmem_ld8(col + 16, cm);
                tmptx::tmem_wait_ld8x2(sm, cm);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const float yv = part[k] - cm[k];
                    const float tv = sm[k] + yv;
                    cm[k] = (tv - sm[k]) - yv;
                    sm[k] = tv;
                    part[k] = 0.f;
                }
                tmptx::tmem_st8(col, sm);
                tmptx::tmem_st8(col + 16, cm);
            }
            tmptx::tmem_wait_st();
        }
    }
    if (!DIVIDED && stop) break;
    // the batch's sums into the FP64 running sums, and the maxima, in pixel order through the
    // exchange buffers (one spare element per 16: the strided writes are conflict-free), so that
    // memory is accessed in whole lines with all of a thread's loads in flight
    double* const staged = reinterpret_cast<double*>(exch);
    auto pad = [](int e) { return e + (e >> 4); };
    const int at = pad(own);
    auto px = [pad](int r) { return pad(2 * P * (r / 2)) + r % 2; };
    constexpr int PER = ROWS * X / NT;   // 16
    __syncthreads();   // every group is done with its transposes
    {
        float send[32];
        tmptx::tmem_ld16(tcomp, send);
        tmptx::tmem_ld16(tcomp + 16, send + 16);
        tmptx::tmem_wait_ld32(send);
        auto sum = [&](int r) { return PC::EXACT ? f64_of(send[2 * r], send[2 * r + 1]) : (double)send[r] - (double)send[16 + r]; };
#pragma unroll
        for (int r = 0; r < 16; r++) staged[at + px(r)] = sum(r);
        tmptx::tmem_ld16(tcomp + 32, send);
        tmptx::tmem_ld16(tcomp + 48, send + 16);
        tmptx::tmem_wait_ld32(send);
#pragma unroll
        for (int r = 0; r < 16; r++) staged[2 * ROWS * EXL + at + px(r)] = sum(r);
    }
    if constexpr (DIVIDED) {
        // (the maxima in the row buffer, whose last copies have been waited for; after a timeout
        // they are no results, but the cluster's barriers are passed all the same)
        float* const maxima = reinterpret_cast<float*>(rows);
        if (stop) tmptx::mbar_wait_bounded(mbar, n & 1, kWaitLimit);
#pragma unroll
        for (int r = 0; r < 16; r++) maxima[at + px(r)] = mip[r];
        tmptx::cluster_sync();
        // this block's share of the pixels: PER / parts per thread
        for (int e = part * PER / parts; e < (part + 1) * PER / parts; e++) {
            const size_t pix = pix0 + tid + e * NT;
            const int x = pad(tid + e * NT);
            double s = a.sum[pix], q = a.sumsq[pix];
            float m = 0.f;
            int won = 0;
            for (int p = 0; p < parts; p++) {
                s += tmptx::cluster_ld_f64(tmptx::cluster_addr(staged + x, p));
                q += tmptx::cluster_ld_f64(tmptx::cluster_addr(staged + 2 * ROWS * EXL + x, p));
                const float mp = tmptx::cluster_ld_f32(tmptx::cluster_addr(maxima + x, p));
                if (p > 0 && mp > m) won = p;
                m = p > 0 ? fmaxf(m, mp) : mp;
            }
            a.sum[pix] = s;
            a.sumsq[pix] = q;
            a.mip[pix] = m;
            if (won) a.best[pix] = __ldcg(a.best_parts + (size_t)(won - 1) * Y * X + pix);
        }
        tmptx::cluster_sync();   // the other blocks have read this one's shared memory
        break;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        double* const dst = (k ? a.sumsq : a.sum) + pix0 + tid;
        double d[PER];
#pragma unroll
        for (int e = 0; e < PER; e++) d[e] = dst[e * NT];
#pragma unroll
        for (int e = 0; e < PER; e++) dst[e * NT] = d[e] + staged[k * 2 * ROWS * EXL + pad(tid + e * NT)];
    }
    __syncthreads();
    float* const stage = reinterpret_cast<float*>(exch);
#pragma unroll
    for (int r = 0; r < 16; r++) stage[at + px(r)] = mip[r];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < PER; e++) a.mip[pix0 + tid + e * NT] = stage[pad(tid + e * NT)];
    __syncthreads();   // the exchange buffers are free again
    }
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    // every warp has finished with its TMEM columns (the barrier above)
    tmptx::tmem_fence_after_sync();
    if (warp == 0) tmptx::tmem_dealloc(*tmem_slot, PC::TMEM_COLS);
    if (stop) {
        // results of these rows are discarded (the host reports the timeout).  The wait for this
        // pair ran out and none was issued after it: wait (bounded again) for its copies
        tmptx::mbar_wait_bounded(mbar, n & 1, kWaitLimit);
        return;
    }
    for (int b = tid; b < a.hist_bins; b += NT) {
        const unsigned int cnt = shist[b];
        if (cnt) atomicAdd(a.hist + b, (unsigned long long)cnt);
    }
}

// --------------------------------------------------------------------------------------
// Prepared micrograph spectrum I'[ky][kx] = I[ky][kx] * exp(+2 pi i (kx*x0/X + ky*y0/Y)) / N
// with the projection placed at (x0, y0) = (X/2 - T/2, Y/2 - T/2), I'[0][0] = 0, and zero
// pitch padding (kx > X/2).  spec: Y*(X/2+1) complex; phases in double.
__global__ void k_prepare_image(const float2* __restrict__ spec, float2* __restrict__ ip, int X, int Y, int XP, int T) {
    const int kx = blockIdx.x * blockDim.x + threadIdx.x;
    const int ky = blockIdx.y;
    if (kx >= XP) return;
    const int hc = X / 2 + 1;
    float2 out = make_float2(0.f, 0.f);
    if (kx < hc && !(kx == 0 && ky == 0)) {
        const long long x0 = X / 2 - T / 2, y0 = Y / 2 - T / 2;
        double sx, cx, sy, cy;
        sincospi(2.0 * (double)((kx * x0) % X) / (double)X, &sx, &cx);
        sincospi(2.0 * (double)((ky * y0) % Y) / (double)Y, &sy, &cy);
        const double pr = cx * cy - sx * sy, pi = cx * sy + sx * cy;
        const float2 v = spec[(size_t)ky * hc + kx];
        const double invn = 1.0 / ((double)X * (double)Y);
        out = make_float2((float)(((double)v.x * pr - (double)v.y * pi) * invn),
                          (float)(((double)v.x * pi + (double)v.y * pr) * invn));
    }
    ip[(size_t)ky * XP + kx] = out;
}

// --------------------------------------------------------------------------------------
__global__ void k_reset_state(float* mip, int* best, double* sum, double* sumsq, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        mip[i] = -FLT_MAX;
        best[i] = -1;
        sum[i] = 0.0;
        sumsq[i] = 0.0;
    }
}

// --------------------------------------------------------------------------------------
// The tensor maps of a correlation buffer C of `cap` orientations.
//   rows      as the row pass reads it: dimensions (8 floats of a column group's row, row of the
//             tile, column group, tile row, orientation), boxes of one row x c_row_box(XP)
//             groups.  L2 promotion to 64 bytes: 0.39 ms for a load-only pass over 2.15 GB
//             against 0.45 without and with 128 or 256 bytes.
//   columns   as k_pass_b_rg writes it: dimensions (a tile, column group, tile row), boxes of
//             256 tiles of one column group
struct CMaps {
    CUtensorMap rows, columns;
};
inline cudaError_t c_tensor_maps(CMaps* maps, float2* C, int XP, int Y, int cap) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
    if (e != cudaSuccess) return e;
    if (found != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    const auto encode = reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn);
    const int R = c_tile_rows(Y);
    const cuuint32_t step[5] = {1, 1, 1, 1, 1};
    {
        const cuuint64_t dim[5] = {8, (cuuint64_t)R, (cuuint64_t)(XP / 4), (cuuint64_t)(Y / R), (cuuint64_t)cap};
        const cuuint64_t stride[4] = {32, 32 * (cuuint64_t)R, (cuuint64_t)XP * 8 * R, (cuuint64_t)XP * 8 * Y};
        const cuuint32_t box[5] = {8, 1, (cuuint32_t)c_row_box(XP), 1, 1};
        const CUresult r = encode(&maps->rows, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, C, dim, stride, box, step,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    const cuuint64_t dim[3] = {8 * (cuuint64_t)R, (cuuint64_t)(XP / 4), (cuuint64_t)cap * (Y / R)};
    const cuuint64_t stride[2] = {32 * (cuuint64_t)R, (cuuint64_t)XP * 8 * R};
    const cuuint32_t box[3] = {8 * (cuuint32_t)R, 1, dim[2] < 256 ? (cuuint32_t)dim[2] : 256};
    const CUresult r = encode(&maps->columns, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, C, dim, stride, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// several resident blocks need the largest shared-memory carveout
template <class K>
cudaError_t configure_cols(K kernel, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}

// --------------------------------------------------------------------------------------
// Launch shapes of one geometry, shared by every entry point.
template <int T, int X, int Y>
struct Launch {
    using PB = PassB<T, Y>;
    using PC = PassC<X>;
    static_assert(Y % PC::ROWS == 0, "pass C blocks hold whole groups of rows");
    using SC = SliceCol<T>;
    using RC = RowC2R<T>;
    static constexpr int pass_b_width = PB::W;   // row pitch alignment (columns)
    // 4096-high micrographs with 256-row pruned transforms: the residue-grouped column pass
    static constexpr bool RG = (T == 256 && Y == 4096);
    // images whose row pass divides its batches (PassC::parts)
    static constexpr bool DIVIDES = 2 * (Y / PC::ROWS) <= PC::MIN_BLOCKS * 160;
    static int pass_c_parts(int nsm) { return DIVIDES ? PC::parts(Y, PC::MIN_BLOCKS * nsm) : 1; }   // most
    static cudaError_t configure_b() {
        cudaError_t e = configure_cols(k_pass_b<T, Y>, PB::SMEM);
        if (RG && e == cudaSuccess)
            e = cudaFuncSetAttribute(k_pass_b_rg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PassBRg::SMEM);
        return e;
    }
    static cudaError_t configure(int XP, int bins) {
        const cudaError_t e = configure_b();
        if (e != cudaSuccess) return e;
        const int smem = (int)PC::smem_bytes(XP, bins);
        if constexpr (DIVIDES) {
            const cudaError_t d = cudaFuncSetAttribute(k_pass_c<X, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (d != cudaSuccess) return d;
        }
        return cudaFuncSetAttribute(k_pass_c<X>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    }
    // slice, projection, normalisation and row transforms
    static void prep(BatchArgs& a, cudaStream_t s) {
        k_slice_colfft<T><<<dim3((T / 2 + 1 + SC::CB - 1) / SC::CB, a.nb), SC::NT, 0, s>>>(a);
        k_row_c2r<T><<<dim3(T / RC::ROWS, a.nb), RC::NT, 0, s>>>(a);
        k_norm<T><<<(a.nb + 7) / 8, 256, 0, s>>>(a, a.norm_pixels > 0 ? a.norm_pixels : (long long)X * Y);
        k_pass_a<T, X><<<dim3(T, a.nb), X / 16, 0, s>>>(a);
    }
    static void pass_b(BatchArgs& a, const CMaps& cmaps, cudaStream_t s, int nsm) {
        const int ngroups = a.XP / (RG ? 4 : PB::W);
        if (RG && ColSchedule::max_items(ngroups, a.nb, nsm) <= PassBRg::MAX_ITEMS)
            k_pass_b_rg<<<nsm, PassBRg::NT, PassBRg::SMEM, s>>>(a, cmaps.columns, ngroups);
        else
            k_pass_b<T, Y><<<PB::BPS * nsm, PB::NT, PB::SMEM, s>>>(a, ngroups);
    }
    static void pass_c(BatchArgs& a, const CMaps& cmaps, cudaStream_t s, int nsm) {
        const int nblocks = Y / PC::ROWS, resident = PC::resident(a.XP, a.hist_bins) * nsm;
        const size_t smem = PC::smem_bytes(a.XP, a.hist_bins);
        if constexpr (DIVIDES) {
            // at least two pairs of orientations for each part
            int parts = a.best_parts ? PC::parts(Y, resident) : 1;
            while (parts > 1 && a.nb < 4 * parts) parts /= 2;
            if (parts > 1) {
                cudaLaunchAttribute cluster;
                cluster.id = cudaLaunchAttributeClusterDimension;
                cluster.val.clusterDim.x = parts;
                cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3(nblocks * parts);
                cfg.blockDim = dim3(PC::NT);
                cfg.dynamicSmemBytes = smem;
                cfg.stream = s;
                cfg.attrs = &cluster;
                cfg.numAttrs = 1;
                cudaLaunchKernelEx(&cfg, k_pass_c<X, true>, a, cmaps.rows, Y, parts);
                return;
            }
        }
        k_pass_c<X><<<nblocks < resident ? nblocks : resident, PC::NT, smem, s>>>(a, cmaps.rows, Y, 1);
    }
};

}  // namespace tmk

#include "tm_tensor.cuh"

namespace tmk {

// Launch shapes of the FP16 tensor-core form of one geometry (row lengths X of
// 1024, 2048 or 4096): k_pass_b with FP16 output in blocks of R rows, and the
// tensor-core row pass.
template <int T, int X, int Y>
struct LaunchTc {
    using PB = PassB<T, Y>;
    using PCT = PassCTc<X>;
    static constexpr int R = PCT::R;
    // height 4096: the tensor-core column pass; other heights: the FP32 column FFTs with FP16 output
    static constexpr bool COL_TC = (Y == 4096);
    using PBT = PassBTc<T, R>;
    static constexpr size_t rows_tab_bytes = (size_t)PCT::B1_BYTES + PCT::B2_BYTES;
    static cudaError_t configure(int XP, int bins) {
        cudaError_t e;
        if constexpr (COL_TC) {
            e = cudaFuncSetAttribute(k_pass_b_tc<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, PBT::SMEM);
            // two CTAs of a pair per SM need the largest shared-memory carveout
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k_pass_b_tc<T, R>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
        } else
            e = configure_cols(k_pass_b<T, Y, R>, PB::SMEM);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(k_pass_c_tc<X>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PCT::smem_bytes(XP, bins));
    }
    static void pass_b(BatchArgs& a, cudaStream_t s, int nsm, const uint4* tabs) {
        if constexpr (COL_TC) {
            // items = (group of 4 columns, orientation); two blocks per SM
            k_pass_b_tc<T, R><<<2 * nsm, PBT::NT, PBT::SMEM, s>>>(a, a.XP / 4, tabs + rows_tab_bytes / 16);
        } else {
            k_pass_b<T, Y, R><<<PB::BPS * nsm, PB::NT, PB::SMEM, s>>>(a, a.XP / PB::W);
        }
    }
    static void pass_c(BatchArgs& a, cudaStream_t s, const uint4* dft) {
        k_pass_c_tc<X><<<Y / R, PCT::NT, PCT::smem_bytes(a.XP, a.hist_bins), s>>>(a, Y, dft);
    }
    // the row pass's DFT operands, then (height 4096) the column pass's
    static constexpr size_t dft_bytes = rows_tab_bytes + (COL_TC ? PBT::dft_bytes : 0);
    static void fill_dft(uint16_t* host) {
        fill_tc_dft<X>(host);
        if constexpr (COL_TC) fill_tc_cols<T, R>(host + rows_tab_bytes / 2);
    }
};

}  // namespace tmk
