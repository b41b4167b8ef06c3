// tm_proposal.cu -- the learned proposal network of the search (C ABI in
// include/tm_b200.h): a 5-layer CNN that reads tiles of the coarse search's
// maps and scores them for the fine search.  The reference has no counterpart;
// its outputs are checked against the FP64 restatement oracle/proposal.py.
//
//   layer 1  conv 3x3, cin -> 32, ReLU, max-pool 2     (tile      -> tile/2)
//   layer 2  conv 3x3, 32 -> 64, ReLU, max-pool 2      (tile/2    -> tile/4)
//   layer 3  conv 3x3, 64 -> 128, ReLU, max-pool 2     (tile/4    -> tile/8)
//   layer 4  conv 3x3, 128 -> 128, ReLU, global max    (tile/8    -> 128)
//   layer 5  fully connected 128 -> 4: objectness logit and a direction
//
// Weights are kept as FP32 master values (Adam state beside them) and used as
// BF16 copies by the forward and the backward-data kernels; activations,
// accumulation and weight gradients are FP32.  The weight gradient is taken
// with respect to the BF16 values the forward used.
//
// Loss of a batch of n tiles with labels (y, t) (y in {0,1}, t a unit vector):
//   L = 1/n sum_i [ w_i BCE(o_i, y_i) + lambda y_i (1 - cos(d_i, t_i)) ]
// with w_i = pos_weight for y_i = 1, else 1, o_i the objectness logit and d_i
// the direction output (only its direction matters: the angular bins are
// ranked by c_b . d).
//
// Every kernel is a bounded loop nest; nothing waits on another block.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>

#include <string>
#include <vector>

#include "../../include/tm_b200.h"
#include "tm_fft.cuh"

namespace tmp {

constexpr int kC1 = 32, kC2 = 64, kC3 = 128, kC4 = 128, kOut = 4;
constexpr int kThreads = 256;

using tmfft::fma2;

// ----------------------------------------------------------------------------------------------
// 3x3 convolution, zero padding 1, NCHW.  out[n][o][y][x] = b[o] + sum_i sum_k
// in[n][i][y+ky-1][x+kx-1] * W(o, i, ky, kx), optionally ReLU.  With FLIP the
// kernel is the backward-data pass of a forward conv whose weights are
// Wf[co][ci][3][3]: W(o, i, ky, kx) = Wf[i][o][2-ky][2-kx] (o runs over the
// forward conv's input channels, i over its output channels), no bias, no ReLU.
// Every output is one chain of multiply-adds over i, then ky, then kx.
//
// Block: a TW x TW tile of output pixels of NI images times COB output channels; a thread computes
// PXT pixels of a row x 8 channels, channels in pairs (two multiply-adds per
// instruction, a pair's weights being adjacent in shared memory): with 4 pixels 48 such instructions per
// input channel and kernel row for 8 shared-memory loads.  (One pixel x 8 channels with
// 9 loads per 8 multiply-adds: the shared-memory pipe bound it at a sixth of the FP32 rate, 200-417
// us for the layers of 128 tiles of 64 x 64; 85-168 now.)  Input channels go through
// shared memory CIB at a time with their halo.
template <int TW_, int PXT_, int CG_, int NI_>
struct ConvTile {
    static constexpr int TW = TW_, PXT = PXT_, CG = CG_, NI = NI_;
    static constexpr int CIB = 8, COT = 8;
    static constexpr int PG = TW * TW / PXT;                            // pixel groups of an image
    static constexpr int COB = CG * COT, NT = NI * PG * CG;
    static constexpr int PITCH = (TW + 2 + 3) / 4 * 4;                  // row pitch of the input tile, 16-byte aligned
};

template <bool FLIP, class CT>
__global__ void __launch_bounds__(CT::NT)
k_conv3x3(const float* __restrict__ in, const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
          float* __restrict__ out, int N, int Ci, int Co, int H, int relu) {
    constexpr int TW = CT::TW, CIB = CT::CIB, PXT = CT::PXT, COB = CT::COB, NT = CT::NT, NI = CT::NI, PITCH = CT::PITCH, E = TW + 2;
    __shared__ __align__(16) float s_in[NI][CIB][E][PITCH];
    __shared__ __align__(16) float s_w[CIB][9][COB];
    const int tiles_x = H / TW;
    const int ty0 = (blockIdx.x / tiles_x) * TW, tx0 = (blockIdx.x % tiles_x) * TW;
    const int co0 = blockIdx.y * COB;
    const int t = threadIdx.x;
    const int pg = t % CT::PG, im = t / CT::PG % NI, cg = t / (CT::PG * NI);
    const int n0 = blockIdx.z * NI, n = n0 + im;
    const int py = pg / (TW / PXT), px = pg % (TW / PXT) * PXT;
    float2 acc[PXT][4];
#pragma unroll
    for (int p = 0; p < PXT; p++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[p][j] = make_float2(0.f, 0.f);
    for (int ci0 = 0; ci0 < Ci; ci0 += CIB) {
        // input tiles with halo
        for (int e = t; e < NI * CIB * E * E; e += NT) {
            const int c = e / (E * E), r = e % (E * E);   // image and channel
            const int yy = ty0 + r / E - 1, xx = tx0 + r % E - 1;
            const int nn = n0 + c / CIB, ci = ci0 + c % CIB;
            float v = 0.0f;
            if ((NI == 1 || nn < N) && ci < Ci && yy >= 0 && yy < H && xx >= 0 && xx < H) v = in[(((size_t)nn * Ci + ci) * H + yy) * H + xx];
            s_in[c / CIB][c % CIB][r / E][r % E] = v;
        }
        // weights of COB output channels x CIB input channels, channel fastest
        for (int e = t; e < COB * CIB * 9; e += NT) {
            const int o = e / (CIB * 9), r = e % (CIB * 9);
            const int c = r / 9, k = r % 9;
            const int co = co0 + o, ci = ci0 + c;
            float v = 0.0f;
            if (co < Co && ci < Ci) {
                if (!FLIP) v = __bfloat162float(w[((size_t)co * Ci + ci) * 9 + k]);
                else v = __bfloat162float(w[((size_t)ci * Co + co) * 9 + (8 - k)]);
            }
            s_w[c][k][o] = v;
        }
        __syncthreads();
#pragma unroll 2
        for (int c = 0; c < CIB; c++) {
#pragma unroll
            for (int ky = 0; ky < 3; ky++) {
                const float* row = &s_in[im][c][py + ky][px];
                float v[PXT + 2];
                if constexpr (PXT == 4) {
                    const float4 a = *reinterpret_cast<const float4*>(row);
                    const float2 b = *reinterpret_cast<const float2*>(row + 4);
                    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y;
                } else {
#pragma unroll
                    for (int p = 0; p < PXT + 2; p++) v[p] = row[p];
                }
#pragma unroll
                for (int kx = 0; kx < 3; kx++) {
                    const float4* wp = reinterpret_cast<const float4*>(&s_w[c][ky * 3 + kx][cg * CT::COT]);
                    const float4 w0 = wp[0], w1 = wp[1];
                    const float2 wj[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y),
                                          make_float2(w1.z, w1.w)};
#pragma unroll
                    for (int p = 0; p < PXT; p++)
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[p][j] = fma2(make_float2(v[p + kx], v[p + kx]), wj[j], acc[p][j]);
                }
            }
        }
        __syncthreads();
    }
    if (NI > 1 && n >= N) return;
    const int y = ty0 + py, x = tx0 + px;
#pragma unroll
    for (int j = 0; j < CT::COT; j++) {
        const int co = co0 + cg * CT::COT + j;
        if (co >= Co) continue;
        const float b = bias ? bias[co] : 0.0f;
#pragma unroll
        for (int p = 0; p < PXT; p++) {
            float v = (j & 1 ? acc[p][j / 2].y : acc[p][j / 2].x) + b;
            if (relu) v = fmaxf(v, 0.0f);
            out[(((size_t)n * Co + co) * H + y) * H + x + p] = v;
        }
    }
}

// Weight and bias gradients of a 3x3 conv on W x W maps: dW[o][i][k] = sum_n sum_p g[n][o][p] *
// in[n][i][p + k - (1,1)], db[o] = sum_n sum_p g[n][o][p].  A block takes 32 output x 8 input
// channels and a share of the pixels, 256 at a time (a band of rows, or several whole maps)
// through shared memory; a thread holds the nine sums of 4 output channels x 1
// input channel over a quarter of them, output channels in pairs: 144 two-wide multiply-adds per 8
// pixels of a row for 38 loads.  The quarters are added in the block, the blocks with
// atomics in FP64 (dW and db are zeroed before the backward pass).  A thread adds 16 pixels in one
// chain and those sums in another: with one chain over all its pixels (256 of 8 x 8 maps, 448 of 16 x 16)
// and FP32 atomics the error was 1.2 times that of one block per channel pair, with these it is 0.6 to
// 0.7 of it (third layer, 128 tiles of 32 and 64), for 0.53 instead of 0.50 ms at 128 tiles of 64.  (One block per channel pair read
// every map from memory once per pair: 0.6-1.95 ms per layer of 128 tiles of 64 x 64; now
// 0.1-0.2 ms.)
template <int W>
struct WGrad {
    static constexpr int OB = 32, IB = 8, PX = 256;
    static constexpr int RB = W * W <= PX ? W : PX / W;        // rows of a map per step
    static constexpr int NI = PX / (RB * W);                   // maps per step
    static constexpr int SL = W < 8 ? W : 8;                   // pixels of a row per inner step
    static constexpr int GP = OB + 4;                          // pitch of a pixel's gradients
    static constexpr int E = W + 2;
    static constexpr int IN = NI * (RB + 2) * E * IB;
    static constexpr int SMEM = (PX * GP + IN) * 4;
    static_assert(PX * GP + IN >= 3 * 64 * 40, "the block reduction reuses the staging buffers");
};

template <int W>
__global__ void __launch_bounds__(kThreads)
k_conv3x3_wgrad(const float* __restrict__ in, const float* __restrict__ g, double* dW, double* db, int N, int Ci, int Co, int units) {
    using WG = WGrad<W>;
    constexpr int OB = WG::OB, IB = WG::IB, PX = WG::PX, RB = WG::RB, NI = WG::NI, SL = WG::SL, GP = WG::GP, E = WG::E;
    extern __shared__ __align__(16) float wsm[];
    float* const s_g = wsm;                 // [pixel][output channel]
    float* const s_in = wsm + PX * GP;      // [map][row][column][input channel], with the halo
    const int itiles = (Ci + IB - 1) / IB;
    const int o0 = blockIdx.x / itiles * OB, i0 = blockIdx.x % itiles * IB;
    const int t = threadIdx.x;
    const int i = t & 7, og = (t >> 3) & 7, pq = t >> 6;   // input channel, group of 4 output channels, quarter
    constexpr int bands = W / RB;
    const int total = (N + NI - 1) / NI * bands;   // steps
    float2 acc[2][10], part[2][10];   // totals and the sums of 16 pixels; tap 9: the bias
    auto zero = [](float2 (&a)[2][10]) {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int k = 0; k < 10; k++) a[h][k] = make_float2(0.f, 0.f);
    };
    zero(acc);
    zero(part);
    for (int u = blockIdx.y * units; u < min(total, (int)(blockIdx.y + 1) * units); u++) {
        const int n0 = u / bands * NI, y0 = u % bands * RB;
        bool unbounded = false;   // an input or a gradient that is infinite or not a number
        // gradients: 4 output channels of a pixel per thread and step
        for (int e = t; e < PX * (OB / 4); e += kThreads) {
            const int p = e % PX, o4 = e / PX * 4;
            const int n = n0 + p / (RB * W), r = p % (RB * W);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (n < N) {
                const float* gp = g + ((size_t)n * Co + o0 + o4) * (W * W) + y0 * W + r;
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = gp[(size_t)j * (W * W)];
#pragma unroll
                for (int j = 0; j < 4; j++) unbounded = unbounded || !(fabsf(v[j]) <= FLT_MAX);
            }
            *reinterpret_cast<float4*>(s_g + p * GP + o4) = make_float4(v[0], v[1], v[2], v[3]);
        }
        // inputs with the halo: 4 input channels of a pixel per thread and step
        for (int e = t; e < NI * (RB + 2) * E * (IB / 4); e += kThreads) {
            const int q = e % (NI * (RB + 2) * E), i4 = e / (NI * (RB + 2) * E) * 4;
            const int n = n0 + q / ((RB + 2) * E), r = q % ((RB + 2) * E);
            const int y = y0 + r / E - 1, x = r % E - 1;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (n < N && y >= 0 && y < W && x >= 0 && x < W) {
                const float* ip = in + ((size_t)n * Ci + i0 + i4) * (W * W) + y * W + x;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (i0 + i4 + j < Ci) v[j] = ip[(size_t)j * (W * W)];
#pragma unroll
                for (int j = 0; j < 4; j++) unbounded = unbounded || !(fabsf(v[j]) <= FLT_MAX);
            }
            *reinterpret_cast<float4*>(s_in + q * IB + i4) = make_float4(v[0], v[1], v[2], v[3]);
        }
        // such an input counts only where its gradient is not zero (the ReLU masks it elsewhere), such a
        // gradient only for the taps inside the map
        const bool masked = __syncthreads_or(unbounded);
        // this quarter's 64 pixels, SL of a row at a time
#pragma unroll 1
        for (int s0 = 64 * pq; s0 < 64 * pq + 64; s0 += SL) {
            const int m = s0 / (RB * W), y = s0 / W % RB, x = s0 % W;
            const float* ip = s_in + ((m * (RB + 2) + y) * E + x) * IB + i;
            float v[3][SL + 2];
#pragma unroll
            for (int ky = 0; ky < 3; ky++)
#pragma unroll
                for (int p = 0; p < SL + 2; p++) v[ky][p] = ip[(ky * E + p) * IB];
#pragma unroll
            for (int p = 0; p < SL; p++) {
                const float4 gv = *reinterpret_cast<const float4*>(s_g + (s0 + p) * GP + 4 * og);
                const float2 ga = make_float2(gv.x, gv.y), gb = make_float2(gv.z, gv.w);
                if (masked) {
#pragma unroll
                    for (int k = 0; k < 9; k++) {
                        const int yy = y0 + y + k / 3 - 1, xx = x + p + k % 3 - 1;
                        if (yy < 0 || yy >= W || xx < 0 || xx >= W) continue;
                        const float b = v[k / 3][p + k % 3];
                        if (ga.x != 0.f) part[0][k].x = fmaf(ga.x, b, part[0][k].x);
                        if (ga.y != 0.f) part[0][k].y = fmaf(ga.y, b, part[0][k].y);
                        if (gb.x != 0.f) part[1][k].x = fmaf(gb.x, b, part[1][k].x);
                        if (gb.y != 0.f) part[1][k].y = fmaf(gb.y, b, part[1][k].y);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 9; k++) {
                        const float2 b = make_float2(v[k / 3][p + k % 3], v[k / 3][p + k % 3]);
                        part[0][k] = fma2(ga, b, part[0][k]);
                        part[1][k] = fma2(gb, b, part[1][k]);
                    }
                }
                part[0][9].x += ga.x; part[0][9].y += ga.y;
                part[1][9].x += gb.x; part[1][9].y += gb.y;
            }
            if ((s0 + SL) % 16 == 0) {
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int k = 0; k < 10; k++) {
                        acc[h][k].x += part[h][k].x;
                        acc[h][k].y += part[h][k].y;
                    }
                zero(part);
            }
        }
        __syncthreads();
    }
    // the quarters' sums: 40 values per (channel group, input channel)
    float* const red = wsm;
    auto value = [&](int e) -> float& {   // e = 10 j + k: output channel j, tap k (9: the bias)
        const int j = e / 10, k = e % 10;
        float2& a = acc[j / 2][k];
        return j & 1 ? a.y : a.x;
    };
    if (pq > 0) {
#pragma unroll
        for (int e = 0; e < 40; e++) red[((pq - 1) * 40 + e) * 64 + (t & 63)] = value(e);
    }
    __syncthreads();
    if (pq == 0 && i0 + i < Ci) {
#pragma unroll
        for (int e = 0; e < 40; e++) {
            const float v = (value(e) + red[e * 64 + t]) + (red[(40 + e) * 64 + t] + red[(80 + e) * 64 + t]);
            const int o = o0 + 4 * og + e / 10, k = e % 10;
            if (k < 9) atomicAdd(&dW[((size_t)o * Ci + i0 + i) * 9 + k], (double)v);
            else if (i0 + i == 0) atomicAdd(&db[o], (double)v);
        }
    }
}

// 2 x 2 max pool (first maximum in row-major order on ties) with its argmax
__global__ void k_maxpool2(const float* __restrict__ in, float* __restrict__ out, unsigned char* __restrict__ arg,
                           long long planes, int H, int W) {
    const int Ho = H / 2, Wo = W / 2;
    const long long total = planes * Ho * Wo;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long pl = e / (Ho * Wo);
        const int r = (int)(e % (Ho * Wo)), y = r / Wo, x = r % Wo;
        const float* ip = in + pl * H * W + (2 * y) * W + 2 * x;
        float m = ip[0];
        int a = 0;
        if (ip[1] > m) { m = ip[1]; a = 1; }
        if (ip[W] > m) { m = ip[W]; a = 2; }
        if (ip[W + 1] > m) { m = ip[W + 1]; a = 3; }
        out[e] = m;
        arg[e] = (unsigned char)a;
    }
}

// gradient through the max pool and the ReLU before it: the selected input of
// each window receives the output gradient when that input was positive
__global__ void k_maxpool2_bwd(const float* __restrict__ gout, const unsigned char* __restrict__ arg,
                               const float* __restrict__ act, float* __restrict__ gin, long long planes, int H, int W) {
    const int Ho = H / 2, Wo = W / 2;
    const long long total = planes * Ho * Wo;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long pl = e / (Ho * Wo);
        const int r = (int)(e % (Ho * Wo)), y = r / Wo, x = r % Wo;
        const long long base = pl * H * W + (2 * y) * W + 2 * x;
        const int a = arg[e];
        const float gv = gout[e];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long long idx = base + (q / 2) * W + q % 2;
            gin[idx] = (q == a && act[idx] > 0.0f) ? gv : 0.0f;
        }
    }
}

// global max over the H*W pixels of each plane (first maximum) with its argmax
__global__ void k_global_max(const float* __restrict__ in, float* __restrict__ out, int* __restrict__ arg,
                             long long planes, int HW) {
    for (long long pl = blockIdx.x * (long long)blockDim.x + threadIdx.x; pl < planes;
         pl += (long long)gridDim.x * blockDim.x) {
        const float* ip = in + pl * HW;
        float m = ip[0];
        int a = 0;
        for (int p = 1; p < HW; p++)
            if (ip[p] > m) {
                m = ip[p];
                a = p;
            }
        out[pl] = m;
        arg[pl] = a;
    }
}

__global__ void k_global_max_bwd(const float* __restrict__ gout, const int* __restrict__ arg,
                                 const float* __restrict__ act, float* __restrict__ gin, long long planes, int HW) {
    const long long total = planes * HW;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long pl = e / HW;
        const int p = (int)(e % HW);
        gin[e] = (p == arg[pl] && act[e] > 0.0f) ? gout[pl] : 0.0f;
    }
}

// fully connected 128 -> 4
__global__ void k_fc(const float* __restrict__ g, const __nv_bfloat16* __restrict__ w, const float* __restrict__ b,
                     float* __restrict__ out, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * kOut) return;
    const int i = e / kOut, j = e % kOut;
    float s = b[j];
    for (int c = 0; c < kC4; c++) s = fmaf(g[(size_t)i * kC4 + c], __bfloat162float(w[j * kC4 + c]), s);
    out[e] = s;
}

// loss terms and the gradient of the outputs; one thread per tile
__global__ void k_loss(const float* __restrict__ out, const float* __restrict__ labels, float* __restrict__ dout,
                       double* loss, int n, float pos_weight, float dir_weight) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* o = out + (size_t)i * kOut;
    const float* l = labels + (size_t)i * 4;
    const float y = l[0];
    const float wgt = y > 0.5f ? pos_weight : 1.0f;
    const float inv_n = 1.0f / (float)n;
    // BCE with logits: max(o, 0) - o y + log(1 + exp(-|o|))
    const float z = o[0];
    const float bce = fmaxf(z, 0.0f) - z * y + log1pf(expf(-fabsf(z)));
    const float sig = 1.0f / (1.0f + expf(-z));
    float li = wgt * bce;
    float* d = dout + (size_t)i * kOut;
    d[0] = inv_n * wgt * (sig - y);
    d[1] = d[2] = d[3] = 0.0f;
    if (y > 0.5f) {
        const float dx = o[1], dy = o[2], dz = o[3];
        const float nn = dx * dx + dy * dy + dz * dz + 1e-12f;
        const float inv = rsqrtf(nn);
        const float dot = dx * l[1] + dy * l[2] + dz * l[3];
        li += dir_weight * (1.0f - dot * inv);
        const float c = -dir_weight * inv_n * inv;
        const float f = dot / nn;
        d[1] = c * (l[1] - f * dx);
        d[2] = c * (l[2] - f * dy);
        d[3] = c * (l[3] - f * dz);
    }
    atomicAdd(loss, (double)(li * inv_n));
}

// FC backward: dW5, db5 (one thread per weight) and dg
__global__ void k_fc_wgrad(const float* __restrict__ g, const float* __restrict__ dout, float* dW, float* db, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kOut * (kC4 + 1)) return;
    const int j = e / (kC4 + 1), c = e % (kC4 + 1);
    float s = 0.0f;
    for (int i = 0; i < n; i++) s = fmaf(dout[(size_t)i * kOut + j], c < kC4 ? g[(size_t)i * kC4 + c] : 1.0f, s);
    if (c < kC4) dW[j * kC4 + c] = s;
    else db[j] = s;
}

__global__ void k_fc_dgrad(const float* __restrict__ dout, const __nv_bfloat16* __restrict__ w, float* __restrict__ dg,
                           int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * kC4) return;
    const int i = e / kC4, c = e % kC4;
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < kOut; j++) s = fmaf(dout[(size_t)i * kOut + j], __bfloat162float(w[j * kC4 + c]), s);
    dg[e] = s;
}

__global__ void k_to_f32(const double* __restrict__ src, float* __restrict__ dst, long long n) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        dst[e] = (float)src[e];
}

__global__ void k_to_bf16(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        dst[e] = __float2bfloat16_rn(src[e]);
}

// Adam (Kingma & Ba 2015) on the FP32 master values, then the BF16 copies
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       __nv_bfloat16* __restrict__ p16, long long n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float ge = g[e];
        const float me = b1 * m[e] + (1.0f - b1) * ge;
        const float ve = b2 * v[e] + (1.0f - b2) * ge * ge;
        m[e] = me;
        v[e] = ve;
        const float pe = p[e] - lr * (me / c1) / (sqrtf(ve / c2) + eps);
        p[e] = pe;
        p16[e] = __float2bfloat16_rn(pe);
    }
}

// ----------------------------------------------------------------------------------------------
struct Layer {
    int ci, co, h;       // input channels, output channels, input height (= width)
    long long w, b;      // offsets of the weights and the bias in the parameter array
};

}  // namespace tmp

struct tm_pnet {
    int device = 0, cin = 0, tile = 0, max_batch = 0, nsm = 148;
    long long nparam = 0;
    tmp::Layer L[5];
    cudaStream_t stream = nullptr;
    float *p = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    double* sums = nullptr;   // of the convolutions' gradients, while the blocks add theirs
    __nv_bfloat16* p16 = nullptr;
    int step = 0;
    // activations (max_batch tiles) and their gradients
    float *x = nullptr, *a1 = nullptr, *q1 = nullptr, *a2 = nullptr, *q2 = nullptr, *a3 = nullptr, *q3 = nullptr,
          *a4 = nullptr, *g = nullptr, *out = nullptr, *lab = nullptr;
    unsigned char *i1 = nullptr, *i2 = nullptr, *i3 = nullptr;
    int* i4 = nullptr;
    float *d_a1 = nullptr, *d_q1 = nullptr, *d_a2 = nullptr, *d_q2 = nullptr, *d_a3 = nullptr, *d_q3 = nullptr,
          *d_a4 = nullptr, *d_g = nullptr, *d_out = nullptr;
    double* d_loss = nullptr;
    std::vector<void*> owned;
    std::string err;
};

namespace {

int pset_err(tm_pnet* c, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    return code;
}

#define PN_CUDA(c, expr)                                                                                     \
    do {                                                                                                     \
        cudaError_t e_ = (expr);                                                                             \
        if (e_ != cudaSuccess) return pset_err(c, TM_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_));    \
    } while (0)

template <typename T>
int palloc(tm_pnet* c, T** ptr, size_t count) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, count * sizeof(T) + 16);
    if (e != cudaSuccess) return pset_err(c, TM_ERR_CUDA, "cudaMalloc(%zu): %s", count * sizeof(T), cudaGetErrorString(e));
    c->owned.push_back(q);
    *ptr = (T*)q;
    return TM_OK;
}

int grid_for(long long n) {
    long long b = (n + 255) / 256;
    return (int)(b < 148LL * 16 ? (b > 0 ? b : 1) : 148LL * 16);
}

// grid (spatial tiles, output-channel groups, groups of images)
template <bool FLIP, class CT>
void conv_launch(tm_pnet* c, const float* in, const float* bias, float* out, const tmp::Layer& l, int n, int relu) {
    const int H = l.h, ci = FLIP ? l.co : l.ci, co = FLIP ? l.ci : l.co;
    const dim3 grid((H / CT::TW) * (H / CT::TW), (co + CT::COB - 1) / CT::COB, (n + CT::NI - 1) / CT::NI);
    tmp::k_conv3x3<FLIP, CT><<<grid, CT::NT, 0, c->stream>>>(in, c->p16 + l.w, bias, out, n, ci, co, H, relu);
}

// The form with one pixel per thread, fewer channels per block and so more blocks while these are
// at most one per SM (then a layer's time is that of one block, whatever their number), else the one with
// the most multiply-adds per load.  128 -> 128 channels, us at 2 / 32 / 128 / 1024 images,
// first form and second: 2 x 2 maps 61 / 69 / 69 / 153 and 66 / 85 / 85 / 109, 4 x 4
// 71 / 72 / 93 / 499 and 89 / 105 / 105 / 221; 2 / 32 / 64 / 128 images: 8 x 8 75 / 77 / 116 / 207 and
// 109 / 110 / 110 / 146, 16 x 16 (64 -> 128) 40 / 79 / 132 / 249 and 56 / 58 / 85 / 163.
template <bool FLIP, class FEW, class MANY>
void conv_few_or_many(tm_pnet* c, const float* in, const float* bias, float* out, const tmp::Layer& l, int n, int relu) {
    const int co = FLIP ? l.ci : l.co, tiles = (l.h / FEW::TW) * (l.h / FEW::TW);
    const long long blocks = (long long)tiles * ((co + FEW::COB - 1) / FEW::COB) * ((n + FEW::NI - 1) / FEW::NI);
    if (blocks <= c->nsm) conv_launch<FLIP, FEW>(c, in, bias, out, l, n, relu);
    else conv_launch<FLIP, MANY>(c, in, bias, out, l, n, relu);
}

template <bool FLIP>
void conv_dispatch(tm_pnet* c, const float* in, const float* bias, float* out, const tmp::Layer& l, int n, int relu) {
    using tmp::ConvTile;
    if (l.h >= 16) conv_few_or_many<FLIP, ConvTile<16, 1, 1, 1>, ConvTile<16, 4, 4, 1>>(c, in, bias, out, l, n, relu);
    else if (l.h == 8) conv_few_or_many<FLIP, ConvTile<8, 1, 4, 1>, ConvTile<8, 4, 8, 1>>(c, in, bias, out, l, n, relu);
    else if (l.h == 4) conv_few_or_many<FLIP, ConvTile<4, 1, 4, 2>, ConvTile<4, 4, 4, 8>>(c, in, bias, out, l, n, relu);
    else conv_few_or_many<FLIP, ConvTile<2, 1, 2, 16>, ConvTile<2, 2, 2, 32>>(c, in, bias, out, l, n, relu);
}

int conv(tm_pnet* c, bool flip, const float* in, const float* bias, float* out, const tmp::Layer& l, int n, int relu) {
    if (flip) conv_dispatch<true>(c, in, nullptr, out, l, n, 0);
    else conv_dispatch<false>(c, in, bias, out, l, n, relu);
    PN_CUDA(c, cudaGetLastError());
    return TM_OK;
}

int forward(tm_pnet* c, int n) {
    using namespace tmp;
    const int h1 = c->tile, h2 = h1 / 2, h3 = h1 / 4, h4 = h1 / 8;
    int rc;
    if ((rc = conv(c, false, c->x, c->p + c->L[0].b, c->a1, c->L[0], n, 1))) return rc;
    k_maxpool2<<<grid_for((long long)n * kC1 * h2 * h2), 256, 0, c->stream>>>(c->a1, c->q1, c->i1, (long long)n * kC1, h1, h1);
    if ((rc = conv(c, false, c->q1, c->p + c->L[1].b, c->a2, c->L[1], n, 1))) return rc;
    k_maxpool2<<<grid_for((long long)n * kC2 * h3 * h3), 256, 0, c->stream>>>(c->a2, c->q2, c->i2, (long long)n * kC2, h2, h2);
    if ((rc = conv(c, false, c->q2, c->p + c->L[2].b, c->a3, c->L[2], n, 1))) return rc;
    k_maxpool2<<<grid_for((long long)n * kC3 * h4 * h4), 256, 0, c->stream>>>(c->a3, c->q3, c->i3, (long long)n * kC3, h3, h3);
    if ((rc = conv(c, false, c->q3, c->p + c->L[3].b, c->a4, c->L[3], n, 1))) return rc;
    k_global_max<<<grid_for((long long)n * kC4), 256, 0, c->stream>>>(c->a4, c->g, c->i4, (long long)n * kC4, h4 * h4);
    k_fc<<<(n * kOut + 127) / 128, 128, 0, c->stream>>>(c->g, c->p16 + c->L[4].w, c->p + c->L[4].b, c->out, n);
    PN_CUDA(c, cudaGetLastError());
    return TM_OK;
}

template <int W>
int wgrad_launch(tm_pnet* c, const float* in, const float* g, const tmp::Layer& l, int n) {
    using WG = tmp::WGrad<W>;
    if (WG::SMEM > 48 * 1024)
        PN_CUDA(c, cudaFuncSetAttribute(tmp::k_conv3x3_wgrad<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, WG::SMEM));
    // about four blocks per SM over the channel tiles and shares of the pixels
    const int tiles = (l.co / WG::OB) * ((l.ci + WG::IB - 1) / WG::IB);
    const int total = (n + WG::NI - 1) / WG::NI * (W / WG::RB);
    int shares = (c->nsm * 4 + tiles - 1) / tiles;
    if (shares > total) shares = total;
    const int units = (total + shares - 1) / shares;
    tmp::k_conv3x3_wgrad<W><<<dim3(tiles, (total + units - 1) / units), tmp::kThreads, WG::SMEM, c->stream>>>(
        in, g, c->sums + l.w, c->sums + l.b, n, l.ci, l.co, units);
    PN_CUDA(c, cudaGetLastError());
    return TM_OK;
}

int wgrad(tm_pnet* c, const float* in, const float* g, const tmp::Layer& l, int n) {
    switch (l.h) {
        case 128: return wgrad_launch<128>(c, in, g, l, n);
        case 64: return wgrad_launch<64>(c, in, g, l, n);
        case 32: return wgrad_launch<32>(c, in, g, l, n);
        case 16: return wgrad_launch<16>(c, in, g, l, n);
        case 8: return wgrad_launch<8>(c, in, g, l, n);
        case 4: return wgrad_launch<4>(c, in, g, l, n);
        default: return wgrad_launch<2>(c, in, g, l, n);
    }
}

// forward + loss + backward into c->grad; the loss sum into c->d_loss
int backward(tm_pnet* c, int n, float pos_weight, float dir_weight) {
    using namespace tmp;
    const int h1 = c->tile, h2 = h1 / 2, h3 = h1 / 4, h4 = h1 / 8;
    int rc;
    if ((rc = forward(c, n))) return rc;
    PN_CUDA(c, cudaMemsetAsync(c->sums, 0, sizeof(double) * c->L[4].w, c->stream));
    PN_CUDA(c, cudaMemsetAsync(c->d_loss, 0, sizeof(double), c->stream));
    k_loss<<<(n + 127) / 128, 128, 0, c->stream>>>(c->out, c->lab, c->d_out, c->d_loss, n, pos_weight, dir_weight);
    k_fc_wgrad<<<(kOut * (kC4 + 1) + 127) / 128, 128, 0, c->stream>>>(c->g, c->d_out, c->grad + c->L[4].w,
                                                                        c->grad + c->L[4].b, n);
    k_fc_dgrad<<<(n * kC4 + 255) / 256, 256, 0, c->stream>>>(c->d_out, c->p16 + c->L[4].w, c->d_g, n);
    k_global_max_bwd<<<grid_for((long long)n * kC4 * h4 * h4), 256, 0, c->stream>>>(c->d_g, c->i4, c->a4, c->d_a4,
                                                                                    (long long)n * kC4, h4 * h4);
    PN_CUDA(c, cudaGetLastError());
    // layer 4
    if ((rc = wgrad(c, c->q3, c->d_a4, c->L[3], n))) return rc;
    if ((rc = conv(c, true, c->d_a4, nullptr, c->d_q3, c->L[3], n, 0))) return rc;
    k_maxpool2_bwd<<<grid_for((long long)n * kC3 * h4 * h4), 256, 0, c->stream>>>(c->d_q3, c->i3, c->a3, c->d_a3,
                                                                                  (long long)n * kC3, h3, h3);
    // layer 3
    if ((rc = wgrad(c, c->q2, c->d_a3, c->L[2], n))) return rc;
    if ((rc = conv(c, true, c->d_a3, nullptr, c->d_q2, c->L[2], n, 0))) return rc;
    k_maxpool2_bwd<<<grid_for((long long)n * kC2 * h3 * h3), 256, 0, c->stream>>>(c->d_q2, c->i2, c->a2, c->d_a2,
                                                                                  (long long)n * kC2, h2, h2);
    // layer 2
    if ((rc = wgrad(c, c->q1, c->d_a2, c->L[1], n))) return rc;
    if ((rc = conv(c, true, c->d_a2, nullptr, c->d_q1, c->L[1], n, 0))) return rc;
    k_maxpool2_bwd<<<grid_for((long long)n * kC1 * h2 * h2), 256, 0, c->stream>>>(c->d_q1, c->i1, c->a1, c->d_a1,
                                                                                  (long long)n * kC1, h1, h1);
    // layer 1 (no gradient of the input)
    if ((rc = wgrad(c, c->x, c->d_a1, c->L[0], n))) return rc;
    k_to_f32<<<grid_for(c->L[4].w), 256, 0, c->stream>>>(c->sums, c->grad, c->L[4].w);
    PN_CUDA(c, cudaGetLastError());
    return TM_OK;
}

int upload(tm_pnet* c, const float* tiles, const float* labels, int n) {
    if (n < 1 || n > c->max_batch) return pset_err(c, TM_ERR_INVALID, "batch %d outside 1..%d", n, c->max_batch);
    if (!tiles) return pset_err(c, TM_ERR_INVALID, "null tiles");
    const size_t per = (size_t)c->cin * c->tile * c->tile;
    PN_CUDA(c, cudaMemcpyAsync(c->x, tiles, sizeof(float) * per * n, cudaMemcpyHostToDevice, c->stream));
    if (labels) PN_CUDA(c, cudaMemcpyAsync(c->lab, labels, sizeof(float) * 4 * n, cudaMemcpyHostToDevice, c->stream));
    return TM_OK;
}

}  // namespace

extern "C" {

int tm_pnet_create(int device, int in_channels, int tile, int max_batch, tm_pnet** out) {
    if (!out) return TM_ERR_INVALID;
    *out = nullptr;
    if (in_channels < 1 || in_channels > 64 || max_batch < 1 || max_batch > 4096) return TM_ERR_INVALID;
    if (tile != 16 && tile != 32 && tile != 64 && tile != 128) return TM_ERR_UNSUPPORTED;
    tm_pnet* c = new tm_pnet();
    c->device = device;
    c->cin = in_channels;
    c->tile = tile;
    c->max_batch = max_batch;
    const int chans[5] = {in_channels, tmp::kC1, tmp::kC2, tmp::kC3, tmp::kC4};
    long long off = 0;
    for (int l = 0; l < 4; l++) {
        c->L[l].ci = chans[l];
        c->L[l].co = chans[l + 1];
        c->L[l].h = tile >> l;
        c->L[l].w = off;
        off += (long long)chans[l] * chans[l + 1] * 9;
        c->L[l].b = off;
        off += chans[l + 1];
    }
    c->L[4].ci = tmp::kC4;
    c->L[4].co = tmp::kOut;
    c->L[4].h = 1;
    c->L[4].w = off;
    off += tmp::kC4 * tmp::kOut;
    c->L[4].b = off;
    off += tmp::kOut;
    c->nparam = off;
    auto fail = [&](int rc) {
        tm_pnet_destroy(c);
        return rc;
    };
    if (cudaSetDevice(device) != cudaSuccess) return fail(TM_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(TM_ERR_CUDA);
    const long long B = max_batch, h = tile;
    int rc = TM_OK;
    rc = rc ? rc : palloc(c, &c->p, c->nparam);
    rc = rc ? rc : palloc(c, &c->grad, c->nparam);
    rc = rc ? rc : palloc(c, &c->sums, c->L[4].w);
    rc = rc ? rc : palloc(c, &c->m, c->nparam);
    rc = rc ? rc : palloc(c, &c->v, c->nparam);
    rc = rc ? rc : palloc(c, &c->p16, c->nparam);
    rc = rc ? rc : palloc(c, &c->x, B * in_channels * h * h);
    rc = rc ? rc : palloc(c, &c->a1, B * tmp::kC1 * h * h);
    rc = rc ? rc : palloc(c, &c->q1, B * tmp::kC1 * h * h / 4);
    rc = rc ? rc : palloc(c, &c->i1, B * tmp::kC1 * h * h / 4);
    rc = rc ? rc : palloc(c, &c->a2, B * tmp::kC2 * h * h / 4);
    rc = rc ? rc : palloc(c, &c->q2, B * tmp::kC2 * h * h / 16);
    rc = rc ? rc : palloc(c, &c->i2, B * tmp::kC2 * h * h / 16);
    rc = rc ? rc : palloc(c, &c->a3, B * tmp::kC3 * h * h / 16);
    rc = rc ? rc : palloc(c, &c->q3, B * tmp::kC3 * h * h / 64);
    rc = rc ? rc : palloc(c, &c->i3, B * tmp::kC3 * h * h / 64);
    rc = rc ? rc : palloc(c, &c->a4, B * tmp::kC4 * h * h / 64);
    rc = rc ? rc : palloc(c, &c->g, B * tmp::kC4);
    rc = rc ? rc : palloc(c, &c->i4, B * tmp::kC4);
    rc = rc ? rc : palloc(c, &c->out, B * tmp::kOut);
    rc = rc ? rc : palloc(c, &c->lab, B * 4);
    rc = rc ? rc : palloc(c, &c->d_a1, B * tmp::kC1 * h * h);
    rc = rc ? rc : palloc(c, &c->d_q1, B * tmp::kC1 * h * h / 4);
    rc = rc ? rc : palloc(c, &c->d_a2, B * tmp::kC2 * h * h / 4);
    rc = rc ? rc : palloc(c, &c->d_q2, B * tmp::kC2 * h * h / 16);
    rc = rc ? rc : palloc(c, &c->d_a3, B * tmp::kC3 * h * h / 16);
    rc = rc ? rc : palloc(c, &c->d_q3, B * tmp::kC3 * h * h / 64);
    rc = rc ? rc : palloc(c, &c->d_a4, B * tmp::kC4 * h * h / 64);
    rc = rc ? rc : palloc(c, &c->d_g, B * tmp::kC4);
    rc = rc ? rc : palloc(c, &c->d_out, B * tmp::kOut);
    rc = rc ? rc : palloc(c, &c->d_loss, 1);
    if (rc) return fail(rc);
    if (cudaMemset(c->p, 0, sizeof(float) * c->nparam) != cudaSuccess ||
        cudaMemset(c->m, 0, sizeof(float) * c->nparam) != cudaSuccess ||
        cudaMemset(c->v, 0, sizeof(float) * c->nparam) != cudaSuccess ||
        cudaMemset(c->p16, 0, sizeof(__nv_bfloat16) * c->nparam) != cudaSuccess)
        return fail(TM_ERR_CUDA);
    *out = c;
    return TM_OK;
}

long long tm_pnet_param_count(const tm_pnet* c) { return c ? c->nparam : -1; }

int tm_pnet_set_params(tm_pnet* c, const float* params) {
    if (!c || !params) return TM_ERR_INVALID;
    PN_CUDA(c, cudaSetDevice(c->device));
    PN_CUDA(c, cudaMemcpyAsync(c->p, params, sizeof(float) * c->nparam, cudaMemcpyHostToDevice, c->stream));
    PN_CUDA(c, cudaMemsetAsync(c->m, 0, sizeof(float) * c->nparam, c->stream));
    PN_CUDA(c, cudaMemsetAsync(c->v, 0, sizeof(float) * c->nparam, c->stream));
    tmp::k_to_bf16<<<grid_for(c->nparam), 256, 0, c->stream>>>(c->p, c->p16, c->nparam);
    PN_CUDA(c, cudaGetLastError());
    PN_CUDA(c, cudaStreamSynchronize(c->stream));
    c->step = 0;
    return TM_OK;
}

int tm_pnet_get_params(tm_pnet* c, float* params) {
    if (!c || !params) return TM_ERR_INVALID;
    PN_CUDA(c, cudaSetDevice(c->device));
    PN_CUDA(c, cudaMemcpyAsync(params, c->p, sizeof(float) * c->nparam, cudaMemcpyDeviceToHost, c->stream));
    PN_CUDA(c, cudaStreamSynchronize(c->stream));
    return TM_OK;
}

int tm_pnet_forward(tm_pnet* c, const float* tiles, int n, float* outputs) {
    if (!c || !outputs) return TM_ERR_INVALID;
    PN_CUDA(c, cudaSetDevice(c->device));
    int rc = upload(c, tiles, nullptr, n);
    if (rc) return rc;
    if ((rc = forward(c, n))) return rc;
    PN_CUDA(c, cudaMemcpyAsync(outputs, c->out, sizeof(float) * tmp::kOut * n, cudaMemcpyDeviceToHost, c->stream));
    PN_CUDA(c, cudaStreamSynchronize(c->stream));
    return TM_OK;
}

int tm_pnet_gradients(tm_pnet* c, const float* tiles, const float* labels, int n, float pos_weight, float dir_weight,
                      double* loss, float* grads) {
    if (!c || !labels || !loss || !grads) return TM_ERR_INVALID;
    PN_CUDA(c, cudaSetDevice(c->device));
    int rc = upload(c, tiles, labels, n);
    if (rc) return rc;
    if ((rc = backward(c, n, pos_weight, dir_weight))) return rc;
    PN_CUDA(c, cudaMemcpyAsync(grads, c->grad, sizeof(float) * c->nparam, cudaMemcpyDeviceToHost, c->stream));
    PN_CUDA(c, cudaMemcpyAsync(loss, c->d_loss, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    PN_CUDA(c, cudaStreamSynchronize(c->stream));
    return TM_OK;
}

int tm_pnet_train_step(tm_pnet* c, const float* tiles, const float* labels, int n, float pos_weight, float dir_weight,
                       float lr, double* loss) {
    if (!c || !labels) return TM_ERR_INVALID;
    PN_CUDA(c, cudaSetDevice(c->device));
    int rc = upload(c, tiles, labels, n);
    if (rc) return rc;
    if ((rc = backward(c, n, pos_weight, dir_weight))) return rc;
    c->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)c->step), c2 = 1.0f - powf(b2, (float)c->step);
    tmp::k_adam<<<grid_for(c->nparam), 256, 0, c->stream>>>(c->p, c->grad, c->m, c->v, c->p16, c->nparam, lr, b1, b2,
                                                           1e-8f, c1, c2);
    PN_CUDA(c, cudaGetLastError());
    if (loss) PN_CUDA(c, cudaMemcpyAsync(loss, c->d_loss, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    PN_CUDA(c, cudaStreamSynchronize(c->stream));
    return TM_OK;
}

const char* tm_pnet_last_error(const tm_pnet* c) { return c ? c->err.c_str() : "null network"; }

int tm_pnet_destroy(tm_pnet* c) {
    if (!c) return TM_OK;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    for (void* q : c->owned) cudaFree(q);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return TM_OK;
}

}  // extern "C"
