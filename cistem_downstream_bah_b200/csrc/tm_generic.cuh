// tm_generic.cuh -- run-time-length transforms for micrograph sizes without
// compiled kernels.
//
// The reference pads a micrograph side to the nearest size whose prime factors
// are small (match_template.cpp:527-575 with ReturnClosestFactorizedUpper,
// functions.cpp:529-577: largest factor 2, then 3, 5, 7, 9, 13, each within
// 10 % growth and a multiple of 4), so a side can carry the primes 2, 3, 5, 7,
// 11 and 13.  The compiled kernels cover the power-of-two widths and the
// 2^a 3^b heights of the common camera formats; every other padded size runs
// on the kernels here, whose FFT lengths are arguments:
//
//   fft_gen        a Stockham transform of a line of length L held in shared
//                  memory (two buffers, ping-pong), radix plan (16, 8, 4, 2,
//                  9, 3, 5, 7, 11, 13) chosen on the host
//   k_pass_a_gen   forward FFT along x of each normalised projection row
//   k_pass_b_gen   per column: forward FFT along y, conjugate multiply with
//                  I', inverse FFT along y
//   k_pass_c_gen   per row: the c2r packing, inverse X/2-point FFT and the
//                  MIP / argmax / compensated sums / histogram update
//   (..._gen2: the same on pairs of lines; the one-line forms take the lengths whose
//   pairs do not fit shared memory)
//   k_w_rows_gen,  the whitening's row r2c and column FFT (with the quadrant
//   k_w_cols_gen   swap and zeroed central pixel)
//
// The arithmetic is the compiled path's (FP32, the same packing and twiddle
// tables; FP64 sums of every value as at compiled widths below 2048, but for the
// longest odd rows, whose sums are FP32, compensated at each value); only the FFT
// organisation differs.  Lines up to
// kGenMaxLen = 8192 points.
#pragma once
#include <type_traits>

#include "tm_fft.cuh"
#include "tm_generic_forms.h"
#include "tm_whiten.cuh"

namespace tmk {

constexpr int kGenMaxStages = 24;
constexpr int kGenNT = 512;
constexpr int kGenMaxLen = 8192;

struct GenPlan {
    int L;                          // transform length
    int n;                          // stages
    int r[kGenMaxStages];           // radices, product L
    int ns[kGenMaxStages];          // product of the earlier radices
    unsigned int mns[kGenMaxStages];   // ceil(2^32 / ns): b / ns = umulhi(b, mns) for b < 2^19, ns > 1
};

// Radix plan of L; false when L has a prime factor above 13 or is too long.
inline bool gen_plan(int L, GenPlan& p) {
    p.L = L;
    p.n = 0;
    if (L < 2 || L > kGenMaxLen) return false;
    int m = L;
    const int order[] = {16, 8, 4, 2, 9, 3, 5, 7, 11, 13};
    for (int r : order)
        while (m % r == 0 && p.n < kGenMaxStages) {
            const int ns = L / m;
            p.ns[p.n] = ns;
            p.mns[p.n] = ns > 1 ? (unsigned int)(((1ULL << 32) + ns - 1) / ns) : 0u;
            p.r[p.n++] = r;
            m /= r;
        }
    return m == 1;
}

// R-point DFT of prime length as R^2 multiplications by compile-time constants
template <int R, int DIR>
__device__ __forceinline__ void dft_naive(float2* e) {
    float2 o[R];
    tmfft::sfor<R>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        float2 acc = e[0];
        tmfft::sfor<R - 1>([&](auto ic) {
            constexpr int i = decltype(ic)::value + 1;
            acc = tmfft::cadd(acc, tmfft::twc<R, (i * k) % R, DIR>(e[i]));
        });
        o[k] = acc;
    });
#pragma unroll
    for (int i = 0; i < R; i++) e[i] = o[i];
}

template <int R, int DIR>
__device__ __forceinline__ void dft_any(float2* e) {
    if constexpr (R == 5 || R == 7 || R == 11 || R == 13) dft_naive<R, DIR>(e);
    else tmfft::dft<R, DIR>(e);
}

// One Stockham stage of radix R over `lines` lines (line stride `stride`), from
// `in` to `out`: butterfly b reads elements b + i L/R, twiddles them by
// W_{Ns R}^{(b mod Ns) i} and writes (b / Ns) Ns R + b mod Ns + i Ns -- the
// pattern of tmfft::fft.
template <int R, int DIR>
__device__ __forceinline__ void gen_stage(const float2* in, float2* out, int stride, int lines, int L, int Ns,
                                          const tmfft::Twiddles& tw) {
    const int nbf = L / R, total = lines * nbf;
    for (int g = threadIdx.x; g < total; g += kGenNT) {
        const int line = g / nbf, b = g - line * nbf;
        const float2* src = in + (size_t)line * stride;
        float2* dst = out + (size_t)line * stride;
        const int jm = b % Ns;
        const float2 w = tw.template w<DIR>(jm * (L / (Ns * R)), L);
        float2 e[R];
#pragma unroll
        for (int i = 0; i < R; i++) e[i] = src[b + i * nbf];
        float2 wp = w;
#pragma unroll
        for (int i = 1; i < R; i++) {
            e[i] = tmfft::cmul(e[i], wp);
            wp = tmfft::cmul(wp, w);
        }
        dft_any<R, DIR>(e);
        const int base = (b / Ns) * Ns * R + jm;
#pragma unroll
        for (int i = 0; i < R; i++) dst[base + i * Ns] = e[i];
    }
    __syncthreads();
}

// Transform of `lines` lines held in shared memory, ping-ponging between buf
// and tmp (both lines x stride); returns the buffer that holds the result.  The
// caller has passed a barrier since buf was filled.  DIR = -1 forward, +1
// inverse, unnormalised.  The twiddle table's length is a multiple of L.
template <int DIR>
__device__ float2* fft_gen(float2* buf, float2* tmp, int stride, int lines, const GenPlan& p, const tmfft::Twiddles& tw) {
    int Ns = 1;
    float2 *in = buf, *out = tmp;
    for (int s = 0; s < p.n; s++) {
        const int R = p.r[s];
        switch (R) {
            case 16: gen_stage<16, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 8: gen_stage<8, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 4: gen_stage<4, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 2: gen_stage<2, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 9: gen_stage<9, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 3: gen_stage<3, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 5: gen_stage<5, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 7: gen_stage<7, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            case 11: gen_stage<11, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
            default: gen_stage<13, DIR>(in, out, stride, lines, p.L, Ns, tw); break;
        }
        Ns *= R;
        float2* sw = in;
        in = out;
        out = sw;
    }
    return in;
}

// ---------------------------------------------------------------------------------------
// k_pass_a_gen: block per (row, orientation); the T normalised samples at the
// start of an X-point line, forward FFT, kx = 0 .. X/2 into A.
template <int T>
__global__ void __launch_bounds__(kGenNT) k_pass_a_gen(BatchArgs a, int X, GenPlan px) {
    extern __shared__ float2 gbuf[];   // 2 x X
    const int row = blockIdx.x, o = blockIdx.y;
    const float2 nrm = a.norm[o];
    const float* prow = a.P + ((size_t)o * T + row) * T;
    for (int i = threadIdx.x; i < X; i += kGenNT)
        gbuf[i] = make_float2(i < T ? (prow[i] - nrm.x) * nrm.y : 0.f, 0.f);
    __syncthreads();
    const float2* f = fft_gen<-1>(gbuf, gbuf + X, X, 1, px, a.tw);
    float2* out = a.A + ((size_t)o * T + row) * a.XP;
    for (int k = threadIdx.x; k <= X / 2; k += kGenNT) out[k] = f[k];
}

// k_pass_b_gen: block per (column, orientation), for the heights whose column pairs do not
// fit shared memory twice (gen_col_pass).
__global__ void __launch_bounds__(kGenNT) k_pass_b_gen(BatchArgs a, int T, int Y, int, GenPlan py) {
    extern __shared__ float2 gbuf[];   // 2 x Y
    const int kx = blockIdx.x, o = blockIdx.y;
    const int XP = a.XP;
    const float2* Ao = a.A + (size_t)o * T * XP + kx;
    for (int n = threadIdx.x; n < Y; n += kGenNT) gbuf[n] = n < T ? Ao[(size_t)n * XP] : make_float2(0.f, 0.f);
    __syncthreads();
    float2* f = fft_gen<-1>(gbuf, gbuf + Y, Y, 1, py, a.twy);
    for (int k = threadIdx.x; k < Y; k += kGenNT) f[k] = cmul_conj(__ldg(a.Ip + (size_t)k * XP + kx), f[k]);
    __syncthreads();
    const float2* z = fft_gen<+1>(f, f == gbuf ? gbuf + Y : gbuf, Y, 1, py, a.twy);
    for (int yy = threadIdx.x; yy < Y; yy += kGenNT) __stcs(a.C + c_index_rt(Y, o, yy, kx, XP), z[yy]);
}
// k_pass_c_gen: block per row y of an odd width whose row pairs do not fit shared memory twice
// (gen_pass_c_pairs): the full X-point inverse of the Hermitian extension, one orientation
// at a time; thread t owns the pixels x = t + kGenNT j and keeps their state in registers over
// the batch.
__global__ void __launch_bounds__(kGenNT, 1)
k_pass_c_gen(BatchArgs a, int X, int Y, GenPlan ph) {
    constexpr int MAXP = 16;
    static_assert(kGenNT * 16 >= kGenMaxLen, "16 pixels per thread cover the longest rows");
    extern __shared__ float2 gbuf[];             // 2 x X, then the histogram
    const int L = X, HC = X / 2 + 1, XP = a.XP, y = blockIdx.x, t = threadIdx.x;
    unsigned int* shist = reinterpret_cast<unsigned int*>(gbuf + 2 * L);
    for (int b = t; b < a.hist_bins; b += kGenNT) shist[b] = 0u;
    float mip[MAXP], fs[MAXP], fq[MAXP], cs[MAXP], cq[MAXP];
    int best[MAXP];
    const size_t rowoff = (size_t)y * X;
#pragma unroll
    for (int j = 0; j < MAXP; j++) {
        const int x = t + kGenNT * j;
        if (x < X) {
            mip[j] = a.mip[rowoff + x];
            best[j] = a.best[rowoff + x];
        }
        fs[j] = fq[j] = cs[j] = cq[j] = 0.f;
    }
    for (int o = 0; o < a.nb; o++) {
        for (int k = t; k < X; k += kGenNT) {
            const int kx = k < HC ? k : X - k;
            float2 v = __ldg(a.C + c_index_rt(Y, o, y, kx, XP));
            if (k >= HC) v = tmfft::conjf2(v);
            if (k == 0) v.y = 0.f;
            gbuf[k] = v;
        }
        __syncthreads();
        const float2* zb = fft_gen<+1>(gbuf, gbuf + L, L, 1, ph, a.tw);
        const int g = (int)(a.gidx0 + o);
#pragma unroll
        for (int j = 0; j < MAXP; j++) {
            const int x = t + kGenNT * j;
            if (x < X) {
                const float val = zb[x].x;
                if (val > mip[j]) { mip[j] = val; best[j] = g; }
                const float ys = val - cs[j];
                const float ts = fs[j] + ys;
                cs[j] = (ts - fs[j]) - ys;
                fs[j] = ts;
                const float yq = fmaf(val, val, -cq[j]);
                const float tq = fq[j] + yq;
                cq[j] = (tq - fq[j]) - yq;
                fq[j] = tq;
                const int bin = __float2int_rz((val - a.hist_min) * a.hist_inv_step);
                if (bin >= 0 && bin < a.hist_bins) atomicAdd(&shist[bin], 1u);
            }
        }
        __syncthreads();   // every output is read before the next orientation's row
    }
#pragma unroll
    for (int j = 0; j < MAXP; j++) {
        const int x = t + kGenNT * j;
        if (x < X) {
            a.mip[rowoff + x] = mip[j];
            a.best[rowoff + x] = best[j];
            a.sum[rowoff + x] += (double)fs[j] - (double)cs[j];
            a.sumsq[rowoff + x] += (double)fq[j] - (double)cq[j];
        }
    }
    __syncthreads();
    for (int b = t; b < a.hist_bins; b += kGenNT) {
        const unsigned int cnt = shist[b];
        if (cnt) atomicAdd(a.hist + b, (unsigned long long)cnt);
    }
}

// ---------------------------------------------------------------------------------------
// The same transforms on pairs of lines (tmfft::Pair: two rows of A, two columns, two
// orientations of a row), 16 bytes per element: the index arithmetic, the twiddle chain and
// the barriers are shared by both, the additions take one instruction for both, and each half
// gets the bits of the scalar transform.  Quotients by a stage's Ns come from a
// reciprocal, twiddles from a stride fixed per stage (three integer divisions per butterfly
// before).  With few warps per SM these kernels wait for memory first of all, so the twiddle
// table and the next item's input lie in shared memory where they fit.  64 orientations at
// 2700 x 2700, line by line -> pairs: rows of A 0.74 -> 0.38 ms, columns 6.3 -> 3.9, rows of
// C 7.0 -> 2.5; what bounds them is the exchange through shared memory once per radix
// (16 bytes per element and stage, in and out).  Where two pairs' buffers do not fit shared
// memory the one-line forms stay.

// One Stockham stage over `lines` (1 or 2) lines.  MUL: the input is I' conj(in), I' of the
// line's two columns at ip + line (pitch ipp float4 per element).
template <int R, int DIR, int NT, bool MUL>
__device__ __forceinline__ void pgen_stage(const float4* in, float4* out, int lines, const GenPlan& p, int s,
                                           const tmfft::Twiddles& tw, const float4* ip, int ipp) {
    using tmfft::Pair;
    const int L = p.L, nbf = L / R, Ns = p.ns[s];
    const unsigned int mns = p.mns[s];
    const int step = tw.lmax / (Ns * R);
    for (int g = threadIdx.x; g < lines * nbf; g += NT) {
        const int line = g >= nbf ? 1 : 0, b = g - line * nbf;
        const float4* src = in + line * L + b;
        const int q = Ns > 1 ? (int)__umulhi((unsigned int)b, mns) : b;
        const int jm = b - q * Ns;
        Pair e[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const float4 f = src[i * nbf];
            e[i] = {make_float2(f.x, f.y), make_float2(f.z, f.w)};
            if constexpr (MUL) {
                const float4 v = __ldg(ip + line + (size_t)(b + i * nbf) * ipp);
                e[i] = tmfft::pmul_conj(make_float2(v.x, v.z), make_float2(v.y, v.w), e[i]);
            }
        }
        if (Ns > 1) {
            float2 w = tw.tab[jm * step];
            if (DIR > 0) w.y = -w.y;
            float2 wp = w;
#pragma unroll
            for (int i = 1; i < R; i++) {
                e[i] = tmfft::pmul(e[i], wp);
                wp = tmfft::cmul(wp, w);
            }
        }
        tmfft::pdft<R, DIR>(e);
        float4* dst = out + line * L + q * (Ns * R) + jm;
#pragma unroll
        for (int i = 0; i < R; i++) dst[i * Ns] = make_float4(e[i].re.x, e[i].re.y, e[i].im.x, e[i].im.y);
    }
    __syncthreads();
}

// Stages s0 .. of the transform of `lines` lines; MUL0: stage s0 multiplies by I' (above).
// The caller has passed a barrier since buf was filled; returns the buffer with the result.
template <int DIR, int NT, bool MUL0>
__device__ __forceinline__ float4* pfft_gen(float4* buf, float4* tmp, int lines, const GenPlan& p, int s0,
                                            const tmfft::Twiddles& tw, const float4* ip = nullptr, int ipp = 0) {
    float4 *in = buf, *out = tmp;
    for (int s = s0; s < p.n; s++) {
        auto stage = [&](auto mul) {
            constexpr bool M = decltype(mul)::value;
            switch (p.r[s]) {
                case 16: pgen_stage<16, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 8: pgen_stage<8, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 4: pgen_stage<4, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 2: pgen_stage<2, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 9: pgen_stage<9, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 3: pgen_stage<3, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 5: pgen_stage<5, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 7: pgen_stage<7, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                case 11: pgen_stage<11, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
                default: pgen_stage<13, DIR, NT, M>(in, out, lines, p, s, tw, ip, ipp); break;
            }
        };
        if constexpr (MUL0) {
            if (s == s0) stage(std::true_type{});
            else stage(std::false_type{});
        } else {
            stage(std::false_type{});
        }
        float4* sw = in;
        in = out;
        out = sw;
    }
    return in;
}

// Fills a line's buffer with its first T elements (value(n)) and zeros, or, where the first
// stage's butterflies then hold one element at most (T <= L / r[0]), with that stage's output:
// each element r[0] times, as the others add nothing.  Returns the first stage left to do.
template <int NT, class Value>
__device__ __forceinline__ int pfill_pruned(float4* buf, int lines, int T, const GenPlan& p, Value value) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int L = p.L, R = p.r[0], nbf = L / R;
    if (T > nbf || p.n < 2) {
        for (int e = threadIdx.x; e < lines * L; e += NT) {
            const int line = e >= L ? 1 : 0, n = e - line * L;
            buf[e] = n < T ? value(line, n) : zero;
        }
        return 0;
    }
    for (int e = threadIdx.x; e < lines * nbf; e += NT) {
        const int line = e >= nbf ? 1 : 0, n = e - line * nbf;
        const float4 v = n < T ? value(line, n) : zero;
        for (int i = 0; i < R; i++) buf[line * L + n * R + i] = v;
    }
    return 1;
}

// k_pass_a_gen2: block per (two rows, orientation)
template <int T>
__global__ void __launch_bounds__(256) k_pass_a_gen2(const __grid_constant__ BatchArgs a, int X, const __grid_constant__ GenPlan px) {
    extern __shared__ __align__(16) float4 pbuf[];   // 2 x X
    const int row = 2 * blockIdx.x, o = blockIdx.y;
    const float2 nrm = a.norm[o];
    const float* prow = a.P + ((size_t)o * T + row) * T;
    const int s0 = pfill_pruned<256>(pbuf, 1, T, px, [&](int, int n) {
        return make_float4((prow[n] - nrm.x) * nrm.y, (prow[T + n] - nrm.x) * nrm.y, 0.f, 0.f);
    });
    __syncthreads();
    const float4* f = pfft_gen<-1, 256, false>(pbuf, pbuf + X, 1, px, s0, a.tw);
    float2* out = a.A + ((size_t)o * T + row) * a.XP;
    for (int k = threadIdx.x; k <= X / 2; k += 256) {
        const float4 z = f[k];
        out[k] = make_float2(z.x, z.z);
        out[a.XP + k] = make_float2(z.y, z.w);
    }
}

// k_pass_b_gen2: block per (LP pairs of adjacent columns, `ob` orientations in turn).
// Shared memory: gen_pass_b_smem.
template <int LP, bool TAB, bool STAGED>
__global__ void __launch_bounds__(kGenNT) k_pass_b_gen2(const __grid_constant__ BatchArgs a, int T, int Y, int ob, const __grid_constant__ GenPlan py) {
    extern __shared__ __align__(16) float4 pbuf[];   // pair c of a buffer at c * Y
    float4* const tmp = pbuf + LP * Y;
    float2* const tab = reinterpret_cast<float2*>(tmp + LP * Y);
    float4* const astage = reinterpret_cast<float4*>(TAB ? tab + Y + Y % 2 : tab);   // [row][pair]
    const int kx0 = blockIdx.x * (2 * LP), o0 = blockIdx.y * ob, o1 = min(a.nb, o0 + ob);
    const int XP = a.XP;
    tmfft::Twiddles tw = a.twy;
    if constexpr (TAB) {
        for (int e = threadIdx.x; e < Y; e += kGenNT) tab[e] = __ldg(a.twy.tab + e);
        tw.tab = tab;
    }
    auto issue_rows = [&](int o) {
        const float2* Ao = a.A + (size_t)o * T * XP + kx0;
        for (int e = threadIdx.x; e < T * LP; e += kGenNT) {
            const float2* src = Ao + (size_t)(e / LP) * XP + 2 * (e % LP);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tmptx::smem_u32(astage + e)), "l"(src) : "memory");
        }
        tmptx::cp_async_commit();
    };
    if constexpr (STAGED) issue_rows(o0);
    for (int o = o0; o < o1; o++) {
        if constexpr (STAGED) tmptx::cp_async_wait<0>();
        __syncthreads();   // the rows (and the table); the previous orientation's output is stored
        const int s0 = pfill_pruned<kGenNT>(pbuf, LP, T, py, [&](int c, int n) {
            const float4 v = STAGED ? astage[n * LP + c]
                                    : __ldg(reinterpret_cast<const float4*>(a.A + ((size_t)o * T + n) * XP + kx0 + 2 * c));
            return make_float4(v.x, v.z, v.y, v.w);
        });
        __syncthreads();
        if constexpr (STAGED) {
            if (o + 1 < o1) issue_rows(o + 1);
        }
        float4* f = pfft_gen<-1, kGenNT, false>(pbuf, tmp, LP, py, s0, tw);
        const float4* z = pfft_gen<+1, kGenNT, true>(f, f == pbuf ? tmp : pbuf, LP, py, 0, tw,
                                                     reinterpret_cast<const float4*>(a.Ip + kx0), XP / 2);
        for (int e = threadIdx.x; e < LP * Y; e += kGenNT) {
            const int yy = e / LP, c = e % LP;
            const float4 v = z[c * Y + yy];
            __stcs(reinterpret_cast<float4*>(a.C + c_index_rt(Y, o, yy, kx0 + 2 * c, XP)), make_float4(v.x, v.z, v.y, v.w));
        }
    }
}

// k_pass_c_gen2: block per row y, two orientations at a time; thread t owns the pixels x = t + NT j
// and keeps their state over the batch: maxima in registers, FP64 sums of every value in TMEM
// (the doubles of pixel j in columns 2 j, sum, and 2 MAXP + 2 j, sum of squares; plain FP32 sums over
// 8 orientations, compensated between the eights, had 6 times the error of sums compensated at each,
// and their registers spilled: 64 orientations at 2700 x 2700 2.86 ms, 2.51 so).  An even width
// uses the c2r packing of k_pass_c (an X/2-point inverse FFT whose outputs hold pixel pairs);
// an odd width (the reference's factorisation can give one, e.g. 3^8) the full X-point
// inverse of the Hermitian extension, the imaginary part of the DC term ignored as FFTW's
// c2r does.  The best orientation goes to memory when a pixel's maximum changes.  256
// threads where two blocks fit an SM (up to 3,072 pixels), else 512.  Shared memory: 2 x L pairs
// | the twiddle table (TAB) | the next pair's rows of C (TAB) | histogram, TMEM slot (no static shared memory:
// the limit is on both together).
__host__ __device__ constexpr size_t gen_pass_c_smem(int X, int XP, int bins, bool tab) {
    return sizeof(float4) * (X % 2 ? 2 * X : X) + (tab ? sizeof(float2) * (X + X % 2 + 2 * XP) : 0) + 4 * ((size_t)bins + 1);
}
// pairs of rows fit shared memory (else k_pass_c_gen)
inline bool gen_pass_c_pairs(int X, int XP, int bins) { return gen_pass_c_smem(X, XP, bins, false) <= kBlockSharedLimit; }

template <bool ODD, int MAXP, int NT, bool TAB>
__global__ void __launch_bounds__(NT, NT == 512 ? 1 : 2)
k_pass_c_gen2(const __grid_constant__ BatchArgs a, int X, int Y, const __grid_constant__ GenPlan ph) {
    extern __shared__ __align__(16) float4 pbuf[];   // 2 x L, L = X/2 or X
    constexpr int WCOLS = 4 * MAXP;                                  // sum, sum of squares
    constexpr uint32_t TCOLS = WCOLS * (NT / 128);
    const int L = ODD ? X : X / 2, HC = X / 2 + 1, XP = a.XP, y = blockIdx.x, t = threadIdx.x, warp = t >> 5;
    float2* const tab = reinterpret_cast<float2*>(pbuf + 2 * L);
    float2* const rows = tab + X + X % 2;                            // two rows of XP
    unsigned int* const shist = reinterpret_cast<unsigned int*>(TAB ? rows + 2 * XP : tab);
    uint32_t* const tmem_slot = shist + a.hist_bins;
    if (warp == 0) {
        tmptx::tmem_alloc(tmem_slot, TCOLS);
        tmptx::tmem_relinquish();
    }
    for (int b = t; b < a.hist_bins; b += NT) shist[b] = 0u;
    tmfft::Twiddles tw = a.tw;
    if constexpr (TAB) {
        for (int e = t; e < X; e += NT) tab[e] = __ldg(a.tw.tab + e);
        tw.tab = tab;
    }
    const size_t rowC = c_index_rt(Y, 0, y, 0, XP), ostep = (size_t)Y * XP;
    const int R4 = 4 * c_tile_rows(Y);
    auto issue_rows = [&](int o) {   // 32-byte pieces of the tiles; an odd batch's last orientation twice
        for (int e = t; e < XP; e += NT) {
            const int h = e >= XP / 2 ? 1 : 0, c = e - h * (XP / 2);   // 16 bytes c of row h
            const float2* src = a.C + (o + h < a.nb ? o + h : o) * ostep + rowC + (size_t)(c >> 1) * R4 + 2 * (c & 1);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tmptx::smem_u32(rows + 2 * e)), "l"(src) : "memory");
        }
        tmptx::cp_async_commit();
    };
    if constexpr (TAB) issue_rows(0);
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    const uint32_t tcomp = *tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(WCOLS * (warp >> 2));
    float mip[MAXP];
    const size_t rowoff = (size_t)y * X;
    {
        float z[8];
#pragma unroll
        for (int j = 0; j < 8; j++) z[j] = 0.f;
#pragma unroll
        for (int j = 0; j < WCOLS; j += 8) tmptx::tmem_st8(tcomp + j, z);
        tmptx::tmem_wait_st();
    }
#pragma unroll
    for (int j = 0; j < MAXP; j++) {
        const int x = t + NT * j;
        mip[j] = x < X ? a.mip[rowoff + x] : FLT_MAX;   // pixels beyond the row never change
    }
    const float2 hmin2 = tmfft::both(a.hist_min), hinv2 = tmfft::both(a.hist_inv_step);
    for (int o = 0; o < a.nb; o += 2) {
        const bool two = o + 1 < a.nb;   // else the second orientation repeats the first
        const float2* c0 = TAB ? rows : a.C + o * ostep + rowC;
        const float2* c1 = TAB ? rows + XP : two ? c0 + ostep : c0;
        auto at = [&](int k) { return TAB ? (size_t)k : (size_t)(k >> 2) * R4 + (k & 3); };
        if constexpr (TAB) {
            tmptx::cp_async_wait<0>();
            __syncthreads();
        }
        if constexpr (ODD) {
            for (int k = t; k < X; k += NT) {
                const size_t e = at(k < HC ? k : X - k);
                float2 v = c0[e], w = c1[e];
                if (k >= HC) { v.y = -v.y; w.y = -w.y; }
                if (k == 0) v.y = w.y = 0.f;
                pbuf[k] = make_float4(v.x, w.x, v.y, w.y);
            }
        } else {
            for (int k = t; k < L; k += NT) {
                const float2 tk = tw.tab[k], wk = make_float2(tk.x, -tk.y);
                float2 z[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float2* row = h ? c1 : c0;
                    float2 hk = row[at(k)], hm = row[at(L - k)];
                    if (k == 0) { hk.y = 0.f; hm.y = 0.f; }
                    const float2 e = make_float2(hk.x + hm.x, hk.y - hm.y);
                    const float2 d = make_float2(hk.x - hm.x, hk.y + hm.y);
                    const float2 od = cmul(d, wk);
                    z[h] = make_float2(e.x - od.y, e.y + od.x);
                }
                pbuf[k] = make_float4(z[0].x, z[1].x, z[0].y, z[1].y);
            }
        }
        __syncthreads();
        if constexpr (TAB) {
            if (o + 2 < a.nb) issue_rows(o + 2);
        }
        // (real part pair, imaginary part pair) per element: an even width's pixel x is pair x
        const float2* zb = reinterpret_cast<const float2*>(pfft_gen<+1, NT, false>(pbuf, pbuf + L, 1, ph, 0, tw));
        const int g = (int)a.gidx0 + o;
#pragma unroll
        for (int j0 = 0; j0 < MAXP; j0 += 4) {   // 4 pixels of both sums at a time
            float sm[8], sq[8];
            tmptx::tmem_ld8(tcomp + 2 * j0, sm);
            tmptx::tmem_ld8(tcomp + 2 * MAXP + 2 * j0, sq);
            tmptx::tmem_wait_ld8x2(sm, sq);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int j = j0 + k, x = t + NT * j;
                float2 v = make_float2(0.f, 0.f);   // (beyond the row: added to sums that are never stored)
                if (x < X) {
                    v = zb[ODD ? 2 * x : x];
                    const float m = fmax3(mip[j], v.x, v.y);
                    if (m > mip[j]) a.best[rowoff + x] = v.x == m ? g : g + 1;
                    mip[j] = m;
                    const float2 bv = tmfft::mul2(tmfft::sub2(v, hmin2), hinv2);
                    const int b0 = __float2int_rz(bv.x), b1 = __float2int_rz(bv.y);
                    if ((unsigned)b0 < (unsigned)a.hist_bins) atomicAdd(&shist[b0], 1u);
                    if (two && (unsigned)b1 < (unsigned)a.hist_bins) atomicAdd(&shist[b1], 1u);
                    if (!two) v.y = 0.f;
                }
                double ds = f64_of(sm[2 * k], sm[2 * k + 1]), dq = f64_of(sq[2 * k], sq[2 * k + 1]);
                const double vx = v.x, vy = v.y;
                ds = (ds + vx) + vy;
                dq = fma(vy, vy, fma(vx, vx, dq));
                f64_to(ds, sm[2 * k], sm[2 * k + 1]);
                f64_to(dq, sq[2 * k], sq[2 * k + 1]);
            }
            tmptx::tmem_st8(tcomp + 2 * j0, sm);
            tmptx::tmem_st8(tcomp + 2 * MAXP + 2 * j0, sq);
        }
        tmptx::tmem_wait_st();
        __syncthreads();   // every output is read before the next pair's rows
    }
#pragma unroll
    for (int j0 = 0; j0 < MAXP; j0 += 4) {
        float sm[8], sq[8];
        tmptx::tmem_ld8(tcomp + 2 * j0, sm);
        tmptx::tmem_ld8(tcomp + 2 * MAXP + 2 * j0, sq);
        tmptx::tmem_wait_ld8x2(sm, sq);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int x = t + NT * (j0 + k);
            if (x < X) {
                a.sum[rowoff + x] += f64_of(sm[2 * k], sm[2 * k + 1]);
                a.sumsq[rowoff + x] += f64_of(sq[2 * k], sq[2 * k + 1]);
                a.mip[rowoff + x] = mip[j0 + k];
            }
        }
    }
    for (int b = t; b < a.hist_bins; b += NT) {
        const unsigned int cnt = shist[b];
        if (cnt) atomicAdd(a.hist + b, (unsigned long long)cnt);
    }
    tmptx::tmem_fence_before_sync();
    __syncthreads();
    tmptx::tmem_fence_after_sync();
    if (warp == 0) tmptx::tmem_dealloc(*tmem_slot, TCOLS);
}

// the row pass for a width X: kernel, threads and shared memory
struct GenRowPass {
    void (*kernel)(BatchArgs, int, int, GenPlan);
    int threads;
    size_t smem;
};
template <bool ODD>
inline GenRowPass gen_row_pass_pairs(int X, int XP, int bins) {
    const size_t full = gen_pass_c_smem(X, XP, bins, true);
    const bool tab = full <= kBlockSharedLimit;
    const size_t smem = tab ? full : gen_pass_c_smem(X, XP, bins, false);
    if (X <= 2048 && full <= 113 * 1024) return {k_pass_c_gen2<ODD, 8, 256, true>, 256, full};
    if (X <= 4096 && full <= 113 * 1024) return {k_pass_c_gen2<ODD, 16, 256, true>, 256, full};
    if (X <= 4096) return {tab ? k_pass_c_gen2<ODD, 8, 512, true> : k_pass_c_gen2<ODD, 8, 512, false>, 512, smem};
    return {tab ? k_pass_c_gen2<ODD, 16, 512, true> : k_pass_c_gen2<ODD, 16, 512, false>, 512, smem};
}
inline GenRowPass gen_row_pass(int X, int XP, int bins) {
    if (!gen_pass_c_pairs(X, XP, bins)) return {k_pass_c_gen, kGenNT, sizeof(float2) * 2 * X + 4 * (size_t)bins};   // long odd rows
    return X % 2 ? gen_row_pass_pairs<true>(X, XP, bins) : gen_row_pass_pairs<false>(X, XP, bins);
}
// the column pass for a height Y: kernel, columns per block and shared memory
struct GenColPass {
    void (*kernel)(BatchArgs, int, int, int, GenPlan);
    int columns;
    size_t smem;
};
inline GenColPass gen_col_pass(int T, int Y) {
    const GenColForm f = gen_col_form(T, Y);
    auto* kernel = f.pairs == 2 ? (f.tab ? k_pass_b_gen2<2, true, true> : k_pass_b_gen2<2, false, true>)
                   : f.pairs == 1 ? (f.tab ? k_pass_b_gen2<1, true, true>
                                     : f.staged ? k_pass_b_gen2<1, false, true> : k_pass_b_gen2<1, false, false>)
                                  : k_pass_b_gen;
    return {kernel, f.columns(), f.smem};
}
// orientations per block: up to 8, which share the table and overlap the loads, as long as there are two
// blocks per SM (352 x 1331, 9 orientations: 0.13 ms with 8, 0.06 one by one)
inline int gen_col_orientations(const GenColPass& p, int XP, int nb, int nsm) {
    if (p.columns == 1) return 1;
    const int ob = (int)((long long)(XP / p.columns) * nb / (2 * nsm));
    return ob < 1 ? 1 : ob > 8 ? 8 : ob;
}

// ---------------------------------------------------------------------------------------
// Whitening transforms of any size (the steps of tmw::k_w_rows / k_w_cols).
template <bool ODD>
__global__ void __launch_bounds__(kGenNT) k_w_rows_gen(const float* __restrict__ img, float2* spec, int X, float mean,
                                                       float vmin, float vmax, tmfft::Twiddles tw, GenPlan ph) {
    extern __shared__ float2 gbuf[];   // 2 x L (L = X/2, or X when X is odd)
    const int HC = X / 2 + 1, y = blockIdx.x;
    const float* src = img + (size_t)y * X;
    float2* row = spec + (size_t)y * HC;
    auto clean = [&](float v) { return (v > vmax || v < vmin) ? mean : v; };
    if constexpr (ODD) {
        // an odd width: the full X-point transform of the real row
        for (int x = threadIdx.x; x < X; x += kGenNT) gbuf[x] = make_float2(clean(src[x]), 0.f);
        __syncthreads();
        const float2* zb = fft_gen<-1>(gbuf, gbuf + X, X, 1, ph, tw);
        for (int k = threadIdx.x; k < HC; k += kGenNT) row[k] = zb[k];
    } else {
        const int H = X / 2;
        for (int n = threadIdx.x; n < H; n += kGenNT) gbuf[n] = make_float2(clean(src[2 * n]), clean(src[2 * n + 1]));
        __syncthreads();
        const float2* zb = fft_gen<-1>(gbuf, gbuf + H, H, 1, ph, tw);
        for (int k = threadIdx.x; k < H; k += kGenNT) {
            const float2 zk = zb[k];
            const float2 zm = zb[k == 0 ? 0 : H - k];
            const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
            const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
            const float2 wo = cmul(o, tw.template w<-1>(k, X));
            row[k] = make_float2(e.x + wo.x, e.y + wo.y);
            if (k == 0) row[H] = make_float2(e.x - o.x, e.y - o.y);
        }
    }
}

__global__ void __launch_bounds__(kGenNT) k_w_cols_gen(float2* spec, int X, int Y, tmfft::Twiddles tw, GenPlan py) {
    extern __shared__ float2 gbuf[];   // 2 x Y: one column
    const int HC = X / 2 + 1, col = blockIdx.x;
    for (int yy = threadIdx.x; yy < Y; yy += kGenNT) gbuf[yy] = spec[(size_t)yy * HC + col];
    __syncthreads();
    const float2* f = fft_gen<-1>(gbuf, gbuf + Y, Y, 1, py, tw);
    // SwapRealSpaceQuadrants as a float phase (Image::PhaseShift, image.cpp:9221-9265), zeroed DC
    const double kPi = 3.14159265359;
    const float sx = (float)(X / 2), sy = (float)(Y / 2);
    const float px = (float)(sx * (float)col * 2.0 * kPi / X);
    for (int yy = threadIdx.x; yy < Y; yy += kGenNT) {
        const float py_ = (float)(sy * (float)tmw::logical(yy, Y) * 2.0 * kPi / Y);
        const float th = -px - py_;
        const float cth = cosf(th), sth = sinf(th);
        float2 v = f[yy];
        v = make_float2(v.x * cth - v.y * sth, v.x * sth + v.y * cth);
        if (col == 0 && yy == 0) v = make_float2(0.f, 0.f);
        spec[(size_t)yy * HC + col] = v;
    }
}

}  // namespace tmk
