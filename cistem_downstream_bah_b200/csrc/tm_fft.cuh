// tm_fft.cuh -- register-resident Stockham FFT building blocks for sm_100a.
//
// An L-point complex transform is spread over P = L / R threads that each hold
// R values in registers.  On entry thread t holds x[t + P*r] (r = 0..R-1); on
// exit it holds X[t + P*r] (natural order, same stride).  Stages use radix R
// while R divides what is left of L, then the largest divisors of R that do
// (a thread then does R/Rs butterflies of radix Rs); between stages the values
// go through a padded shared-memory buffer (Stockham autosort: stage s reads
// element b + r*L/Rs and writes (b/Ns)*Ns*Rs + b%Ns + r*Ns, with Ns the
// product of the earlier radices).  Radices 2, 3, 4, 6, 8, 9, 12, 16, 18 and
// 24 are available, which covers the 2^a 3^b sizes the micrograph
// factorisation produces (match_template.cpp:527-583).
//
// Direction: DIR = -1 forward (exp(-2 pi i k n / L)), +1 inverse
// (unnormalised), matching the reference's FFTW conventions
// (src/core/image.cpp:5085-5113).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace tmfft {

// compile-time loop: f(std::integral_constant<int, i>) for i = 0..N-1
template <class F, int... Is>
__device__ __forceinline__ void sfor_impl(F&& f, std::integer_sequence<int, Is...>) {
    (f(std::integral_constant<int, Is>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F&& f) {
    sfor_impl(f, std::make_integer_sequence<int, N>{});
}

// exp(2 pi i k / n) evaluated at compile time (Taylor series after reducing
// the angle to [-pi, pi]); used for the constants inside the small DFTs
__host__ __device__ constexpr double ct_angle(int k, int n) {
    int m = ((k % n) + n) % n;
    if (2 * m > n) m -= n;
    return 2.0 * 3.14159265358979323846 * (double)m / (double)n;
}
__host__ __device__ constexpr double ct_sin(double x) {
    double term = x, sum = x;
    for (int i = 1; i < 30; i++) {
        term *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double ct_cos(double x) {
    double term = 1.0, sum = 1.0;
    for (int i = 1; i < 30; i++) {
        term *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
        sum += term;
    }
    return sum;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// multiply by -i (DIR=-1) or +i (DIR=+1)
template <int DIR>
__device__ __forceinline__ float2 mul_i(float2 a) {
    return DIR < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// padded shared-memory index: one spare float2 per 16
__device__ __forceinline__ int pad16(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int padded_len(int L) { return L + L / 16; }

// pad16(t + P*r) as a base plus a compile-time offset per r (0 <= t < P, P a
// multiple or a divisor of 16), so the 16 addresses need one register
template <int P>
__device__ __forceinline__ int rd_base(int t) { return (P % 16 == 0) ? t + (t >> 4) : t; }
template <int P>
__host__ __device__ constexpr int rd_off(int r) { return (P % 16 == 0) ? r * (P + P / 16) : P * r + ((P * r) >> 4); }

// pad16(idxD + r*Ns) for the Stockham write of a stage with one radix-R
// butterfly per thread (b = t): idxD = (t/Ns)*Ns*R + t%Ns; valid for Ns == 1
// with R dividing 16, and for Ns a multiple of 16
template <int R>
__device__ __forceinline__ int wr_base(int t, int Ns) {
    return Ns == 1 ? pad16(R * t) : pad16((t / Ns) * Ns * R + (t % Ns));
}
__host__ __device__ constexpr int wr_off(int r, int Ns) { return Ns == 1 ? r : r * (Ns + Ns / 16); }

template <int DIR>
__device__ __forceinline__ void dft2(float2& a, float2& b) {
    float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

template <int DIR>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
    float2 s02 = cadd(a0, a2), d02 = csub(a0, a2);
    float2 s13 = cadd(a1, a3), d13 = mul_i<DIR>(csub(a1, a3));
    a0 = cadd(s02, s13);
    a2 = csub(s02, s13);
    a1 = cadd(d02, d13);
    a3 = csub(d02, d13);
}

// radix-8 in natural order: r = 2*r1 + r2, q = q1 + 4*q2
template <int DIR>
__device__ __forceinline__ void dft8(float2* v) {
    const float h = 0.70710678118654752440f;
    dft4<DIR>(v[0], v[2], v[4], v[6]);   // r2 = 0 -> q1 at v[0,2,4,6]
    dft4<DIR>(v[1], v[3], v[5], v[7]);   // r2 = 1 -> q1 at v[1,3,5,7]
    // twiddle W8^(q1 * r2) on r2 = 1
    v[3] = make_float2((v[3].x + (DIR < 0 ? v[3].y : -v[3].y)) * h, (v[3].y + (DIR < 0 ? -v[3].x : v[3].x)) * h);
    v[5] = mul_i<DIR>(v[5]);
    v[7] = make_float2((-v[7].x + (DIR < 0 ? v[7].y : -v[7].y)) * h, (-v[7].y + (DIR < 0 ? -v[7].x : v[7].x)) * h);
    float2 o[8];
#pragma unroll
    for (int q1 = 0; q1 < 4; q1++) {
        float2 a = v[2 * q1], b = v[2 * q1 + 1];
        o[q1] = cadd(a, b);
        o[q1 + 4] = csub(a, b);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = o[i];
}

// radix-16 in natural order: r = 4*r1 + r2, q = q1 + 4*q2
template <int DIR>
__device__ __forceinline__ void dft16(float2* v) {
#pragma unroll
    for (int r2 = 0; r2 < 4; r2++) dft4<DIR>(v[r2], v[4 + r2], v[8 + r2], v[12 + r2]);
    // v[r2 + 4*q1] now holds u_{r2}[q1]; twiddle by W16^(q1*r2)
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
    const float sg = DIR < 0 ? -1.f : 1.f;
    // (q1, r2) = (1,1): W^1, (1,2): W^2, (1,3): W^3, (2,1): W^2, (2,2): W^4, (2,3): W^6, (3,1): W^3, (3,2): W^6, (3,3): W^9
    const float2 w1 = make_float2(c1, sg * s1), w2 = make_float2(h, sg * h), w3 = make_float2(s1, sg * c1);
    const float2 w6 = make_float2(-h, sg * h), w9 = make_float2(-c1, -sg * s1);
    v[5] = cmul(v[5], w1);
    v[6] = cmul(v[6], w2);
    v[7] = cmul(v[7], w3);
    v[9] = cmul(v[9], w2);
    v[10] = mul_i<DIR>(v[10]);
    v[11] = cmul(v[11], w6);
    v[13] = cmul(v[13], w3);
    v[14] = cmul(v[14], w6);
    v[15] = cmul(v[15], w9);
    float2 o[16];
#pragma unroll
    for (int q1 = 0; q1 < 4; q1++) {
        float2 a0 = v[4 * q1], a1 = v[4 * q1 + 1], a2 = v[4 * q1 + 2], a3 = v[4 * q1 + 3];
        dft4<DIR>(a0, a1, a2, a3);
        o[q1] = a0;
        o[q1 + 4] = a1;
        o[q1 + 8] = a2;
        o[q1 + 12] = a3;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = o[i];
}

template <int DIR>
__device__ __forceinline__ void dft3(float2& a, float2& b, float2& c) {
    // X1,2 = a - (b+c)/2 +- DIR i (sqrt(3)/2) (b-c)
    constexpr float h = 0.86602540378443864676f;
    const float2 sm = cadd(b, c), df = csub(b, c);
    const float2 m = make_float2(fmaf(-0.5f, sm.x, a.x), fmaf(-0.5f, sm.y, a.y));
    const float2 r = mul_i<DIR>(make_float2(h * df.x, h * df.y));
    a = cadd(a, sm);
    b = cadd(m, r);
    c = csub(m, r);
}

// x * W_R^K with W_R = exp(DIR 2 pi i / R), K a compile-time constant
template <int R, int K, int DIR>
__device__ __forceinline__ float2 twc(float2 x) {
    constexpr int k = ((K % R) + R) % R;
    if constexpr (k == 0) return x;
    else if constexpr (4 * k == R) return mul_i<DIR>(x);
    else if constexpr (2 * k == R) return make_float2(-x.x, -x.y);
    else if constexpr (4 * k == 3 * R) return mul_i<-DIR>(x);
    else {
        constexpr float c = (float)ct_cos(ct_angle(k, R));
        constexpr float sn = (float)(DIR * ct_sin(ct_angle(k, R)));
        return cmul(x, make_float2(c, sn));
    }
}

template <int RS, int DIR>
__device__ __forceinline__ void dft(float2* v);

// R1*R2-point DFT in natural order: r = R2*r1 + r2, q = q1 + R1*q2
// (R2 inner transforms of length R1, twiddles W_R^(r2 q1), R1 of length R2)
template <int R1, int R2, int DIR>
__device__ __forceinline__ void dft_pq(float2* v) {
    constexpr int R = R1 * R2;
    float2 u[R];
    sfor<R2>([&](auto r2c) {
        constexpr int r2 = decltype(r2c)::value;
        float2 t[R1];
#pragma unroll
        for (int r1 = 0; r1 < R1; r1++) t[r1] = v[R2 * r1 + r2];
        dft<R1, DIR>(t);
        sfor<R1>([&](auto q1c) {
            constexpr int q1 = decltype(q1c)::value;
            u[r2 * R1 + q1] = twc<R, r2 * q1, DIR>(t[q1]);
        });
    });
#pragma unroll
    for (int q1 = 0; q1 < R1; q1++) {
        float2 t[R2];
#pragma unroll
        for (int r2 = 0; r2 < R2; r2++) t[r2] = u[r2 * R1 + q1];
        dft<R2, DIR>(t);
#pragma unroll
        for (int q2 = 0; q2 < R2; q2++) v[q1 + R1 * q2] = t[q2];
    }
}

template <int RS, int DIR>
__device__ __forceinline__ void dft(float2* v) {
    if constexpr (RS == 16) dft16<DIR>(v);
    else if constexpr (RS == 8) dft8<DIR>(v);
    else if constexpr (RS == 4) dft4<DIR>(v[0], v[1], v[2], v[3]);
    else if constexpr (RS == 2) dft2<DIR>(v[0], v[1]);
    else if constexpr (RS == 3) dft3<DIR>(v[0], v[1], v[2]);
    else if constexpr (RS == 6) dft_pq<3, 2, DIR>(v);
    else if constexpr (RS == 9) dft_pq<3, 3, DIR>(v);
    else if constexpr (RS == 12) dft_pq<4, 3, DIR>(v);
    else if constexpr (RS == 18) dft_pq<9, 2, DIR>(v);
    else if constexpr (RS == 24) dft_pq<8, 3, DIR>(v);
    else static_assert(RS == 1, "unsupported radix");
}

// powers w^0 .. w^(n-1) by a shallow multiplication tree (depth <= 4)
template <int N>
__device__ __forceinline__ void powers(float2 w, float2* p) {
    p[0] = make_float2(1.f, 0.f);
    if constexpr (N > 1) p[1] = w;
    if constexpr (N > 2) p[2] = cmul(w, w);
    if constexpr (N > 3) p[3] = cmul(p[2], w);
    if constexpr (N > 4) {
        p[4] = cmul(p[2], p[2]);
#pragma unroll
        for (int i = 5; i < 8 && i < N; i++) p[i] = cmul(p[4], p[i - 4]);
    }
    if constexpr (N > 8) {
        p[8] = cmul(p[4], p[4]);
#pragma unroll
        for (int i = 9; i < 16 && i < N; i++) p[i] = cmul(p[8], p[i - 8]);
    }
}

// e[r] *= w^r for r = 1..RS-1.  The powers come from a shallow product tree
// (depth <= 4) computed next to their use, so few of them are live at once.
template <int RS>
__device__ __forceinline__ void apply_twiddles(float2* e, float2 w) {
    if constexpr (RS != 2 && RS != 4 && RS != 8 && RS != 16) {
        // w^k by a product tree of depth log2(RS)
        float2 p[RS];
        p[1] = w;
#pragma unroll
        for (int k = 2; k < RS; k++) p[k] = cmul(p[k >> 1], p[k - (k >> 1)]);
#pragma unroll
        for (int k = 1; k < RS; k++) e[k] = cmul(e[k], p[k]);
    } else if constexpr (RS == 2) {
        e[1] = cmul(e[1], w);
    } else if constexpr (RS == 4) {
        const float2 w2 = cmul(w, w);
        e[1] = cmul(e[1], w);
        e[2] = cmul(e[2], w2);
        e[3] = cmul(e[3], cmul(w2, w));
    } else {
        const float2 w2 = cmul(w, w);
        const float2 w3 = cmul(w2, w);
        const float2 w4 = cmul(w2, w2);
        e[1] = cmul(e[1], w);
        e[2] = cmul(e[2], w2);
        e[3] = cmul(e[3], w3);
        e[4] = cmul(e[4], w4);
        e[5] = cmul(e[5], cmul(w4, w));
        e[6] = cmul(e[6], cmul(w4, w2));
        e[7] = cmul(e[7], cmul(w4, w3));
        if constexpr (RS == 16) {
            const float2 w8 = cmul(w4, w4);
            e[8] = cmul(e[8], w8);
            e[9] = cmul(e[9], cmul(w8, w));
            e[10] = cmul(e[10], cmul(w8, w2));
            e[11] = cmul(e[11], cmul(w8, w3));
            const float2 w12 = cmul(w8, w4);
            e[12] = cmul(e[12], w12);
            e[13] = cmul(e[13], cmul(w12, w));
            e[14] = cmul(e[14], cmul(w12, w2));
            e[15] = cmul(e[15], cmul(w12, w3));
        }
    }
}

// Twiddle source: a table of W_LMAX^m = exp(-2 pi i m / LMAX), m = 0..LMAX-1;
// W_L^m = table[(m mod L) * (LMAX / L)] for every L that divides LMAX.
struct Twiddles {
    const float2* __restrict__ tab;
    int lmax;
    template <int DIR>
    __device__ __forceinline__ float2 w(int m, int L) const {
        const int mm = (L & (L - 1)) == 0 ? (m & (L - 1)) : (m % L);
        float2 t = __ldg(tab + (size_t)mm * (lmax / L));
        return DIR < 0 ? t : conjf2(t);
    }
};

// Radix plan of an L-point transform with R values per thread: R while R
// divides what is left, then the largest divisors of R that divide the rest.
// Butterflies are at most radix 24: with R = 32 every stage is a divisor
// (16, ...) and a thread does R / radix butterflies per stage.
constexpr int kMaxRadix = 24;
struct RadixSeq {
    int n;        // stages, -1 if L cannot be split this way
    int r[24];
};
__host__ __device__ constexpr RadixSeq radix_seq(int L, int R) {
    RadixSeq q{0, {}};
    int m = L;
    while (R <= kMaxRadix && m > 1 && m % R == 0 && q.n < 24) {
        q.r[q.n++] = R;
        m /= R;
    }
    while (m > 1) {
        int d = R > kMaxRadix ? kMaxRadix : R;
        while (d > 1 && !(R % d == 0 && m % d == 0)) d--;
        if (d <= 1 || q.n >= 24) return RadixSeq{-1, {}};
        q.r[q.n++] = d;
        m /= d;
    }
    return q;
}
__host__ __device__ constexpr bool plannable(int L, int R) { return L % R == 0 && radix_seq(L, R).n > 0; }

template <int L, int R>
struct Plan {
    static constexpr RadixSeq seq = radix_seq(L, R);
    static_assert(L % R == 0 && seq.n > 0, "transform length cannot be planned with this radix");
    static constexpr int stages = seq.n;
    static constexpr int P = L / R;
    __host__ __device__ static constexpr int radix(int s) { return seq.r[s]; }
    // product of the radices of the stages before s
    __host__ __device__ static constexpr int ns(int s) {
        int n = 1;
        for (int i = 0; i < s; i++) n *= seq.r[i];
        return n;
    }
};

// One cooperative FFT.  `sync` is a callable barrier over all threads that
// use `buf`.  buf has padded_len(L) float2 entries.  The first exchange begins
// with a barrier so that no thread still reads buf from a previous use; a
// caller whose threads have all passed a barrier since buf was last read
// passes FIRST_SYNC = false to skip it.
template <int L, int R, int DIR, bool FIRST_SYNC = true, class Sync>
__device__ __forceinline__ void fft(float2 (&v)[R], int t, float2* buf, const Twiddles& tw, Sync sync) {
    using PL = Plan<L, R>;
    constexpr int P = PL::P;
    sfor<PL::stages>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr int RS = PL::radix(s);
        constexpr int Ns = PL::ns(s);
        constexpr bool last = (s == PL::stages - 1);
        // twiddle base of this stage for the first butterfly, loaded before the
        // exchange so its latency hides behind the barrier and shared loads
        float2 w_first = make_float2(1.f, 0.f);
        if constexpr (s > 0) w_first = tw.template w<DIR>((t % Ns) * (L / (Ns * RS)), L);
        if constexpr (s > 0) {
            // load stage input: x[t + P*r]
            sync();
            if constexpr (P % 16 == 0 || 16 % P == 0) {
                const float2* rb = buf + rd_base<P>(t);
#pragma unroll
                for (int r = 0; r < R; r++) v[r] = rb[rd_off<P>(r)];
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) v[r] = buf[pad16(t + P * r)];
            }
        }
        // butterflies: thread does R/RS of them, b = t + P*u, elements v[u + r*(R/RS)]
#pragma unroll
        for (int u = 0; u < R / RS; u++) {
            const int b = t + P * u;
            float2 e[RS];
#pragma unroll
            for (int r = 0; r < RS; r++) e[r] = v[u + r * (R / RS)];
            if constexpr (s > 0) {
                const int jm = b % Ns;
                const float2 w = (u == 0) ? w_first : tw.template w<DIR>(jm * (L / (Ns * RS)), L);
                apply_twiddles<RS>(e, w);
            }
            dft<RS, DIR>(e);
            if constexpr (last) {
#pragma unroll
                for (int r = 0; r < RS; r++) v[u + r * (R / RS)] = e[r];
            } else {
                if (u == 0 && (FIRST_SYNC || s > 0)) sync();  // previous readers of buf are done
                // base + compile-time offsets equal pad16(idxD + r*Ns) when no
                // 16-element boundary falls inside a butterfly (Ns == 1, R | 16)
                // or every stride is a whole number of 16-blocks (16 | Ns)
                if constexpr (RS == R && ((Ns == 1 && 16 % R == 0) || Ns % 16 == 0)) {
                    float2* wb = buf + wr_base<R>(b, Ns);
#pragma unroll
                    for (int r = 0; r < RS; r++) wb[wr_off(r, Ns)] = e[r];
                } else {
                    const int idxD = (b / Ns) * Ns * RS + (b % Ns);
#pragma unroll
                    for (int r = 0; r < RS; r++) buf[pad16(idxD + r * Ns)] = e[r];
                }
            }
        }
    });
}

// ---- Two transforms at a time -------------------------------------------------------
// The same element of two independent transforms (two orientations, two columns), real
// parts and imaginary parts side by side, so that sm_100's two-wide FP32 instructions
// (add / sub / mul / fma .f32x2) do both with one issue slot; each half is rounded as its
// scalar form, so a transform gives the same bits in a pair as alone.  The FP32 pipe's
// lane rate is that of scalar code (122 FADD lanes per clock and SM measured, 126 two-wide):
// the gain is the issue slots, which bound the transforms of the search (60 % issue active
// with the FP32 pipe at a third to a half).
struct Pair {
    float2 re, im;
};
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tadd.rn.f32x2 s, p, q;\n\t"
        "mov.b64 {%0, %1}, s;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tsub.rn.f32x2 s, p, q;\n\t"
        "mov.b64 {%0, %1}, s;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tmul.rn.f32x2 s, p, q;\n\t"
        "mov.b64 {%0, %1}, s;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// a b + c
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 p, q, s, t;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tmov.b64 s, {%6, %7};\n\t"
        "fma.rn.f32x2 t, p, q, s;\n\tmov.b64 {%0, %1}, t;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ Pair padd(Pair a, Pair b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Pair psub(Pair a, Pair b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + (DIR i) b and a - (DIR i) b
template <int DIR>
__device__ __forceinline__ Pair padd_i(Pair a, Pair b) {
    if constexpr (DIR < 0) return {add2(a.re, b.im), sub2(a.im, b.re)};
    else return {sub2(a.re, b.im), add2(a.im, b.re)};
}
template <int DIR>
__device__ __forceinline__ Pair psub_i(Pair a, Pair b) { return padd_i<-DIR>(a, b); }
// a w for one factor, and a w for a factor of each half (cmul per half: the factor's parts
// would have to be doubled into register pairs for the two-wide form)
__device__ __forceinline__ Pair pmul(Pair a, float2 w) {
    const float2 x = cmul(make_float2(a.re.x, a.im.x), w), y = cmul(make_float2(a.re.y, a.im.y), w);
    return {make_float2(x.x, y.x), make_float2(x.y, y.y)};
}

// a conj(b) with the roles of cmul_conj, b per half
__device__ __forceinline__ Pair pmul_conj(float2 ax, float2 ay, Pair b) {   // a = (ax.x, ay.x), (ax.y, ay.y)
    const float2 x = cmul_conj(make_float2(ax.x, ay.x), make_float2(b.re.x, b.im.x));
    const float2 y = cmul_conj(make_float2(ax.y, ay.y), make_float2(b.re.y, b.im.y));
    return {make_float2(x.x, y.x), make_float2(x.y, y.y)};
}
// a (c + i s) for a compile-time factor, two-wide, rounded as cmul.  The factor's parts are
// immediates inside the instruction block: as operands they are kept in register pairs over
// the surrounding loops, and the kernels with many radices then spill them (the row pass at
// 2700 pixels ran 115 M local loads beside 49 M shared ones).
template <uint32_t C, uint32_t S, uint32_t NS>
__device__ __forceinline__ Pair pmulc_bits(Pair a) {
    Pair r;
    asm("{\n\t.reg .b64 x, y, c, s, n, t, u;\n\tmov.b64 x, {%4, %5};\n\tmov.b64 y, {%6, %7};\n\t"
        "mov.b64 c, {%8, %8};\n\tmov.b64 s, {%9, %9};\n\tmov.b64 n, {%10, %10};\n\t"
        "mul.rn.f32x2 t, y, n;\n\tfma.rn.f32x2 t, x, c, t;\n\tmul.rn.f32x2 u, y, c;\n\tfma.rn.f32x2 u, x, s, u;\n\t"
        "mov.b64 {%0, %1}, t;\n\tmov.b64 {%2, %3}, u;\n\t}"
        : "=f"(r.re.x), "=f"(r.re.y), "=f"(r.im.x), "=f"(r.im.y)
        : "f"(a.re.x), "f"(a.re.y), "f"(a.im.x), "f"(a.im.y), "n"(C), "n"(S), "n"(NS));
    return r;
}

// ROT2: a2 still lacks a factor DIR i
template <int DIR, bool ROT2 = false>
__device__ __forceinline__ void pdft4(Pair& a0, Pair& a1, Pair& a2, Pair& a3) {
    const Pair s02 = ROT2 ? padd_i<DIR>(a0, a2) : padd(a0, a2), d02 = ROT2 ? psub_i<DIR>(a0, a2) : psub(a0, a2);
    const Pair s13 = padd(a1, a3), d13 = psub(a1, a3);
    a0 = padd(s02, s13);
    a2 = psub(s02, s13);
    a1 = padd_i<DIR>(d02, d13);
    a3 = psub_i<DIR>(d02, d13);
}

// dft8 of both halves
template <int DIR>
__device__ __forceinline__ void pdft8(Pair* v) {
    constexpr float h = 0.70710678118654752440f;
    pdft4<DIR>(v[0], v[2], v[4], v[6]);
    pdft4<DIR>(v[1], v[3], v[5], v[7]);
    // v[3] W8 = h (v + DIR i v), v[7] W8^3 = -h (v - DIR i v): the factor h inside the last additions
    const Pair t3 = padd_i<DIR>(v[3], v[3]), t7 = psub_i<DIR>(v[7], v[7]);
    const Pair a0 = v[0], a1 = v[2], a2 = v[4], a3 = v[6], b0 = v[1], b2 = v[5];
    v[0] = padd(a0, b0);
    v[4] = psub(a0, b0);
    v[1] = {fma2(t3.re, both(h), a1.re), fma2(t3.im, both(h), a1.im)};
    v[5] = {fma2(t3.re, both(-h), a1.re), fma2(t3.im, both(-h), a1.im)};
    v[2] = padd_i<DIR>(a2, b2);
    v[6] = psub_i<DIR>(a2, b2);
    v[3] = {fma2(t7.re, both(-h), a3.re), fma2(t7.im, both(-h), a3.im)};
    v[7] = {fma2(t7.re, both(h), a3.re), fma2(t7.im, both(h), a3.im)};
}

// x W_R^K of both halves, as twc
template <int R, int K, int DIR>
__device__ __forceinline__ Pair ptwc(Pair x) {
    constexpr int k = ((K % R) + R) % R;
    if constexpr (k == 0) return x;
    else if constexpr (2 * k == R) return {make_float2(-x.re.x, -x.re.y), make_float2(-x.im.x, -x.im.y)};
    else if constexpr (4 * k == R || 4 * k == 3 * R) {
        constexpr bool plus = (4 * k == R) == (DIR > 0);   // times +i, else -i
        return plus ? Pair{make_float2(-x.im.x, -x.im.y), x.re} : Pair{x.im, make_float2(-x.re.x, -x.re.y)};
    } else {
        constexpr float c = (float)ct_cos(ct_angle(k, R));
        constexpr float sn = (float)(DIR * ct_sin(ct_angle(k, R)));
        return pmulc_bits<__builtin_bit_cast(uint32_t, c), __builtin_bit_cast(uint32_t, sn), __builtin_bit_cast(uint32_t, -sn)>(x);
    }
}

// The 16-point DFT of both halves (rounded as dft16) as its two levels of four 4-point
// transforms with the constants between, so that a caller can put loads, factors and stores
// between the groups of four: level 1 takes x[r2], x[4 + r2], x[8 + r2], x[12 + r2], level 2 leaves
// X[q1], X[q1 + 4], X[q1 + 8], X[q1 + 12].  pdft16_mid takes element (q1, r2) of level 1's results
// at v[4 q1 + r2] or at v[4 r2 + q1] (its factors are symmetric); the factor DIR i of (2, 2),
// v[10], is left to level 2 of q1 = 2 (pdft4's ROT2).
template <int DIR>
__device__ __forceinline__ void pdft16_mid(Pair* v) {
    v[5] = ptwc<16, 1, DIR>(v[5]);
    v[6] = ptwc<16, 2, DIR>(v[6]);
    v[7] = ptwc<16, 3, DIR>(v[7]);
    v[9] = ptwc<16, 2, DIR>(v[9]);
    v[11] = ptwc<16, 6, DIR>(v[11]);
    v[13] = ptwc<16, 3, DIR>(v[13]);
    v[14] = ptwc<16, 6, DIR>(v[14]);
    v[15] = ptwc<16, 9, DIR>(v[15]);
}

// dft3 of both halves (the factor h of its difference inside the last additions)
template <int DIR>
__device__ __forceinline__ void pdft3(Pair& a, Pair& b, Pair& c) {
    constexpr float h = 0.86602540378443864676f, hd = DIR < 0 ? h : -h;
    const Pair sm = padd(b, c), df = psub(b, c);
    const Pair m = {fma2(both(-0.5f), sm.re, a.re), fma2(both(-0.5f), sm.im, a.im)};
    a = padd(a, sm);
    b = {fma2(both(hd), df.im, m.re), fma2(both(-hd), df.re, m.im)};
    c = {fma2(both(-hd), df.im, m.re), fma2(both(hd), df.re, m.im)};
}

// dft9 of both halves, as dft_pq<3, 3>
template <int DIR>
__device__ __forceinline__ void pdft9(Pair* v) {
    sfor<3>([&](auto rc) {
        constexpr int r2 = decltype(rc)::value;
        pdft3<DIR>(v[r2], v[3 + r2], v[6 + r2]);   // -> q1 at v[3 q1 + r2]
        v[3 + r2] = ptwc<9, r2, DIR>(v[3 + r2]);
        v[6 + r2] = ptwc<9, 2 * r2, DIR>(v[6 + r2]);
    });
    Pair o[9];
#pragma unroll
    for (int q1 = 0; q1 < 3; q1++) {
        pdft3<DIR>(v[3 * q1], v[3 * q1 + 1], v[3 * q1 + 2]);
#pragma unroll
        for (int q2 = 0; q2 < 3; q2++) o[q1 + 3 * q2] = v[3 * q1 + q2];
    }
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = o[i];
}

template <int RS, int DIR>
__device__ __forceinline__ void pdft(Pair* v);

// dft_pq of both halves
template <int R1, int R2, int DIR>
__device__ __forceinline__ void pdft_pq(Pair* v) {
    constexpr int R = R1 * R2;
    Pair u[R];
    sfor<R2>([&](auto r2c) {
        constexpr int r2 = decltype(r2c)::value;
        Pair t[R1];
#pragma unroll
        for (int r1 = 0; r1 < R1; r1++) t[r1] = v[R2 * r1 + r2];
        pdft<R1, DIR>(t);
        sfor<R1>([&](auto q1c) {
            constexpr int q1 = decltype(q1c)::value;
            u[r2 * R1 + q1] = ptwc<R, r2 * q1, DIR>(t[q1]);
        });
    });
#pragma unroll
    for (int q1 = 0; q1 < R1; q1++) {
        Pair t[R2];
#pragma unroll
        for (int r2 = 0; r2 < R2; r2++) t[r2] = u[r2 * R1 + q1];
        pdft<R2, DIR>(t);
#pragma unroll
        for (int q2 = 0; q2 < R2; q2++) v[q1 + R1 * q2] = t[q2];
    }
}

// R-point DFT of prime length as R^2 multiplications by compile-time constants
template <int R, int DIR>
__device__ __forceinline__ void pdft_prime(Pair* v) {
    Pair o[R];
    sfor<R>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        Pair acc = v[0];
        sfor<R - 1>([&](auto ic) {
            constexpr int i = decltype(ic)::value + 1;
            acc = padd(acc, ptwc<R, (i * k) % R, DIR>(v[i]));
        });
        o[k] = acc;
    });
#pragma unroll
    for (int i = 0; i < R; i++) v[i] = o[i];
}

template <int DIR>
__device__ __forceinline__ void pdft16(Pair* v) {
#pragma unroll
    for (int g = 0; g < 4; g++) pdft4<DIR>(v[g], v[4 + g], v[8 + g], v[12 + g]);
    pdft16_mid<DIR>(v);
    Pair o[16];
    sfor<4>([&](auto gc) {
        constexpr int g = decltype(gc)::value;
        pdft4<DIR, g == 2>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
#pragma unroll
        for (int k = 0; k < 4; k++) o[g + 4 * k] = v[4 * g + k];
    });
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = o[i];
}

template <int RS, int DIR>
__device__ __forceinline__ void pdft(Pair* v) {
    if constexpr (RS == 16) pdft16<DIR>(v);
    else if constexpr (RS == 8) pdft8<DIR>(v);
    else if constexpr (RS == 4) pdft4<DIR>(v[0], v[1], v[2], v[3]);
    else if constexpr (RS == 9) pdft9<DIR>(v);
    else if constexpr (RS == 3) pdft3<DIR>(v[0], v[1], v[2]);
    else if constexpr (RS == 2) {
        const Pair a = v[0], b = v[1];
        v[0] = padd(a, b);
        v[1] = psub(a, b);
    } else if constexpr (RS == 6) pdft_pq<3, 2, DIR>(v);
    else if constexpr (RS == 12) pdft_pq<4, 3, DIR>(v);
    else if constexpr (RS == 18) pdft_pq<9, 2, DIR>(v);
    else {
        static_assert(RS == 5 || RS == 7 || RS == 11 || RS == 13, "unsupported radix");
        pdft_prime<RS, DIR>(v);
    }
}

// apply_twiddles on both halves, which share the powers of w
template <int RS>
__device__ __forceinline__ void papply_twiddles(Pair* e, float2 w) {
    if constexpr (RS != 2 && RS != 4 && RS != 8 && RS != 16) {
        float2 p[RS];
        p[1] = w;
#pragma unroll
        for (int k = 2; k < RS; k++) p[k] = cmul(p[k >> 1], p[k - (k >> 1)]);
#pragma unroll
        for (int k = 1; k < RS; k++) e[k] = pmul(e[k], p[k]);
    } else {
        float2 p[RS];   // the powers of apply_twiddles: w^k = w^h w^(k - h), h the largest power of 2 below k
        p[1] = w;
#pragma unroll
        for (int k = 2; k < RS; k++) {
            const int h = k > 8 ? 8 : k > 4 ? 4 : k > 2 ? 2 : 1;
            p[k] = k > 12 ? cmul(p[12], p[k - 12]) : cmul(p[h], p[k - h]);
        }
#pragma unroll
        for (int k = 1; k < RS; k++) e[k] = pmul(e[k], p[k]);
    }
}

// The base twiddles of a plan's stages in one array: stage s (from 1) takes Ns entries, entry k being
// W_L^(k L / (Ns RS)), so that neighbouring threads read neighbouring entries.
template <int L, int R>
__host__ __device__ constexpr int stage_table_len(int s = Plan<L, R>::stages) {
    int n = 0;
    for (int i = 1; i < s; i++) n += Plan<L, R>::ns(i);
    return n;
}
template <int L, int R>
__device__ __forceinline__ void fill_stage_table(float2* dst, const Twiddles& tw, int tid, int nthreads) {
    using PL = Plan<L, R>;
    sfor<PL::stages>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        if constexpr (s > 0) {
            constexpr int Ns = PL::ns(s);
            for (int k = tid; k < Ns; k += nthreads) dst[stage_table_len<L, R>(s) + k] = tw.template w<-1>(k * (L / (Ns * PL::radix(s))), L);
        }
    });
}

// Place of element i with one spare element per D (0: none).  An address (t + P r or idxD + r Ns) is a
// base plus a compile-time offset per r where no multiple of D falls inside a step.
template <int D>
__host__ __device__ constexpr int pad_at(int i) { return D ? i + i / (D ? D : 1) : i; }

// fft on both halves.  Element i of a pair is buf[pad_at<D>(i) * WP]: WP pairs side by side, 16
// bytes each, so that 8 lanes (WP pairs of 8 / WP neighbouring t) access 128 different bytes.
// tab: the plan's stage table in shared memory.  act: this thread's outputs are wanted in buf
// (padding lanes of a block pass false).
template <int L, int R, int DIR, int WP, int D, bool FIRST_SYNC = true, class Sync>
__device__ __forceinline__ void pfft(Pair (&v)[R], int t, float4* buf, const float2* tab, bool act, Sync sync) {
    using PL = Plan<L, R>;
    constexpr int P = PL::P;
    sfor<PL::stages>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr int RS = PL::radix(s);
        constexpr int Ns = PL::ns(s);
        constexpr bool last = (s == PL::stages - 1);
        if constexpr (s > 0) {
            sync();
            auto get = [&](Pair& p, const float4* at) {
                const float4 f = *at;
                p = {make_float2(f.x, f.y), make_float2(f.z, f.w)};
            };
            if constexpr (D == 0 || P % (D ? D : 1) == 0 || D % P == 0) {
                const float4* rb = buf + pad_at<D % P == 0 && P < D ? 0 : D>(t) * WP;   // (t below P below D: no spare element)
#pragma unroll
                for (int r = 0; r < R; r++) get(v[r], rb + pad_at<D>(P * r) * WP);
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) get(v[r], buf + pad_at<D>(t + P * r) * WP);
            }
        }
#pragma unroll
        for (int u = 0; u < R / RS; u++) {
            const int b = t + P * u;
            Pair e[RS];
#pragma unroll
            for (int r = 0; r < RS; r++) e[r] = v[u + r * (R / RS)];
            if constexpr (s > 0) {
                const float2 w = tab[stage_table_len<L, R>(s) + (last ? b : b % Ns)];   // b < L / RS, which is the last Ns
                papply_twiddles<RS>(e, DIR < 0 ? w : conjf2(w));
            }
            pdft<RS, DIR>(e);
            if constexpr (last) {
#pragma unroll
                for (int r = 0; r < RS; r++) v[u + r * (R / RS)] = e[r];
            } else {
                if (u == 0 && (FIRST_SYNC || s > 0)) sync();  // previous readers of buf are done
                auto put = [](float4* at, Pair p) { *at = make_float4(p.re.x, p.re.y, p.im.x, p.im.y); };
                if (act) {
                    const int idxD = (b / Ns) * Ns * RS + (b % Ns);
                    if constexpr (D == 0 || Ns % (D ? D : 1) == 0 || (Ns == 1 && D % RS == 0)) {
                        float4* wb = buf + pad_at<D>(idxD) * WP;
#pragma unroll
                        for (int r = 0; r < RS; r++) put(wb + pad_at<D>(r * Ns) * WP, e[r]);
                    } else {
#pragma unroll
                        for (int r = 0; r < RS; r++) put(buf + pad_at<D>(idxD + r * Ns) * WP, e[r]);
                    }
                }
            }
        }
    });
}

}  // namespace tmfft
