// Device FFT building blocks for the docking pipeline (sm_100a, FP32 complex).
//
// Every line transform is a two-level ("four-step") Cooley-Tukey split
// N = R1 * R2 done by a group of threads over a shared-memory line:
//   phase 1: item t in [0,R2) loads x[t + R2*m] (m < R1), does an R1-point DFT
//            in registers, multiplies by W_N^(t*k1) and stores back to the same
//            R1 positions (k1*R2 + t): it reads and writes one position set, so
//            phase 1 needs no barrier between items;
//   phase 2: item u in [0,R1) loads y[u*R2 + n2] (n2 < R2), does an R2-point
//            DFT and yields X[u + R1*k2] in registers for the caller to store.
// Lanes of a warp always index different lines and warps index the butterfly
// item, so the inter-phase twiddle index t*k1 is warp-uniform (broadcast load).
//
// Zero padding: docking grids carry data only in the middle half of each axis
// ([floor(N/4), floor(N/4) + N/2)), so half the inputs of a first pass are
// known zeros (padded_inputs).  The skipped inputs are -0: x + (-0) = x and
// (-0) - x = -x hold for every x, so the compiler drops those adds from the
// codelet (with +0 it may not: +0 + -0 is +0); the outputs are the same bits
// (B200, N = 128: identical records).
//
// The small DFTs are generated at compile time: prime radices 2, 3, 5, 7, 11
// are direct DFTs (radix 4 is a butterfly); composite radices recurse through
// the same four-step split with constant twiddles folded by the compiler.
// Trigonometric constants come from a constexpr Taylor series in double
// (reduced to |x| <= pi), rounded once to float.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>
#include <utility>

namespace mdb {

// ------------------------------------------------------------------ constexpr trig
namespace ct {
constexpr double kPi = 3.14159265358979323846264338327950288;
__host__ __device__ constexpr double sin_series(double x) {
    double term = x, sum = x;
    for (int n = 1; n < 24; ++n) {
        term *= -x * x / ((2.0 * n) * (2.0 * n + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double cos_series(double x) {
    double term = 1.0, sum = 1.0;
    for (int n = 1; n < 24; ++n) {
        term *= -x * x / ((2.0 * n - 1.0) * (2.0 * n));
        sum += term;
    }
    return sum;
}
// angle 2*pi*k/n reduced to (-pi, pi]
__host__ __device__ constexpr double red_angle(long k, long n) {
    long m = ((k % n) + n) % n;
    if (2 * m > n) m -= n;
    return 2.0 * kPi * (double)m / (double)n;
}
__host__ __device__ constexpr float cos2pi(long k, long n) { return (float)cos_series(red_angle(k, n)); }
__host__ __device__ constexpr float sin2pi(long k, long n) { return (float)sin_series(red_angle(k, n)); }

__host__ __device__ constexpr int first_factor(int r) {
    if (r % 4 == 0 && r != 4) return 4;
    for (int p = 2; p * p <= r; ++p)
        if (r % p == 0) return p;
    return r;
}
}  // namespace ct

// ------------------------------------------------------------------ complex helpers
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
__device__ __forceinline__ float2 cmulconj(float2 a, float2 b) {
    return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

template <int I, int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

// a * exp(S * 2 pi i e / R) for a compile-time twiddle: quarter turns are
// swaps and sign flips, odd eighth turns one add pair and a scale by sqrt(1/2),
// the rest a complex multiply by constexpr cos / sin.
template <long E, int R, int S>
__device__ __forceinline__ float2 tw_mul(float2 a) {
    constexpr long e = ((E % R) + R) % R;
    if constexpr (e == 0) {
        return a;
    } else if constexpr ((4 * e) % R == 0) {
        constexpr int q = (int)(4 * e / R);   // 1, 2 or 3 quarter turns
        if constexpr (q == 2) return make_float2(-a.x, -a.y);
        else if constexpr ((q == 1) == (S > 0)) return make_float2(-a.y, a.x);   // times +i
        else return make_float2(a.y, -a.x);                                      // times -i
    } else if constexpr ((8 * e) % R == 0) {
        constexpr int o = (int)(8 * e / R);   // 1, 3, 5 or 7 eighth turns
        constexpr float h = 0.70710678118654752f;
        constexpr float c = (o == 1 || o == 7) ? 1.f : -1.f;                  // sign of cos
        constexpr float sn = (float)S * ((o == 1 || o == 3) ? 1.f : -1.f);    // sign of S sin
        // (a.x c - a.y s, a.x s + a.y c) with |c| = |s| = sqrt(1/2)
        const float re = c > 0 ? (sn > 0 ? a.x - a.y : a.x + a.y) : (sn > 0 ? -a.x - a.y : a.y - a.x);
        const float im = sn > 0 ? (c > 0 ? a.x + a.y : a.x - a.y) : (c > 0 ? a.y - a.x : -a.x - a.y);
        return make_float2(re * h, im * h);
    } else {
        constexpr float c = ct::cos2pi(e, R);
        constexpr float s = (float)S * ct::sin2pi(e, R);
        return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

// ------------------------------------------------------------------ small DFTs
// In-place R-point DFT of v[0..R) with exponent sign S (-1 forward, +1 inverse):
//   v[k] <- sum_n v[n] * exp(S * 2*pi*i*n*k/R)
template <int R, int S, int F = ct::first_factor(R)>
struct Dft;

template <int S>
struct Dft<1, S, 1> {
    __device__ __forceinline__ static void run(float2 *) {}
};

template <int S>
struct Dft<2, S, 2> {
    __device__ __forceinline__ static void run(float2 *v) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <int S>
struct Dft<4, S, 2> {
    __device__ __forceinline__ static void run(float2 *v) {
        const float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
        const float2 t2 = cadd(v[1], v[3]), d = csub(v[1], v[3]);
        // d * (S * i)
        const float2 t3 = (S < 0) ? make_float2(d.y, -d.x) : make_float2(-d.y, d.x);
        v[0] = cadd(t0, t2);
        v[2] = csub(t0, t2);
        v[1] = cadd(t1, t3);
        v[3] = csub(t1, t3);
    }
};

// Prime radix: direct DFT with symmetric pairing of n and R-n.
template <int R, int S>
struct Dft<R, S, R> {
    static_assert(R % 2 == 1 && R >= 3, "odd prime radix");
    __device__ __forceinline__ static void run(float2 *v) {
        constexpr int H = (R - 1) / 2;
        float2 sp[H], sm[H];
        static_for<1, H + 1>([&](auto n_) {
            constexpr int n = decltype(n_)::value;
            sp[n - 1] = cadd(v[n], v[R - n]);
            sm[n - 1] = csub(v[n], v[R - n]);
        });
        float2 out[R];
        float2 dc = v[0];
        static_for<0, H>([&](auto n) { dc = cadd(dc, sp[n]); });
        out[0] = dc;
        static_for<1, H + 1>([&](auto k_) {
            constexpr int k = decltype(k_)::value;
            float2 re = v[0];   // real-cosine part accumulation
            float2 im = make_float2(0.f, 0.f);
            static_for<1, H + 1>([&](auto n_) {
                constexpr int n = decltype(n_)::value;
                constexpr float c = ct::cos2pi((long)n * k, R);
                constexpr float s = (float)S * ct::sin2pi((long)n * k, R);
                re.x += c * sp[n - 1].x;
                re.y += c * sp[n - 1].y;
                // i * s * sm
                im.x += -s * sm[n - 1].y;
                im.y += s * sm[n - 1].x;
            });
            out[k] = cadd(re, im);
            out[R - k] = csub(re, im);
        });
        static_for<0, R>([&](auto k) { v[k] = out[k]; });
    }
};

// Composite radix: R = A * B, input n = B*n1 + n2, output k = k1 + A*k2.
template <int R, int S, int A>
struct Dft {
    static constexpr int B = R / A;
    __device__ __forceinline__ static void run(float2 *v) {
        float2 tmp[R];
        static_for<0, B>([&](auto n2_) {
            constexpr int n2 = decltype(n2_)::value;
            float2 a[A];
            static_for<0, A>([&](auto n1_) {
                constexpr int n1 = decltype(n1_)::value;
                a[n1] = v[B * n1 + n2];
            });
            Dft<A, S>::run(a);
            static_for<0, A>([&](auto k1_) {
                constexpr int k1 = decltype(k1_)::value;
                tmp[k1 * B + n2] = tw_mul<(long)n2 * k1, R, S>(a[k1]);
            });
        });
        static_for<0, A>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            float2 b[B];
            static_for<0, B>([&](auto n2_) { b[decltype(n2_)::value] = tmp[k1 * B + decltype(n2_)::value]; });
            Dft<B, S>::run(b);
            static_for<0, B>([&](auto k2_) { v[k1 + A * decltype(k2_)::value] = b[decltype(k2_)::value]; });
        });
    }
};

// ------------------------------------------------------------------ line plans
// Supported FFT edge lengths and their split N = R1 * R2 (R1 % 4 == 0 where N
// allows it: no input of the first pass is then part padding, part data).
template <int N>
struct Plan;
#define MDB_PLAN(N_, R1_, R2_)                                  \
    template <>                                                  \
    struct Plan<N_> {                                            \
        static constexpr int R1 = R1_;                           \
        static constexpr int R2 = R2_;                           \
        static_assert(R1_ * R2_ == N_, "plan");                  \
    };
MDB_PLAN(16, 4, 4)
MDB_PLAN(21, 3, 7)
MDB_PLAN(25, 5, 5)
MDB_PLAN(27, 3, 9)
MDB_PLAN(18, 6, 3)
MDB_PLAN(20, 4, 5)
MDB_PLAN(22, 2, 11)
MDB_PLAN(24, 4, 6)
MDB_PLAN(28, 4, 7)
MDB_PLAN(30, 6, 5)
MDB_PLAN(32, 4, 8)
MDB_PLAN(33, 3, 11)
MDB_PLAN(35, 5, 7)
MDB_PLAN(36, 4, 9)
MDB_PLAN(40, 8, 5)
MDB_PLAN(42, 6, 7)
MDB_PLAN(44, 4, 11)
MDB_PLAN(45, 5, 9)
MDB_PLAN(48, 4, 12)
MDB_PLAN(49, 7, 7)
MDB_PLAN(50, 10, 5)
MDB_PLAN(54, 6, 9)
MDB_PLAN(55, 5, 11)
MDB_PLAN(56, 8, 7)
MDB_PLAN(60, 4, 15)
MDB_PLAN(63, 7, 9)
MDB_PLAN(64, 8, 8)
MDB_PLAN(66, 6, 11)
MDB_PLAN(70, 10, 7)
MDB_PLAN(72, 8, 9)
MDB_PLAN(75, 5, 15)
MDB_PLAN(77, 7, 11)
MDB_PLAN(81, 9, 9)
MDB_PLAN(80, 8, 10)
MDB_PLAN(84, 12, 7)
MDB_PLAN(88, 8, 11)
MDB_PLAN(90, 10, 9)
MDB_PLAN(96, 8, 12)
MDB_PLAN(98, 14, 7)
MDB_PLAN(99, 9, 11)
MDB_PLAN(100, 20, 5)
MDB_PLAN(105, 7, 15)
MDB_PLAN(108, 12, 9)
MDB_PLAN(110, 10, 11)
MDB_PLAN(112, 8, 14)
MDB_PLAN(120, 8, 15)
MDB_PLAN(126, 14, 9)
MDB_PLAN(128, 8, 16)
MDB_PLAN(132, 12, 11)
MDB_PLAN(140, 20, 7)
MDB_PLAN(144, 16, 9)
MDB_PLAN(150, 10, 15)
MDB_PLAN(154, 14, 11)
MDB_PLAN(160, 16, 10)
MDB_PLAN(162, 18, 9)
MDB_PLAN(168, 12, 14)
MDB_PLAN(176, 16, 11)
MDB_PLAN(180, 12, 15)
MDB_PLAN(192, 12, 16)
MDB_PLAN(196, 14, 14)
MDB_PLAN(198, 18, 11)
MDB_PLAN(200, 20, 10)
MDB_PLAN(210, 14, 15)
MDB_PLAN(216, 12, 18)
MDB_PLAN(220, 20, 11)
MDB_PLAN(224, 16, 14)
// half edges of the staged sizes' complex-to-real pass
MDB_PLAN(121, 11, 11)
MDB_PLAN(125, 5, 25)
MDB_PLAN(135, 5, 27)
MDB_PLAN(147, 7, 21)
// edges above 224 (ng1 of the default grid table up to 160): staged kernels
MDB_PLAN(240, 16, 15)
MDB_PLAN(242, 22, 11)
MDB_PLAN(250, 10, 25)
MDB_PLAN(252, 12, 21)
MDB_PLAN(256, 16, 16)
MDB_PLAN(264, 12, 22)
MDB_PLAN(270, 10, 27)
MDB_PLAN(280, 20, 14)
MDB_PLAN(288, 16, 18)
MDB_PLAN(294, 14, 21)
MDB_PLAN(300, 20, 15)
MDB_PLAN(308, 28, 11)
MDB_PLAN(320, 16, 20)
MDB_PLAN(400, 20, 20)
// edges of the default grid table with ng1 in (160, 220] (staged kernels)
MDB_PLAN(324, 12, 27)
MDB_PLAN(330, 22, 15)
MDB_PLAN(336, 16, 21)
MDB_PLAN(350, 14, 25)
MDB_PLAN(352, 16, 22)
MDB_PLAN(360, 20, 18)
MDB_PLAN(378, 18, 21)
MDB_PLAN(384, 16, 24)
MDB_PLAN(392, 28, 14)
MDB_PLAN(396, 12, 33)
MDB_PLAN(420, 20, 21)
MDB_PLAN(432, 24, 18)
MDB_PLAN(440, 20, 22)
// ng1 in (220, 256]
MDB_PLAN(448, 16, 28)
MDB_PLAN(450, 18, 25)
MDB_PLAN(462, 22, 21)
MDB_PLAN(480, 24, 20)
MDB_PLAN(484, 44, 11)
MDB_PLAN(486, 18, 27)
MDB_PLAN(490, 14, 35)
MDB_PLAN(500, 20, 25)
MDB_PLAN(504, 24, 21)
MDB_PLAN(512, 16, 32)
// their half edges not listed above
MDB_PLAN(165, 11, 15)
MDB_PLAN(175, 7, 25)
MDB_PLAN(189, 7, 27)
MDB_PLAN(225, 15, 15)
MDB_PLAN(231, 11, 21)
MDB_PLAN(243, 9, 27)
MDB_PLAN(245, 7, 35)
#undef MDB_PLAN

// Zero padding of input m of a radix-R1 first pass over stride R2 on an axis
// of length N (data in [floor(N/4), floor(N/4) + N/2)): 0 = padding for every
// item t < R2, 2 = data for every item, 1 = depends on the item.  With
// N % 4 == 0 and R1 % 4 == 0 no input is mixed; other splits have at most two
// mixed inputs, so they prune as well.
template <int N, int R2>
constexpr int pad_state(int m) {
    constexpr int OFF = N / 4, NG = N / 2;
    const int lo = R2 * m, hi = R2 * m + R2 - 1;
    if (hi < OFF || lo >= OFF + NG) return 0;
    return (lo >= OFF && hi < OFF + NG) ? 2 : 1;
}

// The inputs of item t of a pruned first pass: load(y) reads data element
// y in [0, N/2) (axis position y + floor(N/4)).
template <int N, int R1, int R2, class Load>
__device__ __forceinline__ void padded_inputs(float2 (&v)[R1], int t, const Load &load) {
    static_for<0, R1>([&](auto m_) {
        constexpr int m = decltype(m_)::value;
        constexpr int st = pad_state<N, R2>(m);
        const int y = t + R2 * m - N / 4;
        if constexpr (st == 0) v[m] = make_float2(-0.f, -0.f);
        else if constexpr (st == 2) v[m] = load(y);
        else v[m] = (unsigned)y < (unsigned)(N / 2) ? load(y) : make_float2(0.f, 0.f);
    });
}

// Forward phase 1 of item t on a zero-padded line at `b` (axis position 0)
// with element stride `es`, by the line plan of N; tw[j] = exp(-2 pi i j / N).
// The padding is never read.
template <int N>
__device__ __forceinline__ void padded_phase1(float2 *b, int es, int t, const float2 *__restrict__ tw) {
    constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
    float2 v[R1];
    padded_inputs<N, R1, R2>(v, t, [&](int y) { return b[(y + N / 4) * es]; });
    Dft<R1, -1>::run(v);
    static_for<0, R1>([&](auto k1_) {
        constexpr int k1 = decltype(k1_)::value;
        float2 x = v[k1];
        if constexpr (k1 != 0) x = cmul(x, __ldg(&tw[t * k1]));
        b[(k1 * R2 + t) * es] = x;
    });
}

// Phase 2 load + DFT of item u; result out[k2] belongs at element u + R1*k2.
template <int N, int S>
__device__ __forceinline__ void fft_phase2(const float2 *b, int es, int u, float2 (&out)[Plan<N>::R2]) {
    constexpr int R2 = Plan<N>::R2;
    static_for<0, R2>([&](auto n2_) { out[decltype(n2_)::value] = b[(u * R2 + decltype(n2_)::value) * es]; });
    Dft<R2, S>::run(out);
}

}  // namespace mdb
