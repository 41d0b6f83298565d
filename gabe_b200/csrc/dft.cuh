// In-register DFTs of the mixed-radix transforms (fftp.cuh): R points, R a
// power of two times 1, 3, 5 or 7, forward sign e^{-i}, natural order in and
// out.  Complex sums and differences go through the packed two-element FP32
// instructions of sm_100a (one issue slot for both parts: the transforms are
// bound by instruction issue), products with roots of unity stay scalar.
#pragma once

#include <cstdint>
#include <utility>

#include "common.cuh"

namespace gabe {
namespace dft {

// cos and sin of 2 pi a / b at compile time: the angle is folded to the first
// octant, where the Taylor series converges to FP64 rounding in 12 terms.
constexpr double kTwoPi = 6.283185307179586476925286766559;
__host__ __device__ constexpr double taylor_cos(double x) {
    double t = 1., s = 1.;
    for (int n = 1; n <= 12; n++) s += (t *= -x * x / ((2 * n - 1) * (2 * n)));
    return s;
}
__host__ __device__ constexpr double taylor_sin(double x) {
    double t = x, s = x;
    for (int n = 1; n <= 12; n++) s += (t *= -x * x / ((2 * n) * (2 * n + 1)));
    return s;
}
__host__ __device__ constexpr double cos_turn(long long a, long long b) {
    a %= b;
    if (a < 0) a += b;
    if (2 * a > b) a = b - a;                       // cos(2 pi - x) = cos x
    if (4 * a > b) return -cos_turn(b - 2 * a, 2 * b);  // cos(pi - x) = -cos x
    if (8 * a > b) return taylor_sin(kTwoPi * (double)(b - 4 * a) / (double)(4 * b));
    return taylor_cos(kTwoPi * (double)a / (double)b);
}
__host__ __device__ constexpr double sin_turn(long long a, long long b) { return cos_turn(4 * a - b, 4 * b); }

__device__ __forceinline__ float2 add(float2 a, float2 b) {
    float2 r;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)));
    return r;
}
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
    float2 r;
    asm("sub.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)));
    return r;
}
// a + c b with a real c
__device__ __forceinline__ float2 axpy(float c, float2 b, float2 a) {
    float2 r, cc = make_float2(c, c);
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(cc)), "l"(reinterpret_cast<uint64_t &>(b)),
          "l"(reinterpret_cast<uint64_t &>(a)));
    return r;
}
__device__ __forceinline__ float2 scale(float c, float2 b) { return make_float2(c * b.x, c * b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
    return make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}

// v exp(-2 pi i M / R)
template <int M, int R>
__device__ __forceinline__ float2 mul_root(float2 v) {
    constexpr int m = ((M % R) + R) % R;
    if constexpr (m == 0) {
        return v;
    } else if constexpr (4 * m == R) {
        return make_float2(v.y, -v.x);
    } else if constexpr (2 * m == R) {
        return make_float2(-v.x, -v.y);
    } else if constexpr (4 * m == 3 * R) {
        return make_float2(-v.y, v.x);
    } else {
        constexpr float c = (float)cos_turn(m, R), s = (float)sin_turn(m, R);
        return make_float2(v.x * c + v.y * s, v.y * c - v.x * s);
    }
}

template <int I>
struct Int {
    __host__ __device__ constexpr operator int() const { return I; }
};
template <int... I, typename F>
__device__ __forceinline__ void static_for_seq(std::integer_sequence<int, I...>, F &&f) {
    (f(Int<I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F &&f) {
    static_for_seq(std::make_integer_sequence<int, N>{}, static_cast<F &&>(f));
}

// Odd prime P by the definition, folded over x[n] +- x[P-n]:
// X[k], X[P-k] = x0 + sum_n (x[n] + x[P-n]) cos -+ i (x[n] - x[P-n]) sin.
template <int P>
__device__ __forceinline__ void odd(float2 (&x)[P]) {
    constexpr int H = (P - 1) / 2;
    float2 s[H], d[H];
    static_for<H>([&](auto n) {
        s[n] = add(x[1 + n], x[P - 1 - n]);
        d[n] = sub(x[1 + n], x[P - 1 - n]);
    });
    const float2 x0 = x[0];
    static_for<H>([&](auto n) { x[0] = add(x[0], s[n]); });
    static_for<H>([&](auto k) {
        float2 e = x0, o = make_float2(0.f, 0.f);
        static_for<H>([&](auto n) {
            constexpr float c = (float)cos_turn((k + 1) * (n + 1), P), sn = (float)sin_turn((k + 1) * (n + 1), P);
            e = axpy(c, s[n], e);
            if constexpr (n == 0) o = scale(sn, d[n]);
            else o = axpy(sn, d[n], o);
        });
        x[1 + k] = make_float2(e.x + o.y, e.y - o.x);
        x[P - 1 - k] = make_float2(e.x - o.y, e.y + o.x);
    });
}

__host__ __device__ constexpr int odd_part(int r) { return r % 2 ? r : odd_part(r / 2); }

// R points, natural order in and out.
template <int R>
__device__ __forceinline__ void points(float2 (&x)[R]) {
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const float2 a = x[0];
        x[0] = add(a, x[1]);
        x[1] = sub(a, x[1]);
    } else if constexpr (R == 3 || R == 5 || R == 7) {
        odd<R>(x);
    } else {
        // n = Q n1 + n2, k = k1 + P k2: P-point DFTs over n1, roots, Q-point DFTs over n2
        constexpr int P = odd_part(R) > 1 ? odd_part(R) : (R % 4 == 0 && R > 4 ? 4 : 2), Q = R / P;
        float2 z[P][Q];
        static_for<Q>([&](auto n2) {
            float2 t[P];
            static_for<P>([&](auto n1) { t[n1] = x[Q * n1 + n2]; });
            points<P>(t);
            static_for<P>([&](auto k1) { z[k1][n2] = mul_root<n2 * k1, R>(t[k1]); });
        });
        static_for<P>([&](auto k1) {
            points<Q>(z[k1]);
            static_for<Q>([&](auto k2) { x[k1 + P * k2] = z[k1][k2]; });
        });
    }
}

}  // namespace dft
}  // namespace gabe
