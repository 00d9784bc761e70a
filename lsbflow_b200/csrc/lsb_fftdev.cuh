// Device helpers shared by the FFT kernels: complex arithmetic, exactly rounded twiddle
// constants for the small register DFTs, and the register DFT of 1..16 points.
#pragma once
#include <cuda_runtime.h>

namespace lsb {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// scalar type and constructor of a complex vector type (double2 / float2)
template <class V> struct CT;
template <> struct CT<double2> {
    using S = double;
    __device__ static double2 make(double x, double y) { return make_double2(x, y); }
};
template <> struct CT<float2> {
    using S = float;
    __device__ static float2 make(float x, float y) { return make_float2(x, y); }
};

// cos and sin of 2 pi j / 48, j = 0..47, correctly rounded (computed from the series
// definitions in exact decimal arithmetic)
static __device__ constexpr double kC48[48] = {0x1.0000000000000p+0, 0x1.fb9ea92ec689bp-1, 0x1.ee8dd4748bf15p-1, 0x1.d906bcf328d46p-1, 0x1.bb67ae8584caap-1, 0x1.963268b572492p-1, 0x1.6a09e667f3bcdp-1, 0x1.37af93f9513eap-1, 0x1.0000000000000p-1, 0x1.87de2a6aea963p-2, 0x1.0907dc1930690p-2, 0x1.0b5150f6da2d1p-3, 0x0.0p+0, -0x1.0b5150f6da2d1p-3, -0x1.0907dc1930690p-2, -0x1.87de2a6aea963p-2, -0x1.0000000000000p-1, -0x1.37af93f9513eap-1, -0x1.6a09e667f3bcdp-1, -0x1.963268b572492p-1, -0x1.bb67ae8584caap-1, -0x1.d906bcf328d46p-1, -0x1.ee8dd4748bf15p-1, -0x1.fb9ea92ec689bp-1, -0x1.0000000000000p+0, -0x1.fb9ea92ec689bp-1, -0x1.ee8dd4748bf15p-1, -0x1.d906bcf328d46p-1, -0x1.bb67ae8584caap-1, -0x1.963268b572492p-1, -0x1.6a09e667f3bcdp-1, -0x1.37af93f9513eap-1, -0x1.0000000000000p-1, -0x1.87de2a6aea963p-2, -0x1.0907dc1930690p-2, -0x1.0b5150f6da2d1p-3, 0x0.0p+0, 0x1.0b5150f6da2d1p-3, 0x1.0907dc1930690p-2, 0x1.87de2a6aea963p-2, 0x1.0000000000000p-1, 0x1.37af93f9513eap-1, 0x1.6a09e667f3bcdp-1, 0x1.963268b572492p-1, 0x1.bb67ae8584caap-1, 0x1.d906bcf328d46p-1, 0x1.ee8dd4748bf15p-1, 0x1.fb9ea92ec689bp-1};
static __device__ constexpr double kS48[48] = {0x0.0p+0, 0x1.0b5150f6da2d1p-3, 0x1.0907dc1930690p-2, 0x1.87de2a6aea963p-2, 0x1.0000000000000p-1, 0x1.37af93f9513eap-1, 0x1.6a09e667f3bcdp-1, 0x1.963268b572492p-1, 0x1.bb67ae8584caap-1, 0x1.d906bcf328d46p-1, 0x1.ee8dd4748bf15p-1, 0x1.fb9ea92ec689bp-1, 0x1.0000000000000p+0, 0x1.fb9ea92ec689bp-1, 0x1.ee8dd4748bf15p-1, 0x1.d906bcf328d46p-1, 0x1.bb67ae8584caap-1, 0x1.963268b572492p-1, 0x1.6a09e667f3bcdp-1, 0x1.37af93f9513eap-1, 0x1.0000000000000p-1, 0x1.87de2a6aea963p-2, 0x1.0907dc1930690p-2, 0x1.0b5150f6da2d1p-3, 0x0.0p+0, -0x1.0b5150f6da2d1p-3, -0x1.0907dc1930690p-2, -0x1.87de2a6aea963p-2, -0x1.0000000000000p-1, -0x1.37af93f9513eap-1, -0x1.6a09e667f3bcdp-1, -0x1.963268b572492p-1, -0x1.bb67ae8584caap-1, -0x1.d906bcf328d46p-1, -0x1.ee8dd4748bf15p-1, -0x1.fb9ea92ec689bp-1, -0x1.0000000000000p+0, -0x1.fb9ea92ec689bp-1, -0x1.ee8dd4748bf15p-1, -0x1.d906bcf328d46p-1, -0x1.bb67ae8584caap-1, -0x1.963268b572492p-1, -0x1.6a09e667f3bcdp-1, -0x1.37af93f9513eap-1, -0x1.0000000000000p-1, -0x1.87de2a6aea963p-2, -0x1.0907dc1930690p-2, -0x1.0b5150f6da2d1p-3};

// cos and sin of 2 pi j / R for the odd lengths 5, 7 and 9, correctly rounded
static __device__ constexpr double kC5[5] = {0x1.0000000000000p+0, 0x1.3c6ef372fe950p-2, -0x1.9e3779b97f4a8p-1, -0x1.9e3779b97f4a8p-1, 0x1.3c6ef372fe950p-2};
static __device__ constexpr double kS5[5] = {0x0.0p+0, 0x1.e6f0e134454ffp-1, 0x1.2cf2304755a5ep-1, -0x1.2cf2304755a5ep-1, -0x1.e6f0e134454ffp-1};
static __device__ constexpr double kC7[7] = {0x1.0000000000000p+0, 0x1.3f3a0e28bedd1p-1, -0x1.c7b90e3024582p-3, -0x1.cd4bca9cb5c71p-1, -0x1.cd4bca9cb5c71p-1, -0x1.c7b90e3024582p-3, 0x1.3f3a0e28bedd1p-1};
static __device__ constexpr double kS7[7] = {0x0.0p+0, 0x1.904c37505de4bp-1, 0x1.f329c0558e969p-1, 0x1.bc4c04d71abc1p-2, -0x1.bc4c04d71abc1p-2, -0x1.f329c0558e969p-1, -0x1.904c37505de4bp-1};
static __device__ constexpr double kC9[9] = {0x1.0000000000000p+0, 0x1.8836fa2cf5039p-1, 0x1.63a1a7e0b738ap-3, -0x1.0000000000000p-1, -0x1.e11f642522d1cp-1, -0x1.e11f642522d1cp-1, -0x1.0000000000000p-1, 0x1.63a1a7e0b738ap-3, 0x1.8836fa2cf5039p-1};
static __device__ constexpr double kS9[9] = {0x0.0p+0, 0x1.491b7523c161dp-1, 0x1.f838b8c811c17p-1, 0x1.bb67ae8584caap-1, 0x1.5e3a8748a0bf5p-2, -0x1.5e3a8748a0bf5p-2, -0x1.bb67ae8584caap-1, -0x1.f838b8c811c17p-1, -0x1.491b7523c161dp-1};
template <int R>
__device__ __forceinline__ constexpr double odd_cos(int j) { return R == 5 ? kC5[j % 5] : (R == 7 ? kC7[j % 7] : kC9[j % 9]); }
template <int R>
__device__ __forceinline__ constexpr double odd_sin(int j) { return R == 5 ? kS5[j % 5] : (R == 7 ? kS7[j % 7] : kS9[j % 9]); }

// e^{SIGN 2 pi i m / R} for R = 9 or R dividing 48
template <int R, int SIGN, class V = double2>
__device__ __forceinline__ V omega(int m) {
    using S = typename CT<V>::S;
    if constexpr (R == 9) return CT<V>::make((S)odd_cos<9>(m), (S)(SIGN * odd_sin<9>(m)));
    const int j = (m * (48 / R)) % 48;
    return CT<V>::make((S)kC48[j], (S)(SIGN < 0 ? -kS48[j] : kS48[j]));
}

// R-point DFT in registers: 2, 3, 4 directly, 5 and 7 from the sums and differences of the
// pairs (j, R - j), 9 = 3 x 3 and 6, 8, 12, 16 = A*B (A in {4,3}) by one four-step split with
// constant twiddles, 10, 14, 15, 18, 20 and 24 = A*B with coprime factors by the prime-factor map (input
// B a + A b, output k = ka mod A = kb mod B), which needs no twiddles.
template <int R, int SIGN, class V>
__device__ __forceinline__ void dft_reg(V (&v)[R]) {
    using S = typename CT<V>::S;
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const V a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 3) {
        const S h = (S)kS48[16];  // sin(2 pi / 3)
        const V t1 = cadd(v[1], v[2]);
        const V t2 = CT<V>::make(v[0].x - (S)0.5 * t1.x, v[0].y - (S)0.5 * t1.y);
        const V d = csub(v[1], v[2]);
        // SIGN < 0: X1 = t2 - i h d, X2 = t2 + i h d
        const V ihd = CT<V>::make(-h * d.y, h * d.x);
        v[0] = cadd(v[0], t1);
        if (SIGN < 0) {
            v[1] = csub(t2, ihd);
            v[2] = cadd(t2, ihd);
        } else {
            v[1] = cadd(t2, ihd);
            v[2] = csub(t2, ihd);
        }
    } else if constexpr (R == 4) {
        const V a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const V c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        if (SIGN < 0) {
            v[1] = CT<V>::make(b.x + d.y, b.y - d.x);
            v[3] = CT<V>::make(b.x - d.y, b.y + d.x);
        } else {
            v[1] = CT<V>::make(b.x - d.y, b.y + d.x);
            v[3] = CT<V>::make(b.x + d.y, b.y - d.x);
        }
    } else if constexpr (R == 5 || R == 7) {
        constexpr int H = (R - 1) / 2;
        V a[H], b[H];  // x_j + x_{R-j}, x_j - x_{R-j}
#pragma unroll
        for (int j = 0; j < H; ++j) {
            a[j] = cadd(v[j + 1], v[R - 1 - j]);
            b[j] = csub(v[j + 1], v[R - 1 - j]);
        }
        const V x0 = v[0];
#pragma unroll
        for (int j = 0; j < H; ++j) v[0] = cadd(v[0], a[j]);
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            V e = x0, o = CT<V>::make((S)0, (S)0);
#pragma unroll
            for (int j = 1; j <= H; ++j) {
                const S cc = (S)odd_cos<R>(j * k), ss = (S)(SIGN * odd_sin<R>(j * k));
                e = CT<V>::make(fma(cc, a[j - 1].x, e.x), fma(cc, a[j - 1].y, e.y));
                o = CT<V>::make(fma(-ss, b[j - 1].y, o.x), fma(ss, b[j - 1].x, o.y));  // i s b
            }
            v[k] = cadd(e, o);
            v[R - k] = csub(e, o);
        }
    } else if constexpr (R == 10 || R == 14 || R == 15 || R == 18 || R == 20 || R == 24) {
        constexpr int A = (R == 20) ? 4 : ((R == 15 || R == 24) ? 3 : 2), B = R / A;
        V w[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int a = 0; a < A; ++a) w[b][a] = v[(B * a + A * b) % R];
            dft_reg<A, SIGN>(w[b]);
        }
#pragma unroll
        for (int ka = 0; ka < A; ++ka) {
            V u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) u[b] = w[b][ka];
            dft_reg<B, SIGN>(u);
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (k % A == ka) v[k] = u[k % B];
        }
    } else {
        constexpr int A = (R % 4 == 0) ? 4 : 3;
        constexpr int B = R / A;
        V w[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            V u[A];
#pragma unroll
            for (int a = 0; a < A; ++a) u[a] = v[B * a + b];
            dft_reg<A, SIGN>(u);
#pragma unroll
            for (int ka = 0; ka < A; ++ka) w[b][ka] = (b > 0 && ka > 0) ? cmul(u[ka], omega<R, SIGN, V>(b * ka)) : u[ka];
        }
#pragma unroll
        for (int ka = 0; ka < A; ++ka) {
            V u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) u[b] = w[b][ka];
            dft_reg<B, SIGN>(u);
#pragma unroll
            for (int kb = 0; kb < B; ++kb) v[ka + A * kb] = u[kb];
        }
    }
}


}  // namespace lsb
