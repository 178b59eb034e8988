// Small inverse transforms in registers (radix 2, 4, 8, 32) and tables of roots of unity, for the
// channelizer kernels (chan_fused.cuh, chan_fft1024.cu).
#pragma once

#include "ptx.cuh"

#include <cuda_runtime.h>

namespace rfx {
namespace fft {

// The transform's roots of unity, rounded once from double. Built at compile time: sine and
// cosine by their Taylor series on [0, pi / 4], the other octants by symmetry.
template <int N>
struct Roots {
    float v[2 * N];   // e^{2 pi i k / N}: re, im
};

constexpr double taylor(double a, bool cosine)
{
    double term = cosine ? 1.0 : a;
    double sum = term;
    for (int k = cosine ? 1 : 2; k < 30; k += 2) {
        term *= -a * a / (static_cast<double>(k) * (k + 1));
        sum += term;
    }
    return sum;
}

template <int N>
constexpr Roots<N> make_roots()
{
    Roots<N> r{};
    constexpr double kPi = 3.14159265358979323846264338327950288;
    constexpr int kOctant = N / 8;
    for (int k = 0; k < N; ++k) {
        const int oct = k / kOctant;
        const int rem = k % kOctant;
        // Angle within the octant, mirrored in odd octants.
        const double a = 2.0 * kPi * ((oct & 1) ? kOctant - rem : rem) / N;
        const double c = taylor(a, true);
        const double s = taylor(a, false);
        double re = 0.0;
        double im = 0.0;
        switch (oct) {
        case 0: re = c; im = s; break;
        case 1: re = s; im = c; break;
        case 2: re = -s; im = c; break;
        case 3: re = -c; im = s; break;
        case 4: re = -c; im = -s; break;
        case 5: re = -s; im = -c; break;
        case 6: re = s; im = -c; break;
        default: re = c; im = -s; break;
        }
        r.v[2 * k] = static_cast<float>(re);
        r.v[2 * k + 1] = static_cast<float>(im);
    }
    return r;
}

// ---- small transforms in registers (inverse: w = e^{+2 pi i / r}) -----------------------------

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// a + i b and a - i b.
__device__ __forceinline__ f32x2 add_i(f32x2 a, f32x2 b)
{
    const float2 p = unpack2(a);
    const float2 q = unpack2(b);
    return pack2(p.x - q.y, p.y + q.x);
}

__device__ __forceinline__ f32x2 sub_i(f32x2 a, f32x2 b)
{
    const float2 p = unpack2(a);
    const float2 q = unpack2(b);
    return pack2(p.x + q.y, p.y - q.x);
}

__device__ __forceinline__ f32x2 cmul(f32x2 a, float2 w)
{
    const float2 p = unpack2(a);
    return pack2(__fmaf_rn(p.x, w.x, -__fmul_rn(p.y, w.y)),
                 __fmaf_rn(p.x, w.y, __fmul_rn(p.y, w.x)));
}

template <int r>
__device__ __forceinline__ void small_dft(f32x2* v)
{
    if constexpr (r == 2) {
        const f32x2 a = v[0];
        v[0] = add2(a, v[1]);
        v[1] = sub2(a, v[1]);
    } else if constexpr (r == 4) {
        const f32x2 s0 = add2(v[0], v[2]);
        const f32x2 d0 = sub2(v[0], v[2]);
        const f32x2 s1 = add2(v[1], v[3]);
        const f32x2 d1 = sub2(v[1], v[3]);
        v[0] = add2(s0, s1);
        v[1] = add_i(d0, d1);
        v[2] = sub2(s0, s1);
        v[3] = sub_i(d0, d1);
    } else {
        static_assert(r == 8, "radix 2, 4 or 8");
        constexpr float c = 0.70710678118654752440f;
        const f32x2 s0 = add2(v[0], v[4]);
        const f32x2 d0 = sub2(v[0], v[4]);
        const f32x2 s1 = add2(v[1], v[5]);
        const f32x2 d1 = sub2(v[1], v[5]);
        const f32x2 s2 = add2(v[2], v[6]);
        const f32x2 d2 = sub2(v[2], v[6]);
        const f32x2 s3 = add2(v[3], v[7]);
        const f32x2 d3 = sub2(v[3], v[7]);
        // Even outputs: the 4-point transform of s.
        const f32x2 e0 = add2(s0, s2);
        const f32x2 e1 = sub2(s0, s2);
        const f32x2 e2 = add2(s1, s3);
        const f32x2 e3 = sub2(s1, s3);
        v[0] = add2(e0, e2);
        v[4] = sub2(e0, e2);
        v[2] = add_i(e1, e3);
        v[6] = sub_i(e1, e3);
        // Odd outputs: w8 d1 = c (1 + i) d1 and w8^3 d3 = c (-1 + i) d3.
        const f32x2 f0 = add_i(d0, d2);
        const f32x2 f1 = sub_i(d0, d2);
        const float2 p = unpack2(d1);
        const float2 q = unpack2(d3);
        const f32x2 g1 = pack2(p.x - p.y, p.y + p.x);
        const f32x2 g3 = pack2(-q.x - q.y, q.x - q.y);
        const f32x2 h0 = add2(g1, g3);
        const f32x2 h1 = sub2(g1, g3);
        const f32x2 cc = pack2(c, c);
        const f32x2 nc = pack2(-c, -c);
        v[1] = fma2(cc, h0, f0);
        v[5] = fma2(nc, h0, f0);
        const float2 a = unpack2(f1);
        const float2 b = unpack2(h1);
        v[3] = pack2(__fmaf_rn(-c, b.y, a.x), __fmaf_rn(c, b.x, a.y));
        v[7] = pack2(__fmaf_rn(c, b.y, a.x), __fmaf_rn(-c, b.x, a.y));
    }
}

// 32 points, as 4 x 8: v[n] in, v[k] out, n = a + 4 b, k = c + 8 d:
//   sum_a w32^(a c) w4^(a d) [ sum_b v[a + 4 b] w8^(b c) ].
__device__ __forceinline__ void dft32(f32x2 (&v)[32])
{
    // cos(2 pi j / 32), j = 0 .. 8.
    constexpr float kC[9] = {1.0f,
                             0.98078528040323044913f,
                             0.92387953251128675613f,
                             0.83146961230254523708f,
                             0.70710678118654752440f,
                             0.55557023301960222474f,
                             0.38268343236508977173f,
                             0.19509032201612826785f,
                             0.0f};
    f32x2 t[4][8];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            t[a][b] = v[a + 4 * b];
        }
        small_dft<8>(t[a]);
#pragma unroll
        for (int c = 1; c < 8; ++c) {
            if (a > 0) {
                const int j = a * c;          // 1 .. 21: quadrants 0 to 2 of the circle
                const int q = j / 8;
                const int r = j % 8;
                const float re = q == 0 ? kC[r] : q == 1 ? -kC[8 - r] : -kC[r];
                const float im = q == 0 ? kC[8 - r] : q == 1 ? kC[r] : -kC[8 - r];
                t[a][c] = cmul(t[a][c], make_float2(re, im));
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        f32x2 w[4] = {t[0][c], t[1][c], t[2][c], t[3][c]};
        small_dft<4>(w);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            v[c + 8 * d] = w[d];
        }
    }
}

}  // namespace fft
}  // namespace rfx
