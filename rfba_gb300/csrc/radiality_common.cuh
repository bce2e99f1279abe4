// Device code shared by the radiality kernel (radiality.cu) and its adjoint
// (adjoint.cu): packed f32x2 arithmetic, the warp-uniform tables, the smoothed
// gradient and the separable passes' helpers.
#pragma once

#include <cuda_runtime.h>

#include "srrf_internal.h"

namespace rfba {
namespace {

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int V>
struct IntC {
    static constexpr int value = V;
};

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
// v with its sign flipped where d < 0
__device__ __forceinline__ float flip_sign(float v, float d) {
    return __int_as_float(__float_as_int(v) ^ (__float_as_int(d) & 0x80000000));
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ int floordiv(int a, int b) {  // b > 0
    int q = a / b;
    return (a % b != 0 && a < 0) ? q - 1 : q;
}

// Division of 0 <= c < 65536 by d >= 2 with one multiply-high.
struct FastDiv {
    unsigned m;
    __device__ explicit FastDiv(int d) : m(0xffffffffu / (unsigned)d + 1u) {}
    __device__ int operator()(int c) const { return (int)__umulhi((unsigned)c, m); }
};

// The warp-uniform tables of a launch. They travel in the kernel's parameters
// when they fit (UN > 1): the compiler then keeps the tap weights and point
// constants in uniform registers, which a packed FMA takes as one operand
// without using a vector register read port. The ports are what bounds the
// point loop: FMAs with three different vector register operands run at 80
// lanes per clock and SM here, with a uniform operand at 112 of 128 (measured
// side by side). Rings too large for the parameters (AxesinRing above 12 or 13)
// read the same records from global memory.
template <int UN>
struct UTab {
    float4 q[UN];
};
template <int UN>
__device__ __forceinline__ float4 uget(const UTab<UN>& ut, const float4* g, int i) {
    if constexpr (UN > 1)
        return ut.q[i];
    else
        return __ldg(g + i);
}

// gradKernel's smoothed gradient (kernel.cu:73-124) at four coarse cells that
// follow each other along the innermost axis, from the clamped input tile
// (base: the first cell's voxel; x stride 1, mid stride sv, inner rows at
// row(k)): Gx = sum over i in [1, mR], j in [-yR, yR], k in [-zR, zR] of
// I(+i, j, k) - I(-i, j, k), and likewise for the other axes, in tile axis
// order. Ranges (1, 1, 1, 1) share their 6 x 9 loads between the four cells;
// with smoothing off the reference's central difference is the case mR = 1 and
// all lateral ranges 0. Integer inputs make the sums exact in float whatever
// the order. ORDERED adds the terms in the reference's order, i outside j outside k in
// the volume's x, y, z, whichever axis is innermost (y_inner: y is, and mid is z), so
// that a float input's gradient does not depend on the plan.
template <bool ORDERED = false, class Row>
__device__ __forceinline__ void gradient4(int mode, const int gr[4], Row&& row, int sv, float (&g)[3][4],
                                          bool y_inner = false) {
    if (mode == 1) {
        float v[6][3][3];  // [w - 1 .. w + 4][mid][x]
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float* r = row(k - 1);
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int i = 0; i < 3; ++i) v[k][j][i] = r[(j - 1) * sv + (i - 1)];
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            float gx = 0.f, gm = 0.f, gn = 0.f;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    if (!ORDERED) gx += v[w + b][a][2] - v[w + b][a][0];
                    gm += v[w + b][2][a] - v[w + b][0][a];
                    gn += ORDERED ? v[w + 2][b][a] - v[w][b][a] : v[w + 2][a][b] - v[w][a][b];
                }
            if (ORDERED) {
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const float(&u)[3] = v[w + b][a];
                        const float(&s)[3] = v[w + a][b];
                        gx += y_inner ? s[2] - s[0] : u[2] - u[0];
                    }
            }
            g[0][w] = gx;
            g[1][w] = gm;
            g[2][w] = gn;
        }
    } else if (mode == 2) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float* r = row(w);
            g[0][w] = r[1] - r[-1];
            g[1][w] = r[sv] - r[-sv];
            g[2][w] = row(w + 1)[0] - row(w - 1)[0];
        }
    } else {
        const int mR = gr[0], xR = gr[1], yR = gr[2], zR = gr[3];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            float gx = 0.f, gm = 0.f, gn = 0.f;
            auto I = [&](int dx, int dm, int dn) { return row(w + dn)[dm * sv + dx]; };
            const bool swap = ORDERED && y_inner;
            const int oR = swap ? zR : yR, pR = swap ? yR : zR;
            for (int i = 1; i <= mR; ++i)
                for (int j = -oR; j <= oR; ++j)
                    for (int k = -pR; k <= pR; ++k)
                        gx += swap ? I(i, k, j) - I(-i, k, j) : I(i, j, k) - I(-i, j, k);
            for (int j = 1; j <= mR; ++j)
                for (int i = -xR; i <= xR; ++i)
                    for (int k = -zR; k <= zR; ++k) gm += I(i, j, k) - I(i, -j, k);
            for (int k = 1; k <= mR; ++k)
                for (int i = -xR; i <= xR; ++i)
                    for (int j = -yR; j <= yR; ++j) gn += I(i, j, k) - I(i, j, -k);
            g[0][w] = gx;
            g[1][w] = gm;
            g[2][w] = gn;
        }
    }
}

// Four taps along x (src, src + 1, ..) at four cells of the innermost axis.
__device__ __forceinline__ void filter4(float4 w, const float4* src, float (&r)[4]) {
    const float4 u0 = src[0], u1 = src[1], u2 = src[2], u3 = src[3];
    r[0] = fmaf(w.w, u3.x, fmaf(w.z, u2.x, fmaf(w.y, u1.x, w.x * u0.x)));
    r[1] = fmaf(w.w, u3.y, fmaf(w.z, u2.y, fmaf(w.y, u1.y, w.x * u0.y)));
    r[2] = fmaf(w.w, u3.z, fmaf(w.z, u2.z, fmaf(w.y, u1.z, w.x * u0.z)));
    r[3] = fmaf(w.w, u3.w, fmaf(w.z, u2.w, fmaf(w.y, u1.w, w.x * u0.w)));
}
// Four taps, four cells of the innermost axis at once.
__device__ __forceinline__ float4 filter_cells(float4 w, float4 c0, float4 c1, float4 c2, float4 c3) {
    const float2 w0 = dup(w.x), w1 = dup(w.y), w2 = dup(w.z), w3 = dup(w.w);
    const float2 l = fma2(w3, lo2(c3), fma2(w2, lo2(c2), fma2(w1, lo2(c1), mul2(w0, lo2(c0)))));
    const float2 h = fma2(w3, hi2(c3), fma2(w2, hi2(c2), fma2(w1, hi2(c1), mul2(w0, hi2(c0)))));
    return make_float4(l.x, l.y, h.x, h.y);
}
// The same along the tile's mid axis (rows src, src + stride, ..).
__device__ __forceinline__ float4 filter_rows(float4 w, const float4* src, int stride) {
    return filter_cells(w, src[0], src[stride], src[2 * stride], src[3 * stride]);
}
// Cell w of a column into the packed halves (compile-time w).
template <int CH, int NH>
__device__ __forceinline__ void put_half(float2 (&T)[NH], int w, float v) {
    if (w < NH) T[w].x = v;
    if (w >= CH && w - CH < NH) T[w - CH].y = v;
}

// Sum of what the packed halves hold for cell w (compile-time w).
template <int CH, int NH>
__device__ __forceinline__ float get_halves(const float2 (&T)[NH], int w) {
    return w >= NH + CH ? 0.f : w >= NH ? T[w - CH].y : w < CH ? T[w].x : T[w].x + T[w - CH].y;
}

}  // namespace
}  // namespace rfba
