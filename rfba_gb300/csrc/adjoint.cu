// Differentiable SRRF path (sm_103a): drift resampling, and the adjoint of a
// scalar objective on the map with respect to the input voxels and the
// per-volume drift shifts. The reference has no derivatives; the forward it
// differentiates is the reference's radiality (kernel.cu:44-287) and temporal
// reduction (TRA kernel.cu:291-327, TRAC with ITC 0 kernel.cu:469-507) on
// volumes resampled by the drift operator
//     I'_t(x) = sum_{i,j,k} c(x + d_x - i) c(y + d_y - j) c(z + d_z - k) I_t[clamp(i, j, k)],
// c = the reference's Catmull-Rom kernel (kernel.cu:128-138), applied one axis
// at a time (x, then y, then z).
//
// Backward, per call:
//   1. temporal adjoint, one thread per subvoxel: dL/drad_t and dL/dI_t from
//      dL/dmap and the stored radiality/intensity stacks;
//   2. radiality adjoint, persistent over (tile, time) like the forward: the
//      interpolated gradient at every ring sample is recomputed (not stored),
//      the derivative of the radiality term is pushed back through the transposed
//      passes, and the tile's contribution to dL/dI' is added to global memory;
//   3. the drift operator's transpose gives dL/dI, and dL/dd_t is the sum over
//      the volume of dL/dI'_t times the resampling with derivative weights on
//      one axis.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "radiality_common.cuh"
#include "shared_limit.h"
#include "srrf_internal.h"

namespace rfba {
namespace {

// Bounds check of a computed global index: out of range records the first
// offence (site in the top byte, index below) and the access is skipped.
__device__ __forceinline__ bool in_range(long long i, long long n, unsigned long long* err, int site) {
    if (i >= 0 && i < n) return true;
    if (err) atomicCAS(err, 0ull, ((unsigned long long)site << 56) | ((unsigned long long)i & 0x00ffffffffffffffull));
    return false;
}

// Catmull-Rom kernel and its derivative (a = 0.5), kernel.cu:128-138.
__device__ __forceinline__ float cr(float xx) {
    const float a = 0.5f;
    const float x = fabsf(xx);
    if (x < 1.f) return x * x * (x * (2.f - a) + (a - 3.f)) + 1.f;
    if (x < 2.f) return ((-a * x + 5.f * a) * x - 8.f * a) * x + 4.f * a;
    return 0.f;
}
__device__ __forceinline__ float dcr(float xx) {
    const float a = 0.5f;
    const float x = fabsf(xx), s = xx < 0.f ? -1.f : 1.f;
    if (x < 1.f) return s * (3.f * (2.f - a) * x * x + 2.f * (a - 3.f) * x);
    if (x < 2.f) return s * ((-3.f * a * x + 10.f * a) * x - 8.f * a);
    return 0.f;
}

// ---------------------------------------------------------------------------
// Transpose of the drift operator on one axis: a gather over the outputs whose
// clamped taps hit each input position. Away from the axis's ends an output xo hits
// position c with one tap, c - floor(xo + d), so at most eight outputs in a row are
// looked at and one weight formed for each; at the ends, where clamped taps pile up,
// every output's four taps are tried. One warp a row (t, z, y) with x across its
// lanes, so y's and z's weights are formed once a row. 60 volumes of 64^3, per axis:
// x 0.22, y 0.13, z 0.13 ms against 0.35 when each voxel divided its index in 64 bits
// and formed the weight of each of the 28 pairs of output and tap; floor 0.02.
__device__ __forceinline__ float end_weight(int xo, float d, int c, int len) {
    const float pos = (float)xo + d;
    const int base = (int)floorf(pos);
    float w = 0.f;
#pragma unroll
    for (int k = -1; k <= 2; ++k)
        if (clampi(base + k, 0, len - 1) == c) w += cr(pos - (float)(base + k));
    return w;
}
template <int AXIS>
__global__ void __launch_bounds__(256) shift_adjoint_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                            int W, int H, int D, int T,
                                                            const float* __restrict__ shifts) {
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)D * H, stride = AXIS == 0 ? 1 : (AXIS == 1 ? W : (long long)W * H);
    const int len = AXIS == 0 ? W : (AXIS == 1 ? H : D);
    for (long long r = blockIdx.x * 8LL + (threadIdx.x >> 5); r < rows * T; r += gridDim.x * 8LL) {
        const int t = (int)(r / rows), zy = (int)(r - t * rows);
        const int z = zy / H, y = zy - z * H;
        const float d = shifts[3 * t + AXIS];
        constexpr int N = 8;
        float w[N];
        int first = 0;
        auto weights = [&](int c) {
            first = (int)floorf((float)c - d) - 3;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int xo = (int)((unsigned)first + j);
                const float pos = (float)xo + d;
                const int k = c - (int)floorf(pos);
                w[j] = xo >= 0 && xo < len && k >= -1 && k <= 2 ? cr(pos - (float)c) : 0.f;
            }
        };
        const int c0 = AXIS == 1 ? y : z;
        if (AXIS != 0) weights(c0);
        for (int x = lane; x < W; x += 32) {
            const int c = AXIS == 0 ? x : c0;
            const long long i = r * W + x;
            const float* line = src + (i - c * stride);
            float acc = 0.f;
            if (c > 0 && c < len - 1) {
                if (AXIS == 0) weights(c);
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (w[j] != 0.f) acc = fmaf(w[j], __ldg(line + (first + j) * stride), acc);
            } else {
                const int lo = c == 0 ? 0 : max((int)floorf((float)c - d) - 3, 0);
                const int hi = c == len - 1 ? len - 1 : min((int)ceilf((float)c - d) + 3, len - 1);
                for (int xo = lo; xo <= hi; ++xo) {
                    const float we = end_weight(xo, d, c, len);
                    if (we != 0.f) acc = fmaf(we, __ldg(line + xo * stride), acc);
                }
            }
            dst[i] = acc;
        }
    }
}

// Drift operator on all three axes at once: the x-, y- and z-passes with
// per-axis index clamping compose to one 4 x 4 x 4 tensor-product stencil with
// clamped indices. mode 0 writes I'_t; mode 1 adds, per volume, the sums over
// voxels of g * dI'/dd_a (a = x, y, z: derivative weights on axis a) into
// out[3 t + a] (FP64, one atomic per block and axis). A warp takes 32 columns of x
// at one y and walks L planes of z, keeping the last four planes' x- and y-passes in
// registers: a step reads one plane's 16 taps instead of four planes' 64. The
// passes and their sums are the stencil's. Bound by the taps' load instructions: 60
// volumes of 64^3 take 0.17 ms (mode 0) and 0.43 (mode 1), 0.56 and 0.82 with all 64
// taps a voxel.
constexpr int kDriftThreads = 256;
template <int MODE>
__global__ void __launch_bounds__(kDriftThreads) drift3d_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                                const float* __restrict__ g, int W, int H, int D,
                                                                int L, const float* __restrict__ shifts,
                                                                double* __restrict__ out) {
    const int t = blockIdx.y;
    const long long nv = (long long)W * H * D;
    const float* st = src + (long long)t * nv;
    const float dx = shifts[3 * t], dy = shifts[3 * t + 1], dz = shifts[3 * t + 2];
    double acc[3] = {0.0, 0.0, 0.0};
    const int nx = (W + 31) / 32, nz = (D + L - 1) / L;
    // every index is clamped into the volume, so no tap can leave it
    for (long long i = blockIdx.x * (kDriftThreads / 32LL) + (threadIdx.x >> 5); i < (long long)nx * H * nz;
         i += gridDim.x * (kDriftThreads / 32LL)) {
        const long long q = i / nx;
        const int x = (int)(i - q * nx) * 32 + (threadIdx.x & 31);
        const int y = (int)(q % H), z0 = (int)(q / H) * L;
        if (x >= W) continue;
        const float px = (float)x + dx, py = (float)y + dy;
        const int bx = (int)floorf(px), by = (int)floorf(py);
        float wx[4], ex[4], wy[4], ey[4];
        long long ty[4];  // a tap's row in a plane
        int ix[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            wx[k] = cr(px - (float)(bx + k - 1));
            wy[k] = cr(py - (float)(by + k - 1));
            if (MODE == 1) {
                ex[k] = dcr(px - (float)(bx + k - 1));
                ey[k] = dcr(py - (float)(by + k - 1));
            }
            ty[k] = (long long)clampi(by + k - 1, 0, H - 1) * W;
            ix[k] = clampi(bx + k - 1, 0, W - 1);
        }
        // a plane's x pass per row, then its y pass
        float s[4], s_dx[4], s_dy[4];
        auto plane = [&](int z, int k) {
            const float* rp = st + (long long)clampi(z, 0, D - 1) * H * W;
            float v[4][4];
#pragma unroll
            for (int ky = 0; ky < 4; ++ky)
#pragma unroll
                for (int kx = 0; kx < 4; ++kx) v[ky][kx] = __ldg(rp + ty[ky] + ix[kx]);
            float sy = 0.f, sy_dx = 0.f, sy_dy = 0.f;
#pragma unroll
            for (int ky = 0; ky < 4; ++ky) {
                float sx = 0.f, sx_d = 0.f;
#pragma unroll
                for (int kx = 0; kx < 4; ++kx) {
                    sx = fmaf(wx[kx], v[ky][kx], sx);
                    if (MODE == 1) sx_d = fmaf(ex[kx], v[ky][kx], sx_d);
                }
                sy = fmaf(wy[ky], sx, sy);
                if (MODE == 1) {
                    sy_dx = fmaf(wy[ky], sx_d, sy_dx);
                    sy_dy = fmaf(ey[ky], sx, sy_dy);
                }
            }
            s[k] = sy;
            if (MODE == 1) {
                s_dx[k] = sy_dx;
                s_dy[k] = sy_dy;
            }
        };
        int held = 0;
        for (int z = z0; z < min(z0 + L, D); ++z) {
            const float pz = (float)z + dz;
            const int bz = (int)floorf(pz);
            if (z == z0 || (bz != held && bz != held + 1)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) plane(bz + k - 1, k);
            } else if (bz != held) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    s[k] = s[k + 1];
                    if (MODE == 1) {
                        s_dx[k] = s_dx[k + 1];
                        s_dy[k] = s_dy[k + 1];
                    }
                }
                plane(bz + 2, 3);
            }
            held = bz;
            float v = 0.f, gx_ = 0.f, gy_ = 0.f, gz_ = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float wz = cr(pz - (float)(bz + k - 1));
                v = fmaf(wz, s[k], v);
                if (MODE == 1) {
                    gx_ = fmaf(wz, s_dx[k], gx_);
                    gy_ = fmaf(wz, s_dy[k], gy_);
                    gz_ = fmaf(dcr(pz - (float)(bz + k - 1)), s[k], gz_);
                }
            }
            const long long o = (long long)t * nv + ((long long)z * H + y) * W + x;
            if (MODE == 0) {
                dst[o] = v;
            } else {
                const double gg = g[o];
                acc[0] += gg * gx_;
                acc[1] += gg * gy_;
                acc[2] += gg * gz_;
            }
        }
    }
    if (MODE == 1) {
        __shared__ double red[3][kDriftThreads];
#pragma unroll
        for (int a = 0; a < 3; ++a) red[a][threadIdx.x] = acc[a];
        __syncthreads();
        for (int s2 = kDriftThreads / 2; s2 > 0; s2 >>= 1) {
            if (threadIdx.x < s2)
#pragma unroll
                for (int a = 0; a < 3; ++a) red[a][threadIdx.x] += red[a][threadIdx.x + s2];
            __syncthreads();
        }
        if (threadIdx.x < 3) atomicAdd(out + 3 * t + threadIdx.x, red[threadIdx.x][0]);
    }
}

// ---------------------------------------------------------------------------
// Temporal adjoint, one thread per subvoxel of the single block. FP32 with
// compensated (Kahan) sums over t: FP64 arithmetic runs at a small fraction of
// the FP32 rate on this GPU and would make this HBM-sized pass compute-bound.
struct KSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// Adjoint of TRAC with ITC 1 (kernel.cu:437-555) for one subvoxel; r, I its
// radiality and intensity series (stride V), m and IW the level-0 mean and
// intensity weight. The forward bins the series in place level after level
// (entry t < nB - k becomes the mean of entries tk .. tk + k - 1, entry 0
// reading itself as 0, entries past the series reading 0; the rest keep their
// values) and sums per level AB (reset) and ABC / ABCD, CD, AC, BD, AD, BC (not
// reset) around m; out = sum_l |C_l| / nB_l. Reverse mode over the levels with
// O(T) memory per subvoxel: one forward sweep gives each level's sums, hence
// d out / d(each level's partial sums) as suffix sums over the levels; then,
// from the deepest level up, the level's array state is replayed from r into
// S (the dL/dI buffer, free until the end) and the gradient with respect to
// that state is formed in place in Gd (the dL/dS buffer): the level's own
// sums' derivatives plus its transposed binning of the next level's gradient,
// walking the entries downwards so that every entry a later bin reads is still
// the next level's. The level-0 mean takes minus the sum of all direct terms
// over T. FP32 with compensated sums in the forward sweep.
constexpr int kMaxLevels = 32;

__device__ void trac_itc1_adjoint(const float* r, const float* I, long long V, int T, int k, int iw, int renorm,
                                  int poscon, float g, float m, float IW, float* Gd, float* S) {
    float Cl[kMaxLevels], ABl[kMaxLevels], CDa[kMaxLevels], ACa[kMaxLevels], BDa[kMaxLevels], ADa[kMaxLevels],
        BCa[kMaxLevels];
    int nbl[kMaxLevels];
    const float invk = 1.f / (float)k;
    // binning of one level in place (the forward's order)
    auto bin_level = [&](int nb) {
        for (int t = 0; t < nb - k; ++t) {
            float nv = 0.f;
            if (t * k < nb)
                for (int j = 0; j < k; ++j) {
                    const int src = t * k + j;
                    const float rv = (src == t || src >= T) ? 0.f : S[(long long)src * V];
                    nv += rv / (float)k;
                }
            S[(long long)t * V] = nv;
        }
    };
    for (int t = 0; t < T; ++t) S[(long long)t * V] = r[(long long)t * V];
    KSum ABC, ABCD, CD, AC, BD, AD, BC;
    float out_raw = 0.f;
    int L = 0, nB = T;
    while (nB > k && L < kMaxLevels) {
        KSum AB;
        for (int t = 0; t < nB - k; ++t) {
            const float A = S[(long long)t * V] - m, B = S[(long long)(t + 1) * V] - m;
            AB.add(A * B);
            if (k >= 3) {
                const float C = S[(long long)(t + 2) * V] - m;
                if (k == 3) ABC.add(A * B * C);
                if (k == 4) {
                    const float D = S[(long long)(t + 3) * V] - m;
                    ABCD.add(A * B * C * D);
                    CD.add(C * D);
                    AC.add(A * C);
                    BD.add(B * D);
                    AD.add(A * D);
                    BC.add(B * C);
                }
            }
        }
        bin_level(nB);
        const float C = k == 2 ? AB.s : (k == 3 ? ABC.s : ABCD.s - AB.s * CD.s - AC.s * BD.s - AD.s * BC.s);
        Cl[L] = C;
        ABl[L] = AB.s;
        CDa[L] = CD.s;
        ACa[L] = AC.s;
        BDa[L] = BD.s;
        ADa[L] = AD.s;
        BCa[L] = BC.s;
        nbl[L] = nB;
        out_raw += fabsf(C) / (float)nB;
        ++L;
        nB = nB / k;
    }
    // d out / d(partial sums of each level): suffix sums over the levels
    float wM[kMaxLevels], wAB[kMaxLevels], wCD[kMaxLevels], wAC[kMaxLevels], wBD[kMaxLevels], wAD[kMaxLevels],
        wBC[kMaxLevels];
    {
        float ss = 0.f, scd = 0.f, sac = 0.f, sbd = 0.f, sad = 0.f, sbc = 0.f;
        for (int l = L - 1; l >= 0; --l) {
            const float sl = (Cl[l] > 0.f ? 1.f : (Cl[l] < 0.f ? -1.f : 0.f)) / (float)nbl[l];
            ss += sl;
            scd -= sl * ABl[l];
            sac -= sl * BDa[l];
            sbd -= sl * ACa[l];
            sad -= sl * BCa[l];
            sbc -= sl * ADa[l];
            wM[l] = k == 2 ? sl : ss;
            wAB[l] = -sl * CDa[l];
            wCD[l] = scd;
            wAC[l] = sac;
            wBD[l] = sbd;
            wAD[l] = sad;
            wBC[l] = sbc;
        }
    }
    for (int t = 0; t < T; ++t) Gd[(long long)t * V] = 0.f;
    float dm = 0.f;
    for (int l = L - 1; l >= 0; --l) {
        // replay level l's state
        for (int t = 0; t < T; ++t) S[(long long)t * V] = r[(long long)t * V];
        int nb = T;
        for (int j = 0; j < l; ++j) {
            bin_level(nb);
            nb /= k;
        }
        const int N = nb - k;
        auto sv = [&](int t) { return S[(long long)t * V] - m; };
        for (int p = T - 1; p >= 0; --p) {
            // transposed binning: entries at or past N keep their value, entry
            // p feeds bin p / k
            float gp = p >= N ? Gd[(long long)p * V] : 0.f;
            const int tb = p / k;
            if (tb < N && tb * k < nb && p != tb) gp += Gd[(long long)tb * V] * invk;
            // this level's sums: the products starting at t = p - q hold entry p
            float dp = 0.f;
            for (int q = 0; q < k; ++q) {
                const int t = p - q;
                if (t < 0 || t >= N) continue;
                const float A = sv(t), B = sv(t + 1);
                if (k == 2) {
                    dp += wM[l] * (q == 0 ? B : A);
                } else if (k == 3) {
                    const float C = sv(t + 2);
                    dp += wM[l] * (q == 0 ? B * C : (q == 1 ? A * C : A * B));
                } else {
                    const float C = sv(t + 2), D = sv(t + 3);
                    if (q == 0) dp += wM[l] * B * C * D + wAB[l] * B + wAC[l] * C + wAD[l] * D;
                    if (q == 1) dp += wM[l] * A * C * D + wAB[l] * A + wBD[l] * D + wBC[l] * C;
                    if (q == 2) dp += wM[l] * A * B * D + wCD[l] * D + wAC[l] * A + wBC[l] * B;
                    if (q == 3) dp += wM[l] * A * B * C + wCD[l] * C + wBD[l] * B + wAD[l] * A;
                }
            }
            Gd[(long long)p * V] = gp + dp;
            dm += dp;
        }
    }
    const float invT = 1.f / (float)T;
    const float scale = iw ? IW : 1.f;
    for (int t = 0; t < T; ++t) {
        const float rv = r[(long long)t * V], Iv = I[(long long)t * V];
        float gr = g * (scale * (Gd[(long long)t * V] - dm * invT) + (iw ? out_raw * Iv * invT : 0.f));
        const float gi = iw ? g * out_raw * rv * invT : 0.f;
        if (renorm) gr *= 0.5f;
        if (poscon && !(rv > 0.f)) gr = 0.f;
        Gd[(long long)t * V] = gr;
        S[(long long)t * V] = Iv > 0.f ? gi : 0.f;
    }
}

__global__ void temporal_adjoint_kernel(const BlockDev* __restrict__ blocks, const float* __restrict__ rad,
                                        const float* __restrict__ inten, const float* __restrict__ gmap, int T,
                                        int method, int itc, int order, int iw, int renorm, int poscon,
                                        float* __restrict__ gS, float* __restrict__ gI, long long nmap,
                                        unsigned long long* err) {
    const BlockDev& B = blocks[0];
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= B.vox) return;
    const long long V = B.vox;
    const long long nx = B.nreg[0], ny = B.nreg[1];
    const long long x = v % nx, y = (v / nx) % ny, z = v / (nx * ny);
    const long long gidx = B.out_offset + x * B.out_stride[0] + y * B.out_stride[1] + z * B.out_stride[2];
    if (!in_range(gidx, nmap, err, 5)) return;
    const float g = gmap[gidx];
    const float* r = rad + v;
    const float* I = inten + v;
    // first pass: sums
    KSum ms, iws;
    bool finite = isfinite(g);
    for (int t = 0; t < T; ++t) {
        const float rv = r[t * V];
        finite = finite && isfinite(rv);
        ms.add(rv);
        iws.add(rv * I[t * V]);
    }
    if (!finite) {
        for (int t = 0; t < T; ++t) {
            gS[t * V + v] = 0.f;
            gI[t * V + v] = 0.f;
        }
        return;
    }
    const float invT = 1.f / (float)T;
    if (method == 0 || method == 2) {
        // TRM (kernel.cu:332-366): the first argmax of the seeded maximum carries
        // the derivative. TRPPM (kernel.cu:372-419): d/dr_t of ((sum r+)^2 +
        // sum r+^2) / 2 / count is (sum r+ + r_t) / count where r_t > 0.
        int arg = -1;
        float mip = 0.f;
        KSum s1, s2, si;
        for (int t = 0; t < T; ++t) {
            const float rv = r[t * V], Iv = I[t * V];
            if (method == 0) {
                const float val = iw ? rv * Iv : rv;
                if (val > mip) {
                    mip = val;
                    arg = t;
                }
            } else {
                const float rp = fmaxf(rv, 0.f);
                s1.add(rp);
                s2.add(rp * rp);
                si.add(Iv);
            }
        }
        const float count = fmaxf(0.5f * (float)T * (float)(T + 1), 1.f);
        const float scale = iw ? si.s * invT : 1.f;
        const float pps = 0.5f * (s1.s * s1.s + s2.s) / count;
        for (int t = 0; t < T; ++t) {
            const float rv = r[t * V], Iv = I[t * V];
            float gr = 0.f, gi = 0.f;
            if (method == 0) {
                if (t == arg) {
                    gr = g * (iw ? Iv : 1.f);
                    gi = iw ? g * rv : 0.f;
                }
            } else {
                gr = rv > 0.f ? g * (s1.s + rv) / count * scale : 0.f;
                gi = iw ? g * pps * invT : 0.f;
            }
            if (renorm) gr *= 0.5f;
            if (poscon && !(rv > 0.f)) gr = 0.f;
            gS[t * V + v] = gr;
            gI[t * V + v] = Iv > 0.f ? gi : 0.f;
        }
        return;
    }
    if (method == 3 && itc == 1) {
        trac_itc1_adjoint(r, I, V, T, order, iw, renorm, poscon, g, ms.s * invT, iws.s * invT, gS + v, gI + v);
        return;
    }
    const float m = ms.s * invT;
    const float IW = iws.s * invT;
    const float scale_iw = iw ? IW : 1.f;
    float C = 0.f, AB = 0.f, CD = 0.f, AC = 0.f, BD = 0.f, AD = 0.f, BC = 0.f;
    // sum over s of dC/da_s, in closed form from window sums of the same pass:
    // order 2: S0 + S1; order 3: P12 + P02 + P01; order 4: the four triple sums
    // minus each lag's three single-sum x pair-sum terms
    float sumd = 0.f;
    const int N = T - order;
    if (method == 3) {
        KSum c1, s4, ab, cd, ac, bd, ad, bc, s0, s1, s2, s3, p012, p013, p023, p123;
        for (int t = 0; t < N; ++t) {
            const float A = r[t * V] - m, Bv = r[(t + 1) * V] - m;
            s0.add(A);
            s1.add(Bv);
            if (order == 2) c1.add(A * Bv);
            if (order >= 3) {
                const float Cv = r[(t + 2) * V] - m;
                s2.add(Cv);
                if (order == 3) {
                    c1.add(A * Bv * Cv);
                    ab.add(A * Bv);
                    ac.add(A * Cv);
                    bc.add(Bv * Cv);
                }
                if (order == 4) {
                    const float Dv = r[(t + 3) * V] - m;
                    s3.add(Dv);
                    s4.add(A * Bv * Cv * Dv);
                    ab.add(A * Bv);
                    cd.add(Cv * Dv);
                    ac.add(A * Cv);
                    bd.add(Bv * Dv);
                    ad.add(A * Dv);
                    bc.add(Bv * Cv);
                    p012.add(A * Bv * Cv);
                    p013.add(A * Bv * Dv);
                    p023.add(A * Cv * Dv);
                    p123.add(Bv * Cv * Dv);
                }
            }
        }
        C = c1.s;
        AB = ab.s, CD = cd.s, AC = ac.s, BD = bd.s, AD = ad.s, BC = bc.s;
        if (order == 4) C = s4.s - AB * CD - AC * BD - AD * BC;
        if (order == 2) {
            sumd = s0.s + s1.s;
        } else if (order == 3) {
            sumd = BC + AC + AB;
        } else {
            sumd = (p123.s + p023.s + p013.s + p012.s) - (s1.s * CD + s2.s * BD + s3.s * BC) -
                   (s0.s * CD + s3.s * AC + s2.s * AD) - (s3.s * AB + s0.s * BD + s1.s * AD) -
                   (s2.s * AB + s1.s * AC + s0.s * BC);
        }
    }
    // dC/da_s for every s, then centring (dC/dr_t = dC/da_t - mean_s dC/da_s)
    auto dCda = [&](int s) -> float {
        float d = 0.f;
        auto a = [&](int t) -> float { return (t >= 0 && t < T) ? r[t * V] - m : 0.f; };
        for (int l = 0; l < order; ++l) {
            const int t0 = s - l;  // the product starting at t0 contains a_s at lag l
            if (t0 < 0 || t0 >= N) continue;
            if (order == 2) d += a(t0 + 1 - l);
            else if (order == 3) {
                float p = 1.f;
                for (int q = 0; q < 3; ++q)
                    if (q != l) p *= a(t0 + q);
                d += p;
            } else {
                const float A = a(t0), Bv = a(t0 + 1), Cv = a(t0 + 2), Dv = a(t0 + 3);
                if (l == 0) d += Bv * Cv * Dv - Bv * CD - Cv * BD - Dv * BC;
                if (l == 1) d += A * Cv * Dv - A * CD - Dv * AC - Cv * AD;
                if (l == 2) d += A * Bv * Dv - Dv * AB - A * BD - Bv * AD;
                if (l == 3) d += A * Bv * Cv - Cv * AB - Bv * AC - A * BC;
            }
        }
        return d;
    };
    const float mean_d = sumd * invT;
    const float sgn = C > 0.f ? 1.f : (C < 0.f ? -1.f : 0.f);
    const float aC = fabsf(C);
    for (int t = 0; t < T; ++t) {
        const float rv = r[t * V], Iv = I[t * V];
        float gr, gi;
        if (method == 1) {
            gr = g * (iw ? Iv : 1.f) * invT;
            gi = iw ? g * rv * invT : 0.f;
        } else {
            gr = g * (sgn * invT * scale_iw * (dCda(t) - mean_d) + (iw ? aC * invT * Iv * invT : 0.f));
            gi = iw ? g * aC * invT * rv * invT : 0.f;
        }
        if (renorm) gr *= 0.5f;
        if (poscon && !(rv > 0.f)) gr = 0.f;
        gS[t * V + v] = gr;
        gI[t * V + v] = Iv > 0.f ? gi : 0.f;
    }
}

// ---------------------------------------------------------------------------
// Radiality adjoint, on the forward's plan and tiles (16 x kTileRows columns, one
// per thread, two halves of a column in a register pair; see radiality.cu). Every
// (tile, time point) recomputes the interpolated gradient at each ring sample and
// pushes the derivative back through the passes, transposed and in reverse order:
//
//   point   with the forward's scaled frame values (dot, cp, E, c2 = cp^2 + E^2, g2 =
//           dot^2 + c2, s = sqrt(c2 / g2)) and K = dL/ds,
//             ds = ((1 - s^2) (cp dcp + E dE) - s^2 dot ddot) / sqrt(c2 g2),
//           so with k = K / sqrt(c2 g2), b = s^2 k, m = k - b:
//             dE = m E, dZ = m cp - kappa b dot, -dP = kappa m cp + b dot;
//   third   transposed along the innermost axis in registers, over the points of a
//           pair;
//   second  transposed along x: the lanes of a row exchange their columns through
//           shared memory, plane by plane, sorted by x phase. Lane u then
//           gathers coarse cell u: for each phase and tap one shift of the row, so the
//           weights are uniform and no two lanes add to the same place;
//   first   transposed along the mid axis as a gather over the tile's rows, once per
//           ring value of that axis;
//   stencil transposed as a gather over the cells' 3^3 neighbourhood, and one global
//           atomic add per input voxel of the tile.
//
// Where two lanes of a warp updated the same shared-memory rows in turn (the second
// pass along y, two phases for magnifications above 2), short-scoreboard and barrier
// waits kept the FMA pipe at 43 %.
__device__ __forceinline__ float4 f4fma(float s, float4 a, float4 c) {
    return make_float4(fmaf(s, a.x, c.x), fmaf(s, a.y, c.y), fmaf(s, a.z, c.z), fmaf(s, a.w, c.w));
}

// Ring samples whose gradient nearly vanishes or nearly follows the ring direction
// amplify the rounding of the interpolated gradient into the derivative, by |g|^2 of
// the column over |g| |g_perp| of the sample. With the passes in the plan's order single
// voxels of dL/dI came out up to 5e-3 away from those with passes along x, then y, then
// z, on one of four drift series: neither is the more accurate (on a crop at 4 x 4 x 2
// both are 2.1e-5 from 64 bits), but dL/dI is to be the same whatever the plan. So below
// a bound on c2 g2, this factor times the square of the sum of |g|^2 over four cells of
// the column, the point loop takes the derivative at the bound, which costs no operation
// more than the guard against 0 does, and marks the subvoxel; fix_marked then adds what
// is missing, from the derivative in the fixed order. Samples under the bound are ten in a
// million on a series of 60 volumes of 64^3 at mag 2 (82 thousand; correcting them takes
// 0.3 of the pair's 42.2 ms), and two of a subvoxel's 62 where a whole volume is a ramp
// along a ring direction (12 volumes of 64^3 then take 20 to 29 ms instead of 6).
constexpr float kSampleBound = 6e-9f;

// The derivative of one sample's sine term with respect to (-P, E, Z), times K.
struct Derivative {
    float P, E, Z;
};
__device__ __forceinline__ Derivative sample_derivative(float P, float E, float Z, float h, float c, float wun, float un,
                                                        float gS, float inv) {
    const float dot = fmaf(c, Z, __fmul_rn(h, P)), cp = fmaf(h, Z, __fmul_rn(-c, P));
    const float c2 = fmaf(cp, cp, __fmul_rn(E, E)), sn = c2 * inv;
    const float k = flip_sign(wun * fmaf(sn, -un, 1.f), dot) * gS * inv;
    const float b = sn * sn * k, m = k - b;
    return Derivative{fmaf(c, m * cp, h * (b * dot)), m * E, fmaf(h, m * cp, -c * (b * dot))};
}

// What the correction needs of a tile and time point.
struct FixTile {
    const FwdParams* p;
    const float4* fix;
    const float4* gt;  // gradient planes [NQ][nv][nu]
    float4* gu;        // dL/dU planes [NQ][ty][nu]
    const float* wx;   // the x values' tap weights
    const float* wm;   // the tile rows' mid weights and first tap cells
    const int* base;
    const float* gS;
    long long zstride;
};

// Four taps along x (weights w) at innermost cell c of a row of planes [quad][rows][nu].
__device__ __forceinline__ float along_x(const float4* row, int quad, int c, const float* w) {
    const float* g = reinterpret_cast<const float*>(row + (c >> 2) * quad) + (c & 3);
    return fmaf(w[3], g[12], fmaf(w[2], g[8], fmaf(w[1], g[4], w[0] * g[0])));
}

// A store that the compiler knows to be to shared memory: through a generic pointer, in a
// function that is called, it counts as one that may reach the caller's locals.
__device__ __forceinline__ void store_shared(float* p, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "f"(v) : "memory");
}

// The correction of a pair's samples below the bound: each half of the warp takes its own
// row's columns, one subvoxel after another. Of this lane's column, u0, ax, bound and sbase are its first x cell, x
// weight index, bound and place in the stacks, marked its subvoxels that have such a
// sample. Adds to dL/dU what the derivative in the fixed order exceeds the one at the bound
// by: u = |u| (h x' + c z), x' = (ca, sb) in the x-y plane, the gradient interpolated along
// x, then y, turned by (ca, sb), then along z; a half's lanes 4 o + i take plane o of z and
// row i of y. The point loop's frame is this one times scale. Nothing here depends on other tiles or
// launches. A call takes 1.9 us, out of line so that the point loop keeps its registers
// (60 volumes of 64^3 at mag 2: 1 pair of a warp in 115 comes here).
template <int MZ, int CZ>
__device__ __noinline__ void fix_marked(const FixTile& f, int pair, int u0, int ax, float bound, long long sbase,
                                        unsigned int marked) {
    constexpr int NQ = tile_quads(CZ);
    const unsigned int full = 0xffffffffu;
    const FwdParams& p = *f.p;
    const int lane = threadIdx.x & 31, o = (lane >> 2) & 3, i = lane & 3;
    const bool y_inner = p.ax1 == 2;
    const float4 r3 = __ldg(p.utab + p.u_pair + 4 * pair + 3);
    const int half = lane & 16, row = threadIdx.x / kTileX;
    const float* wm = f.wm + 4 * row;
    // a half that has no column or subvoxel left goes along with the other's, its own kept out
    for (unsigned int open = (__ballot_sync(full, marked != 0) >> half) & 0xffff; __any_sync(full, open != 0);
         open &= open - 1) {
        const int src = open ? half + __ffs(open) - 1 : lane;
        const int su = __shfl_sync(full, u0, src);
        const float* wx = f.wx + 4 * __shfl_sync(full, ax, src);
        const float least = __shfl_sync(full, bound, src);
        const long long at = __shfl_sync(full, sbase, src);
        const unsigned int subvoxels = __shfl_sync(full, marked, src);
        for (unsigned int left = open ? subvoxels : 0; __any_sync(full, left != 0); left &= left - 1) {
            const int z = left ? __ffs(left) - 1 : 0;
            const float gS = left ? f.gS[at + z * f.zstride] : 0.f;
#pragma unroll 1
            for (int qi = __float_as_int(r3.x); qi < __float_as_int(r3.y); ++qi) {
                const float4 fr = __ldg(f.fix + 2 * qi), wt = __ldg(f.fix + 2 * qi + 1);
                const float4 c = __ldg(p.utab + p.u_pt + 3 * qi + 2);
                // weights along the innermost axis: every second word of their record
                const float* wi = reinterpret_cast<const float*>(p.utab + p.u_wz + 2 * (__float_as_int(c.x) + z % MZ));
                const int w0 = z / MZ + ((__float_as_int(c.y) >> (z % MZ)) & 1);
                float v[3];
                {
                    const float4* row0 = f.gt + (f.base[row] + (y_inner ? o : i)) * p.NU + su;
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        v[d] = along_x(row0 + (d == 0 ? 0 : (d == 1) == y_inner ? 2 : 1) * NQ * p.NV * p.NU, p.NV * p.NU,
                                       w0 + (y_inner ? i : o), wx);
                }
                // the sums over y of each z, then over z
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass) {
                    float acc[3];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float w = y_inner == (pass == 0) ? __ldg(wi + 2 * k) : wm[k];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const float u = __shfl_sync(full, v[d], half + (pass == 0 ? 4 * o + k : 4 * k));
                            acc[d] = k ? fmaf(w, u, acc[d]) : w * u;
                        }
                    }
                    v[0] = pass == 0 ? fmaf(acc[1], fr.y, __fmul_rn(acc[0], fr.x)) : acc[0];
                    v[1] = pass == 0 ? fmaf(acc[1], fr.x, __fmul_rn(acc[0], -fr.y)) : acc[1];
                    v[2] = acc[2];
                }
                const float P = v[0], E = v[1], Z = v[2], hh = fr.z, cc = fr.w;
                const float dot = fmaf(cc, Z, __fmul_rn(hh, P)), cp = fmaf(hh, Z, __fmul_rn(-cc, P));
                const float c2 = fmaf(cp, cp, __fmul_rn(E, E)), xx = c2 * fmaf(dot, dot, c2);
                const float scale = wt.z, s4 = scale * scale * scale * scale;
                const Derivative e = sample_derivative(P, E, Z, hh, cc, wt.x, wt.y, gS, rsqrt_approx(fmaxf(xx, kGuard)));
                const Derivative q = sample_derivative(P, E, Z, hh, cc, wt.x, wt.y, gS,
                                                       scale * scale * rsqrt_approx(fmaxf(xx * s4, least)));
                const float dP = q.P - e.P, dE = e.E - q.E;
                const float dG[3] = {fmaf(dE, -fr.y, dP * fr.x), fmaf(dE, fr.x, dP * fr.y), e.Z - q.Z};
                if (left) {
                    const int w = w0 + o;
                    const float spread = __ldg(wi + 2 * o) * wx[i];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int k = d == 0 ? 0 : (d == 1) == y_inner ? 2 : 1;
                        float* g = reinterpret_cast<float*>(f.gu + ((k * NQ + (w >> 2)) * p.TY + row) * p.NU + su + i) +
                                   (w & 3);
                        store_shared(g, fmaf(dG[d], spread, *g));
                    }
                }
                __syncwarp();
            }
        }
    }
}

template <int MZ, int CZ, int UN>
__global__ void __maxnreg__(kAdjRegs)
    radiality_adjoint_kernel(const __grid_constant__ FwdParams p, const __grid_constant__ AdjParams a,
                             const __grid_constant__ UTab<UN> ut) {
    constexpr int CH = CZ / 2;
    constexpr int HZ = MZ * CH;
    constexpr int FZ = MZ * CZ;
    constexpr int NH = CH + 4;
    constexpr int NW = CZ + 4;
    constexpr int NQ = tile_quads(CZ);
    static_assert(FZ <= 32, "a column's marks fit a word");
    extern __shared__ float4 smem4[];

    const int NU = p.NU, NV = p.NV, TY = p.TY;
    const int gplane = NQ * NV * NU, uplane = NQ * TY * NU;
    // Shared layout: [G][dL/dG][U, sharing its place with the input tile and the
    // intensity's cells][dL/dU][exchange rows][lane tables]
    float4* gt = smem4;
    float4* gg = gt + 3 * gplane;
    float4* ut4 = gg + 3 * gplane;
    float4* gu = ut4 + p.u_region;
    float4* ex = gu + 3 * uplane;
    float* inp = reinterpret_cast<float*>(ut4);
    float4* icell = ut4;
    const int mx = p.mag[0], my = p.mag[1];
    const int a1 = p.ax1, a2 = p.ax2;
    // exchange row: four zeros, then per x phase the tile's coarse cells and four zeros
    const int nxc = adj_cells(mx), exw = 4 + mx * nxc;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int warp = tid >> 5, half = (tid >> 4) & 1;
    float4* ex_warp = ex + warp * (2 * NQ * exw);  // [quad][row of the warp][exw]
    float* tab = reinterpret_cast<float*>(ex + (nthr >> 5) * (2 * NQ * exw));
    __shared__ unsigned int s_item;
    __shared__ int2 s_row[kMaxThreads / kTileX];
    __shared__ int s_base[kMaxThreads / kTileX];
    __shared__ alignas(16) float s_weight[kMaxThreads / kTileX * 4];

    const int xf = tid & (kTileX - 1);
    const int q = tid / kTileX;
    for (int i = tid; i < p.lane_words; i += nthr) tab[i] = p.lane[i];
    const float* wx = tab + p.l_wx;
    const int* offx = reinterpret_cast<const int*>(tab + p.l_offx);
    const float* wy = tab + p.l_wm;
    const int* offy = reinterpret_cast<const int*>(tab + p.l_offm);
    const int NIX = p.NIX, NIY = p.NIY, NIZ = p.NIZ, R = p.R;
    const int nin = NIX * NIY * NIZ;
    const FastDiv div_nu(NU), div_nv(NV), div_nix(NIX), div_nixy(NIX * NIY);
    const float* in = static_cast<const float*>(p.in);
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);

    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(p.work_counter, 1u);
        __syncthreads();
        const long long item = s_item;
        if (item >= p.nitems) break;
        const int tile_i = (int)(item % p.ntiles);
        const int chunk = (int)(item / p.ntiles);
        const TileDesc td = p.tiles[tile_i];
        const BlockDev& B = p.blocks[td.block];
        const int bw = B.size[0], bh = B.size[a1], bd = B.size[a2];
        const int X0 = B.lo[0] + td.t[0] * kTileX;
        const int Y0 = B.lo[a1] + td.t[a1] * TY;
        const int Z0 = (B.lo[a2] / MZ) * MZ + td.t[a2] * FZ;
        const int cx0 = floordiv(X0, mx) - 2;
        const int cy0 = floordiv(Y0, my) - 2;
        const int cz0 = Z0 / MZ - 2;
        const int X = X0 + xf, Y = Y0 + q;
        const int xi = floordiv(X, mx), xr = X - xi * mx;
        if (xf == 0) {
            const int yi = floordiv(Y, my);
            s_row[q] = make_int2(yi - cy0 - 2, Y - yi * my);  // first tap row at offset 0, phase
        }
        // exchange slots that no lane of this tile fills read as zero
        for (int i = tid & 31; i < 2 * NQ * exw; i += 32) ex_warp[i] = zero4;
        const int ex_put = half * exw + xr * nxc + (xi - cx0 - 2) + 4;
        const bool in_tile = X < B.hi[0] && Y < B.hi[a1];
        const long long V = B.vox;
        const long long ystride = a1 == 1 ? B.nreg[0] : (long long)B.nreg[0] * B.nreg[1];
        const long long zstride = a1 == 1 ? (long long)B.nreg[0] * B.nreg[1] : B.nreg[0];
        const int zlo = B.lo[a2], zhi = B.hi[a2];
        const long long v0 = (long long)(Y - B.lo[a1]) * ystride + (X - B.lo[0]) + (Z0 - zlo) * zstride;

        const int t0 = p.t_lo + chunk * p.t_chunk;
        const int t1 = min(p.t_hi > 0 ? p.t_hi : p.T, t0 + p.t_chunk);
        for (int t = t0; t < t1; ++t) {
            const long long sbase = B.stack_off + (long long)(t - p.stack_t0) * V + v0;
            const long long tbase = (long long)t * p.D * p.H * p.W;
            // dL/dS or dL/dI of this thread's subvoxels
            auto stack_value = [&](const float* st, int z) -> float {
                const int Z = Z0 + z;
                const long long i = sbase + z * zstride;
                return in_tile && Z >= zlo && Z < zhi && in_range(i, a.n_stack, a.err, 9) ? st[i] : 0.f;
            };
            auto global_row = [&](int iy, int iz) -> long long {
                const int by = B.origin[a1] + clampi(cy0 - R + iy, 0, bh - 1);
                const int bz = B.origin[a2] + clampi(cz0 - R + iz, 0, bd - 1);
                return tbase + (a1 == 1 ? (long long)bz * p.H + by : (long long)by * p.H + bz) * p.W + B.origin[0];
            };
            __syncthreads();  // the previous time point is done with the input tile's place
            for (int r = q, iy = q, iz = 0; r < NIY * NIZ; r += TY, iy += TY) {
                while (iy >= NIY) {
                    iy -= NIY;
                    ++iz;
                }
                const long long rowg = global_row(iy, iz);
                for (int ix = xf; ix < NIX; ix += kTileX) {
                    const long long gi = rowg + clampi(cx0 - R + ix, 0, bw - 1);
                    inp[r * NIX + ix] = in_range(gi, a.n_in, a.err, 8) ? __ldg(in + gi) : 0.f;
                }
            }
            __syncthreads();
            for (int c = tid; c < gplane; c += nthr) {
                const int row = div_nu(c), u = c - row * NU;
                const int wq = div_nv(row), v = row - wq * NV, w0 = wq * 4;
                const int cu = cx0 + u, cv = cy0 + v, cw = cz0 + w0;
                float g[3][4];
#pragma unroll
                for (int k = 0; k < 3; ++k)
#pragma unroll
                    for (int w = 0; w < 4; ++w) g[k][w] = 0.f;
                if (cu >= 0 && cu < bw && cv >= 0 && cv < bh && cw + 3 >= 0 && cw < bd) {
                    const float* base = inp + (v + R) * NIX + (u + R);
                    gradient4<true>(p.grad_mode, p.gr, [&](int k) { return base + (w0 + R + k) * (NIY * NIX); }, NIX, g,
                                    a1 == 2);
#pragma unroll
                    for (int w = 0; w < 4; ++w)
                        if (cw + w < 0 || cw + w >= bd) g[0][w] = g[1][w] = g[2][w] = 0.f;
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    gt[k * gplane + c] = make_float4(g[k][0], g[k][1], g[k][2], g[k][3]);
                    gg[k * gplane + c] = zero4;
                }
            }
            float2 gS[HZ];
#pragma unroll
            for (int z = 0; z < HZ; ++z) gS[z] = make_float2(stack_value(a.gS, z), stack_value(a.gS, z + HZ));

            // x pass transposed of one plane: every lane lays down its column, then lane u
            // gathers cell u of its row (and a second one where a row has more than 16
            // cells) and adds it to, or stores it in, dst
            auto x_transpose = [&](const float2(&g)[NH], int xval, int mask, float4* dst, bool add) {
                __syncwarp();  // the row's previous readers
#pragma unroll
                for (int wq = 0; wq < NQ; ++wq)
                    ex_warp[ex_put + wq * (2 * exw)] =
                        make_float4(get_halves<CH>(g, wq * 4), get_halves<CH>(g, wq * 4 + 1),
                                    get_halves<CH>(g, wq * 4 + 2), get_halves<CH>(g, wq * 4 + 3));
                __syncwarp();
                for (int u0 = 0; u0 < NU; u0 += kTileX) {
                    const float4* from = ex_warp + half * exw + 4 + min(u0 + xf, NU - 1);
                    float2 lo[NQ], hi[NQ];
#pragma unroll
                    for (int wq = 0; wq < NQ; ++wq) lo[wq] = hi[wq] = make_float2(0.f, 0.f);
                    for (int r = 0; r < mx; ++r) {
                        const float4 wa = uget(ut, p.utab, p.u_wx + 2 * (xval * mx + r));
                        const float4 wb = uget(ut, p.utab, p.u_wx + 2 * (xval * mx + r) + 1);
                        const float4* src = from + r * nxc - ((mask >> r) & 1);
#pragma unroll
                        for (int wq = 0; wq < NQ; ++wq) {
                            const float4* sw = src + wq * (2 * exw);
                            const float4 g0 = sw[0], g1 = sw[-1], g2 = sw[-2], g3 = sw[-3];
                            lo[wq] = fma2(hi2(wb), lo2(g3), fma2(lo2(wb), lo2(g2), fma2(hi2(wa), lo2(g1), fma2(lo2(wa), lo2(g0), lo[wq]))));
                            hi[wq] = fma2(hi2(wb), hi2(g3), fma2(lo2(wb), hi2(g2), fma2(hi2(wa), hi2(g1), fma2(lo2(wa), hi2(g0), hi[wq]))));
                        }
                    }
                    if (u0 + xf < NU) {
                        float4* d = dst + q * NU + u0 + xf;
#pragma unroll
                        for (int wq = 0; wq < NQ; ++wq) {
                            const float4 o4 = add ? d[wq * (TY * NU)] : zero4;
                            d[wq * (TY * NU)] = make_float4(o4.x + lo[wq].x, o4.y + lo[wq].y, o4.z + hi[wq].x, o4.w + hi[wq].y);
                        }
                    }
                }
            };
            // first pass transposed: dL/dU planes [y][u] into cells [v][u]. One thread takes
            // a column of rows; their first tap cell steps by 0 or 1, so a window of four
            // cells slides along and every cell is written by one thread (testing all rows
            // for every cell took 15 % of the kernel).
            auto mid_transpose = [&](const float4* src, float4* dst, int planes) {
                for (int c = tid; c < planes * NQ * NU; c += nthr) {
                    const int pw = div_nu(c), u = c - pw * NU;
                    const float4* col = src + pw * TY * NU + u;
                    float4* cell = dst + (pw * NV + s_base[0]) * NU + u;
                    float2 l0 = make_float2(0.f, 0.f), h0 = l0, l1 = l0, h1 = l0, l2 = l0, h2 = l0, l3 = l0, h3 = l0;
                    auto flush = [&]() {
                        const float4 o4 = *cell;
                        *cell = make_float4(o4.x + l0.x, o4.y + l0.y, o4.z + h0.x, o4.w + h0.y);
                        cell += NU;
                        l0 = l1, h0 = h1, l1 = l2, h1 = h2, l2 = l3, h2 = h3;
                        l3 = h3 = make_float2(0.f, 0.f);
                    };
                    int b = s_base[0];
                    for (int y = 0; y < TY; ++y) {
                        if (s_base[y] != b) {
                            ++b;
                            flush();
                        }
                        const float4 w = *reinterpret_cast<const float4*>(s_weight + y * 4);
                        const float4 g = col[y * NU];
                        const float2 gl = lo2(g), gh = hi2(g);
                        l0 = fma2(dup(w.x), gl, l0), h0 = fma2(dup(w.x), gh, h0);
                        l1 = fma2(dup(w.y), gl, l1), h1 = fma2(dup(w.y), gh, h1);
                        l2 = fma2(dup(w.z), gl, l2), h2 = fma2(dup(w.z), gh, h2);
                        l3 = fma2(dup(w.w), gl, l3), h3 = fma2(dup(w.w), gh, h3);
                    }
                    for (int k = 0; k < 4; ++k) flush();
                }
            };
            // the tile rows' first tap cell and weights for a ring value of the mid axis
            auto row_table = [&](int mval) {
                if (xf < 4) {
                    const int i = mval * my + s_row[q].y;
                    if (xf == 0) s_base[q] = s_row[q].x + offy[i];
                    s_weight[q * 4 + xf] = wy[i * 4 + xf];
                }
            };

            for (int gi = 0; gi < p.ngroups; ++gi) {
                const float4 grp = uget(ut, p.utab, p.u_grp + gi);
                __syncthreads();  // gt built / the previous group's dL/dU folded into the cells
                row_table(__float_as_int(grp.x));
                __syncthreads();
                // first pass, a column of rows to a thread as above
                for (int c = tid; c < 3 * NQ * NU; c += nthr) {
                    const int pw = div_nu(c), u = c - pw * NU;
                    int b = s_base[0];
                    const float4* src = gt + (pw * NV + b) * NU + u;
                    float4 c0 = src[0], c1 = src[NU], c2 = src[2 * NU], c3 = src[3 * NU];
                    for (int y = 0; y < TY; ++y) {
                        if (s_base[y] != b) {
                            ++b;
                            src += NU;
                            c0 = c1, c1 = c2, c2 = c3, c3 = src[3 * NU];
                        }
                        const int at = (pw * TY + y) * NU + u;
                        ut4[at] = filter_cells(*reinterpret_cast<const float4*>(s_weight + y * 4), c0, c1, c2, c3);
                        gu[at] = zero4;
                    }
                }
                __syncthreads();
                for (int pi = __float_as_int(grp.y); pi < __float_as_int(grp.z); ++pi) {
                    const float4 r0 = uget(ut, p.utab, p.u_pair + 4 * pi);
                    const float4 r1 = uget(ut, p.utab, p.u_pair + 4 * pi + 1);
                    const float4 r2 = uget(ut, p.utab, p.u_pair + 4 * pi + 2);
                    const float4 r3 = uget(ut, p.utab, p.u_pair + 4 * pi + 3);
                    const int xv = __float_as_int(r2.w), ax = xv * mx + xr;
                    const float4 wv = *reinterpret_cast<const float4*>(wx + ax * 4);
                    const float4* ubase = ut4 + q * NU + xi - cx0 - 2 + offx[ax];
                    const int pa = __float_as_int(r2.x), pb = __float_as_int(r2.y), pc = __float_as_int(r2.z);
                    float2 TP[NH], TE[NH], TZ[NH];
#pragma unroll
                    for (int wq = 0; wq < NQ; ++wq) {
                        float A[4], Bv[4], Cv[4];
                        filter4(wv, ubase + pa * uplane + wq * TY * NU, A);
                        filter4(wv, ubase + pb * uplane + wq * TY * NU, Bv);
                        filter4(wv, ubase + pc * uplane + wq * TY * NU, Cv);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            put_half<CH>(TP, wq * 4 + k, A[k]);
                            put_half<CH>(TE, wq * 4 + k, Bv[k]);
                            put_half<CH>(TZ, wq * 4 + k, Cv[k]);
                        }
                    }
#pragma unroll
                    for (int w = 0; w < NH; ++w) {
                        const float2 A = TP[w], Bv = TE[w];
                        TP[w] = fma2(hi2(r0), Bv, mul2(lo2(r0), A));
                        TE[w] = fma2(hi2(r1), Bv, mul2(lo2(r1), A));
                    }
                    // the bound, and whether it is above the guard (kGuard, in this frame): with
                    // gradients of 1e-8 or so every sample is below the guard, and none is fixed
                    float bound = r3.w;
                    bool fixing;
                    {
                        constexpr int w = NH / 2;
                        const float2 lo = fma2(TZ[w - 1], TZ[w - 1], fma2(TE[w - 1], TE[w - 1], mul2(TP[w - 1], TP[w - 1])));
                        const float2 g = fma2(TZ[w], TZ[w], fma2(TE[w], TE[w], fma2(TP[w], TP[w], lo)));
                        const float rel = (g.x + g.y) * (g.x + g.y) * kSampleBound;
                        fixing = rel > bound && rel < 1e38f;
                        if (fixing) bound = rel;
                    }
                    unsigned int marked = 0;
                    float2 gP[NH], gE[NH], gZ[NH];  // gP with the sign turned
#pragma unroll
                    for (int w = 0; w < NH; ++w) gP[w] = gE[w] = gZ[w] = make_float2(0.f, 0.f);
                    for (int qi = __float_as_int(r3.x); qi < __float_as_int(r3.y); ++qi) {
                        const float4 c0 = uget(ut, p.utab, p.u_pt + 3 * qi);
                        const float4 c1 = uget(ut, p.utab, p.u_pt + 3 * qi + 1);
                        const float4 c2i = uget(ut, p.utab, p.u_pt + 3 * qi + 2);
                        const int offmask = __float_as_int(c2i.y);
                        float wun = c1.z;  // 2 weight |u|, in a vector register (see radiality.cu)
                        asm volatile("" : "+f"(wun));
                        auto zpass = [&](auto OFF, int zr, float2 w0, float2 w1, float2 w2, float2 w3) {
                            constexpr int o = decltype(OFF)::value;
                            float lowest = 1e38f;  // c2 g2 over these samples
#pragma unroll
                            for (int zi = 0; zi < CH; ++zi) {
                                const float2 P = fma2(w3, TP[zi + o + 3], fma2(w2, TP[zi + o + 2], fma2(w1, TP[zi + o + 1], mul2(w0, TP[zi + o]))));
                                const float2 E = fma2(w3, TE[zi + o + 3], fma2(w2, TE[zi + o + 2], fma2(w1, TE[zi + o + 1], mul2(w0, TE[zi + o]))));
                                const float2 Zc = fma2(w3, TZ[zi + o + 3], fma2(w2, TZ[zi + o + 2], fma2(w1, TZ[zi + o + 1], mul2(w0, TZ[zi + o]))));
                                const float2 dot = fma2(lo2(c0), Zc, P);
                                const float2 cp = fma2(hi2(c0), P, Zc);
                                const float2 c2 = fma2(cp, cp, mul2(E, E));
                                const float2 g2 = fma2(dot, dot, c2);
                                const float2 xx = mul2(c2, g2);
                                lowest = fminf(lowest, fminf(xx.x, xx.y));
                                // 1 / sqrt(c2 g2), at most that at the bound; where g is parallel to
                                // u (c2 = 0) every product below carries a factor c2, cp or E and
                                // vanishes
                                const float2 inv = make_float2(rsqrt_approx(fmaxf(xx.x, bound)),
                                                               rsqrt_approx(fmaxf(xx.y, bound)));
                                const float2 sn = mul2(c2, inv);
                                // K = dL/ds = dL/dS sign(dot) 2 weight |u| (1 - |u| s)
                                const float2 om = mul2(fma2(sn, lo2(c1), dup(wun)), gS[zi * MZ + zr]);
                                const float2 k = mul2(make_float2(flip_sign(om.x, dot.x), flip_sign(om.y, dot.y)), inv);
                                const float2 b = mul2(mul2(sn, sn), k);
                                const float2 m = fma2(b, dup(-1.0f), k);
                                const float2 mc = mul2(m, cp), bd2 = mul2(b, dot), dE = mul2(m, E);
                                const float2 dP = fma2(lo2(c0), mc, bd2);   // -dL/dP
                                const float2 dZ = fma2(hi2(c0), bd2, mc);
                                gP[zi + o] = fma2(w0, dP, gP[zi + o]);
                                gE[zi + o] = fma2(w0, dE, gE[zi + o]);
                                gZ[zi + o] = fma2(w0, dZ, gZ[zi + o]);
                                gP[zi + o + 1] = fma2(w1, dP, gP[zi + o + 1]);
                                gE[zi + o + 1] = fma2(w1, dE, gE[zi + o + 1]);
                                gZ[zi + o + 1] = fma2(w1, dZ, gZ[zi + o + 1]);
                                gP[zi + o + 2] = fma2(w2, dP, gP[zi + o + 2]);
                                gE[zi + o + 2] = fma2(w2, dE, gE[zi + o + 2]);
                                gZ[zi + o + 2] = fma2(w2, dZ, gZ[zi + o + 2]);
                                gP[zi + o + 3] = fma2(w3, dP, gP[zi + o + 3]);
                                gE[zi + o + 3] = fma2(w3, dE, gE[zi + o + 3]);
                                gZ[zi + o + 3] = fma2(w3, dZ, gZ[zi + o + 3]);
                            }
                            if (fixing && lowest < bound) {
#pragma unroll
                                for (int zi = 0; zi < CH; ++zi) {
                                    const float2 P = fma2(w3, TP[zi + o + 3], fma2(w2, TP[zi + o + 2], fma2(w1, TP[zi + o + 1], mul2(w0, TP[zi + o]))));
                                    const float2 E = fma2(w3, TE[zi + o + 3], fma2(w2, TE[zi + o + 2], fma2(w1, TE[zi + o + 1], mul2(w0, TE[zi + o]))));
                                    const float2 Zc = fma2(w3, TZ[zi + o + 3], fma2(w2, TZ[zi + o + 2], fma2(w1, TZ[zi + o + 1], mul2(w0, TZ[zi + o]))));
                                    const float2 dot = fma2(lo2(c0), Zc, P);
                                    const float2 cp = fma2(hi2(c0), P, Zc);
                                    const float2 c2 = fma2(cp, cp, mul2(E, E));
                                    const float2 xx = mul2(c2, fma2(dot, dot, c2));
                                    const int z = zi * MZ + zr;
                                    if (xx.x < bound && gS[z].x != 0.f) marked |= 1u << z;
                                    if (xx.y < bound && gS[z].y != 0.f) marked |= 1u << (z + HZ);
                                }
                            }
                        };
#pragma unroll
                        for (int zr = 0; zr < MZ; ++zr) {
                            const float4 wa = uget(ut, p.utab, p.u_wz + 2 * (__float_as_int(c2i.x) + zr));
                            const float4 wb = uget(ut, p.utab, p.u_wz + 2 * (__float_as_int(c2i.x) + zr) + 1);
                            if ((offmask >> zr) & 1)
                                zpass(IntC<1>{}, zr, lo2(wa), hi2(wa), lo2(wb), hi2(wb));
                            else
                                zpass(IntC<0>{}, zr, lo2(wa), hi2(wa), lo2(wb), hi2(wb));
                        }
                    }
                    // out of the pair's frame (transposed)
                    {
                        const float2 na = make_float2(-r0.x, -r0.y), nb = make_float2(-r0.z, -r0.w);
#pragma unroll
                        for (int w = 0; w < NH; ++w) {
                            const float2 P = gP[w], E = gE[w];
                            gP[w] = fma2(lo2(r1), E, mul2(na, P));
                            gE[w] = fma2(hi2(r1), E, mul2(nb, P));
                        }
                    }
                    const int mask = __float_as_int(r3.z);
                    x_transpose(gP, xv, mask, gu + pa * uplane, true);
                    x_transpose(gE, xv, mask, gu + pb * uplane, true);
                    x_transpose(gZ, xv, mask, gu + pc * uplane, true);
                    if (__any_sync(0xffffffffu, marked != 0)) {
                        __syncwarp();  // the row's sums above
                        const FixTile f = {&p, a.fix, gt, gu, wx, s_weight, s_base, a.gS, zstride};
                        fix_marked<MZ, CZ>(f, pi, xi - cx0 - 2 + offx[ax], ax, bound, sbase, marked);
                    }
                }
                __syncthreads();
                mid_transpose(gu, gg, 3);
            }
            // intensity at the subvoxel centre: the same passes with ring value 0
            {
                float2 gW[NH];
#pragma unroll
                for (int w = 0; w < NH; ++w) gW[w] = make_float2(0.f, 0.f);
#pragma unroll
                for (int zr = 0; zr < MZ; ++zr) {
                    const int m0 = (2 * zr + 1 >= MZ) ? 1 : 0;
                    const float4 qz = uget(ut, p.utab, p.u_wi + zr);
#pragma unroll
                    for (int zi = 0; zi < CH; ++zi) {
                        const int z = zi * MZ + zr;
                        const float2 gi = make_float2(stack_value(a.gI, z), stack_value(a.gI, z + HZ));
                        gW[zi + m0] = fma2(dup(qz.x), gi, gW[zi + m0]);
                        gW[zi + m0 + 1] = fma2(dup(qz.y), gi, gW[zi + m0 + 1]);
                        gW[zi + m0 + 2] = fma2(dup(qz.z), gi, gW[zi + m0 + 2]);
                        gW[zi + m0 + 3] = fma2(dup(qz.w), gi, gW[zi + m0 + 3]);
                    }
                }
                __syncthreads();  // the last group's dL/dU is folded into the cells
                row_table(p.zero_m);
                for (int c = tid; c < gplane; c += nthr) icell[c] = zero4;
                x_transpose(gW, p.zero_x, p.zero_xoff, gu, false);
                __syncthreads();
                mid_transpose(gu, icell, 1);
            }
            __syncthreads();
            // stencil transpose onto the input tile positions, then into dL/dI'. Cells
            // outside the tile grid or the block do not depend on the input. With ranges
            // (1, 1, 1, 1) the cell at offset d adds -(dx Gx + dm Gm + dn Gn), so per position
            // of the x-mid plane sA = sum of -(dx Gx + dm Gm) and sB = sum of Gn over its nine
            // neighbours are formed first, four cells of the innermost axis at a time
            // (straight from the cells the scattered single-word reads took a seventh of
            // the kernel's shared-memory cycles).
            float4 *sA = gt, *sB = gu;  // [quad][NIY][NIX]
            if (p.grad_mode == 1) {
                for (int i = tid; i < NQ * NIY * NIX; i += nthr) {
                    const int wq = div_nixy(i);
                    const int rem = i - wq * (NIX * NIY);
                    const int iy = div_nix(rem), ix = rem - iy * NIX;
                    float4 A = zero4, Bs = zero4;
#pragma unroll
                    for (int dm = 0; dm < 3; ++dm)
#pragma unroll
                        for (int dx = 0; dx < 3; ++dx) {
                            const int uu = ix - R + dx - 1, vv = iy - R + dm - 1;
                            if (uu < 0 || uu >= NU || cx0 + uu < 0 || cx0 + uu >= bw || vv < 0 || vv >= NV ||
                                cy0 + vv < 0 || cy0 + vv >= bh)
                                continue;
                            const float4* c = gg + (wq * NV + vv) * NU + uu;
                            if (dx != 1) A = f4fma(dx == 0 ? 1.f : -1.f, c[0], A);
                            if (dm != 1) A = f4fma(dm == 0 ? 1.f : -1.f, c[gplane], A);
                            Bs = f4fma(1.f, c[2 * gplane], Bs);
                        }
                    sA[i] = A;
                    sB[i] = Bs;
                }
                __syncthreads();
            }
            const float* gf = reinterpret_cast<const float*>(gg);
            const float* icf = reinterpret_cast<const float*>(icell);
            for (int i = tid; i < nin; i += nthr) {
                const int iz = div_nixy(i);
                const int rem = i - iz * (NIX * NIY);
                const int iy = div_nix(rem), ix = rem - iy * NIX;
                const int u = ix - R, v = iy - R, w = iz - R;  // cell with the same position
                float acc = 0.f;
                auto inside = [&](int uu, int vv, int ww) {
                    return uu >= 0 && uu < NU && vv >= 0 && vv < NV && ww >= 0 && ww < NW && cx0 + uu >= 0 &&
                           cx0 + uu < bw && cy0 + vv >= 0 && cy0 + vv < bh && cz0 + ww >= 0 && cz0 + ww < bd;
                };
                if (inside(u, v, w)) acc = icf[((w >> 2) * NV + v) * (4 * NU) + u * 4 + (w & 3)];
                if (p.grad_mode == 1) {
                    const float* fa = reinterpret_cast<const float*>(sA) + 4 * rem;
                    const float* fb = reinterpret_cast<const float*>(sB) + 4 * rem;
#pragma unroll
                    for (int dn = 0; dn < 3; ++dn) {
                        const int ww = w + dn - 1;
                        if (ww < 0 || ww >= NW || cz0 + ww < 0 || cz0 + ww >= bd) continue;
                        const int at = (ww >> 2) * (4 * NIX * NIY) + (ww & 3);
                        acc += fa[at];
                        if (dn != 1) acc += dn == 0 ? fb[at] : -fb[at];
                    }
                } else {
                    const int mR = p.gr[0], xR = p.gr[1], yR = p.gr[2], zR = p.gr[3];
                    auto G = [&](int plane, int du, int dv, int dw) -> float {
                        const int uu = u + du, vv = v + dv, ww = w + dw;
                        return inside(uu, vv, ww) ? gf[plane * 4 * gplane + ((ww >> 2) * NV + vv) * (4 * NU) + uu * 4 + (ww & 3)]
                                                  : 0.f;
                    };
                    // Gx(c) = sum_{i>0, j, k} I(c + (i, j, k)) - I(c + (-i, j, k))
                    for (int ii = 1; ii <= mR; ++ii)
                        for (int j = -yR; j <= yR; ++j)
                            for (int k = -zR; k <= zR; ++k) acc += G(0, -ii, -j, -k) - G(0, ii, -j, -k);
                    for (int jj = 1; jj <= mR; ++jj)
                        for (int ii = -xR; ii <= xR; ++ii)
                            for (int k = -zR; k <= zR; ++k) acc += G(1, -ii, -jj, -k) - G(1, -ii, jj, -k);
                    for (int kk = 1; kk <= mR; ++kk)
                        for (int ii = -xR; ii <= xR; ++ii)
                            for (int j = -yR; j <= yR; ++j) acc += G(2, -ii, -j, -kk) - G(2, -ii, -j, kk);
                }
                if (acc != 0.f) {
                    const long long gidx = global_row(iy, iz) + clampi(cx0 - R + ix, 0, bw - 1);
                    if (in_range(gidx, a.n_in, a.err, 10)) atomicAdd(a.gin + gidx, acc);
                }
            }
        }
    }
}

template <class F>
int with_adj_kernel(const FwdParams& p, F&& f) {
    auto go = [&](auto mz) -> int {
        constexpr int MZ = decltype(mz)::value;
        constexpr int CZ = adj_cz(MZ);
        if (p.u_count > kUTabMax) return f(radiality_adjoint_kernel<MZ, CZ, 1>, IntC<1>{});
        if (p.cz < CZ) return f(radiality_adjoint_kernel<MZ, CZ / 2, kUTabMax>, IntC<kUTabMax>{});
        return f(radiality_adjoint_kernel<MZ, CZ, kUTabMax>, IntC<kUTabMax>{});
    };
    switch (p.mag[2]) {
        case 1: return go(IntC<1>{});
        case 2: return go(IntC<2>{});
        case 3: return go(IntC<3>{});
        case 4: return go(IntC<4>{});
        case 5: return go(IntC<5>{});
        case 6: return go(IntC<6>{});
        case 7: return go(IntC<7>{});
        case 8: return go(IntC<8>{});
    }
    return (int)cudaErrorInvalidValue;
}

}  // namespace

// float4s of the place that U, the input tile and the intensity's cells share
int radiality_adjoint_u_region(const FwdParams& p) {
    const int nq = tile_quads(p.cz);
    return std::max(std::max(3 * nq * p.TY * p.NU, (p.NIX * p.NIY * p.NIZ + 3) / 4), nq * p.NV * p.NU);
}

size_t radiality_adjoint_smem_bytes(const FwdParams& p) {
    const int nq = tile_quads(p.cz), warps = p.TY * kTileX / 32;
    const size_t f4 = (size_t)6 * nq * p.NV * p.NU + p.u_region + (size_t)3 * nq * p.TY * p.NU +
                      (size_t)warps * 2 * nq * (4 + p.mag[0] * adj_cells(p.mag[0]));
    return (f4 * sizeof(float4) + (size_t)p.lane_words * sizeof(float) + 15) & ~(size_t)15;
}

int launch_radiality_adjoint(const FwdParams& p, const FwdPlan& plan, const AdjParams& a, int grid, size_t smem,
                             void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return with_adj_kernel(p, [&](auto k, auto n) -> int {
        constexpr int UN = decltype(n)::value;
        const cudaError_t e = allow_shared(k, smem, kStaticShared);
        if (e != cudaSuccess) return (int)e;
        UTab<UN> tab;
        std::memset(&tab, 0, sizeof tab);
        if (UN > 1) std::memcpy(tab.q, plan.adj_utab.data(), plan.adj_utab.size() * sizeof(float));
        k<<<grid, p.TY * kTileX, smem, st>>>(p, a, tab);
        return (int)cudaGetLastError();
    });
}

int radiality_adjoint_max_ctas_per_sm(const FwdParams& p, int* out) {
    const size_t smem = radiality_adjoint_smem_bytes(p);
    return with_adj_kernel(p, [&](auto k, auto) -> int {
        const cudaError_t e = allow_shared(k, smem, kStaticShared);
        if (e != cudaSuccess) return (int)e;
        return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k, p.TY * kTileX, smem);
    });
}

int launch_temporal_adjoint(const BlockDev* blocks, long long vox, const float* rad, const float* inten,
                            const float* gmap, int T, int method, int itc, int order, int iw, int renorm, int poscon,
                            float* gS, float* gI, long long nmap, unsigned long long* err, void* stream) {
    if (vox == 0) return 0;
    const long long grid = (vox + 127) / 128;
    temporal_adjoint_kernel<<<(unsigned)grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        blocks, rad, inten, gmap, T, method, itc, order, iw, renorm, poscon, gS, gI, nmap, err);
    return (int)cudaGetLastError();
}

int launch_shift_adjoint(const float* src, float* dst, int W, int H, int D, int T, int axis, const float* shifts,
                         int sms, void* stream) {
    const long long rows = (long long)D * H * T;
    const unsigned grid = (unsigned)std::min<long long>((rows + 7) / 8, 64LL * sms);
    auto k = axis == 0 ? shift_adjoint_kernel<0> : axis == 1 ? shift_adjoint_kernel<1> : shift_adjoint_kernel<2>;
    k<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(src, dst, W, H, D, T, shifts);
    return (int)cudaGetLastError();
}

namespace {
__global__ void d2f_kernel(const double* s, float* d, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = (float)s[i];
}
}  // namespace

int launch_double_to_float(const double* src, float* dst, int n, void* stream) {
    if (n <= 0) return 0;
    d2f_kernel<<<(n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(src, dst, n);
    return (int)cudaGetLastError();
}

int launch_drift3d(const float* src, float* dst, const float* g, int W, int H, int D, int T, const float* shifts,
                   int mode, double* out, int sms, void* stream) {
    // walks of 16 planes (19 planes' taps for 16 of output) where they leave every SM
    // its warps, else of 4, whose chain of loads is shorter
    const long long cols = (long long)((W + 31) / 32) * H;
    const int L = cols * ((D + 15) / 16) * T >= 16LL * sms ? 16 : 4;
    const long long warps = cols * ((D + L - 1) / L);
    dim3 grid((unsigned)std::min<long long>((warps + 7) / 8, 64LL * sms), (unsigned)T);
    auto k = mode == 0 ? drift3d_kernel<0> : drift3d_kernel<1>;
    k<<<grid, kDriftThreads, 0, static_cast<cudaStream_t>(stream)>>>(src, dst, g, W, H, D, L, shifts, out);
    return (int)cudaGetLastError();
}

}  // namespace rfba
