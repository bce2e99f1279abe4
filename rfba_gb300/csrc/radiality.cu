// Fused gradient + Catmull-Rom magnification + radiality kernel (sm_103a).
//
// Replaces the reference's gradKernel (kernel.cu:44-125) and calculateRadiality
// (kernel.cu:186-253, with interpolateG kernel.cu:141-169, _calculateDk
// kernel.cu:174-183 and interpolateIntensity kernel.cu:257-287) by one
// persistent kernel. Per work item (block, subvoxel tile, time chunk) and time
// point:
//
//   1. the input tile plus halo is staged into shared memory by a TMA tensor
//      copy (requested one time point ahead) and converted to float with the
//      reference's block-edge clamp (its fminf/fmaxf clamps); inputs whose rows
//      a tensor map cannot address are read with plain loads instead;
//   2. the smoothed gradient of every coarse cell the tile's taps reach is formed
//      in shared memory, one plane per component, four cells of the tile's
//      innermost axis to a float4;
//   3. the ring's n^2 samples are reduced to their distinct points (62 for
//      n = 12) and factorised per axis: Catmull-Rom interpolation is separable,
//      and a sample's taps along an axis depend only on the subvoxel's phase
//      there and the ring point's coordinate. For each distinct value along the
//      tile's mid axis the filtered planes U are formed once in shared memory;
//   4. each thread owns one column of subvoxels along the innermost axis, its
//      lower and upper half packed in register pairs. For each (mid, x) pair of
//      ring values it filters U along x into a column and turns it into the
//      pair's frame; for each ring point of the pair it filters the column along
//      the innermost axis (the tap offset per phase is uniform over the warp, so
//      both offsets are unrolled with static register indices) and accumulates
//      the radiality term, on packed f32x2 FMAs (two subvoxels per instruction);
//   5. radiality and interpolated intensity per subvoxel and time point are
//      written to the stack that the temporal kernel reduces.
//
// What bounds it: the point loop's 20 packed FMAs and 4 MUFUs per point and two
// subvoxels (of 28 warp instructions), 5 of 7.5 ms for four volumes of 128 x
// 128 x 64 at 4 x 4 x 2 (134 M subvoxels x 62 points), where the FMA pipe is 69 %
// busy; in isolation that loop takes 58 clocks per warp and two subvoxels on one
// SM partition against 41 for its FMAs alone, 51 without the MUFUs. The register
// file is what is in the way: it serves two operands per lane and clock, so an
// FMA whose three operands are different vector registers runs at two thirds of
// the rate (80 against 112 to 118 lanes per clock and SM, measured). Hence the
// uniform tables below, the frame that needs no products for the projection, and
// sqrt(weight) folded into 1 - Dk/r so that the square is the accumulating FMA.
// With (x, y) pairs, y columns and 22 packed FMAs per point the same four volumes
// took 10.8 ms.
//
// The radiality term of a sample with interpolated gradient g and ring offset
// rho (kernel.cu:224-240), with u = rho / r: the pair's frame turns (x, mid) so that
// u lies in its P-Z plane, and scales every component alike (FwdPlan in
// srrf_internal.h). Then with kappa the tangent of u's elevation dot = P + kappa Z is
// g.u, cp = Z - kappa P and E are the part of g perpendicular to u, up to the scale,
//   Dk / r = |u| sin(angle(g, u)) = |u| sqrt(|g_perp|^2 / |g|^2),
//   D = (1 - Dk/r)^2,   S -= D if g.u > 0, S += D otherwise
// (at g.u = 0 the sample is perpendicular to g and D vanishes, whatever the sign).
// The perpendicular part is formed directly, so Dk has full relative accuracy
// even when g is almost parallel to u; g = 0 gives 0 * inf = NaN exactly as the
// reference's 0/0 does. Coordinates are local (phase + ring offset), so no
// precision is lost at large volume coordinates. The sample window test
// (kernel.cu:146) makes a whole subvoxel NaN; it is evaluated on the host per
// axis with the reference's float arithmetic and applied here as a per-block
// valid box.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include <cudaTypedefs.h>

#include "radiality_common.cuh"
#include "shared_limit.h"
#include "srrf_internal.h"

namespace rfba {
namespace {

// ---- TMA staging of the input tile ----------------------------------------
// The tile's input box (x rounded down to a 16-byte boundary, so the box is
// wider by up to 15 bytes) is copied by one cp.async.bulk.tensor per time point
// into a staging area, completion signalled on an mbarrier. The next time
// point's box is requested as soon as the current one has been converted, so
// the copy overlaps the radiality work. Coordinates outside the volume read
// zeros; the reference's block-edge clamp is applied when the staging area is
// converted to float (clamped positions always lie inside the box).
__device__ __forceinline__ unsigned smem_u32(const void* ptr) {
    return (unsigned)__cvta_generic_to_shared(ptr);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_load_box(void* dst, const CUtensorMap* map, uint64_t* bar, unsigned bytes, int x,
                                             int y, int z, int t) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(t), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait for the staging phase: false once about a second of wall time
// (%globaltimer) has passed without the phase completing, whatever the time a
// single try_wait suspends for; an iteration cap backs the clock up.
constexpr unsigned long long kWaitLimitNs = 1000000000ull;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (int i = 1; i < (1 << 26); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 15) == 0 && global_ns() - t0 > kWaitLimitNs) return false;
    }
    return false;
}

template <int MZ, int CZ, int UN>
__global__ void __maxnreg__(fwd_regs(MZ, CZ))
    radiality_kernel(const __grid_constant__ FwdParams p, const __grid_constant__ CUtensorMap tmap,
                     const __grid_constant__ UTab<UN> ut) {
    // the tile's two halves along its innermost axis share one register pair: cell
    // w of the lower half and cell w + CH of the upper one
    constexpr int CH = CZ / 2;
    constexpr int HZ = MZ * CH;
    constexpr int FZ = MZ * CZ;
    constexpr int NH = CH + 4;
    constexpr int NQ = tile_quads(CZ);
    extern __shared__ float4 smem4[];

    // Shared layout: [G planes][U planes, the input tile from plane 1 on][lane tables][TMA staging, 128-byte aligned].
    // Planes are [NQ][NV or TY][NU] float4 over four cells of the innermost axis.
    const int NU = p.NU, NV = p.NV;
    const int uplane = NQ * p.TY * NU;
    float4* gt = smem4;
    float4* ut4 = gt + 3 * NQ * NV * NU;
    float* inp = reinterpret_cast<float*>(ut4 + uplane);  // [NIZ][NIY][NIX], dead once G and the intensity's plane are built
    float* tab = reinterpret_cast<float*>(ut4 + p.u_region);
    unsigned char* stage = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(tab + p.lane_words) + 127) & ~(uintptr_t)127);  // [box z][box y][tma_bx]
    __shared__ unsigned int s_item;
    __shared__ int2 s_row[kMaxThreads / kTileX];
    __shared__ alignas(8) uint64_t s_bar;
    const bool use_tma = p.use_tma != 0;
    unsigned phase = 0;
    if (use_tma && threadIdx.x == 0) {
        mbar_init(&s_bar, 1);
        fence_mbar_init();
    }

    const int nthr = blockDim.x;
    const int tid = threadIdx.x;
    const int mx = p.mag[0], my = p.mag[1];
    const int a1 = p.ax1, a2 = p.ax2;  // volume axes of the tile's mid and innermost axis
    // one column (X, Y) per thread
    const int xf = tid & (kTileX - 1);
    const int q = tid / kTileX;                   // 0 .. TY - 1
    const int TY = p.TY;

    for (int i = tid; i < p.lane_words; i += nthr) tab[i] = p.lane[i];
    const float* wx = tab + p.l_wx;
    const int* offx = reinterpret_cast<const int*>(tab + p.l_offx);
    const float* wy = tab + p.l_wm;
    const int* offy = reinterpret_cast<const int*>(tab + p.l_offm);

    const int NIX = p.NIX, NIY = p.NIY, NIZ = p.NIZ, R = p.R;
    const FastDiv div_nu(NU), div_nv(NV), div_ty(TY);
    const int es = p.in_u16 ? 2 : 4;
    const int box1 = a1 == 1 ? NIY : NIZ;  // rows of the staged box along the volume's y

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

        // Tile geometry (block-local fine and coarse coordinates; y is the tile's
        // mid axis and z its innermost axis).
        const int X0 = B.lo[0] + td.t[0] * kTileX;
        const int Y0 = B.lo[a1] + td.t[a1] * p.TY;
        const int Z0 = (B.lo[a2] / MZ) * MZ + td.t[a2] * FZ;
        const int cx0 = floordiv(X0, mx) - 2;
        const int cy0 = floordiv(Y0, my) - 2;
        const int cz0 = Z0 / MZ - 2;
        const int X = X0 + xf;
        const int Y = Y0 + q;
        const int xi = floordiv(X, mx), xr = X - xi * mx;
        if (xf == 0) {
            const int yi = floordiv(Y, my);
            s_row[q] = make_int2(yi - cy0 - 2, Y - yi * my);  // first tap row at offset 0, phase
        }
        const bool in = X < B.hi[0] && Y < B.hi[a1];
        const long long V = B.vox;
        const long long ystride = a1 == 1 ? B.nreg[0] : (long long)B.nreg[0] * B.nreg[1];
        const long long zstride = a1 == 1 ? (long long)B.nreg[0] * B.nreg[1] : B.nreg[0];
        const int zlo = B.lo[a2], zhi = B.hi[a2];
        const long long v0 = (long long)(Y - B.lo[a1]) * ystride + (X - B.lo[0]) + (Z0 - zlo) * zstride;
        const bool rad = X >= B.rad_lo[0] && X <= B.rad_hi[0] && Y >= B.rad_lo[a1] && Y <= B.rad_hi[a1];
        // rows without a valid sample only take part in the shared work
        const bool work = __any_sync(0xffffffffu, in && rad);

        const int t0 = p.t_lo + chunk * p.t_chunk;
        const int t1 = min(p.t_hi > 0 ? p.t_hi : p.T, t0 + p.t_chunk);
        // TMA box origin: x rounded down to a 16-byte boundary; the offset back
        // (0 .. 16 bytes / element size - 1) is where the tile starts in a staged row
        const int kal = 16 / es;
        const int gx0 = B.origin[0] + cx0 - R;
        const int box_ox = ((gx0 % kal) + kal) % kal;
        auto issue = [&](int tt) {
            int c[3];
            c[a1] = B.origin[a1] + cy0 - R;
            c[a2] = B.origin[a2] + cz0 - R;
            tma_load_box(stage, &tmap, &s_bar, (unsigned)(p.tma_bx * NIY * NIZ * es), gx0 - box_ox, c[1], c[2], tt);
        };
        if (use_tma && tid == 0) {
            fence_proxy_async();  // the previous item's generic reads of the staging area come first
            // failure-detection test hook: without the request the wait below
            // runs out, the CTA records the timeout and leaves
            if (!p.test_skip_copy) issue(t0);
        }
        for (int t = t0; t < t1; ++t) {
            const long long sbase = B.stack_off + (long long)(t - p.stack_t0) * V;
            // 1. input tile with block-edge clamp; 16 lanes per row, one division
            //    per row
            if (use_tma) {
                const bool ok = mbar_wait_bounded(&s_bar, phase);
                if (__syncthreads_or(!ok)) {
                    // the copy did not land: record it, give it a bounded time to
                    // finish so no write is pending into this CTA's shared memory
                    if (tid == 0) {
                        if (p.err) atomicCAS(p.err, 0ull, (0x54ull << 56) | (unsigned long long)item);
                        mbar_wait_bounded(&s_bar, phase);
                    }
                    return;
                }
                phase ^= 1u;
                auto unpack = [&](auto* st) {
                    for (int r = q, iy = q, iz = 0; r < NIY * NIZ; r += TY, iy += TY) {
                        while (iy >= NIY) {
                            iy -= NIY;
                            ++iz;
                        }
                        const int sy = clampi(cy0 - R + iy, 0, bh - 1) - (cy0 - R);
                        const int sz = clampi(cz0 - R + iz, 0, bd - 1) - (cz0 - R);
                        const auto* srow = st + (a1 == 1 ? sz * box1 + sy : sy * box1 + sz) * p.tma_bx + box_ox;
                        float* rows = inp + r * NIX;
                        for (int ix = xf; ix < NIX; ix += kTileX)
                            rows[ix] = (float)srow[clampi(cx0 - R + ix, 0, bw - 1) - (cx0 - R)];
                    }
                };
                if (p.in_u16)
                    unpack(reinterpret_cast<const uint16_t*>(stage));
                else
                    unpack(reinterpret_cast<const float*>(stage));
                __syncthreads();
                if (tid == 0 && t + 1 < t1) {
                    fence_proxy_async();  // the staging area's generic reads before the next async write
                    issue(t + 1);
                }
            } else {
                const long long tbase = (long long)t * p.D * p.H * p.W;
                __syncthreads();  // the tile shares the U planes, read until here by the previous time point
                for (int r = q, iy = q, iz = 0; r < NIY * NIZ; r += TY, iy += TY) {
                    while (iy >= NIY) {
                        iy -= NIY;
                        ++iz;
                    }
                    const int by = B.origin[a1] + clampi(cy0 - R + iy, 0, bh - 1);
                    const int bz = B.origin[a2] + clampi(cz0 - R + iz, 0, bd - 1);
                    const long long rowg =
                        tbase + (a1 == 1 ? (long long)bz * p.H + by : (long long)by * p.H + bz) * p.W + B.origin[0];
                    float* rows = inp + r * NIX;
                    for (int ix = xf; ix < NIX; ix += kTileX) {
                        const long long gi = rowg + clampi(cx0 - R + ix, 0, bw - 1);
                        rows[ix] = p.in_u16 ? (float)__ldg(static_cast<const uint16_t*>(p.in) + gi)
                                            : __ldg(static_cast<const float*>(p.in) + gi);
                    }
                }
                __syncthreads();
            }
            // 2. gradient planes, and the intensity filtered along the mid axis (ring
            //    value 0) in U plane 0. Cells outside the block are 0.
            for (int c = tid; c < NQ * NV * NU; c += nthr) {
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
                    auto row = [&](int k) { return base + (w0 + R + k) * (NIY * NIX); };
                    gradient4(p.grad_mode, p.gr, row, NIX, g);
#pragma unroll
                    for (int w = 0; w < 4; ++w)
                        if (cw + w < 0 || cw + w >= bd) g[0][w] = g[1][w] = g[2][w] = 0.f;
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) gt[k * (NQ * NV * NU) + c] = make_float4(g[k][0], g[k][1], g[k][2], g[k][3]);
            }
            for (int c = tid; c < uplane; c += nthr) {
                const int r = div_nu(c), u = c - r * NU;
                const int wq = div_ty(r), y = r - wq * TY, w0 = wq * 4;
                const int2 ri = s_row[y];
                const float4 wv = *reinterpret_cast<const float4*>(wy + (p.zero_m * my + ri.y) * 4);
                const int v = ri.x + offy[p.zero_m * my + ri.y];
                const bool uin = cx0 + u >= 0 && cx0 + u < bw;
                const float wk[4] = {wv.x, wv.y, wv.z, wv.w};
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const bool vin = uin && cy0 + v + k >= 0 && cy0 + v + k < bh;
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const int cw = cz0 + w0 + w;
                        const float x = inp[((w0 + w + R) * NIY + (v + k + R)) * NIX + u + R];
                        acc[w] = fmaf(wk[k], vin && cw >= 0 && cw < bd ? x : 0.f, acc[w]);
                    }
                }
                ut4[c] = make_float4(acc[0], acc[1], acc[2], acc[3]);
            }
            __syncthreads();
            // intensity at the subvoxel centre (interpolateIntensity)
            {
                const float4 wv = *reinterpret_cast<const float4*>(wx + (p.zero_x * mx + xr) * 4);
                const float4* src = ut4 + q * NU + xi - cx0 - 2 + offx[p.zero_x * mx + xr];
                float2 Tw[NH];
#pragma unroll
                for (int wq = 0; wq < NQ; ++wq) {
                    float u[4];
                    filter4(wv, src + wq * TY * NU, u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) put_half<CH>(Tw, wq * 4 + k, u[k]);
                }
                const bool okc = X >= B.int_lo[0] && X <= B.int_hi[0] && Y >= B.int_lo[a1] && Y <= B.int_hi[a1];
                const int ilo = B.int_lo[a2], ihi = B.int_hi[a2];
                float* dst = p.int_stack + sbase + v0;
#pragma unroll
                for (int zr = 0; zr < MZ; ++zr) {
                    // exactly the reference's 4 taps (kernel.cu:268-283), so a
                    // non-finite voxel reaches the same subvoxels: they start one
                    // coarse cell later when floor((zr + 0.5) / mz - 0.5) = 0,
                    // i.e. when 2 zr + 1 >= mz
                    const int m0 = (2 * zr + 1 >= MZ) ? 1 : 0;
                    const float4 qz = uget(ut, p.utab, p.u_wi + zr);
#pragma unroll
                    for (int zi = 0; zi < CH; ++zi) {
                        float2 acc = mul2(dup(qz.x), Tw[zi + m0]);
                        acc = fma2(dup(qz.y), Tw[zi + m0 + 1], acc);
                        acc = fma2(dup(qz.z), Tw[zi + m0 + 2], acc);
                        acc = fma2(dup(qz.w), Tw[zi + m0 + 3], acc);
                        const int z = zi * MZ + zr, Z = Z0 + z;
                        if (in && Z >= zlo && Z < zhi)
                            dst[z * zstride] = okc && Z >= ilo && Z <= ihi ? fmaxf(acc.x, 0.f) : 0.f;
                        if (in && Z + HZ >= zlo && Z + HZ < zhi)
                            dst[(z + HZ) * zstride] = okc && Z + HZ >= ilo && Z + HZ <= ihi ? fmaxf(acc.y, 0.f) : 0.f;
                    }
                }
            }

            float2 S[HZ];
#pragma unroll
            for (int z = 0; z < HZ; ++z) S[z] = make_float2(0.f, 0.f);

            for (int gi = 0; gi < p.ngroups; ++gi) {
                const float4 grp = uget(ut, p.utab, p.u_grp + gi);
                __syncthreads();  // gt ready / previous U consumed
                // 3. the gradient planes filtered along the mid axis for this group's
                //    ring value
                {
                    const int b0 = __float_as_int(grp.x) * my;
                    for (int c = tid; c < 3 * uplane; c += nthr) {
                        const int r = div_nu(c), u = c - r * NU;
                        const int pw = div_ty(r), y = r - pw * TY;
                        const int2 ri = s_row[y];
                        ut4[c] = filter_rows(*reinterpret_cast<const float4*>(wy + (b0 + ri.y) * 4),
                                             gt + (pw * NV + ri.x + offy[b0 + ri.y]) * NU + u, NU);
                    }
                }
                __syncthreads();
                // 4. pairs of this mid value
                if (!work) continue;
                for (int pi = __float_as_int(grp.y); pi < __float_as_int(grp.z); ++pi) {
                    const float4 r0 = uget(ut, p.utab, p.u_pair + 4 * pi);
                    const float4 r1 = uget(ut, p.utab, p.u_pair + 4 * pi + 1);
                    const float4 r2 = uget(ut, p.utab, p.u_pair + 4 * pi + 2);
                    const float4 r3 = uget(ut, p.utab, p.u_pair + 4 * pi + 3);
                    const int a = __float_as_int(r2.w) * mx + xr;
                    const float4 wv = *reinterpret_cast<const float4*>(wx + a * 4);
                    const float4* ubase = ut4 + q * NU + xi - cx0 - 2 + offx[a];
                    const float4* pa = ubase + __float_as_int(r2.x) * uplane;
                    const float4* pb = ubase + __float_as_int(r2.y) * uplane;
                    const float4* pc = ubase + __float_as_int(r2.z) * uplane;
                    // x pass of the three planes, in the pair's plane order, then into the
                    // pair's frame on both halves at once (on single cells, before the
                    // halves are packed, the same products took 8.4 instead of 7.5 ms on
                    // four volumes of 128 x 128 x 64 at 4 x 4 x 2)
                    float2 TP[NH], TE[NH], TZ[NH];
#pragma unroll
                    for (int wq = 0; wq < NQ; ++wq) {
                        float A[4], Bv[4], Cv[4];
                        filter4(wv, pa + wq * TY * NU, A);
                        filter4(wv, pb + wq * TY * NU, Bv);
                        filter4(wv, pc + wq * TY * NU, Cv);
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
                    for (int qi = __float_as_int(r3.x); qi < __float_as_int(r3.y); ++qi) {
                        const float4 c0 = uget(ut, p.utab, p.u_pt + 3 * qi);
                        const float4 c1 = uget(ut, p.utab, p.u_pt + 3 * qi + 1);
                        const float4 c2i = uget(ut, p.utab, p.u_pt + 3 * qi + 2);
                        const int offmask = __float_as_int(c2i.y);
                        // in a vector register: an FMA takes one uniform operand, a second
                        // one would be copied in front of every use
                        float root = c1.z;
                        asm volatile("" : "+f"(root));
                        auto zpass = [&](auto OFF, int zr, float2 w0, float2 w1, float2 w2, float2 w3) {
                            constexpr int o = decltype(OFF)::value;
#pragma unroll
                            for (int zi = 0; zi < CH; ++zi) {
                                const int z = zi * MZ + zr;
                                const float2 P = fma2(w3, TP[zi + o + 3], fma2(w2, TP[zi + o + 2], fma2(w1, TP[zi + o + 1], mul2(w0, TP[zi + o]))));
                                const float2 E = fma2(w3, TE[zi + o + 3], fma2(w2, TE[zi + o + 2], fma2(w1, TE[zi + o + 1], mul2(w0, TE[zi + o]))));
                                const float2 Zc = fma2(w3, TZ[zi + o + 3], fma2(w2, TZ[zi + o + 2], fma2(w1, TZ[zi + o + 1], mul2(w0, TZ[zi + o]))));
                                const float2 dot = fma2(lo2(c0), Zc, P);         // along the ring direction
                                const float2 cp = fma2(hi2(c0), P, Zc);          // across it
                                const float2 c2 = fma2(cp, cp, mul2(E, E));      // |g_perp|^2
                                const float2 g2 = fma2(dot, dot, c2);            // |g|^2
                                // sin = sqrt(c2) / sqrt(g2): g parallel to u gives 0, g = 0
                                // gives 0 * inf = NaN (the reference's 0/0).
                                const float2 sn = mul2(make_float2(sqrt_approx(c2.x), sqrt_approx(c2.y)),
                                                       make_float2(rsqrt_approx(g2.x), rsqrt_approx(g2.y)));
                                const float2 om = fma2(sn, lo2(c1), dup(root));  // sqrt(weight) (1 - Dk/r)
                                S[z] = fma2(om, make_float2(flip_sign(om.x, dot.x), flip_sign(om.y, dot.y)), S[z]);
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
                }
            }

            // 5. finalize and store radiality (S holds the sum with the sign of the
            //    projection; converging samples count positive)
            const int rlo = B.rad_lo[a2], rhi = B.rad_hi[a2];
            float* dst = p.rad_stack + sbase + v0;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int z = 0; z < HZ; ++z) {
                    const int Z = Z0 + h * HZ + z;
                    if (!in || Z < zlo || Z >= zhi) continue;
                    float r = rad && Z >= rlo && Z <= rhi ? (h ? S[z].y : S[z].x) * p.neg_weight
                                                          : __int_as_float(0x7fc00000);
                    if (p.renorm) r = 0.5f + r * 0.5f;
                    if (p.poscon) r = fmaxf(r, 0.f);
                    dst[(h * HZ + z) * zstride] = r;
                }
        }
    }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda
// link dependency).
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
        else
            cudaGetLastError();
    });
    return fn;
}

// 4D tensor map (x, y, z, t) of the input with the tile's staging box; false
// (plain loads) when TMA staging is off for this launch or the input cannot be
// described (base or row pitch not 16-byte aligned).
bool encode_input_map(const FwdParams& p, CUtensorMap* map) {
    std::memset(map, 0, sizeof *map);
    const int es = p.in_u16 ? 2 : 4;
    if (p.tma_bx <= 0) return false;
    if ((reinterpret_cast<uintptr_t>(p.in) & 15) != 0 || ((long long)p.W * es) % 16 != 0) return false;
    if (p.tma_bx > 256 || p.NIY > 256 || p.NIZ > 256 || (p.tma_bx * es) % 16 != 0) return false;
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dim[4] = {(cuuint64_t)p.W, (cuuint64_t)p.H, (cuuint64_t)p.D, (cuuint64_t)p.T};
    const cuuint64_t stride[3] = {(cuuint64_t)p.W * es, (cuuint64_t)p.W * p.H * es, (cuuint64_t)p.W * p.H * p.D * es};
    const bool zin = p.ax2 == 2;
    const cuuint32_t box[4] = {(cuuint32_t)p.tma_bx, (cuuint32_t)(zin ? p.NIY : p.NIZ),
                               (cuuint32_t)(zin ? p.NIZ : p.NIY), 1u};
    const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    const CUresult r = fn(map, es == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                          const_cast<void*>(p.in), dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

size_t g4_words(const FwdParams& p) {  // float4s of the G planes
    const int nq = tile_quads(p.cz);
    return (size_t)3 * nq * p.NV * p.NU;
}

// f(kernel, table size) for the launch's z magnification and table form
template <class F>
int with_kernel(const FwdParams& p, F&& f) {
    auto go = [&](auto mz) -> int {
        constexpr int MZ = decltype(mz)::value;
        auto depth = [&](auto cz) -> int {
            constexpr int CZ = decltype(cz)::value;
            if (p.u_count > kUTabMax) return f(radiality_kernel<MZ, CZ, 1>, IntC<1>{});
            if (p.u_count > kUTabSmall) return f(radiality_kernel<MZ, CZ, kUTabMax>, IntC<kUTabMax>{});
            return f(radiality_kernel<MZ, CZ, kUTabSmall>, IntC<kUTabSmall>{});
        };
        if constexpr (MZ <= kDeepMag)
            if (p.cz == 8) return depth(IntC<8>{});
        if constexpr (MZ >= kFlatMag)
            if (p.cz == 2) return depth(IntC<2>{});
        return depth(IntC<4>{});
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

// float4s of the U planes, which also hold the input tile (from plane 1 on)
// while the gradient is formed
int radiality_u_region(const FwdParams& p) {
    const int nq = tile_quads(p.cz);
    const int plane = nq * p.TY * p.NU;
    return std::max(3 * plane, plane + (p.NIX * p.NIY * p.NIZ + 3) / 4);
}

size_t radiality_smem_bytes(const FwdParams& p) {
    size_t b = sizeof(float4) * (g4_words(p) + (size_t)p.u_region) + sizeof(float) * (size_t)p.lane_words;
    if (p.tma_bx > 0) b += 128 + (size_t)p.tma_bx * p.NIY * p.NIZ * (p.in_u16 ? 2 : 4);  // 128-byte aligned start
    return (b + 15) & ~(size_t)15;
}

int radiality_tma_box_x(const FwdParams& p) {
    const int es = p.in_u16 ? 2 : 4;
    const int al = 16 / es;
    if (((long long)p.W * es) % 16 != 0) return 0;
    const char* e = std::getenv("RFBA_TMA");
    if (e && e[0] == '0' && e[1] == 0) return 0;
    const int bx = ((p.NIX + al - 1 + al - 1) / al) * al;  // NIX + up to al - 1 of alignment slack
    return bx <= 256 ? bx : 0;
}

int launch_radiality(const FwdParams& p, const FwdPlan& plan, int grid, size_t smem, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return with_kernel(p, [&](auto k, auto n) -> int {
        constexpr int UN = decltype(n)::value;
        const cudaError_t e = allow_shared(k, smem, kStaticShared);
        if (e != cudaSuccess) return (int)e;
        FwdParams q = p;
        CUtensorMap map;
        q.use_tma = encode_input_map(p, &map) ? 1 : 0;
        UTab<UN> tab;
        if (UN > 1) {
            std::memcpy(tab.q, plan.utab.data(), plan.utab.size() * sizeof(float));
            std::memset(reinterpret_cast<char*>(tab.q) + plan.utab.size() * sizeof(float), 0,
                        sizeof tab.q - plan.utab.size() * sizeof(float));
        } else {
            std::memset(&tab, 0, sizeof tab);
        }
        k<<<grid, p.TY * kTileX, smem, st>>>(q, map, tab);
        return (int)cudaGetLastError();
    });
}

int radiality_max_ctas_per_sm(const FwdParams& p, int* out) {
    const size_t smem = radiality_smem_bytes(p);
    return with_kernel(p, [&](auto k, auto) -> int {
        const cudaError_t e = allow_shared(k, smem, kStaticShared);
        if (e != cudaSuccess) return (int)e;
        return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k, p.TY * kTileX, smem);
    });
}

}  // namespace rfba
