// Temporal reduction of the radiality stack (sm_103a).
//
// One thread per output subvoxel reduces its radiality series rad[t] and the
// interpolated intensity series I[t] into the map value, with the reference's
// exact semantics:
//   TRM   kernel.cu:332-366  max(0, max_t rad*I)            (IW=0: rad)
//   TRA   kernel.cu:291-327  (1/T) sum_t rad*I              (IW=0: rad)
//   TRPPM kernel.cu:372-419  sum_{t0<=t1} r0+ r1+ / count * mean_t I, computed as
//                            ((sum r+)^2 + sum r+^2) / 2 / (T(T+1)/2): the same
//                            sum with every pair visited once, O(T) instead of O(T^2)
//   TRAC  kernel.cu:423-555  lag-1 cumulants of order 2/3/4 around the mean of
//                            the unweighted series; ITC=1 repeats on the series
//                            binned in place by the order, with the reference's
//                            accumulator carry-over (only AB is reset per level)
//                            and its binning order (entry 0 is cleared before it
//                            is read).
// All temporal sums are FP32 with Kahan compensation. The ITC=1 binning read
// one past the end of an odd-length series (beyond the reference's allocation)
// is defined as 0.
#include <cuda_runtime.h>

#include "shared_limit.h"
#include "srrf_internal.h"

namespace rfba {
namespace {

struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// The region and the voxel in it of output subvoxel gid.
__device__ __forceinline__ const BlockDev& locate(const TemporalParams& p, long long gid, long long* v) {
    int lo = 0, hi = p.nblocks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.vox_prefix[mid] <= gid) lo = mid;
        else hi = mid - 1;
    }
    *v = gid - p.vox_prefix[lo];
    return p.blocks[lo];
}

// Voxel v's place in the output.
__device__ __forceinline__ long long out_index(const BlockDev& B, long long v) {
    const long long nx = B.nreg[0], ny = B.nreg[1];
    long long x, y, z;
    if (v < 0x7fffffffLL) {
        // 32-bit division: a 64-bit one is a long integer sequence per thread
        const unsigned vv = (unsigned)v, ux = (unsigned)nx, uy = (unsigned)ny;
        const unsigned q = vv / ux;
        x = vv - q * ux;
        y = q % uy;
        z = q / uy;
    } else {
        x = v % nx;
        y = (v / nx) % ny;
        z = v / (nx * ny);
    }
    return B.out_offset + x * B.out_stride[0] + y * B.out_stride[1] + z * B.out_stride[2];
}

__global__ void __launch_bounds__(256) temporal_kernel(const TemporalParams p) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= p.total_vox) return;
    long long v;
    const BlockDev& B = locate(p, gid, &v);
    const long long V = B.vox;
    float* rad = p.rad_stack + B.stack_off + v;
    const float* inten = p.int_stack + B.stack_off + v;
    const int T = p.T;
    float result;

    if (p.method == 1) {  // TRA
        Kahan k;
        if (p.iw == 1)
            for (int t = 0; t < T; ++t) k.add(rad[t * V] * inten[t * V]);
        else
            for (int t = 0; t < T; ++t) k.add(rad[t * V]);
        result = k.s / (float)T;
    } else if (p.method == 0) {  // TRM
        float mip = 0.f;
        for (int t = 0; t < T; ++t) mip = fmaxf(p.iw == 1 ? rad[t * V] * inten[t * V] : rad[t * V], mip);
        result = mip;
    } else if (p.method == 2) {  // TRPPM
        Kahan s1, s2, si;
        for (int t = 0; t < T; ++t) {
            const float r = fmaxf(rad[t * V], 0.f);
            s1.add(r);
            s2.add(r * r);
            if (p.iw == 1) si.add(inten[t * V]);
        }
        const float count = fmaxf(0.5f * (float)T * (float)(T + 1), 1.f);
        float pps = (0.5f * (s1.s * s1.s + s2.s)) / count;
        if (p.iw == 1) pps *= si.s / (float)T;
        result = pps;
    } else {  // TRAC
        const int k = p.order;
        Kahan km, kiw;
        for (int t = 0; t < T; ++t) {
            const float r = rad[t * V];
            kiw.add(r * inten[t * V]);
            km.add(r);
        }
        const float mean = km.s / (float)T;
        const float IW = kiw.s / (float)T;
        Kahan AB, ABC, ABCD, CD, AC, BD, AD, BC;
        float out = 0.f;
        if (p.itc != 1) {
            float A = rad[0] - mean;
            float Bv = T > 1 ? rad[V] - mean : 0.f;
            float C = T > 2 ? rad[2 * V] - mean : 0.f;
            for (int t = 0; t < T - k; ++t) {
                const float Dv = (k == 4) ? rad[(t + 3) * V] - mean : 0.f;
                AB.add(A * Bv);
                if (k == 3) ABC.add(A * Bv * C);
                if (k == 4) {
                    ABCD.add(A * Bv * C * Dv);
                    CD.add(C * Dv);
                    AC.add(A * C);
                    BD.add(Bv * Dv);
                    AD.add(A * Dv);
                    BC.add(Bv * C);
                }
                A = Bv;
                Bv = C;
                C = (k == 4) ? Dv : ((t + 3 < T) ? rad[(t + 3) * V] - mean : 0.f);
            }
            if (k == 3) out = fabsf(ABC.s) / (float)T;
            else if (k == 4) out = fabsf(ABCD.s - AB.s * CD.s - AC.s * BD.s - AD.s * BC.s) / (float)T;
            else out = fabsf(AB.s) / (float)T;
        } else {
            int nB = T;
            while (nB > k) {
                AB = Kahan();
                for (int t = 0; t < nB - k; ++t) {
                    const int tBin = t * k;
                    const float A = rad[t * V] - mean;
                    const float Bv = rad[(t + 1) * V] - mean;
                    AB.add(A * Bv);
                    if (k == 3) {
                        const float C = rad[(t + 2) * V] - mean;
                        ABC.add(A * Bv * C);
                    }
                    if (k == 4) {
                        const float C = rad[(t + 2) * V] - mean;
                        const float Dv = rad[(t + 3) * V] - mean;
                        ABCD.add(A * Bv * C * Dv);
                        CD.add(C * Dv);
                        AC.add(A * C);
                        BD.add(Bv * Dv);
                        AD.add(A * Dv);
                        BC.add(Bv * C);
                    }
                    float nv = 0.f;
                    if (tBin < nB) {
                        // entry t is cleared before the bin reads it (t = 0 reads itself
                        // as 0); a read past the end of the series at level 0 is 0
                        for (int j = 0; j < k; ++j) {
                            const int src = tBin + j;
                            const float rv = (src == t || src >= T) ? 0.f : rad[(long long)src * V];
                            nv += rv / (float)k;
                        }
                    }
                    rad[t * V] = nv;
                }
                if (k == 3) out += fabsf(ABC.s) / (float)nB;
                else if (k == 4) out += fabsf(ABCD.s - AB.s * CD.s - AC.s * BD.s - AD.s * BC.s) / (float)nB;
                else out += fabsf(AB.s) / (float)nB;
                nB = nB / k;
            }
        }
        if (p.iw == 1) out = IW * out;
        result = out;
    }

    p.out[out_index(B, v)] = result;
}

// TRAC with ITC=1, each thread's series in its own column of shared memory: the
// stacks are read once, where temporal_kernel reads the radiality again for the
// cumulants and reads, writes and re-reads every level in place, each step waiting on
// the last one's memory. The whole column is copied by cp.async at the start, so each
// thread has T loads in flight, and only its own thread uses it: no barrier. Bound by
// HBM up to T = 50 or so, then by the latency of the sums at few warps an SM (a column
// is 512 T bytes a CTA). 3.5e8 subvoxel-volumes, order 2 and 4, ms:
//   T        20           50           100          200          450       floor
//   here     0.76, 0.96   0.74, 1.01   1.06, 1.23   1.71, 1.91   2.87, 3.18   0.41
//   in place 2.02, 1.62   2.27, 1.88   2.93, 2.54   3.78, 3.20   4.41, 3.42
// so every T whose column fits goes here. With ITC=0 the series is only read twice and
// temporal_kernel is as fast (0.72 against 0.73 ms at T = 100) or faster (0.77 against
// 1.14 at 200): it stays there. The arithmetic and its order are temporal_kernel's.
constexpr int kColThreads = 128;
constexpr size_t kColMaxSmem = 227 * 1024;
template <int K>
__global__ void __launch_bounds__(kColThreads) trac_itc_kernel(const __grid_constant__ TemporalParams p) {
    extern __shared__ float col[];
    const long long gid = (long long)blockIdx.x * kColThreads + threadIdx.x;
    if (gid >= p.total_vox) return;
    long long v;
    const BlockDev& B = locate(p, gid, &v);
    const long long V = B.vox;
    const float* __restrict__ rad = p.rad_stack + B.stack_off + v;
    const float* __restrict__ inten = p.int_stack + B.stack_off + v;
    const int T = p.T;
    float* s = col + threadIdx.x;
    auto at = [&](int t) -> float& { return s[t * kColThreads]; };

    const unsigned dst = (unsigned)__cvta_generic_to_shared(s);
    for (int t = 0; t < T; ++t)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + t * kColThreads * 4), "l"(rad + t * V)
                     : "memory");
    Kahan km, kiw;
    if (p.iw == 1) {
        constexpr int U = 8;
        float w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = u < T ? __ldcs(inten + u * V) : 0.f;
        asm volatile("cp.async.wait_all;" ::: "memory");
        int t = 0;
        for (; t + U <= T; t += U) {
            float n[U];
#pragma unroll
            for (int u = 0; u < U; ++u) n[u] = t + U + u < T ? __ldcs(inten + (t + U + u) * V) : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float r = at(t + u);
                kiw.add(r * w[u]);
                km.add(r);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) w[u] = n[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t + u < T) {
                const float r = at(t + u);
                kiw.add(r * w[u]);
                km.add(r);
            }
    } else {
        asm volatile("cp.async.wait_all;" ::: "memory");
        for (int t = 0; t < T; ++t) km.add(at(t));
    }
    const float mean = km.s / (float)T;
    Kahan AB, ABC, ABCD, CD, AC, BD, AD, BC;
    auto join = [&](float A, float Bv, float C, float Dv) {
        AB.add(A * Bv);
        if (K == 3) ABC.add(A * Bv * C);
        if (K == 4) {
            ABCD.add(A * Bv * C * Dv);
            CD.add(C * Dv);
            AC.add(A * C);
            BD.add(Bv * Dv);
            AD.add(A * Dv);
            BC.add(Bv * C);
        }
    };
    auto cumulant = [&](int n) {
        if (K == 3) return fabsf(ABC.s) / (float)n;
        if (K == 4) return fabsf(ABCD.s - AB.s * CD.s - AC.s * BD.s - AD.s * BC.s) / (float)n;
        return fabsf(AB.s) / (float)n;
    };
    float out = 0.f;
    for (int nB = T; nB > K; nB /= K) {
        AB = Kahan();
        for (int t = 0; t < nB - K; ++t) {
            join(at(t) - mean, at(t + 1) - mean, K > 2 ? at(t + (K > 2 ? 2 : 0)) - mean : 0.f, at(t + K - 1) - mean);
            // entry t is cleared before its bin reads it; a read past the end is 0
            float nv = 0.f;
            if (t * K < nB) {
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    const int src = t * K + j;
                    nv += (src == t || src >= T ? 0.f : at(src)) / (float)K;
                }
            }
            at(t) = nv;
        }
        out += cumulant(nB);
    }
    if (p.iw == 1) out = (kiw.s / (float)T) * out;
    p.out[out_index(B, v)] = out;
}

}  // namespace

int launch_temporal(const TemporalParams& p, void* stream) {
    if (p.total_vox == 0) return 0;
    const size_t smem = (size_t)p.T * kColThreads * sizeof(float);
    if (p.method == 3 && p.itc == 1 && smem <= kColMaxSmem) {
        void (*k)(TemporalParams) = p.order == 3   ? trac_itc_kernel<3>
                                    : p.order == 4 ? trac_itc_kernel<4>
                                                   : trac_itc_kernel<2>;
        if (smem > 48 * 1024) {
            const cudaError_t e = allow_shared(k, smem, 0);
            if (e != cudaSuccess) return (int)e;
        }
        const long long grid = (p.total_vox + kColThreads - 1) / kColThreads;
        k<<<(unsigned)grid, kColThreads, smem, static_cast<cudaStream_t>(stream)>>>(p);
        return (int)cudaGetLastError();
    }
    const long long grid = (p.total_vox + 255) / 256;
    temporal_kernel<<<(unsigned)grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    return (int)cudaGetLastError();
}

}  // namespace rfba
