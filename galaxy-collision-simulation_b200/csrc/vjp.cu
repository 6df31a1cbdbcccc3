// vjp.cu -- vector-Jacobian product of the direct accelerations (the adjoint kernel).
//
// No reference counterpart (the reference has no gradients).  With
//     a_k = G sum_{j != k} m_j d s^-3/2,   d = x_j - x_k,   s = |d|^2 + eps^2,
// and a cotangent l_k on a_k, L = sum_k l_k . a_k has
//     dL/dx_k = G sum_j [ s^-3/2 A - 3 s^-5/2 (A . d) d ],  A = m_k l_j - m_j l_k,
//     dL/dm_k = -G sum_j s^-3/2 (l_j . d),
// which is a gather over j with the forward kernel's tiling: the sources stage
// (x_j, m_j, l_j) -- 7 words -- in shared memory and each thread keeps IPT targets.
// A self pair has d = 0, and its A is zero up to the rounding of one product (m_k l_k - m_k l_k by a
// fused multiply-add), so with eps > 0 it adds at most 2^-53 (mixed: 2^-24) of m_k |l_k| eps^-3.
// Forms: FP64 (refined rsqrt) and mixed (FP32 pair arithmetic on offsets from a per-tile
// FP64 origin, the sums of each source tile added up in FP64).  A j-split keeps systems of any
// size spread over all SMs: grid and fused ordered reduction as in the forward kernels (force.cuh).
#include "gx_device.cuh"
#include "vjp.cuh"

#include <algorithm>
#include <cfloat>

namespace gx {
namespace {

// This CTA's four sums per target: written out, or left as partial sums of its chunk.
__device__ __forceinline__ void vjp_write(const VjpArgs& a, int64_t t, double vx, double vy, double vz, double h) {
    a.gx[t] = a.G * vx;
    a.gy[t] = a.G * vy;
    a.gz[t] = a.G * vz;
    if (a.gm) a.gm[t] = -a.G * h;
}

__device__ __forceinline__ void vjp_store(const VjpArgs& a, int chunk, int64_t t, const double (&v)[4]) {
    if (a.nsplit == 1) {
        vjp_write(a, t, v[0], v[1], v[2], v[3]);
    } else {
        const size_t base = (size_t)chunk * 4 * (size_t)a.n + (size_t)t;
#pragma unroll
        for (int c = 0; c < 4; ++c) a.part[base + (size_t)c * (size_t)a.n] = v[c];
    }
}

// The CTA that takes the tile's last ticket adds its chunks' partial sums in chunk order (read
// through L2, after a fence); no CTA waits for another.
template <int BLOCK, int IPT>
__device__ __forceinline__ void vjp_finish(const VjpArgs& a, int64_t tile) {
    if (a.nsplit <= 1) return;
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&a.tile_count[tile], 1u) == (unsigned)a.nsplit - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = tile * (BLOCK * IPT) + k * BLOCK + threadIdx.x;
        if (t >= a.n) continue;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
        for (int c = 0; c < a.nsplit; ++c) {
            const size_t base = (size_t)c * 4 * (size_t)a.n + (size_t)t;
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q] += __ldcg(a.part + base + (size_t)q * (size_t)a.n);
        }
        vjp_write(a, t, s[0], s[1], s[2], s[3]);
    }
}

// FP64: 35 FP64 operations per pair (3 differences, 3 FMA, 5 for the rsqrt, 2 for its powers, 3 for
// l_j . d, 6 for A, 3 for A . d, 3 for its factor, 7 FMA into the sums).  Bound by the FP64 pipe:
// N = 16,384 632 us = 87% of the measured rate, against 720 us
// with 42 operations (l_k . d, products not fused into the sums).
template <int BLOCK, int IPT, int JT, bool EPS0>
__global__ void __launch_bounds__(BLOCK) vjp_f64_kernel(const VjpArgs a) {
    static_assert(JT % BLOCK == 0, "tile shape");
    __shared__ __align__(16) double2 sxy[JT];
    __shared__ __align__(16) double2 szm[JT];
    __shared__ __align__(16) double2 sl01[JT];
    __shared__ double sl2[JT];
    const int tid = threadIdx.x;
    const int64_t tile = blockIdx.x / a.nsplit;
    const int chunk = (int)(blockIdx.x % a.nsplit);
    const int64_t t0 = tile * (BLOCK * IPT);
    double xk[IPT], yk[IPT], zk[IPT], mk[IPT], lk[IPT][3], acc[IPT][4];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid, i = t < a.n ? t : t0;
        xk[k] = a.x[i];
        yk[k] = a.y[i];
        zk[k] = a.z[i];
        mk[k] = a.m[i];
        lk[k][0] = a.lx[i];
        lk[k][1] = a.ly[i];
        lk[k][2] = a.lz[i];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] = 0.0;
    }
    const int64_t jb = (int64_t)chunk * a.j_chunk, je = min(a.n, jb + a.j_chunk);
    for (int64_t j0 = jb; j0 < je; j0 += JT) {
#pragma unroll
        for (int r = 0; r < JT / BLOCK; ++r) {
            const int jj = r * BLOCK + tid;
            const int64_t j = j0 + jj;
            const bool in = j < je;
            sxy[jj] = in ? make_double2(a.x[j], a.y[j]) : make_double2(0.0, 0.0);
            szm[jj] = in ? make_double2(a.z[j], a.m[j]) : make_double2(0.0, 0.0);
            sl01[jj] = in ? make_double2(a.lx[j], a.ly[j]) : make_double2(0.0, 0.0);
            sl2[jj] = in ? a.lz[j] : 0.0;
        }
        __syncthreads();
#pragma unroll 2
        for (int jj = 0; jj < JT; ++jj) {
            const double2 xy = sxy[jj], zm = szm[jj], l01 = sl01[jj];
            const double l2 = sl2[jj];
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const double dx = xy.x - xk[k], dy = xy.y - yk[k], dz = zm.x - zk[k];
                const double s = fma(dz, dz, fma(dy, dy, fma(dx, dx, a.eps2)));
                double y = rsqrt_f64(s);
                if (EPS0) y = (s == 0.0) ? 0.0 : y;
                const double y2 = y * y;
                const double i3 = y2 * y;
                const double ljd = fma(l2, dz, fma(l01.y, dy, l01.x * dx));
                const double A0 = fma(mk[k], l01.x, -(zm.y * lk[k][0]));
                const double A1 = fma(mk[k], l01.y, -(zm.y * lk[k][1]));
                const double A2 = fma(mk[k], l2, -(zm.y * lk[k][2]));
                const double B = fma(A2, dz, fma(A1, dy, A0 * dx));
                const double c3 = i3 * (-3.0 * y2) * B;
                acc[k][0] = fma(c3, dx, fma(i3, A0, acc[k][0]));
                acc[k][1] = fma(c3, dy, fma(i3, A1, acc[k][1]));
                acc[k][2] = fma(c3, dz, fma(i3, A2, acc[k][2]));
                acc[k][3] = fma(i3, ljd, acc[k][3]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        if (t < a.n) vjp_store(a, chunk, t, acc[k]);
    }
    vjp_finish<BLOCK, IPT>(a, tile);
}

// Mixed precision, two TARGETS per packed .f32x2 lane pair (sources pre-duplicated in shared
// memory as (x,x,y,y) (z,z,m,m) (l0,l0,l1,l1) (l2,l2)).  Per source and target pair: 29
// packed FP32 instructions + 2 MUFU rsqrt.  The two gradient terms are accumulated apart,
// G = sum s^-3/2 A and W = sum s^-5/2 (A.d) d; after every source tile their FP32 sums go into
// FP64 ones as G - 3W, so a target keeps 4 of these.  A . d is taken from A itself (3 operations;
// m_k (l_j . d) - m_j (l_k . d) took 5, and cancels where l varies little).
// Bound by the FP32 FMA pipe: N = 16,384 286 us = 76% of the measured rate (N = 40,000 1.63 ms,
// 79%), against 368 us with 31 operations, four targets and seven compensated sums per target (196
// registers: 8 warps per SM) and a reduction launch.
template <int BLOCK, int IPT, int JT, bool EPS0>
__global__ void __launch_bounds__(BLOCK) vjp_mixed_kernel(const VjpArgs a) {
    static_assert(JT % BLOCK == 0 && IPT % 2 == 0, "tile shape");
    constexpr int NP = IPT / 2;
    __shared__ __align__(16) float4 sA[JT], sB[JT], sC[JT];
    __shared__ __align__(8) float2 sD[JT];
    __shared__ double sred[6][BLOCK / 32];

    const int tid = threadIdx.x;
    const int64_t tile = blockIdx.x / a.nsplit;
    const int chunk = (int)(blockIdx.x % a.nsplit);
    const int64_t t0 = tile * (BLOCK * IPT);
    double org[3];
    f2 XK[NP], YK[NP], ZK[NP], MK[NP], NL0[NP], NL1[NP], NL2[NP];
    {
        int64_t idx[IPT];
        double bx[IPT], by[IPT], bz[IPT];
        double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int64_t t = t0 + k * BLOCK + tid;
            idx[k] = t < a.n ? t : t0;
            bx[k] = a.x[idx[k]];
            by[k] = a.y[idx[k]];
            bz[k] = a.z[idx[k]];
            lo[0] = fmin(lo[0], bx[k]); hi[0] = fmax(hi[0], bx[k]);
            lo[1] = fmin(lo[1], by[k]); hi[1] = fmax(hi[1], by[k]);
            lo[2] = fmin(lo[2], bz[k]); hi[2] = fmax(hi[2], bz[k]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = warp_min(lo[c]);
            hi[c] = warp_max(hi[c]);
        }
        if ((tid & 31) == 0)
            for (int c = 0; c < 3; ++c) {
                sred[c][tid >> 5] = lo[c];
                sred[3 + c][tid >> 5] = hi[c];
            }
        __syncthreads();
        for (int c = 0; c < 3; ++c) {
            double l = sred[c][0], h = sred[3 + c][0];
            for (int w = 1; w < BLOCK / 32; ++w) {
                l = fmin(l, sred[c][w]);
                h = fmax(h, sred[3 + c][w]);
            }
            org[c] = 0.5 * (l + h);
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const int k0 = 2 * q, k1 = 2 * q + 1;
            XK[q] = pk2(__double2float_rn(bx[k0] - org[0]), __double2float_rn(bx[k1] - org[0]));
            YK[q] = pk2(__double2float_rn(by[k0] - org[1]), __double2float_rn(by[k1] - org[1]));
            ZK[q] = pk2(__double2float_rn(bz[k0] - org[2]), __double2float_rn(bz[k1] - org[2]));
            MK[q] = pk2(__double2float_rn(a.m[idx[k0]]), __double2float_rn(a.m[idx[k1]]));
            NL0[q] = pk2(-__double2float_rn(a.lx[idx[k0]]), -__double2float_rn(a.lx[idx[k1]]));
            NL1[q] = pk2(-__double2float_rn(a.ly[idx[k0]]), -__double2float_rn(a.ly[idx[k1]]));
            NL2[q] = pk2(-__double2float_rn(a.lz[idx[k0]]), -__double2float_rn(a.lz[idx[k1]]));
        }
    }
    double acc[IPT][4];
#pragma unroll
    for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] = 0.0;
    const f2 E2 = pk2(a.eps2f, a.eps2f);
    const f2 Z0 = pk2(0.f, 0.f);
    const int64_t jb = (int64_t)chunk * a.j_chunk, je = min(a.n, jb + a.j_chunk);
    for (int64_t j0 = jb; j0 < je; j0 += JT) {
#pragma unroll
        for (int r = 0; r < JT / BLOCK; ++r) {
            const int jj = r * BLOCK + tid;
            const int64_t j = j0 + jj;
            float qx = 0.f, qy = 0.f, qz = 0.f, qm = 0.f, l0 = 0.f, l1 = 0.f, l2 = 0.f;
            if (j < je) {
                qx = __double2float_rn(a.x[j] - org[0]);
                qy = __double2float_rn(a.y[j] - org[1]);
                qz = __double2float_rn(a.z[j] - org[2]);
                qm = __double2float_rn(a.m[j]);
                l0 = __double2float_rn(a.lx[j]);
                l1 = __double2float_rn(a.ly[j]);
                l2 = __double2float_rn(a.lz[j]);
            }
            sA[jj] = make_float4(qx, qx, qy, qy);
            sB[jj] = make_float4(qz, qz, qm, qm);
            sC[jj] = make_float4(l0, l0, l1, l1);
            sD[jj] = make_float2(l2, l2);
        }
        __syncthreads();
        f2 G[NP][3], W[NP][3], H[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            G[q][0] = G[q][1] = G[q][2] = Z0;
            W[q][0] = W[q][1] = W[q][2] = Z0;
            H[q] = Z0;
        }
#pragma unroll 4
        for (int jj = 0; jj < JT; ++jj) {
            f2 X, Y, Z, M, L0, L1;
            lds_v2b64(reinterpret_cast<const float*>(&sA[jj]), X, Y);
            lds_v2b64(reinterpret_cast<const float*>(&sB[jj]), Z, M);
            lds_v2b64(reinterpret_cast<const float*>(&sC[jj]), L0, L1);
            const f2 L2 = *reinterpret_cast<const f2*>(&sD[jj]);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const f2 dX = sub2(X, XK[q]), dY = sub2(Y, YK[q]), dZ = sub2(Z, ZK[q]);
                f2 S = fma2(dX, dX, E2);
                S = fma2(dY, dY, S);
                S = fma2(dZ, dZ, S);
                float s0, s1;
                upk2(S, s0, s1);
                float y0 = rsqrt_f32(s0), y1 = rsqrt_f32(s1);
                if (EPS0) {
                    y0 = (s0 == 0.f) ? 0.f : y0;
                    y1 = (s1 == 0.f) ? 0.f : y1;
                }
                const f2 Yv = pk2(y0, y1);
                const f2 Y2 = mul2(Yv, Yv);
                const f2 I3 = mul2(Y2, Yv);
                f2 LJD = mul2(L0, dX);                            // l_j . d
                LJD = fma2(L1, dY, LJD);
                LJD = fma2(L2, dZ, LJD);
                const f2 A0 = fma2(MK[q], L0, mul2(M, NL0[q]));  // m_k l_j - m_j l_k
                const f2 A1 = fma2(MK[q], L1, mul2(M, NL1[q]));
                const f2 A2 = fma2(MK[q], L2, mul2(M, NL2[q]));
                f2 B = mul2(A0, dX);                              // A . d
                B = fma2(A1, dY, B);
                B = fma2(A2, dZ, B);
                const f2 C = mul2(I3, mul2(Y2, B));
                G[q][0] = fma2(I3, A0, G[q][0]);
                G[q][1] = fma2(I3, A1, G[q][1]);
                G[q][2] = fma2(I3, A2, G[q][2]);
                W[q][0] = fma2(C, dX, W[q][0]);
                W[q][1] = fma2(C, dY, W[q][1]);
                W[q][2] = fma2(C, dZ, W[q][2]);
                H[q] = fma2(I3, LJD, H[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            float g0, g1, w0, w1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                upk2(G[q][c], g0, g1);
                upk2(W[q][c], w0, w1);
                acc[2 * q][c] += fma(-3.0, (double)w0, (double)g0);
                acc[2 * q + 1][c] += fma(-3.0, (double)w1, (double)g1);
            }
            upk2(H[q], g0, g1);
            acc[2 * q][3] += (double)g0;
            acc[2 * q + 1][3] += (double)g1;
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        if (t < a.n) vjp_store(a, chunk, t, acc[k]);
    }
    vjp_finish<BLOCK, IPT>(a, tile);
}

#define VMIX(E) {kMixed, 128, 2, 256, E, (const void*)&vjp_mixed_kernel<128, 2, 256, E>}
#define VF64(B, I, J, E) {kF64, B, I, J, E, (const void*)&vjp_f64_kernel<B, I, J, E>}

const VjpVariant kVjp[] = {
    VMIX(false), VMIX(true),
    VF64(64, 1, 128, false), VF64(64, 1, 128, true),
    VF64(64, 2, 256, false), VF64(64, 2, 256, true),
};

}  // namespace

// The variant for n bodies.  Mixed: two targets per thread (N = 16,384 286 us; four targets 294, more
// registers and fewer blocks).  FP64: one target per thread and short passes for small systems
// (N = 1000 19 us, two targets 42; N = 8192 175 against 178), two above (N = 40,000 3.65 ms
// against 3.69).
const VjpVariant& vjp_variant(int64_t n, int precision, bool eps0) {
    return kVjp[(precision == kMixed ? 0 : n < 12000 ? 2 : 4) + (eps0 ? 1 : 0)];
}

// Chunks of two passes (N = 16,384, mixed, sources per chunk 256: 304 us, 512: 288, 2048: 324; FP64
// 512: 632, 2048: 755), of one where that leaves the SMs without two blocks each; at most 64, and
// at most 256 MB of partial sums.
int vjp_split(const VjpVariant& v, int64_t n, int sms) {
    const int64_t chunk = vjp_tiles(v, n) * ((n + 2 * v.jt - 1) / (2 * v.jt)) < 2 * sms ? v.jt : 2 * v.jt;
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>(64, (256ll << 20) / (32 * std::max<int64_t>(n, 1))));
    return (int)std::max<int64_t>(1, std::min(most, (n + chunk - 1) / chunk));
}

cudaError_t launch_vjp(const VjpVariant& v, const VjpArgs& args, cudaStream_t st) {
    if (args.n <= 0) return cudaSuccess;
    const int64_t blocks = vjp_tiles(v, args.n) * args.nsplit;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    VjpArgs a = args;
    void* params[] = {(void*)&a};
    return cudaLaunchKernel(v.fn, dim3((unsigned)blocks), dim3(v.block), params, 0, st);
}

}  // namespace gx
