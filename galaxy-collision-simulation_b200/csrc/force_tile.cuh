// force_tile.cuh -- per-tile bodies of the direct-sum kernels, shared by the one-system
// kernels (force.cu) and the persistent batched kernels (batch.cu).
//
// Pair term of the reference (cpp/direct/direct_solver.cpp:8-23, cpp/cuda/cuda_solver.cu:63-106):
//     a_i = G * sum_{j != i} m_j (x_j - x_i) / (|x_j - x_i|^2 + eps^2)^(3/2)
//
// A tile is BLOCK*IPT consecutive target ordinals [t0, t0 + BLOCK*IPT) held in registers
// (IPT per thread); the sources of one chunk stream through shared memory JT at a time and
// every shared-memory load of a source is reused by IPT targets.  Three arithmetic forms:
//   * mixed  -- sources are staged as FP32 offsets from an FP64 origin (the centre of the
//               bounding box of the tile's targets); the pair term runs in FP32 (12 FP32
//               FMA-pipe operations + 1 MUFU rsqrt per interaction), two sources per
//               packed .f32x2 instruction; the per-j-tile FP32 partial sums are folded into a
//               compensated (TwoSum) accumulator; the result is FP64.
//   * f64    -- FP64 pair term with a refined hardware rsqrt (16 FP64 pipe operations).
//   * exact  -- FP64 with the reference's operation order, IEEE sqrt and division and no
//               contraction; j ascending, i == j skipped: bit-identical to
//               compute_direct_accelerations_for_targets (direct_solver.cpp:59-83).
// A self pair (same body as target and source) has a zero offset and so adds exactly 0
// when eps > 0; with eps == 0 the eps0 variants select s == 0 pairs away, as the
// reference's `if (s2 == 0.0)` does.
//
// Every function here contains __syncthreads(): call it with block-uniform arguments.
#pragma once

#include "force.cuh"
#include "gx_device.cuh"

#include <cfloat>

namespace gx {


// Body index of target ordinal t.  An index-list entry outside [0, n_src) (device index
// arrays are not checked on the host) is replaced by body 0 for the loads, and
// write_result() stores NaN for that target instead of its sum.
__device__ __forceinline__ bool target_ok(const ForceArgs& a, int64_t t) {
    if (!a.tgt_idx) return true;
    const int64_t i = a.tgt_idx[t];
    return i >= 0 && i < a.n_src;
}

__device__ __forceinline__ int64_t target_body(const ForceArgs& a, int64_t t) {
    if (!a.tgt_idx) return a.t_begin + t;
    const int64_t i = a.tgt_idx[t];
    return (i >= 0 && i < a.n_src) ? i : 0;
}

// Final FP64 result of target t (body index `body`): store, then the optional closing kick
// v += a*dt in the reference's rounding (integrator.cpp:7-11, no contraction).
__device__ __forceinline__ void write_result(const ForceArgs& a, int64_t t, int64_t body,
                                             double fx, double fy, double fz) {
    if (!target_ok(a, t)) {
        a.ax[t] = a.ay[t] = a.az[t] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    a.ax[t] = fx;
    a.ay[t] = fy;
    a.az[t] = fz;
    if (a.vx) {
        a.vx[body] = dadd(a.vx[body], dmul(fx, a.kick_dt));
        a.vy[body] = dadd(a.vy[body], dmul(fy, a.kick_dt));
        a.vz[body] = dadd(a.vz[body], dmul(fz, a.kick_dt));
    }
}

__device__ __forceinline__ void write_partial(const ForceArgs& a, int chunk, int64_t t, double sx,
                                              double sy, double sz) {
    const size_t base = (size_t)chunk * 3 * (size_t)a.n_tgt + (size_t)t;
    a.part[base] = sx;
    a.part[base + (size_t)a.n_tgt] = sy;
    a.part[base + 2 * (size_t)a.n_tgt] = sz;
}

// Fused reduction, run by every CTA after its tile body has written its partial sums: the
// CTA that takes the tile's last ticket adds the tile's nsplit partials in chunk order --
// the sums force_reduce_kernel forms -- and writes the results.  Each thread fences its
// own partial stores before the ticket is taken; the last CTA reads the partials from L2
// (ld.global.cg), so no stale L1 line can be seen.  No CTA waits for another.
template <int BLOCK, int IPT>
__device__ __forceinline__ void finish_tile(const ForceArgs& a, const int64_t tile, const int64_t t0) {
    if (a.nsplit <= 1 || !a.tile_count) return;
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&a.tile_count[tile], 1u) == (unsigned)a.nsplit - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + threadIdx.x;
        if (t >= a.n_tgt) continue;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int c = 0; c < a.nsplit; ++c) {
            const size_t base = (size_t)c * 3 * (size_t)a.n_tgt + (size_t)t;
            s0 += __ldcg(a.part + base);
            s1 += __ldcg(a.part + base + (size_t)a.n_tgt);
            s2 += __ldcg(a.part + base + 2 * (size_t)a.n_tgt);
        }
        write_result(a, t, target_body(a, t), a.G * s0, a.G * s1, a.G * s2);
    }
    if (threadIdx.x == 0) a.tile_count[tile] = 0u;
}


// ---------------------------------------------------------------------------------------
// Mixed precision.
// ---------------------------------------------------------------------------------------
template <int BLOCK, int IPT, int JT, bool PACKED, bool EPS0>
__device__ __forceinline__ void mixed_tile(const ForceArgs& a, const int64_t t0, const int chunk) {
    static_assert(JT % BLOCK == 0 && JT % 4 == 0 && BLOCK % 32 == 0, "tile shape");
    constexpr int NW = BLOCK / 32;
    __shared__ __align__(16) float sx[JT];
    __shared__ __align__(16) float sy[JT];
    __shared__ __align__(16) float sz[JT];
    __shared__ __align__(16) float sm[JT];
    __shared__ double sred[6][NW];

    const int tid = threadIdx.x;
    const int64_t first_body = target_body(a, t0);

    double bx[IPT], by[IPT], bz[IPT];
    int64_t body[IPT];
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        body[k] = t < a.n_tgt ? target_body(a, t) : first_body;
        bx[k] = a.x[body[k]];
        by[k] = a.y[body[k]];
        bz[k] = a.z[body[k]];
        lo[0] = fmin(lo[0], bx[k]); hi[0] = fmax(hi[0], bx[k]);
        lo[1] = fmin(lo[1], by[k]); hi[1] = fmax(hi[1], by[k]);
        lo[2] = fmin(lo[2], bz[k]); hi[2] = fmax(hi[2], bz[k]);
    }
    // Origin of the tile: centre of the bounding box of its targets (padding lanes repeat
    // a real target, so they do not widen the box).
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = warp_min(lo[c]);
        hi[c] = warp_max(hi[c]);
    }
    if ((tid & 31) == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sred[c][tid >> 5] = lo[c];
            sred[3 + c][tid >> 5] = hi[c];
        }
    }
    __syncthreads();
    double org[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double l = sred[c][0], h = sred[3 + c][0];
#pragma unroll
        for (int w = 1; w < NW; ++w) {
            l = fmin(l, sred[c][w]);
            h = fmax(h, sred[3 + c][w]);
        }
        org[c] = 0.5 * (l + h);
    }

    float xi[IPT], yi[IPT], zi[IPT];
    CompF cx[IPT], cy[IPT], cz[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        xi[k] = __double2float_rn(bx[k] - org[0]);
        yi[k] = __double2float_rn(by[k] - org[1]);
        zi[k] = __double2float_rn(bz[k] - org[2]);
        cx[k].init();
        cy[k].init();
        cz[k].init();
    }

    const int64_t jb = (int64_t)chunk * a.j_chunk;
    const int64_t je = min(a.n_src, jb + a.j_chunk);
    const float e2 = a.eps2f;

    for (int64_t j0 = jb; j0 < je; j0 += JT) {
#pragma unroll
        for (int r = 0; r < JT / BLOCK; ++r) {
            const int jj = r * BLOCK + tid;
            const int64_t j = j0 + jj;
            float qx = 0.f, qy = 0.f, qz = 0.f, qm = 0.f;
            if (j < je) {
                qx = __double2float_rn(a.x[j] - org[0]);
                qy = __double2float_rn(a.y[j] - org[1]);
                qz = __double2float_rn(a.z[j] - org[2]);
                qm = __double2float_rn(a.m[j]);
            }
            sx[jj] = qx;
            sy[jj] = qy;
            sz[jj] = qz;
            sm[jj] = qm;
        }
        __syncthreads();

        if constexpr (PACKED) {
            f2 XI[IPT], YI[IPT], ZI[IPT], PX[IPT], PY[IPT], PZ[IPT];
            const f2 E2 = pk2(e2, e2);
            const f2 Z0 = pk2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                XI[k] = pk2(xi[k], xi[k]);
                YI[k] = pk2(yi[k], yi[k]);
                ZI[k] = pk2(zi[k], zi[k]);
                PX[k] = Z0;
                PY[k] = Z0;
                PZ[k] = Z0;
            }
#pragma unroll 2
            for (int jj = 0; jj < JT; jj += 4) {
                f2 X[2], Y[2], Z[2], M[2];
                lds_v2b64(sx + jj, X[0], X[1]);
                lds_v2b64(sy + jj, Y[0], Y[1]);
                lds_v2b64(sz + jj, Z[0], Z[1]);
                lds_v2b64(sm + jj, M[0], M[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int k = 0; k < IPT; ++k) {
                        const f2 dX = sub2(X[h], XI[k]);
                        const f2 dY = sub2(Y[h], YI[k]);
                        const f2 dZ = sub2(Z[h], ZI[k]);
                        f2 R = fma2(dX, dX, E2);
                        R = fma2(dY, dY, R);
                        R = fma2(dZ, dZ, R);
                        float r0, r1;
                        upk2(R, r0, r1);
                        float i0 = rsqrt_f32(r0), i1 = rsqrt_f32(r1);
                        if (EPS0) {
                            i0 = (r0 == 0.f) ? 0.f : i0;
                            i1 = (r1 == 0.f) ? 0.f : i1;
                        }
                        const f2 I = pk2(i0, i1);
                        f2 T = mul2(I, I);
                        T = mul2(T, I);
                        const f2 W = mul2(M[h], T);
                        PX[k] = fma2(dX, W, PX[k]);
                        PY[k] = fma2(dY, W, PY[k]);
                        PZ[k] = fma2(dZ, W, PZ[k]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                float l0, l1;
                upk2(PX[k], l0, l1);
                cx[k].add(l0 + l1);
                upk2(PY[k], l0, l1);
                cy[k].add(l0 + l1);
                upk2(PZ[k], l0, l1);
                cz[k].add(l0 + l1);
            }
        } else {
            float px[IPT], py[IPT], pz[IPT];
#pragma unroll
            for (int k = 0; k < IPT; ++k) px[k] = py[k] = pz[k] = 0.f;
#pragma unroll 4
            for (int jj = 0; jj < JT; ++jj) {
                const float qx = sx[jj], qy = sy[jj], qz = sz[jj], qm = sm[jj];
#pragma unroll
                for (int k = 0; k < IPT; ++k) {
                    const float dx = qx - xi[k], dy = qy - yi[k], dz = qz - zi[k];
                    float r = fmaf(dx, dx, e2);
                    r = fmaf(dy, dy, r);
                    r = fmaf(dz, dz, r);
                    float iv = rsqrt_f32(r);
                    if (EPS0) iv = (r == 0.f) ? 0.f : iv;
                    const float w = qm * (iv * iv * iv);
                    px[k] = fmaf(dx, w, px[k]);
                    py[k] = fmaf(dy, w, py[k]);
                    pz[k] = fmaf(dz, w, pz[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                cx[k].add(px[k]);
                cy[k].add(py[k]);
                cz[k].add(pz[k]);
            }
        }
        __syncthreads();
    }

#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        if (t >= a.n_tgt) continue;
        if (a.nsplit == 1)
            write_result(a, t, body[k], a.G * cx[k].value(), a.G * cy[k].value(), a.G * cz[k].value());
        else
            write_partial(a, chunk, t, cx[k].value(), cy[k].value(), cz[k].value());
    }
}

// ---------------------------------------------------------------------------------------
// Mixed precision, targets packed: the same arithmetic as mixed_tile, but each packed
// .f32x2 instruction serves two TARGETS against one source.  Sources are staged in shared
// memory already duplicated ((x, x, y, y), (z, z, m, m): two 16-byte loads per source), so a
// target pair keeps one 64-bit register per coordinate and per accumulator instead of two:
// 6 registers fewer per target, which buys occupancy or more targets per thread.
// ORG: targets per origin when that is a multiple of the CTA's own tile (0: the tile); the origin,
// and with it every bit of the result, is then that of a CTA with the whole ORG targets.
// ---------------------------------------------------------------------------------------
template <int BLOCK, int IPT, int JT, bool EPS0, int UNROLL = 4, int ORG = 0>
__device__ __forceinline__ void mixed_tp_tile(const ForceArgs& a, const int64_t t0, const int chunk) {
    static_assert(JT % BLOCK == 0 && BLOCK % 32 == 0 && IPT % 2 == 0, "tile shape");
    constexpr int NW = BLOCK / 32;
    constexpr int NP = IPT / 2;
    __shared__ __align__(16) float4 sA[JT];  // (x, x, y, y)
    __shared__ __align__(16) float4 sB[JT];  // (z, z, m, m)
    __shared__ double sred[6][NW];

    const int tid = threadIdx.x;
    const int64_t first_body = target_body(a, t0);
    double bx[IPT], by[IPT], bz[IPT];
    int64_t body[IPT];
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        body[k] = t < a.n_tgt ? target_body(a, t) : first_body;
        bx[k] = a.x[body[k]];
        by[k] = a.y[body[k]];
        bz[k] = a.z[body[k]];
        lo[0] = fmin(lo[0], bx[k]); hi[0] = fmax(hi[0], bx[k]);
        lo[1] = fmin(lo[1], by[k]); hi[1] = fmax(hi[1], by[k]);
        lo[2] = fmin(lo[2], bz[k]); hi[2] = fmax(hi[2], bz[k]);
    }
    if constexpr (ORG != 0) {  // the other targets that share the origin
        static_assert(ORG % (BLOCK * IPT) == 0, "whole tiles share an origin");
        const int64_t g0 = t0 / ORG * ORG;
        for (int64_t t = g0 + tid; t < min(g0 + ORG, a.n_tgt); t += BLOCK) {
            if (t >= t0 && t < t0 + BLOCK * IPT) continue;
            const int64_t i = target_body(a, t);
            const double v[3] = {a.x[i], a.y[i], a.z[i]};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = fmin(lo[c], v[c]);
                hi[c] = fmax(hi[c], v[c]);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = warp_min(lo[c]);
        hi[c] = warp_max(hi[c]);
    }
    if ((tid & 31) == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sred[c][tid >> 5] = lo[c];
            sred[3 + c][tid >> 5] = hi[c];
        }
    }
    __syncthreads();
    double org[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double l = sred[c][0], h = sred[3 + c][0];
#pragma unroll
        for (int w = 1; w < NW; ++w) {
            l = fmin(l, sred[c][w]);
            h = fmax(h, sred[3 + c][w]);
        }
        org[c] = 0.5 * (l + h);
    }

    f2 XI[NP], YI[NP], ZI[NP];
    CompF cx[IPT], cy[IPT], cz[IPT];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        XI[q] = pk2(__double2float_rn(bx[2 * q] - org[0]), __double2float_rn(bx[2 * q + 1] - org[0]));
        YI[q] = pk2(__double2float_rn(by[2 * q] - org[1]), __double2float_rn(by[2 * q + 1] - org[1]));
        ZI[q] = pk2(__double2float_rn(bz[2 * q] - org[2]), __double2float_rn(bz[2 * q + 1] - org[2]));
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        cx[k].init();
        cy[k].init();
        cz[k].init();
    }

    const int64_t jb = (int64_t)chunk * a.j_chunk;
    const int64_t je = min(a.n_src, jb + a.j_chunk);
    const f2 E2 = pk2(a.eps2f, a.eps2f);
    const f2 Z0 = pk2(0.f, 0.f);

    for (int64_t j0 = jb; j0 < je; j0 += JT) {
#pragma unroll
        for (int r = 0; r < JT / BLOCK; ++r) {
            const int jj = r * BLOCK + tid;
            const int64_t j = j0 + jj;
            float qx = 0.f, qy = 0.f, qz = 0.f, qm = 0.f;
            if (j < je) {
                qx = __double2float_rn(a.x[j] - org[0]);
                qy = __double2float_rn(a.y[j] - org[1]);
                qz = __double2float_rn(a.z[j] - org[2]);
                qm = __double2float_rn(a.m[j]);
            }
            sA[jj] = make_float4(qx, qx, qy, qy);
            sB[jj] = make_float4(qz, qz, qm, qm);
        }
        __syncthreads();
        f2 PX[NP], PY[NP], PZ[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) PX[q] = PY[q] = PZ[q] = Z0;
        const auto source = [&](const int jj) {
            f2 X, Y, Z, M;
            lds_v2b64(reinterpret_cast<const float*>(&sA[jj]), X, Y);
            lds_v2b64(reinterpret_cast<const float*>(&sB[jj]), Z, M);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const f2 dX = sub2(X, XI[q]);
                const f2 dY = sub2(Y, YI[q]);
                const f2 dZ = sub2(Z, ZI[q]);
                f2 R = fma2(dX, dX, E2);
                R = fma2(dY, dY, R);
                R = fma2(dZ, dZ, R);
                float r0, r1;
                upk2(R, r0, r1);
                float i0 = rsqrt_f32(r0), i1 = rsqrt_f32(r1);
                if (EPS0) {
                    i0 = (r0 == 0.f) ? 0.f : i0;
                    i1 = (r1 == 0.f) ? 0.f : i1;
                }
                const f2 I = pk2(i0, i1);
                f2 T = mul2(I, I);
                T = mul2(T, I);
                const f2 W = mul2(M, T);
                PX[q] = fma2(dX, W, PX[q]);
                PY[q] = fma2(dY, W, PY[q]);
                PZ[q] = fma2(dZ, W, PZ[q]);
            }
        };
        if constexpr (ORG != 0) {  // many short chunks: without the massless rest of a last pass
            static_assert(JT % UNROLL == 0, "whole groups of sources");
            const int cnt = (int)min((int64_t)JT, je - j0);
            for (int jg = 0; jg < cnt; jg += UNROLL)
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) source(jg + u);
        } else {
#pragma unroll UNROLL
            for (int jj = 0; jj < JT; ++jj) source(jj);
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            float p0, p1;
            upk2(PX[q], p0, p1);
            cx[2 * q].add(p0);
            cx[2 * q + 1].add(p1);
            upk2(PY[q], p0, p1);
            cy[2 * q].add(p0);
            cy[2 * q + 1].add(p1);
            upk2(PZ[q], p0, p1);
            cz[2 * q].add(p0);
            cz[2 * q + 1].add(p1);
        }
        __syncthreads();
    }

#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        if (t >= a.n_tgt) continue;
        if (a.nsplit == 1)
            write_result(a, t, body[k], a.G * cx[k].value(), a.G * cy[k].value(), a.G * cz[k].value());
        else
            write_partial(a, chunk, t, cx[k].value(), cy[k].value(), cz[k].value());
    }
}

// ---------------------------------------------------------------------------------------
// FP64 with a refined hardware rsqrt: bound by the FP64 pipe, 16 operations per interaction
// (3 subtractions, 3 FMA, 7 for the weight m s^-3/2 in inv_cube_f64, 3 FMA).  N = 49,999:
// 2.48 ms = 1008 Gint/s, 95% of the measured pipe rate; 2.68 ms with one wave of blocks, 2.94 ms
// with the rsqrt refined first and cubed after (17 operations) as well.
// ---------------------------------------------------------------------------------------
template <int BLOCK, int IPT, int JT, bool EPS0, bool SHORT = false>
__device__ __forceinline__ void f64_tile(const ForceArgs& a, const int64_t t0, const int chunk) {
    static_assert(JT % BLOCK == 0 && JT % 2 == 0, "tile shape");
    __shared__ __align__(16) double sx[JT];
    __shared__ __align__(16) double sy[JT];
    __shared__ __align__(16) double sz[JT];
    __shared__ __align__(16) double sm[JT];

    const int tid = threadIdx.x;
    const int64_t first_body = target_body(a, t0);
    double xi[IPT], yi[IPT], zi[IPT], fx[IPT], fy[IPT], fz[IPT];
    int64_t body[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        body[k] = t < a.n_tgt ? target_body(a, t) : first_body;
        xi[k] = a.x[body[k]];
        yi[k] = a.y[body[k]];
        zi[k] = a.z[body[k]];
        fx[k] = fy[k] = fz[k] = 0.0;
    }
    const int64_t jb = (int64_t)chunk * a.j_chunk;
    const int64_t je = min(a.n_src, jb + a.j_chunk);
    const double e2 = a.eps2;

    for (int64_t j0 = jb; j0 < je; j0 += JT) {
#pragma unroll
        for (int r = 0; r < JT / BLOCK; ++r) {
            const int jj = r * BLOCK + tid;
            const int64_t j = j0 + jj;
            const bool in = j < je;
            sx[jj] = in ? a.x[j] : 0.0;
            sy[jj] = in ? a.y[j] : 0.0;
            sz[jj] = in ? a.z[j] : 0.0;
            sm[jj] = in ? a.m[j] : 0.0;
        }
        __syncthreads();
        const auto source = [&](const int jj) {
            const double qx = sx[jj], qy = sy[jj], qz = sz[jj], qm = sm[jj];
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const double dx = qx - xi[k], dy = qy - yi[k], dz = qz - zi[k];
                double r = fma(dx, dx, e2);
                r = fma(dy, dy, r);
                r = fma(dz, dz, r);
                double w = inv_cube_f64(r, qm);
                if (EPS0) w = (r == 0.0) ? 0.0 : w;
                fx[k] = fma(dx, w, fx[k]);
                fy[k] = fma(dy, w, fy[k]);
                fz[k] = fma(dz, w, fz[k]);
            }
        };
        if constexpr (SHORT) {  // many short chunks: without the massless rest of a last pass
            const int cnt = (int)min((int64_t)JT, je - j0);
            for (int jg = 0; jg < cnt; jg += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u) source(jg + u);
        } else {
#pragma unroll 4
            for (int jj = 0; jj < JT; ++jj) source(jj);
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = t0 + k * BLOCK + tid;
        if (t >= a.n_tgt) continue;
        if (EPS0 && sum_overflowed(fx[k], fy[k], fz[k])) {
            fx[k] = fy[k] = fz[k] = 0.0;
            for (int64_t j = jb; j < je; ++j) {
                const double dx = a.x[j] - xi[k], dy = a.y[j] - yi[k], dz = a.z[j] - zi[k];
                const double w = inv_cube_first(fma(dz, dz, fma(dy, dy, fma(dx, dx, e2))), a.m[j]);
                fx[k] = fma(dx, w, fx[k]);
                fy[k] = fma(dy, w, fy[k]);
                fz[k] = fma(dz, w, fz[k]);
            }
        }
        if (a.nsplit == 1)
            write_result(a, t, body[k], a.G * fx[k], a.G * fy[k], a.G * fz[k]);
        else
            write_partial(a, chunk, t, fx[k], fy[k], fz[k]);
    }
}

// ---------------------------------------------------------------------------------------
// FP64 in the reference's operation order (bit-identical to direct_solver.cpp:59-83).
//
// Every target's sum runs over the sources one after the other, but the terms themselves do
// not depend on it.  A CTA owns TG targets: PW warps compute terms (a warp takes 32 / TG sources
// side by side, U of them in flight per thread) into a shared buffer, and the remaining warps --
// one lane per target and component -- add the previous pass's terms in ascending source order
// while the next pass is computed (two buffers, one barrier per pass).  The addition chain of
// a target is then the only serial part, and a few thousand targets already occupy every SM.
// Bound by the FP64 pipe (31 operations per pair) and the shared-memory traffic of the terms
// (14 of the 16 cycles that the pipe needs for 32 pairs).  N = 16,384: 0.82 ms (327 Gint/s)
// against 3.03 ms with one thread per target and IEEE square root and division source by
// source; N = 1000: 20 us.
// Self pairs and s2 == 0 pairs add +0.0, which leaves the sum unchanged: it starts at +0.0 and,
// in round-to-nearest, is -0.0 only when both addends are.
// ---------------------------------------------------------------------------------------
// The terms of U staged sources s0, s0 + SS, ... at one target, in the reference's operations:
// component c of term u goes to out[u * OU + c * OC].  check (uniform over the warp): the warp
// has a target among the staged sources, self being this thread's slot (its term is zero).
template <int U, int SS, int OU, int OC>
__device__ __forceinline__ void exact_terms(const double2* sxy, const double2* szg, int s0, double xi, double yi,
                                            double zi, double e2, int self, bool check, double* out) {
    double rx[U], ry[U], rz[U], g[U], s2[U], inv[U];
    ExactGuard guard;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const double2 xy = sxy[s0 + u * SS], zg = szg[s0 + u * SS];
        rx[u] = dsub(xy.x, xi);
        ry[u] = dsub(xy.y, yi);
        rz[u] = dsub(zg.x, zi);
        g[u] = zg.y;
        s2[u] = dadd(dadd(dadd(dmul(rx[u], rx[u]), dmul(ry[u], ry[u])), dmul(rz[u], rz[u])), e2);
        inv[u] = exact_inv(s2[u], guard);
    }
    if (check || !guard.clean()) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            inv[u] = ieee_inv(s2[u]);
            if (s2[u] == 0.0 || s0 + u * SS == self) rx[u] = ry[u] = rz[u] = g[u] = inv[u] = 0.0;
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const double scale = dmul(g[u], dmul(dmul(inv[u], inv[u]), inv[u]));
        out[u * OU] = dmul(rx[u], scale);
        out[u * OU + OC] = dmul(ry[u], scale);
        out[u * OU + 2 * OC] = dmul(rz[u], scale);
    }
}

template <int TG, int PW, int U>
struct ExactShape {
    static constexpr int SPW = 32 / TG;              // sources a warp takes side by side
    static constexpr int NS = PW * U * SPW;          // sources per pass
    static constexpr int AW = (3 * TG + 31) / 32;    // adding warps
    static constexpr int BLOCK = 32 * (PW + AW);
    static constexpr int JT = 32 * PW > NS ? 32 * PW : NS;  // sources staged at a time
};

template <int TG, int PW, int U>
__device__ __forceinline__ void exact_tile(const ForceArgs& a, const int64_t t0) {
    using S = ExactShape<TG, PW, U>;
    constexpr int NS = S::NS, JT = S::JT, PT = 32 * PW, PF = JT / PT;
    static_assert(32 % TG == 0 && JT % PT == 0 && JT % NS == 0, "shape");
    __shared__ __align__(16) double2 sxy[JT];
    __shared__ __align__(16) double2 szg[JT];  // z and G m (rounded as the reference rounds it)
    __shared__ double s_con[2][NS * 3 * TG];   // term of source s, component c, target t: (3 s + c) TG + t
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool producer = warp < PW;
    const int tgt = lane % TG, sub = lane / TG;
    const int64_t t = t0 + tgt;
    const int64_t body = target_body(a, t < a.n_tgt ? t : t0);
    const double xi = a.x[body], yi = a.y[body], zi = a.z[body];
    const double G = a.G, e2 = a.eps2;
    const int slot = (warp - PW) * 32 + lane;  // adding lanes: component slot / TG of target slot % TG
    double f = 0.0;
    double px[PF], py[PF], pz[PF], pm[PF];  // the next tile's sources on their way
    auto fetch = [&](int64_t j0) {
#pragma unroll
        for (int r = 0; r < PF; ++r) {
            const int64_t j = max(min(j0 + r * PT + tid, a.n_src - 1), (int64_t)0);
            px[r] = a.x[j];
            py[r] = a.y[j];
            pz[r] = a.z[j];
            pm[r] = a.m[j];
        }
    };
    if (producer) fetch(0);
    int buf = 0;
    for (int64_t j0 = 0; j0 < a.n_src; j0 += JT) {
        if (producer) {
#pragma unroll
            for (int r = 0; r < PF; ++r) {
                sxy[r * PT + tid] = make_double2(px[r], py[r]);
                szg[r * PT + tid] = make_double2(pz[r], dmul(G, pm[r]));
            }
        }
        __syncthreads();
        if (producer && j0 + JT < a.n_src) fetch(j0 + JT);
        const int cnt = (int)min((int64_t)JT, a.n_src - j0);
        const int self = (int)min(max(body - j0, (int64_t)-1), (int64_t)JT);  // the target's own slot, if here
        const bool check = __any_sync(0xffffffffu, self >= 0 && self < JT);
        for (int p0 = 0; p0 < cnt; p0 += NS, buf ^= 1) {
            if (producer) {
                const int s0 = p0 + warp * U * S::SPW + sub;
                double* const out = &s_con[buf][(s0 - p0) * 3 * TG + tgt];
                exact_terms<U, S::SPW, 3 * S::SPW * TG, TG>(sxy, szg, s0, xi, yi, zi, e2, self, check, out);
            }
            __syncthreads();
            if (!producer && slot < 3 * TG) {
                const double* c = &s_con[buf][slot];
                if (cnt - p0 >= NS) {
#pragma unroll
                    for (int s = 0; s < NS; ++s) f = dadd(f, c[s * 3 * TG]);
                } else {
                    for (int s = 0; s < cnt - p0; ++s) f = dadd(f, c[s * 3 * TG]);
                }
            }
        }
    }
    __syncthreads();
    if (!producer && slot < 3 * TG) s_con[0][slot] = f;
    __syncthreads();
    if (tid < TG && t < a.n_tgt) write_result(a, t, body, s_con[0][tid], s_con[0][TG + tid], s_con[0][2 * TG + tid]);
}

// The same sum with one target per thread: U terms at a time, independent of one another, then
// their additions in order.  30 FP64 operations per pair and no exchange of terms, for as many
// targets as fill the SMs.  N = 65,536: 10.2 ms (420 Gint/s, 74% of the measured pipe rate);
// one source at a time with IEEE square root and division took 15.4 ms.
template <int BLOCK, int JT, int U>
__device__ __forceinline__ void exact_serial_tile(const ForceArgs& a, const int64_t t0) {
    static_assert(JT % BLOCK == 0 && JT % U == 0, "tile shape");
    constexpr int PF = JT / BLOCK;
    __shared__ __align__(16) double2 sxy[2][JT];
    __shared__ __align__(16) double2 szg[2][JT];
    const int tid = threadIdx.x;
    const int64_t t = t0 + tid;
    const int64_t body = target_body(a, t < a.n_tgt ? t : t0);
    const double xi = a.x[body], yi = a.y[body], zi = a.z[body];
    const double G = a.G, e2 = a.eps2;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    double px[PF], py[PF], pz[PF], pm[PF];
    auto fetch = [&](int64_t j0) {
#pragma unroll
        for (int r = 0; r < PF; ++r) {
            const int64_t j = max(min(j0 + r * BLOCK + tid, a.n_src - 1), (int64_t)0);
            px[r] = a.x[j];
            py[r] = a.y[j];
            pz[r] = a.z[j];
            pm[r] = a.m[j];
        }
    };
    fetch(0);
    int buf = 0;
    for (int64_t j0 = 0; j0 < a.n_src; j0 += JT, buf ^= 1) {
#pragma unroll
        for (int r = 0; r < PF; ++r) {
            sxy[buf][r * BLOCK + tid] = make_double2(px[r], py[r]);
            szg[buf][r * BLOCK + tid] = make_double2(pz[r], dmul(G, pm[r]));
        }
        __syncthreads();
        if (j0 + JT < a.n_src) fetch(j0 + JT);
        const int cnt = (int)min((int64_t)JT, a.n_src - j0);
        const int self = (int)min(max(body - j0, (int64_t)-1), (int64_t)JT);
        const bool check = __any_sync(0xffffffffu, self >= 0 && self < JT);
        for (int s0 = 0; s0 < cnt; s0 += U) {
            double c[3 * U];
            exact_terms<U, 1, 3, 1>(sxy[buf], szg[buf], s0, xi, yi, zi, e2, self, check, c);
            if (s0 + U <= cnt) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    fx = dadd(fx, c[3 * u]);
                    fy = dadd(fy, c[3 * u + 1]);
                    fz = dadd(fz, c[3 * u + 2]);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (s0 + u >= cnt) break;
                    fx = dadd(fx, c[3 * u]);
                    fy = dadd(fy, c[3 * u + 1]);
                    fz = dadd(fz, c[3 * u + 2]);
                }
            }
        }
    }
    if (t < a.n_tgt) write_result(a, t, body, fx, fy, fz);
}

}  // namespace gx
