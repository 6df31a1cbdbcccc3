// fmm.cu -- FMM far field on the device: leaf moments (P2M), the upward pass (M2M) and
// the multipole evaluation at every target (M2P).
//
// Moments.  FastMultipoleSolver::p2m_m2m / compute_multipole_moments
// (cpp/fmm/fmm_solver.cpp:157-208) with add_multipole_point / add_multipole_shifted_child
// (cpp/fmm/multipole.cpp:218-252) are restated with the reference's operations in the
// reference's order and no contraction (dadd/dmul), so masses, centres of mass and the 31
// moments of every node are bit-identical to the reference's (for masses >= 0).  Leaves first
// (one warp per leaf; lane k owns moment 4 + k), then the internal nodes, deepest first (a block
// per node, a warp per child).
//
// M2P.  multipole_acceleration (multipole.cpp:254-296) builds the degree-4 Taylor
// polynomial of (d + u)_c |d + u|_eps^-3 in the source offset u by truncated polynomial
// products and contracts it with the moments.  Those Taylor coefficients are the
// Cartesian derivatives of the softened potential phi(r) = (r.r + eps^2)^-1/2:
//     a_c = -G sum_k 1/k! M^(k)_{i1..ik} d^(k+1) phi / dr_i1..dr_ik dr_c  at r = d,
// with d = centre of mass - target and M^(k) the raw k-th moment tensor (M^(0) = mass,
// M^(1) = 0 about the centre of mass).  Writing g_n = (-1)^n (2n-1)!! s^-(2n+1)/2,
// s = d.d + eps^2, the derivative tensors are sums of g_n times products of d's and
// Kronecker deltas, and the contraction per order is
//     k=0: -m g1 d
//     k=2: -1/2  [ g3 M[dd] d + g2 (tr M d + 2 M[d]) ]
//     k=3: -1/6  [ g4 O[ddd] d + g3 (3 (w.d) d + 3 O[dd]) + 3 g2 w ]
//     k=4: -1/24 [ g5 H[dddd] d + g4 (6 T2[dd] d + 4 H[ddd]) + g3 (3 tr2 d + 12 T2[d]) ]
// (w, T2, tr2 are the traces stored in the node record).  This is the same polynomial,
// evaluated in about 170 FP64 operations per (target, node) pair instead of the
// reference's polynomial algebra; only rounding differs.  Moments of degree above the
// effective order are left out exactly as evaluate_component does (:205-216).
#include "fmm.cuh"
#include "gx_device.cuh"

#include <algorithm>
#include <atomic>

namespace gx {
namespace {

constexpr int kMomBlock = 256;  // 8 warps, one node each
constexpr int kM2PBlock = 128;

// binomial (multipole.cpp:57-76) for n <= 4.
constexpr int binom4(int n, int k) {
    return (k < 0 || k > n) ? 0 : (k == 0 || k == n) ? 1 : n == 2 ? 2 : n == 3 ? 3 : (k == 2 ? 6 : 4);
}

constexpr int kMaxShiftTerms = 12;  // (2+1)(1+1)(1+1): the most multi-indices below a degree-4 one

// Index tables, evaluated at compile time.  Moment slot k (0..34) is the reference's
// exponent order (multipole.cpp:16-26): degree ascending, then the x exponent descending,
// then the y exponent descending.  For every moment alpha of degree 2..4 (slot 4 + a) the
// terms of add_multipole_shifted_child (multipole.cpp:227-252) in the reference's beta
// order: beta <= alpha componentwise, degree-1 betas left out (their moment is 0 about the
// child's centre of mass, and adding the zero product never changes a sum that starts at
// +0), each with the binomial product and the exponents of the shift.
struct MomentTables {
    int ex[35] = {}, ey[35] = {}, ez[35] = {};
    int nterm[31] = {};
    double bin[31][kMaxShiftTerms] = {};
    int kb[31][kMaxShiftTerms] = {}, dx[31][kMaxShiftTerms] = {}, dy[31][kMaxShiftTerms] = {},
        dz[31][kMaxShiftTerms] = {};
};

constexpr MomentTables make_moment_tables() {
    MomentTables t;
    int k = 0;
    for (int d = 0; d <= 4; ++d)
        for (int x = d; x >= 0; --x)
            for (int y = d - x; y >= 0; --y) {
                t.ex[k] = x;
                t.ey[k] = y;
                t.ez[k] = d - x - y;
                ++k;
            }
    for (int a = 0; a < 31; ++a) {
        const int ka = 4 + a, ax = t.ex[ka], ay = t.ey[ka], az = t.ez[ka];
        int n = 0;
        for (int b = 0; b < 35; ++b) {
            const int bx = t.ex[b], by = t.ey[b], bz = t.ez[b];
            if (bx > ax || by > ay || bz > az || bx + by + bz == 1) continue;
            t.bin[a][n] = (double)(binom4(ax, bx) * binom4(ay, by) * binom4(az, bz));
            t.kb[a][n] = b;
            t.dx[a][n] = ax - bx;
            t.dy[a][n] = ay - by;
            t.dz[a][n] = az - bz;
            ++n;
        }
        t.nterm[a] = n;
    }
    return t;
}

__device__ const MomentTables kTab = make_moment_tables();

// Traces of the moments (record slots 35..45), one lane each: slot 35 + t of the record from
// mom[k] = moment 4 + k (shared memory).
__device__ const signed char kTrace[11][3] = {{0, 3, 5},    {6, 9, 11},   {7, 12, 14},  {8, 13, 15},
                                              {16, 19, 21}, {17, 22, 24}, {18, 23, 25}, {19, 26, 28},
                                              {20, 27, 29}, {21, 28, 30}, {0, 0, 0}};
__device__ __forceinline__ double trace_of(const double* mom, int t) {
    auto sum3 = [&](int k) { return mom[kTrace[k][0]] + mom[kTrace[k][1]] + mom[kTrace[k][2]]; };
    return t < 10 ? sum3(t) : sum3(4) + sum3(7) + sum3(9);
}

// Leaf moments: p2m_m2m leaf branch (fmm_solver.cpp:162-167, 180-181) and
// compute_multipole_moments leaf branch (:187-193).  One warp per node; the warp of an
// internal node only enters it as its octet's parent (the children of the o-th split node are
// nodes 1 + 8 o ..).  The leaf's bodies are staged 32 at a time in shared memory and every lane
// runs the reference's sequential sums over them.  For the moments (lane k for moment 4 + k),
// lane q first puts the powers of body q's offset, as pow_int (multipole.cpp:43-49) computes
// them, beside one another (rows of 33: the lanes of a warp read up to five rows at one body
// without a bank conflict).  A massless leaf gets its cell centre as centre of mass, as in the
// reference.  Bound by latency (dependent loads, the sums, three divisions): N = 65,536 leaf 64
// 13 us, N = 2^20 leaf 16 205 us; with every lane computing and selecting the powers of
// every body 40 and 346 us.
constexpr int kPowRow = 33;
__global__ void __launch_bounds__(kMomBlock) fmm_leaf_kernel(const FmmArgs a) {
    __shared__ double s_pow[kMomBlock / 32][15 * kPowRow];  // rows 5 c + e; first x, y, z, m in rows 1, 6, 11, 14
    __shared__ double s_m[kMomBlock / 32][32];
    const int wl = threadIdx.x >> 5;
    const int w = (int)((blockIdx.x * (unsigned)kMomBlock + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= fmm_nodes(a)) return;
    const int c0 = a.node_child[w];
    if (c0 >= 0) {
        if (lane == 0) a.octet_parent[(c0 - 1) >> 3] = w;
        return;
    }
    const int b = a.node_beg[w], e = a.node_end[w];
    double* r = a.rec + (size_t)w * kFmmRec;
    double* const pw = s_pow[wl];
    double* const sm = s_m[wl];
    double x = 0.0, y = 0.0, z = 0.0;  // this lane's body of the staged chunk
    auto stage = [&](int k0) {
        __syncwarp();
        if (k0 + lane < e) {
            const int i = a.perm[k0 + lane];
            x = a.x[i];
            y = a.y[i];
            z = a.z[i];
            pw[1 * kPowRow + lane] = x;
            pw[6 * kPowRow + lane] = y;
            pw[11 * kPowRow + lane] = z;
            sm[lane] = a.m[i];
        }
        __syncwarp();
        return min(32, e - k0);
    };
    double mass = 0.0, wx = 0.0, wy = 0.0, wz = 0.0;
    for (int k0 = b; k0 < e; k0 += 32) {
        const int cnt = stage(k0);
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) {
            const double mi = sm[q];
            mass = dadd(mass, mi);
            wx = dadd(wx, dmul(pw[1 * kPowRow + q], mi));
            wy = dadd(wy, dmul(pw[6 * kPowRow + q], mi));
            wz = dadd(wz, dmul(pw[11 * kPowRow + q], mi));
        }
    }
    // lanes 0..2 divide one component each
    double com = 0.0;
    if (lane < 3) {
        const double num = lane == 0 ? wx : lane == 1 ? wy : wz;
        const double* cell = lane == 0 ? a.node_cx : lane == 1 ? a.node_cy : a.node_cz;
        com = mass > 0.0 ? __ddiv_rn(num, mass) : cell[w];
    }
    const double cx = __shfl_sync(0xffffffffu, com, 0), cy = __shfl_sync(0xffffffffu, com, 1);
    const double cz = __shfl_sync(0xffffffffu, com, 2);
    const int ks = lane < 31 ? 4 + lane : 0;
    const double* rx = pw + kTab.ex[ks] * kPowRow;
    const double* ry = pw + (5 + kTab.ey[ks]) * kPowRow;
    const double* rz = pw + (10 + kTab.ez[ks]) * kPowRow;
    double v = 0.0;
    for (int k0 = b; k0 < e; k0 += 32) {
        const int cnt = e - b > 32 ? stage(k0) : e - b;
        __syncwarp();
        if (lane < cnt) {
            auto powers = [&](double u, double* p) {
                const double u2 = dmul(u, u), u3 = dmul(u2, u);
                p[0] = 1.0;
                p[kPowRow] = u;
                p[2 * kPowRow] = u2;
                p[3 * kPowRow] = u3;
                p[4 * kPowRow] = dmul(u3, u);
            };
            powers(dsub(x, cx), pw + lane);
            powers(dsub(y, cy), pw + 5 * kPowRow + lane);
            powers(dsub(z, cz), pw + 10 * kPowRow + lane);
        }
        __syncwarp();
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) v = dadd(v, dmul(sm[q], dmul(dmul(rx[q], ry[q]), rz[q])));
    }
    __syncwarp();
    pw[lane] = v;
    if (lane < 31) r[4 + lane] = v;
    else r[kRecMass] = mass;
    if (lane < 3) r[lane] = com;
    __syncwarp();
    if (lane < 11) r[kRecTrQ + lane] = trace_of(pw, lane);
}

// Internal node: p2m_m2m (fmm_solver.cpp:168-181) over the children in octant order, then
// add_multipole_shifted_child per child (multipole.cpp:227-252), with the reference's operations
// in its order.  One block per node at a time: the 8 children's records are staged in shared
// memory, warp c computes child c's shifted contribution to every moment (lane a for moment
// 4 + a), and warp 0 adds the 8 contributions in child order, as the reference does.  A massless
// child adds exact zeros to every sum in the reference and is skipped here (masses are >= 0).
// The terms of a moment (binomial product, slot of the child's moment, powers of the shift) differ
// from lane to lane, so they are read from tables: in shared memory, term by term across the
// lanes, and the powers of a child's shift beside them, all free of bank conflicts (in global
// memory they cost some 1800 L1 wavefronts per child: N = 2^20 leaf 16 750 us).
constexpr int kM2MBlock = 256;
struct M2MShared {
    double bin[kMaxShiftTerms][32];
    int term[kMaxShiftTerms][32];  // kb | dx << 8 | dy << 12 | dz << 16
    double child[8][kRecTrQ];
    double pow[8][3][6];
    double val[8][32];
    double mom[32];
    int node;
};

__device__ __forceinline__ void m2m_tables(M2MShared& s) {
    for (int i = threadIdx.x; i < kMaxShiftTerms * 32; i += kM2MBlock) {
        const int q = i >> 5, l = i & 31;
        const bool in = l < 31 && q < kTab.nterm[l];
        s.bin[q][l] = in ? kTab.bin[l][q] : 0.0;
        // slot of the child's moment: the mass for moment 0
        const int kb = in ? (kTab.kb[l][q] == 0 ? kRecMass : kTab.kb[l][q]) : kRecMass;
        s.term[q][l] = in ? kb | kTab.dx[l][q] << 8 | kTab.dy[l][q] << 12 | kTab.dz[l][q] << 16 : kb;
    }
}

// All threads of the block, for the same internal node w with children c0 .. c0 + 7; tables filled
// (before a barrier).  Ends with a barrier.
__device__ __forceinline__ void m2m_node(const FmmArgs& a, const int w, const int c0, M2MShared& s) {
    const int tid = threadIdx.x, c = tid >> 5, lane = tid & 31;
    for (int k = tid; k < 8 * kRecTrQ; k += kM2MBlock)
        s.child[k / kRecTrQ][k % kRecTrQ] = __ldcg(&a.rec[(size_t)(c0 + k / kRecTrQ) * kFmmRec + k % kRecTrQ]);
    __syncthreads();
    double mass = 0.0, wx = 0.0, wy = 0.0, wz = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double cm = s.child[q][kRecMass];
        if (!(cm > 0.0)) continue;
        mass = dadd(mass, cm);
        wx = dadd(wx, dmul(s.child[q][0], cm));
        wy = dadd(wy, dmul(s.child[q][1], cm));
        wz = dadd(wz, dmul(s.child[q][2], cm));
    }
    // lane 0..2 of every warp divides its component
    const double num = lane == 0 ? wx : lane == 1 ? wy : wz;
    const double* cell = lane == 0 ? a.node_cx : lane == 1 ? a.node_cy : a.node_cz;
    double com = 0.0;
    const double* cr = s.child[c];
    if (lane < 3) {
        com = mass > 0.0 ? __ddiv_rn(num, mass) : cell[w];
        // powers 0..4 of the child's shift, as pow_int computes them
        const double v = dsub(cr[lane], com);
        double* pw = s.pow[c][lane];
        const double v2 = dmul(v, v), v3 = dmul(v2, v);
        pw[0] = 1.0;
        pw[1] = v;
        pw[2] = v2;
        pw[3] = v3;
        pw[4] = dmul(v3, v);
    }
    __syncwarp();
    if (cr[kRecMass] > 0.0) {
        const int nt = lane < 31 ? kTab.nterm[lane] : 0;
        double value = 0.0;
#pragma unroll
        for (int q = 0; q < kMaxShiftTerms; ++q) {
            const int t = s.term[q][lane];
            const double sf = dmul(dmul(dmul(s.bin[q][lane], s.pow[c][0][t >> 8 & 15]), s.pow[c][1][t >> 12 & 15]),
                                   s.pow[c][2][t >> 16]);
            const double next = dadd(value, dmul(sf, cr[t & 255]));
            if (q < nt && sf != 0.0) value = next;
        }
        s.val[c][lane] = value;
    }
    __syncthreads();
    if (c == 0) {
        double* r = a.rec + (size_t)w * kFmmRec;
        double total = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (s.child[q][kRecMass] > 0.0) total = dadd(total, s.val[q][lane]);
        s.mom[lane] = total;
        if (lane < 31) r[4 + lane] = total;
        if (lane < 3) r[lane] = com;
        if (lane == 3) r[kRecMass] = mass;
        __syncwarp();
        if (lane < 11) r[kRecTrQ + lane] = trace_of(s.mom, lane);
    }
    __syncthreads();  // the staging arrays are free for the next node
}

// The octets [ob, oe) (one level's split nodes), level by level.
__global__ void __launch_bounds__(kM2MBlock) fmm_m2m_kernel(const FmmArgs a, int ob, int oe) {
    __shared__ M2MShared s;
    m2m_tables(s);
    for (int o = ob + blockIdx.x; o < oe; o += gridDim.x) m2m_node(a, a.octet_parent[o], 1 + 8 * o, s);
}

// Every internal node in one launch, without a barrier per level.  Blocks take the octets from
// a ticket counter in decreasing order; levels are numbered top down, so a node comes after all
// its children.  A block waits (thread c for child c) until the flag of each internal child's
// octet is set, computes the node and sets its own flag.  A block only waits for nodes whose
// tickets were taken before its own, by blocks already running, so the wait always ends; it is
// bounded all the same (timeout_ns of the global timer), and a wait that gives up sets bit 0 of
// err[0] and err[1] (the evaluation is then redone).  Child records are read through L2
// (__ldcg), since another SM wrote them in this launch.
// Bound by the latency of one node per level: N = 65,536 leaf 64 (9 levels) 40 us, N = 2^20 leaf 16
// 235 us, against 79 and 750 us with the tables in global memory (and a ticket per node, or a
// launch per level).  (Eight lanes per node with the shift terms as straight-line code:
// 110 and 156 us; its 80 KB of instructions are fetched anew on every level.)
__device__ __forceinline__ unsigned long long m2m_clock() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__global__ void __launch_bounds__(kM2MBlock) fmm_m2m_tree_kernel(const FmmArgs a, int* ticket, int* ready, int* err,
                                                                 unsigned long long timeout_ns) {
    __shared__ M2MShared s;
    m2m_tables(s);
    const int octets = (fmm_nodes(a) - 1) >> 3;  // -1 >> 3 = -1 when there are no nodes
    for (;;) {
        if (threadIdx.x == 0) s.node = atomicAdd(ticket, 1);
        __syncthreads();
        const int o = octets - 1 - s.node;
        if (o < 0) return;
        const int c0 = 1 + 8 * o;
        if (threadIdx.x < 8) {
            const int gc = a.node_child[c0 + threadIdx.x];
            if (gc >= 0) {
                const int* f = ready + ((gc - 1) >> 3);
                const unsigned long long t0 = m2m_clock();
                int v = 0;
                for (unsigned it = 0;; ++it) {
                    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
                    if (v) break;
                    if ((it & 255) == 255 && m2m_clock() - t0 > timeout_ns) {
                        atomicOr(err, 1);
                        atomicOr(err + 1, 1);
                        break;
                    }
                }
            }
        }
        __syncthreads();
        m2m_node(a, a.octet_parent[o], c0, s);  // ends with a block barrier; warp 0 wrote the record
        if (threadIdx.x < 32) {
            __threadfence();
            __syncwarp();
            if (threadIdx.x == 0)
                asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(ready + o), "r"(1) : "memory");
        }
    }
}

__device__ __forceinline__ double rsqrt_t(double s) { return rsqrt_f64(s); }
__device__ __forceinline__ float rsqrt_t(float s) { return rsqrt_f32(s); }

// One far node's contribution at one target (without the factor G), from the offset d =
// centre of mass - target and the node's values r[k] = record slot k (k >= 3).  T = double
// is the FP64 far field; T = float the mixed-precision one (d taken in FP64, then rounded).
template <int P, typename T>
__device__ __forceinline__ void m2p_terms(const T* __restrict__ r, const T dx, const T dy, const T dz, const T eps2,
                                          T& fx, T& fy, T& fz) {
    const T s = dx * dx + dy * dy + dz * dz + eps2;
    if (s == T(0)) return;  // h0 == 0 (multipole.cpp:272-275)
    const T ri = rsqrt_t(s);
    const T r2 = ri * ri;
    const T g1 = -ri * r2;
    T cd = -r[kRecMass] * g1;  // coefficient of d
    T vx = T(0), vy = T(0), vz = T(0);
    if (P >= 2) {
        const T g2 = T(-3.0) * g1 * r2, g3 = T(-5.0) * g2 * r2;
        const T mx = r[4] * dx + r[5] * dy + r[6] * dz;
        const T my = r[5] * dx + r[7] * dy + r[8] * dz;
        const T mz = r[6] * dx + r[8] * dy + r[9] * dz;
        const T mdd = dx * mx + dy * my + dz * mz;
        cd -= T(0.5) * (g3 * mdd + g2 * r[kRecTrQ]);
        vx -= g2 * mx;
        vy -= g2 * my;
        vz -= g2 * mz;
        if (P >= 4) {
            const T g4 = T(-7.0) * g3 * r2, g5 = T(-9.0) * g4 * r2;
            // degree-2 monomials of d weighted 2/nu!
            const T qxx = dx * dx, qxy = T(2.0) * dx * dy, qxz = T(2.0) * dx * dz, qyy = dy * dy,
                    qyz = T(2.0) * dy * dz, qzz = dz * dz;
            const T ox = r[10] * qxx + r[11] * qxy + r[12] * qxz + r[13] * qyy + r[14] * qyz + r[15] * qzz;
            const T oy = r[11] * qxx + r[13] * qxy + r[14] * qxz + r[16] * qyy + r[17] * qyz + r[18] * qzz;
            const T oz = r[12] * qxx + r[14] * qxy + r[15] * qxz + r[17] * qyy + r[18] * qyz + r[19] * qzz;
            const T oddd = dx * ox + dy * oy + dz * oz;
            const T wd = r[kRecW] * dx + r[kRecW + 1] * dy + r[kRecW + 2] * dz;
            cd -= g4 * oddd * T(1.0 / 6.0) + T(0.5) * g3 * wd;
            vx -= T(0.5) * (g3 * ox + g2 * r[kRecW]);
            vy -= T(0.5) * (g3 * oy + g2 * r[kRecW + 1]);
            vz -= T(0.5) * (g3 * oz + g2 * r[kRecW + 2]);
            // degree-3 monomials of d weighted 6/mu!
            const T cxxx = qxx * dx, cxxy = T(3.0) * qxx * dy, cxxz = T(3.0) * qxx * dz, cxyy = T(3.0) * dx * qyy,
                    cxyz = T(3.0) * qxy * dz, cxzz = T(3.0) * dx * qzz, cyyy = qyy * dy, cyyz = T(3.0) * qyy * dz,
                    cyzz = T(3.0) * dy * qzz, czzz = qzz * dz;
            const T hx = r[20] * cxxx + r[21] * cxxy + r[22] * cxxz + r[23] * cxyy + r[24] * cxyz + r[25] * cxzz +
                         r[26] * cyyy + r[27] * cyyz + r[28] * cyzz + r[29] * czzz;
            const T hy = r[21] * cxxx + r[23] * cxxy + r[24] * cxxz + r[26] * cxyy + r[27] * cxyz + r[28] * cxzz +
                         r[30] * cyyy + r[31] * cyyz + r[32] * cyzz + r[33] * czzz;
            const T hz = r[22] * cxxx + r[24] * cxxy + r[25] * cxxz + r[27] * cxyy + r[28] * cxyz + r[29] * cxzz +
                         r[31] * cyyy + r[32] * cyyz + r[33] * cyzz + r[34] * czzz;
            const T hdddd = dx * hx + dy * hy + dz * hz;
            const T* Tq = r + kRecT2;  // xx xy xz yy yz zz
            const T tx2 = Tq[0] * dx + Tq[1] * dy + Tq[2] * dz;
            const T ty2 = Tq[1] * dx + Tq[3] * dy + Tq[4] * dz;
            const T tz2 = Tq[2] * dx + Tq[4] * dy + Tq[5] * dz;
            const T tdd = dx * tx2 + dy * ty2 + dz * tz2;
            cd -= g5 * hdddd * T(1.0 / 24.0) + T(0.25) * g4 * tdd + T(0.125) * g3 * r[kRecTr2];
            const T k4 = g4 * T(1.0 / 6.0), k3 = T(0.5) * g3;
            vx -= k4 * hx + k3 * tx2;
            vy -= k4 * hy + k3 * ty2;
            vz -= k4 * hz + k3 * tz2;
        }
    }
    fx += cd * dx + vx;
    fy += cd * dy + vy;
    fz += cd * dz + vz;
}

// A staged record at one target: the FP64 record, or the mixed record (kRec32 layout).
template <int P>
__device__ __forceinline__ void m2p_one(const double* __restrict__ r, double tx, double ty, double tz, double eps2,
                                        double& fx, double& fy, double& fz) {
    m2p_terms<P, double>(r, r[0] - tx, r[1] - ty, r[2] - tz, eps2, fx, fy, fz);
}
template <int P>
__device__ __forceinline__ void m2p_one(const float* __restrict__ r, double tx, double ty, double tz, float eps2,
                                        float& fx, float& fy, float& fz) {
    const double* com = reinterpret_cast<const double*>(r);
    m2p_terms<P, float>(r + 3, (float)(com[0] - tx), (float)(com[1] - ty), (float)(com[2] - tz), eps2, fx, fy, fz);
}

// The mixed-precision records (kRec32) from the FP64 ones, one thread per 16 bytes (13 per
// node) so that both sides are read and written in whole sectors.  Bound by HBM: N = 2^20 leaf 16
// (282,000 nodes, 158 MB) 25 us, against 155 us with one thread per node.
constexpr int kRec32Pieces = kRec32 / 4;
__global__ void __launch_bounds__(256) fmm_rec32_kernel(const FmmArgs a) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t k = i / kRec32Pieces;
    const int p = (int)(i - k * kRec32Pieces);
    if (k >= fmm_nodes(a)) return;
    const double* r = a.rec + (size_t)k * kFmmRec;
    float4 v;
    float* f = reinterpret_cast<float*>(&v);
    if (p == 0) {
        reinterpret_cast<double2*>(&v)[0] = make_double2(r[0], r[1]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int slot = 4 * p + q - 3;  // float 4 p + q holds slot 4 p + q - 3 of the record
            f[q] = slot <= kRecTr2 ? __double2float_rn(r[slot]) : 0.0f;
        }
        if (p == 1) reinterpret_cast<double*>(&v)[0] = r[2];  // floats 4 and 5: the third coordinate
    }
    reinterpret_cast<float4*>(a.rec32 + (size_t)k * kRec32)[p] = v;
}

constexpr int kM2PSub = 64;     // node records per shared-memory buffer
constexpr int kM2PStages = 2;   // buffers in the cp.async ring
// Elements of a node record that an order reads, staged in 16-byte pieces one after the other, and
// the records that a warp stages at once with a lane per piece.
template <int P, typename T>
__host__ __device__ constexpr int m2p_pieces() {
    constexpr int elems = sizeof(T) == 8 ? (P == 0 ? 4 : P == 2 ? kRecTrQ + 1 : 46)
                                         : (P == 0 ? 7 : P == 2 ? kRecTrQ + 4 : kRecTr2 + 4);
    return (elems * (int)sizeof(T) + 15) / 16;
}
template <int P, typename T>
__host__ __device__ constexpr int m2p_per_pass() {
    int n = 1;
    while (2 * n * m2p_pieces<P, T>() <= 32) n *= 2;
    return n;
}
template <int P, typename T>
constexpr size_t m2p_dyn_smem() { return (size_t)kM2PStages * kM2PSub * m2p_pieces<P, T>() * 16; }

__device__ __forceinline__ void cp_async16(const unsigned s, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Work item = (target leaf, up to kM2PChunk far nodes).  The item's node records stream
// through a ring of kM2PStages shared-memory buffers: while the block evaluates one, cp.async
// fills the next ones.  Thread t evaluates target t % W against nodes t / W, t / W + S, ...
// of each buffer (W = the leaf's targets, at most one block; S = block / W node slots, so at
// most W - 1 threads idle); a buffer is filled with a multiple of S records, so every slot
// evaluates the same number of nodes between barriers.  The S partial sums of a target are
// added in slot order, so results do not depend on scheduling.
// A lane copies one 16-byte piece of a record per pass (two mixed records or one FP64 record per
// warp), and reads its list entries one buffer ahead.  The mixed form is bound by instruction issue:
// N = 2^20 leaf 16 (624 M pairs, five targets per leaf: a record is staged for every five pairs)
// 7.04 ms, against 7.72 with pieces dealt out over the block (15 instructions each, and list
// reads just before the copies); seven blocks per SM take 0.1 to 0.3 ms less than six or eight.
// A ring per warp, without block barriers, took 7.9 ms: records shared by two warps are copied
// twice, and its steps cost more instructions than the barriers.  FP64 is bound by its pipe
// (66 %): N = 65,536 leaf 64 231 us either way.
template <int P, typename T>
__global__ void __launch_bounds__(kM2PBlock, (sizeof(T) == 4 ? 7 : 4)) fmm_m2p_kernel(const FmmArgs a) {
    constexpr bool F64 = sizeof(T) == 8;
    constexpr int PIECES = m2p_pieces<P, T>();
    constexpr int kStride = PIECES * 16 / (int)sizeof(T);  // elements of a staged record
    constexpr size_t kGlobal = (size_t)(F64 ? kFmmRec : kRec32) * sizeof(T);  // bytes of a record
    constexpr int kPerPass = m2p_per_pass<P, T>(), kBlockPass = kM2PBlock / 32 * kPerPass;
    constexpr int kPasses = (kM2PSub + kBlockPass - 1) / kBlockPass;
    const char* rec = F64 ? reinterpret_cast<const char*>(a.rec) : reinterpret_cast<const char*>(a.rec32);
    const T eps2 = F64 ? (T)a.eps2 : (T)a.eps2f;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ double s_red[kM2PBlock * 3];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31;
    // the record and piece that the lane stages of each pass
    const int rl = lane < kPerPass * PIECES ? (tid >> 5) * kPerPass + lane / PIECES : kM2PSub;
    const char* const rec_piece = rec + 16 * (lane % PIECES);
    const unsigned dst = (unsigned)__cvta_generic_to_shared(s_raw) + rl * (PIECES * 16) + 16 * (lane % PIECES);
    if (a.overflow && *a.overflow) return;
    const int n_items = fmm_items(a);
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const M2PItem w = a.items[it];
        if (w.leaf < 0) continue;
        const int cnt = w.count;
        const int tb = a.leaf_off[w.leaf], nt = a.leaf_off[w.leaf + 1] - tb;
        const int W = min(nt, kM2PBlock);
        const int S = kM2PBlock / W;
        const int q = tid / W, tl = tid - q * W;
        const int R = S <= kM2PSub ? S * (kM2PSub / S) : kM2PSub;  // records per buffer
        const int nsub = (cnt + R - 1) / R;
        // the nodes of the lane's records of a buffer, read one buffer ahead of the copies
        int node[kPasses];
        auto nodes_of = [&](int sc) {
            const int m = min(R, cnt - sc * R);
            const int* const list = a.far_node + w.fb + sc * R + rl;
#pragma unroll
            for (int u = 0; u < kPasses; ++u)
                if (rl + u * kBlockPass < m) node[u] = __ldg(list + u * kBlockPass);
        };
        // fills buffer sc % kM2PStages with records sc * R ..
        auto stage = [&](int sc) {
            const int m = min(R, cnt - sc * R);
            const unsigned to = dst + (sc % kM2PStages) * (kM2PSub * PIECES * 16);
#pragma unroll
            for (int u = 0; u < kPasses; ++u)
                if (rl + u * kBlockPass < m)
                    cp_async16(to + u * (kBlockPass * PIECES * 16), rec_piece + (size_t)(unsigned)node[u] * kGlobal);
            cp_async_commit();
            nodes_of(sc + 1);
        };
        for (int t0 = 0; t0 < nt; t0 += W) {
            const int t = t0 + tl;
            T fx = T(0), fy = T(0), fz = T(0);
            int i = -1;
            double tx = 0.0, ty = 0.0, tz = 0.0;
            if (q < S && t < nt) {
                i = a.leaf_part[tb + t];
                if (i >= a.t_begin && i < a.t_end) {
                    tx = a.x[i];
                    ty = a.y[i];
                    tz = a.z[i];
                } else {
                    i = -1;
                }
            }
            nodes_of(0);
            stage(0);
            for (int sc = 0; sc < nsub; ++sc) {
                cp_async_wait<0>();
                __syncthreads();  // buffer sc is complete, and every thread is done with buffer sc - 1
                if (sc + 1 < nsub) stage(sc + 1);
                const T* buf = reinterpret_cast<const T*>(s_raw) + (sc % kM2PStages) * (kM2PSub * kStride);
                const int m = min(R, cnt - sc * R);
                if (i >= 0)
                    for (int j = q; j < m; j += S) m2p_one<P>(buf + j * kStride, tx, ty, tz, eps2, fx, fy, fz);
            }
            s_red[tid * 3 + 0] = (double)fx;
            s_red[tid * 3 + 1] = (double)fy;
            s_red[tid * 3 + 2] = (double)fz;
            __syncthreads();
            if (q == 0 && i >= 0) {
                double sx = 0.0, sy = 0.0, sz = 0.0;
                for (int k = 0; k < S; ++k) {
                    const int o = (k * W + tl) * 3;
                    sx += s_red[o];
                    sy += s_red[o + 1];
                    sz += s_red[o + 2];
                }
                if (w.nchunks == 1) {
                    a.ax[i] = a.ax[i] + a.G * sx;
                    a.ay[i] = a.ay[i] + a.G * sy;
                    a.az[i] = a.az[i] + a.G * sz;
                } else {
                    const size_t o = (size_t)(w.scratch + (int64_t)w.chunk * nt + t) * 3;
                    a.scratch[o] = sx;
                    a.scratch[o + 1] = sy;
                    a.scratch[o + 2] = sz;
                }
            }
            __syncthreads();
        }
        if (w.nchunks > 1) {
            // The CTA that completes the leaf's last chunk adds the partials in chunk order.
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = (atomicAdd(&a.done[w.leaf], 1) == w.nchunks - 1);
            __syncthreads();
            if (s_last) {
                __threadfence();
                for (int t = tid; t < nt; t += kM2PBlock) {
                    const int i = a.leaf_part[tb + t];
                    if (i < a.t_begin || i >= a.t_end) continue;
                    double sx = 0.0, sy = 0.0, sz = 0.0;
                    for (int c = 0; c < w.nchunks; ++c) {
                        const size_t o = (size_t)(w.scratch + (int64_t)c * nt + t) * 3;
                        sx += __ldcg(&a.scratch[o]);
                        sy += __ldcg(&a.scratch[o + 1]);
                        sz += __ldcg(&a.scratch[o + 2]);
                    }
                    a.ax[i] = a.ax[i] + a.G * sx;
                    a.ay[i] = a.ay[i] + a.G * sy;
                    a.az[i] = a.az[i] + a.G * sz;
                }
            }
            __syncthreads();
        }
    }
}

template <int P, typename T>
cudaError_t launch_m2p_order(const FmmArgs& a, cudaStream_t st) {
    // the shared-memory opt-in is a per-device setting of the kernel
    static std::atomic<unsigned long long> set_on{0};
    constexpr size_t smem = m2p_dyn_smem<P, T>();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(set_on.load() & bit)) {
        e = cudaFuncSetAttribute(fmm_m2p_kernel<P, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        set_on.fetch_or(bit);
    }
    fmm_m2p_kernel<P, T><<<std::min(a.n_items, 1 << 20), kM2PBlock, smem, st>>>(a);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_m2p_type(const FmmArgs& a, cudaStream_t st) {
    switch (a.order) {
        case 0: return launch_m2p_order<0, T>(a, st);
        case 2: return launch_m2p_order<2, T>(a, st);
        default: return launch_m2p_order<4, T>(a, st);
    }
}

}  // namespace

int fmm_effective_order(int expansion_order) {
    int p = std::min(4, std::max(0, expansion_order));
    if (p == 1 || p == 3) ++p;
    return p;
}

cudaError_t launch_fmm_moments_tree(const FmmArgs& a, int* ticket, int* ready, int* err, int sms, cudaStream_t st) {
    constexpr int wpb = kMomBlock / 32;
    if (a.n_nodes == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(ready, 0, fmm_octets(a.n_nodes) * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(ticket, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    fmm_leaf_kernel<<<(a.n_nodes + wpb - 1) / wpb, kMomBlock, 0, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const int grid = (int)std::min<int64_t>((int64_t)fmm_octets(a.n_nodes), (int64_t)sms * 8);
    fmm_m2m_tree_kernel<<<grid, kM2MBlock, 0, st>>>(a, ticket, ready, err, 1000000000ull);
    return cudaGetLastError();
}

// ax += nx, ay += ny, az += nz: the near field, computed into its own arrays while the far
// field ran, added to it (one rounding, as when the near kernel adds to the far field).
__global__ void __launch_bounds__(256) fmm_add_near_kernel(int64_t n, double* ax, double* ay, double* az,
                                                           const double* nx, const double* ny, const double* nz) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        ax[i] = ax[i] + nx[i];
        ay[i] = ay[i] + ny[i];
        az[i] = az[i] + nz[i];
    }
}

cudaError_t launch_fmm_add_near(int64_t n, double* ax, double* ay, double* az, const double* nx, const double* ny,
                                const double* nz, int sms, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, (int64_t)sms * 8);
    fmm_add_near_kernel<<<(unsigned)blocks, 256, 0, st>>>(n, ax, ay, az, nx, ny, nz);
    return cudaGetLastError();
}

cudaError_t launch_fmm_moments(const FmmArgs& a, const int32_t* level_off_host, int n_levels, int sms,
                               cudaStream_t st) {
    constexpr int wpb = kMomBlock / 32;
    if (a.n_nodes == 0) return cudaSuccess;
    fmm_leaf_kernel<<<(a.n_nodes + wpb - 1) / wpb, kMomBlock, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    for (int d = n_levels - 2; d >= 0; --d) {  // octets whose children are level d + 1
        const int ob = (level_off_host[d + 1] - 1) >> 3, oe = (level_off_host[d + 2] - 1) >> 3;
        if (oe <= ob) continue;
        fmm_m2m_kernel<<<std::min(oe - ob, sms * 8), kM2MBlock, 0, st>>>(a, ob, oe);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_fmm_m2p(const FmmArgs& a, bool mixed, cudaStream_t st) {
    if (a.n_items == 0) return cudaSuccess;
    if (!mixed) return launch_m2p_type<double>(a, st);
    fmm_rec32_kernel<<<(unsigned)(((int64_t)a.n_nodes * kRec32Pieces + 255) / 256), 256, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_m2p_type<float>(a, st);
}

}  // namespace gx
