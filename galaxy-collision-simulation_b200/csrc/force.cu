// force.cu -- one-system direct-sum kernels (one CTA per target tile and source chunk,
// chunk-minor), the ordered j-split reduction (fused into the last CTA of each tile, or a
// second kernel) and the table of compiled variants.  The arithmetic lives in
// force_tile.cuh.
#include "force_tile.cuh"

#include <mutex>

namespace gx {
namespace {

// Ordered reduction of the j-split partial sums, then G and the epilogue (the unfused path).
__global__ void __launch_bounds__(256) force_reduce_kernel(const ForceArgs a) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= a.n_tgt) return;
    double s[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < a.nsplit; ++c) {
        const size_t base = (size_t)c * 3 * (size_t)a.n_tgt + (size_t)t;
        s[0] += a.part[base];
        s[1] += a.part[base + (size_t)a.n_tgt];
        s[2] += a.part[base + 2 * (size_t)a.n_tgt];
    }
    write_result(a, t, target_body(a, t), a.G * s[0], a.G * s[1], a.G * s[2]);
}

template <int BLOCK, int IPT, int JT, bool PACKED, bool EPS0>
__global__ void __launch_bounds__(BLOCK) force_mixed_kernel(const ForceArgs a) {
    const int64_t tile = blockIdx.x / a.nsplit;
    mixed_tile<BLOCK, IPT, JT, PACKED, EPS0>(a, tile * (BLOCK * IPT), (int)(blockIdx.x % a.nsplit));
    finish_tile<BLOCK, IPT>(a, tile, tile * (BLOCK * IPT));
}

template <int BLOCK, int IPT, int JT, bool EPS0, int MINB, int UNROLL = 4>
__global__ void __launch_bounds__(BLOCK, MINB) force_mixed_tp_kernel(const ForceArgs a) {
    const int64_t tile = blockIdx.x / a.nsplit;
    mixed_tp_tile<BLOCK, IPT, JT, EPS0, UNROLL>(a, tile * (BLOCK * IPT), (int)(blockIdx.x % a.nsplit));
    finish_tile<BLOCK, IPT>(a, tile, tile * (BLOCK * IPT));
}

template <int BLOCK, int IPT, int JT, bool EPS0>
__global__ void __launch_bounds__(BLOCK) force_f64_kernel(const ForceArgs a) {
    const int64_t tile = blockIdx.x / a.nsplit;
    f64_tile<BLOCK, IPT, JT, EPS0>(a, tile * (BLOCK * IPT), (int)(blockIdx.x % a.nsplit));
    finish_tile<BLOCK, IPT>(a, tile, tile * (BLOCK * IPT));
}

template <int TG, int PW, int U>
__global__ void __launch_bounds__(ExactShape<TG, PW, U>::BLOCK) force_exact_kernel(const ForceArgs a) {
    exact_tile<TG, PW, U>(a, (int64_t)blockIdx.x * TG);
}

template <int BLOCK, int JT, int U>
__global__ void __launch_bounds__(BLOCK) force_exact_serial_kernel(const ForceArgs a) {
    exact_serial_tile<BLOCK, JT, U>(a, (int64_t)blockIdx.x * BLOCK);
}

#define MIXED(B, I, J, P, E) {kMixed, B, I, J, P, E, (const void*)&force_mixed_kernel<B, I, J, P, E>}
#define MIXTP(B, I, J, E, MB) {kMixed, B, I, J, 2, E, (const void*)&force_mixed_tp_kernel<B, I, J, E, MB>}
#define MIXTPU(B, I, J, MB, U) {kMixed, B, I, J, 2, 0, (const void*)&force_mixed_tp_kernel<B, I, J, false, MB, U>}
#define F64(B, I, J, E) {kF64, B, I, J, 0, E, (const void*)&force_f64_kernel<B, I, J, E>}
#define EXSER(B, J, U) {kF64Exact, B, 1, J, 0, 1, (const void*)&force_exact_serial_kernel<B, J, U>}
#define EXACT(T, W, U)                                                                             \
    {kF64Exact, ExactShape<T, W, U>::BLOCK, 1, ExactShape<T, W, U>::JT, 0, 1,                      \
     (const void*)&force_exact_kernel<T, W, U>, T}

const ForceVariant kVariants[] = {
    // mixed, targets packed
    MIXTPU(256, 6, 512, 1, 8),
    MIXTPU(128, 8, 512, 1, 8),
    MIXTPU(128, 6, 512, 2, 16),
    MIXTP(128, 8, 512, false, 1),
    MIXTPU(256, 4, 512, 2, 16),
    MIXTPU(64, 8, 256, 1, 8),
    // mixed, sources packed; the scalar entry measures what packing buys
    MIXED(128, 8, 512, true, false),
    MIXED(64, 4, 256, true, false),
    MIXED(256, 4, 512, false, false),
    // softening 0
    MIXED(256, 4, 512, true, true),
    MIXED(64, 4, 256, true, true),
    F64(256, 2, 256, false),
    F64(128, 2, 256, false),
    F64(256, 1, 256, false),
    F64(128, 4, 256, false),
    F64(64, 2, 128, false),
    F64(256, 2, 256, true),
    F64(64, 2, 128, true),
    EXACT(16, 8, 2),
    EXSER(64, 128, 8),
    // twins of the fifth and the eighth mixed variant: the same tiles over other threads
    {kMixed, 512, 2, 512, 2, 0, (const void*)&force_mixed_tp_kernel<512, 2, 512, false, 1, 8>, 0, 4},
    {kMixed, 256, 1, 256, 1, 0, (const void*)&force_mixed_kernel<256, 1, 256, true, false>, 0, 7},
};
// Which exact variant (the two above, in that order) for n_tgt targets.  The serial kernel
// needs one thread per target and fills the SMs from 592 warps of targets up; below, and until
// its second round of warps is well filled, the cooperative one is faster in spite of the terms
// it passes through shared memory.  Measured with n targets and n sources, cooperative /
// serial: n = 1000 20 / 71 us, 4000 73 / 231, 16,384 821 / 886, 19,000 1195 / 1574, 30,000
// 2682 / 2483 us, 65,536 12.3 / 10.2 ms.
constexpr int64_t kExactCoopTargets = 27000;

constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

}  // namespace

const ForceVariant* force_variants(int* count) {
    *count = kNumVariants;
    return kVariants;
}

int force_variant_ids(int precision, int eps0, int* ids, int max_ids) {
    int c = 0;
    for (int i = 0; i < kNumVariants; ++i) {
        const ForceVariant& v = kVariants[i];
        if (v.precision != precision) continue;
        if (precision != kF64Exact && v.eps0 != eps0) continue;
        if (c < max_ids) ids[c] = i;
        ++c;
    }
    return c;
}

int64_t force_tiles(const ForceVariant& v, int64_t n_tgt) {
    const int64_t tile = v.targets ? v.targets : (int64_t)v.block * v.ipt;
    return (n_tgt + tile - 1) / tile;
}

int force_exact_variant(int64_t n_tgt) {
    static const int first = [] {
        int i = 0;
        while (kVariants[i].precision != kF64Exact) ++i;
        return i;
    }();
    return first + (n_tgt <= kExactCoopTargets ? 0 : 1);
}

cudaError_t force_launch(const ForceVariant& v, const ForceArgs& args, cudaStream_t stream) {
    if (args.n_tgt <= 0) return cudaSuccess;
    const int ns = v.precision == kF64Exact ? 1 : args.nsplit;
    const int64_t blocks = force_tiles(v, args.n_tgt) * ns;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    ForceArgs a = args;
    void* params[] = {(void*)&a};
    cudaError_t e = cudaLaunchKernel(v.fn, dim3((unsigned)blocks), dim3(v.block), params, 0, stream);
    if (e != cudaSuccess || args.nsplit <= 1 || args.tile_count) return e;
    force_reduce_kernel<<<(unsigned)((args.n_tgt + 255) / 256), 256, 0, stream>>>(a);
    return cudaGetLastError();
}

int force_occupancy(const ForceVariant& v) {
    static std::mutex mu;
    static int cache[64] = {0};
    const int idx = (int)(&v - kVariants);
    std::lock_guard<std::mutex> lock(mu);
    if (idx >= 0 && idx < 64 && cache[idx] > 0) return cache[idx];
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, v.fn, v.block, 0) != cudaSuccess || nb < 1) nb = 1;
    if (idx >= 0 && idx < 64) cache[idx] = nb;
    return nb;
}

}  // namespace gx
