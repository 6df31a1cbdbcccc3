// vjp.cuh -- launcher of the adjoint (vector-Jacobian product) kernel.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gx {

struct VjpArgs {
    const double* x;
    const double* y;
    const double* z;
    const double* m;
    const double* lx;  // cotangent on the accelerations
    const double* ly;
    const double* lz;
    int64_t n;
    int64_t j_chunk;  // sources per chunk, a multiple of the variant's jt
    int nsplit;       // chunks
    double* gx;
    double* gy;
    double* gz;
    double* gm;    // nullable
    double* part;  // nsplit * 4 * n when nsplit > 1
    unsigned* tile_count;  // then also one zeroed ticket per target tile
    double G;
    double eps2;
    float eps2f;
};

struct VjpVariant {
    int precision, block, ipt, jt;
    bool eps0;
    const void* fn;
};
// The variant and the source split for n bodies.
const VjpVariant& vjp_variant(int64_t n, int precision, bool eps0);
int vjp_split(const VjpVariant& v, int64_t n, int sms);
inline int64_t vjp_tiles(const VjpVariant& v, int64_t n) {
    const int64_t tile = (int64_t)v.block * v.ipt;
    return (n + tile - 1) / tile;
}
cudaError_t launch_vjp(const VjpVariant& v, const VjpArgs& a, cudaStream_t st);

}  // namespace gx
