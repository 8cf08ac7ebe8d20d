// pml_post.cuh -- the PML multiply after the sixth stage, one block's share;
// used by its own kernels (misc.cu) and by the chained form's step kernel
// (stage_chain.cu).
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"

namespace pstd {

// After the sixth stage, for every PML domain (kernel/Solver.cpp:85,
// kernel/core/Domain.cpp:716-725): keep p0 = px + py from before the multiply
// (the reference does not recompute p0 after it), then px *= ax, py *= ay.
// vx and vy of non-rigid domains were attenuated in the stage epilogue; rigid
// domains (fields in the fixed buffer) get all four multiplies here.
// one (row, 128-column chunk) block `lb` of PML domain doms[idx[dj]]
__device__ __forceinline__ void pml_post_block(int dj, int lb, const int* idx, const DevDomain* doms, float* set,
                                               float* fixed, float* p0, const float* __restrict__ att) {
    const DevDomain d = doms[idx[dj]];
    float* base = d.fixed ? fixed : set;
    const int chunks = (d.nx + 1 + 127) >> 7;   // vx rows have nx + 1 columns
    const int r = lb / chunks, i = ((lb - r * chunks) << 7) + threadIdx.x;
    if (r < d.ny && i < d.nx) {
        const long long e = (long long)r * d.pitch_p + i;
        const float px = __ldcg(base + d.o_px + e), py = __ldcg(base + d.o_py + e);
        p0[d.o_p0 + e] = __fadd_rn(px, py);
        if (d.att_xp >= 0) base[d.o_px + e] = __fmul_rn(px, att[d.att_xp + i]);
        if (d.att_yp >= 0) base[d.o_py + e] = __fmul_rn(py, att[d.att_yp + r]);
    }
    if (d.fixed) {
        if (r < d.ny && i < d.nx + 1 && d.att_xv >= 0) {
            const long long e = d.o_vx + (long long)r * d.pitch_vx + i;
            base[e] = __fmul_rn(__ldcg(base + e), att[d.att_xv + i]);
        }
        if (r < d.ny + 1 && i < d.nx && d.att_yv >= 0) {
            const long long e = d.o_vy + (long long)r * d.pitch_vy + i;
            base[e] = __fmul_rn(__ldcg(base + e), att[d.att_yv + r]);
        }
    }
}

// the domain of flat block b: the last k with off[k] <= b (off ascends, off[0] = 0)
__device__ __forceinline__ int pml_domain_of(const int* off, int n, int b) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

}  // namespace pstd
