// stage_chain.cu -- the chained form: one launch per RK stage over the
// four-strip jobs of every transform length, launched with programmatic stream
// serialisation, and one launch after the sixth stage for the PML multiply,
// the receivers and the step flags.
//
// Per-length launches fork and join the lengths of every stage: a stage of a
// small scene (200 x 200 cells, lengths 128 and 512) took 13-14 us of which the
// kernels' data moves need well under one.  Here a stage is one node, its CTAs
// are resident (with job record and tables read) when the previous stage ends,
// and a step is seven nodes in a row instead of fifteen with forks.
//
// Three families: 0 has small jobs of 128 threads and tables in shared memory
// (many SMs: scenes that do not fill the GPU); 1 has 256 threads and more
// strips per job; 2 has family 0's jobs with 256 threads and smaller radices,
// because in a small scene a stage lasts as long as its last CTA and a CTA as
// long as one thread's passes.  Step of the 200 x 200 scene: per-length launches
// 61 us, family 0 55, 1 66, 2 49; of a 611 x 405 scene in six domains: 93, 89,
// 86, 109.  The plan times them on the scene's own steps against the per-length
// launches and keeps the fastest.
#include "pml_post.cuh"
#include "stage_quad.cuh"

namespace pstd {

struct ChainFam0 {
    static constexpr int NT = 128, MINB = 4;
    using C32 = QCfg<32, 4, 128, 4, 8, 4, 0, 0, 1>;
    using C64 = QCfg<64, 4, 128, 4, 8, 8, 0, 0, 1>;
    using C128 = QCfg<128, 4, 128, 4, 4, 4, 8, 0, 1>;
    using C256 = QCfg<256, 2, 128, 4, 4, 8, 8, 0, 1>;
    using C512 = QCfg<512, 2, 128, 4, 8, 8, 8, 0, 1>;
    using C1024 = QCfg<1024, 1, 128, 4, 4, 4, 8, 8, 1>;
    using C2048 = QCfg<2048, 1, 128, 4, 4, 8, 8, 8, 1>;
    using C4096 = QCfg<4096, 1, 128, 4, 8, 8, 8, 8, 1>;
    using C8192 = QCfg<8192, 1, 128, 4, 16, 8, 8, 8, 0>;
};
struct ChainFam1 {
    static constexpr int NT = 256, MINB = 3;
    using C32 = QCfg<32, 16, 256, 3, 8, 4>;
    using C64 = QCfg<64, 16, 256, 3, 8, 8>;
    using C128 = QCfg<128, 16, 256, 3, 4, 4, 8>;
    using C256 = QCfg<256, 8, 256, 3, 4, 8, 8>;
    using C512 = QCfg<512, 4, 256, 3, 8, 8, 8>;
    using C1024 = QCfg<1024, 2, 256, 3, 4, 4, 8, 8>;
    using C2048 = QCfg<2048, 1, 256, 3, 4, 8, 8, 8>;
    using C4096 = QCfg<4096, 1, 256, 3, 8, 8, 8, 8>;
    using C8192 = QCfg<8192, 1, 256, 3, 16, 8, 8, 8>;
};

// family 0's job sizes with twice the threads and smaller radices: shorter
// passes for the last CTA of a stage
struct ChainFam2 {
    static constexpr int NT = 256, MINB = 2;
    using C32 = QCfg<32, 8, 256, 2, 4, 8, 0, 0, 1>;
    using C64 = QCfg<64, 8, 256, 2, 4, 4, 4, 0, 1>;
    using C128 = QCfg<128, 8, 256, 2, 4, 4, 8, 0, 1>;
    using C256 = QCfg<256, 4, 256, 2, 4, 4, 4, 4, 1>;
    using C512 = QCfg<512, 2, 256, 2, 4, 4, 4, 8, 1>;
    using C1024 = QCfg<1024, 1, 256, 2, 4, 4, 8, 8, 1>;
    using C2048 = QCfg<2048, 1, 256, 2, 4, 8, 8, 8, 1>;
    using C4096 = QCfg<4096, 1, 256, 2, 8, 8, 8, 8, 1>;
    using C8192 = QCfg<8192, 1, 256, 2, 16, 8, 8, 8, 0>;
};

// (not inlined: every length keeps its own register allocation)
template <class C>
__device__ __noinline__ void chain_job(float4* sm, const StageArgs& A, const QJob& J, int tid) {
    quad_job<C>(sm, A, J, A.tw + J.ttab, tid);
}

template <class F>
__global__ void __launch_bounds__(F::NT, F::MINB) stage_chain(const __grid_constant__ StageArgs A) {
    extern __shared__ __align__(16) float4 smc[];
    const QJob& J = A.qjobs[blockIdx.x];
    const int tid = threadIdx.x;
    if (J.kind & JK_COPY) {
        grid_wait();
        grid_release();
        copy_axis<F::NT>(A, A.doms[J.dom], J.kind & JK_Y, tid);
        return;
    }
    switch (J.L) {
        case 32: chain_job<typename F::C32>(smc, A, J, tid); break;
        case 64: chain_job<typename F::C64>(smc, A, J, tid); break;
        case 128: chain_job<typename F::C128>(smc, A, J, tid); break;
        case 256: chain_job<typename F::C256>(smc, A, J, tid); break;
        case 512: chain_job<typename F::C512>(smc, A, J, tid); break;
        case 1024: chain_job<typename F::C1024>(smc, A, J, tid); break;
        case 2048: chain_job<typename F::C2048>(smc, A, J, tid); break;
        case 4096: chain_job<typename F::C4096>(smc, A, J, tid); break;
        case 8192: chain_job<typename F::C8192>(smc, A, J, tid); break;
        default: break;
    }
}

template <class F>
static const StageVariant* chain_variants(int L) {
    static const StageVariant v[] = {
        make_quad_variant<typename F::C32>("L32 (chained)"),     make_quad_variant<typename F::C64>("L64 (chained)"),
        make_quad_variant<typename F::C128>("L128 (chained)"),   make_quad_variant<typename F::C256>("L256 (chained)"),
        make_quad_variant<typename F::C512>("L512 (chained)"),   make_quad_variant<typename F::C1024>("L1024 (chained)"),
        make_quad_variant<typename F::C2048>("L2048 (chained)"), make_quad_variant<typename F::C4096>("L4096 (chained)"),
        make_quad_variant<typename F::C8192>("L8192 (chained)"),
    };
    for (const StageVariant& x : v)
        if (x.L == L) return &x;
    return nullptr;
}

const StageVariant* chain_variant(int L, int fam) {
    return fam == 2 ? chain_variants<ChainFam2>(L) : fam == 1 ? chain_variants<ChainFam1>(L) : chain_variants<ChainFam0>(L);
}

template <class F>
static cudaError_t prepare_fam() {
    return cudaFuncSetAttribute(stage_chain<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, F::C8192::SMEM);
}
cudaError_t prepare_chain(int fam) {
    return fam == 2 ? prepare_fam<ChainFam2>() : fam == 1 ? prepare_fam<ChainFam1>() : prepare_fam<ChainFam0>();
}

// launch `kernel` so that it may start while its predecessor in the stream drains
template <class... P, class... Q>
static cudaError_t launch_pdl(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st, Q&&... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e == cudaErrorNotSupported || e == cudaErrorInvalidValue) {   // a stream without the attribute: plain order
        cudaGetLastError();
        cfg.numAttrs = 0;
        e = cudaLaunchKernelEx(&cfg, kernel, args...);
    }
    return e;
}

cudaError_t launch_chain(int fam, int n_jobs, const StageArgs& a, size_t smem, cudaStream_t st) {
    if (n_jobs <= 0) return cudaSuccess;
    return fam == 2   ? launch_pdl(stage_chain<ChainFam2>, n_jobs, ChainFam2::NT, smem, st, a)
           : fam == 1 ? launch_pdl(stage_chain<ChainFam1>, n_jobs, ChainFam1::NT, smem, st, a)
                      : launch_pdl(stage_chain<ChainFam0>, n_jobs, ChainFam0::NT, smem, st, a);
}

// After the sixth stage: blocks below `pml_blocks` do the PML multiply
// (pml_post_block), the block after them the receivers (receiver_kernel's
// sample: they read air domains, the multiply writes PML domains) and clears
// the scenes' first-step flags.
__global__ void __launch_bounds__(128) step_post_kernel(const int* idx, int n_pml, const int* off, int pml_blocks,
                                                        const DevDomain* doms, float* set, float* fixed, float* p0,
                                                        const float* __restrict__ att, const DevReceiver* rec, int n_rec,
                                                        float* ring, int ring_cap, int* counter, int* first_step,
                                                        int n_scenes) {
    int dj = 0;
    if ((int)blockIdx.x < pml_blocks) dj = pml_domain_of(off, n_pml, (int)blockIdx.x);
    grid_wait();
    grid_release();
    if ((int)blockIdx.x < pml_blocks) {
        pml_post_block(dj, (int)blockIdx.x - off[dj], idx, doms, set, fixed, p0, att);
        return;
    }
    for (int i = threadIdx.x; i < n_scenes; i += blockDim.x) first_step[i] = 0;
    if (!ring) return;   // spectral receivers have their own launches
    const int step = *counter;
    for (int r = threadIdx.x; r < n_rec; r += blockDim.x) {
        const DevReceiver q = rec[r];
        const DevDomain& d = doms[q.dom];
        const long long e = (long long)q.row * d.pitch_p + q.col;
        ring[(long long)(step % ring_cap) * n_rec + r] = __fadd_rn(set[d.o_px + e], set[d.o_py + e]);
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = step + 1;
}

cudaError_t launch_step_post(const int* idx, int n_pml, const int* off, int pml_blocks, const DevDomain* doms, float* set,
                             float* fixed, float* p0, const float* att, const DevReceiver* rec, int n_rec, float* ring,
                             int ring_cap, int* counter, int* first_step, int n_scenes, cudaStream_t st) {
    if (n_pml <= 0) pml_blocks = 0;
    return launch_pdl(step_post_kernel, pml_blocks + 1, 128, 0, st, idx, n_pml, off, pml_blocks, doms, set, fixed, p0, att,
                      rec, n_rec, ring, ring_cap, counter, first_step, n_scenes);
}

}  // namespace pstd
