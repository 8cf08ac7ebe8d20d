// stage_serve.cu -- the stage kernel configurations of the serving loop's
// per-length persistent form: one per transform length, each compiled as
// the device-count kernel (stage_quad_dev).  They are the
// configurations the autotuner picks on batches of scenes like the serving
// stream (cells log-uniform 64x64 .. 1024x768, 50-cell PML), so a server
// gets tuned arithmetic without timing variants on live scenes.  Each is also
// in the length's list of variants (a solo run pinned to it computes the same).
#include "stage_quad.cuh"

namespace pstd {

const StageVariant* serve_variant(int L) {
    static const StageVariant v[] = {
        make_quad_dev_variant<QCfg<32, 8, 64, 8, 8, 4>>("L32 quad8 nt64 r8.4 (serving)"),
        make_quad_dev_variant<QCfg<64, 8, 64, 8, 8, 8>>("L64 quad8 nt64 r8.8 (serving)"),
        make_quad_dev_variant<QCfg<128, 8, 128, 7, 4, 4, 8>>("L128 quad8 nt128 r4.4.8 (serving)"),
        make_quad_dev_variant<QCfg<256, 4, 128, 7, 4, 8, 8>>("L256 quad4 nt128 r4.8.8 (serving)"),
        make_quad_dev_variant<QCfg<512, 2, 128, 7, 8, 8, 8>>("L512 quad2 nt128 r8.8.8 (serving)"),
        make_quad_dev_variant<QCfg<1024, 2, 128, 4, 16, 8, 8>>("L1024 quad2 nt128 r16.8.8 (serving)"),
        make_quad_dev_variant<QCfg<2048, 2, 256, 2, 16, 16, 8>>("L2048 quad2 nt256 r16.16.8 (serving)"),
        make_quad_dev_variant<QCfg<4096, 1, 256, 3, 8, 8, 8, 8>>("L4096 quad1 nt256 r8.8.8.8 (serving)"),
        make_quad_dev_variant<QCfg<8192, 1, 512, 1, 16, 8, 8, 8>>("L8192 quad1 nt512 r16.8.8.8 (serving)"),
    };
    for (const StageVariant& x : v)
        if (x.L == L) return &x;
    return nullptr;
}

}  // namespace pstd
