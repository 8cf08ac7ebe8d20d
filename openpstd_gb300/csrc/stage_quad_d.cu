// four-strip stage kernel variants with a fused last pass, transform
// lengths 1024 .. 8192
#include "stage_quad.cuh"

namespace pstd {

const StageVariant* stage_variants_quad_d(int L, int* n) {
    static const StageVariant v1024[] = {
        make_quad_variant<QCfg<1024, 2, 128, 4, 16, 8, 8, 0, 0, 1>>("L1024 quad2 nt128 mb4 r16.8.8 fused"),
        make_quad_variant<QCfg<1024, 1, 128, 7, 8, 16, 8, 0, 0, 1>>("L1024 quad1 nt128 mb7 r8.16.8 fused"),
        make_quad_variant<QCfg<1024, 1, 64, 8, 16, 8, 8, 0, 0, 1>>("L1024 quad1 nt64 mb8 r16.8.8 fused"),
    };
    static const StageVariant v2048[] = {
        make_quad_variant<QCfg<2048, 1, 128, 4, 16, 16, 8, 0, 0, 1>>("L2048 quad1 nt128 mb4 r16.16.8 fused"),
        make_quad_variant<QCfg<2048, 2, 256, 2, 16, 16, 8, 0, 0, 1>>("L2048 quad2 nt256 mb2 r16.16.8 fused"),
        make_quad_variant<QCfg<2048, 1, 256, 3, 4, 8, 8, 8, 0, 1>>("L2048 quad1 nt256 mb3 r4.8.8.8 fused"),
    };
    static const StageVariant v4096[] = {
        make_quad_variant<QCfg<4096, 1, 256, 2, 16, 16, 16, 0, 0, 1>>("L4096 quad1 nt256 mb2 r16.16.16 fused"),
        make_quad_variant<QCfg<4096, 1, 256, 3, 8, 8, 8, 8, 0, 1>>("L4096 quad1 nt256 mb3 r8.8.8.8 fused"),
    };
    static const StageVariant v8192[] = {
        make_quad_variant<QCfg<8192, 1, 512, 1, 16, 8, 8, 8, 0, 1>>("L8192 quad1 nt512 mb1 r16.8.8.8 fused"),
        make_quad_variant<QCfg<8192, 1, 1024, 1, 16, 8, 8, 8, 0, 1>>("L8192 quad1 nt1024 mb1 r16.8.8.8 fused"),
    };
    switch (L) {
        case 1024: *n = 3; return v1024;
        case 2048: *n = 3; return v2048;
        case 4096: *n = 2; return v4096;
        case 8192: *n = 2; return v8192;
        default: *n = 0; return nullptr;
    }
}

}  // namespace pstd
