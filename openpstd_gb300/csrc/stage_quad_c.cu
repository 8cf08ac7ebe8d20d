// four-strip stage kernel variants with a fused last pass, transform
// lengths 128 .. 512
#include "stage_quad.cuh"

namespace pstd {

const StageVariant* stage_variants_quad_c(int L, int* n) {
    static const StageVariant v128[] = {
        make_quad_variant<QCfg<128, 8, 128, 7, 4, 4, 8, 0, 0, 1>>("L128 quad8 nt128 mb7 r4.4.8 fused"),
        make_quad_variant<QCfg<128, 8, 128, 6, 8, 16, 0, 0, 0, 1>>("L128 quad8 nt128 mb6 r8.16 fused"),
        make_quad_variant<QCfg<128, 8, 64, 10, 16, 8, 0, 0, 0, 1>>("L128 quad8 nt64 mb10 r16.8 fused"),
        make_quad_variant<QCfg<128, 8, 128, 6, 4, 4, 8, 0, 0, 1>>("L128 quad8 nt128 mb6 r4.4.8 fused"),
    };
    static const StageVariant v256[] = {
        make_quad_variant<QCfg<256, 4, 128, 7, 4, 8, 8, 0, 0, 1>>("L256 quad4 nt128 mb7 r4.8.8 fused"),
        make_quad_variant<QCfg<256, 8, 128, 4, 16, 16, 0, 0, 0, 1>>("L256 quad8 nt128 mb4 r16.16 fused"),
    };
    static const StageVariant v512[] = {
        make_quad_variant<QCfg<512, 2, 128, 7, 8, 8, 8, 0, 0, 1>>("L512 quad2 nt128 mb7 r8.8.8 fused"),
        make_quad_variant<QCfg<512, 2, 128, 6, 8, 8, 8, 0, 0, 1>>("L512 quad2 nt128 mb6 r8.8.8 fused"),
    };
    switch (L) {
        case 128: *n = 4; return v128;
        case 256: *n = 2; return v256;
        case 512: *n = 2; return v512;
        default: *n = 0; return nullptr;
    }
}

}  // namespace pstd
