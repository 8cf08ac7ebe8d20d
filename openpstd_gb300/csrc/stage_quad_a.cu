// four-strip stage kernel variants for transform lengths 32 .. 512
#include "stage_quad.cuh"

namespace pstd {

const StageVariant* stage_variants_quad_a(int L, int* n) {
    static const StageVariant v32[] = {
        make_quad_variant<QCfg<32, 8, 64, 8, 8, 4>>("L32 quad8 nt64 r8.4"),
    };
    static const StageVariant v64[] = {
        make_quad_variant<QCfg<64, 8, 64, 8, 8, 8>>("L64 quad8 nt64 r8.8"),
    };
    static const StageVariant v128[] = {
        make_quad_variant<QCfg<128, 8, 128, 6, 8, 16>>("L128 quad8 nt128 r8.16"),
        make_quad_variant<QCfg<128, 8, 128, 7, 4, 4, 8>>("L128 quad8 nt128 r4.4.8"),
        make_quad_variant<QCfg<128, 8, 128, 6, 4, 4, 8>>("L128 quad8 nt128 mb6 r4.4.8"),
        make_quad_variant<QCfg<128, 8, 64, 10, 16, 8>>("L128 quad8 nt64 r16.8"),
        make_quad_variant<QCfg<128, 16, 128, 5, 16, 8>>("L128 quad16 nt128 r16.8"),
        make_quad_variant<QCfg<128, 4, 64, 14, 4, 4, 8, 0, 1>>("L128 quad4 nt64 r4.4.8 tsm"),
    };
    static const StageVariant v256[] = {
        make_quad_variant<QCfg<256, 8, 128, 5, 16, 16>>("L256 quad8 nt128 r16.16"),
        make_quad_variant<QCfg<256, 4, 128, 7, 4, 8, 8>>("L256 quad4 nt128 r4.8.8"),
        make_quad_variant<QCfg<256, 8, 256, 3, 4, 8, 8>>("L256 quad8 nt256 r4.8.8"),
        make_quad_variant<QCfg<256, 2, 64, 12, 4, 8, 8, 0, 1>>("L256 quad2 nt64 r4.8.8 tsm"),
    };
    static const StageVariant v512[] = {
        make_quad_variant<QCfg<512, 2, 128, 7, 8, 8, 8>>("L512 quad2 nt128 r8.8.8"),
        make_quad_variant<QCfg<512, 2, 128, 6, 8, 8, 8>>("L512 quad2 nt128 mb6 r8.8.8"),
        make_quad_variant<QCfg<512, 4, 256, 3, 8, 8, 8>>("L512 quad4 nt256 r8.8.8"),
        make_quad_variant<QCfg<512, 1, 64, 14, 8, 8, 8>>("L512 quad1 nt64 r8.8.8"),
        make_quad_variant<QCfg<512, 2, 128, 6, 8, 8, 8, 0, 1>>("L512 quad2 nt128 r8.8.8 tsm"),
        make_quad_variant<QCfg<512, 1, 64, 12, 8, 8, 8, 0, 1>>("L512 quad1 nt64 r8.8.8 tsm"),
    };
    switch (L) {
        case 32: *n = 1; return v32;
        case 64: *n = 1; return v64;
        case 128: *n = 6; return v128;
        case 256: *n = 4; return v256;
        case 512: *n = 6; return v512;
        default: *n = 0; return nullptr;
    }
}

}  // namespace pstd
