// dg_stage_p4.cu -- compiled launch variants of the stage kernel for order p = 4
// (elements per CTA, threads per CTA, variable groups, residual arithmetic; then the
// optional flags: all groups' pencils in one phase, single coefficient buffer, unfused
// volume, row-split traces and lifts, one face-flux point per thread, face fluxes from
// the face kernel, face lifts added in the inverse mass's first pass; then the minimum
// of resident CTAs per SM asked of the compiler).  Contexts on non-affine meshes use the
// general-geometry (kGE) entries only, the others never do.  The
// first variant of each precision whose threshold of elements per SM the mesh reaches is
// the default (the measured best); dg_tune_stage may pick another.
#include "dg_stage.cuh"
#include "dg_small.cuh"

namespace dgk {

static const StageVariant kVariants4[] = {
    make_small_variant<4, 1, 64, 2, 4, 1, double>(make_column_variant<4, 1, 64, double, 4, 5, 64, 1>(0)),
    make_column_variant<4, 1, 64, double, 4, 5, 64, 1>(0),
    make_variant<4, 1, 128, 1, double, kUF | kSB | kFX | kMG, 4>(),
    make_variant<4, 1, 128, 1, double, kUF | kSB | kFX, 4>(),
    make_variant<4, 1, 128, 1, double, kUF | kRS | kSB | kK1, 4>(),
    make_variant<4, 1, 128, 1, double, kUF | kRS | kSB | kK1>(),
    make_variant<4, 1, 64, 2, double>(),
    make_small_variant<4, 1, 64, 3, 6, 1, float>(make_column_variant<4, 1, 64, float, 8, 5, 64, 1>(0)),
    make_column_variant<4, 1, 64, float, 8, 5, 64, 1>(0),
    make_variant<4, 1, 128, 1, float, kUF | kSB | kFX | kMG>(),
    make_variant<4, 1, 128, 1, float, kUF | kSB | kFX>(),
    make_variant<4, 1, 128, 1, float, kUF | kSB>(),
    make_variant<4, 1, 128, 1, float, kUF | kRS | kSB>(),
    make_variant<4, 1, 128, 2, float, kPZ>(),
    // general (trilinear) geometry: the variants of non-affine meshes.  In
    // mixed precision with the face kernel 119 -> 96 us per RK stage at 13^3 bent
    // elements, from 3 elements per SM (8^3: 32.5 -> 26.5, 6^3: 16.4 against 18.5).  The
    // FP64 column form is slower here (131 against 118 us: four CTAs per SM for want of
    // registers do not cover the 125 KB matrix of each element)
    make_variant<4, 1, 128, 1, double, kUF | kRS | kSB | kK1 | kGE>(),
    from_per_sm(make_variant<4, 1, 128, 1, float, kUF | kSB | kGE | kFX>(), 3),
    make_variant<4, 1, 128, 1, float, kUF | kSB | kGE>(),
    make_variant<4, 1, 96, 1, double, kUF | kRS | kSB | kK1 | kGE>(),
    make_variant<4, 1, 128, 1, double, kUF | kRS | kSB | kGE | kFX>(),
};

int stage_variants_p4(const StageVariant** out)
{
    *out = kVariants4;
    return static_cast<int>(sizeof(kVariants4) / sizeof(kVariants4[0]));
}

}  // namespace dgk
