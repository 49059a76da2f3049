// dg_stage_p5.cu -- compiled launch variants of the stage kernel for order p = 5
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

static const StageVariant kVariants5[] = {
    make_small_variant<5, 1, 128, 1, 4, 1, double>(make_column_variant<5, 1, 64, double, 4, 5, 64, 1>(0)),
    make_small_variant<5, 1, 64, 2, 4, 1, double>(make_column_variant<5, 1, 64, double, 4, 5, 64, 1>(0)),
    make_column_variant<5, 1, 64, double, 4, 5, 64, 1>(0),
    make_variant<5, 1, 256, 1, double, kUF | kRS | kSB | kFX | kMG, 2>(),
    make_variant<5, 1, 256, 1, double, kUF | kRS | kSB | kFX, 2>(),
    make_variant<5, 1, 128, 1, double, kUF | kRS | kSB | kFX>(),
    // forward Euler and residuals beside the one-launch RK4 steps: one launch, ahead of
    // the column form's two up to the largest such mesh (an update, 3^3 elements 18.8 ->
    // 12.7 us, 6^3 22.7 -> 18.4; p <= 4: column form ahead or equal)
    beside_small(make_variant<5, 1, 256, 1, double, kUF | kRS | kSB | kK1, 2>()),
    make_variant<5, 1, 128, 3, double>(),
    make_small_variant<5, 1, 96, 2, 6, 1, float>(make_column_variant<5, 1, 64, float, 6, 8, 128, 1>(0)),
    make_small_variant<5, 1, 64, 3, 6, 1, float>(make_column_variant<5, 1, 64, float, 6, 8, 128, 1>(0)),
    make_column_variant<5, 1, 64, float, 6, 8, 128, 1>(0),
    make_variant<5, 1, 256, 1, float, kUF | kSB | kFX | kMG, 3>(),
    make_variant<5, 1, 128, 1, float, kUF | kRS | kSB | kFX>(),
    make_variant<5, 1, 256, 1, float, kUF | kSB | kFX, 3>(),
    make_variant<5, 1, 256, 1, float, kUF | kRS | kSB | kK1, 3>(),
    make_variant<5, 1, 128, 2, float, kSB>(),
    make_variant<5, 1, 64, 2, float>(),
    // general (trilinear) geometry: the variants of non-affine meshes.  With
    // the face kernel 137 -> 126 us per RK stage at 10^3 bent elements in FP64 (8^3:
    // 70.7 against 71.2), from 4 elements per SM; in mixed precision 153 -> 143, left to
    // dg_tune_stage because its FP32 sums round differently from the default's (1e-9 of
    // the state after a few steps).  The FP64 column form takes 168 us
    from_per_sm(make_variant<5, 1, 256, 1, double, kUF | kRS | kSB | kGE | kFX, 2>(), 4),
    make_variant<5, 1, 256, 1, double, kUF | kRS | kSB | kK1 | kGE, 2>(),
    make_variant<5, 1, 128, 1, float, kUF | kRS | kSB | kK1 | kGE>(),
    make_variant<5, 1, 128, 1, double, kUF | kRS | kSB | kK1 | kGE>(),
    make_variant<5, 1, 256, 1, float, kUF | kRS | kSB | kK1 | kGE, 3>(),
    make_variant<5, 1, 256, 1, float, kUF | kRS | kSB | kGE | kFX, 3>(),
};

int stage_variants_p5(const StageVariant** out)
{
    *out = kVariants5;
    return static_cast<int>(sizeof(kVariants5) / sizeof(kVariants5[0]));
}

}  // namespace dgk
