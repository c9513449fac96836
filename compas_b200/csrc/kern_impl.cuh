// Instantiation and launch of the stage kernels of one model and dimension (included once by each
// kern_*.cu translation unit).
#pragma once

#include <algorithm>
#include <type_traits>

#include "launch.h"
#include "stage_kernel.cuh"

namespace compas {

// Launch shapes of the stage kernels (threads per CTA, CTAs per SM) among which the autotuner picks;
// the tile is 8^3 in 3D and 16^2 in 2D for every shape. The register budget is set per SM
// sub-partition (16384 registers each, warps dealt round-robin). Shape 0 is the default where nothing is
// tuned and the tiles fill the GPU; default_shape (compas_b200.cu) has the rule for fewer.
//
// stage_tile (FACES = false): its passes have 512 (3D) or 18 x 16 x components (2D) reconstruction items and
// 576 or 272 faces, so 288 threads fill both nearly evenly; in 3D mixed, 320 (ten warps, the most that the
// registers of 288 leave room for) do better for being more warps. B200, us per stage: 128^3 SIXEQS WENO5
// mixed with 192 / 256 / 288 / 320 threads x 2 (TMA halos) 570 / 518 / 546 / 513, WENO5B 288 / 320 627 / 586;
// 96^3 FP64 288 x 2 / 576 x 1 / 384 x 1 764 / 810 / 888; 1024 x 512 FIVEEQS WENO5B mixed 144 x 4 / 192 x 3 /
// 288 x 2 87 / 93 / 95, FP64 288 x 2 / 192 x 3 / 144 x 4 254 / 276 / 298.
// stage_tile_faces (FACES = true): 576 (3D) or 272 (2D) faces a direction and one thread each.
template <bool FACES, int D, bool MIX, int S>
struct ShapeParams;
template <bool MIX> struct ShapeParams<false, 3, MIX, 0> { static constexpr int NT = MIX ? 320 : 288, MINB = 2; };
template <bool MIX> struct ShapeParams<false, 3, MIX, 1> { static constexpr int NT = 576, MINB = 1; };
template <> struct ShapeParams<false, 3, true, 2> { static constexpr int NT = 256, MINB = 2; };
template <> struct ShapeParams<false, 3, false, 2> { static constexpr int NT = 384, MINB = 1; };
template <> struct ShapeParams<false, 2, true, 0> { static constexpr int NT = 144, MINB = 4; };
template <> struct ShapeParams<false, 2, true, 2> { static constexpr int NT = 288, MINB = 2; };
template <> struct ShapeParams<false, 2, false, 0> { static constexpr int NT = 288, MINB = 2; };
template <> struct ShapeParams<false, 2, false, 2> { static constexpr int NT = 144, MINB = 4; };
template <bool MIX> struct ShapeParams<false, 2, MIX, 1> { static constexpr int NT = 512, MINB = 1; };
template <bool MIX> struct ShapeParams<true, 3, MIX, 0> { static constexpr int NT = 192, MINB = 2; };
template <bool MIX> struct ShapeParams<true, 3, MIX, 1> { static constexpr int NT = 256, MINB = 2; };
template <bool MIX> struct ShapeParams<true, 3, MIX, 2> { static constexpr int NT = 288, MINB = 2; };
template <bool MIX> struct ShapeParams<true, 2, MIX, 0> { static constexpr int NT = 272, MINB = 2; };
template <bool MIX> struct ShapeParams<true, 2, MIX, 1> { static constexpr int NT = 272, MINB = 1; };
template <bool MIX> struct ShapeParams<true, 2, MIX, 2> { static constexpr int NT = 136, MINB = 4; };

// In 2D, shape 1 of the single-box kernel takes 8^2 tiles: a box of few tiles is bound by the time of one
// tile, and four small ones on four SMs take a fraction of it (more halo, 2.5 conversions a cell for 1.75, so
// not where the larger tiles fill the GPU). LIST: the box-list kernel, whose tile counts are those of 16^2.
template <class M, bool FACES, bool MIX, int S, bool LIST = false>
struct LaunchShape {
    static constexpr bool SMALL = (M::D == 2 && !FACES && !LIST && S == 1);
    static constexpr int TS = SMALL ? kTile2 / 2 : (M::D == 2) ? kTile2 : kTile3;
    static constexpr int TZ = (M::D == 2) ? 1 : TS;
    static constexpr int NT = SMALL ? 192 : ShapeParams<FACES, M::D, MIX, S>::NT;
    static constexpr int MINB = SMALL ? 2 : ShapeParams<FACES, M::D, MIX, S>::MINB;
};

// One CTA per tile of the box.
template <class M, int SCHEME, bool MIX, int VAR, int SH>
static cudaError_t launch_stage_v(const StageArgs& a, cudaStream_t st) {
    using S = LaunchShape<M, SCHEME == 2 || VAR == kVarThinc, MIX, SH>;
    constexpr size_t SMEM = tile_smem<M, SCHEME, MIX, VAR, S::TS, S::TZ, S::MINB>();
    auto kern = stage_kernel<M, SCHEME, MIX, VAR, S::TS, S::TS, S::TZ, S::NT, S::MINB>;
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const long long tiles = a.tile_count > 0 ? (long long)a.tile_count
                                             : (long long)((a.g.n[0] + S::TS - 1) / S::TS) *
                                                   ((a.g.n[1] + S::TS - 1) / S::TS) * ((a.g.n[2] + S::TZ - 1) / S::TZ);
    kern<<<(unsigned)tiles, S::NT, SMEM, st>>>(a);
    return cudaGetLastError();
}

// One box with the y/z halo slabs staged by TMA (3D mixed form; the maps describe a.Us).
template <class M, int SCHEME, int SH>
static cudaError_t launch_stage_tma(const StageArgs& a, const TmaMaps& tm, cudaStream_t st) {
    using S = LaunchShape<M, false, true, SH>;
    constexpr size_t SMEM = tile_smem<M, SCHEME, true, kVarTma, S::TS, S::TZ, S::MINB>();
    auto kern = stage_kernel_tma<M, SCHEME, true, S::TS, S::TS, S::TZ, S::NT, S::MINB>;
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const long long tiles = a.tile_count > 0 ? (long long)a.tile_count
                                             : (long long)((a.g.n[0] + S::TS - 1) / S::TS) *
                                                   ((a.g.n[1] + S::TS - 1) / S::TS) * ((a.g.n[2] + S::TZ - 1) / S::TZ);
    kern<<<(unsigned)tiles, S::NT, SMEM, st>>>(a, tm);
    return cudaGetLastError();
}

template <class M, int SCHEME, bool MIX>
static cudaError_t launch_stage_var(const KernelChoice& k, const StageArgs& a, cudaStream_t st, const TmaMaps* tm) {
    if constexpr (SCHEME == 2) {
        // GODUNOV / MUSCL: the plain right-hand side, ordinary halo loads (the tuner's TMA candidate
        // runs this form too)
        if (k.phase_field || k.thinc) return cudaErrorNotSupported;
        switch (k.shape) {
            case 1: return launch_stage_v<M, 2, MIX, kVarPlain, 1>(a, st);
            case 2: return launch_stage_v<M, 2, MIX, kVarPlain, 2>(a, st);
            default: return launch_stage_v<M, 2, MIX, kVarPlain, 0>(a, st);
        }
    } else {
    if constexpr (M::D == 3 && MIX && M::KIND != kModelFiveN && M::KIND != kModelSixN) {
        if (tm && tm->valid && !k.thinc && !k.phase_field) {
            switch (k.shape) {
                case 1: return launch_stage_tma<M, SCHEME, 1>(a, *tm, st);
                case 2: return launch_stage_tma<M, SCHEME, 2>(a, *tm, st);
                default: return launch_stage_tma<M, SCHEME, 0>(a, *tm, st);
            }
        }
    }
    if constexpr (M::KIND == kModelFiveN || M::KIND == kModelSixN) {
        // FIVEEQS_NPHASE, SIXEQS_IE_NPHASE: the plain hyperbolic right-hand side only
        if (k.phase_field || k.thinc) return cudaErrorNotSupported;
    } else {
        // the THINC and Phase-Field variants run at shape 0
        if (k.phase_field) return launch_stage_v<M, SCHEME, MIX, kVarPhaseField, 0>(a, st);
        if (k.thinc) return launch_stage_v<M, SCHEME, MIX, kVarThinc, 0>(a, st);
    }
    switch (k.shape) {
        case 1: return launch_stage_v<M, SCHEME, MIX, kVarPlain, 1>(a, st);
        case 2: return launch_stage_v<M, SCHEME, MIX, kVarPlain, 2>(a, st);
        default: return launch_stage_v<M, SCHEME, MIX, kVarPlain, 0>(a, st);
    }
    }
}

// The kernels of one precision form (MIX); the two forms are separate translation units (built in
// parallel).
template <class M, bool MIX>
static cudaError_t launch_stage_m(const KernelChoice& k, const StageArgs& a, cudaStream_t st, const TmaMaps* tm) {
    if (k.limiter < 5) return launch_stage_var<M, 2, MIX>(k, a, st, tm);  // GODUNOV / MUSCL / WENO3 family
    return (k.limiter == 6) ? launch_stage_var<M, 6, MIX>(k, a, st, tm) : launch_stage_var<M, 5, MIX>(k, a, st, tm);
}

// Persistent box-list launch: one resident wave of CTAs walks the tiles of every box.
template <class M, int SCHEME, bool MIX, int SH>
static cudaError_t launch_list_v(const ListArgs& L, cudaStream_t st) {
    using S = LaunchShape<M, SCHEME == 2, MIX, SH, true>;
    constexpr size_t SMEM = tile_smem<M, SCHEME, MIX, kVarPlain, S::TS, S::TZ, S::MINB>();
    auto kern = stage_list_kernel<M, SCHEME, MIX, S::TS, S::TS, S::TZ, S::NT, S::MINB>;
    static int grid = 0;
    if (!grid) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
        if (e != cudaSuccess) return e;
        int dev = 0, sms = 0, per = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, S::NT, SMEM)) != cudaSuccess) return e;
        grid = sms * std::max(per, 1);
    }
    kern<<<grid, S::NT, SMEM, st>>>(L);
    return cudaGetLastError();
}

template <class M, int SCHEME, bool MIX>
static cudaError_t launch_list_s(const KernelChoice& k, const ListArgs& L, cudaStream_t st) {
    switch (k.shape) {
        case 1: return launch_list_v<M, SCHEME, MIX, 1>(L, st);
        case 2: return launch_list_v<M, SCHEME, MIX, 2>(L, st);
        default: return launch_list_v<M, SCHEME, MIX, 0>(L, st);
    }
}

template <class M, bool MIX>
static cudaError_t launch_list_m(const KernelChoice& k, const ListArgs& L, cudaStream_t st) {
    if (k.limiter < 5) return launch_list_s<M, 2, MIX>(k, L, st);  // GODUNOV / MUSCL / WENO3 family
    return (k.limiter == 6) ? launch_list_s<M, 6, MIX>(k, L, st) : launch_list_s<M, 5, MIX>(k, L, st);
}

}  // namespace compas

// PREC 0: the plain FP64 form (launch_*_<name>_p0), PREC 1: the mixed form (launch_*_<name>_p1).
#define COMPAS_DEFINE_LAUNCHERS(name, Model, PREC)                                                   \
    namespace compas {                                                                              \
    cudaError_t launch_stage_##name##_p##PREC(const KernelChoice& k, const StageArgs& a, cudaStream_t st, \
                                              const TmaMaps* tm) {                                  \
        return launch_stage_m<Model, PREC == 1>(k, a, st, tm);                                      \
    }                                                                                               \
    cudaError_t launch_list_##name##_p##PREC(const KernelChoice& k, const ListArgs& L, cudaStream_t st) { \
        return launch_list_m<Model, PREC == 1>(k, L, st);                                           \
    }                                                                                               \
    }
