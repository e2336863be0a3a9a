// tile.cuh - the register tile kernels' work units, shared by the two-phase
// kernels (step.cu) and the interleaved step kernel (step_inter.cu): the
// V-phase and T-phase arithmetic of one 4-cell chunk (whole or one output
// group at a time), the tile geometry, and the per-tile unit loop.
//
// Reference kernels: FD_V Float/main.cu:64-192, Half/main.cu:156-268; FD_T
// Float/main.cu:194-295, Half/main.cu:270-371.
#pragma once
#include <type_traits>

#include "post.cuh"
#include "shot.h"

namespace bpk {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kSegCells = 128;
// 3D tiles: the 8 rows of a tile are 8/TZ consecutive y rows of TZ consecutive
// z planes, so the z neighbours of most rows are rows of the same tile (2D
// tiles are 8 consecutive z rows).  Measured on B200 (192^3, 200^3 order 4,
// 552 x 552 x 424; all shapes bit-identical): FP32 is fastest with 1 x 8
// (up to 8 % over 8 x 1), COMP16, in the register kernels that order 4 still
// runs, with 4 x 2.
__host__ __device__ constexpr int tile_tz(int prec) {
    return prec == BP_PREC_FP32 ? 8 : (prec == BP_PREC_COMP16 ? 2 : 1);
}

// Binary search of the shot owning tile t (tile0 ascending).
__device__ __forceinline__ int locate_shot(const ShotDesc* shots, int nshots, long long t) {
    int lo = 0, hi = nshots - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (shots[mid].tile0 <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

#ifndef BP_RS_SPLIT
#define BP_RS_SPLIT 1
#endif
// Resident CTAs per SM the 2D phase kernels are register-limited to (1 = no
// limit).  Measured on B200 for the 4040 x 2040 order-2 grid: FP32 is fastest
// at 3 (80 registers; the V phase spills 12-16 bytes, 40 in the form for tiles of
// more units than warps); FP64 at 2 (128 registers; uncapped it takes ~150, one
// CTA per SM, and runs 40 % slower).  2D COMP16 runs the staged kernels, whose
// caps are in step_async.cu.
#ifndef BP_MINB_F32
#define BP_MINB_F32 3
#endif
#ifndef BP_MINB_F64
#define BP_MINB_F64 2
#endif
// 3D: uncapped, the kernels take 128-240 registers.  FP32 is fastest at 2 CTAs
// (128 registers, no spills) now that a chunk's memory variables and
// coefficients are loaded in batches: us per step on B200 at 3 -> 2 CTAs, 200^3
// order 2 557 -> 417, order 4 588 -> 444, 104^3 order 4 123 -> 83, 140 x 130 x
// 120 199 -> 147, and 192^3 with the reference's rounding 525 -> 405.  COMP16
// (order 4), taken one output group at a time (v_chunk_g/t_chunk_g, next to no
// spills), is fastest at 4 CTAs (64 registers) on the 552 x 552 x 424 and 200^3
// grids; FP64 at 2 (128 registers; uncapped it takes 196-240, one CTA per SM).
#ifndef BP_MINB3_F32
#define BP_MINB3_F32 2
#endif
#ifndef BP_MINB3_C16
#define BP_MINB3_C16 4
#endif
#ifndef BP_MINB3_F64
#define BP_MINB3_F64 2
#endif
// Compensated-BF16 storage (FP32 arithmetic, 3-byte values, a two-instruction
// decode): its own caps.
#ifndef BP_MINB_B24
#define BP_MINB_B24 3
#endif
#ifndef BP_MINB_B24_V
#define BP_MINB_B24_V 3
#endif
// (3D at 2 CTAs: 140 x 130 x 120 order 4 198 -> 184 us per step, 296 x 296 x 232
// 1462 -> 1437, against 3)
#ifndef BP_MINB3_B24
#define BP_MINB3_B24 2
#endif
template <int DIM, int ORD, class P, bool VPHASE>
__host__ __device__ constexpr int phase_min_blocks() {
    if (P::store == BP_PREC_CBF16) return DIM == 3 ? BP_MINB3_B24 : (VPHASE ? BP_MINB_B24_V : BP_MINB_B24);
    if (DIM == 3) return P::prec == BP_PREC_FP32 ? BP_MINB3_F32 : P::prec == BP_PREC_COMP16 ? BP_MINB3_C16 : BP_MINB3_F64;
    return P::prec == BP_PREC_FP32 ? BP_MINB_F32 : BP_MINB_F64;
}
// How a tile learns its step index: 1 = once per shot per launch, 0 = a read
// of the step counter per tile (measured faster for FP32 at 80 registers).
#ifndef BP_TILE_LOOP_F32
#define BP_TILE_LOOP_F32 0
#endif
#ifndef BP_TILE_LOOP_C16
#define BP_TILE_LOOP_C16 1
#endif
template <class P>
__host__ __device__ constexpr bool step_once_per_shot() {
    return P::prec == BP_PREC_COMP16 ? BP_TILE_LOOP_C16 : P::prec == BP_PREC_FP32 ? BP_TILE_LOOP_F32 : 1;
}

// Phases whose neighbour-field and coefficient loads take the read-only path
// (bit 0 = V, bit 1 = T), for the whole-chunk form of FP32.  Measured on B200:
// the T phase 2.5 % faster in 2D (4040 x 2040) and 1-2 % in 3D (192^3, 200^3
// order 4, 552 x 552 x 424); the V phase unchanged in 2D, up to 4 % slower in 3D.
#ifndef BP_NC_F32_2D
#define BP_NC_F32_2D 2
#endif
#ifndef BP_NC_F32_3D
#define BP_NC_F32_3D 2
#endif
template <int DIM, class P, bool VPHASE>
__host__ __device__ constexpr bool read_only_loads() {
    return kReadOnlyPath ||
           (P::prec == BP_PREC_FP32 && (((DIM == 2 ? BP_NC_F32_2D : BP_NC_F32_3D) >> (VPHASE ? 0 : 1)) & 1));
}

// ---------------------------------------------------------------------------
// Where a chunk's field values come from.  GlobalSrc loads them from the field
// arrays (NC: through the read-only path); AsyncSrc (async.cuh) from the
// warp's shared-memory slots, which asynchronous copies have filled.
// span: cells x0 - HW .. x0 + 3 + HW of the chunk's row; rows: the chunk's cells
// in rows -HW .. HW along y (AX 1) or z (AX 2); own: the chunk's cells.
template <int ORD, class P, bool NC, bool AHEAD = true>
struct GlobalSrc : SrcForm {
    static constexpr bool kAhead = AHEAD;
    using R = typename P::real;
    const ShotDesc& S;
    cidx c;
    int x0;
    __device__ __forceinline__ GlobalSrc(const ShotDesc& S_, cidx c_, int x0_) : S(S_), c(c_), x0(x0_) {}
    template <int F>
    __device__ __forceinline__ void span(R (&v)[4 + ORD]) const {
        load_span<ORD, P, NC>(S.f[F], S.flo[F], c - x0, x0, S.nx, v);
    }
    template <int F, int AX>
    __device__ __forceinline__ void rows(R (&a)[ORD + 1][4]) const {
        load_rows<ORD, P, NC>(S.f[F], S.flo[F], c, AX == 1 ? S.pitch : (cidx)S.plane, a);
    }
    template <int F>
    __device__ __forceinline__ void own(R (&v)[4]) const {
        P::ld4(S.f[F], S.flo[F], c, v);
    }
};

// Difference along x of field F at the chunk (FWD: at x + 1/2), divided by H as
// deriv_q's Q says; false if that does not hold for one of the four.
template <int ORD, class P, int F, bool FWD, int Q, class Src>
__device__ __forceinline__ bool d_span(const ShotDesc& S, const Src& src, typename P::real (&d)[4]) {
    typename P::real v[4 + ORD];
    src.template span<F>(v);
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const typename P::real q = FWD ? dfwd<ORD>(v, j) : dbwd<ORD>(v, j);
        if constexpr (Q) ok = deriv_q<P, Q>(q, S, d[j]) && ok;
        else d[j] = deriv_div<P>(q, S);
    }
    return ok;
}
// Difference across rows (AX 1: y, 2: z) of field F at the chunk, divided by
// the spacing.
template <int ORD, class P, int F, int AX, bool FWD, int Q, class Src>
__device__ __forceinline__ bool d_rows(const ShotDesc& S, const Src& src, int z, typename P::real (&d)[4]) {
    using R = typename P::real;
    R a[ORD + 1][4];
    src.template rows<F, AX>(a);
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        R t[ORD + 1];
#pragma unroll
        for (int k = 0; k <= ORD; k++) t[k] = a[k][j];
        const R q = FWD ? rfwd<ORD>(t) : rbwd<ORD>(t);
        if constexpr (Q) ok = deriv_q<P, Q>(q, S, d[j]) && ok;
        else if constexpr (AX == 2) d[j] = deriv_z<P, FWD>(q, S, z);
        else d[j] = deriv_div<P>(q, S);
    }
    return ok;
}
// Runs differences(Q) for a chunk: as the policy divides, or in two operations
// and, where these do not hold, again through quot_y.
template <class P, class Fn>
__device__ __forceinline__ void differences(const ShotDesc& S, const Fn& fn) {
    if constexpr (two_op_policy<P>()) {
        if (!S.h_two_ops || !fn(std::integral_constant<int, 1>{})) fn(std::integral_constant<int, 2>{});
    } else {
        fn(std::integral_constant<int, 0>{});
    }
}

// ---------------------------------------------------------------------------
// V phase for one 4-cell chunk: FD_V (Float/main.cu:103-191).
// NC: read-only-path loads of the coefficients; ids: the chunk's tuple indices
// (indexed medium)
template <int DIM, int ORD, class P, bool RS, bool NC, class Src>
__device__ __forceinline__ void v_chunk(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                        typename P::real r, unsigned mask, unsigned ids) {
    VState<typename P::real> V;
    V.mids = ids;
    // ---- derivatives of the old stresses (x1..s3, Float/main.cu:115-128) ----
    differences<P>(S, [&](auto q) {
        constexpr int Q = decltype(q)::value;
        bool ok = true;
        ok = d_span<ORD, P, BP_F_TXX, true, Q>(S, src, V.x1) && ok;
        ok = d_span<ORD, P, BP_F_P, true, Q>(S, src, V.s1) && ok;
        ok = d_span<ORD, P, BP_F_TXZ, false, Q>(S, src, V.z2) && ok;
        ok = d_rows<ORD, P, BP_F_TXZ, 2, false, Q>(S, src, z, V.x3) && ok;
        ok = d_rows<ORD, P, BP_F_TZZ, 2, true, Q>(S, src, z, V.z1) && ok;
        ok = d_rows<ORD, P, BP_F_P, 2, true, Q>(S, src, z, V.s3) && ok;
        if constexpr (DIM == 3) {
            ok = d_span<ORD, P, BP_F_TXY, false, Q>(S, src, V.y2) && ok;
            ok = d_rows<ORD, P, BP_F_TXY, 1, false, Q>(S, src, z, V.x2) && ok;
            ok = d_rows<ORD, P, BP_F_TYY, 1, true, Q>(S, src, z, V.y1) && ok;
            ok = d_rows<ORD, P, BP_F_TYZ, 2, false, Q>(S, src, z, V.y3) && ok;
            ok = d_rows<ORD, P, BP_F_TYZ, 1, false, Q>(S, src, z, V.z3) && ok;
            ok = d_rows<ORD, P, BP_F_P, 1, true, Q>(S, src, z, V.s2) && ok;
        }
        return ok;
    });
    v_tail<DIM, ORD, P, false, RS, NC>(S, c, x0, y, z, r, mask, V, TailOut::v_of(S), src);
}

// ---------------------------------------------------------------------------
// T phase for one 4-cell chunk: FD_T (Float/main.cu:232-294).
template <int DIM, int ORD, class P, bool RS, bool NC, class Src>
__device__ __forceinline__ void t_chunk(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                        typename P::real r, unsigned mask, unsigned ids) {
    TState<typename P::real> T;
    T.mids = ids;
    differences<P>(S, [&](auto q) {
        constexpr int Q = decltype(q)::value;
        bool ok = true;
        ok = d_span<ORD, P, BP_F_VUX, false, Q>(S, src, T.uxx) && ok;
        ok = d_span<ORD, P, BP_F_VWX, false, Q>(S, src, T.wx) && ok;
        ok = d_span<ORD, P, BP_F_VUZ, true, Q>(S, src, T.uzx) && ok;
        ok = d_rows<ORD, P, BP_F_VUZ, 2, false, Q>(S, src, z, T.uzz) && ok;
        ok = d_rows<ORD, P, BP_F_VWZ, 2, false, Q>(S, src, z, T.wz) && ok;
        ok = d_rows<ORD, P, BP_F_VUX, 2, true, Q>(S, src, z, T.uxz) && ok;
        if constexpr (DIM == 3) {
            ok = d_span<ORD, P, BP_F_VUY, true, Q>(S, src, T.uyx) && ok;
            ok = d_rows<ORD, P, BP_F_VUY, 1, false, Q>(S, src, z, T.uyy) && ok;
            ok = d_rows<ORD, P, BP_F_VWY, 1, false, Q>(S, src, z, T.wy) && ok;
            ok = d_rows<ORD, P, BP_F_VUX, 1, true, Q>(S, src, z, T.uxy) && ok;
            ok = d_rows<ORD, P, BP_F_VUY, 2, true, Q>(S, src, z, T.uyz) && ok;
            ok = d_rows<ORD, P, BP_F_VUZ, 1, true, Q>(S, src, z, T.uzy) && ok;
        }
        return ok;
    });
    t_tail<DIM, ORD, P, false, RS, NC>(S, c, x0, y, z, r, mask, T, TailOut::t_of(S), src);
}

// ---------------------------------------------------------------------------
// Chunks taken one output group at a time.  v_chunk/t_chunk form all the
// derivatives of a chunk before the CPML and the updates: twelve in 3D, so 48
// values (96 in FP64) are live at once and the capped kernels spill.  Here each
// velocity component (and each shear stress, then the normal stresses and
// the pressure) loads, differences, CPML-corrects and stores only what it
// needs.  Every element goes through the same operations in the same order
// as in v_tail/t_tail, so the results are bit-identical.
// Which phases take this form, per dimension and precision (bit 0 = V, bit 1
// = T).  Measured on B200 (3D: 192^3 and 552 x 552 x 424 order 2, 200^3
// order 4; 2D: 4040 x 2040 order 2): 3D COMP16 both (12-16 % off the step,
// its spills gone); 2D COMP16, here the interleaved kernel alone, the T phase (13 %
// off it, the V phase 2 % slower grouped); FP64 both in 3D: the T phase with 2 CTAs per SM 25-30 % off
// the 3D step, the V phase, which spills 516-860 bytes as a whole chunk (an axis'
// memory variables at once) and none grouped, us per step 140 x 130 x 120 345 ->
// 312, order 4 366 -> 334, 200 x 190 x 180 905 -> 825, 296 x 296 x 232 2760 -> 2536,
// order 4 3295 -> 3000; FP32 neither (10-20 % slower, its latency-bound phases
// losing the loads they had in flight).
#ifndef BP_GROUP3_C16
#define BP_GROUP3_C16 3
#endif
#ifndef BP_GROUP3_F32
#define BP_GROUP3_F32 0
#endif
#ifndef BP_GROUP3_F64
#define BP_GROUP3_F64 3
#endif
#ifndef BP_GROUP2_C16
#define BP_GROUP2_C16 2
#endif
#ifndef BP_GROUP2_F32
#define BP_GROUP2_F32 0
#endif
#ifndef BP_GROUP2_F64
#define BP_GROUP2_F64 0
#endif
template <int DIM, class P, bool VPHASE>
__host__ __device__ constexpr bool grouped() {
    const int m = DIM == 3 ? (P::prec == BP_PREC_COMP16 ? BP_GROUP3_C16 : P::prec == BP_PREC_FP32 ? BP_GROUP3_F32 : BP_GROUP3_F64)
                           : (P::prec == BP_PREC_COMP16 ? BP_GROUP2_C16 : P::prec == BP_PREC_FP32 ? BP_GROUP2_F32 : BP_GROUP2_F64);
    return (m >> (VPHASE ? 0 : 1)) & 1;
}

// Masked cells feed zero derivatives into the memory variables.
template <class R>
__device__ __forceinline__ void mask0(R (&d)[4], unsigned mask) {
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(mask >> j & 1u)) d[j] = 0;
}
// CPML of one derivative on the slab of `axis` (slot k, half-grid profile if
// half); nothing outside that slab.  Slabs hold 3 slots per phase in 2D, 4 in 3D.
template <int DIM, bool RS, class R, bool EX = false>
__device__ __forceinline__ void cpml_g(const ShotDesc& S, void* const (&psi)[3], int axis, int k, bool half,
                                       cidx si, int x0, int y, int z, R (&d)[4], R r) {
    if (si < 0) return;
    const void* pb = half ? S.pb2[axis] : S.pb[axis];
    const void* pe = half ? S.pe2[axis] : S.pe[axis];
    cpml_slot<DIM == 3 ? 4 : 3, RS, R, EX>(d, psi[axis], S.slab_cells[axis], k, si, axis == 0,
                                        axis == 0 ? x0 : (axis == 1 ? y : z), x0, pb, pe, r);
}

// One velocity component AX (0 = x, 1 = y, 2 = z) of the V phase
// (Float/main.cu:103-191 for that component).
template <int DIM, int ORD, class P, bool RS, int AX, class Src>
__device__ __forceinline__ void v_comp(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                       typename P::real r, unsigned mask, unsigned ids,
                                       const typename P::real (&rf)[4]) {
    using R = typename P::real;
    // dx, dy, dz: the stress derivatives summed into this component (dy in 3D
    // only); dp: the pressure derivative along AX.  Slots as in v_tail.
    R dx[4], dy[4], dz[4], dp[4];
    differences<P>(S, [&](auto q) {
        constexpr int Q = decltype(q)::value;
        bool ok = true;
        if constexpr (AX == 0) {
            ok = d_span<ORD, P, BP_F_TXX, true, Q>(S, src, dx) && ok;                          // x1
            if constexpr (DIM == 3) ok = d_rows<ORD, P, BP_F_TXY, 1, false, Q>(S, src, z, dy) && ok;   // x2
            ok = d_rows<ORD, P, BP_F_TXZ, 2, false, Q>(S, src, z, dz) && ok;                           // x3
            ok = d_span<ORD, P, BP_F_P, true, Q>(S, src, dp) && ok;                            // s1
        } else if constexpr (AX == 1) {
            ok = d_span<ORD, P, BP_F_TXY, false, Q>(S, src, dx) && ok;                         // y2
            ok = d_rows<ORD, P, BP_F_TYY, 1, true, Q>(S, src, z, dy) && ok;                            // y1
            ok = d_rows<ORD, P, BP_F_TYZ, 2, false, Q>(S, src, z, dz) && ok;                           // y3
            ok = d_rows<ORD, P, BP_F_P, 1, true, Q>(S, src, z, dp) && ok;                              // s2
        } else {
            ok = d_span<ORD, P, BP_F_TXZ, false, Q>(S, src, dx) && ok;                         // z2
            if constexpr (DIM == 3) ok = d_rows<ORD, P, BP_F_TYZ, 1, false, Q>(S, src, z, dy) && ok;   // z3
            ok = d_rows<ORD, P, BP_F_TZZ, 2, true, Q>(S, src, z, dz) && ok;                            // z1
            ok = d_rows<ORD, P, BP_F_P, 2, true, Q>(S, src, z, dp) && ok;                              // s3
        }
        return ok;
    });
    if constexpr (P::prec == BP_PREC_COMP16 && RS) {
        scale4(dx, r); scale4(dz, r); scale4(dp, r);
        if constexpr (DIM == 3) scale4(dy, r);
    }
    mask0(dx, mask); mask0(dz, mask); mask0(dp, mask);
    if constexpr (DIM == 3) mask0(dy, mask);
    void* const psi[3] = {S.psiV[0], S.psiV[1], S.psiV[2]};
    const cidx s0 = slab_index(S, 0, x0, y, z), s2 = slab_index(S, 2, x0, y, z);
    const cidx s1 = DIM == 3 ? slab_index(S, 1, x0, y, z) : -1;
    if constexpr (AX == 0) {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 0, true, s0, x0, y, z, dx, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 1, true, s0, x0, y, z, dp, r);
        if constexpr (DIM == 3) cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 0, false, s1, x0, y, z, dy, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 0, false, s2, x0, y, z, dz, r);
    } else if constexpr (AX == 1) {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 3, false, s0, x0, y, z, dx, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 1, true, s1, x0, y, z, dy, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 2, true, s1, x0, y, z, dp, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 3, false, s2, x0, y, z, dz, r);
    } else {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 2, false, s0, x0, y, z, dx, r);
        if constexpr (DIM == 3) cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 3, false, s1, x0, y, z, dy, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 1, true, s2, x0, y, z, dz, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 2, true, s2, x0, y, z, dp, r);
    }
    // the divergence in v_tail's summation order: x1 (+x2) +x3, y1+y2+y3, z1+z2 (+z3)
    R sum[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (DIM == 2) sum[j] = AX == 0 ? dx[j] + dz[j] : dz[j] + dx[j];
        else if constexpr (AX == 0) sum[j] = dx[j] + dy[j] + dz[j];
        else if constexpr (AX == 1) sum[j] = dy[j] + dx[j] + dz[j];
        else sum[j] = dz[j] + dx[j] + dy[j];
    }
    constexpr int fu = AX == 0 ? BP_F_VUX : AX == 1 ? BP_F_VUY : BP_F_VUZ;
    constexpr int fw = AX == 0 ? BP_F_VWX : AX == 1 ? BP_F_VWY : BP_F_VWZ;
    constexpr int crho = AX == 0 ? VC_RHO_X : AX == 1 ? VC_RHO_Y : VC_RHO_Z;
    constexpr int cc1 = AX == 0 ? VC_CC1_X : AX == 1 ? VC_CC1_Y : VC_CC1_Z;
    constexpr int cc2 = AX == 0 ? VC_CC2_X : AX == 1 ? VC_CC2_Y : VC_CC2_Z;
    R rho[4], c1[4], c2[4], vu[4], vw[4], nu[4], nw[4];
    vcoef4<P>(S, crho, c, ids, rho);
    vcoef4<P>(S, cc1, c, ids, c1);
    vcoef4<P>(S, cc2, c, ids, c2);
    src.template own<fu>(vu);
    src.template own<fw>(vw);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (P::prec == BP_PREC_COMP16) {
            const R wo = RS ? mulr(vw[j], r) : vw[j], uo = RS ? mulr(vu[j], r) : vu[j];
            R rr = rf[j] * rho[j];
            const R wn = fma_rn(-c2[j], dp[j], fma_rn(c1[j], wo, -mul_rn(rr * c2[j], sum[j])));   // as v_tail
            nw[j] = wn;
            nu[j] = uo + rho[j] * sum[j] - rr * (wn - wo);
        } else {
            R wo = vw[j];
            const R num = wo * c2[j] - S.dtr<R>() * (rf[j] * rho[j] * sum[j] + dp[j]);
            const R wn = (c1[j] == (R)0) ? (R)0 : quot<P, DIM>(num, c1[j]);
            nw[j] = wn;
            nu[j] = vu[j] + S.dtr<R>() * rho[j] * sum[j] - rf[j] * rho[j] * (wn - wo);
        }
        if (!(mask >> j & 1u)) { nw[j] = vw[j]; nu[j] = vu[j]; }
    }
    P::st4(S.f[fw], S.flo[fw], c, nw);
    P::st4(S.f[fu], S.flo[fu], c, nu);
}

template <int DIM, int ORD, class P, bool RS, class Src>
__device__ __forceinline__ void v_chunk_g(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                          typename P::real r, unsigned mask, unsigned ids) {
    typename P::real rf[4];
    vcoef4<P>(S, VC_RHOF, c, ids, rf);
    v_comp<DIM, ORD, P, RS, 0>(S, src, c, x0, y, z, r, mask, ids, rf);
    if constexpr (DIM == 3) v_comp<DIM, ORD, P, RS, 1>(S, src, c, x0, y, z, r, mask, ids, rf);
    v_comp<DIM, ORD, P, RS, 2>(S, src, c, x0, y, z, r, mask, ids, rf);
}

// Old value of a stress field at the chunk, with this step's rescale.
template <int F, class P, bool RS, class Src>
__device__ __forceinline__ void ld_old(const Src& src, typename P::real r, typename P::real (&o)[4]) {
    src.template own<F>(o);
    if constexpr (P::prec == BP_PREC_COMP16 && RS) scale4(o, r);
}
template <class P>
__device__ __forceinline__ void st_new(const ShotDesc& S, int f, cidx c, unsigned mask,
                                       typename P::real (&nv)[4], const typename P::real (&ov)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(mask >> j & 1u)) nv[j] = ov[j];
    P::st4(S.f[f], S.flo[f], c, nv);
}

// One shear stress of the T phase: SH 0 = txy, 1 = tyz (3D only), 2 = txz
// (Float/main.cu:232-294 for that stress).
template <int DIM, int ORD, class P, bool RS, int SH, class Src>
__device__ __forceinline__ void t_shear(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                        typename P::real r, unsigned mask, unsigned ids, void* const (&psi)[3]) {
    using R = typename P::real;
    R a[4], b[4];    // the two derivatives, in the order of the update's sum
    differences<P>(S, [&](auto q) {
        constexpr int Q = decltype(q)::value;
        bool ok = true;
        if constexpr (SH == 0) {
            ok = d_rows<ORD, P, BP_F_VUX, 1, true, Q>(S, src, z, a) && ok;        // uxy
            ok = d_span<ORD, P, BP_F_VUY, true, Q>(S, src, b) && ok;      // uyx
        } else if constexpr (SH == 1) {
            ok = d_rows<ORD, P, BP_F_VUY, 2, true, Q>(S, src, z, a) && ok;        // uyz
            ok = d_rows<ORD, P, BP_F_VUZ, 1, true, Q>(S, src, z, b) && ok;        // uzy
        } else {
            ok = d_rows<ORD, P, BP_F_VUX, 2, true, Q>(S, src, z, a) && ok;        // uxz
            ok = d_span<ORD, P, BP_F_VUZ, true, Q>(S, src, b) && ok;      // uzx
        }
        return ok;
    });
    mask0(a, mask); mask0(b, mask);
    if constexpr (SH == 0) {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 3, true, slab_index(S, 0, x0, y, z), x0, y, z, b, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 2, true, slab_index(S, 1, x0, y, z), x0, y, z, a, r);
    } else if constexpr (SH == 1) {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 3, true, slab_index(S, 1, x0, y, z), x0, y, z, b, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 3, true, slab_index(S, 2, x0, y, z), x0, y, z, a, r);
    } else {
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 2, true, slab_index(S, 0, x0, y, z), x0, y, z, b, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 2, true, slab_index(S, 2, x0, y, z), x0, y, z, a, r);
    }
    constexpr int f = SH == 0 ? BP_F_TXY : SH == 1 ? BP_F_TYZ : BP_F_TXZ;
    constexpr int cm = SH == 0 ? TC_MUXY : SH == 1 ? TC_MUYZ : TC_MUXZ;
    R mu[4], o[4], n[4];
    tcoef4<P>(S, cm, c, ids, mu);
    ld_old<f, P, RS>(src, r, o);
    const R dt = S.dtr<R>();
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (P::prec == BP_PREC_COMP16) n[j] = o[j] + mu[j] * (a[j] + b[j]);
        else n[j] = o[j] + mu[j] * dt * (a[j] + b[j]);
    }
    st_new<P>(S, f, c, mask, n, o);
}

template <int DIM, int ORD, class P, bool RS, class Src>
__device__ __forceinline__ void t_chunk_g(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                          typename P::real r, unsigned mask, unsigned ids) {
    using R = typename P::real;
    void* const psi[3] = {S.psiT[0], S.psiT[1], S.psiT[2]};
    if constexpr (DIM == 3) {
        t_shear<DIM, ORD, P, RS, 0>(S, src, c, x0, y, z, r, mask, ids, psi);
        t_shear<DIM, ORD, P, RS, 1>(S, src, c, x0, y, z, r, mask, ids, psi);
    }
    t_shear<DIM, ORD, P, RS, 2>(S, src, c, x0, y, z, r, mask, ids, psi);

    // normal stresses and pressure: the divergence derivatives (uyy, wy in 3D)
    R uxx[4], uyy[4], uzz[4], wx[4], wy[4], wz[4];
    differences<P>(S, [&](auto q) {
        constexpr int Q = decltype(q)::value;
        bool ok = true;
        ok = d_span<ORD, P, BP_F_VUX, false, Q>(S, src, uxx) && ok;
        ok = d_span<ORD, P, BP_F_VWX, false, Q>(S, src, wx) && ok;
        if constexpr (DIM == 3) {
            ok = d_rows<ORD, P, BP_F_VUY, 1, false, Q>(S, src, z, uyy) && ok;
            ok = d_rows<ORD, P, BP_F_VWY, 1, false, Q>(S, src, z, wy) && ok;
        }
        ok = d_rows<ORD, P, BP_F_VUZ, 2, false, Q>(S, src, z, uzz) && ok;
        ok = d_rows<ORD, P, BP_F_VWZ, 2, false, Q>(S, src, z, wz) && ok;
        return ok;
    });
    mask0(uxx, mask); mask0(wx, mask); mask0(uzz, mask); mask0(wz, mask);
    if constexpr (DIM == 3) { mask0(uyy, mask); mask0(wy, mask); }
    {
        const cidx s0 = slab_index(S, 0, x0, y, z);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 0, false, s0, x0, y, z, uxx, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 0, 1, false, s0, x0, y, z, wx, r);
        if constexpr (DIM == 3) {
            const cidx s1 = slab_index(S, 1, x0, y, z);
            cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 0, false, s1, x0, y, z, uyy, r);
            cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 1, 1, false, s1, x0, y, z, wy, r);
        }
        const cidx s2 = slab_index(S, 2, x0, y, z);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 0, false, s2, x0, y, z, uzz, r);
        cpml_g<DIM, RS, typename P::real, P::exact>(S, psi, 2, 1, false, s2, x0, y, z, wz, r);
    }
    R cC[4], cM[4], cH[4], cH2[4], o[4], n[4];
    const R dt = S.dtr<R>();
    tcoef4<P>(S, TC_C, c, ids, cC);
    tcoef4<P>(S, TC_M, c, ids, cM);
    ld_old<BP_F_P, P, RS>(src, r, o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (DIM == 3) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = o[j] - cC[j] * (uxx[j] + uyy[j] + uzz[j]) - cM[j] * (wx[j] + wy[j] + wz[j]);
            else
                n[j] = o[j] - dt * (cC[j] * (uxx[j] + uyy[j] + uzz[j]) + cM[j] * (wx[j] + wy[j] + wz[j]));
        } else {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = o[j] - cC[j] * (uxx[j] + uzz[j]) - cM[j] * (wx[j] + wz[j]);
            else
                n[j] = o[j] - dt * (cC[j] * (uxx[j] + uzz[j]) + cM[j] * (wx[j] + wz[j]));
        }
    }
    st_new<P>(S, BP_F_P, c, mask, n, o);
    tcoef4<P>(S, TC_H, c, ids, cH);
    tcoef4<P>(S, TC_H2U, c, ids, cH2);
    ld_old<BP_F_TXX, P, RS>(src, r, o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (DIM == 3) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(o[j], cH2[j], (uyy[j] + uzz[j]), cH[j], uxx[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = o[j] + dt * (cH2[j] * (uyy[j] + uzz[j]) + cH[j] * uxx[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        } else {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(o[j], cH2[j], uzz[j], cH[j], uxx[j], cC[j], (wx[j] + wz[j]));
            else
                n[j] = o[j] + dt * (cH2[j] * uzz[j] + cH[j] * uxx[j] + cC[j] * (wx[j] + wz[j]));
        }
    }
    st_new<P>(S, BP_F_TXX, c, mask, n, o);
    if constexpr (DIM == 3) {
        ld_old<BP_F_TYY, P, RS>(src, r, o);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(o[j], cH2[j], (uxx[j] + uzz[j]), cH[j], uyy[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = o[j] + dt * (cH2[j] * (uxx[j] + uzz[j]) + cH[j] * uyy[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        }
        st_new<P>(S, BP_F_TYY, c, mask, n, o);
    }
    ld_old<BP_F_TZZ, P, RS>(src, r, o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (DIM == 3) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(o[j], cH2[j], (uxx[j] + uyy[j]), cH[j], uzz[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = o[j] + dt * (cH2[j] * (uxx[j] + uyy[j]) + cH[j] * uzz[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        } else {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(o[j], cH2[j], uxx[j], cH[j], uzz[j], cC[j], (wx[j] + wz[j]));
            else
                n[j] = o[j] + dt * (cH2[j] * uxx[j] + cH[j] * uzz[j] + cC[j] * (wx[j] + wz[j]));
        }
    }
    st_new<P>(S, BP_F_TZZ, c, mask, n, o);
}

// ---------------------------------------------------------------------------
// The cells of the chunk at x0 the phases update, as a 4-bit mask (0: none).
template <int ORD>
__device__ __forceinline__ unsigned chunk_mask(const ShotDesc& S, int x0) {
    const int hw = ORD / 2;
    unsigned mask = 0;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (x0 + j >= hw && x0 + j < S.nx - hw) mask |= 1u << j;
    return mask;
}
// Whether the phases update row (y, z).
template <int DIM, int ORD>
__device__ __forceinline__ bool row_updated(const ShotDesc& S, int y, int z) {
    const int hw = ORD / 2;
    return z >= hw && z < S.nz - hw && (DIM == 2 || (y >= hw && y < S.ny - hw));
}

// One chunk of one phase: cells x0 .. x0 + 3 of row (y, z), mask of them updated
// (it: the step index, r: the COMP16 rescale factor of that step).  post (T
// phase only): the chunk also records the receivers in its cells and, if it
// holds the source cell, injects the next source sample, in place of the
// post-step kernel k_post.
template <int DIM, int ORD, class P, bool VPHASE, bool NC, bool GROUPED, class Src>
__device__ __forceinline__ void chunk_work(const ShotDesc& S, const Src& src, cidx c, int x0, int y, int z,
                                           typename P::real r, unsigned mask, unsigned ids, int it, int post) {
    using R = typename P::real;
    constexpr bool C16 = P::prec == BP_PREC_COMP16;
    // COMP16: the rescale products only on the steps whose factor is not
    // exactly 1 (a uniform branch; the products are never fused, so both
    // forms give the same bits when r == 1)
    if (C16 && (r != (R)1 || !BP_RS_SPLIT)) {
        if constexpr (GROUPED) {
            if constexpr (VPHASE) v_chunk_g<DIM, ORD, P, C16>(S, src, c, x0, y, z, r, mask, ids);
            else t_chunk_g<DIM, ORD, P, C16>(S, src, c, x0, y, z, r, mask, ids);
        } else {
            if constexpr (VPHASE) v_chunk<DIM, ORD, P, C16, NC>(S, src, c, x0, y, z, r, mask, ids);
            else t_chunk<DIM, ORD, P, C16, NC>(S, src, c, x0, y, z, r, mask, ids);
        }
    } else {
        if constexpr (GROUPED) {
            if constexpr (VPHASE) v_chunk_g<DIM, ORD, P, false>(S, src, c, x0, y, z, r, mask, ids);
            else t_chunk_g<DIM, ORD, P, false>(S, src, c, x0, y, z, r, mask, ids);
        } else {
            if constexpr (VPHASE) v_chunk<DIM, ORD, P, false, NC>(S, src, c, x0, y, z, r, mask, ids);
            else t_chunk<DIM, ORD, P, false, NC>(S, src, c, x0, y, z, r, mask, ids);
        }
    }
    if constexpr (!VPHASE)
        if (post) post_chunk<DIM, P>(S, it, c, x0, y, z);
}
// The same from the field arrays.  NCOK = false: no read-only-path loads (the
// interleaved step kernel reads arrays that the same launch writes).
template <int DIM, int ORD, class P, bool VPHASE, bool NCOK>
__device__ __forceinline__ void chunk_unit(const ShotDesc& S, int x0, int y, int z, typename P::real r, int it,
                                           int post) {
    if (!row_updated<DIM, ORD>(S, y, z)) return;
    const unsigned mask = chunk_mask<ORD>(S, x0);
    if (!mask) return;
    // the interleaved kernel's FP64 V phase, at one CTA per SM, takes whole chunks
    // (200 x 190 x 180 1649 us per step, 1829 grouped; order 4 1698 and 1855)
    constexpr bool GROUPED = grouped<DIM, P, VPHASE>() && (NCOK || !VPHASE || P::prec != BP_PREC_FP64);
    constexpr bool NC = read_only_loads<DIM, P, VPHASE>() && NCOK && !GROUPED;
    const cidx c = x0 + y * S.pitch + z * (cidx)S.plane;
    // an indexed medium's tuple indices first: their load overlaps the field loads
    unsigned ids = 0;
    if (med_on<P>(S)) ids = med_ids(S, c);
    // The interleaved kernel holds both phases in one function and spills in 2D
    // with the coefficients loaded ahead (FP32, us per step ahead -> not: 4040 x
    // 2040 layered 229 -> 206, per-cell 257 -> 243, 817 x 1073 32.8 -> 31.7; the
    // reference's rounding 232 -> 224, but 253 -> 261 per-cell, 41 -> 44: ahead).
    constexpr bool AHEAD = NCOK || DIM == 3 || P::exact;
    const GlobalSrc<ORD, P, NC, AHEAD> src(S, c, x0);
    chunk_work<DIM, ORD, P, VPHASE, NC, GROUPED>(S, src, c, x0, y, z, r, mask, ids, it, post);
}

// The (row, segment) units of tile (rb, sb) of shot S in one phase: the
// rectangular tiling of the interleaved step kernel, whose bands are whole row
// blocks.  Warp w takes units w, w + 8, ...; consecutive warps take
// consecutive rows.
template <int DIM, int ORD, class P, bool VPHASE, bool MU, bool NCOK>
__device__ __forceinline__ void tile_units(const ShotDesc& S, int rb, int sb, int warp, int lane, typename P::real r,
                                           int it, int post) {
    const int lr = S.tile_lr, units = 1 << (lr + S.tile_ls);
    auto unit = [&](int u) {
        const int ri = u & ((1 << lr) - 1);
        const int seg = (sb << S.tile_ls) + (u >> lr);
        if (seg >= S.nseg) return;
        int y, z;
        if constexpr (DIM == 3) {
            const int ltz = S.tile_ltz, lty = lr - ltz;
            const int nyb = (S.ny + (1 << lty) - 1) >> lty;
            const int zb = rb / nyb, yb = rb - zb * nyb;
            y = (yb << lty) + (ri & ((1 << lty) - 1));
            z = (zb << ltz) + (ri >> lty);
            if (y >= S.ny) return;
        } else {
            y = 0;
            z = (rb << lr) + ri;
        }
        chunk_unit<DIM, ORD, P, VPHASE, NCOK>(S, seg * kSegCells + lane * 4, y, z, r, it, post);
    };
    // MU: tiles of more units than warps (16-row or 8 x 2 tiles); the
    // one-unit form keeps no loop state live across the chunk code, which
    // spills more of the 2D FP32 V phase's 80 registers
    if constexpr (MU) {
        for (int u = warp; u < units; u += kWarps) unit(u);
    } else {
        if (warp < units) unit(warp);
    }
}

// n / d for 0 <= n < 2^31 by a product with the divisor's reciprocal
// (magic_of): exact for every such n.
__device__ __forceinline__ int div_magic(int n, unsigned m, int s) {
    return (int)(((unsigned long long)(unsigned)n * m) >> s);
}

// Cell of chunk q of the flat tiling (row ri of its row block), false past the
// shot's chunks.  The chunks of the row blocks follow each other, cpr of them a
// row (row_chunks, step.cu), and a warp takes 32 consecutive ones: its lanes are
// full where a row is no multiple of 128 cells.  Measured on B200 against rows
// cut into 128-cell segments, whose last segment is 8-86 % empty (FP32, us per
// step, segments -> flat): 200^3 order 2 544 -> 465, order 4 591 -> 515; 424 x
// 424 x 328 per-cell medium 4408 -> 3390; 817 x 1073 23.7 -> 20.6; 192^3
// reference rounding 746 -> 626; FP64 1040 x 540 56.5 -> 41.7; 4040 x 2040
// (1 % empty) unchanged.  The kernels wait on loads, so a warp's work counts
// whether its lanes are full or not.
template <int DIM>
__device__ __forceinline__ bool flat_cell(const ShotDesc& S, int q, int ri, int& x0, int& y, int& z) {
    if (q >= S.nchunk_f) return false;
    const int blk = div_magic(q, S.cpr_m, S.cpr_s);
    x0 = (q - blk * S.cpr) * 4;
    if constexpr (DIM == 3) {
        const int ltz = S.tile_ltz, lty = S.tile_lr - ltz;
        const int zb = div_magic(blk, S.nyb_m, S.nyb_s);
        y = ((blk - zb * S.nyb) << lty) + (ri & ((1 << lty) - 1));
        z = (zb << ltz) + (ri >> lty);
        return y < S.ny && z < S.nz;
    } else {
        y = 0;
        z = (blk << S.tile_lr) + ri;
        return z < S.nz;
    }
}

// The units of tile lt of shot S in the flat tiling.
template <int DIM, int ORD, class P, bool VPHASE, bool MU, bool NCOK>
__device__ __forceinline__ void flat_units(const ShotDesc& S, int lt, int warp, int lane, typename P::real r, int it,
                                           int post) {
    const int lr = S.tile_lr, units = 1 << (lr + S.tile_ls);
    auto unit = [&](int u) {
        const int ri = u & ((1 << lr) - 1);
        const int q = (((lt << S.tile_ls) + (u >> lr)) << 5) + lane;
        int x0, y, z;
        if (!flat_cell<DIM>(S, q, ri, x0, y, z)) return;
        chunk_unit<DIM, ORD, P, VPHASE, NCOK>(S, x0, y, z, r, it, post);
    };
    if constexpr (MU) {
        for (int u = warp; u < units; u += kWarps) unit(u);
    } else {
        if (warp < units) unit(warp);
    }
}

// L2 prefetch of this warp's unit of tile lt: the FP32 fields, a 128-byte line
// of one array per lane (no registers held, nothing waited for).
template <int DIM>
__device__ __forceinline__ void flat_prefetch(const ShotDesc& S, int lt, int warp, int lane) {
    const int lr = S.tile_lr;
    const int q = (((lt << S.tile_ls) + (warp >> lr)) << 5) + (lane & 3) * 8;
    int x0, y, z;
    if (!flat_cell<DIM>(S, q, warp & ((1 << lr) - 1), x0, y, z)) return;
    const cidx c = x0 + y * S.pitch + z * (cidx)S.plane;
#pragma unroll
    for (int f = 0; f < BP_NFIELDS; f += 8) {
        const int a = f + (lane >> 2);
        if (a < BP_NFIELDS && S.f[a])
            asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const float*>(S.f[a]) + c));
    }
}

}  // namespace bpk
