// stencil.cuh - per-chunk stencil arithmetic shared by the phase kernels:
// staggered differences, the division by H, span/row loads, the CPML memory
// update, and the tails of FD_V / FD_T (rescale, mask, CPML, update, store)
// that both the tile kernels (step.cu) and the marching kernels
// (step_march.cu) call, so both produce bit-identical results.
#pragma once
#include "common.cuh"

namespace bpk {

// Correctly rounded quotients without the divide routine's slow path.
//
// The compiler's IEEE division leaves its inline sequence for operands far from
// 1, and a wavefield is full of them: ahead of the wavefront the scheme's own
// domain of influence advances a cell per step, and its values fall off to
// subnormal numbers, which then fill the grid out to the borders.  Here a tiny
// dividend is scaled up by a power of two (exactly) and the quotient back down,
// and the quotient is formed from the divisor's reciprocal y by two residual
// corrections q += y (a - q b) with exact fused residuals (Markstein, IBM J.
// Res. Dev. 34(1), 1990), which round correctly where nothing under- or
// overflows.  A subnormal result must not be rounded twice, so q is first
// rounded to odd (Boldo and Melquiond, IEEE Trans. Comput. 57(4), 2008): 24 bits
// to odd, then to at most 22 to nearest, is one rounding to nearest (FP64: 53
// and 51).  The binade below the smallest normal (one bit more) and quotients
// out of range (infinite, NaN) take the division itself.  Equal to a / b bit for bit
// (tests/test_gpu_quotient.py).
template <class R> struct QuotRange;
template <> struct QuotRange<float> {
    static constexpr float small = 0x1p-30f, up = 0x1p64f, down = 0x1p-64f, lo = 0x1p-61f, sub = 0x1p-63f, hi = 0x1p120f;
};
template <> struct QuotRange<double> {
    static constexpr double small = 0x1p-300, up = 0x1p600, down = 0x1p-600, lo = 0x1p-420, sub = 0x1p-423, hi = 0x1p1000;
};
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ int bits_of(float a) { return __float_as_int(a); }
__device__ __forceinline__ long long bits_of(double a) { return __double_as_longlong(a); }
__device__ __forceinline__ float of_bits(int a) { return __int_as_float(a); }
__device__ __forceinline__ double of_bits(long long a) { return __longlong_as_double(a); }

// a / b for y = 1 / b to within an ulp
template <class R>
__device__ __forceinline__ R quot_y(R a, R b, R y) {
    using Q = QuotRange<R>;
    const bool tiny = fabs(a) < Q::small;
    const R t = mul_rn(a, tiny ? Q::up : (R)1);
    R q = mul_rn(t, y);
    q = fma_rn(fma_rn(-q, b, t), y, q);
    q = fma_rn(fma_rn(-q, b, t), y, q);
    if (fabs(q) >= Q::lo && fabs(q) < Q::hi) return mul_rn(q, tiny ? Q::down : (R)1);
    if (a == (R)0) return mul_rn(a, b);            // the zero with the quotient's sign
    if (tiny && fabs(q) < Q::sub) {
        const R r = fma_rn(-q, b, t);              // a up - q b, exact
        auto w = bits_of(q);
        if (r != (R)0) w = (w + ((bits_of(r) ^ bits_of(b) ^ w) >> (8 * sizeof(R) - 1))) | 1;
        return mul_rn(of_bits(w), Q::down);
    }
    return a / b;
}
// the reciprocal of b to within an ulp (0, infinite or NaN where b is out of range)
__device__ __forceinline__ float recip(float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return fma_rn(fma_rn(-b, y, 1.0f), y, y);
}

// num / c1 of the friction update.  FP32 through quot_y: 296 x 296 x 232 1194 ->
// 1078 us per step, 4040 x 2040 165.9 -> 162.1 (B200, order 2).  CBF16 in 2D too,
// after a test for zero, which is what the quiet grid ahead of the domain of
// influence divides: the 4040 x 2040 layered run of 8000 steps, 180.3 us per
// step with the division (158 early, 192 late), 169.1 without the test (164,
// 175), 165.1 with it (156, 175); order 4 201.7, 190.5 and 186.0; 817 x 1073 at
// step 1500 24.0, 22.3 and 22.0.  In 3D CBF16 keeps the division: 200 x 190 x 180
// 367 against 376 at step 600, 296 x 296 x 232 965 against 975 early, though 1208
// against 1092 late.  So does FP64.
// TEST0: FP32 tests for zero as well (SrcForm).
template <class P, int DIM, bool TEST0 = false>
__device__ __forceinline__ typename P::real quot(typename P::real a, typename P::real b) {
    if constexpr (P::store == BP_PREC_FP32 && !TEST0) return quot_y<float>(a, b, recip(b));
    else if constexpr (P::store == BP_PREC_FP32 || (P::store == BP_PREC_CBF16 && DIM == 2))
        return a == 0.0f ? a * b : quot_y<float>(a, b, recip(b));
    else return a == (typename P::real)0 ? a * b : a / b;
}

// Differences divided by H with IEEE rounding: FP64 and the reference's rounding
// (PolF32R).  H is one number, so 1/H is held as the unevaluated sum inv + lo
// and a / H = fma(a, inv, a lo), two operations, correctly rounded for every a
// where that holds for the H at hand (Brisebarre, Muller and Raina, IEEE Trans.
// Comput. 53(8), 2004; const_divisor in divisor.h decides it exactly).  That
// leaves out tiny and huge differences (and -0), the rim of the scheme's domain
// of influence ahead of the wavefront: a chunk is differenced in two operations first,
// and again through quot_y if any of its differences was one of those.  Measured
// on B200 (us per step, once the field has spread / in the first 130 steps):
// 192^3 reference rounding, order 2, 630 / 745 -> 404 / 585; 200 x 190 x 180 order
// 4 698 / 914 -> 442 / 739; FP64 4040 x 2040 533 / 510 -> 408 / 376, 168^3 809 ->
// 675.  One out-of-line call for the rim of each difference instead spilled
// around the calls (FP64 168^3 1106, order 4 932).
template <class P>
__host__ __device__ constexpr bool two_op_policy() { return P::prec == BP_PREC_FP64 || P::exact; }
// Q 0: the policy's own division; 1: two operations (false: not for this
// difference); 2: quot_y
template <class P, int Q>
__device__ __forceinline__ bool deriv_q(typename P::real a, const ShotDesc& S, typename P::real& q) {
    using R = typename P::real;
    R h, inv, lo, least, most;
    if constexpr (sizeof(R) == 8) { h = S.hd; inv = S.inv_hd; lo = S.inv_hd_lo; least = (R)0x1p-860; most = (R)0x1p900; }
    else { h = S.h; inv = S.inv_h; lo = S.inv_h_lo; least = (R)0x1p-80f; most = (R)0x1p100f; }
    if constexpr (Q == 2) {
        q = quot_y<R>(a, h, inv);
        return true;
    } else {
        q = fma_rn(a, inv, mul_rn(a, lo));        // +0 for +0 too
        bool zero;
        if constexpr (sizeof(R) == 8) zero = __double_as_longlong(a) == 0;
        else zero = __float_as_int(a) == 0;
        return (fabs(a) >= least && fabs(a) < most) || zero;
    }
}

template <class P>
__device__ __forceinline__ typename P::real deriv_div(typename P::real a, const ShotDesc& S) {
    // FP32: the reference divides by H.  q = a * (1/H) refined by one residual
    // step, q += (a - q H) * (1/H), with the exact fused residual a - q H,
    // matches the IEEE quotient a / H to within one ulp (equal in all but rare
    // near-tie cases) in 3 instructions instead of a full divide.
    // COMP16 (own arithmetic) multiplies by 1/H; FP64 and the reference's
    // rounding go through deriv_q.
    static_assert(!two_op_policy<P>(), "correctly rounded differences take deriv_q");
    if constexpr (P::prec == BP_PREC_FP32) {
        const float q = a * S.inv_h;
        return __fmaf_rn(__fmaf_rn(-q, S.h, a), S.inv_h, q);
    } else return a * S.inv_h;
}

// A difference along z divided by the row spacing: H on a uniform grid
// (deriv_div), the row's factor on a variable one (PolF32G; FWD: the forward
// difference of rows z, z+1, else the backward one of rows z-1, z).
template <class P, bool FWD>
__device__ __forceinline__ typename P::real deriv_z(typename P::real a, const ShotDesc& S, int z) {
    if constexpr (P::graded) return __fmul_rn(a, S.zf[FWD ? z : S.nz + z]);   // never contracted into a later add
    else return deriv_div<P>(a, S);
}

// Staggered difference from a span v[j] = f(x0 - HW + j).
template <int ORD, class R>
__device__ __forceinline__ R dfwd(const R* v, int j) {   // at x0+j+1/2
    constexpr int HW = ORD / 2;
    if constexpr (ORD == 2) return v[HW + j + 1] - v[HW + j];
    else return (R)1.125 * (v[HW + j + 1] - v[HW + j]) + (R)(-1.0 / 24.0) * (v[HW + j + 2] - v[HW + j - 1]);
}
template <int ORD, class R>
__device__ __forceinline__ R dbwd(const R* v, int j) {   // at x0+j-1/2
    constexpr int HW = ORD / 2;
    if constexpr (ORD == 2) return v[HW + j] - v[HW + j - 1];
    else return (R)1.125 * (v[HW + j] - v[HW + j - 1]) + (R)(-1.0 / 24.0) * (v[HW + j + 1] - v[HW + j - 2]);
}
// Difference across rows: a[k] = f(row + k - HW) for one cell.
template <int ORD, class R>
__device__ __forceinline__ R rfwd(const R* a) {
    constexpr int HW = ORD / 2;
    if constexpr (ORD == 2) return a[HW + 1] - a[HW];
    else return (R)1.125 * (a[HW + 1] - a[HW]) + (R)(-1.0 / 24.0) * (a[HW + 2] - a[HW - 1]);
}
template <int ORD, class R>
__device__ __forceinline__ R rbwd(const R* a) {
    constexpr int HW = ORD / 2;
    if constexpr (ORD == 2) return a[HW] - a[HW - 1];
    else return (R)1.125 * (a[HW] - a[HW - 1]) + (R)(-1.0 / 24.0) * (a[HW + 1] - a[HW - 2]);
}

// Load f(x0 - HW .. x0 + 3 + HW) of one row; x neighbours clamped into the row
// (clamped values only feed cells that are never updated).
template <int ORD, class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void load_span(const void* p, const int8_t* lo, cidx rowbase, int x0, int nx,
                                          typename P::real (&v)[4 + ORD]) {
    constexpr int HW = ORD / 2;
    typename P::real c[4];
    P::template ld4<NC>(p, lo, rowbase + x0, c);
#pragma unroll
    for (int j = 0; j < 4; j++) v[HW + j] = c[j];
#pragma unroll
    for (int k = 1; k <= HW; k++) {
        int xl = x0 - k; xl = xl < 0 ? 0 : xl;
        int xr = x0 + 3 + k; xr = xr > nx - 1 ? nx - 1 : xr;
        v[HW - k] = P::template ld1<NC>(p, lo, rowbase + xl);
        v[HW + 3 + k] = P::template ld1<NC>(p, lo, rowbase + xr);
    }
}

// Load the 4 cells of rows row-HW .. row+HW (offsets along y or z).
template <int ORD, class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void load_rows(const void* p, const int8_t* lo, cidx c, cidx stride,
                                          typename P::real (&a)[ORD + 1][4]) {
    constexpr int HW = ORD / 2;
#pragma unroll
    for (int k = 0; k <= ORD; k++) P::template ld4<NC>(p, lo, c + (k - HW) * stride, a[k]);
}

// Product by the COMP16 rescale factor, never fused into a neighbouring add:
// the kernels skip it when the factor is exactly 1 (all steps but one in a
// hundred), and x * 1 == x only holds if no FMA ever absorbs the product.
template <class R>
__device__ __forceinline__ R mulr(R x, R r) {
    if constexpr (sizeof(R) == 4) return __fmul_rn(x, r);
    else return __dmul_rn(x, r);
}
template <class R>
__device__ __forceinline__ void scale4(R (&v)[4], R r) {
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = mulr(v[j], r);
}

// New ψ of one cell: ψ e + b (e prev + ∂).  EX (FP32 only): e prev + ∂ fused,
// then added times b to the float product ψ e with one rounding, as the
// reference's double-promoted expression rounds it (Float/main.cu:130-158).
template <bool EX, class R>
__device__ __forceinline__ R cpml_psi(R ps, R pv, R d, R bb, R ee) {
    if constexpr (EX) return __fmaf_rn(bb, __fmaf_rn(ee, pv, d), __fmul_rn(ps, ee));
    else return ps * ee + bb * (ee * pv + d);
}

// CPML memory update of one derivative slot for a 4-cell chunk
// (Float/main.cu:130-158):  ψ = ψ e + b (e prev + ∂),  prev = ∂,  ∂ += ψ,
// with b = -DT d / 2 precomputed.  The x axis has per-cell tables; the y and z
// axes one value per chunk.  Old ψ/prev are multiplied by the state rescale r.
template <bool RS, class R, bool EX = false>
__device__ __forceinline__ void cpml_x(R (&d)[4], R* psi, R* prev, const R* b, const R* e, int x0, R r) {
    R ps[4], pv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        ps[j] = RS ? mulr(psi[j], r) : psi[j];
        pv[j] = RS ? mulr(prev[j], r) : prev[j];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        R ee = e[x0 + j], bb = b[x0 + j];
        R np = cpml_psi<EX>(ps[j], pv[j], d[j], bb, ee);
        ps[j] = np;
        pv[j] = d[j];
        d[j] = d[j] + np;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) { psi[j] = ps[j]; prev[j] = pv[j]; }
}
template <bool RS, class R, bool EX = false>
__device__ __forceinline__ void cpml_s(R (&d)[4], R* psi, R* prev, R bb, R ee, R r) {
    R ps[4], pv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        ps[j] = RS ? mulr(psi[j], r) : psi[j];
        pv[j] = RS ? mulr(prev[j], r) : prev[j];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        R np = cpml_psi<EX>(ps[j], pv[j], d[j], bb, ee);
        ps[j] = np;
        pv[j] = d[j];
        d[j] = d[j] + np;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) { psi[j] = ps[j]; prev[j] = pv[j]; }
}

// Vector access helpers for the memory variables (ψ in fp32 or fp64).
template <class R>
struct PsiIO {
    __device__ __forceinline__ static void ld(const R* p, R (&v)[4]) {
        if constexpr (sizeof(R) == 4) {
            float4 t = *reinterpret_cast<const float4*>(p);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
            v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
        }
    }
    __device__ __forceinline__ static void st(R* p, const R (&v)[4]) {
        if constexpr (sizeof(R) == 4) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
            reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
        }
    }
};

// One derivative slot of one axis: memory variables k (ψ) and NS+k (prev) of
// the (phase, axis) slab array; fwd selects the half-grid profile.
template <int NS, bool RS, class R, bool EX = false>
__device__ __forceinline__ void cpml_slot(R (&d)[4], void* base, long long cells, int k, cidx sidx,
                                          bool xaxis, int pos, int x0, const void* pb, const void* pe, R r,
                                          void* out = nullptr, bool st = true) {
    R* ps = static_cast<R*>(base) + (long long)k * cells + sidx;
    R* pv = static_cast<R*>(base) + (long long)(NS + k) * cells + sidx;
    R psv[4], pvv[4];
    PsiIO<R>::ld(ps, psv);
    PsiIO<R>::ld(pv, pvv);
    const R* b = static_cast<const R*>(pb);
    const R* e = static_cast<const R*>(pe);
    if (xaxis) cpml_x<RS, R, EX>(d, psv, pvv, b, e, x0, r);
    else cpml_s<RS, R, EX>(d, psv, pvv, b[pos], e[pos], r);
    if (out) {       // double-buffered memory variables: the new values go to `out`
        ps = static_cast<R*>(out) + (long long)k * cells + sidx;
        pv = static_cast<R*>(out) + (long long)(NS + k) * cells + sidx;
    }
    if (st) {
        PsiIO<R>::st(ps, psv);
        PsiIO<R>::st(pv, pvv);
    }
}

// The memory variables of every slot of one axis at once (slot k: derivative
// d[k], the half-grid profile if half bit k): all the loads before the first
// store, so a chunk waits once for an axis instead of once per slot (the
// compiler cannot move a load over a store to the same type).  Measured on B200,
// us per step, slot by slot -> at once (FP32 where not named): 296 x 296 x 232
// 1740 -> 1553, 4040 x 2040 179 -> 166, 817 x 1073 21.2 -> 19.3, 200^3 order 2
// 492 -> 482; FP64 1040 x 540 40.0 -> 38.1.
template <int NS, bool RS, class R, bool EX = false, bool SLOTWISE = false>
__device__ __forceinline__ void cpml_axis(R (*const (&d)[NS])[4], unsigned half, void* base, long long cells,
                                          cidx sidx, bool xaxis, int pos, int x0, const void* pb, const void* pe,
                                          const void* pb2, const void* pe2, R r, void* out, bool st) {
    if constexpr (SLOTWISE) {
#pragma unroll
        for (int k = 0; k < NS; k++)
            cpml_slot<NS, RS, R, EX>(*d[k], base, cells, k, sidx, xaxis, pos, x0, (half >> k & 1) ? pb2 : pb,
                                     (half >> k & 1) ? pe2 : pe, r, out, st);
        return;
    }
    R ps[NS][4], pv[NS][4];
#pragma unroll
    for (int k = 0; k < NS; k++) {
        PsiIO<R>::ld(static_cast<const R*>(base) + (long long)k * cells + sidx, ps[k]);
        PsiIO<R>::ld(static_cast<const R*>(base) + (long long)(NS + k) * cells + sidx, pv[k]);
    }
    R* o = static_cast<R*>(out ? out : base);
#pragma unroll
    for (int k = 0; k < NS; k++) {
        const R* b = static_cast<const R*>((half >> k & 1) ? pb2 : pb);
        const R* e = static_cast<const R*>((half >> k & 1) ? pe2 : pe);
        if (xaxis) cpml_x<RS, R, EX>(*d[k], ps[k], pv[k], b, e, x0, r);
        else cpml_s<RS, R, EX>(*d[k], ps[k], pv[k], b[pos], e[pos], r);
    }
    if (st) {
#pragma unroll
        for (int k = 0; k < NS; k++) {
            PsiIO<R>::st(o + (long long)k * cells + sidx, ps[k]);
            PsiIO<R>::st(o + (long long)(NS + k) * cells + sidx, pv[k]);
        }
    }
}

// Slab memory-variable index of a chunk for one axis, or -1 outside the slab.
__device__ __forceinline__ cidx slab_index(const ShotDesc& S, int axis, int x0, int y, int z) {
    const Slab& sl = S.slab[axis];
    if (axis == 0) {
        int sx = sl.index(x0);
        if (sx < 0) return -1;
        return (z * S.ny + y) * sl.width + sx;
    } else if (axis == 1) {
        int sy = sl.index(y);
        if (sy < 0) return -1;
        return (z * sl.width + sy) * S.pitch + x0;
    } else {
        int sz = sl.index(z);
        if (sz < 0) return -1;
        return (sz * S.ny + y) * S.pitch + x0;
    }
}

// ---------------------------------------------------------------------------
// Everything of the V phase after the stress derivatives: COMP16 rescale,
// masking, CPML memory variables, divergence, the velocity updates and their
// stores.  PRE: the caller has already loaded the coefficients and old
// velocities into V (the marching kernel); otherwise they are loaded here.
// RS: old state is multiplied by the COMP16 rescale r; the kernels pass false
// when r is exactly 1, which gives the same bits without the products.
// Where a phase tail stores: the field arrays (and COMP16 residuals) of the
// new state, and the memory variables it reads (psi_in) and writes (psi_out).
// In place, the single-buffered kernels' case, everything is the descriptor's
// own; the fused step kernel (step_fused.cu) reads one copy of the state and
// writes the other, and computes without storing on its halo cells.
struct TailOut {
    void* const* f;
    int8_t* const* flo;
    void* const* psi_in;
    void* const* psi_out;        // nullptr: in place
    bool store;                  // false: compute only (the fused kernel's halo cells)
    __device__ __forceinline__ static TailOut v_of(const ShotDesc& S) { return TailOut{S.f, S.flo, S.psiV, nullptr, true}; }
    __device__ __forceinline__ static TailOut t_of(const ShotDesc& S) { return TailOut{S.f, S.flo, S.psiT, nullptr, true}; }
};

// Coefficients of a chunk: from the per-cell arrays, or from the tuple table
// of an indexed medium (float policies only; FP64 shots are never indexed).
template <class P>
__device__ __forceinline__ bool med_on(const ShotDesc& S) {
    if constexpr (sizeof(typename P::real) == 4) return S.med_idx != nullptr;
    else return false;
}
// Component q of group g of the chunk's four tuples.
template <class R>
__device__ __forceinline__ void med_comp4(const ShotDesc& S, unsigned ids, int g, int q, R (&o)[4]) {
    float4 t[4];
    med_group4(S, ids, g, t);
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = (R)(q == 0 ? t[j].x : q == 1 ? t[j].y : q == 2 ? t[j].z : t[j].w);
}
// One V-phase coefficient (VCoef k) of the chunk at c (ids: its tuple indices).
template <class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void vcoef4(const ShotDesc& S, int k, cidx c, unsigned ids, typename P::real (&o)[4]) {
    if (med_on<P>(S)) {
        const int g = (k == VC_RHO_Y || k == VC_CC1_Y || k == VC_CC2_Y) ? MED_V_Y
                      : (k == VC_RHO_Z || k == VC_CC1_Z || k == VC_CC2_Z) ? MED_V_Z : MED_V_X;
        const int q = k == VC_RHOF ? 3 : (k == VC_RHO_X || k == VC_RHO_Y || k == VC_RHO_Z) ? 0
                      : (k == VC_CC1_X || k == VC_CC1_Y || k == VC_CC1_Z) ? 1 : 2;
        med_comp4(S, ids, g, q, o);
        return;
    }
    P::template ld4<NC>(S.vc[k], S.vclo[k], c, o);
}
// One T-phase coefficient (TCoef k) of the chunk at c.
template <class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void tcoef4(const ShotDesc& S, int k, cidx c, unsigned ids, typename P::real (&o)[4]) {
    if (med_on<P>(S)) {
        const int g = (k == TC_C || k == TC_M || k == TC_H || k == TC_H2U) ? MED_T_A : MED_T_B;
        const int q = (k == TC_C || k == TC_MUXZ) ? 0 : (k == TC_M || k == TC_MUXY) ? 1
                      : (k == TC_H || k == TC_MUYZ) ? 2 : 3;
        med_comp4(S, ids, g, q, o);
        return;
    }
    P::template ld4<NC>(S.tc[k], S.tclo[k], c, o);
}

// How the tails load what they need besides the derivatives, by where a chunk's
// values come from (the sources below and in tile.cuh and async.cuh).  kAhead: FP32
// loads every axis' coefficients and old velocities before the first axis'
// stores, and divides without a test for zero.  kSlotwise: the CPML memory
// variables slot by slot.
struct SrcForm {
    static constexpr bool kAhead = true, kSlotwise = false;
};

// The chunk's old values of a field the phase updates, from its array.
template <class P>
struct ArraySrc : SrcForm {
    const ShotDesc& S;
    cidx c;
    __device__ __forceinline__ ArraySrc(const ShotDesc& S_, cidx c_) : S(S_), c(c_) {}
    template <int F>
    __device__ __forceinline__ void own(typename P::real (&v)[4]) const { P::ld4(S.f[F], S.flo[F], c, v); }
};

// The same with the tuple indices loaded here: one test of the medium's form per
// coefficient, on which the compiler joins consecutive ones.  With a second test
// around the index load the fused kernel of a per-cell medium waited for every
// coefficient in turn (4040 x 2040 FP32 676 us per step, 417 this way; order 4
// 1200 and 1000; COMP16 1026 and 943; B200).
template <class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void vcoef4(const ShotDesc& S, int k, cidx c, typename P::real (&o)[4]) {
    if (med_on<P>(S)) vcoef4<P, NC>(S, k, c, med_ids(S, c), o);
    else P::template ld4<NC>(S.vc[k], S.vclo[k], c, o);
}
template <class P, bool NC = kReadOnlyPath>
__device__ __forceinline__ void tcoef4(const ShotDesc& S, int k, cidx c, typename P::real (&o)[4]) {
    if (med_on<P>(S)) tcoef4<P, NC>(S, k, c, med_ids(S, c), o);
    else P::template ld4<NC>(S.tc[k], S.tclo[k], c, o);
}

template <class R>
struct VState {
    R x1[4], x3[4], s1[4], z1[4], z2[4], s3[4];       // derivatives (2D and 3D)
    R x2[4], y1[4], y2[4], y3[4], s2[4], z3[4];       // 3D only
    R rf[4], rho_x[4], c1_x[4], c2_x[4], vu_x[4], vw_x[4], rho_z[4], c1_z[4], c2_z[4], vu_z[4], vw_z[4];
    R rho_y[4], c1_y[4], c2_y[4], vu_y[4], vw_y[4];
    unsigned mids;                 // indexed medium: the chunk's four tuple indices (set before the tail)
};

// On return V's old-velocity members (vu_*, vw_*) hold the new velocities as a
// later load of the stored values returns them.
template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath, class Src>
__device__ __forceinline__ void v_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, VState<typename P::real>& V, const TailOut& O, const Src& src) {
    using R = typename P::real;
    auto &x1 = V.x1, &x3 = V.x3, &s1 = V.s1, &z1 = V.z1, &z2 = V.z2, &s3 = V.s3;
    auto &x2 = V.x2, &y1 = V.y1, &y2 = V.y2, &y3 = V.y3, &s2 = V.s2, &z3 = V.z3;
    auto &rf = V.rf, &rho_x = V.rho_x, &c1_x = V.c1_x, &c2_x = V.c2_x, &vu_x = V.vu_x, &vw_x = V.vw_x;
    auto &rho_z = V.rho_z, &c1_z = V.c1_z, &c2_z = V.c2_z, &vu_z = V.vu_z, &vw_z = V.vw_z;
    auto &rho_y = V.rho_y, &c1_y = V.c1_y, &c2_y = V.c2_y, &vu_y = V.vu_y, &vw_y = V.vw_y;
    const bool med = med_on<P>(S);
    auto load_axis = [&](int crho, int ccc1, int ccc2, R (&rho)[4], R (&c1)[4], R (&c2)[4]) {
        if (med) {
            // one group per cell: (rho, cc1, cc2, rhof) of this axis
            const int g = crho == VC_RHO_X ? MED_V_X : crho == VC_RHO_Y ? MED_V_Y : MED_V_Z;
            float4 t[4];
            med_group4(S, V.mids, g, t);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                rho[j] = (R)t[j].x; c1[j] = (R)t[j].y; c2[j] = (R)t[j].z;
                if (g == MED_V_X) rf[j] = (R)t[j].w;
            }
        } else {
            P::template ld4<NC>(S.vc[crho], S.vclo[crho], c, rho);
            P::template ld4<NC>(S.vc[ccc1], S.vclo[ccc1], c, c1);
            P::template ld4<NC>(S.vc[ccc2], S.vclo[ccc2], c, c2);
        }
    };
    // the rescale factor applies to old stresses: scale their derivatives
    if constexpr (P::prec == BP_PREC_COMP16 && RS) {
        scale4(x1, r); scale4(s1, r); scale4(z2, r); scale4(x3, r); scale4(z1, r); scale4(s3, r);
        if constexpr (DIM == 3) { scale4(x2, r); scale4(y1, r); scale4(y2, r); scale4(y3, r); scale4(s2, r); scale4(z3, r); }
    }
    // masked cells (never updated) feed zero derivatives into the memory variables
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(mask >> j & 1u)) {
            x1[j] = 0; s1[j] = 0; z2[j] = 0; x3[j] = 0; z1[j] = 0; s3[j] = 0;
            if constexpr (DIM == 3) { x2[j] = 0; y1[j] = 0; y2[j] = 0; y3[j] = 0; s2[j] = 0; z3[j] = 0; }
        }

    // ---- CPML memory variables on the slabs (Float/main.cu:130-158) ----
    {
        constexpr int NS = DIM == 3 ? 4 : 3;
        // half-grid profile for the forward differences (bits by slot)
        auto axis = [&](R (*const (&d)[NS])[4], unsigned half, int a, int pos) {
            const cidx si = slab_index(S, a, x0, y, z);
            if (si >= 0)
                cpml_axis<NS, RS, R, P::exact, Src::kSlotwise>(d, half, O.psi_in[a], S.slab_cells[a], si, a == 0, pos, x0, S.pb[a],
                                               S.pe[a], S.pb2[a], S.pe2[a], r, O.psi_out ? O.psi_out[a] : nullptr, O.store);
        };
        if constexpr (DIM == 3) {
            R (*const dx[NS])[4] = {&x1, &s1, &z2, &y2};
            R (*const dy[NS])[4] = {&x2, &y1, &s2, &z3};
            R (*const dz[NS])[4] = {&x3, &z1, &s3, &y3};
            axis(dx, 0x3u, 0, x0);
            axis(dy, 0x6u, 1, y);
            axis(dz, 0x6u, 2, z);
        } else {
            R (*const dx[NS])[4] = {&x1, &s1, &z2};
            R (*const dz[NS])[4] = {&x3, &z1, &s3};
            axis(dx, 0x3u, 0, x0);
            axis(dz, 0x6u, 2, z);
        }
    }

    // ---- stress divergence per axis ----
    R sumx[4], sumz[4], sumy[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (DIM == 3) {
            sumx[j] = x1[j] + x2[j] + x3[j];
            sumy[j] = y1[j] + y2[j] + y3[j];
            sumz[j] = z1[j] + z2[j] + z3[j];
        } else {
            sumx[j] = x1[j] + x3[j];
            sumz[j] = z1[j] + z2[j];
        }
    }

    // ---- velocity updates per axis (Float/main.cu:106-113,160-190) ----
    auto axis_update = [&](const R (&sum)[4], const R (&dp)[4], int fu, int fw, const R (&rho)[4],
                           const R (&c1)[4], const R (&c2)[4], R (&vu)[4], R (&vw)[4]) {
        R nu[4], nw[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16) {
                // Half/main.cu:256-262 with Bt = (rhof rho^-1) Bp formed here
                const R wo = RS ? mulr(vw[j], r) : vw[j], uo = RS ? mulr(vu[j], r) : vu[j];
                R rr = rf[j] * rho[j];                    // rhof * rho^-1
                // one contraction for every kernel family: the result must not
                // depend on which products the compiler fuses here
                const R wn = fma_rn(-c2[j], dp[j], fma_rn(c1[j], wo, -mul_rn(rr * c2[j], sum[j])));
                nw[j] = wn;
                nu[j] = uo + rho[j] * sum[j] - rr * (wn - wo);
            } else {
                R wo = vw[j];
                const R num = wo * c2[j] - S.dtr<R>() * (rf[j] * rho[j] * sum[j] + dp[j]);
                const R wn = (c1[j] == (R)0) ? (R)0 : quot<P, DIM, !Src::kAhead>(num, c1[j]);
                nw[j] = wn;
                nu[j] = vu[j] + S.dtr<R>() * rho[j] * sum[j] - rf[j] * rho[j] * (wn - wo);
            }
            if (!(mask >> j & 1u)) { nw[j] = vw[j]; nu[j] = vu[j]; }
        }
        P::st4_rt(O.f[fw], O.flo[fw], c, nw, O.store);
        P::st4_rt(O.f[fu], O.flo[fu], c, nu, O.store);
#pragma unroll
        for (int j = 0; j < 4; j++) { vw[j] = nw[j]; vu[j] = nu[j]; }
    };
    // FP32 loads every axis' coefficients and old velocities before the first
    // axis' stores, so the chunk waits for them once.  Measured on B200 (us per
    // step): 424 x 424 x 328 per-cell medium 3066 -> 2887, 296 x 296 x 232 1495 ->
    // 1436, 4040 x 2040 per-cell 205.8 -> 202.9, indexed 162.6 -> 163.4.  The
    // 3-byte and FP64 forms spill and lose: COMP16 2D 259 -> 321, CBF16 296 x
    // 296 x 232 1681 -> 1791, FP64 168^3 814 -> 899.
    constexpr bool kAhead = P::store == BP_PREC_FP32 && Src::kAhead;
    auto load_x = [&] {
        if (!med) P::template ld4<NC>(S.vc[VC_RHOF], S.vclo[VC_RHOF], c, rf);   // indexed: with the x group
        load_axis(VC_RHO_X, VC_CC1_X, VC_CC2_X, rho_x, c1_x, c2_x);
        src.template own<BP_F_VUX>(vu_x);
        src.template own<BP_F_VWX>(vw_x);
    };
    auto load_y = [&] {
        if constexpr (DIM == 3) {
            load_axis(VC_RHO_Y, VC_CC1_Y, VC_CC2_Y, rho_y, c1_y, c2_y);
            src.template own<BP_F_VUY>(vu_y);
            src.template own<BP_F_VWY>(vw_y);
        }
    };
    auto load_z = [&] {
        load_axis(VC_RHO_Z, VC_CC1_Z, VC_CC2_Z, rho_z, c1_z, c2_z);
        src.template own<BP_F_VUZ>(vu_z);
        src.template own<BP_F_VWZ>(vw_z);
    };
    if constexpr (!PRE) {
        load_x();
        if constexpr (kAhead) {
            if constexpr (DIM == 3) load_y();
            load_z();
        }
    }
    axis_update(sumx, s1, BP_F_VUX, BP_F_VWX, rho_x, c1_x, c2_x, vu_x, vw_x);
    if constexpr (DIM == 3) {
        if constexpr (!PRE && !kAhead) load_y();
        axis_update(sumy, s2, BP_F_VUY, BP_F_VWY, rho_y, c1_y, c2_y, vu_y, vw_y);
    }
    if constexpr (!PRE && !kAhead) load_z();
    axis_update(sumz, s3, BP_F_VUZ, BP_F_VWZ, rho_z, c1_z, c2_z, vu_z, vw_z);
}

template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath>
__device__ __forceinline__ void v_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, VState<typename P::real>& V) {
    v_tail<DIM, ORD, P, PRE, RS, NC>(S, c, x0, y, z, r, mask, V, TailOut::v_of(S), ArraySrc<P>(S, c));
}
template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath>
__device__ __forceinline__ void v_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, VState<typename P::real>& V, const TailOut& O) {
    v_tail<DIM, ORD, P, PRE, RS, NC>(S, c, x0, y, z, r, mask, V, O, ArraySrc<P>(S, c));
}

// ---------------------------------------------------------------------------
// COMP16's new normal stress.  c w, shared by the normal stresses, is rounded by
// itself: written out, so that every kernel family stores the same bits.
__device__ __forceinline__ float c16_normal(float o, float h2, float e2, float h, float e, float c, float w) {
    return __fadd_rn(__fmaf_rn(h, e, __fmaf_rn(h2, e2, o)), __fmul_rn(c, w));
}

// Everything of the T phase after the velocity derivatives: masking, CPML
// memory variables, the pressure and stress updates and their stores.  PRE:
// the caller has already loaded the moduli and the old stresses into T, the
// latter multiplied by the COMP16 rescale (the marching kernel).
template <class R>
struct TState {
    R uxx[4], uzz[4], wx[4], wz[4], uxz[4], uzx[4];   // derivatives (2D and 3D)
    R uyy[4], wy[4], uxy[4], uyx[4], uyz[4], uzy[4];   // 3D only
    R cC[4], cM[4], cH[4], cH2[4], mxz[4], op[4], oxx[4], ozz[4], oxz[4];
    R mxy[4], myz[4], oyy[4], oxy[4], oyz[4];
    unsigned mids;                 // indexed medium: the chunk's four tuple indices (set before the tail)
};

// On return T's old-stress members (op, oxx, ...) hold the new values.
template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath, class Src>
__device__ __forceinline__ void t_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, TState<typename P::real>& T, const TailOut& O, const Src& src) {
    using R = typename P::real;
    auto &uxx = T.uxx, &uzz = T.uzz, &wx = T.wx, &wz = T.wz, &uxz = T.uxz, &uzx = T.uzx;
    auto &uyy = T.uyy, &wy = T.wy, &uxy = T.uxy, &uyx = T.uyx, &uyz = T.uyz, &uzy = T.uzy;
    auto &cC = T.cC, &cM = T.cM, &cH = T.cH, &cH2 = T.cH2, &mxz = T.mxz;
    auto &op = T.op, &oxx = T.oxx, &ozz = T.ozz, &oxz = T.oxz;
    auto &mxy = T.mxy, &myz = T.myz, &oyy = T.oyy, &oxy = T.oxy, &oyz = T.oyz;
    auto load_state = [&]() {
        if (med_on<P>(S)) {
            const unsigned ids = T.mids;
            float4 a[4], b[4];
            med_group4(S, ids, MED_T_A, a);
            med_group4(S, ids, MED_T_B, b);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                cC[j] = (R)a[j].x; cM[j] = (R)a[j].y; cH[j] = (R)a[j].z; cH2[j] = (R)a[j].w; mxz[j] = (R)b[j].x;
                if constexpr (DIM == 3) { mxy[j] = (R)b[j].y; myz[j] = (R)b[j].z; }
            }
        } else {
            P::template ld4<NC>(S.tc[TC_C], S.tclo[TC_C], c, cC);
            P::template ld4<NC>(S.tc[TC_M], S.tclo[TC_M], c, cM);
            P::template ld4<NC>(S.tc[TC_H], S.tclo[TC_H], c, cH);
            P::template ld4<NC>(S.tc[TC_H2U], S.tclo[TC_H2U], c, cH2);
            P::template ld4<NC>(S.tc[TC_MUXZ], S.tclo[TC_MUXZ], c, mxz);
            if constexpr (DIM == 3) {
                P::template ld4<NC>(S.tc[TC_MUXY], S.tclo[TC_MUXY], c, mxy);
                P::template ld4<NC>(S.tc[TC_MUYZ], S.tclo[TC_MUYZ], c, myz);
            }
        }
        src.template own<BP_F_P>(op);
        src.template own<BP_F_TXX>(oxx);
        src.template own<BP_F_TZZ>(ozz);
        src.template own<BP_F_TXZ>(oxz);
        if constexpr (DIM == 3) {
            src.template own<BP_F_TYY>(oyy);
            src.template own<BP_F_TXY>(oxy);
            src.template own<BP_F_TYZ>(oyz);
        }
        if constexpr (P::prec == BP_PREC_COMP16 && RS) {     // old state takes this step's rescale
            scale4(op, r); scale4(oxx, r); scale4(ozz, r); scale4(oxz, r);
            if constexpr (DIM == 3) { scale4(oyy, r); scale4(oxy, r); scale4(oyz, r); }
        }
    };
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(mask >> j & 1u)) {
            uxx[j] = 0; wx[j] = 0; uzx[j] = 0; uzz[j] = 0; wz[j] = 0; uxz[j] = 0;
            if constexpr (DIM == 3) { uyx[j] = 0; uyy[j] = 0; wy[j] = 0; uxy[j] = 0; uyz[j] = 0; uzy[j] = 0; }
        }

    // ---- CPML (Float/main.cu:252-285).  The velocities are this step's, but the
    // stored ψ/prev of this phase are old state and take the rescale r ----
    {
        constexpr int NS = DIM == 3 ? 4 : 3;
        auto axis = [&](R (*const (&d)[NS])[4], unsigned half, int a, int pos) {
            const cidx si = slab_index(S, a, x0, y, z);
            if (si >= 0)
                cpml_axis<NS, RS, R, P::exact, Src::kSlotwise>(d, half, O.psi_in[a], S.slab_cells[a], si, a == 0, pos, x0, S.pb[a],
                                               S.pe[a], S.pb2[a], S.pe2[a], r, nullptr, O.store);
        };
        if constexpr (DIM == 3) {
            R (*const dx[NS])[4] = {&uxx, &wx, &uzx, &uyx};
            R (*const dy[NS])[4] = {&uyy, &wy, &uxy, &uzy};
            R (*const dz[NS])[4] = {&uzz, &wz, &uxz, &uyz};
            axis(dx, 0xcu, 0, x0);
            axis(dy, 0xcu, 1, y);
            axis(dz, 0xcu, 2, z);
        } else {
            R (*const dx[NS])[4] = {&uxx, &wx, &uzx};
            R (*const dz[NS])[4] = {&uzz, &wz, &uxz};
            axis(dx, 0x4u, 0, x0);
            axis(dz, 0x4u, 2, z);
        }
    }

    // ---- pressure and stress updates (Float/main.cu:287-293) ----
    if constexpr (!PRE) load_state();
    const R dt = S.dtr<R>();
    auto finish = [&](int f, R (&nv)[4], R (&ov)[4]) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (!(mask >> j & 1u)) nv[j] = ov[j];
        if (O.store) P::st4(O.f[f], O.flo[f], c, nv);
#pragma unroll
        for (int j = 0; j < 4; j++) ov[j] = nv[j];
    };
    R n[4];
    if constexpr (DIM == 3) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = op[j] - cC[j] * (uxx[j] + uyy[j] + uzz[j]) - cM[j] * (wx[j] + wy[j] + wz[j]);
            else
                n[j] = op[j] - dt * (cC[j] * (uxx[j] + uyy[j] + uzz[j]) + cM[j] * (wx[j] + wy[j] + wz[j]));
        }
        finish(BP_F_P, n, op);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(oxx[j], cH2[j], (uyy[j] + uzz[j]), cH[j], uxx[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = oxx[j] + dt * (cH2[j] * (uyy[j] + uzz[j]) + cH[j] * uxx[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        }
        finish(BP_F_TXX, n, oxx);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(oyy[j], cH2[j], (uxx[j] + uzz[j]), cH[j], uyy[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = oyy[j] + dt * (cH2[j] * (uxx[j] + uzz[j]) + cH[j] * uyy[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        }
        finish(BP_F_TYY, n, oyy);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(ozz[j], cH2[j], (uxx[j] + uyy[j]), cH[j], uzz[j], cC[j], (wx[j] + wy[j] + wz[j]));
            else
                n[j] = ozz[j] + dt * (cH2[j] * (uxx[j] + uyy[j]) + cH[j] * uzz[j] + cC[j] * (wx[j] + wy[j] + wz[j]));
        }
        finish(BP_F_TZZ, n, ozz);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16) n[j] = oxy[j] + mxy[j] * (uxy[j] + uyx[j]);
            else n[j] = oxy[j] + mxy[j] * dt * (uxy[j] + uyx[j]);
        }
        finish(BP_F_TXY, n, oxy);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16) n[j] = oyz[j] + myz[j] * (uyz[j] + uzy[j]);
            else n[j] = oyz[j] + myz[j] * dt * (uyz[j] + uzy[j]);
        }
        finish(BP_F_TYZ, n, oyz);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16) n[j] = oxz[j] + mxz[j] * (uxz[j] + uzx[j]);
            else n[j] = oxz[j] + mxz[j] * dt * (uxz[j] + uzx[j]);
        }
        finish(BP_F_TXZ, n, oxz);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = op[j] - cC[j] * (uxx[j] + uzz[j]) - cM[j] * (wx[j] + wz[j]);
            else
                n[j] = op[j] - dt * (cC[j] * (uxx[j] + uzz[j]) + cM[j] * (wx[j] + wz[j]));
        }
        finish(BP_F_P, n, op);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(oxx[j], cH2[j], uzz[j], cH[j], uxx[j], cC[j], (wx[j] + wz[j]));
            else
                n[j] = oxx[j] + dt * (cH2[j] * uzz[j] + cH[j] * uxx[j] + cC[j] * (wx[j] + wz[j]));
        }
        finish(BP_F_TXX, n, oxx);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16)
                n[j] = c16_normal(ozz[j], cH2[j], uxx[j], cH[j], uzz[j], cC[j], (wx[j] + wz[j]));
            else
                n[j] = ozz[j] + dt * (cH2[j] * uxx[j] + cH[j] * uzz[j] + cC[j] * (wx[j] + wz[j]));
        }
        finish(BP_F_TZZ, n, ozz);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if constexpr (P::prec == BP_PREC_COMP16) n[j] = oxz[j] + mxz[j] * (uxz[j] + uzx[j]);
            else n[j] = oxz[j] + mxz[j] * dt * (uxz[j] + uzx[j]);
        }
        finish(BP_F_TXZ, n, oxz);
    }
}

template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath>
__device__ __forceinline__ void t_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, TState<typename P::real>& T) {
    t_tail<DIM, ORD, P, PRE, RS, NC>(S, c, x0, y, z, r, mask, T, TailOut::t_of(S), ArraySrc<P>(S, c));
}
template <int DIM, int ORD, class P, bool PRE, bool RS, bool NC = kReadOnlyPath>
__device__ __forceinline__ void t_tail(const ShotDesc& S, cidx c, int x0, int y, int z, typename P::real r,
                                       unsigned mask, TState<typename P::real>& T, const TailOut& O) {
    t_tail<DIM, ORD, P, PRE, RS, NC>(S, c, x0, y, z, r, mask, T, O, ArraySrc<P>(S, c));
}

}  // namespace bpk
