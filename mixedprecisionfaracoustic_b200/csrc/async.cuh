// async.cuh - a warp's field values in shared memory, filled by asynchronous
// copies: what the staged tile kernels (step_async.cu) read in place of the
// field arrays.
#pragma once
#include "tile.cuh"

namespace bpk {

// One staged row of a unit: the chunks of field f in the row `off` rows away
// along y (ax 1) or z (ax 2), or the chunks themselves (ax 0).
struct SlotId {
    int f, ax, off;
};
struct SlotTable {
    SlotId s[48];
    int n;
    int left[8], right[8], nl, nr;      // slots read across their left / right edge
};
// The rows one phase reads (V: FD_V, T: FD_T), the fields it updates among them.
template <int DIM, int ORD, bool V>
constexpr SlotTable slot_table() {
    SlotTable t{};
    constexpr int HW = ORD / 2;
    t.n = 0; t.nl = 0; t.nr = 0;
    auto row = [&](int f, int ax, int off) { t.s[t.n++] = SlotId{f, ax, off}; };
    // x differences: forward reads 1 .. HW cells to the right (HW - 1 to the left), backward the mirror
    auto centre = [&](int f, bool span, bool fwd) {
        if (span && (fwd || ORD == 4)) t.right[t.nr++] = t.n;
        if (span && (!fwd || ORD == 4)) t.left[t.nl++] = t.n;
        row(f, 0, 0);
    };
    auto across = [&](int f, int ax, bool fwd) {
        for (int o = fwd ? 1 - HW : -HW; o <= (fwd ? HW : HW - 1); o++)
            if (o != 0) row(f, ax, o);
    };
    if (V) {
        centre(BP_F_TXX, true, true);
        centre(BP_F_P, true, true);
        centre(BP_F_TXZ, true, false);
        centre(BP_F_TZZ, false, false);
        across(BP_F_TXZ, 2, false);
        across(BP_F_TZZ, 2, true);
        across(BP_F_P, 2, true);
        if (DIM == 3) {
            centre(BP_F_TXY, true, false);
            centre(BP_F_TYY, false, false);
            centre(BP_F_TYZ, false, false);
            across(BP_F_TXY, 1, false);
            across(BP_F_TYY, 1, true);
            across(BP_F_TYZ, 1, false);
            across(BP_F_TYZ, 2, false);
            across(BP_F_P, 1, true);
        }
        row(BP_F_VUX, 0, 0); row(BP_F_VWX, 0, 0);
        if (DIM == 3) { row(BP_F_VUY, 0, 0); row(BP_F_VWY, 0, 0); }
        row(BP_F_VUZ, 0, 0); row(BP_F_VWZ, 0, 0);
    } else {
        centre(BP_F_VUX, true, false);
        centre(BP_F_VWX, true, false);
        centre(BP_F_VUZ, true, true);
        centre(BP_F_VWZ, false, false);
        across(BP_F_VUZ, 2, false);
        across(BP_F_VWZ, 2, false);
        across(BP_F_VUX, 2, true);
        if (DIM == 3) {
            centre(BP_F_VUY, true, true);
            centre(BP_F_VWY, false, false);
            across(BP_F_VUY, 1, false);
            across(BP_F_VWY, 1, false);
            across(BP_F_VUX, 1, true);
            across(BP_F_VUY, 2, true);
            across(BP_F_VUZ, 1, true);
        }
        row(BP_F_P, 0, 0); row(BP_F_TXX, 0, 0); row(BP_F_TZZ, 0, 0); row(BP_F_TXZ, 0, 0);
        if (DIM == 3) { row(BP_F_TYY, 0, 0); row(BP_F_TXY, 0, 0); row(BP_F_TYZ, 0, 0); }
    }
    return t;
}
__host__ __device__ constexpr int slot_of(const SlotTable& t, int f, int ax, int off) {
    for (int i = 0; i < t.n; i++)
        if (t.s[i].f == f && (off == 0 ? t.s[i].ax == 0 : (t.s[i].ax == ax && t.s[i].off == off))) return i;
    return -1;
}

// A COMP16 slot: 34 chunks, the 32 lanes' between one to the left of lane 0 and
// one to the right of lane 31; the hi words, then the residuals.
constexpr int kSlotHi = 34 * 8, kSlotBytes = kSlotHi + 34 * 4;

template <int B>
__device__ __forceinline__ void copy_async(void* smem, const void* g) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(g), "n"(B) : "memory");
}
// Starts the copy of the chunk at cell offset i of field f into entry e of a slot.
__device__ __forceinline__ void slot_fill(const ShotDesc& S, char* slot, int e, int f, cidx i) {
    copy_async<8>(slot + e * 8, static_cast<const uint16_t*>(S.f[f]) + i);
    copy_async<4>(slot + kSlotHi + e * 4, S.flo[f] + i);
}

// Source of a chunk's field values (tile.cuh) over the warp's slots.
template <int DIM, int ORD, class P, bool V>
struct AsyncSrc : SrcForm {
    static_assert(P::store == BP_PREC_COMP16, "the slots hold COMP16 chunks");
    using R = typename P::real;
    static constexpr SlotTable T = slot_table<DIM, ORD, V>();
    static constexpr int kBytes = T.n * kSlotBytes;
    char* w;          // the warp's slots
    int lane;
    __device__ __forceinline__ AsyncSrc(char* w_, int lane_) : w(w_), lane(lane_) {}

    template <int I>
    __device__ __forceinline__ void get4(R (&v)[4]) const {
        static_assert(I >= 0, "the slot table lacks a row");
        char* s = w + I * kSlotBytes;
        P::ld4(s, reinterpret_cast<const int8_t*>(s + kSlotHi), (lane + 1) * 4, v);
    }
    template <int I>
    __device__ __forceinline__ R get1(int k) const {        // cell k of the chunk, -HW .. 3 + HW
        char* s = w + I * kSlotBytes;
        return P::ld1(s, reinterpret_cast<const int8_t*>(s + kSlotHi), (lane + 1) * 4 + k);
    }
    template <int F>
    __device__ __forceinline__ void span(R (&v)[4 + ORD]) const {
        constexpr int HW = ORD / 2, I = slot_of(T, F, 0, 0);
        R q[4];
        get4<I>(q);
#pragma unroll
        for (int j = 0; j < 4; j++) v[HW + j] = q[j];
#pragma unroll
        for (int k = 1; k <= HW; k++) {
            v[HW - k] = get1<I>(-k);
            v[HW + 3 + k] = get1<I>(3 + k);
        }
    }
    template <int F, int AX, int O>
    __device__ __forceinline__ void row(R (&v)[4]) const {
        constexpr int I = slot_of(T, F, AX, O);
        // rows the difference does not read are not staged, nor used
        if constexpr (I >= 0) get4<I>(v);
        else v[0] = v[1] = v[2] = v[3] = (R)0;
    }
    template <int F, int AX>
    __device__ __forceinline__ void rows(R (&a)[ORD + 1][4]) const {
        if constexpr (ORD == 2) {
            row<F, AX, -1>(a[0]); row<F, AX, 0>(a[1]); row<F, AX, 1>(a[2]);
        } else {
            row<F, AX, -2>(a[0]); row<F, AX, -1>(a[1]); row<F, AX, 0>(a[2]); row<F, AX, 1>(a[3]); row<F, AX, 2>(a[4]);
        }
    }
    template <int F>
    __device__ __forceinline__ void own(R (&v)[4]) const {
        get4<slot_of(T, F, 0, 0)>(v);
    }

    // Starts the copies of every row of the lane's chunk at cell c (x0: its
    // first x), the warp's edge chunks by its first and last lane.
    __device__ __forceinline__ static void fill(const ShotDesc& S, char* w, int lane, cidx c, int x0) {
        const cidx sy = S.pitch, sz = S.plane;
        fill_rows<0>(S, w, lane, c, sy, sz);
        if (lane == 0 && x0 > 0) fill_edges<true, 0>(S, w, 0, c - 4);
        if (lane == 31 && x0 + 4 < S.nx) fill_edges<false, 0>(S, w, 33, c + 4);
    }
    template <int I>
    __device__ __forceinline__ static void fill_rows(const ShotDesc& S, char* w, int lane, cidx c, cidx sy, cidx sz) {
        if constexpr (I < T.n) {
            constexpr SlotId d = T.s[I];
            slot_fill(S, w + I * kSlotBytes, lane + 1, d.f, c + (d.ax == 1 ? d.off * sy : d.ax == 2 ? d.off * sz : 0));
            fill_rows<I + 1>(S, w, lane, c, sy, sz);
        }
    }
    template <bool LEFT, int K>
    __device__ __forceinline__ static void fill_edges(const ShotDesc& S, char* w, int e, cidx c) {
        if constexpr (K < (LEFT ? T.nl : T.nr)) {
            constexpr int I = LEFT ? T.left[K] : T.right[K];
            slot_fill(S, w + I * kSlotBytes, e, T.s[I].f, c);
            fill_edges<LEFT, K + 1>(S, w, e, c);
        }
    }
};

}  // namespace bpk
