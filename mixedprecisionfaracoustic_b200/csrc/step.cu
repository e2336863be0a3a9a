// step.cu - the hot path: velocity phase, stress phase and post-step kernels.
//
// Reference kernels replaced (Zhitao-Zhang/MixedPrecisionFarAcoustic):
//   FD_V   Float/main.cu:64-192,  Half/main.cu:156-268  -> k_phase (VPHASE)
//   FD_T   Float/main.cu:194-295, Half/main.cu:270-371  -> k_phase (T)
//   Source Float/main.cu:45-59,   Half/main.cu:135-151  -> k_post (inject)
//   trace capture Float/main.cu:1075-1093               -> k_post (record)
//   ScaleHalfArray/ScaleCompressedArray Half/main.cu:102-114: folded into
//   k_phase as a per-step factor on every old state value.
//
// Work decomposition: a tile is 8 rows x 128 cells of one shot; a CTA of 8
// warps takes one tile at a time (one row per warp, 4 consecutive x cells per
// lane, 16-byte vector accesses along x; the 128 cells run on into the next
// row block where a row ends, flat_cell in tile.cuh).  CTAs loop over the tile
// table of all shots of a batch, so one launch advances every shot by one phase.
// Neighbour rows (y, z) are re-read through L1/L2; DRAM sees each array once
// per phase.  The CPML memory variables exist on the slabs only; a chunk
// touches them only when it lies in a slab of that axis.
#include "tile.cuh"

namespace bpk {

// PF: a CTA starts the L2 prefetch of its next tile before it works on a tile.
// FP32 launches of indexed media take it from kAheadTiles tiles a CTA on: 4040 x
// 2040 order 2 153.7 -> 148.0 us per step, order 4 163.2 -> 157.9, 200^3 order 2
// 409 -> 403 (B200).  Everything else loses by it: per-cell media, whose
// coefficients keep DRAM busy (4040 x 2040 196 -> 221, 424 x 424 x 328 2742 ->
// 3392), the 3-byte and FP64 formats, which wait less on loads (COMP16 255 ->
// 264, FP64 532 -> 614), and some short launches (817 x 1073 19.2 -> 20.0).  Around
// the line, without -> with: 2D order 2 at 3, 6, 8, 10 and 14 tiles a CTA 33.7 -> 32.7,
// 52.4 -> 51.5, 70.7 -> 67.6, 94.4 -> 89.5, 119.8 -> 113.0; 3D 73.1 -> 74.4, 119.7 ->
// 118.8, 158.0 -> 158.6, 181.8 -> 174.5, 251.9 -> 245.2.
constexpr int kAheadTiles = 8;
template <int DIM, int ORD, class P, bool VPHASE, bool MU, bool PF = false>
__global__ void __launch_bounds__(kThreads, (phase_min_blocks<DIM, ORD, P, VPHASE>())) k_phase(const ShotDesc* __restrict__ shots, int nshots,
                                                     long long ntiles, int k, int post) {
    using R = typename P::real;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The descriptor of the tile's shot is staged in shared memory whenever the
    // shot changes, so the ~100 pointers and extents the chunk code reads are
    // shared-memory broadcasts instead of per-warp global loads.
    __shared__ ShotDesc sdesc;
    int cur = -1;
    bool live = false;
    int it_cur = 0;
    R r = (R)1;
    // A CTA's tiles: blockIdx.x, + gridDim.x, ... in the V phase, the same ones
    // from the last back in the T phase, which so starts on what the V phase
    // touched last and finds it in L2, on the SM (and die) that touched it: c1
    // 4040 x 2040 FP32 162 -> 154 us per step on B200, per-cell 201 -> 196, 200^3
    // order 4 444 -> 436, 1640 x 1140 53.9 -> 51.5; grids that fit in L2
    // unchanged, where reversing the order across the CTAs, so that a tile
    // changes its SM, cost them 8 %.
    const long long G = gridDim.x;
    const bool back = !VPHASE && ntiles > G;
    const long long t0 = back ? blockIdx.x + (ntiles - 1 - blockIdx.x) / G * G : blockIdx.x;
    for (long long t = t0; t >= 0 && t < ntiles; t += back ? -G : G) {
        const int si = nshots == 1 ? 0 : locate_shot(shots, nshots, t);
        if (si != cur) {                      // uniform across the CTA
            __syncthreads();
            const long long* src = reinterpret_cast<const long long*>(shots + si);
            long long* dst = reinterpret_cast<long long*>(&sdesc);
            for (int w = threadIdx.x; w < (int)(sizeof(ShotDesc) / 8); w += blockDim.x) dst[w] = src[w];
            __syncthreads();
            cur = si;
            if constexpr (step_once_per_shot<P>()) {
                // the step index and the COMP16 rescale are fixed for the
                // whole launch: read them once per shot, not once per tile
                const int it = *sdesc.step_base + k;
                it_cur = it;
                live = !sdesc.done && it < sdesc.nt;
                if constexpr (P::prec == BP_PREC_COMP16) r = live ? sdesc.rtab[it] : 1.0f;
            }
        }
        const ShotDesc& S = sdesc;
        if constexpr (step_once_per_shot<P>()) {
            if (!live) continue;
        } else {
            const int it = *S.step_base + k;
            if (S.done || it >= S.nt) continue;
            it_cur = it;
            if constexpr (P::prec == BP_PREC_COMP16) r = S.rtab[it];
        }
        if constexpr (PF) {
            const long long tn = back ? t - G : t + G;
            if (tn >= S.tile0 && tn < ntiles) flat_prefetch<DIM>(S, (int)(tn - S.tile0), warp, lane);
        }
        flat_units<DIM, ORD, P, VPHASE, MU, true>(S, (int)(t - S.tile0), warp, lane, r, it_cur, post);
    }
}

// The phase of a single shot: its descriptor is a kernel parameter, so the
// pointers and extents are constant-bank operands where k_phase loads them from
// shared memory for every use, and a launch starts on its step counter instead
// of on the descriptor.  Measured on B200, us per step, k_phase -> this: 4040 x
// 2040 FP32 147.3 -> 144.3, order 4 155.7 -> 151.6, CBF16 186.4 -> 180.3 (over 8000
// steps), FP64 408 -> 398; 3041 x 1547 order 4 CBF16 137 -> 129; 200^3 order 4 435 -> 427; 424 x 424 x
// 328 2743 -> 2690; 192^3 reference rounding 404 -> 387.
template <int DIM, int ORD, class P, bool VPHASE, bool PF>
__global__ void __launch_bounds__(kThreads, (phase_min_blocks<DIM, ORD, P, VPHASE>()))
    k_phase_one(const __grid_constant__ ShotDesc S, int ntiles, int k, int post) {
    using R = typename P::real;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int it = *S.step_base + k;
    if (S.done || it >= S.nt) return;
    R r = (R)1;
    if constexpr (P::prec == BP_PREC_COMP16) r = S.rtab[it];
    const int G = gridDim.x;
    const bool back = !VPHASE && ntiles > G;           // tile order as in k_phase
    const int t0 = back ? blockIdx.x + (ntiles - 1 - (int)blockIdx.x) / G * G : blockIdx.x;
    for (int t = t0; t >= 0 && t < ntiles; t += back ? -G : G) {
        if constexpr (PF) {
            const int tn = back ? t - G : t + G;
            if (tn >= 0 && tn < ntiles) flat_prefetch<DIM>(S, tn, warp, lane);
        }
        flat_units<DIM, ORD, P, VPHASE, false, true>(S, t, warp, lane, r, it, post);
    }
}

// ---------------------------------------------------------------------------
// Post-step kernel: records the five seismogram components of step it at the
// unique receiver cells, then injects the source sample of step it+1 (the
// reference's Source kernel runs at the top of the next step, so the order
// record(it) -> inject(it+1) -> FD_V(it+1) is unchanged).  The thread that
// records the source cell, if any, injects after its own reads; otherwise
// thread 0 of the shot's first block does.
template <class P>
__global__ void k_post(const ShotDesc* __restrict__ shots, int k, int do_record) {
    const ShotDesc& S = shots[blockIdx.y];
    const int it = *S.step_base + k;
    if (S.done || it >= S.nt) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (do_record && r < S.nrec) record<P>(S, it, r, S.rec_idx[r]);
    const bool owner = (S.src_rec >= 0) ? (r == S.src_rec) : (blockIdx.x == 0 && threadIdx.x == 0);
    if (owner) inject<P>(S, it + 1);
}


// Injection of step it = *step_base + k alone (before the first step).
template <class P>
__global__ void k_inject(const ShotDesc* __restrict__ shots, int nshots, int k) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nshots) return;
    const ShotDesc& S = shots[s];
    if (S.done) return;
    inject<P>(S, *S.step_base + k);
}

// Advances the per-shot step base by n after a chunk of n steps.
__global__ void k_advance(const ShotDesc* __restrict__ shots, int nshots, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nshots) return;
    const ShotDesc& S = shots[s];
    if (S.done) return;
    int v = *S.step_base + n;
    *S.step_base = v > S.nt ? S.nt : v;
}

// Snapshot: copies field f (physical units) of one shot, either the x-z slice
// at y = sy or the whole padded volume, into a dense float array.
template <class P>
__global__ void k_snapshot(const ShotDesc* __restrict__ shots, int shot, int f, int slice_y, float* out, int it) {
    using R = typename P::real;
    const ShotDesc& S = shots[shot];
    const long long n = slice_y >= 0 ? (long long)S.nx * S.nz : (long long)S.nx * S.ny * S.nz;
    R sc = (R)1;
    if constexpr (P::prec == BP_PREC_COMP16) {
        const bool vel = f <= BP_F_VWZ;
        sc = (vel ? S.out_vel : S.out_stress) / S.dyn[it];
    }
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        int x = (int)(q % S.nx);
        long long rest = q / S.nx;
        int y, z;
        if (slice_y >= 0) { y = slice_y; z = (int)rest; }
        else { y = (int)(rest % S.ny); z = (int)(rest / S.ny); }
        const long long i = x + (long long)y * S.pitch + (long long)z * S.plane;
        out[q] = (float)(P::ld1(S.f[f], S.flo[f], i) * sc);
    }
}

// Full-field read in double precision (physical units) for bp_get_field*.
template <class P>
__global__ void k_field_f64(const ShotDesc* __restrict__ shots, int f, double* out) {
    const ShotDesc& S = shots[0];
    const long long n = (long long)S.nx * S.ny * S.nz;
    double sc = 1.0;
    if constexpr (P::prec == BP_PREC_COMP16) {
        const int it = *S.step_base;
        const int itc = it > 0 ? it - 1 : 0;
        sc = (double)((f <= BP_F_VWZ ? S.out_vel : S.out_stress) / S.dyn[itc < S.nt ? itc : S.nt - 1]);
    }
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        int x = (int)(q % S.nx);
        long long rest = q / S.nx;
        int y = (int)(rest % S.ny), z = (int)(rest / S.ny);
        const long long i = x + (long long)y * S.pitch + (long long)z * S.plane;
        out[q] = (double)P::ld1(S.f[f], S.flo[f], i) * sc;
    }
}

// Coefficient read-back (decoded to float) over the dense padded grid.
template <class P>
__global__ void k_coef(const ShotDesc* __restrict__ shots, int which, float* out) {
    const ShotDesc& S = shots[0];
    const void* p = which < VC_COUNT ? S.vc[which] : S.tc[which - VC_COUNT];
    const int8_t* lo = which < VC_COUNT ? S.vclo[which] : S.tclo[which - VC_COUNT];
    const long long n = (long long)S.nx * S.ny * S.nz;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        int x = (int)(q % S.nx);
        long long rest = q / S.nx;
        int y = (int)(rest % S.ny), z = (int)(rest / S.ny);
        out[q] = p ? (float)P::ld1(p, lo, x + (long long)y * S.pitch + (long long)z * S.plane) : 0.0f;
    }
}

// ---------------------------------------------------------------------------
// Host-side launchers (explicit instantiation over dim x order x precision).

// Shared-memory carveout of the phase kernels, in percent of the SM's unified
// L1/shared storage (their only shared data is the shot descriptor; the rest
// serves as L1 for the neighbour re-reads); -1 leaves the driver's choice.
#ifndef BP_L1_CARVEOUT
#define BP_L1_CARVEOUT -1
#endif
template <int D, int O, class P, bool V, bool M>
static void phase_carveout() {
    if constexpr (BP_L1_CARVEOUT >= 0) {
        static bool set = false;                       // once per kernel
        if (!set) {
            cudaFuncSetAttribute(k_phase<D, O, P, V, M>, cudaFuncAttributePreferredSharedMemoryCarveout, BP_L1_CARVEOUT);
            set = true;
        }
    }
}

// One shot (its descriptor on the host) at a tile shape of at most one unit a warp.
template <class P, bool PF = false>
static cudaError_t launch_one(int dim, int order, bool v, const ShotDesc& S, int ntiles, int k, int grid, cudaStream_t st,
                              int post) {
#define BPK_ONE(D, O)                                                                                         \
    if (dim == D && order == O) {                                                                             \
        if (v) k_phase_one<D, O, P, true, PF><<<grid, kThreads, 0, st>>>(S, ntiles, k, 0);                    \
        else k_phase_one<D, O, P, false, PF><<<grid, kThreads, 0, st>>>(S, ntiles, k, post);                  \
        return cudaGetLastError();                                                                            \
    }
    if constexpr (std::is_same_v<P, PolF32>) {     // 2D only with the prefetch, 3D order 4 only without
        BPK_ONE(3, 2)
        if constexpr (PF) { BPK_ONE(2, 2) BPK_ONE(2, 4) }
        else { BPK_ONE(3, 4) }
    } else if constexpr (P::graded) {
        BPK_ONE(2, 2) BPK_ONE(3, 2)
    } else {
        BPK_ONE(2, 2) BPK_ONE(2, 4) BPK_ONE(3, 2) BPK_ONE(3, 4)
    }
#undef BPK_ONE
    return cudaErrorInvalidValue;
}

template <class P>
struct Launch {
    static cudaError_t phase(int dim, int order, bool v, const ShotDesc* d_shots, int nshots, long long ntiles,
                             int k, int grid, cudaStream_t st, int post, bool multi) {
#define BPK_LAUNCH(D, O)                                                                                        \
    if (dim == D && order == O) {                                                                               \
        if (multi) {                                                                                            \
            if (v) { phase_carveout<D, O, P, true, true>();                                                     \
                     k_phase<D, O, P, true, true><<<grid, kThreads, 0, st>>>(d_shots, nshots, ntiles, k, 0); }  \
            else { phase_carveout<D, O, P, false, true>();                                                      \
                   k_phase<D, O, P, false, true><<<grid, kThreads, 0, st>>>(d_shots, nshots, ntiles, k, post); } \
        } else {                                                                                                \
            if (v) { phase_carveout<D, O, P, true, false>();                                                    \
                     k_phase<D, O, P, true, false><<<grid, kThreads, 0, st>>>(d_shots, nshots, ntiles, k, 0); } \
            else { phase_carveout<D, O, P, false, false>();                                                     \
                   k_phase<D, O, P, false, false><<<grid, kThreads, 0, st>>>(d_shots, nshots, ntiles, k, post); } \
        }                                                                                                       \
        return cudaGetLastError();                                                                              \
    }
        if constexpr (P::graded) {           // the variable z grid: order 2 only
            BPK_LAUNCH(2, 2) BPK_LAUNCH(3, 2)
        } else if constexpr (P::prec == BP_PREC_COMP16) {   // the others: step_async.cu
            BPK_LAUNCH(3, 4)
        } else {
            BPK_LAUNCH(2, 2) BPK_LAUNCH(2, 4) BPK_LAUNCH(3, 2) BPK_LAUNCH(3, 4)
        }
#undef BPK_LAUNCH
        return cudaErrorInvalidValue;
    }
};

}  // namespace bpk

// C++ entry points used by the host code (sim.cu, batch.cu).
namespace bpk {
// COMP16 phases that take the kernels of step_async.cu: all but 3D order 4,
// whose 37 staged rows (15 KB a warp) leave too few warps on an SM: 240 x 230 x
// 220 per-cell medium 1588 us per step staged, 1434 from the register tiles (140
// x 130 x 120 uniform 262 and 280; B200).
static bool c16_async(int dim, int order) { return dim == 2 || order == 2; }

template <int D, int O>
static cudaError_t launch_ahead(bool v, const ShotDesc* d, int n, long long ntiles, int k, int grid, cudaStream_t st, int post) {
    if (v) k_phase<D, O, PolF32, true, false, true><<<grid, kThreads, 0, st>>>(d, n, ntiles, k, 0);
    else k_phase<D, O, PolF32, false, false, true><<<grid, kThreads, 0, st>>>(d, n, ntiles, k, post);
    return cudaGetLastError();
}
cudaError_t launch_phase(int prec, int dim, int order, bool vphase, const ShotDesc* d_shots, int nshots,
                         long long ntiles, int k, int grid, cudaStream_t st, int post, int rounding, bool multi,
                         bool graded, bool indexed, bool dense, const ShotDesc* one) {
    if (nshots != 1 || multi) one = nullptr;
    if (graded) {
        if (prec != BP_PREC_FP32 || rounding != BP_ROUND_FAST || order != 2) return cudaErrorInvalidValue;
        return one ? launch_one<PolF32G>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post)
                   : Launch<PolF32G>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
    }
    if (prec == BP_PREC_FP32 && rounding == BP_ROUND_REFERENCE)
        return one ? launch_one<PolF32R>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post)
                   : Launch<PolF32R>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
    if (prec == BP_PREC_FP32 && indexed && !multi && ntiles >= (long long)kAheadTiles * grid) {
        if (one && (dim == 2 || order == 2)) return launch_one<PolF32, true>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post);
        if (dim == 2 && order == 2) return launch_ahead<2, 2>(vphase, d_shots, nshots, ntiles, k, grid, st, post);
        if (dim == 2) return launch_ahead<2, 4>(vphase, d_shots, nshots, ntiles, k, grid, st, post);
        if (order == 2) return launch_ahead<3, 2>(vphase, d_shots, nshots, ntiles, k, grid, st, post);
    }
    // 2D FP32 otherwise keeps the staged descriptor: 4040 x 2040 per-cell 195.6 us
    // per step, 198.0 with the parameter; 817 x 1073 19.2 and 19.4
    if (prec == BP_PREC_FP32)
        return one && dim == 3 ? launch_one<PolF32>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post)
                   : Launch<PolF32>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
    if (prec == BP_PREC_COMP16 && c16_async(dim, order))
        return launch_phase_async(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, one, dense);
    // 3D order 4: the V phase spills 200 bytes with the descriptor as a parameter
    // and none without, for the same time (us per step, 296 x 296 x 232 uniform 2630
    // and 2600, per-cell 3053 and 3057; 200 x 190 x 180 787 and 788)
    if (prec == BP_PREC_COMP16)
        return Launch<PolC16>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
    if (prec == BP_PREC_CBF16)
        return one ? launch_one<PolB24>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post)
                   : Launch<PolB24>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
    return one ? launch_one<PolF64>(dim, order, vphase, *one, (int)ntiles, k, grid, st, post)
                   : Launch<PolF64>::phase(dim, order, vphase, d_shots, nshots, ntiles, k, grid, st, post, multi);
}

cudaError_t launch_post(int prec, const ShotDesc* d_shots, int nshots, int max_rec, int k, int do_record,
                        cudaStream_t st) {
    dim3 grid((max_rec + 127) / 128 > 0 ? (max_rec + 127) / 128 : 1, nshots);
    if (prec == BP_PREC_FP32) k_post<PolF32><<<grid, 128, 0, st>>>(d_shots, k, do_record);
    else if (prec == BP_PREC_COMP16) k_post<PolC16><<<grid, 128, 0, st>>>(d_shots, k, do_record);
    else if (prec == BP_PREC_CBF16) k_post<PolB24><<<grid, 128, 0, st>>>(d_shots, k, do_record);
    else k_post<PolF64><<<grid, 128, 0, st>>>(d_shots, k, do_record);
    return cudaGetLastError();
}

cudaError_t launch_inject(int prec, const ShotDesc* d_shots, int nshots, int k, cudaStream_t st) {
    int g = (nshots + 127) / 128;
    if (prec == BP_PREC_FP32) k_inject<PolF32><<<g, 128, 0, st>>>(d_shots, nshots, k);
    else if (prec == BP_PREC_COMP16) k_inject<PolC16><<<g, 128, 0, st>>>(d_shots, nshots, k);
    else if (prec == BP_PREC_CBF16) k_inject<PolB24><<<g, 128, 0, st>>>(d_shots, nshots, k);
    else k_inject<PolF64><<<g, 128, 0, st>>>(d_shots, nshots, k);
    return cudaGetLastError();
}

cudaError_t launch_advance(const ShotDesc* d_shots, int nshots, int n, cudaStream_t st) {
    k_advance<<<(nshots + 127) / 128, 128, 0, st>>>(d_shots, nshots, n);
    return cudaGetLastError();
}

cudaError_t launch_snapshot(int prec, const ShotDesc* d_shots, int shot, int f, int slice_y, float* out, int it,
                            cudaStream_t st) {
    if (prec == BP_PREC_FP32) k_snapshot<PolF32><<<296, 256, 0, st>>>(d_shots, shot, f, slice_y, out, it);
    else if (prec == BP_PREC_COMP16) k_snapshot<PolC16><<<296, 256, 0, st>>>(d_shots, shot, f, slice_y, out, it);
    else if (prec == BP_PREC_CBF16) k_snapshot<PolB24><<<296, 256, 0, st>>>(d_shots, shot, f, slice_y, out, it);
    else k_snapshot<PolF64><<<296, 256, 0, st>>>(d_shots, shot, f, slice_y, out, it);
    return cudaGetLastError();
}

cudaError_t launch_field_f64(int prec, const ShotDesc* d_shots, int f, double* out, cudaStream_t st) {
    if (prec == BP_PREC_FP32) k_field_f64<PolF32><<<296, 256, 0, st>>>(d_shots, f, out);
    else if (prec == BP_PREC_COMP16) k_field_f64<PolC16><<<296, 256, 0, st>>>(d_shots, f, out);
    else if (prec == BP_PREC_CBF16) k_field_f64<PolB24><<<296, 256, 0, st>>>(d_shots, f, out);
    else k_field_f64<PolF64><<<296, 256, 0, st>>>(d_shots, f, out);
    return cudaGetLastError();
}

int phase_occupancy(int prec, int dim, int order, bool vphase, int rounding, bool dense) {
    int n = 0;
    const void* fn = nullptr;
#define BPK_FN(PP, D, O)                                                                   \
    if (dim == D && order == O)                                                            \
        fn = vphase ? (const void*)k_phase<D, O, PP, true, false> : (const void*)k_phase<D, O, PP, false, false>;
    if (prec == BP_PREC_FP32 && rounding == BP_ROUND_REFERENCE) {
        BPK_FN(PolF32R, 2, 2) BPK_FN(PolF32R, 2, 4) BPK_FN(PolF32R, 3, 2) BPK_FN(PolF32R, 3, 4)
    } else if (prec == BP_PREC_FP32) { BPK_FN(PolF32, 2, 2) BPK_FN(PolF32, 2, 4) BPK_FN(PolF32, 3, 2) BPK_FN(PolF32, 3, 4) }
    else if (prec == BP_PREC_COMP16 && c16_async(dim, order)) return phase_async_occupancy(dim, order, vphase, dense);
    else if (prec == BP_PREC_COMP16) { BPK_FN(PolC16, 3, 4) }
    else if (prec == BP_PREC_CBF16) { BPK_FN(PolB24, 2, 2) BPK_FN(PolB24, 2, 4) BPK_FN(PolB24, 3, 2) BPK_FN(PolB24, 3, 4) }
    else { BPK_FN(PolF64, 2, 2) BPK_FN(PolF64, 2, 4) BPK_FN(PolF64, 3, 2) BPK_FN(PolF64, 3, 4) }
#undef BPK_FN
    if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, 0) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

cudaError_t launch_coef(int prec, const ShotDesc* d_shots, int which, float* out, cudaStream_t st) {
    if (prec == BP_PREC_FP32) k_coef<PolF32><<<296, 256, 0, st>>>(d_shots, which, out);
    else if (prec == BP_PREC_COMP16) k_coef<PolC16><<<296, 256, 0, st>>>(d_shots, which, out);
    else if (prec == BP_PREC_CBF16) k_coef<PolB24><<<296, 256, 0, st>>>(d_shots, which, out);
    else k_coef<PolF64><<<296, 256, 0, st>>>(d_shots, which, out);
    return cudaGetLastError();
}

int phase_threads() { return kThreads; }

static int ilog2(int v) {
    int l = 0;
    while ((1 << (l + 1)) <= v) l++;
    return l;
}
static bool pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

// Chunks per row of the flat tiling, n for a row without gaps.  Rows that start
// on 64-byte boundaries of the field arrays (FP32: 128-byte lines where that
// adds at most 6 % of empty chunks) keep a warp's pieces of two rows from
// sharing the memory's fetch unit with other warps: 296 x 296 x 232 with a
// per-cell medium reads 3.03 GB in the V phase without gaps, 2.57 GB with 80
// chunks for 74, and takes 1435 -> 1190 (76) or 1267 (80) us per step; CBF16
// there 1690 -> 1374, COMP16 1323 -> 1287 (uniform, 80).  Gaps above 9 % cost
// more than they save (CBF16 140 x 130 x 120, 35 chunks: 208 us without, 228 at
// 40).  2D COMP16, bound by its codec's instructions, takes none (4040 x 2040:
// 222 us without, 227 with).
static int row_chunks(int n, int dim, int prec) {
    const int a64 = prec == BP_PREC_FP64 ? 2 : prec == BP_PREC_FP32 ? 4 : 8;
    auto up = [&](int a) { return (n + a - 1) / a * a; };
    if (prec == BP_PREC_FP32 && (up(2 * a64) - n) * 100 <= 6 * n) return up(2 * a64);
    if ((dim == 3 || prec != BP_PREC_COMP16) && (up(a64) - n) * 100 <= 9 * n) return up(a64);
    return n;
}

// Reciprocal of d >= 1 for div_magic: p = 31 + ceil(log2 d), m = ceil(2^p / d)
// < 2^32, and n m >> p = n / d for every 0 <= n < 2^31.
static void magic_of(int d, unsigned& m, int& s) {
    s = 31;
    while ((1LL << (s - 31)) < d) s++;
    m = (unsigned)(((1ULL << s) + d - 1) / d);
}

TileShape default_tile_shape(int dim, int prec) {
    TileShape t;
    t.rows = kWarps;
    t.segs = 1;
    t.tz = dim == 3 ? tile_tz(prec) : 1;
    return t;
}

bool valid_tile_shape(int dim, const TileShape& t) {
    if (!pow2(t.rows) || t.rows < 4 || t.rows > 32 || !pow2(t.segs) || t.segs > 4) return false;
    if (dim == 3 && t.tz != 0 && (!pow2(t.tz) || t.tz > t.rows)) return false;
    return true;
}

long long apply_tile_shape(ShotDesc& S, int dim, int prec, TileShape t) {
    if (dim == 3 && t.tz == 0) t.tz = tile_tz(prec) < t.rows ? tile_tz(prec) : t.rows;
    if (dim == 2) t.tz = 1;
    S.tile_lr = ilog2(t.rows);
    S.tile_ls = ilog2(t.segs);
    S.tile_ltz = ilog2(t.tz);
    S.nseg_t = (S.nseg + t.segs - 1) / t.segs;
    const int ty = dim == 3 ? t.rows / t.tz : 1;
    S.nyb = dim == 3 ? (S.ny + ty - 1) / ty : 1;
    const long long blocks = dim == 3 ? (long long)S.nyb * ((S.nz + t.tz - 1) / t.tz) : (S.nrows + t.rows - 1) / t.rows;
    S.cpr = row_chunks((S.nx + 3) / 4, dim, prec);
    magic_of(S.cpr, S.cpr_m, S.cpr_s);
    magic_of(S.nyb, S.nyb_m, S.nyb_s);
    S.nchunk_f = (int)(blocks * S.cpr);
    return (blocks * S.cpr + 32LL * t.segs - 1) / (32LL * t.segs);
}
int seg_cells() { return kSegCells; }
}  // namespace bpk
