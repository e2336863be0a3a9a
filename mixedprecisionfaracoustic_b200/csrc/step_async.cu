// step_async.cu - the COMP16 phase kernels: a unit's field rows come into the
// warp's own shared memory by asynchronous copies, all started before the first
// is waited for.
//
// Reference kernels replaced: FD_V (Half/main.cu:156-268), FD_T (:270-371).
//
// COMP16 holds two arrays a field and decodes every value it loads, so a chunk
// that loads into registers needs 2-4 times FP32's: the register tile kernels
// spilled 250-1100 bytes a thread in 2D and took their chunks one output at a
// time in 3D, waiting for each output's loads.  Here the copies hold no
// registers, a unit waits once, and the values are decoded as they are used.
// Warps are independent: a warp fills its slots, waits for its own copies and
// works; other resident warps cover the wait.
#include "async.cuh"

namespace bpk {

// Warps per CTA and CTAs per SM: 24 warps at 80 registers in 2D, 16 at 128 in
// 3D, where 24 spill.  Measured on B200 (us per step, register tiles -> staged):
// 4040 x 2040 order 2 254.5 -> 222, order 4 343 -> 310 (2 CTAs: 233 and 319; 4:
// 280 and more); 817 x 1073 41.5 -> 34.2; 296 x 296 x 232 uniform 2075 -> 1287 (3
// CTAs: 2640), per-cell medium 2545 -> 1940; 140 x 130 x 120 228 -> 172.  With the
// descriptor as a parameter and the four-value codec: 177, 227, 27, 980, 1620 and
// 152.  Large 2D order-2 launches of per-cell media wait on their coefficients and
// take 32 warps (DENSE, indexed_form in runner.h; indexed media 177 -> 181 by it).  Taking the chunk
// one output at a time (as the register tiles do in 3D) costs 10-35 % here, and
// copies of the next unit under way while one is worked on cost occupancy: 50 %
// slower.
template <int DIM, int ORD, class P, bool VPHASE, bool DENSE>
struct AsyncShape {
    using Src = AsyncSrc<DIM, ORD, P, VPHASE>;
    static constexpr int NW = 8, MINB = DIM == 2 ? (DENSE ? 4 : 3) : 2, kSmem = NW * Src::kBytes;
};

// Waits for this thread's copies.
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The units of tile lt this warp takes.
template <int DIM, int ORD, class P, bool VPHASE>
__device__ __forceinline__ void async_units(const ShotDesc& S, char* mine, int lt, int warp, int lane,
                                            typename P::real r, int it, int post) {
    using C = AsyncShape<DIM, ORD, P, VPHASE, false>;
    using Src = typename C::Src;
    const int lr = S.tile_lr, units = 1 << (lr + S.tile_ls);
    for (int u = warp; u < units; u += C::NW) {
        const int q = (((lt << S.tile_ls) + (u >> lr)) << 5) + lane;
        int x0, y, z;
        const bool on = flat_cell<DIM>(S, q, u & ((1 << lr) - 1), x0, y, z) && row_updated<DIM, ORD>(S, y, z);
        const cidx c = on ? x0 + y * S.pitch + z * (cidx)S.plane : 0;
        unsigned ids = 0;
        if (on) {
            // every chunk of an updated row, also one whose own cells are
            // not updated: its neighbour lane differences across into it
            Src::fill(S, mine, lane, c, x0);
            if (med_on<P>(S)) ids = med_ids(S, c);
        }
        wait_copies();
        __syncwarp();
        const unsigned mask = on ? chunk_mask<ORD>(S, x0) : 0;
        if (mask) {
            const Src src(mine, lane);
            chunk_work<DIM, ORD, P, VPHASE, false, false>(S, src, c, x0, y, z, r, mask, ids, it, post);
        }
        __syncwarp();                     // every lane has read before the slots are filled again
    }
}

template <int DIM, int ORD, class P, bool VPHASE, bool DENSE>
__global__ void __launch_bounds__(AsyncShape<DIM, ORD, P, VPHASE, DENSE>::NW * 32, (AsyncShape<DIM, ORD, P, VPHASE, DENSE>::MINB))
    k_phase_async(const ShotDesc* __restrict__ shots, int nshots, long long ntiles, int k, int post) {
    using R = typename P::real;
    using C = AsyncShape<DIM, ORD, P, VPHASE, DENSE>;
    using Src = typename C::Src;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ ShotDesc sdesc;
    extern __shared__ __align__(16) char slots[];
    char* const mine = slots + warp * Src::kBytes;
    int cur = -1, it = 0;
    bool live = false;
    R r = (R)1;
    // tiles in the order of k_phase (step.cu): the T phase from the last back
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
            it = *sdesc.step_base + k;
            live = !sdesc.done && it < sdesc.nt;
            if constexpr (P::prec == BP_PREC_COMP16) r = live ? sdesc.rtab[it] : 1.0f;
        }
        if (!live) continue;
        const ShotDesc& S = sdesc;
        async_units<DIM, ORD, P, VPHASE>(S, mine, (int)(t - S.tile0), warp, lane, r, it, post);
    }
}

// The same for a single shot, its descriptor a kernel parameter (k_phase_one).
template <int DIM, int ORD, class P, bool VPHASE, bool DENSE>
__global__ void __launch_bounds__(AsyncShape<DIM, ORD, P, VPHASE, DENSE>::NW * 32, (AsyncShape<DIM, ORD, P, VPHASE, DENSE>::MINB))
    k_phase_async_one(const __grid_constant__ ShotDesc S, int ntiles, int k, int post) {
    using R = typename P::real;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    extern __shared__ __align__(16) char slots[];
    const int it = *S.step_base + k;
    if (S.done || it >= S.nt) return;
    R r = (R)1;
    if constexpr (P::prec == BP_PREC_COMP16) r = S.rtab[it];
    const int G = gridDim.x;
    const bool back = !VPHASE && ntiles > G;
    const int t0 = back ? blockIdx.x + (ntiles - 1 - (int)blockIdx.x) / G * G : blockIdx.x;
    for (int t = t0; t >= 0 && t < ntiles; t += back ? -G : G)
        async_units<DIM, ORD, P, VPHASE>(S, slots + warp * AsyncShape<DIM, ORD, P, VPHASE, DENSE>::Src::kBytes, t, warp, lane, r,
                                         it, post);
}

// The kernels use more dynamic shared memory than a launch may without this
// (set per device, so before every launch that is not a graph replay).
template <int D, int O, class P, bool V, bool DN>
static cudaError_t allow_smem() {
    cudaError_t e = cudaFuncSetAttribute(k_phase_async_one<D, O, P, V, DN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         AsyncShape<D, O, P, V, DN>::kSmem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(k_phase_async<D, O, P, V, DN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                AsyncShape<D, O, P, V, DN>::kSmem);
}
template <int D, int O, class P, bool V, bool DN>
static cudaError_t launch_a(const ShotDesc* d, int nshots, long long ntiles, int k, int grid, cudaStream_t st, int post,
                            const ShotDesc* one) {
    using C = AsyncShape<D, O, P, V, DN>;
    cudaError_t e = allow_smem<D, O, P, V, DN>();
    if (e != cudaSuccess) return e;
    if (one) k_phase_async_one<D, O, P, V, DN><<<grid, C::NW * 32, C::kSmem, st>>>(*one, (int)ntiles, k, post);
    else k_phase_async<D, O, P, V, DN><<<grid, C::NW * 32, C::kSmem, st>>>(d, nshots, ntiles, k, post);
    return cudaGetLastError();
}
template <int D, int O, class P, bool V, bool DN>
static int occupancy_a() {
    int n = 0;
    if (allow_smem<D, O, P, V, DN>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_phase_async<D, O, P, V, DN>, AsyncShape<D, O, P, V, DN>::NW * 32,
                                                      AsyncShape<D, O, P, V, DN>::kSmem) != cudaSuccess)
        return 1;
    return n > 0 ? n : 1;
}

#define BPK_EACH(X) X(2, 2) X(2, 4) X(3, 2)
cudaError_t launch_phase_async(int dim, int order, bool v, const ShotDesc* d, int nshots, long long ntiles, int k,
                               int grid, cudaStream_t st, int post, const ShotDesc* one, bool indexed) {
#define BPK_LAUNCH(D, O)                                                                                            \
    if (dim == D && order == O) {                                                                                   \
        if (D == 2 && O == 2 && !indexed)                                                                                     \
            return v ? launch_a<D, O, PolC16, true, D == 2 && O == 2>(d, nshots, ntiles, k, grid, st, 0, one)                 \
                     : launch_a<D, O, PolC16, false, D == 2 && O == 2>(d, nshots, ntiles, k, grid, st, post, one);            \
        return v ? launch_a<D, O, PolC16, true, false>(d, nshots, ntiles, k, grid, st, 0, one)                      \
                 : launch_a<D, O, PolC16, false, false>(d, nshots, ntiles, k, grid, st, post, one);                 \
    }
    BPK_EACH(BPK_LAUNCH)
#undef BPK_LAUNCH
    return cudaErrorInvalidValue;
}
int phase_async_occupancy(int dim, int order, bool v, bool indexed) {
#define BPK_OCC(D, O)                                                                                               \
    if (dim == D && order == O) {                                                                                   \
        if (D == 2 && O == 2 && !indexed)                                                                                     \
            return v ? occupancy_a<D, O, PolC16, true, D == 2 && O == 2>() : occupancy_a<D, O, PolC16, false, D == 2 && O == 2>();      \
        return v ? occupancy_a<D, O, PolC16, true, false>() : occupancy_a<D, O, PolC16, false, false>();            \
    }
    BPK_EACH(BPK_OCC)
#undef BPK_OCC
    return 1;
}
}  // namespace bpk
