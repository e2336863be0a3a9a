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
// 152.  Large 2D order-2 shots of per-cell media wait on their coefficients and
// take 32 warps (DENSE, dense_form in runner.h; indexed media 177 -> 181 by it).  Taking the chunk
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

template <int DIM, int ORD, class P, bool VPHASE>
__global__ void __launch_bounds__(AsyncShape<DIM, ORD, P, VPHASE, false>::NW * 32, (AsyncShape<DIM, ORD, P, VPHASE, false>::MINB))
    k_phase_async(const ShotDesc* __restrict__ shots, int nshots, long long ntiles, int k, int post) {
    using R = typename P::real;
    using Src = typename AsyncShape<DIM, ORD, P, VPHASE, false>::Src;
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
            r = live ? sdesc.rtab[it] : 1.0f;
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
    const R r = S.rtab[it];
    const int G = gridDim.x;
    const bool back = !VPHASE && ntiles > G;
    const int t0 = back ? blockIdx.x + (ntiles - 1 - (int)blockIdx.x) / G * G : blockIdx.x;
    for (int t = t0; t >= 0 && t < ntiles; t += back ? -G : G)
        async_units<DIM, ORD, P, VPHASE>(S, slots + warp * AsyncShape<DIM, ORD, P, VPHASE, DENSE>::Src::kBytes, t, warp, lane, r,
                                         it, post);
}

// The kernels use more dynamic shared memory than a launch may without this
// (set per device, so before every launch that is not a graph replay).
template <class K>
static cudaError_t allow_smem(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
template <int D, int O, class P, bool V, bool DN = false>
static cudaError_t launch_single(const ShotDesc& S, long long ntiles, int k, int grid, cudaStream_t st, int post) {
    using C = AsyncShape<D, O, P, V, DN>;
    cudaError_t e = allow_smem(k_phase_async_one<D, O, P, V, DN>, C::kSmem);
    if (e != cudaSuccess) return e;
    k_phase_async_one<D, O, P, V, DN><<<grid, C::NW * 32, C::kSmem, st>>>(S, (int)ntiles, k, post);
    return cudaGetLastError();
}
template <int D, int O, class P, bool V>
static cudaError_t launch_table(const ShotDesc* d, int nshots, long long ntiles, int k, int grid, cudaStream_t st, int post) {
    using C = AsyncShape<D, O, P, V, false>;
    cudaError_t e = allow_smem(k_phase_async<D, O, P, V>, C::kSmem);
    if (e != cudaSuccess) return e;
    k_phase_async<D, O, P, V><<<grid, C::NW * 32, C::kSmem, st>>>(d, nshots, ntiles, k, post);
    return cudaGetLastError();
}
template <class K>
static int occupancy_a(K kernel, int threads, int bytes) {
    int n = 0;
    if (allow_smem(kernel, bytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, bytes) != cudaSuccess)
        return 1;
    return n > 0 ? n : 1;
}

#define BPK_EACH(X) X(2, 2) X(2, 4) X(3, 2)
// dense: the shape for per-cell media, 2D order-2 single shots only
cudaError_t launch_phase_async(int dim, int order, bool v, const ShotDesc* d, int nshots, long long ntiles, int k,
                               int grid, cudaStream_t st, int post, const ShotDesc* one, bool dense) {
    if (dense) {
        if (dim != 2 || order != 2 || !one) return cudaErrorInvalidValue;
        return v ? launch_single<2, 2, PolC16, true, true>(*one, ntiles, k, grid, st, 0)
                 : launch_single<2, 2, PolC16, false, true>(*one, ntiles, k, grid, st, post);
    }
#define BPK_LAUNCH(D, O)                                                                                            \
    if (dim == D && order == O) {                                                                                   \
        if (one) return v ? launch_single<D, O, PolC16, true>(*one, ntiles, k, grid, st, 0)                         \
                          : launch_single<D, O, PolC16, false>(*one, ntiles, k, grid, st, post);                    \
        return v ? launch_table<D, O, PolC16, true>(d, nshots, ntiles, k, grid, st, 0)                              \
                 : launch_table<D, O, PolC16, false>(d, nshots, ntiles, k, grid, st, post);                         \
    }
    BPK_EACH(BPK_LAUNCH)
#undef BPK_LAUNCH
    return cudaErrorInvalidValue;
}
int phase_async_occupancy(int dim, int order, bool v, bool dense) {
#define BPK_OCC(KERNEL, D, O, V, DN) occupancy_a(KERNEL, AsyncShape<D, O, PolC16, V, DN>::NW * 32, AsyncShape<D, O, PolC16, V, DN>::kSmem)
    if (dense && dim == 2 && order == 2)
        return v ? BPK_OCC((k_phase_async_one<2, 2, PolC16, true, true>), 2, 2, true, true)
                 : BPK_OCC((k_phase_async_one<2, 2, PolC16, false, true>), 2, 2, false, true);
#define BPK_EACH_OCC(D, O)                                                                                          \
    if (dim == D && order == O)                                                                                     \
        return v ? BPK_OCC((k_phase_async<D, O, PolC16, true>), D, O, true, false)                                  \
                 : BPK_OCC((k_phase_async<D, O, PolC16, false>), D, O, false, false);
    BPK_EACH(BPK_EACH_OCC)
#undef BPK_EACH_OCC
#undef BPK_OCC
    return 1;
}
}  // namespace bpk
