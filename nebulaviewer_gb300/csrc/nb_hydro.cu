// One RK2 stage of the isothermal-Euler update: MUSCL reconstruction (minmod / van Leer /
// MC) + HLL or Rusanov face flux, unsplit x->y->z divergence, wind and jet sources, the
// convex RK combination a*U0 + b*(U + dt*dU), density floor and velocity cap.
//
// Follows nebula3d.py:76-151 (hydro_stage, Rusanov) and sim.py:423-498 (hydro_stage_hll)
// with the face fluxes of nebula3d.py:54-72 / sim.py:397-420.  In the exact build every float
// operation is the reference's, in the reference's order (-fmad=false), so a stage is
// bit-identical to the float32 oracle; the fast build contracts a*b+c, holds two cells in every
// paired FP32 register and shares one approximate reciprocal per density.
//
// GB300 layout: a block owns a 32 (k) x TJ (j) column of cells and marches along i over an
// i-chunk.  Each (j,k) plane tile with a 2-cell halo is brought into shared memory by TMA (five
// 3-D tiled loads: rho, mx, my, mz, xi; mbarrier-tracked, bounded waits).  One raw slot: plane
// p+1 is requested as soon as plane p has been converted, and lands while plane p's faces and
// update are computed.  A plane is converted once to primitives (rho, u, v, w) and (c^2, c) in
// shared memory; every face flux is evaluated once (the reference evaluates each face twice).
// The two builds' tiles differ from there: nb_hydro_pair.cuh (fast), nb_hydro_exact.cuh (exact).
// Sources: the wind loop over the active stars in ionized cells, the jet loop over the tile's list
// of stars whose jet can reach it.  Stage 2 also reduces the CFL max speed of the new state
// (nebula3d.py:154-162) into one atomic.
#include <cmath>
#include <type_traits>

#include "nb_internal.cuh"

namespace {

constexpr int TK = 32;            // cells per tile along k (one warp)
constexpr int RAWW = 40;          // raw tile width along k: [k0-4, k0+36), 16-byte aligned start

template <int LIM>
__device__ __forceinline__ float slope_lim(float a, float b) {
    if (a * b <= 0.0f) return 0.0f;
    if (LIM == 2) {                                           // sim.py:366-372 mc_lim
        float s = a > 0.0f ? 1.0f : -1.0f;
        return s * fminr(fminr(2.0f * fabsf(a), 2.0f * fabsf(b)), 0.5f * fabsf(a + b));
    }
    if (LIM == 1) return 2.0f * a * b / (a + b);              // sim.py:375-380 vl_lim
    if (fabsf(a) < fabsf(b)) return a;                        // nebula3d.py:40-46 minmod
    return b;
}

// Where a tile lies: its first column, row and plane, and the end of its i-chunk.
struct HydroTile {
    int k0, j0, i0, i_end;
    __device__ __forceinline__ HydroTile(const HydroLaunch& L, int tile, int nx, int tj) {
        int kt, jt, ci;
        if (L.order == 0) {                       // sweep order 0: k tiles fastest, then j, then i-chunks
            kt = tile % L.tiles_k;
            tile /= L.tiles_k;
            jt = tile % L.tiles_j;
            ci = tile / L.tiles_j;
        } else {                                  // sweep order 1: i-chunks fastest, then k, then j
            ci = tile % L.n_chunks;
            tile /= L.n_chunks;
            kt = tile % L.tiles_k;
            jt = tile / L.tiles_k;
        }
        k0 = kt * TK;
        j0 = jt * tj;
        // n_chunks = ceil(nx / chunk_i) chunks of equal depth (within one plane): no short last chunk
        i0 = (int)((long long)ci * nx / L.n_chunks);
        i_end = (int)((long long)(ci + 1) * nx / L.n_chunks);
    }
};

// The stars whose jet (nebula3d.py:131-149: strength > 0, an active star, r < jet_r) can reach
// a cell centre of this tile, in star order, by one warp: the distance from the star to the box of
// the tile's cell centres, less a margin of two cells for the float rounding of the per-cell
// distance, must be below jet_r.  Stars left out add exactly nothing to any cell here.
__device__ __forceinline__ void jet_list(const HydroLaunch& L, const HydroTile& t, int ny, int nz, int tj, float dx,
                                         float jet_r, int nstars, int tk, int* n_jet_p, unsigned char* jet_ix) {
    const float bx0 = ((float)t.i0 + 0.5f) * dx, bx1 = ((float)(t.i_end - 1) + 0.5f) * dx;
    const float by0 = ((float)t.j0 + 0.5f) * dx, by1 = ((float)(min(t.j0 + tj, ny) - 1) + 0.5f) * dx;
    const float bz0 = ((float)t.k0 + 0.5f) * dx, bz1 = ((float)(min(t.k0 + TK, nz) - 1) + 0.5f) * dx;
    const float reach = jet_r + 2.0f * dx;
    int n = 0;
    for (int s0 = 0; s0 < nstars; s0 += 32) {
        const int s = s0 + tk;
        bool keep = false;
        if (s < nstars) {
            const float4 st = L.sw[s].w, jt = L.sw[s].jet;
            if (jt.w > 0.0f && st.w > 0.0f) {
                const float ex = fmaxf(0.0f, fmaxf(bx0 - st.x, st.x - bx1));
                const float ey = fmaxf(0.0f, fmaxf(by0 - st.y, st.y - by1));
                const float ez = fmaxf(0.0f, fmaxf(bz0 - st.z, st.z - bz1));
                keep = !(ex * ex + ey * ey + ez * ez >= reach * reach);    // NaN keeps the star
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) jet_ix[n + __popc(m & ((1u << tk) - 1u))] = (unsigned char)s;
        n += __popc(m);
    }
    if (tk == 0) *n_jet_p = n;
}

// a tile's CFL max speed into its instance (red: one float per warp of shared memory)
__device__ __forceinline__ void hydro_smax(const HydroLaunch& L, float v, float* red, int warps) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxr(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.0f;
        for (int w = 0; w < warps; ++w) m = fmaxr(m, red[w]);
        atomicMax(L.smax_bits, __float_as_uint(m));
    }
}

}  // namespace

#if defined(NB_ARITH_FAST) && NB_ARITH_FAST
#include "nb_hydro_pair.cuh"
#else
#include "nb_hydro_exact.cuh"
#endif

namespace {

// A TMA wait gave up: record it and let the raw slot's copy land (a bounded wait); the block's shared
// memory lives until thread 0 has left.  No barrier: warps may come here a march step apart.
template <int TJ>
__device__ __forceinline__ void hydro_abort(unsigned char* smem, unsigned* status, unsigned ph0, unsigned limit) {
    using SM = HydroSmem<TJ>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SM::FIXED - SM::BAR_BYTES);
    if (threadIdx.x == 0) {                      // the load that may still be in flight
        atomicOr(status, NB_DEV_TMA_TIMEOUT);
        mbar_wait_limited(&bar[0], ph0 & 1u, &limit);
    }
}

// the barriers, and the block's work rotation (hydro_tile) from the slot of its first warp: the
// blocks resident on an SM occupy different groups of 8 slots and so take different rotations
template <int TJ>
__device__ __forceinline__ void hydro_init_bars(unsigned char* smem, int* rot) {
    using SM = HydroSmem<TJ>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SM::FIXED - SM::BAR_BYTES);
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        bar[2] = 0;                              // no wait has given up
        fence_mbar_init();
        *rot = (int)((warp_slot() >> 3) * HYDRO_ROT_STEP & 3u);
    }
    __syncthreads();
}

template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32>
__global__ void __launch_bounds__(HYDRO_THREADS, HYDRO_MINB) hydro_stage_kernel(const HydroLaunch L) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int rot;
    hydro_init_bars<TJ>(smem, &rot);
    unsigned ph0 = 0;
    bool failed = false;
    hydro_tile<SOLVER, LIM, TJ, STAGE2, I32>(L, blockIdx.x, smem, ph0, failed, rot);
    if (failed) hydro_abort<TJ>(smem, L.status, ph0, L.wait_limit);
}

// Persistent batched stage: blocks take (instance, tile) work items from a list spanning many
// instances of different sizes, in list order, through one atomic counter (reset by the
// batched control kernel before every step).  A block whose bounded wait gave up computes nothing
// more: it keeps taking items and flags the instance of each one it leaves undone, so every
// instance with an unwritten tile reports NB_DEV_TMA_TIMEOUT.
// records in global memory: their loaded fields need an 80-register budget in the exact build
constexpr int HYDRO_BATCH_MINB = HYDRO_MINB < 3 ? HYDRO_MINB : 3;
template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32>
__global__ void __launch_bounds__(HYDRO_THREADS, HYDRO_BATCH_MINB)
hydro_batch_kernel(const HydroLaunch* __restrict__ Ls, const int2* __restrict__ work, int n_work,
                   unsigned* counter) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int item, rot;
    hydro_init_bars<TJ>(smem, &rot);
    unsigned ph0 = 0;
    bool failed = false;                         // block-uniform (hydro_tile sets it after a barrier)
    const HydroLaunch* last = nullptr;
    for (;;) {
        if (threadIdx.x == 0) item = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int it = item;
        if (it >= n_work) break;
        const int2 w = work[it];
        if (!Ls[w.x].active) {                   // an idle slot of the batch: nothing to do
            __syncthreads();
            continue;
        }
        last = &Ls[w.x];
        hydro_tile<SOLVER, LIM, TJ, STAGE2, I32>(*last, w.y, smem, ph0, failed, rot);
        if (failed) break;
        __syncthreads();
    }
    if (failed && last) {
        hydro_abort<TJ>(smem, last->status, ph0, last->wait_limit);
        // the items this block would still have taken are left undone: flag their instances (the
        // counter grows by one per turn, so the loop ends)
        if (threadIdx.x == 0)
            for (unsigned it; (it = atomicAdd(counter, 1u)) < (unsigned)n_work;)
                atomicOr(Ls[work[it].x].status, NB_DEV_TMA_TIMEOUT);
    }
}

// The same persistent stage with the stage records in the kernel parameter (batches of at most
// NB_BATCH_PARAM_MAX instances, 32-bit offsets): a record's fields come from the constant bank,
// as the single-instance kernel's do, so it fits the same registers and blocks / SM.  The active flags
// (changed between graph replays) and the status words are read from the device copy Lg.
template <int SOLVER, int LIM, int TJ, bool STAGE2>
__global__ void __launch_bounds__(HYDRO_THREADS, HYDRO_MINB)
hydro_batch_param_kernel(const __grid_constant__ NbBatchRecords R, const HydroLaunch* __restrict__ Lg,
                         const int2* __restrict__ work, int n_work, unsigned* counter) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int item, rot;
    hydro_init_bars<TJ>(smem, &rot);
    unsigned ph0 = 0;
    bool failed = false;                         // block-uniform (hydro_tile sets it after a barrier)
    int last = -1;
    for (;;) {
        if (threadIdx.x == 0) item = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int it = item;
        if (it >= n_work) break;
        const int2 w = work[it];
        if (!Lg[w.x].active) {                   // an idle slot of the batch: nothing to do
            __syncthreads();
            continue;
        }
        last = w.x;
        hydro_tile<SOLVER, LIM, TJ, STAGE2, true>(R.L[w.x], w.y, smem, ph0, failed, rot);
        if (failed) break;
        __syncthreads();
    }
    if (failed && last >= 0) {
        hydro_abort<TJ>(smem, Lg[last].status, ph0, Lg[last].wait_limit);
        if (threadIdx.x == 0)                    // flag the instances of the items left undone
            for (unsigned it; (it = atomicAdd(counter, 1u)) < (unsigned)n_work;)
                atomicOr(Lg[work[it].x].status, NB_DEV_TMA_TIMEOUT);
    }
}

template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32>
cudaError_t run_kernel(const HydroLaunch& L, cudaStream_t s) {
    auto kern = hydro_stage_kernel<SOLVER, LIM, TJ, STAGE2, I32>;
    const int smem = HydroSmem<TJ>::bytes(L.nstars_host);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)                        // the largest shared-memory carveout: 2 blocks of 112 KB (fast), 4 of 57 (exact) per SM
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    const int blocks = L.tiles_k * L.tiles_j * L.n_chunks;
    kern<<<blocks, HYDRO_THREADS, smem, s>>>(L);
    return cudaGetLastError();
}

template <int SOLVER, int LIM, int TJ>
cudaError_t run_stage(const HydroLaunch& L, cudaStream_t s) {
    const bool s2 = L.smax_bits || L.u0[0] != L.in[0];
    if (L.idx32) return s2 ? run_kernel<SOLVER, LIM, TJ, true, true>(L, s) : run_kernel<SOLVER, LIM, TJ, false, true>(L, s);
    return s2 ? run_kernel<SOLVER, LIM, TJ, true, false>(L, s) : run_kernel<SOLVER, LIM, TJ, false, false>(L, s);
}

template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32>
cudaError_t run_batch_kernel(const HydroLaunch* Ls, const NbBatchRecords* rec, const int2* work, int n_work,
                             unsigned* counter, int max_stars, int grid, cudaStream_t s) {
    const int smem = HydroSmem<TJ>::bytes(max_stars);
    if (I32 && rec) {
        auto kern = hydro_batch_param_kernel<SOLVER, LIM, TJ, STAGE2>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        kern<<<grid, HYDRO_THREADS, smem, s>>>(*rec, Ls, work, n_work, counter);
        return cudaGetLastError();
    }
    auto kern = hydro_batch_kernel<SOLVER, LIM, TJ, STAGE2, I32>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    kern<<<grid, HYDRO_THREADS, smem, s>>>(Ls, work, n_work, counter);
    return cudaGetLastError();
}

template <int SOLVER, int LIM, int TJ>
cudaError_t run_batch(const HydroLaunch* Ls, const NbBatchRecords* rec, const int2* work, int n_work,
                      unsigned* counter, int max_stars, int stage2, int idx32, int grid, cudaStream_t s) {
    if (idx32)
        return stage2 ? run_batch_kernel<SOLVER, LIM, TJ, true, true>(Ls, rec, work, n_work, counter, max_stars, grid, s)
                      : run_batch_kernel<SOLVER, LIM, TJ, false, true>(Ls, rec, work, n_work, counter, max_stars, grid, s);
    return stage2 ? run_batch_kernel<SOLVER, LIM, TJ, true, false>(Ls, nullptr, work, n_work, counter, max_stars, grid, s)
                  : run_batch_kernel<SOLVER, LIM, TJ, false, false>(Ls, nullptr, work, n_work, counter, max_stars, grid, s);
}

}  // namespace

int nb_hydro_tile_j() { return HYDRO_TJ; }

// The i-chunk depth of a stage alone on the GPU: blocks = columns x chunks run in rounds of `sms` x
// HYDRO_MINB, each of the depth's planes and four halo planes (and about half a plane to start); a
// last round with fewer blocks on an SM has cheaper planes.  The blocks are as long as one another but
// for the winds and jets: `sources` stars with one add HYDRO_WIND of a plane each where a warp has an
// ionized cell or one in a jet's reach, and that gas may fill one block and miss the next, so a block's
// share of it is time at the end that no other block fills.  The least time over all chunk counts.
// With a fixed depth of 20 a small grid left SMs idle for 24 serial planes and the last round was
// often nearly empty: stages 1 + 2 (fast) at 64^3 76 -> 33 us, 128^3 96 -> 88, 192^3 251 -> 235,
// 256^3 523 -> 502 (depths 4, 15, 48, 37).  Without the winds in it the rule gave one chunk a column at
// 384^3 for any stars, and the GPU then waited for the few columns in the ionized gas: stages 1 + 2 there
// with 6 / 24 / 64 / 256 stars 1657 / 2100 / 3429 / 11557 -> 1625 / 1662 / 1814 / 3287 us (depths 96, 35,
// 24, 12), at 256^3 with 256 stars 2046 -> 1301 (37 -> 8); exact build, 256^3, 24 stars 1219 -> 1167.
// Eight stars with jets and no winds, 200^3: 419 -> 336 us (67 -> 20).
int nb_hydro_depth(int nx, long long columns, int sms, int sources) {
    int best = nx;
    double least = 0.0;
    for (int n = 1, last = 0; n <= nx; ++n) {
        const int depth = (nx + n - 1) / n;
        if (depth == last) continue;                       // the same depth with fewer chunks came before
        last = depth;
        const long long blocks = columns * ((nx + depth - 1) / depth), round = (long long)sms * HYDRO_MINB;
        const long long rest = blocks % round;
        const double t = ((double)(blocks / round) + HYDRO_PLANE[(rest + sms - 1) / sms]) * (depth + 4.5) +
                         HYDRO_WIND * sources * depth;
        if (least == 0.0 || t < least) {
            least = t;
            best = depth;
        }
        if (depth == 1) break;
    }
    return best;
}

// The depth of a batch's stages, whose persistent blocks (`slots` of them) take tiles in turn: deep
// chunks convert fewer halo planes (4.5 per chunk), shallow ones end together (half a chunk idle at the
// end, and a chunk's wind work, as above); the sum is least at the depth whose square is 9 planes' worth
// of each block's share, less by the instance's own sources (a batch step of seven 128^3 with one star and a
// 96^3 with 256 stars 2438 -> 1243 us; 1413 with the most windy instance's depth for all).
int nb_hydro_depth_batch(double column_planes, int slots, int sources) {
    const double d = std::sqrt(9.0 * column_planes / (slots > 0 ? slots : 1) / (1.0 + 2.0 * HYDRO_WIND * sources));
    return d < 2.0 ? 2 : (d > 128.0 ? 128 : (int)d);
}

int nb_hydro_idx32(long long ncell) { return ncell <= HYDRO_IDX32_CELLS; }

// resident blocks per SM of the persistent stage kernel (sizes its grid)
int nb_hydro_batch_blocks_per_sm(int solver, int limiter, int max_stars, int idx32, int params) {
    constexpr int TJ = HYDRO_TJ;
    const int smem = HydroSmem<TJ>::bytes(max_stars);
    auto occ = [&](auto kern) {
        int n = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, HYDRO_THREADS, smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n;
    };
    int n;
    if (idx32 && params) {
        if (solver == NB_SOLVER_RUSANOV)
            n = occ(hydro_batch_param_kernel<NB_SOLVER_RUSANOV, 0, TJ, true>);
        else if (limiter == NB_LIM_VANLEER)
            n = occ(hydro_batch_param_kernel<NB_SOLVER_HLL, NB_LIM_VANLEER, TJ, true>);
        else if (limiter == NB_LIM_MC)
            n = occ(hydro_batch_param_kernel<NB_SOLVER_HLL, NB_LIM_MC, TJ, true>);
        else
            n = occ(hydro_batch_param_kernel<NB_SOLVER_HLL, NB_LIM_MINMOD, TJ, true>);
        return n > 0 ? n : HYDRO_MINB;
    }
    if (solver == NB_SOLVER_RUSANOV)
        n = idx32 ? occ(hydro_batch_kernel<NB_SOLVER_RUSANOV, 0, TJ, true, true>)
                  : occ(hydro_batch_kernel<NB_SOLVER_RUSANOV, 0, TJ, true, false>);
    else if (limiter == NB_LIM_VANLEER)
        n = idx32 ? occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_VANLEER, TJ, true, true>)
                  : occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_VANLEER, TJ, true, false>);
    else if (limiter == NB_LIM_MC)
        n = idx32 ? occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_MC, TJ, true, true>)
                  : occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_MC, TJ, true, false>);
    else
        n = idx32 ? occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_MINMOD, TJ, true, true>)
                  : occ(hydro_batch_kernel<NB_SOLVER_HLL, NB_LIM_MINMOD, TJ, true, false>);
    return n > 0 ? n : HYDRO_BATCH_MINB;
}

cudaError_t nb_launch_hydro(const HydroLaunch& L, int solver, int limiter, cudaStream_t s) {
    constexpr int TJ = HYDRO_TJ;
    if (solver == NB_SOLVER_RUSANOV) return run_stage<NB_SOLVER_RUSANOV, 0, TJ>(L, s);
    switch (limiter) {
        case NB_LIM_VANLEER: return run_stage<NB_SOLVER_HLL, NB_LIM_VANLEER, TJ>(L, s);
        case NB_LIM_MC: return run_stage<NB_SOLVER_HLL, NB_LIM_MC, TJ>(L, s);
        default: return run_stage<NB_SOLVER_HLL, NB_LIM_MINMOD, TJ>(L, s);
    }
}

cudaError_t nb_launch_hydro_batch(const HydroLaunch* Ls, const NbBatchRecords* rec, const int2* work, int n_work,
                                  unsigned* counter, int max_stars, int stage2, int idx32, int solver, int limiter,
                                  int grid, cudaStream_t s) {
    constexpr int TJ = HYDRO_TJ;
    if (solver == NB_SOLVER_RUSANOV)
        return run_batch<NB_SOLVER_RUSANOV, 0, TJ>(Ls, rec, work, n_work, counter, max_stars, stage2, idx32, grid, s);
    switch (limiter) {
        case NB_LIM_VANLEER:
            return run_batch<NB_SOLVER_HLL, NB_LIM_VANLEER, TJ>(Ls, rec, work, n_work, counter, max_stars, stage2, idx32,
                                                                grid, s);
        case NB_LIM_MC:
            return run_batch<NB_SOLVER_HLL, NB_LIM_MC, TJ>(Ls, rec, work, n_work, counter, max_stars, stage2, idx32, grid,
                                                           s);
        default:
            return run_batch<NB_SOLVER_HLL, NB_LIM_MINMOD, TJ>(Ls, rec, work, n_work, counter, max_stars, stage2, idx32,
                                                               grid, s);
    }
}
