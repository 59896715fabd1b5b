// The exact build's hydro stage tile: one cell per thread, every float operation the reference's.
//
// A plane is converted once to primitives (rho, u, v, w) and (c^2, c) in shared memory (each
// thread's own and halo cell, at offsets computed once per tile); every limited y / z slope and every
// face flux is evaluated once (the reference evaluates each face twice) and shared through shared
// memory (y faces and slopes), warp shuffle (z faces) or registers (x faces; each cell's limited x
// slope is also carried to the next face).  Once-per-cell slopes pay here, where a slope costs a
// product, two compares and two selects per component (stages -5.5%).  Paired FP32 is not usable:
// the assembler fuses a dependent mul.rn.f32x2 -> add.rn.f32x2 into one fused multiply-add even with
// explicit round-to-nearest modifiers and -fmad=false (13% of random operands differ by an ulp).
#pragma once
#include "nb_internal.cuh"

namespace {

constexpr int PW = 36;                // primitive tile width along k: [k0-2, k0+34)
constexpr int HYDRO_THREADS = 256;
constexpr int HYDRO_TJ = 8;           // tile rows along j (one warp per row; 16 measured 2% slower)
constexpr long long HYDRO_IDX32_CELLS = (1LL << 31) - 1;       // signed cell offsets
constexpr int HYDRO_MINB = 4;         // resident blocks per SM the register budget is sized for (64 regs)
constexpr float HYDRO_PLANE[HYDRO_MINB + 1] = {0.0f, 0.59f, 0.72f, 0.86f, 1.0f};   // a plane's time by blocks on an SM
constexpr double HYDRO_WIND = 0.04;   // one star's wind over an ionized plane of a tile, in planes (nb_hydro_depth)
constexpr int HYDRO_ROT_STEP = 1;     // resident blocks start their extra work one scheduler apart

__device__ __forceinline__ float comp(const float4& v, int c) {
    return c == 0 ? v.x : (c == 1 ? v.y : (c == 2 ? v.z : v.w));
}

// Face flux between cells b and c along axis AX (1 = x, 2 = y, 3 = z: the velocity
// component normal to the face).  cs = (c^2, c) of a cell.
//   dot((0, L1, L2, L3), e_AX) == 0 + L_AX exactly (the other products are +-0 and the
//   velocities are finite), and e_c * (rho c^2) == +0 for c != AX.
// The limited slope (4 components) of cell b between its neighbours a and c along one axis:
// slope_lim(b - a, c - b).  A face's right slope is the next face's left slope along the same
// axis (same operands, same bits), which the x march carries from face to face.
template <int LM>
__device__ __forceinline__ float4 slopes_scalar(const float4 qa, const float4 qb, const float4 qc) {
    float sl[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) sl[c] = slope_lim<LM>(comp(qb, c) - comp(qa, c), comp(qc, c) - comp(qb, c));
    return make_float4(sl[0], sl[1], sl[2], sl[3]);
}

// the face flux from the two cells and their limited slopes
template <int SOLVER, int AX>
__device__ __forceinline__ float4 face_flux_sl(const float4 qb, const float4 qc, const float4 sl,
                                                      const float4 sr, const float2 csb, const float2 csc,
                                                      const float floor_) {
    float L[4], R[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        L[c] = comp(qb, c) + 0.5f * comp(sl, c);
        R[c] = comp(qc, c) - 0.5f * comp(sr, c);
    }
    const float rL = fmaxq(L[0], floor_), rR = fmaxq(R[0], floor_);
    const float unL = 0.0f + L[AX], unR = 0.0f + R[AX];
    const float UL[4] = {rL, rL * L[1], rL * L[2], rL * L[3]};
    const float UR[4] = {rR, rR * R[1], rR * R[2], rR * R[3]};
    const float pL = rL * csb.x, pR = rR * csc.x;
    float FL[4], FR[4], F[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        FL[c] = UL[c] * unL + (c == AX ? pL : 0.0f);
        FR[c] = UR[c] * unR + (c == AX ? pR : 0.0f);
    }
    if (SOLVER == NB_SOLVER_RUSANOV) {
        const float amax = fmaxq(fabsf(unL) + csb.y, fabsf(unR) + csc.y);
        const float ha = 0.5f * amax;
#pragma unroll
        for (int c = 0; c < 4; ++c) F[c] = 0.5f * (FL[c] + FR[c]) - ha * (UR[c] - UL[c]);
        return make_float4(F[0], F[1], F[2], F[3]);
    }
    const float SL = fminq(unL - csb.y, unR - csc.y);
    const float SR = fmaxq(unL + csb.y, unR + csc.y);
    if (SL >= 0.0f) return make_float4(FL[0], FL[1], FL[2], FL[3]);
    if (SR <= 0.0f) return make_float4(FR[0], FR[1], FR[2], FR[3]);
    const float slsr = SL * SR, den = SR - SL;
#pragma unroll
    for (int c = 0; c < 4; ++c) F[c] = (SR * FL[c] - SL * FR[c] + slsr * (UR[c] - UL[c])) / den;
    return make_float4(F[0], F[1], F[2], F[3]);
}

template <int SOLVER, int LIM>
__device__ __forceinline__ float4 cell_slopes(const float4 qa, const float4 qb, const float4 qc) {
    return slopes_scalar<SOLVER == NB_SOLVER_HLL ? LIM : 0>(qa, qb, qc);
}

// The x face between cells b and c of the march: `slope` holds cell b's limited slope on entry
// (the previous face's right slope) and cell c's on return.
template <int SOLVER, int LIM>
__device__ __forceinline__ float4 face_flux_x(const float4 qb, const float4 qc, const float4 qd, const float2 csb,
                                              const float2 csc, const float floor_, float4& slope) {
    const float4 sl = slope;
    slope = cell_slopes<SOLVER, LIM>(qb, qc, qd);
    return face_flux_sl<SOLVER, 1>(qb, qc, sl, slope, csb, csc, floor_);
}

template <int TJ>
struct HydroSmem {
    static constexpr int RAW_FIELD = (TJ + 4) * RAWW;                     // floats per field
    static constexpr int RAW_BYTES = 5 * RAW_FIELD * 4;                      // one raw slot
    static constexpr int PRIM_BYTES = 3 * (TJ + 4) * PW * 16;               // planes p-2, p-1, p
    static constexpr int CS_BYTES = 3 * (TJ + 4) * PW * 8;
    static constexpr int SY_BYTES = (TJ + 2) * TK * 16;                     // y slopes, rows j0-1 .. j0+TJ
    static constexpr int SZ_BYTES = TJ * (TK + 2) * 16;                     // z slopes, columns k0-1 .. k0+TK
    static constexpr int FACE_BYTES = ((TJ + 1) * TK + TJ) * 16;            // y faces; the z faces k0-1/2
    static constexpr int BAR_BYTES = 64;
    static constexpr int FIXED = RAW_BYTES + PRIM_BYTES + CS_BYTES + SY_BYTES + SZ_BYTES + FACE_BYTES + BAR_BYTES;
    // star tables: positions / wind weights and jets (2 x float4 per star), then the tile's jet
    // list: a count and the indices (one byte each) of the stars whose jet can reach the tile
    __host__ __device__ static int jet_list_offset(int nstars) { return FIXED + nstars * 32; }
    static int bytes(int nstars) { return jet_list_offset(nstars) + 16 + ((nstars + 15) & ~15); }
};

// One (j,k) tile column of one instance, marched over its i-chunk.  Called once per block by
// the single-instance kernel and once per work item by the persistent batched kernel.  The
// two mbarriers and their phases persist across calls: every load a call issues, it waits for.
// `rot` (0-3, the same in every thread of the block) spreads the per-plane work that only some
// warps do -- the y faces below the tile, the z faces before it, the z-halo conversion and the TMA
// issue -- over warps of four different schedulers (warp w is issued by scheduler w mod 4 when a
// block's warp slots start at a multiple of 4), rotated from block to block; any value gives the
// same results.
template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32 = false>
__device__ __forceinline__ void hydro_tile(const HydroLaunch& L, int tile, unsigned char* smem, unsigned& ph0,
                                           bool& failed, int rot) {
    static_assert(TJ == 8, "the halo and edge-face warp assignment assumes 8 warps of 32 threads");
    using Idx = typename std::conditional<I32, int, long long>::type;     // the own cell's offset
    using SM = HydroSmem<TJ>;
    {
        // an opaque zero added to the shared-memory base: the compiler then derives the tiles'
        // addresses from one register rather than holding several precomputed bases (measured at
        // 256^3: stage spills 4 -> 0 bytes, stages -3%, the same code otherwise)
        unsigned zero = 0;
        asm volatile("" : "+r"(zero));
        smem += zero;
    }
    float* raw = reinterpret_cast<float*>(smem);                                   // [5][TJ+4][40]
    float4* prim = reinterpret_cast<float4*>(smem + SM::RAW_BYTES);                // [4 or 3][TJ+4][36]
    float2* cs = reinterpret_cast<float2*>(smem + SM::RAW_BYTES + SM::PRIM_BYTES); // [3][TJ+4][36]
    float4* sy = reinterpret_cast<float4*>(smem + SM::RAW_BYTES + SM::PRIM_BYTES + SM::CS_BYTES);  // [TJ+2][32]
    float4* sz = sy + (TJ + 2) * TK;                                               // [TJ][34]
    float4* fy = sz + TJ * (TK + 2);                                               // [TJ+1][32]
    float4* fz0 = fy + (TJ + 1) * TK;                                              // [TJ]
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SM::FIXED - SM::BAR_BYTES);
    float4* sw_w = reinterpret_cast<float4*>(smem + SM::FIXED);
    const NbConst& C = *L.c;
    const int nx = C.nx, ny = C.ny, nz = C.nz, nstars = L.no_sources ? 0 : C.nstars;
    float4* sw_j = sw_w + nstars;

    const int tid = threadIdx.x, tk = tid & 31, tj = tid >> 5;
    const HydroTile tl(L, tile, nx, TJ);
    const int k0 = tl.k0, j0 = tl.j0, i0 = tl.i0, i_end = tl.i_end;
    const int P0 = i0 - 2, P1 = i_end + 1;

    const float floor_ = C.floor_, cn2 = C.cn2, ci2 = C.ci2, vmax = C.vmax, dx = C.dx;
    const float dt = L.use_override ? L.dt_override : L.st->dt_f;
    const float pulse = L.use_override ? L.pulse_override : L.st->pulse_f;
    const float wind = L.no_sources ? 0.0f : C.wind_f, jet_cos = C.jet_cos_f, jet_r = C.jet_r_f;
    const float a = L.a, b = L.b;

    int* n_jet_p = reinterpret_cast<int*>(smem + SM::jet_list_offset(nstars));
    unsigned char* jet_ix = smem + SM::jet_list_offset(nstars) + 16;
    for (int s = tid; s < nstars; s += blockDim.x) {
        sw_w[s] = L.sw[s].w;
        sw_j[s] = L.sw[s].jet;
    }
    constexpr unsigned TX_BYTES = 5u * SM::RAW_FIELD * 4u;
    auto issue = [&](int p) {                    // plane p into the raw slot, tracked by bar[0]
        if (!L.maps) return;                     // failure-path test: the wait for it runs out
        const int pc = iclampd(p, 0, nx - 1);
        fence_proxy_async();                     // the slot's previous contents were read by this block
        mbar_expect_tx(&bar[0], TX_BYTES);
#pragma unroll
        for (int f = 0; f < 4; ++f)
            tma_load_3d(raw + f * SM::RAW_FIELD, &L.maps[L.map_in + f], k0 - 4, j0 - 2, pc, &bar[0]);
        tma_load_3d(raw + 4 * SM::RAW_FIELD, &L.maps[NB_MAP_XI], k0 - 4, j0 - 2, pc, &bar[0]);
    };
    // the per-plane extra work, on warps of schedulers rot, rot+1, rot+2 and rot+3 (mod 4): the y
    // faces below the tile (role bit 1), the z faces before it (bit 2), the z-halo conversion,
    // the TMA issue (bit 4); with once-per-cell slopes also the slopes of the halo cells the faces
    // read: the y slopes of row j0-1 (bit 8) and of row j0+TJ (bit 16), the z slopes of columns
    // k0-1 and k0+TK (bit 32)
    const int w_zhalo = 4 + ((rot + 2) & 3);
    const unsigned role = (tj == rot ? 1u : 0u) | (tj == ((rot + 1) & 3) && tk < TJ ? 2u : 0u) |
                          (tid == (4 + ((rot + 3) & 3)) * 32 ? 4u : 0u) |
                          (tj == 4 + (rot & 3) ? 8u : 0u) |
                          (tj == 4 + ((rot + 1) & 3) ? 16u : 0u) |
                          (tj == 4 + ((rot + 3) & 3) && tk < 2 * TJ ? 32u : 0u);
    if (role & 4u) issue(P0);
    if (tj == 0) jet_list(L, tl, ny, nz, TJ, dx, jet_r, nstars, tk, n_jet_p, jet_ix);

    float4 fx_prev = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xslope = make_float4(0.f, 0.f, 0.f, 0.f);    // limited x slope of the march's cell p-2
    float vmax_local = 0.0f;

    // clamped global -> raw-tile coordinates
    auto raw_at = [&](int jj, int kk) {      // jj, kk: prim-tile coords
        const int jc = iclampd(j0 - 2 + jj, 0, ny - 1) - (j0 - 2);
        const int kc = iclampd(k0 - 2 + kk, 0, nz - 1) - (k0 - 4);
        return jc * RAWW + kc;
    };
    const int own = (tj + 2) * PW + tk + 2;          // this thread's cell in a prim / cs tile
    // the cells this thread converts in every plane: its own, and one of the 4 TK + 4 TJ cells of
    // the halo strips (corners are never read): warps 0-3 one row of the y strips each, warp
    // w_zhalo the z strips; their offsets, computed once per tile, clamp to the domain in the raw tile
    const bool has_halo = tj < 4 || tj == w_zhalo;
    const int raw_own = raw_at(tj + 2, tk + 2);
    int prim_halo = 0, raw_halo = 0;
    if (has_halo) {
        int jj, kk;
        if (tj < 4) {
            jj = tj < 2 ? tj : TJ + tj;
            kk = 2 + tk;
        } else {
            const int hh = tk;
            jj = 2 + (hh >> 2);
            const int q = hh & 3;
            kk = q < 2 ? q : 32 + q;
        }
        prim_halo = jj * PW + kk;
        raw_halo = raw_at(jj, kk);
    }
    const int j = j0 + tj, k = k0 + tk;
    const bool inside = j < ny && k < nz;
    constexpr int PSLOT = (TJ + 4) * PW;

    for (int p = P0; p <= P1; ++p) {
        // slots of planes p, p-1, p-2 in the three-plane rings of primitives and sound speeds
        const int cq = (p - P0) % 3;
        const int cq1 = cq == 0 ? 2 : cq - 1;
        const int cq2 = cq1 == 0 ? 2 : cq1 - 1;
        const int ps = cq;
        // own-cell values of plane i = p - 2 the epilogue needs, issued before the flux work
        const int i = p - 2;
        const Idx cell = ((Idx)i * ny + j) * nz + k;
        const bool work = p >= i0 + 2;
        float u00 = 0.f, u01 = 0.f, u02 = 0.f, u03 = 0.f, ur = 0.f, umx = 0.f, umy = 0.f, umz = 0.f, uxi = 0.f;
        if (work && inside) {
            ur = L.in[0][cell]; umx = L.in[1][cell]; umy = L.in[2][cell]; umz = L.in[3][cell];
            uxi = L.xi[cell];
            if (STAGE2) {                        // early: read only at the end, 4 more live registers
                u00 = L.u0[0][cell]; u01 = L.u0[1][cell]; u02 = L.u0[2][cell]; u03 = L.u0[3][cell];
            }
        }
        const int jj = tj + 2, kk = tk + 2;
        if (work) {
            // ---- the limited y and z slopes of every cell of plane i that the faces read, each
            // evaluated once (a face's two slopes are its cells' slopes along its axis: the same
            // operands, the same bits).  Plane i was converted two planes ago and the previous
            // plane's faces are done (its second barrier), so no barrier is needed here, and this
            // work overlaps the wait for plane p's tile.
            const float4* q = prim + cq2 * PSLOT;
            const float4 qo = q[jj * PW + kk];
            sy[(tj + 1) * TK + tk] = cell_slopes<SOLVER, LIM>(q[(jj - 1) * PW + kk], qo, q[(jj + 1) * PW + kk]);
            sz[tj * (TK + 2) + tk + 1] = cell_slopes<SOLVER, LIM>(q[jj * PW + kk - 1], qo, q[jj * PW + kk + 1]);
            if (role & 8u)                       // row j0-1: primitive rows 0..2
                sy[tk] = cell_slopes<SOLVER, LIM>(q[0 * PW + kk], q[1 * PW + kk], q[2 * PW + kk]);
            if (role & 16u)                      // row j0+TJ: primitive rows TJ+1..TJ+3
                sy[(TJ + 1) * TK + tk] = cell_slopes<SOLVER, LIM>(q[(TJ + 1) * PW + kk], q[(TJ + 2) * PW + kk],
                                                                  q[(TJ + 3) * PW + kk]);
            if (role & 32u) {                    // columns k0-1 (lanes 0..TJ-1) and k0+TK (lanes TJ..2TJ-1)
                const int r = tk & (TJ - 1);
                const int c0 = tk < TJ ? 0 : TK + 1;
                const int b = (r + 2) * PW + c0;
                sz[r * (TK + 2) + c0] = cell_slopes<SOLVER, LIM>(q[b], q[b + 1], q[b + 2]);
            }
        }
        const bool ok = mbar_wait_limited(&bar[0], ph0, &L.wait_limit);
        if (ok) ph0 ^= 1u;                       // a timed-out wait keeps its parity for the abort wait
        if (__syncthreads_or(!ok)) { failed = true; break; }
        const float* rb = raw;
        float4* pp = prim + ps * PSLOT;
        float2* cp = cs + cq * PSLOT;
        // ---- convert plane p: the own cell, then (has_halo) one cell of the halo strips
        auto convert = [&](int o, int pi) {
            const float r = fmaxq(rb[o], floor_);
            const float xv = rb[4 * SM::RAW_FIELD + o];
            const float c2 = cn2 + xv * (ci2 - cn2);
            pp[pi] = make_float4(r, rb[SM::RAW_FIELD + o] / r, rb[2 * SM::RAW_FIELD + o] / r,
                                 rb[3 * SM::RAW_FIELD + o] / r);
            cp[pi] = make_float2(c2, sqrtf(c2));
        };
        convert(raw_own, own);
        if (has_halo) convert(raw_halo, prim_halo);
        __syncthreads();                         // every thread is done with the raw slot
        if ((role & 4u) && p + 1 <= P1) issue(p + 1);
        if (p < P0 + 2) continue;
        if (p == P0 + 2) {                       // the x slope of plane P0+1 (planes P0, P0+1, P0+2)
            xslope = cell_slopes<SOLVER, LIM>(prim[cq2 * PSLOT + own], prim[cq1 * PSLOT + own], pp[own]);
            continue;
        }
        // x face (p-2)+1/2 from the own column of planes p-2..p and the carried slope of p-2
        const float4 fx_new = face_flux_x<SOLVER, LIM>(prim[cq2 * PSLOT + own], prim[cq1 * PSLOT + own], pp[own],
                                                       cs[cq2 * PSLOT + own], cs[cq1 * PSLOT + own], floor_, xslope);
        if (!work) { fx_prev = fx_new; continue; }
        // ---- the y and z faces of cell plane i, from the cells and their slopes
        const float4* q = prim + cq2 * PSLOT;
        const float2* c = cs + cq2 * PSLOT;
        const float4 fyp = face_flux_sl<SOLVER, 2>(q[jj * PW + kk], q[(jj + 1) * PW + kk], sy[(tj + 1) * TK + tk],
                                                   sy[(tj + 2) * TK + tk], c[jj * PW + kk], c[(jj + 1) * PW + kk],
                                                   floor_);
        const float4 fzp = face_flux_sl<SOLVER, 3>(q[jj * PW + kk], q[jj * PW + kk + 1], sz[tj * (TK + 2) + tk + 1],
                                                   sz[tj * (TK + 2) + tk + 2], c[jj * PW + kk], c[jj * PW + kk + 1],
                                                   floor_);
        fy[(tj + 1) * TK + tk] = fyp;
        if (role & 1u) {                        // the y face below the tile: (j0-1)+1/2
            fy[tk] = face_flux_sl<SOLVER, 2>(q[1 * PW + kk], q[2 * PW + kk], sy[tk], sy[TK + tk], c[1 * PW + kk],
                                             c[2 * PW + kk], floor_);
        } else if (role & 2u) {                 // the z face before the tile in row tk: (k0-1)+1/2
            const int r2 = (tk + 2) * PW;
            fz0[tk] = face_flux_sl<SOLVER, 3>(q[r2 + 1], q[r2 + 2], sz[tk * (TK + 2)], sz[tk * (TK + 2) + 1],
                                              c[r2 + 1], c[r2 + 2], floor_);
        }
        __syncthreads();
        const float4 fym = fy[tj * TK + tk];
        // the z face k-1/2 is the lower lane's k+1/2; lane 0 takes the face before the tile
        float4 fzm = make_float4(__shfl_up_sync(0xffffffffu, fzp.x, 1), __shfl_up_sync(0xffffffffu, fzp.y, 1),
                                 __shfl_up_sync(0xffffffffu, fzp.z, 1), __shfl_up_sync(0xffffffffu, fzp.w, 1));
        if (tk == 0) fzm = fz0[tj];
        const float4 fxp = fx_new, fxm = fx_prev;
        fx_prev = fx_new;
        // div = 0 + (fR-fL)_x, then += (fR-fL)_y, then += (fR-fL)_z  (nebula3d.py:87-109)
        float du0, du1, du2, du3;
        float d0 = 0.0f + (fxp.x - fxm.x), d1 = 0.0f + (fxp.y - fxm.y);
        float d2 = 0.0f + (fxp.z - fxm.z), d3 = 0.0f + (fxp.w - fxm.w);
        d0 = d0 + (fyp.x - fym.x); d1 = d1 + (fyp.y - fym.y); d2 = d2 + (fyp.z - fym.z); d3 = d3 + (fyp.w - fym.w);
        d0 = d0 + (fzp.x - fzm.x); d1 = d1 + (fzp.y - fzm.y); d2 = d2 + (fzp.z - fzm.z); d3 = d3 + (fzp.w - fzm.w);
        // ---- sources and RK combination (nebula3d.py:111-151)
        if (C.dx_pow2) {
            const float sc = C.inv_dx;
            du0 = -d0 * sc; du1 = -d1 * sc; du2 = -d2 * sc; du3 = -d3 * sc;
        } else {
            du0 = -d0 / dx; du1 = -d1 / dx; du2 = -d2 / dx; du3 = -d3 / dx;
        }
        const float px = ((float)i + 0.5f) * dx, py = ((float)j + 0.5f) * dx, pz = ((float)k + 0.5f) * dx;
        const float x_ion = uxi;
        if (wind > 0.0f && x_ion > 0.01f) {
            float ax = 0.0f, ay = 0.0f, az = 0.0f;
            for (int s = 0; s < nstars; ++s) {
                const float4 st = sw_w[s];
                if (st.w > 0.0f) {
                    const float rx = px - st.x, ry = py - st.y, rz = pz - st.z;
                    const float r2 = ((rx * rx + ry * ry) + rz * rz) + 0.0004f;     // 0 + x*x == x*x
                    const float f = st.w / (r2 * sqrtf(r2));
                    ax = ax + rx * f; ay = ay + ry * f; az = az + rz * f;
                }
            }
            const float wx = wind * x_ion;
            ax = ax * wx; ay = ay * wx; az = az * wx;
            du0 = du0 + 0.0f;
            du1 = du1 + ur * ax; du2 = du2 + ur * ay; du3 = du3 + ur * az;
        }
        float jx = 0.0f, jy = 0.0f, jz = 0.0f;
        const int n_jet = *n_jet_p;
        for (int m = 0; m < n_jet; ++m) {
            const int s = jet_ix[m];
            const float4 jt = sw_j[s];
            const float4 st = sw_w[s];
            {
                const float rx = px - st.x, ry = py - st.y, rz = pz - st.z;
                const float r = sqrtf((rx * rx + ry * ry) + rz * rz);
                if (r < jet_r && r > 1e-6f) {
                    const float cth = (((0.0f + rx * jt.x) + ry * jt.y) + rz * jt.z) / r;
                    if (fabsf(cth) > jet_cos) {
                        const float f = (cth > 0.0f ? 1.0f : -1.0f) * jt.w * pulse / (r * r + 0.0004f);
                        jx = jx + jt.x * f; jy = jy + jt.y * f; jz = jz + jt.z * f;
                    }
                }
            }
        }
        du0 = du0 + 0.0f;
        du1 = du1 + ur * jx; du2 = du2 + ur * jy; du3 = du3 + ur * jz;
        if (!STAGE2) {
            u00 = ur; u01 = umx; u02 = umy; u03 = umz;
        }
        const float un0 = ur + dt * du0, un1 = umx + dt * du1, un2 = umy + dt * du2, un3 = umz + dt * du3;
        const float o0 = a * u00 + b * un0, o1 = a * u01 + b * un1, o2 = a * u02 + b * un2, o3 = a * u03 + b * un3;
        const float r = fmaxq(o0, floor_);
        float vx = o1 / r, vy = o2 / r, vz = o3 / r;
        const float sp = sqrtf((vx * vx + vy * vy) + vz * vz);
        if (sp > vmax) {
            const float f = vmax / sp;
            vx = vx * f; vy = vy * f; vz = vz * f;
        }
        const float m1 = r * vx, m2 = r * vy, m3 = r * vz;
        if (inside) {
            L.out[0][cell] = r;
            L.out[1][cell] = m1;
            L.out[2][cell] = m2;
            L.out[3][cell] = m3;
            if (STAGE2 && L.smax_bits) {         // nebula3d.py:158-162 on the new state
                const float v = fabsf(m1 / r) + fabsf(m2 / r) + fabsf(m3 / r) + c[own].y;
                vmax_local = fmaxq(v, vmax_local);
            }
        }
    }
    if (failed) return;
    if (STAGE2 && L.smax_bits) hydro_smax(L, vmax_local, reinterpret_cast<float*>(fy), TJ);
}

}  // namespace
