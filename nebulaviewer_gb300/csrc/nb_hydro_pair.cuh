// The fast build's hydro stage tile: two rows per thread on paired FP32.
//
// A block owns a 32 (k) x 16 (j) column of cells and marches along i.  Thread (w, lane) of its eight
// warps holds the cells of rows j = j0 + 2w and j + 1 at k = k0 + lane as one pair in every
// register: each float operation of the reconstruction, the flux and the update is one f32x2
// instruction for two cells (sm_100+ add/sub/mul/fma.rn.f32x2), and no half ever has to be moved to
// make a pair -- pairs of a cell's components need broadcast operands and cost the flux about a
// third more instructions.  The two rows are neighbours, so the y slopes and the face between them
// are shared in registers.
//
// One block barrier per plane.  At march step p (plane p's tile has landed):
//   convert plane p to primitives (own pair, and on three warps one pair of the halo strips) into slot
//   p mod 3, keeping the own cells' raw values for the update two steps on;
//   barrier; request plane p+1's tile;
//   x face (p-2)+1/2 from the own column, and with it the update of plane p-2;
//   y and z faces of plane p-1 (its slot is complete since the barrier), kept in registers but for
//   the face above each row pair, which the next warp reads a step later from shared memory.
// The faces at the tile's lower y and z edges and the state beyond its upper z edge are extra work
// of two warps, done a step ahead.  128 registers, 112 KB of shared memory, two blocks per SM at any
// number of stars.
//
// Bound: the shared-memory data pipe, 81 / 79% of its peak wavefronts in stage 1 / 2 (a 16-byte access is four
// a warp), with 16 warps a SM to hide it: issue is 56% and DRAM 31 / 42%; a warp waits on fixed latencies
// 1.2 cycles an instruction, on shared memory 0.9, on the barrier 0.9.  313 / 337 thread instructions a cell where
// pairs of components took 528 / 559.  Measured at 256^3 (sheet, chosen depth of 37 planes): stage 1 309 -> 243 us,
// stage 2 338 -> 260 us (2.49 and 3.36 TB/s of their 36 and 52 B a cell); 192^3 145 -> 115, 160 -> 123 us.
// Grids of up to 8 rows leave half a tile idle: 512 x 8 x 512 110 -> 131 us for both stages.
// Tried on this tile and slower or level: the own cells' values read again from global memory (one
// address instruction and a pointer load per access, +12%), shuffles along k (+3%), the march unrolled
// by two (instructions -5%, instruction fetch stalls +), a ninth and tenth warp for the edge work (96
// registers: stage 1 level, stage 2 +20%), the next tile prefetched to L2 (level).
#pragma once
#include "nb_f32x2.cuh"
#include "nb_internal.cuh"

namespace {

constexpr int HYDRO_TJ = 16;          // tile rows along j (two rows per warp)
constexpr int HYDRO_THREADS = 256;    // eight warps
constexpr int PPW = 36;               // pairs per row of a plane: columns k0-2 .. k0+33
constexpr long long HYDRO_IDX32_CELLS = (1LL << 31) - 1;       // signed cell offsets
constexpr int HYDRO_MINB = 2;         // resident blocks per SM (128 registers, 112 KB of shared memory each)
constexpr float HYDRO_PLANE[HYDRO_MINB + 1] = {0.0f, 0.74f, 1.0f};   // a plane's time by blocks on an SM
constexpr double HYDRO_WIND = 0.04;   // one star's wind over an ionized plane of a tile, in planes (nb_hydro_depth)
constexpr int HYDRO_ROT_STEP = 2;     // two resident blocks place their extra work two schedulers apart

// an approximate reciprocal (<= 1 ulp)
__device__ __forceinline__ float vrcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ F2 vrcp(F2 a) { return mk2(vrcp(lo(a)), vrcp(hi(a))); }
__device__ __forceinline__ float vmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ F2 vmax(F2 a, float b) { return mk2(fmaxf(lo(a), b), fmaxf(hi(a), b)); }
// max(a, b, 0) in one instruction (sm_100+)
__device__ __forceinline__ float vmax0(float a, float b) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(0.0f));
    return r;
}
__device__ __forceinline__ F2 vmax0(F2 a, F2 b) { return mk2(vmax0(lo(a), lo(b)), vmax0(hi(a), hi(b))); }
__device__ __forceinline__ float vabs_add(float a, float c) { return vadd(fabsf(a), c); }
__device__ __forceinline__ F2 vabs_add(F2 a, F2 c) { return mk2(vabs_add(lo(a), lo(c)), vabs_add(hi(a), hi(c))); }
__device__ __forceinline__ float vmaxv(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ F2 vmaxv(F2 a, F2 b) { return mk2(fmaxf(lo(a), lo(b)), fmaxf(hi(a), hi(b))); }
template <typename T>
__device__ __forceinline__ T vset(float a);
template <>
__device__ __forceinline__ float vset<float>(float a) { return a; }
template <>
__device__ __forceinline__ F2 vset<F2>(float a) { return mk2(a, a); }

// min.xorsign.abs: min(|a|, |b|) with the sign sign(a) xor sign(b)
__device__ __forceinline__ float min_xorsign(float a, float b) {
    float r;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// The limited slope between the differences a and b.  Minmod in three ALU operations and no product:
// m = min_xorsign(a, b) is min(|a|, |b|) when a and b have the same sign, <= 0 otherwise;
// min_xorsign(a, max(m, 0)) puts a's sign on it.  The value is nebula3d.py:40-46's (a or b, the
// smaller magnitude), but that a zero result may be -0, and that an underflowing product a * b, where
// the reference returns 0, gives the smaller magnitude.
template <int LIM>
__device__ __forceinline__ float slope1(float a, float b) {
    if (LIM == 0) return min_xorsign(a, fmaxf(min_xorsign(a, b), 0.0f));
    return slope_lim<LIM>(a, b);
}
template <int LIM>
__device__ __forceinline__ F2 slope1(F2 a, F2 b) {
    return mk2(slope1<LIM>(lo(a), lo(b)), slope1<LIM>(hi(a), hi(b)));
}

// a state's density, velocity normal to a face and two transverse velocities; (c^2, c) beside it
template <typename T>
struct St {
    T r, n, s, t;
};
template <typename T>
struct Cs {
    T c2, c;
};

// The face flux (nebula3d.py:54-72, sim.py:397-420) of the reconstructed states L and R, normal
// component second.  HLL with S_L = -m and S_R = s clamped to m, s >= 0 (the early returns of
// sim.py:410-413 up to the rounding of s / s) and Rusanov are one form,
//   F = a F_L + b F_R + k (U_L - U_R),   HLL: a = s / (s + m), b = m / (s + m), k = a m = b s
//                                         Rusanov: a = b = 1/2, m = s = max(|u| + c), k = s / 2.
// With U = r (1, u, v, w) and F = U u + p, the left state's part of every component but the
// pressure is G_L (1, u, v, w), G_L = a r_L u_L + k r_L = a r_L (u_L + m) >= 0, and the right one's
// G_R (1, u, v, w), G_R = b r_R (u_R - s) <= 0: 28 pair operations instead of the 40 of evaluating U,
// F_L and F_R by component.  The mass flux takes r_L - r_R as one difference (as the component form
// does: no cancellation between G_L and G_R).  Each side's G comes from its own state, so each
// velocity is carried with its own side's rounding: G_R as the mass flux less G_L (one operation
// less, level in time: 246 / 266 us at 256^3 against 245 / 265) rounds at the left side's size, and a
// dense cell beside thin fast gas then costs the thin side's momentum up to 300 times the rounding of
// its terms, in one direction of the axis only.  Errors of a stage against float64, start of the
// component form -> this: level or smaller in smooth, rough, still, hot and cold gas and at fronts.
template <int SOLVER, typename T>
__device__ __forceinline__ St<T> flux(const St<T>& L, const Cs<T>& cl, const St<T>& R, const Cs<T>& cr,
                                      const float floor_) {
    const T rL = vmax(L.r, floor_), rR = vmax(R.r, floor_);
    T a, b, m, s;
    if (SOLVER == NB_SOLVER_RUSANOV) {
        a = b = vset<T>(0.5f);
        m = s = vmaxv(vabs_add(L.n, cl.c), vabs_add(R.n, cr.c));
    } else {
        m = vmax0(vsub(cl.c, L.n), vsub(cr.c, R.n));
        s = vmax0(vadd(L.n, cl.c), vadd(R.n, cr.c));
        const T inv = vrcp(vadd(s, m));
        a = vmul(s, inv);
        b = vmul(m, inv);
    }
    const T aL = vmul(a, rL), bR = vmul(b, rR);
    St<T> F;
    F.r = vfma(aL, L.n, vfma(bR, R.n, vmul(vmul(a, m), vsub(rL, rR))));
    const T gL = vmul(aL, vadd(L.n, m)), gR = vmul(bR, vsub(R.n, s));
    const T p = vfma(a, vmul(rL, cl.c2), vmul(b, vmul(rR, cr.c2)));
    F.n = vfma(gL, L.n, vfma(gR, R.n, p));
    F.s = vfma(gL, L.s, vmul(gR, R.s));
    F.t = vfma(gL, L.t, vmul(gR, R.t));
    return F;
}

// b + 0.5 s and b - 0.5 s, the states at a cell's upper and lower face
template <typename T>
__device__ __forceinline__ St<T> up(const St<T>& b, const St<T>& s) {
    const T h = vset<T>(0.5f);
    return {vfma(h, s.r, b.r), vfma(h, s.n, b.n), vfma(h, s.s, b.s), vfma(h, s.t, b.t)};
}
template <typename T>
__device__ __forceinline__ St<T> down(const St<T>& b, const St<T>& s) {
    const T h = vset<T>(-0.5f);
    return {vfma(h, s.r, b.r), vfma(h, s.n, b.n), vfma(h, s.s, b.s), vfma(h, s.t, b.t)};
}
template <typename T>
__device__ __forceinline__ St<T> diff(const St<T>& b, const St<T>& a) {
    return {vsub(b.r, a.r), vsub(b.n, a.n), vsub(b.s, a.s), vsub(b.t, a.t)};
}
template <int LIM, typename T>
__device__ __forceinline__ St<T> slopes(const St<T>& a, const St<T>& b) {
    return {slope1<LIM>(a.r, b.r), slope1<LIM>(a.n, b.n), slope1<LIM>(a.s, b.s), slope1<LIM>(a.t, b.t)};
}
__device__ __forceinline__ St<float> lo(const St<F2>& a) { return {lo(a.r), lo(a.n), lo(a.s), lo(a.t)}; }
__device__ __forceinline__ St<float> hi(const St<F2>& a) { return {hi(a.r), hi(a.n), hi(a.s), hi(a.t)}; }
__device__ __forceinline__ St<F2> mk2(const St<float>& a, const St<float>& b) {
    return {mk2(a.r, b.r), mk2(a.n, b.n), mk2(a.s, b.s), mk2(a.t, b.t)};
}
// A stored state is (r, u, v, w); the face along an axis takes its normal component second.
// Each of these is its own inverse.
template <typename T>
__device__ __forceinline__ St<T> y_order(const St<T>& a) { return {a.r, a.s, a.n, a.t}; }
template <typename T>
__device__ __forceinline__ St<T> z_order(const St<T>& a) { return {a.r, a.t, a.s, a.n}; }

// Shared memory of a tile, as byte offsets (every access is one register and an immediate).
template <int TJ>
struct HydroSmem {
    static constexpr int NP = TJ / 2;                                        // row pairs, one per warp
    static constexpr int RAW_FIELD = (TJ + 4) * RAWW * 4;                    // one field of the raw slot
    static constexpr int PLANE = (NP + 2) * PPW * 16;                        // one array over a plane with its halo
    // a slot: (r0 r1 u0 u1), (v0 v1 w0 w1) and (c2_0 c2_1 c_0 c_1) of every pair, then the own cells' raw
    // (rho, mx) and (my, mz), [256] each
    static constexpr int OWN = 3 * PLANE;
    static constexpr int PER = HYDRO_THREADS * 16;                           // 16 bytes per thread
    static constexpr int RAW = 0;                                            // five fields: plane p as loaded
    static constexpr int SLOT = OWN + 2 * PER;
    // a warp's exchange along k, [2 halves][256], and beside it the edges [parity][side][NP] of each half:
    // side 0 the z face before the tile, side 1 the lower state of the cell after it
    static constexpr int ZX = (RAW + 5 * RAW_FIELD + 511) / 512 * 512;
    static constexpr int ZE = ZX + PER, ZE_PAR = 256, ZE_SIDE = 128;         // ZE: a multiple of 512
    static constexpr int ZX_HALF = PER + 512;
    static constexpr int FY = ZX + 2 * ZX_HALF;                              // the y face below each pair, [parity][256]
    static constexpr int XI = FY + 2 * PER;                                  // the own cells' xi, [parity][256]
    static constexpr int PRIM = XI + PER;                                    // slots of planes p-2, p-1, p
    static constexpr int BAR_BYTES = 64;
    static constexpr int FIXED = PRIM + 3 * SLOT + BAR_BYTES;
    static constexpr int FLAG = FIXED - BAR_BYTES + 16;                      // after two mbarriers: a wait gave up
    // The tile's jet list: a count and the indices (one byte each) of the stars whose jet can reach the tile.
    // The stars' weights and jets are read through L1, by all lanes at once: two blocks leave 1.3 KB of an
    // SM's shared memory, and with the tables there (32 B a star) from 38 stars on only one block was resident.
    // Stages 1 + 2 at 256^3 with the tables there -> this, in 37-plane chunks: 6 stars 512 -> 514 us, 40 stars
    // 846 -> 618, 128 stars 1343 -> 1135, 256 stars 2369 -> 2074; without winds from 38 stars on 662 -> 491.
    static constexpr int JETS = FIXED;
    static int bytes(int nstars) { return JETS + 16 + ((nstars + 15) & ~15); }
    static_assert(HYDRO_MINB * (JETS + 16 + NB_MAX_STARS + 1024) <= 228 * 1024, "two blocks per SM");
};

// One (j,k) tile column of one instance, marched over its i-chunk.  Called once per block by
// the single-instance kernel and once per work item by the persistent batched kernel.  The
// two mbarriers and their phases persist across calls: every load a call issues, it waits for.
// `rot` (0-3, the same in every thread of the block) places the per-plane work that only some warps
// do on warps of four different schedulers (warp w is issued by scheduler w mod 4 when a block's
// warp slots start at a multiple of 4); any value gives the same results.
template <int SOLVER, int LIM, int TJ, bool STAGE2, bool I32 = false>
__device__ __forceinline__ void hydro_tile(const HydroLaunch& L, int tile, unsigned char* smem, unsigned& ph0,
                                           bool& failed, int rot) {
    static_assert(TJ == 16, "eight warps of two rows each");
    constexpr int LM = SOLVER == NB_SOLVER_HLL ? LIM : 0;
    using Idx = typename std::conditional<I32, int, long long>::type;     // the own cells' offsets
    using SM = HydroSmem<TJ>;
    constexpr int NP = SM::NP, ROW = PPW * 16;
    {
        // an opaque zero on the shared-memory base keeps the compiler from holding several precomputed
        // bases (stage 1 -3%, stage 2 -4% at 256^3)
        unsigned zero = 0;
        asm volatile("" : "+r"(zero));
        smem += zero;
    }
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SM::FIXED - SM::BAR_BYTES);
    const NbConst& C = *L.c;
    const int nx = C.nx, ny = C.ny, nz = C.nz, nstars = L.no_sources ? 0 : C.nstars;

    const int tid = threadIdx.x, tk = tid & 31, tj = tid >> 5;
    const HydroTile tl(L, tile, nx, TJ);
    const int k0 = tl.k0, j0 = tl.j0, i0 = tl.i0, i_end = tl.i_end;
    const int P0 = i0 - 2, P1 = i_end + 1;

    const float floor_ = C.floor_, cn2 = C.cn2, dci2 = C.ci2 - C.cn2, vcap = C.vmax, dx = C.dx;
    const float dt = L.use_override ? L.dt_override : L.st->dt_f;
    const float pulse = L.use_override ? L.pulse_override : L.st->pulse_f;
    const float wind = L.no_sources ? 0.0f : C.wind_f, jet_cos = C.jet_cos_f, jet_r = C.jet_r_f;

    int* n_jet_p = reinterpret_cast<int*>(smem + SM::JETS);
    unsigned char* jet_ix = smem + SM::JETS + 16;
    auto issue = [&](int p, int to, uint64_t* b) {           // plane p into the raw slot at `to`, tracked by b
        if (!L.maps) return;                     // failure-path test: the wait for it runs out
        const int pc = iclampd(p, 0, nx - 1);
        fence_proxy_async();                     // the slot's previous contents were read by this block
        mbar_expect_tx(b, 5u * SM::RAW_FIELD);
#pragma unroll
        for (int f = 0; f < 5; ++f)
            tma_load_3d(smem + to + f * SM::RAW_FIELD, &L.maps[f < 4 ? L.map_in + f : NB_MAP_XI], k0 - 4, j0 - 2, pc, b);
    };
    // The second plane of a march lands in the last primitive slot, which is free until the third is
    // converted, so the first two loads are in flight together.
    static_assert(5 * SM::RAW_FIELD <= SM::SLOT, "a raw slot fits a primitive slot");
    constexpr int SECOND = SM::PRIM + 2 * SM::SLOT;
    // the warps with extra work: y faces below the tile; z faces before it and states after it; the
    // z halo strips; the tile request; the two y halo row pairs (on the other four warps)
    const bool w_yedge = tj == rot, w_zedge = tj == ((rot + 1) & 3), w_issue = tid == ((rot + 3) & 3) * 32;
    const int w_zhalo = (rot + 2) & 3, w_ylo = 4 + ((rot + 2) & 3), w_yhi = 4 + ((rot + 3) & 3);
    if (w_issue) {
        issue(P0, SM::RAW, &bar[0]);
        issue(P0 + 1, SECOND, &bar[1]);
    }
    if (tj == 0) jet_list(L, tl, ny, nz, TJ, dx, jet_r, nstars, tk, n_jet_p, jet_ix);

    auto ld4 = [&](int o) -> float4 { return *reinterpret_cast<const float4*>(smem + o); };
    auto st4 = [&](int o, F2 u, F2 v) { *reinterpret_cast<float4*>(smem + o) = make_float4(lo(u), hi(u), lo(v), hi(v)); };
    auto state = [&](int o, int half) -> St<F2> {            // a state in two 16-byte halves
        const float4 x = ld4(o), y = ld4(o + half);
        return {mk2(x.x, x.y), mk2(x.z, x.w), mk2(y.x, y.y), mk2(y.z, y.w)};
    };
    auto load = [&](int o) { return state(SM::PRIM + o, SM::PLANE); };
    auto load_c = [&](int o) -> Cs<F2> {
        const float4 x = ld4(SM::PRIM + o + 2 * SM::PLANE);
        return {mk2(x.x, x.y), mk2(x.z, x.w)};
    };
    // clamped global -> byte offset in a raw field of halo-tile row jj (0 .. TJ+3), column kk (0 .. 35)
    auto raw_at = [&](int jj, int kk) {
        const int jc = iclampd(j0 - 2 + jj, 0, ny - 1) - (j0 - 2);
        const int kc = iclampd(k0 - 2 + kk, 0, nz - 1) - (k0 - 4);
        return (jc * RAWW + kc) * 4;
    };
    // the pairs this thread converts in every plane: its own and, on three warps, one of the halo
    // strips (corners are never read); offsets computed once per tile, clamped to the domain
    const bool has_halo = tj == w_zhalo || tj == w_ylo || tj == w_yhi;
    const int raw_own0 = raw_at(2 * tj + 2, tk + 2), raw_own1 = raw_at(2 * tj + 3, tk + 2);
    int halo = 0, raw_halo0 = 0, raw_halo1 = 0;              // halo: relative to the own pair's place
    if (has_halo) {
        int pr = tj == w_ylo ? 0 : NP + 1, kk = tk + 2;
        if (tj == w_zhalo) {
            pr = 1 + (tk >> 2);
            kk = (tk & 3) < 2 ? (tk & 3) : 32 + (tk & 3);
        }
        halo = (pr - tj - 1) * ROW + (kk - tk - 2) * 16;
        raw_halo0 = raw_at(2 * pr, kk);
        raw_halo1 = raw_at(2 * pr + 1, kk);
    }
    const int j = j0 + 2 * tj, k = k0 + tk;
    const bool in0 = j < ny && k < nz, in1 = j + 1 < ny && k < nz;
    // a plane's offset of the own pair's cells, clamped to the grid (a cell outside it is never stored)
    const Idx plane = (Idx)ny * nz, at = (Idx)min(j, ny - 1) * nz + min(k, nz - 1);
    const int up_row = j + 1 < ny ? nz : 0;

    const float ab = L.a + L.b, bdt = L.b * dt, kdiv = -__fdiv_rn(bdt, dx);
    const float src = kdiv != 0.0f ? __fdiv_rn(bdt, kdiv) : 0.0f;       // -dx, such that kdiv src is b dt
    float vmax_local = 0.0f;
    St<F2> Lx{}, fxp{}, S{};                         // plane p-1's upper x state; the last x face; plane p-2's y and
    St<float> f1{};                                  // z differences, and its face between the two rows
    F2 u0[4];                                        // stage 2: u0 of the plane the next step updates
    // offsets that a step leaves for the next: the own pair in the slots of planes p, p-1, p-2; the own
    // 16 bytes of the parity of p - P0; where the next lane's lower state and the previous lane's face are
    const int own = (tj + 1) * ROW + (tk + 2) * 16, raw_place = SM::OWN + tid * 16 - own;
    int o0 = own, o1 = own + 2 * SM::SLOT, o2 = own + SM::SLOT, t0 = tid * 16;
    int z_up = tk == 31 ? SM::ZE + SM::ZE_SIDE + SM::ZE_PAR + tj * 16 : SM::ZX + tid * 16 + 16;
    int z_dn = tk == 0 ? SM::ZE + SM::ZE_PAR + tj * 16 : SM::ZX + tid * 16 - 16;
    const int z_up_par = tk == 31 ? SM::ZE_PAR : 0, z_dn_par = tk == 0 ? SM::ZE_PAR : 0;
    int n_jet = 0;

    // One march step.  FULL: x faces, update and y / z faces; otherwise (the first three planes) only the
    // conversion and the x states.  The first full step's update (plane i0-1) and the last one's y / z
    // faces (plane i_end) come to nothing: the one is not stored, the others are not read.
    auto step = [&](const int p, auto full, auto second) -> bool {
        constexpr bool FULL = decltype(full)::value, SEC = decltype(second)::value;   // SEC: plane P0+1
        constexpr int RAW = SEC ? SECOND : SM::RAW;
        const int i = p - 2;
        if (FULL && (wind > 0.0f || n_jet > 0)) {
            // ---- wind and jets of plane i (nebula3d.py:111-149), into its flux differences, which
            // the update scales by kdiv
            const float4 u = ld4(SM::PRIM + o2 + raw_place);
            const float2 x = *reinterpret_cast<const float2*>(smem + SM::XI + (t0 >> 1));
            const F2 rho = vmul(vset<F2>(src), mk2(u.x, u.y));
            const float px = ((float)i + 0.5f) * dx, py0 = ((float)j + 0.5f) * dx, py1 = ((float)(j + 1) + 0.5f) * dx;
            const float pz = ((float)k + 0.5f) * dx;
            if (wind > 0.0f && (x.x > 0.01f || x.y > 0.01f)) {
                // an inactive star adds exactly nothing (a zero weight at the origin: no branch, so that
                // four stars' loads and reciprocals are under way together)
                F2 ax = vset<F2>(0.0f), ay = ax, az = ax;
#pragma unroll 4
                for (int s = 0; s < nstars; ++s) {
                    float4 st = __ldg(&L.sw[s].w);
                    if (!(st.w > 0.0f)) st = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const float rx = px - st.x, rz = pz - st.z;
                    const F2 ry = mk2(py0 - st.y, py1 - st.y);
                    const F2 r2 = vadd(vfma(ry, ry, vset<F2>(rx * rx + rz * rz)), vset<F2>(0.0004f));
                    const F2 f = vmul(vset<F2>(st.w), vrcp(vmul(r2, mk2(sqrtf(lo(r2)), sqrtf(hi(r2))))));
                    ax = vfma(vset<F2>(rx), f, ax);
                    ay = vfma(ry, f, ay);
                    az = vfma(vset<F2>(rz), f, az);
                }
                // cells at or below an ionized fraction of 0.01 take no wind
                const F2 wx = vmul(rho, mk2(x.x > 0.01f ? wind * x.x : 0.0f, x.y > 0.01f ? wind * x.y : 0.0f));
                S.n = vfma(wx, ax, S.n);
                S.s = vfma(wx, ay, S.s);
                S.t = vfma(wx, az, S.t);
            }
            if (n_jet > 0) {
                float jx[2] = {0.0f, 0.0f}, jy[2] = {0.0f, 0.0f}, jz[2] = {0.0f, 0.0f};
                for (int m = 0; m < n_jet; ++m) {
                    const int s = jet_ix[m];
                    const float4 jt = __ldg(&L.sw[s].jet), st = __ldg(&L.sw[s].w);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float rx = px - st.x, ry = (h ? py1 : py0) - st.y, rz = pz - st.z;
                        const float r = sqrtf((rx * rx + ry * ry) + rz * rz);
                        if (r < jet_r && r > 1e-6f) {
                            const float cth = (((0.0f + rx * jt.x) + ry * jt.y) + rz * jt.z) / r;
                            if (fabsf(cth) > jet_cos) {
                                const float f = (cth > 0.0f ? 1.0f : -1.0f) * jt.w * pulse / (r * r + 0.0004f);
                                jx[h] = jx[h] + jt.x * f; jy[h] = jy[h] + jt.y * f; jz[h] = jz[h] + jt.z * f;
                            }
                        }
                    }
                }
                S.n = vfma(rho, mk2(jx[0], jx[1]), S.n);
                S.s = vfma(rho, mk2(jy[0], jy[1]), S.s);
                S.t = vfma(rho, mk2(jz[0], jz[1]), S.t);
            }
        }
        const bool ok = mbar_wait_limited(&bar[SEC ? 1 : 0], SEC ? ph0 >> 1 : ph0 & 1u, &L.wait_limit);
        if (ok) ph0 ^= SEC ? 2u : 1u;            // a timed-out wait keeps its parity for the abort wait
        // ---- convert plane p: the own pair, and on three warps one pair of the halo strips
        auto convert = [&](int r0, int r1, int o, auto own_cells) -> St<F2> {
            auto rd = [&](int f) {
                return mk2(*reinterpret_cast<const float*>(smem + RAW + f * SM::RAW_FIELD + r0),
                           *reinterpret_cast<const float*>(smem + RAW + f * SM::RAW_FIELD + r1));
            };
            const F2 w0 = rd(0), w1 = rd(1), w2 = rd(2), w3 = rd(3), x = rd(4);
            if (decltype(own_cells)::value) {
                st4(SM::PRIM + o + raw_place, w0, w1);
                st4(SM::PRIM + o + raw_place + SM::PER, w2, w3);
                *reinterpret_cast<float2*>(smem + SM::XI + (t0 >> 1)) = make_float2(lo(x), hi(x));
            }
            const F2 r = vmax(w0, floor_), ri = vrcp(r);
            const St<F2> q = {r, vmul(w1, ri), vmul(w2, ri), vmul(w3, ri)};
            const F2 c2 = vfma(x, vset<F2>(dci2), vset<F2>(cn2));
            st4(SM::PRIM + o, q.r, q.n);
            st4(SM::PRIM + o + SM::PLANE, q.s, q.t);
            st4(SM::PRIM + o + 2 * SM::PLANE, c2, mk2(sqrtf(lo(c2)), sqrtf(hi(c2))));
            return q;
        };
        if (has_halo) convert(raw_halo0, raw_halo1, o0 + halo, std::false_type{});
        const St<F2> q = convert(raw_own0, raw_own1, o0, std::true_type{});
        // the only barrier of a plane: plane p's slot and the faces of the step before are complete,
        // and the raw slot is read.  A wait that gave up is told by a flag: cheaper than a barrier that
        // reduces.  A warp still reading it here may see it set for the next step and leave one step early;
        // it meets no further barrier, and the others' barrier does not wait for warps that have exited.
        volatile unsigned* gave_up = reinterpret_cast<unsigned*>(smem + SM::FLAG);
        if (!ok) *gave_up = 1u;
        __syncthreads();
        if (*gave_up) return false;
        if (w_issue && p < P1) {
            // into the raw slot just read: the next plane (the first step's: the third, the second being
            // under way; the second step read another slot)
            if (!SEC) issue(p == P0 ? p + 2 : p + 1, SM::RAW, &bar[0]);
            if (STAGE2 && L.map_u0 >= 0 && L.maps && p >= i0 && p < i_end) {     // u0 of plane p, read a step on
#pragma unroll
                for (int f = 0; f < 4; ++f) tma_prefetch_3d(&L.maps[L.map_u0 + f], max(k0 - 4, 0), max(j0 - 2, 0), p);
            }
        }
        // ---- x: the limited slope of plane p-1 and the face (p-2)+1/2
        St<F2> fx;
        {
            const St<F2> q1 = load(o1);
            const St<F2> sx = slopes<LM>(diff(q1, load(o2)), diff(q, q1));
            if (FULL) fx = flux<SOLVER>(Lx, load_c(o2), down(q1, sx), load_c(o1), floor_);
            Lx = up(q1, sx);
        }
        // ---- update of plane i = p - 2 (nebula3d.py:87-151)
        if (FULL) {
            const float4 fm = ld4(SM::FY + t0);              // the y face below the pair
            S.r = mk2(lo(S.r) + (f1.r - fm.x), hi(S.r));
            S.n = mk2(lo(S.n) + (f1.n - fm.y), hi(S.n));
            S.s = mk2(lo(S.s) + (f1.s - fm.z), hi(S.s));
            S.t = mk2(lo(S.t) + (f1.t - fm.w), hi(S.t));
            // a U0 + b (U + dt dU) as (a + b) U + (a (U0 - U) + b dt dU): U0 - U is small beside U, so the sum
            // is rounded once at U's size (in stage 1 U0 is U).  The density's error against float64 after three
            // steps is 0.8 times that of the sum as written; a U0 + b U formed a step early, which keeps 8
            // registers free and is 4% faster, makes it 1.15 times
            const St<F2> u = state(SM::PRIM + o2 + raw_place, SM::PER);
            const F2 kd = vset<F2>(kdiv), ab2 = vset<F2>(ab), a2 = vset<F2>(L.a);
            auto comb = [&](F2 fn, F2 fo, F2 sd, F2 un, F2 uo) {
                const F2 dv = vadd(vsub(fn, fo), sd);
                return STAGE2 ? vfma(ab2, un, vfma(kd, dv, vmul(a2, vsub(uo, un)))) : vfma(kd, dv, vmul(ab2, un));
            };
            const F2 o[4] = {comb(fx.r, fxp.r, S.r, u.r, u0[0]), comb(fx.n, fxp.n, S.n, u.n, u0[1]),
                             comb(fx.s, fxp.s, S.s, u.s, u0[2]), comb(fx.t, fxp.t, S.t, u.t, u0[3])};
            fxp = fx;
            const F2 r = vmax(o[0], floor_);
            // one reciprocal for the three velocities and the max speed; the speed cap without a branch
            // (min(1, vmax / |v|): exactly 1 below the cap)
            const F2 ri = vrcp(r);
            F2 vx = vmul(o[1], ri), vy = vmul(o[2], ri), vz = vmul(o[3], ri);
            const F2 v2 = vfma(vz, vz, vfma(vy, vy, vmul(vx, vx)));
            const F2 cf = mk2(fminf(1.0f, vcap * rsqrtf(lo(v2))), fminf(1.0f, vcap * rsqrtf(hi(v2))));
            vx = vmul(vx, cf); vy = vmul(vy, cf); vz = vmul(vz, cf);
            const F2 m1 = vmul(r, vx), m2 = vmul(r, vy), m3 = vmul(r, vz);
            const Idx cell = (Idx)i * plane + at, cell1 = cell + up_row;
            const bool st0 = in0 && p >= i0 + 2, st1 = in1 && p >= i0 + 2;
            if (st0) {
                L.out[0][cell] = lo(r); L.out[1][cell] = lo(m1); L.out[2][cell] = lo(m2); L.out[3][cell] = lo(m3);
            }
            if (st1) {
                L.out[0][cell1] = hi(r); L.out[1][cell1] = hi(m1); L.out[2][cell1] = hi(m2); L.out[3][cell1] = hi(m3);
            }
            if (STAGE2) {                        // nebula3d.py:158-162 on the new state
                const F2 w1 = vmul(m1, ri), w2 = vmul(m2, ri), w3 = vmul(m3, ri), cc = load_c(o2).c;
                if (st0) vmax_local = fmaxf(fabsf(lo(w1)) + fabsf(lo(w2)) + fabsf(lo(w3)) + lo(cc), vmax_local);
                if (st1) vmax_local = fmaxf(fabsf(hi(w1)) + fabsf(hi(w2)) + fabsf(hi(w3)) + hi(cc), vmax_local);
            }
            if (STAGE2 && p < P1) {              // u0 of the next step's plane: on its way during the faces
                const Idx next = cell + plane, next1 = next + up_row;
#pragma unroll
                for (int f = 0; f < 4; ++f) u0[f] = mk2(L.u0[f][next], L.u0[f][next1]);
            }
        }
        // ---- y and z faces of plane p - 1
        if (FULL) {
            const St<F2> q1 = load(o1);
            const Cs<F2> c1 = load_c(o1);
            {
                // z: the state below the upper face comes from the next lane, the face below from the
                // previous one (lanes 31 and 0: from the edge work of the step before), through the
                // warp's own exchange rows: 8 accesses where shuffles take 16 and the edges' selects
                const St<F2> qz = z_order(q1), qb = z_order(load(o1 + 16));
                const St<F2> sz = slopes<LM>(diff(qz, z_order(load(o1 - 16))), diff(qb, qz));
                const int x = SM::ZX + (t0 & (SM::PER - 1));
                auto put = [&](const St<F2>& v) {
                    st4(x, v.r, v.n);
                    st4(x + SM::ZX_HALF, v.s, v.t);
                };
                put(down(qz, sz));
                __syncwarp();
                const St<F2> f = flux<SOLVER>(up(qz, sz), c1, state(z_up, SM::ZX_HALF), load_c(o1 + 16), floor_);
                __syncwarp();                    // every lane has read its lower state
                put(f);
                __syncwarp();
                S = z_order(diff(f, state(z_dn, SM::ZX_HALF)));
            }
            {
                // y: the faces above row j (between the pair's rows) and above row j + 1
                const St<F2> qy = y_order(q1);
                const St<float> qm = hi(y_order(load(o1 - ROW)));
                const St<F2> pn = y_order(load(o1 + ROW));
                const Cs<F2> cn = load_c(o1 + ROW);
                const St<float> dA = diff(lo(qy), qm), dB = diff(hi(qy), lo(qy)), dC = diff(lo(pn), hi(qy));
                const St<float> dD = diff(hi(pn), lo(pn));
                const St<float> sB = slopes<LM>(dB, dC);
                const St<F2> f = y_order(flux<SOLVER>(up(qy, mk2(slopes<LM>(dA, dB), sB)), c1,
                                                      mk2(down(hi(qy), sB), down(lo(pn), slopes<LM>(dC, dD))),
                                                      {mk2(hi(c1.c2), lo(cn.c2)), mk2(hi(c1.c), lo(cn.c))}, floor_));
                f1 = lo(f);
                const St<float> f2 = hi(f);
                S.r = mk2(lo(S.r), hi(S.r) + (f2.r - f1.r));
                S.n = mk2(lo(S.n), hi(S.n) + (f2.n - f1.n));
                S.s = mk2(lo(S.s), hi(S.s) + (f2.s - f1.s));
                S.t = mk2(lo(S.t), hi(S.t) + (f2.t - f1.t));
                if (tj < NP - 1)
                    *reinterpret_cast<float4*>(smem + SM::FY + (t0 ^ SM::PER) + TK * 16) =
                        make_float4(f2.r, f2.n, f2.s, f2.t);
            }
        }
        // ---- the z face before the tile and the states after it of plane p, for the next step
        if (w_zedge && p >= i0 && p < i_end && tk < 2 * NP) {
            const int pr = tk & (NP - 1), o = o0 - own + (pr + 1) * ROW + (tk < NP ? 16 : 33 * 16);
            const St<F2> qa = z_order(load(o)), qb = z_order(load(o + 16)), qc = z_order(load(o + 32));
            const St<F2> dab = diff(qb, qa);
            St<F2> R = down(qb, slopes<LM>(dab, diff(qc, qb)));          // the lower state of cell k0 or k0+32
            if (tk < NP)
                R = flux<SOLVER>(up(qa, slopes<LM>(diff(qa, z_order(load(o - 16))), dab)), load_c(o), R, load_c(o + 16),
                                 floor_);
            const int e = SM::ZE + (t0 >= SM::PER ? SM::ZE_PAR : 0) + (tk < NP ? 0 : SM::ZE_SIDE) + pr * 16;
            st4(e, R.r, R.n);
            st4(e + SM::ZX_HALF, R.s, R.t);
        }
        // ---- the y face below the tile, (j0-1)+1/2, of plane p - 1
        if (FULL && w_yedge) {
            const int o = o1 - own + (tk + 2) * 16;
            const St<F2> pa = y_order(load(o)), pb = y_order(load(o + ROW));
            const Cs<F2> ca = load_c(o), cb = load_c(o + ROW);
            const St<float> dm = diff(lo(pb), hi(pa));
            const St<float> f = y_order(flux<SOLVER, float>(
                up(hi(pa), slopes<LM>(diff(hi(pa), lo(pa)), dm)), {hi(ca.c2), hi(ca.c)},
                down(lo(pb), slopes<LM>(dm, diff(hi(pb), lo(pb)))), {lo(cb.c2), lo(cb.c)}, floor_));
            *reinterpret_cast<float4*>(smem + SM::FY + ((t0 ^ SM::PER) & SM::PER) + tk * 16) =
                make_float4(f.r, f.n, f.s, f.t);
        }
        const int o3 = o2;
        o2 = o1;
        o1 = o0;
        o0 = o3;
        t0 ^= SM::PER;
        z_up ^= z_up_par;
        z_dn ^= z_dn_par;
        return true;
    };
    if (!step(P0, std::false_type{}, std::false_type{}) || !step(P0 + 1, std::false_type{}, std::true_type{})) {
        if (tid == 0) mbar_wait_limited(&bar[1], ph0 >> 1, &L.wait_limit);     // the second plane's load, still in flight
        failed = true;
        return;
    }
    if (!step(P0 + 2, std::false_type{}, std::false_type{})) { failed = true; return; }
    n_jet = *n_jet_p;
    for (int p = P0 + 3; p <= P1; ++p)
        if (!step(p, std::true_type{}, std::false_type{})) { failed = true; return; }
    if (STAGE2 && L.smax_bits) hydro_smax(L, vmax_local, reinterpret_cast<float*>(smem + SM::FY), NP);
}

}  // namespace
