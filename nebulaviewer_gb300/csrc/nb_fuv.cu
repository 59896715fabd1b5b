// Dust-attenuated FUV field G0 = sum_star L exp(-tau_FUV) / r^2.  Follows
// nebula3d.py:320-352 (cast_fuv: per-ray dust optical depth binned on a coarse spherical
// grid att[r, u, phi]) and nebula3d.py:355-388 (apply_fuv: trilinear att / r^2 per cell),
// as driven by sim.py:949-985 (fuv_field, fp16 store of G0).
//
// GB300 design: cast_fuv marches a ray with a group of G lanes, the optical depth being an
// inclusive group scan over a Kahan-compensated carry; a lane that crosses into new radial
// bins writes them, and a ray stops once its optical depth passes 120 (exp(-tau) is 0.0f from
// there on: its remaining bins are written as 0).  Density and ionized fraction are sampled at the
// same corners, so they are first packed as (rho, xi) pairs into free scratch: one 8-byte gather per
// corner.  All rays of all active stars are one launch, into one attenuation table per star.  An
// entry is the pair (att(r), att(min(r + 1, nr - 1))) as one float2 (the ray writes each bin into
// its own pair and its lower neighbour's), so a trilinear sample of apply_fuv is four 8-byte gathers
// instead of eight 4-byte ones; values and arithmetic are those of the plain table
// (NB_TUNE_FUV_PAIRS = 0), bit for bit, in whichever order the entries lie.  apply_fuv accumulates
// every active star for a cell in one register, in the reference's star order (so the float32 sum
// is the reference's), and stores G0 once as fp16.
//
// Both kernels were bound by L1 wavefronts (a gather takes one per 128-byte line it touches).  The
// table lies in bricks of 4 u x 4 r, one line each (a ray still writes whole 32-byte sectors), the
// rays of a brick are cast together, and a warp of the apply takes 4 x 2 x 4 cells instead of 32
// along k: 21 lines per cell group and star instead of 48.  apply_fuv at 64^3 / 192^3 / 256^3 /
// 384^3 with six stars: 29 / 262 / 563 / 1954 -> 24 / 178 / 396 / 1299 us (cells alone 458 at
// 256^3), now issue bound (88%); cast_fuv with its pack 630 -> 589 us at 256^3 (whole pairs where
// a ray fills its last bins), level at 128^3 and dearer below, where the table keeps the plain order
// (nb_fuv_bricks).  The cast is bound by L1 (90% of its data pipe) and by the chain of a segment (loads,
// scan, ballots).  The pack keeps to 8 B a cell, stage planes 0-1, because a render pack's voxels lie in
// planes 2-3: each cell packed with its upper neighbour (four 16-byte gathers a sample) was 3% faster.
#include "nb_rayutil.cuh"

namespace {

__global__ void __launch_bounds__(256) pack_rx_kernel(const float* __restrict__ rho, const float* __restrict__ xi,
                                                      float2* __restrict__ rx, long long n) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        rx[q] = make_float2(rho[q], xi[q]);
}

// An entry's offset is the sum of three: of its phi, its u and its r.
template <int L>
__device__ __forceinline__ int fuv_phi(int ip, int nu, int nr) {
    return ip * (L == FUV_BRICKS ? nu * nr : nr);
}
template <int L>
__device__ __forceinline__ int fuv_u(int iu, int nphi, int nr) {
    return L == FUV_BRICKS ? 4 * iu + (iu >> 2) * (4 * nr - 16) : iu * (nphi * nr);
}
template <int L>
__device__ __forceinline__ int fuv_r(int ir) {
    return L == FUV_BRICKS ? ir + 12 * (ir >> 2) : ir;
}

template <int G, int L>
__global__ void __launch_bounds__(256, 5) cast_fuv_kernel(const NbConst* __restrict__ c, const NbStarW* __restrict__ sw,
                                                       const float4* __restrict__ dirs,
                                                       const float2* __restrict__ rx,
                                                       float* __restrict__ att, int nstars,
                                                       const float* star_override, float tau_cut) {
    const int nr = c->fnr, nu = c->fnu, nphi = c->fnphi, nray = nu * nphi;
    const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) / G * G));
    if (gid >= (long long)nray * nstars) return;
    // below 2^32 (fnu * fnphi * nstars; nb_create checks it): 32-bit division
    const int s = (int)((unsigned)gid / (unsigned)nray), ray = (int)((unsigned)gid - (unsigned)s * (unsigned)nray);
    float sx, sy, sz;
    if (star_override) {
        sx = star_override[0]; sy = star_override[1]; sz = star_override[2];
    } else {
        const NbStarW w = sw[s];
        if (!w.active) return;
        sx = w.w.x; sy = w.w.y; sz = w.w.z;
    }
    // bricks: four u in turn, so that the rays of a line of the table are cast together
    const int iu = L == FUV_BRICKS ? ray / (4 * nphi) * 4 + (ray & 3) : ray / nphi;
    const int ip = L == FUV_BRICKS ? (ray >> 2) % nphi : ray % nphi;
    float* const table = L == FUV_REF ? att : att + (L == FUV_PLAIN ? 1 : 2) * ((long long)s * nray * nr);
    const int at = fuv_phi<L>(ip, nu, nr) + fuv_u<L>(iu, nphi, nr);
    auto put = [&](int b, float v) {
        if (L == FUV_REF) {
            att[((long long)b * nu + iu) * nphi + ip] = v;
        } else if (L == FUV_PLAIN) {
            table[at + b] = v;
        } else {                                 // bin b is pair b's .x and pair b-1's .y
            float* p = table + 2 * (long long)at;
            p[2 * fuv_r<L>(b)] = v;
            if (b > 0) p[2 * fuv_r<L>(b - 1) + 1] = v;
            if (b == nr - 1) p[2 * fuv_r<L>(b) + 1] = v;
        }
    };
    // every bin from b0 on: whole pairs
    auto fill = [&](int b0, float v) {
        if (L == FUV_REF || L == FUV_PLAIN) {
            for (int b = b0 + lane; b < nr; b += G) put(b, v);
        } else {
            float2* p = reinterpret_cast<float2*>(table) + at;
            for (int b = b0 + lane; b < nr; b += G) p[fuv_r<L>(b)] = make_float2(v, v);
            if (lane == 0 && b0 > 0 && b0 < nr) p[fuv_r<L>(b0 - 1)].y = v;
        }
    };
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const float dx = c->dx, inv_dx = c->inv_dx, dr = c->dr_f, binr = c->binr_f, kappa = c->kappa_f;
    const bool pow2 = c->dx_pow2 != 0;
    const float4 d = dirs[iu * nphi + ip];
    float t0, t1;
    nb_box_range(sx, sy, sz, d.x, d.y, d.z, c->bmax, t0, t1);
    const int n0 = trunc_i(t0 / dr);
    const int n1 = min(c->nsteps, trunc_i(t1 / dr) + 2);
    float hi = 0.0f, comp = 0.0f;      // Kahan-compensated optical depth carried between segments
    int ib = 0;                        // first bin not yet written
    bool stopped = false;
    for (int base = n0; base < n1; base += G) {
        const int n = base + lane;
        const bool valid = n < n1;
        const float r = ((float)n + 0.5f) * dr;
        float dtau = 0.0f;
        int nb = ib;
        if (valid) {
            const float qx = sx + d.x * r, qy = sy + d.y * r, qz = sz + d.z * r;
            const float2 nx_i = sample_n2(rx, nx, ny, nz, qx, qy, qz, dx, inv_dx, pow2);   // (n_tot, x_i)
            dtau = kappa * nx_i.x * (1.0f - 0.92f * nx_i.y) * dr;
            nb = trunc_i(r / binr);
        }
        float incl = dtau;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const float v = __shfl_up_sync(gmask, incl, o, G);
            if (lane >= o) incl = incl + v;
        }
        const float tau = hi + (incl - comp);
        // bins [prev, min(nb, nr)) take exp(-tau) of this sample (nb never decreases along a ray)
        int prev = __shfl_up_sync(gmask, nb, 1, G);
        if (lane == 0) prev = ib;
        const bool stop = valid && nb >= nr;
        // Past tau_cut (> 0) exp(-tau) is 0.0f (exp(-120) ~ 8e-53 lies far below the least float
        // denormal) and stays 0 along the ray (dtau >= 0): the bins from here on are all 0.
        const bool dark = tau_cut > 0.0f && valid && tau > tau_cut;
        const unsigned bal = __ballot_sync(gmask, stop || dark);
        const unsigned mine = G == 32 ? bal : (bal >> ((threadIdx.x & 31) / G * G)) & ((1u << G) - 1u);
        const int first_stop = mine ? __ffs(mine) - 1 : G;
        if (valid && lane <= first_stop && nb > prev) {
            const float v = expf(-tau);
            const int e = min(nb, nr);
            for (int b = prev; b < e; ++b) put(b, v);
        }
        if (mine) {                              // a lane ran out of bins or into the dark
            const int e_first = __shfl_sync(gmask, min(nb, nr), first_stop, G);
            fill(e_first, 0.0f);
            stopped = true;
            break;
        }
        const int last = min(G, n1 - base) - 1;
        ib = __shfl_sync(gmask, nb, last, G);
        const float total = __shfl_sync(gmask, incl, G - 1, G);
        const float y = total - comp;
        const float tsum = hi + y;
        comp = (tsum - hi) - y;
        hi = tsum;
    }
    if (!stopped) fill(ib, expf(-(hi - comp)));
}

template <bool HALF, int L>
__global__ void __launch_bounds__(256, 6) apply_fuv_kernel(const NbConst* __restrict__ c, const NbStarW* __restrict__ sw,
                                                        const float* __restrict__ att, int nstars,
                                                        void* __restrict__ g0, int li) {
    __shared__ float4 st[NB_MAX_STARS];
    __shared__ float lum[NB_MAX_STARS];
    __shared__ int act[NB_MAX_STARS];
    __shared__ float4 rowtab[8][NB_ROW_STARS + 1];       // + 1: the eight rows of a warp in different banks
    for (int s = threadIdx.y * blockDim.x + threadIdx.x; s < nstars; s += blockDim.x * blockDim.y) {
        st[s] = sw[s].w;
        lum[s] = sw[s].lum_f;
        act[s] = sw[s].active;
    }
    __syncthreads();
    const int nx = c->nx, ny = c->ny, nz = c->nz, nr = c->fnr, nu = c->fnu, nphi = c->fnphi;
    const float dx = c->dx, binr = c->binr_f;
    const float two_pi = 2.0f * pi_f();
    const int colmul = fuv_phi<L>(1, nu, nr);   // offsets within a star's table are below 2^31
    const int C_plane_on = c->plane_on;
    const float* C_plane_g0 = c->plane_g0;
    // a block takes 2^li x 2^lj rows, a warp 4 cells of each of them at a time
    const int lj = 3 - li, nbj = (ny + (1 << lj) - 1) >> lj, bi = blockIdx.x / nbj, bj = blockIdx.x - bi * nbj;
    // (without pairs 32 cells of one row: four stars at 128^3 88 us, 98 with two stars in flight, 104 with the patch)
    const int row = L == FUV_PLAIN ? threadIdx.y : threadIdx.x >> 2;
    // per-row azimuth constants (star_row_table): the same values the per-cell form computes
    float4* tab = nullptr;
    if (nstars <= NB_ROW_STARS) {
        const int r = threadIdx.y, i = (bi << li) + (r >> lj), j = (bj << lj) + (r & ((1 << lj) - 1));
        star_row_table(st, act, nstars, ((float)i + 0.5f) * dx, ((float)j + 0.5f) * dx, nphi, colmul, rowtab[r]);
        __syncthreads();
        tab = rowtab[row];
    }
    const int wi = (bi << li) + (row >> lj), wj = (bj << lj) + (row & ((1 << lj) - 1));
    if (wi >= nx || wj >= ny) return;
    const float px = ((float)wi + 0.5f) * dx, py = ((float)wj + 0.5f) * dx;
    const long long base = ((long long)wi * ny + wj) * nz;
    for (int k = L == FUV_PLAIN ? threadIdx.x : threadIdx.y * 4 + (threadIdx.x & 3); k < nz; k += 32) {
        const long long q = base + k;
        const float pz = ((float)k + 0.5f) * dx;
        float g = 0.0f;
        for (int s = 0; s < nstars; ++s) {
            if (!act[s]) continue;
            const float4 sp = st[s];
            const float rz = pz - sp.z;
            float r, tp;
            int pw[2];
            if (tab) {
                const float4 tb = tab[s];
                r = fmaxq(sqrtf(tb.x + rz * rz), 1e-6f);                          // (rx^2 + ry^2) + rz^2
                tp = tb.y;
                pw[0] = __float_as_int(tb.z);
                pw[1] = __float_as_int(tb.w);
            } else {
                const float rx = px - sp.x, ry = py - sp.y;
                r = fmaxq(sqrtf((rx * rx + ry * ry) + rz * rz), 1e-6f);             // 0 + x*x == x*x
                float phi = atan2f(ry, rx);
                if (phi < 0.0f) phi = phi + two_pi;
                const float fp = phi / two_pi * (float)nphi - 0.5f;
                const int ip = (int)floorf(fp);
                tp = fp - (float)ip;
                pw[0] = wrap_index(ip, nphi) * colmul;
                pw[1] = wrap_index(ip + 1, nphi) * colmul;
            }
            const float u = rz / r;
            const float fr = r / binr - 0.5f;
            const float fu = (u + 1.0f) * 0.5f * (float)nu - 0.5f;
            const float flr = floorf(fr), flu = floorf(fu);
            const int ir = (int)flr, iu = (int)flu;
            const float tr = fr - flr, tu = fu - flu;
            const long long tab0 = (long long)s * nu * nphi * nr;
            const int ua = fuv_u<L>(iclampd(iu, 0, nu - 1), nphi, nr), ub = fuv_u<L>(iclampd(iu + 1, 0, nu - 1), nphi, nr);
            float v[2][2][2];                    // [r corner][u corner][phi corner]
            if (L != FUV_PLAIN) {
                // pair rc = (att(rc), att(min(rc + 1, nr - 1))): the two r corners, except at ir = -1,
                // where both clamp to r = 0 (the pair's .x)
                const float2* ap = reinterpret_cast<const float2*>(att) + tab0;
                const int rc = fuv_r<L>(iclampd(ir, 0, nr - 1));
#pragma unroll
                for (int bb = 0; bb < 2; ++bb)
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        const float2 pr = __ldg(ap + ((bb ? ub : ua) + pw[cc] + rc));
                        v[0][bb][cc] = pr.x;
                        v[1][bb][cc] = ir < 0 ? pr.x : pr.y;
                    }
            } else {
                const float* as = att + tab0;
#pragma unroll
                for (int aa = 0; aa < 2; ++aa)
#pragma unroll
                    for (int bb = 0; bb < 2; ++bb)
#pragma unroll
                        for (int cc = 0; cc < 2; ++cc) {
                            const int rr = iclampd(ir + aa, 0, nr - 1);
                            v[aa][bb][cc] = __ldg(as + ((bb ? ub : ua) + pw[cc] + rr));
                        }
            }
            float acc = 0.0f;
#pragma unroll
            for (int aa = 0; aa < 2; ++aa)
#pragma unroll
                for (int bb = 0; bb < 2; ++bb)
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        const float wgt = (aa == 0 ? 1.0f - tr : tr) * (bb == 0 ? 1.0f - tu : tu) * (cc == 0 ? 1.0f - tp : tp);
                        acc = acc + wgt * v[aa][bb][cc];
                    }
            const float r2 = fmaxq(r * r, 0.0004f);
            const float term = lum[s] * acc / r2;      // rounded before the sum in both builds
            g = __fadd_rn(g, term);                     // the reference's star order
        }
        if (C_plane_on) g = g + __ldg(C_plane_g0 + q);      // the -x plane source, after the stars
        if (HALF)
            reinterpret_cast<__half*>(g0)[q] = __float2half_rn(g);
        else
            reinterpret_cast<float*>(g0)[q] = g;
    }
}

// FUV of the -x plane source (no reference counterpart): per column, the dust optical depth
// of nebula3d.py:343 summed along +x to each cell centre; G0 term = L exp(-tau).
__global__ void __launch_bounds__(256) plane_fuv_kernel(const NbConst* __restrict__ c, const float* __restrict__ rho,
                                                        const float* __restrict__ xi, float* __restrict__ g) {
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= ny * nz) return;
    const float kappa = c->kappa_f, dx = c->dx, lum = c->plane_lum_f;
    const long long plane = (long long)ny * nz;
    float tau = 0.0f;
    for (int i = 0; i < nx; ++i) {
        const long long q = i * plane + col;
        const float dtau = kappa * __ldg(rho + q) * (1.0f - 0.92f * __ldg(xi + q)) * dx;
        g[q] = lum * expf(-(tau + 0.5f * dtau));
        tau = tau + dtau;
    }
}

}  // namespace

cudaError_t nb_launch_plane_fuv(const NbConst* c, const float* rho, const float* xi, float* g, int ny, int nz,
                                cudaStream_t s) {
    const int cols = ny * nz;
    plane_fuv_kernel<<<(cols + 255) / 256, 256, 0, s>>>(c, rho, xi, g);
    return cudaGetLastError();
}

// The layout of an instance's table where it holds pairs.  Bricks where they need no padding (a table is then
// as large as in the other orders; every ray budget a simulation chooses for itself is a multiple of 4) and
// where the cells that read it are many enough: a ray's bins then lie in four times as many lines, which costs
// the cast what the table's size says, and the apply gains what the cells' number says.  Cast + apply of six
// stars, bricks and [u][phi][r], at entries / cells of 1024 (16^3) 97 and 84 us, 16 (64^3) 156 and 156, 8
// (80^3) 187 and 191, 5 (96^3) 213 and 228, 2 (128^3) 285 and 323; thin grids, three stars: 12 x 300 x 200 at
// 11 119 and 113, 16 x 512 x 64 at 8 79 and 72, 512 x 512 x 4 at 4 136 and 138.  ([u][phi][r] with the cells
// along k, before the bricks: 87 at 16^3, 164 at 64^3, 232 at 96^3, 85 at 16 x 512 x 64.)
int nb_fuv_bricks(int fnr, int fnu, int fnphi, long long ncell) {
    return fnr % 4 == 0 && fnu % 4 == 0 && (long long)fnr * fnu * fnphi <= 6 * ncell;
}

cudaError_t nb_launch_cast_fuv(const NbConst* c, const NbStarW* sw, const float4* dirs, const float* rho,
                               const float* xi, float* att, int nstars, int group, const float* star_override,
                               cudaStream_t s, int fnu, int fnphi, void* rx_scratch, long long ncell,
                               float tau_cut, int layout) {
    float2* rx = static_cast<float2*>(rx_scratch);
    {
        const long long b = (ncell + 255) / 256;
        pack_rx_kernel<<<(int)(b < 152LL * 16 ? (b < 1 ? 1 : b) : 152LL * 16), 256, 0, s>>>(rho, xi, rx, ncell);
    }
    const long long threads = (long long)fnu * fnphi * nstars * group;
    const int blocks = (int)((threads + 255) / 256);
#define NB_FUV_LAUNCH(G, L) \
    cast_fuv_kernel<G, L><<<blocks, 256, 0, s>>>(c, sw, dirs, rx, att, nstars, star_override, tau_cut)
#define NB_FUV_GROUPS(L)                          \
    switch (group) {                              \
        case 8: NB_FUV_LAUNCH(8, L); break;       \
        case 16: NB_FUV_LAUNCH(16, L); break;     \
        default: NB_FUV_LAUNCH(32, L); break;     \
    }
    if (layout == FUV_REF) {
        NB_FUV_LAUNCH(32, FUV_REF);
    } else if (layout == FUV_BRICKS) {
        NB_FUV_GROUPS(FUV_BRICKS)
    } else if (layout == FUV_PAIRS) {
        NB_FUV_GROUPS(FUV_PAIRS)
    } else {
        NB_FUV_GROUPS(FUV_PLAIN)
    }
#undef NB_FUV_GROUPS
#undef NB_FUV_LAUNCH
    return cudaGetLastError();
}

cudaError_t nb_launch_apply_fuv(const NbConst* c, const NbStarW* sw, const float* att, int nstars, void* g0,
                                cudaStream_t s, int nx, int ny, int half, int layout) {
    // 4 x 2 rows a block, or another split where that leaves far more lanes without a row (thin and small
    // grids): 2 x 4 and 1 x 8 rows took 10% longer at 192^3 and 256^3
    int li = 2, blocks = ((nx + 3) / 4) * ((ny + 1) / 2);
    const int b2 = ((nx + 1) / 2) * ((ny + 3) / 4), b1 = nx * ((ny + 7) / 8);
    if (b2 < blocks - blocks / 10) li = 1, blocks = b2;
    if (b1 < blocks - blocks / 10) li = 0, blocks = b1;
#define NB_FUV_APPLY(L)                                                                                   \
    (half ? apply_fuv_kernel<true, L><<<blocks, dim3(32, 8), 0, s>>>(c, sw, att, nstars, g0, li)          \
          : apply_fuv_kernel<false, L><<<blocks, dim3(32, 8), 0, s>>>(c, sw, att, nstars, g0, li))
    if (layout == FUV_BRICKS) NB_FUV_APPLY(FUV_BRICKS);
    else if (layout == FUV_PAIRS) NB_FUV_APPLY(FUV_PAIRS);
    else NB_FUV_APPLY(FUV_PLAIN);
#undef NB_FUV_APPLY
    return cudaGetLastError();
}
