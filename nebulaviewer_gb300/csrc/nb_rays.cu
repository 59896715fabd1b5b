// Stromgren ionization: per-star ray casting of the recombination column, the front
// apply (max-merge of xi, min-merge of the signed front distance) and the 7-point
// smoothing of xi.  Follows nebula3d.py:195-315 (sample_n, box_range, cast_rays, rf_at,
// apply_front, smooth_xi) as driven by sim.py:927-947 (ionize).
//
// GB300 design:
//  * cast_rays: a group of G lanes (1 to 32; 1 by default) marches one ray, G consecutive
//    samples at a time; the recombination column sum(n^2 r^2 dr) is added to a Kahan-compensated
//    carry (G > 1: an inclusive group scan; two lanes take it from one exchange), and the
//    first sample whose column passes Q is found with one ballot.  That march is warp-uniform: a
//    warp's groups loop together until all are done, and the trilinear sampler has no branches.
//    The one-lane march (cast_ray1) is a plain loop of its own.
//    All rays of all active stars are one launch, a warp a bundle of neighbouring directions.
//  * The front table holds, per (star, phi, u), the pair (rf(u), rf(min(u + 1, nu - 1))) as one
//    float2 (cast_rays writes each front into its own pair and its lower neighbour's), so the
//    bilinear lookup of apply_front is two 8-byte gathers instead of four 4-byte ones; the values
//    and the arithmetic are those of the plain table (NB_TUNE_FRONT_PAIRS = 0), bit for bit.
//  * apply_front: one pass over the grid merges the active stars, in star order, into one
//    register pair per cell (the reference makes S passes).  With up to 32 stars, each star's
//    front-radius range (merged by the ray cast) lets a 32-cell row segment leave out the stars that
//    cannot change its xi or front distance (the same bits).  The float32 front distance is
//    rounded once to the fp16 dfront (sim.py:980-985, 511-514).
//  * smooth_xi writes the final xi and reduces the CFL max speed of the step from it
//    (nebula3d.py:154-162), so an ionizing step needs no separate max-speed pass.
#include <cstring>

#include "nb_f32x2.cuh"
#include "nb_rays_rule.h"
#include "nb_rayutil.cuh"

namespace {

// The place of direction (iu, ip) in the order of the ionizing ray cast.  A warp takes 8 (u) x 4 (phi)
// neighbouring directions where the ray grid divides so: the bundle stays within a few cells, so its rays
// share cache lines and end within a few samples of one another, and its fronts fill whole sectors of the
// [phi][u] table (32 neighbours along phi span an arc ten times as wide).
__device__ __forceinline__ int ray_place(int iu, int ip, int nu, int nphi) {
    if ((nu & 7) || (nphi & 3)) return iu * nphi + ip;
    return (((ip >> 2) * (nu >> 3) + (iu >> 3)) << 5) + (ip & 3) * 8 + (iu & 7);
}

// Ray directions of nebula3d.py:253-256 / 329-332 in float32; cos/sin of the float32 angle
// are evaluated in FP64 and rounded (the correctly rounded float32 value in all but
// vanishingly rare double-rounding cases).  Computed once per ray grid.
__global__ void ray_dirs_kernel(int nu, int nphi, float4* __restrict__ dirs) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nu * nphi) return;
    const int iu = id / nphi, ip = id % nphi;
    const float u = -1.0f + ((float)iu + 0.5f) * 2.0f / (float)nu;
    const float s = sqrtf(fmaxr(1.0f - u * u, 0.0f));
    const float phi = ((float)ip + 0.5f) * 2.0f * pi_f() / (float)nphi;
    const float cph = (float)cos((double)phi), sph = (float)sin((double)phi);
    dirs[id] = make_float4(s * cph, s * sph, u, 0.0f);
}
// The directions in the order of the ionizing ray cast (a kernel of its own: with other stores in
// ray_dirs_kernel the fast build rounds u differently at some nu); .w: the direction's place ip * nu + iu in a
// [phi][u] table, its sign bit set at the first and last u (the cast does no index division).
__global__ void ray_order_kernel(int nu, int nphi, const float4* __restrict__ dirs, float4* __restrict__ out) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nu * nphi) return;
    const int iu = id / nphi, ip = id % nphi;
    const int w = (ip * nu + iu) | (iu == 0 || iu == nu - 1 ? 0x80000000 : 0);
    float4 d = dirs[id];
    d.w = __int_as_float(w);
    out[ray_place(iu, ip, nu, nphi)] = d;
}

// nebula3d.py:247-270 cast_rays: the ray along d of star (sx, sy, sz, Q), G lanes per ray; every
// lane of the group gets the front radius.
template <int G>
__device__ __forceinline__ float cast_ray(const NbConst& C, const float4 d, const float* __restrict__ rho, float sx,
                                         float sy, float sz, float Q, int lane, unsigned gmask, bool live) {
    // Warp-uniform march: every lane of the warp runs the loop until all of its groups are done
    // (`live` false: the group has no ray), a finished group's lanes
    // only carry predicated-off values, so the warp never diverges inside the loop.
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const float dx = C.dx, inv_dx = C.inv_dx, dr = C.dr_f;
    const bool pow2 = C.dx_pow2 != 0;
    float t0, t1;
    nb_box_range(sx, sy, sz, d.x, d.y, d.z, C.bmax, t0, t1);
    const int n0 = trunc_i(t0 / dr);
    const int n1 = min(C.nsteps, trunc_i(t1 / dr) + 2);
    float hi = 0.0f, comp = 0.0f;          // Kahan-compensated column carried between segments
    float rf = C.diag_f;
    bool done = !live || n0 >= n1;
    for (int base = n0;; base += G) {
        if (__all_sync(0xffffffffu, done)) break;
        const int n = base + lane;
        const bool valid = !done && n < n1;
        const float r = ((float)n + 0.5f) * dr;
        const float nv = sample_n(rho, nx, ny, nz, sx + d.x * r, sy + d.y * r, sz + d.z * r, dx, inv_dx, pow2);
        const float inc = valid ? nv * nv * r * r * dr : 0.0f;
        float incl, excl, total, other = 0.0f;
        if (G == 1) {
            incl = inc;
            excl = 0.0f;
            total = inc;
        } else if (G == 2) {
            // one exchange gives the pair's scan: lane 1 adds lane 0's term (inc1 + inc0, the
            // general scan's operation) and both take that sum as the total
            other = __shfl_xor_sync(gmask, inc, 1, 2);
            incl = lane ? inc + other : inc;
            excl = lane ? other : 0.0f;
            total = lane ? incl : other + inc;
        } else {
            incl = inc;
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const float v = __shfl_up_sync(gmask, incl, o, G);
                if (lane >= o) incl = incl + v;
            }
            excl = __shfl_up_sync(gmask, incl, 1, G);
            if (lane == 0) excl = 0.0f;
            total = __shfl_sync(gmask, incl, G - 1, G);
        }
        const float col = hi + (excl - comp);
        const bool cross = valid && (col + inc > Q);
        const unsigned bal = __ballot_sync(0xffffffffu, cross);
        const unsigned mine = G == 32 ? bal : (bal >> ((threadIdx.x & 31) / G * G)) & ((1u << G) - 1u);
        float rfc = 0.0f;
        if (bal) {                               // some group of the warp crossed (warp-uniform)
            if (G <= 2) {
                // the pair's first crossing lane, from the terms both lanes hold
                const int p = G == 1 ? 0 : ((mine & 1u) ? 0 : 1);
                const float inc0 = lane ? other : inc;
                const float rp = ((float)(base + p) + 0.5f) * dr;
                const float colp = hi + ((p ? inc0 : 0.0f) - comp);
                const float incp = p == lane ? inc : other;
                rfc = rp - 0.5f * dr + dr * (Q - colp) / fmaxr(incp, 1e-20f);
            } else {
                const float rfl = r - 0.5f * dr + dr * (Q - col) / fmaxr(inc, 1e-20f);
                rfc = __shfl_sync(gmask, rfl, mine ? __ffs(mine) - 1 : 0, G);
            }
        }
        if (!done) {
            if (mine) {
                rf = rfc;
                done = true;
            } else {
                const float y = total - comp;
                const float tsum = hi + y;
                comp = (tsum - hi) - y;
                hi = tsum;
                done = base + G >= n1;
            }
        }
    }
    return rf;
}

// c + a b, as the build contracts it
__device__ __forceinline__ float mac(float a, float b, float c) {
#if NB_ARITH_FAST
    return fmaf(a, b, c);
#else
    return vadd(c, vmul(a, b));
#endif
}
// sample_n and the sample range out of line: cast_ray1 needs them only near the box's faces
__device__ __noinline__ float sample_n_call(const float* __restrict__ a, const NbConst& C, float px, float py, float pz) {
    return sample_n(a, C.nx, C.ny, C.nz, px, py, pz, C.dx, C.inv_dx, C.dx_pow2 != 0);
}
__device__ __noinline__ int2 ray_range(const NbConst& C, float sx, float sy, float sz, float dxr, float dyr, float dzr) {
    float t0, t1;
    nb_box_range(sx, sy, sz, dxr, dyr, dzr, C.bmax, t0, t1);
    return make_int2(trunc_i(t0 / C.dr_f), min(C.nsteps, trunc_i(t1 / C.dr_f) + 2));
}

// cast_ray with one lane per ray, as a plain loop, where nb_rays_small allows it: the same bits (the
// products and sums are spelled out where a contraction would change them).  Along the part of the ray
// that lies a cell inside the box, [i0, i1], the eight corners lie at fixed steps from the lower one, and
// neither a clamp nor a test of the domain is needed; nb_rays_small keeps the rounding of i0 and i1, which
// may be approximate, and of the positions below the half cell to spare.  floor(g) is g added to 1.5 x 2^23 rounded down, whose bits also
// hold the index: no conversion instruction (those issue at an eighth of the rate).  Samples before i0 and
// after i1 are sample_n's.  A star inside that part starts at sample 0, so a ray that ends within it never
// needs its exact range, which costs eight divisions.
// Issue bound (72% of the slots; 484 instructions a warp at 256^3 with six stars and 512 x 1024 rays), the
// gathers' cache lines next (51%).  cast_rays with the march over sample_n in 32 rays along phi -> this:
// 59 -> 35 us at 64^3, 105 -> 60 at 192^3, 118 -> 64 at 256^3; exact build 69 -> 38, 88 -> 48 at 128^3,
// 126 -> 76 at 192^3.  Two samples at a time (loads of both in flight) measured 8% slower, the clamped form
// of the corners everywhere 13% slower.
__device__ __forceinline__ float cast_ray1(const NbConst& C, const float4 d, const float* __restrict__ rho, float sx,
                                           float sy, float sz, float Q) {
    const float dr = C.dr_f, dx = C.dx;
    const float o[3] = {sx, sy, sz}, v[3] = {d.x, d.y, d.z};
    float i0 = 0.0f, i1 = 1e9f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float w = rcp_approx(v[a]), ta = (dx - o[a]) * w, tb = ((C.bmax[a] - dx) - o[a]) * w;
        i0 = fmaxf(i0, fminf(ta, tb));
        i1 = fminf(i1, fmaxf(ta, tb));
    }
    // a star that is no number (every position of its rays is none either) stays with sample_n
    if (!(fabsf(sx) + fabsf(sy) + fabsf(sz) < 1e30f)) i1 = -1.0f;
    const bool inside = i0 == 0.0f && i1 > 0.0f;
    const float inv_dr = rcp_approx(dr);
    float nf = 0.5f, end = (float)C.nsteps;              // n + 1/2 (exact: nb_rays_small)
    float sum = 0.0f, comp = 0.0f, rf = C.diag_f;        // Kahan-compensated column
    auto crosses = [&](float nv, float r) -> bool {
        const float inc = vmul(vmul(vmul(vmul(nv, nv), r), r), dr), col = sum - comp;
        if (vadd(col, inc) > Q) {
            rf = fmaf(-0.5f, dr, r) + dr * (Q - col) / fmaxf(inc, 1e-20f);
            return true;
        }
        const float y = vsub(inc, comp), t = sum + y;
        comp = (t - sum) - y;
        sum = t;
        return false;
    };
    auto by_call = [&](float r) {
        return sample_n_call(rho, C, mac(d.x, r, sx), mac(d.y, r, sy), mac(d.z, r, sz));
    };
    if (!inside) {
        const int2 n = ray_range(C, sx, sy, sz, d.x, d.y, d.z);
        nf = (float)n.x + 0.5f;
        end = (float)n.y;
        for (const float in0 = i0 * inv_dr; nf < end && !(nf >= in0); nf += 1.0f) {
            const float r = vmul(nf, dr);
            if (crosses(by_call(r), r)) return rf;
        }
    }
    const float inv_dx = C.inv_dx, M = 12582912.0f, in1 = fminf(i1 * inv_dr, end);
    const bool pow2 = C.dx_pow2 != 0;
    const int ny = C.ny, nz = C.nz, sx1 = ny * nz;
    const unsigned Mb = 0x4B400000u, k = (Mb * (unsigned)ny + Mb) * (unsigned)nz + Mb;   // the bits of M in an index
    for (; nf < in1; nf += 1.0f) {
        const float r = vmul(nf, dr), px = mac(d.x, r, sx), py = mac(d.y, r, sy), pz = mac(d.z, r, sz);
        float gx, gy, gz;
        if (pow2) {                                      // an exact product
            gx = fmaf(px, inv_dx, -0.5f);
            gy = fmaf(py, inv_dx, -0.5f);
            gz = fmaf(pz, inv_dx, -0.5f);
        } else {                                         // the quotient is rounded before the subtraction
            gx = vadd(px / dx, -0.5f);
            gy = vadd(py / dx, -0.5f);
            gz = vadd(pz / dx, -0.5f);
        }
        const float mx = __fadd_rd(gx, M), my = __fadd_rd(gy, M), mz = __fadd_rd(gz, M);
        const float fx = gx - (mx - M), fy = gy - (my - M), fz = gz - (mz - M);
        const unsigned e = (__float_as_uint(mx) * (unsigned)ny + __float_as_uint(my)) * (unsigned)nz +
                           (__float_as_uint(mz) - k);
        const float *p00 = rho + e, *p01 = p00 + nz, *p10 = p00 + sx1, *p11 = p10 + nz;
#if NB_ARITH_FAST
        const F2 a0 = mk2(__ldg(p00), __ldg(p00 + 1)), a1 = mk2(__ldg(p10), __ldg(p10 + 1));
        const F2 b0 = mk2(__ldg(p01), __ldg(p01 + 1)), b1 = mk2(__ldg(p11), __ldg(p11 + 1));
        const F2 x2 = mk2(fx, fx), y2 = mk2(fy, fy);
        const F2 a = vfma(vsub(a1, a0), x2, a0), b = vfma(vsub(b1, b0), x2, b0), c = vfma(vsub(b, a), y2, a);
        const float c0 = lo(c), c1 = hi(c);
#else
        const float a0 = __ldg(p00), a1 = __ldg(p10), b0 = __ldg(p01), b1 = __ldg(p11);
        const float A0 = __ldg(p00 + 1), A1 = __ldg(p10 + 1), B0 = __ldg(p01 + 1), B1 = __ldg(p11 + 1);
        const float a = mac(a1 - a0, fx, a0), b = mac(b1 - b0, fx, b0), c0 = mac(b - a, fy, a);
        const float A = mac(A1 - A0, fx, A0), B = mac(B1 - B0, fx, B0), c1 = mac(B - A, fy, A);
#endif
        if (crosses(mac(vsub(c1, c0), fz, c0), r)) return rf;
    }
    if (inside) end = (float)ray_range(C, sx, sy, sz, d.x, d.y, d.z).y;
    for (; nf < end; nf += 1.0f) {
        const float r = vmul(nf, dr);
        if (crosses(by_call(r), r)) return rf;
    }
    return rf;
}

// Each star's least and largest front radius, for apply_front's culling: order-preserving bits of the
// floats (a NaN orders above every number), merged by one minimum and one maximum per warp.
__device__ __forceinline__ unsigned front_key(float v) {
    const unsigned b = __float_as_uint(v);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float front_of_key(unsigned k) {
    return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu));
}
// Every thread of the block calls it; `on`: the lane holds a front of star s of `bounds`, `id` tells the
// stars of a block apart.  A block whose rays are all one star's merges once: two atomics per warp on a
// handful of addresses took longer than the marches (133 us at every grid size).
__device__ __forceinline__ void merge_front(uint2* bounds, int id, int s, float rf, bool on) {
    __shared__ unsigned part[2][8];
    __shared__ int first;
    if (threadIdx.x == 0) first = id;
    __syncthreads();
    const unsigned k = front_key(rf);
    if (__syncthreads_and(on && id == first)) {
        const unsigned mn = __reduce_min_sync(0xffffffffu, k), mx = __reduce_max_sync(0xffffffffu, k);
        if ((threadIdx.x & 31) == 0) {
            part[0][threadIdx.x >> 5] = mn;
            part[1][threadIdx.x >> 5] = mx;
        }
        __syncthreads();
        if (threadIdx.x < 8) {
            const unsigned m = __reduce_min_sync(0xffu, part[0][threadIdx.x]);
            const unsigned x = __reduce_max_sync(0xffu, part[1][threadIdx.x]);
            if (threadIdx.x == 0) {
                atomicMin(&bounds[s].x, m);
                atomicMax(&bounds[s].y, x);
            }
        }
    } else if (on) {
        atomicMin(&bounds[s].x, k);
        atomicMax(&bounds[s].y, k);
    }
}

// The front of the ray along d of star s into an instance's table [star][phi][u]: one float, or (pairs)
// the .x of its own float2 pair and the .y of the pair below it (and of its own at the last u).
__device__ __forceinline__ void put_front(float* rfront, bool pairs, int s, long long nray, int nu, const float4 d,
                                          float rf) {
    const int w = __float_as_int(d.w);
    const long long e = (long long)s * nray + (w & 0x7fffffff);
    if (!pairs) {
        rfront[e] = rf;
        return;
    }
    float* p = rfront + 2 * e;
    p[0] = rf;
    // w < 0: the first u (below 0) or the last (above 0), or both where nu is 1
    if (w >= 0 || (d.z > 0.0f && nu > 1)) p[-1] = rf;
    if (w < 0 && (d.z > 0.0f || nu == 1)) p[1] = rf;
}

// The front radius along d.  SMALL: cast_ray1.
template <int G, bool SMALL>
__device__ __forceinline__ float cast_dir(const NbConst& C, const float4 d, const float* __restrict__ rho, float sx,
                                          float sy, float sz, float Q, int lane, unsigned gmask, bool live) {
    if (SMALL) return live ? cast_ray1(C, d, rho, sx, sy, sz, Q) : 0.0f;
    return cast_ray<G>(C, d, rho, sx, sy, sz, Q, lane, gmask, live);
}

// Resident blocks per SM of the ray kernel: 5 (48 registers); at 6 (40 registers) the warp-uniform
// march spills 44-84 bytes.
#define NB_CAST_RAYS_MINB 5
// blockIdx.y: the star
template <int G, bool PAIRS, bool SMALL>
__global__ void __launch_bounds__(256, NB_CAST_RAYS_MINB)
    cast_rays_kernel(const NbConst* __restrict__ c, const NbStarW* __restrict__ sw, const float4* __restrict__ dirs,
                     const float* __restrict__ rho, float* __restrict__ rfront, uint2* bounds,
                     const float* star_override, float q_override) {
    const int nray = c->nu * c->nphi, s = blockIdx.y;
    const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) / G * G));
    // no early exit: every thread reaches the march's warp-wide operations and the merge's barriers
    const bool in = gid < nray;
    const float4 d = dirs[in ? (int)gid : 0];
    if (star_override) {
        const float rf = cast_dir<G, SMALL>(*c, d, rho, star_override[0], star_override[1], star_override[2],
                                            q_override, lane, gmask, in);
        const int e = __float_as_int(d.w) & 0x7fffffff, ip = e / c->nu;
        if (in && lane == 0) rfront[(e - ip * c->nu) * c->nphi + ip] = rf;
        return;
    }
    const NbStarW w = sw[s];
    const bool live = in && w.active;
    const float rf = cast_dir<G, SMALL>(*c, d, rho, w.w.x, w.w.y, w.w.z, w.q_f, lane, gmask, live);
    // the instance's table is [star][phi][u] (u fastest: the cells of a warp share phi)
    if (live && lane == 0) put_front(rfront, PAIRS, s, nray, c->nu, d, rf);
    if (bounds) merge_front(bounds, s, s, rf, live);
}

// Rays of every star of every listed instance: job e owns groups [job[e].ray0, job[e+1].ray0).
// `J` holds the job records (global memory, or the kernel parameter of the param form); the active
// flags always come from `Jd`, the device copy (they change between replays of a captured step).
template <int G, bool SMALL, typename Jobs>
__device__ __forceinline__ void cast_rays_batch_body(const Jobs& J, const NbRayJob* __restrict__ Jd, int n_jobs,
                                                     long long n_groups) {
    const long long gid0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) / G * G));
    // no early exit: every thread reaches the march's warp-wide operations and the merge's barriers
    const bool in = gid0 < n_groups;
    const long long gid = in ? gid0 : 0;
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {                          // last job with ray0 <= gid
        const int mid = (lo + hi + 1) >> 1;
        if (J[mid].ray0 <= gid) lo = mid; else hi = mid - 1;
    }
    const NbRayJob& job = J[lo];
    const NbConst& C = *job.c;
    const int nray = C.nu * C.nphi;
    const long long local = gid - job.ray0;
    const unsigned l32 = (unsigned)local;        // below 2^32 within a job (nb_create): 32-bit division
    const int s = (int)(l32 / (unsigned)nray);
    const float4 d = job.dirs[l32 - (unsigned)s * (unsigned)nray];
    const bool star = in && s < job.nstars && Jd[lo].active;
    NbStarW w{};
    if (star) w = job.sw[s];
    const bool live = star && w.active;
    const float rf = cast_dir<G, SMALL>(C, d, job.rho, w.w.x, w.w.y, w.w.z, w.q_f, lane, gmask, live);
    if (live && lane == 0) put_front(job.rfront, job.pairs != 0, s, nray, C.nu, d, rf);
    // the lanes of a warp may belong to two jobs: (job, star) pairs are told apart
    merge_front(job.front_bounds, lo * NB_MAX_STARS + s, s, rf, live && job.front_bounds);
}

template <int G, bool SMALL>
__global__ void __launch_bounds__(256) cast_rays_batch_kernel(const NbRayJob* __restrict__ jobs, int n_jobs,
                                                              long long n_groups) {
    cast_rays_batch_body<G, SMALL>(jobs, jobs, n_jobs, n_groups);
}

// the job records in the kernel parameter (constant bank): 48 registers, 5 blocks / SM
template <int G, bool SMALL>
__global__ void __launch_bounds__(256, NB_CAST_RAYS_MINB)
    cast_rays_batch_param_kernel(const __grid_constant__ NbRayJobs P, const NbRayJob* __restrict__ jobs, int n_jobs,
                                 long long n_groups) {
    cast_rays_batch_body<G, SMALL>(P.J, jobs, n_jobs, n_groups);
}

// The stars that can change xi or the front distance of the 32-cell segment [kb, kb + 32) of a
// row, as a mask (1 <= nstars <= NB_ROW_STARS).  Over the segment a star's
// r - rf lies in [LB, UB]: LB = (least distance to the segment) - (largest front radius of the
// star), UB = (largest distance) - (smallest front radius).  A star with LB at or above both
// min(1e3, least UB over the stars) and width / 2, plus a margin of one cell for float rounding,
// gives every cell of the segment val = 0 (no xi) and an r - rf above another star's (no front
// distance): leaving it out changes no bit.  A NaN bound (NaN radii or positions, whose min /
// max merges depend on order) keeps every active star.
// Computed for per_pass = 32 / nstars consecutive segments [kb0 + 32 g, kb0 + 32 g + 32) at once:
// lane g * nstars + s bounds star s over segment g, each segment's least upper bound is gathered
// from its nstars lanes, and lane g returns segment g's mask (bit s: star s).  One warp pass per
// per_pass segments: the culling costs ~per_pass times fewer instructions per cell.
__device__ __forceinline__ unsigned segment_masks(const float4* st, const int* act, const float4* tab,
                                                  const float2* bnd, int nstars, int kb0, int per_pass, int nz,
                                                  float dx, float width) {
    const int lane = threadIdx.x;
    const int g = lane / nstars, s = lane - g * nstars;
    const int kb = kb0 + 32 * g;
    const bool on = g < per_pass && kb < nz && act[s];
    float lb = __int_as_float(0x7f800000), ub = lb;       // +inf: the lane bounds no star
    bool bad = false;
    if (on) {
        const float sz = st[s].z, d2 = tab[s].x;
        const float2 b = bnd[s];                          // (least, largest) front radius
        const float z0 = ((float)kb + 0.5f) * dx, z1 = ((float)(min(kb + 31, nz - 1)) + 0.5f) * dx;
        const float en = fmaxf(0.0f, fmaxf(z0 - sz, sz - z1));
        const float ex = fmaxf(fabsf(sz - z0), fabsf(sz - z1));
        lb = sqrtf(d2 + en * en) - b.y;
        ub = sqrtf(d2 + ex * ex) - b.x;
        bad = isnan(lb) || isnan(ub);
    }
    const int base = min(g * nstars, 31);
    float m = __int_as_float(0x7f800000);
    for (int t = 0; t < nstars; ++t) m = fminf(m, __shfl_sync(0xffffffffu, ub, min(base + t, 31)));
    const float thr = fmaxf(fminf(1e3f, m), 0.5f * width) + dx;
    const unsigned keep = __ballot_sync(0xffffffffu, on && lb < thr);
    const unsigned all = __ballot_sync(0xffffffffu, on);
    const unsigned nan = __ballot_sync(0xffffffffu, bad);
    if (lane >= per_pass) return 0u;
    const int sh = lane * nstars;
    const unsigned full = nstars == 32 ? 0xffffffffu : ((1u << nstars) - 1u);
    return ((nan >> sh) & full) ? (all >> sh) & full : (keep >> sh) & full;
}

// nebula3d.py:273-307 rf_at + apply_front over one row (i, j), fused over the active stars,
// with the fp16 store of the front distance (sim.py:942, 980-985).  `tab`: this warp's row
// table (NB_ROW_STARS entries) or null for the per-cell form; `bnd`: each star's (least, largest)
// front radius, or null to merge every active star in every segment.  PAIRS: the front table
// holds (u, u + 1) pairs.
template <bool PAIRS>
__device__ __forceinline__ void apply_front_row(const NbConst& C, const float4* st, const int* act, int nstars,
                                                const float* __restrict__ rfront, float* __restrict__ xi_raw,
                                                void* __restrict__ dfront, bool half, int row, float4* tab,
                                                const float2* bnd) {
    const int nx = C.nx, ny = C.ny, nz = C.nz, nu = C.nu, nphi = C.nphi;
    if (row >= nx * ny) return;
    const int i = row / ny, j = row - (row / ny) * ny;
    const long long base = (long long)row * nz;
    const float dx = C.dx, width = C.width;
#if NB_ARITH_FAST
    const float inv_width = 1.0f / width;
#endif
    const float two_pi = 2.0f * pi_f();
    const float px = ((float)i + 0.5f) * dx, py = ((float)j + 0.5f) * dx;
    const long long rstride = (long long)nu * nphi;
    if (tab && nstars > NB_ROW_STARS) tab = nullptr;
    if (!tab) bnd = nullptr;
    if (tab) star_row_table(st, act, nstars, px, py, nphi, nu, tab);
    const unsigned row_stars = tab ? __ballot_sync(0xffffffffu, (int)threadIdx.x < nstars && act[threadIdx.x]) : 0u;
    constexpr int SG = 2;                       // stars whose gathers are in flight together
    // the culling masks of per_pass segments come from one pass (segment_masks): lane g holds
    // segment g's, broadcast when that segment's cells are merged
    if (nstars < 1) bnd = nullptr;
    const int per_pass = bnd ? 32 / nstars : 1;
    for (int kb0 = 0; kb0 < nz; kb0 += 32 * per_pass) {
      const unsigned masks = bnd ? segment_masks(st, act, tab, bnd, nstars, kb0, per_pass, nz, dx, width) : 0u;
      for (int g = 0; g < per_pass; ++g) {
        const int kb = kb0 + 32 * g;
        if (kb >= nz) break;                     // uniform over the warp
        const unsigned seg = bnd ? __shfl_sync(0xffffffffu, masks, g) : row_stars;
        const int k = kb + (int)threadIdx.x;
        if (k >= nz) continue;
        const long long q = base + k;
        const float pz = ((float)k + 0.5f) * dx;
        float xi = 0.0f, df = 1e3f;
        unsigned left = seg;                     // mask form: the segment's stars in star order
        for (int s0 = 0; tab ? left != 0u : s0 < nstars; s0 += SG) {
            float r[SG], tu[SG], tp[SG], g00[SG], g01[SG], g10[SG], g11[SG];
            bool on[SG];
#pragma unroll
            for (int e = 0; e < SG; ++e) {
                int s;
                if (tab) {
                    on[e] = left != 0u;
                    s = on[e] ? __ffs(left) - 1 : 0;
                    left &= left - 1u;
                } else {
                    s = s0 + e;
                    on[e] = s < nstars && act[s];
                }
                if (!on[e]) continue;                   // an empty slot's values are never read
                const float4 sp = st[s];
                const float* rfs = rfront + (long long)s * rstride;
                const float rz = pz - sp.z;
                int c0, c1;                      // phi columns times nu (table [phi][u])
                if (tab) {
                    const float4 tb = tab[s];
                    r[e] = fmaxq(sqrtf(tb.x + rz * rz), 1e-6f);                  // (rx^2 + ry^2) + rz^2
                    tp[e] = tb.y;
                    c0 = __float_as_int(tb.z);
                    c1 = __float_as_int(tb.w);
                } else {
                    const float rx = px - sp.x, ry = py - sp.y;
                    r[e] = fmaxq(sqrtf((rx * rx + ry * ry) + rz * rz), 1e-6f);     // 0 + x*x == x*x
                    float phi = atan2f(ry, rx);
                    if (phi < 0.0f) phi = phi + two_pi;
                    const float fp = phi / two_pi * (float)nphi - 0.5f;
                    const int ip = (int)floorf(fp);
                    tp[e] = fp - (float)ip;
                    c0 = wrap_index(ip, nphi) * nu;
                    c1 = wrap_index(ip + 1, nphi) * nu;
                }
#if NB_ARITH_FAST
                const float u = rz * rcp_approx(r[e]);
#else
                const float u = rz / r[e];
#endif
                const float fu = (u + 1.0f) * 0.5f * (float)nu - 0.5f;
                const int iu = (int)floorf(fu);
                tu[e] = fu - (float)iu;
                const int u0 = max(iu, 0), u1 = min(iu + 1, nu - 1);    // u in [-1, 1]: iu in [-1, nu - 1]
                if (PAIRS) {
                    // pair u0 = (rf(u0), rf(min(u0 + 1, nu - 1))): the two u corners, except at iu = -1,
                    // where both corners clamp to u = 0 (the pair's .x)
                    const float2* rp = reinterpret_cast<const float2*>(rfront) + (long long)s * rstride;
                    const float2 p0 = __ldg(rp + c0 + u0), p1 = __ldg(rp + c1 + u0);
                    g00[e] = p0.x;
                    g01[e] = p1.x;
                    g10[e] = iu < 0 ? p0.x : p0.y;
                    g11[e] = iu < 0 ? p1.x : p1.y;
                } else {
                    g00[e] = __ldg(rfs + c0 + u0);
                    g01[e] = __ldg(rfs + c1 + u0);
                    g10[e] = __ldg(rfs + c0 + u1);
                    g11[e] = __ldg(rfs + c1 + u1);
                }
            }
#pragma unroll
            for (int e = 0; e < SG; ++e) {
                if (!on[e]) continue;
                const float ra = g00[e] * (1.0f - tp[e]) + g01[e] * tp[e];
                const float rb = g10[e] * (1.0f - tp[e]) + g11[e] * tp[e];
                const float rf = ra * (1.0f - tu[e]) + rb * tu[e];
#if NB_ARITH_FAST
                // clamped to [0, 1] by the saturating form of the multiply-add; merged by one max
                xi = fmaxf(xi, __saturatef((rf - r[e]) * inv_width + 0.5f));
#else
                const float val = fminr(fmaxr(0.0f, (rf - r[e]) / width + 0.5f), 1.0f);
                if (val > xi) xi = val;              // in star order, as the reference merges
#endif
                df = fminq(df, r[e] - rf);
            }
        }
        if (C.plane_on) {                        // the -x plane-parallel source: same merge rules
            const float xf = __ldg(C.plane_xf + (long long)j * nz + k);
            const float val = fminr(fmaxr(0.0f, (xf - px) / width + 0.5f), 1.0f);
            if (val > xi) xi = val;
            df = fminr(df, px - xf);
        }
        xi_raw[q] = xi;
        if (half)
            reinterpret_cast<__half*>(dfront)[q] = __float2half_rn(df);
        else
            reinterpret_cast<float*>(dfront)[q] = df;
      }
    }
}

// the (least, largest) front radius per star into shared memory (after load_stars' barrier)
__device__ __forceinline__ void load_front_bounds(const uint2* bounds, int nstars, float2* bnd, int tlin) {
    for (int s = tlin; s < nstars; s += blockDim.x * blockDim.y)
        bnd[s] = make_float2(front_of_key(bounds[s].x), front_of_key(bounds[s].y));
    __syncthreads();
}

__device__ __forceinline__ int load_stars(const NbStarW* sw, int nstars, float4* st, int* act) {
    const int tlin = threadIdx.y * blockDim.x + threadIdx.x;
    for (int s = tlin; s < nstars; s += blockDim.x * blockDim.y) {
        st[s] = sw[s].w;
        act[s] = sw[s].active;
    }
    __syncthreads();
    return tlin;
}

template <bool HALF, bool PAIRS>
__global__ void __launch_bounds__(256, 4) apply_front_kernel(const NbConst* __restrict__ c,
                                                          const NbStarW* __restrict__ sw,
                                                          const float* __restrict__ rfront, int nstars,
                                                          float* __restrict__ xi_raw, void* __restrict__ dfront,
                                                          unsigned* smax_reset, const uint2* __restrict__ bounds) {
    __shared__ float4 st[NB_MAX_STARS];
    __shared__ int act[NB_MAX_STARS];
    __shared__ float4 tab[8][NB_ROW_STARS];
    __shared__ float2 bnd[NB_ROW_STARS];
    const int tlin = load_stars(sw, nstars, st, act);
    if (smax_reset && blockIdx.x == 0 && tlin == 0) *smax_reset = 0u;
    if (bounds) load_front_bounds(bounds, nstars, bnd, tlin);    // only with nstars <= NB_ROW_STARS
    apply_front_row<PAIRS>(*c, st, act, nstars, rfront, xi_raw, dfront, HALF, blockIdx.x * blockDim.y + threadIdx.y,
                           tab[threadIdx.y], bounds ? bnd : nullptr);
}

// Rows of every listed instance; job e owns blocks [job[e].blk0, job[e+1].blk0) (8 rows each).
__global__ void __launch_bounds__(256) apply_front_batch_kernel(const NbRayJob* __restrict__ jobs, int n_jobs) {
    __shared__ float4 st[NB_MAX_STARS];
    __shared__ int act[NB_MAX_STARS];
    __shared__ float4 tab[8][NB_ROW_STARS];
    __shared__ float2 bnd[NB_ROW_STARS];
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].blk0 <= (long long)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const NbRayJob& J = jobs[lo];
    if (!J.active) return;                       // uniform over the block
    const int lb = (int)(blockIdx.x - J.blk0);
    const int tlin = load_stars(J.sw, J.nstars, st, act);
    if (lb == 0 && tlin == 0) *J.smax = 0u;
    if (J.front_bounds) load_front_bounds(J.front_bounds, J.nstars, bnd, tlin);     // uniform over the block
    if (J.pairs)
        apply_front_row<true>(*J.c, st, act, J.nstars, J.rfront, J.xi_raw, J.dfront, J.half != 0,
                              lb * blockDim.y + threadIdx.y, tab[threadIdx.y], J.front_bounds ? bnd : nullptr);
    else
        apply_front_row<false>(*J.c, st, act, J.nstars, J.rfront, J.xi_raw, J.dfront, J.half != 0,
                               lb * blockDim.y + threadIdx.y, tab[threadIdx.y], J.front_bounds ? bnd : nullptr);
}

// nebula3d.py:310-315 smooth_xi (+ sim.py:941 copy back) of one row, then the CFL max speed
// (nebula3d.py:154-162) of the state with the new xi.
__device__ __forceinline__ float smooth_row(const NbConst& C, const float* __restrict__ src, float* __restrict__ xi,
                                            const float* __restrict__ rho, const float* __restrict__ mx,
                                            const float* __restrict__ my, const float* __restrict__ mz, bool smax,
                                            int row) {
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const float cn2 = C.cn2, ci2 = C.ci2;
    float m = 0.0f;
    if (row >= nx * ny) return m;
    const int i = row / ny, j = row - (row / ny) * ny;
    const long long base = (long long)row * nz;
    const long long sj = nz, si = (long long)ny * nz;
    const long long dxm = i > 0 ? si : 0, dxp = i < nx - 1 ? si : 0;
    const long long dym = j > 0 ? sj : 0, dyp = j < ny - 1 ? sj : 0;
#pragma unroll 4
    for (int k = threadIdx.x; k < nz; k += 32) {
        const long long q = base + k;
        const float xm = __ldg(src + q - dxm), xp = __ldg(src + q + dxp);
        const float ym = __ldg(src + q - dym), yp = __ldg(src + q + dyp);
        const float zm = __ldg(src + q - (k > 0 ? 1 : 0)), zp = __ldg(src + q + (k < nz - 1 ? 1 : 0));
        const float mm = (xm + xp + ym + yp + zm + zp) / 6.0f;
        const float x = 0.5f * __ldg(src + q) + 0.5f * mm;
        xi[q] = x;
        if (smax) {
            const float r = rho[q];
#if NB_ARITH_FAST
            const float ri = 1.0f / r;               // one division for the three velocities
            const float v = fabsf(mx[q] * ri) + fabsf(my[q] * ri) + fabsf(mz[q] * ri) + sqrtf(cn2 + x * (ci2 - cn2));
#else
            const float v = fabsf(mx[q] / r) + fabsf(my[q] / r) + fabsf(mz[q] / r) + sqrtf(cn2 + x * (ci2 - cn2));
#endif
            m = fmaxr(v, m);
        }
    }
    return m;
}

__device__ __forceinline__ void block_max_to(float m, unsigned* smax_bits) {
    for (int o = 16; o > 0; o >>= 1) m = fmaxr(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float red[32];
    if (threadIdx.x == 0) red[threadIdx.y] = m;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        float b = 0.0f;
        for (int w = 0; w < (int)blockDim.y; ++w) b = fmaxr(b, red[w]);
        atomicMax(smax_bits, __float_as_uint(b));
    }
}

__global__ void __launch_bounds__(256) smooth_kernel(const NbConst* __restrict__ c, const float* __restrict__ src,
                                                     float* __restrict__ xi, const float* __restrict__ rho,
                                                     const float* __restrict__ mx, const float* __restrict__ my,
                                                     const float* __restrict__ mz, unsigned* smax_bits) {
    const float m = smooth_row(*c, src, xi, rho, mx, my, mz, smax_bits != nullptr,
                               blockIdx.x * blockDim.y + threadIdx.y);
    if (smax_bits) block_max_to(m, smax_bits);
}

__global__ void __launch_bounds__(256) smooth_batch_kernel(const NbRayJob* __restrict__ jobs, int n_jobs) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].blk0 <= (long long)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const NbRayJob& J = jobs[lo];
    if (!J.active) return;                       // uniform over the block
    const int lb = (int)(blockIdx.x - J.blk0);
    const float m = smooth_row(*J.c, J.xi_raw, J.xi, J.rho, J.mx, J.my, J.mz, true, lb * blockDim.y + threadIdx.y);
    block_max_to(m, J.smax);
}

// Plane-parallel ionizing source on the -x face (no reference counterpart): per (j,k) column, the
// recombination column sum n^2 dx along +x in cell order, the front where it passes the flux F,
// interpolated inside the crossing cell as cast_rays does (nebula3d.py:262-268); no front: rcap.
__global__ void __launch_bounds__(256) plane_front_kernel(const NbConst* __restrict__ c, const float* __restrict__ rho,
                                                          float* __restrict__ xf) {
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= ny * nz) return;
    const float F = c->plane_F_f, dx = c->dx;
    float sum = 0.0f, x = c->diag_f;
    const long long plane = (long long)ny * nz;
    for (int i = 0; i < nx; ++i) {
        const float n = __ldg(rho + i * plane + col);
        const float inc = n * n * dx;
        if (sum + inc > F) {
            x = ((float)i + 0.5f) * dx - 0.5f * dx + dx * (F - sum) / fmaxr(inc, 1e-20f);
            break;
        }
        sum = sum + inc;
    }
    xf[col] = x;
}

}  // namespace

cudaError_t nb_launch_plane_front(const NbConst* c, const float* rho, float* xf, int ny, int nz, cudaStream_t s) {
    const int cols = ny * nz;
    plane_front_kernel<<<(cols + 255) / 256, 256, 0, s>>>(c, rho, xf);
    return cudaGetLastError();
}

cudaError_t nb_launch_ray_dirs(int nu, int nphi, float4* dirs, cudaStream_t s) {
    const int n = nu * nphi;
    ray_dirs_kernel<<<(n + 255) / 256, 256, 0, s>>>(nu, nphi, dirs);
    return cudaGetLastError();
}

cudaError_t nb_launch_ray_order(int nu, int nphi, const float4* dirs, float4* out, cudaStream_t s) {
    const int n = nu * nphi;
    ray_order_kernel<<<(n + 255) / 256, 256, 0, s>>>(nu, nphi, dirs, out);
    return cudaGetLastError();
}

int nb_rays_small(const NbConst& c) { return nb_march_unclamped(c.nx, c.ny, c.nz, c.nsteps, c.dr_f, c.dx) ? 1 : 0; }

cudaError_t nb_launch_cast_rays(const NbConst* c, const NbStarW* sw, const float4* dirs, const float* rho,
                                float* rfront, int nstars, int group, uint2* bounds, const float* star_override,
                                float q_override, cudaStream_t s, int nu, int nphi, int pairs, int small) {
    const long long threads = (long long)nu * nphi * group;
    const dim3 blocks((unsigned)((threads + 255) / 256), (unsigned)nstars);
#define NB_RAYS_LAUNCH(G, SM)                                                                                      \
    (pairs ? cast_rays_kernel<G, true, SM><<<blocks, 256, 0, s>>>(c, sw, dirs, rho, rfront, bounds, \
                                                                  star_override, q_override)                        \
           : cast_rays_kernel<G, false, SM><<<blocks, 256, 0, s>>>(c, sw, dirs, rho, rfront, bounds,                \
                                                                   star_override, q_override))
    switch (group) {
        case 1:
            if (small) NB_RAYS_LAUNCH(1, true);
            else NB_RAYS_LAUNCH(1, false);
            break;
        case 2: NB_RAYS_LAUNCH(2, false); break;
        case 4: NB_RAYS_LAUNCH(4, false); break;
        case 8: NB_RAYS_LAUNCH(8, false); break;
        case 16: NB_RAYS_LAUNCH(16, false); break;
        default: NB_RAYS_LAUNCH(32, false); break;
    }
#undef NB_RAYS_LAUNCH
    return cudaGetLastError();
}

cudaError_t nb_launch_apply_front(const NbConst* c, const NbStarW* sw, const float* rfront, int nstars,
                                  float* xi_raw, void* dfront, unsigned* smax_reset, cudaStream_t s, int nx, int ny,
                                  int half, const uint2* bounds, int pairs) {
    const dim3 blk(32, 8);
    const int blocks = rowwalk_blocks(nx, ny);
    if (nstars < 1 || nstars > NB_ROW_STARS) bounds = nullptr;
    if (half && pairs)
        apply_front_kernel<true, true><<<blocks, blk, 0, s>>>(c, sw, rfront, nstars, xi_raw, dfront, smax_reset, bounds);
    else if (half)
        apply_front_kernel<true, false><<<blocks, blk, 0, s>>>(c, sw, rfront, nstars, xi_raw, dfront, smax_reset, bounds);
    else if (pairs)
        apply_front_kernel<false, true><<<blocks, blk, 0, s>>>(c, sw, rfront, nstars, xi_raw, dfront, smax_reset, bounds);
    else
        apply_front_kernel<false, false><<<blocks, blk, 0, s>>>(c, sw, rfront, nstars, xi_raw, dfront, smax_reset, bounds);
    return cudaGetLastError();
}

cudaError_t nb_launch_smooth(const NbConst* c, const float* xi_raw, float* xi, const float* rho, const float* mx,
                             const float* my, const float* mz, unsigned* smax_bits, cudaStream_t s, int nx, int ny) {
    smooth_kernel<<<rowwalk_blocks(nx, ny), dim3(32, 8), 0, s>>>(c, xi_raw, xi, rho, mx, my, mz, smax_bits);
    return cudaGetLastError();
}

cudaError_t nb_launch_ionize_batch(const NbRayJob* jobs, const NbRayJob* host_jobs, int n_jobs, long long n_groups,
                                   long long n_blocks, int group, int small, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    const long long threads = n_groups * group;
    const long long blocks = (threads + 255) / 256;
    if (blocks > 0 && host_jobs && n_jobs <= NB_BATCH_PARAM_MAX) {
        NbRayJobs P;
        std::memset(&P, 0, sizeof(P));
        std::memcpy(P.J, host_jobs, sizeof(NbRayJob) * n_jobs);
        const unsigned nb = (unsigned)blocks;
        switch (group) {
            case 1:
                if (small)
                    cast_rays_batch_param_kernel<1, true><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups);
                else
                    cast_rays_batch_param_kernel<1, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups);
                break;
            case 2: cast_rays_batch_param_kernel<2, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups); break;
            case 4: cast_rays_batch_param_kernel<4, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups); break;
            case 8: cast_rays_batch_param_kernel<8, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups); break;
            case 16: cast_rays_batch_param_kernel<16, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups); break;
            default: cast_rays_batch_param_kernel<32, false><<<nb, 256, 0, s>>>(P, jobs, n_jobs, n_groups); break;
        }
    } else if (blocks > 0) {
        switch (group) {
            case 1:
                if (small)
                    cast_rays_batch_kernel<1, true><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups);
                else
                    cast_rays_batch_kernel<1, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups);
                break;
            case 2: cast_rays_batch_kernel<2, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups); break;
            case 4: cast_rays_batch_kernel<4, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups); break;
            case 8: cast_rays_batch_kernel<8, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups); break;
            case 16: cast_rays_batch_kernel<16, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups); break;
            default: cast_rays_batch_kernel<32, false><<<(unsigned)blocks, 256, 0, s>>>(jobs, n_jobs, n_groups); break;
        }
    }
    apply_front_batch_kernel<<<(unsigned)n_blocks, dim3(32, 8), 0, s>>>(jobs, n_jobs);
    smooth_batch_kernel<<<(unsigned)n_blocks, dim3(32, 8), 0, s>>>(jobs, n_jobs);
    return cudaGetLastError();
}
