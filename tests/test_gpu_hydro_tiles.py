"""The fast build's hydro stage (two rows per thread, 32 x 16 tiles, march along i) at the sizes where
its tiles end: one row, an odd row, a row past a tile, partial k tiles, chunks of one plane.

Against the CPU oracle's restatement of the reference kernel: a stage adds dt / dx times six face
fluxes to a state, each within some twenty roundings of 2^-24 of rho (|v| + c)^2, and
dt (|v| + c) / dx <= 0.3, so the two stay within 6 x 20 x 0.3 x 6e-8 = 2.2e-6 of the largest
rho (|v| + c); asserted at 1e-5, the path's tolerance for one step.  The bits depend neither on the
chunk depth nor on the tile sweep order: every face is evaluated with the same operations wherever
a tile or a chunk ends."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = ((1, 1, 4), (2, 15, 32), (5, 16, 36), (3, 17, 28), (4, 33, 100), (21, 47, 64))
SCHEMES = (("hll", "minmod"), ("hll", "vanleer"), ("hll", "mc"), ("rusanov", "minmod"))


def stages(sim, lib, U, dt, pulse):
    g = [[torch.full_like(U[0], float("nan")) for _ in range(4)] for _ in range(2)]
    F = lambda ts: lib.f4([t.data_ptr() for t in ts])  # noqa: E731
    lib.check(sim._lib.nb_hydro_stage(sim._h, F(U), F(U), F(g[0]), 0.0, 1.0, dt, pulse), sim._h, "stage 1")
    lib.check(sim._lib.nb_hydro_stage(sim._h, F(g[0]), F(U), F(g[1]), 0.5, 0.5, dt, pulse), sim._h, "stage 2")
    torch.cuda.synchronize()
    return [[t.cpu().numpy() for t in s] for s in g]


@pytest.mark.parametrize("solver,lim", SCHEMES)
@pytest.mark.parametrize("shape", SHAPES)
def test_fast_stage_at_tile_edges(shape, solver, lim):
    import oracle as O
    from nebulaviewer_gb300 import _lib, autotune as at, build, sim as S
    from nebulaviewer_gb300.params import make_params, sound_speeds
    build.build(verbose=False)
    dx = 0.02
    rng = np.random.default_rng(sum(shape))
    rho = np.exp(rng.normal(0.0, 1.5, shape)).astype(np.float32)
    mom = [(rho * rng.normal(0.0, 2.0, shape)).astype(np.float32) for _ in range(3)]
    xi = (rng.random(shape) * (rng.random(shape) < 0.7)).astype(np.float32)
    L = np.array(shape) * dx
    stars = [(float(p[0]), float(p[1]), float(p[2]), float(q), 0.0) for p, q in zip(rng.random((3, 3)) * L, rng.random(3))]
    jets, jkinds = [(0.0, 0.6, 0.8)] * 3, ["jet", "none", "proto"]
    P = dict(q_main=1.0, q_ramp=0.0, wind=0.5, jet=3.0, jet_proto=2.0, jet_r=0.1, jet_angle=40.0, solver=solver,
             limiter=lim, floor=2e-3, cfl=0.3, cn2=1.0, ci2=144.0, vmax=30.0)
    sim = S.Sim.from_state(shape, dx, rho, stars, ["main"] * 3, jets, jkinds, P, mom=mom, rays=(8, 16),
                           fuv_grid=(4, 4, 8), start_main=False, arith="fast")
    sim._xi.copy_(torch.as_tensor(xi, device="cuda"))
    Pm = make_params(base=P)
    cn2, ci2, vmax = sound_speeds(Pm)
    o = O.OracleSim(shape, dx, rho, stars, ["main"] * 3, jets, jkinds, Pm, rays=(8, 16), fuv_grid=(4, 4, 8), mom=mom,
                    start_main=False, cn2=cn2, ci2=ci2, vmax=vmax)
    o._set_star_weights()
    c = np.sqrt(cn2 + xi * (ci2 - cn2))
    speed = sum(np.abs(m) for m in mom) / rho + c
    dt, pulse = float(np.float32(0.3 * dx / speed.max())), 1.3
    U = [torch.as_tensor(a, device="cuda") for a in [rho] + mom]
    got = stages(sim, _lib, U, dt, pulse)
    Un = [rho] + mom
    ref = [[np.zeros(shape, np.float32) for _ in range(4)] for _ in range(2)]
    kw = dict(stars=o.star_arr, nstars=3, wind=0.5, jets=o.jet_arr, jet_cos=math.cos(math.radians(40.0)), jet_r=0.1,
              pulse=pulse, dt=dt, dx=dx, floor_=2e-3, cn2=cn2, ci2=ci2, vmax=vmax, solver=1 if solver == "hll" else 0,
              lim={"minmod": 0, "vanleer": 1, "mc": 2}[lim])
    o.K.hydro_stage(Un, xi, Un, ref[0], a=0.0, b=1.0, **kw)
    o.K.hydro_stage(ref[0], xi, Un, ref[1], a=0.5, b=0.5, **kw)
    scale = [float(rho.max())] + [float((rho * speed).max())] * 3
    for s in range(2):
        for f in range(4):
            top = max(scale[f], float(np.abs(ref[s][f]).max()))
            assert float(np.abs(got[s][f] - ref[s][f]).max()) <= 1e-5 * top, (s, f)
    for chunk, order in ((1, 0), (2, 1), (3, 0), (64, 1)):
        at.put(sim, "chunk_i", chunk)
        at.put(sim, "tile_order", order)
        again = stages(sim, _lib, U, dt, pulse)
        for s in range(2):
            for f in range(4):
                assert np.array_equal(again[s][f].view(np.int32), got[s][f].view(np.int32)), (chunk, order, s, f)
    sim.close()
