"""The fast build's hydro stage over the star counts a scene may have, to the library's 256: against the
oracle's restatement of the reference kernel (winds of active and inactive stars, jets), and its time.

A stage's own rounding is within 2.2e-6 of the largest rho (|v| + c) (six fluxes of twenty roundings times
dt / dx).  The winds add dt rho w sum(q r / (r^2 + 4e-4)^1.5), each term within ten roundings: with w scaled
by the star count their sum stays below the largest speed, so 1e-6 of the same scale.  Asserted at 1e-5."""
import ctypes as C
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nstars", (1, 3, 4, 5, 33, 38, 70, 256))
def test_winds_and_jets_of_many_stars(nstars):
    import oracle as O
    from nebulaviewer_gb300 import _lib, build, sim as S
    from nebulaviewer_gb300.params import make_params, sound_speeds
    build.build(verbose=False)
    shape, dx = (5, 18, 36), 0.02
    rng = np.random.default_rng(nstars)
    rho = np.exp(rng.normal(0.0, 1.0, shape)).astype(np.float32)
    mom = [(rho * rng.normal(0.0, 2.0, shape)).astype(np.float32) for _ in range(3)]
    xi = (rng.random(shape) * (rng.random(shape) < 0.7)).astype(np.float32)
    L = np.array(shape) * dx
    stars = [(*(float(v) for v in rng.random(3) * L), float(rng.uniform(0.1, 1.0)), 0.0 if s % 4 != 2 else 1e3)
             for s in range(nstars)]
    jets, jkinds = [(0.0, 0.6, 0.8)] * nstars, ["jet" if s % 3 == 0 else "none" for s in range(nstars)]
    P = dict(q_main=1.0, q_ramp=0.0, wind=0.5 / nstars, jet=3.0 / nstars, jet_r=0.1, jet_angle=40.0, floor=2e-3, cfl=0.3,
             cn2=1.0, ci2=144.0, vmax=60.0, max_stars=nstars)
    sim = S.Sim.from_state(shape, dx, rho, stars, ["main"] * nstars, jets, jkinds, P, mom=mom, rays=(8, 16),
                           fuv_grid=(4, 4, 8), start_main=False, arith="fast")
    sim._xi.copy_(torch.as_tensor(xi, device="cuda"))
    Pm = make_params(base=P)
    cn2, ci2, vmax = sound_speeds(Pm)
    o = O.OracleSim(shape, dx, rho, stars, ["main"] * nstars, jets, jkinds, Pm, rays=(8, 16), fuv_grid=(4, 4, 8),
                    mom=mom, start_main=False, cn2=cn2, ci2=ci2, vmax=vmax)
    o._set_star_weights()
    speed = sum(np.abs(m) for m in mom) / rho + np.sqrt(cn2 + xi * (ci2 - cn2))
    dt, pulse = float(np.float32(0.3 * dx / speed.max())), 1.3
    U = [torch.as_tensor(a, device="cuda") for a in [rho] + mom]
    out = [torch.full_like(U[0], float("nan")) for _ in range(4)]
    F = lambda ts: _lib.f4([t.data_ptr() for t in ts])  # noqa: E731
    _lib.check(sim._lib.nb_hydro_stage(sim._h, F(U), F(U), F(out), 0.0, 1.0, dt, pulse), sim._h, "nb_hydro_stage")
    torch.cuda.synchronize()
    ref = [np.zeros(shape, np.float32) for _ in range(4)]
    o.K.hydro_stage([rho] + mom, xi, [rho] + mom, ref, a=0.0, b=1.0, stars=o.star_arr, nstars=nstars, wind=P["wind"],
                    jets=o.jet_arr, jet_cos=math.cos(math.radians(40.0)), jet_r=0.1, pulse=pulse, dt=dt, dx=dx,
                    floor_=2e-3, cn2=cn2, ci2=ci2, vmax=vmax, solver=1, lim=0)
    for c in range(4):
        top = max(float(rho.max()) if c == 0 else float((rho * speed).max()), float(np.abs(ref[c]).max()))
        assert float(np.abs(out[c].cpu().numpy() - ref[c]).max()) <= 1e-5 * top, c
    sim.close()


def stage_ms(sim, passes=5):
    """the least time of a step's two stages, by the library's event timers"""
    lib, best = sim._lib, math.inf
    ms, n = (C.c_double * 16)(), (C.c_longlong * 16)()
    lib.nb_profile(sim._h, 1)
    for _ in range(passes + 1):
        sim.step(2)
        lib.nb_profile_read(sim._h, ms, n)
        best = min(best, ms[1] / n[1] + ms[2] / n[2])
    lib.nb_profile(sim._h, 0)
    return best


def sheet(res, nstars, wind):
    from nebulaviewer_gb300 import build, ics
    from nebulaviewer_gb300.sim import Sim
    build.build(verbose=False)
    ic = ics.sheet(res=res, seed=4, nstars=nstars, device="cuda")
    ic["P"]["wind"] = wind
    return Sim.from_state(ic["shape"], ic["dx"], ic["rho"], ic["stars"], ic["kinds"], ic["jets"], ic["jkinds"], ic["P"],
                          mom=ic["mom"], rays=(64, 128), fuv_grid=(16, 16, 32), arith="fast")


def test_idle_stars_do_not_slow_the_stage():
    """the stars' tables take no room from the tiles: without winds the stages of 256 stars are as fast as
    those of one (a resident block less per SM is 1.35 times as long)"""
    t = {}
    for nstars in (1, 256):
        s = sheet(224, nstars, 0.0)
        t[nstars] = stage_ms(s)
        s.close()
    assert t[256] <= 1.15 * t[1], t


def test_chosen_depth_with_many_winds():
    """the depth chosen for a grid counts its stars' winds: many winds make the ionized tiles the slow ones,
    and few deep chunks then leave the GPU waiting for them.  The chosen depth is within a quarter of the
    better of two fixed ones (one for the whole column was three times as slow)."""
    from nebulaviewer_gb300 import autotune as at
    for res, nstars in ((192, 256), (384, 64)):
        s = sheet(res, nstars, 0.5)
        s.step(12)
        chosen, t = stage_ms(s), {}
        for depth in (8, 24):
            at.put(s, "chunk_i", depth)
            t[depth] = stage_ms(s)
        assert chosen <= 1.25 * min(t.values()), (res, nstars, chosen, t)
        s.close()


def test_chosen_depths_of_a_batch_with_one_windy_instance():
    """a batch's chunk depths count each instance's own winds: a step with the chosen ones takes at most a
    quarter more than with a fixed depth (with the same deep chunks for all it was 1.7 times as long)"""
    from nebulaviewer_gb300 import autotune as at
    from nebulaviewer_gb300.batch import BatchSim

    def step_ms(depth):
        sims = [sheet(128, 1, 0.5) for _ in range(7)] + [sheet(96, 256, 0.5)]
        for s in sims if depth else ():
            at.put(s, "chunk_i", depth)
        b = BatchSim(sims)
        b.step(6)
        torch.cuda.synchronize()
        best = math.inf
        for _ in range(5):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            b.step(6)
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]) / 6)
        b.close()
        for s in sims:
            s.close()
        return best
    t = {d: step_ms(d) for d in (None, 8, 20)}
    assert t[None] <= 1.25 * min(t[8], t[20]), t
