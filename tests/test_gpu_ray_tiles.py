"""The ionizing-ray kernel where its forms end: grids of one or two cells on an axis, odd grids, stars in
a corner, on a cell centre, on a face and outside the box, ray grids that do and do not divide into the
8 x 4 bundles of a warp -- each star's fronts against the CPU oracle's restatement of the reference kernel.

Both sum the same samples n^2 r^2 dr with compensation; positions and interpolation differ by a few
roundings, so a front moves by a few 1e-7 of the box: asserted at the path's 1e-5 of the largest radius.
A sample within rounding of the box's face may be inside for one and outside for the other: at most
0.1% of the rays (the path's bound on the ionized mask) may differ by more."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ("exact", "fast"))
@pytest.mark.parametrize("rays", ((8, 4), (6, 10), (16, 12), (64, 128)))
@pytest.mark.parametrize("shape", ((1, 1, 4), (1, 6, 8), (5, 2, 4), (9, 7, 12), (20, 31, 24)))
def test_fronts_against_oracle(shape, rays, arith):
    import oracle as O
    from nebulaviewer_gb300 import _lib, build, sim as S
    build.build(verbose=False)
    dx = 0.03
    rng = np.random.default_rng(7 * sum(shape) + rays[0])
    rho = np.exp(rng.normal(0.0, 0.7, shape)).astype(np.float32)
    L = np.array(shape) * dx
    P = dict(q_main=1.0, q_ramp=0.0, wind=0.0)
    sim = S.Sim.from_state(shape, dx, rho, [(float(L[0] / 2), float(L[1] / 2), float(L[2] / 2), 1.0, 0.0)], ["main"],
                           [(0.0, 0.0, 1.0)], ["none"], P, rays=rays, fuv_grid=(4, 4, 8), start_main=False, arith=arith)
    K = O.Kernels(np.float32)
    out = torch.zeros(rays, device="cuda")
    stars = ((0.5, 0.5, 0.5), (1e-3, 1e-3, 1e-3), (1.5 / shape[0], 0.5, 2.5 / shape[2]), (0.0, 0.5, 0.5), (1.2, 0.4, 0.6))
    for at in stars:
        xyz = [float(np.float32(a * l)) for a, l in zip(at, L)]
        for Q in (2e-5, 3e-3, 1e3):
            _lib.check(sim._lib.nb_cast_rays(sim._h, (C.c_double * 3)(*xyz), Q, C.c_void_p(out.data_ptr())), sim._h, "rays")
            ref = K.cast_rays(rho, tuple(xyz), Q, sim.dr, sim.nsteps, dx, sim.diag, tuple(L), rays[0], rays[1])
            off = np.abs(out.cpu().numpy() - ref) > 1e-5 * float(np.abs(ref).max())
            assert off.mean() <= 1e-3, (at, Q, float(off.mean()))
    sim.close()
