"""The unclamped one-lane march of the ionizing rays gives the general march's bits: the same fields, stars
and rays through an instance whose sample limit is past the unclamped march's (2^22), which the library
sends to the general march.  Grids from four cells an axis on, cell sizes that are powers of two and not,
sample steps of a cell and half a cell, stars within, on cell centres and faces, in a corner and outside,
direction tables that do and do not divide into the warp's bundles, fronts within and beyond the box."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = ((4, 4, 4), (4, 64, 8), (17, 30, 36), (64, 64, 64), (50, 61, 68), (7, 5, 256))


def instance(sim, P, dx, rays, fast, nsteps):
    """a second handle on the Sim's fields with this sample limit"""
    from nebulaviewer_gb300 import _lib, sim as S
    d = S.instance_desc(sim.shape, dx, P, rays, (4, 4, 8), fast, 1)
    n = sim._n
    d.nsteps = nsteps
    d.f = _lib.NbFields(sim._rho.data_ptr(), sim._mx.data_ptr(), sim._my.data_ptr(), sim._mz.data_ptr(),
                        sim._xi.data_ptr(), sim._stage.data_ptr(), sim._dfront.data_ptr(), sim._g0.data_ptr())
    assert n == int(np.prod(sim.shape))
    d.stream = sim._stream.cuda_stream
    h = C.c_void_p()
    _lib.check(sim._lib.nb_create(C.byref(d), C.byref(h)), None, "nb_create", sim._lib)
    return h


@pytest.mark.parametrize("arith", ("exact", "fast"))
@pytest.mark.parametrize("rays", ((8, 4), (33, 50), (96, 128)))
@pytest.mark.parametrize("shape", SHAPES)
def test_same_bits_as_the_general_march(shape, rays, arith):
    from nebulaviewer_gb300 import _lib, build, sim as S
    from nebulaviewer_gb300.params import make_params
    build.build(verbose=False)
    rng = np.random.default_rng(3 * sum(shape) + rays[0])
    rho = np.exp(rng.normal(0.0, 1.0, shape)).astype(np.float32)
    for dx in (1.0 / 64, 0.013):
        L = np.array(shape) * dx
        P = dict(q_main=1.0, q_ramp=0.0, wind=0.0, max_stars=1)
        sim = S.Sim.from_state(shape, dx, rho, [(*(float(v) / 2 for v in L), 1.0, 0.0)], ["main"], [(0.0, 0.0, 1.0)],
                               ["none"], P, rays=rays, fuv_grid=(4, 4, 8), start_main=False, arith=arith)
        lib = sim._lib
        places = [0.5 * L, np.full(3, 1e-3) * L, np.array([1.5, 1.5, 1.5]) * dx, np.array([0.0, 0.4, 0.6]) * L,
                  np.array([dx, 0.3 * L[1], L[2] - dx]), 1.0 * L, np.array([-0.1, 0.3, 0.4]) * L,
                  np.array([1.2, -0.2, 0.5]) * L] + [rng.random(3) * L for _ in range(4)]
        for fast in (True, False):
            hs = [instance(sim, make_params(base=P), dx, rays, fast, n) for n in (3000, (1 << 22) + 1)]
            out = [torch.zeros(rays, device="cuda") for _ in hs]
            for at in places:
                xyz = (C.c_double * 3)(*(float(np.float32(v)) for v in at))
                for Q in (1e-6, 1e-3, 1.0, 1e30):
                    for h, o in zip(hs, out):
                        _lib.check(lib.nb_cast_rays(h, xyz, Q, C.c_void_p(o.data_ptr())), h, "nb_cast_rays", lib)
                    torch.cuda.synchronize()
                    assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32)), (dx, fast, at, Q)
            for h in hs:
                lib.nb_destroy(h)
        sim.close()
