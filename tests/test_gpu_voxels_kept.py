"""The voxels `Sim.render_pack` returns are a view of the stage block (planes 2-3 after the prefilter, 0-1
without it).  A FUV pass packs its samples into planes 0-1 and leaves the smoothed voxels as they are."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LOOK = {"c_ha": (0.33, 0.675, 1.5), "c_o3": (0.45, 1.125, 1.5), "c_s2": (1.2, 0.66, 0.3), "c_dg": (0.07, 0.035, 0.01),
        "c_sh": (0.02, 0.007, 0.009), "gs": 12.0, "ambient": 0.1, "edge": 0.08}


@pytest.mark.parametrize("arith", ("exact", "fast"))
@pytest.mark.parametrize("shape", ((6, 5, 4), (17, 30, 36), (48, 48, 48)))
def test_fuv_pass_leaves_the_voxels(shape, arith):
    import ctypes as C
    from nebulaviewer_gb300 import _lib, build, ics
    from nebulaviewer_gb300.sim import Sim
    build.build(verbose=False)
    ic = ics.sheet(res=min(shape) * 2, seed=4, nstars=3, device="cuda", shape=shape)
    s = Sim.from_state(ic["shape"], ic["dx"], ic["rho"], ic["stars"], ic["kinds"], ic["jets"], ic["jkinds"], ic["P"],
                       mom=ic["mom"], rays=(16, 32), fuv_grid=(8, 8, 16), arith=arith)
    s.step(2)
    s.update_render_fields(force=True)
    vox = s.render_pack(dict(LOOK, inv_L=[1.0 / v for v in s.L], dx=s.dx))
    want = vox.numpy().copy()
    out = torch.zeros((8, 8, 16), device="cuda")
    xyz = (C.c_double * 3)(*[0.4 * v for v in s.L])
    for call in (s.fuv_field, lambda: s.update_render_fields(force=True),
                 lambda: _lib.check(s._lib.nb_cast_fuv(s._h, xyz, C.c_void_p(out.data_ptr())), s._h, "nb_cast_fuv")):
        call()
        torch.cuda.synchronize()
        assert np.array_equal(vox.numpy().view(np.uint16), want.view(np.uint16))
    s.close()
