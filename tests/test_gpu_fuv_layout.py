"""The order of the FUV table on both sides of its rule (bricks of 4 u x 4 r where six times the cells reach the
table's entries, [u][phi][r] below): G0 has the bits of the table without pairs either way, in both builds."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# fuv_grid (8, 12, 16): 1536 entries a star, the line at 256 cells
SHAPES = ((3, 21, 4), (4, 16, 4), (1, 4, 64), (2, 9, 16), (63, 1, 4), (64, 1, 4), (16, 16, 4), (7, 9, 8))


@pytest.mark.parametrize("arith", ("exact", "fast"))
@pytest.mark.parametrize("nstars", (1, 33))
@pytest.mark.parametrize("shape", SHAPES)
def test_g0_has_the_same_bits_in_every_order(shape, nstars, arith):
    from nebulaviewer_gb300 import autotune as at, build, sim as S
    build.build(verbose=False)
    dx = 0.03
    rng = np.random.default_rng(sum(shape) + nstars)
    rho = np.exp(rng.normal(0.0, 0.7, shape)).astype(np.float32)
    L = np.array(shape) * dx
    stars = [(*(float(v) for v in rng.random(3) * L), float(rng.uniform(0.2, 2.0)), 0.0) for _ in range(nstars)]
    P = dict(q_main=1.0, q_ramp=0.0, wind=0.0, fp32_fields=True, max_stars=nstars)
    g0 = []
    for grid in ((8, 12, 16), (8, 10, 16)):          # the second never divides into bricks
        sim = S.Sim.from_state(shape, dx, rho, stars, ["main"] * nstars, [(0.0, 0.0, 1.0)] * nstars, ["none"] * nstars, P,
                               rays=(8, 16), fuv_grid=grid, arith=arith)
        out = {}
        for pairs in (0, 1):
            at.put(sim, "fuv_pairs", pairs)
            sim.fuv_field()
            torch.cuda.synchronize()
            out[pairs] = sim.g0.numpy().astype(np.float32)
        assert np.isfinite(out[1]).all() and out[1].max() > 0
        assert np.array_equal(out[0].view(np.int32), out[1].view(np.int32)), grid
        g0.append(out[1])
        sim.close()
    assert not np.array_equal(g0[0], g0[1])          # two grids, two tables
