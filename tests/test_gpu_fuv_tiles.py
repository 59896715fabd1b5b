"""The FUV apply where its tiles end: grids thinner than a block's rows, odd grids, FUV tables that do and
do not divide into bricks.  The table's order changes no bit (pairs, in bricks or not, against the plain
table), and the float32 field agrees with the CPU oracle's restatement of the reference kernels.

Both sum the same samples and interpolate the same table entries; positions, exponentials and quotients
differ by a few roundings (fast build: approximate ones), so G0 is asserted at the path's 1e-4 of the
largest value.  A cell whose bin or a sample whose side of the box's face is decided by rounding may take
another entry: at most 0.1% of the cells may differ by more."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ("exact", "fast"))
@pytest.mark.parametrize("grid", ((4, 4, 8), (5, 6, 7), (8, 12, 16), (6, 8, 5), (32, 64, 64)))
@pytest.mark.parametrize("shape", ((1, 1, 4), (1, 6, 8), (5, 2, 4), (2, 9, 36), (9, 7, 12), (20, 31, 24)))
def test_g0_against_oracle_and_plain_table(shape, grid, arith):
    import oracle as O
    from nebulaviewer_gb300 import autotune as at, build, sim as S
    build.build(verbose=False)
    dx = 0.03
    rng = np.random.default_rng(5 * sum(shape) + grid[0])
    rho = np.exp(rng.normal(0.0, 0.7, shape)).astype(np.float32)
    L = np.array(shape) * dx
    stars = [(float(a * L[0]), float(b * L[1]), float(c * L[2]), q, 0.0)
             for a, b, c, q in ((0.47, 0.53, 0.51, 1.0), (0.11, 0.83, 0.29, 0.5), (0.9, 0.2, 0.7, 2.0))]
    P = dict(q_main=1.0, q_ramp=0.0, wind=0.0, fp32_fields=True)
    sim = S.Sim.from_state(shape, dx, rho, stars, ["main"] * 3, [(0.0, 0.0, 1.0)] * 3, ["none"] * 3, P, rays=(8, 16),
                           fuv_grid=grid, arith=arith)
    g0 = {}
    for pairs in (0, 1):
        at.put(sim, "fuv_pairs", pairs)
        sim.fuv_field()
        torch.cuda.synchronize()
        g0[pairs] = sim.g0.numpy().astype(np.float32)
    assert np.array_equal(g0[0].view(np.int32), g0[1].view(np.int32))
    K = O.Kernels(np.float32)
    xi = sim.xi.numpy()
    ref = np.zeros(shape, np.float32)
    binr = sim.diag / grid[0]
    for st in stars:
        att = K.cast_fuv(rho, xi, st[:3], sim.P["kappa_fuv"], sim.dr, sim.nsteps, dx, binr, tuple(L), *grid)
        K.apply_fuv(att, st[:3], st[3] / sim.P["q_main"], dx, binr, ref)
    assert np.isfinite(g0[1]).all() and ref.max() > 0
    off = np.abs(g0[1] - ref) > 1e-4 * float(ref.max())
    assert off.mean() <= 1e-3, float(off.mean())
    sim.close()
