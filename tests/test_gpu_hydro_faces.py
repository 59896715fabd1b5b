"""The hydro stage's rounding at a contact of dense, slow, cold gas and thin, fast, hot gas (a density step
of 1e5), along each axis and in both directions, against the oracle's float64 restatement of the reference
kernel.

A face flux F = a F_L + b F_R + k (U_L - U_R), 0 <= a, b <= 1 and 0 <= k <= the largest wave speed S, is a
sum of the two sides' own terms r v_c (|u| + S) (normal component: + r c^2).  Twenty roundings of 2^-24 of
those terms -- each side's mass with its own velocity, so that the digits of k r_dense never reach the thin
side's velocity -- bound the error of a face, and a cell's is dt / dx times that of its six faces and ten
roundings of its own new value.  The sides' largest values stand for their cells'."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPE, DX = (18, 37, 44), 0.02
ULP = 2.0 ** -24


def contact(axis, flip, seed):
    """rho, v, xi and the dense side's mask"""
    rng = np.random.default_rng(seed)
    n = SHAPE[axis]
    m = np.arange(n) < n // 2
    dense = np.broadcast_to((m ^ flip).reshape([-1 if a == axis else 1 for a in range(3)]), SHAPE)
    noise = lambda: 1.0 + 0.1 * rng.uniform(-1, 1, SHAPE)  # noqa: E731
    rho = np.where(dense, 300.0, 0.004) * noise()
    v = [np.where(dense, 1e-4, s * 20.0) * noise() for s in rng.choice((-1.0, 1.0), 3)]
    xi = np.where(dense, 0.0, 1.0)
    rho = rho.astype(np.float32)
    return rho, [(rho * c).astype(np.float32) for c in v], xi.astype(np.float32), dense


def allowance(rho, mom, xi, dense, ref, dt, cn2, ci2):
    """the bound above, per component and cell"""
    r64 = rho.astype(np.float64)
    v = [np.abs(m / r64) for m in mom]
    c2 = cn2 + xi.astype(np.float64) * (ci2 - cn2)
    S = float((np.sqrt(c2) + np.max(v, axis=0)).max())
    terms = [[], []]                              # by side (thin, dense): along each axis, per component
    for side in (0, 1):
        w = dense if side else ~dense
        r, vm, cc = float(r64[w].max()), [float(x[w].max()) for x in v], float(c2[w].max())
        for ax in range(3):
            f = vm[ax] + S
            terms[side].append([r * f] + [r * vm[c] * f + (r * cc if c == ax else 0.0) for c in range(3)])
    out = [10 * ULP * np.abs(u) for u in ref]
    for ax in range(3):
        pad = np.concatenate([dense.take([0], ax), dense, dense.take([-1], ax)], ax)
        n = SHAPE[ax]
        for c in range(4):
            t = np.where(pad, terms[1][ax][c], terms[0][ax][c])
            cell = t.take(range(1, n + 1), ax)
            # a face takes both its cells' terms where the sides differ
            for lo in (0, 2):
                other = pad.take(range(lo, lo + n), ax) != dense
                out[c] = out[c] + dt / DX * 20 * ULP * (cell + np.where(other, t.take(range(lo, lo + n), ax), 0.0))
    return out


@pytest.mark.parametrize("solver", ("hll", "rusanov"))
@pytest.mark.parametrize("flip", (False, True))
@pytest.mark.parametrize("axis", (0, 1, 2))
def test_contact_of_dense_and_thin_gas(axis, flip, solver):
    import oracle as O
    from nebulaviewer_gb300 import _lib, build, sim as S
    from nebulaviewer_gb300.params import make_params, sound_speeds
    build.build(verbose=False)
    P = dict(q_main=1.0, wind=0.0, jet=0.0, solver=solver, limiter="minmod", floor=2e-3, cfl=0.3, cn2=1.0, ci2=144.0,
             vmax=72.0)
    cn2, ci2, vmax = sound_speeds(make_params(base=P))
    rho, mom, xi, dense = contact(axis, flip, 10 * axis + flip)
    speed = sum(np.abs(m) for m in mom) / rho + np.sqrt(cn2 + xi * (ci2 - cn2))
    dt = float(np.float32(0.3 * DX / speed.max()))
    sim = S.Sim.from_state(SHAPE, DX, rho, [], [], [], [], P, mom=mom, rays=(8, 16), fuv_grid=(4, 4, 8),
                           start_main=False, arith="fast")
    sim._xi.copy_(torch.as_tensor(xi, device="cuda"))
    U = [torch.as_tensor(a, device="cuda") for a in [rho] + mom]
    out = [torch.full_like(U[0], float("nan")) for _ in range(4)]
    F = lambda ts: _lib.f4([t.data_ptr() for t in ts])  # noqa: E731
    _lib.check(sim._lib.nb_hydro_stage(sim._h, F(U), F(U), F(out), 0.0, 1.0, dt, 0.0), sim._h, "nb_hydro_stage")
    torch.cuda.synchronize()
    K = O.Kernels(np.float64)
    Un = [a.astype(np.float64) for a in [rho] + mom]
    ref = [np.zeros(SHAPE) for _ in range(4)]
    K.hydro_stage(Un, xi.astype(np.float64), Un, ref, a=0.0, b=1.0, stars=np.zeros((1, 4)), nstars=0, wind=0.0,
                  jets=np.zeros((1, 4)), jet_cos=1.0, jet_r=0.0, pulse=0.0, dt=dt, dx=DX, floor_=2e-3, cn2=cn2,
                  ci2=ci2, vmax=vmax, solver=1 if solver == "hll" else 0, lim=0)
    tol = allowance(rho, mom, xi, dense, ref, dt, cn2, ci2)
    for c in range(4):
        worst = float((np.abs(out[c].cpu().numpy() - ref[c]) / tol[c]).max())
        assert worst <= 1.0, (c, worst)
    sim.close()
