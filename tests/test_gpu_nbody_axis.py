"""DOP853 n-body systems with three lanes to a body (few systems of up to ten bodies in a
static frame) against a lane per body (many systems) and the oracle: systems that fill
the warp, one more body than fits, several turns of pulling bodies, bodies without a
pull between them, and unlike bodies side by side.

The two forms add the pulls and the norm in another order: units in the last place per
step, 1e-12 of the state over 40 Myr; the oracle is held to the 1e-11 of the n-body
parity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members,massive,null", [(1, 1, 0), (4, 4, 1), (10, 0, None), (10, 10, 4), (10, 4, 3), (11, 5, 2)])
def test_three_lanes_to_a_body(oracle, members, massive, null):
    import gala_gb300 as g
    from gala_gb300 import workloads as W
    from gala_gb300.nbody import BODY_DTYPE, integrate_systems, pack_bodies

    mw = W.mw_composite()
    H = g.Hamiltonian(mw)
    kinds = [lambda: g.PlummerPotential(2e9, 0.5), lambda: g.KeplerPotential(1e7), lambda: g.NFWPotential(m=3e9, r_s=2.0),
             lambda: g.MiyamotoNagaiPotential(1e9, 0.5, 0.2), lambda: g.HernquistPotential(1e9, 0.7)]
    one = [None if i == null else kinds[i % len(kinds)]() for i in range(massive)]
    base = np.ascontiguousarray(W.mw_ics(3 * members, seed=40 + members).T.reshape(3, members, 6))
    t = np.arange(41.0)
    got = {}
    for n in (3, 8 * 200 + 1):  # more than eight per SM
        w0 = np.ascontiguousarray(np.tile(base, (n // 3 + 1, 1, 1))[:n])
        bodies = pack_bodies([one] * n) if massive else np.zeros((n, 0), dtype=BODY_DTYPE)
        w, st, stats = integrate_systems(H, bodies, w0, t, atol=1e-12, rtol=1e-10, out_stride=4, return_stats=True)
        assert bool((st == 1).all())
        last, _ = integrate_systems(H, bodies, w0, t, atol=1e-12, rtol=1e-10, save_all=False)
        got[n] = w[:3].cpu().numpy(), stats[:3].cpu().numpy(), last[:3].cpu().numpy()
    few, many = got.values()
    scale = np.maximum(np.linalg.norm(many[0], axis=-1, keepdims=True), 1.0)
    assert np.all(np.abs(few[0] - many[0]) <= 1e-12 * scale)
    assert np.all(np.abs(few[2] - many[0][:, -1]) <= 1e-12 * scale[:, -1])
    assert np.array_equal(few[1], many[1])
    ref, idid = oracle.nbody_dop853(mw, pack_bodies([one])[0] if massive else np.zeros(0, dtype=BODY_DTYPE), massive, base[0], t,
                                    atol=1e-12, rtol=1e-10)
    assert idid == 1 and np.all(np.abs(few[0][0] - ref[::4]) <= 1e-11 * scale[0])
