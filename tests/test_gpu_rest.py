"""Films at rest and torn faces: the cells whose trace ends before it starts."""
import numpy as np
import pytest

import _parity as P

pytestmark = pytest.mark.gpu


# Parallel chains, serial chains.  (On the smallest grids neighbouring points
# are so far apart that the interpolation rounds at any fraction.)
@pytest.mark.parametrize("nT", [64, 512])
def test_a_film_at_rest_stays_where_it_is(gpulib, nT):
    """No speed, no displacement: the maps and the surfactant come out of the
    advection bit for bit as they went in (an interpolation at a fraction of
    0 is exact)."""
    from soapbubble_gb300 import synth
    from soapbubble_gb300.bubble import GpuBubble, make_params
    f = synth.make_fields("c0", nT, 5)
    uph, uth = synth.wind_from_stream(nT, 9, max_speed=1.0)
    with GpuBubble(make_params(nT, 0.02, force_reinit=1)) as gb:
        gb.upload_fields(f.eta, f.gamma, uth, uph, f.uair_init, f.vair_init)
        gb.step(3, 0.4, 0.02)  # maps away from the identity
        gb.upload("u_theta", np.zeros_like(uth))
        gb.upload("u_phi", np.zeros_like(uph))
        maps = {k: gb.download(k) for k in ("fwd_t", "fwd_p", "bwd_t", "bwd_p")}
        gamma = gb.download("gamma")
        gb.step(1, 0.4, 0.02)
        for k, m in maps.items():
            np.testing.assert_array_equal(gb.download(k), m, err_msg=k)
        np.testing.assert_array_equal(gb.download_system("gamma_adv"), gamma)


# Faces torn singly, in blocks and in whole rows; the samples around them leave
# the torn ones out (step parity's 1e-5 and 1e-4 cells, and the same faces torn
# afterwards).
@pytest.mark.parametrize("nT", [32, 64, 512])
def test_torn_faces_match_oracle(oracle, gpulib, nT):
    from soapbubble_gb300 import synth
    from soapbubble_gb300.bubble import GpuBubble, make_params
    f = synth.make_fields("c0", nT, 5)
    uph, uth = synth.wind_from_stream(nT, 9, max_speed=1.0)
    rng = np.random.Generator(np.random.PCG64(nT))
    for u in (uth, uph):
        u[rng.random(u.shape) < 0.02] = np.nan
        u[nT // 4: nT // 4 + 3, 5: nT // 2] = np.nan
        u[nT // 2, :] = np.nan
    op = oracle.default_params(nT, dt_s=0.01)
    op.t = 0.4
    op.force_reinit = 0
    ob = oracle.OracleBubble(op, f.eta, f.gamma, uth, uph, f.uair_init, f.vair_init)
    with GpuBubble(make_params(nT, 0.01, solver_tol=1e-10, solver_max_iter=2000, force_reinit=1)) as gb:
        P.sync_state(gb, ob)
        gb.step(1, 0.4, 0.01)
        adv = ob.copy()
        adv.update_maps()
        adv.advection()
        for t, p in P.MAPS[:2]:
            assert P.map_err_cells(gb.download(t), gb.download(p), adv.a[t], adv.a[p], nT) <= 1e-4
        assert P.rel_err(gb.download_system("eta_adv"), adv.a["eta"]) <= 1e-5
        assert P.rel_err(gb.download_system("gamma_adv"), adv.a["gamma"]) <= 1e-5
        ob.step()
        for k, o in (("u_theta", "uth"), ("u_phi", "uph")):
            got = gb.download(k)
            np.testing.assert_array_equal(np.isnan(got), np.isnan(ob.a[o]), err_msg=k)
            assert P.rel_err(got, ob.a[o]) <= 1e-5


def test_a_step_from_rest_costs_no_more_than_one_in_motion(gpulib):
    """The first step after an upload: cells that do not move take one form of
    the chains, not both.  A trace that stays costs less than one that moves,
    so 15 % is left to the clock; both forms took 1.5 times as long."""
    from soapbubble_gb300 import synth
    from soapbubble_gb300.bubble import GpuBubble, make_params
    f = synth.make_fields("c1", 512, 5)
    still = [np.zeros_like(f.uth), np.zeros_like(f.uph)]
    rest, motion = [], []
    with GpuBubble(make_params(512, 0.002)) as gb:
        for _ in range(8):
            gb.upload_fields(f.eta, f.gamma, *still, f.uair_init, f.vair_init)
            for times in (rest, motion):
                ms = np.zeros(16)
                gb.step_timed(1, 0.0, 0.002, ms)
                times.append(ms[:2])
    assert np.all(np.min(rest, axis=0) <= 1.15 * np.min(motion, axis=0)), (rest, motion)
