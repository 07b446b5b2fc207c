"""The chain kernels (sb_chain.cu): their fast forms, the general forms beside
them, and the two ways of dealing a cell's chains to threads.

Fields after advection and map entries are compared with the FP64 oracle at
the tolerances of the step parity tests (1e-5 normwise, 1e-4 cells); the two
ways do the same operations in the same order, so they agree bit for bit."""
import numpy as np
import pytest

import _parity as P

pytestmark = pytest.mark.gpu


# Rows beside the poles at every speed; traces of a fraction of a cell, of
# several cells over a pole, and (speed 8, dt 0.1) arcs beyond the fast forms;
# the smallest grid, whose entries lie further apart than the fast slerp takes.
@pytest.mark.parametrize("nT,speed,dt", [(8, 0.5, 0.02), (32, 8.0, 0.1), (64, 2.0, 0.1), (256, 1.0, 0.02)])
def test_advection_matches_oracle(oracle, gpulib, nT, speed, dt):
    from soapbubble_gb300 import synth
    from soapbubble_gb300.bubble import GpuBubble, make_params
    f = synth.make_fields("c0", nT, 5)
    uph, uth = synth.wind_from_stream(nT, 9, max_speed=speed)
    op = oracle.default_params(nT, dt_s=dt)
    op.t = 0.4
    op.force_reinit = 0
    ob = oracle.OracleBubble(op, f.eta, f.gamma, uth, uph, f.uair_init, f.vair_init)
    for _ in range(2):  # maps and accumulators away from their start, the same wind again
        ob.update_maps()
        ob.advection()
        ob.a["uth"][...], ob.a["uph"][...] = uth, uph
    with GpuBubble(make_params(nT, dt, solver_max_iter=2000, force_reinit=1)) as gb:
        P.sync_state(gb, ob)
        ob.update_maps()
        ob.advection()
        gb.step(1, 0.4, dt)
        for t, p in P.MAPS[:2]:
            err = P.map_err_cells(gb.download(t), gb.download(p), ob.a[t], ob.a[p], nT)
            assert err <= 1e-4, (t, err)
        assert P.rel_err(gb.download_system("eta_adv"), ob.a["eta"]) <= 1e-5
        adv = gb.download_system("gamma_adv")
        whole = adv < 25.0  # a broken cell's gamma is replaced by its maximum
        assert whole.mean() > 0.9
        assert np.max(np.abs(adv - ob.a["gamma"])[whole]) <= 1e-5 * np.abs(ob.a["gamma"]).max()


# Alone a 64- or 256-row bubble has its chains in parallel (below one thread
# per cell of a full chip); in a set of more than 152 * 1024 cells a thread
# runs them one after the other.
@pytest.mark.parametrize("sizes", [[16, 256, 256], [64] * 20, [256, 512, 8]])
def test_serial_and_parallel_chains_agree(gpulib, sizes):
    from soapbubble_gb300 import synth
    from soapbubble_gb300.bubble import GpuBatch, GpuBubble, make_params
    assert sum(2 * n * n for n in sizes) > 152 * 1024
    fields = [synth.make_fields("c0", n, 40 + k) for k, n in enumerate(sizes)]

    def bubbles(ks):
        out = []
        for k in ks:
            g = GpuBubble(make_params(sizes[k], 0.02))
            f = fields[k]
            uph, uth = synth.wind_from_stream(sizes[k], 70 + k, max_speed=2.0)
            if k == 0:
                uph[sizes[k] // 2, :3] = np.nan  # torn faces take the general forms
            g.upload_fields(f.eta, f.gamma, uth, uph, f.uair_init, f.vair_init)
            out.append(g)
        return out

    alone = bubbles([0, len(sizes) - 1])
    members = bubbles(range(len(sizes)))
    try:
        with GpuBatch(members) as batch:
            batch.step(3, 0.2, 0.02)
            batch.synchronize()
            for g in alone:
                g.step(3, 0.2, 0.02)
                g.synchronize(require_converged=False)
            for one, many in zip(alone, (members[0], members[-1])):
                for name in ("eta", "gamma", "u_theta", "u_phi", "eta_delta", "gamma_delta", "fwd_t", "bwd_p"):
                    np.testing.assert_array_equal(one.download(name), many.download(name), err_msg=name)
                assert one.stats().distortion == many.stats().distortion
    finally:
        for g in alone + members:
            g.close()
