"""The discrete adjoint on the GPU: its gradient against the tangent-linear
reference (the oracle on dual numbers, same frozen dt sequence) and against
central differences of the GPU forward, for random directions in the bed and
the Manning field; and the same gradient whatever the checkpoint interval."""
import numpy as np
import pytest

from tlm import tlm_misfit

pytestmark = pytest.mark.gpu


def case(swe, nx=40, ny=30, steps=30, seed=21):
    from water_simulator_b200 import workloads
    c = workloads.adjoint_case(nx=nx, ny=ny, dx=10.0, n_gauges=6, seed=seed, hump=0.4)
    # observations from the perturbed bed
    truth = swe.MisfitAdjoint(nx, ny, 10.0, c["b_true"], c["eta0"], manning_field=c["n"], gauges=c["gauges"],
                              steps=steps, checkpoint_every=7)
    _, eta = truth.forward()
    truth.close()
    return c, eta


def gradient(swe, c, obs, steps, every=7):
    adj = swe.MisfitAdjoint(c["nx"], c["ny"], c["dx"], c["b"], c["eta0"], manning_field=c["n"], gauges=c["gauges"],
                            steps=steps, checkpoint_every=every)
    adj.set_observations(obs)
    J, _ = adj.forward()
    gb, gn = adj.backward()
    dts = adj.dt_sequence()
    return adj, J, gb, gn, dts


def test_adjoint_matches_tangent_linear(swe):
    steps = 30
    c, obs = case(swe, steps=steps)
    adj, J, gb, gn, dts = gradient(swe, c, obs, steps)
    rng = np.random.default_rng(1)
    for trial in range(4):
        db = rng.normal(0, 1, c["b"].shape)
        dn = rng.normal(0, 1e-3, c["n"].shape) if trial >= 2 else np.zeros(c["n"].shape)
        Jt, dJ, dts_t = tlm_misfit(c, c["b"], c["n"], db, dn, steps, obs)
        assert abs(Jt - J) <= 1e-12 * abs(J)
        got = float(np.dot(gb, db.reshape(-1)) + np.dot(gn, dn.reshape(-1)))
        assert abs(got - dJ) <= 1e-8 * abs(dJ), (trial, got, dJ)
    assert np.all(gb.reshape(c["ny"] + 4, c["nx"] + 4)[:2] == 0)          # ghosts carry no gradient
    adj.close()


def test_adjoint_against_central_differences(swe):
    steps = 30
    c, obs = case(swe, steps=steps, seed=22)
    adj, J, gb, gn, dts = gradient(swe, c, obs, steps)
    rng = np.random.default_rng(2)

    def J_at(b, n):
        f = swe.MisfitAdjoint(c["nx"], c["ny"], c["dx"], b, c["eta0"], manning_field=n, gauges=c["gauges"],
                              steps=steps, checkpoint_every=steps)
        f.set_observations(obs)
        f.dt_sequence(fixed=dts)
        v, _ = f.forward()
        f.close()
        return v

    for trial in range(20):
        db = rng.normal(0, 1, c["b"].shape)
        dn = rng.normal(0, 1e-3, c["n"].shape)
        want = float(np.dot(gb, db.reshape(-1)) + np.dot(gn, dn.reshape(-1)))
        errs = []
        for eps in (1e-4, 1e-5, 1e-6, 1e-7):
            fd = (J_at(c["b"] + eps * db, c["n"] + eps * dn) - J_at(c["b"] - eps * db, c["n"] - eps * dn)) / (2 * eps)
            errs.append(abs(fd - want) / abs(want))
        assert min(errs) <= 1e-5, (trial, errs)
    adj.close()


def test_gradient_independent_of_checkpointing(swe):
    steps = 23
    c, obs = case(swe, steps=steps, seed=23)
    ref = None
    for every in (1, 5, 23):
        adj, J, gb, gn, _ = gradient(swe, c, obs, steps, every)
        if ref is None:
            ref = (gb, gn)
        else:
            assert np.array_equal(gb, ref[0]) and np.array_equal(gn, ref[1])
        adj.close()


def test_gauges_sharing_a_cell(swe):
    """Gauges may repeat a cell: their contributions add in gauge order."""
    steps = 20
    c, _ = case(swe, steps=steps, seed=24)
    g = np.asarray(c["gauges"], dtype=np.int32)
    c["gauges"] = np.concatenate([g, g[:2], g[:1]]).astype(np.int32)
    rng = np.random.default_rng(3)
    obs = rng.normal(2.0, 0.05, (steps, len(c["gauges"])))
    adj, J, gb, gn, dts = gradient(swe, c, obs, steps)
    db = rng.normal(0, 1, c["b"].shape)
    dn = rng.normal(0, 1e-3, c["n"].shape)
    Jt, dJ, _ = tlm_misfit(c, c["b"], c["n"], db, dn, steps, obs)
    assert abs(Jt - J) <= 1e-12 * abs(J)
    got = float(np.dot(gb, db.reshape(-1)) + np.dot(gn, dn.reshape(-1)))
    assert abs(got - dJ) <= 1e-8 * abs(dJ), (got, dJ)
    adj.close()


BOUNDARY_CASES = {
    "outflow_we": {"west": "outflow", "east": "outflow"},
    "periodic_all": {"west": "periodic", "east": "periodic", "south": "periodic", "north": "periodic"},
    "flather_west": {"west": ("flather", 2.05, 0.0), "east": "outflow"},
    "flather_sn_periodic_we": {"south": ("flather", 2.0, 0.01), "north": ("flather", 1.95, -0.02),
                               "west": "periodic", "east": "periodic"},
    "mixed": {"east": ("flather", 2.0, 0.0), "south": "outflow", "north": "periodic"},
    "tide_west": {"west": ("tide", 2.0, [0.3, 0.1], [2 * 3.141592653589793 / 600, 2 * 3.141592653589793 / 250],
                           [0.0, 40.0], 0.05), "east": "outflow"},
}


@pytest.mark.parametrize("name", list(BOUNDARY_CASES))
def test_adjoint_boundaries_match_tangent_linear(swe, name):
    """Outflow, periodic and Flather sides, constant or tidal
    (src/swe.mjs:1026-1126): the forward equals the oracle's, the gradient
    its tangent-linear model."""
    from water_simulator_b200 import workloads
    bcs = BOUNDARY_CASES[name]
    steps, nx, ny = 24, 40, 30
    c = workloads.adjoint_case(nx=nx, ny=ny, dx=10.0, n_gauges=6, seed=31, hump=0.4)
    kw = dict(manning_field=c["n"], gauges=c["gauges"], steps=steps, checkpoint_every=7, boundaries=bcs)
    truth = swe.MisfitAdjoint(nx, ny, 10.0, c["b_true"], c["eta0"], **kw)
    _, obs = truth.forward()
    truth.close()
    adj = swe.MisfitAdjoint(nx, ny, 10.0, c["b"], c["eta0"], **kw)
    adj.set_observations(obs)
    J, _ = adj.forward()
    gb, gn = adj.backward()
    rng = np.random.default_rng(5)
    for trial in range(3):
        db = rng.normal(0, 1, c["b"].shape)
        dn = rng.normal(0, 1e-3, c["n"].shape) if trial else np.zeros(c["n"].shape)
        Jt, dJ, _ = tlm_misfit(c, c["b"], c["n"], db, dn, steps, obs, bcs=bcs)
        assert abs(Jt - J) <= 1e-12 * abs(J), (name, Jt, J)
        got = float(np.dot(gb, db.reshape(-1)) + np.dot(gn, dn.reshape(-1)))
        assert abs(got - dJ) <= 1e-8 * abs(dJ), (name, trial, got, dJ)
    g2 = gb.reshape(ny + 4, nx + 4)
    assert np.all(g2[:2] == 0) and np.all(g2[-2:] == 0) and np.all(g2[:, :2] == 0) and np.all(g2[:, -2:] == 0)
    adj.close()


def test_adjoint_boundary_refusals(swe):
    c = swe.MisfitAdjoint(8, 8, 10.0, np.zeros(144), 1.0, gauges=[50], steps=2)
    with pytest.raises(ValueError):
        c.set_boundary("west", "sponge")
    with pytest.raises(KeyError):
        c.set_boundary("up", "reflect")
    c.close()


TIDE_WEST = {"west": ("tide", 2.0, [0.3], [2 * 3.141592653589793 / 250], [40.0], 0.05)}


@pytest.mark.parametrize("bad", [0.0, -0.5, np.inf, np.nan])
@pytest.mark.parametrize("bcs", [None, TIDE_WEST], ids=["walls", "tide"])
@pytest.mark.parametrize("at", [0, 5, 11])
def test_a_refused_step_changes_nothing(swe, at, bcs, bad):
    """A dt that step() refuses leaves the state as it was: the later steps are
    those of the run without it, and the gradient is that run's, with the
    misfit of the repeated state counted twice, for any checkpoint interval."""
    from water_simulator_b200 import workloads
    c = workloads.adjoint_case(nx=40, ny=30, dx=10.0, n_gauges=6, seed=33, hump=0.4)
    n = 11
    rng = np.random.default_rng(8)
    obs = rng.normal(2.0, 0.05, (n, 6))

    def handle(steps, every):
        return swe.MisfitAdjoint(40, 30, 10.0, c["b"], c["eta0"], manning_field=c["n"], gauges=c["gauges"],
                                 steps=steps, checkpoint_every=every, boundaries=bcs)

    plain = handle(n, n)
    plain.set_observations(obs)
    _, eta = plain.forward()
    dts = plain.dt_sequence()
    if at > 0:                                     # twice the residual of the state that repeats
        twice = obs.copy()
        twice[at - 1] = eta[at - 1] - 2 * (eta[at - 1] - obs[at - 1])
        plain.set_observations(twice)
    plain.forward()
    want = plain.backward()
    plain.close()
    got = []
    for every in (1, 5, n + 1):
        adj = handle(n + 1, every)
        adj.dt_sequence(fixed=np.insert(dts, at, bad))
        _, e0 = adj.forward()
        assert np.array_equal(np.delete(e0, at, axis=0), eta)
        assert at == 0 or np.array_equal(e0[at], eta[at - 1])
        adj.set_observations(np.insert(obs, at, obs[at - 1] if at > 0 else e0[0], axis=0))
        adj.forward()
        got.append(adj.backward())
        adj.close()
    for g in got[1:]:
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1])
    for g, w in zip(got[0], want):                 # 2r + 2r against 4r, at most 12 steps of rounding apart
        assert np.max(np.abs(g - w)) <= 1e-11 * np.max(np.abs(w))


@pytest.mark.parametrize("refused", [None, 0, 6])
@pytest.mark.parametrize("bcs", [None, {"west": ("flather", 2.05, 0.0), "east": "outflow"}], ids=["walls", "flather"])
def test_gauges_in_ghost_cells(swe, bcs, refused):
    """Gauges in ghost cells (a corner among them) read what the step left there,
    after a refused step the filled ghosts: the gradient against central
    differences with the dt sequence held, the same for any checkpoint interval."""
    from water_simulator_b200 import workloads
    nx, ny, steps = 24, 18, 12
    W = nx + 4
    c = workloads.adjoint_case(nx=nx, ny=ny, dx=10.0, n_gauges=2, seed=35, hump=0.4)
    g = np.concatenate([c["gauges"], [9 * W + 1, 9 * W + 2, 1 * W + 1, (ny + 2) * W + 7]]).astype(np.int32)
    rng = np.random.default_rng(9)
    obs = rng.normal(2.0, 0.05, (steps, len(g)))

    def handle(b, n, every, dts=None):
        adj = swe.MisfitAdjoint(nx, ny, 10.0, b, c["eta0"], manning_field=n, gauges=g, steps=steps,
                                checkpoint_every=every, boundaries=bcs)
        adj.set_observations(obs)
        if dts is not None:
            adj.dt_sequence(fixed=dts)
        return adj

    first = handle(c["b"], c["n"], steps)
    first.forward()
    dts = first.dt_sequence()
    first.close()
    if refused is not None:
        dts[refused] = 0.0
    got = []
    for every in (1, 5, steps):
        adj = handle(c["b"], c["n"], every, dts)
        _, eta = adj.forward()
        if refused is not None and bcs is None:    # the wall's ghost is its neighbour's mirror
            assert np.all(eta[refused, 2] == eta[refused, 3])
        got.append(adj.backward())
        adj.close()
    for q in got[1:]:
        assert np.array_equal(q[0], got[0][0]) and np.array_equal(q[1], got[0][1])

    def J_at(b, n):
        f = handle(b, n, steps, dts)
        v, _ = f.forward()
        f.close()
        return v

    for trial in range(4):
        db = rng.normal(0, 1, c["b"].shape)
        dn = rng.normal(0, 1e-3, c["n"].shape)
        want = float(np.dot(got[0][0], db.reshape(-1)) + np.dot(got[0][1], dn.reshape(-1)))
        errs = []
        for eps in (1e-4, 1e-5, 1e-6, 1e-7):
            fd = (J_at(c["b"] + eps * db, c["n"] + eps * dn) - J_at(c["b"] - eps * db, c["n"] - eps * dn)) / (2 * eps)
            errs.append(abs(fd - want) / abs(want))
        assert min(errs) <= 1e-5, (trial, errs)


def test_an_incomplete_tile_copy_is_reported(swe):
    """The status bit that a tile copy past its bound sets (put there by the
    test hook): forward() raises SWE_ETIMEOUT, backward() asks for a new
    forward pass, and without the bit the handle works as before."""
    c, obs = case(swe, steps=6)
    adj, J, gb, gn, _ = gradient(swe, c, obs, 6, 4)
    adj.debug_status(4)
    with pytest.raises(swe.SweError) as e:
        adj.forward()
    assert e.value.code == -4                      # SWE_ETIMEOUT
    with pytest.raises(swe.SweError) as e:
        adj.backward()
    assert e.value.code == -1                      # SWE_EINVAL: no forward pass
    adj.debug_status(0)
    assert adj.forward()[0] == J
    again = adj.backward()
    assert np.array_equal(again[0], gb) and np.array_equal(again[1], gn)
    adj.close()
