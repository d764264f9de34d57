"""The diagnostics' sums against the reference's own order, bit for bit, and
their partials apart from the stages'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(x):
    """One running sum, left to right."""
    return float(np.cumsum(np.asarray(x, dtype=np.float64))[-1])


def depths(kind, n, rng):
    x = rng.uniform(0.0, 3.0, n)
    if kind == "ties":                        # multiples of half an ulp of the sum
        x = rng.integers(0, 1 << 20, n) * 2.0 ** -30
        x[0] = 2.0 ** 23 + 1
    elif kind == "dry_first":
        x[: (2 * n) // 3] = 0.0
    elif kind == "wide":                      # many binades, up and down
        x = 10.0 ** rng.uniform(-30, 9, n)
    elif kind == "equal":
        x[:] = 0.1
    elif kind == "none":
        x[:] = 0.0
    elif kind == "subnormal":
        x = rng.integers(0, 9, n) * 5e-324
        x[-1] = 1e-300
    elif kind == "negative":
        x[n // 2] = -0.25
    elif kind == "lost":
        x[n // 3] = np.nan
    elif kind == "infinite":
        x[n // 2], x[n // 4] = np.inf, 1e308
        x[n // 8] = 1e308
    return x


@pytest.mark.parametrize("nx,ny", [(1, 1), (64, 64), (4097, 1), (4096, 3), (97, 211), (1030, 517)])
@pytest.mark.parametrize("kind", ["uniform", "ties", "dry_first", "wide", "equal", "none", "subnormal", "negative", "lost",
                                  "infinite"])
def test_volume_is_the_running_sum(swe, kind, nx, ny):
    rng = np.random.default_rng(nx * ny)
    h = np.full((ny + 4, nx + 4), 7.0)
    h[2:-2, 2:-2] = depths(kind, nx * ny, rng).reshape(ny, nx)
    sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=0.0, eta0=0.0)
    sim.h = h
    with np.errstate(over="ignore", invalid="ignore"):
        want = chain(h[2:-2, 2:-2].reshape(-1)) * 2.0 * 2.0
    for _ in range(2):
        got = sim.volume()
        assert got == want or (np.isnan(got) and np.isnan(want))
    sim.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (127, 9), (128, 8), (129, 17), (300, 600)])
def test_energy_and_maxima(swe, nx, ny):
    rng = np.random.default_rng(nx + ny)
    shape = (ny + 4, nx + 4)
    b, h = rng.uniform(-2.0, 0.5, shape), np.maximum(rng.uniform(-0.5, 3.0, shape), 0.0)
    hu, hv = h * rng.normal(0, 1, shape), h * rng.normal(0, 1, shape)
    hu[2, 2], hv[2, 2] = 1e-250, 0.0          # a cell outside the tame range
    sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=b, eta0=0.0)
    sim.h, sim.hu, sim.hv = h, hu, hv
    i = (slice(2, -2), slice(2, -2))
    B, H = b[i], h[i]
    u, v = sim.vel(hu[i].reshape(-1), H.reshape(-1)).reshape(ny, nx), sim.vel(hv[i].reshape(-1), H.reshape(-1)).reshape(ny, nx)
    term = np.where(H > 0, 0.5 * H * (u * u + v * v) + 0.5 * swe.G * H * (H + 2 * B), 0.0)
    assert sim.energy() == chain([chain(r) for r in term]) * 2.0 * 2.0
    wet = H > 1e-3
    assert sim.maxSurfaceDeviation(0.25) == float(np.max(np.where(wet, np.abs(B + H - 0.25), 0.0)))
    assert abs(sim.maxSpeed() - float(np.max(np.where(wet, np.hypot(u, v), 0.0)))) <= 4e-16 * sim.maxSpeed()
    assert sim.finite()
    c = np.sqrt(swe.G * H)
    rate = float(np.max(np.where(wet, (np.abs(u) + c) / 2.0 + (np.abs(v) + c) / 2.0, 0.0)))
    assert sim.maxDt() == (0.45 / rate if rate > 0 else np.inf)
    sim.close()


def test_a_diagnostic_between_steps_leaves_the_time_step_alone(swe):
    """Tiles of settled land keep their partials from step to step: a
    reduction in between must not put its own in their place."""
    from water_simulator_b200 import workloads
    b, h = workloads.beach_dam_break(nx=512, ny=160, dx=8.0)
    sims = [swe.ShallowWater(nx=512, ny=160, dx=8.0, bed=b, eta0=b + h, manning=0.03) for _ in range(2)]
    for k in range(8):
        for sim in sims:
            sim.step()
        sims[0].maxSurfaceDeviation(1e7)
        sims[0].maxSpeed()
        sims[0].volume()
        assert sims[0].maxDt() == sims[1].maxDt()
    for sim in sims:
        sim.run(4)
    assert np.array_equal(sims[0].field("h"), sims[1].field("h")) and sims[0].t == sims[1].t
    for sim in sims:
        sim.close()


@pytest.mark.parametrize("minDepth", [0.0, 1e-3, 1e15, 1e18, 1e19, 1e77, np.float64(1e80), np.inf])
def test_energy_for_any_min_depth(swe, minDepth):
    """The velocities' desingularisation is minDepth^4, infinite from about
    1e77 on: the velocities are 0 then and the energy is the potential one.
    The same bits as the velocities of the operators at every minDepth."""
    rng = np.random.default_rng(5)
    nx, ny = 130, 9
    b, h = rng.uniform(-1, 0.5, (ny + 4, nx + 4)), rng.uniform(0.5, 3.0, (ny + 4, nx + 4))
    with np.errstate(over="ignore"):
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=b, eta0=0.0, minDepth=minDepth)
    hu, hv = h * rng.normal(0, 1, h.shape), h * rng.normal(0, 1, h.shape)
    sim.h, sim.hu, sim.hv = h, hu, hv
    i = (slice(2, -2), slice(2, -2))
    B, H = b[i], h[i]
    u, v = (sim.vel(q[i].reshape(-1), H.reshape(-1)).reshape(ny, nx) for q in (hu, hv))
    term = 0.5 * H * (u * u + v * v) + 0.5 * swe.G * H * (H + 2 * B)
    assert np.all(np.isfinite(term))
    assert sim.energy() == chain([chain(r) for r in term]) * 2.0 * 2.0
    sim.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 5001), (4, 33), (5, 4), (127, 40), (128, 3), (129, 65), (1025, 2), (5001, 3),
                                   (1, 300_007), (620_003, 1)])
def test_reductions_reach_every_cell(swe, nx, ny):
    """The largest value is found, and one lost cell seen, wherever it lies:
    narrow and low grids share the blocks' threads out differently."""
    rng = np.random.default_rng(nx + ny)
    shape = (ny + 4, nx + 4)
    h = rng.uniform(1.0, 2.0, shape)
    sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=0.0, eta0=0.0)
    cells = [(0, 0), (ny - 1, nx - 1), (ny - 1, 0), (0, nx - 1)] + [(rng.integers(ny), rng.integers(nx)) for _ in range(4)]
    for j, i in cells:
        x = h.copy()
        x[j + 2, i + 2] = 9.0
        sim.h = x
        assert sim.maxSurfaceDeviation(0.0) == 9.0 and sim.finite()
        c = np.sqrt(swe.G * 9.0)
        assert sim.maxDt() == 0.45 / (c / 2.0 + c / 2.0)
        hu = np.zeros(shape)
        hu[j + 2, i + 2] = 3.0
        sim.hu = hu
        u = sim.vel(3.0, 9.0)
        assert abs(sim.maxSpeed() - u) <= 4e-16 * u
        sim.hu = np.zeros(shape)
    for j, i in [(0, 0), (ny + 3, nx + 3), (ny + 1, 1), (rng.integers(ny + 4), rng.integers(nx + 4))]:   # ghosts too
        hv = np.zeros(shape)
        hv[j, i] = np.nan
        sim.hv = hv
        assert not sim.finite()
    sim.close()


@pytest.mark.parametrize("cells", [1024, 7167, 7168, 7169])
@pytest.mark.parametrize("kind", ["uniform", "wide", "negative", "lost"])
def test_volume_where_the_plain_chain_ends(swe, kind, cells):
    """Up to 7168 cells the sum is the plain chain, from there on cut into runs."""
    h = depths(kind, cells, np.random.default_rng(cells))
    sim = swe.ShallowWater(nx=cells, ny=1, dx=2.0, bed=0.0, eta0=0.0)
    x = np.full((5, cells + 4), 7.0)
    x[2, 2:-2] = h
    sim.h = x
    got, want = sim.volume(), chain(h) * 2.0 * 2.0
    assert got == want or (np.isnan(got) and np.isnan(want))
    sim.close()
