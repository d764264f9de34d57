"""Every GPU parity case of test_parity_gpu.py again, with the stage run by
the two tiled kernels (k_split_faces, k_split_cells) instead of the fused
row-marching kernel: the same bit-for-bit comparison against the oracle."""
import pytest

from test_parity_gpu import *  # noqa: F401,F403  (the cases themselves)


@pytest.fixture(autouse=True)
def _stage_kernels(monkeypatch):
    monkeypatch.setenv("SWE_B200_STAGE", "split")


def test_the_handles_run_the_tiled_kernels(swe):
    import ctypes
    sim = swe.ShallowWater(nx=40, ny=30, dx=1.0, bed=-1.0, eta0=0.0)
    impl = ctypes.c_int(-1)
    swe._lib.check(swe.load_library().swe_get_stage_kernels(sim._h, ctypes.byref(impl)))
    assert impl.value == 1
    sim.close()


@pytest.mark.parametrize("case", ["beach", "sphere", "beach_sponge"])
def test_tiled_and_fused_give_the_same_bits(swe, case, monkeypatch):
    """Down to the sign of zero: the tiled pair (with its dry-tile skip and
    the tiles it settles to +0 without computing them) against the fused
    kernel, after many steps of a flooding beach, of a sphere with land, and
    of the beach with a sponge over its dry east end (the sponge pours water
    onto dry tiles, so no tile may settle under it)."""
    import numpy as np
    from water_simulator_b200 import workloads

    def make():
        if case in ("beach", "beach_sponge"):
            b, h = workloads.beach_dam_break(nx=256, ny=96, dx=8.0)
            sim = swe.ShallowWater(nx=256, ny=96, dx=8.0, bed=b, eta0=b + h, manning=0.03)
            sim.boundaries = {"west": swe.flather(lambda t: 0.0, lambda t: 0.0)}
            if case == "beach_sponge":
                eta_ref = float(np.max(b)) + 0.5
                sim.forcing = swe.makeSponge(sim, side="east", width=40, strength=0.05, etaRef=eta_ref)
            return sim
        c = workloads.globe_tide(nx=180, ny=90, lat0=-80.0, lat1=80.0, modes=12)
        return swe.ShallowWater(nx=180, ny=90, bed=c["b"], eta0=c["eta0"] + (c["b"] < 0) * 0.5,
                                sphere={"R": 6371e3, "lat0": -80.0, "lat1": 80.0, "omega": 7.2921e-5})

    out = {}
    for impl in ("fused", "split"):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        sim = make()
        assert sim.run(200) == 200
        out[impl] = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")] + [sim.t]
        sim.close()
    for a, b in zip(out["fused"][:3], out["split"][:3]):
        assert np.array_equal(a, b)
    assert out["fused"][3] == out["split"][3]


def test_dry_tile_flags_follow_host_writes(swe, monkeypatch):
    """The cell kernel records which tiles it left with h == 0 everywhere,
    and the next face kernel skips tiles whose 3 x 3 neighbourhood is so
    recorded.  Every other writer of the state clears those records: water
    poured onto dry land by the host, dryClean, friction, and a switch to
    the fused kernels and back.  Through all of them the tiled pair stays
    bit-identical (uint64 patterns) to the fused kernel."""
    import ctypes
    import numpy as np
    from water_simulator_b200 import workloads
    lib = swe.load_library()

    def scenario(impl):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        b, h = workloads.beach_dam_break(nx=256, ny=96, dx=8.0)
        sim = swe.ShallowWater(nx=256, ny=96, dx=8.0, bed=b, eta0=b + h, manning=0.03)
        sim.boundaries = {"west": swe.flather(lambda t: 0.0, lambda t: 0.0)}
        assert sim.run(40) == 40
        hh = np.array(sim.field("h")).reshape(sim.H, sim.W)
        assert (hh[30:70, 160:240] == 0).all()            # dry land, tiles deep inside it
        hh[40:60, 170:230] += 0.7                         # a pond poured onto it
        sim.h = hh.reshape(-1)
        assert sim.run(30) == 30
        sim.dryClean()
        assert sim.run(10) == 10
        sim.applyFriction(sim.maxDt())
        assert sim.run(10) == 10
        other = 0 if impl == "split" else 1               # there and back
        mine = 1 - other
        swe._lib.check(lib.swe_set_stage_kernels(sim._h, other))
        assert sim.run(5) == 5
        swe._lib.check(lib.swe_set_stage_kernels(sim._h, mine))
        assert sim.run(25) == 25
        out = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")] + [sim.t]
        sim.close()
        return out

    fused, split = scenario("fused"), scenario("split")
    for a, b in zip(fused[:3], split[:3]):
        assert np.array_equal(a, b)
    assert fused[3] == split[3]


@pytest.mark.parametrize("nx,ny", [(256, 96), (255, 97), (30, 9)])
def test_tensor_map_tile_copies_give_the_same_bits(swe, monkeypatch, nx, ny):
    """The face kernel's state tile and the cell kernel's face and depth
    tiles fetched by tensor-map copies (even padded width) against the
    per-element loads (SWE_B200_TMA=0): the same bits after 150 steps of a
    flooding beach with friction, tiles at every edge of the grid and tiles
    beside dry ones included (the copies fill outside the grid with zeros,
    and faces of dry tiles are read as +0 either way).  An odd padded width
    always takes the per-element loads."""
    import numpy as np
    from water_simulator_b200 import workloads

    def run(tma):
        monkeypatch.setenv("SWE_B200_TMA", "1" if tma else "0")
        b, h = workloads.beach_dam_break(nx=nx, ny=ny, dx=8.0 * 256 / nx)
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=8.0 * 256 / nx, bed=b, eta0=b + h, manning=0.03)
        sim.boundaries = {"west": swe.flather(swe.Tide({}, msl=0.0).signal()), "north": swe.outflow}
        assert sim.run(150) == 150
        out = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")] + [sim.t]
        sim.close()
        return out

    a, b = run(True), run(False)
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)
    assert a[3] == b[3]


@pytest.mark.parametrize("nx,ny", [(256, 96), (512, 384)])
def test_face_tile_list_gives_the_same_bits(swe, monkeypatch, nx, ny):
    """The face kernel over the list of tiles that do not settle, on a grid
    of resident CTAs, against one CTA per tile (SWE_B200_FACE_LIST=0): the
    same bits after 150 steps of a flooding beach, where most tiles settle
    and the list changes as the water moves."""
    import numpy as np
    from water_simulator_b200 import workloads

    def run(on):
        monkeypatch.setenv("SWE_B200_FACE_LIST", "1" if on else "0")
        b, h = workloads.beach_dam_break(nx=nx, ny=ny, dx=8.0 * 256 / nx)
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=8.0 * 256 / nx, bed=b, eta0=b + h, manning=0.03)
        sim.boundaries = {"west": swe.flather(swe.Tide({}, msl=0.0).signal())}
        assert sim.run(150) == 150
        out = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")] + [sim.t, sim.massFloored]
        sim.close()
        return out

    a, b = run(True), run(False)
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)
    assert a[3:] == b[3:]


@pytest.mark.parametrize("nx,ny", [(2050, 1800), (1801, 2047)])
def test_looped_tile_lists_give_the_same_bits(swe, monkeypatch, nx, ny):
    """A grid on which more than 8192 tiles settle and more than 4736 are
    listed, so that the listed kernels' CTAs take several tiles each: the
    same bits as without the lists (SWE_B200_FACE_LIST=0).  An odd width has
    no tensor map of the state."""
    import numpy as np
    from water_simulator_b200 import workloads

    X = np.arange(nx + 4)[None, :] / nx + 0 * np.arange(ny + 4)[:, None]
    b = 40.0 * (X - 0.35) + workloads.uniform_noise(7, X.shape, -0.2, 0.2)
    eta = np.maximum(b, np.where(X < 0.33, 0.5, 0.0))

    def run(on):
        monkeypatch.setenv("SWE_B200_FACE_LIST", "1" if on else "0")
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=b, eta0=eta, manning=0.03)
        assert sim.run(150) == 150 and sim.run(20) == 20
        out = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")] + [sim.t, sim.massFloored]
        sim.close()
        return out

    a, b_ = run(True), run(False)
    for x, y in zip(a[:3], b_[:3]):
        assert np.array_equal(x, y)
    assert a[3:] == b_[3:]


@pytest.mark.parametrize("side", ["west", "east", "south", "north", "inside"])
@pytest.mark.parametrize("nx,ny", [(96, 40), (97, 41)])
def test_a_single_limited_cell_next_to_a_tile(swe, monkeypatch, nx, ny, side):
    """The cell kernel looks for limited cells in a tile and in the cells
    beside it, and reads theta only then.  A cell of thin, fast water on each
    side of the tile of columns 32 to 63 and rows 16 to 23 (padded), and
    inside it, on dry land: 0.9 s at 26 m/s would take 2.3 times what it
    holds over one 10 m face.  The same bits as the fused kernel, which forms
    theta for every cell."""
    import numpy as np

    j, i = {"west": (18, 31), "east": (19, 64), "south": (15, 40), "north": (24, 50), "inside": (20, 45)}[side]

    def run(impl):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        b = np.zeros((ny + 4, nx + 4))
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=10.0, bed=b, eta0=b)
        state = {f: b.copy() for f in ("h", "hu", "hv")}
        state["h"][17:22, 34:38] = 0.5               # calm, so that the tile has water of its own
        state["h"][j, i], state["hu"][j, i], state["hv"][j, i] = 0.05, 1.3, -0.9
        for f, v in state.items():
            setattr(sim, f, v.reshape(-1))
        for _ in range(3):
            sim.step(0.9)
        out = [sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv")]
        sim.close()
        return out

    for x, y in zip(run("fused"), run("split")):
        assert np.array_equal(x, y)


def _bits(sim):
    import numpy as np
    return [sim.field(f).view(np.uint64).copy() for f in ("b", "h", "hu", "hv")], (sim.t, sim.massFloored)


def _fused_and_split(monkeypatch, scenario):
    import numpy as np
    out = {}
    for impl in ("fused", "split"):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        out[impl] = scenario()
    for a, b in zip(out["fused"], out["split"]):
        for x, y in zip(a[0], b[0]):
            assert np.array_equal(x, y)
        assert a[1] == b[1]


@pytest.mark.parametrize("sides", ["walls", "mixed"])
@pytest.mark.parametrize("nx,ny", [(604, 244), (604, 252), (801, 503), (1180, 1020), (1180, 1028)])
def test_wet_grids_of_several_waves_give_the_fused_kernels_bits(swe, monkeypatch, nx, ny, sides):
    """589, 608, 1664, 4736 and 4773 tiles: on the second to the fourth the face
    kernel fills the ghosts and prepares the step, once a run of 128 steps or
    more has found that few tiles settle; the first never settles, the last is
    too large.  Then runs with a fixed dt, to a given time, past it (refused
    steps) and single steps, which settle again."""
    import numpy as np
    from water_simulator_b200 import workloads

    X, Y = np.meshgrid(np.arange(nx + 4) / 40.0, np.arange(ny + 4) / 30.0)
    b = 0.4 * np.sin(X) * np.cos(Y) + workloads.uniform_noise(3, X.shape, -0.1, 0.1)
    b[ny // 2:ny // 2 + 20, 40:90] = 3.0              # an island

    def scenario():
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=5.0, bed=b, eta0=np.where(X < 5, 2.4, 2.0))
        if sides == "mixed":
            sim.boundaries = {"west": swe.flather(swe.Tide({"M2": [0.4, 30.0]}, msl=2.1).signal()), "east": swe.outflow,
                              "south": swe.periodic, "north": swe.periodic}
        assert sim.run(133) == 133
        out = [_bits(sim)]
        assert sim.run(5, dt=0.2) == 5
        done = sim.run(40, tEnd=sim.t + 1.0)
        assert 0 < done < 40 and sim.run(3, tEnd=sim.t) == 0
        out.append(_bits(sim))
        for _ in range(2):
            sim.step()
        sim.step(0.1)
        assert sim.run(9) == 9
        out.append(_bits(sim))
        sim.close()
        return out

    _fused_and_split(monkeypatch, scenario)


@pytest.mark.parametrize("case", ["beach", "sphere", "beach_sponge", "host_writes"])
def test_settling_grids_of_several_waves_give_the_fused_kernels_bits(swe, monkeypatch, case):
    """Grids of more than 592 tiles, which alone settle: a flooding beach, a
    sphere with land, a sponge that pours water onto dry tiles, and a state that
    the host, dryClean, friction and the fused kernels write in between."""
    import numpy as np
    from water_simulator_b200 import workloads
    lib = swe.load_library()

    def beach():
        b, h = workloads.beach_dam_break(nx=640, ny=320, dx=8.0 * 256 / 640)
        sim = swe.ShallowWater(nx=640, ny=320, dx=8.0 * 256 / 640, bed=b, eta0=b + h, manning=0.03)
        sim.boundaries = {"west": swe.flather(swe.Tide({}, msl=0.0).signal())}
        return sim, b

    def scenario():
        if case == "sphere":
            c = workloads.globe_tide(nx=720, ny=360, lat0=-80.0, lat1=80.0, modes=12)
            sim = swe.ShallowWater(nx=720, ny=360, bed=c["b"], eta0=c["eta0"] + (c["b"] < 0) * 0.5,
                                   sphere={"R": 6371e3, "lat0": -80.0, "lat1": 80.0, "omega": 7.2921e-5})
            assert sim.run(150) == 150
            out = [_bits(sim)]
            sim.close()
            return out
        sim, b = beach()
        if case == "beach_sponge":
            sim.forcing = swe.makeSponge(sim, side="east", width=60, strength=0.05, etaRef=float(np.max(b)) + 0.5)
        assert sim.run(150) == 150
        out = [_bits(sim)]
        if case == "host_writes":
            hh = np.array(sim.field("h")).reshape(sim.H, sim.W)
            assert (hh[100:220, 400:600] == 0).all()      # dry land, tiles deep inside it
            hh[140:180, 430:560] += 0.7                   # a pond poured onto it
            sim.h = hh.reshape(-1)
            assert sim.run(30) == 30
            out.append(_bits(sim))
            sim.dryClean()
            assert sim.run(10) == 10
            sim.applyFriction(sim.maxDt())
            assert sim.run(10) == 10
            mine = 0 if monkeypatch_impl() == "fused" else 1
            swe._lib.check(lib.swe_set_stage_kernels(sim._h, 1 - mine))
            assert sim.run(5) == 5
            swe._lib.check(lib.swe_set_stage_kernels(sim._h, mine))
            assert sim.run(25) == 25
        for _ in range(4):
            sim.step()
            sim.maxSurfaceDeviation(1e7)                  # its partials are not the stages'
        assert sim.run(33) == 33
        out.append(_bits(sim))
        sim.close()
        return out

    def monkeypatch_impl():
        import os
        return os.environ["SWE_B200_STAGE"]

    _fused_and_split(monkeypatch, scenario)
