"""The branch-free face arithmetic (swe_math.cuh, the "tame" functions):
correctly rounded wherever the face kernel takes it, and the tiled kernels'
choice between it and the operators against the fused kernel, which has the
operators only, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def square_roots_near_a_boundary(most=63):
    """The doubles in [1, 4) whose square root lies within about 2^-51 ulp of
    a midpoint between doubles: x 2^k = M^2 + d for an odd M of 54 bits and
    |d| <= most, found by lifting the roots of M^2 = -d mod 2^k bit by bit."""
    out = set()
    for k, ulp in ((54, 2.0 ** -52), (55, 2.0 ** -51)):
        for d in range(-most, most + 1):
            if -d % 8 != 1:                     # an odd square is 1 mod 8
                continue
            roots = {1, 3, 5, 7}
            for b in range(3, k):
                roots = {c for r in roots for c in (r, r + (1 << b)) if (c * c + d) % (1 << (b + 1)) == 0}
            for M in {r % (1 << 54) for r in roots}:
                if M >= 1 << 53 and (M * M + d) % (1 << k) == 0 and 1 << 52 <= (M * M + d) >> k < 1 << 53:
                    out.add(((M * M + d) >> k) * ulp)
    return sorted(out)


def test_the_boundary_cases_are_found():
    roots = square_roots_near_a_boundary()
    assert len(roots) == 24 and 1 + 2.0 ** -52 in roots


@pytest.mark.gpu
def test_tame_functions_round_correctly(tmp_path):
    exe = str(tmp_path / "tame_math")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-I" + os.path.join(ROOT, "water-simulator_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "tame_math.cu")], check=True, capture_output=True, text=True)
    text = "\n".join(x.hex() for x in square_roots_near_a_boundary())
    r = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    bad = {n: int(v) for n, v in (line.split() for line in r.stdout.splitlines())}
    assert len(bad) == 10 and not any(bad.values()), bad


PLANTS = {                                       # values planted in (h, hu) cells here and there
    "none": [],
    "tiny": [(1e-40, 1e-45), (1.5, 1e-250), (2.0, -5e-324), (1e-320, 0.0)],
    "huge": [(1e13, 1.0), (2.0, 1e31), (1e200, 1e150)],
    "ones": [(2.0 - 2.0 ** -52, 1.0), (1.0 - 2.0 ** -53, -0.5), (4.0 - 2.0 ** -51, 1.0), (2.0 - 2.0 ** -52, 0.0)],
    "lost": [(np.nan, 0.0), (np.inf, 1.0), (1.0, -np.inf), (-0.5, 0.25), (-0.0, -0.0)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("plant", sorted(PLANTS))
@pytest.mark.parametrize("nx,ny", [(1, 1), (32, 8), (61, 19), (70, 41)])
@pytest.mark.parametrize("kw", [{}, {"limiter": "minmod"}, {"limiter": "central", "order": 1}, {"minDepth": 1e-30},
                                {"minDepth": 0.0}, {"dx": 1e-25}, {"sphere": {"lat0": -60.0, "lat1": 60.0}}],
                         ids=lambda k: "-".join(k) or "plain")
def test_tame_tiles_and_the_others_give_the_fused_kernels_bits(swe, monkeypatch, plant, nx, ny, kw):
    rng = np.random.default_rng(nx + 7 * ny)
    shape = (ny + 4, nx + 4)
    b = rng.uniform(-0.3, 0.3, shape)
    h = np.where(rng.random(shape) < 0.15, 0.0, rng.uniform(0.0, 3.0, shape))
    hu, hv = (h * rng.normal(0.0, 2.0, shape) * (rng.random(shape) < 0.8) for _ in range(2))
    h[:, shape[1] // 2:] = 2.0 - b[:, shape[1] // 2:]              # a lake at rest beside it
    hu[:, shape[1] // 2:] = 0.0
    for k, (x, q) in enumerate(PLANTS[plant]):
        j, i = 2 + (5 * k) % ny, 2 + (11 * k + 3) % nx
        h[j, i], hu[j, i] = x, q
    args = dict(nx=nx, ny=ny, bed=b, eta0=0.0, manning=0.0)
    args.update(kw)
    if "sphere" not in kw:
        args.setdefault("dx", 2.0)
    out = []
    for impl in ("fused", "split"):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        sim = swe.ShallowWater(**args)
        sim.h, sim.hu, sim.hv = h, hu, hv
        for _ in range(2):
            sim.step(1e-3)
        out.append([sim.field(f).copy() for f in ("h", "hu", "hv")])
        sim.close()
    for x, y in zip(*out):
        assert np.array_equal(np.isnan(x), np.isnan(y))
        fine = ~np.isnan(x)
        assert np.array_equal(x[fine].view(np.uint64), y[fine].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(28, 4), (29, 5), (590, 244), (589, 245), (1000, 1140), (1001, 1200)])
@pytest.mark.parametrize("sides", ["mixed", "periodic", "tide"])
def test_every_size_of_step_gives_the_fused_kernels_bits(swe, monkeypatch, nx, ny, sides):
    """A step's launches depend on the grid's size (ghosts and dt within the
    face kernel, one wave or several, one block to close or 32, tile lists)
    and on whether its width is even: all against the fused kernels."""
    rng = np.random.default_rng(nx)
    b = rng.uniform(-0.3, 0.3, (ny + 4, nx + 4))
    b[:, (2 * nx) // 3:] = 3.0                   # dry land, settled tiles on the larger grids
    eta = np.where(np.arange(nx + 4) < nx // 3, 2.0, 1.2)[None, :].repeat(ny + 4, 0)
    out = []
    for impl in ("fused", "split"):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        sim = swe.ShallowWater(nx=nx, ny=ny, dx=2.0, bed=b, eta0=eta, manning=0.0, coriolis=1e-4)
        if sides == "periodic":
            sim.boundaries = {s: swe.periodic for s in ("west", "east", "south", "north")}
        elif sides == "tide":
            sim.boundaries.west = swe.flather(swe.Tide({"M2": [0.3, 20.0], "S2": [0.1, 5.0]}, msl=2.0).signal())
        else:
            sim.boundaries = {"west": swe.flather(lambda t: 2.0, lambda t: 0.1), "east": swe.outflow,
                              "south": swe.reflect, "north": swe.outflow}
        sim.step(1e-3)
        assert sim.run(5) == 5 if sides != "mixed" else sim.run(2) == 2
        t_end = sim.t + 1.5 * sim.maxDt()
        sim.run(6, tEnd=t_end)                  # the third step of these is refused
        out.append([sim.field(f).view(np.uint64).copy() for f in ("h", "hu", "hv", "b")] + [sim.t, sim.maxDt()])
        sim.close()
    for x, y in zip(out[0][:4], out[1][:4]):
        assert np.array_equal(x, y)
    assert out[0][4:] == out[1][4:]


@pytest.mark.gpu
def test_a_flather_side_that_is_set_again_or_changed(swe, monkeypatch):
    """A driver sets its Flather sides before every run: the same values leave
    the captured steps alone, others take effect at once."""
    def tide(a):
        return swe.flather(swe.Tide({"M2": [a, 30.0]}, msl=2.0).signal())
    out = []
    for impl in ("fused", "split"):
        monkeypatch.setenv("SWE_B200_STAGE", impl)
        sim = swe.ShallowWater(nx=90, ny=40, dx=5.0, bed=0.0, eta0=2.0, manning=0.0)
        for west in (tide(0.5), tide(0.5), tide(0.25), swe.reflect, tide(0.25), tide(0.5)):
            sim.boundaries.west = west
            sim.run(64)
        out.append([sim.field(f).copy() for f in ("h", "hu", "hv")] + [sim.t])
        sim.close()
    assert all(np.array_equal(x, y) for x, y in zip(out[0][:3], out[1][:3])) and out[0][3] == out[1][3]
    assert np.max(np.abs(out[0][1])) > 0
