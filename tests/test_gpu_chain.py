"""Chains of fused steps: several steps in one call (the sediment gather runs
in the next step's first kernel) against the same steps one call at a time,
bit for bit, with and without talus passes, by direct launches and by graph,
for batches of unlike worlds, and where k_transport's strips and chunks end
unevenly."""
import time

import numpy as np
import pytest

import hydrogen as H

pytestmark = pytest.mark.gpu


def make(n, cfg="config2", smooth=False, seed=0, graph=H.HG_AUTO, thermal=True):
    w = H.World(n)
    w.init_heightmap(H.noise(seed=seed))
    H.configure(w, cfg)
    s = H.settings_config2() if thermal else H.settings_config1()
    if smooth:
        s.Kspeed[1] = 2.0
    w.set_erosion(s)
    w.set_options(H.options(H.RAIN_BERNOULLI, p=0.02, seed=seed, graph=graph))
    return w


def assert_same(a, b, ctx):
    for f in H.STATE_FIELDS:
        x, y = a.download(f), b.download(f)
        assert np.array_equal(x, y), f"{ctx} {f}: {np.count_nonzero(x != y)} cells differ"
    assert a.step_count == b.step_count


@pytest.mark.parametrize("thermal", [True, False])
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("calls", [[2], [3, 1, 2], [5], [9, 8, 3]])
def test_chained_steps_equal_single_steps(thermal, graph, calls):
    a, b = make(192, graph=graph, thermal=thermal), make(192, graph=graph, thermal=thermal)
    for k in calls:
        a.step(k, H.MODE_FUSED)
        for _ in range(k):
            b.step(1, H.MODE_FUSED)
        assert_same(a, b, f"after {a.step_count} steps")


@pytest.mark.parametrize("smooth", [False, True])
def test_batch_of_unlike_worlds_in_a_chain(smooth):
    def worlds():
        return [make(64, seed=1), make(320, seed=2, thermal=False), make(192, seed=3, smooth=smooth),
                make(128, cfg="config1", seed=4)]

    a, b = worlds(), worlds()
    batch = H.Batch(a)
    batch.step(5)
    batch.step(1)
    batch.sync()
    for w in b:
        w.step(6, H.MODE_PLAIN)
    for i, (x, y) in enumerate(zip(a, b)):
        assert_same(x, y, f"terrain {i}")
    batch.close()


@pytest.mark.parametrize("n", [64, 960, 1536])
def test_strips_and_chunks_against_per_pass(n):
    a, b = make(n, seed=5), make(n, seed=5)
    a.step(3, H.MODE_FUSED)
    b.step(3, H.MODE_PLAIN)
    assert_same(a, b, f"{n}")


def make2(n, seed=0, thermal=True, dirt_talus=True):
    w = H.World(n, layers=2)
    w.init_reference_heightmap(H.map_settings(hmap_dims=(n, n), seed=0.1 * seed, scale=0.006))
    s = H.ErosionSettings()
    H.check(H.lib.hg_default_erosion_settings(H.ctypes.byref(s)))
    s.d_t, s.G = 0.02, 9.81
    s.Kalpha[0], s.Kalpha[1] = 0.6, 0.4
    if not thermal:
        s.Kspeed[0] = 0.0
    if not dirt_talus:
        s.Kspeed[1] = 0.0
    w.set_erosion(s)
    w.set_rain(H.rain_uniform(0.5, 1))
    w.set_options(H.options(H.RAIN_BERNOULLI, p=0.02, seed=seed))
    return w


@pytest.mark.parametrize("n", [64, 192, 832])
@pytest.mark.parametrize("thermal,dirt_talus", [(True, True), (True, False), (False, True), (False, False)])
def test_two_layer_chain_against_per_pass(n, thermal, dirt_talus):
    a, b = make2(n, 1, thermal, dirt_talus), make2(n, 1, thermal, dirt_talus)
    for k in (3, 1, 4):
        a.step(k, H.MODE_FUSED)
        b.step(k, H.MODE_PLAIN)
        for f in H.STATE_FIELDS + ["dirt", "sediment_dirt"]:
            x, y = a.download(f), b.download(f)
            assert np.array_equal(x, y), f"{f} after {a.step_count}: {np.count_nonzero(x != y)} cells differ"


@pytest.mark.parametrize("n", [72, 760, 776, 2040, 2056])
@pytest.mark.parametrize("rain", ["uniform", "bernoulli"])
def test_joined_passes_against_single_ones(n, rain):
    """The per-pass step joins passes (the gather in the talus launch up to a
    side of 768, in its own above; marching talus warps from 2048 up): the bits
    of the passes run one by one."""
    worlds = []
    for _ in range(2):
        w = H.World(n)
        w.init_heightmap(H.noise(seed=5))
        H.configure(w, "config2")
        if rain == "uniform":
            w.set_rain(H.rain_uniform(0.01, 2))
            w.set_options(H.options(H.RAIN_UNIFORM))
        else:
            w.set_options(H.options(H.RAIN_BERNOULLI, p=0.05, seed=3))
        worlds.append(w)
    a, b = worlds
    for k in range(4):
        a.step(1, H.MODE_PLAIN)
        b.run_pass("rain")
        b.run_pass("flux")
        b.run_pass("erosion")
        b.run_pass("sediment")
        b.run_pass("thermal_flux")
        b.run_pass("thermal_transport")
        b.step_count = k + 1
    for f in ("rock", "water", "sediment", "flux_l", "flux_r", "flux_t", "flux_b", "vel_u", "vel_v", "vel_z"):
        x, y = a.download(f), b.download(f)
        assert np.array_equal(x, y), f"{f}: {np.count_nonzero(x != y)} cells differ"


@pytest.mark.parametrize("n", [384, 448, 2112, 4160])
def test_forms_of_the_talus_launch_against_per_pass(n):
    """Either side of the lines between rows, tiles and marching warps: a chain
    (launches with and without the gather) and a single step."""
    a, b = make(n, seed=6), make(n, seed=6)
    a.step(3, H.MODE_FUSED)
    a.step(1, H.MODE_FUSED)
    b.step(4, H.MODE_PLAIN)
    assert_same(a, b, f"{n}")
    a.close()
    b.close()


def test_marching_batch_against_per_pass():
    """Two groups of two worlds, each group large enough for marching warps
    with the gather too."""
    def worlds():
        return [make(2944, seed=k, thermal=k != 2, graph=0) for k in range(4)]

    a, b = worlds(), worlds()
    batch = H.Batch(a)
    batch.step(3)
    batch.step(1)
    batch.sync()
    for w in b:
        w.step(4, H.MODE_PLAIN)
    for i, (x, y) in enumerate(zip(a, b)):
        assert_same(x, y, f"terrain {i}")
    batch.close()
    for w in a + b:
        w.close()


def test_talus_launch_of_a_middle_sized_world():
    """At 1024² the talus passes with the sediment gather take about as long as
    the rest of the step; a warp per strip of four rows took 1.75 times that."""
    w = make(1024)
    w.set_options(H.options(H.RAIN_UNIFORM))
    w.step(8, H.MODE_FUSED)

    def us(which, k=40):
        best = 1e9
        for _ in range(10):
            w.sync()
            t0 = time.perf_counter()
            for _ in range(k):
                w.fused_pass(which)
            w.sync()
            best = min(best, (time.perf_counter() - t0) / k)
        return best * 1e6

    us(0), us(1)
    hydro, transport = us(0), us(1)
    w.close()
    assert transport < 1.45 * hydro, f"{transport:.1f} us, {hydro:.1f} us"


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("n", [512, 576, 4160])
def test_tiles_of_8_rows_either_side_of_the_small_launch(n, graph):
    """Tiles of 8 rows on request: a block of 256 threads in small launches, of
    128 in larger ones, a world alone and in a batch."""
    def world(k):
        w = make(n, seed=k)
        w.set_options(H.options(H.RAIN_BERNOULLI, p=0.02, seed=k, tile=(64, 8), graph=graph))
        return w

    a, b = world(7), world(7)
    a.step(3, H.MODE_FUSED)
    a.step(1, H.MODE_FUSED)
    b.step(4, H.MODE_PLAIN)
    assert_same(a, b, f"{n}")
    if n < 4096:
        ws, small = [world(8), make(64, seed=9)], [world(8), make(64, seed=9)]
        batch = H.Batch(ws)
        batch.step(3)
        batch.sync()
        for x, y in zip(ws, small):
            y.step(3, H.MODE_PLAIN)
            assert_same(x, y, f"batch {n}")
        batch.close()
    a.close()
    b.close()


def test_tiles_of_8_rows_keep_up_at_4096():
    """Single steps without talus by tiles of 8 and of 16 rows (1.15 times when a
    thread of an 8-row tile had one pair of cells at every size)."""
    w = make(4096, thermal=False)
    us = {}
    for rows in (16, 8):
        w.set_options(H.options(H.RAIN_UNIFORM, tile=(64, rows), graph=0))
        us[rows] = 1e9
        for _ in range(6):
            w.sync()
            t0 = time.perf_counter()
            for _ in range(12):
                w.step(1, H.MODE_FUSED)
            w.sync()
            us[rows] = min(us[rows], (time.perf_counter() - t0) / 12 * 1e6)
    w.close()
    assert us[8] < 1.07 * us[16], us
