"""The bit-plane kernel with one band per SM: identical (whole numbers) to the per-half-sweep kernels
from bands of one row to the largest it holds (every number of words per draw warp and update lane), on
regions whose rows differ in width, in every random mode; epochs; coupling from the past; and
failure detection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(rt, shape):
    D = rt.DominoTiler
    d = D.AztecDiamond(shape) if isinstance(shape, int) else D.Rectangle(*shape)
    return D.MaxTiling(d), D.MinTiling(d)


def _chains(rt, tiler, starts, launch, steps):
    n = rt.side_of(starts[0])
    s = rt.DominoSampler(n, len(starts), tiler)
    for c, t in enumerate(starts):
        s.load(c, t)
    s.set_launch(*launch)
    info = s.engine_info()
    for part, seed in steps:
        if tiler.rng == "fast":
            s.run_fast(seed, -part, part)
        else:
            s.seed(seed)
            s.run(rt.mt19937_colours(seed, part))
    out = [s.store(c) for c in range(len(starts))]
    s.close()
    return out, info


@pytest.mark.parametrize("rng", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("shape,bands", [(9, 152), (31, 17), (64, 40), (100, 152), (150, 20), (333, 152), (430, 60), (512, 152),
                                         ((40, 301), 152), ((301, 40), 152), ((260, 700), 152), ((500, 498), 100)])
def test_grid_equals_per_half_sweep_kernels(rt, rng, shape, bands):
    tmax, tmin = _start(rt, shape)
    n = rt.side_of(tmax)
    tiler = rt.DominoTiler(rule="cftp_twoperiodic", rng="fast" if rng == "fast" else "tinymt", a=1.0, b=0.7,
                           fast_stream=5)
    if rng == "table":
        tiler.LoadTinyMT(np.random.RandomState(n).randint(0, 2**32, size=((n - 2) * (n // 2 - 2), 3), dtype=np.uint32))
    steps = [(70, 11), (1, 4), (2, 5), (61, 12)]
    for starts in ([tmin], [tmin, tmax]):
        got, info = _chains(rt, tiler, starts, (0, bands, 0), steps)
        assert info["engine"] == 4 and 3 <= info["bands"] <= bands
        want, _ = _chains(rt, tiler, starts, (1, 0, 0), steps)
        for g, w in zip(got, want):
            assert np.array_equal(g, w), (shape, rng, bands)


@pytest.mark.parametrize("order", [700, 1024, 1200])
@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_largest_diamonds(rt, order, rng):
    # 1200: more words a band than the registers hold in TinyMT mode, which goes to the other kernels
    tmax, tmin = _start(rt, order)
    tiler = rt.DominoTiler(rule="cftp", rng=rng)
    got, _ = _chains(rt, tiler, [tmin, tmax], (0, 0, 0), [(40, 3)])
    want, _ = _chains(rt, tiler, [tmin, tmax], (1, 0, 0), [(40, 3)])
    assert all(np.array_equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_cftp_on_the_grid_equals_the_per_half_sweep_kernels(rt, rng):
    tmax, tmin = _start(rt, (30, 400))  # few rows: coalesces soon, too wide for a cluster in TinyMT mode
    runs = []
    for engine in (0, 1):
        tiler = rt.DominoTiler(rule="cftp", rng=rng, engine=engine)
        runs.append(tiler.cftp(tmax, tmin, driver_seed=8, first_steps=400, schedule=1, max_attempts=20))
    (a, sa), (b, sb) = runs
    assert np.array_equal(a, b)
    for key in ("attempts", "total_steps", "final_steps", "flip_attempts"):
        assert sa[key] == sb[key]


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_grid_wait_gives_up_and_the_sampler_stays_usable(rt, rng):
    """Band 1 publishes none of its boundary words and a wait gives up after 4096 polls: every band
    leaves, the host reads RT_ERR_TIMEOUT, and the sampler then repeats a fresh sampler's walk."""
    tmax, tmin = _start(rt, 64)
    n = rt.side_of(tmax)
    tiler = rt.DominoTiler(rule="cftp", rng=rng)
    cols = rt.mt19937_colours(77, 64)

    def fresh():
        s = rt.DominoSampler(n, 2, tiler)
        s.load(0, tmin)
        s.load(1, tmax)
        s.set_launch(0, 40, 0)
        return s

    def go(s):
        if rng == "fast":
            s.run_fast(5, 0, 64)
        else:
            s.seed(5)
            s.run(cols)
        s.sync()

    s = fresh()
    assert s.engine_info()["bands"] > 16
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, 1, 4096) == rt.RT_OK
    with pytest.raises(rt.RTError) as err:
        go(s)
    assert err.value.status == rt.RT_ERR_TIMEOUT
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, -1, 0) == rt.RT_OK
    s.load(0, tmin)
    s.load(1, tmax)
    go(s)
    got = [s.store(0), s.store(1)]
    s.close()
    ref = fresh()
    go(ref)
    want = [ref.store(0), ref.store(1)]
    ref.close()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("rng", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("shape", [1, 2, 5, 16, 24, 61, 64, 96, 150, 200, 250, (8, 90), (300, 20), (64, 448), (301, 442)])
def test_automatic_depth_equals_per_half_sweep_kernels(rt, rng, shape):
    # 12, 8, .. 2 runs between exchanges (fewer in TinyMT mode): launches of fewer runs than that, of a whole number
    # of them and of others
    tmax, tmin = _start(rt, shape)
    n = rt.side_of(tmax)
    tiler = rt.DominoTiler(rule="cftp_twoperiodic", rng="fast" if rng == "fast" else "tinymt", a=1.0, b=0.7,
                           fast_stream=5)
    if rng == "table":
        tiler.LoadTinyMT(np.random.RandomState(n).randint(0, 2**32, size=((n - 2) * (n // 2 - 2), 3), dtype=np.uint32))
    steps = [(48, 11), (1, 4), (5, 5), (121, 12)]
    for starts in ([tmin], [tmin, tmax]):
        got, info = _chains(rt, tiler, starts, (0, 0, 0), steps)
        assert info["engine"] == 4
        want, _ = _chains(rt, tiler, starts, (1, 0, 0), steps)
        for g, w in zip(got, want):
            assert np.array_equal(g, w), (shape, rng)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("gap", [3, 8, 14, 40])
def test_components_apart(rt, rng, gap):
    # Two diamonds one above the other, of different columns, with rows between them that hold nothing that can flip
    blocks = [_start(rt, order) for order in (9, 14)]
    sides = [rt.side_of(b[0]) for b in blocks]
    n = sum(sides) + gap + 60
    n += n % 2
    starts = []
    for which in (0, 1):
        g = np.zeros((n, n), np.int32)
        row = 2
        for (pair, side, col) in zip(blocks, sides, (40, 4)):
            g[row:row + side, col:col + side] = pair[which].reshape(side, side)
            row += side + gap - gap % 2
        starts.append(g.ravel().copy())
    tiler = rt.DominoTiler(rule="cftp", rng=rng, fast_stream=1)
    steps = [(90, 3), (31, 4)]
    for use in (starts[:1], starts):
        got, info = _chains(rt, tiler, use, (0, 0, 0), steps)
        assert info["engine"] == 4
        want, _ = _chains(rt, tiler, use, (1, 0, 0), steps)
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
