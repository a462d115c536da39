"""Kernels that the size-based choices reach only on certain domains, each on one that reaches it (the planned
route is checked), against the per-half-sweep kernels or the oracle: the cluster's couplings, every number of
words a draw warp of the one-band-per-SM kernel in fast mode, its waits that give up, and walks longer than
one launch."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER, GRID = 1, 2


def _route(rt):
    out = (C.c_int32 * 4)()
    assert rt.lib().rt_test_route(out) == rt.RT_OK
    return dict(zip(("engine", "form", "bands", "depth"), out))


def _start(rt, shape):
    D = rt.DominoTiler
    d = D.AztecDiamond(shape) if isinstance(shape, int) else D.Rectangle(*shape)
    return D.MaxTiling(d), D.MinTiling(d)


@pytest.mark.parametrize("rng,shape,schedule,firsts", [
    ("tinymt", (20, 1000), 1, (64, 500)), ("tinymt", (4, 1200), 1, (2, 16, 100, 2000)),
    ("tinymt", (4, 1200), 0, (40, 150)), ("tinymt", (2, 1300), 1, (2, 5, 12, 30, 64)),
    ("fast", (2, 3000), 1, (1, 8, 200)), ("fast", (4, 3000), 1, (4, 32, 1000))])
def test_cluster_couplings(rt, rng, shape, schedule, firsts):
    """Short first look-backs end in different attempts, so in different ones of the four clusters; a long one
    coalesces in several at once."""
    tmax, tmin = _start(rt, shape)
    seen = set()
    for first in firsts:
        runs = []
        for engine in (0, 1):
            tiler = rt.DominoTiler(rule="cftp", rng=rng, engine=engine)
            runs.append(tiler.cftp(tmax, tmin, 31 + first, first_steps=first, schedule=schedule, max_attempts=30))
            if engine == 0:
                assert _route(rt)["form"] == CLUSTER
        (a, sa), (b, sb) = runs
        assert np.array_equal(a, b)
        for key in ("attempts", "total_steps", "final_steps", "flip_attempts"):
            assert sa[key] == sb[key]
        seen.add((sa["attempts"] - 1) % 4)
    assert len(seen) >= 2


def _run(rt, s, rng, seed, steps):
    if rng == "fast":
        s.run_fast(seed, -steps, steps)
    else:
        s.seed(seed)
        s.run(rt.mt19937_colours(seed, steps))


@pytest.mark.parametrize("chains", [1, 2])
def test_words_per_draw_warp_in_fast_mode(rt, chains):
    seen = set()
    for order in (600, 800, 1024, 1300):
        starts = _start(rt, order)[:chains]
        n = rt.side_of(starts[0])
        out = []
        for launch in ((0, 152, 0), (1, 0, 0)):
            s = rt.DominoSampler(n, chains, rt.DominoTiler(rule="cftp_twoperiodic", rng="fast", a=1.0, b=0.6))
            for c, t in enumerate(starts):
                s.load(c, t)
            s.set_launch(*launch)
            info = s.engine_info()
            if launch[0] == 0 and _route(rt)["form"] == GRID:
                assert _route(rt)["depth"] == 1
                seen.add(info["units_per_thread"])
            for steps, seed in ((33, 3), (2, 4), (1, 5)):
                _run(rt, s, "fast", seed, steps)
            out.append([s.store(c) for c in range(chains)])
            s.close()
        assert all(np.array_equal(a, b) for a, b in zip(*out)), order
    assert {8, 12, 16} <= seen, seen


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("steps", [40, 200])
def test_an_exchange_after_every_run_gives_up(rt, rng, steps):
    tmax, tmin = _start(rt, 600)
    n = rt.side_of(tmax)
    out = []
    for silent in (True, False):
        s = rt.DominoSampler(n, 2, rt.DominoTiler(rule="cftp", rng=rng))
        s.set_launch(0, 152, 0)
        for c, t in enumerate((tmin, tmax)):
            s.load(c, t)
        if silent:
            s.engine_info()
            route = _route(rt)
            assert route["form"] == GRID and route["depth"] == 1 and route["bands"] > 16
            assert rt.lib().rt_dm_sampler_test_silent_band(s.h, 1, 4096) == rt.RT_OK
            with pytest.raises(rt.RTError) as err:
                _run(rt, s, rng, 5, steps)
                s.sync()
            assert err.value.status == rt.RT_ERR_TIMEOUT
            assert rt.lib().rt_dm_sampler_test_silent_band(s.h, -1, 0) == rt.RT_OK
            for c, t in enumerate((tmin, tmax)):
                s.load(c, t)
        _run(rt, s, rng, 5, steps)
        s.sync()
        out.append([s.store(c) for c in (0, 1)])
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("rng,shape", [("tinymt", (4, 4)), ("fast", (4, 4)), ("tinymt", (18, 34))])  # one CTA, bands
def test_bibone_walk_of_two_launches(rt, orc, shape, rng):
    T = rt.TriangleDimerTiler
    steps = (1 << 18) + 77
    got = T.RhombusBrick(*shape)
    want, n = got.copy(), rt.side_of(got)
    if rng == "fast":
        orc.td_walk_fast(want, n, 0, steps, 5, 0)
    else:
        orc.td_walk_tinymt(want, n, steps, 5)
    T(rng=rng).Walk(got, steps, 5)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_recttri_walk_of_two_launches(rt, orc, rng):
    R = rt.RectTriangleTiler
    steps = (1 << 20) + 77
    got = R.minHex(2)
    want, n = got.copy(), rt.side_of(got)
    if rng == "fast":
        orc.rt_walk_fast(want, n, 0, steps, 5, 0)
    else:
        orc.rt_walk_tinymt(want, n, steps, 5)
    R(rng=rng).Walk(got, steps, 5)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("rng,side", [("tinymt", 5), ("fast", 5), ("tinymt", 36)])  # one CTA, a cluster
def test_lozenge_walk_of_two_launches(rt, orc, side, rng):
    L = rt.LozengeTiler
    steps = (1 << 16) + 77
    got = L.MinTiling(L.Hexagon(side))
    want, n = got.copy(), rt.side_of(got)
    if rng == "fast":
        orc.lz_walk_fast(want, n, 0, steps, 5, 0)
    else:
        orc.lz_walk_tinymt(want, n, steps, 5)
    L(rng=rng).Walk(got, steps, 5)
    assert np.array_equal(got, want)
