"""The lozenge bit-plane engine (engine 0): identical (whole numbers) to the per-step kernels in each of
its three forms - one CTA, one cluster, one band per SM - at the sizes where the form changes, on
regions with a corner removed, for both rules, every random mode, one and two chains; and inputs
that it leaves to the byte kernels."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walk(rt, start, steps, seed, mode, engine, q=None):
    n = int(np.sqrt(start.size))
    tiler = rt.LozengeTiler(rng="fast" if mode == "fast" else "tinymt", fast_stream=9, q=q, engine=engine)
    if mode == "table":
        tiler.LoadTinyMT(np.random.RandomState(n).randint(0, 2**32, size=(n * n // 3 - 7, 3), dtype=np.uint32))
    t = start.copy()
    tiler.Walk(t, steps, seed)
    return t


@pytest.mark.parametrize("mode", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("side", [1, 2, 3, 14, 15, 16, 31, 32, 33, 39, 41, 47, 125, 127, 203, 206])
def test_hexagon_walks_equal_the_per_step_kernels(rt, mode, side):
    L = rt.LozengeTiler
    d = L.Hexagon(side)
    q = 0.97 if side % 2 else None
    for start in (L.MinTiling(d), L.MaxTiling(d)):
        steps = 900 if side < 50 else 200
        assert np.array_equal(_walk(rt, start, steps, 40 + side, mode, 0, q), _walk(rt, start, steps, 40 + side, mode, 1, q))


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("n,m", [(9, 4), (24, 10), (60, 30), (140, 35)])
def test_hexagon_without_a_corner(rt, mode, n, m):
    L = rt.LozengeTiler
    start = L.MinTiling(L.AlmostHexDomain(n, m))
    a = _walk(rt, start, 400, 8, mode, 0)
    assert np.array_equal(a, _walk(rt, start, 400, 8, mode, 1)) and not np.array_equal(a, start)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("side", [4, 13, 18])
def test_cftp_equals_the_per_step_kernels(rt, mode, side):
    L = rt.LozengeTiler
    d = L.Hexagon(side)
    tmax, tmin = L.MaxTiling(d), L.MinTiling(d)
    (a, sa), (b, sb) = (L(rng=mode, engine=e).cftp(tmax, tmin, 70 + side, first_steps=64, schedule=1, max_attempts=20)
                        for e in (0, 1))
    assert np.array_equal(a, b)
    for key in ("attempts", "total_steps", "final_steps", "flip_attempts"):
        assert sa[key] == sb[key]


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("side", [150, 260])
def test_two_chains_on_many_bands(rt, mode, side):
    L = rt.LozengeTiler
    d = L.Hexagon(side)
    tmax, tmin = L.MaxTiling(d), L.MinTiling(d)
    outs = []
    for engine in (0, 1):
        with pytest.raises(rt.RTError) as e:  # one short attempt: the top chain comes back uncoalesced
            L(rng=mode, engine=engine).cftp(tmax, tmin, 5, first_steps=60, max_attempts=1)
        assert e.value.status == rt.RT_ERR_NOT_COALESCED
        o = L(rng=mode, engine=engine).opts()
        out, st = np.zeros_like(tmax), rt.CftpStats()
        rt.lib().rt_lozenge_cftp(tmax.ctypes.data, tmin.ctypes.data, int(np.sqrt(tmax.size)), 5, 60, 0, 1, C.byref(o),
                                 out.ctypes.data, C.byref(st))
        outs.append((out, st.flip_attempts))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
def test_states_that_are_no_tilings(rt, mode):
    rng = np.random.default_rng(4)
    start = rng.choice(np.array([0, 25, 38, 63, 7], np.int32), size=30 * 30).astype(np.int32)
    assert np.array_equal(_walk(rt, start, 40, 3, mode, 0), _walk(rt, start, 40, 3, mode, 1))
    # a tiling that reaches the vertices which are never rebuilt: row 1
    L = rt.LozengeTiler
    t = L.MinTiling(L.Hexagon(6))
    n = int(np.sqrt(t.size))
    first = int(np.nonzero(t.reshape(n, n).any(1))[0][0])
    up = np.roll(t.reshape(n, n), -(first - 1), axis=0).ravel().copy()
    assert np.array_equal(_walk(rt, up, 200, 3, mode, 0), _walk(rt, up, 200, 3, mode, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("rng,schedule", [("fast", 1), ("tinymt", 0), ("tinymt", 1)])
def test_attempts_side_by_side_return_the_smallest(rt, rng, schedule):
    # The first look-back decides which of the four CTAs runs the attempt that coalesces; several coalesce at once
    # where the first is already long enough, and the chain must then be the first one's.
    L = rt.LozengeTiler
    sizes = ((2, (1, 4, 16, 512)), (9, (8, 32, 128, 8192)))
    if schedule == 0:  # look-backs grow by 2 first only
        sizes = ((2, (4, 16, 512)), (9, (512, 1024, 8192)))
    for side, firsts in sizes:
        d = L.Hexagon(side)
        tmax, tmin = L.MaxTiling(d), L.MinTiling(d)
        seen = set()
        for first in firsts:
            runs = [L(rng=rng, engine=engine).cftp(tmax, tmin, 77 + first, first_steps=first, schedule=schedule,
                                                   max_attempts=36) for engine in (0, 1)]
            (a, sa), (b, sb) = runs
            assert np.array_equal(a, b)
            keys = ("attempts", "total_steps", "final_steps", "flip_attempts")
            assert [sa[k] for k in keys] == [sb[k] for k in keys]
            seen.add(sa["attempts"])
        assert len(seen) >= 2
