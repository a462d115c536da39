"""Rectangle-triangle walks on the cluster kernel: identical (whole numbers) to the oracle from one
CTA to sixteen, on sizes around its plan's edges, in every random mode, with moves across the
seams between CTAs; and states that are not tilings, which keep to the per-step kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walk(rt, orc, start, steps, seed, mode, weights=None):
    n = int(np.sqrt(start.size))
    tiler = rt.RectTriangleTiler(rng="fast" if mode == "fast" else "tinymt", fast_stream=7, weights=weights)
    a, b = start.copy(), start.copy()
    if mode == "fast":
        orc.rt_walk_fast(b, n, 0, steps, seed, 7, weights)
    elif mode == "table":
        params = np.random.RandomState(n).randint(0, 2**32, size=(n * n // 3 - 5, 3), dtype=np.uint32)
        tiler.LoadTinyMT(params)
        orc.rt_walk_tinymt(b, n, steps, seed, weights, params=params)
    else:
        orc.rt_walk_tinymt(b, n, steps, seed, weights)
    tiler.Walk(a, steps, seed)
    return a, b


@pytest.mark.parametrize("mode", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("side,steps", [(2, 300), (3, 301), (8, 900), (21, 700), (22, 700), (40, 500), (75, 300), (120, 120)])
def test_cluster_walk_equals_the_oracle(rt, orc, side, steps, mode):
    w = np.random.default_rng(side).uniform(0.6, 1.6, size=9) if side % 2 else None
    for start in (orc.rt_hex(side, False), orc.rt_hex(side, True)):
        a, b = _walk(rt, orc, start, steps, 1000 + side, mode, w)
        assert np.array_equal(a, b)
        assert not np.array_equal(a, start)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
def test_moves_everywhere_cross_the_seams(rt, orc, mode):
    # the sloped start moves all over the hexagon at once
    start = rt.RectTriangleTiler.slopeHex(60)
    a, b = _walk(rt, orc, start, 400, 5, mode)
    assert np.array_equal(a, b)
    assert int((a != start).sum()) > 3000


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
def test_states_that_are_no_tilings(rt, orc, mode):
    rng = np.random.default_rng(3)
    states = np.array([0, 0x122133, 0x331221, 0x8ebbe8, 0x47d47a, 0x6699cf, 0x123456], np.int32)
    start = rng.choice(states, size=21 * 21).astype(np.int32)  # digits differ between vertices
    a, b = _walk(rt, orc, start, 60, 9, mode)
    assert np.array_equal(a, b)
    rim = orc.rt_hex(5, False).reshape(18, 18)
    rim[0, 4] = 0x331221  # a vertex that is never rebuilt
    a, b = _walk(rt, orc, rim.ravel(), 60, 9, mode)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("side", [255, 330])
def test_largest_sizes_match_the_oracle(rt, orc, side):
    # TinyMT: 255 is near the largest the registers hold, 330 beyond it
    start = orc.rt_hex(side, False)
    for mode in ("tinymt", "fast"):
        a, b = _walk(rt, orc, start, 40, 3, mode)
        assert np.array_equal(a, b)
