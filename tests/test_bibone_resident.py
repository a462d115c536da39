"""Bibone walks on the resident kernel (dimers as bit planes): identical (whole numbers) to the oracle on regions
from one word to many, with edges at a word's edge, in one CTA and in bands that exchange rows every few steps
(steps not a multiple of the depth), in every random mode; the statistics; and input that is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walk(rt, orc, start, steps, seed, mode):
    n = int(np.sqrt(start.size))
    tiler = rt.TriangleDimerTiler(rng="fast" if mode == "fast" else "tinymt", fast_stream=11)
    a, b = start.copy(), start.copy()
    if mode == "fast":
        orc.td_walk_fast(b, n, 0, steps, seed, 11)
    elif mode == "table":
        params = np.random.RandomState(n).randint(0, 2**32, size=((n // 2) ** 2 - 3, 3), dtype=np.uint32)
        tiler.LoadTinyMT(params)
        orc.td_walk_tinymt(b, n, steps, seed, params=params)
    else:
        orc.td_walk_tinymt(b, n, steps, seed)
    stats = tiler.Walk(a, steps, seed)
    return a, b, stats


@pytest.mark.parametrize("mode", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("rows,cols", [(1, 2), (2, 2), (5, 6), (3, 58), (60, 4), (26, 26), (29, 30), (61, 90), (126, 34),
                                       (30, 122), (170, 168)])
def test_rhombus_walks_equal_the_oracle(rt, orc, rows, cols, mode):
    a, b, _ = _walk(rt, orc, rt.TriangleDimerTiler.RhombusBrick(rows, cols), 700, 5 + rows, mode)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("n,m", [(6, 0), (18, 5), (47, 0), (90, 21), (200, 40)])
def test_cone_walks_equal_the_oracle(rt, orc, n, m, mode):
    a, b, _ = _walk(rt, orc, rt.TriangleDimerTiler.IceCreamCone(n, m), 500, 17 + n, mode)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
def test_largest_sizes_equal_the_oracle(rt, orc, mode):
    # TinyMT: an exchange every step; fast mode: many words a row
    a, b, _ = _walk(rt, orc, rt.TriangleDimerTiler.RhombusBrick(420, 700), 60, 3, mode)
    assert np.array_equal(a, b)


def test_flip_attempts_count_the_covered_sites_of_each_class(rt):
    T = rt.TriangleDimerTiler
    t = T.RhombusBrick(12, 18)  # every class's share of 216 sites: 1/2, 1/3 and 1/6
    st = T(rng="fast").Walk(t.copy(), 900, 4)
    assert 216 // 6 * 900 < st["flip_attempts"] < 216 // 2 * 900 and st["total_steps"] == 900
    one = [T(rng="fast", fast_stream=k).Walk(t.copy(), 1, 4)["flip_attempts"] for k in range(60)]
    assert set(one) == {108, 72, 36}


def test_refused_input_is_left_as_it_was(rt):
    T = rt.TriangleDimerTiler
    t = T.RhombusBrick(8, 8)
    bad = t.copy()
    bad[np.nonzero(bad)[0][3]] ^= 4
    keep = bad.copy()
    with pytest.raises(rt.RTError) as e:
        T(rng="fast").Walk(bad, 5, 1)
    assert e.value.status == rt.RT_ERR_INVALID_ARGUMENT and np.array_equal(bad, keep)
    n = int(np.sqrt(t.size))
    d = T.Dimers(t)
    d[(n // 2) * 5 + 4] |= 2  # a second dimer at a vertex
    twice = T.FromDimers(d, n)
    with pytest.raises(rt.RTError, match="share a vertex"):
        T().Walk(twice, 5, 1)
