"""Walks of a few steps on small inputs keep to the kernels that need little set-up; longer walks and larger
inputs go to the resident ones.  The two sides of each line, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("side", [2, 20, 21, 42, 44, 45])
@pytest.mark.parametrize("steps", [0, 1, 3, 4, 7, 8])
def test_recttri(rt, orc, side, steps, mode):
    start = rt.RectTriangleTiler.slopeHex(side)
    n = rt.side_of(start)
    tiler = rt.RectTriangleTiler(rng="fast" if mode == "fast" else "tinymt", fast_stream=7)
    got, want = start.copy(), start.copy()
    if mode == "fast":
        orc.rt_walk_fast(want, n, 0, steps, 11, 7, None)
    elif mode == "table":
        params = np.random.RandomState(n).randint(0, 2**32, size=(n * n // 3 - 5, 3), dtype=np.uint32)
        tiler.LoadTinyMT(params)
        orc.rt_walk_tinymt(want, n, steps, 11, None, params=params)
    else:
        orc.rt_walk_tinymt(want, n, steps, 11, None)
    tiler.Walk(got, steps, 11)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("side", [1, 2, 9, 30, 60])
@pytest.mark.parametrize("steps", [0, 1, 2, 9])
def test_lozenge(rt, orc, side, steps, mode):
    L = rt.LozengeTiler
    start = L.MinTiling(L.Hexagon(side))
    got, want = start.copy(), start.copy()
    if mode == "fast":
        orc.lz_walk_fast(want, rt.side_of(start), 0, steps, 11, 7)
    else:
        orc.lz_walk_tinymt(want, rt.side_of(start), steps, 11)
    L(rng=mode, fast_stream=7).Walk(got, steps, 11)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("mode", ["tinymt", "fast"])
@pytest.mark.parametrize("rows,cols", [(4, 4), (20, 12), (41, 40), (42, 42), (43, 40), (44, 44)])
@pytest.mark.parametrize("steps", [0, 1, 12])
def test_bibone(rt, orc, rows, cols, steps, mode):
    T = rt.TriangleDimerTiler
    start = T.RhombusBrick(rows, cols)
    n = rt.side_of(start)
    got, want = start.copy(), start.copy()
    if mode == "fast":
        orc.td_walk_fast(want, n, 0, steps, 11, 7)
    else:
        orc.td_walk_tinymt(want, n, steps, 11)
    stats = T(rng=mode, fast_stream=7).Walk(got, steps, 11)
    assert np.array_equal(got, want)
    assert stats["total_steps"] == steps
    bad = start.copy()
    bad[n + 1] ^= 4  # no dimer configuration
    with pytest.raises(rt.RTError) as err:
        T(rng=mode).Walk(bad, steps, 11)
    assert err.value.status == rt.RT_ERR_INVALID_ARGUMENT
