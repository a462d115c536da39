"""Failure detection of the resident kernels whose calls make their own state: band 1 publishes nothing and
every wait gives up after a few thousand polls.  The call returns RT_ERR_TIMEOUT, leaves the caller's state as
it was, and the next call is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _silent(rt, call, state):
    before = state.copy()
    assert rt.lib().rt_test_silent_band(1, 4096, 0, 1 << 20) == rt.RT_OK
    try:
        with pytest.raises(rt.RTError) as err:
            call()
        assert err.value.status == rt.RT_ERR_TIMEOUT
    finally:
        assert rt.lib().rt_test_silent_band(-1, 0, 0, 0) == rt.RT_OK
    assert np.array_equal(state, before)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("side", [56, 200])  # one cluster, one band per SM
@pytest.mark.parametrize("steps", [40, 200])
def test_lozenge(rt, orc, side, steps, rng):
    L = rt.LozengeTiler
    t = L.MinTiling(L.Hexagon(side))
    want = t.copy()
    if rng == "fast":
        orc.lz_walk_fast(want, rt.side_of(t), 0, steps, 5, 0)
    else:
        orc.lz_walk_tinymt(want, rt.side_of(t), steps, 5)
    tiler = L(rng=rng)
    _silent(rt, lambda: tiler.Walk(t, steps, 5), t)
    tiler.Walk(t, steps, 5)
    assert np.array_equal(t, want)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("rows,cols", [(70, 64), (200, 200)])
def test_bibone(rt, orc, rows, cols, rng):
    T = rt.TriangleDimerTiler
    t = T.RhombusBrick(rows, cols)
    want = t.copy()
    if rng == "fast":
        orc.td_walk_fast(want, rt.side_of(t), 0, 40, 5, 0)
    else:
        orc.td_walk_tinymt(want, rt.side_of(t), 40, 5)
    tiler = T(rng=rng)
    _silent(rt, lambda: tiler.Walk(t, 40, 5), t)
    tiler.Walk(t, 40, 5)
    assert np.array_equal(t, want)


@pytest.mark.parametrize("n", [40, 100, 190, 512, 700])  # depths 4, 4, 3, 2 and 1
def test_six_vertex_walk(rt, orc, n):
    S = rt.SixVertexTiler
    h = S.MinHeight(n)
    want = h.copy()
    orc.sv_walk(want, n, 0, 4 * 20, 5, 0, 1.0, 1.0, 1.5)
    tiler = S(1.0, 1.0, 1.5)
    _silent(rt, lambda: tiler.Walk(h, 20, 5), h)
    tiler.Walk(h, 20, 5)
    assert np.array_equal(h, want)


def test_six_vertex_coupling(rt, orc):
    S = rt.SixVertexTiler
    tiler = S(1.0, 1.0, 1.5)
    top, bottom = S.MaxHeight(48), S.MinHeight(48)
    _silent(rt, lambda: tiler.cftp(top, bottom, 5, first_sweeps=64, max_attempts=8), top)
    got, stats = tiler.cftp(top, bottom, 5, first_sweeps=64, max_attempts=8)
    want = orc.sv_cftp(top, bottom, 48, 5, 0, 64, 8, 1.0, 1.0, 1.5)
    assert np.array_equal(got, want[0])
