"""Walks convert their tilings on the device only where it has room for the words; without it they do so on
the host, with the same results and the same refusals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(rt):
    yield lambda n: rt.lib().rt_test_alloc_limit(n)
    rt.lib().rt_test_alloc_limit(0)


@pytest.mark.parametrize("n", [200, 512])
def test_six_vertex(rt, limit, n):
    S = rt.SixVertexTiler
    start = S.MinHeight(n)
    want = start.copy()
    S(1.0, 1.0, 1.5).Walk(want, 20, 4)
    assert limit(2 * (n + 1) ** 2) == rt.RT_OK  # half of the heights
    got = start.copy()
    S(1.0, 1.0, 1.5).Walk(got, 20, 4)
    assert np.array_equal(got, want)
    bad = start.copy()
    bad[5] += 2
    with pytest.raises(rt.RTError) as err:
        S(1.0, 1.0, 1.5).Walk(bad, 20, 4)
    assert err.value.status == rt.RT_ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_bibone(rt, limit, rng):
    T = rt.TriangleDimerTiler
    start = T.RhombusBrick(200, 200)
    n = rt.side_of(start)
    want = start.copy()
    stats = T(rng=rng).Walk(want, 30, 4)
    assert limit(2 * n * n) == rt.RT_OK
    got = start.copy()
    again = T(rng=rng).Walk(got, 30, 4)
    assert np.array_equal(got, want)
    assert again["flip_attempts"] == stats["flip_attempts"]
    bad = start.copy()
    bad[n + 1] ^= 4
    with pytest.raises(rt.RTError) as err:
        T(rng=rng).Walk(bad, 30, 4)
    assert err.value.status == rt.RT_ERR_INVALID_ARGUMENT


def test_too_little_for_the_state_itself(rt, limit):
    S = rt.SixVertexTiler
    assert limit(1000) == rt.RT_OK
    h = S.MinHeight(512)
    with pytest.raises(rt.RTError) as err:
        S(1.0, 1.0, 1.5).Walk(h, 20, 4)
    assert err.value.status == rt.RT_ERR_OUT_OF_MEMORY
    assert np.array_equal(h, S.MinHeight(512))
