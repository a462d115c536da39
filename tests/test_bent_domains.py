"""Long bent domains: few words a row, but a bounding box that no cluster's windows hold.  The automatic
choice declines the cluster kernel there and takes another, with the same chains."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bent(rt, side, wide):
    m = side + 1 - side % 2
    d = np.zeros((m, m), np.int32)
    d[2:side - 3, 2:2 + wide] = 1
    d[side - 3 - wide:side - 3, 2:side - 3 - (side - 5) % 2] = 1
    d = d.ravel()
    return rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("side,wide,chains", [(3000, 40, 1), (2000, 40, 2), (1200, 40, 2), (700, 24, 1)])
def test_automatic_choice_equals_the_per_half_sweep_kernels(rt, rng, side, wide, chains):
    starts = _bent(rt, side, wide)[:chains]
    n = rt.side_of(starts[0])
    got = []
    for engine in (0, 1):
        s = rt.DominoSampler(n, chains, rt.DominoTiler(rule="cftp", rng=rng, engine=engine))
        for c, t in enumerate(starts):
            s.load(c, t)
        if rng == "fast":
            s.run_fast(5, 0, 40)
        else:
            s.seed(5)
            s.run(rt.mt19937_colours(5, 40))
        got.append([s.store(c) for c in range(chains)])
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_coupling(rt, rng):
    tmax, tmin = _bent(rt, 2000, 40)
    got = []
    for engine in (0, 1):
        with pytest.raises(rt.RTError) as err:
            rt.DominoTiler(rule="cftp", rng=rng, engine=engine).cftp(tmax, tmin, 3, first_steps=10, max_attempts=2)
        got.append(err.value.status)
    assert got == [rt.RT_ERR_NOT_COALESCED] * 2
