"""A server's CTAs hold every admissible side as bit planes, also those that would take more shared memory
than the largest (their draws then run fewer steps ahead)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_side", [40, 130, 140, 200, 288])
def test_every_side_runs_as_planes(rt, max_side):
    s = rt.Server(slots=4, max_side=max_side)
    for model, step in ((0, 2), (1, 3)):
        periods = {n: rt.lib().rt_server_test_period(s.h, model, n) for n in range(12, max_side + 1, step)}
        assert min(periods.values()) >= 2, periods
    s.close()


@pytest.mark.parametrize("side", [47, 50, 57])
def test_samples_of_such_sides(rt, side):
    L = rt.LozengeTiler
    d = L.Hexagon(side)
    tmax, tmin = L.MaxTiling(d), L.MinTiling(d)
    assert 102 <= rt.side_of(tmax) <= 130
    job = dict(model="lozenge", tmax=tmax, tmin=tmin, seed=5, stream=2, rule="cftp", first_steps=100, max_attempts=2)
    server = rt.Server(slots=4, max_side=130)
    out, attempts, look_back = server.wait(server.submit(job))
    server.close()
    samples, want, _ = rt.cftp_batch([job])
    assert np.array_equal(out, samples[0])
    assert attempts == want[0] and look_back == 600
