"""The batch kernel's bit planes: sizes on both sides of a 32-cell word, and instances that the planes cannot hold
(a stray edge, flip candidates at cells that are never rebuilt), against the single-instance fast mode."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(rt, model, size):
    T = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    d = T.AztecDiamond(size) if model == "domino" else T.Hexagon(size)
    return T.MaxTiling(d), T.MinTiling(d)


def _same(rt, jobs):
    outs, attempts, _ = rt.cftp_batch(jobs)
    for job, out, att in zip(jobs, outs, attempts):
        if job["model"] == "domino":
            tiler = rt.DominoTiler(rule=job["rule"], rng="fast", a=job["a"], b=job["b"], fast_stream=job["stream"])
        else:
            tiler = rt.LozengeTiler(rng="fast", fast_stream=job["stream"])
        ref, st = tiler.cftp(job["tmax"], job["tmin"], job["seed"], first_steps=job["first_steps"], schedule=1,
                             max_attempts=20)
        assert att == st["attempts"] and np.array_equal(out, ref), (job["model"], len(out))


def _job(model, pair, k, rule="cftp", b=1.0):
    return {"model": model, "tmax": pair[0], "tmin": pair[1], "seed": 900 + k, "stream": k, "rule": rule, "a": 1.0, "b": b,
            "first_steps": 16, "max_attempts": 20}


# colour-array rows of order + 3 cells (dominoes) and of about side + 1 cells (lozenges)
@pytest.mark.parametrize("model,sizes", [("domino", (1, 2, 13, 28, 29, 30)), ("lozenge", (2, 3, 29, 30, 31, 32))])
def test_sizes_around_a_word(rt, model, sizes):
    jobs = [_job(model, _pair(rt, model, s), k) for k, s in enumerate(sizes)]
    if model == "domino":
        jobs += [_job(model, _pair(rt, model, s), 50 + s, "cftp_twoperiodic", 0.9) for s in (2, 13, 28)]
    _same(rt, jobs)
    _same(rt, jobs[:1])  # alone: CTAs without an instance of their own run its later attempts


@pytest.mark.parametrize("model,size", [("domino", 6), ("domino", 11), ("lozenge", 4), ("lozenge", 7)])
def test_stray_edge(rt, model, size):
    pair = [t.copy() for t in _pair(rt, model, size)]
    for t in pair:
        t[0] = 8  # an edge to the right that its other end does not have
    _same(rt, [_job(model, pair, 1), _job(model, _pair(rt, model, size), 2)])


# A domain of which a corner lies in the first row or column, which is never rebuilt: the chains need not meet, and
# the result is the top chain of the one attempt.
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("model,size", [("domino", 6), ("lozenge", 5)])
def test_candidates_at_the_border(rt, orc, model, size, axis):
    pair = []
    for t in _pair(rt, model, size):
        n = int(round(len(t) ** 0.5))
        g = t.reshape(n, n)
        s = min(int(np.nonzero(x.reshape(n, n))[axis].min()) for x in _pair(rt, model, size))
        s -= s % (2 if model == "domino" else 3)
        pair.append(np.roll(g, -s, axis).ravel().copy())
    job = dict(_job(model, pair, 3), max_attempts=1)
    outs, attempts, _ = rt.cftp_batch([job])
    ref = pair[0].copy()
    if model == "domino":
        orc.walk_fast(ref, n, -32, 32, job["seed"], job["stream"], rule=1)
    else:
        orc.lz_walk_fast(ref, n, -48, 48, job["seed"], job["stream"])
    assert np.array_equal(outs[0], ref)
