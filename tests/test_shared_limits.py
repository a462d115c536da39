"""Callers of different sizes share a kernel: the shared memory that one plan needs must not lower what
another's launch may ask for.  Samplers, servers and threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sampler(rt, order, rng, launch):
    D = rt.DominoTiler
    d = D.AztecDiamond(order)
    tmax, tmin = D.MaxTiling(d), D.MinTiling(d)
    engine, bands = launch
    s = rt.DominoSampler(rt.side_of(tmax), 2, D(rule="cftp", rng=rng, engine=engine))
    s.load(0, tmin)
    s.load(1, tmax)
    s.set_launch(0, bands, 0)
    return s


def _run(rt, s, rng, seed):
    if rng == "fast":
        s.run_fast(seed, 0, 30)
    else:
        s.seed(seed)
        s.run(rt.mt19937_colours(seed, 30))


@pytest.mark.parametrize("rng,launch,large,small", [
    ("tinymt", (0, 152), 150, 60), ("tinymt", (0, 152), 500, 430), ("tinymt", (0, 16), 200, 150),
    ("tinymt", (4, 0), 512, 64), ("tinymt", (2, 0), 400, 200), ("tinymt", (3, 0), 300, 100),
    ("fast", (0, 152), 100, 30), ("fast", (0, 16), 200, 150), ("fast", (2, 0), 400, 200)])
def test_samplers_in_turn(rt, rng, launch, large, small):
    """The large one is planned first, the small one then, and the large one runs again."""
    want = _sampler(rt, large, rng, launch)
    a = _sampler(rt, large, rng, launch)
    _run(rt, a, rng, 5)
    b = _sampler(rt, small, rng, launch)
    _run(rt, b, rng, 6)
    _run(rt, a, rng, 7)
    for seed in (5, 7):
        _run(rt, want, rng, seed)
    for c in (0, 1):
        assert np.array_equal(a.store(c), want.store(c))
    for s in (a, b, want):
        s.close()


def test_servers_of_two_sizes(rt):
    D = rt.DominoTiler
    d = D.AztecDiamond(8)
    job = dict(model="domino", tmax=D.MaxTiling(d), tmin=D.MinTiling(d), seed=3, stream=1, rule="cftp",
               a=1.0, b=1.0, first_steps=16, max_attempts=16)
    large = rt.Server(slots=8, max_side=200)
    small = rt.Server(slots=8, max_side=40)
    out = [s.wait(s.submit(job))[0] for s in (large, small)]
    assert np.array_equal(*out)
    large.close()
    small.close()


@pytest.mark.parametrize("model", ["bibone", "recttri", "lozenge", "six"])
def test_walks_from_two_threads(rt, model):
    T, R, L, S = rt.TriangleDimerTiler, rt.RectTriangleTiler, rt.LozengeTiler, rt.SixVertexTiler
    if model == "bibone":
        tiler, starts = T(rng="fast"), [T.RhombusBrick(200, 300), T.RhombusBrick(40, 60)]
    elif model == "recttri":
        tiler, starts = R(rng="fast"), [R.minHex(120), R.minHex(60)]
    elif model == "lozenge":
        tiler, starts = L(rng="fast"), [L.MinTiling(L.Hexagon(k)) for k in (100, 70)]
    else:
        tiler, starts = S(1.0, 1.0, 1.5), [S.MinHeight(600), S.MinHeight(300)]
    want = []
    for t in starts:
        want.append(t.copy())
        tiler.Walk(want[-1], 30, 4)
    errors = []

    def work(k):
        try:
            for _ in range(150):
                t = starts[k].copy()
                tiler.Walk(t, 30, 4)
                if not np.array_equal(t, want[k]):
                    errors.append("differs")
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
