"""The bit-plane kernel in one thread-block cluster: identical (whole numbers) to the oracle and
to the per-half-sweep kernels at the edges of its plan - one word, rows that start or end at a
word's edge, one row per CTA, more CTAs than rows, the largest domain it holds and the first it
does not - for every random mode, one and two chains, epochs, and coupling from the past."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(rt, shape):
    D = rt.DominoTiler
    d = D.AztecDiamond(shape) if isinstance(shape, int) else D.Rectangle(*shape)
    return D.MaxTiling(d), D.MinTiling(d)


def _chains(rt, tiler, starts, launch, steps):
    n = rt.side_of(starts[0])
    s = rt.DominoSampler(n, len(starts), tiler)
    for c, t in enumerate(starts):
        s.load(c, t)
    s.set_launch(*launch)
    info = s.engine_info()
    for part, seed in steps:
        if tiler.rng == "fast":
            s.run_fast(seed, -part, part)
        else:
            s.seed(seed)
            s.run(rt.mt19937_colours(seed, part))
    out = [s.store(c) for c in range(len(starts))]
    s.close()
    return out, info


@pytest.mark.parametrize("rng", ["tinymt", "table", "fast"])
@pytest.mark.parametrize("shape", [1, 2, 7, 16, 31, (2, 130), (130, 2), (3, 64), (62, 61), (126, 130), 100])
def test_cluster_equals_per_half_sweep_kernels(rt, rng, shape):
    tmax, tmin = _start(rt, shape)
    n = rt.side_of(tmax)
    tiler = rt.DominoTiler(rule="cftp_twoperiodic", rng="fast" if rng == "fast" else "tinymt", a=1.0, b=0.7,
                           fast_stream=5)
    if rng == "table":
        tiler.LoadTinyMT(np.random.RandomState(n).randint(0, 2**32, size=((n - 2) * (n // 2 - 2), 3), dtype=np.uint32))
    steps = [(90, 11), (41, 12)]
    for starts in ([tmin], [tmin, tmax]):
        want, _ = _chains(rt, tiler, starts, (1, 0, 0), steps)
        for ctas in (1, 3, 16):
            got, info = _chains(rt, tiler, starts, (0, ctas, 0), steps)
            if info["engine"] != 4 or info["bands"] > ctas:
                assert ctas < 16  # more words than so few CTAs hold
                continue
            for g, w in zip(got, want):
                assert np.array_equal(g, w), (shape, rng, ctas)


@pytest.mark.parametrize("shape", [4, 9, 40, (30, 97)])
def test_cluster_walks_and_epochs_equal_the_oracle(rt, orc, shape):
    tmax, _ = _start(rt, shape)
    n = rt.side_of(tmax)
    g, o = tmax.copy(), tmax.copy()
    rt.DominoTiler(rule="plain").Walk(g, [120, 33], [5, 77])  # the automatic choice
    orc.walk_epochs_tinymt(o, n, [120, 33], [5, 77], rule=0, a=0.7, b=1.0)
    assert np.array_equal(g, o)


@pytest.mark.parametrize("order", [3, 8, 12, 20])
@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_cluster_cftp_equals_the_per_half_sweep_kernels(rt, order, rng):
    tmax, tmin = _start(rt, order)
    runs = []
    for engine in (0, 1):
        tiler = rt.DominoTiler(rule="cftp", rng=rng, engine=engine)
        runs.append(tiler.cftp(tmax, tmin, driver_seed=31 + order, first_steps=16, schedule=1, max_attempts=20))
    (a, sa), (b, sb) = runs
    assert np.array_equal(a, b)
    for key in ("attempts", "total_steps", "final_steps", "flip_attempts"):
        assert sa[key] == sb[key]


@pytest.mark.parametrize("order,rng", [(215, "tinymt"), (240, "tinymt"), (230, "fast")])
def test_largest_domains(rt, order, rng):
    # 240 in TinyMT mode: more words than the cluster's registers hold, so another kernel's 16 bands
    tmax, tmin = _start(rt, order)
    tiler = rt.DominoTiler(rule="cftp", rng=rng)
    want, _ = _chains(rt, tiler, [tmax, tmin], (1, 0, 0), [(30, 3)])
    got, info = _chains(rt, tiler, [tmax, tmin], (0, 16, 0), [(30, 3)])
    assert info["engine"] == 4 and info["bands"] == 16
    assert all(np.array_equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
def test_cluster_wait_gives_up_and_the_sampler_stays_usable(rt, rng):
    """CTA 1 sends none of its boundary words and a wait gives up after 4096 polls: every CTA
    leaves, the host reads RT_ERR_TIMEOUT, and the sampler then repeats a fresh sampler's walk."""
    tmax, tmin = _start(rt, 40)
    n = rt.side_of(tmax)
    tiler = rt.DominoTiler(rule="cftp", rng=rng)
    cols = rt.mt19937_colours(77, 64)

    def fresh():
        s = rt.DominoSampler(n, 2, tiler)
        s.load(0, tmin)
        s.load(1, tmax)
        s.set_launch(0, 4, 0)
        return s

    def go(s):
        if rng == "fast":
            s.run_fast(5, 0, 64)
        else:
            s.seed(5)
            s.run(cols)
        s.sync()

    s = fresh()
    assert s.engine_info()["bands"] == 4
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, 1, 4096) == rt.RT_OK
    with pytest.raises(rt.RTError) as err:
        go(s)
    assert err.value.status == rt.RT_ERR_TIMEOUT
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, -1, 0) == rt.RT_OK
    s.load(0, tmin)
    s.load(1, tmax)
    go(s)
    got = [s.store(0), s.store(1)]
    s.close()
    ref = fresh()
    go(ref)
    want = [ref.store(0), ref.store(1)]
    ref.close()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("rng,schedule", [("fast", 1), ("tinymt", 0), ("tinymt", 1)])
def test_attempts_side_by_side_return_the_smallest(rt, rng, schedule):
    # The first look-back decides which of the four clusters runs the attempt that coalesces; several coalesce at once
    # where the first is already long enough, and the chain must then be the first one's.
    D = rt.DominoTiler
    sizes = ((3, (1, 2, 4, 8, 256)), (12, (4, 16, 64, 256, 4096)))
    if schedule == 0:  # look-backs grow by 2 first only
        sizes = ((3, (2, 4, 8, 256)), (12, (128, 256, 512, 4096)))
    for order, firsts in sizes:
        d = D.AztecDiamond(order)
        tmax, tmin = D.MaxTiling(d), D.MinTiling(d)
        seen = set()
        for first in firsts:
            runs = [D(rule="cftp", rng=rng, engine=engine).cftp(tmax, tmin, 77 + first, first_steps=first,
                                                                schedule=schedule, max_attempts=36)
                    for engine in (0, 1)]
            (a, sa), (b, sb) = runs
            assert np.array_equal(a, b)
            assert {k: sa[k] for k in ("attempts", "total_steps", "final_steps", "flip_attempts")} == {
                k: sb[k] for k in ("attempts", "total_steps", "final_steps", "flip_attempts")}
            seen.add(sa["attempts"])
        assert len(seen) >= 3
