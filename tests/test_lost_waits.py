"""A bounded wait that gave up is reported, whatever becomes of the engine whose launch it was: the
sampler may plan another engine before it reads the launch's error word (another number of swept
chains, tilings loaded, a coupling whose table entry asks for other bands)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(rt, order):
    D = rt.DominoTiler
    d = D.AztecDiamond(order)
    return D.MaxTiling(d), D.MinTiling(d)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("bands,order", [(4, 40), (40, 64)])
@pytest.mark.parametrize("change", ["active", "load"])
def test_the_engine_goes_before_its_error_is_read(rt, rng, bands, order, change):
    tmax, tmin = _start(rt, order)
    s = rt.DominoSampler(rt.side_of(tmax), 2, rt.DominoTiler(rule="cftp", rng=rng))
    s.load(0, tmin)
    s.load(1, tmax)
    s.set_launch(0, bands, 0)
    cols = rt.mt19937_colours(77, 64)

    def go():
        if rng == "fast":
            s.run_fast(5, 0, 64)
        else:
            s.run(cols)

    if rng == "tinymt":
        s.seed(5)
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, 1, 4096) == rt.RT_OK
    go()
    assert rt.lib().rt_dm_sampler_test_silent_band(s.h, -1, 0) == rt.RT_OK
    if change == "active":
        s.set_active(1)
    else:
        s.load(1, tmax)
    with pytest.raises(rt.RTError) as err:
        go()
        s.sync()
    assert err.value.status == rt.RT_ERR_TIMEOUT
    go()  # reported once
    s.sync()
    s.close()


def test_early_epoch_of_a_coupling(rt, tmp_path):
    """The second attempt is two launches: the first one's band 1 publishes nothing.  The table asks for
    other bands than a coupling's first choice, k_deep, does."""
    tmax, tmin = _start(rt, 160)
    table = tmp_path / "tune.txt"
    tiler = rt.DominoTiler(rule="cftp", rng="tinymt")
    args = dict(driver_seed=9, first_steps=30, schedule=0, max_attempts=2)
    for bands in (152, 100):
        table.write_text(f"domino 6 32768 2 tinymt 4 {bands} 0\n")
        rt.tune_load(table)
        try:
            assert rt.lib().rt_test_silent_band(1, 4096, 1, 1) == rt.RT_OK
            with pytest.raises(rt.RTError) as err:
                tiler.cftp(tmax, tmin, **args)
            assert err.value.status == rt.RT_ERR_TIMEOUT
            assert rt.lib().rt_test_silent_band(-1, 0, 0, 0) == rt.RT_OK
            with pytest.raises(rt.RTError) as err:
                tiler.cftp(tmax, tmin, **args)
            assert err.value.status == rt.RT_ERR_NOT_COALESCED
        finally:
            rt.lib().rt_test_silent_band(-1, 0, 0, 0)
            rt.tune_clear()
