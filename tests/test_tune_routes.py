"""What the autotuner measures is what its table entry then runs: each candidate shape that a sampler takes is
written as an entry, and a sampler that follows the table plans the same kernel with as many bands."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _route(rt):
    out = (C.c_int32 * 4)()
    assert rt.lib().rt_test_route(out) == rt.RT_OK
    return tuple(out)


@pytest.mark.parametrize("rng", ["tinymt", "fast"])
@pytest.mark.parametrize("order", [24, 130, 420])
def test_entries_run_what_was_measured(rt, tmp_path, order, rng):
    from randomtilingspublic_gb300 import autotune

    rt.tune_clear()
    D = rt.DominoTiler
    d = D.AztecDiamond(order)
    tmax, tmin = D.MaxTiling(d), D.MinTiling(d)
    n = rt.side_of(tmax)
    path, taken = tmp_path / "tune.txt", 0
    for shape in autotune.candidates(autotune._sm_count()):
        if shape[0] == 2 and shape[2] not in (512, 1024):
            continue
        got = autotune.measure(rt, n, 2, rng, tmax, tmin, shape, half_sweeps=8, reps=1)
        if got is None:
            continue
        measured, used = _route(rt), got[1]
        entry = dict(n_lo=6, n_hi=32768, chains=2, rng=rng, engine=used[0], bands=used[1], threads=used[2], us=1.0,
                     order=order, N=n)
        autotune.write_table([entry], path)
        rt.tune_load(path)
        try:
            s = autotune._sampler(rt, n, 2, rng, tmax, tmin)
            info = s.engine_info()
            s.close()
            assert info["tuned"] and info["engine"] == used[0]
            assert _route(rt) == measured, (shape, used)
        finally:
            rt.tune_clear()
        taken += 1
    assert taken >= 4
