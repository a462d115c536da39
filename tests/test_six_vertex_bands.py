"""The resident six-vertex engine against the oracle: one band and many, exchanges every 4, 3, 2 and 1 sweeps,
five distinct thresholds (a = b) and nine, sizes on both sides of each rule of its launch shape."""
import numpy as np
import pytest

ABC = [(1.0, 1.0, 1.5), (0.8, 1.2, 1.5)]


# n: rows that move and words a row set the form: 16 rows of one word (n = 32) is the last single band, 128 / 129
# the first rows of three words, 192 / 193 of four; 608 / 609 bands of two rows and of more.
@pytest.mark.gpu
@pytest.mark.parametrize("abc", ABC)
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 34, 64, 65, 66, 127, 128, 129, 130, 192, 193, 194, 257])
def test_walk_matches_oracle(rt, orc, n, abc):
    S = rt.SixVertexTiler
    for sweeps, top in ((1, True), (6, False), (13, True)):
        a = S.MaxHeight(n) if top else S.MinHeight(n)
        b = a.copy()
        S(*abc, fast_stream=3).Walk(a, sweeps, 77 + sweeps)
        orc.sv_walk(b, n, 0, 4 * sweeps, 77 + sweeps, 3, *abc)
        assert np.array_equal(a, b), (n, sweeps, top)


@pytest.mark.gpu
@pytest.mark.parametrize("abc", ABC)
@pytest.mark.parametrize("n,sweeps", [(512, 101), (608, 33), (610, 33), (1024, 17), (2049, 9), (2600, 5)])
def test_walk_matches_sub_sweep_kernels(rt, n, sweeps, abc):
    S = rt.SixVertexTiler
    a, b = S.MinHeight(n), S.MinHeight(n)
    S(*abc, engine=2).Walk(a, sweeps, 9)
    S(*abc, engine=1).Walk(b, sweeps, 9)
    assert np.array_equal(a, b)


@pytest.mark.gpu
def test_walk_in_several_launches(rt):
    # 2^14 sweeps a launch: the states change buffers between launches
    S = rt.SixVertexTiler
    for n in (9, 40):
        a, b = S.MinHeight(n), S.MinHeight(n)
        S(1.0, 1.0, 1.2).Walk(a, 2 * (1 << 14) + 3, 4)
        S(1.0, 1.0, 1.2, engine=1).Walk(b, 2 * (1 << 14) + 3, 4)
        assert np.array_equal(a, b)


# Attempts run side by side in groups: the first look-back decides which of a group coalesces first.
@pytest.mark.gpu
@pytest.mark.parametrize("abc", [(1.0, 1.0, 1.5), (0.9, 0.7, 1.1)])
@pytest.mark.parametrize("n", [3, 16, 32, 33, 40, 66])
def test_cftp_matches_sub_sweep_kernels(rt, n, abc):
    S = rt.SixVertexTiler
    for first in (1, 3, 16, 600) if n < 40 else (16, 600):
        out, st = S(*abc, fast_stream=1).cftp(S.MaxHeight(n), S.MinHeight(n), 21, first_sweeps=first, max_attempts=16)
        ref, sr = S(*abc, fast_stream=1, engine=1).cftp(S.MaxHeight(n), S.MinHeight(n), 21, first_sweeps=first,
                                                        max_attempts=16)
        assert np.array_equal(out, ref)
        for key in ("attempts", "total_steps", "final_steps", "flip_attempts"):
            assert st[key] == sr[key], (first, key)


@pytest.mark.gpu
def test_engine_two_serves_and_refuses_what_it_did(rt):
    S = rt.SixVertexTiler
    n = 4600  # would fit in 16 CTAs' shared memory
    a, b = S.MinHeight(n), S.MinHeight(n)
    S(engine=2).Walk(a, 2, 1)
    S(engine=1).Walk(b, 2, 1)
    assert np.array_equal(a, b)
    h = S.MinHeight(6000)
    with pytest.raises(rt.RTError):
        S(engine=2).Walk(h, 1, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [95, 96, 97, 127, 128, 160])
def test_heights_packed_on_the_device(rt, orc, n):
    # sizes around the rule and around words of 32 points; heights of any parity and offset
    S = rt.SixVertexTiler
    for off in (0, 1, -6):
        a = S.MaxHeight(n) + np.int32(off)
        b = a.copy()
        S(0.9, 1.0, 1.3, fast_stream=2).Walk(a, 9, 31)
        orc.sv_walk(b, n, 0, 36, 31, 2, 0.9, 1.0, 1.3)
        assert np.array_equal(a, b)
    for y, x in ((0, 0), (n, n), (n // 2, n), (3, 64)):
        bad = S.MinHeight(n)
        bad[y * (n + 1) + x] += 1
        kept = bad.copy()
        with pytest.raises(rt.RTError, match="not a height function"):
            S().Walk(bad, 3, 1)
        assert np.array_equal(bad, kept)
