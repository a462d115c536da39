"""Device height functions of domains whose rows and columns are all short: diagonal strips of 2 x 2
blocks, in both directions, and zigzags of them, against the host's; and that their time stays within
reach of a diamond's of the same side (spread along lines alone, a strip one block wide takes 140 times
as long at side 1004, with the passes inside tiles less than 20)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _strip(blocks, wide, kind):
    m = 2 * blocks + 3
    d = np.zeros((m, m), np.int32)
    for a in range(blocks):
        b0 = a if kind == "down" else blocks - 1 - a
        if kind == "zigzag":
            b0 = abs((a + 20) % 80 - 40) % blocks
        for b in range(max(0, b0 - wide + 1), min(blocks, b0 + wide)):
            d[1 + 2 * a:3 + 2 * a, 1 + 2 * b:3 + 2 * b] = 1
    t = np.zeros((m + 1, m + 1), np.int32)  # horizontal dominoes from odd columns
    left = d[:, 1:m - 1:2]
    t[:m, 2:m:2] |= 2 * left
    t[1:, 2:m:2] |= left
    return d.ravel(), t.ravel()


@pytest.mark.parametrize("kind", ["down", "up", "zigzag"])
@pytest.mark.parametrize("blocks,wide", [(1, 1), (3, 1), (15, 1), (16, 1), (17, 1), (31, 2), (60, 3), (200, 1), (200, 6)])
def test_equal_to_the_host(rt, blocks, wide, kind):
    d, t = _strip(blocks, wide, kind)
    D = rt.DominoTiler
    assert np.array_equal(D.TilingToHeightfuncDevice(t, d), D.TilingToHeightfunc(t, d))


def test_time_against_a_diamond(rt):
    torch = pytest.importorskip("torch")
    D = rt.DominoTiler
    diamond = D.AztecDiamond(499)
    best = []
    for d, t in ((diamond, D.MinTiling(diamond)), _strip(500, 1, "down")):
        n = rt.side_of(t)
        s = rt.DominoSampler(n, 1, D(rule="cftp"))
        s.load(0, t)
        s.set_domain(d)
        h = torch.empty(n * n, dtype=torch.int32, device="cuda")
        times = []
        for _ in range(6):
            s.sync()
            t0 = time.perf_counter()
            s.accumulate_heights(0, 0, h.data_ptr())
            s.sync()
            times.append(time.perf_counter() - t0)
        s.close()
        best.append(min(times))
    assert best[1] < 50 * best[0], best
