"""The caller's height buffer is only copied to: a byte address between two words does, and a call that
is refused leaves it as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,offset", [(3, 2), (40, 1), (40, 4), (200, 6)])
def test_heights_at_any_address(rt, order, offset):
    torch = pytest.importorskip("torch")
    D = rt.DominoTiler
    d = D.AztecDiamond(order)
    t = D.MaxTiling(d)
    n = rt.side_of(t)
    s = rt.DominoSampler(n, 1, D(rule="cftp"))
    s.load(0, t)
    buf = torch.full((4 * n * n + 16,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(rt.RTError):  # no domain yet
        s.accumulate_heights(0, 0, buf.data_ptr() + offset)
    assert bool((buf == 7).all())
    s.set_domain(d)
    sums = torch.zeros(n * n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    s.accumulate_heights(0, sums.data_ptr(), buf.data_ptr() + offset)
    s.sync()
    s.close()
    raw = buf.cpu().numpy()
    got = raw[offset:offset + 4 * n * n].copy().view(np.int32)
    want = D.TilingToHeightfunc(t, d)
    assert np.array_equal(got, want)
    assert (raw[:offset] == 7).all() and (raw[offset + 4 * n * n:] == 7).all()
    assert np.array_equal(sums.cpu().numpy(), np.where(want != np.iinfo(np.int32).max, want, 0))
