"""The persistent tile walk of the pairwise MI kernel where it can go wrong: many tiles per CTA, one example, more rows
than the table of logarithms holds, values that are no category, and each way of writing the operands."""
import numpy as np
import pytest

from tests.test_gpu_pairwise_mi import _data

pytestmark = pytest.mark.gpu


def _mi64(data, c, pc):
    rows, v = data.shape
    oh = np.zeros((rows, v, c), np.float32)
    r, j = np.nonzero(data < c)
    oh[r, j, data[r, j]] = 1.0
    oh = oh.reshape(rows, v * c)
    joint = (oh.T @ oh).astype(np.float64).reshape(v, c, v, c).transpose(0, 2, 1, 3)   # counts, exact in float32
    single = (oh.sum(0, dtype=np.float64).reshape(v, c) + pc / c) / (rows + pc)
    p = (joint + pc / c ** 2) / (rows + pc)
    return (p * (np.log(p) - np.log(single)[:, None, :, None] - np.log(single)[None, :, None, :])).sum((2, 3))


# (categories, variables, rows): 2926 and 1892 tiles (20 and 13 per CTA); one example; rows past the table with 128-row
# tails; two-variable words, four-row groups, byte stores and variables wider than a tile, aligned and not
@pytest.mark.parametrize("c,v,rows,beyond", [
    (32, 600, 130, 0), (8, 1900, 64, 0), (4, 50, 1, 0), (2, 131, 8193, 0), (16, 20, 9001, 0), (64, 30, 257, 0),
    (128, 9, 1030, 0), (256, 5, 700, 0), (2, 300, 1601, 3), (8, 70, 515, 40), (32, 18, 400, 200)])
def test_tiles(c, v, rows, beyond):
    """Cells are sums of c^2 terms p (log p - ...) in float32: 1e-5 of the largest entry bounds their rounding."""
    from lvd_pg_b200 import api
    data = _data(c, v, rows, c + v)
    if beyond:   # values that are no category count nowhere
        data[np.random.default_rng(1).random(data.shape) < 0.1] = c + beyond if c + beyond < 256 else 255
    want = _mi64(data, c, 0.1)
    got = api.pairwise_mi(data, c, 0.1).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
    if c <= 32:
        assert np.array_equal(got, got.T)
