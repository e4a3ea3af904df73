"""The cell sort's order of arrivals from beyond the face neighbours, at the
edges of its segment sizes (one lane, a warp's sorts of 32 to 512, and rank
counting beyond)."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case
from pydsmc import gpu

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 12, 13, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 700]


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
def test_far_arrivals_in_source_order(block, precision):
    """Particles two cells upstream of a target fly into it in one step; the
    target holds them in their source order (their Ir is their number)."""
    raw, dm, mess = block
    cc = dm.cells["cellXY"]
    h = 1.0 / 12
    rs = np.random.RandomState(2)
    # columns of cells away from the removed block and the sides, each with one source and one target
    src = [int(np.argmin(((cc - np.array([(2.5 + 6 * (i % 2)) * h, (0.5 + i // 8) * 0.0625, (0.5 + (i % 8)) * 0.0625])) ** 2)
                         .sum(1))) for i in range(len(SIZES))]
    assert len(set(src)) == len(src)
    dst = [int(np.argmin(((cc - (cc[s] + np.array([2 * h, 0, 0]))) ** 2).sum(1))) for s in src]
    cell = np.concatenate([np.full(m, s) for m, s in zip(SIZES, src)]).astype(np.int32)
    tag = np.arange(cell.shape[0], dtype=float)
    order = np.argsort(cell, kind="stable")
    cell, want = cell[order], {}
    x = cc[cell] + (rs.random_sample((cell.shape[0], 3)) - 0.5) * np.array([0.2 * h, 0.01, 0.01])
    v = np.zeros_like(x)
    v[:, 0] = 2 * h / float(mess["dtime"])
    for s, d in zip(src, dst):
        want[d] = tag[cell == s]
    with make_case(dm, mess, precision=precision) as case:
        case.upload_particles(x, v, tag, cell)
        case.step(1, gpu.STAGE_MOVE | gpu.STAGE_SORT)
        _, _, ir, c = case.download_particles()
    assert c.shape[0] == cell.shape[0]
    for d, w in want.items():
        assert np.array_equal(ir[c == d], w), d
