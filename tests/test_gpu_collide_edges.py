"""Collisions at the ends of the classes by particle count that the FP64 path
has (a lane's cells 12, a warp's arena 376, a block's 3,072; FP32: 16, 512,
4,096), and of cells run in place (claims in shared memory up to 27,648 and
20,480 particles, in the cell-id slots beyond): FP64 against the oracle,
mixed by the momentum of each cell and by its bits on a second run."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle, rel_close
from pydsmc import gpu

pytestmark = pytest.mark.gpu


def _fill(dm, mess, counts, seed):
    rs = np.random.RandomState(seed)
    cell = np.sort(np.repeat(rs.permutation(dm.ncell)[: len(counts)], counts)).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    return x, u + sig * rs.standard_normal(x.shape), -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0])), cell


def _collide(dm, mess, parts, **kw):
    with make_case(dm, mess, seed=11, **kw) as case:
        case.upload_particles(*parts)
        case.collisionDSMC()
        return case.download_particles(), case.cell_state(), case.counters()


def _with_pairs(dm, parts, pairs):
    """The block's constants with about this many candidate pairs in all."""
    mess = I.block_mess(dm, 20).copy()
    mess["Neff"] = float(mess["Neff"]) * pairs / max(_collide(dm, mess, parts)[2]["candidate_pairs"], 1)
    return mess


def test_fp64_class_ends_match_oracle(block):
    """At most 2 pairs a particle in the largest cells: states to 1e-9 for 97%
    of the particles (the bound of the full tetrahedral step), majorants and
    pair remainders likewise and exactly."""
    raw, dm, mess = block
    counts = [11, 12, 13, 375, 376, 377, 3071, 3072, 3073]
    parts = _fill(dm, mess, counts, 8)
    mess = _with_pairs(dm, parts, 9000)
    (_, vg, irg, cg), cs, cnt = _collide(dm, mess, parts)
    o = make_oracle(dm, mess, seed=11)
    o.set_particles(*parts)
    o.step(0, gpu.STAGE_COLLIDE)
    _, vo, iro, co = o.particles()
    assert np.array_equal(cg, co)
    assert np.array_equal(cs[1], o.cell_state()[1])
    assert cnt["candidate_pairs"] == o.counters()["candidate_pairs"] > 8000
    ok = rel_close(vg, vo, 1e-9, 1e-12).all(1) & rel_close(irg, iro, 1e-9, 1e-12)
    assert ok.mean() >= 0.97, ok.mean()


def test_mixed_cells_in_place_lose_no_write(block):
    """A collision changes the sum of its two particles' velocities by the
    rounding of their mean (counted twice) and of the two results, each at most
    half an ulp h of the largest component, without bias: over k collisions a
    deviation of sqrt(6 k / 3) h < 2 h sqrt(k). The bound is eight of these.
    A write lost changes the sum by the order of the thermal speed, 1. Collisions
    of a cell: at most its candidate pairs, which go with n (n - 1)."""
    raw, dm, mess = block
    counts = [4095, 4096, 4097, 20480, 20481]
    parts = _fill(dm, mess, counts, 8)
    mess = _with_pairs(dm, parts, 70000)
    runs = [_collide(dm, mess, parts, precision=gpu.PRECISION_MIXED) for _ in range(2)]
    for a, b in zip(runs[0][0], runs[1][0]):
        assert np.array_equal(a, b)
    for a, b in zip(runs[0][1], runs[1][1]):
        assert np.array_equal(a, b)
    (_, vg, irg, cg), _, cnt = runs[0]
    cell, v = parts[3], parts[1].astype(np.float32).astype(np.float64)
    assert np.array_equal(cg, cell)
    h = 2.0 ** (np.ceil(np.log2(max(np.abs(vg).max(), np.abs(v).max()))) - 25.0)
    n = np.bincount(cell, minlength=dm.ncell).astype(float)
    k = cnt["candidate_pairs"] * n * (n - 1.0) / (n * (n - 1.0)).sum()
    assert cnt["collisions"] > 20000
    for d in range(3):
        lost = np.abs(np.bincount(cell, vg[:, d], dm.ncell) - np.bincount(cell, v[:, d], dm.ncell))
        assert np.all(lost <= 8.0 * 2.0 * h * np.sqrt(k)), (lost.max(), d)
