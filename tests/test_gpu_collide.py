"""Collisions of cells at the edges of the collision pass's classes: one lane
(16 particles), a warp's arena (512), a block's arena (4,096), in place
beyond it, and the pair counts that move a cell to a block (1,024) and to
the front of the list (8,192)."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle, rel_close
from pydsmc import gpu

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 15, 16, 17, 33, 64, 255, 256, 257, 511, 512, 513, 1024, 1500, 4095, 4096, 4097]


def _fill(dm, mess, seed):
    rs = np.random.RandomState(seed)
    pick = rs.permutation(dm.ncell)[: len(COUNTS)]
    cell = np.repeat(pick, COUNTS).astype(np.int32)
    cell = np.sort(cell)
    lo, hi = I.cell_boxes(dm)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    u, sig, tN = I.freestream(mess)
    return x, u + sig * rs.standard_normal((cell.shape[0], 3)), -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0])), cell


def _mess(dm, pairs_of_largest):
    """The block's constants with the real particles per simulated one such
    that the 4,097-particle cell has about this many candidate pairs (crmax
    starts at 3)."""
    mess = I.block_mess(dm, 20).copy()
    case_pairs = {}
    with make_case(dm, mess, seed=1) as case:
        x, v, ir, cell = _fill(dm, mess, 5)
        case.upload_particles(x, v, ir, cell)
        case.collisionDSMC()
        case_pairs = case.counters()["candidate_pairs"]
    total = sum(n * (n - 1) for n in COUNTS)
    mess["Neff"] = float(mess["Neff"]) * pairs_of_largest * total / (4097 * 4096) / max(case_pairs, 1)
    return mess


@pytest.mark.parametrize("pairs", [9000, 70000])
def test_fp64_cell_classes_match_oracle(block, pairs):
    """One pass: pair counts and remainders exact. At 9,000 pairs in the
    largest cell (4.4 a particle at most) the states agree to 1e-9 for 97%
    of the particles, the bound of the full tetrahedral step (30 pairs a
    particle); at 70,000 (34 a particle, more than there) momentum and
    energy of every cell are kept to rounding."""
    raw, dm, _ = block
    mess = _mess(dm, pairs)
    x, v, ir, cell = _fill(dm, mess, 5)
    with make_case(dm, mess, seed=11) as case:
        case.upload_particles(x, v, ir, cell)
        case.collisionDSMC()
        _, vg, irg, cg = case.download_particles()
        cs, cnt = case.cell_state(), case.counters()
    o = make_oracle(dm, mess, seed=11)
    o.set_particles(x, v, ir, cell)
    o.step(0, gpu.STAGE_COLLIDE)
    _, vo, iro, co = o.particles()
    oc, ocnt = o.cell_state(), o.counters()
    assert np.array_equal(cg, co)
    assert np.array_equal(cs[1], oc[1])
    assert cnt["candidate_pairs"] == ocnt["candidate_pairs"]
    assert cnt["big_cells"] == sum(n > 512 for n in COUNTS)
    assert abs(cnt["collisions"] - ocnt["collisions"]) <= 1e-3 * ocnt["collisions"] + 2
    if pairs == 9000:
        ok = rel_close(vg, vo, 1e-9, 1e-12).all(1) & rel_close(irg, iro, 1e-9, 1e-12)
        assert ok.mean() >= 0.97, ok.mean()
        assert rel_close(cs[0], oc[0], 1e-9).mean() >= 0.97
    for q0, q1 in ((v, vg), ((0.5 * (v ** 2).sum(1) + ir)[:, None], (0.5 * (vg ** 2).sum(1) + irg)[:, None])):
        a = np.stack([np.bincount(cell, weights=q0[:, k]) for k in range(q0.shape[1])])
        b = np.stack([np.bincount(cell, weights=q1[:, k]) for k in range(q1.shape[1])])
        assert np.allclose(a, b, rtol=1e-11, atol=1e-9)


@pytest.mark.parametrize("pairs", [9000, 70000])
def test_mixed_cell_classes_conserve(block, pairs):
    """The mixed pass over the same cells: FP64's pair counts, momentum and
    energy of every cell to FP32 rounding (a collision rounds each component
    by at most a few 2^-24 of a speed of about 3; a particle takes part in at
    most some 70, and a cell adds up at most 4,097), and the same bits
    again."""
    raw, dm, _ = block
    mess = _mess(dm, pairs)
    x, v, ir, cell = _fill(dm, mess, 5)
    outs = []
    for _ in range(2):
        with make_case(dm, mess, seed=11, precision=gpu.PRECISION_MIXED) as case:
            case.upload_particles(x, v, ir, cell)
            case.collisionDSMC()
            _, vg, irg, cg = case.download_particles()
            outs.append((vg, irg, case.cell_state()[0], case.cell_state()[1], case.counters()))
    for a, b in zip(outs[0][:4], outs[1][:4]):
        assert np.array_equal(a, b)
    with make_case(dm, mess, seed=11) as case:
        case.upload_particles(x, v, ir, cell)
        case.collisionDSMC()
        assert np.array_equal(case.cell_state()[1], outs[0][3])
        assert case.counters()["candidate_pairs"] == outs[0][4]["candidate_pairs"]
    vg, irg = outs[0][:2]
    e0, e1 = 0.5 * (v ** 2).sum(1) + ir, 0.5 * (vg ** 2).sum(1) + irg
    n = np.bincount(cell)
    for q0, q1 in ((v[:, 0], vg[:, 0]), (v[:, 1], vg[:, 1]), (v[:, 2], vg[:, 2]), (e0, e1)):
        d = np.abs(np.bincount(cell, weights=q1) - np.bincount(cell, weights=q0))
        assert np.all(d <= 70 * 16 * 2.0 ** -24 * np.maximum(n, 1)), d.max()
    assert (vg != v.astype(np.float32)).any(1).sum() > 0.5 * len(cell)


def test_fp64_cells_at_the_arenas_ends_match_oracle(block):
    """A warp's FP64 arena (376) and a block's (2,048), a lane's cells (12),
    as in test_fp64_cell_classes_match_oracle at 9,000 pairs."""
    raw, dm, _ = block
    mess = _mess(dm, 9000)
    counts = [11, 12, 13, 375, 376, 377, 2047, 2048, 2049]
    rs = np.random.RandomState(8)
    cell = np.sort(np.repeat(rs.permutation(dm.ncell)[: len(counts)], counts)).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    v, ir = u + sig * rs.standard_normal(x.shape), -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0]))
    with make_case(dm, mess, seed=11) as case:
        case.upload_particles(x, v, ir, cell)
        case.collisionDSMC()
        _, vg, irg, cg = case.download_particles()
        cs = case.cell_state()
    o = make_oracle(dm, mess, seed=11)
    o.set_particles(x, v, ir, cell)
    o.step(0, gpu.STAGE_COLLIDE)
    _, vo, iro, co = o.particles()
    assert np.array_equal(cg, co)
    assert np.array_equal(cs[1], o.cell_state()[1])
    ok = rel_close(vg, vo, 1e-9, 1e-12).all(1) & rel_close(irg, iro, 1e-9, 1e-12)
    assert ok.mean() >= 0.97, ok.mean()


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
def test_who_takes_a_cell_does_not_matter(precision):
    """100 cells of 200 particles and some 700 pairs, and 100 of 10 particles:
    alone, blocks take the first and half warps the second; among 500 of the
    one kind and 5,580 of the other, warps and single lanes. The same bits."""
    raw, dm = I.block_mesh(8)
    mess = I.block_mess(dm, 20).copy()
    vol = np.asarray(dm.cells["area"], dtype=float)
    order = np.argsort(np.abs(vol - np.median(vol)), kind="stable")
    rs = np.random.RandomState(2)
    n = np.full(dm.ncell, 10)
    n[order[:500]] = 200
    cell = np.repeat(np.arange(dm.ncell), n).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    v, ir = u + sig * rs.standard_normal(x.shape), -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0]))
    few = np.zeros(dm.ncell, bool)
    few[order[:100]] = True
    few[order[500:600]] = True
    few = few[cell]
    only = few & (n[cell] == 200)
    with make_case(dm, mess, seed=1, precision=precision) as case:
        case.upload_particles(x[only], v[only], ir[only], cell[only])
        case.collisionDSMC()
        mess["Neff"] = float(mess["Neff"]) * 700.0 * 100 / case.counters()["candidate_pairs"]
    outs = []
    for keep in (few, np.ones(few.shape, bool)):
        with make_case(dm, mess, seed=9, precision=precision) as case:
            case.upload_particles(x[keep], v[keep], ir[keep], cell[keep])
            case.collisionDSMC()
            _, vg, irg, _ = case.download_particles()
            outs.append((vg[few[keep]], irg[few[keep]], case.counters()["candidate_pairs"]))
    assert 100 * 512 < outs[0][2] < 100 * 1024
    assert np.array_equal(outs[0][0], outs[1][0])
    assert np.array_equal(outs[0][1], outs[1][1])
    assert (outs[0][0] != v[few].astype(outs[0][0].dtype)).any(1).mean() > 0.5


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
def test_cells_beyond_a_blocks_arena(block, precision):
    """Cells run in place: at the end of a block's arena (3,072 in FP64, 4,096
    in FP32) and of the claims that fit its memory (27,648 and 20,480), with
    3.4 pairs a particle at most. FP64 against the oracle as in
    test_fp64_cell_classes_match_oracle; mixed keeps every cell's momentum and
    energy to the bound of test_mixed_cell_classes_conserve. The claims leave
    no trace in the cell ids."""
    raw, dm, _ = block
    mess = _mess(dm, 1000)
    counts = [3072, 3073, 27648, 27649] if precision == gpu.PRECISION_FP64 else [4096, 4097, 20480, 20481]
    rs = np.random.RandomState(8)
    cell = np.sort(np.repeat(rs.permutation(dm.ncell)[: len(counts)], counts)).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    v, ir = u + sig * rs.standard_normal(x.shape), -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0]))
    with make_case(dm, mess, seed=11, precision=precision) as case:
        case.upload_particles(x, v, ir, cell)
        case.collisionDSMC()
        _, vg, irg, cg = case.download_particles()
        cnt = case.counters()
    assert np.array_equal(cg, cell)
    assert cnt["collisions"] > 0.05 * len(cell)
    if precision == gpu.PRECISION_FP64:
        o = make_oracle(dm, mess, seed=11)
        o.set_particles(x, v, ir, cell)
        o.step(0, gpu.STAGE_COLLIDE)
        _, vo, iro, co = o.particles()
        assert np.array_equal(co, cell)
        ok = rel_close(vg, vo, 1e-9, 1e-12).all(1) & rel_close(irg, iro, 1e-9, 1e-12)
        assert ok.mean() >= 0.97, ok.mean()
    e0, e1 = 0.5 * (v ** 2).sum(1) + ir, 0.5 * (vg ** 2).sum(1) + irg
    n = np.bincount(cell)
    for q0, q1 in ((v[:, 0], vg[:, 0]), (v[:, 1], vg[:, 1]), (v[:, 2], vg[:, 2]), (e0, e1)):
        d = np.abs(np.bincount(cell, weights=q1) - np.bincount(cell, weights=q0))
        assert np.all(d <= 70 * 16 * 2.0 ** -24 * np.maximum(n, 1)), d.max()
