"""Deletions of the GSIS particle update at the ends of their batches (32 draws)
and of the slot table in shared memory (1,024 particles, global memory
beyond), against the oracle: the same particles kept, in the same order, and
after the linear map the same velocities and internal energies bit for bit
(copies and IEEE arithmetic in the same order). In mixed precision the kept
particles are those of the oracle, by their stored positions."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle
from pydsmc import gpu

pytestmark = pytest.mark.gpu

COUNTS = [31, 32, 33, 64, 65, 66, 200, 1023, 1024, 1025, 1500]
DELETE = [1, 31, 32, 33, 64, 65]


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
def test_deletion_batches_match_oracle(block, precision):
    raw, dm, mess = block
    rs = np.random.RandomState(31)
    jobs = [(n, r) for n in COUNTS for r in DELETE + [n - 2, n - 1, n] if 0 < r <= n]
    pick = np.sort(rs.permutation(dm.ncell)[: len(jobs)])
    have, keep = np.full(dm.ncell, 3), np.full(dm.ncell, 3)
    for c, (n, r) in zip(pick, jobs):
        have[c], keep[c] = n, n - r
    cell = np.repeat(np.arange(dm.ncell), have).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    x = lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((cell.shape[0], 3))
    v = u + sig * rs.standard_normal(x.shape)
    ir = -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0]))
    ns = np.empty((dm.ncell, 6))
    # the count the update draws is keep or, once in 10^6, one more
    ns[:, 0] = (keep + 1e-6) * float(mess["Neff"]) / (dm.cells["area"] * float(mess["n_ref"]))
    ns[:, 1:4] = u + 0.3 * rs.standard_normal((dm.ncell, 3))
    ns[:, 4:6] = tN * rs.uniform(0.7, 1.4, (dm.ncell, 2))
    with make_case(dm, mess, seed=9, precision=precision) as case:
        case.upload_particles(x, v, ir, cell)
        rep = case.molecular_velocity_change(ns, None)
        xg, vg, irg, cg = case.download_particles()
    o = make_oracle(dm, mess, seed=9)
    o.set_particles(x, v, ir, cell)
    orep = o.molecular_velocity_change(ns, None)
    xo, vo, iro, co = o.particles()
    assert rep == orep and rep["removed"] >= sum(r for _, r in jobs) - 2
    assert np.array_equal(cg, co)
    if precision == gpu.PRECISION_MIXED:
        assert np.array_equal(xg, I.fp32_positions(dm, xo, co))
    else:
        assert np.array_equal(xg, xo) and np.array_equal(vg, vo) and np.array_equal(irg, iro)
