"""The FP64 acceptance of a collision pair, which FP32 settles unless the
variate lies within 2^-13 of the estimate: the same pairs collide as in the
oracle's FP64 test, over some 4e5 pairs, of which some hundred lie that near.
A decision could differ by rounding only for a variate within about 1e-9 of the
acceptance (states agree to that after the few collisions a particle has
here), 4e-4 expected."""
import ctypes as C

import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle
from pydsmc import gpu

pytestmark = pytest.mark.gpu


def _sigma_c(mess, eta, crmax):
    """The majorant of the pair count but for constants (collisionDiameter,
    src/ProcessDSMC.cpp:2626-2645)."""
    cr = crmax * float(mess["v_rms"])
    return cr * (2.0 * float(mess["kB"]) * float(mess["T_ref"]) / float(mess["p_mass_r"]) / cr ** 2) ** eta


# 1 - 2 eta: the library's gas, both ends and the sign of what FP32 settles, and
# beyond it, where FP64 decides alone
@pytest.mark.parametrize("eta", [0.24, 0.0, 0.9, -3.4999, 4.4999, -3.51, 4.51])
@pytest.mark.parametrize("crmax", [3.0, 1.0])
def test_the_same_pairs_collide(block, eta, crmax):
    raw, dm, mess = block
    # the library's gas has 630,040 candidate pairs here at crmax 3: 500 a cell
    neff = float(mess["Neff"]) * 500.0 * dm.ncell / 630040.0
    neff *= _sigma_c(mess, float(mess["eta"]), 3.0) / _sigma_c(mess, eta, crmax)
    mess = mess.copy()
    mess["eta"], mess["Neff"] = eta, neff
    x, v, ir, cell = I.fill_inputs(dm, mess, 400, 17)
    cr = np.full(dm.ncell, crmax)
    with make_case(dm, mess, seed=21) as case:
        case.upload_particles(x, v, ir, cell)
        case.set_cell_state(crmax=cr)
        case.collisionDSMC()
        vg, c = case.download_particles()[1], case.counters()
    o = make_oracle(dm, mess, seed=21)
    o.set_particles(x, v, ir, cell)
    o.lib.oracle_set_cell_state(o.h, cr.ctypes.data_as(C.c_void_p), None, None)
    o.step(0, gpu.STAGE_COLLIDE)
    vo, oc = o.particles()[1], o.counters()
    assert c["candidate_pairs"] == oc["candidate_pairs"]
    assert 450 * dm.ncell < c["candidate_pairs"] < 550 * dm.ncell
    assert c["collisions"] == oc["collisions"] > 0
    assert np.array_equal((vg != v).any(1), (vo != v).any(1))
