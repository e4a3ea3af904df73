"""FP64 sampling (statistic_macro) where a warp takes runs of several cells:
meshes of as many cells as make its runs 1, 2, 3 and 32 cells long with a
shorter last one, with empty cells first, in the middle and last in a run and
cells of 1, 31, 32, 33, 65 and 300 particles. The oracle adds the same terms in
the same order, each operation rounded on its own, so every sum, field, window
count and sparse state is the same bit for bit; four steps take the window
through two exchanges."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle
from pydsmc import gpu
from pydsmc import mesh as M

pytestmark = pytest.mark.gpu

BOXES = {1: (13, 11, 9), 2: (31, 23, 21), 3: (29, 28, 28), 32: (61, 61, 62)}


def _run_length(ncell):
    import torch
    return max(1, min(32, ncell // (torch.cuda.get_device_properties(0).multi_processor_count * 48)))


@pytest.mark.parametrize("run", sorted(BOXES))
def test_fp64_sampling_runs_match_oracle(run):
    dm = M.build_dsmc_mesh(M.hex_box(*BOXES[run], 1.0, 0.8, 0.6))
    mess = I.block_mess(dm, 5)
    group = _run_length(dm.ncell)
    if group != run:
        pytest.skip(f"runs of {group} cells on this device")
    assert run == 1 or dm.ncell % run
    rs = np.random.RandomState(3)
    n = rs.choice([0, 1, 2, 3, 31, 32, 33, 65], dm.ncell, p=[0.3, 0.3, 0.2, 0.14, 0.02, 0.02, 0.01, 0.01])
    first = np.arange(0, dm.ncell, run)
    n[first[1::3]] = 0                                        # the first cell of a run
    n[np.minimum(first + run // 2, dm.ncell - 1)[2::5]] = 0   # one inside it
    n[np.minimum(first + run - 1, dm.ncell - 1)[::4]] = 0     # the last
    n[-1] = 33
    n[first[7]] = 300
    n[first[9]: first[9] + run] = 0                           # all of a run
    cell = np.repeat(np.arange(dm.ncell), n).astype(np.int32)
    u, sig, tN = I.freestream(mess)
    v = u + sig * rs.standard_normal((cell.shape[0], 3))
    ir = -0.5 * tN * np.log(1.0 - rs.random_sample(cell.shape[0]))
    x = dm.cells["cellXY"][cell]
    kw = dict(nss=2, nscheme=3, nevery=1, nrepeat=2)
    o = make_oracle(dm, mess, **kw)
    o.set_particles(x, v, ir, cell)
    with make_case(dm, mess, keep_step_moments=1, **kw) as case:
        case.upload_particles(x, v, ir, cell)
        case.statistic_macroPre()
        o.macro_pre()
        for k in range(1, 5):
            case.step(k, gpu.STAGE_SAMPLE)
            o.step(k, gpu.STAGE_SAMPLE)
            assert np.array_equal(case.step_moments(), o.step_moments()), k
        assert (case.step_moments()[:, 0] == n).all()
        for which in (gpu.MACRO_LOCAL, gpu.MACRO_RECORD, gpu.MACRO_FINAL_RECORD):
            assert np.array_equal(case.macro(which), o.macro(which)), which
        g, w = case.counts(), o.counts()
        for k in ("ppc", "window_samples", "window_valid", "sparse_state"):
            assert np.array_equal(g[k], w[k]), k
    assert len(np.unique(w["sparse_state"])) > 1
