"""Particle upload, download and the tracing check at the edges of the
transfer's blocks (65,536 values) and of the tracing check's chunks (131,072
particles)."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle, rel_close
from pydsmc import gpu

pytestmark = pytest.mark.gpu


def _particles(dm, mess, n, seed):
    rs = np.random.RandomState(seed)
    cell = np.sort(rs.randint(0, dm.ncell, size=n)).astype(np.int32)
    lo, hi = I.cell_boxes(dm)
    u, sig, tN = I.freestream(mess)
    return (lo[cell] + (hi[cell] - lo[cell]) * rs.random_sample((n, 3)), u + sig * rs.standard_normal((n, 3)),
            -0.5 * tN * np.log(1.0 - rs.random_sample(n)), cell)


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
@pytest.mark.parametrize("n", [1, 65535, 65536, 65537, 200001])
def test_upload_download_round_trip(block, n, precision):
    """What comes back is what went up (mixed: its FP32 rounding), from
    cell-major arrays and from shuffled ones, whose cells keep their order."""
    raw, dm, mess = block
    x, v, ir, cell = _particles(dm, mess, n, 3)
    mixed = precision == gpu.PRECISION_MIXED
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    o = np.random.RandomState(4).permutation(n)
    with make_case(dm, mess, precision=precision) as case:
        for order in (np.arange(n), o):
            case.upload_particles(x[order], v[order], ir[order], cell[order])
            want = order[np.argsort(cell[order], kind="stable")]
            xg, vg, irg, cg = case.download_particles()
            assert np.array_equal(cg, cell[want])
            assert np.array_equal(xg, I.fp32_positions(dm, x[want], cell[want]) if mixed else x[want])
            assert np.array_equal(vg, f32(v[want]) if mixed else v[want])
            assert np.array_equal(irg, f32(ir[want]) if mixed else ir[want])


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
def test_download_between_move_and_sort(block, precision):
    """Slots of removed particles (cell -1) are still there; every other
    particle lies in its cell, to the rounding of an FP32 offset."""
    raw, dm, mess = block
    x, v, ir, cell = _particles(dm, mess, 70000, 3)
    lo, hi = I.cell_boxes(dm)
    with make_case(dm, mess, precision=precision) as case:
        case.upload_particles(x, v, ir, cell)
        case.advection(1)
        xg, vg, irg, cg = case.download_particles()
        cnt = case.counters()
    removed = cnt["removed"] + cnt["dropped"] + cnt["lost"]
    live = cg >= 0
    assert removed > 0 and (~live).sum() == removed
    assert np.all(xg[live] >= lo[cg[live]] - 1e-6) and np.all(xg[live] <= hi[cg[live]] + 1e-6)


@pytest.mark.parametrize("n", [65537, 131072, 131075])
def test_trace_in_chunks_matches_oracle(block, n):
    """With wall re-emission, whose random streams are numbered by particle:
    the second chunk continues the numbering."""
    raw, dm, mess = block
    x, v, dt, cell = I.trace_inputs(dm, mess, n, 6)
    with make_case(dm, mess, seed=5) as case:
        g = case.trace(x, v, dt, cell, stop_at_wall=False)
    o = make_oracle(dm, mess, seed=5).trace(x, v, dt, cell, stop_at_wall=False)
    for k in ("cell", "ifout", "face", "tri", "ncross"):
        assert np.array_equal(g[k], o[k]), k
    for k in ("x", "v", "dt"):
        assert np.all(rel_close(g[k], o[k], 1e-9, 1e-12)), k


def test_trace_memory_grows(block):
    """A small call, a larger one and the small one again, on one handle,
    against fresh handles."""
    raw, dm, mess = block
    x, v, dt, cell = I.trace_inputs(dm, mess, 70001, 6)
    with make_case(dm, mess, seed=5, precision=gpu.PRECISION_MIXED) as case:
        kept = [case.trace(x[:n], v[:n], dt[:n], cell[:n], stop_at_wall=False) for n in (33, 70001, 33)]
    for n, g in zip((33, 70001, 33), kept):
        with make_case(dm, mess, seed=5, precision=gpu.PRECISION_MIXED) as case:
            f = case.trace(x[:n], v[:n], dt[:n], cell[:n], stop_at_wall=False)
        for k in f:
            assert np.array_equal(f[k], g[k]), k
