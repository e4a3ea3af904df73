"""The tracing check where the FP32 exit test has the least room: meshes far from
the origin and of very small and large cells, particles on faces, edges and
corners, at rest, along the axes, slow and fast, with short and long flights.
Each decision and the final state against the oracle's FP64 trace, on the state
that the precision stores. The walls are outlets: a re-emission (behind an
unmapped face, where the flight goes on) draws its velocity in the precision."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle, rel_close
from pydsmc import gpu
from pydsmc import mesh as M

pytestmark = pytest.mark.gpu


def _mesh(scale, shift, tets=False):
    if tets:
        from pydsmc import capsule
        raw = capsule.capsule_mesh(**I.CAPSULE_SMALL)
    else:
        raw = M.block_case_mesh(scale=8)
    raw.points[...] = raw.points * scale + np.asarray(shift)
    return M.build_dsmc_mesh(raw)


def _particles(dm, n, seed):
    rs = np.random.RandomState(seed)
    P = dm.points.reshape(-1, 3)
    cell = rs.randint(0, dm.ncell, size=n).astype(np.int32)
    face = dm.cells["cell2face"][cell, rs.randint(0, 4, n)]
    tri = P[dm.edges["faceMap"][face, :3]]
    cc = dm.cells["cellXY"][cell]
    size = np.abs(tri - cc[:, None]).max((1, 2))[:, None]
    w = rs.dirichlet(np.ones(3), n)
    kind = np.arange(n) % 6
    w[kind == 1] = np.array([0.5, 0.5, 0.0])               # on an edge
    w[kind == 2] = np.array([1.0, 0.0, 0.0])               # on a corner
    x = np.einsum("nk,nkd->nd", w, tri)                    # on a face
    inside = (kind >= 3)[:, None]
    x = np.where(inside, cc + (x - cc) * rs.random_sample((n, 1)), x)
    x[kind == 3] = cc[kind == 3]                           # the centre
    v = rs.standard_normal((n, 3))
    axis = np.arange(n) % 7 == 0
    v[axis] = np.eye(3)[rs.randint(0, 3, axis.sum())] * rs.choice([-1.0, 1.0], axis.sum())[:, None]
    mag = rs.choice([0.0, 1e-24, 1e-12, 1.0, 1e6], n, p=[0.05, 0.05, 0.1, 0.7, 0.1])
    dt = np.where(mag > 0.0, size[:, 0] / np.maximum(mag, 1e-300), 1.0) * rs.choice([1e-6, 0.3, 5.0], n)
    return x, v * mag[:, None], dt, cell


@pytest.mark.parametrize("precision", [gpu.PRECISION_FP64, gpu.PRECISION_MIXED])
@pytest.mark.parametrize("scale,shift,tets", [(1.0, (0, 0, 0), False), (1.0, (3e3, -1e4, 2e4), False),
                                              (1e-5, (0, 0, 0), False), (1e5, (0, 0, 0), False),
                                              (1.0, (0, 0, 0), True), (1.0, (-2e4, 5e3, 0), True)])
def test_trace_extremes_match_oracle(precision, scale, shift, tets):
    dm = _mesh(scale, shift, tets)
    mess = I.block_mess(dm, 20)
    x, v, dt, cell = _particles(dm, 60000, 4)
    with make_case(dm, mess, zones=I.NOWALL_ZONES, seed=5, precision=precision) as case:
        g = case.trace(x, v, dt, cell, stop_at_wall=True)
    if precision == gpu.PRECISION_MIXED:
        x, v = I.fp32_state(dm, x, v, cell)
    o = make_oracle(dm, mess, zones=I.NOWALL_ZONES, seed=5).trace(x, v, dt, cell, stop_at_wall=True)
    for k in ("cell", "ifout", "face", "tri", "ncross"):
        assert np.array_equal(g[k], o[k]), (k, int((g[k] != o[k]).sum()))
    assert np.array_equal(g["dt"], o["dt"])
    if precision == gpu.PRECISION_FP64:
        assert np.array_equal(g["x"], o["x"]) and np.array_equal(g["v"], o["v"])
    assert (o["ncross"] > 0).sum() > 5000 and (o["ifout"] == 0).sum() > 5000
