"""The move's kernels by mesh kind (they unroll over the mesh's face count)
and by particle count (shares of a thread, a block and the work list),
against the oracle's transport, FP64, states to 1e-9 and cells exact: both
sides trace every particle by the same FP64 operations, wall re-emission
differing in the last bits of CUDA's functions against libm, which a few
crossings do not carry past that."""
import numpy as np
import pytest

import inputs as I
from gpu_util import make_case, make_oracle, rel_close
from pydsmc import gpu
from pydsmc import mesh as M

pytestmark = pytest.mark.gpu

STAGES = gpu.STAGE_INJECT | gpu.STAGE_MOVE | gpu.STAGE_SORT
ZONES = I.REF_ZONES + [(7, gpu.ROLE_SPECULAR, 0)]


def _mesh(kind):
    if kind == "pyramid":
        return M.build_dsmc_mesh(M.pyramid_box(5, 4, 3, 1.0, 0.8, 0.6))
    if kind == "wedge":
        return M.build_dsmc_mesh(M.prism_box(6, 5, 4, 1.0, 0.8, 0.6))
    raw = M.block_case_mesh(scale=4)
    if kind == "warped":     # one node off its place: its cells' quads are not planar, the others are
        p = raw.points.copy()
        inner = np.nonzero(np.all((p > 0.1) & (p < np.array([0.3, 0.2, 0.2])), axis=1))[0][0]
        p[inner] += np.array([0.013, -0.009, 0.007])
        raw.points[...] = p
    return M.build_dsmc_mesh(raw)


def _points(dm, cell, rs):
    """Random points of the cells: the centroid moved towards a corner of a
    face by less than the whole way (the cells are star-shaped from it)."""
    P = dm.points.reshape(-1, 3)
    face = dm.cells["cell2face"][cell, 0]
    w = rs.dirichlet(np.ones(4), size=cell.shape[0])
    nodes = dm.edges["faceMap"][face, :3]
    tri = P[nodes]
    return w[:, :1] * dm.cells["cellXY"][cell] + np.einsum("nk,nkd->nd", w[:, 1:], tri)


def _transport(dm, mess, n, seed, precision=gpu.PRECISION_FP64, steps=2, **shape):
    rs = np.random.RandomState(seed)
    cell = np.sort(rs.randint(0, dm.ncell, size=n)).astype(np.int32)
    x = _points(dm, cell, rs)
    u, sig, tN = I.freestream(mess)
    v = u + 3.0 * sig * rs.standard_normal((n, 3))
    ir = -0.5 * tN * np.log(1.0 - rs.random_sample(n))
    with make_case(dm, mess, zones=ZONES, seed=13, precision=precision) as case:
        if shape:
            case.set_launch_shape(**shape)
        case.upload_particles(x, v, ir, cell)
        for s in range(1, steps + 1):
            case.step(s, STAGES)
        case.sync()
        g, c = case.download_particles(), case.counters()
    return (x, v, ir, cell), g, c


@pytest.mark.parametrize("kind", ["hexahedron", "wedge", "pyramid", "warped"])
def test_transport_by_mesh_kind_matches_oracle(kind):
    dm = _mesh(kind)
    mess = I.block_mess(dm, 20)
    start, (xg, vg, irg, cg), c = _transport(dm, mess, 20 * dm.ncell, 5)
    o = make_oracle(dm, mess, zones=ZONES, seed=13)
    o.set_particles(*start)
    for s in (1, 2):
        o.step(s, STAGES)
    xo, vo, iro, co = o.particles()
    assert np.array_equal(cg, co)
    for a, b in ((xg, xo), (vg, vo), (irg, iro)):
        assert np.all(rel_close(a, b, 1e-9, 1e-12))
    oc = o.counters()
    for k in ("injected", "removed", "dropped", "lost", "wall_hits", "crossings"):
        assert c[k] == oc[k], k
    assert c["crossings"] > dm.ncell


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 1023, 1025, 4099])
def test_transport_by_count_and_share(n):
    """Few particles: the stay pass's shares per thread and the chunks of the
    tracing pass; the same bits for every shape, and the oracle's cells."""
    dm = _mesh("hexahedron")
    mess = I.block_mess(dm, 20)
    ref = None
    for per in (1, 2, 4):
        for threads in (128, 256):
            start, g, _ = _transport(dm, mess, n, 7, stay_per_thread=per, move_threads=threads)
            if ref is None:
                ref = g
                o = make_oracle(dm, mess, zones=ZONES, seed=13)
                o.set_particles(*start)
                for s in (1, 2):
                    o.step(s, STAGES)
                assert np.array_equal(g[3], o.particles()[3])
            for a, b in zip(ref, g):
                assert np.array_equal(a, b)
