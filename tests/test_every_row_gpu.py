"""The walk over the rows near a face gives the faces of the walk over every row
(AM_OPT_EVERY_ROW), bit for bit in every form: the same regions in the same order, the
same polygons, the same count of FP64 walks -- near-equal hits, whose order only
rounding decides, included."""
import numpy as np
import pytest
import torch

from analyticmesh_gb300 import _lib, engine, workloads as wl
from test_dead_units_gpu import with_dead_units
from test_near_list_gpu import clustered

pytestmark = pytest.mark.gpu

BOX = ([[1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0], [0, -1, 0], [0, 0, -1]], [-0.3, -0.35, -0.4] * 2)

# name: network, level (None: the mean on the sphere of radius 1/2), box, region limit
CASES = {
    "sphere128x4": (lambda: wl.sphere(), 0.0, False, 0),
    "rows128": (lambda: wl.geometric([64, 64], 4, perturb=0.02), 0.0, False, 0),
    "rows129": (lambda: wl.geometric([64, 65], 5, perturb=0.02), 0.0, False, 0),
    "rows200_one_layer": (lambda: wl.geometric([200], 7, perturb=0.02), 0.0, False, 0),
    "box48x3": (lambda: wl.geometric([48, 48, 48], 12, perturb=0.05), 0.0, True, 0),
    "skips24x8": (lambda: wl.geometric([24] * 8, 9, skips=[[0], [1, 1, 0], [1, 0, 1]] + [[0]] * 5,
                                       tm_shapes=[[0, 0], [24, 3]]), 0.0, False, 0),
    "clustered90x2": (lambda: clustered(90, 2, 8), None, False, 0),
    "clustered240": (lambda: clustered(240, 1, 9), None, False, 0),
    "dead160x2": (lambda: with_dead_units([160, 160], 5, 0.7, 0.0), None, False, 0),
    "deep": (lambda: wl.deep(), wl.DEEP_ISO, False, 300000),
    "large_skip": (lambda: wl.large_skip(), 0.0, False, 100000),
}


def compare_walks(net, st, pt, level, form, limit):
    out, walks = [], []
    for every in (0, 1):
        eng = engine.Engine(form, net.nodes, net.arc_table, net.num_extra)
        eng.set_option(_lib.AM_OPT_EVERY_ROW, every)
        if limit:
            eng.set_option(_lib.AM_OPT_MAX_REGIONS, limit)
        try:
            eng.run_net(net, st, pt, level)
        except _lib.AmError as ex:
            assert limit and ex.status == _lib.AM_ERR_CAPACITY, str(ex)
        out.append(eng.regions())
        walks.append(eng.stats()["num_fp64_walks"])
        eng.close()
    a, b = out
    assert a.num > 500 and walks[0] == walks[1]
    for x, y in ((a.bits, b.bits), (a.nverts, b.nverts), (a.status, b.status), (a.start, b.start)):
        assert np.array_equal(x, y)
    used = np.arange(a.edges.shape[1])[None, :] < a.nverts[:, None]
    assert np.array_equal(a.edges[used], b.edges[used])
    assert np.array_equal(a.verts[used].view(np.int64), b.verts[used].view(np.int64))


@pytest.mark.parametrize("form", ["float32", "mixed", "float64"])
@pytest.mark.parametrize("name", list(CASES))
def test_faces_of_the_list_and_of_every_row_are_equal(name, form):
    factory, level, boxed, limit = CASES[name]
    if form == "float64" and name in ("deep", "large_skip"):
        limit //= 4
    m = factory()
    if level is None:
        x = torch.nn.functional.normalize(torch.randn(2048, 3, generator=torch.Generator().manual_seed(1)), dim=1) * 0.5
        with torch.no_grad():
            level = float(m(x).double().mean())
    box = BOX if boxed else (None, None)
    net = wl.net_arrays(m, *box)
    st, pt = wl.seeds_for(m, init_num=96, seed=3, iso=level, w_extra=box[0], b_extra=box[1])
    compare_walks(net, st, pt, level, form, limit)


@pytest.mark.parametrize("form", ["float32", "mixed", "float64"])
@pytest.mark.parametrize("scale,shift", [(1e-2, 0), (1e-3, 0), (1e-4, 0), (1e3, 0), (1.0, 20.0), (1e-2, 0.3)])
@pytest.mark.parametrize("name", ["sphere128x4", "deep"])
def test_faces_of_small_large_and_distant_shapes(name, scale, shift, form):
    """The shape scaled, and moved by `shift` along a diagonal: the list's margin goes with
    the coordinates' size."""
    factory, level, _, _ = CASES[name]
    m = factory()
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=96, seed=3, iso=level)
    t = shift * np.array([0.6, -0.3, 0.7])
    net.W[0] = net.W[0] / scale
    net.b[0] = net.b[0] - net.W[0] @ t
    compare_walks(net, st, pt * scale + t, level, form, 60000)
