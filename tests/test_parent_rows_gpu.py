"""Rows taken from the parent region (the composition starts after the layer a
region was entered through): the same regions, rows and polygons bit for bit,
whether a region finds its parent's rows or composes every layer."""
import numpy as np
import pytest

from analyticmesh_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu

NETS = {
    "plain48x3": lambda: wl.geometric([48, 48, 48], 12, perturb=0.05),
    # an identity and a transform between hidden layers, one into the output
    "skips24x4": lambda: wl.geometric([24, 24, 24, 24], 9, skips=[[0], [1, 1, 0], [1, 2, 1], [1, 3, 2]],
                                      tm_shapes=[[0, 0], [24, 24], [1, 24]]),
    "one_layer": lambda: wl.geometric([40], 5, perturb=0.02),
    "streamed260x2": lambda: wl.geometric([60, 260, 130], 6, perturb=0.02),
}


@pytest.mark.parametrize("form", ["float32", "mixed", "float64"])
@pytest.mark.parametrize("name", list(NETS))
def test_parents_rows_and_composed_rows_agree(name, form):
    """One network marched with waves of several sizes: whole levels (every
    parent's rows are there), and as a batch member with a ring of 2 x 16 and
    2 x 300 slots (most parents' rows have been overwritten, or some)."""
    m = NETS[name]()
    net = wl.net_arrays(m, *([[[0.0, 0.0, 1.0]], [-0.2]] if name == "skips24x4" else []))
    st, pt = wl.seeds_for(m, init_num=64, seed=3, w_extra=net.w_extra, b_extra=net.b_extra)
    ref = engine.march(net, st, pt, form)
    a = ref.regions()
    assert a.num > 300
    for chunk in (16, 300):
        eng = engine.Engine(form, net.nodes, net.arc_table, net.num_extra)
        eng.set_option(_lib.AM_OPT_CHUNK, chunk)
        engine.run_batch([eng], [net], [st], [pt])
        b = eng.regions()
        for x, y in ((a.bits, b.bits), (a.nverts, b.nverts), (a.status, b.status), (a.start, b.start)):
            assert np.array_equal(x, y), chunk
        used = np.arange(a.edges.shape[1])[None, :] < a.nverts[:, None]  # (slots behind the polygon are not written)
        assert np.array_equal(a.edges[used], b.edges[used]), chunk
        assert np.array_equal(a.verts[used].view(np.int64), b.verts[used].view(np.int64)), chunk
        eng.close()
    ref.close()
