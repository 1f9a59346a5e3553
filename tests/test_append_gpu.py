"""The one-pass append: the regions and their order do not depend on how many
rows a wave has (one to many per block, the last block partly filled), nor on
the number of seeds in the last warp."""
import numpy as np
import pytest

from analyticmesh_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seeds", [1, 31, 32, 33, 257])
def test_regions_and_order_with_any_number_of_seeds(seeds):
    m = wl.geometric([40, 40], 7, perturb=0.02)
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=400, seed=3)
    st, pt = st[:seeds], pt[:seeds]
    out = []
    for chunk in (0, 1, 33):
        eng = engine.march(net, st, pt, "float64", options={_lib.AM_OPT_CHUNK: chunk} if chunk else {})
        out.append(eng.regions())
        eng.close()
    a = out[0]
    assert a.num > 200
    for b in out[1:]:
        for x, y in ((a.bits, b.bits), (a.start, b.start), (a.nverts, b.nverts)):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("chunk", [9728, 9729, 30000])
def test_waves_of_more_rows_than_warps(chunk):
    """9,728 rows fill the grid of 152 SMs with one row per warp."""
    m = wl.sphere()
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=1024, seed=7)
    out = []
    for c in (4000, chunk):
        eng = engine.march(net, st, pt, "float32", options={_lib.AM_OPT_CHUNK: c})
        out.append(eng.regions())
        eng.close()
    a, b = out
    assert a.num > 200000
    for x, y in ((a.bits, b.bits), (a.start, b.start), (a.nverts, b.nverts)):
        assert np.array_equal(x, y)
