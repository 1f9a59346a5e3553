"""The widest layers that the tensor-core composition's shared memory takes."""
import pytest
import torch

from analyticmesh_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8160, 8192])
def test_a_wide_first_layer_marches_in_the_mixed_form(width):
    m = wl.geometric([width], 5, perturb=0.01)
    net = wl.net_arrays(m)
    x = torch.nn.functional.normalize(torch.randn(2048, 3, generator=torch.Generator().manual_seed(1)), dim=1) * 0.5
    with torch.no_grad():
        level = float(m(x).double().mean())
    st, pt = wl.seeds_for(m, init_num=16, seed=3, iso=level)
    eng = engine.Engine("mixed", net.nodes, net.arc_table, net.num_extra)
    eng.set_option(_lib.AM_OPT_CHUNK, 500)
    eng.set_option(_lib.AM_OPT_MAX_REGIONS, 2000)
    with pytest.raises(_lib.AmError) as ex:
        eng.run_net(net, st, pt, level)
    assert ex.value.status == _lib.AM_ERR_CAPACITY, str(ex.value)  # the region limit, not the widths
    assert eng.stats()["num_regions"] > 2000 and eng.error_report(500)["max_abs_f"] <= 1e-5
    eng.close()
