"""The append while other work holds the SMs: its blocks then start late, some
after the block that finishes the wave has moved the queue on.  Every network of a
batch of small ones beside wide ones gives the regions it gives alone, in the same
order, on every repeat and on engines that are used again."""
import numpy as np
import pytest

from analyticmesh_gb300 import engine, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["mixed", "float32"])
def test_small_networks_beside_wide_ones_repeat_their_own_regions(form):
    models = [wl.geometric([24 + 8 * (i % 5)] * (2 + i % 3), 200 + i, perturb=0.01) for i in range(10)]
    models[3:3] = [wl.sphere()]
    models.append(wl.geometric([128] * 4, 222, perturb=0.01))
    nets = [wl.net_arrays(m) for m in models]
    seeds = [wl.seeds_for(m, init_num=64, seed=30 + i) for i, m in enumerate(models)]
    alone = []
    for net, (st, pt) in zip(nets, seeds):
        e = engine.march(net, st, pt, form)
        alone.append(e.regions())
        e.close()
    assert all(r.num > 50 for r in alone)
    engines = [engine.Engine(form, n.nodes, n.arc_table, n.num_extra) for n in nets]
    for repeat in range(4):
        engine.run_batch(engines, nets, [s[0] for s in seeds], [s[1] for s in seeds])
        for i, (e, want) in enumerate(zip(engines, alone)):
            got = e.regions()
            assert got.num == want.num, (repeat, i)
            for x, y in ((got.bits, want.bits), (got.start, want.start), (got.nverts, want.nverts)):
                assert np.array_equal(x, y), (repeat, i)
    for e in engines:
        e.close()


@pytest.mark.parametrize("chunk", [9, 17, 48])
def test_waves_shorter_than_a_small_largest_wave(chunk):
    """Graph-driven waves of every length up to a largest wave of a few rows."""
    m = wl.geometric([40, 40], 7, perturb=0.02)
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=400, seed=3)
    out = []
    for c in (None, chunk):
        e = engine.march(net, st[:8], pt[:8], "float64", chunk=c)
        out.append(e.regions())
        e.close()
    a, b = out
    assert a.num > 200
    for x, y in ((a.bits, b.bits), (a.start, b.start), (a.nverts, b.nverts)):
        assert np.array_equal(x, y)
