"""Dead units (all-zero rows, rows that are constants) in more rows than the near list
holds: the faces are the oracle's, in every form as many as without a list."""
import numpy as np
import pytest
import torch

from analyticmesh_gb300 import engine, workloads as wl
from oracle import compare, oracle

pytestmark = pytest.mark.gpu


def with_dead_units(widths, seed, share, bias):
    m = wl.geometric(widths, seed, perturb=0.02)
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for lin in m.linears[:-1]:
            dead = torch.randperm(lin.weight.shape[0], generator=g)[:int(share * lin.weight.shape[0])]
            lin.weight[dead] = 0.0
            lin.bias[dead] = bias
    return m


@pytest.mark.parametrize("bias", [0.0, -0.3, 0.3], ids=["zero", "negative", "positive"])
@pytest.mark.parametrize("widths,share", [([66, 65], 0.3), ([160, 160], 0.7), ([300], 0.8)], ids=["131", "320", "300"])
def test_faces_among_dead_units_are_the_oracles(widths, share, bias):
    m = with_dead_units(widths, 5, share, bias)
    x = torch.nn.functional.normalize(torch.randn(2048, 3, generator=torch.Generator().manual_seed(1)), dim=1) * 0.5
    with torch.no_grad():
        level = float(m(x).double().mean())
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=96, seed=3, iso=level)
    ref = oracle.run_oracle(net, st, pt, dtype="float64", iso=level)
    eng = engine.march(net, st, pt, "float64", iso=level)
    assert eng.stats()["num_faces"] > 100
    c = compare.canonical(eng.regions(), ref, tol=1e-9)
    assert c["only_a"] == 0 and c["only_b"] == 0, c
    assert c["faces_mismatch"] == 0 and c["faces_only_a"] == 0 and c["faces_only_b"] == 0, c
    total = eng.stats()["num_regions"]
    for form in ("float32", "mixed"):
        e = engine.march(net, st, pt, form, iso=level)
        assert abs(e.stats()["num_regions"] - total) <= 0.01 * total + 4, form
        e.close()
    eng.close()
