"""The walk over the planes near a face (at most 128 rows of a region) against the
oracle's walk over every row: row counts around 128, where the list starts to
leave rows out, and planes so unevenly spread that the radius taken from the
parent is far too small or too large (repeats, and faces walked over every row)."""
import numpy as np
import pytest
import torch

from analyticmesh_gb300 import engine, workloads as wl
from oracle import compare, oracle

pytestmark = pytest.mark.gpu


def clustered(width, depth, seed):
    """Two thirds of the first layer's planes pass within 1e-2 of one point near
    the surface, the others are spread as usual."""
    m = wl.geometric([width] * depth, seed, perturb=0.02)
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        w, b = m.linears[0].weight, m.linears[0].bias
        n = 2 * width // 3
        at = torch.tensor([0.45, 0.1, -0.05])
        b[:n] = -(w[:n] @ at) + 1e-2 * w[:n].norm(dim=1) * torch.randn(n, generator=g)
    return m


NETS = {
    "rows127": (lambda: wl.geometric([42, 42, 43], 3, perturb=0.02), 0),
    "rows128": (lambda: wl.geometric([64, 64], 4, perturb=0.02), 0),
    "rows129": (lambda: wl.geometric([64, 65], 5, perturb=0.02), 0),
    "rows126+6": (lambda: wl.geometric([63, 63], 6, perturb=0.02), 6),
    "rows200_one_layer": (lambda: wl.geometric([200], 7, perturb=0.02), 0),
    "clustered90x2": (lambda: clustered(90, 2, 8), 0),
    "clustered240": (lambda: clustered(240, 1, 9), 0),
}


@pytest.mark.parametrize("name", list(NETS))
def test_faces_from_the_near_list_are_the_oracles(name):
    factory, extra = NETS[name]
    m = factory()
    box = ([[1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0], [0, -1, 0], [0, 0, -1]], [-0.6] * 6) if extra else (None, None)
    level = 0.0
    if name.startswith("clustered"):  # a closed level of the moved planes' network
        x = torch.nn.functional.normalize(torch.randn(2048, 3, generator=torch.Generator().manual_seed(1)), dim=1) * 0.5
        with torch.no_grad():
            level = float(m(x).double().mean())
    net = wl.net_arrays(m, *box)
    st, pt = wl.seeds_for(m, init_num=96, seed=3, iso=level, w_extra=box[0], b_extra=box[1])
    ref = oracle.run_oracle(net, st, pt, dtype="float64", iso=level)
    eng = engine.march(net, st, pt, "float64", iso=level)
    c = compare.canonical(eng.regions(), ref, tol=1e-9)
    assert c["only_a"] == 0 and c["only_b"] == 0, c
    assert c["faces_mismatch"] == 0 and c["faces_only_a"] == 0 and c["faces_only_b"] == 0, c
    # the other forms visit the float64 form's regions up to slivers, and their
    # vertices lie on the surface: the forms' own bound on |f(v)|
    total = eng.stats()["num_regions"]
    for form in ("float32", "mixed"):
        e = engine.march(net, st, pt, form, iso=level)
        assert abs(e.stats()["num_regions"] - total) <= 0.01 * total + 4, form
        if form == "mixed":
            assert e.error_report(0)["max_abs_f"] <= 1e-5
        e.close()
    eng.close()


@pytest.mark.parametrize("widths", [[29], [30], [61], [62], [31, 62], [62, 63]], ids=lambda w: "rows%d" % (sum(w) + 3))
def test_seeds_whose_nearest_pairs_are_shut_out(widths):
    """A box corner inside the surface: at its seeds most pairs of near planes meet
    outside it, so the start search goes on for many pairs.  Row counts around
    those of a lane's rows (32, 64, 128), against the oracle's search."""
    m = wl.geometric(widths, 11, perturb=0.05)
    corner = ([[1, 0, 0], [0, 1, 0], [0, 0, 1]], [-0.05, 0.02, -0.1])
    net = wl.net_arrays(m, *corner)
    st, pt = wl.seeds_for(m, init_num=200, seed=5, w_extra=corner[0], b_extra=corner[1])
    ref = oracle.run_oracle(net, st, pt, dtype="float64")
    eng = engine.march(net, st, pt, "float64")
    c = compare.canonical(eng.regions(), ref, tol=1e-9)
    assert c["only_a"] == 0 and c["only_b"] == 0, c
    assert c["faces_mismatch"] == 0 and c["faces_only_a"] == 0 and c["faces_only_b"] == 0, c
    eng.close()
