"""Calls that meet the end of the device's memory: the status, and the engine usable
afterwards.  The memory is held by plain allocations for the time of the call."""
import contextlib

import numpy as np
import pytest
import torch

from analyticmesh_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory_left(mib):
    """All of the device's memory but about `mib` MiB is taken."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        for block in (4 << 30, 256 << 20, 32 << 20, 12 << 20):  # (from 10 MiB on each is an allocation of its own)
            while torch.cuda.mem_get_info()[0] > (mib << 20) + block:
                held.append(torch.empty(block, dtype=torch.uint8, device="cuda"))
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _same(a, b):
    return a.num == b.num and np.array_equal(a.bits, b.bits) and np.array_equal(a.nverts, b.nverts)


@pytest.mark.parametrize("left", [4, 600], ids=["wave_buffers", "rows"])
@pytest.mark.parametrize("form", ["float32", "mixed"])
def test_rows_that_do_not_fit_leave_the_engine_usable(form, left):
    m = wl.sphere()
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=1024, seed=1)
    eng = engine.march(net, st, pt, form, chunk=1000)
    want = eng.regions()
    assert want.num > 200000
    with memory_left(left):
        with pytest.raises(_lib.AmError) as ex:
            eng.region_rows(0, 200000)  # 1.6 GB of rows beside 30 MB of wave buffers
        assert ex.value.status == _lib.AM_ERR_OUT_OF_MEMORY, str(ex.value)
    rows, _ = eng.region_rows(5, 40)
    assert np.isfinite(rows).all()
    eng.run_net(net, st, pt)
    assert _same(eng.regions(), want)
    eng.close()


def _held(f):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = f()
    return out, before - torch.cuda.mem_get_info()[0]


def test_a_given_wave_bounds_the_rows():
    """1,000 regions of 4,096 rows: two waves' rows are 131 MB."""
    m = wl.large_skip()
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=512, seed=3)

    def march(eng):
        try:
            eng.run_net(net, st, pt)
        except _lib.AmError as ex:
            assert ex.status == _lib.AM_ERR_CAPACITY
        return eng.stats()["num_regions"]

    eng = engine.Engine("mixed", net.nodes, net.arc_table, net.num_extra)
    eng.set_option(_lib.AM_OPT_MAX_REGIONS, 20000)
    eng.set_option(_lib.AM_OPT_CHUNK, 1000)
    n, held = _held(lambda: march(eng))
    assert n > 20000 and held < (1 << 30), held
    want = eng.regions()
    eng.set_option(_lib.AM_OPT_CHUNK, 0)
    march(eng)  # the history of the default
    got = eng.regions()
    both = min(got.num, want.num)
    assert np.array_equal(got.bits[:both], want.bits[:both])
    eng.set_option(_lib.AM_OPT_CHUNK, 1000)
    march(eng)
    rest = _held(eng.close)[1]
    assert -rest < (2 << 30), rest  # the default's rows were given back before


def test_the_rows_make_room_for_the_mesh_and_the_report():
    m = wl.sphere()
    net = wl.net_arrays(m)
    st, pt = wl.seeds_for(m, init_num=1024, seed=1)
    plain = engine.march(net, st, pt, "float32")
    mesh, rep = plain.combine(), plain.error_report(0)
    plain.close()
    for use in ("mesh", "report", "run"):
        eng = engine.march(net, st, pt, "float32")
        with memory_left(4):
            if use == "mesh":
                got = eng.combine()
                assert np.array_equal(got.verts, mesh.verts) and np.array_equal(got.face_indices, mesh.face_indices)
            elif use == "report":
                assert eng.error_report(0) == rep
            else:  # a larger wave's buffers
                eng.set_option(_lib.AM_OPT_CHUNK, 100000)
                eng.run_net(net, st, pt)
        eng.run_net(net, st, pt)
        assert eng.stats()["num_faces"] == len(mesh.face_sizes)
        eng.close()
