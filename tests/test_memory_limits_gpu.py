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
