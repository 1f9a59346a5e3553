"""Arguments where a caller may have them: on the host, on the device, and on the device
at addresses that are not aligned to their elements.  The same regions and vertices."""
import ctypes as C

import numpy as np
import pytest
import torch

from analyticmesh_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu


def _at(array, dtype, off):
    """(keep-alive, address) of a device copy of `array`, `off` bytes past a 256-byte boundary."""
    raw = torch.from_numpy(np.ascontiguousarray(array, dtype).reshape(-1).view(np.uint8).copy())
    buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
    buf[off:off + raw.numel()] = raw.cuda()
    assert buf.data_ptr() % 256 == 0
    return buf, buf.data_ptr() + off


@pytest.mark.parametrize("form", ["float32", "mixed", "float64"])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_device_arguments_at_any_address(form, off):
    m = wl.geometric([24, 24, 24], 9, skips=[[0], [1, 0, 0], [0]], tm_shapes=[[24, 3]])
    net = wl.net_arrays(m, [[0.0, 0.0, 1.0]], [-0.2])
    st, pt = wl.seeds_for(m, init_num=64, seed=3, w_extra=net.w_extra, b_extra=net.b_extra)
    want = engine.march(net, st, pt, form)
    a = want.regions()
    assert a.num > 100
    dt = np.float64 if form == "float64" else np.float32
    keep = []

    def ptr(x, dtype=dt):
        buf, p = _at(x, dtype, off)
        keep.append(buf)
        return p

    eng = engine.Engine(form, net.nodes, net.arc_table, net.num_extra)
    n = len(net.W)
    shapes = np.ascontiguousarray([s for t in net.tms for s in t.shape] or [0], np.int32)
    args = [(C.c_void_p * n)(*[ptr(w) for w in net.W]), (C.c_void_p * n)(*[ptr(b) for b in net.b]), ptr(st, np.uint8),
            ptr(pt), st.shape[0], (C.c_void_p * len(net.tms))(*[ptr(t) for t in net.tms]),
            shapes.ctypes.data_as(C.POINTER(C.c_int32)), len(net.tms), ptr(net.w_extra), ptr(net.b_extra)]
    torch.cuda.synchronize()  # (the copies above; the engine has a stream of its own)
    rc = _lib.lib().am_analytic_marching(eng.h, *args, 0.0, 0, None)
    _lib.check(rc, eng.h)
    b = eng.regions()
    for x, y in ((a.bits, b.bits), (a.nverts, b.nverts), (a.start, b.start)):
        assert np.array_equal(x, y)
    used = np.arange(a.edges.shape[1])[None, :] < a.nverts[:, None]
    assert np.array_equal(a.verts[used].view(np.int64), b.verts[used].view(np.int64))
    eng.close()
    want.close()
