"""What the kernels' sources may name.  The same library serves one GPU and every rank
of a run on several, where a bulk load into several CTAs' shared memory is closed."""
import glob
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_kernel_loads_into_several_ctas_shared_memory():
    files = [p for e in ("*.cu", "*.cuh", "*.h", "*.cpp") for p in glob.glob(os.path.join(ROOT, "analyticmesh_gb300", "csrc", e))]
    assert len(files) > 10
    for p in files:
        text = open(p).read()
        assert "multicast" not in text and "__cluster_dims__" not in text, p
