"""The composition's algorithmic FLOPs that the bench line divides by: of the layers that
a region does not share with the region it was entered from."""
import numpy as np

import bench
from analyticmesh_gb300 import workloads as wl


def test_flops_are_counted_from_the_layer_a_region_was_entered_through():
    m = wl.geometric([6, 5, 4], 3, skips=[[0], [1, 1, 0], [1, 0, 1]], tm_shapes=[[4, 6], [1, 3]])
    net = wl.net_arrays(m)
    # linears 6 -> 5, 5 -> 4 (+ 4 x 6 from hidden layer 1), 4 -> 1 (+ 1 x 3 from the input)
    per = {1: 8 * (30 + 20 + 24 + 4 + 3), 2: 8 * (20 + 24 + 4 + 3), 3: 8 * (4 + 3)}
    for first, want in per.items():
        assert bench.composition_flops(net.nodes, net.arc_table, net.tms, first) == want
    starts = np.array([-1, 0, 5, 6, 10, 11, 14, -1], np.int32)
    assert bench.marching_flops(net, starts) == 4 * per[1] + 2 * per[2] + 2 * per[3]
