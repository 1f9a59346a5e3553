"""The rules of csrc/am_rules.h over their whole ranges."""
import ctypes as C

import pytest

from rules_cpu import rules


@pytest.mark.parametrize("sms", [1, 4, 148, 152])
def test_append_shared_memory_holds_every_waves_span(tmp_path, sms):
    """Room for the span of every row count up to the largest wave's; every row is in
    one block's span."""
    L = rules(tmp_path, """
int worst(int rows_max, int sms) { // rows whose span does not fit or whose spans miss a row; 0: none
    const int grid = append_grid(rows_max, sms), room = append_span_room(rows_max, grid);
    for (int rows = 1; rows <= rows_max; ++rows) {
        const int span = append_span(rows, grid), blocks = append_blocks_used(rows, grid);
        if (span > room || blocks > grid || (long long)span * blocks < rows) return rows;
    }
    return room > kAppendSpanMax ? -1 : 0;
}""")
    for rows_max in list(range(1, 130)) + [9727, 9728, 9729, 31008, 262144, 4096 * 8 * sms + 1]:
        assert L.worst(rows_max, sms) == 0, rows_max


@pytest.mark.parametrize("kind,device,address,element,want", [
    (1, 0, 0x7000, 4, True), (1, 0, 0x7004, 4, True), (1, 0, 0x7004, 8, False), (1, 0, 0x7001, 4, False),
    (1, 0, 0x7002, 4, False), (1, 0, 0x7001, 1, True),  # (states are bytes)
    (1, 1, 0x7000, 4, False), (1, 1, 0x7000, 1, False),  # another GPU's memory
    (2, 1, 0x7000, 8, True), (2, 0, 0x7003, 4, False),  # managed: every device's
    (0, 0, 0x7000, 4, False), (0, -1, 0x7000, 1, False),  # host
])
def test_callers_memory_that_kernels_read_where_it_is(tmp_path, kind, device, address, element, want):
    L = rules(tmp_path, """
int in_place(int type, int device, uint64_t address, int element) {
    return read_in_place((MemoryType)type, device, 0, address, element);
}""")
    assert bool(L.in_place(kind, device, C.c_uint64(address), element)) is want
