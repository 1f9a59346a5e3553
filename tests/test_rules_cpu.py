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


def test_near_list_radius_recovers_from_any_value(tmp_path):
    """The radius a region hands to its children is finite and positive whatever it came
    from, and generations whose lists count the planes within it (a density of planes
    per radius, up to a network's rows) come to lists of about the target."""
    L = rules(tmp_path, "float child(float T, int listed) { return child_reach(T, listed, 64); }\n"
                        "int groups(int finite) { return seed_groups(finite); }\n"
                        "float clamped(float T) { return clamp_reach(T); }")
    L.child.restype = L.clamped.restype = C.c_float
    L.child.argtypes, L.clamped.argtypes = [C.c_float, C.c_int], [C.c_float]
    inf = float("inf")
    for T in (inf, float("nan"), -1.0, 0.0, 1e-45, 1e-30, 1e-3, 1.0, 1e18, 3.4e38):
        for listed in (-1, 0, 1, 16, 64, 128, 12800):
            assert 0 < L.child(T, listed) <= 1.0001e18, (T, listed)
        assert 0 < L.clamped(T) < inf
        for rows, density in ((200, 300.0), (4096, 2e4), (12800, 1e6)):
            t = L.child(T, 64)
            for _ in range(120):  # 48 decades by 64 / 200 or by 4 a generation: 97 or 80
                t = L.child(t, min(rows, int(density * t)))
            assert 32 <= min(rows, density * t) <= 128, (T, rows, t)
    for finite in range(0, 129):
        assert L.groups(finite) == min(finite, 60)


def test_a_seeds_warp_among_more_than_2_to_the_27(tmp_path):
    L = rules(tmp_path, "long long row(unsigned b, unsigned n, unsigned t) { return warp_row(b, n, t); }")
    L.row.restype = C.c_longlong
    for row in (0, 1, 7, 8, 2**27 - 1, 2**27, 2**27 + 9, 2**31 - 2):
        for lane in (0, 31):
            assert L.row(row // 8, 256, row % 8 * 32 + lane) == row


@pytest.mark.parametrize("fp64", [0, 1])
def test_lanes_of_the_rule_between_near_equal_hits(tmp_path, fp64):
    """The lanes that a face's warps had when a block of eight warps held the rows of up to
    eight faces (a power of two) in 73 KB of shared memory."""
    L = rules(tmp_path, "int lanes(int fp64, int ALLP, int warps) { return hit_rule_lanes(fp64, ALLP, warps); }")
    for allp in range(8, 12808, 8):
        face = 32 * allp + 1120 if fp64 else 16 * allp + 1056
        faces = 1
        while 2 * faces <= 8 and 2 * faces * face <= 73 * 1024:
            faces *= 2
        assert L.lanes(fp64, allp, 0) == 32 * (8 // faces), allp
        assert L.lanes(fp64, allp, 4) == 128


def test_slots_of_the_ring_of_rows(tmp_path):
    """Never less than a wave; a given wave size bounds it whatever the network, and the
    ring then does not grow with the waves (a ring that grows loses its history)."""
    L = rules(tmp_path, "long long slots(int wave, int chunk, int units, long long row_bytes, int batch, int given) {"
                        " return ring_slots(wave, chunk, units, row_bytes, batch, given); }")
    L.slots.restype = C.c_longlong
    L.slots.argtypes = [C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_int, C.c_int]
    for units in (1, 512, 12800):
        row = 16 * ((units + 7) // 8 * 8)
        for chunk in (1, 1000, 524288):
            full = chunk + 48 * units
            for wave in {1, min(300, chunk), chunk}:
                given = L.slots(wave, chunk, units, row, 0, 1)
                assert given == max(2 * chunk, min(full, (64 << 20) // row))
                assert given * row <= max(2 * chunk * row, 64 << 20)
                assert L.slots(wave, chunk, units, row, 1, 0) == L.slots(wave, chunk, units, row, 1, 1) == 2 * wave
                assert L.slots(wave, chunk, units, row, 0, 0) == full
    assert L.slots(50000, 1000, 4096, 65536, 0, 1) == 100000
    assert L.slots(5000, 1000, 512, 8192, 0, 0) == 5000 + 48 * 512
