// am_rules.h -- rules of sizes and of the host path as plain functions, without CUDA,
// so that they can be checked over their whole range on the CPU.
#pragma once

#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define AM_RULE __host__ __device__ inline
#else
#define AM_RULE inline
#endif

namespace am {

// ---------------------------------------------------------------- callers' memory
// May kernels on device `current` read a caller's array of `element`-byte values where
// it is?  Managed memory and memory of the same device, aligned to its elements; all
// else -- host memory, another device's memory (there need be no peer mapping), an
// odd address (a load that is not aligned faults) -- is copied to the device first.
enum MemoryType : int { kMemHost = 0, kMemDevice = 1, kMemManaged = 2 };
AM_RULE bool read_in_place(MemoryType type, int device, int current, uint64_t address, int element)
{
    return (type == kMemManaged || (type == kMemDevice && device == current)) && address % (uint64_t)element == 0;
}

// ---------------------------------------------------------------- seeds
// the row of a warp per row, in 64 bits: 2^27 rows are 2^32 threads
AM_RULE long long warp_row(unsigned block, unsigned block_threads, unsigned thread)
{
    return ((long long)block * block_threads + thread) >> 5;
}

// ---------------------------------------------------------------- ring of rows
// Slots wanted for the constraint rows of waves of up to `wave` regions (the largest:
// `chunk`) and the history in which their regions find their parents.  A parent is at
// most about one level of the breadth-first queue away, and a level held 28 to 39
// regions per hidden unit on the benchmark networks (512 .. 4,096 units): 48 a unit.
// Where memory is bounded, two waves, which reach the parents while a wave holds a
// whole level: of the largest size at once where the caller gave it (a ring that grows
// loses its history), of the present one in a batch, whose members' waves grow.  A
// given size does not keep the history from 64 MiB: waves smaller than a level would
// find no parent in two of them (3-42-10-12-92-125-246-1, mixed, 200 K regions in waves
// of 64 on GB300: composition 130 ms without it, 124 with it).
constexpr long long kRingBytes = 64ll << 20;
constexpr size_t kRingFree = size_t(256) << 20; // from here on a ring asks how much memory is free
AM_RULE long long ring_slots(int wave, int chunk, int units, long long row_bytes, bool batch, bool given)
{
    const long long most = chunk > wave ? chunk : wave, all = most + 48ll * units;
    if (batch) return 2ll * wave;
    if (!given) return all;
    const long long small = kRingBytes / row_bytes < all ? kRingBytes / row_bytes : all;
    return 2ll * most > small ? 2ll * most : small;
}

// ---------------------------------------------------------------- near list
// A near list's radius stays a finite, positive number: a region's children scale
// theirs from it, so that one that is infinite, zero or NaN would be every
// descendant's.  (1e18: its square is still finite.)
constexpr float kReachMin = 1e-30f, kReachMax = 1e18f;
AM_RULE float clamp_reach(float T)
{
    const float t = T < kReachMax ? T : kReachMax; // (NaN: the largest)
    return t > kReachMin ? t : kReachMin;
}
// the radius of a region's children, its own list having `listed` rows within T: a
// ball holds about as many planes per radius (at most four times as large)
AM_RULE float child_reach(float T, int listed, int target)
{
    const int least = target / 4;
    return clamp_reach(T * ((float)target / (float)(listed > least ? listed : least)));
}
// groups of rows, of those with a plane at a finite distance, that a seed's radius
// is to reach
AM_RULE int seed_groups(int finite) { return finite < 60 ? finite : 60; }

// ---------------------------------------------------------------- near-equal hits
// Lanes of the rule that says which of two planes hit at nearly the same place comes
// first (am_polygon.cu).  Rounding decides there, and a few regions of a marching depend
// on it, so the rule stays what it was when eight warps a block scanned faces' rows from
// 73 KB of shared memory: 32 lanes for each warp that a face of this many rows had.
// `warps` (AM_OPT_FACE_WARPS) > 0: that many instead.
AM_RULE int hit_rule_lanes(bool fp64_rows, int ALLP, int warps)
{
    if (warps > 0) return 32 * warps;
    const int one = fp64_rows ? 256 : 512, two = fp64_rows ? 544 : 1096, four = fp64_rows ? 1128 : 2264;
    return ALLP <= one ? 32 : (ALLP <= two ? 64 : (ALLP <= four ? 128 : 256));
}

// ---------------------------------------------------------------- append
constexpr int kAppendWarps = 8;    // per block; a row is a warp's
constexpr int kAppendSpanMax = 4096; // most rows per block: their winners and prefixes in shared memory

// blocks of the grid for at most rows_max rows
AM_RULE int append_grid(int rows_max, int sms)
{
    const int fill = (rows_max + kAppendWarps - 1) / kAppendWarps, most = 8 * sms;
    const int least = (rows_max + kAppendSpanMax - 1) / kAppendSpanMax;
    const int n = fill < most ? fill : most;
    return n > least ? n : least;
}
// what a wave of `rows` rows makes of it: a row per warp at least, one block at least
// (for the step), `span` rows per block
AM_RULE int append_blocks_used(int rows, int grid)
{
    const int fill = (rows + kAppendWarps - 1) / kAppendWarps;
    const int n = fill < grid ? fill : grid;
    return n > 1 ? n : 1;
}
AM_RULE int append_span(int rows, int grid)
{
    const int blocks = append_blocks_used(rows, grid);
    return (rows + blocks - 1) / blocks;
}
// the largest span of any wave of at most rows_max rows: while the grid is not full a
// span has up to kAppendWarps rows, whatever rows_max / grid is (rows_max 9: two
// blocks, five rows each, but eight rows are one block's)
AM_RULE int append_span_room(int rows_max, int grid)
{
    const int full = (rows_max + grid - 1) / grid;
    return full > kAppendWarps ? full : kAppendWarps;
}

} // namespace am
