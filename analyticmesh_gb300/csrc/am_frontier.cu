// am_frontier.cu -- region hash set and the append-only region store.
//
// The reference keeps visited regions as 32-bit FNV-1 fingerprints in an
// open-addressing table and accepts a region as new when its fingerprint is
// absent (backend/inc/hash.h:33-67) -- two different regions with the same
// fingerprint silently lose one.  This store keeps every region's full
// packed key; a table slot holds (fingerprint, id) and a fingerprint match
// is confirmed by comparing the keys.
//
// New regions are appended in candidate order (append_kernel), so the region
// ids of a run do not depend on thread scheduling.
#include <algorithm>
#include <cuda/atomic>
#include <cuda_runtime.h>

#include "am_device.cuh"
#include "am_internal.h"
#include "am_rules.h"

namespace am {

namespace {

__device__ __forceinline__ unsigned long long load_slot(const unsigned long long *p)
{
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> a(*const_cast<unsigned long long *>(p));
    return a.load(cuda::memory_order_relaxed);
}

// a warp per state: a word is one coalesced 32-byte read and a ballot (a thread
// per state read bytes N apart from its neighbours')
__global__ void seed_pack_kernel(const uint8_t *states, int S, int N, int W, uint32_t *keys, uint64_t *hash, int *zeroed,
                                 SeedPoints pt)
{
    if (zeroed && blockIdx.x == 0 && threadIdx.x == 0) *zeroed = 0;
    const int lane = threadIdx.x & 31;
    const long long s = warp_row(blockIdx.x, blockDim.x, threadIdx.x);
    if (s >= S) return;
    if (pt.dst && lane < 3) { // (FP32 to FP64 is exact)
        const size_t q = (size_t)s * 3 + lane;
        const double v = pt.pbytes == 8 ? ((const double *)pt.src)[q] : (double)((const float *)pt.src)[q];
        if (pt.tbytes == 8) ((double *)pt.dst)[q] = v;
        else ((float *)pt.dst)[q] = (float)v;
    }
    const uint8_t *row = states + (size_t)s * N;
    uint64_t h = 0;
    for (int w0 = 0; w0 < W; w0 += 32) {
        uint32_t mine = 0;
#pragma unroll 8
        for (int u = 0; u < 32; ++u) {
            if (w0 + u >= W) break;
            const int q = 32 * (w0 + u) + lane;
            const uint32_t word = __ballot_sync(0xffffffffu, q < N && row[q] != 0);
            if (lane == u) mine = word;
        }
        if (w0 + lane < W) {
            keys[(size_t)s * W + w0 + lane] = mine;
            h += word_term(mine, w0 + lane);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    if (lane == 0) hash[s] = h;
}

__global__ void seed_insert_kernel(const uint32_t *keys, const uint64_t *hash, int S, int W, HashDev hs, int32_t *rec,
                                   int *err)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const uint64_t h = hash[s];
    const uint32_t fp = fp_of(h);
    const unsigned long long mine = slot_value(fp, 1, (uint32_t)s);
    const uint32_t *key = keys + (size_t)s * W;
    unsigned long long slot = h & hs.mask;
    int r = -1, probe = 0;
    for (; probe < kMaxProbes; ++probe) {
        unsigned long long cur = load_slot(hs.slots + slot);
        if (cur == kEmpty) {
            const unsigned long long old = atomicCAS(hs.slots + slot, kEmpty, mine);
            if (old == kEmpty) {
                r = (int)slot;
                break;
            }
            cur = old;
        }
        if ((uint32_t)(cur >> 32) == fp) {
            const uint32_t *other = keys + (size_t)((uint32_t)cur & 0x7fffffffu) * W;
            bool eq = true;
            for (int w = 0; w < W && eq; ++w) eq = (other[w] == key[w]);
            if (eq) {
                atomicMin(hs.slots + slot, mine);
                r = (int)slot;
                break;
            }
        }
        slot = (slot + (unsigned long long)probe + 1ull) & hs.mask;
    }
    if (probe == kMaxProbes) atomicOr(err, kErrTableFull);
    rec[s] = r;
}

constexpr int kAppendThreads = 32 * kAppendWarps;
constexpr int kSpinIters = 1 << 24; // bound of the wait for an earlier block's count

struct AppendArgs {
    int mode;              // 0 children of a chunk, 1 seeds
    NetDev net;
    RegionsDev reg;
    ChunkDev ch;
    HashDev hs;
    const uint32_t *seed_keys;
    const uint64_t *seed_hash;
    const void *seed_points; // [S][3] TS
    int n_items;           // seeds
    long long *tail;
    AppendScratch *sc;
    int *err;
};

// An append's rows are 32 candidates each: the edge slots of one region of the
// wave, or 32 seeds.  Is this lane's candidate of row r the one in its slot?
__device__ __forceinline__ bool is_winner(const AppendArgs &a, int r, int lane, long long head)
{
    const int q = r * 32 + lane;
    if (a.mode == 1 && q >= a.n_items) return false;
    const int rec = a.ch.rec[q];
    if (rec < 0) return false;
    const uint32_t myid = a.mode == 1 ? (uint32_t)q
                                      : (uint32_t)((long long)r * a.net.ALL + a.reg.edges[(size_t)(head + r) * kVMax + lane]);
    return (uint32_t)load_slot(a.hs.slots + rec) == ((1u << 31) | (myid & 0x7fffffffu));
}

// (the whole warp) the winners `won` of row r become the regions from rid0 on.  A
// lane each for their records, so that a row costs one chain of loads whatever
// its winners; the keys' words by the warp.  (Measured on GB300, frontier phase:
// with the winners one after the other 0.90 ms for 3-[128]x4-1 and 12.8 for
// 3-[512]x8-1, this way 0.79 and 11.7.)
template <typename TS>
__device__ __forceinline__ void append_row(const AppendArgs &a, int r, uint32_t won, long long rid0, long long head, int lane)
{
    const int W = a.net.W;
    const long long rid = rid0 + __popc(won & ((1u << lane) - 1u));
    bool mine = (won >> lane) & 1u;
    if (mine && rid >= a.reg.cap) {
        atomicOr(a.err, kErrCapacity);
        mine = false;
    }
    const uint32_t writes = __ballot_sync(0xffffffffu, mine);
    const long long parent = head + r; // (children)
    const int q = r * 32 + lane;       // the candidate: edge slot or seed
    int k = -1;
    TS m[3] = {TS(0), TS(0), TS(0)};
    uint64_t h = 0;
    if (a.mode == 1) {
        if (mine) {
            h = a.seed_hash[q];
            const TS *pt = (const TS *)a.seed_points + (size_t)q * 3;
#pragma unroll
            for (int c = 0; c < 3; ++c) m[c] = pt[c];
        }
    } else {
        const int n = a.reg.nv[parent]; // (a winner is one of the polygon's edges)
        const uint64_t ph = a.reg.hash[parent];
        TS v[3] = {TS(0), TS(0), TS(0)};
        if (lane < n) {
            k = a.reg.edges[(size_t)parent * kVMax + lane];
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] = ((const TS *)a.reg.verts)[((size_t)parent * kVMax + lane) * 3 + c];
        }
        const int after = lane + 1 < n ? lane + 1 : 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TS w = __shfl_sync(0xffffffffu, v[c], after);
            m[c] = (v[c] + w) / TS(2);
        }
        if (mine) h = flip_hash(ph, a.reg.keys[(size_t)parent * W + (k >> 5)], k);
    }
    if (mine) {
        TS *mid = (TS *)a.reg.mid + (size_t)rid * 4;
#pragma unroll
        for (int c = 0; c < 3; ++c) mid[c] = m[c];
        mid[3] = TS(0);
        a.reg.start[rid] = k;
        a.reg.parent[rid] = a.mode == 1 ? -1 : (int32_t)parent;
        a.reg.hash[rid] = h;
        a.reg.nv[rid] = 0;
        a.reg.status[rid] = 0;
        a.hs.slots[a.ch.rec[q]] = slot_value(fp_of(h), 0, (uint32_t)rid);
    }
    for (int w0 = 0; w0 < W; w0 += 32) {
        const int w = w0 + lane;
        const uint32_t p = a.mode != 1 && w < W ? a.reg.keys[(size_t)parent * W + w] : 0u;
        for (uint32_t b = writes; b; b &= b - 1u) {
            const int i = __ffs(b) - 1;
            const int ki = __shfl_sync(0xffffffffu, k, i);
            const long long to = __shfl_sync(0xffffffffu, rid, i);
            if (w >= W) continue;
            const uint32_t word = a.mode == 1 ? a.seed_keys[(size_t)(r * 32 + i) * W + w] : p ^ (w == (ki >> 5) ? 1u << (ki & 31) : 0u);
            a.reg.keys[(size_t)to * W + w] = word;
        }
    }
}

// graph-driven loop: retire the wave, take the next one from the queue and
// go on while it is non-empty, no error bit is set, its children fit and the
// queue has not outgrown the wave buffers of a batch member
__device__ void wave_step(WaveCtl &c, cudaGraphConditionalHandle cond)
{
    if (c.count > 0) c.waves++;
    c.head += c.count;
    const long long rem = c.tail - c.head;
    c.count = (int)(rem < (long long)c.chunk_cap ? (rem > 0 ? rem : 0) : (long long)c.chunk_cap);
    c.work = 0u;
    for (int i = 0; i < kMaxLayers; ++i) c.ccount[i] = 0;
    const int err = *(volatile int *)&c.err;
    const bool go = c.count > 0 && err == 0 &&
                    c.tail + (long long)c.count * kVMax <= c.limit && c.waves < c.max_waves &&
                    c.tail <= c.stop_tail && rem <= (long long)c.grow_at;
    cudaGraphSetConditional(cond, go ? 1u : 0u);
}

// Appends the winners of all rows at the tail, in candidate order, in one pass:
// a block takes the next span of rows (a ticket: a block waits for earlier
// tickets only, which have started), counts its winners, publishes the count,
// adds up the counts before it, and writes.  (A winner's slot becomes a
// region's while later blocks still count; a candidate that reads it then is not
// the winner either way.)  The last block to finish moves the tail and, in the
// graph-driven loop, the queue.  The counts carry the append's number, so that
// nothing has to be cleared between appends.  Measured on GB300 against a count
// kernel, a write kernel (a thread per winner) and a step kernel, frontier phase:
// 3-[512]x8-1 17.4 -> 11.7 ms, 3-[256]x6-1 2.5 -> 2.1 ms; with a quarter of the
// blocks (a warp then walks several rows one after the other) 19.5 and 3.1 ms.
template <typename TS>
__global__ void __launch_bounds__(kAppendThreads) append_kernel(AppendArgs a, cudaGraphConditionalHandle cond, int step)
{
    extern __shared__ uint32_t sh[]; // the span's winners, then their prefix
    __shared__ int s_ticket;
    __shared__ int s_part[kAppendWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    long long head = 0;
    int rows;
    if (a.mode == 1) {
        rows = (a.n_items + 31) / 32;
    } else if (a.ch.ctl) { // (not head and count: wave_step moves them while blocks are still to come)
        head = a.ch.ctl->append_head;
        rows = a.ch.ctl->append_count;
    } else {
        head = a.ch.head;
        rows = a.ch.count;
    }
    const int blocks = append_blocks_used(rows, (int)gridDim.x);
    if ((int)blockIdx.x >= blocks) return;
    const int span = append_span(rows, (int)gridDim.x);
    if (tid == 0) s_ticket = (int)atomicAdd(&a.sc->ticket, 1u);
    __syncthreads();
    const int ticket = s_ticket;
    const uint32_t epoch = a.sc->epoch + 1u;
    const long long tail = *a.tail; // (moved by the last block only)
    const int r0 = min(rows, ticket * span), n = min(rows - r0, span);
    uint32_t *won = sh, *pre = sh + span;
#pragma unroll 4
    for (int r = warp; r < n; r += kAppendWarps) {
        const uint32_t b = __ballot_sync(0xffffffffu, is_winner(a, r0 + r, lane, head));
        if (lane == 0) won[r] = b;
    }
    __syncthreads();
    // exclusive prefix over the span's rows
    int total = 0;
    for (int q = 0; q < n; q += kAppendThreads) {
        const int v = q + tid < n ? __popc(won[q + tid]) : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_part[warp] = x;
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kAppendWarps; ++w) {
            if (w < warp) before += s_part[w];
            all += s_part[w];
        }
        if (q + tid < n) pre[q + tid] = (uint32_t)(total + before + x - v);
        total += all;
        __syncthreads();
    }
    // publish, and the counts of the earlier tickets
    volatile unsigned long long *entry = a.sc->entry;
    if (tid == 0) entry[ticket] = ((unsigned long long)epoch << 32) | (uint32_t)total;
    int sum = 0;
    for (int t = tid; t < ticket; t += kAppendThreads) {
        unsigned long long e = entry[t];
        for (int i = 0; (uint32_t)(e >> 32) != epoch; e = entry[t])
            if (++i >= kSpinIters) {
                atomicOr(a.err, kErrWait);
                break;
            }
        sum += (int)(uint32_t)e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) s_part[warp] = sum;
    __syncthreads();
    long long base = tail;
#pragma unroll
    for (int w = 0; w < kAppendWarps; ++w) base += s_part[w];
    for (int r = warp; r < n; r += kAppendWarps) {
        const uint32_t b = won[r];
        if (b) append_row<TS>(a, r0 + r, b, base + (long long)pre[r], head, lane);
    }
    if (tid == 0) {
        if (ticket == blocks - 1) a.sc->new_tail = base + total;
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&a.sc->done, 1u) == (unsigned)blocks - 1u) {
            __threadfence();
            *a.tail = *(volatile long long *)&a.sc->new_tail;
            a.sc->ticket = 0u;
            a.sc->done = 0u;
            a.sc->epoch = epoch;
            if (step) wave_step(*a.ch.ctl, cond);
        }
    }
}

// Class of every region of the wave (ChunkDev): class j's list gets the wave
// position, split[position] the number of leading rows that come from the
// parent's slot (0 for class 1, whose layer-1 rows are the network's own).
// The order within a class does not matter: a region's rows do not depend on
// the tile it is composed in.
__global__ void wave_classes_kernel(NetDev net, RegionsDev reg, ChunkDev ch)
{
    long long head;
    int count;
    chunk_range(ch, head, count);
    const long long rows_from = ch.ctl ? *(volatile const long long *)&ch.ctl->rows_from : ch.rows_from;
    // a slot that this wave writes holds no parent any more
    const long long oldest = max(rows_from, head + count - (long long)ch.ring);
    const int lane = threadIdx.x & 31;
    const int layers = net.n_lin - 1;
    for (int r0 = (int)(blockIdx.x * blockDim.x + threadIdx.x) - lane; r0 < count; r0 += (int)(gridDim.x * blockDim.x)) {
        const int rl = r0 + lane;
        int c = 0;
        if (rl < count) {
            const int par = reg.parent[head + rl], k = reg.start[head + rl];
            c = 1;
            if (par >= oldest && par >= 0 && k >= 0)
                while (c < layers && k >= net.hoff[c + 1]) ++c;
            ch.split[rl] = c > 1 ? net.hoff[c + 1] : 0;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, c);
        const int first = __ffs(peers) - 1;
        int base = 0;
        if (c > 0 && lane == first) base = atomicAdd(ch.ccount + c - 1, __popc(peers));
        base = __shfl_sync(0xffffffffu, base, first);
        if (c > 0) ch.order[(size_t)(c - 1) * ch.order_cap + base + __popc(peers & ((1u << lane) - 1u))] = rl;
    }
}

// run statistics: faces (>= 3 vertices), the largest polygon, and one count
// per failure status
__global__ void region_stats_kernel(const int32_t *nv, const int8_t *status, long long n, unsigned long long *out)
{
    __shared__ unsigned int s[kStatsCount];
    if (threadIdx.x < kStatsCount) s[threadIdx.x] = 0u;
    __syncthreads();
    unsigned int faces = 0, vmax = 0, verts = 0, bad[4] = {0u, 0u, 0u, 0u};
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
        const int v = nv[r];
        faces += v >= 3 ? 1u : 0u;
        vmax = max(vmax, (unsigned int)max(v, 0));
        verts += (unsigned int)min(max(v, 0), kVMax);
        const int st = status[r];
        if (st >= kNoStart && st <= kSingular) bad[st - kNoStart]++;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        faces += __shfl_xor_sync(0xffffffffu, faces, o);
        vmax = max(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        verts += __shfl_xor_sync(0xffffffffu, verts, o);
#pragma unroll
        for (int b = 0; b < 4; ++b) bad[b] += __shfl_xor_sync(0xffffffffu, bad[b], o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s[0], faces);
        atomicMax(&s[1], vmax);
        for (int b = 0; b < 4; ++b) atomicAdd(&s[2 + b], bad[b]);
        atomicAdd(&s[6], verts);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(out, (unsigned long long)s[0]);
        atomicMax(out + 1, (unsigned long long)s[1]);
        for (int b = 0; b < 5; ++b) atomicAdd(out + 2 + b, (unsigned long long)s[2 + b]);
    }
}

__global__ void rehash_kernel(RegionsDev reg, long long n, HashDev hs, int *err)
{
    const long long rid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (rid >= n) return;
    const uint64_t h = reg.hash[rid];
    const unsigned long long v = slot_value(fp_of(h), 0, (uint32_t)rid);
    unsigned long long slot = h & hs.mask;
    for (int probe = 0; probe < kMaxProbes; ++probe) {
        if (atomicCAS(hs.slots + slot, kEmpty, v) == kEmpty) return;
        slot = (slot + (unsigned long long)probe + 1ull) & hs.mask;
    }
    atomicOr(err, kErrTableFull);
}

} // namespace

void launch_seed_pack(const uint8_t *states, int S, int N, int W, uint32_t *keys, uint64_t *hash, cudaStream_t st,
                      int *zeroed, const SeedPoints &points)
{
    if (S <= 0) return;
    seed_pack_kernel<<<((unsigned)S + 7u) / 8u, 256, 0, st>>>(states, S, N, W, keys, hash, zeroed, points);
}

void launch_seed_insert(const uint32_t *keys, const uint64_t *hash, int S, int W, const HashDev &hs, int32_t *rec,
                        int *d_err, cudaStream_t st)
{
    if (S <= 0) return;
    seed_insert_kernel<<<(S + 127) / 128, 128, 0, st>>>(keys, hash, S, W, hs, rec, d_err);
}

int append_blocks(int rows_max) { return append_grid(rows_max, device_sms()); }

void launch_append(int mode, int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch,
                   const HashDev &hs, const uint32_t *seed_keys, const uint64_t *seed_hash, const void *seed_points,
                   int n_items, long long *d_tail, AppendScratch *sc, int blocks_cap, int *d_err, cudaStream_t st,
                   const cudaGraphConditionalHandle *cond)
{
    const int rows = mode == 1 ? (n_items + 31) / 32 : ch.count; // graph-driven loop: the largest wave
    if (rows <= 0) return;
    AppendArgs a;
    a.mode = mode;
    a.net = net;
    a.reg = reg;
    a.ch = ch;
    a.hs = hs;
    a.seed_keys = seed_keys;
    a.seed_hash = seed_hash;
    a.seed_points = seed_points;
    a.n_items = n_items;
    a.tail = d_tail;
    a.sc = sc;
    a.err = d_err;
    const int nb = append_blocks(rows);
    if (nb > blocks_cap) { // the host sizes the scratch for the largest wave
        int e = kErrCapacity;
        cudaMemcpyAsync(d_err, &e, sizeof(int), cudaMemcpyHostToDevice, st);
        return;
    }
    const size_t smem = sizeof(uint32_t) * 2 * (size_t)append_span_room(rows, nb);
    const cudaGraphConditionalHandle h = cond ? *cond : cudaGraphConditionalHandle{};
    if (prec == kFloat32)
        append_kernel<float><<<nb, kAppendThreads, smem, st>>>(a, h, cond ? 1 : 0);
    else
        append_kernel<double><<<nb, kAppendThreads, smem, st>>>(a, h, cond ? 1 : 0);
}

void launch_wave_classes(const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, cudaStream_t st)
{
    const int grid = std::min((ch.count + 255) / 256, 2 * device_sms());
    if (grid > 0) wave_classes_kernel<<<grid, 256, 0, st>>>(net, reg, ch);
}

void launch_region_stats(const int32_t *nv, const int8_t *status, long long n, unsigned long long *out,
                         cudaStream_t st)
{
    if (n <= 0) return;
    const int grid = (int)std::min<long long>((n + 255) / 256, 4ll * device_sms());
    region_stats_kernel<<<grid, 256, 0, st>>>(nv, status, n, out);
}

void launch_rehash(const RegionsDev &reg, long long n, const HashDev &hs, int *d_err, cudaStream_t st)
{
    if (n <= 0) return;
    rehash_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(reg, n, hs, d_err);
}

} // namespace am
