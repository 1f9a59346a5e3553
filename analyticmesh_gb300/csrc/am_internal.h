// am_internal.h -- shared types of the GB300 Analytic Marching engine
// (host driver <-> kernels).  Not part of the C ABI.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace am {

constexpr int kMaxLayers = 24;   // linear layers
constexpr int kMaxSkips = 4;     // additive connections into one layer
constexpr int kVMax = 32;        // polygon capacity (vertices / edges per face)
constexpr int kWalkSteps = 96;   // bound on walk iterations (vertices + merges)
constexpr int kTopK = 64;        // seed start search: pairs x <= 812 use the 57 nearest planes
constexpr int kMaxProbes = 4096; // hash probe bound
constexpr uint64_t kEmpty = ~0ull;
constexpr int kMaxWaves = 1 << 20; // bound on the waves of one graph launch

enum Precision : int { kFloat32 = 0, kFloat64 = 1, kMixed = 2 };

// Region status codes (poly_status)
enum : int8_t { kOk = 0, kNoStart = 1, kOpen = 2, kTruncated = 3, kSingular = 4 };

// Device error bits.  kErrWait: a bounded wait inside a kernel (a
// tensor-core pipeline barrier) ran out; the kernel stopped issuing work and
// returned, and its results are not valid.  kErrNonFinite: a weight, bias,
// transform or extra constraint is NaN or infinite.
enum : int { kErrTableFull = 1, kErrWait = 2, kErrCapacity = 4, kErrNonFinite = 8 };

struct SkipDev {
    int from;        // 0 = network input, h >= 1 = hidden layer h
    int kind;        // 0 identity, 1 transform
    const void *tmt; // transform, transposed and padded: [dec][Mp]
    int Mp;
};

// A network resident on the device in the layouts the kernels read.
struct NetDev {
    int n_lin;                    // linear layers
    int N, E, ALL, ALLP, W;       // hidden units, extra rows, N+E, padded, key words
    int nodes[kMaxLayers + 1];
    int hoff[kMaxLayers + 1];     // first constraint row of hidden layer h (h >= 1)
    const void *Wt[kMaxLayers];   // linear i transposed and padded: [nodes[i]][Mp[i]]
    int Mp[kMaxLayers];
    const void *bias[kMaxLayers]; // [nodes[i+1]]
    const void *W0;               // linear 0 as given: [nodes[1]][3]
    int nskip[kMaxLayers];        // connections into linear i
    SkipDev skip[kMaxLayers][kMaxSkips];
    const void *w_extra;          // [E][3]
    const void *b_extra;          // [E]
};

// Region store: append-only, indexed by region id (rid).
struct RegionsDev {
    uint32_t *keys;     // [cap][W] packed activation bits
    uint64_t *hash;     // [cap]
    void *mid;          // [cap][4] TS: seed point / edge midpoint, radius of the near list for the region's children (am_polygon.cu)
    int32_t *start;     // [cap] start plane (-1 = seed)
    int32_t *parent;    // [cap] the region it was entered from (-1 = seed)
    int32_t *nv;        // [cap] polygon vertex count
    int8_t *status;     // [cap]
    void *verts;        // [cap][kVMax][3] TS
    int32_t *edges;     // [cap][kVMax] plane of the edge leaving vertex i
    long long cap;
};

struct HashDev {
    unsigned long long *slots;
    unsigned long long mask;
};

// Wave control block in device memory.  The host-driven loop reads tail and
// err after every wave; the graph-driven loop keeps head and count here too,
// so the kernels of a captured wave read their range from the device and the last
// block of the append advances the queue and decides whether to go on.
struct WaveCtl {
    long long tail;     // regions in the store (appends advance it)
    int err;            // device error bits
    int pad0;
    long long head;     // first region of the current wave (graph-driven loop)
    int count;          // regions in the current wave
    int waves;          // waves completed
    long long limit;    // go on only while tail + count * kVMax <= limit
    int chunk_cap;      // largest wave
    unsigned int work;  // next region of the wave for the polygon warps
    int max_waves;      // waves one graph launch may run
    int grow_at;        // stop while more regions than this wait (a batch member's wave buffers grow with its queue)
    long long stop_tail; // stop after the wave that takes tail past this (a region limit)
    long long rows_from; // regions before this have no rows in the ring (it was reallocated)
    int ccount[kMaxLayers]; // regions of the wave per class (see ChunkDev)
    // the range of the wave whose children the append takes: a copy of head and
    // count that the wave's polygon kernel makes.  The append's last block moves head
    // and count on while other blocks of its grid may not have started yet; those
    // read this copy, which nothing writes before the append has ended.
    long long append_head;
    int append_count;
    int pad1;
};

// the control block's device / pinned allocation: WaveCtl, then the run's
// statistics counters (faces, largest polygon, then one count per status
// kNoStart .. kSingular, then the polygon vertices, reduced at the end of a run),
// then the count of faces walked again with FP64 predicates (accumulated during
// the run), then the weld's counts
constexpr int kStatsCount = 7;
constexpr int kFp64Slot = kStatsCount;
constexpr int kWeldSlot = kFp64Slot + 1; // vertices, faces, face indices
constexpr size_t kStatsOff = (sizeof(WaveCtl) + 15) / 16 * 16;
constexpr size_t kCtlBytes = kStatsOff + (kStatsCount + 4) * sizeof(unsigned long long);

// A wave of regions.  The constraint rows live in a ring: region id r's rows
// are at slot r % ring until a later wave takes the slot, so that a region
// finds its parent's rows there.  A region entered through a plane of hidden
// layer j has its parent's activations in layers 1 .. j - 1 and so its
// parent's affine maps in layers 1 .. j, bit for bit; only the layers after j
// are composed (class j), and the rows of the layers up to j come from the
// parent's slot (the polygon kernel, which reads every row anyway, copies them
// into the region's own).  Class 1 is composed from layer 1 on: seeds, regions
// entered through layer 1, and regions whose parent's rows have been overwritten.
struct ChunkDev {
    long long head;     // first rid of the chunk
    int count;          // regions in the chunk
    void *cons;         // [ring or count][ALLP][4] TC constraint rows
    void *eq;           // [count][4] TC face plane (b already offset by iso)
    int32_t *rec;       // [count * kVMax] hash slot claimed by each child, -1 none
    WaveCtl *ctl = nullptr; // set: head and count come from the device (graph-driven loop)
    int ring = 0;       // slots of cons; 0: no ring, rows at the wave position, every region class 1
    int order_cap = 0;  // wave positions per class list
    int32_t *order = nullptr;  // [n_lin - 1][order_cap] wave positions by class (class c's list at c - 1)
    int32_t *split = nullptr;  // [count] leading rows that come from the parent's slot
    int32_t *ccount = nullptr; // [n_lin - 1] regions per class
    long long rows_from = 0;   // host-driven loop: WaveCtl::rows_from
};

#ifdef __CUDACC__
// the wave's range, from the launch or from the device
__device__ __forceinline__ void chunk_range(const ChunkDev &ch, long long &head, int &count)
{
    if (ch.ctl) {
        head = *(volatile const long long *)&ch.ctl->head;
        count = *(volatile const int *)&ch.ctl->count;
    } else {
        head = ch.head;
        count = ch.count;
    }
}
// slot of a region's rows: of the region at wave position rl, and of region rid
__device__ __forceinline__ uint32_t row_slot(const ChunkDev &ch, long long head, int rl)
{
    return ch.ring ? (uint32_t)(head + rl) % (uint32_t)ch.ring : (uint32_t)rl;
}
__device__ __forceinline__ uint32_t ring_slot(const ChunkDev &ch, int rid) { return (uint32_t)rid % (uint32_t)ch.ring; }
#endif

struct Tolerances {
    double eps;         // feasibility (geometric distance), reference FP_EPS
    double same_eps;    // vertex merge (L1), reference FP_SAME_EPS
    double par_eps;     // a plane counts as crossing an edge line when w.d > par_eps |w| |d|
};

// launchers (stream-ordered, no synchronisation)
// nonfinite: device flag, non-zero when a weight may not be finite (null: all are)
void launch_compose(int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, double iso, int *d_err,
                    cudaStream_t st, const int *nonfinite = nullptr);
// rule_warps: sets the rule between near-equal hits (hit_rule_lanes)
// every_row: no near list
// nfp64: counts the faces the mixed form walks again with FP64 predicates
void launch_polygon(int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, const HashDev &hs,
                    const Tolerances &tol, int rule_warps, bool every_row, unsigned long long *nfp64, int *d_err,
                    cudaStream_t st);
// zeroed: an int set to zero as well (optional); points: S x 3 seed points of
// pbytes-byte floats, converted to tbytes-byte ones in dst (optional)
struct SeedPoints {
    const void *src = nullptr;
    void *dst = nullptr;
    int pbytes = 0, tbytes = 0;
};
void launch_seed_pack(const uint8_t *states, int S, int N, int W, uint32_t *keys, uint64_t *hash, cudaStream_t st,
                      int *zeroed = nullptr, const SeedPoints &points = SeedPoints());
void launch_seed_insert(const uint32_t *keys, const uint64_t *hash, int S, int W, const HashDev &hs, int32_t *rec,
                        int *d_err, cudaStream_t st);
// append of the winners.  mode 0: children of a wave, mode 1: seeds.  cond: the
// graph-driven loop's condition, which the append's last block sets after it has
// advanced ctl to the next wave.
struct AppendScratch {
    unsigned int ticket, done; // zero between appends
    unsigned int epoch;        // appends made
    unsigned int pad;
    long long new_tail;
    unsigned long long entry[1]; // [blocks] winners per block, tagged with the append's number
};
inline size_t append_scratch_bytes(int blocks) { return sizeof(AppendScratch) + sizeof(unsigned long long) * (size_t)blocks; }
int append_blocks(int rows_max);
void launch_append(int mode, int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch,
                   const HashDev &hs, const uint32_t *seed_keys, const uint64_t *seed_hash, const void *seed_points,
                   int n_items, long long *d_tail, AppendScratch *sc, int blocks_cap, int *d_err, cudaStream_t st,
                   const cudaGraphConditionalHandle *cond = nullptr);
void launch_rehash(const RegionsDev &reg, long long n, const HashDev &hs, int *d_err, cudaStream_t st);
void launch_region_stats(const int32_t *nv, const int8_t *status, long long n, unsigned long long *out,
                         cudaStream_t st);
// class lists and splits of a wave (ChunkDev); ccount must be zero
void launch_wave_classes(const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, cudaStream_t st);
int device_sms();
// the network's parameters into the engine's layouts, every value checked for NaN
// and infinity (kErrNonFinite), in one launch
struct LoadList {
    struct Item {
        const void *src; // device memory
        void *dst;
        int M, K, Mp;    // M x K to [K][Mp] (zero padding); Mp = 0: K values as they are
    } item[64];
    int count;
};
void launch_load(int prec, const LoadList &list, int *d_err, cudaStream_t st);
struct PrepareList { // FP32 linears to transpose and pad
    struct Item {
        const float *src;
        float *dst;
        int M, K, Mp;
    } item[kMaxLayers];
    int count;
};
void launch_prepare_list(const PrepareList &list, int *nonfinite, cudaStream_t st);

// error report (am_verify.cu): out[0] max |f(v)| bits, out[1] max vertex
// error bits, out[2] vertices, out[3] vertices left out (singular), out[4] faces
void launch_gather_keys(const uint32_t *keys, int W, const long long *ids, int count, uint32_t *out, cudaStream_t st);
void launch_to_double(const void *src, long long n, void *dst, cudaStream_t st);
void launch_verify(int ts_bytes, const RegionsDev &reg, const long long *ids, int count, const double *rows,
                   const double *eq, int ALLP, int ALL, unsigned long long *out, cudaStream_t st);

} // namespace am
