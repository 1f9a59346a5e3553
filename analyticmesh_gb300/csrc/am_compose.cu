// am_compose.cu -- region affine composition (SIMT form, fp32 / fp64).
//
// For every region of a chunk, compose the affine map of every hidden unit
// under the region's activation state and write the sign-flipped constraint
// rows C_k = (1 - 2 s_k) [w_k | b_k] plus the face plane (w_eq, b_eq - iso).
// Same mathematics as the reference's fill_constraints + offset_b_equ
// (backend/inc/process.h:18-203), organised GB300-first.  Connections into the
// output layer are composed too (the reference's loop stops before them,
// process.h:42).
//
// One warp owns a region: its lanes hold 32 x RPL output units x 4 columns in
// registers and walk over the *active* units of the operand only (an inactive
// unit's column of W meets an all-zero row of X: skipping it changes no bit of
// the sums, about half the units are inactive, and each region has its own).
// The weights stream through shared memory once per tile of up to 16 regions: a
// copy warp brings [32 units x up to 256 rows] blocks into a ring of stages
// with bulk copies, and the regions' warps pass through the ring on their own,
// up to a ring apart, because their active counts differ (a block barrier
// per 32 units would cost the slowest of 16 each time).  A warp reads only rows
// it has written itself (or its parent's), so nothing else is shared.
//
// What bounds it: the FMA pipe and the issue slots in fp32 (per active unit
// 4 RPL FMAs, RPL + 1 shared loads), the FP64 pipe in fp64.  Measured on GB300:
// see compose_kernel.
#include <algorithm>
#include <cuda_runtime.h>

#include "am_device.cuh"
#include "am_internal.h"
#include "am_umma.cuh"

namespace am {

namespace {

constexpr int kKC = 32;                 // operand units per block
constexpr int kWait = 1 << 22;
constexpr int kPadBytes = 2048;         // lanes beyond a pass's last row read past the block's end
constexpr int kStagesMax = 4;

// FP32: one CTA of sixteen regions per SM.  FP64: four of four, so that a wave's
// regions spread more evenly over the SMs and every round of tiles ends sooner
// (the weights' extra traffic is nothing against the FP64 pipe's time: measured
// 31.1 against 33.3 ms, and the same in FP32 3.1 against 3.1).
template <typename T>
struct Cfg {
    static constexpr bool f64 = sizeof(T) == 8;
    static constexpr int warps = f64 ? 4 : 16;          // regions per tile at most
    static constexpr int threads = 32 * warps + 32;     // + the copy warp
    static constexpr int ctas = f64 ? 4 : 1;            // per SM
    static constexpr int stages = f64 ? 3 : 4;
    static constexpr int stage_bytes = (f64 ? 16 : 32) * 1024; // kKC units x pass rows
    static constexpr int rows = stage_bytes / (kKC * (int)sizeof(T)); // per pass: 256 FP32, 64 FP64
    static constexpr size_t smem =
        (size_t)stages * stage_bytes + kPadBytes + (size_t)warps * kKC * (sizeof(vec4_t<T>) + sizeof(uint32_t));
};

struct Ring {
    uint64_t full[kStagesMax], empty[kStagesMax];
    int abort;
};

__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ bool ring_wait(uint64_t *bar, uint32_t parity, int *err, volatile int *abort)
{
    if (*abort) return false;
    if (umma::mbar_wait(bar, parity, kWait)) return true;
    if (err) atomicOr(err, kErrWait);
    *abort = 1;
    return false;
}

// The products of linear i: job 0 is the linear on hidden layer i, the others
// its transforms from earlier hidden layers.
struct Job {
    const void *wt;
    int Mp, src;
};
__device__ __forceinline__ int jobs_of(const NetDev &net, int i)
{
    int n = 1;
    for (int s = 0; s < net.nskip[i]; ++s) n += net.skip[i][s].kind == 1 && net.skip[i][s].from >= 1;
    return n;
}
__device__ __forceinline__ Job job_of(const NetDev &net, int i, int job)
{
    if (job > 0)
        for (int s = 0, q = 0; s < net.nskip[i]; ++s)
            if (net.skip[i][s].kind == 1 && net.skip[i][s].from >= 1 && ++q == job)
                return Job{net.skip[i][s].tmt, net.skip[i][s].Mp, net.skip[i][s].from};
    return Job{net.Wt[i], net.Mp[i], i};
}

// (the copy warp) the weight blocks of every tile of the CTA, in the order the
// regions' warps consume them
template <typename T>
__device__ void produce(const NetDev &net, const WavePlan &plan, int rounds, unsigned char *ws, Ring &ring, int *err)
{
    const int lane = threadIdx.x & 31;
    volatile int *abort = &ring.abort;
    int h = 0;
    int last[Cfg<T>::stages]; // (lane 0's view, the same in every lane) the last block copied into each stage
    for (int s = 0; s < Cfg<T>::stages; ++s) last[s] = -1;
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        for (int i = plan_class(plan, t); i < net.n_lin; ++i)
            for (int mb = 0; mb < net.nodes[i + 1]; mb += Cfg<T>::rows)
                for (int job = 0, nj = jobs_of(net, i); job < nj; ++job) {
                    const Job jb = job_of(net, i, job);
                    const int K = net.nodes[jb.src], ld = min(Cfg<T>::rows, jb.Mp - mb);
                    for (int k0 = 0; k0 < K; k0 += kKC, ++h) {
                        const int s = h % Cfg<T>::stages;
                        int go = 1;
                        if (lane == 0)
                            go = h < Cfg<T>::stages || ring_wait(ring.empty + s, (uint32_t)(h / Cfg<T>::stages - 1) & 1u, err, abort);
                        if (!__shfl_sync(0xffffffffu, go, 0)) continue;
                        const int kc = min(kKC, K - k0);
                        const uint32_t row = (uint32_t)(ld * sizeof(T));
                        const T *src = (const T *)jb.wt + (size_t)k0 * jb.Mp + mb;
                        unsigned char *dst = ws + (size_t)s * Cfg<T>::stage_bytes;
                        if (lane == 0) umma::mbar_expect_tx(ring.full + s, row * (uint32_t)kc);
                        __syncwarp();
                        if (ld == jb.Mp) { // whole rows of W^T: one contiguous run
                            if (lane == 0) umma::bulk_g2s(dst, src, row * (uint32_t)kc, ring.full + s);
                        } else if (lane < kc) {
                            umma::bulk_g2s(dst + (size_t)lane * row, src + (size_t)lane * jb.Mp, row, ring.full + s);
                        }
#pragma unroll
                        for (int q = 0; q < Cfg<T>::stages; ++q)
                            if (q == s) last[q] = h;
                    }
                }
    }
    // nothing lands in shared memory after the CTA has left (bounded)
    if (lane == 0)
#pragma unroll
        for (int s = 0; s < Cfg<T>::stages; ++s)
            if (last[s] >= 0) umma::mbar_wait(ring.full + s, (uint32_t)(last[s] / Cfg<T>::stages) & 1u, kWait);
    __syncwarp();
}

// A region's state in its warp.
template <typename T>
struct Region {
    T *cons;
    size_t rstride;
    int4 ri;
    int jend, lane;
    const uint32_t *key;
    vec4_t<T> *xs;  // the warp's packed operand block: rows ...
    uint32_t *offs; // ... and where their units' weights are in the ring
    bool dense;
};

// the products of the packed units i .. i + U - 1, in order
template <typename T, int RPL, int U>
__device__ __forceinline__ void units(const Region<T> &g, const unsigned char *w, int i, T acc[RPL][4])
{
    vec4_t<T> x[U];
    T wu[U][RPL];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        x[u] = g.xs[i + u];
        const T *p = reinterpret_cast<const T *>(w + g.offs[i + u]);
#pragma unroll
        for (int j = 0; j < RPL; ++j) wu[u][j] = p[32 * j];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < RPL; ++j) {
            acc[j][0] = fma_t(wu[u][j], x[u].x, acc[j][0]);
            acc[j][1] = fma_t(wu[u][j], x[u].y, acc[j][1]);
            acc[j][2] = fma_t(wu[u][j], x[u].z, acc[j][2]);
            acc[j][3] = fma_t(wu[u][j], x[u].w, acc[j][3]);
        }
}

// the same for a linear of one unit (the output): lane c of four takes column c,
// a quarter of the multiply-adds of a lane per unit (the FP64 pipe issues an
// instruction at the same cost however few lanes are active)
template <typename T>
__device__ __forceinline__ void unit_face(const Region<T> &g, const unsigned char *w0, int i, T &acc)
{
    const T x = reinterpret_cast<const T *>(g.xs + i)[g.lane & 3];
    acc = fma_t(*reinterpret_cast<const T *>(w0 + g.offs[i]), x, acc);
}

// one pass (32 RPL units of linear i from mb on; RPL 0: its only unit, in acc's
// first element by column) over every job's blocks
template <typename T, int RPL>
__device__ void pass(const NetDev &net, int i, int mb, const Region<T> &g, const unsigned char *ws, Ring &ring, int &h,
                     int *err, T (*acc)[4])
{
    volatile int *abort = &ring.abort;
    for (int job = 0, nj = jobs_of(net, i); job < nj; ++job) {
        const Job jb = job_of(net, i, job);
        const int K = net.nodes[jb.src], rows0 = net.hoff[jb.src], ld = min(Cfg<T>::rows, jb.Mp - mb);
        const T *src = g.cons + (size_t)(uint32_t)(rows0 < g.jend ? g.ri.y : g.ri.x) * g.rstride + (size_t)rows0 * 4;
        auto load = [&](int k0, bool &on) {
            const int k = k0 + g.lane;
            on = k < K && key_bit(g.key, rows0 + k);
            vec4_t<T> c;
            c.x = c.y = c.z = c.w = T(0);
            if (on) c = ld4<T>(src + (size_t)k * 4);
            return c;
        };
        bool on;
        vec4_t<T> c = load(0, on);
        for (int k0 = 0; k0 < K; k0 += kKC, ++h) {
            const T sg = rows0 + k0 + g.lane == g.ri.z ? T(1) : T(-1); // (C = -A where active)
            vec4_t<T> x;
            x.x = sg * c.x;
            x.y = sg * c.y;
            x.z = sg * c.z;
            x.w = sg * c.w;
            // the block's active units, packed in order: the operand row and the
            // offset of the unit's weights in the ring
            const int s = h % Cfg<T>::stages;
            const uint32_t off = (uint32_t)(s * Cfg<T>::stage_bytes + g.lane * ld * (int)sizeof(T));
            const bool take = g.dense ? k0 + g.lane < K : on;
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            const int n = __popc(mask), at = __popc(mask & ((1u << g.lane) - 1u));
            if (!on) x.x = x.y = x.z = x.w = T(0);
            if (take) {
                g.xs[at] = x;
                g.offs[at] = off;
            }
            __syncwarp();
            if (k0 + kKC < K) c = load(k0 + kKC, on);
            // (the warp decides as one: after an abort nobody reads the ring)
            const bool ok = __all_sync(0xffffffffu, ring_wait(ring.full + s, (uint32_t)(h / Cfg<T>::stages) & 1u, err, abort));
            if (ok) {
                const unsigned char *w = ws + g.lane * sizeof(T);
                // U units' loads in flight (the FP64 pipe is slow enough for one)
                constexpr int U = sizeof(T) == 8 ? 1 : (RPL > 4 ? 2 : 4);
                int i = 0;
                if constexpr (RPL == 0) {
#pragma unroll 4
                    for (; i < n; ++i) unit_face<T>(g, ws, i, acc[0][0]);
                } else {
                    for (; i + U <= n; i += U) units<T, RPL, U>(g, w, i, acc);
                    for (; U > 1 && i < n; ++i) units<T, RPL, 1>(g, w, i, acc);
                }
            }
            __syncwarp();
            if (g.lane == 0) umma::mbar_arrive(ring.empty + s);
        }
    }
}

// bias, connections without a product (identities, the input), the output
template <typename T>
__device__ __forceinline__ void store_unit(const NetDev &net, int i, int m, const Region<T> &g, const T *acc, T iso,
                                           T *eq)
{
    T v[4] = {acc[0], acc[1], acc[2], acc[3] + ((const T *)net.bias[i])[m]};
    for (int s = 0; s < net.nskip[i]; ++s) {
        const SkipDev &sk = net.skip[i][s];
        if (sk.kind == 0) {
            if (sk.from == 0) {
                if (m < 3) v[m] += T(1);
            } else {
                const int row = net.hoff[sk.from] + m;
                if (key_bit(g.key, row)) {
                    const vec4_t<T> c = tile_row<T>(g.cons, g.rstride, g.ri, row, g.jend);
                    v[0] -= c.x;
                    v[1] -= c.y;
                    v[2] -= c.z;
                    v[3] -= c.w;
                }
            }
        } else if (sk.from == 0) {
            const T *tt = (const T *)sk.tmt; // [3][Mp]
            v[0] += tt[m];
            v[1] += tt[(size_t)sk.Mp + m];
            v[2] += tt[2 * (size_t)sk.Mp + m];
        }
    }
    vec4_t<T> o;
    if (i < net.n_lin - 1) {
        const int row = net.hoff[i + 1] + m;
        const T sg = key_bit(g.key, row) ? T(-1) : T(1);
        o.x = sg * v[0];
        o.y = sg * v[1];
        o.z = sg * v[2];
        o.w = sg * v[3];
        st4<T>(g.cons + (size_t)(uint32_t)g.ri.x * g.rstride + (size_t)row * 4, o);
    } else {
        o.x = v[0];
        o.y = v[1];
        o.z = v[2];
        o.w = v[3] - iso;
        st4<T>(eq, o);
    }
}

template <typename T>
__device__ void face_pass(const NetDev &net, int i, const Region<T> &g, const unsigned char *ws, Ring &ring, int &h, int *err,
                          T iso, T *eq)
{
    T acc[1][4];
    acc[0][0] = T(0);
    pass<T, 0>(net, i, 0, g, ws, ring, h, err, acc);
    T v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = __shfl_sync(0xffffffffu, acc[0][0], c);
    if (g.lane == 0) store_unit<T>(net, i, 0, g, v, iso, eq);
}

template <typename T, int RPL>
__device__ void linear_pass(const NetDev &net, int i, int mb, const Region<T> &g, const unsigned char *ws, Ring &ring,
                            int &h, int *err, T iso, T *eq)
{
    T acc[RPL][4];
#pragma unroll
    for (int j = 0; j < RPL; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[j][c] = T(0);
    pass<T, RPL>(net, i, mb, g, ws, ring, h, err, acc);
#pragma unroll
    for (int j = 0; j < RPL; ++j) {
        const int m = mb + 32 * j + g.lane;
        if (m < net.nodes[i + 1]) store_unit<T>(net, i, m, g, acc[j], iso, eq);
    }
}

// Measured on GB300, composition of all 265 K regions of 3-[128]x4-1 in waves of
// 7 K (parents' rows on both sides): fp32 2.7 ms, fp64 28.5 ms; a 16-region x
// 64-row register tile per CTA over every unit, operand staged behind two block
// barriers per 32 units, took 6.6 and 71 ms.  8,192 given states, every layer
// (weights transposed and keys packed in the same call): 112 us against 238.
// (Two neighbouring units per fma.rn.f32x2 and the operand's columns doubled, 13
// instructions per active unit instead of 22, measured the same in fp32: the
// chain of a block -- rows, packing, ring, products -- bounds it.)
template <typename T>
__global__ void __launch_bounds__(Cfg<T>::threads, Cfg<T>::ctas) compose_kernel(NetDev net, RegionsDev reg, ChunkDev ch, T iso,
                                                              const int *nonfinite, int *err)
{
    extern __shared__ __align__(128) unsigned char ws[]; // the weight ring, then the warps' operand blocks
    __shared__ Ring ring;
    __shared__ WavePlan plan;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    long long head;
    int count;
    chunk_range(ch, head, count);
    if (count <= 0) return;
    // as few regions per tile as fill the grid: a small wave spreads over every SM
    if (warp == 0) plan_wave(plan, ch, net.n_lin - 1, count, (int)gridDim.x, Cfg<T>::warps, 1);
    if (tid == 32) {
        ring.abort = 0;
        for (int s = 0; s < Cfg<T>::stages; ++s) {
            umma::mbar_init(ring.full + s, 1);
            umma::mbar_init(ring.empty + s, Cfg<T>::warps);
        }
        umma::fence_mbar_init();
    }
    __syncthreads();
    const int rounds = plan_rounds(plan, (int)gridDim.x);
    if (warp == Cfg<T>::warps) {
        produce<T>(net, plan, rounds, ws, ring, err);
        return;
    }
    Region<T> g;
    g.cons = (T *)ch.cons;
    g.rstride = (size_t)net.ALLP * 4;
    g.lane = lane;
    {
        unsigned char *pack = ws + (size_t)Cfg<T>::stages * Cfg<T>::stage_bytes + kPadBytes;
        g.xs = reinterpret_cast<vec4_t<T> *>(pack) + warp * kKC;
        g.offs = reinterpret_cast<uint32_t *>(pack + (size_t)Cfg<T>::warps * kKC * sizeof(vec4_t<T>)) + warp * kKC;
    }
    // a weight that is not finite meets the zeros of inactive units too (NaN,
    // as in a dense product): then no unit is skipped
    g.dense = nonfinite && *nonfinite != 0;
    int h = 0;
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        const int cls = plan_class(plan, t);
        const bool live = warp < tile_nreg(plan, t, cls);
        if (!live) { // no region for this warp: it gives its share of every block back
            for (int i = cls; i < net.n_lin; ++i)
                for (int mb = 0; mb < net.nodes[i + 1]; mb += Cfg<T>::rows)
                    for (int job = 0, nj = jobs_of(net, i); job < nj; ++job)
                        for (int k0 = 0, K = net.nodes[job_of(net, i, job).src]; k0 < K; k0 += kKC, ++h) {
                            const int s = h % Cfg<T>::stages;
                            __all_sync(0xffffffffu, ring_wait(ring.full + s, (uint32_t)(h / Cfg<T>::stages) & 1u, err, &ring.abort));
                            if (lane == 0) umma::mbar_arrive(ring.empty + s);
                        }
            continue;
        }
        g.ri = tile_region(plan, reg, ch, head, t, cls, warp);
        g.jend = cls > 1 ? net.hoff[cls + 1] : 0;
        g.key = reg.keys + (size_t)(head + g.ri.w) * net.W;
        T *own = g.cons + (size_t)(uint32_t)g.ri.x * g.rstride;
        T *eq = (T *)ch.eq + (size_t)g.ri.w * 4;
        // class 1: hidden layer 1 = linear 0 rows, sign-flipped; extra constraints as given
        if (cls == 1) {
            const T *W0 = (const T *)net.W0;
            const T *b0 = (const T *)net.bias[0];
            for (int m = lane; m < net.nodes[1]; m += 32) {
                const T sg = key_bit(g.key, m) ? T(-1) : T(1);
                vec4_t<T> c;
                c.x = sg * W0[3 * m + 0];
                c.y = sg * W0[3 * m + 1];
                c.z = sg * W0[3 * m + 2];
                c.w = sg * b0[m];
                st4<T>(own + (size_t)m * 4, c);
            }
        }
        const T *we = (const T *)net.w_extra;
        const T *be = (const T *)net.b_extra;
        for (int e = lane; e < net.E; e += 32) {
            vec4_t<T> c;
            c.x = we[3 * e + 0];
            c.y = we[3 * e + 1];
            c.z = we[3 * e + 2];
            c.w = be[e];
            st4<T>(own + (size_t)(net.N + e) * 4, c);
        }
        __syncwarp(); // the rows written above are other lanes' operand
        for (int i = cls; i < net.n_lin; ++i) {
            for (int mb = 0; mb < net.nodes[i + 1]; mb += Cfg<T>::rows) {
                const int n = (min(Cfg<T>::rows, net.nodes[i + 1] - mb) + 31) / 32;
                if (i == net.n_lin - 1) face_pass<T>(net, i, g, ws, ring, h, err, iso, eq); // (one unit)
                else if (n <= 1) linear_pass<T, 1>(net, i, mb, g, ws, ring, h, err, iso, eq);
                else if (n <= 2 || Cfg<T>::f64) linear_pass<T, 2>(net, i, mb, g, ws, ring, h, err, iso, eq);
                else if constexpr (!Cfg<T>::f64) {
                    if (n <= 3) linear_pass<T, 3>(net, i, mb, g, ws, ring, h, err, iso, eq);
                    else if (n <= 4) linear_pass<T, 4>(net, i, mb, g, ws, ring, h, err, iso, eq);
                    else if (n <= 6) linear_pass<T, 6>(net, i, mb, g, ws, ring, h, err, iso, eq);
                    else linear_pass<T, 8>(net, i, mb, g, ws, ring, h, err, iso, eq);
                }
            }
            __syncwarp(); // layer i + 1's rows become the next operand
        }
    }
}

template <typename T>
__global__ void load_kernel(LoadList list, int *err)
{
    const LoadList::Item &it = list.item[blockIdx.y];
    const T *src = (const T *)it.src;
    T *dst = (T *)it.dst;
    const long long n = it.Mp ? (long long)it.K * it.Mp : it.K;
    bool bad = false;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        T v;
        if (it.Mp) {
            const int k = (int)(q / it.Mp), m = (int)(q % it.Mp);
            v = m < it.M ? src[(size_t)m * it.K + k] : T(0);
        } else {
            v = src[q];
        }
        bad |= !isfinite(v);
        dst[q] = v;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, kErrNonFinite);
}

// FP32 linears transposed and padded in one launch (blockIdx.y); *nonfinite set
// where a value is not finite
__global__ void prepare_list_kernel(PrepareList list, int *nonfinite)
{
    const PrepareList::Item &it = list.item[blockIdx.y];
    const int n = it.K * it.Mp;
    bool bad = false;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int k = q / it.Mp, m = q % it.Mp;
        const float v = m < it.M ? it.src[(size_t)m * it.K + k] : 0.f;
        bad |= !isfinite(v);
        it.dst[q] = v;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(nonfinite, 1);
}

} // namespace

void launch_load(int prec, const LoadList &list, int *d_err, cudaStream_t st)
{
    if (list.count <= 0) return;
    long long most = 1;
    for (int b = 0; b < list.count; ++b)
        most = std::max(most, (long long)list.item[b].K * std::max(list.item[b].Mp, 1));
    const dim3 grid((unsigned)std::min<long long>((most + 255) / 256, 256), (unsigned)list.count);
    if (prec == kFloat64)
        load_kernel<double><<<grid, 256, 0, st>>>(list, d_err);
    else
        load_kernel<float><<<grid, 256, 0, st>>>(list, d_err);
}

template <typename T>
static void launch_one(const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, T iso, const int *nonfinite,
                       int *d_err, cudaStream_t st)
{
    cudaFuncSetAttribute(compose_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<T>::smem);
    const int slots = device_sms() * Cfg<T>::ctas;
    const int grid = ch.ctl ? slots : std::min(slots, ch.count);
    compose_kernel<T><<<grid, Cfg<T>::threads, Cfg<T>::smem, st>>>(net, reg, ch, iso, nonfinite, d_err);
}

void launch_compose(int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, double iso, int *d_err,
                    cudaStream_t st, const int *nonfinite)
{
    if (!ch.ctl && ch.count <= 0) return;
    if (prec == kFloat64)
        launch_one<double>(net, reg, ch, iso, nonfinite, d_err, st);
    else
        launch_one<float>(net, reg, ch, (float)iso, nonfinite, d_err, st);
}

void launch_prepare_list(const PrepareList &list, int *nonfinite, cudaStream_t st)
{
    if (list.count > 0) prepare_list_kernel<<<dim3(64, (unsigned)list.count), 256, 0, st>>>(list, nonfinite);
}

} // namespace am
