// am_compose_tc.cu -- region affine composition on the 5th-generation tensor
// cores (the mixed-precision form).
//
// Same mathematics as am_compose.cu (the reference's fill_constraints,
// backend/inc/process.h:18-193): for every region, A_{l+1} = W_l diag(s_l) A_l
// (+ b_l, + skips), C = (1 - 2 s) A.  One CTA owns a tile of regions (4
// columns each, UMMA N = 4 x regions, chosen per launch from the chunk size so
// that small frontier waves still spread over every SM) and keeps the masked
// operand X_l = diag(s_l) A_l on chip the whole way through the network, as
// bf16 terms in shared memory (MN-major core matrices without swizzle): the B
// operand of tcgen05.mma.  The layer
// weights are the A operand (K-major); they are pre-split and
// stored in global memory as the exact shared-memory image of their 128 x 64
// blocks, so one bulk copy (cp.async.bulk, completing on an mbarrier) stages a
// block while the tensor core works on the previous one, and the first blocks
// of the next layer land while the epilogue of this one runs.
//
// Every operand is split into three bf16 terms, x = hi + mid + lo (24
// significant bits, as fp32); a block issues the six products whose weight is
// at least 2^-16 -- hh, hm, mh, hl, lh, mm.  A two-term split leaves ~2^-17
// of every operand unrepresented, which moved vertices by ~1.5e-5 and changed
// near-degenerate walk decisions.  The tensor core's fp32 accumulation error
// grows with the number of accumulate steps into one accumulator, so the
// dominant hh product and the five small correction products accumulate in
// two separate TMEM accumulators that the epilogue adds once: fp32-level
// constraint rows.  The epilogue (sixteen warps; the warps w with equal w % 4
// share TMEM lanes 32 (w % 4).. and split the columns) reads the accumulators with
// tcgen05.ld (one TMEM lane per output unit), adds bias and skips, writes the
// sign-flipped constraint rows to HBM for the polygon kernel, and writes the
// next layer's masked operand straight back into shared memory.  The face
// plane (output layer, one row) is a 4 x K dot product per region in fp32,
// from the operand in shared memory.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "am_device.cuh"
#include "am_internal.h"
#include "am_tc.h"
#include "am_umma.cuh"

namespace am {

namespace {

constexpr int kThreads = 512;
constexpr int kWaitIters = 1 << 22;
constexpr int kFaceSumBytes = kThreads * 16; // face-plane partial sums: a float4 per thread

// x = hi + mid + lo in bf16 for two values at once (round to nearest each)
__device__ __forceinline__ void split2(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l)
{
    const __nv_bfloat162 hb = __floats2bfloat162_rn(a, b);
    const float2 hf = __bfloat1622float2(hb);
    const float ra = a - hf.x, rb = b - hf.y;
    const __nv_bfloat162 mb = __floats2bfloat162_rn(ra, rb);
    const float2 mf = __bfloat1622float2(mb);
    const __nv_bfloat162 lb = __floats2bfloat162_rn(ra - mf.x, rb - mf.y);
    h = *reinterpret_cast<const uint32_t *>(&hb);
    m = *reinterpret_cast<const uint32_t *>(&mb);
    l = *reinterpret_cast<const uint32_t *>(&lb);
}

// The masked operand X (ncols x Kp) is kept as three bf16 terms in 64-deep blocks.
// The operand image: a term of a 64-deep block is ncols / 8 chunks of eight
// columns, a chunk 64 rows of 16 bytes.  That is the canonical MN-major layout
// without swizzle (eight rows of a chunk: 128 contiguous bytes), so a warp whose
// lanes hold consecutive rows stores 512 contiguous bytes, in scratch (the streamed
// operand) as in shared memory, and any multiple of 16 columns will do.  (Measured on GB300: the
// products run at the same rate as from a 128-byte swizzle, 64 cycles at 128
// columns; with the swizzled layout, two regions x 16 rows per warp item, the
// composition of ragged widths with connections took 1.95 ms against 1.72, of
// 128 x 4 1.80 against 1.74.)
__host__ __device__ __forceinline__ uint32_t op_term_bytes(int ncols) { return (uint32_t)ncols * 128u; }
__device__ __forceinline__ void op_put8(uint8_t *blk, uint32_t term, int chunk, int k, const float *x)
{
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split2(x[2 * i], x[2 * i + 1], h[i], m[i], l[i]);
    uint8_t *p = blk + chunk * 1024 + k * 16;
    *reinterpret_cast<uint4 *>(p) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(p + term) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(p + 2 * term) = make_uint4(l[0], l[1], l[2], l[3]);
}

// the whole operand in shared memory
struct XOp {
    uint8_t *xs;
    uint32_t term; // bytes of a term of a block
    __device__ __forceinline__ uint8_t *block(int kb) const { return xs + (size_t)kb * 3 * term; }
    // columns 8 chunk .. 8 chunk + 7 of row k
    __device__ __forceinline__ void put8(int chunk, int k, const float *x) const { op_put8(block(k >> 6), term, chunk, k & 63, x); }
    // hi + mid + lo of region r's columns of row k
    __device__ __forceinline__ void get4(int r, int k, float *v) const
    {
        const uint8_t *p = block(k >> 6) + (r >> 1) * 1024 + (k & 63) * 16 + (r & 1) * 8;
        const uint2 h = *reinterpret_cast<const uint2 *>(p), m = *reinterpret_cast<const uint2 *>(p + term),
                    l = *reinterpret_cast<const uint2 *>(p + 2 * term);
        const uint32_t hw[2] = {h.x, h.y}, mw[2] = {m.x, m.y}, lw[2] = {l.x, l.y};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&hw[i]));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&mw[i]));
            const float2 c = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&lw[i]));
            v[2 * i] = a.x + b.x + c.x;
            v[2 * i + 1] = a.y + b.y + c.y;
        }
    }
};

// the connections of linear i that are no product (identities, the input) added
// to unit m of a region
__device__ __forceinline__ void add_skips(const NetDev &net, int i, int m, const float *cons, size_t rstride, const int4 &ri,
                                          int jend, const uint32_t *key, float (&o)[4])
{
    for (int s = 0; s < net.nskip[i]; ++s) {
        const SkipDev &sk = net.skip[i][s];
        if (sk.kind == 0) {
            if (sk.from == 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (m == c) o[c] += 1.f;
            } else {
                const int srow = net.hoff[sk.from] + m;
                if (key_bit(key, srow)) {
                    const float4 c = tile_row<float>(cons, rstride, ri, srow, jend);
                    o[0] -= c.x;
                    o[1] -= c.y;
                    o[2] -= c.z;
                    o[3] -= c.w;
                }
            }
        } else if (sk.from == 0) {
            const float *tt = (const float *)sk.tmt;
            o[0] += tt[m];
            o[1] += tt[(size_t)sk.Mp + m];
            o[2] += tt[2 * (size_t)sk.Mp + m];
        }
    }
}

// X[n = 4r + c][k] = s_k(r) ? -C[r][src + k][c] : 0 for k < K, 0 to the end of the
// last block.  A warp item is two regions x 32 rows, a row per lane: loads and
// stores of 512 contiguous bytes.
__device__ void stage_x_from_rows(const XOp &X, int R, const float *cons, size_t rstride, const int4 *ri, int jend,
                                  const uint32_t *keys, int W, int nreg, int src, int K)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool par = src < jend;
    constexpr int kU = 2, kWarpsM = kThreads / 32;
    const int n = R * ((K + 63) / 64);
    // the items' loads before the first is used (measured on GB300: one by one the
    // rows of 32 regions x 128 units took 15 K cycles, most of a tile's time)
    for (int q0 = warp; q0 < n; q0 += kU * kWarpsM) {
        float4 v[kU][2];
        unsigned other = 0u; // rows with the other sign
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = q0 + u * kWarpsM, kb = q / R, in = q - kb * R;
            const int k = kb * 64 + (in & 1) * 32 + lane;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = (in >> 1) * 2 + e;
                v[u][e] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (q < n && r < nreg && k < K && key_bit(keys + (size_t)r * W, src + k)) {
                    const int4 g = ri[r];
                    v[u][e] = ld4<float>(cons + (size_t)(uint32_t)(par ? g.y : g.x) * rstride + (size_t)(src + k) * 4);
                    if (src + k == g.z) other |= 1u << (2 * u + e);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = q0 + u * kWarpsM, kb = q / R, in = q - kb * R;
            if (q >= n) break;
            const float s0 = (other >> (2 * u)) & 1u ? 1.f : -1.f, s1 = (other >> (2 * u + 1)) & 1u ? 1.f : -1.f;
            const float4 a = v[u][0], b = v[u][1];
            const float x[8] = {s0 * a.x, s0 * a.y, s0 * a.z, s0 * a.w, s1 * b.x, s1 * b.y, s1 * b.z, s1 * b.w};
            X.put8(in >> 1, kb * 64 + (in & 1) * 32 + lane, x);
        }
    }
}

__device__ __forceinline__ int mat_blocks(const TcMat &m) { return (m.Mp / 128) * (m.Kp / 64); }
__device__ __forceinline__ bool tc_skip(const SkipDev &sk) { return sk.kind == 1 && sk.from >= 1; }

// global weight block g in the order the layers consume them: linear i's
// blocks (M tile outer, K block inner), then its skip transforms
__device__ const uint8_t *block_ptr(const NetDev &net, const TcNet &tc, int g)
{
    for (int i = 1; i <= net.n_lin - 2; ++i) {
        int nb = mat_blocks(tc.lin[i]);
        if (g < nb) return tc.lin[i].blocks + (size_t)g * kWBlockBytes;
        g -= nb;
        for (int s = 0; s < net.nskip[i]; ++s)
            if (tc_skip(net.skip[i][s])) {
                nb = mat_blocks(tc.skip[i][s]);
                if (g < nb) return tc.skip[i][s].blocks + (size_t)g * kWBlockBytes;
                g -= nb;
            }
    }
    return nullptr;
}

// blocks of the linears before `end` (total: end = n_lin - 1)
__device__ int blocks_before(const NetDev &net, const TcNet &tc, int end)
{
    int n = 0;
    for (int i = 1; i < end; ++i) {
        n += mat_blocks(tc.lin[i]);
        for (int s = 0; s < net.nskip[i]; ++s)
            if (tc_skip(net.skip[i][s])) n += mat_blocks(tc.skip[i][s]);
    }
    return n;
}

// Weight-block pipeline.  A copy warp (its lane 0) streams every weight block
// of the CTA's tiles, in the order the products consume them: block h goes
// into stage h % nstage once block h - nstage's products have completed (done
// barrier).  Thread 0 issues the products of block h once its bytes have
// landed (full barrier).  Phase parity of either barrier for block h is
// (h / nstage) & 1.  h counts on across the CTA's tiles, so the next tile's
// first blocks load during this tile's last layer and every layer's first
// blocks during the previous layer's epilogue.  (Measured on GB300: with the
// copies issued by thread 0 between its products, each block cost it a wait
// for the previous block's products before the refill, and the tensor pipe
// stood idle most of the time.)
//
// Every wait is bounded.  A wait that runs out sets the error bit kErrWait
// and the CTA's abort flag: from then on no copy and no product is issued,
// the other threads skip the epilogues, and before the CTA returns the copy
// warp waits (again bounded) for its copies in flight and thread 0 for the
// products in flight, so that nothing lands in shared memory or TMEM after
// the CTA has released them.  The host reports kErrWait as a failed run.
struct WPipe {
    uint64_t *full, *done;
    uint8_t *ws;
    int nstage;
    int *err;
    int consumed;          // (warp 0) blocks whose products were issued
    volatile int *abort;   // the CTA's abort flag (shared memory)
};

__device__ __forceinline__ bool wp_wait(WPipe &p, uint64_t *bar, uint32_t parity)
{
    if (umma::mbar_wait(bar, parity, kWaitIters)) return true;
    atomicOr(p.err, kErrWait);
    *p.abort = 1;
    return false;
}

// (the copy warp's lane 0) every weight block of the CTA's tiles, nstage
// blocks ahead of the products at most; a tile of class c consumes the blocks
// of linear c on
__device__ void wp_produce(WPipe &p, const NetDev &net, const TcNet &tc, const WavePlan &plan, int rounds)
{
    int last[4] = {-1, -1, -1, -1}; // the last block copied into each stage
    const int total = blocks_before(net, tc, net.n_lin - 1);
    int h = 0;
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        for (int b = blocks_before(net, tc, plan_class(plan, t)); b < total; ++b, ++h) {
            const int s = h % p.nstage;
            if (*p.abort) continue;
            if (h >= p.nstage && !wp_wait(p, p.done + s, (uint32_t)((h - p.nstage) / p.nstage) & 1u)) continue;
            umma::mbar_expect_tx(p.full + s, (uint32_t)kWBlockBytes);
            umma::bulk_g2s(p.ws + (size_t)s * kWBlockBytes, block_ptr(net, tc, b), (uint32_t)kWBlockBytes, p.full + s);
            last[s] = h;
        }
    }
    // nothing lands in shared memory after the CTA has left (bounded)
    for (int s = 0; s < p.nstage; ++s)
        if (last[s] >= 0) umma::mbar_wait(p.full + s, (uint32_t)(last[s] / p.nstage) & 1u, kWaitIters);
}

// The six products of one K step (terms t of the weights, u of the operand, of
// weight 2^-8(t+u), t + u <= 2), the same A consecutively: hh into the main
// accumulator, the others into the correction's.
__device__ __forceinline__ void issue_step(uint32_t d_main, uint32_t d_corr, uint64_t ad, uint64_t xd, uint64_t xu,
                                           uint32_t idesc, bool fresh)
{
    umma::mma_bf16_a<1>(d_main, ad, xd, idesc, fresh ? 0u : 1u);
    umma::mma_bf16_a<2>(d_corr, ad, xd + xu, idesc, fresh ? 0u : 1u);
    umma::mma_bf16_a<3>(d_corr, ad, xd + 2 * xu, idesc, 1u);
    umma::mma_bf16_a<1>(d_corr, ad + 1024u, xd, idesc, 1u);
    umma::mma_bf16_a<3>(d_corr, ad + 1024u, xd + xu, idesc, 1u);
    umma::mma_bf16_a<0>(d_corr, ad + 2048u, xd, idesc, 1u);
}

// (warp 0, one elected lane issuing: see issue_streamed) D[mt] (+)= M . X over all
// K blocks of the operand in shared memory: six products per K step (terms t, u of
// weight 2^-8(t+u), t + u <= 2)
__device__ void gemm_issue(WPipe &p, const TcMat &m, int mtiles, const XOp &X, int ncols, uint32_t tmem, bool first, int &g)
{
    const uint32_t idesc = umma::idesc_bf16_bmn(128, ncols);
    const uint64_t xd0 = umma::desc_mn(umma::smem_addr(X.xs), 128u, 1024u);
    const uint64_t xu = X.term >> 4, xj = 16u; // to the next term and K step (16 rows of every chunk)
    const int kblocks = m.Kp / 64;
    for (int mt = 0; mt < mtiles; ++mt) {
        for (int kb = 0; kb < kblocks; ++kb) {
            const int s = g % p.nstage;
            const bool ok = *p.abort == 0 && wp_wait(p, p.full + s, (uint32_t)(g / p.nstage) & 1u);
            if (!__all_sync(0xffffffffu, ok)) return;
            umma::fence_after();
            const uint32_t a0 = umma::smem_addr(p.ws + (size_t)s * kWBlockBytes);
            const uint32_t d_main = tmem + (uint32_t)(mt * ncols);            // hh
            const uint32_t d_corr = tmem + (uint32_t)((mtiles + mt) * ncols); // the rest
            const bool fresh = first && kb == 0;
            // A: term t at +16 KB (1024 units), K step j at +32 B (2 units)
            const uint64_t ad = umma::desc_sw128(a0), xd = xd0 + 3u * xu * (uint64_t)kb;
            if (umma::elect()) {
#pragma unroll
                for (int j = 0; j < 4; ++j) issue_step(d_main, d_corr, ad + 2u * j, xd + xj * j, xu, idesc, fresh && j == 0);
                umma::commit(umma::smem_addr(p.done + s)); // frees the stage for the copy warp
            }
            __syncwarp();
            p.consumed = g + 1;
            ++g;
        }
    }
}

// (thread 0) after the last block of a layer: wait until its products are in TMEM
__device__ void gemm_finish(WPipe &p, int g)
{
    if (*p.abort) return;
    const int last = g - 1;
    if (!wp_wait(p, p.done + last % p.nstage, (uint32_t)(last / p.nstage) & 1u)) return;
    umma::fence_before();
}

// (every thread, after the block barrier that follows gemm_finish) observe
// the same completion before reading the accumulators
__device__ __forceinline__ void gemm_observe(const WPipe &p, int last)
{
    if (!umma::mbar_wait(p.done + last % p.nstage, (uint32_t)(last / p.nstage) & 1u, kWaitIters)) atomicOr(p.err, kErrWait);
    umma::fence_after();
}

// (thread 0, aborting CTA) wait, bounded, for the products of the last
// committed block
__device__ void wp_drain(WPipe &p)
{
    if (p.consumed > 0)
        umma::mbar_wait(p.done + (p.consumed - 1) % p.nstage, (uint32_t)((p.consumed - 1) / p.nstage) & 1u, kWaitIters);
}

// the 512 threads of the resident tile (not the copy warp)
__device__ __forceinline__ void bar_main() { asm volatile("bar.sync 2, %0;" ::"r"(kThreads) : "memory"); }

// words between two regions' keys in shared memory: odd, so that lanes
// reading consecutive regions' bits hit distinct banks
__host__ __device__ __forceinline__ int key_stride(int W) { return W | 1; }

__global__ void __launch_bounds__(kThreads + 32, 1) compose_tc_kernel(NetDev net, TcNet tc, RegionsDev reg, ChunkDev ch,
                                                                  float iso, int slots, int *err)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[4];
    __shared__ uint32_t tslot;
    __shared__ int s_last;
    __shared__ int s_abort; // a pipeline wait ran out (thread 0 or the copy warp)
    __shared__ int s_stop;  // thread 0's view of it, published before a tile barrier: uniform
    __shared__ WavePlan plan;
    __shared__ int4 ri[64]; // the tile's regions (at most 256 columns)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    long long head;
    int count;
    chunk_range(ch, head, count);
    if (count <= 0) return;
    const int KW = key_stride(net.W); // odd: lanes on consecutive regions read distinct banks
    uint8_t *base = smem_raw + ((1024u - (umma::smem_addr(smem_raw) & 1023u)) & 1023u);
    XOp X;
    X.xs = base;
    // (the layout is the widest tile's)
    uint8_t *ws = base + (size_t)(tc.kp_max / 64) * 3 * op_term_bytes(tc.ncols_max);      // nstage weight blocks
    uint32_t *keys = reinterpret_cast<uint32_t *>(ws + (size_t)tc.nstage * kWBlockBytes); // the tile's bits
    // per CTA, for every tile: linear 0 as (w0, w1, w2, b) per unit and the
    // face-plane weights (the output linear's only row)
    float4 *w0s = reinterpret_cast<float4 *>(keys + (size_t)(tc.ncols_max / 4) * key_stride(net.W));
    float *wls = reinterpret_cast<float *>(w0s + net.nodes[1]);
    float *fsum = reinterpret_cast<float *>(reinterpret_cast<uintptr_t>(wls + net.nodes[net.n_lin - 1] + 3) & ~(uintptr_t)15);
    WPipe pp{bars, bars + 2, ws, tc.nstage, err, 0, &s_abort};
    if (warp == 0) { // one tile per resident slot while the wave is small, the widest tile otherwise
        plan_wave(plan, ch, net.n_lin - 1, count, slots, tc.ncols_max / 4, 4);
        if (lane == 0) {
            s_abort = 0;
            s_stop = 0;
            for (int b = 0; b < 4; ++b) umma::mbar_init(bars + b, 1);
            umma::fence_mbar_init();
        }
    } else {
        const float *W0 = (const float *)net.W0;
        const float *b0 = (const float *)net.bias[0];
        for (int m = tid - 32; m < net.nodes[1]; m += kThreads)
            w0s[m] = make_float4(W0[3 * m], W0[3 * m + 1], W0[3 * m + 2], b0[m]);
        const int il = net.n_lin - 1;
        const float *wl = (const float *)net.Wt[il]; // [K][Mp], column 0
        for (int k = tid - 32; k < net.nodes[il]; k += kThreads) wls[k] = wl[(size_t)k * net.Mp[il]];
    }
    __syncthreads(); // the plan; barriers initialised, for the copy warp too
    const int R = plan.R, ncols = 4 * R;
    if ((int)blockIdx.x >= plan.tile0[plan.layers]) return;
    const int rounds = plan_rounds(plan, (int)gridDim.x);
    int tmem_cols = 32;
    while (tmem_cols < 2 * tc.mtiles_max * ncols) tmem_cols <<= 1;
    const size_t rstride = (size_t)net.ALLP * 4;
    X.term = op_term_bytes(ncols);
    if (warp == 0) umma::tmem_alloc(&tslot, (uint32_t)tmem_cols); // (read after a tile's barriers)
    if (warp == kThreads / 32) { // the copy warp: the weight blocks of every tile
        if (lane == 0) wp_produce(pp, net, tc, plan, rounds);
        __syncwarp();
        __syncthreads(); // the tile threads' last barrier
        return;
    }
    int g = 0; // next weight block (thread 0)
    // epilogue: warp w reads TMEM lanes 32 (w % 4).. and every (kThreads / 128)-th column block
    const int q4 = warp & 3, cgrp = warp >> 2, ngrp = kThreads / 128;

    float *cons = (float *)ch.cons;
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        const int cls = plan_class(plan, t);
        const int jend = cls > 1 ? net.hoff[cls + 1] : 0; // rows before this are in the parent's slot
        const int nreg = tile_nreg(plan, t, cls);
        bar_main(); // the previous tile is done with the keys and the operand
        if (tid < nreg) ri[tid] = tile_region(plan, reg, ch, head, t, cls, tid);
        for (int rr = warp; rr < R; rr += kThreads / 32) { // (beside it) a region's words together in flight
            const uint32_t *key = reg.keys + (size_t)(rr < nreg ? head + tile_pos(plan, ch, t, cls, rr) : 0) * net.W;
#pragma unroll 2
            for (int w = lane; w < net.W; w += 32) keys[rr * KW + w] = rr < nreg ? key[w] : 0u;
        }
        bar_main(); // every thread reads every region's bits below

        // class 1: hidden layer 1 = linear 0 rows (sign-flipped); the extra constraints
        {
            const int n1 = net.nodes[1];
            for (int rr = warp; cls == 1 && rr < nreg; rr += kThreads / 32)
                for (int m = lane; m < n1; m += 32) {
                    const float sg = key_bit(keys + (size_t)rr * KW, m) ? -1.f : 1.f;
                    const float4 w = w0s[m];
                    st4<float>(cons + (size_t)(uint32_t)ri[rr].x * rstride + (size_t)m * 4,
                               make_float4(sg * w.x, sg * w.y, sg * w.z, sg * w.w));
                }
            const float *we = (const float *)net.w_extra;
            const float *be = (const float *)net.b_extra;
            for (int q = tid; q < nreg * net.E; q += kThreads) {
                const int rr = q / net.E, e = q % net.E;
                st4<float>(cons + (size_t)(uint32_t)ri[rr].x * rstride + (size_t)(net.N + e) * 4,
                           make_float4(we[3 * e], we[3 * e + 1], we[3 * e + 2], be[e]));
            }
        }
        if (cls > 1) { // the operand of linear cls, from the parent's rows
            stage_x_from_rows(X, R, cons, rstride, ri, jend, keys, KW, nreg, net.hoff[cls], net.nodes[cls]);
        } else {
            const int n1 = net.nodes[1];
            // X_1 = diag(s_1) [W0 | b0], two regions x 32 units at a time
            for (int q = warp; q < R * ((n1 + 63) / 64); q += kThreads / 32) {
                const int kb = q / R, in = q - kb * R, k = kb * 64 + (in & 1) * 32 + lane;
                const float4 w = k < n1 ? w0s[k] : make_float4(0.f, 0.f, 0.f, 0.f);
                float x[8];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = (in >> 1) * 2 + e;
                    const bool on = r < nreg && k < n1 && key_bit(keys + (size_t)r * KW, k);
                    x[4 * e] = on ? w.x : 0.f;
                    x[4 * e + 1] = on ? w.y : 0.f;
                    x[4 * e + 2] = on ? w.z : 0.f;
                    x[4 * e + 3] = on ? w.w : 0.f;
                }
                X.put8(in >> 1, k, x);
            }
        }
        umma::fence_proxy_async();
        umma::fence_before();
        bar_main();
        umma::fence_after();
        const uint32_t tmem = tslot;

        for (int i = cls; i <= net.n_lin - 2; ++i) {
            const int M = net.nodes[i + 1];
            const int mtiles = (M + 127) / 128;
            if (warp == 0) gemm_issue(pp, tc.lin[i], mtiles, X, ncols, tmem, true, g);
            for (int s = 0; s < net.nskip[i]; ++s) {
                const SkipDev &sk = net.skip[i][s];
                if (tc_skip(sk)) {
                    // the operand is about to be overwritten: the products so far must be done
                    if (tid == 0) {
                        gemm_finish(pp, g);
                        if (*pp.abort) s_stop = 1;
                    }
                    bar_main();
                    if (s_stop) break; // written by thread 0 before the barrier: uniform
                    stage_x_from_rows(X, R, cons, rstride, ri, jend, keys, KW, nreg, net.hoff[sk.from], net.nodes[sk.from]);
                    umma::fence_proxy_async();
                    bar_main();
                    if (warp == 0) gemm_issue(pp, tc.skip[i][s], mtiles, X, ncols, tmem, false, g);
                }
            }
            // the first M tile's bias, loaded while the products run
            const float *bias = (const float *)net.bias[i];
            float bnext = q4 * 32 + lane < M ? bias[q4 * 32 + lane] : 0.f;
            if (tid == 0) {
                gemm_finish(pp, g);
                if (*pp.abort) s_stop = 1;
                s_last = g - 1;
            }
            __syncwarp();
            bar_main();
            if (s_stop) break; // no epilogue: the accumulators are not complete
            gemm_observe(pp, s_last);
            // epilogue: accumulators -> constraint rows (HBM) and the next operand (smem)
            const int Kn = (M + 63) / 64 * 64; // next operand's padded K (the face plane reads it too)
            for (int c = warp; c < R / 2; c += kThreads / 32)
                for (int k = M + lane; k < Kn; k += 32) {
                    const float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    X.put8(c, k, z);
                }
            for (int mt = 0; mt < mtiles; ++mt) {
                const int m = mt * 128 + q4 * 32 + lane;
                const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
                const float bm = bnext;
                if (mt + 1 < mtiles) bnext = m + 128 < M ? bias[m + 128] : 0.f;
                const int row = net.hoff[i + 1] + m;
                for (int cb = cgrp; cb < ncols / 16; cb += ngrp) {
                    // the four regions' slots and key words, read ahead of the accumulators
                    uint32_t slot[4], kw[4];
                    #pragma unroll
                    for (int qq = 0; qq < 4; ++qq) {
                        slot[qq] = (uint32_t)ri[cb * 4 + qq].x;
                        kw[qq] = m < M ? keys[(cb * 4 + qq) * KW + (row >> 5)] : 0u;
                    }
                    float v[16], vc[16];
                    umma::tmem_ld16x2(lane_base + (uint32_t)(mt * ncols + cb * 16),
                                      lane_base + (uint32_t)((mtiles + mt) * ncols + cb * 16), v, vc);
                    if (m >= M) continue;
                    float x[16]; // next operand, columns cb * 16 .. + 15 of row k = m
                    #pragma unroll
                    for (int qq = 0; qq < 4; ++qq) {
                        const int r = cb * 4 + qq;
                        float o[4] = {v[4 * qq] + vc[4 * qq], v[4 * qq + 1] + vc[4 * qq + 1],
                                      v[4 * qq + 2] + vc[4 * qq + 2], v[4 * qq + 3] + vc[4 * qq + 3] + bm};
                        if (net.nskip[i] && r < nreg) add_skips(net, i, m, cons, rstride, ri[r], jend, keys + (size_t)r * KW, o);
                        const bool act = r < nreg && ((kw[qq] >> (row & 31)) & 1u);
                        const float sg = act ? -1.f : 1.f;
                        if (r < nreg)
                            st4<float>(cons + (size_t)slot[qq] * rstride + (size_t)row * 4,
                                       make_float4(sg * o[0], sg * o[1], sg * o[2], sg * o[3]));
                        #pragma unroll
                        for (int c = 0; c < 4; ++c) x[4 * qq + c] = act ? o[c] : 0.f;
                    }
                    X.put8(cb * 2, m, x);
                    X.put8(cb * 2 + 1, m, x + 8);
                }
            }
            umma::fence_proxy_async();
            umma::fence_before();
            bar_main();
            umma::fence_after();
        }

        if (s_stop) break;
        // face plane: w_eq = W_L . X_L (+ b_L, + connections into the output layer)
        // in fp32 from the operand in shared memory (hi + mid + lo is exact):
        // lanes take regions (consecutive regions share operand rows), the
        // warps split K, partial sums meet in shared memory
        {
            const int i = net.n_lin - 1;
            const int K = net.nodes[i];
            const float bl = ((const float *)net.bias[i])[0];
            constexpr int kWarps = kThreads / 32;
            for (int r0 = 0; r0 < R; r0 += 32) {
                // thread (region fr of these 32, K residue fw): sixteen
                // consecutive rows of two regions per warp and step
                const int fr = 2 * warp + (lane & 1), fw = lane >> 1, r = r0 + fr;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                if (r < R)
#pragma unroll 4
                    for (int k = fw; k < K; k += kWarps) {
                        const float w = wls[k];
                        float x[4];
                        X.get4(r, k, x);
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[c] = fmaf(w, x[c], acc[c]);
                    }
                // partial sums: [residue][region][4]
                reinterpret_cast<float4 *>(fsum)[fw * 32 + fr] = make_float4(acc[0], acc[1], acc[2], acc[3]);
                bar_main();
                if (tid < 128) {
                    const int rr = tid >> 2, c = tid & 3, rg = r0 + rr;
                    float a = 0.f;
                    for (int w = 0; w < kWarps; ++w) a += fsum[(w * 32 + rr) * 4 + c];
                    if (rg < nreg) {
                        const uint32_t *key = keys + (size_t)rg * KW;
                        auto crow = [&](int row) { // component c of a constraint row
                            const float v = cons[(size_t)(uint32_t)(row < jend ? ri[rg].y : ri[rg].x) * rstride + (size_t)row * 4 + c];
                            return row == ri[rg].z ? -v : v;
                        };
                        for (int s = 0; s < net.nskip[i]; ++s) {
                            const SkipDev &sk = net.skip[i][s];
                            if (sk.kind == 0) {
                                if (sk.from >= 1 && net.nodes[sk.from] == 1 && key_bit(key, net.hoff[sk.from]))
                                    a -= crow(net.hoff[sk.from]);
                            } else if (sk.from == 0) {
                                if (c < 3) a += ((const float *)sk.tmt)[(size_t)c * sk.Mp];
                            } else {
                                const float *tt = (const float *)sk.tmt; // [dec][Mp]
                                const int hs = net.hoff[sk.from];
                                for (int k = 0; k < net.nodes[sk.from]; ++k)
                                    if (key_bit(key, hs + k)) a -= tt[(size_t)k * sk.Mp] * crow(hs + k);
                            }
                        }
                        if (c == 3) a += bl - iso;
                        ((float *)ch.eq)[(size_t)ri[rg].w * 4 + c] = a;
                    }
                }
                bar_main();
            }
        }
    } // tiles
    if (tid == 0 && *pp.abort) wp_drain(pp);
    umma::fence_before();
    __syncthreads(); // with the copy warp
    if (warp == 0) umma::tmem_dealloc(tslot, (uint32_t)tmem_cols);
}

// ---------------------------------------------------------------- streamed operand
// Wide layers: three bf16 terms of a resident K x ncols operand leave room for
// only a few regions per tile, and every tile streams all weight blocks again.
// Here the operand lives in a scratch area of device memory per CTA (in L2 while
// it is used), as the shared-memory image of its 64-deep K blocks, and is copied
// one block at a time into a two-stage ring by a copy warp of its own, as the
// weights are by another.  Sixteen row warps write it: the blocks of the layer
// the tile starts from out of the parents' rows, once per tile, and every
// later layer's in the epilogue that computes its rows.  K blocks are the outer
// loop of the products, so one block of the operand serves every M tile of a
// pass, and the tile is as wide as TMEM allows (two accumulators per M tile in
// 512 columns).  A pass's accumulators are in two halves, so that the row warps
// read out one half while the products go into the other (pass_group).
// What bounds it (measured on GB300, 3-[512]x8-1 with connections, 32 regions a
// tile): a pass of eight operand blocks takes 47 K cycles, its products 25 K.  The
// row warps' stores -- 31 bytes a cycle and SM, whoever issues them -- need 10 K
// per pass for rows and operand, mostly beside the products; the products wait
// for the first half's operand (8 K) and accumulators (4 K) around the passes'
// ends, and lose about 400 cycles per weight block to barriers between blocks.
// With the row warps rebuilding every block of every pass in shared memory from
// the rows the composition took 308 ms of a marching, this way 275 ms (a weight
// block copied once per CTA; shared by two CTAs 274); with six
// layers of 256 units 16.5 and 15.4 ms.
// The operand values, the order of the products into each accumulator and the
// epilogue and face-plane arithmetic are those of compose_tc_kernel, so both
// kernels give the same bits.
constexpr int kSBuild = 512;            // threads of the row warps (16)
constexpr int kSThreads = kSBuild + 96; // + the issuing warp and the weight- and operand-copy warps
constexpr int kSFaceSumBytes = kSBuild * 16;

__device__ __forceinline__ int jobs_of(const NetDev &net, int i)
{
    int n = 1;
    for (int s = 0; s < net.nskip[i]; ++s) n += tc_skip(net.skip[i][s]) ? 1 : 0;
    return n;
}

// product job `job` of linear i: 0 = the linear itself on hidden layer i,
// q >= 1 = its q-th tensor-core connection (a transform of an earlier layer)
__device__ const TcMat &job_mat(const NetDev &net, const TcNet &tc, int i, int job, int &src)
{
    src = i;
    if (job > 0) {
        int q = 0;
        for (int s = 0; s < net.nskip[i]; ++s)
            if (tc_skip(net.skip[i][s]) && ++q == job) {
                src = net.skip[i][s].from;
                return tc.skip[i][s];
            }
    }
    return tc.lin[i];
}

// 64-deep operand blocks of a pass over linear i: those of its product jobs
__device__ __forceinline__ int pass_blocks(const NetDev &net, const TcNet &tc, int i)
{
    int n = 0, src;
    const int njobs = jobs_of(net, i);
    for (int job = 0; job < njobs; ++job) n += job_mat(net, tc, i, job, src).Kp / 64;
    return n;
}

// Hidden layers whose operand a tile of class c needs and does not compute: c
// itself, written first, and then in ascending order the earlier ones that feed a
// tensor-core connection.
__device__ __forceinline__ uint32_t parent_operands(const NetDev &net, int cls)
{
    uint32_t mask = cls <= net.n_lin - 2 ? 1u << cls : 0u;
    for (int i = cls; i <= net.n_lin - 2; ++i)
        for (int s = 0; s < net.nskip[i]; ++s)
            if (tc_skip(net.skip[i][s]) && net.skip[i][s].from <= cls) mask |= 1u << net.skip[i][s].from;
    return mask;
}
__device__ __forceinline__ int op_blocks(const NetDev &net, int layer) { return (net.nodes[layer] + 63) / 64; }
// blocks written before layer `layer`'s, of the layers in `mask`
__device__ __forceinline__ int parent_blocks_before(const NetDev &net, uint32_t mask, int cls, int layer)
{
    if (layer == cls) return 0;
    int n = op_blocks(net, cls);
    for (int l = 1; l < layer; ++l)
        if (l != cls && ((mask >> l) & 1u)) n += op_blocks(net, l);
    return n;
}

// Operand blocks taken together, from block b of a pass of n blocks: the first
// two and the last two when the pass has tiles in both halves.  Within such a
// pair the first half's products come before the second half's, so that the
// first half's accumulators are complete two products early: their epilogue and
// the next pass's first operand blocks run under the second half's products, and
// the second half's epilogue under the next pass's first ones.  Each accumulator
// receives its products in the order of the blocks either way.
__device__ __forceinline__ int pass_group(int b, int n, bool two)
{
    return two && ((b == 0 && n >= 2) || (b == n - 2 && n >= 4)) ? 2 : 1;
}

__device__ __forceinline__ void bar_rows() { asm volatile("bar.sync 1, %0;" ::"r"(kSBuild) : "memory"); }

// Bounded wait of the streamed kernel: false at once when the CTA is
// aborting, and false -- with the error bit kErrWait and the abort flag set --
// when the wait runs out.  An aborting CTA keeps its arrive / commit / barrier
// sequence (so that no thread waits on a partner that gave up) but issues no
// copy or product and skips the epilogue work.
__device__ __forceinline__ bool swait(uint64_t *bar, uint32_t parity, int *err, volatile int *abort)
{
    // the phase test and the abort flag's load overlap (the issuing
    // thread's critical path between two blocks of products)
    const bool ready = umma::mbar_test(bar, parity);
    const int ab = *abort;
    if (ab) return false;
    if (ready || umma::mbar_wait(bar, parity, kWaitIters)) return true;
    atomicOr(err, kErrWait);
    *abort = 1;
    return false;
}

// the same decided as one warp
__device__ __forceinline__ bool wwait(uint64_t *bar, uint32_t parity, int *err, volatile int *abort)
{
    return __all_sync(0xffffffffu, swait(bar, parity, err, abort));
}

// (one thread of its own warp) the weight blocks through the nstage ring, in
// the order the products consume them -- tile, layer, group of M tiles, operand
// blocks (pass_group), half of the group, M tile --
// running ahead of the products by up to nstage blocks: block h goes into
// stage h % nstage once the products of block h - nstage have completed.
// Measured on GB300: with the copies issued from the same thread as the
// products, every block cost that thread a wait for the previous block's
// products before its refill (about as long as the 24 products themselves),
// so the tensor pipe was idle most of the time.
__device__ void produce_streamed(const NetDev &net, const TcNet &tc, uint8_t *ws, uint64_t *wfull, uint64_t *wdone,
                                 int half, const WavePlan &plan, int rounds, int *err, volatile int *abort)
{
    const int nst = tc.nstage;
    int h = 0;
    int ps = 0;        // stage of block h (h % nst) ...
    uint32_t pph = 0u; // ... and (h / nst) & 1, kept incrementally
    int last[4] = {-1, -1, -1, -1}; // the last block copied into each stage
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        for (int i = plan_class(plan, t); i <= net.n_lin - 2; ++i) {
            const int mtl = (net.nodes[i + 1] + 127) / 128, mper = (mtl + tc.mgroups - 1) / tc.mgroups;
            const int nblk = pass_blocks(net, tc, i);
            for (int mt0 = 0; mt0 < mtl; mt0 += mper) {
                const int mt1 = min(mtl, mt0 + mper), mh = min(mt1, mt0 + half);
                int job0 = 0, kb0 = 0; // block b
                for (int b = 0, gs; b < nblk; b += gs) {
                    gs = pass_group(b, nblk, mh < mt1);
                    int job = 0, kb = 0;
                    for (int part = 0; part < 2; ++part) {
                        job = job0;
                        kb = kb0;
                        for (int u = 0; u < gs; ++u) {
                            int src;
                            const TcMat &m = job_mat(net, tc, i, job, src);
                            const int kblocks = m.Kp / 64;
                            for (int mt = part ? mh : mt0; mt < (part ? mt1 : mh); ++mt, ++h) {
                                const int s = ps;
                                const uint32_t ph = pph; // phase of block h - nst's products
                                if (++ps == nst) {
                                    ps = 0;
                                    pph ^= 1u;
                                }
                                if (h >= nst && !swait(wdone + s, ph ^ 1u, err, abort)) continue;
                                if (*abort) continue;
                                umma::mbar_expect_tx(wfull + s, (uint32_t)kWBlockBytes);
                                umma::bulk_g2s(ws + (size_t)s * kWBlockBytes, m.blocks + (size_t)(mt * kblocks + kb) * kWBlockBytes,
                                               (uint32_t)kWBlockBytes, wfull + s);
                                last[s] = h;
                            }
                            if (++kb == kblocks) {
                                kb = 0;
                                ++job;
                            }
                        }
                    }
                    job0 = job;
                    kb0 = kb;
                }
            }
        }
    }
    // nothing lands in shared memory after the CTA has left: the last copy of
    // every stage (bounded)
    for (int s = 0; s < nst; ++s)
        if (last[s] >= 0) umma::mbar_wait(wfull + s, (uint32_t)(last[s] / nst) & 1u, kWaitIters);
}

// A walk over the CTA's weight blocks in the order the products take them (that
// of produce_streamed), and what each block needs and completes.
struct ProductWalk {
    int rd, i, mt0, mt1, mh, b, gs, part, u, mt; // round, linear, M tiles of the pass [mt0, mh, mt1), group, half, block of it, M tile
    int mper, mtl, nblk;
    int pass[2], xb; // passes with a first / second half, and operand blocks, before this one's
    __device__ __forceinline__ bool first_of_pass() const { return b + u == 0; }
    __device__ __forceinline__ bool new_operand() const { return part == 0 && mt == mt0; }
    __device__ __forceinline__ bool new_half() const { return b + u == 0 && mt == (part ? mh : mt0); }
    __device__ __forceinline__ bool last_of_operand() const { return mt == mt1 - 1; }
    __device__ __forceinline__ bool last_of_half() const { return b + gs == nblk && u == gs - 1 && (mt == mh - 1 || mt == mt1 - 1); }
    __device__ __forceinline__ int operand() const { return xb + u; }
    __device__ __forceinline__ int half_pass() const { return part ? pass[1] : pass[0]; }

    __device__ __forceinline__ void enter_group()
    {
        gs = pass_group(b, nblk, mh < mt1);
        part = u = 0;
        mt = mt0;
    }
    __device__ __forceinline__ void enter_pass()
    {
        mt1 = min(mtl, mt0 + mper);
        mh = min(mt1, mt0 + half_);
        b = 0;
        enter_group();
    }
    __device__ __forceinline__ void enter_layer(const NetDev &net, const TcNet &tc)
    {
        mtl = (net.nodes[i + 1] + 127) / 128;
        mper = (mtl + tc.mgroups - 1) / tc.mgroups;
        nblk = pass_blocks(net, tc, i);
        mt0 = 0;
        enter_pass();
    }
    // the first tile from round rd on that has products
    __device__ __forceinline__ bool enter_tile(const NetDev &net, const TcNet &tc, const WavePlan &plan, int rounds)
    {
        for (; rd < rounds; ++rd) {
            const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
            if (t < 0) continue;
            i = plan_class(plan, t);
            if (i > net.n_lin - 2) continue;
            enter_layer(net, tc);
            return true;
        }
        return false;
    }
    __device__ __forceinline__ bool start(const NetDev &net, const TcNet &tc, const WavePlan &plan, int rounds, int half)
    {
        half_ = half;
        rd = pass[0] = pass[1] = xb = 0;
        return enter_tile(net, tc, plan, rounds);
    }
    __device__ __forceinline__ bool next(const NetDev &net, const TcNet &tc, const WavePlan &plan, int rounds)
    {
        if (++mt < (part ? mt1 : mh)) return true;
        if (++u < gs) {
            mt = part ? mh : mt0;
            return true;
        }
        if (part == 0 && mh < mt1) {
            part = 1;
            u = 0;
            mt = mh;
            return true;
        }
        xb += gs;
        b += gs;
        if (b < nblk) {
            enter_group();
            return true;
        }
        ++pass[0];
        pass[1] += mh < mt1;
        mt0 += mper;
        if (mt0 < mtl) {
            enter_pass();
            return true;
        }
        if (++i <= net.n_lin - 2) {
            enter_layer(net, tc);
            return true;
        }
        ++rd;
        return enter_tile(net, tc, plan, rounds);
    }

private:
    int half_;
};

// (one warp, one elected lane issuing: the walk's values are the same in every
// lane, so the descriptors stay in uniform registers) the products: operand and
// weight blocks from the copy warps' rings, six products per K step into the main
// (hi.hi) and the correction accumulator of each M tile.  The tensor pipe takes
// two or three products ahead (measured on GB300: 24 products are issued in 1,495
// of the 1,766 cycles they take), so a gap of more than about 150 cycles in the
// issuing stream leaves it idle: the walk's next step and the look at the next
// block's barriers are made between the K steps, and a block's end costs a commit
// and a branch (with the bookkeeping and waits between the blocks, the pipe stood
// for 800 to 900 cycles per block of 1,536).  The commits that free the operand
// stages and publish the accumulators are made whatever happens, so that the
// row warps never wait on a partner that gave up.
__device__ void issue_streamed(const NetDev &net, const TcNet &tc, uint8_t *ws, uint64_t *wfull, uint64_t *wdone,
                               uint8_t *xs0, uint64_t *xfull, uint64_t *xdone, uint64_t *accdone, uint64_t *accfree,
                               uint32_t tmem, int ncols, int half, const WavePlan &plan, int rounds, int *err,
                               volatile int *abort)
{
    const int nst = tc.nstage;
    int consumed = 0;
    int s = 0;        // stage of weight block h (h % nst) ...
    uint32_t ph = 0u; // ... and its phase parity ((h / nst) & 1), kept incrementally
    // weight stage q's descriptor = wd0 + q * wstep (start address field)
    const uint64_t wd0 = umma::desc_sw128(umma::smem_addr(ws));
    const uint64_t wstep = (uint64_t)(kWBlockBytes >> 4);
    // operand descriptors of the two stages; term and K step (16 rows of every chunk) add constant offsets
    const uint32_t term = op_term_bytes(ncols);
    const uint64_t xd0 = umma::desc_mn(umma::smem_addr(xs0), 128u, 1024u);
    const uint64_t xu = term >> 4, xj = 16u;
    const uint32_t idesc = umma::idesc_bf16_bmn(128, ncols);
    ProductWalk w;
    bool more = w.start(net, tc, plan, rounds, half);
    bool ready = false, ok = true;
    int last_s = 0;
    uint32_t last_ph = 0u;
    while (more) {
        const int xs = w.operand() & 1;
        if (w.new_operand()) ok = true;
        if (!ready) { // in order: the block's waits that apply (seen before, when ready)
            if (w.new_half() && w.half_pass() > 0) ok = wwait(accfree + w.part, (uint32_t)(w.half_pass() - 1) & 1u, err, abort) && ok;
            if (w.new_operand()) ok = wwait(xfull + xs, (uint32_t)(w.operand() >> 1) & 1u, err, abort) && ok;
            ok = wwait(wfull + s, ph, err, abort) && ok;
        }
        umma::fence_after();
        const uint32_t d_main = tmem + (uint32_t)(2 * (w.mt - w.mt0) * ncols), d_corr = d_main + (uint32_t)ncols;
        const uint64_t ad = wd0 + wstep * (uint64_t)s; // term t at +16 KB, K step j at +32 B
        const uint64_t xd = xd0 + (uint64_t)xs * (3u * xu);
        const bool fresh = w.first_of_pass();
        const bool xlast = w.last_of_operand(), hlast = w.last_of_half();
        const uint32_t abar = umma::smem_addr(accdone + w.part);
        const uint32_t xbar = umma::smem_addr(xdone + xs), wbar = umma::smem_addr(wdone + s);
        const bool go = ok;
        if (go && umma::elect()) issue_step(d_main, d_corr, ad, xd, xu, idesc, fresh);
        __syncwarp();
        if (go) ++consumed;
        const int s_last = s;
        const uint32_t ph_last = ph;
        if (++s == nst) {
            s = 0;
            ph ^= 1u;
        }
        more = w.next(net, tc, plan, rounds);
        if (go && umma::elect()) issue_step(d_main, d_corr, ad + 2u, xd + xj, xu, idesc, false);
        __syncwarp();
        ready = go && more && umma::mbar_test(wfull + s, ph);
        if (ready && w.new_operand()) ready = umma::mbar_test(xfull + (w.operand() & 1), (uint32_t)(w.operand() >> 1) & 1u);
        if (ready && w.new_half() && w.half_pass() > 0) ready = umma::mbar_test(accfree + w.part, (uint32_t)(w.half_pass() - 1) & 1u);
        ready = __all_sync(0xffffffffu, ready);
        if (go && umma::elect()) issue_step(d_main, d_corr, ad + 4u, xd + 2u * xj, xu, idesc, false);
        __syncwarp();
        if (umma::elect()) {
            if (go) {
                issue_step(d_main, d_corr, ad + 6u, xd + 3u * xj, xu, idesc, false);
                umma::commit(wbar); // the copy warp may refill the stage
            }
            if (xlast) umma::commit(xbar); // the operand stage is free once these complete
            if (hlast) umma::commit(abar); // the half's accumulators are complete
        }
        __syncwarp();
        if (go) {
            last_s = s_last;
            last_ph = ph_last;
        }
    }
    // the last products have completed before TMEM is released
    if (consumed > 0 && !umma::mbar_wait(wdone + last_s, last_ph, kWaitIters)) atomicOr(err, kErrWait);
}

// Progress of the row warps, for the operand copy, a count per warp: [0] operand
// blocks written from the parents' rows, [1], [2] passes whose first / second half
// has been read out and written.  (Counts and not barrier phases: the copy may
// look at one long after the next has been raised.)
struct Progress {
    uint32_t n[3][kSBuild / 32];
};
__device__ __forceinline__ void progress_set(uint32_t *c, uint32_t v)
{
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(umma::smem_addr(c)), "r"(v) : "memory");
}
// (one warp) every row warp has reached `target`
__device__ __forceinline__ bool progress_wait(const uint32_t *c, uint32_t target, int *err, volatile int *abort)
{
    const uint32_t mine = umma::smem_addr(c + (threadIdx.x & (kSBuild / 32 - 1)));
    for (int it = 0; it < kWaitIters; ++it) {
        uint32_t v;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(mine) : "memory");
        if (__all_sync(0xffffffffu, (int32_t)(v - target) >= 0)) return true;
        if (__any_sync(0xffffffffu, *abort != 0)) return false;
        __nanosleep(32);
    }
    if ((threadIdx.x & 31) == 0) atomicOr(err, kErrWait);
    *abort = 1;
    return false;
}

// (a warp of its own, one lane copying) the operand blocks through the two-stage ring, in
// the order the products consume them, each once the row warps have written it
// and the stage is free.  Rows written by other threads are read here by the
// copy engine: every writer fences (generic to async proxy) before its warp counts.
__device__ void copy_operand(const NetDev &net, const TcNet &tc, uint8_t *xs0, uint64_t *xfull, uint64_t *xdone,
                             const Progress &prog, const uint8_t *xg, int ncols, int half, const WavePlan &plan,
                             int rounds, int *err, volatile int *abort)
{
    const uint32_t bytes = 3u * op_term_bytes(ncols);
    const bool lead = (threadIdx.x & 31) == 0;
    int xb = 0;
    uint32_t pass = 0, conv = 0;
    int last0 = -1, last1 = -1; // the last block copied into each stage
    for (int rd = 0; rd < rounds; ++rd) {
        const int t = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
        if (t < 0) continue;
        const int cls = plan_class(plan, t);
        const uint32_t mask = parent_operands(net, cls);
        uint32_t prev_pass = 0;
        int prev_mper = 1;
        for (int i = cls; i <= net.n_lin - 2; ++i) {
            const int mtl = (net.nodes[i + 1] + 127) / 128, mper = (mtl + tc.mgroups - 1) / tc.mgroups;
            const uint32_t layer_pass = pass;
            const int njobs = jobs_of(net, i);
            for (int mt0 = 0; mt0 < mtl; mt0 += mper, ++pass)
                for (int job = 0; job < njobs; ++job) {
                    int src;
                    const int nkb = job_mat(net, tc, i, job, src).Kp / 64;
                    const uint32_t before = src <= cls ? conv + (uint32_t)parent_blocks_before(net, mask, cls, src) : 0u;
                    for (int kb = 0; kb < nkb; ++kb, ++xb) {
                        const int xs = xb & 1, fl = xb >> 1;
                        bool ok = fl < 1 || wwait(xdone + xs, (uint32_t)(fl - 1) & 1u, err, abort);
                        if (ok && mt0 == 0) {
                            if (src <= cls) {
                                ok = progress_wait(prog.n[0], before + (uint32_t)kb + 1u, err, abort);
                            } else if (job == 0) { // the M tile of linear i - 1 that computes these rows
                                const int mt = kb / 2, g = mt / prev_mper, part = mt - g * prev_mper >= half ? 1 : 0;
                                ok = progress_wait(prog.n[1 + part], prev_pass + (uint32_t)g + 1u, err, abort);
                            } // (a connection's source was complete before the job before it)
                        }
                        if (!ok) continue;
                        if (lead) {
                            umma::mbar_expect_tx(xfull + xs, bytes);
                            uint8_t *dst = xs0 + (size_t)xs * bytes;
                            const uint8_t *from = xg + tc.xoff[src] + (size_t)kb * bytes;
                            for (uint32_t q = 0; q < bytes; q += bytes / 3) umma::bulk_g2s(dst + q, from + q, bytes / 3, xfull + xs);
                        }
                        __syncwarp();
                        if (xs) last1 = xb;
                        else last0 = xb;
                    }
                }
            prev_pass = layer_pass;
            prev_mper = mper;
        }
        for (int l = 1; l <= cls; ++l)
            if ((mask >> l) & 1u) conv += (uint32_t)op_blocks(net, l);
    }
    // nothing lands in shared memory after the CTA has left (bounded)
    if (last0 >= 0) umma::mbar_wait(xfull, (uint32_t)(last0 >> 1) & 1u, kWaitIters);
    if (last1 >= 0) umma::mbar_wait(xfull + 1, (uint32_t)(last1 >> 1) & 1u, kWaitIters);
}

__global__ void __launch_bounds__(kSThreads, 1) compose_tcs_kernel(NetDev net, TcNet tc, RegionsDev reg, ChunkDev ch,
                                                                    float iso, int slots, int *err)
{
    extern __shared__ uint8_t smem_raw[];
    // wfull[3], wdone[3] (weight ring), xfull[2], xdone[2] (operand ring), accdone[2], accfree[2] (per half)
    __shared__ uint64_t bars[14];
    __shared__ Progress prog;
    __shared__ uint32_t tslot;
    __shared__ int s_abort; // a wait ran out: nothing more is issued, epilogues are skipped
    __shared__ WavePlan plan;
    __shared__ int4 ri[64]; // the tile's regions (at most 256 columns)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    long long head;
    int count;
    chunk_range(ch, head, count);
    if (count <= 0) return;
    // one tile per resident slot while the wave is small, the widest tile otherwise
    if (warp == 0) plan_wave(plan, ch, net.n_lin - 1, count, slots, tc.ncols_max / 4, 4);
    __syncthreads();
    const int R = plan.R, ncols = 4 * R;
    if ((int)blockIdx.x >= plan.tile0[plan.layers]) return;
    const int rounds = plan_rounds(plan, (int)gridDim.x);
    int tmem_cols = 32;
    const int mper_max = (tc.mtiles_max + tc.mgroups - 1) / tc.mgroups;
    while (tmem_cols < 2 * mper_max * ncols) tmem_cols <<= 1;
    const int half = (mper_max + 1) / 2; // M tiles of a group's first half
    const size_t rstride = (size_t)net.ALLP * 4;
    const int KW = key_stride(net.W); // odd: lanes on consecutive regions read distinct banks

    uint8_t *base = smem_raw + ((1024u - (umma::smem_addr(smem_raw) & 1023u)) & 1023u);
    const uint32_t term = op_term_bytes(ncols); // one term of one K block of the operand
    uint8_t *xs0 = base;                        // two stages of hi, mid, lo
    uint8_t *xg = tc.xbuf + (size_t)blockIdx.x * tc.xcta;
    uint8_t *ws = base + 6 * (size_t)term;
    uint32_t *keys = reinterpret_cast<uint32_t *>(ws + (size_t)tc.nstage * kWBlockBytes);
    float4 *w0s = reinterpret_cast<float4 *>(keys + (size_t)(tc.ncols_max / 4) * key_stride(net.W));
    float *wls = reinterpret_cast<float *>(w0s + net.nodes[1]);
    // the face plane's partial sums use the operand ring: it is idle then
    // (the tile's products are complete, the next tile's operand not begun)
    float *fsum = reinterpret_cast<float *>(base);
    uint64_t *wfull = bars, *wdone = bars + 3, *xfull = bars + 6, *xdone = bars + 8, *accdone = bars + 10, *accfree = bars + 12;

    volatile int *abort = &s_abort;
    if (tid == 0) {
        s_abort = 0;
        for (int b = 0; b < 3; ++b) {
            umma::mbar_init(wfull + b, 1);
            umma::mbar_init(wdone + b, 1);
        }
        umma::mbar_init(xfull, 1);
        umma::mbar_init(xfull + 1, 1);
        umma::mbar_init(xdone, 1);
        umma::mbar_init(xdone + 1, 1);
        umma::mbar_init(accdone, 1);
        umma::mbar_init(accdone + 1, 1);
        umma::mbar_init(accfree, kSBuild / 32); // (one arrival per row warp)
        umma::mbar_init(accfree + 1, kSBuild / 32);
        for (int w = 0; w < kSBuild / 32; ++w) prog.n[0][w] = prog.n[1][w] = prog.n[2][w] = 0u;
        umma::fence_mbar_init();
    }
    if (warp == 0) umma::tmem_alloc(&tslot, (uint32_t)tmem_cols);
    {
        const float *W0 = (const float *)net.W0;
        const float *b0 = (const float *)net.bias[0];
        for (int m = tid; m < net.nodes[1]; m += kSThreads)
            w0s[m] = make_float4(W0[3 * m], W0[3 * m + 1], W0[3 * m + 2], b0[m]);
        const int il = net.n_lin - 1;
        const float *wl = (const float *)net.Wt[il]; // [K][Mp], column 0
        for (int k = tid; k < net.nodes[il]; k += kSThreads) wls[k] = wl[(size_t)k * net.Mp[il]];
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tslot;

    if (warp == kSBuild / 32) {
        issue_streamed(net, tc, ws, wfull, wdone, xs0, xfull, xdone, accdone, accfree, tmem, ncols, half, plan,
                       rounds, err, abort);
        __syncwarp(); // the warp reaches the block barrier below converged
    } else if (warp == kSBuild / 32 + 1) {
        if (lane == 0) produce_streamed(net, tc, ws, wfull, wdone, half, plan, rounds, err, abort);
        __syncwarp();
    } else if (warp == kSBuild / 32 + 2) {
        copy_operand(net, tc, xs0, xfull, xdone, prog, xg, ncols, half, plan, rounds, err, abort);
        __syncwarp();
    } else {
        // the row warps: operand blocks from the parents' rows, epilogues, the face plane
        const int q4 = warp & 3, cgrp = warp >> 2, ngrp = kSBuild / 128;
        uint32_t pass = 0, pass1 = 0, nconv = 0; // passes read out, those of two halves, operand blocks written from parents' rows
        float *cons = (float *)ch.cons;
        for (int rd = 0; rd < rounds; ++rd) {
            const int tile = plan_tile(plan, rd, (int)blockIdx.x, (int)gridDim.x);
            if (tile < 0) continue;
            const int cls = plan_class(plan, tile);
            const int jend = cls > 1 ? net.hoff[cls + 1] : 0; // rows before this are in the parent's slot
            const int nreg = tile_nreg(plan, tile, cls);
            bar_rows(); // the previous tile is done with the keys
            if (tid < nreg) ri[tid] = tile_region(plan, reg, ch, head, tile, cls, tid);
            for (int rr = warp; rr < R; rr += kSBuild / 32) { // (beside it) a region's words together in flight
                const uint32_t *key = reg.keys + (size_t)(rr < nreg ? head + tile_pos(plan, ch, tile, cls, rr) : 0) * net.W;
#pragma unroll 4
                for (int w = lane; w < net.W; w += 32) keys[rr * KW + w] = rr < nreg ? key[w] : 0u;
            }
            bar_rows();
            // class 1: hidden layer 1 = linear 0 rows (sign-flipped); the extra constraints
            const int n1 = net.nodes[1];
            for (int rr = warp; cls == 1 && rr < nreg; rr += kSBuild / 32)
                for (int m = lane; m < n1; m += 32) {
                    const float sg = key_bit(keys + (size_t)rr * KW, m) ? -1.f : 1.f;
                    const float4 w = w0s[m];
                    st4<float>(cons + (size_t)(uint32_t)ri[rr].x * rstride + (size_t)m * 4,
                               make_float4(sg * w.x, sg * w.y, sg * w.z, sg * w.w));
                }
            const float *we = (const float *)net.w_extra;
            const float *be = (const float *)net.b_extra;
            for (int q = tid; q < nreg * net.E; q += kSBuild) {
                const int rr = q / net.E, e = q % net.E;
                st4<float>(cons + (size_t)(uint32_t)ri[rr].x * rstride + (size_t)(net.N + e) * 4,
                           make_float4(we[3 * e], we[3 * e + 1], we[3 * e + 2], be[e]));
            }
            bar_rows(); // layer-1 rows written by every row warp

            // The operand of the layers the parents computed:
            // X[4r + c][k] = s_k(r) ? -C[r][k][c] : 0, block by block.  A warp
            // item is two regions x 32 rows, a row per lane: loads and stores of
            // 512 contiguous bytes.  Two items' rows are loaded before the two
            // before them are stored.  Raw values are kept and signed when
            // stored; `other` marks the rows whose sign is the other one (the
            // plane the region was entered through).
            const int cpb = ((R + 15) / 16 + 1) / 2; // chunks of two items per warp and block
            const uint32_t xblk = 3u * term;
            const uint32_t pmask = parent_operands(net, cls);
            for (uint32_t left = pmask; left;) {
                const int layer = (left >> cls) & 1u ? cls : __ffs(left) - 1;
                left &= ~(1u << layer);
                const int K = net.nodes[layer], rows0 = net.hoff[layer];
                const bool par = rows0 < jend;
                auto load = [&](int kb, int j, float4 *v) {
                    unsigned other = 0u;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int q = warp + 16 * (2 * j + (u >> 1)), r = (q >> 1) * 2 + (u & 1);
                        const int k = kb * 64 + (q & 1) * 32 + lane;
                        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (r < nreg && k < K && key_bit(keys + (size_t)r * KW, rows0 + k)) {
                            const int4 g = ri[r];
                            if (rows0 + k == g.z) other |= 1u << u;
                            v[u] = ld4<float>(cons + (size_t)(uint32_t)(par ? g.y : g.x) * rstride + (size_t)(rows0 + k) * 4);
                        }
                    }
                    return other;
                };
                const int n = op_blocks(net, layer) * cpb;
                float4 a[4], b[4];
                unsigned ao = load(0, 0, a), bo = 0u;
                int kb = 0, j = 0;
                for (int c = 0; c < n; ++c) {
                    const int k0 = kb, j0 = j;
                    if (++j == cpb) {
                        j = 0;
                        ++kb;
                    }
                    if (c + 1 < n) bo = load(kb, j, b);
                    uint8_t *blk = xg + tc.xoff[layer] + (size_t)k0 * xblk;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int q = warp + 16 * (2 * j0 + u);
                        if (q >= R) continue;
                        const float s0 = (ao >> (2 * u)) & 1u ? 1.f : -1.f, s1 = (ao >> (2 * u + 1)) & 1u ? 1.f : -1.f;
                        const float x[8] = {s0 * a[2 * u].x,     s0 * a[2 * u].y,     s0 * a[2 * u].z,     s0 * a[2 * u].w,
                                            s1 * a[2 * u + 1].x, s1 * a[2 * u + 1].y, s1 * a[2 * u + 1].z, s1 * a[2 * u + 1].w};
                        op_put8(blk, term, q >> 1, (q & 1) * 32 + lane, x);
                    }
                    if (j == 0) { // the block's last chunk
                        ++nconv;
                        // (the fence waits for the stores: later blocks two together)
                        if (k0 < 4 || (k0 & 1) == 1 || c + 1 == n) {
                            umma::fence_proxy_async_all();
                            __syncwarp();
                            if (lane == 0) progress_set(&prog.n[0][warp], nconv);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) a[u] = b[u];
                    ao = bo;
                }
            }
            // The epilogue of a half pass reads its accumulators (warp w: TMEM
            // lanes 32 (w % 4).., column blocks cgrp, cgrp + ngrp, ... of each M
            // tile), and stores their rows and the next layer's operand.
            const int ncb = ncols / 16;
            const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
            for (int i = cls; i <= net.n_lin - 2; ++i) {
                const int M = net.nodes[i + 1], mtiles = (M + 127) / 128;
                const int mper = (mtiles + tc.mgroups - 1) / tc.mgroups;
                const float *bias = (const float *)net.bias[i];
                uint8_t *xl = i < net.n_lin - 2 ? xg + tc.xoff[i + 1] : nullptr;
                const int Kx = (M + 63) / 64 * 64; // operand rows, zero beyond M
                for (int part = 0, mt0 = 0; mt0 < mtiles;) {
                    const int e1 = min(mtiles, mt0 + mper), eh = min(e1, mt0 + half);
                    const int ma = part ? eh : mt0, mb = part ? e1 : eh;
                    const int mA = ma * 128 + q4 * 32 + lane;
                    const float bA = ma < mb && mA < M ? bias[mA] : 0.f; // loaded while the products run
                    // the half's products are in TMEM; the TMEM loads below are
                    // warp-collective, so the warp decides as one
                    bool acc_ok = swait(accdone + part, (part ? pass1 : pass) & 1u, err, abort);
                    acc_ok = __all_sync(0xffffffffu, acc_ok) && !__any_sync(0xffffffffu, *abort != 0);
                    umma::fence_after();
                    // accumulators -> registers: main + correction, sixteen columns
                    // at a time; once the half's last ones are out, the products
                    // may overwrite it.  Then + bias and connections -> rows and
                    // the next operand.
                    int c = cgrp, mt = ma;
                    bool have = acc_ok && ma < mb && c < ncb;
                    if (!have) {
                        umma::fence_before();
                        __syncwarp();
                        if (lane == 0) umma::mbar_arrive(accfree + part);
                    }
                    while (have) {
                        const int c0 = c, m = mt * 128 + q4 * 32 + lane, row = net.hoff[i + 1] + m;
                        const float bm = mt == ma ? bA : (m < M ? bias[m] : 0.f);
                        uint8_t *xrow = xl && m < Kx ? xl + (size_t)(m >> 6) * xblk : nullptr;
                        float *rowp = cons + (size_t)row * 4;
                        const int lim = m < M ? nreg : 0; // regions with a row here
                        // the four regions' slots and key bits, read ahead of the accumulators
                        uint32_t slot[4];
                        unsigned acts = 0u;
#pragma unroll
                        for (int qq = 0; qq < 4; ++qq) {
                            slot[qq] = (uint32_t)ri[c0 * 4 + qq].x;
                            if (c0 * 4 + qq < lim && key_bit(keys + (size_t)(c0 * 4 + qq) * KW, row)) acts |= 1u << qq;
                        }
                        float sum[4][4];
                        {
                            const uint32_t ta = lane_base + (uint32_t)(2 * (mt - mt0) * ncols + c0 * 16);
                            float vc[16];
                            umma::tmem_ld16x2(ta, ta + (uint32_t)ncols, &sum[0][0], vc);
#pragma unroll
                            for (int e = 0; e < 16; ++e) sum[e >> 2][e & 3] += vc[e];
                        }
                        c += ngrp;
                        if (c >= ncb) {
                            c = cgrp;
                            have = ++mt < mb;
                        }
                        if (!have) {
                            umma::fence_before(); // TMEM read out before the next products overwrite it
                            __syncwarp();
                            if (lane == 0) umma::mbar_arrive(accfree + part);
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float x[8];
#pragma unroll
                            for (int q2 = 0; q2 < 2; ++q2) {
                                const int qq = 2 * h + q2, r = c0 * 4 + qq;
                                float(&o)[4] = sum[qq];
                                o[3] += bm;
                                const bool act = (acts >> qq) & 1u;
                                if (r < lim) {
                                    if (net.nskip[i])
                                        add_skips(net, i, m, cons, rstride, ri[r], jend, keys + (size_t)r * KW, o);
                                    const float sg = act ? -1.f : 1.f;
                                    st4<float>(rowp + (size_t)slot[qq] * rstride, make_float4(sg * o[0], sg * o[1], sg * o[2], sg * o[3]));
                                }
#pragma unroll
                                for (int e = 0; e < 4; ++e) x[4 * q2 + e] = act ? o[e] : 0.f;
                            }
                            if (xrow) op_put8(xrow, term, c0 * 2 + h, m & 63, x);
                        }
                    }
                    umma::fence_proxy_async_all(); // the operand's rows, for the copy
                    __syncwarp();
                    if (lane == 0) progress_set(&prog.n[1 + part][warp], pass + 1u);
                    if (part == 0 && eh < e1) {
                        part = 1;
                    } else {
                        pass1 += part;
                        ++pass;
                        part = 0;
                        mt0 += mper;
                    }
                }
                bar_rows(); // rows of hidden layer i + 1 written by every row warp
            }

            // face plane: w_eq = W_L . X_L, X_L = -C of the last hidden layer
            // where active; lanes take regions, the warps split K, partial
            // sums meet in shared memory (the order of compose_tc_kernel)
            {
                const int i = net.n_lin - 1;
                const int K = net.nodes[i], rows0 = net.hoff[i];
                const float bl = ((const float *)net.bias[i])[0];
                constexpr int kWarps = kSBuild / 32;
                const bool live = !*abort; // per thread: the barriers below are kept either way
                for (int r0 = 0; r0 < R; r0 += 32) {
                    // thread (region fr of these 32, K residue fw): sixteen
                    // consecutive rows of two regions per warp and step
                    const int fr = 2 * warp + (lane & 1), fw = lane >> 1, r = r0 + fr;
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    if (live && r < nreg) {
                        const int4 g = ri[r];
                        const float *cr = cons + (size_t)(uint32_t)(rows0 < jend ? g.y : g.x) * rstride + (size_t)rows0 * 4;
#pragma unroll 4
                        for (int k = fw; k < K; k += kWarps) {
                            const float w = wls[k];
                            float x[4] = {0.f, 0.f, 0.f, 0.f};
                            if (key_bit(keys + (size_t)r * KW, rows0 + k)) {
                                const float4 c = ld4<float>(cr + (size_t)k * 4);
                                x[0] = -c.x, x[1] = -c.y, x[2] = -c.z, x[3] = -c.w;
                            }
                            const float wk = rows0 + k == g.z ? -w : w; // (the parent's sign)
#pragma unroll
                            for (int c = 0; c < 4; ++c) acc[c] = fmaf(wk, x[c], acc[c]);
                        }
                    }
                    reinterpret_cast<float4 *>(fsum)[fw * 32 + fr] = make_float4(acc[0], acc[1], acc[2], acc[3]);
                    bar_rows();
                    if (live && tid < 128) {
                        const int rr = tid >> 2, c = tid & 3, rg = r0 + rr;
                        float a = 0.f;
                        for (int w = 0; w < kWarps; ++w) a += fsum[(w * 32 + rr) * 4 + c];
                        if (rg < nreg) {
                            const uint32_t *key = keys + (size_t)rg * KW;
                            auto crow = [&](int row) { // component c of a constraint row
                                const float v = cons[(size_t)(uint32_t)(row < jend ? ri[rg].y : ri[rg].x) * rstride + (size_t)row * 4 + c];
                                return row == ri[rg].z ? -v : v;
                            };
                            for (int s = 0; s < net.nskip[i]; ++s) {
                                const SkipDev &sk = net.skip[i][s];
                                if (sk.kind == 0) {
                                    if (sk.from >= 1 && net.nodes[sk.from] == 1 && key_bit(key, net.hoff[sk.from]))
                                        a -= crow(net.hoff[sk.from]);
                                } else if (sk.from == 0) {
                                    if (c < 3) a += ((const float *)sk.tmt)[(size_t)c * sk.Mp];
                                } else {
                                    const float *tt = (const float *)sk.tmt; // [dec][Mp]
                                    const int hs = net.hoff[sk.from];
                                    for (int k = 0; k < net.nodes[sk.from]; ++k)
                                        if (key_bit(key, hs + k)) a -= tt[(size_t)k * sk.Mp] * crow(hs + k);
                                }
                            }
                            if (c == 3) a += bl - iso;
                            ((float *)ch.eq)[(size_t)ri[rg].w * 4 + c] = a;
                        }
                    }
                    bar_rows();
                }
            }
        }
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tslot, (uint32_t)tmem_cols);
}

// src (M x K fp32, row-major) -> three bf16 terms as the shared-memory image
// of 128 x 64 blocks (K-major, 128-byte swizzle), zero padding to Mp x Kp
__global__ void pack_weights_kernel(const float *src, int M, int K, int Mp, int Kp, uint8_t *dst)
{
    const long long n = (long long)Mp * Kp;
    const int kblocks = Kp / 64;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int m = (int)(q / Kp), k = (int)(q % Kp);
        const float v = (m < M && k < K) ? src[(size_t)m * K + k] : 0.f;
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        const float r1 = v - __bfloat162float(h);
        const __nv_bfloat16 md = __float2bfloat16_rn(r1);
        const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(md));
        const int mt = m >> 7, r = m & 127, kb = k >> 6, kk = k & 63;
        uint8_t *blk = dst + (size_t)(mt * kblocks + kb) * kWBlockBytes;
        const uint32_t off = (uint32_t)(r * 128 + ((((kk >> 3) ^ (r & 7)) & 7) << 4) + ((kk & 7) << 1));
        *reinterpret_cast<__nv_bfloat16 *>(blk + off) = h;
        *reinterpret_cast<__nv_bfloat16 *>(blk + 16384 + off) = md;
        *reinterpret_cast<__nv_bfloat16 *>(blk + 32768 + off) = lo;
    }
}

} // namespace

int device_sms()
{
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms[dev] = n > 0 ? n : 148;
    }
    return sms[dev];
}

size_t tc_smem_bytes(const TcNet &tc, int ncols, int W)
{
    if (tc.streamed) { // two operand stages of one K block each (the face-plane sums reuse them)
        return 1024 + std::max<size_t>(6 * (size_t)op_term_bytes(ncols), (size_t)kSFaceSumBytes) + (size_t)tc.nstage * kWBlockBytes +
               (size_t)(tc.ncols_max / 4) * key_stride(W) * 4 + 16 * (size_t)tc.n1 + 4 * (size_t)tc.k_last + 16;
    }
    return 1024 + (size_t)(tc.kp_max / 64) * 3 * op_term_bytes(ncols) + (size_t)tc.nstage * kWBlockBytes + (size_t)(tc.ncols_max / 4) * key_stride(W) * 4 +
           16 * (size_t)tc.n1 + 4 * (size_t)tc.k_last + 16 + (size_t)kFaceSumBytes;
}

size_t tc_smem_cap()
{
    static const size_t own = [] { // (a rounded figure would refuse widths that fit: a layer of 8,192 units has 464 bytes to spare)
        cudaFuncAttributes a = {}, b = {};
        if (cudaFuncGetAttributes(&a, compose_tc_kernel) != cudaSuccess || cudaFuncGetAttributes(&b, compose_tcs_kernel) != cudaSuccess) {
            cudaGetLastError();
            return (size_t)2048;
        }
        return std::max(a.sharedSizeBytes, b.sharedSizeBytes);
    }();
    return 227u * 1024u - own;
}

void launch_compose_tc(const NetDev &net, const TcNet &tc, const RegionsDev &reg, const ChunkDev &ch, double iso,
                       int *d_err, cudaStream_t st)
{
    if (!ch.ctl && ch.count <= 0) return;
    const int sms = device_sms();
    const size_t smem = tc_smem_bytes(tc, tc.ncols_max, net.W);
    const int slots = sms; // one resident tile per SM, the wave's tiles strided over them
    if (tc.streamed) {
        cudaFuncSetAttribute(compose_tcs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        const int grid = std::min(slots, tc.xctas);
        compose_tcs_kernel<<<grid, kSThreads, smem, st>>>(net, tc, reg, ch, (float)iso, grid, d_err);
        return;
    }
    cudaFuncSetAttribute(compose_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    compose_tc_kernel<<<slots, kThreads + 32, smem, st>>>(net, tc, reg, ch, (float)iso, slots, d_err);
}

void launch_pack_weights(const float *src, int M, int K, int Mp, int Kp, void *dst, cudaStream_t st)
{
    const long long n = (long long)Mp * Kp;
    if (n <= 0) return;
    const int grid = (int)std::min<long long>((n + 255) / 256, 4096);
    pack_weights_kernel<<<grid, 256, 0, st>>>(src, M, K, Mp, Kp, (uint8_t *)dst);
}

} // namespace am
