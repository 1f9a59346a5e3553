// am_polygon.cu -- face polygon of every region of a wave, a warp per face,
// plus the frontier insert of its neighbours.
//
// The face of a region is the polygon {x : w_eq.x + b_eq = 0, C_k(x) <= 0 for
// all k}.  The reference finds it by a pivot walk that tries candidate planes
// in order of distance from a seed point, one 3x3 solve plus an N-row
// feasibility scan per candidate, one candidate per region per round with a
// host round trip between rounds (backend/inc/kernel.h:1258-1320).  Here one
// warp owns a face and the walk is ray shooting along the current edge line: a
// pass over the rows gives the first plane the line hits, and the vertex is the
// 3x3 solve of (edge plane, hit plane, face plane).  The walk goes
// counter-clockwise about w_eq, which is the orientation the reference's
// correctNormalDirection enforces (kernel.h:1325-1370).  Zero-length edges
// (vertices closer than FP_SAME_EPS in L1) are merged and spawn no neighbour,
// as in cudaUpdateVert_kernel (kernel.h:1197-1205).
//
// The near list.  A face is small against the distance of most of its rows'
// planes, so the warp streams the rows once from global memory, keeps the
// normalised rows of the planes within a distance T of the walk's start point p
// in shared memory (about kTarget of them, at most kList) and walks over those.
// A row left out has a plane farther than T from p, so within the ball of
// radius D < T around p it is neither violated, nor near zero, nor hit: every
// decision of the walk is the one over all rows as long as the walk's points
// stay in the ball, which is checked at every step (see ball_radius for the
// margin).  T comes from the parent's count, scaled (a plane count in a ball
// grows with its radius); a seed's from a first pass over the rows.  A walk that
// leaves its ball is repeated with a larger T, and then over every row.
//
// Which of two rows that the line hits at nearly the same parameter comes first
// is decided by rounding.  The rule is the scan's over all rows by `ways` lanes
// with two interleaved chains each: within a chain fractions are compared by
// cross products in row order, between lanes by quotient and row.  A scan over
// the list takes the smallest quotient if no other is within 1e-5 of it (any
// rule gives that row), the rule's quotient and row if the candidates within
// 1e-5 belong to different lanes, and otherwise gives up: the face is walked
// over all rows with the rule itself.
//
// Seed regions (start == -1) first find a polygon vertex exactly as the
// reference's calcStartIdx does (kernel.h:799-856): planes ordered by signed
// geometric distance from the seed point, pairs enumerated by get_i_j up to
// x = min((ALL-1)(ALL-2), 812), the first pair whose vertex satisfies every
// other constraint within FP_EPS wins.  Those pairs only involve the 57
// nearest planes, which the list holds.
//
// Every edge on a hidden unit's plane gives a neighbour: the key with that
// bit flipped.  Its hash is updated in O(1) and it is inserted into the
// region hash set (full-key comparison on fingerprint match); among equal new
// keys the smallest (parent, plane) id wins, so the result is deterministic.
#include <algorithm>
#include <cuda/atomic>
#include <cuda_runtime.h>

#include "am_device.cuh"
#include "am_internal.h"
#include "am_rules.h"

namespace am {

namespace {

constexpr int kList = 128;      // rows of the near list (four per lane)
constexpr int kTarget = 64;     // and how many it aims at (80 and 48 measured 1 to 7 % slower)
constexpr int kDirect = 512;    // rows up to which a walk that left its ball goes on to every row (face_slow)
constexpr int kFaceWarps = 4;   // faces per block
constexpr int kBlocks = 8;      // blocks per SM
constexpr int kUnroll = 4;      // FP32 rows per lane in flight (half as many FP64 ones)
constexpr unsigned kFull = 0xffffffffu;
constexpr int kNoHit = 0x7fffffff;

template <typename T>
__device__ __forceinline__ unsigned long long order_key(T d);
template <>
__device__ __forceinline__ unsigned long long order_key<float>(float d)
{
    if (d != d) return 0ull;
    uint32_t u = __float_as_uint(d);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return (unsigned long long)u;
}
template <>
__device__ __forceinline__ unsigned long long order_key<double>(double d)
{
    if (d != d) return 0ull;
    unsigned long long u = (unsigned long long)__double_as_longlong(d);
    u = (u >> 63) ? ~u : (u | 0x8000000000000000ull);
    return u;
}

// (key, index) pairs: a is ahead of b when its distance is larger, ties by lower index
__device__ __forceinline__ bool ahead(unsigned long long ka, int ia, unsigned long long kb, int ib)
{
    return ka > kb || (ka == kb && ia < ib);
}

__device__ __forceinline__ bool finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite_bits(double v)
{
    return ((uint32_t)(__double_as_longlong(v) >> 52) & 0x7ffu) != 0x7ffu;
}

// Products and sums with the roundings fixed, not left to the compiler's
// contraction (which depends on the code around them): they decide the walk, and
// the list and the scan over every row must agree.
__device__ __forceinline__ float mul_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_t(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
// a0 b0 + a1 b1 + a2 b2
template <typename T>
__device__ __forceinline__ T dot3(T a0, T b0, T a1, T b1, T a2, T b2)
{
    return fma_t(a2, b2, fma_t(a0, b0, mul_t(a1, b1)));
}
// a b - c d
template <typename T>
__device__ __forceinline__ T diff2(T a, T b, T c, T d)
{
    return fma_t(a, b, -mul_t(c, d));
}

// ---------------------------------------------------------------- rows
// A region's constraint rows in global memory: the first nsplit in the parent's
// slot (the plane the region was entered through with the other sign), the rest
// in its own.
template <typename TC>
struct GlobalRows {
    const vec4_t<TC> *par, *own;
    int nsplit, flip, n;
    __device__ __forceinline__ vec4_t<TC> raw(int k) const
    {
        vec4_t<TC> v = k < nsplit ? par[k] : own[k];
        if (k == flip) {
            v.x = -v.x;
            v.y = -v.y;
            v.z = -v.z;
            v.w = -v.w;
        }
        return v;
    }
    __device__ __forceinline__ vec4_t<TC> get(int k) const;
    __device__ __forceinline__ int name(int k) const { return k; }
};

// Normalised (|w| = 1, zero rows become 0.x + sign(b) inf): signed geometric
// distances are then plain dot products, the same quantity the reference's
// feasibility test computes as (w.x + b) * rsqrt(|w|^2) (kernel.h:729-795).
template <typename TC>
__device__ __forceinline__ vec4_t<TC> normalised(vec4_t<TC> v)
{
    const TC n2 = dot3(v.x, v.x, v.y, v.y, v.z, v.z);
    if (n2 > TC(0)) {
        const TC inv = rsqrt(n2); // as the reference's distance normalisation
        v.x = mul_t(v.x, inv);
        v.y = mul_t(v.y, inv);
        v.z = mul_t(v.z, inv);
        v.w = mul_t(v.w, inv);
    } else {
        v.w = v.w > TC(0) ? TC(INFINITY) : (v.w < TC(0) ? TC(-INFINITY) : TC(NAN));
    }
    return v;
}
template <typename TC>
__device__ __forceinline__ vec4_t<TC> GlobalRows<TC>::get(int k) const
{
    return normalised<TC>(raw(k));
}

// The near list of a face (shared memory); rows are named by their position.
template <typename TC>
struct NearList {
    vec4_t<TC> row[kList];
    uint16_t idx[kList];
};
template <typename TC>
struct ListRows {
    const NearList<TC> *l;
    int n;
    __device__ __forceinline__ vec4_t<TC> get(int j) const { return l->row[j]; }
    __device__ __forceinline__ int name(int j) const { return l->idx[j]; } // the row's plane
};

// The vertex of planes ra, rb and the face plane, solved by the warp: lane
// L = 0..3 (and its copies L + 4, L + 8, ...) computes Cramer's determinant
// with column L - 1 replaced by -b (L = 0: none), then divides by the lane-0
// determinant -- the same arithmetic as solve3 on one lane, in two dependent
// sequences (determinant, divide) instead of seven, which matters because the
// SM's FP64 pipe issues a warp instruction at the same cost however few lanes
// are active (for the same reason a conversion to FP64 is spread over eight
// lanes).  Every lane returns the vertex in the solve precision (V) and rounded
// to the scan precision (Vc); false if a coordinate is not finite.
template <typename TC>
__device__ __forceinline__ TC component(const vec4_t<TC> &v, int c)
{
    return c < 2 ? (c == 0 ? v.x : v.y) : (c == 2 ? v.z : v.w);
}
template <typename TC, typename TS>
__device__ __forceinline__ bool warp_solve(const vec4_t<TC> &ra, const vec4_t<TC> &rb, const TS *eqv, TS *V, TC *Vc,
                                           int lane)
{
    TS m[8] = {(TS)ra.x, (TS)ra.y, (TS)ra.z, (TS)ra.w, (TS)rb.x, (TS)rb.y, (TS)rb.z, (TS)rb.w};
    if (sizeof(TS) > sizeof(TC)) {
        const int c = lane & 7;
        const TS cs = (TS)component<TC>(c < 4 ? ra : rb, c & 3);
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = __shfl_sync(kFull, cs, j);
    }
    const int L = lane & 3;
    const TS a00 = L == 1 ? -m[3] : m[0], a01 = L == 2 ? -m[3] : m[1], a02 = L == 3 ? -m[3] : m[2];
    const TS a10 = L == 1 ? -m[7] : m[4], a11 = L == 2 ? -m[7] : m[5], a12 = L == 3 ? -m[7] : m[6];
    const TS a20 = L == 1 ? -eqv[3] : eqv[0], a21 = L == 2 ? -eqv[3] : eqv[1], a22 = L == 3 ? -eqv[3] : eqv[2];
    const TS d = det3<TS>(a00, a01, a02, a10, a11, a12, a20, a21, a22);
    const TS d0 = __shfl_sync(kFull, d, 0);
    const TS x = d / d0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        V[j] = __shfl_sync(kFull, x, j + 1);
        Vc[j] = (TC)V[j];
    }
    return finite_bits(V[0]) && finite_bits(V[1]) && finite_bits(V[2]);
}

// L1 distance test |V - P|_1 < eps.  With TS wider than TC it is decided on
// the scan-precision copies when the rounding margin allows -- Vc and Pc are
// V and P rounded to nearest, so the TC sum is within 2^-23 (|Vc|_1 + |Pc|_1)
// + 3 ulp of the exact one; 2^-21 (|Vc|_1 + |Pc|_1 + d) bounds both -- and
// returns -1 ("near") otherwise, for the caller to decide in TS.
template <typename TC, typename TS>
__device__ __forceinline__ int same_filter(const TC *Vc, TC px, TC py, TC pz, TS eps)
{
    const TC d = fabs(Vc[0] - px) + fabs(Vc[1] - py) + fabs(Vc[2] - pz);
    const TC mag = fabs(Vc[0]) + fabs(Vc[1]) + fabs(Vc[2]) + fabs(px) + fabs(py) + fabs(pz);
    const TC margin = TC(4.76837158203125e-7) * (mag + d); // 2^-21
    const TC e = (TC)eps;
    if (d >= e + margin) return 0;
    if (d + margin < e) return 1;
    return -1;
}

// ---------------------------------------------------------------- the ball
// A row left out has its plane farther than T from p, up to the rounding of the
// FP32 test: a few 1e-7 of the coordinates' size s = |p|_1 + T, which bounds the
// points of the ball and, beside their distance, the planes' offsets.  For a point x
// with |x - p| <= D its value is below -(T - D), and the edge line reaches its plane
// beyond |x - p| = T; with T - D >= D / 16 + 1e-4 s the computed quotient of such a
// row is larger than that of any hit within the ball, whatever the line's angle to
// the plane: with m = T - D, t the hit's distance (<= 2 D) and a the row's slope, the
// computed quotient is at least (a (t + m) - 1e-6 s) / (a + 5e-7) and
// (m - 1e-6 s) / (a + 5e-7), and m^2 > 5e-6 D s puts one of the two above t for every
// a (m^2 >= 4 (D / 16) (1e-4 s) = 2.5e-5 D s).  The bound goes with the scale of the
// coordinates.  The mixed form's near-zero predicates (1e-6 and 2e-6) do not: there m
// is 4e-6 more, so that a row left out is never near zero.  (With s = 1 + |p|_1, which
// does not shrink with the shape, every face of a shape of 1e-3 was walked over every
// row: 3-[128]x4-1 scaled by 1e-3, polygon phase on GB300 in float64 / mixed / float32
// 30.0 / 13.6 / 4.9 ms, with this size 9.2 / 7.7 / 1.9; at scale 1 9.2 / 3.1 / 1.9.)
struct Ball {
    float x, y, z, d2; // centre, squared radius (< 0: nothing is inside, infinite: every row is in the list)
    __device__ __forceinline__ bool in(float px, float py, float pz) const
    {
        const float dx = px - x, dy = py - y, dz = pz - z;
        return d2 == INFINITY || dx * dx + dy * dy + dz * dz <= d2; // (NaN: outside)
    }
};
__device__ __forceinline__ float coord_size(const Ball &b, float T) { return fabsf(b.x) + fabsf(b.y) + fabsf(b.z) + T; }
template <bool kPredicates> // (the mixed form)
__device__ __forceinline__ float ball_radius2(const Ball &b, float T)
{
    if (T == INFINITY) return INFINITY;
    const float D = (T - 1e-4f * coord_size(b, T) - (kPredicates ? 4e-6f : 0.f)) * (16.f / 17.f);
    return D > 0.f ? D * D : -1.f;
}

// The rows within T of the ball's centre go into the list.  The test compares
// squares, without the square root, the centre scaled by 1 / T: a row is left out
// if g < 0 and (g / T)^2 > |w|^2 (NaN: kept).  n counts them all; at most kList
// are stored (raw; finish_list normalises).
template <typename TC>
struct Sieve {
    float bx, by, bz, bw;
    NearList<TC> *list;
    int n, lane;
    __device__ __forceinline__ Sieve(const Ball &ball, float T, NearList<TC> *l, int ln) : list(l), n(0), lane(ln)
    {
        bw = 1.f / T; // (T infinite: 0, every row is kept)
        bx = ball.x * bw;
        by = ball.y * bw;
        bz = ball.z * bw;
    }
    // this lane's row of a block of 32 (k: its plane; in: there is one)
    __device__ __forceinline__ void take(const vec4_t<TC> &v, int k, bool in)
    {
        const float x = (float)v.x, y = (float)v.y, z = (float)v.z, w = (float)v.w;
        const float g = fmaf(x, bx, fmaf(y, by, fmaf(z, bz, w * bw)));
        const float n2 = fmaf(x, x, fmaf(y, y, z * z));
        const bool keep = in && !(g < 0.f && g * g > n2);
        const unsigned b = __ballot_sync(kFull, keep);
        if (b) {
            const int pos = n + __popc(b & ((1u << lane) - 1u));
            if (keep && pos < kList) {
                list->row[pos] = v;
                list->idx[pos] = (uint16_t)k;
            }
            n += __popc(b);
        }
    }
    __device__ __forceinline__ void finish() const
    {
        __syncwarp();
        for (int j = lane; j < min(n, kList); j += 32) list->row[j] = normalised<TC>(list->row[j]);
        __syncwarp();
    }
};

// A pass over the rows by plain loads (a repeat with another T: rare).  A row of zeros
// (a dead unit) is no plane -- NaN once normalised, it is never hit, near or violated --
// and is left out; the kernel's own pass keeps it, since looking for it costs every face.
template <typename TC>
__device__ int collect(const GlobalRows<TC> &g, float T, const Ball &ball, NearList<TC> *list, int lane)
{
    Sieve<TC> sv(ball, T, list, lane);
    __syncwarp();
    for (int k = lane; k - lane < g.n; k += 32) {
        const bool in = k < g.n;
        vec4_t<TC> v;
        v.x = v.y = v.z = v.w = TC(0);
        if (in) v = g.raw(k);
        sv.take(v, k, in && !(v.x == TC(0) && v.y == TC(0) && v.z == TC(0) && v.w == TC(0)));
    }
    sv.finish();
    return sv.n;
}

// The pass over a face's rows, straight from global memory, the parent's rows into
// the region's slot as well: kUnroll rows per lane in flight.  Measured on GB300
// (3-[512]x8-1, polygon phase): 4 rows and 32 warps per SM 146 ms, 8 rows and 24
// warps 158, 2 rows 151, 40 warps 158; a per-warp ring of bulk copies into shared
// memory with the next face's chunks under way, 226 (its state spilled).
template <typename TC, bool kCopy>
__device__ __forceinline__ void stream_part(const vec4_t<TC> *src, vec4_t<TC> *copy, int k0, int k1, int flip, Sieve<TC> &sv)
{
    constexpr int U = sizeof(TC) == 4 ? kUnroll : kUnroll / 2;
    const int lane = sv.lane;
    for (; k0 < k1; k0 += 32 * U) {
        vec4_t<TC> v[U];
        const vec4_t<TC> *s = src + k0 + lane;
        if (k0 + 32 * U <= k1) {
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = s[32 * u];
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u].x = v[u].y = v[u].z = v[u].w = TC(0);
                if (k0 + 32 * u + lane < k1) v[u] = s[32 * u];
            }
        }
        if (kCopy) { // (the plane the region was entered through is a parent's row)
            if (flip >= k0 && flip < k0 + 32 * U) {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k0 + 32 * u + lane == flip) {
                        v[u].x = -v[u].x;
                        v[u].y = -v[u].y;
                        v[u].z = -v[u].z;
                        v[u].w = -v[u].w;
                    }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + 32 * u + lane < k1) copy[k0 + 32 * u + lane] = v[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) sv.take(v[u], k0 + 32 * u + lane, k0 + 32 * u + lane < k1);
    }
}

// the list position of plane k (in the list)
template <typename TC>
__device__ __forceinline__ int position(const NearList<TC> *list, int n, int k, int lane)
{
    for (int j = 0; j < n; j += 32) {
        const unsigned b = __ballot_sync(kFull, j + lane < n && (int)list->idx[j + lane] == k);
        if (b) return j + __ffs(b) - 1;
    }
    return -1;
}

// A radius that holds about kTarget rows: every lane's rows in four groups, the
// smallest distance of each; T is the distance that 60 of the 128 groups reach
// (rows spread evenly over the groups: ln(1 / (1 - 60 / 128)) rows per group), or all
// of them where fewer have a row with a normal (dead units).
template <typename TC>
__device__ float seed_radius(const GlobalRows<TC> &g, const Ball &ball, int lane)
{
    unsigned m[4] = {0x7f800000u, 0x7f800000u, 0x7f800000u, 0x7f800000u};
    const int per = (g.n + 127) / 128; // rows of a lane per group
    for (int i = 0, k = lane; k < g.n; ++i, k += 32) {
        const vec4_t<TC> v = g.raw(k);
        const float x = (float)v.x, y = (float)v.y, z = (float)v.z, w = (float)v.w;
        const float c = -(x * ball.x + y * ball.y + z * ball.z + w) * rsqrtf(x * x + y * y + z * z);
        const unsigned key = c > 0.f ? __float_as_uint(c) : (c != c ? 0x7f800000u : 0u);
        const int q = i / per;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j == q) m[j] = min(m[j], key);
    }
    int finite = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) finite += m[j] < 0x7f800000u;
    const int need = seed_groups(__reduce_add_sync(kFull, finite));
    if (need == 0) return kReachMax;
    unsigned lo = 0u, hi = 0x7f800000u;
    for (int it = 0; it < 20; ++it) {
        const unsigned mid = (lo + hi) / 2u;
        int c = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) c += m[j] <= mid;
        if (__reduce_add_sync(kFull, c) >= need) hi = mid;
        else lo = mid;
    }
    return clamp_reach(__uint_as_float(hi));
}

// ---------------------------------------------------------------- scans
// What a scan along an edge line found: the first plane (position), or none, or
// (list only) that the rule between near-equal hits needs every row.
enum : int { kHit = 0, kNone = 1, kGiveUp = 2 };

template <typename TC>
struct Line {
    TC d0, d1, d2, thr; // direction (not normalised), parallel threshold
    TC c0, c1, c2;      // current point
    int e, prev;        // the planes it lies on
};
// the same in FP64, for the mixed form's predicates near zero (the threshold is
// worked out where a row is near zero: few steps)
struct Line64 {
    double d0, d1, d2, par_eps, c0, c1, c2;
    __device__ __forceinline__ double thr() const { return par_eps * sqrt(dot3(d0, d0, d1, d1, d2, d2)); }
};

// The rule over the list, `t` exact quotients by candidate: the smallest
// (quotient, row) unless two candidates share a lane of the rule.
// tf[j]: approximate quotient of the lane's row j (infinite: no candidate).
template <typename TC, typename Exact>
__device__ __forceinline__ int choose(const ListRows<TC> &rows, const float (&tf)[kList / 32], int ways, int lane, int &bk,
                                      float &bt, Exact exact)
{
    float lmin = tf[0];
    int lj = 0;
#pragma unroll
    for (int j = 1; j < kList / 32; ++j)
        if (tf[j] < lmin) {
            lmin = tf[j];
            lj = j;
        }
    const unsigned mb = __reduce_min_sync(kFull, __float_as_uint(lmin)); // (quotients are not negative)
    if (mb >= 0x7f800000u) return kNone;
    bt = __uint_as_float(mb);
    const float lim = bt * 1.00001f;
    int c = 0;
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) c += tf[j] <= lim;
    const unsigned any = __ballot_sync(kFull, c > 0);
    if (__popc(any) == 1 && __ballot_sync(kFull, c > 1) == 0u) {
        const int src = __ffs(any) - 1;
        bk = __shfl_sync(kFull, lane + 32 * lj, src);
        return kHit;
    }
    // several hits within 1e-5: by the rule (rare)
    int lane_of[kList / 32]; // the rule's lane of each of this lane's candidates
    double bq = INFINITY;    // quotients in FP64 hold the FP32 ones exactly
    int bi = kNoHit, bp = kNoHit;
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) {
        const bool cand = tf[j] <= lim;
        const int pos = lane + 32 * j;
        const int k = cand ? (int)rows.l->idx[pos] : -1;
        lane_of[j] = cand ? k % ways : -1 - pos;
        if (cand) {
            const double q = exact(j);
            if (q < bq || (q == bq && k < bi)) {
                bq = q;
                bi = k;
                bp = pos;
            }
        }
    }
    bool clash = false;
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) {
        unsigned left = __ballot_sync(kFull, lane_of[j] >= 0);
        while (left) {
            const int src = __ffs(left) - 1;
            left &= left - 1u;
            const int w = __shfl_sync(kFull, lane_of[j], src);
#pragma unroll
            for (int i = 0; i < kList / 32; ++i)
                if (lane_of[i] == w && !(i == j && lane == src)) clash = true;
        }
    }
    if (__any_sync(kFull, clash)) return kGiveUp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double oq = __shfl_xor_sync(kFull, bq, o);
        const int oi = __shfl_xor_sync(kFull, bi, o), op = __shfl_xor_sync(kFull, bp, o);
        if (oq < bq || (oq == bq && oi < bi)) {
            bq = oq;
            bi = oi;
            bp = op;
        }
    }
    bk = bp;
    return kHit;
}

// First hit along the edge line over the list: min over crossing planes of
// t = max(0, -g) / a.  kNear: `near` is set when a row other than the two the
// current point lies on has |g| < 1e-6 there (the rows are normalised, so g is
// a distance): a predicate near zero, which the mixed form takes again in FP64.
template <typename TC, bool kNear>
__device__ __forceinline__ int scan(const ListRows<TC> &rows, const Line<TC> &ln, int ways, int lane, int &bk, float &bt,
                                    bool &near)
{
    float tf[kList / 32];
    TC num[kList / 32], den[kList / 32];
    bool nr = false;
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) {
        const int pos = lane + 32 * j;
        tf[j] = INFINITY;
        num[j] = den[j] = TC(1);
        if (32 * j < rows.n && pos < rows.n && pos != ln.e && pos != ln.prev) {
            const vec4_t<TC> r = rows.get(pos);
            const TC a = dot3(r.x, ln.d0, r.y, ln.d1, r.z, ln.d2);
            TC g = -(dot3(r.x, ln.c0, r.y, ln.c1, r.z, ln.c2) + r.w);
            if (kNear) nr = nr || fabs(g) < TC(1e-6);
            if (a > ln.thr) {
                g = g > TC(0) ? g : TC(0);
                num[j] = g;
                den[j] = a;
                const float q = __fdividef((float)g, (float)a);
                tf[j] = q <= 3.4e38f ? q : 3.4e38f; // (a candidate stays one)
            }
        }
    }
    if (kNear) near = near || __any_sync(kFull, nr);
    return choose<TC>(rows, tf, ways, lane, bk, bt, [&](int j) { return (double)(num[j] / den[j]); });
}

// The mixed form's scan with FP64 predicates (over FP32 rows): every row is
// evaluated in FP32 from the FP32 copy of the current point, and again in
// FP64 from the FP64 current point when that value is within 2e-6 of zero --
// a sign or feasibility decision near zero, taken in FP64.  The first hit is
// the smaller of the FP32 candidates' best and the FP64 candidates' best,
// compared in FP64, ties to the lower row.
struct Cand64 {
    double t;
    bool ok;
};
__device__ __forceinline__ Cand64 near_zero64(const float4 &r, const Line64 &l)
{
    Cand64 c{0.0, false};
    const double a = dot3<double>(r.x, l.d0, r.y, l.d1, r.z, l.d2);
    if (!(a > l.thr())) return c;
    double num = -(dot3<double>(r.x, l.c0, r.y, l.c1, r.z, l.c2) + (double)r.w);
    num = num > 0.0 ? num : 0.0;
    c.t = num / a;
    c.ok = true;
    return c;
}
__device__ __forceinline__ int scan_wide(const ListRows<float> &rows, const Line<float> &ln, const Line64 &l64, int ways,
                                         int lane, int &bk, float &bt)
{
    float tf[kList / 32], num[kList / 32], den[kList / 32]; // den 0: the quotient itself is in q
    double q[kList / 32];
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) {
        const int pos = lane + 32 * j;
        tf[j] = INFINITY;
        q[j] = 0.0;
        num[j] = den[j] = 0.f;
        if (32 * j < rows.n && pos < rows.n && pos != ln.e && pos != ln.prev) {
            const float4 r = rows.get(pos);
            const float g = dot3(r.x, ln.c0, r.y, ln.c1, r.z, ln.c2) + r.w;
            if (fabsf(g) < 2e-6f) {
                const Cand64 c = near_zero64(r, l64);
                if (c.ok) {
                    q[j] = c.t;
                    tf[j] = (float)c.t <= 3.4e38f ? (float)c.t : 3.4e38f;
                }
            } else {
                const float a = dot3(r.x, ln.d0, r.y, ln.d1, r.z, ln.d2);
                if (a > ln.thr) {
                    num[j] = -g > 0.f ? -g : 0.f;
                    den[j] = a;
                    const float t = __fdividef(num[j], a);
                    tf[j] = t <= 3.4e38f ? t : 3.4e38f;
                }
            }
        }
    }
    return choose<float>(rows, tf, ways, lane, bk, bt,
                         [&](int j) { return den[j] != 0.f ? (double)num[j] / (double)den[j] : q[j]; });
}

// The rule itself over every row: `ways` lanes, 32 at a time, two interleaved
// chains each (rows of a chain come in increasing order, so a later row never
// wins a tie against the chain's earlier choice).
template <typename TC, bool kNear>
__device__ int scan(const GlobalRows<TC> &rows, const Line<TC> &ln, int ways, int lane, int &bk_out, float &bt_out, bool &near)
{
    TC wt = TC(INFINITY);
    int wk = kNoHit;
    bool nr = false;
    for (int l0 = 0; l0 < ways; l0 += 32) {
        TC bnum = TC(1), bden = TC(0), bnum1 = TC(1), bden1 = TC(0);
        int bk = kNoHit, bk1 = kNoHit;
        auto consider = [&](int k, TC &bn, TC &bd, int &bi) {
            const vec4_t<TC> r = rows.get(k);
            const TC a = dot3(r.x, ln.d0, r.y, ln.d1, r.z, ln.d2);
            TC num = -(dot3(r.x, ln.c0, r.y, ln.c1, r.z, ln.c2) + r.w);
            if (k == ln.e || k == ln.prev) return;
            if (kNear) nr = nr || fabs(num) < TC(1e-6);
            if (!(a > ln.thr)) return;
            num = num > TC(0) ? num : TC(0);
            if (mul_t(num, bd) < mul_t(bn, a)) {
                bn = num;
                bd = a;
                bi = k;
            }
        };
        int k = l0 + lane;
        for (; k + ways < rows.n; k += 2 * ways) {
            consider(k, bnum, bden, bk);
            consider(k + ways, bnum1, bden1, bk1);
        }
        if (k < rows.n) consider(k, bnum, bden, bk);
        const TC lhs = mul_t(bnum1, bden), rhs = mul_t(bnum, bden1);
        if (bk1 != kNoHit && (lhs < rhs || (lhs == rhs && bk1 < bk))) {
            bnum = bnum1;
            bden = bden1;
            bk = bk1;
        }
        const TC bt = bk == kNoHit ? TC(INFINITY) : bnum / bden;
        if (bt < wt || (bt == wt && bk < wk)) {
            wt = bt;
            wk = bk;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const TC ot = __shfl_xor_sync(kFull, wt, o);
        const int ok = __shfl_xor_sync(kFull, wk, o);
        if (ot < wt || (ot == wt && ok < wk)) {
            wt = ot;
            wk = ok;
        }
    }
    if (kNear) near = near || __any_sync(kFull, nr);
    bk_out = wk;
    bt_out = (float)wt;
    return wk == kNoHit ? kNone : kHit;
}
__device__ int scan_wide(const GlobalRows<float> &rows, const Line<float> &ln, const Line64 &l64, int ways, int lane,
                         int &bk_out, float &bt_out)
{
    double wt = INFINITY;
    int wk = kNoHit;
    for (int l0 = 0; l0 < ways; l0 += 32) {
        float bnum = 1.f, bden = 0.f;
        int bk = kNoHit, tk = kNoHit;
        double tn = INFINITY;
        for (int k = l0 + lane; k < rows.n; k += ways) {
            if (k == ln.e || k == ln.prev) continue;
            const float4 r = rows.get(k);
            const float g = dot3(r.x, ln.c0, r.y, ln.c1, r.z, ln.c2) + r.w;
            if (fabsf(g) < 2e-6f) {
                const Cand64 c = near_zero64(r, l64);
                if (c.ok && (c.t < tn || (c.t == tn && k < tk))) {
                    tn = c.t;
                    tk = k;
                }
                continue;
            }
            const float a = dot3(r.x, ln.d0, r.y, ln.d1, r.z, ln.d2);
            if (!(a > ln.thr)) continue;
            const float num = -g > 0.f ? -g : 0.f;
            const float lhs = mul_t(num, bden), rhs = mul_t(bnum, a);
            if (lhs < rhs || (lhs == rhs && k < bk)) {
                bnum = num;
                bden = a;
                bk = k;
            }
        }
        double bt = bk == kNoHit ? INFINITY : (double)bnum / (double)bden;
        if (tk != kNoHit && (tn < bt || (tn == bt && tk < bk))) {
            bt = tn;
            bk = tk;
        }
        if (bt < wt || (bt == wt && bk < wk)) {
            wt = bt;
            wk = bk;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ot = __shfl_xor_sync(kFull, wt, o);
        const int ok = __shfl_xor_sync(kFull, wk, o);
        if (ot < wt || (ot == wt && ok < wk)) {
            wt = ot;
            wk = ok;
        }
    }
    bk_out = wk;
    bt_out = (float)wt;
    return wk == kNoHit ? kNone : kHit;
}

// ---------------------------------------------------------------- walk
// A face while it is walked.  Lane i ends with vertex i (vx, vy, vz) and the
// plane of the edge leaving it (ve); lane j records step j's hit plane (sbk) and
// merge decision (sdec, 0 append, 1 merge with the previous vertex, 2 merge with
// the first), nsteps the steps taken.  Planes are the row source's positions.
template <typename TS>
struct Face {
    TS vx, vy, vz;
    int ve, n;
    bool closed;
    int8_t status;
    int sbk, sdec, nsteps;
};

// One face walk from the start plane s: the scan in TC (kWide: FP64 predicates
// near zero), vertices solved in TS.  kNear: `near` is set when some step's scan
// met a row within 1e-6 of the current point.  kWalked, or (list only; the face is
// not valid) kLeft: a point left the ball, kUndecided: the rule between near-equal
// hits needs every row, whatever the ball's size.
enum : int { kWalked = 0, kAgain = 1, kLeft = 2, kUndecided = 3 };
template <typename TC, typename TS, bool kWide, bool kNear, typename Rows>
__device__ int walk(const Rows &rows, const Ball &ball, int ways, const vec4_t<TC> &eqc, const TS *eqv, const TS *p,
                     int s, TC par_eps, TS same_eps, int lane, Face<TS> &f, bool &near)
{
    TS last[3] = {0, 0, 0}, first[3] = {0, 0, 0}; // vertices appended last and first (every lane)
    f.vx = f.vy = f.vz = TS(0);
    f.ve = -1;
    f.n = 0;
    f.closed = false;
    f.status = kOk;
    f.sbk = -1;
    f.sdec = 0;
    f.nsteps = 0;
    near = false;
    Line<TC> ln;
    ln.e = s;
    ln.prev = -1;
    ln.c0 = (TC)p[0]; // current point, scan precision
    ln.c1 = (TC)p[1];
    ln.c2 = (TC)p[2];
    Line64 l64; // and in FP64 for the wide scan
    if (kWide) {
        l64.c0 = p[0];
        l64.c1 = p[1];
        l64.c2 = p[2];
    }
    if (!ball.in((float)ln.c0, (float)ln.c1, (float)ln.c2)) return kLeft;
    for (int step = 0; step < kWalkSteps; ++step) {
        f.nsteps = step + 1;
        // direction of the edge line: w_eq x w_e (counter-clockwise about w_eq)
        const vec4_t<TC> r = rows.get(ln.e);
        ln.d0 = diff2(eqc.y, r.z, eqc.z, r.y);
        ln.d1 = diff2(eqc.z, r.x, eqc.x, r.z);
        ln.d2 = diff2(eqc.x, r.y, eqc.y, r.x);
        ln.thr = par_eps * sqrt(dot3(ln.d0, ln.d0, ln.d1, ln.d1, ln.d2, ln.d2));
        int bk;
        float bt;
        int what;
        if constexpr (kWide) {
            const double rx = r.x, ry = r.y, rz = r.z;
            l64.d0 = diff2((double)eqv[1], rz, (double)eqv[2], ry);
            l64.d1 = diff2((double)eqv[2], rx, (double)eqv[0], rz);
            l64.d2 = diff2((double)eqv[0], ry, (double)eqv[1], rx);
            l64.par_eps = (double)par_eps;
            what = scan_wide(rows, ln, l64, ways, lane, bk, bt);
        } else {
            what = scan<TC, kNear>(rows, ln, ways, lane, bk, bt, near);
        }
        if (what == kGiveUp) return kUndecided;
        if (what == kNone) { // the edge line never leaves the region (or its ball)
            if (ball.d2 != INFINITY) return kLeft;
            f.status = kOpen;
            break;
        }
        if (!ball.in((float)ln.c0 + bt * (float)ln.d0, (float)ln.c1 + bt * (float)ln.d1, (float)ln.c2 + bt * (float)ln.d2))
            return kLeft;
        // vertex = 3x3 solve of (edge plane, hit plane, face plane)
        TS V[3];
        TC Vc[3];
        if (!warp_solve<TC, TS>(r, rows.get(bk), eqv, V, Vc, lane)) {
            f.status = kSingular;
            break;
        }
        // 0 append, 1 zero-length edge on e (merge), 2 zero-length closing edge;
        // decided in the solve precision (on the scan-precision copies
        // where the rounding margin settles it)
        int decision = 0;
        if (f.n > 0) {
            int s1 = -1, s2 = 0;
            if (sizeof(TS) > sizeof(TC)) {
                s1 = same_filter<TC, TS>(Vc, (TC)last[0], (TC)last[1], (TC)last[2], same_eps);
                if (bk == s && s1 == 0) s2 = same_filter<TC, TS>(Vc, (TC)first[0], (TC)first[1], (TC)first[2], same_eps);
            }
            if (s1 == 1) {
                decision = 1;
            } else if (s1 == 0 && s2 != -1) {
                decision = s2 == 1 ? 2 : 0;
            } else {
                if (fabs(V[0] - last[0]) + fabs(V[1] - last[1]) + fabs(V[2] - last[2]) < same_eps)
                    decision = 1;
                else if (bk == s && fabs(V[0] - first[0]) + fabs(V[1] - first[1]) + fabs(V[2] - first[2]) < same_eps)
                    decision = 2;
            }
        }
        if (lane == step) {
            f.sbk = bk;
            f.sdec = decision;
        }
        if (decision == 1 && lane == f.n - 1) f.ve = bk; // the edge on e has zero length
        if (decision == 0) {
            if (lane == f.n) {
                f.vx = V[0];
                f.vy = V[1];
                f.vz = V[2];
                f.ve = bk;
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                last[j] = V[j];
                if (f.n == 0) first[j] = V[j];
            }
            f.n++;
        }
        if (bk == s) {
            f.closed = true;
            break;
        }
        if (f.n >= kVMax) {
            f.status = kTruncated;
            break;
        }
        ln.prev = ln.e;
        ln.e = bk;
        ln.c0 = Vc[0];
        ln.c1 = Vc[1];
        ln.c2 = Vc[2];
        if (kWide) {
            l64.c0 = V[0];
            l64.c1 = V[1];
            l64.c2 = V[2];
        }
        if (!ball.in((float)ln.c0, (float)ln.c1, (float)ln.c2)) return kLeft;
    }
    if (!f.closed && f.status == kOk) f.status = kTruncated;
    return kWalked;
}

// Mixed form: the walk runs in the scan precision TC (solves included, as the
// plain form does), then every vertex is solved again in TS -- four lanes per
// vertex (the four Cramer determinants), eight vertices per warp instruction
// -- and every merge decision is taken again on the TS vertices.  When all
// decisions agree, the face is the TS walk's face: the same hit planes, the
// same TS vertices.  Returns kAgain, and the caller walks again with every
// predicate and every solve in TS, when a scan met a row within 1e-6 of the
// current point other than the two it lies on (a sign or feasibility test
// near zero), when the TC walk did not close normally, took more than 32
// steps or met a vertex that is not finite in TS, or when a decision comes
// out differently in TS; kLeft and kUndecided as walk does.
template <typename TC, typename TS, typename Rows>
__device__ int walk_refined(const Rows &rows, const Ball &ball, int ways, const vec4_t<TC> &eqc, const TS *eqv,
                            const TS *p, int s, TC par_eps, TS same_eps, int lane, Face<TS> &f)
{
    const unsigned full = kFull;
    const TC eqf[4] = {eqc.x, eqc.y, eqc.z, eqc.w};
    const TC pf[3] = {(TC)p[0], (TC)p[1], (TC)p[2]};
    Face<TC> w;
    bool near;
    const int how = walk<TC, TC, false, true>(rows, ball, ways, eqc, eqf, pf, s, par_eps, (TC)same_eps, lane, w, near);
    if (how != kWalked) return how;
    const int sbk = w.sbk, sdec = w.sdec, nsteps = w.nsteps;
    // a predicate near zero: the caller walks again with FP64 predicates
    if (near || w.status != kOk || !w.closed || nsteps < 1 || nsteps > 32) return kAgain;

    // step j's vertex in TS, into lane j
    const int G = lane >> 2, L = lane & 3, gbase = lane & ~3;
    TS rx = 0, ry = 0, rz = 0;
    bool planes_ok = true;
    for (int r0 = 0; r0 < nsteps; r0 += 8) {
        const int j = min(r0 + G, nsteps - 1);            // the step this lane group solves
        const int pb = __shfl_sync(full, sbk, j);          // its hit plane
        const int pj = __shfl_sync(full, sbk, max(j - 1, 0));
        const int pa = j == 0 ? s : pj;                    // and the edge plane it walked on
        const bool in = (unsigned)pa < (unsigned)rows.n && (unsigned)pb < (unsigned)rows.n;
        planes_ok = planes_ok && in;
        // lane t of the group converts components 2t, 2t + 1 of [row a | row b]
        const vec4_t<TC> rr = rows.get(in ? (L < 2 ? pa : pb) : 0);
        const TS c0 = (TS)(L & 1 ? rr.z : rr.x);
        const TS c1 = (TS)(L & 1 ? rr.w : rr.y);
        TS m[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            m[2 * t] = __shfl_sync(full, c0, gbase | t);
            m[2 * t + 1] = __shfl_sync(full, c1, gbase | t);
        }
        const TS a00 = L == 1 ? -m[3] : m[0], a01 = L == 2 ? -m[3] : m[1], a02 = L == 3 ? -m[3] : m[2];
        const TS a10 = L == 1 ? -m[7] : m[4], a11 = L == 2 ? -m[7] : m[5], a12 = L == 3 ? -m[7] : m[6];
        const TS a20 = L == 1 ? -eqv[3] : eqv[0], a21 = L == 2 ? -eqv[3] : eqv[1], a22 = L == 3 ? -eqv[3] : eqv[2];
        const TS d = det3<TS>(a00, a01, a02, a10, a11, a12, a20, a21, a22);
        const TS x = d / __shfl_sync(full, d, gbase);
        const int src = ((lane - r0) & 7) * 4 + 1;
        const TS v0 = __shfl_sync(full, x, src), v1 = __shfl_sync(full, x, src + 1), v2 = __shfl_sync(full, x, src + 2);
        if (lane >= r0 && lane < r0 + 8) {
            rx = v0;
            ry = v1;
            rz = v2;
        }
    }
    const bool mine = lane < nsteps;
    if (!__all_sync(full, planes_ok && (!mine || (finite_bits(rx) && finite_bits(ry) && finite_bits(rz))))) return kAgain;

    // the decisions again, on the TS vertices: step j against the last
    // vertex appended before it and, on the closing step, the first vertex
    const unsigned amask = __ballot_sync(full, mine && sdec == 0);
    const unsigned before = lane > 0 ? (amask & ((1u << lane) - 1u)) : 0u;
    const int la = before ? 31 - __clz(before) : 0;
    const TC Vc[3] = {(TC)rx, (TC)ry, (TC)rz};
    const TC lx = __shfl_sync(full, Vc[0], la), ly = __shfl_sync(full, Vc[1], la), lz = __shfl_sync(full, Vc[2], la);
    const TC f0 = __shfl_sync(full, Vc[0], 0), f1 = __shfl_sync(full, Vc[1], 0), f2 = __shfl_sync(full, Vc[2], 0);
    const bool check = mine && lane > 0;
    int s1 = same_filter<TC, TS>(Vc, lx, ly, lz, same_eps);
    int s2 = sbk == s ? same_filter<TC, TS>(Vc, f0, f1, f2, same_eps) : 0;
    if (__any_sync(full, check && (s1 < 0 || (s1 == 0 && s2 < 0)))) {
        const TS Lx = __shfl_sync(full, rx, la), Ly = __shfl_sync(full, ry, la), Lz = __shfl_sync(full, rz, la);
        const TS Fx = __shfl_sync(full, rx, 0), Fy = __shfl_sync(full, ry, 0), Fz = __shfl_sync(full, rz, 0);
        if (check && s1 < 0) s1 = (fabs(rx - Lx) + fabs(ry - Ly) + fabs(rz - Lz) < same_eps) ? 1 : 0;
        if (check && s2 < 0) s2 = (fabs(rx - Fx) + fabs(ry - Fy) + fabs(rz - Fz) < same_eps) ? 1 : 0;
    }
    const int dec = s1 == 1 ? 1 : (sbk == s && s2 == 1 ? 2 : 0);
    if (!__all_sync(full, !check || dec == sdec)) return kAgain;

    // vertex o is the o-th appended step; its edge is the hit plane of the
    // last step before the next append, a closing merge excepted
    f.n = __popc(amask);
    const int so = lane < f.n ? (int)__fns(amask, 0, lane + 1) : 0;
    const int snext = lane + 1 < f.n ? (int)__fns(amask, 0, lane + 2) : nsteps;
    int kl = (snext - 1) & 31;
    if (__shfl_sync(full, sdec, kl) == 2) kl = (kl - 1) & 31;
    const int e_out = __shfl_sync(full, sbk, kl);
    const TS ox = __shfl_sync(full, rx, so), oy = __shfl_sync(full, ry, so), oz = __shfl_sync(full, rz, so);
    if (lane < f.n) {
        f.vx = ox;
        f.vy = oy;
        f.vz = oz;
        f.ve = e_out;
    } else {
        f.vx = f.vy = f.vz = TS(0);
        f.ve = -1;
    }
    f.closed = true;
    f.status = kOk;
    return kWalked;
}

template <typename TC, typename TS, typename Rows>
__device__ int walk_fp64(const Rows &rows, const Ball &ball, int ways, const vec4_t<TC> &eqc, const TS *p,
                                       int s, TC par_eps, TS same_eps, int lane, Face<TS> &f)
{
    const TS eqv[4] = {(TS)eqc.x, (TS)eqc.y, (TS)eqc.z, (TS)eqc.w};
    bool near;
    return walk<TC, TS, true, false>(rows, ball, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f, near);
}

// The whole walk of a form over one row source (kLeft, kUndecided: as walk).
template <typename TC, typename TS, typename Rows>
__device__ int face_walk(const Rows &rows, const Ball &ball, int ways, const vec4_t<TC> &eqc, const TS *eqv, const TS *p,
                          int s, TC par_eps, TS same_eps, int lane, Face<TS> &f, bool &again)
{
    again = false;
    if constexpr (sizeof(TS) > sizeof(TC)) { // scan-precision walk, vertices refined in the solve precision
        const int r = walk_refined<TC, TS>(rows, ball, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f);
        if (r != kAgain) return r;
        again = true; // FP64 predicates and FP64 solves
        return walk_fp64<TC, TS>(rows, ball, ways, eqc, p, s, par_eps, same_eps, lane, f);
    } else {
        bool near;
        return walk<TC, TS, false, false>(rows, ball, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f, near);
    }
}

// ---------------------------------------------------------------- seeds
// Start vertex of a seed region: the start plane's position and the vertex in
// p, -1 when no pair is feasible, -2 when the list cannot decide (it does not
// surely hold the nearest planes).  Every row outside the list holds at a point
// of the ball; elsewhere the rows are tested one by one.
template <typename TC, typename TS, typename Rows>
__device__ int seed_start(const Rows &rows, const GlobalRows<TC> &all, const Ball &ball, float T, const TS *eqv, TS *p, TC eps,
                          int lane)
{
    // pairs x <= 812 reach sorted positions up to 56: keep the 64 nearest,
    // position q in lane q % 32, register q / 32
    const int ksel = all.n < kTopK ? all.n : kTopK;
    if (rows.n < ksel) return -2;
    int top0 = -1, top1 = -1;
    unsigned long long pk = ~0ull;
    int pi = -1;
    const TC pc[3] = {(TC)p[0], (TC)p[1], (TC)p[2]};
    if (rows.n <= kList) { // each row's rank among all, its key computed once
        constexpr int kPer = kList / 32;
        unsigned long long key[kPer];
        int rank[kPer];
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            const int k = lane + 32 * t;
            key[t] = 0ull;
            rank[t] = k < rows.n ? 0 : kNoHit;
            if (k < rows.n) {
                const vec4_t<TC> v = rows.get(k);
                key[t] = order_key(dot3(v.x, pc[0], v.y, pc[1], v.z, pc[2]) + v.w);
            }
        }
#pragma unroll
        for (int t = 0; t < kPer; ++t)
            for (int l = 0; l < 32 && 32 * t + l < rows.n; ++l) {
                const unsigned long long ok = __shfl_sync(kFull, key[t], l);
#pragma unroll
                for (int u = 0; u < kPer; ++u) rank[u] += ahead(ok, 32 * t + l, key[u], lane + 32 * u);
            }
        for (int sel = 0; sel < ksel; ++sel) {
            int mine = -1;
#pragma unroll
            for (int t = 0; t < kPer; ++t)
                if (rank[t] == sel) mine = lane + 32 * t;
            const int at = __shfl_sync(kFull, mine, __ffs(__ballot_sync(kFull, mine >= 0)) - 1);
            if (lane == (sel & 31)) {
                if (sel < 32) top0 = at;
                else top1 = at;
            }
            pi = at;
        }
    } else
    for (int sel = 0; sel < ksel; ++sel) {
        unsigned long long bk = 0ull;
        int bi = kNoHit;
        for (int k = lane; k < rows.n; k += 32) {
            const vec4_t<TC> v = rows.get(k);
            const TC d = dot3(v.x, pc[0], v.y, pc[1], v.z, pc[2]) + v.w;
            const unsigned long long key = order_key(d);
            const bool below = key < pk || (key == pk && k > pi);
            if (below && ahead(key, k, bk, bi)) {
                bk = key;
                bi = k;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(kFull, bk, o);
            const int oi = __shfl_xor_sync(kFull, bi, o);
            if (ahead(ok, oi, bk, bi)) {
                bk = ok;
                bi = oi;
            }
        }
        if (lane == (sel & 31)) {
            if (sel < 32) top0 = bi;
            else top1 = bi;
        }
        pk = bk;
        pi = bi;
    }
    if (ball.d2 != INFINITY) { // the farthest chosen plane well inside T: no plane left out is nearer
        const vec4_t<TC> v = rows.get(pi);
        const float c = -(float)(dot3(v.x, pc[0], v.y, pc[1], v.z, pc[2]) + v.w);
        if (!(c < T * 0.999f - 1e-5f * coord_size(ball, T))) return -2;
    }
    int x_max = (all.n - 1) * (all.n - 2);
    if (x_max > 812) x_max = 812;
    if (x_max < 0) x_max = 0;
    // eight pairs at a time, four lanes per pair (its Cramer determinants, the
    // arithmetic of warp_solve); their vertices are tested one after the other,
    // the first that every other row admits wins
    const int G = lane >> 2, L = lane & 3, gbase = lane & ~3;
    // the rows in FP32, held by the lanes: a vertex that one of them shuts out by
    // more than the FP32 error (a row's and a determinant's rounding, a quotient's,
    // a product's, three sums': 9 x 2^-24 of the products' sizes; 2^-20 asked for)
    // needs neither the divisions nor a test in TC.  (FP64 is what a seed's search
    // costs: 813 pairs.  Measured on GB300, eight boxes around 64 x 3 networks in
    // FP64, a batch of marchings: 8.0 ms with every pair divided and tested row
    // after row and the nearest planes picked one by one, 7.4 ms this way.)
    constexpr int kPer = kList / 32;
    const bool held = rows.n <= kList;
    float4 fr[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        fr[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (held && lane + 32 * t < rows.n) {
            const vec4_t<TC> r = rows.get(lane + 32 * t);
            fr[t] = make_float4((float)r.x, (float)r.y, (float)r.z, (float)r.w);
        }
    }
    const float feps = (float)eps + 1e-30f;
    for (int x0 = 0; x0 <= x_max; x0 += 8) {
        int i, j;
        get_i_j(min(x0 + G, x_max), all.n, i, j);
        const int ri0 = __shfl_sync(kFull, top0, i & 31), ri1 = __shfl_sync(kFull, top1, i & 31);
        const int rj0 = __shfl_sync(kFull, top0, j & 31), rj1 = __shfl_sync(kFull, top1, j & 31);
        const int ri = i < 32 ? ri0 : ri1;
        const int rj = j < 32 ? rj0 : rj1;
        // lane t of the group converts components 2t, 2t + 1 of [row i | row j]
        const vec4_t<TC> rr = rows.get(L < 2 ? ri : rj);
        const TS c0 = (TS)(L & 1 ? rr.z : rr.x), c1 = (TS)(L & 1 ? rr.w : rr.y);
        TS m[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            m[2 * t] = __shfl_sync(kFull, c0, gbase | t);
            m[2 * t + 1] = __shfl_sync(kFull, c1, gbase | t);
        }
        const TS a00 = L == 1 ? -m[3] : m[0], a01 = L == 2 ? -m[3] : m[1], a02 = L == 3 ? -m[3] : m[2];
        const TS a10 = L == 1 ? -m[7] : m[4], a11 = L == 2 ? -m[7] : m[5], a12 = L == 3 ? -m[7] : m[6];
        const TS a20 = L == 1 ? -eqv[3] : eqv[0], a21 = L == 2 ? -eqv[3] : eqv[1], a22 = L == 3 ? -eqv[3] : eqv[2];
        const TS d = det3<TS>(a00, a01, a02, a10, a11, a12, a20, a21, a22);
        const TS d0 = __shfl_sync(kFull, d, gbase);
        unsigned shut = 0u; // pairs of the eight that some row shuts out for certain
        if (held) {
            // (a quotient of determinants that FP32 does not hold to its precision shuts nothing out)
            const float fd = (float)d, f0 = (float)d0;
            const float fx = d == TS(0) ? 0.f : (fminf(fabsf(fd), fabsf(f0)) < 1e-30f ? NAN : fd / f0);
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                const float a = __shfl_sync(kFull, fx, 4 * g + 1), b = __shfl_sync(kFull, fx, 4 * g + 2),
                            c = __shfl_sync(kFull, fx, 4 * g + 3);
                const int gi = __shfl_sync(kFull, ri, 4 * g), gj = __shfl_sync(kFull, rj, 4 * g);
#pragma unroll
                for (int t = 0; t < kPer; ++t) {
                    const int k = lane + 32 * t;
                    const float d = fr[t].x * a + fr[t].y * b + fr[t].z * c + fr[t].w;
                    const float z = fabsf(fr[t].x * a) + fabsf(fr[t].y * b) + fabsf(fr[t].z * c) + fabsf(fr[t].w);
                    if (d > feps + z * 9.5367431640625e-7f && k != gi && k != gj) shut |= 1u << g;
                }
            }
            shut = __reduce_or_sync(kFull, shut);
        }
        if (shut == 0xffu) continue;
        const TS xv = d / d0;
        for (int g = 0; g < 8 && x0 + g <= x_max; ++g) {
            if ((shut >> g) & 1u) continue;
            const TS v[3] = {__shfl_sync(kFull, xv, 4 * g + 1), __shfl_sync(kFull, xv, 4 * g + 2),
                             __shfl_sync(kFull, xv, 4 * g + 3)};
            const TC vc[3] = {(TC)v[0], (TC)v[1], (TC)v[2]};
            const int pi_ = __shfl_sync(kFull, ri, 4 * g), pj_ = __shfl_sync(kFull, rj, 4 * g);
            bool bad = false;
            for (int k = lane; k < rows.n; k += 32) {
                if (k == pi_ || k == pj_) continue;
                const vec4_t<TC> r = rows.get(k);
                if (dot3(r.x, vc[0], r.y, vc[1], r.z, vc[2]) + r.w > eps) bad = true;
            }
            if (__any_sync(kFull, bad)) continue;
            if (!ball.in((float)vc[0], (float)vc[1], (float)vc[2])) {
                const int ki = rows.name(pi_), kj = rows.name(pj_);
                for (int k = lane; k < all.n; k += 32) {
                    if (k == ki || k == kj) continue;
                    const vec4_t<TC> r = all.get(k);
                    if (dot3(r.x, vc[0], r.y, vc[1], r.z, vc[2]) + r.w > eps) bad = true;
                }
                if (__any_sync(kFull, bad)) continue;
            }
            p[0] = v[0];
            p[1] = v[1];
            p[2] = v[2];
            return pi_;
        }
    }
    return -1;
}

// What the kernel needs of a face's walk.
template <typename TS>
struct Result {
    TS vx, vy, vz; // lane i: vertex i
    int ve;        // and the plane of the edge leaving it (-1: none)
    int n, start;  // vertices; start plane
    bool closed, again;
    int8_t status;
    float T;       // radius of the list used last, and the rows in it
    int listed;
};

// Everything but the common face (a region with a parent whose FP32 walk stays in
// its list and needs no FP64 predicate): seeds, repeats with another radius, FP64
// predicates, every row.  Kept out of the kernel's registers.  `what`: kAgain, only
// the FP64 predicates are asked for, on the list as it is; kLeft or kUndecided, the
// walk over the list as it is (n rows within T) has failed.  `every_row`: no list.
// A larger ball costs a pass over the rows and may fail again (an edge that never
// ends does for certain), so it is tried only where a walk over every row costs
// more: on up to kDirect rows a step of that takes a few rows per lane as the list's
// does.  Measured on GB300, polygon phase in float64 / mixed / float32: 3-[50]x3-1 with
// connections, 192 of 14,397 faces open, 2.5 / 0.98 / 0.73 ms with the failed walk made
// again and larger balls tried, 1.8 / 0.76 / 0.53 this way; widths 8 to 87 with many
// near-equal hits 10.4 / 3.4 / 2.8 and 6.2 / 2.2 / 1.8; the benchmark networks alike.
template <typename TC, typename TS>
__device__ __noinline__ void face_slow(const GlobalRows<TC> &all, NearList<TC> *list, int ways, const vec4_t<TC> &eqc,
                                       const TS *mid, int start, TC eps, TC par_eps, TS same_eps, int lane, int what,
                                       int n, float T, bool every_row, Result<TS> &out)
{
    const bool is_seed = start < 0;
    const TS eqv[4] = {(TS)eqc.x, (TS)eqc.y, (TS)eqc.z, (TS)eqc.w};
    TS p[3] = {mid[0], mid[1], mid[2]};
    Ball ball{(float)p[0], (float)p[1], (float)p[2], -1.f};
    Face<TS> f;
    bool done = false, wide = false, found = false;
    int s = start, s_plane = start;
    auto clear = [&] {
        f.vx = f.vy = f.vz = TS(0);
        f.n = 0;
        f.ve = -1;
        f.closed = false;
        f.status = kNoStart;
    };
    clear();
    if (is_seed) {
        T = all.n > kList ? seed_radius<TC>(all, ball, lane) : INFINITY;
        n = -1;
    }
    bool use_list = !every_row && what != kUndecided;
    auto larger = [&](bool direct) { // a larger ball, if it is worth a pass
        if (n > 3 * kList / 4 || T >= kReachMax || (direct && all.n <= kDirect)) return false;
        T *= fminf((float)kList * 0.85f / (float)max(n, 1), 3.f);
        n = -1;
        return true;
    };
    if (use_list && !is_seed && what == kLeft && n <= kList) use_list = larger(true);
    if (n > kList) { // (only if dead units are in it is the same ball worth another pass)
        bool dead = false;
        for (int j = lane; j < kList; j += 32) dead = dead || list->row[j].w != list->row[j].w;
        if (__any_sync(kFull, dead)) n = -1;
    }
    for (int tries = 0; tries < 5 && !done && use_list; ++tries) {
        if (n < 0) n = collect<TC>(all, T, ball, list, lane);
        if (n > kList) { // a smaller ball
            T = clamp_reach(T * ((float)kTarget / (float)n));
            n = -1;
            continue;
        }
        const ListRows<TC> rows{list, n};
        ball.d2 = ball_radius2<(sizeof(TS) > sizeof(TC))>(ball, T);
        TS q[3] = {p[0], p[1], p[2]};
        if (!is_seed) {
            s = position<TC>(list, n, start, lane);
        } else {
            s = seed_start<TC, TS>(rows, all, ball, T, eqv, q, eps, lane);
            if (s == -1) { // no feasible start
                done = true;
                s_plane = -1;
                break;
            }
        }
        int how = kLeft;
        if (s >= 0) {
            if constexpr (sizeof(TS) > sizeof(TC)) {
                if (what == kAgain) {
                    wide = true;
                    how = walk_fp64<TC, TS>(rows, ball, ways, eqc, q, s, par_eps, same_eps, lane, f);
                } else {
                    how = face_walk<TC, TS>(rows, ball, ways, eqc, eqv, q, s, par_eps, same_eps, lane, f, wide);
                }
            } else {
                how = face_walk<TC, TS>(rows, ball, ways, eqc, eqv, q, s, par_eps, same_eps, lane, f, wide);
            }
            s_plane = list->idx[s];
        }
        what = kLeft;
        done = how == kWalked;
        if (done) {
            if (f.ve >= 0) f.ve = list->idx[f.ve];
        } else if (how == kUndecided || !larger(s >= 0)) {
            if (is_seed && s >= 0) { // the start vertex found is every row's too
                found = true;
                p[0] = q[0];
                p[1] = q[1];
                p[2] = q[2];
            }
            break;
        }
    }
    if (!done) { // every row
        const Ball whole{0.f, 0.f, 0.f, INFINITY};
        clear();
        wide = false;
        s = start;
        if (found) s = s_plane;
        else if (is_seed) s = seed_start<TC, TS>(all, all, whole, INFINITY, eqv, p, eps, lane);
        if (s >= 0) face_walk<TC, TS>(all, whole, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f, wide);
        s_plane = s;
    }
    out.vx = f.vx;
    out.vy = f.vy;
    out.vz = f.vz;
    out.ve = f.ve;
    out.n = f.n;
    out.start = s_plane;
    out.closed = f.closed;
    out.again = wide;
    out.status = f.status;
    out.T = T;
    out.listed = n;
}

// ---------------------------------------------------------------- neighbours
__device__ __forceinline__ long long next_work(WaveCtl *ctl, int lane)
{
    unsigned int v = 0;
    if (lane == 0) v = atomicAdd(&ctl->work, 1u);
    return (long long)__shfl_sync(0xffffffffu, v, 0);
}

__device__ __forceinline__ unsigned long long load_slot(const unsigned long long *p)
{
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> a(*const_cast<unsigned long long *>(p));
    return a.load(cuda::memory_order_relaxed);
}

// Insert the neighbours across the planes kv >= 0 (one per lane; the parent's
// key with that bit flipped) into the region hash set.  Every lane probes for its
// own key, so that the slots of all edges are read at once; where fingerprints
// match, the whole warp compares the keys (lane l takes words l, l + 32, ...).
// Returns the slot claimed for a new candidate (or the candidate slot this one
// now shares), -1 when the key is a committed region already.  Among equal
// candidate keys the smallest (parent, plane) id stays in the slot, so the
// result does not depend on timing.  Region entries (tag 0) point at the region
// store; candidate entries (tag 1) carry (wave position, plane) and point at
// the parent's key.
__device__ int insert_edges(const RegionsDev &reg, const HashDev &hs, long long head, int ALL, int W, const uint32_t *pkey,
                            uint64_t phash, long long rl, int kv, int lane, int *err)
{
    int got = -1;
    bool open = kv >= 0;
    uint32_t fp = 0;
    unsigned long long mine = 0, slot = 0;
    if (open) {
        const uint64_t h = flip_hash(phash, pkey[kv >> 5], kv);
        fp = fp_of(h);
        mine = slot_value(fp, 1, (uint32_t)(rl * ALL + kv));
        slot = h & hs.mask;
    }
    for (int probe = 0; probe < kMaxProbes; ++probe) {
        unsigned long long cur = 0ull;
        bool match = false;
        if (open) {
            cur = load_slot(hs.slots + slot);
            if (cur == kEmpty) {
                const unsigned long long old = atomicCAS(hs.slots + slot, kEmpty, mine);
                if (old == kEmpty) {
                    got = (int)slot;
                    open = false;
                }
                cur = old;
            }
            match = open && (uint32_t)(cur >> 32) == fp;
        }
        unsigned todo = __ballot_sync(kFull, match);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            const uint32_t id = (uint32_t)__shfl_sync(kFull, (uint32_t)cur & 0x7fffffffu, src);
            const bool cand = __shfl_sync(kFull, (uint32_t)cur >> 31, src) != 0u;
            const int k = __shfl_sync(kFull, kv, src);
            const uint32_t *other = reg.keys + (size_t)(cand ? head + id / ALL : (long long)id) * W;
            const int ok2 = cand ? (int)(id % ALL) : -1;
            const int kw = k >> 5, ow = ok2 >= 0 ? ok2 >> 5 : -1;
            const uint32_t kb = 1u << (k & 31), ob = ok2 >= 0 ? 1u << (ok2 & 31) : 0u;
            bool differ = false;
            for (int w = lane; w < W; w += 32) {
                const uint32_t a = pkey[w] ^ (w == kw ? kb : 0u);
                const uint32_t b = other[w] ^ (w == ow ? ob : 0u);
                differ = differ || a != b;
            }
            if (!__any_sync(kFull, differ) && lane == src) {
                open = false;
                if (cand) {
                    atomicMin(hs.slots + slot, mine);
                    got = (int)slot;
                }
            }
        }
        if (!__any_sync(kFull, open)) return got;
        slot = (slot + (unsigned long long)probe + 1ull) & hs.mask;
    }
    if (open) atomicOr(err, kErrTableFull);
    return got;
}

// ---------------------------------------------------------------- kernel
// TC is the scan precision, TS the solve precision.
//
// What bounds it: the rows from HBM on wide networks (65.7 KB read and on average
// 32 KB written per face of 4,104 rows), latency and issue slots on narrow ones,
// the FP64 pipe where TS or TC is double.  A warp per face, rather than a group
// that scans every row at every step from shared memory, because with the list a
// step is four rows per lane and the rest of it (solve, decisions) is the same for
// every warp of a group.  Measured on GB300, polygon phase of a whole marching:
//   3-[512]x8-1 mixed (6.8 M faces)      378 ms -> 143 ms
//   3-[256]x6-1 mixed (1.28 M)            29.4  -> 15.0
//   3-[128]x4-1 mixed / fp32 / fp64 (265 K) 3.2 / 2.4 / 28.8 -> 2.7 / 1.7 / 8.5
template <typename TC, typename TS>
__global__ void __launch_bounds__(32 * kFaceWarps, kBlocks) polygon_kernel(NetDev net, RegionsDev reg, ChunkDev ch, HashDev hs,
                                                                     Tolerances tol, int ways, bool every_row,
                                                                     unsigned long long *nfp64, int *err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    NearList<TC> *list = reinterpret_cast<NearList<TC> *>(smem_raw) + wib;
    const int ALL = net.ALL, N = net.N, W = net.W;
    const TC eps = (TC)tol.eps, par_eps = (TC)tol.par_eps;
    const TS same_eps = (TS)tol.same_eps;
    long long head;
    int count;
    chunk_range(ch, head, count);
    if (ch.ctl && blockIdx.x == 0 && threadIdx.x == 0) { // the wave's range for the append
        ch.ctl->append_head = head;
        ch.ctl->append_count = count;
    }
    // a region per warp: by launch position, or (fixed grid of the
    // graph-driven loop) from the wave's work counter
    long long rl_next = (long long)blockIdx.x * kFaceWarps + wib;
    for (;;) {
        const long long rl = ch.ctl ? next_work(ch.ctl, lane) : rl_next;
        rl_next += (long long)gridDim.x * kFaceWarps;
        if (rl >= count) break;
        const long long rid = head + rl;
        vec4_t<TC> *own = reinterpret_cast<vec4_t<TC> *>((TC *)ch.cons + (size_t)row_slot(ch, head, (int)rl) * net.ALLP * 4);
        const int start = reg.start[rid], parent = reg.parent[rid];
        GlobalRows<TC> all;
        all.n = ALL;
        all.own = own;
        all.nsplit = ch.split ? ch.split[rl] : 0;
        all.flip = all.nsplit ? start : -1;
        all.par = all.nsplit ? reinterpret_cast<const vec4_t<TC> *>((const TC *)ch.cons + (size_t)ring_slot(ch, parent) * net.ALLP * 4)
                             : own;
        const TS *midp = (const TS *)reg.mid + (size_t)rid * 4;

        // ------------------------------------------------ near list, walk
        Result<TS> r;
        r.T = INFINITY; // few rows: all of them
        int what = kLeft;
        if (start >= 0) {
            if (ALL > kList) r.T = (float)((const TS *)reg.mid)[(size_t)parent * 4 + 3];
            const Ball centre{(float)midp[0], (float)midp[1], (float)midp[2], -1.f};
            Sieve<TC> sv(centre, r.T, list, lane);
            stream_part<TC, true>(all.par, own, 0, all.nsplit, all.flip, sv);
            stream_part<TC, false>(own, nullptr, all.nsplit, ALL, -1, sv);
            sv.finish();
            r.listed = sv.n;
            if (sv.n <= kList && !every_row) {
                const vec4_t<TC> eqc = ld4<TC>((const TC *)ch.eq + (size_t)rl * 4); // scan precision copy
                const TS eqv[4] = {(TS)eqc.x, (TS)eqc.y, (TS)eqc.z, (TS)eqc.w};
                const TS p[3] = {midp[0], midp[1], midp[2]};
                Ball ball{(float)p[0], (float)p[1], (float)p[2], -1.f};
                ball.d2 = ball_radius2<(sizeof(TS) > sizeof(TC))>(ball, r.T);
                const ListRows<TC> rows{list, sv.n};
                const int s = position<TC>(list, sv.n, start, lane);
                Face<TS> f;
                if (s >= 0) {
                    if constexpr (sizeof(TS) > sizeof(TC)) {
                        what = walk_refined<TC, TS>(rows, ball, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f);
                    } else {
                        bool near;
                        what = walk<TC, TS, false, false>(rows, ball, ways, eqc, eqv, p, s, par_eps, same_eps, lane, f, near);
                    }
                }
                r.vx = f.vx;
                r.vy = f.vy;
                r.vz = f.vz;
                r.n = f.n;
                r.closed = f.closed;
                r.status = f.status;
                r.ve = what == kWalked && f.ve >= 0 ? (int)list->idx[f.ve] : -1;
                r.start = start;
            }
        }
        if (what != kWalked) {
            Result<TS> o;
            const vec4_t<TC> eqc = ld4<TC>((const TC *)ch.eq + (size_t)rl * 4);
            face_slow<TC, TS>(all, list, ways, eqc, midp, start, eps, par_eps, same_eps, lane, what, r.listed, r.T, every_row, o);
            r = o;
            if (r.again && lane == 0) atomicAdd(nfp64, 1ull);
        }

        // ------------------------------------------------ outputs
        const int nv = r.n, ve = r.ve;
        if (lane == 0) {
            reg.nv[rid] = nv;
            reg.status[rid] = r.status;
            ((TS *)reg.mid)[(size_t)rid * 4 + 3] = (TS)child_reach(r.T, r.listed, kTarget);
        }
        if (lane < nv) {
            TS *vo = (TS *)reg.verts + ((size_t)rid * kVMax + lane) * 3;
            vo[0] = r.vx;
            vo[1] = r.vy;
            vo[2] = r.vz;
            reg.edges[(size_t)rid * kVMax + lane] = ve;
        }

        // ------------------------------------------------ neighbours
        // the plane crossed by edge `lane` where a neighbour is to be inserted
        int kv = -1;
        if (lane < nv && ve >= 0 && ve < N && (r.closed || lane < nv - 1) && !(start >= 0 && ve == r.start)) kv = ve;
        ch.rec[(size_t)rl * kVMax + lane] =
            insert_edges(reg, hs, head, ALL, W, reg.keys + (size_t)rid * W, reg.hash[rid], rl, kv, lane, err);
        __syncwarp();
    }
}

} // namespace

template <typename TC, typename TS>
static void launch_one(const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, const HashDev &hs,
                       const Tolerances &tol, int *d_err, int ways, bool every_row, unsigned long long *nfp64, cudaStream_t st)
{
    auto k = polygon_kernel<TC, TS>;
    const size_t smem = sizeof(NearList<TC>) * kFaceWarps;
    int per_sm = 1; // as many blocks as stay resident
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * kFaceWarps, smem);
    long long grid = (long long)device_sms() * std::max(per_sm, 1);
    if (!ch.ctl) grid = std::min<long long>(grid, (ch.count + kFaceWarps - 1) / kFaceWarps);
    k<<<(unsigned)grid, 32 * kFaceWarps, smem, st>>>(net, reg, ch, hs, tol, ways, every_row, nfp64, d_err);
}

void launch_polygon(int prec, const NetDev &net, const RegionsDev &reg, const ChunkDev &ch, const HashDev &hs,
                    const Tolerances &tol, int rule_warps, bool every_row, unsigned long long *nfp64, int *d_err, cudaStream_t st)
{
    if (!ch.ctl && ch.count <= 0) return;
    const int ways = hit_rule_lanes(prec == kFloat64, net.ALLP, rule_warps);
    if (prec == kFloat64)
        launch_one<double, double>(net, reg, ch, hs, tol, d_err, ways, every_row, nfp64, st);
    else if (prec == kMixed)
        launch_one<float, double>(net, reg, ch, hs, tol, d_err, ways, every_row, nfp64, st);
    else
        launch_one<float, float>(net, reg, ch, hs, tol, d_err, ways, every_row, nfp64, st);
}

} // namespace am
