// Differentiable density calibration: forward run with a time-averaged bilinear
// density splat, MSE loss against a target density, and the hand-written adjoint
// of the kinematic step with respect to per-entity speeds and per-road speed
// factors.
//
// Forward (k_adj_forward, one thread per entity, all ticks in registers): the
// move step of the plain path with step length speed*factor[road]*dt; every K
// ticks the state is checkpointed; each position is splatted with cell-centred
// bilinear weights into a gw x gh grid over the world.  Weights are accumulated
// per entity in registers as fixed point (units of 2^-31) while the entity stays in
// the same 2 x 2 cell block and flushed with 64-bit integer atomics when it leaves:
// integer addition is associative, so the density is bit-identical from run to
// run whatever the order of the flushes.
//
// Discrete events (the tick at which an entity reaches its road end and the road
// it picks) are held fixed: the gradient is that of the piecewise-smooth model
// with the forward's event schedule.  Every natural forward stores the schedule
// (one bit per entity and tick); a forward can replay it, so that finite
// differences can be taken on the same model, and the backward always does.
//
// Backward, per segment of K ticks from the last to the first
// (k_adj_backward): recompute the segment from its checkpoint with the recorded
// events, store its positions, then sweep backwards:
//   a_t += (1/T) d splat(p_t)/dp . lambda,     lambda = dL/dD = 2/G (D - D*)
//   snap tick:     a_{t-1} = 0 (p_t = road end does not depend on p, speed, factor)
//   otherwise:     n = (target - p_{t-1})/L, l = s*f*dt, g = n . a_t
//                  dL/ds += g*f*dt,  dL/df_road += g*s*dt,
//                  a_{t-1} = a_t - (l/L)(a_t - n g)
// Speed gradients are owned by their entity (no reduction).  Road-factor
// contributions are flushed as (road, value) records, one per road visit per
// segment, then packed, sorted by road with the stable onesweep radix sort and summed
// per road in a fixed order: a deterministic segmented reduction, no float atomics.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "msim_chain.cuh"
#include "msim_internal.h"
#include "msim_kernels.cuh"

namespace msim {
namespace {

constexpr uint32_t kRecPerSeg = 8;  // road-visit records per entity and segment
constexpr uint32_t kRecBlock = 1024;  // entities whose records one block packs

struct AdjArgs {
    DeviceMap map;
    uint32_t n, ticks, K, sched_words;
    float dt, inv_cw, inv_ch;
    uint32_t gw, gh, fbits;
    const float2* pos0;
    const uint32_t* head0;
    const uint4* rng0;
    const float* speed;
    float2* ck_pos;
    uint32_t* ck_head;
    uint4* ck_rng;
    unsigned long long* dacc;
    uint32_t* sched;  // one bit per entity and tick
    uint32_t lanes;   // entities per warp (adj_entity)
    uint32_t* err;
};

// Threads of a block of the forward and backward kernels, and blocks per SM.  Both are
// bound by issue.  Forward: one warp a block, so that a slow warp keeps no finished one's
// place (262,144 entities 1.68 ms; 128 threads 1.80; before the paired instructions, as
// the figures that follow).  Backward: the history (800 B per
// entity at K = 100) of the resident threads then mostly stays in the L2 it is read back
// from (7 blocks of 128 threads 2.63 ms; 6 3.01, 8 at fewer registers 2.96, 24 of 32 2.94).
constexpr uint32_t kAdjForwardThreads = 32;
constexpr int kAdjForwardBlocks = 32;
constexpr uint32_t kAdjThreads = 128;
constexpr int kAdjBackwardBlocks = 7;

// The entity of a thread: `lanes` entities to a warp (32, fewer for small counts: the
// road ends and cell changes of one entity hold up the others of its warp).
__device__ __forceinline__ uint32_t adj_entity(uint32_t n, uint32_t lanes) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    const uint64_t e = (uint64_t)warp * lanes + lane;
    return lane < lanes && e < n ? (uint32_t)e : 0xffffffffu;
}

// Cell coordinates of a position: u = x * (gw / W) - 1/2 in binary32 (cell-centred),
// then U = floor(u * 2^fbits) as an integer (exact: a binary32 u below 2^(30-fbits)
// has no fractional bits beyond fbits once truncated there).  The cell is
// U >> fbits and the fraction fx = (U mod 2^fbits) / 2^fbits; fbits is the largest
// value (at most 22) that keeps U in 31 bits for the grid.
struct Splat {
    int i0, j0;
    uint32_t fx, fy;  // fractions in units of 2^-fbits
};
__device__ __forceinline__ int fixed_coord(float u, uint32_t fbits) {
    const float lim = __int_as_float((127 + 30 - (int)fbits) << 23);  // 2^(30 - fbits)
    u = fminf(fmaxf(u, -lim), lim);                                  // off-grid positions stay off-grid
    return __float2int_rd(__fmul_rn(u, __int_as_float((127 + (int)fbits) << 23)));
}
__device__ __forceinline__ Splat splat_of(float ux, float uy, uint32_t fbits) {
    const int U = fixed_coord(ux, fbits);
    const int V = fixed_coord(uy, fbits);
    const uint32_t mask = (1u << fbits) - 1u;
    Splat s;
    s.i0 = U >> fbits;  // arithmetic shift: floor
    s.j0 = V >> fbits;
    s.fx = (uint32_t)U & mask;
    s.fy = (uint32_t)V & mask;
    return s;
}
// The same without conversions while a position stays in the cell (fi, fj) of an
// earlier splat: u - fi towards zero is in [0, 1) exactly when floor(u) = fi (u - fi is
// exact for u >= 0; for u in [-1, 0) its truncation keeps every bit above 2^-24), and
// adding 2^(23 - fbits) towards zero leaves the fraction's first fbits bits as the low
// bits of the sum.  An entity stays about a hundred ticks in a cell.
struct CellFrame {
    float2 back;  // (-fi, -fj); NaN: no cell
    float one;    // 2^(23 - fbits)
};
__device__ __forceinline__ float2 add2_rz(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rz.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 cell_coords(float2 p, float2 inv_c) { return plus(both(-0.5f), mul2(p, inv_c)); }
__device__ __forceinline__ bool in_cell(const CellFrame& c, float2 u, float2& w) {
    const float2 d = add2_rz(u, c.back);
    w = add2_rz(d, both(c.one));
    return max(__float_as_uint(d.x), __float_as_uint(d.y)) < 0x3f800000u;
}
__device__ __forceinline__ float frame_one(uint32_t fbits) { return __int_as_float((150 - (int)fbits) << 23); }

// Per-entity sums over the ticks spent in one 2 x 2 cell block: the tick count and
// the sums of fx, fy and fx*fy give the four bilinear corner weights exactly.
struct BlockSums {
    uint32_t n;
    unsigned long long sx, sy, sxy;
};
__device__ __forceinline__ void flush_block(unsigned long long* dacc, uint32_t gw, uint32_t gh, int i0, int j0,
                                            const BlockSums& b, uint32_t fbits) {
    const unsigned long long F = 1ull << fbits;
    // corner weights in units of 2^-2fbits, then in the accumulator's 2^-31
    const unsigned long long w[4] = {(unsigned long long)b.n * F * F - F * (b.sx + b.sy) + b.sxy, F * b.sx - b.sxy,
                                     F * b.sy - b.sxy, b.sxy};
    const uint32_t sh = 2u * fbits - 31u;
    const int ci[4] = {i0, i0 + 1, i0, i0 + 1}, cj[4] = {j0, j0, j0 + 1, j0 + 1};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned long long v = w[k] >> sh;
        if (v && ci[k] >= 0 && cj[k] >= 0 && ci[k] < (int)gw && cj[k] < (int)gh)
            atomicAdd(&dacc[(size_t)cj[k] * gw + ci[k]], v);
    }
}

// Sums of blocks an entity has left, one per thread, until a lane of the warp leaves a
// second one: then every lane that has one flushes it.  An entity changes its cell once
// in about 70 ticks, so some lane of a warp does in 37 % of its ticks; waiting for the second
// change brings the flushes of about eight lanes together.
struct LeftBlocks {
    int i[kAdjForwardThreads], j[kAdjForwardThreads];
    uint32_t n[kAdjForwardThreads];  // 0: none
    unsigned long long sx[kAdjForwardThreads], sy[kAdjForwardThreads], sxy[kAdjForwardThreads];
};
__device__ __forceinline__ void flush_left(LeftBlocks& left, const AdjArgs& a) {
    const uint32_t t = threadIdx.x;
    if (left.n[t]) {
        flush_block(a.dacc, a.gw, a.gh, left.i[t], left.j[t], BlockSums{left.n[t], left.sx[t], left.sy[t], left.sxy[t]},
                    a.fbits);
        left.n[t] = 0u;
    }
}

// REPLAY: the stored event schedule is forced; else events come from the step and the
// schedule is stored.  Ticks run in stretches of at most 32 that end where a schedule
// word or a checkpoint does, so a tick itself is the step, the cell test and three
// sums (32-bit within a stretch).  Bound by issue (83 % active): 105 warp instructions
// per tick against 190 with the road reloaded, two conversions and a flush at every
// cell change; 262,144 entities x 2,000 ticks 3.13 -> 1.68 ms, with the coordinates in
// paired instructions 1.59, at 32 blocks per SM 1.57.
template <int RNG, bool REPLAY>
__global__ __launch_bounds__(kAdjForwardThreads, kAdjForwardBlocks) void k_adj_forward(AdjArgs a) {
    __shared__ LeftBlocks left;
    chain_enter();
    const uint32_t e = adj_entity(a.n, a.lanes);
    left.n[threadIdx.x] = 0u;
    const unsigned warp_mask = __ballot_sync(0xffffffffu, e != 0xffffffffu);
    if (e == 0xffffffffu) return;
    float2 p = a.pos0[e];
    uint32_t h = a.head0[e];
    uint4 r = a.rng0[e];
    const float s = a.speed[e];
    Leg l{};
    if (!leg_load<true>(a.map, a.dt, s, h, l, a.err)) {  // unreachable: headings come from the initializer
        h = 0u;
        leg_load<true>(a.map, a.dt, s, h, l, a.err);
    }
    const uint32_t low = (1u << a.fbits) - 1u;
    CellFrame c{both(__int_as_float(0x7fc00000)), frame_one(a.fbits)};  // in no cell yet
    int bi = INT32_MIN, bj = INT32_MIN;
    BlockSums acc{0u, 0ull, 0ull, 0ull};
    size_t ck = e;
    uint32_t until_ck = 0, bits = 0;
    for (uint32_t t = 0; t < a.ticks;) {
        if (until_ck == 0) {
            a.ck_pos[ck] = p;
            a.ck_head[ck] = h;
            a.ck_rng[ck] = r;
            ck += a.n;
            until_ck = a.K;
        }
        const uint32_t first = t & 31u;
        const uint32_t len = min(min(32u - first, until_ck), a.ticks - t);
        uint32_t* word = a.sched + (size_t)e * a.sched_words + (t >> 5);
        if (REPLAY) bits = *word >> first;
        uint32_t sx = 0u, sy = 0u, began = 0u;  // sums and first tick of this stretch in the block
#pragma unroll 2
        for (uint32_t k = 0; k < len; k++) {
            const int force = REPLAY ? (int)(bits & 1u) : -1;
            const bool snapped = step_leg<true, true>(a.map, a.dt, s, p, h, l, a.err, force,
                                                [&]() { return rng_next<RNG>(r); });
            if (REPLAY) bits >>= 1;
            else if (snapped) bits |= 1u << (first + k);
            const float2 u = cell_coords(p, make_float2(a.inv_cw, a.inv_ch));
            float2 w;
            const bool stays = in_cell(c, u, w);
            uint32_t fx = __float_as_uint(w.x) & low, fy = __float_as_uint(w.y) & low;
            bool leaves = false;
            Splat sp{};
            if (!stays) {
                sp = splat_of(u.x, u.y, a.fbits);
                fx = sp.fx;
                fy = sp.fy;
                leaves = sp.i0 != bi || sp.j0 != bj;
            }
            if (__any_sync(warp_mask, leaves && left.n[threadIdx.x] != 0u)) flush_left(left, a);
            if (leaves) {
                acc.n += k - began;
                if (acc.n) {
                    left.i[threadIdx.x] = bi;
                    left.j[threadIdx.x] = bj;
                    left.n[threadIdx.x] = acc.n;
                    left.sx[threadIdx.x] = acc.sx + sx;
                    left.sy[threadIdx.x] = acc.sy + sy;
                    left.sxy[threadIdx.x] = acc.sxy;
                }
                bi = sp.i0;
                bj = sp.j0;
                c.back = make_float2(-(float)bi, -(float)bj);
                acc = BlockSums{0u, 0ull, 0ull, 0ull};
                sx = sy = 0u;
                began = k;
            }
            sx += fx;
            sy += fy;
            acc.sxy += (unsigned long long)fx * fy;
        }
        acc.n += len - began;
        acc.sx += sx;
        acc.sy += sy;
        t += len;
        until_ck -= len;
        if (!REPLAY && ((t & 31u) == 0u || t == a.ticks)) {
            *word = bits;
            bits = 0u;
        }
    }
    flush_left(left, a);
    if (acc.n) flush_block(a.dacc, a.gw, a.gh, bi, bj, acc, a.fbits);
}

// density, lambda = 2/G (D - D*), per-block partial sums of (D - D*)^2
__global__ __launch_bounds__(256) void k_adj_loss(const unsigned long long* __restrict__ dacc,
                                                  const float* __restrict__ target, uint32_t G, uint32_t ticks,
                                                  float* density, float* lambda, double* partial) {
    __shared__ double s_sum[256];
    chain_enter();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    double d2 = 0.0;
    if (g < G) {
        const double D = (double)dacc[g] * 0x1p-31 / (double)ticks;
        const double diff = D - (double)target[g];
        density[g] = (float)D;
        lambda[g] = (float)(2.0 / (double)G * diff);
        d2 = diff * diff;
    }
    s_sum[threadIdx.x] = d2;
    __syncthreads();
    for (uint32_t o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s_sum[threadIdx.x] += s_sum[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = s_sum[0];
}

// The blocks' partial sums in a fixed order: strided by thread, then a tree (one thread
// adding 1,024 partials one after another took 54 us).
__global__ __launch_bounds__(256) void k_adj_loss_final(const double* partial, uint32_t blocks, uint32_t G,
                                                        double* loss) {
    __shared__ double s_sum[256];
    chain_enter();
    double s = 0.0;
    for (uint32_t b = threadIdx.x; b < blocks; b += 256u) s += partial[b];
    s_sum[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s_sum[threadIdx.x] += s_sum[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = s_sum[0] / (double)G;
}

struct AdjBack {
    AdjArgs f;
    uint32_t segments;
    const float* lambda;
    float2* hist_pos;     // [K + 1][n]: the segment's positions, its checkpoint first
    uint32_t* hist_head;  // [K][n]: headings before the segment's road ends, in order
    double* gspeed;
    float* gspeed_out;    // by entity id (may be NULL)
    const uint32_t* perm;
    uint2* rec;           // [n][segments * kRecPerSeg]: road, float bits of the gradient part
    uint32_t* rec_count;  // [n]
    uint32_t* rec_block;  // records per kRecBlock entities (accumulated)
    uint32_t num_roads;
};

__device__ __forceinline__ float lam_at(const float* lambda, uint32_t gw, uint32_t gh, int i, int j) {
    return (i < 0 || j < 0 || i >= (int)gw || j >= (int)gh) ? 0.f : __ldg(&lambda[(size_t)j * gw + i]);
}

// 1 / sqrt(d2) by the hardware instruction (rsqrtf's bits for normal d2, without its
// test for subnormal ones); 0 for d2 = 0, where the adjoint's terms then vanish.
__device__ __forceinline__ float inv_length(float d2) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d2));
    return d2 >= 1.17549435e-38f ? y : d2 > 0.f ? rsqrtf(d2) : 0.f;
}

// Gradient of the splat at a position, scaled by cells per metre and 1 / ticks, as two
// linear functions of the cell fractions: x = x0 + fy * x1, y = y0 + fx * y1.
struct SplatGrad {
    float x0, x1, y0, y1;
};
__device__ __noinline__ SplatGrad splat_grad(const float* lambda, uint32_t gw, uint32_t gh, int i, int j, float sx,
                                             float sy) {
    const float l00 = lam_at(lambda, gw, gh, i, j), l10 = lam_at(lambda, gw, gh, i + 1, j);
    const float l01 = lam_at(lambda, gw, gh, i, j + 1), l11 = lam_at(lambda, gw, gh, i + 1, j + 1);
    SplatGrad g;
    g.x0 = (l10 - l00) * sx;
    g.x1 = ((l11 - l01) - (l10 - l00)) * sx;
    g.y0 = (l01 - l00) * sy;
    g.y1 = ((l11 - l10) - (l01 - l00)) * sy;
    return g;
}

// Backward of one entity, segment by segment from the last to the first: recompute
// the segment's positions from its checkpoint (the event decisions from the schedule,
// the road choices from the checkpointed RNG, both exact; the position update with
// the hardware reciprocal square root, since the adjoint needs the positions only to
// about 1e-6 relative and snaps put them back on exact road ends), then sweep
// backwards over them.  The road's leg and the cell's gradient stay in registers until a
// road end or a cell change, the leg's gradient parts are summed before they are scaled,
// headings are kept only for road ends (12 -> 8 B of history per tick), ticks run in
// stretches of one schedule word, and all segments run in one launch, which a launch per
// segment rounded up to two waves each.  262,144 entities x 2,000 ticks 5.06 -> 2.63 ms,
// with the coordinates in paired instructions 2.52.
template <int RNG>
__global__ __launch_bounds__(kAdjThreads, kAdjBackwardBlocks) void k_adj_backward(AdjBack b) {
    chain_enter();
    const AdjArgs& a = b.f;
    const uint32_t e = adj_entity(a.n, a.lanes);
    if (e == 0xffffffffu) return;
    const size_t n = a.n;
    const float s = a.speed[e];
    const uint32_t* sched = a.sched + (size_t)e * a.sched_words;
    uint2* rec = b.rec + (size_t)e * b.segments * kRecPerSeg;
    uint32_t* ends = b.hist_head + e;
    const float invT = 1.0f / (float)a.ticks;
    const float sx = a.inv_cw * invT, sy = a.inv_ch * invT;
    const float scale = __int_as_float((127 - (int)a.fbits) << 23);  // 2^-fbits
    float2 adj = make_float2(0.f, 0.f);
    double gspeed = 0.0;
    uint32_t records = 0;
    CellFrame c{both(__int_as_float(0x7fc00000)), frame_one(a.fbits)};
    SplatGrad sg{};
    for (uint32_t seg = b.segments; seg-- > 0;) {
        const uint32_t t0 = seg * a.K, t1 = t0 + min(a.K, a.ticks - t0);  // ticks t0 + 1 .. t1
        const size_t ck = (size_t)seg * n + e;
        float2 p = a.ck_pos[ck];
        uint32_t h = a.ck_head[ck];
        uint4 r = a.ck_rng[ck];
        Leg l{};
        if (!leg_load<true>(a.map, a.dt, s, h, l, a.err)) {  // unreachable: the forward's headings
            h = 0u;
            leg_load<true>(a.map, a.dt, s, h, l, a.err);
        }
        float2* at = b.hist_pos + e;  // the segment's positions, its checkpoint first
        *at = p;
        uint32_t num_ends = 0;
        for (uint32_t t = t0; t < t1;) {  // recompute with the recorded events
            const uint32_t first = t & 31u, len = min(32u - first, t1 - t);
            uint32_t bits = __brev(sched[t >> 5]) << first;  // the next tick's event in the sign bit
            t += len;
#pragma unroll 4
            for (uint32_t k = 0; k < len; k++) {
                if ((int)bits >= 0) {
                    const float2 d = sub2(make_float2(l.tx, l.ty), p), dd = mul2(d, d);
                    p = plus(p, mul2(d, both(inv_length(dd.x + dd.y) * l.step)));
                } else {
                    p.x = l.tx;
                    p.y = l.ty;
                    ends[(size_t)num_ends++ * n] = h;
                    road_end<true>(a.map, a.dt, s, h, l, a.err, [&]() { return rng_next<RNG>(r); });
                }
                bits <<= 1;
                at += n;
                *at = p;
            }
        }
        // reverse sweep: p is the position after the tick, the history (fetched kAhead
        // ticks early) holds the one before it
        constexpr uint32_t kAhead = 4;
        float2 ahead[kAhead];
        uint32_t left = t1 - t0;  // ticks to sweep; the position before the next one is hist[left - 1]
#pragma unroll
        for (uint32_t q = 0; q < kAhead; q++) {
            if (q < left) at -= n;
            ahead[q] = *at;
        }
        float gs = 0.f, cur_sum = 0.f;
        uint32_t cur_road = b.num_roads, nrec = 0;
        uint32_t road = h & kHeadRoad;
        float f = a.map.factor ? __ldg(&a.map.factor[road]) : 1.0f;
        float part = 0.f;  // sum of n . adj over the leg
        bool any = false;
        auto record = [&]() {
            if (cur_road == b.num_roads) return;
            if (nrec < kRecPerSeg) {
                rec[records++] = make_uint2(cur_road, __float_as_uint(cur_sum));
                nrec++;
            } else {
                atomicOr(a.err, kErrOob);
            }
        };
        auto end_leg = [&]() {
            if (!any) return;
            if (road != cur_road) {
                record();
                cur_road = road;
                cur_sum = 0.f;
            }
            cur_sum += part * s * a.dt;
            gs += part * f * a.dt;
            part = 0.f;
            any = false;
        };
        for (uint32_t t = t1; t > t0;) {
            const uint32_t word_from = (t - 1u) & ~31u, from = max(word_from, t0), len = t - from;
            uint32_t bits = sched[word_from >> 5] << (31u - ((t - 1u) & 31u));  // this tick's event in the sign bit
            t = from;
#pragma unroll 4
            for (uint32_t k = 0; k < len; k++) {
                const float2 pp = ahead[0];
#pragma unroll
                for (uint32_t q = 0; q + 1u < kAhead; q++) ahead[q] = ahead[q + 1u];
                left--;
                if (left >= kAhead) at -= n;  // else the checkpoint again, not used
                ahead[kAhead - 1u] = *at;
                {  // + (1/T) d splat(p_t)/dp . lambda
                    const float2 u = cell_coords(p, make_float2(a.inv_cw, a.inv_ch));
                    float2 w, fr;  // fr: the cell fractions
                    if (in_cell(c, u, w)) {
                        fr = add2(w, both(-c.one));  // exact: fbits bits
                    } else {
                        const Splat sp = splat_of(u.x, u.y, a.fbits);
                        sg = splat_grad(b.lambda, a.gw, a.gh, sp.i0, sp.j0, sx, sy);
                        fr = make_float2((float)sp.fx * scale, (float)sp.fy * scale);  // exact: fewer than 24 bits
                        c.back = make_float2(-(float)sp.i0, -(float)sp.j0);
                    }
                    adj = add2(adj, make_float2(__fmaf_rn(fr.y, sg.x1, sg.x0), __fmaf_rn(fr.x, sg.y1, sg.y0)));
                }
                if ((int)bits >= 0) {
                    const float2 d = sub2(make_float2(l.tx, l.ty), pp);
                    const float d2 = __fmaf_rn(d.x, d.x, d.y * d.y);
                    const float inv = inv_length(d2);
                    const float g = __fmaf_rn(d.x, adj.x, d.y * adj.y) * inv;  // n . adj
                    part += g;
                    any = any || d2 > 0.f;
                    const float2 across = fma2(d, both(g * -inv), adj);  // adj - n g
                    adj = fma2(across, both(l.step * -inv), adj);
                } else {
                    end_leg();
                    adj = make_float2(0.f, 0.f);
                    h = ends[(size_t)--num_ends * n];  // the road before this tick
                    road = h & kHeadRoad;
                    l = leg_of<false>(a.map, a.dt, s, road, __ldg(&a.map.road_pos[road]), (h & kHeadToEnd) != 0);
                    f = a.map.factor ? __ldg(&a.map.factor[road]) : 1.0f;
                }
                bits <<= 1;
                p = pp;
            }
        }
        end_leg();
        record();
        gspeed += (double)gs;
    }
    b.gspeed[e] = gspeed;
    if (b.gspeed_out) b.gspeed_out[b.perm[e]] = (float)gspeed;
    b.rec_count[e] = records;
    if (records) atomicAdd(&b.rec_block[e / kRecBlock], records);
}

// Road gradients: the entities' records (about 30 of the 160 places of an entity are
// used at K = 100) are packed in entity order, sorted by road with the stable radix
// sort and summed per road.  One block: the exclusive scan of the records per
// kRecBlock entities (rec_block is left zeroed for the next backward), the total, and
// zeroed digit counts.
__global__ __launch_bounds__(1024) void k_adj_rec_scan(uint32_t* rec_block, uint32_t* rec_base, uint32_t blocks,
                                                       uint32_t* total, uint32_t* hist) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_run;
    chain_enter();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid < kMaxPasses * kRadix) hist[tid] = 0u;
    if (tid == 0) s_run = 0u;
    __syncthreads();
    for (uint32_t b0 = 0; b0 < blocks; b0 += 1024u) {
        const uint32_t i = b0 + tid;
        const uint32_t v = i < blocks ? rec_block[i] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t before = s_run;
        for (uint32_t w = 0; w < warp; w++) before += s_warp[w];
        if (i < blocks) {
            rec_base[i] = before + incl - v;
            rec_block[i] = 0u;
        }
        __syncthreads();
        if (tid == 1023u) s_run = before + incl;
        __syncthreads();
    }
    if (tid == 0) *total = s_run;
}

// One block per kRecBlock entities: their records end to end, 256 at a time (the
// entity of a record by binary search in the scanned counts), and the roads' digits.
__global__ __launch_bounds__(256) void k_adj_rec_pack(const uint2* __restrict__ rec,
                                                      const uint32_t* __restrict__ rec_count,
                                                      const uint32_t* __restrict__ rec_base, uint32_t n, uint32_t places,
                                                      uint32_t passes, uint32_t* __restrict__ key,
                                                      uint32_t* __restrict__ val, uint32_t* hist) {
    constexpr uint32_t kPer = kRecBlock / 256u;
    __shared__ uint32_t s_first[kRecBlock + 1];  // records before each entity of the block
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    chain_enter();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid; i < passes * kRadix; i += 256u) s_hist[i] = 0u;
    const uint32_t e0 = blockIdx.x * kRecBlock;
    uint32_t v[kPer], sum = 0u;
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++) {
        const uint32_t e = e0 + tid * kPer + k;
        v[k] = e < n ? rec_count[e] : 0u;
        sum += v[k];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t run = incl - sum;
    for (uint32_t w = 0; w < warp; w++) run += s_warp[w];
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++) {
        s_first[tid * kPer + k] = run;
        run += v[k];
    }
    if (tid == 255u) s_first[kRecBlock] = run;
    __syncthreads();
    const uint32_t count = s_first[kRecBlock], base = rec_base[blockIdx.x];
    for (uint32_t i = tid; i < count; i += 256u) {
        uint32_t o = 0;  // last entity that begins at or before record i
#pragma unroll
        for (uint32_t st = kRecBlock / 2u; st > 0; st >>= 1)
            if (s_first[o + st] <= i) o += st;
        const uint2 x = rec[(size_t)(e0 + o) * places + (i - s_first[o])];
        key[base + i] = x.x;
        val[base + i] = x.y;
        for (uint32_t ps = 0; ps < passes; ps++) atomicAdd(&s_hist[ps * kRadix + ((x.x >> (8u * ps)) & 0xffu)], 1u);
    }
    __syncthreads();
    for (uint32_t i = tid; i < passes * kRadix; i += 256u)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// One warp per road: its run of the sorted records by two binary searches (lanes 0 and
// 1), summed in double strided by lane, then a tree: a fixed order.
__global__ __launch_bounds__(256) void k_adj_road_sum(const uint32_t* __restrict__ key, const float* __restrict__ val,
                                                      const uint32_t* __restrict__ total, uint32_t num_roads,
                                                      double* gfactor, float* out, const uint32_t* err) {
    chain_enter();
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t rd = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (rd >= num_roads || (*err & kErrTimeout)) return;  // uniform per warp
    uint32_t lo = 0, hi = *total;
    const uint32_t want = rd + (lane & 1u);  // first record of road `want` or later
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (key[mid] < want) lo = mid + 1u;
        else hi = mid;
    }
    const uint32_t from = __shfl_sync(FULL, lo, 0), to = __shfl_sync(FULL, lo, 1);
    double s = 0.0;
    for (uint32_t q = from + lane; q < to; q += 32u) s += (double)val[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
    if (lane == 0) {
        gfactor[rd] = s;
        if (out) out[rd] = (float)s;
    }
}

// Entities are kept in spatial order inside the context (perm[i] = entity id of
// internal index i); this moves a per-entity array across that boundary.
__global__ void k_adj_gather(const float* __restrict__ in, const uint32_t* __restrict__ perm, uint32_t n,
                             float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[perm[i]];
}

int cuda_fail(cudaError_t e, const char* what) {
    cudaGetLastError();
    return fail(MSIM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
#define ACK(expr, what)                                    \
    do {                                                   \
        cudaError_t e_ = (expr);                           \
        if (e_ != cudaSuccess) return cuda_fail(e_, what); \
    } while (0)

}  // namespace
}  // namespace msim

using namespace msim;

struct msim_adj {
    int device = 0;
    cudaStream_t stream = nullptr;
    msim_adj_params p{};
    uint32_t n = 0, R = 0, C = 0, S = 0, sched_words = 0, passes = 1;
    float world_w = 0, world_h = 0;
    std::vector<void*> allocs;
    float4* road_pos = nullptr;
    uint4* road_conn = nullptr;
    uint32_t* conn = nullptr;
    float* speed = nullptr;
    float* factor = nullptr;
    float* target = nullptr;
    float2* pos0 = nullptr;
    uint32_t* head0 = nullptr;
    uint4* rng0 = nullptr;
    float2* ck_pos = nullptr;
    uint32_t* ck_head = nullptr;
    uint4* ck_rng = nullptr;
    unsigned long long* dacc = nullptr;
    float* density = nullptr;
    float* lambda = nullptr;
    double* partial = nullptr;
    double* loss = nullptr;
    uint32_t* sched = nullptr;
    float2* hist_pos = nullptr;
    uint32_t* hist_head = nullptr;
    double* gspeed = nullptr;
    double* gfactor = nullptr;
    uint2* rec = nullptr;             // road-visit records, a fixed place count per entity
    uint32_t* rec_used = nullptr;     // records of each entity
    uint32_t* rec_block = nullptr;    // records per kRecBlock entities (zero between backwards)
    uint32_t* rec_base = nullptr;     // their exclusive scan
    uint32_t* rec_total = nullptr;
    uint32_t* sk[2] = {nullptr, nullptr};
    uint32_t* sv[2] = {nullptr, nullptr};
    uint32_t* hist = nullptr;
    uint32_t* lookback = nullptr;
    uint32_t* tickets = nullptr;
    uint32_t* sort_dirty = nullptr;   // look-back words each region's last pass published
    bool sort_clean = false;          // regions, tickets and extents are as the chained passes expect
    uint32_t lanes = 32;
    uint32_t* err = nullptr;
    StatusWord status_host;          // page-locked copy of *err
    uint32_t* perm = nullptr;        // device: entity id of each internal index
    std::vector<uint32_t> hperm;     // host copy
    size_t rec_count = 0;
    size_t sort_region = 0;           // look-back words per pass
    bool sort_large = false;          // 4096-record tiles (else 1024)
    bool have_forward = false;
    bool have_backward = false;
    bool have_sched = false;
    uint32_t last_mode = 0;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    cudaEvent_t ph[6] = {};  // forward: kernel start/end, loss end; backward: start, sweeps end, end
};

namespace {

template <typename T>
int aalloc(msim_adj* a, T** ptr, size_t count) {
    void* raw = nullptr;
    if (!device_malloc(&raw, std::max<size_t>(count, 1) * sizeof(T)))
        return fail(MSIM_ERR_NOMEM, "device allocation failed in the adjoint context");
    a->allocs.push_back(raw);
    *ptr = static_cast<T*>(raw);
    return MSIM_OK;
}

void free_adj(msim_adj* a) {
    for (void* p : a->allocs) cudaFree(p);
    a->allocs.clear();
    if (a->t0) cudaEventDestroy(a->t0);
    if (a->t1) cudaEventDestroy(a->t1);
    for (cudaEvent_t& ev : a->ph)
        if (ev) cudaEventDestroy(ev);
    if (a->stream) cudaStreamDestroy(a->stream);
}

// Fraction bits of the splat's fixed-point cell coordinates: the largest value
// (at most 22, at least 16) with |u| * 2^fbits below 2^30 for u in (-1, max(gw, gh)).
uint32_t splat_fraction_bits(uint32_t gw, uint32_t gh) {
    const uint32_t g = std::max(gw, gh);
    uint32_t b = 0;
    while ((1ull << b) < (uint64_t)g + 1u) b++;
    const int fb = 30 - (int)b;
    return (uint32_t)std::max(16, std::min(22, fb));
}

// Entities per warp: 32, halved (to kAdjMinLanes) while that leaves the schedulers
// fewer than two warps each.  Small counts are bound by the latency of a tick, and the
// road end or cell change of one lane adds to every lane of its warp.
constexpr uint32_t kAdjMinLanes = 8;
uint32_t adj_lanes(uint32_t n, int sms) {
    uint32_t lanes = 32;
    while (lanes > kAdjMinLanes && n / lanes < 8u * (uint32_t)std::max(sms, 1)) lanes /= 2;
    return lanes;
}
unsigned adj_blocks(const msim_adj* a, uint32_t threads) {
    const uint64_t warps = ((uint64_t)a->n + a->lanes - 1u) / a->lanes;
    return (unsigned)((warps * 32u + threads - 1u) / threads);
}

AdjArgs fwd_args(msim_adj* a) {
    AdjArgs f{};
    f.map.road_pos = a->road_pos;
    f.map.road_conn = a->road_conn;
    f.map.conn = a->conn;
    f.map.factor = a->factor;
    f.map.num_roads = a->R;
    f.map.num_conn = a->C;
    f.n = a->n;
    f.ticks = a->p.ticks;
    f.K = a->p.checkpoint_interval;
    f.sched_words = a->sched_words;
    f.dt = a->p.dt;
    f.inv_cw = (float)((double)a->p.grid_w / (double)a->world_w);
    f.inv_ch = (float)((double)a->p.grid_h / (double)a->world_h);
    f.fbits = splat_fraction_bits(a->p.grid_w, a->p.grid_h);
    f.gw = a->p.grid_w;
    f.gh = a->p.grid_h;
    f.pos0 = a->pos0;
    f.head0 = a->head0;
    f.rng0 = a->rng0;
    f.speed = a->speed;
    f.ck_pos = a->ck_pos;
    f.ck_head = a->ck_head;
    f.ck_rng = a->ck_rng;
    f.dacc = a->dacc;
    f.sched = a->sched;
    f.lanes = a->lanes;
    f.err = a->err;
    return f;
}

int check_status(msim_adj* a) {
    ACK(cudaMemcpyAsync(a->status_host, a->err, sizeof(uint32_t), cudaMemcpyDeviceToHost, a->stream),
        "read device status");
    ACK(cudaStreamSynchronize(a->stream), "cudaStreamSynchronize");
    const uint32_t h = *static_cast<volatile uint32_t*>(a->status_host);
    if (h) {
        ACK(cudaMemset(a->err, 0, sizeof(uint32_t)), "clear device status");
        a->sort_clean = false;
        if (h & kErrTimeout) return fail(MSIM_ERR_TIMEOUT, "a bounded device wait gave up in the road-gradient sort");
        return fail(MSIM_ERR_OOB, "device-side index check failed in the adjoint (or more than 8 road visits per "
                                  "entity in one checkpoint segment)");
    }
    return MSIM_OK;
}

}  // namespace

namespace {
// host scatter of an internal-order array to entity-id order
template <typename T>
void to_entity_order(const std::vector<uint32_t>& perm, const T* in, T* out, size_t width = 1) {
    for (size_t i = 0; i < perm.size(); i++)
        for (size_t w = 0; w < width; w++) out[(size_t)perm[i] * width + w] = in[i * width + w];
}
}  // namespace

extern "C" {

int msim_adj_create(const msim_map* map, const msim_adj_params* params, msim_adj** out) {
    if (!out) return fail(MSIM_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (!map || !params) return fail(MSIM_ERR_INVALID, "NULL argument");
    int rc = validate_map(*map);
    if (rc != MSIM_OK) return rc;
    const msim_adj_params& p = *params;
    if (p.num_entities == 0 || p.num_entities >= (1u << 28)) return fail(MSIM_ERR_INVALID, "num_entities out of range");
    if (p.ticks == 0 || p.checkpoint_interval == 0) return fail(MSIM_ERR_INVALID, "ticks and checkpoint_interval must be > 0");
    if (p.grid_w == 0 || p.grid_h == 0 || (uint64_t)p.grid_w * p.grid_h > (1ull << 26) || p.grid_w > 16384u ||
        p.grid_h > 16384u)
        return fail(MSIM_ERR_INVALID, "density grid size out of range");
    if (p.rng_kind > 1 || p.placement > 1) return fail(MSIM_ERR_INVALID, "unknown rng_kind or placement");
    if (!(p.dt > 0.f) || !(p.speed_max >= p.speed_min)) return fail(MSIM_ERR_INVALID, "bad dt or speed range");
    if (map->num_roads >= (1u << 30)) return fail(MSIM_ERR_INVALID, "too many roads");
    msim_adj* a = new (std::nothrow) msim_adj();
    if (!a) return fail(MSIM_ERR_NOMEM, "out of host memory");
    auto bail = [&](int code) {
        free_adj(a);
        delete a;
        return code;
    };
    cudaGetDevice(&a->device);
    a->p = p;
    a->n = p.num_entities;
    a->R = map->num_roads;
    a->C = map->num_connections;
    a->world_w = map->width;
    a->world_h = map->height;
    a->S = (p.ticks + p.checkpoint_interval - 1) / p.checkpoint_interval;
    a->sched_words = (p.ticks + 31) / 32;
    uint32_t bits = 1;
    while ((1ull << bits) <= a->R) bits++;  // keys 0..R (R = unused record)
    a->passes = (bits + 7) / 8;
    if (a->passes > kMaxPasses) return bail(fail(MSIM_ERR_INVALID, "too many roads for the record sort"));
    a->rec_count = (size_t)a->S * a->n * kRecPerSeg;
    if (a->rec_count >= (1ull << 30)) return bail(fail(MSIM_ERR_INVALID, "ticks x entities too large for the record sort"));
    // about one record place in six is used: 1024-record tiles where 4096-record ones
    // would leave most of the chip idle
    a->sort_large = a->rec_count >= (1u << 22);
    a->sort_region = a->sort_large ? (a->rec_count + kSortTile - 1) / kSortTile * kRadix
                                   : sort_lookback_words((uint32_t)a->rec_count);
    int sms = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, a->device);
    a->lanes = adj_lanes(a->n, sms);
    cudaError_t e = cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return bail(cuda_fail(e, "cudaStreamCreate"));
    if (!a->status_host.take())
        return bail(fail(MSIM_ERR_NOMEM, "page-locked allocation of the status word failed"));
    cudaEventCreate(&a->t0);
    cudaEventCreate(&a->t1);
    for (cudaEvent_t& ev : a->ph) cudaEventCreate(&ev);
    const size_t n = a->n, G = (size_t)p.grid_w * p.grid_h, K = p.checkpoint_interval;
    if ((rc = aalloc(a, &a->road_pos, a->R)) || (rc = aalloc(a, &a->road_conn, a->R)) ||
        (rc = aalloc(a, &a->conn, (size_t)a->C + 1)) || (rc = aalloc(a, &a->speed, n)) ||
        (rc = aalloc(a, &a->factor, a->R)) || (rc = aalloc(a, &a->target, G)) || (rc = aalloc(a, &a->pos0, n)) ||
        (rc = aalloc(a, &a->head0, n)) || (rc = aalloc(a, &a->rng0, n)) || (rc = aalloc(a, &a->ck_pos, a->S * n)) ||
        (rc = aalloc(a, &a->ck_head, a->S * n)) || (rc = aalloc(a, &a->ck_rng, a->S * n)) ||
        (rc = aalloc(a, &a->dacc, G)) || (rc = aalloc(a, &a->density, G)) || (rc = aalloc(a, &a->lambda, G)) ||
        (rc = aalloc(a, &a->partial, (G + 255) / 256)) || (rc = aalloc(a, &a->loss, 1)) ||
        (rc = aalloc(a, &a->sched, n * a->sched_words)) || (rc = aalloc(a, &a->hist_pos, (K + 1) * n)) ||
        (rc = aalloc(a, &a->hist_head, K * n)) || (rc = aalloc(a, &a->gspeed, n)) ||
        (rc = aalloc(a, &a->gfactor, a->R)) || (rc = aalloc(a, &a->rec, a->rec_count)) ||
        (rc = aalloc(a, &a->rec_used, n)) || (rc = aalloc(a, &a->rec_block, (n + kRecBlock - 1) / kRecBlock)) ||
        (rc = aalloc(a, &a->rec_base, (n + kRecBlock - 1) / kRecBlock)) || (rc = aalloc(a, &a->rec_total, 1)) ||
        (rc = aalloc(a, &a->sk[0], a->rec_count)) ||
        (rc = aalloc(a, &a->sk[1], a->rec_count)) || (rc = aalloc(a, &a->sv[0], a->rec_count)) ||
        (rc = aalloc(a, &a->sv[1], a->rec_count)) || (rc = aalloc(a, &a->hist, (size_t)kMaxPasses * kRadix)) ||
        (rc = aalloc(a, &a->lookback, a->passes * a->sort_region)) ||
        (rc = aalloc(a, &a->tickets, (size_t)kMaxPasses)) || (rc = aalloc(a, &a->sort_dirty, (size_t)kMaxPasses)) ||
        (rc = aalloc(a, &a->err, 1)) || (rc = aalloc(a, &a->perm, n)))
        return bail(rc);
    std::vector<uint32_t> conn(a->C + 1);
    if (a->C) std::memcpy(conn.data(), map->connections, sizeof(uint32_t) * a->C);
    conn[a->C] = a->C ? map->connections[a->C - 1] : 0u;
    std::vector<float> ones(a->R, 1.0f);
    e = cudaMemcpy(a->road_pos, map->road_pos, sizeof(float4) * a->R, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(a->road_conn, map->road_conn, sizeof(uint4) * a->R, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(a->conn, conn.data(), sizeof(uint32_t) * (a->C + 1), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(a->factor, ones.data(), sizeof(float) * a->R, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(a->err, 0, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(a->rec_block, 0, sizeof(uint32_t) * ((n + kRecBlock - 1) / kRecBlock));
    if (e == cudaSuccess) e = cudaMemset(a->target, 0, sizeof(float) * G);
    if (e != cudaSuccess) return bail(cuda_fail(e, "adjoint set-up"));
    // initial entity state: the deterministic initializer of msim_init_entities
    DeviceMap m{};
    m.road_pos = a->road_pos;
    m.road_conn = a->road_conn;
    m.conn = a->conn;
    m.num_roads = a->R;
    m.num_conn = a->C;
    EntityState st{};
    st.pos = a->pos0;
    st.head = a->head0;
    st.rng = a->rng0;
    st.speed = a->speed;
    st.slot_id = a->hist_head;  // scratch for the slot ids the initializer writes
    e = launch_init_entities(a->stream, m, st, a->n, p.rng_kind, p.seed, p.placement, p.speed_min, p.speed_max);
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    if (e != cudaSuccess) return bail(cuda_fail(e, "adjoint entity init"));
    // spatial order: entities sorted (stably) by the Morton code of their initial
    // density cell, so a warp's cell gathers and flushes touch nearby cells
    {
        std::vector<float2> pos(n);
        std::vector<uint32_t> head(n), spd(n);
        std::vector<uint4> rng(n);
        e = cudaMemcpy(pos.data(), a->pos0, sizeof(float2) * n, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(head.data(), a->head0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(rng.data(), a->rng0, sizeof(uint4) * n, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(spd.data(), a->speed, sizeof(float) * n, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return bail(cuda_fail(e, "adjoint spatial order"));
        const double sx = (double)p.grid_w / (double)a->world_w, sy = (double)p.grid_h / (double)a->world_h;
        std::vector<uint32_t> key(n);
        for (size_t i = 0; i < n; i++) {
            const double cx = std::min(std::max((double)pos[i].x * sx, 0.0), (double)p.grid_w - 1.0);
            const double cy = std::min(std::max((double)pos[i].y * sy, 0.0), (double)p.grid_h - 1.0);
            key[i] = morton2((uint32_t)cx, (uint32_t)cy);
        }
        a->hperm.resize(n);
        for (size_t i = 0; i < n; i++) a->hperm[i] = (uint32_t)i;
        std::stable_sort(a->hperm.begin(), a->hperm.end(), [&](uint32_t x, uint32_t y) { return key[x] < key[y]; });
        std::vector<float2> pos2(n);
        std::vector<uint32_t> head2(n), spd2(n);
        std::vector<uint4> rng2(n);
        for (size_t i = 0; i < n; i++) {
            const uint32_t id = a->hperm[i];
            pos2[i] = pos[id];
            head2[i] = head[id];
            rng2[i] = rng[id];
            spd2[i] = spd[id];
        }
        e = cudaMemcpy(a->pos0, pos2.data(), sizeof(float2) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(a->head0, head2.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(a->rng0, rng2.data(), sizeof(uint4) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(a->speed, spd2.data(), sizeof(float) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(a->perm, a->hperm.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return bail(cuda_fail(e, "adjoint spatial order"));
    }
    *out = a;
    return MSIM_OK;
}


int msim_adj_destroy(msim_adj* a) {
    if (!a) return MSIM_OK;
    cudaSetDevice(a->device);
    cudaStreamSynchronize(a->stream);
    free_adj(a);
    delete a;
    return MSIM_OK;
}

int msim_adj_get_initial_state(msim_adj* a, float* pos, uint32_t* heading, uint32_t* rng, float* speed) {
    if (!a) return fail(MSIM_ERR_INVALID, "NULL argument");
    cudaSetDevice(a->device);
    ACK(cudaStreamSynchronize(a->stream), "sync");
    const size_t n = a->n;
    std::vector<uint32_t> tmp(4 * n);
    if (pos) {
        ACK(cudaMemcpy(tmp.data(), a->pos0, sizeof(float2) * n, cudaMemcpyDeviceToHost), "download");
        to_entity_order(a->hperm, reinterpret_cast<const float*>(tmp.data()), pos, 2);
    }
    if (heading) {
        ACK(cudaMemcpy(tmp.data(), a->head0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost), "download");
        to_entity_order(a->hperm, tmp.data(), heading);
    }
    if (rng) {
        ACK(cudaMemcpy(tmp.data(), a->rng0, sizeof(uint4) * n, cudaMemcpyDeviceToHost), "download");
        to_entity_order(a->hperm, tmp.data(), rng, 4);
    }
    // the current speeds: the initializer's until a forward passes others
    if (speed) {
        ACK(cudaMemcpy(tmp.data(), a->speed, sizeof(float) * n, cudaMemcpyDeviceToHost), "download");
        to_entity_order(a->hperm, reinterpret_cast<const float*>(tmp.data()), speed);
    }
    return MSIM_OK;
}

int msim_adj_forward(msim_adj* a, const float* d_speed, const float* d_factor, const float* d_target,
                     float* d_density, uint32_t mode, double* loss) {
    msim::NvtxRange range("msim_adj_forward");
    if (!a) return fail(MSIM_ERR_INVALID, "NULL argument");
    if (mode > 2) return fail(MSIM_ERR_INVALID, "mode must be 0 (natural), 1 (record events) or 2 (replay events)");
    if (mode == 2 && !a->have_sched) return fail(MSIM_ERR_INVALID, "no recorded event schedule to replay");
    cudaSetDevice(a->device);
    const size_t n = a->n, G = (size_t)a->p.grid_w * a->p.grid_h;
    if (d_speed) {
        k_adj_gather<<<(unsigned)((n + 255) / 256), 256, 0, a->stream>>>(d_speed, a->perm, a->n, a->speed);
        ACK(cudaGetLastError(), "speed");
    }
    if (d_factor)
        ACK(cudaMemcpyAsync(a->factor, d_factor, sizeof(float) * a->R, cudaMemcpyDeviceToDevice, a->stream), "factor");
    if (d_target)
        ACK(cudaMemcpyAsync(a->target, d_target, sizeof(float) * G, cudaMemcpyDeviceToDevice, a->stream), "target");
    ACK(cudaMemsetAsync(a->dacc, 0, sizeof(unsigned long long) * G, a->stream), "memset density");
    const AdjArgs f = fwd_args(a);
    const unsigned blocks = adj_blocks(a, kAdjForwardThreads);
    cudaEventRecord(a->ph[0], a->stream);
    if (a->p.rng_kind == 1) {
        if (mode == MSIM_ADJ_REPLAY) k_adj_forward<1, true><<<blocks, kAdjForwardThreads, 0, a->stream>>>(f);
        else k_adj_forward<1, false><<<blocks, kAdjForwardThreads, 0, a->stream>>>(f);
    } else {
        if (mode == MSIM_ADJ_REPLAY) k_adj_forward<0, true><<<blocks, kAdjForwardThreads, 0, a->stream>>>(f);
        else k_adj_forward<0, false><<<blocks, kAdjForwardThreads, 0, a->stream>>>(f);
    }
    ACK(cudaGetLastError(), "k_adj_forward");
    cudaEventRecord(a->ph[1], a->stream);
    const unsigned gb = (unsigned)((G + 255) / 256);
    ACK(launch_chained(k_adj_loss, gb, 256, a->stream, a->dacc, a->target, (uint32_t)G, a->p.ticks, a->density,
                       a->lambda, a->partial),
        "k_adj_loss");
    ACK(launch_chained(k_adj_loss_final, 1, 256, a->stream, a->partial, gb, (uint32_t)G, a->loss), "k_adj_loss_final");
    cudaEventRecord(a->ph[2], a->stream);
    if (d_density)
        ACK(cudaMemcpyAsync(d_density, a->density, sizeof(float) * G, cudaMemcpyDeviceToDevice, a->stream), "density");
    if (loss) ACK(cudaMemcpyAsync(loss, a->loss, sizeof(double), cudaMemcpyDeviceToHost, a->stream), "loss");
    int rc = check_status(a);
    if (rc != MSIM_OK) return rc;
    a->have_forward = true;
    a->last_mode = mode;
    a->have_sched = true;
    return MSIM_OK;
}

int msim_adj_backward(msim_adj* a, float* d_grad_speed, float* d_grad_factor) {
    msim::NvtxRange range("msim_adj_backward");
    if (!a) return fail(MSIM_ERR_INVALID, "NULL argument");
    if (!a->have_forward) return fail(MSIM_ERR_INVALID, "backward needs a forward first");
    cudaSetDevice(a->device);
    AdjBack b{};
    b.f = fwd_args(a);
    b.segments = a->S;
    b.lambda = a->lambda;
    b.hist_pos = a->hist_pos;
    b.hist_head = a->hist_head;
    b.gspeed = a->gspeed;
    b.gspeed_out = d_grad_speed;
    b.perm = a->perm;
    b.rec = a->rec;
    b.rec_count = a->rec_used;
    b.rec_block = a->rec_block;
    b.num_roads = a->R;
    cudaEventRecord(a->ph[3], a->stream);
    if (a->p.rng_kind == 1) k_adj_backward<1><<<adj_blocks(a, kAdjThreads), kAdjThreads, 0, a->stream>>>(b);
    else k_adj_backward<0><<<adj_blocks(a, kAdjThreads), kAdjThreads, 0, a->stream>>>(b);
    ACK(cudaGetLastError(), "k_adj_backward");
    cudaEventRecord(a->ph[4], a->stream);
    // road gradients: the records packed, stably sorted by road, summed per road
    const uint32_t rec_blocks = (a->n + kRecBlock - 1u) / kRecBlock;
    ACK(launch_chained(k_adj_rec_scan, 1, 1024, a->stream, a->rec_block, a->rec_base, rec_blocks, a->rec_total, a->hist),
        "k_adj_rec_scan");
    ACK(launch_chained(k_adj_rec_pack, rec_blocks, 256, a->stream, a->rec, a->rec_used, a->rec_base, a->n,
                       a->S * kRecPerSeg, a->passes, a->sk[0], a->sv[0], a->hist),
        "k_adj_rec_pack");
    // with two or more passes each clears the next one's look-back words and ticket
    const bool chained = a->passes >= 2;
    if (!a->sort_clean || !chained) {
        ACK(cudaMemsetAsync(a->lookback, 0, sizeof(uint32_t) * a->passes * a->sort_region, a->stream), "memset lookback");
        ACK(cudaMemsetAsync(a->tickets, 0, sizeof(uint32_t) * kMaxPasses, a->stream), "memset tickets");
        ACK(cudaMemsetAsync(a->sort_dirty, 0, sizeof(uint32_t) * kMaxPasses, a->stream), "memset look-back extents");
    }
    a->sort_clean = false;  // until every pass has launched
    for (uint32_t ps = 0; ps < a->passes; ps++) {
        SweepChain ch;
        const uint32_t nx = (ps + 1u) % a->passes;
        ch.next_lookback = a->lookback + nx * a->sort_region;
        ch.next_ticket = a->tickets + nx;
        ch.next_dirty = a->sort_dirty + nx;
        ch.my_dirty = a->sort_dirty + ps;
        ACK(launch_onesweep(a->stream, a->sk[ps & 1], a->sv[ps & 1], a->sk[(ps + 1) & 1], a->sv[(ps + 1) & 1],
                            (uint32_t)a->rec_count, 8u * ps, a->hist + ps * kRadix, a->lookback + ps * a->sort_region,
                            a->tickets + ps, a->err, a->rec_total, chained ? &ch : nullptr, kDefaultSpinLimit,
                            a->sort_large),
            "k_onesweep");
    }
    a->sort_clean = true;
    ACK(launch_chained(k_adj_road_sum, (a->R + 7u) / 8u, 256, a->stream, a->sk[a->passes & 1],
                       reinterpret_cast<const float*>(a->sv[a->passes & 1]), a->rec_total, a->R, a->gfactor, d_grad_factor,
                       a->err),
        "k_adj_road_sum");
    cudaEventRecord(a->ph[5], a->stream);
    a->have_backward = true;
    return check_status(a);
}

int msim_adj_phase_times(msim_adj* a, float ms[4]) {
    if (!a || !ms) return fail(MSIM_ERR_INVALID, "NULL argument");
    if (!a->have_forward || !a->have_backward) return fail(MSIM_ERR_INVALID, "needs a forward and a backward first");
    cudaSetDevice(a->device);
    ACK(cudaStreamSynchronize(a->stream), "sync");
    ACK(cudaEventElapsedTime(&ms[0], a->ph[0], a->ph[1]), "cudaEventElapsedTime");
    ACK(cudaEventElapsedTime(&ms[1], a->ph[1], a->ph[2]), "cudaEventElapsedTime");
    ACK(cudaEventElapsedTime(&ms[2], a->ph[3], a->ph[4]), "cudaEventElapsedTime");
    ACK(cudaEventElapsedTime(&ms[3], a->ph[4], a->ph[5]), "cudaEventElapsedTime");
    return MSIM_OK;
}

int msim_adj_get_gradients_f64(msim_adj* a, double* grad_speed, double* grad_factor) {
    if (!a) return fail(MSIM_ERR_INVALID, "NULL argument");
    cudaSetDevice(a->device);
    ACK(cudaStreamSynchronize(a->stream), "sync");
    if (grad_speed) {
        std::vector<double> tmp(a->n);
        ACK(cudaMemcpy(tmp.data(), a->gspeed, sizeof(double) * a->n, cudaMemcpyDeviceToHost), "download");
        to_entity_order(a->hperm, tmp.data(), grad_speed);
    }
    if (grad_factor) ACK(cudaMemcpy(grad_factor, a->gfactor, sizeof(double) * a->R, cudaMemcpyDeviceToHost), "download");
    return MSIM_OK;
}

int msim_adj_get_schedule(msim_adj* a, uint32_t* words) {
    if (!a || !words) return fail(MSIM_ERR_INVALID, "NULL argument");
    if (!a->have_sched) return fail(MSIM_ERR_INVALID, "no recorded event schedule");
    cudaSetDevice(a->device);
    ACK(cudaStreamSynchronize(a->stream), "sync");
    std::vector<uint32_t> tmp((size_t)a->n * a->sched_words);
    ACK(cudaMemcpy(tmp.data(), a->sched, sizeof(uint32_t) * tmp.size(), cudaMemcpyDeviceToHost), "download schedule");
    to_entity_order(a->hperm, tmp.data(), words, a->sched_words);
    return MSIM_OK;
}

int msim_adj_timer_begin(msim_adj* a) {
    if (!a) return fail(MSIM_ERR_INVALID, "NULL argument");
    ACK(cudaEventRecord(a->t0, a->stream), "cudaEventRecord");
    return MSIM_OK;
}

int msim_adj_timer_end(msim_adj* a, float* ms) {
    if (!a || !ms) return fail(MSIM_ERR_INVALID, "NULL argument");
    ACK(cudaEventRecord(a->t1, a->stream), "cudaEventRecord");
    ACK(cudaEventSynchronize(a->t1), "cudaEventSynchronize");
    ACK(cudaEventElapsedTime(ms, a->t0, a->t1), "cudaEventElapsedTime");
    return MSIM_OK;
}

}  // extern "C"
