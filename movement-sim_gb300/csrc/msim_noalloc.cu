// msim_query_neighbours_noalloc: the radius neighbour query (the neighbour sets of
// msim_step with MSIM_STEP_NEIGHBOURS) for positions the caller already holds on the
// device, without allocating any memory.
//
// Who needs this: callers that cannot call cudaMalloc at the point where they
// want neighbour sets.  cudaMalloc may synchronise the whole device and is not
// permitted while the calling thread is capturing a stream into a CUDA graph; a
// host application that hands all device memory to its own pool at start-up, or
// a tick loop that must never block in the allocator, cannot create an msim
// context (which allocates its buffers in msim_create and its export staging on
// first use).  This entry point takes device pointers for its inputs and
// outputs and keeps every intermediate (cell counts and starts, ranks, positions and
// ids in cell order) in one file-scope __device__ array of fixed size, so it calls no
// cudaMalloc, cudaFree or other allocating routine.
//
// The array is shared by every call on a device and keeps the last call's
// contents; each call clears what must start at zero.  Calls whose GPU work
// overlaps (two streams, or two host threads) race on the array: serialise them.
//
// At up to 262,144 entities everything lies in L2 and a call is bound by the latency of
// its chain, so the entities are binned by a counting sort - rank by atomic, one scan of
// the cells, scatter - instead of radix passes over 4,096-key tiles (25 blocks at
// 100,000 entities, 17 us a pass), cells lie row by row so that a box is one run per
// row, and the four kernels start under their predecessors' tails.  100,003 entities,
// 2 m, 16 ids: 97 -> 23 us a call (one memset for counts and cursor; with two, 28).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include <cuda_runtime.h>

#include "msim_chain.cuh"
#include "msim_internal.h"
#include "msim_kernels.cuh"

namespace msim {
namespace {

// Capacity: MSIM_NOALLOC_MAX_ENTITIES entities, up to 512 x 512 cells.
constexpr uint32_t kMaxN = MSIM_NOALLOC_MAX_ENTITIES;
constexpr uint32_t kMaxSide = 512;
constexpr uint32_t kMaxCells = kMaxSide * kMaxSide;
constexpr uint32_t kScanCells = 1024;  // cells of one scan block: whole rows (the row pitch is a power of two)
// word offsets inside the scratch array
constexpr size_t kOffCursor = 0;                       // of the scan blocks; zeroed with the counts that follow
constexpr size_t kOffCount = kOffCursor + 64;          // entities per cell
constexpr size_t kOffStart = kOffCount + kMaxCells;
constexpr size_t kOffRank = kOffStart + kMaxCells;     // of each entity inside its cell
constexpr size_t kOffId = kOffRank + kMaxN;            // in cell order
constexpr size_t kOffPos = kOffId + kMaxN;
constexpr size_t kScratchWords = kOffPos + 2ull * kMaxN;  // ~6 MB

static __device__ __align__(256) uint32_t g_noalloc_scratch[kScratchWords];

struct CellGrid {
    float inv_cell, radius, d2_limit;
    uint32_t nx, ny, pitch;  // cell (x, y) is y * pitch + x
};

__device__ __forceinline__ uint32_t cell_of(const CellGrid& g, float2 p) {
    return tile_coord(p.y, g.inv_cell, g.ny) * g.pitch + tile_coord(p.x, g.inv_cell, g.nx);
}

__global__ __launch_bounds__(256) void k_noalloc_rank(const float2* __restrict__ pos, uint32_t n, CellGrid g,
                                                      uint32_t* count, uint32_t* __restrict__ rank,
                                                      uint32_t* status) {
    chain_enter();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i == 0 && status) *status = 0u;  // nothing below waits or can leave its range
    if (i < n) rank[i] = atomicAdd(&count[cell_of(g, pos[i])], 1u);
}

// Starts of kScanCells cells; the blocks take their places from a cursor in any order
// (a box's run never leaves a block's cells).
__global__ __launch_bounds__(256) void k_noalloc_scan(const uint32_t* __restrict__ count, uint32_t cells,
                                                      uint32_t* __restrict__ start, uint32_t* cursor) {
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_base;
    chain_enter();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t c = blockIdx.x * kScanCells + tid * 4u;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c < cells) v = *reinterpret_cast<const uint4*>(count + c);  // the table ends on whole quads
    const uint32_t sum = v.x + v.y + v.z + v.w;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8u; w++) {
        before += w < warp ? s_warp[w] : 0u;
        all += s_warp[w];
    }
    if (tid == 0) s_base = atomicAdd(cursor, all);
    __syncthreads();
    if (c >= cells) return;
    uint4 o;
    o.x = s_base + before + incl - sum;
    o.y = o.x + v.x;
    o.z = o.y + v.y;
    o.w = o.z + v.z;
    *reinterpret_cast<uint4*>(start + c) = o;
}

__global__ __launch_bounds__(256) void k_noalloc_scatter(const float2* __restrict__ pos, uint32_t n, CellGrid g,
                                                         const uint32_t* __restrict__ start,
                                                         const uint32_t* __restrict__ rank,
                                                         float2* __restrict__ cell_pos, uint32_t* __restrict__ cell_id) {
    chain_enter();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    const float2 p = pos[i];
    const uint32_t q = start[cell_of(g, p)] + rank[i];
    if (q >= n) return;  // only if the caller rewrites pos meanwhile; never write out of range
    cell_pos[q] = p;
    cell_id[q] = i;
}

// A thread's list of ids in shared memory, a column of words.
struct Column {
    uint32_t* at0;
    __device__ __forceinline__ uint32_t& operator[](uint32_t k) const { return at0[k * kQueryThreads]; }
};
// id goes down from place k of a heap (largest first) of n ids.
__device__ __forceinline__ void sift_down(Column c, uint32_t k, uint32_t n, uint32_t id) {
    for (;;) {
        uint32_t child = 2u * k + 1u;
        if (child >= n) break;
        uint32_t x = c[child];
        if (child + 1u < n) {
            const uint32_t y = c[child + 1u];
            if (y > x) {
                x = y;
                child++;
            }
        }
        if (x <= id) break;
        c[k] = x;
        k = child;
    }
    c[k] = id;
}
// The warp puts the m ids of a column in ascending order; m up to 32 K.
template <uint32_t K>
__device__ __forceinline__ void order_column(Column c, uint32_t m, uint32_t lane) {
    uint32_t x[K], rank[K];
#pragma unroll
    for (uint32_t k = 0; k < K; k++) {
        x[k] = lane + 32u * k < m ? c[lane + 32u * k] : MSIM_NO_NEIGHBOUR;
        rank[k] = 0u;
    }
    for (uint32_t j = 0; j < m; j++) {
        const uint32_t y = c[j];
#pragma unroll
        for (uint32_t k = 0; k < K; k++) rank[k] += y < x[k] ? 1u : 0u;
    }
    __syncwarp();  // every id is read
#pragma unroll
    for (uint32_t k = 0; k < K; k++)
        if (lane + 32u * k < m) c[rank[k]] = x[k];
}

// The query, one thread per entity in cell order: per row of its box one run of positions,
// four loads in flight.  With lists the positions are tested 32 at a time into a mask and
// the hits taken afterwards, two ids in flight, so that the lanes of a warp take theirs
// together: the entries of a cell come in no order of ids, and one insertion at a time held
// up the other lanes (100,003 entities about spots, 42 neighbours, 16 ids 361 -> 193 us).  The
// thread's list lies in shared memory, ascending up to kAscending ids; longer lists go on in
// no order (insertion into 200 ids moved 100 for each), become a heap once they are full, and
// are put in order by the warp in the end (262,144 about spots, 200 ids 2.5 -> 1.2 ms).
// Registers for 12 and 6 blocks per SM: at 16 the compiler spills (262,144 spread, 4 ids 25.3
// us for 23.7), and with many ids the shared memory allows no more.
// The lists are written by the whole warp (see k_export_nbr), 16 bytes a lane with QUADS
// (cap a multiple of 4 and idx_out on a 16-byte boundary).
constexpr uint32_t kAscending = 32;
enum Lists : int { kCounts, kShort, kLong };  // cap 0, up to kAscending, above
template <Lists LISTS, bool QUADS>
__global__ __launch_bounds__(kQueryThreads, LISTS == kLong ? 6 : 12) void k_noalloc_query(const uint32_t* __restrict__ cell_id,
                                                                 const float2* __restrict__ cell_pos,
                                                                 const uint32_t* __restrict__ start,
                                                                 const uint32_t* __restrict__ cell_count, CellGrid g,
                                                                 uint32_t n, uint32_t cap,
                                                                 uint32_t* __restrict__ count_out,
                                                                 uint32_t* __restrict__ idx_out) {
    constexpr uint32_t FULL = 0xffffffffu;
    extern __shared__ uint32_t s_list[];
    chain_enter();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t p = blockIdx.x * kQueryThreads + tid;
    const Column list{s_list + tid};
    uint32_t count = 0, id = 0xffffffffu;
    uint32_t m = 0, last = MSIM_NO_NEIGHBOUR;  // ids held; the largest of a full list
    if (p < n) {
        id = cell_id[p];
        const float2 me = cell_pos[p];
        // margin for the rounding of me -/+ reach at this position's magnitude
        const float mag = fmaxf(fabsf(me.x), fabsf(me.y));
        const float reach =
            __fadd_rn(__fmul_rn(g.radius, 1.00000095367431640625f), __fmul_rn(mag, 1.9073486328125e-6f));
        const uint32_t x0 = tile_coord(__fsub_rn(me.x, reach), g.inv_cell, g.nx);
        const uint32_t x1 = tile_coord(__fadd_rn(me.x, reach), g.inv_cell, g.nx);
        const uint32_t y0 = tile_coord(__fsub_rn(me.y, reach), g.inv_cell, g.ny);
        const uint32_t y1 = tile_coord(__fadd_rn(me.y, reach), g.inv_cell, g.ny);
        for (uint32_t y = y0; y <= y1; y++) {
            const uint32_t c0 = y * g.pitch + x0, c1 = y * g.pitch + x1;
            const uint32_t from = start[c0], to = min(start[c1] + cell_count[c1], n);
            if constexpr (LISTS == kCounts) {
                for (uint32_t q0 = from; q0 < to; q0 += 4u) {
                    float2 o[4];
#pragma unroll
                    for (uint32_t u = 0; u < 4u; u++) o[u] = cell_pos[min(q0 + u, to - 1u)];
#pragma unroll
                    for (uint32_t u = 0; u < 4u; u++)
                        if (q0 + u < to && q0 + u != p && in_range_fast(o[u], me, g.radius, g.d2_limit)) count++;
                }
            } else {
                for (uint32_t q0 = from; q0 < to; q0 += 32u) {
                    uint32_t hits = 0u;
                    for (uint32_t k = 0; k < 32u && q0 + k < to; k += 4u) {
                        float2 o[4];
#pragma unroll
                        for (uint32_t u = 0; u < 4u; u++) o[u] = cell_pos[min(q0 + k + u, to - 1u)];
#pragma unroll
                        for (uint32_t u = 0; u < 4u; u++) {
                            const uint32_t q = q0 + k + u;
                            const bool hit = q < to && q != p && in_range_fast(o[u], me, g.radius, g.d2_limit);
                            hits |= hit ? 1u << (k + u) : 0u;
                        }
                    }
                    count += (uint32_t)__popc(hits);
                    while (hits) {
                        constexpr uint32_t kIds = 2;
                        uint32_t other[kIds];
#pragma unroll
                        for (uint32_t u = 0; u < kIds; u++) {
                            other[u] = hits ? cell_id[q0 + (uint32_t)__ffs(hits) - 1u] : MSIM_NO_NEIGHBOUR;
                            hits &= hits - 1u;
                        }
#pragma unroll
                        for (uint32_t u = 0; u < kIds; u++) {
                            if (other[u] >= last) continue;
                            if (LISTS == kLong && m == cap) {
                                sift_down(list, 0u, cap, other[u]);
                                last = list[0];
                                continue;
                            }
                            uint32_t j = m < cap ? m++ : cap - 1u;
                            if (LISTS == kShort || j < kAscending) {
                                while (j > 0) {
                                    const uint32_t prev = list[j - 1u];
                                    if (prev <= other[u]) break;
                                    list[j] = prev;
                                    j--;
                                }
                            }
                            list[j] = other[u];
                            if (m < cap) continue;
                            if (LISTS == kLong)
                                for (uint32_t k = cap / 2u; k-- > 0;) sift_down(list, k, cap, list[k]);
                            last = list[LISTS == kLong ? 0u : cap - 1u];
                        }
                    }
                }
            }
        }
        if (id < n) count_out[id] = count;
    }
    if (LISTS == kCounts) return;
    __syncwarp();
    const uint32_t kept = m;
    const uint32_t* const col = s_list + warp * 32u;
    if constexpr (LISTS == kLong) {
        for (uint32_t todo = __ballot_sync(FULL, m > kAscending); todo; todo &= todo - 1u) {
            const uint32_t e = (uint32_t)__ffs(todo) - 1u, held = __shfl_sync(FULL, m, e);
            const Column c{s_list + warp * 32u + e};
            if (held <= 64u) order_column<2>(c, held, lane);
            else order_column<kMaxCap / 32u>(c, held, lane);
        }
        __syncwarp();
    }
    if constexpr (QUADS) {
        const uint32_t quads = cap >> 2;
        for (uint32_t i = lane; i < quads * 32u; i += 32u) {
            const uint32_t e = i / quads, j = (i - e * quads) * 4u;
            const uint32_t eid = __shfl_sync(FULL, id, e), ek = __shfl_sync(FULL, kept, e);
            if (eid >= n) continue;
            uint4 v;
            v.x = j < ek ? col[j * kQueryThreads + e] : MSIM_NO_NEIGHBOUR;
            v.y = j + 1u < ek ? col[(j + 1u) * kQueryThreads + e] : MSIM_NO_NEIGHBOUR;
            v.z = j + 2u < ek ? col[(j + 2u) * kQueryThreads + e] : MSIM_NO_NEIGHBOUR;
            v.w = j + 3u < ek ? col[(j + 3u) * kQueryThreads + e] : MSIM_NO_NEIGHBOUR;
            *reinterpret_cast<uint4*>(idx_out + (size_t)eid * cap + j) = v;
        }
    } else {
        for (uint32_t e = 0; e < 32u; e++) {
            const uint32_t eid = __shfl_sync(FULL, id, e), ek = __shfl_sync(FULL, kept, e);
            if (eid >= n) continue;  // uniform
            for (uint32_t j = lane; j < cap; j += 32u)
                idx_out[(size_t)eid * cap + j] = j < ek ? col[j * kQueryThreads + e] : MSIM_NO_NEIGHBOUR;
        }
    }
}

using Query = void (*)(const uint32_t*, const float2*, const uint32_t*, const uint32_t*, CellGrid, uint32_t, uint32_t,
                       uint32_t*, uint32_t*);
const Query kQueries[3][2] = {{k_noalloc_query<kCounts, false>, k_noalloc_query<kCounts, false>},
                              {k_noalloc_query<kShort, false>, k_noalloc_query<kShort, true>},
                              {k_noalloc_query<kLong, false>, k_noalloc_query<kLong, true>}};

// Per-device set-up: the scratch array's device address (the host-side symbol is
// only a stand-in, never a usable device pointer) and the query's shared-memory limit.
// Both end with the device's CUDA context, so another one sets them up again.
struct DeviceSlot {
    unsigned long long context = 0;  // the CUDA context it was set up in (0: none)
    uint32_t* scratch = nullptr;
};
constexpr int kCarveout = 45;  // percent of the largest; 60 and 75: 2 to 5 % slower at 262,144
std::mutex g_setup_mutex;
DeviceSlot g_slots[64];

int setup_device(int dev, DeviceSlot** out) {
    if (dev < 0 || dev >= 64) return fail(MSIM_ERR_INVALID, "device ordinal out of range for the no-allocation path");
    std::lock_guard<std::mutex> lk(g_setup_mutex);
    DeviceSlot& slot = g_slots[dev];
    unsigned long long context = 0;
    if (!cuda_context_id(&context) && (cudaSetDevice(dev) != cudaSuccess || !cuda_context_id(&context)))
        return fail(MSIM_ERR_CUDA, "no CUDA context for the no-allocation query");
    if (slot.context != context) {
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess || !ptr)
            return fail(MSIM_ERR_CUDA, std::string("cudaGetSymbolAddress(no-allocation scratch) failed: ") +
                                           cudaGetErrorString(e));
        for (const Query q : {kQueries[kLong][0], kQueries[kLong][1]})
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(q, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kMaxCap * kQueryThreads * sizeof(uint32_t)));
        if (e != cudaSuccess)
            return fail(MSIM_ERR_CUDA, std::string("cudaFuncSetAttribute failed: ") + cudaGetErrorString(e));
        // The kernels that start under their predecessors' tails find the shared memory of an
        // SM as those left it.  A small query's blocks were put on the few SMs whose shared
        // memory had already been set for them (20,000 entities in one cell, 157 blocks, 4 ids:
        // 11.6 ms for 3.4), so the chain asks for one setting; with longer lists it is the
        // memory itself that spreads the blocks.
        for (const void* k : {(const void*)k_noalloc_rank, (const void*)k_noalloc_scan, (const void*)k_noalloc_scatter,
                              (const void*)kQueries[kShort][0], (const void*)kQueries[kShort][1]})
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveout);
        if (e != cudaSuccess)
            return fail(MSIM_ERR_CUDA, std::string("cudaFuncSetAttribute failed: ") + cudaGetErrorString(e));
        slot.scratch = static_cast<uint32_t*>(ptr);
        slot.context = context;
    }
    *out = &slot;
    return MSIM_OK;
}

}  // namespace
}  // namespace msim

using namespace msim;

extern "C" int msim_query_neighbours_noalloc(const float* d_pos, uint32_t n, float world_w, float world_h,
                                             float radius, uint32_t cap, uint32_t* d_count, uint32_t* d_idx,
                                             uint32_t* d_status, void* stream) {
    if (n > kMaxN)
        return fail(MSIM_ERR_INVALID, "n = " + std::to_string(n) + " exceeds the no-allocation limit of " +
                                          std::to_string(kMaxN) + " entities");
    if (cap > kMaxCap) return fail(MSIM_ERR_INVALID, "cap must be <= " + std::to_string(kMaxCap));
    if (!std::isfinite(radius) || radius < 0.f) return fail(MSIM_ERR_INVALID, "radius must be finite and >= 0");
    if (!(world_w > 0.f) || !(world_h > 0.f) || !std::isfinite(world_w) || !std::isfinite(world_h))
        return fail(MSIM_ERR_INVALID, "world_w and world_h must be positive and finite");
    if (n && (!d_pos || !d_count || (cap && !d_idx)))
        return fail(MSIM_ERR_INVALID, "d_pos, d_count (and d_idx when cap > 0) are required");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(MSIM_ERR_CUDA, std::string("cudaGetDevice failed: ") + cudaGetErrorString(e));
    DeviceSlot* slot = nullptr;
    int rc = setup_device(dev, &slot);
    if (rc != MSIM_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint32_t* w = slot->scratch;
    if (n == 0) {
        if (d_status && cudaMemsetAsync(d_status, 0, sizeof(uint32_t), s) != cudaSuccess)
            return fail(MSIM_ERR_CUDA, "cudaMemsetAsync failed");
        return MSIM_OK;
    }

    // cells no smaller than the radius (a box spans at most three), about two per entity,
    // at most 512 a side
    const double largest = std::max((double)world_w, (double)world_h);
    double cell = std::max((double)radius * (1.0 + 0x1p-20),
                           std::sqrt((double)world_w * (double)world_h / (2.0 * (double)n)));
    cell = std::max(std::max(cell, largest / (double)kMaxSide * (1.0 + 1e-6)), 1e-3);
    CellGrid g{};
    g.nx = (uint32_t)std::min<double>(std::max(1.0, std::ceil((double)world_w / cell)), kMaxSide);
    g.ny = (uint32_t)std::min<double>(std::max(1.0, std::ceil((double)world_h / cell)), kMaxSide);
    g.pitch = 4;
    while (g.pitch < g.nx) g.pitch *= 2;
    g.inv_cell = (float)(1.0 / cell);
    g.radius = radius;
    g.d2_limit = sqrt_limit(radius);
    const uint32_t cells = g.pitch * g.ny;
    const float2* pos = reinterpret_cast<const float2*>(d_pos);
    float2* cell_pos = reinterpret_cast<float2*>(w + kOffPos);
    uint32_t *count = w + kOffCount, *cursor = w + kOffCursor;
    const unsigned blocks = (n + 255u) / 256u;
    const bool quads = (cap & 3u) == 0u && (reinterpret_cast<uintptr_t>(d_idx) & 15u) == 0u;

    bool ok = cudaMemsetAsync(cursor, 0, sizeof(uint32_t) * (kOffCount - kOffCursor + cells), s) == cudaSuccess;
    ok = ok && launch_chained(k_noalloc_rank, blocks, 256, s, pos, n, g, count, w + kOffRank, d_status) == cudaSuccess;
    ok = ok && launch_chained(k_noalloc_scan, (cells + kScanCells - 1u) / kScanCells, 256, s, count, cells,
                              w + kOffStart, cursor) == cudaSuccess;
    ok = ok && launch_chained(k_noalloc_scatter, blocks, 256, s, pos, n, g, w + kOffStart, w + kOffRank, cell_pos,
                              w + kOffId) == cudaSuccess;
    ok = ok && launch_chained_shared(kQueries[cap == 0 ? kCounts : cap <= kAscending ? kShort : kLong][quads],
                              (n + kQueryThreads - 1) / kQueryThreads, kQueryThreads,
                              (size_t)cap * kQueryThreads * sizeof(uint32_t), s, w + kOffId, cell_pos, w + kOffStart,
                              count, g, n, cap, d_count, d_idx) == cudaSuccess;
    if (!ok) return fail(MSIM_ERR_CUDA, std::string("no-allocation neighbour query: ") + cudaGetErrorString(cudaGetLastError()));
    return MSIM_OK;
}
