// Index update by counting (included by msim_kernels.cu inside its namespace).
//
// After the first neighbour tick the index is built by a counting sort: the move step
// takes a rank for every entity from its key's counter (k_step), a chained scan turns the
// counters into the key-start table (k_mark) and every entity goes to its key's start
// plus its rank (k_place).  Three kernels and no dependence on the previous order, where
// splitting that order, sorting its changed entries in three radix passes, merging and
// filling the table took seven (with the move step 117 -> 50 us at 1 M entities, 531 ->
// 388 at 16 M).  k_mark moves 12 bytes per key, k_place 36 per entity.  The order of equal keys follows the atomics; nothing
// observable depends on it (neighbour sets are sets, lists are sorted by id).

constexpr uint32_t kScanThreads = 256;
constexpr uint32_t kScanRows = 4;                                // 16-byte loads per thread
constexpr uint32_t kScanTile = kScanThreads * kScanRows * 4u;    // 4096 keys per block

// kstart[k] = entities with keys below k, for k <= num_keys; the counters are left zero
// for the next update.  Tiles are taken in ticket order and look back 32 predecessors per
// round of loads; a tile's sum is published before its own offsets are computed.
__global__ __launch_bounds__(kScanThreads) void k_mark(uint32_t* __restrict__ key_count, uint32_t num_keys, uint32_t n,
                                                      uint32_t* __restrict__ kstart, uint32_t* lookback,
                                                      uint32_t* ticket, uint32_t num_tiles, uint32_t* err,
                                                      uint32_t spin_limit) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr uint32_t NW = kScanThreads / 32;
    __shared__ uint32_t s_sum[kScanRows * NW];  // per (row, warp), then their exclusive scan
    __shared__ uint32_t s_tile, s_before;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    chain_enter();
    if (index_failed(err)) return;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= num_tiles) return;  // only when the ticket did not start at zero; uniform per block
    const uint32_t base = tile * kScanTile;
    uint4 v[kScanRows];
    uint32_t incl[kScanRows];
#pragma unroll
    for (uint32_t r = 0; r < kScanRows; r++) {
        const uint32_t k = base + r * kScanThreads * 4u + tid * 4u;
        v[r] = make_uint4(0u, 0u, 0u, 0u);
        if (k < num_keys) v[r] = *reinterpret_cast<const uint4*>(key_count + k);  // a multiple of four keys
    }
#pragma unroll
    for (uint32_t r = 0; r < kScanRows; r++) {
        incl[r] = v[r].x + v[r].y + v[r].z + v[r].w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl[r], o);
            if (lane >= (uint32_t)o) incl[r] += y;
        }
        if (lane == 31) s_sum[r * NW + warp] = incl[r];
    }
    __syncthreads();
    if (warp == 0) {
        static_assert(kScanRows * NW == 32, "one sum per lane");
        const uint32_t sum = s_sum[lane];
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        s_sum[lane] = x - sum;
        const uint32_t all = __shfl_sync(FULL, x, 31);
        if (lane == 0) st_relaxed(lookback + tile, (tile == 0 ? kFlagPrefix : kFlagAgg) | all);
        uint32_t before = 0u;
        if (tile > 0) {
            int32_t j = (int32_t)tile - 1;
            uint32_t spins = 0u;
            for (;;) {
                const int32_t idx = j - (int32_t)lane;
                const uint32_t w = idx >= 0 ? ld_relaxed(lookback + idx) : kFlagPrefix;
                const unsigned prefix = __ballot_sync(FULL, (w & kFlagPrefix) != 0u);
                const unsigned not_ready = __ballot_sync(FULL, (w & kFlagMask) == 0u);
                const uint32_t first = prefix ? (uint32_t)(__ffs(prefix) - 1) : 32u;
                const unsigned needed = first == 32u ? FULL : (0xffffffffu >> (31u - first));
                if (not_ready & needed) {  // a predecessor has not published: poll again
                    if (++spins > spin_limit) {
                        if (lane == 0) atomicOr(err, kErrTimeout);
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                before += __reduce_add_sync(FULL, lane <= first ? w & kValueMask : 0u);
                if (first < 32u) break;
                j -= 32;
            }
            if (lane == 0) st_relaxed(lookback + tile, kFlagPrefix | ((before + all) & kValueMask));
        }
        if (lane == 0) s_before = before;
    }
    __syncthreads();
    const uint32_t before = s_before;
#pragma unroll
    for (uint32_t r = 0; r < kScanRows; r++) {
        const uint32_t k = base + r * kScanThreads * 4u + tid * 4u;
        if (k >= num_keys) continue;
        uint4 o;
        o.x = before + s_sum[r * NW + warp] + incl[r] - (v[r].x + v[r].y + v[r].z + v[r].w);
        o.y = o.x + v[r].x;
        o.z = o.y + v[r].y;
        o.w = o.z + v[r].z;
        *reinterpret_cast<uint4*>(kstart + k) = o;
        *reinterpret_cast<uint4*>(key_count + k) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (tile == num_tiles - 1u && tid == 0) kstart[num_keys] = n;
}

// Every slot to its place in the sorted order: sorted_slot, and where wanted its position
// and the slot's own place (rank).
__global__ __launch_bounds__(256) void k_place(const uint32_t* __restrict__ key, const uint32_t* __restrict__ key_rank,
                                               const uint32_t* __restrict__ kstart, uint32_t num_keys, uint32_t n,
                                               const float2* __restrict__ pos, uint32_t* __restrict__ sorted_slot,
                                               float2* __restrict__ sorted_pos, uint32_t* __restrict__ rank,
                                               uint32_t* err) {
    chain_enter();
    if (index_failed(err)) return;
    const uint32_t s = blockIdx.x * 256u + threadIdx.x;
    if (s >= n) return;
    const uint32_t k = key[s], r = key_rank[s];
    float2 p = make_float2(0.f, 0.f);
    if (sorted_pos) p = pos[s];
    const uint32_t q = k < num_keys ? kstart[k] + r : n;
    if (q >= n) {  // unreachable: keys, counters and ranks come from the same step
        atomicOr(err, kErrOob);
        return;
    }
    sorted_slot[q] = s;
    if (sorted_pos) sorted_pos[q] = p;
    if (rank) rank[s] = q;
}
