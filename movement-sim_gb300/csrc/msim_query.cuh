// Key-start table and radius neighbour query (included by msim_kernels.cu inside
// its namespace).

// ---- key-start table ------------------------------------------------------------
// kstart[k] = first sorted position whose key is >= k, for every k in
// [0, num_keys]; kstart[num_keys] = n.  Keys >= num_keys (never produced by valid
// inputs) count as num_keys - 1.  A tile's run is [kstart[t << ybits],
// kstart[(t + 1) << ybits]); a band run inside it is two independent loads.

__device__ __forceinline__ uint32_t clamped_key(const uint32_t* __restrict__ sk, uint32_t q, uint32_t num_keys) {
    const uint32_t k = sk[q];
    return k < num_keys ? k : num_keys - 1u;
}

// One thread per position q in [0, n]: q owns the entries (key[q-1], key[q]] (q = n:
// up to num_keys).  Gaps of at most kGapDirect entries (almost all of them) are
// written by the thread itself; gaps up to kGapWarp entries by the whole warp (the
// lanes' gaps laid end to end, 32 coalesced entries per store); longer ones are cut
// into chunks of kGapChunk entries, appended to a list with one atomic per warp
// (disjoint entries, so the append order does not matter) and filled by
// k_kstart_fill.
constexpr uint32_t kGapDirect = 8;
constexpr uint32_t kGapWarp = 256;
constexpr uint32_t kGapChunk = 4096;

// Writes kstart[from + r] = value for r < len, for every lane of the warp (all lanes
// call it; a lane with nothing to write passes len = 0).
__device__ __forceinline__ void fill_key_gaps(uint32_t from, uint32_t len, uint32_t value, uint32_t lane,
                                              uint32_t* __restrict__ kstart, uint4* __restrict__ chunks,
                                              uint32_t* chunk_count, uint32_t chunk_cap) {
    constexpr uint32_t FULL = 0xffffffffu;
    if (len <= kGapDirect) {
        for (uint32_t r = 0; r < len; r++) kstart[from + r] = value;
    }
    // medium gaps: the warp writes them together
    const uint32_t wlen = len > kGapDirect && len <= kGapWarp ? len : 0u;
    if (__any_sync(FULL, wlen != 0u)) {
        uint32_t incl = wlen;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t excl = incl - wlen;
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        for (uint32_t base = 0; base < total; base += 32u) {
            const uint32_t i = base + lane;
            uint32_t owner = 0;
#pragma unroll
            for (uint32_t st = 16; st > 0; st >>= 1) {
                const uint32_t v = __shfl_sync(FULL, incl, owner + st - 1u);
                if (v <= i) owner += st;
            }
            const uint32_t o_excl = __shfl_sync(FULL, excl, owner);
            const uint32_t o_from = __shfl_sync(FULL, from, owner);
            const uint32_t o_val = __shfl_sync(FULL, value, owner);
            if (i < total) kstart[o_from + (i - o_excl)] = o_val;
        }
    }
    // long gaps: chunks, one list append per warp
    const uint32_t m = len > kGapWarp ? (len + kGapChunk - 1u) / kGapChunk : 0u;
    if (__any_sync(FULL, m != 0u)) {
        uint32_t incl = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        uint32_t base = 0;
        if (lane == 31) base = atomicAdd(chunk_count, total);
        base = __shfl_sync(FULL, base, 31) + (incl - m);
        if (m) {
            if (base + m > chunk_cap) {  // unreachable: chunk_cap bounds every key space; stay correct anyway
                for (uint32_t r = 0; r < len; r++) kstart[from + r] = value;
            } else {
                for (uint32_t c = 0; c < m; c++) {
                    const uint32_t off = c * kGapChunk;
                    chunks[base + c] =
                        make_uint4(from + off, len - off < kGapChunk ? len - off : kGapChunk, value, 0u);
                }
            }
        }
    }
}

__global__ __launch_bounds__(256) void k_kstart_pos(const uint32_t* __restrict__ sk, uint32_t n,
                                                    uint32_t* __restrict__ kstart, uint32_t num_keys,
                                                    uint4* __restrict__ chunks, uint32_t* chunk_count,
                                                    uint32_t chunk_cap, const uint32_t* __restrict__ sv,
                                                    const float2* __restrict__ pos, float2* __restrict__ sorted_pos,
                                                    const uint32_t* err) {
    chain_enter();
    if (index_failed(err)) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (sorted_pos && q < n) {  // positions in sorted order, for the query's candidate reads
        const uint32_t slot = sv[q];
        sorted_pos[q] = slot < n ? pos[slot] : make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
    }
    uint32_t from = 0, len = 0;
    if (q <= n) {
        from = q ? clamped_key(sk, q - 1u, num_keys) + 1u : 0u;
        const uint32_t to = q < n ? clamped_key(sk, q, num_keys) : num_keys;  // inclusive
        len = to >= from ? to - from + 1u : 0u;
    }
    fill_key_gaps(from, len, q, lane, kstart, chunks, chunk_count, chunk_cap);
}

__global__ __launch_bounds__(256) void k_kstart_fill(const uint4* __restrict__ chunks,
                                                     const uint32_t* __restrict__ chunk_count, uint32_t chunk_cap,
                                                     uint32_t* __restrict__ kstart, const uint32_t* err) {
    chain_enter();
    if (index_failed(err)) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t count = min(*chunk_count, chunk_cap);
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < count; c += warps) {
        const uint4 ch = chunks[c];
        for (uint32_t r = lane; r < ch.y; r += 32u) kstart[ch.x + r] = ch.z;
    }
}

// Chunk-list capacity that no key space can exceed: every chunked gap has more than
// kGapWarp entries, and adds at most one partial chunk.
inline uint32_t kstart_chunk_cap(uint64_t num_keys) {
    return (uint32_t)((num_keys + 1u) / (kGapWarp + 1u) + (num_keys + 1u) / kGapChunk + 2u);
}

// Positions in sorted order (NaN for a slot out of range), for the key-start paths
// that do not gather them on the way.
__global__ __launch_bounds__(256) void k_gather_pos(const uint32_t* __restrict__ sv, const float2* __restrict__ pos,
                                                    uint32_t n, float2* __restrict__ sorted_pos,
                                                    const uint32_t* err) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n || index_failed(err)) return;
    const uint32_t slot = sv[q];
    sorted_pos[q] = slot < n ? pos[slot] : make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
}

// One thread per table entry, binary search over the sorted keys: for key spaces
// much smaller than the number of positions (many positions per key).
__global__ __launch_bounds__(256) void k_kstart_search(const uint32_t* __restrict__ sk, uint32_t n,
                                                       uint32_t* __restrict__ kstart, uint32_t num_keys,
                                                       const uint32_t* err) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > num_keys || index_failed(err)) return;
    uint32_t lo = 0, hi = n;  // first position with clamped key >= k
    if (k == num_keys) {
        lo = n;
    } else {
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (clamped_key(sk, mid, num_keys) < k) lo = mid + 1u;
            else hi = mid;
        }
    }
    kstart[k] = lo;
}

// ---- radius neighbour query ------------------------------------------------------
// A warp queries 32 consecutive sorted positions (mostly one or two tiles).  Each
// lane's box [pos - reach, pos + reach] covers one to four tiles (more only when the
// tile side is below 2 x reach); for every tile the lane reads the run of the y bands
// its box overlaps from the key-start table.  The warp lays all non-empty runs of its
// lanes end to end in a shared run list (flat start, start position, owner lane) and
// tests 32 (owner, candidate) pairs per iteration, so every lane is busy whatever the
// run lengths; the run of each pair comes from a bit mask of the runs that start in
// the current window of 32 pairs.  Every candidate is tested with the predicate of
// random_move.comp:551-562; candidate positions come from the sorted copy, read in
// runs.  A hit counts for the owner and, for the first KEEP hits, keeps the
// candidate's sorted position; ids are looked up only for those.  The lists of entities
// with more than KEEP neighbours are made afterwards (lists_from_pairs, longer_lists).  The
// predicate is symmetric (fl(a - b) = -fl(b - a)), so the pair count is half the sum of the counts,
// and a pair of entities of the same warp (most pairs: consecutive sorted entities
// share their band runs) is tested once, by the lower lane, which credits both.  Each
// warp writes its lists contiguously at warp * 32 * cap and adds its count sum to one
// of kPairBins counters; the kernel has no block-wide barrier.
//
// KEEP (chosen by kDenseNeighbours and kCrowdNeighbours): sparse populations keep 8 and
// count every hit with a shared atomic; dense ones keep 32, crowds 48, and a looked-up
// window counts an owner's hits by ballot - its pairs lie side by side, where up to 32
// atomics on its counter took turns - with atomics only for the credited lanes.  (Read
// back from pair lists the hits thin out: one atomic per owner's run of pairs there was 15 %
// slower than one per hit; counts alone take an atomic per hit everywhere.)  Lists of more
// than eight are ranked in shared memory.  1 M entities with 4.5 neighbours 170 -> 83 us per
// tick, 200,000 with 14.6 261 -> 50.  A few warps with many lists beyond KEEP decide how
// long a crowd's query takes (a list looked up again cost about 4 us, and half the time half
// of the SMs stood idle), so those come from the kept pairs where there are any, and crowds
// keep more at fewer blocks resident.
constexpr uint32_t kRuns = 4;                  // runs per lane and round
constexpr uint32_t kWarpRuns = 32u * kRuns;    // run-list capacity of a warp

// Pair lists, for the ticks that reuse an index.  The index does not change between
// those ticks and entities move little, so a query can keep, per warp, the pairs it
// tested that lie within radius + 2 x (the displacement of the next few ticks): every pair
// in range in one of those ticks is among them, and their queries test the kept pairs
// alone - no tiles, bands or key starts per entity, no search for the run of a pair, and
// a quarter of the pairs.  One word per pair: owner lane | the candidate's sorted
// position (PairStore::places words per warp; kNoPairs: more than that, look them up); and
// the entity id of every sorted position, read beside the candidate's position so that
// a hit keeps the id itself.
// Bound by issue in sparse populations (79 % issue active at 4 M entities; 375 warp
// instructions a warp against 770), by the latency of its three dependent loads in small
// and in dense ones.  1 M entities at 2 m 30.6 us looked up, 19.3 from pairs, 38
// for the query that keeps them; the 16 M tick 532 -> 371 us, the 1 M tick 44.3 -> 34.6,
// reference mode at 1 M 122 -> 105.  Keeping runs instead of pairs gave 31.1 us at 1 M,
// ids beside the pairs 42 us for the keeping query.
constexpr uint32_t kPairOwnerShift = 27;
constexpr uint32_t kPairPosition = (1u << kPairOwnerShift) - 1u;
constexpr uint32_t kNoPairs = 0xffffffffu;
// looked up; looked up and kept; read back; looked up in boxes widened by *PairStore::disp
enum PairLists : int { kPairsFound, kPairsKept, kPairsUsed, kPairsWidened };

struct PairStore {
    uint32_t* pairs;
    uint32_t* sizes;
    uint32_t* ids;
    uint32_t places;  // per warp
    float near2;  // pairs up to this squared distance are kept
    const uint32_t* disp;  // kPairsWidened: the tick's largest displacement d (float bits)
    float widen_limit;     // and the d up to which the query runs
};

template <int KEEP, bool LIST>
struct QueryShared {
    float2 me[kQueryThreads];
    uint32_t cnt[kQueryThreads];
    uint32_t id[kQueryThreads];                // kept pairs: the entities' ids
    // A warp's words: rows of one word per lane for the sorted positions of the first hits
    // (DENSE: the owner's own from the front, those credited by lower lanes from the back),
    // then the run list.  Together they hold the warp's longer lists once the others are
    // written out.
    static constexpr uint32_t kKept = LIST ? KEEP : 0, kRows = kKept + 3u * kRuns;
    uint32_t words[kQueryThreads / 32][kRows * 32u];
    __device__ __forceinline__ uint32_t& place(uint32_t warp, uint32_t c, uint32_t lane) {
        return words[warp][c * 32u + lane];
    }
    // of run j: its start position minus its flat start, its flat start, its owner lane
    __device__ __forceinline__ uint32_t& rq(uint32_t warp, uint32_t j) { return words[warp][kKept * 32u + j]; }
    __device__ __forceinline__ uint32_t& rfs(uint32_t warp, uint32_t j) {
        return words[warp][kKept * 32u + kWarpRuns + j];
    }
    __device__ __forceinline__ uint32_t& rown(uint32_t warp, uint32_t j) {
        return words[warp][kKept * 32u + 2u * kWarpRuns + j];
    }
};

// Bits [from, to) of a word, both clamped to 0 .. 32.
__device__ __forceinline__ uint32_t bit_range(int from, int to) {
    from = max(from, 0);
    to = min(to, 32);
    return to > from ? (0xffffffffu >> (32 - (to - from))) << from : 0u;
}

// A hit of owner and candidate q by atomics on their counters; kept for the owner is
// `theirs`, for a credited lane `mine` (sorted positions or ids).
template <bool LIST, int KEEP>
__device__ __forceinline__ void count_hit(QueryShared<KEEP, LIST>& sh, uint32_t warp, uint32_t owner, uint32_t q,
                                          uint32_t pwarp, uint32_t theirs, uint32_t mine) {
    constexpr bool DENSE = LIST && KEEP != kQueryKeep;
    const uint32_t ot = warp * 32u + owner, other = q - pwarp;
    const uint32_t c = atomicAdd(&sh.cnt[ot], 1u);
    if (LIST && c < (uint32_t)KEEP) sh.place(warp, DENSE ? KEEP - 1 - c : c, owner) = theirs;
    if (other < 32u) {  // a higher lane of this warp: the pair counts for it too
        const uint32_t om = warp * 32u + other;
        const uint32_t c2 = atomicAdd(&sh.cnt[om], 1u);
        if (LIST && c2 < (uint32_t)KEEP) sh.place(warp, DENSE ? KEEP - 1 - c2 : c2, other) = mine;
    }
}

// own: DENSE: the lane's hits as owner so far.  KEPT: near pairs are appended to the
// warp's places (near_count so far).
template <bool LIST, int KEEP, bool KEPT>
__device__ __forceinline__ void query_runs(const uint32_t (&lo_in)[kRuns], const uint32_t (&len_in)[kRuns],
                                           uint32_t lane, uint32_t warp, uint32_t pwarp, QueryShared<KEEP, LIST>& sh,
                                           const float2* __restrict__ sorted_pos, const TileGrid& g, uint32_t& own,
                                           PairStore store, uint32_t& near_count) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr bool DENSE = LIST && KEEP != kQueryKeep;
    // A pair of entities of this warp is tested once, by the lower lane, which credits
    // both (the predicate is symmetric, and an in-range pair lies in both entities'
    // runs).  So a lane skips the warp's positions up to its own: a run that starts at
    // or after the warp's first position starts after the owner instead (a run that
    // starts before it is kept whole; the loop skips those positions).  At 16 M about
    // 4.7 of the 5.3 candidates of an entity lie in its own warp.
    uint32_t lo[kRuns], len[kRuns];
#pragma unroll
    for (uint32_t k = 0; k < kRuns; k++) {
        lo[k] = lo_in[k];
        len[k] = len_in[k];
        if (len[k] && lo[k] >= pwarp) {
            const uint32_t hi = lo[k] + len[k];
            const uint32_t from = lo[k] > pwarp + lane ? lo[k] : pwarp + lane + 1u;
            lo[k] = from;
            len[k] = hi > from ? hi - from : 0u;
        }
    }
    uint32_t flat = 0, nr = 0;
#pragma unroll
    for (uint32_t k = 0; k < kRuns; k++) {
        flat += len[k];
        nr += len[k] ? 1u : 0u;
    }
    uint32_t fi = flat, ri = nr;  // inclusive warp prefixes of candidates and runs
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t yf = __shfl_up_sync(FULL, fi, o);
        const uint32_t yr = __shfl_up_sync(FULL, ri, o);
        if (lane >= (uint32_t)o) {
            fi += yf;
            ri += yr;
        }
    }
    const uint32_t total = __shfl_sync(FULL, fi, 31);
    const uint32_t runs = __shfl_sync(FULL, ri, 31);
    uint32_t j = ri - nr, fs = fi - flat;
#pragma unroll
    for (uint32_t k = 0; k < kRuns; k++) {
        if (len[k]) {
            sh.rq(warp, j) = lo[k] - fs;
            sh.rfs(warp, j) = fs;
            sh.rown(warp, j) = lane;
            j++;
            fs += len[k];
        }
    }
    __syncwarp();  // the run list is visible to the whole warp
    uint32_t ra = 0;  // first run that starts at or after the current window
    for (uint32_t base = 0; base < total; base += 32u) {
        const uint32_t rr = ra + lane;
        const uint32_t off = (rr < runs ? sh.rfs(warp, rr) : 0xffffffffu) - base;
        const uint32_t marks = __reduce_or_sync(FULL, off < 32u ? (1u << off) : 0u);
        const uint32_t le = marks & (0xffffffffu >> (31u - lane));
        const uint32_t run = ra + (uint32_t)__popc(le) - 1u;  // le == 0: the run begun before the window
        ra += (uint32_t)__popc(marks);
        const uint32_t i = base + lane;
        if constexpr (!DENSE && !KEPT) {
            if (i >= total) continue;
            const uint32_t q = sh.rq(warp, run) + i;
            const uint32_t owner = sh.rown(warp, run);
            if (q - pwarp <= owner) continue;  // the owner itself or a lower lane: tested from there
            if (!in_range_fast(sorted_pos[q], sh.me[warp * 32u + owner], g.radius, g.d2_limit)) continue;
            count_hit<LIST, KEEP>(sh, warp, owner, q, pwarp, q, pwarp + owner);
        } else {
            uint32_t q = 0u, owner = lane, other = 0u;
            bool hit = false, near = false;
            if (i < total) {
                q = sh.rq(warp, run) + i;
                owner = sh.rown(warp, run);
                other = q - pwarp;
                if (other > owner) {
                    const float2 o = sorted_pos[q], me = sh.me[warp * 32u + owner];
                    hit = in_range_fast(o, me, g.radius, g.d2_limit);
                    if (KEPT) {
                        const float ex = __fsub_rn(o.x, me.x), ey = __fsub_rn(o.y, me.y);
                        near = __fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)) <= store.near2;
                    }
                }
            }
            if constexpr (KEPT) {
                const uint32_t m = __ballot_sync(FULL, near);
                const uint32_t at = near_count + (uint32_t)__popc(m & lanemask_lt());
                if (near && at < store.places)
                    store.pairs[(size_t)(pwarp >> 5) * store.places + at] = q | (owner << kPairOwnerShift);
                near_count += (uint32_t)__popc(m);
            }
            if constexpr (!DENSE) {
                if (hit) count_hit<LIST, KEEP>(sh, warp, owner, q, pwarp, q, pwarp + owner);
                continue;
            }
            const uint32_t hits = __ballot_sync(FULL, hit);
            const uint32_t mine = bit_range((int)(fi - flat - base), (int)(fi - base));  // this lane's pairs
            if (LIST) {
                const uint32_t before = __shfl_sync(FULL, own, owner), pairs = __shfl_sync(FULL, mine, owner);
                const uint32_t c = before + (uint32_t)__popc(hits & pairs & lanemask_lt());
                if (hit && c < (uint32_t)KEEP) sh.place(warp, c, owner) = q;
            }
            own += (uint32_t)__popc(hits & mine);
            if (hit && other < 32u) {
                const uint32_t om = warp * 32u + other;
                const uint32_t c2 = atomicAdd(&sh.cnt[om], 1u);
                if (LIST && c2 < (uint32_t)KEEP) sh.place(warp, KEEP - 1 - c2, other) = pwarp + owner;
            }
        }
    }
    __syncwarp();  // before the run list is rewritten
}

// Inclusive prefix sums over the warp, and the first lane whose sum exceeds i (31 when
// none does).
__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}
__device__ __forceinline__ uint32_t first_above(uint32_t ends, uint32_t i) {
    uint32_t o = 0;
#pragma unroll
    for (uint32_t st = 16; st > 0; st >>= 1)
        if (__shfl_sync(0xffffffffu, ends, o + st - 1u) <= i) o += st;
    return min(o, 31u);
}

// The ascending lists of the lanes with count > 0 (more than KEEP neighbours; 0 for the
// others, whose lists are written) of a warp whose pairs are kept, by this tick's query or
// an earlier one: those pairs again, every id into its entity's part of the keep words (the
// lists end to end, as many lanes at a time as fit), then each id to its rank among its
// list.  place: the lane's list in out.  False: a list alone is too long for the words.
template <int KEEP>
__device__ __noinline__ bool lists_from_pairs(const uint32_t* pairs, uint32_t size,
                                              const uint32_t* __restrict__ sorted_slot,
                                              const uint32_t* __restrict__ slot_id,
                                              const float2* __restrict__ sorted_pos, float radius, float d2_limit,
                                              uint32_t n, uint32_t pwarp, uint32_t count, uint32_t place,
                                              uint32_t cap, QueryShared<KEEP, true>& sh, uint32_t* out) {
    constexpr uint32_t FULL = 0xffffffffu, kWords = 32u * QueryShared<KEEP, true>::kRows;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (__any_sync(FULL, count > kWords)) return false;
    uint32_t* const words = &sh.place(warp, 0u, 0u);
    auto id_of = [&](uint32_t q) {
        const uint32_t s2 = sorted_slot[q];
        return s2 < n ? (slot_id ? slot_id[s2] : s2) : 0xffffffffu;
    };
    sh.id[warp * 32u + lane] = pwarp + lane < n ? id_of(pwarp + lane) : 0xffffffffu;
    const uint32_t ends = warp_inclusive(count, lane);
    for (uint32_t from = 0; from < 32u;) {  // lanes from .. to - 1
        const uint32_t before = __shfl_sync(FULL, ends - count, from);
        const uint32_t to = (uint32_t)__popc(__ballot_sync(FULL, lane < from || ends - before <= kWords));
        const uint32_t total = __shfl_sync(FULL, ends, to - 1u) - before;
        sh.cnt[warp * 32u + lane] = ends - count - before;  // next free word
        __syncwarp();
        const uint32_t wanted = __ballot_sync(FULL, count != 0u && lane - from < to - from);
        constexpr uint32_t kAtOnce = 4;  // per lane: each pair's loads wait for it
        for (uint32_t base = lane; base < size; base += 32u * kAtOnce) {
            uint32_t pair[kAtOnce], id[kAtOnce], who[kAtOnce];  // who: bit 0 the owner, bit 1 the other lane
            float2 pos[kAtOnce];
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; k++) pair[k] = base + 32u * k < size ? pairs[base + 32u * k] : kNoPairs;
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; k++) {
                const uint32_t q = pair[k] & kPairPosition, other = q - pwarp;
                who[k] = 0u;
                if (base + 32u * k < size)
                    who[k] = ((wanted >> (pair[k] >> kPairOwnerShift)) & 1u) |
                             (other < 32u ? ((wanted >> other) & 1u) << 1 : 0u);
                if (who[k]) {
                    id[k] = id_of(q);
                    pos[k] = sorted_pos[q];
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; k++) {
                const uint32_t owner = pair[k] >> kPairOwnerShift, other = (pair[k] & kPairPosition) - pwarp;
                if (!who[k] || !in_range_fast(pos[k], sh.me[warp * 32u + owner], radius, d2_limit)) continue;
                if (who[k] & 1u) words[atomicAdd(&sh.cnt[warp * 32u + owner], 1u)] = id[k];
                if (who[k] & 2u) words[atomicAdd(&sh.cnt[warp * 32u + other], 1u)] = sh.id[warp * 32u + owner];
            }
        }
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32u) {
            const uint32_t i = base + lane, o = first_above(ends, i + before);
            const uint32_t m = __shfl_sync(FULL, count, o), first = __shfl_sync(FULL, ends, o) - m - before;
            const uint32_t at = __shfl_sync(FULL, place, o);
            if (i >= total) continue;
            const uint32_t id = words[i];
            uint32_t rank = 0;
#pragma unroll 8
            for (uint32_t k = 0; k < m; k++) rank += words[first + k] < id ? 1u : 0u;
            if (rank < cap) out[at + rank] = id;
        }
        __syncwarp();  // before the words are used again
        from = to;
    }
    return true;
}

// The ascending list of lane o's entity (more than KEEP neighbours) by the whole warp: its
// runs again, 64 candidates at a time, every hit's id into the warp's words, then each id to
// its rank among them.  Ranks cost the square of the ids held (200,000 entities with 727
// neighbours, 64 ids: 17.8 ms with all of them, 6.5 so), so with `full` held the cap
// smallest stay and larger ids are skipped from then on: any number of neighbours fits.
template <uint32_t ROWS>
__device__ __noinline__ void list_by_warp(const uint32_t* __restrict__ sorted_slot,
                                          const float2* __restrict__ sorted_pos, const uint32_t* __restrict__ slot_id,
                                          const uint32_t* __restrict__ kstart, const TileGrid& g, float reach,
                                          uint32_t n, uint32_t p, float2 me, uint32_t cap, uint32_t* words, uint32_t* out) {
    constexpr uint32_t FULL = 0xffffffffu, kNone = 0xffffffffu;
    static_assert(2u * kMaxCap + 64u <= ROWS * 32u, "a full buffer and the hits of a round");
    const uint32_t lane = threadIdx.x & 31u;
    const float ylo = __fsub_rn(me.y, reach), yhi = __fadd_rn(me.y, reach);
    const uint32_t x0 = tile_coord(__fsub_rn(me.x, reach), g.inv_cell, g.tiles_x);
    const uint32_t x1 = tile_coord(__fadd_rn(me.x, reach), g.inv_cell, g.tiles_x);
    const uint32_t y0 = tile_coord(ylo, g.inv_cell, g.tiles_y), y1 = tile_coord(yhi, g.inv_cell, g.tiles_y);
    const uint32_t nx = x1 - x0 + 1u, slots = nx * (y1 - y0 + 1u);
    const uint32_t full = max(2u * cap, 384u);
    uint32_t m = 0, below = kNone;  // ids held; only smaller ones are still wanted
    auto rank_of = [&](uint32_t id) {
        uint32_t rank = 0;
        for (uint32_t j = 0; j < m; j++) rank += words[j] < id ? 1u : 0u;
        return rank;
    };
    for (uint32_t j0 = 0; j0 < slots; j0 += 32u) {  // a tile's run per lane
        const uint32_t j = j0 + lane;
        uint32_t lo = 0, len = 0;
        if (j < slots) {
            const uint32_t jy = j / nx, tx = x0 + (j - jy * nx), ty = y0 + jy;
            const uint32_t t = morton2(tx, ty) << g.ybits;
            lo = kstart[t | (g.ybits ? y_band(g, ylo, ty) : 0u)];
            const uint32_t hi = min(kstart[(t | (g.ybits ? y_band(g, yhi, ty) : 0u)) + 1u], n);
            len = hi > lo ? hi - lo : 0u;
        }
        const uint32_t ends = warp_inclusive(len, lane), total = __shfl_sync(FULL, ends, 31);
        for (uint32_t base = 0; base < total; base += 64u) {  // the runs end to end, two candidates per lane
            uint32_t q[2], id[2];
            bool hit[2];
#pragma unroll
            for (uint32_t k = 0; k < 2u; k++) {
                const uint32_t i = base + 32u * k + lane, o = first_above(ends, i);
                q[k] = __shfl_sync(FULL, lo, o) + (i - (__shfl_sync(FULL, ends, o) - __shfl_sync(FULL, len, o)));
                hit[k] = i < total && q[k] != p;
            }
#pragma unroll
            for (uint32_t k = 0; k < 2u; k++) {
                hit[k] = hit[k] && in_range_fast(sorted_pos[q[k]], me, g.radius, g.d2_limit);
                const uint32_t s2 = hit[k] ? sorted_slot[q[k]] : n;
                id[k] = s2 < n ? (slot_id ? slot_id[s2] : s2) : kNone;
            }
#pragma unroll
            for (uint32_t k = 0; k < 2u; k++) {
                const uint32_t hits = __ballot_sync(FULL, id[k] < below);
                if (id[k] < below) words[m + (uint32_t)__popc(hits & lanemask_lt())] = id[k];
                m += (uint32_t)__popc(hits);
            }
            if (m < full) continue;
            __syncwarp();
            uint32_t last = 0u;  // the cap-th smallest, of the lane that holds it
            for (uint32_t i = lane; i < m; i += 32u)
                if (rank_of(words[i]) == cap - 1u) last = words[i];
            below = __reduce_max_sync(FULL, last);
            uint32_t kept = 0;
            for (uint32_t i0 = 0; i0 < m; i0 += 32u) {  // towards the front, behind the reads
                const uint32_t x = i0 + lane < m ? words[i0 + lane] : kNone;
                const uint32_t stay = __ballot_sync(FULL, x <= below && x != kNone);
                if ((stay >> lane) & 1u) words[kept + (uint32_t)__popc(stay & lanemask_lt())] = x;
                kept += (uint32_t)__popc(stay);
                __syncwarp();
            }
            m = kept;
        }
    }
    __syncwarp();
    for (uint32_t i = lane; i < m; i += 32u) {
        const uint32_t rank = rank_of(words[i]);
        if (rank < cap) out[rank] = words[i];
    }
    __syncwarp();  // before the words are used again
}

// How a lane holds the smallest ids it has met: in a column of the warp's words in no order,
// the largest replaced and every id ranked in the end; in a column, ascending, by insertion;
// or by insertion in its place of the output.
enum HeldIds : int { kUnordered, kOrdered, kInPlace };

// The ascending lists of the lanes with count > 0 (more than KEEP neighbours), each by its
// own lane, `width` lanes at a time.  Candidates are tested 32 at a time into a mask and the
// hits taken afterwards, so that the lanes take theirs together.
template <HeldIds HELD>
__device__ __forceinline__ void lists_by_lane(const uint32_t* __restrict__ sorted_slot,
                                              const float2* __restrict__ sorted_pos,
                                              const uint32_t* __restrict__ slot_id,
                                              const uint32_t* __restrict__ kstart, const TileGrid& g, float reach,
                                              uint32_t n, uint32_t p, uint32_t count, uint32_t cap, uint32_t width,
                                              uint32_t* words, uint32_t* out) {
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t kept = min(count, cap), step = HELD == kInPlace ? 1u : width;
    uint32_t todo = __ballot_sync(FULL, count != 0u);
    while (todo) {
        const uint32_t column = (uint32_t)__popc(todo & lanemask_lt());
        const bool mine = ((todo >> (threadIdx.x & 31u)) & 1u) && column < width;
        todo &= ~__ballot_sync(FULL, mine);
        if (mine) {
            uint32_t* const list = HELD == kInPlace ? out : words + column;
            uint32_t m = 0, top = 0u, at = 0u;  // ids held; kUnordered: the largest and its place once all are
            const float2 me = sorted_pos[p];
            const float ylo = __fsub_rn(me.y, reach), yhi = __fadd_rn(me.y, reach);
            const uint32_t x0 = tile_coord(__fsub_rn(me.x, reach), g.inv_cell, g.tiles_x);
            const uint32_t x1 = tile_coord(__fadd_rn(me.x, reach), g.inv_cell, g.tiles_x);
            const uint32_t y0 = tile_coord(ylo, g.inv_cell, g.tiles_y), y1 = tile_coord(yhi, g.inv_cell, g.tiles_y);
            for (uint32_t ty = y0; ty <= y1; ty++) {
                for (uint32_t tx = x0; tx <= x1; tx++) {
                    const uint32_t t = morton2(tx, ty) << g.ybits;
                    const uint32_t q1 = min(kstart[(t | (g.ybits ? y_band(g, yhi, ty) : 0u)) + 1u], n);
                    for (uint32_t q0 = kstart[t | (g.ybits ? y_band(g, ylo, ty) : 0u)]; q0 < q1; q0 += 32u) {
                        uint32_t hits = 0u;
                        for (uint32_t k = 0; k < 32u && q0 + k < q1; k += 4u) {
#pragma unroll
                            for (uint32_t u = 0; u < 4u; u++) {
                                const uint32_t q = min(q0 + k + u, q1 - 1u);  // past the end: the last one's again
                                const bool hit = q != p && in_range_fast(sorted_pos[q], me, g.radius, g.d2_limit);
                                hits |= hit ? 1u << (q - q0) : 0u;
                            }
                        }
                        while (hits) {
                            const uint32_t s2 = sorted_slot[q0 + (uint32_t)__ffs(hits) - 1u];
                            hits &= hits - 1u;
                            if (s2 >= n) continue;
                            const uint32_t id = slot_id ? slot_id[s2] : s2;
                            if constexpr (HELD == kUnordered) {
                                if (m < kept) at = m++;
                                else if (id >= top) continue;
                                list[at * step] = id;
                                if (m < kept) continue;
                                top = 0u;
#pragma unroll 4
                                for (uint32_t j = 0; j < kept; j++) {
                                    const uint32_t x = list[j * step];
                                    if (x >= top) {
                                        top = x;
                                        at = j;
                                    }
                                }
                            } else {
                                uint32_t j = m;
                                if (m < kept) m++;
                                else if (id < list[(kept - 1u) * step]) j = kept - 1u;
                                else continue;
                                while (j > 0 && list[(j - 1u) * step] > id) {
                                    list[j * step] = list[(j - 1u) * step];
                                    j--;
                                }
                                list[j * step] = id;
                            }
                        }
                    }
                }
            }
            if constexpr (HELD == kOrdered) {
                for (uint32_t j = 0; j < m; j++) out[j] = list[j * step];
            } else if constexpr (HELD == kUnordered) {
                for (uint32_t i = 0; i < m; i += 2u) {
                    const uint32_t a = list[i * step], b = i + 1u < m ? list[(i + 1u) * step] : 0xffffffffu;
                    uint32_t ra = 0, rb = 0;
#pragma unroll 4
                    for (uint32_t j = 0; j < m; j++) {
                        const uint32_t x = list[j * step];
                        ra += x < a ? 1u : 0u;
                        rb += x < b ? 1u : 0u;
                    }
                    out[ra] = a;
                    if (i + 1u < m) out[rb] = b;
                }
            }
        }
        __syncwarp();  // before the next lanes use the words
    }
}

// The ascending lists of the lanes with count > KEEP (0 for the others, whose lists are
// written), looked up again.  The only call of the kernel's tail, so that nothing stays live
// across it.
// Sparse populations have such lists where entities stand at one point; their ids then come
// in a few ascending stretches, which suits insertion (1 M entities at the road starts, about
// 30 neighbours, us per tick, by insertion / ranked in the end: 16 ids 178 / 199, 64 ids 234 /
// 300).  In one turn of the warp's lanes, or two while the walk that is done twice is short;
// lists of up to 96 ids in the output, where a third turn cost more than the slower
// memory (3,000 entities on one spot, 64 ids: 2.2 ms, in four turns 4.7, list by list 3.7);
// longer ones list by list (the same with 256 ids 6.8 ms, in the output 12).
// In dense populations ids come in no order: ranked in the end 8 / 32 ids of 82 neighbours
// 216 / 296 us at 50,000, by insertion 229 / 407, list by list 418 / 416.  A list alone costs
// the warp what about 16 lanes' lists cost at once, more with longer lists, and two turns are
// slower than list by list (64 ids of 570 neighbours, 1 M: 27 / 22 ms).
template <int KEEP>
__device__ __noinline__ void longer_lists(const uint32_t* __restrict__ sorted_slot,
                                          const float2* __restrict__ sorted_pos,
                                          const uint32_t* __restrict__ slot_id, const uint32_t* __restrict__ kstart,
                                          const TileGrid& g, float reach, uint32_t n, uint32_t p, uint32_t count,
                                          uint32_t cap, uint32_t* words, uint32_t* out) {
    constexpr uint32_t FULL = 0xffffffffu, kRows = QueryShared<KEEP, true>::kRows;
    uint32_t longer = __ballot_sync(FULL, count != 0u);
    const uint32_t lanes = (uint32_t)__popc(longer), most = __reduce_max_sync(FULL, min(count, cap));
    if constexpr (KEEP == kQueryKeep) {
        uint32_t width = 32u;
        while (most * width > kRows * 32u) width >>= 1;
        const bool short_walk = __reduce_max_sync(FULL, count) <= 16u * most;
        if (lanes <= (short_walk ? 2u * width : width)) {
            lists_by_lane<kOrdered>(sorted_slot, sorted_pos, slot_id, kstart, g, reach, n, p, count, cap, width, words,
                                    out);
            return;
        }
        if (most <= 96u) {
            lists_by_lane<kInPlace>(sorted_slot, sorted_pos, slot_id, kstart, g, reach, n, p, count, cap, 32u, words,
                                    out);
            return;
        }
    } else if (most <= kRows && lanes >= 16u + most / 4u) {
        lists_by_lane<kUnordered>(sorted_slot, sorted_pos, slot_id, kstart, g, reach, n, p, count, cap, 32u, words, out);
        return;
    }
    const float2 me = sorted_pos[min(p, n - 1u)];
    for (; longer; longer &= longer - 1u) {
        const int o = __ffs(longer) - 1;
        list_by_warp<kRows>(sorted_slot, sorted_pos, slot_id, kstart, g, reach, n, p - (threadIdx.x & 31u) + (uint32_t)o,
                            make_float2(__shfl_sync(FULL, me.x, o), __shfl_sync(FULL, me.y, o)), cap, words,
                            reinterpret_cast<uint32_t*>(
                                __shfl_sync(FULL, reinterpret_cast<unsigned long long>(out), o)));
    }
}

// Resident blocks per SM.  Sparse and counts alone: 16 (64 warps), at 40 registers (12
// blocks) the symmetric pair loop gained nothing (0.435 against 0.437 ms at 16 M), at 32 it
// takes 0.395; reading back dense pair lists takes six in flight per lane and 12.  Lists of
// dense populations: as many as their places in shared memory allow.
constexpr int query_blocks(bool list, int keep, PairLists pairs) {
    if (keep == kQueryKeep) return 16;
    if (!list) return pairs == kPairsUsed ? 12 : 16;
    return keep == kQueryKeepDense ? 9 : 7;
}
template <bool LIST, int KEEP, PairLists PAIRS>
__global__ __launch_bounds__(kQueryThreads, query_blocks(LIST, KEEP, PAIRS)) void k_query(const uint32_t* __restrict__ kstart,
                                                         const uint32_t* __restrict__ sorted_slot,
                                                         const float2* __restrict__ sorted_pos,
                                                         const uint32_t* __restrict__ slot_id,
                                                         const __grid_constant__ TileGrid g,
                                                         uint32_t n, uint32_t cap, uint32_t* __restrict__ count_out,
                                                         uint32_t* __restrict__ list,
                                                         unsigned long long* __restrict__ pair_bins,
                                                         unsigned long long* __restrict__ next_bins,
                                                         const uint32_t* err, uint32_t* __restrict__ count_by_id,
                                                         PairStore store) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ QueryShared<KEEP, LIST> sh;
    // read first, tested once the other first loads are in flight (they stay in range
    // whatever an index update left behind)
    const uint32_t status = err ? ld_relaxed(err) : 0u;
    float reach = g.reach;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31;
    const uint32_t warp = tid >> 5;
    const uint32_t p = blockIdx.x * kQueryThreads + tid;
    const uint32_t pwarp = p - lane;
    const bool valid = p < n;
    float2 me = make_float2(0.f, 0.f);
    constexpr bool DENSE = LIST && KEEP != kQueryKeep;
    // pairs in flight per lane (dense 2 / 4 / 6: 1 M entities with 4.5 neighbours 90.9 / 87.5 /
    // 85.9 us per tick)
    constexpr uint32_t kPairsAtOnce = KEEP != kQueryKeep ? 6 : 2;
    const uint32_t* pairs = PAIRS == kPairsUsed ? store.pairs + (size_t)(p >> 5) * store.places : nullptr;
    uint32_t size = kNoPairs;
    uint32_t pair[kPairsAtOnce], my_id = 0u;
    if (PAIRS == kPairsUsed) {  // the first pairs, their number, position and id in flight together
        size = store.sizes[p >> 5];
#pragma unroll
        for (uint32_t k = 0; k < kPairsAtOnce; k++) pair[k] = pairs[lane + 32u * k];
        my_id = valid ? store.ids[p] : 0u;
    }
    if (valid) me = sorted_pos[p];
    if (status & kErrTimeout) return;  // an index update gave up (index_failed)
    if (PAIRS == kPairsWidened) {
        // an entity within the radius now lay within reach + d when the index was built;
        // a d past the limit (or not finite) leaves the query to the host
        const float d = __uint_as_float(*store.disp);
        if (!(d <= store.widen_limit)) return;
        reach = __fadd_ru(reach, __fmul_ru(d, 1.0f + 0x1p-20f));  // d was measured with one rounding
    }
    sh.me[tid] = me;
    sh.cnt[tid] = 0u;
    uint32_t own = 0u, near_count = 0u;
    if (PAIRS == kPairsKept && valid) {
        const uint32_t s2 = sorted_slot[p];
        store.ids[p] = s2 < n ? (slot_id ? slot_id[s2] : s2) : 0xffffffffu;
    }
    const bool have_ids = PAIRS == kPairsUsed && size != kNoPairs;  // uniform per warp
    if (have_ids) {
        sh.id[tid] = my_id;
        __syncwarp();
        for (uint32_t base = 0; base < size; base += 32u * kPairsAtOnce) {
            float2 o[kPairsAtOnce];
            uint32_t id[kPairsAtOnce];
#pragma unroll
            for (uint32_t k = 0; k < kPairsAtOnce; k++) {
                if (base + 32u * k + lane >= size) continue;
                const uint32_t q = pair[k] & kPairPosition;
                o[k] = sorted_pos[q];
                if (LIST) id[k] = store.ids[q];
            }
#pragma unroll
            for (uint32_t k = 0; k < kPairsAtOnce; k++) {
                const uint32_t i = base + 32u * k + lane;
                if (i >= size) continue;
                const uint32_t owner = pair[k] >> kPairOwnerShift;
                if (in_range_fast(o[k], sh.me[warp * 32u + owner], g.radius, g.d2_limit))
                    count_hit<LIST, KEEP>(sh, warp, owner, pair[k] & kPairPosition, pwarp, id[k],
                                                 sh.id[warp * 32u + owner]);
                if (i + 32u * kPairsAtOnce < size) pair[k] = pairs[i + 32u * kPairsAtOnce];
            }
        }
    } else {
    uint32_t x0 = 1, x1 = 0, y0 = 1, y1 = 0;  // empty box for invalid lanes
    float ylo = 0.f, yhi = 0.f;
    if (valid) {
        ylo = __fsub_rn(me.y, reach);
        yhi = __fadd_rn(me.y, reach);
        x0 = tile_coord(__fsub_rn(me.x, reach), g.inv_cell, g.tiles_x);
        x1 = tile_coord(__fadd_rn(me.x, reach), g.inv_cell, g.tiles_x);
        y0 = tile_coord(ylo, g.inv_cell, g.tiles_y);
        y1 = tile_coord(yhi, g.inv_cell, g.tiles_y);
    }
    const uint32_t nx = x1 >= x0 ? x1 - x0 + 1u : 0u, ny = y1 >= y0 ? y1 - y0 + 1u : 0u;
    if (__all_sync(FULL, nx <= 2u && ny <= 2u)) {
        // at most 2 x 2 tiles (always when the tile side is at least 2 x reach): the
        // tiles' Morton codes by increments; the row y0 runs from the lower box edge's
        // band up (to the last band when the box reaches row y1), row y1 from band 0
        const uint32_t top = (1u << g.ybits) - 1u;
        const uint32_t b_lo = g.ybits ? y_band(g, ylo, y0) : 0u;
        const uint32_t b_hi = g.ybits ? y_band(g, yhi, y1) : 0u;
        const uint32_t m00 = morton2_tile(x0, y0);
        const uint32_t m10 = morton_inc_x(m00);
        const uint32_t tiles[kRuns] = {m00, m10, morton_inc_y(m00), morton_inc_y(m10)};
        const bool have[kRuns] = {nx >= 1u && ny >= 1u, nx == 2u && ny >= 1u, nx >= 1u && ny == 2u,
                                  nx == 2u && ny == 2u};
        uint32_t lo[kRuns], len[kRuns];
#pragma unroll
        for (uint32_t k = 0; k < kRuns; k++) {
            lo[k] = 0u;
            len[k] = 0u;
            if (__any_sync(FULL, have[k]) && have[k]) {
                const uint32_t t = tiles[k] << g.ybits;
                const uint32_t bl = k < 2u ? b_lo : 0u;
                const uint32_t bh = k < 2u ? (ny == 2u ? top : b_hi) : b_hi;
                lo[k] = kstart[t | bl];
                uint32_t hi = kstart[(t | bh) + 1u];
                if (hi > n) hi = n;
                len[k] = hi > lo[k] ? hi - lo[k] : 0u;
            }
        }
        query_runs<LIST, KEEP, PAIRS == kPairsKept>(lo, len, lane, warp, pwarp, sh, sorted_pos, g, own,
                                                           store, near_count);
    } else {
        // general boxes (tile side below 2 x reach): kRuns tiles per round
        const uint32_t nslots = nx * ny;
        const uint32_t max_slots = __reduce_max_sync(FULL, nslots);
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < max_slots; j0 += kRuns) {
            uint32_t lo[kRuns], len[kRuns];
#pragma unroll
            for (uint32_t k = 0; k < kRuns; k++) {
                const uint32_t j = j0 + k;
                lo[k] = 0u;
                len[k] = 0u;
                if (j < nslots) {
                    const uint32_t jy = j / nx;
                    const uint32_t tx = x0 + (j - jy * nx), ty = y0 + jy;
                    const uint32_t t = morton2(tx, ty) << g.ybits;
                    const uint32_t b0 = g.ybits ? y_band(g, ylo, ty) : 0u;
                    const uint32_t b1 = g.ybits ? y_band(g, yhi, ty) : 0u;
                    lo[k] = kstart[t | b0];
                    uint32_t hi = kstart[(t | b1) + 1u];
                    if (hi > n) hi = n;
                    len[k] = hi > lo[k] ? hi - lo[k] : 0u;
                }
            }
            query_runs<LIST, KEEP, PAIRS == kPairsKept>(lo, len, lane, warp, pwarp, sh, sorted_pos, g, own,
                                                           store, near_count);
        }
    }
    if (PAIRS == kPairsKept && lane == 0) store.sizes[p >> 5] = near_count <= store.places ? near_count : kNoPairs;
    }
    __syncwarp();
    const uint32_t count = valid ? sh.cnt[tid] + own : 0u;
    if (valid) {
        count_out[p] = count;
        // slots that hold their own entity: the count also goes straight to its id's
        // place (the host tick downloads these, with no export pass after the query)
        if (count_by_id) count_by_id[sorted_slot[p]] = count;
    }
    const uint32_t warp_sum = __reduce_add_sync(FULL, count);  // every pair is seen from both ends
    // the next query's counters (a memset for them stood between two queries)
    if (p < kPairBins) next_bins[p] = 0ull;
    if (lane == 0 && warp_sum) atomicAdd(&pair_bins[(p >> 5) & (kPairBins - 1u)], (unsigned long long)warp_sum);
    if constexpr (LIST) {
        const uint32_t kept = count < cap ? count : cap;
        uint32_t incl = kept;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        uint32_t* out = list + (size_t)(p >> 5) * 32u * cap + (incl - kept);
        // the warp's largest list that was kept bounds the (warp-uniform) loops below
        const uint32_t listed = count <= (uint32_t)KEEP ? count : 0u;
        const uint32_t wmax = __reduce_max_sync(FULL, listed);
        if (!DENSE || wmax <= kSortInRegisters) {
            uint32_t id[kSortInRegisters];  // ascending; unused slots hold 0xffffffff
#pragma unroll
            for (int i = 0; i < kSortInRegisters; i++) {  // all fetches of a lane in flight together
                id[i] = 0xffffffffu;
                if ((uint32_t)i < wmax) {
                    const uint32_t k = DENSE && (uint32_t)i >= own ? (uint32_t)i + (uint32_t)KEEP - listed : (uint32_t)i;
                    const uint32_t x = (uint32_t)i < listed ? sh.place(warp, k, lane) : 0xffffffffu;
                    if (have_ids) {
                        id[i] = x;
                        continue;
                    }
                    const uint32_t s2 = (uint32_t)i < listed ? sorted_slot[x] : n;
                    id[i] = s2 < n ? (slot_id ? slot_id[s2] : s2) : 0xffffffffu;  // NULL: slot = id
                }
            }
            uint32_t keep[kSortInRegisters];
#pragma unroll
            for (int i = 0; i < kSortInRegisters; i++) keep[i] = 0xffffffffu;
#pragma unroll
            for (int i = 0; i < kSortInRegisters; i++) {
                if ((uint32_t)i >= wmax) continue;  // uniform
                // keep[0..i) is sorted and slot i is free: insert there and sink it, i
                // compare-exchanges (w (w - 1) / 2 in all for a warp's largest list w)
                keep[i] = id[i];
#pragma unroll
                for (int j = i; j > 0; j--) {
                    const uint32_t lo = min(keep[j - 1], keep[j]), hi = max(keep[j - 1], keep[j]);
                    keep[j - 1] = lo;
                    keep[j] = hi;
                }
            }
#pragma unroll
            for (int i = 0; i < kSortInRegisters; i++) {
                if ((uint32_t)i >= wmax) break;  // uniform
                if ((uint32_t)i < min(listed, cap)) out[i] = keep[i];
            }
        } else {
            // longer lists: every id to rows 0 .. of its lane's column (row i of the list lies
            // at i, or at i + KEEP - listed for the credited ones: never below i), then two
            // elements of a column per lane, the warp's pairs of elements end to end: each
            // element to its rank in its column
#pragma unroll 4
            for (uint32_t i = 0; i < wmax; i++) {
                if (i < listed) {
                    const uint32_t x = sh.place(warp, i < own ? i : i + (uint32_t)KEEP - listed, lane);
                    const uint32_t s2 = have_ids ? n : sorted_slot[x];
                    sh.place(warp, i, lane) = have_ids ? x : s2 < n ? (slot_id ? slot_id[s2] : s2) : 0xffffffffu;
                }
            }
            __syncwarp();
            const uint32_t couples = (listed + 1u) / 2u;
            uint32_t li = couples;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, li, o);
                if (lane >= (uint32_t)o) li += y;
            }
            const uint32_t total = __shfl_sync(FULL, li, 31);
            const uint32_t place = incl - kept;  // the lane's first place in the warp's output
            uint32_t* warp_out = out - place;
            for (uint32_t base = 0; base < total; base += 32u) {
                const uint32_t i = base + lane;
                uint32_t o = 0;  // first lane whose inclusive prefix exceeds i
#pragma unroll
                for (uint32_t st = 16; st > 0; st >>= 1) {
                    const uint32_t v = __shfl_sync(FULL, li, o + st - 1u);
                    if (v <= i) o += st;
                }
                o &= 31u;
                const uint32_t m = __shfl_sync(FULL, listed, o), to = __shfl_sync(FULL, place, o);
                const uint32_t first = __shfl_sync(FULL, li - couples, o);
                if (i < total) {
                    const uint32_t* col = &sh.place(warp, 0u, o);
                    const uint32_t j = 2u * (i - first);
                    const uint32_t a = col[j * 32u];
                    const uint32_t b = j + 1u < m ? col[(j + 1u) * 32u] : 0xffffffffu;
                    uint32_t ra = 0, rb = 0;
#pragma unroll 4
                    for (uint32_t k = 0; k < m; k++) {
                        const uint32_t x = col[k * 32u];
                        ra += x < a ? 1u : 0u;
                        rb += x < b ? 1u : 0u;
                    }
                    if (ra < cap) warp_out[to + ra] = a;
                    if (j + 1u < m && rb < cap) warp_out[to + rb] = b;
                }
            }
        }
        // a few in a million in a sparse population, unless entities stand at one point
        const uint32_t beyond = count > (uint32_t)KEEP ? count : 0u;
        if (!__any_sync(FULL, beyond != 0u)) return;
        __syncwarp();  // the kept lists are written out: their words are free
        if constexpr (DENSE && (PAIRS == kPairsUsed || PAIRS == kPairsKept)) {
            const uint32_t known = PAIRS == kPairsUsed ? size : near_count <= store.places ? near_count : kNoPairs;
            if (known != kNoPairs &&
                lists_from_pairs<KEEP>(store.pairs + (size_t)(p >> 5) * store.places, known, sorted_slot, slot_id, sorted_pos,
                                       g.radius, g.d2_limit, n, pwarp, beyond, incl - kept, cap, sh,
                                       list + (size_t)(p >> 5) * 32u * cap))
                return;
        }
        longer_lists<KEEP>(sorted_slot, sorted_pos, slot_id, kstart, g, reach, n, p, beyond, cap,
                           &sh.place(warp, 0u, 0u), out);
    }
}
