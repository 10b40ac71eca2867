// Seed batch generation, neighbour sampling, per-hop dedup and relabel.
//
// A batch is one launch that empties the id map and takes the seed slice, then two launches per hop on one
// stream, with every size kept on the device:
//   hop_sample  : G lanes per input node read its CSR range, draw the neighbours (Philox4x32-10 counter RNG)
//                 and enter every neighbour into the batch-local id map with the minimum of its entry
//                 numbers (input * fanout + slot: the order of the edges, without knowing how many edges the
//                 inputs before it have)
//   hop_finish  : one scan over the entries that counts edges and new nodes together; edges leave at their
//                 final positions, new nodes get their local ids in order of first appearance, every edge
//                 gets the local id of its source; the CTA of the last tile advances the counters
// The edge order (input after input, slot after slot) and the node order (first appearance in
// that edge order) do not depend on scheduling, so a host replay reproduces them bit for bit.
//
// Replaces batch_generate / random_sample / construct_graph / counter_update / ClearPosMap of
// sampling_server/src/engine/operator_impl.cu:28-91,178-317,598-604: the O(N) bitmap and
// position_map become a batch-local open-addressing map that stays in L2, the fixed <<<16,512>>>
// grid becomes a grid sized from the SM count, and the blocking counter read-backs disappear.
#include "common.cuh"
#include <cstdlib>

namespace legion {

static constexpr unsigned kFull = 0xFFFFFFFFu;

// Programmatic dependent launch.  A kernel launched with the attribute may be scheduled while its
// predecessor in the stream is still running; it must not touch the predecessor's results before
// pdl_wait() returns (all prerequisite grids complete, their writes visible).  pdl_trigger() lets the
// successor of THIS kernel be scheduled as soon as every CTA of this kernel has started.  Both are
// no-ops for a kernel launched the ordinary way.  The point: a hop is two kernels of 5-25 us, and the
// drain / launch / ramp-up between two of them costs as much as a quarter of one.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint32_t mix32(uint32_t h)
{
    h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16;
    return h;
}

// One probe of map slot `m` for `key`.  True: the slot is the key's, and its value is at most `cand`.
// A slot is read, claimed and lowered as one 8-byte word, the value in its upper half, so that its accesses never
// overlap in part: a key that is met for the first time costs one load and one compare-and-swap, a key whose value is
// already below `cand` (a seed, a node of an earlier hop, a hub that other inputs have reached) one load.  Values (never
// negative) only fall and keys never change once written, so a stale read can only lead to an atomic that changes
// nothing.
__device__ __forceinline__ bool map_claim(MapSlot *m, int32_t key, int32_t cand)
{
    const unsigned long long empty = ((unsigned long long)(uint32_t)kEmptyVal << 32) | (uint32_t)kEmptyKey;
    const unsigned long long mine = ((unsigned long long)(uint32_t)cand << 32) | (uint32_t)key;
    unsigned long long *const word = reinterpret_cast<unsigned long long *>(m);
    unsigned long long w = __ldcg(word);
    if (w == empty) {
        w = atomicCAS(word, empty, mine);
        if (w == empty) return true;
    }
    if ((int32_t)(uint32_t)w != key) return false;
    if (w > mine) atomicMin(word, mine);
    return true;
}

// Enters `key` and lowers its value to `cand`; returns the slot.
// The front region is tried first (kFrontProbes slots from the key's home slot).  Slots never empty
// during a batch, so every thread that carries the same key sees the same first usable slot there, or
// finds all of them taken by other keys and moves on to the back region, like every other thread
// with that key.
__device__ __forceinline__ int32_t map_insert_min(MapSlot *map, MapDims dims, int32_t key, int32_t cand,
                                                  int32_t *ctl)
{
    const uint32_t h = mix32((uint32_t)key);
    uint32_t s = h & dims.front_mask;
    for (int probe = 0; probe < kFrontProbes; ++probe) {
        if (map_claim(&map[s], key, cand)) return (int32_t)s;
        s = (s + 1) & dims.front_mask;
    }
    if (ctl[CTL_BACK_DIRTY] == 0) ctl[CTL_BACK_DIRTY] = 1;
    MapSlot *back = map + dims.front_mask + 1;
    s = mix32(h ^ 0x9E3779B9u) & dims.back_mask;
    for (uint32_t probe = 0; probe <= dims.back_mask; ++probe) {
        if (map_claim(&back[s], key, cand)) return (int32_t)(dims.front_mask + 1 + s);
        s = (s + 1) & dims.back_mask;
    }
    atomicCAS(&ctl[CTL_ERROR], DERR_NONE, DERR_MAP_FULL);
    return 0;
}

__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                              uint32_t k0, uint32_t k1, uint32_t &o0, uint32_t &o1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        uint32_t n0 = hi1 ^ c1 ^ k0;
        uint32_t n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    o0 = c0; o1 = c1;
}

// one bounded draw in [0, n): 64 random bits times n, high half
__device__ __forceinline__ uint32_t draw_below(uint32_t input_index, uint32_t lane, uint32_t round,
                                               uint32_t hop, uint32_t batch_id, uint32_t k0, uint32_t k1,
                                               uint32_t n)
{
    uint32_t w0, w1;
    philox4x32_10(input_index, round * 32u + lane, hop, batch_id, k0, k1, w0, w1);
    unsigned long long r64 = ((unsigned long long)w1 << 32) | w0;
    return (uint32_t)__umul64hi(r64, (unsigned long long)n);
}

// m distinct values of [0, n) in lanes 0..m-1 of every group of G lanes (m <= G, m < n; m, n and the node are the
// group's own).  All 32 lanes take part; lanes >= m of a group hold a dummy that can never compare equal.  A lane
// keeps its draw unless a lane of its group that already holds the value, or a lower lane that drew it in the same
// round, exists.
template <int G>
__device__ __forceinline__ uint32_t draw_distinct(int m, uint32_t n, uint32_t input_index, uint32_t hop,
                                                  uint32_t batch_id, uint32_t k0, uint32_t k1, int max_rounds, int lane)
{
    const int sub = lane & (G - 1);
    const unsigned group = (G == 32 ? kFull : ((1u << (G & 31)) - 1u)) << (lane & ~(G - 1));
    bool kept = sub >= m;
    uint32_t x = 0x80000000u | (uint32_t)lane;
    for (int r = 0; r < max_rounds; ++r) {
        const unsigned keptmask = __ballot_sync(kFull, kept);
        if (keptmask == kFull) return x;
        if (!kept) x = draw_below(input_index, (uint32_t)sub, (uint32_t)r, hop, batch_id, k0, k1, n);
        const unsigned peers = __match_any_sync(kFull, x) & group;
        if (!kept) kept = ((peers & keptmask) == 0u) && ((__ffs(peers) - 1) == lane);
    }
    // Lanes still without a value after max_rounds take the next free value, in lane order.
    unsigned keptmask = __ballot_sync(kFull, kept);
    for (int guard = 0; guard < G && keptmask != kFull; ++guard) {
        const unsigned open = ~keptmask & group;
        const int l = open != 0u ? __ffs(open) - 1 : lane;
        uint32_t cand = __shfl_sync(kFull, x, l);
        for (int it = 0; it < 64; ++it) {
            const unsigned clash = __ballot_sync(kFull, open != 0u && kept && sub < m && x == cand);
            if (clash == 0u) break;
            if (clash & group) cand = (cand + 1u) % n;
        }
        if (lane == l && open != 0u) { x = cand; kept = true; }
        keptmask = __ballot_sync(kFull, kept);
    }
    return x;
}

// exclusive scan over the CTA (kScanThreads threads); smem holds 8 ints
__device__ __forceinline__ int block_excl_scan(int x, int *total, int *smem)
{
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int t = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) smem[warp] = incl;
    __syncthreads();
    int wo = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        int s = smem[w];
        if (w < warp) wo += s;
        tot += s;
    }
    __syncthreads();
    *total = tot;
    return wo + incl - x;
}

// ---- batch start -----------------------------------------------------------------------------

// First kernel of every batch: empties the id map, zeroes the counters, stores the batch's parameters (the only
// values of the batch that are passed by value) and takes the seed slice with its labels (batch_generate,
// operator_impl.cu:28-56).  The front region of the map is always cleared; the back region only if the last batch
// on this pipe put anything there.  The seeds enter the map with the first hop.
__global__ void batch_start_kernel(uint4 *slots2, int64_t n_pairs, int32_t *ctl, int32_t *nc, int32_t *ec,
                                   BatchCtl *bctl, BatchCtl value, int64_t back_pairs, int32_t *ids, int32_t *labels)
{
    __shared__ int s_dirty;
    if (threadIdx.x == 64) {
        // the CTA that is the last to have read the flag lowers it; nothing enters the map before the next kernel
        s_dirty = __ldcg(&ctl[CTL_BACK_DIRTY]);  // final since the end of the last batch's sampling
        __threadfence();
        if (atomicAdd(&ctl[CTL_TICKET_D], 1) == (int)gridDim.x - 1) {
            ctl[CTL_BACK_DIRTY] = 0;
            ctl[CTL_TICKET_D] = 0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 32) *bctl = value;
    if (blockIdx.x == 0 && threadIdx.x < 16) {
        // the error words are sticky, and the dirty flag and its ticket belong to the CTAs of this kernel
        if (threadIdx.x == CTL_LATE_ERROR && ctl[CTL_LATE_ERROR] != DERR_NONE) {
            if (ctl[CTL_ERROR] == DERR_NONE) ctl[CTL_ERROR] = ctl[CTL_LATE_ERROR];
        }
        if (threadIdx.x != CTL_ERROR && threadIdx.x != CTL_BAD_IDS && threadIdx.x != CTL_BACK_DIRTY && threadIdx.x != CTL_TICKET_D)
            ctl[threadIdx.x] = threadIdx.x == CTL_N_NODES ? value.size : 0;
        nc[threadIdx.x] = 0;  // cudaMemsetAsync of both counters, operator_impl.cu:158-159
        ec[threadIdx.x] = 0;
        __syncwarp(0xFFFFu);
        if (threadIdx.x == 0) {  // counter_update of op 0, operator_impl.cu:60-65
            nc[1] = value.size;
            nc[LEGION_INTRABATCH_CON * 3] = value.size;
            nc[LEGION_INTRABATCH_CON * 3 - 1] = value.hop_num;
        }
    }
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < value.size; idx += gridDim.x * blockDim.x) {
        const int64_t pos = value.first + idx;
        int32_t id = -1, label = -1;
        if (pos < value.total_cap) {  // operator_impl.cu:41-43
            id = value.all_ids[pos];
            label = value.all_labels[pos];
            if (id >= value.n_nodes) {  // not a node of this graph: skipped like an overrun slot, and reported
                id = -1;
                ctl[CTL_BAD_IDS] = 1;
            }
        }
        ids[idx] = id;
        labels[idx] = label;
    }
    const uint4 empty = make_uint4((uint32_t)kEmptyKey, (uint32_t)kEmptyVal, (uint32_t)kEmptyKey,
                                   (uint32_t)kEmptyVal);
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_pairs; i += step) slots2[i] = empty;
    __syncthreads();
    if (s_dirty == 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < back_pairs; i += step) slots2[n_pairs + i] = empty;
}

// ---- one hop -----------------------------------------------------------------------------------

// A stretch of a hop's inputs (launch_sample_hop).
struct HopPart {
    int32_t first, count, last;
};
__device__ __forceinline__ int part_inputs(const HopPart &p, int inputs) { return max(0, min(p.count, inputs - p.first)); }

// Lanes that share an input node: the fanout, rounded up to 8, 16 or 32.
static inline int group_lanes(int fanout) { return fanout <= 8 ? 8 : fanout <= 16 ? 16 : 32; }

// A warp takes a chunk of consecutive input nodes: one coalesced load of their ids and one round of loads of their
// CSR ranges for all of them, then 32 / G nodes at a time, G lanes each, draw their neighbours.
// Entry i * fanout + s of `rec` holds (neighbour id, its map slot) of slot s of input i, or slot -1.
// Bound by latency: neighbour id from HBM, map slot and compare-and-swap in L2, one after the other; small chunks
// keep every warp of the chip on its own chain.
// In the batch's first hop the seeds enter the map too, each with its position.
// PART: the launch takes the inputs [part.first, part.first + part.count) of the hop.
template <int G, bool PART>
__global__ void __launch_bounds__(256, 6)
hop_sample_kernel(const int64_t *__restrict__ indptr, const int32_t *__restrict__ indices, const int32_t *ids,
                  int32_t fanout, uint32_t hop, const BatchCtl *__restrict__ b, int2 *rec, MapSlot *map, MapDims mask,
                  int32_t *ctl, const int32_t *nc, uint8_t *edge_cnt, uint32_t *tile_state, int64_t max_entries, HopPart part)
{
    pdl_wait();
    pdl_trigger();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, n_threads = gridDim.x * blockDim.x;
    const int late = ctl[CTL_LATE_ERROR];
    const int known = ctl[CTL_N_NODES];
    const int inputs = !PART || part.first == 0 ? known : ctl[CTL_HOP_N];
    if (tid == 0) {
        ctl[CTL_TILE] = 0;
        if (!PART || part.first == 0) ctl[CTL_HOP_N] = known;
        ctl[CTL_PART_N] = known;
        ctl[CTL_PART_E] = ctl[CTL_E_TOTAL];
        if (late != DERR_NONE) atomicCAS(&ctl[CTL_ERROR], DERR_NONE, late);
    }
    if (ctl[CTL_ERROR] != DERR_NONE || late != DERR_NONE) return;
    const int lo = PART ? part.first : 0;
    const int n = PART && !part.last ? part_inputs(part, inputs) : inputs - lo;
    // (cannot happen unless a captured sequence of ops is replayed behind others than it was captured behind)
    if (n > 0 && (int64_t)n * fanout > max_entries) {
        if (threadIdx.x == 0) atomicCAS(&ctl[CTL_ERROR], DERR_NONE, DERR_EDGE_OVERFLOW);
        return;
    }
    const uint32_t k = (uint32_t)fanout;
    // the tiles that hop_finish_kernel is about to scan have not been counted yet
    for (int t = tid, n_tiles = (n * fanout + kTile - 1) / kTile; t < n_tiles; t += n_threads) tile_state[t] = 0;
    const uint32_t batch_id = b->global_batch, k0 = b->k0, k1 = b->k1;
    const int max_rounds = b->max_rounds;
    const int n_limit = b->n_nodes;
    const bool seeds_in = ctl[CTL_SEEDS_IN] != 0;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const unsigned group = (G == 32 ? kFull : ((1u << (G & 31)) - 1u)) << (lane & ~(G - 1));
    constexpr int NPW = 32 / G;  // nodes that a warp works on together
    const int n_warps = n_threads >> 5;
    int chunk = (n + n_warps - 1) / n_warps;
    chunk = min(32, (chunk + NPW - 1) / NPW * NPW);
    // this hop's per-destination edge counts start behind those of the hops before it, whose destinations were the
    // nodes known when each began (node_counter words 9 .. 9 + hop - 1)
    int cnt0 = 0;
    for (uint32_t h = 0; h < hop; ++h) cnt0 += __ldcg(&nc[LEGION_INTRABATCH_CON * 3 + h]);
    for (int64_t first = (int64_t)(tid >> 5) * chunk; first < n; first += (int64_t)n_warps * chunk) {
        const int here = min(chunk, n - (int)first);
        int64_t my_start = 0;
        int32_t my_deg = 0;
        if (lane < here) {
            const int32_t id = __ldcg(&ids[lo + first + lane]);
            if (id >= 0) {
                if (id < n_limit) {
                    my_start = __ldg(&indptr[id]);
                    my_deg = (int32_t)(__ldg(&indptr[id + 1]) - my_start);
                } else {  // a neighbour id that the topology itself got wrong is never followed
                    ctl[CTL_BAD_IDS] = 1;
                }
            }
            edge_cnt[cnt0 + lo + first + lane] = (uint8_t)min((uint32_t)my_deg, k);
            if (!seeds_in && id >= 0) map_insert_min(map, mask, id, lo + (int)first + lane, ctl);
        }
        for (int j0 = 0; j0 < here; j0 += NPW) {
            const int j = j0 + lane / G;
            const int64_t start = __shfl_sync(kFull, (long long)my_start, j & 31);
            const uint32_t deg_j = (uint32_t)__shfl_sync(kFull, my_deg, j & 31);
            const uint32_t deg = j < here ? deg_j : 0u;
            const uint32_t i = (uint32_t)first + (uint32_t)j;  // of this launch's inputs
            // drawn: deg >= 2k draws the k positions to take, k < deg < 2k the deg - k positions to leave out
            const bool leave_out = deg > k && deg < 2 * k;
            const int m = deg <= k ? 0 : leave_out ? (int)(deg - k) : (int)k;
            const uint32_t x = draw_distinct<G>(m, deg, (uint32_t)lo + i, hop, batch_id, k0, k1, max_rounds, lane);
            int out_slot = -1, out_slot2 = -1;   // slot of this lane's first edge, second edge in out_slot2
            uint32_t pos = sub, pos2 = sub + G;
            if (!leave_out) {
                if ((uint32_t)sub < min(deg, k)) out_slot = sub;
                if (deg > k) pos = x;
            }
            if (__any_sync(kFull, leave_out)) {
                // positions 0 .. deg - 1 without the drawn ones; deg < 2k <= 2G, so two per lane
                const bool drawn = leave_out && sub < m;
                const uint32_t out0 = __reduce_or_sync(group, drawn && x < 32u ? 1u << x : 0u);
                const uint32_t out1 = G == 32 ? __reduce_or_sync(group, drawn && x >= 32u ? 1u << (x - 32u) : 0u) : 0u;
                if (leave_out) {
                    const uint32_t keep0 = ~out0 & (deg >= 32u ? 0xFFFFFFFFu : (1u << deg) - 1u);
                    if ((keep0 >> sub) & 1u) out_slot = __popc(keep0 & ((1u << sub) - 1u));
                    if (G == 32) {
                        const uint32_t keep1 = ~out1 & (deg <= 32u ? 0u : (1u << (deg - 32u)) - 1u);
                        if ((keep1 >> sub) & 1u) out_slot2 = __popc(keep0) + __popc(keep1 & ((1u << sub) - 1u));
                    } else {
                        if ((keep0 >> (sub + (G & 31))) & 1u) out_slot2 = __popc(keep0 & ((1u << (sub + (G & 31))) - 1u));
                    }
                }
            }
            const int e0 = (int)(i * k);
            int32_t u = 0, u2 = 0;
            if (out_slot >= 0) u = __ldg(&indices[start + pos]);
            if (out_slot2 >= 0) u2 = __ldg(&indices[start + pos2]);
            if (out_slot >= 0) {
                const int e = e0 + out_slot;
                rec[e] = make_int2(u, map_insert_min(map, mask, u, kNewBase + e, ctl));
            }
            if (out_slot2 >= 0) {
                const int e = e0 + out_slot2;
                rec[e] = make_int2(u2, map_insert_min(map, mask, u2, kNewBase + e, ctl));
            }
            if (j < here && (uint32_t)sub >= deg && (uint32_t)sub < k) rec[e0 + sub] = make_int2(-1, -1);
        }
    }
}

constexpr uint32_t kTileCounted = 0x80000000u;
// reads of a wait inside the scan before it gives up (legion_set_tunable "scan_wait_limit"); about a second
constexpr int kScanWaitLimit = 1 << 20;
int g_scan_wait_limit = kScanWaitLimit;

// The end of a hop that found c nodes and e edges: counter_update for op_id (a multiple of LEGION_INTRABATCH_CON) on
// both counter arrays, held one word per lane by the warp that calls; with a mirror (the last hop) both arrays also go
// to page-locked host memory, one posted store per lane: the host learns the sizes of the batch without a copy-engine
// transfer queued behind other batches' exports.  The end of a part that is not the hop's last (`closes` false) only
// adds to the words that count the hop.  A hop that failed has found nothing: the batch ends with the hops before it.
__device__ __forceinline__ void advance_counters(int word, int c, int e, int n0, int e_base, int op_id, int32_t *ctl, int32_t *nc,
                                                 int32_t *ec, int32_t *mirror, bool closes, bool failed)
{
    constexpr int C = LEGION_INTRABATCH_CON;
    const int lane = threadIdx.x & 31, h = op_id / C;
    const int known = __shfl_sync(kFull, word, 0) + __shfl_sync(kFull, word, 1);
    const int found = failed ? 0 : __shfl_sync(kFull, word, C * 2) + c;                     // operator_impl.cu:281
    const int done = __shfl_sync(kFull, word, 16) + __shfl_sync(kFull, word, 17);
    const int drawn = failed ? 0 : __shfl_sync(kFull, word, 18) + e;                        // operator_impl.cu:282
    bool changed = true;                                                                    // operator_impl.cu:66-80
    if (!closes) {
        if (lane == C * 2) nc[C * 2] = found;
        if (lane == 16 + 2) ec[2] = drawn;
        changed = false;
    } else if (lane == 0) word = known;
    else if (lane == 1) word = found;
    else if (lane == C * 2 || lane == 16 + 2) word = 0;
    else if (lane == C * 2 + 1 || lane == C * 3 + h) word = known + found;
    else if (lane == 16) word = done;
    else if (lane == 17 || lane == 16 + C * 3 + h) word = drawn;
    else if (lane == 16 + C * 4 + h) word = done;
    else changed = false;
    if (changed) *(lane < 16 ? nc + lane : ec + (lane - 16)) = word;
    if (mirror != nullptr) mirror[lane] = word;
    if (lane == 0) {
        ctl[CTL_N_NODES] = n0 + c;
        ctl[CTL_E_TOTAL] = e_base + e;
        ctl[CTL_SEEDS_IN] = 1;
    }
}

// One pass over the entries of a hop, in tiles of 1024.  A CTA counts its tile's edges and the entries that
// reached a node first, publishes both counts, adds up the counts of the tiles before it (each CTA reads them all,
// one word per tile, so nothing is passed from tile to tile) and places its edges and new nodes.
// Tiles are handed out in order by a ticket and a CTA publishes its counts before it waits for others, so the
// lowest unfinished tile never waits: whatever else shares the GPU, every wait ends.  All waits are bounded
// (DERR_SCAN_TIMEOUT).  A CTA that gives up, or whose edges do not fit, places nothing more but still hands out and
// counts tiles, so that the CTA of the last tile always closes the hop.
// The CTA of the last tile knows the hop's totals as soon as it has added up the others' and advances the counters
// there and then: no CTA waits for the end of all others (the two that did, one of them behind a fence over the stores
// of the whole CTA, were 4 of the 9-11 us that the launch took on two tiles).
// The local id of a node that another entry reached first is written to its map slot by that entry's CTA, which has
// an earlier tile, or the same one.
// Bound by L2 latency: record, map slot, counts, map slot.  Four entries per thread: four map reads in flight and fewer
// counts to add up.  (Tiles of 256 in small hops, for more CTAs: eight batches of 800 seeds, [25,10], 267 against 264 us,
// and 295 where hop 2 used them too; one batch alone the same.)
template <bool PART>
__global__ void __launch_bounds__(kScanThreads, 6)
hop_finish_kernel(const int2 *__restrict__ rec, int32_t fanout, uint32_t *tile_state, int32_t *ids, MapSlot *map,
                  int32_t *src_global, int32_t *agg_src, int32_t *agg_dst, int32_t *ctl, int32_t *nc, int32_t *ec, int op_id,
                  const BatchCtl *__restrict__ b, int last_hop, int64_t max_nodes, int64_t max_edges, HopPart part,
                  int wait_limit)
{
    pdl_wait();
    pdl_trigger();
    constexpr int IPT = kTile / kScanThreads, TILE = kTile;
    static_assert(IPT == 4, "records are read as two 16-byte vectors per thread");
    __shared__ int smem[kScanThreads / 32];
    __shared__ int s_edges[kScanThreads / 32], s_new[kScanThreads / 32];
    __shared__ int s_tile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl[CTL_TILE], 1);
    const int n0 = ctl[CTL_PART_N];
    const int e_base = ctl[CTL_PART_E];
    const int inputs = PART ? part_inputs(part, ctl[CTL_HOP_N]) : n0;
    const bool closes = !PART || part.last;
    const bool ok = ctl[CTL_ERROR] == DERR_NONE;  // raised before this kernel: nobody raises it while it runs
    // both counter arrays, one word per lane of the first warp (only this kernel changes what it uses of them)
    const int counter = threadIdx.x < 16 ? nc[threadIdx.x] : threadIdx.x < 32 ? ec[threadIdx.x - 16] : 0;
    int32_t *const mirror = last_hop && closes ? b->mirror : nullptr;
    const int total = ok ? inputs * fanout : 0;
    const int n_tiles = (total + TILE - 1) / TILE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int next = 0, edges = 0, fresh = 0;  // tiles before `next` hold `edges` edges and `fresh` new nodes
    int failed = DERR_NONE;
    if (n_tiles == 0 && blockIdx.x == 0 && warp == 0)
        advance_counters(counter, 0, 0, n0, e_base, op_id, ctl, nc, ec, mirror, closes, !ok);
    for (;;) {
        __syncthreads();
        const int tile = s_tile;
        if (tile >= n_tiles) break;
        const int base = tile * TILE + threadIdx.x * IPT;
        int u[IPT], slot[IPT], val[IPT];
        // rec is padded to whole tiles
        const int4 *r4 = reinterpret_cast<const int4 *>(rec + base);
        const int4 r0 = __ldcs(r4), r1 = __ldcs(r4 + 1);
        u[0] = r0.x; slot[0] = r0.y; u[1] = r0.z; slot[1] = r0.w;
        u[2] = r1.x; slot[2] = r1.y; u[3] = r1.z; slot[3] = r1.w;
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            if (base + j >= total) slot[j] = -1;
            val[j] = slot[j] >= 0 ? __ldcg(&map[slot[j]].val) : 0;
        }
        int count = 0;  // edges in the low half, new nodes in the high half: both at most 1024
#pragma unroll
        for (int j = 0; j < IPT; ++j) count += (slot[j] >= 0 ? 1 : 0) + (slot[j] >= 0 && val[j] == kNewBase + base + j ? 1 << 16 : 0);
        int tile_count;
        int mine = block_excl_scan(count, &tile_count, smem);
        if (threadIdx.x == 0) *(volatile uint32_t *)&tile_state[tile] = kTileCounted | (uint32_t)tile_count;
        int se = 0, sn = 0;
        bool late = failed != DERR_NONE;
        for (int q = next + threadIdx.x; q < tile && !late; q += kScanThreads) {
            uint32_t w = __ldcg(&tile_state[q]);
            for (int spin = 0; (w & kTileCounted) == 0u && spin < wait_limit; ++spin) w = *(volatile uint32_t *)&tile_state[q];
            if ((w & kTileCounted) == 0u) {
                // said before it is settled: the CTA of the last tile, should it have seen this count, then sees the word
                atomicCAS(&ctl[CTL_LATE_ERROR], DERR_NONE, DERR_SCAN_TIMEOUT);
                __threadfence();
                w = *(volatile uint32_t *)&tile_state[q];
            }
            late = (w & kTileCounted) == 0u || wait_limit < 0;
            se += (int)(w & 0xFFFFu);
            sn += (int)((w & ~kTileCounted) >> 16);
        }
        se = __reduce_add_sync(kFull, se);
        sn = __reduce_add_sync(kFull, sn);
        if (lane == 0) { s_edges[warp] = se; s_new[warp] = sn; }
        if (__syncthreads_or(late ? 1 : 0) && failed == DERR_NONE) failed = DERR_SCAN_TIMEOUT;
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; ++w) { edges += s_edges[w]; fresh += s_new[w]; }
        const int tile_edges = tile_count & 0xFFFF, tile_new = tile_count >> 16;
        // (in the pool's order they always fit: legion_pool_create sizes both buffers for it)
        if (failed == DERR_NONE && (int64_t)e_base + edges + tile_edges > max_edges) failed = DERR_EDGE_OVERFLOW;
        if (failed == DERR_NONE && (int64_t)n0 + fresh + tile_new > max_nodes) failed = DERR_NODE_OVERFLOW;
        if (failed != DERR_NONE && threadIdx.x == 0) atomicCAS(&ctl[CTL_LATE_ERROR], DERR_NONE, failed);
        if (tile == n_tiles - 1 && warp == 0)
            advance_counters(counter, fresh + tile_new, edges + tile_edges, n0, e_base, op_id, ctl, nc, ec, mirror, closes,
                             failed != DERR_NONE);
        if (failed == DERR_NONE) {
            int at = e_base + edges + (mine & 0xFFFF);
            int local = n0 + fresh + (mine >> 16);
            int dst = base / fanout, in_row = base - dst * fanout;
            if (PART) dst += part.first;
            int where[IPT];
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                where[j] = -1;
                if (slot[j] >= 0) {
                    src_global[at] = u[j];
                    agg_dst[at] = dst;
                    if (val[j] == kNewBase + base + j) {
                        ids[local] = u[j];
                        __stcg(&map[slot[j]].val, local);
                        val[j] = local++;
                    }
                    if (val[j] < kNewBase) agg_src[at] = val[j];
                    else where[j] = at;  // first reached by another entry of this hop
                    ++at;
                }
                if (++in_row == fanout) { in_row = 0; ++dst; }
            }
            const bool last_tile = tile == n_tiles - 1 && warp == 0;
            const int others = last_tile ? *(volatile int32_t *)&ctl[CTL_LATE_ERROR] : DERR_NONE;
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                if (where[j] < 0) continue;
                int v = __ldcg(&map[slot[j]].val);
                for (int spin = 0; v >= kNewBase && spin < wait_limit; ++spin) {
                    v = *(volatile int32_t *)&map[slot[j]].val;
                    if ((spin & 1023) == 1023 && *(volatile int32_t *)&ctl[CTL_LATE_ERROR] != DERR_NONE) break;
                }
                if (v >= kNewBase) {
                    atomicCAS(&ctl[CTL_LATE_ERROR], DERR_NONE, DERR_SCAN_TIMEOUT);
                    v = 0;  // a local id all the same: the batch is reported, not left with an index that is none
                }
                agg_src[where[j]] = v;
            }
            // a CTA that gave up while this one did not: the hop is closed once more, without what it found
            if (last_tile && __any_sync(kFull, others != DERR_NONE))
                advance_counters(counter, 0, 0, n0, e_base, op_id, ctl, nc, ec, mirror, closes, true);
        }
        if (n_tiles <= (int)gridDim.x) break;  // a tile for every CTA
        edges += tile_edges;
        fresh += tile_new;
        next = tile + 1;
        if (threadIdx.x == 0) s_tile = atomicAdd(&ctl[CTL_TILE], 1);
    }
}

// ---- launchers -----------------------------------------------------------------------------------

// 1: the kernels of a batch after its first are launched as programmatic dependents; 0: never; -1: by the rule below
// (legion_set_tunable "pdl"; start value from the environment variable LEGION_PDL)
static int pdl_from_env()
{
    const char *v = getenv("LEGION_PDL");
    if (v == nullptr || (v[0] != '0' && v[0] != '1') || v[1] != 0) return -1;
    return v[0] - '0';
}
int g_pdl = pdl_from_env();
// front region of the id map = worst-case slots >> this; -1: sized by legion_pool_create's own rule
// (legion_set_tunable "map_front_shift")
int g_map_front_shift = -1;

// The rule: batches that have the GPU to themselves, in pools of one pipe, and small ones, whose launches are mostly start
// and drain.  Measured, us a batch, ordinary against dependent launches, fanout [25,10], all rows cached: one pipe
// 59.3 / 51.6 (pool of 65,494 nodes), 71.7 / 65.0 (228,800), 120 / 114 (2.3 M); two pipes 23.3 / 22.3, 29.6 / 29.1,
// 64.2 / 66.3; four pipes 13.2 / 12.9, 18.6 / 18.7, 51.9 / 56.0, and at 128,700 nodes 15.3 / 15.1: with several pipes the
// others' kernels fill the gaps, and the CTAs that wait take registers from them.
constexpr int64_t kDependentNodes = 1 << 16;

template <typename... KArgs, typename... Args>
static cudaError_t launch_dep(const LegionPool *p, void (*kernel)(KArgs...), int grid, int block, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    const bool dependent = g_pdl < 0 ? p->pipes == 1 || p->max_nodes <= kDependentNodes : g_pdl == 1;
    cfg.attrs = dependent ? at : nullptr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

static inline int grid_for(int64_t items, int per_cta, int cap)
{
    int64_t g = (items + per_cta - 1) / per_cta;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

const void *batch_start_kernel_address() { return (const void *)batch_start_kernel; }

BatchCtl make_batch_ctl(const LegionPool *p, const LegionCache *c, const int32_t *all_ids, const int32_t *all_labels,
                        int32_t total_cap, int64_t first, int32_t size, int64_t n_nodes)
{
    BatchCtl v;
    v.all_ids = all_ids;
    v.all_labels = all_labels;
    v.first = first;
    v.total_cap = total_cap;
    v.size = size;
    v.hop_num = p->hop_num;
    v.global_batch = p->global_batch;
    v.k0 = (uint32_t)p->rng_seed;
    v.k1 = (uint32_t)(p->rng_seed >> 32);
    v.max_rounds = p->max_rounds;
    v.clock = (c != nullptr && c->kind == 1) ? c->clock : 0;
    v.n_nodes = (n_nodes > 0 && n_nodes < 0x7FFFFFFF) ? (int32_t)n_nodes : 0x7FFFFFFF;
    // two mirrors per pipe when batches are sampled ahead of the hand-off: the next batch on the pipe may finish its
    // sampling before the host has read the counters of the one before
    v.mirror = p->h_stage[p->pipe] + 2 * (size_t)p->batch_size + 32 +
               (p->slots < p->pipes ? 32 * (p->mirror_flip[p->pipe] & 1) : 0);
    return v;
}

int launch_batch_generate(cudaStream_t s, LegionPool *p, const BatchCtl &v)
{
    const int pipe = p->pipe;
    p->hop_inputs[pipe] = p->batch_size;
    const int64_t n_pairs = ((int64_t)p->map_front_mask + 1) / 2;
    const int64_t back_pairs = ((int64_t)p->map_mask + 1) / 2;
    // sized for the front region and the seeds; when the back region has to be cleared too, the CTAs loop longer
    int64_t threads = n_pairs / 4 > p->batch_size ? n_pairs / 4 : p->batch_size;
    batch_start_kernel<<<grid_for(threads, 256, p->sm_count * 8), 256, 0, s>>>(
        reinterpret_cast<uint4 *>(p->map[pipe]), n_pairs, p->ctl[pipe], p->node_counter[pipe], p->edge_counter[pipe],
        p->bctl[pipe], v, back_pairs, p->ids[pipe], p->labels[pipe]);
    LG_LAUNCH_CHECK();
    return LEGION_OK;
}

template <int G, bool PART>
static cudaError_t launch_hop_sample(cudaStream_t s, LegionPool *p, const LegionGraph *g, int32_t fanout, int32_t hop,
                                     int64_t inputs, HopPart part)
{
    const int pipe = p->pipe;
    return launch_dep(p, hop_sample_kernel<G, PART>, grid_for(inputs, 8 * (32 / G), p->sm_count * 6), 256, s, g->indptr, g->indices, p->ids[pipe], fanout,
                      (uint32_t)hop, p->bctl[pipe], p->edge_rec[pipe], p->map[pipe], MapDims{ p->map_front_mask, p->map_mask },
                      p->ctl[pipe], p->node_counter[pipe], p->edge_cnt[pipe], p->tile_state[pipe], p->max_hop_edges, part);
}

template <bool PART>
static int launch_hop_pair(cudaStream_t s, LegionPool *p, const LegionGraph *g, int32_t fanout, int32_t hop, int32_t op_id,
                           int64_t inputs, HopPart part)
{
    const int pipe = p->pipe;
    switch (group_lanes(fanout)) {
    case 8: LG_CUDA((launch_hop_sample<8, PART>(s, p, g, fanout, hop, inputs, part))); break;
    case 16: LG_CUDA((launch_hop_sample<16, PART>(s, p, g, fanout, hop, inputs, part))); break;
    default: LG_CUDA((launch_hop_sample<32, PART>(s, p, g, fanout, hop, inputs, part))); break;
    }
    LG_CUDA(launch_dep(p, hop_finish_kernel<PART>, grid_for(inputs * fanout, kTile, p->sm_count * 8), kScanThreads, s, p->edge_rec[pipe],
                       fanout, p->tile_state[pipe], p->ids[pipe], p->map[pipe], p->src_global[pipe], p->agg_src[pipe],
                       p->agg_dst[pipe], p->ctl[pipe], p->node_counter[pipe], p->edge_counter[pipe], op_id, p->bctl[pipe],
                       hop + 1 == p->hop_num ? 1 : 0, p->max_nodes, p->max_edges, part, g_scan_wait_limit));
    return LEGION_OK;
}

// In the pool's order every hop's entries (inputs * fanout) fit the records, which legion_pool_create sizes for that.  The
// ops may also come in another order, or more than once; a hop that then could have more inputs is sampled in parts of
// as many as fit, one pair of launches each.  The nodes of an earlier part have their local ids when a later one meets
// them, so the result is that of one pair over all inputs.
int launch_sample_hop(cudaStream_t s, LegionPool *p, const LegionGraph *g, int32_t fanout, int32_t hop, int32_t op_id)
{
    int64_t inputs = p->batch_size;
    for (int h = 0; h < hop; ++h) inputs += inputs * p->fanout[h];  // in the pool's order
    if (inputs < p->hop_inputs[p->pipe]) inputs = p->hop_inputs[p->pipe];
    const int64_t known = inputs + inputs * fanout;
    p->hop_inputs[p->pipe] = known < p->max_nodes ? known : p->max_nodes;
    if (inputs * fanout <= p->max_hop_edges) return launch_hop_pair<false>(s, p, g, fanout, hop, op_id, inputs, HopPart{ 0, 0, 1 });
    const int64_t fit = p->max_hop_edges / fanout;
    for (int64_t first = 0; first < inputs; first += fit) {
        const int rc = launch_hop_pair<true>(s, p, g, fanout, hop, op_id, fit,
                                             HopPart{ (int32_t)first, (int32_t)fit, first + fit >= inputs ? 1 : 0 });
        if (rc != LEGION_OK) return rc;
    }
    return LEGION_OK;
}

}  // namespace legion
