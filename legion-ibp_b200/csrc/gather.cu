// Cache lookup fused with the feature gather.
//
// One warp owns up to 32 consecutive rows of the segment: every lane looks up one id (one coalesced id
// load, one 4-byte table read), turns the answer into a source pointer (this GPU's partition, a
// peer's partition reached by plain loads over NVLink, or the pinned host table reached by
// zero-copy loads), and the warp then copies the rows four at a time with 16-byte loads so that
// 4 x 512 B per warp are in flight before the first store.  Stores are streaming (the trainer
// reads the rows once).  Hit / miss sets leave the kernel in cache_index exactly as FindFeat
// would have written them.
//
// Replaces bght::bcht::find + multiGPU_feat_cache_lookup (sampling_server/src/cache/cache.cu:157-192,
// 743-781; cache/cache_impl.cuh:239-303: thread-per-float, 4-byte loads, 32-64 CTAs) and
// static_retrieve_kernel + static_transfer_kernel (comp_cache/static_cache_kernel.cuh:185-266).
#include "common.cuh"
#include <cstdlib>

#include <cuda_fp8.h>
#include <string.h>

namespace legion {

static constexpr unsigned kFull = 0xFFFFFFFFu;

// List of the rows of a batch whose source is the host table (see miss_begin).
struct MissSink {
    int2 *rows;      // (position in ids, host table row)
    int32_t *count;  // [0] number of entries
    int32_t *hist;   // entries per stretch of 1 << shift rows, or nullptr
    int32_t *rank;
    int32_t shift, n_rows;  // rows of the table
};

// Hand-off of a batch that was sampled ahead.  A pool with fewer hand-off slots than pipes samples into private
// buffers; when the batch's turn comes, its block structure (ids, labels, both edge lists, both counter arrays: ~3 MB for a
// paper100M-shaped batch) is copied into the slot that the consumer reads (the buffers of engine/ipc_service.cu:163-169).
// Sizes are read from the counters on the device.  All of the grid takes part.
struct Publish {
    const int32_t *ids, *labels, *src, *dst, *nc, *ec;
    int32_t *o_ids, *o_labels, *o_src, *o_dst, *o_nc, *o_ec;  // o_ids nullptr: nothing to hand off
};
__device__ __forceinline__ void publish_copy(const Publish &p)
{
    const int hops = p.nc[LEGION_INTRABATCH_CON * 3 - 1];
    const int n = p.nc[LEGION_INTRABATCH_CON * 3 + hops];
    const int n_lab = p.nc[LEGION_INTRABATCH_CON * 3];
    const int e = p.ec[0] + p.ec[1];
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    // every array is padded to whole 1024-element tiles, so whole 16-byte vectors may be copied
    for (int i = tid; i * 4 < n; i += step) reinterpret_cast<int4 *>(p.o_ids)[i] = reinterpret_cast<const int4 *>(p.ids)[i];
    for (int i = tid; i * 4 < e; i += step) {
        const int4 a = reinterpret_cast<const int4 *>(p.src)[i], b = reinterpret_cast<const int4 *>(p.dst)[i];
        reinterpret_cast<int4 *>(p.o_src)[i] = a;
        reinterpret_cast<int4 *>(p.o_dst)[i] = b;
    }
    for (int i = tid; i < n_lab; i += step) p.o_labels[i] = p.labels[i];
    if (blockIdx.x == 0 && threadIdx.x < 16) {
        // words 2 and 3 are the snapshot of the lookup, which segment_of leaves there
        if (threadIdx.x != 2 && threadIdx.x != 3) p.o_nc[threadIdx.x] = p.nc[threadIdx.x];
        p.o_ec[threadIdx.x] = p.ec[threadIdx.x];
    }
}

struct GatherParams {
    const int32_t *ids;
    int32_t *nc;  // node_counter of the pipe
    int32_t *nc_out;  // where the snapshot of the lookup goes: the same, or the hand-off slot's
    int32_t op_id;
    const int32_t *lut;
    int32_t capacity, kg, ki;
    const uint8_t *part[LEGION_MAX_DEVICE + 1];  // part[kg]: this GPU's private copies of rows that peers hold
    const uint8_t *host;
    int64_t n_nodes;
    uint8_t *dst;
    int32_t *cache_index;
    unsigned long long *stats;
    int32_t row_bytes;   // bytes of one output row
    int32_t slot_bytes;  // bytes of one cached row
    int32_t feature_len; // elements per row (quantised codecs)
    int32_t *err;        // device error word of the pipe (sticky), or nullptr
    // rows of uncached seeds that the copy engine staged in device memory for this batch: entry r < stage_n of the
    // id list, when it misses the cache, is row stage_pos[r] - stage_base of stage_rows (nullptr: no staging)
    const uint8_t *stage_rows;
    const int32_t *stage_pos;
    int32_t stage_base, stage_n;
    int32_t n_rows;      // rows of a list of the caller's own; -1: the segment of op_id in the counters
    int32_t rows_per_warp; // fixed by a tunable; 0: chosen by the length of the list
    MissSink miss;
    Publish pub;
};

// A missed row that sits in the batch's staging area is served from there like a cached row; `where` 4 keeps
// it out of the hit / miss counters and off the miss list.
__device__ __forceinline__ void use_staged(const GatherParams &p, int index, int &where, const uint8_t *&src)
{
    if (where == 2 && p.stage_rows != nullptr && index < p.stage_n) {
        src = p.stage_rows + (int64_t)(__ldg(&p.stage_pos[index]) - p.stage_base) * p.row_bytes;
        where = 4;
    }
}

__device__ __forceinline__ const uint8_t *shfl_ptr(const uint8_t *p, int src)
{
    unsigned long long v = (unsigned long long)p;
    unsigned lo = __shfl_sync(kFull, (unsigned)v, src);
    unsigned hi = __shfl_sync(kFull, (unsigned)(v >> 32), src);
    return (const uint8_t *)(((unsigned long long)hi << 32) | lo);
}

// Segment of a lookup op: the seeds (op 1) or the nodes found by hop h (op 3h+1).  Taken from
// the cumulative counts nc[9+h], which are written once per batch, so that a gather may overlap
// the sampling of the next hop on another stream.  Block 0 also leaves the (offset, size)
// snapshot that counter_update writes for a lookup op (operator_impl.cu:85-87).
__device__ __forceinline__ void segment_of(const int32_t *nc, int32_t *nc_out, int op_id, int &off, int &n, int n_rows = -1)
{
    if (n_rows >= 0) {
        off = 0;
        n = n_rows;
        return;
    }
    if (op_id == kOpGatherAll) {
        // every node of the batch in one launch (the runner's choice: one long gather instead of one
        // short one per hop); the snapshot words get the values the last per-hop lookup would leave
        const int hops = nc[LEGION_INTRABATCH_CON * 3 - 1];
        off = 0;
        n = nc[LEGION_INTRABATCH_CON * 3 + hops];
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const int last = hops > 0 ? nc[LEGION_INTRABATCH_CON * 3 + hops - 1] : 0;
            nc_out[2] = last;
            nc_out[3] = n - last;
        }
        return;
    }
    const int h = op_id / LEGION_INTRABATCH_CON;
    off = h > 0 ? nc[LEGION_INTRABATCH_CON * 3 + h - 1] : 0;
    n = nc[LEGION_INTRABATCH_CON * 3 + h] - off;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        nc_out[(op_id % LEGION_INTRABATCH_CON) * 2] = off;
        nc_out[(op_id % LEGION_INTRABATCH_CON) * 2 + 1] = n;
    }
}

// Looks one id up and resolves it to a source row.  `where`: 0 local, 1 peer, 2 host, 3 none.
// A table entry >= 0 is the global cache index; LEGION_CACHEMISS_FLAG (-2) means "row `id` of the
// host table"; an entry <= -3 means "row -(entry + 3) of the host table", for host tables that are
// not laid out in id order (legion_cache_fill_static_rows).  `host_row` is the row to fetch on a miss;
// gidx leaves as the reference's FindFeat would write it.
__device__ __forceinline__ const uint8_t *resolve(const GatherParams &p, int32_t id, int32_t &gidx, int &where,
                                                  int32_t &host_row)
{
    gidx = LEGION_CACHEMISS_FLAG;
    where = 3;
    host_row = id;
    if (id < 0 || id >= p.n_nodes) return nullptr;  // not a node: nothing is read, the output row stays as it is
    if (p.lut != nullptr) gidx = __ldg(&p.lut[id]);
    if (gidx >= 0) {
        int d = gidx / p.capacity;
        int row = gidx - d * p.capacity;
        const uint8_t *base = d <= LEGION_MAX_DEVICE ? p.part[d] : nullptr;
        if (base != nullptr) {
            where = (d == p.ki || d == p.kg) ? 0 : 1;
            return base + (int64_t)row * p.slot_bytes;
        }
        gidx = LEGION_CACHEMISS_FLAG;  // the table names a partition this call was not given: served as a miss
    }
    if (gidx <= -3) host_row = -(gidx + 3);
    gidx = LEGION_CACHEMISS_FLAG;
    if (p.host != nullptr) {
        where = 2;
        return p.host + ((int64_t)host_row % p.n_nodes) * (int64_t)p.row_bytes;
    }
    return nullptr;
}

// Rows served by the host table are not copied by the hit kernels: the warp appends them to the
// batch's miss list (one atomicAdd per warp, ranks by ballot) and clears their source pointer.
// The list holds (position in `ids`, row of the host table), so the miss kernel needs nothing else of the batch
// and may still run while the next batch on the same pipe is being sampled; it empties the list.
__device__ __forceinline__ void defer_misses(int2 *miss_rows, int32_t *miss_count, int row, int32_t id, int where,
                                             const uint8_t *&src, int lane)
{
    unsigned m = __ballot_sync(kFull, where == 2);
    if (m == 0u) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(&miss_count[0], __popc(m));
    base = __shfl_sync(kFull, base, 0);
    if (where == 2) {
        miss_rows[base + __popc(m & ((1u << lane) - 1u))] = make_int2(row, id);
        src = nullptr;
    }
}

// The same in two halves, for a kernel that wants the row copies of the chunk in flight before it needs the
// list position: the first half counts the chunk's misses, asks for their place in the list (the atomic's answer
// travels while the rows do) and clears their source pointers; the second half writes the entries.
// With `hist` an entry is also counted in its stretch of the host table and carries its number there, from which
// miss_order_kernel makes a list by rising table row.
__host__ __device__ __forceinline__ int miss_stretch(int32_t host_row, int32_t n_rows, int32_t shift)
{
    return (int)((uint32_t)(host_row < n_rows ? host_row : host_row % n_rows) >> shift);
}
struct MissTicket {
    unsigned mask;
    int base, rank;
};
__device__ __forceinline__ MissTicket miss_begin(const MissSink &m, int32_t host_row, int where, const uint8_t *&src, int lane)
{
    MissTicket t;
    t.mask = __ballot_sync(kFull, where == 2);
    t.base = t.rank = 0;
    if (t.mask != 0u && lane == 0) t.base = atomicAdd(&m.count[0], __popc(t.mask));
    if (where == 2) {
        src = nullptr;
        if (m.hist != nullptr) t.rank = atomicAdd(&m.hist[miss_stretch(host_row, m.n_rows, m.shift)], 1);
    }
    return t;
}
__device__ __forceinline__ void miss_finish(const MissSink &m, const MissTicket &t, int row, int32_t host_row, int where, int lane)
{
    if (t.mask == 0u) return;
    const int at = __shfl_sync(kFull, t.base, 0) + __popc(t.mask & ((1u << lane) - 1u));
    if (where != 2) return;
    m.rows[at] = make_int2(row, host_row);
    if (m.hist != nullptr) m.rank[at] = t.rank;
}

// Hit / miss counters of a CTA, added to the cache's counters once per CTA (three atomics on three words that
// every warp of every gather would otherwise hit).
__device__ __forceinline__ void count_where(int *cta_counts, int where, int lane)
{
    unsigned m0 = __ballot_sync(kFull, where == 0);
    unsigned m1 = __ballot_sync(kFull, where == 1);
    unsigned m2 = __ballot_sync(kFull, where == 2);
    if (lane == 0) {
        if (m0) atomicAdd(&cta_counts[0], __popc(m0));
        if (m1) atomicAdd(&cta_counts[1], __popc(m1));
        if (m2) atomicAdd(&cta_counts[2], __popc(m2));
    }
}

__device__ __forceinline__ void add_stats(unsigned long long *stats, int where, int lane)
{
    unsigned m0 = __ballot_sync(kFull, where == 0);
    unsigned m1 = __ballot_sync(kFull, where == 1);
    unsigned m2 = __ballot_sync(kFull, where == 2);
    if (stats != nullptr && lane == 0) {
        if (m0) atomicAdd(&stats[0], (unsigned long long)__popc(m0));
        if (m1) atomicAdd(&stats[1], (unsigned long long)__popc(m1));
        if (m2) atomicAdd(&stats[2], (unsigned long long)__popc(m2));
    }
}

// The two halves of resolve(), for callers that fetch the table entry of the next chunk early.
__device__ __forceinline__ int32_t lookup_raw(const GatherParams &p, int32_t id)
{
    return (id >= 0 && id < p.n_nodes && p.lut != nullptr) ? __ldg(&p.lut[id]) : LEGION_CACHEMISS_FLAG;
}
__device__ __forceinline__ const uint8_t *decode_raw(const GatherParams &p, int32_t id, int32_t raw, int32_t &gidx,
                                                     int &where, int32_t &host_row)
{
    gidx = LEGION_CACHEMISS_FLAG;
    where = 3;
    host_row = id;
    if (id < 0 || id >= p.n_nodes) return nullptr;  // not a node: nothing is read, the output row stays as it is
    if (raw >= 0) {
        int d = raw / p.capacity;
        int row = raw - d * p.capacity;
        const uint8_t *base = d <= LEGION_MAX_DEVICE ? p.part[d] : nullptr;
        if (base != nullptr) {
            gidx = raw;
            where = (d == p.ki || d == p.kg) ? 0 : 1;
            return base + (int64_t)row * p.slot_bytes;
        }
        // the table names a partition this call was not given: served as a miss
    }
    if (raw <= -3) host_row = -(raw + 3);
    if (p.host != nullptr) {
        where = 2;
        return p.host + ((int64_t)host_row % p.n_nodes) * (int64_t)p.row_bytes;
    }
    return nullptr;
}

// Rows a warp looks up and copies at a time: 32, one per lane, or fewer when the list is so short that the warps of
// the grid can hold all of it with fewer each.
__device__ __forceinline__ int rows_per_warp_for(int n, int n_warps, int least)
{
    int rpw = 32;
    while (rpw > least && (int64_t)n_warps * (rpw >> 1) >= n) rpw >>= 1;
    return rpw;
}

// Rows whose size is a multiple of 16 bytes.  VPL = 16-byte vectors per lane per row,
// R = rows copied together (R * VPL * 512 bytes in flight per warp).  A warp looks up to 32 ids up, one per
// lane, then copies their rows R at a time; while the first rows of a chunk are in flight it already
// fetches the id and the table entry of its next chunk, so that only the first lookup of a warp is
// exposed.  Long lists are bound by HBM; a list that does not give every warp 32 rows, by the chain id -> table ->
// row and the rounds behind it, so a warp then takes fewer rows, down to 4, and more SMs have some.
template <int VPL, int R>
__global__ void __launch_bounds__(256) gather_vec_kernel(GatherParams p)
{
    __shared__ int cta_counts[3];
    if (threadIdx.x < 3) cta_counts[threadIdx.x] = 0;
    __syncthreads();
    if (p.pub.o_ids != nullptr) publish_copy(p.pub);
    int off, n;
    segment_of(p.nc, p.nc_out, p.op_id, off, n, p.n_rows);
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int row_vec = p.row_bytes >> 4;
    const int rpw = p.rows_per_warp > 0 ? p.rows_per_warp : rows_per_warp_for(n, n_warps, 4);
    int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blockIdx.x * (blockDim.x >> 5) * rpw >= n) return;  // the whole CTA is past the end
    int32_t id = (lane < rpw && c * rpw + lane < n) ? __ldg(&p.ids[off + c * rpw + lane]) : -1;
    int32_t raw = lookup_raw(p, id);
    for (; c * rpw < n; c += n_warps) {
        const int r = c * rpw + lane;
        int32_t gidx, host_row;
        int where;
        const uint8_t *src = decode_raw(p, id, raw, gidx, where, host_row);
        if (lane < rpw && r < n) p.cache_index[off + r] = gidx;
        use_staged(p, off + r, where, src);
        if (p.stats != nullptr) count_where(cta_counts, where, lane);
        const MissTicket ticket = miss_begin(p.miss, host_row, where, src, lane);
        const int rows_here = min(rpw, n - c * rpw);
        uint8_t *dst_base = p.dst + (int64_t)(off + c * rpw) * p.row_bytes;
        const int rn = (c + n_warps) * rpw + lane;
        id = (lane < rpw && rn < n) ? __ldg(&p.ids[off + rn]) : -1;
        for (int j0 = 0; j0 < rows_here; j0 += R) {
            uint4 v[R][VPL];
            const uint8_t *sp[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                sp[jj] = shfl_ptr(src, (j0 + jj) & 31);
                if (j0 + jj >= rows_here) sp[jj] = nullptr;
            }
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
#pragma unroll
                for (int q = 0; q < VPL; ++q) {
                    int idx = lane + 32 * q;
                    if (sp[jj] != nullptr && idx < row_vec)
                        v[jj][q] = *reinterpret_cast<const uint4 *>(sp[jj] + idx * 16);
                }
            }
            if (j0 == 0) raw = lookup_raw(p, id);
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
#pragma unroll
                for (int q = 0; q < VPL; ++q) {
                    int idx = lane + 32 * q;
                    if (sp[jj] != nullptr && idx < row_vec)
                        __stcs(reinterpret_cast<uint4 *>(dst_base + (int64_t)(j0 + jj) * p.row_bytes + idx * 16),
                               v[jj][q]);
                }
            }
        }
        miss_finish(p.miss, ticket, off + r, host_row, where, lane);
    }
    __syncthreads();
    if (p.stats != nullptr && threadIdx.x < 3 && cta_counts[threadIdx.x] != 0)
        atomicAdd(&p.stats[threadIdx.x], (unsigned long long)cta_counts[threadIdx.x]);
}

// ---- the same gather with the copy engine of the SM (bulk asynchronous copies) -----------------------
//
// A warp looks 32 ids up, one per lane, as above; then every lane whose row is held in GPU memory issues
// ONE bulk copy global -> shared for its whole row (cp.async.bulk, completion counted in bytes on the
// warp's mbarrier), the warp waits for the barrier, and every lane issues ONE bulk copy shared -> global
// into the output row.  No row data passes through registers, so a warp keeps 32 rows (16 KB for
// 512-byte rows) in flight with a handful of registers, and three CTAs of four warps hold 192 KB of
// reads in flight per SM.  Rows, shared-memory slots and output rows are 16-byte aligned and a multiple
// of 16 bytes long, which is all that the untiled bulk copy asks for; no multicast, no tensor map.
// Every wait is bounded: on a timeout the warp raises DERR_BULK_TIMEOUT, waits once more (again bounded) for
// the copies it issued and leaves.  After that error the pipe's output rows are invalid and the caller must
// stop issuing work on this context (legion_pool_device_error reports it): a copy that is still on its way
// when the CTA retires would land in shared memory that no longer belongs to it.
constexpr int kBulkWarps = 4;
constexpr int kBulkWaitLimit = 1 << 20;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (int spin = 0; spin < kBulkWaitLimit; ++spin) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

__global__ void __launch_bounds__(kBulkWarps * 32) gather_bulk_kernel(GatherParams p)
{
    extern __shared__ __align__(128) uint8_t bulk_smem[];          // [warp][32 rows][row_bytes]
    __shared__ __align__(8) unsigned long long bars[kBulkWarps];
    int off, n;
    segment_of(p.nc, p.nc_out, p.op_id, off, n);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t row_bytes = (uint32_t)p.row_bytes;
    uint8_t *my_rows = bulk_smem + (size_t)warp * 32 * row_bytes;
    const uint32_t my_slot = smem_addr(my_rows + (size_t)lane * row_bytes);
    const uint32_t bar = smem_addr(&bars[warp]);
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    uint32_t parity = 0;
    bool store_pending = false;
    int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c * 32 < n) {
        int32_t id = (c * 32 + lane < n) ? __ldg(&p.ids[off + c * 32 + lane]) : -1;
        int32_t raw = lookup_raw(p, id);
        for (; c * 32 < n; c += n_warps) {
            const int r = c * 32 + lane;
            int32_t gidx, host_row;
            int where;
            const uint8_t *src = decode_raw(p, id, raw, gidx, where, host_row);
            if (r < n) p.cache_index[off + r] = gidx;
            add_stats(p.stats, where, lane);
            defer_misses(p.miss.rows, p.miss.count, off + r, host_row, where, src, lane);
            const int rn = (c + n_warps) * 32 + lane;
            id = (rn < n) ? __ldg(&p.ids[off + rn]) : -1;
            const unsigned hits = __ballot_sync(kFull, src != nullptr);
            // the previous chunk's stores must have read their rows out of shared memory
            if (store_pending) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            if (hits != 0u) {
                if (lane == 0) {
                    const uint32_t tx = (uint32_t)__popc(hits) * row_bytes;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(tx) : "memory");
                }
                __syncwarp();
                if (src != nullptr)
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                        :: "r"(my_slot), "l"(src), "r"(row_bytes), "r"(bar) : "memory");
            }
            raw = lookup_raw(p, id);  // the next chunk's table entries travel while the rows do
            if (hits != 0u) {
                const bool done = mbar_wait(bar, parity);
                parity ^= 1u;
                if (!__all_sync(kFull, done)) {
                    if (lane == 0 && p.err != nullptr) atomicCAS(p.err, DERR_NONE, DERR_BULK_TIMEOUT);
                    mbar_wait(bar, parity ^ 1u);  // one more bounded wait for the copies that are still on their way
                    break;
                }
                if (src != nullptr) {
                    uint8_t *dst = p.dst + (int64_t)(off + r) * p.row_bytes;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                 :: "l"(dst), "r"(my_slot), "r"(row_bytes) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    store_pending = true;
                }
            }
        }
    }
    // nothing of this CTA may still be in flight when its shared memory is given back
    if (store_pending) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Rows that are not whole 16-byte vectors (rows of F floats with F odd, ...) or longer than 2048 bytes.  T = the
// widest of 16, 8 and 4 bytes that divides the row.  The rows of a warp are consecutive in the output, so they are
// copied as one flat run of T's: lane l takes elements l, l + 32, ... of the run, whatever row they fall into, U of
// them in flight.  Bound by HBM when the rows are many; when they are few (a list that does not give every warp
// 32 rows), by the chain id -> table -> row, so a warp then takes fewer rows, down to 4.
// Measured, 75 floats a row, against one row after the other per warp with one load in flight: a batch of 1,237
// seeds and fanout [15,10] through the operators (28 k rows in three gathers) 275 -> 152 us.
template <typename T, int U>
__global__ void __launch_bounds__(256) gather_flat_kernel(GatherParams p)
{
    __shared__ const uint8_t *s_src[8][32];
    __shared__ int cta_counts[3];
    if (threadIdx.x < 3) cta_counts[threadIdx.x] = 0;
    __syncthreads();
    if (p.pub.o_ids != nullptr) publish_copy(p.pub);
    int off, n;
    segment_of(p.nc, p.nc_out, p.op_id, off, n, p.n_rows);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int rpw = rows_per_warp_for(n, n_warps, 4);
    const int per_row = p.row_bytes / (int)sizeof(T);
    const int row0 = lane / per_row, col0 = lane - row0 * per_row;   // where the lane's first element falls
    const int d_row = 32 / per_row, d_col = 32 - d_row * per_row;    // and how far 32 elements on
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * rpw < n; c += n_warps) {
        const int r = c * rpw + lane;
        const bool mine = lane < rpw && r < n;
        const int32_t id = mine ? __ldg(&p.ids[off + r]) : -1;
        int32_t gidx, host_row;
        int where;
        const uint8_t *src = resolve(p, id, gidx, where, host_row);
        if (mine) p.cache_index[off + r] = gidx;
        use_staged(p, off + r, where, src);
        if (p.stats != nullptr) count_where(cta_counts, where, lane);
        const MissTicket ticket = miss_begin(p.miss, host_row, where, src, lane);
        s_src[warp][lane] = src;
        __syncwarp();
        const int total = min(rpw, n - c * rpw) * per_row;
        T *dst = reinterpret_cast<T *>(p.dst + (int64_t)(off + c * rpw) * p.row_bytes);
        int row = row0, col = col0;
        for (int i0 = lane; i0 < total; i0 += 32 * U) {
            T v[U];
            bool ok[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ok[u] = false;
                if (i0 + 32 * u < total) {
                    const uint8_t *sp = s_src[warp][row];
                    ok[u] = sp != nullptr;
                    if (ok[u]) v[u] = reinterpret_cast<const T *>(sp)[col];
                }
                row += d_row;
                col += d_col;
                if (col >= per_row) {
                    col -= per_row;
                    ++row;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (ok[u]) __stcs(&dst[i0 + 32 * u], v[u]);
        }
        miss_finish(p.miss, ticket, off + r, host_row, where, lane);
        __syncwarp();
    }
    __syncthreads();
    if (p.stats != nullptr && threadIdx.x < 3 && cta_counts[threadIdx.x] != 0)
        atomicAdd(&p.stats[threadIdx.x], (unsigned long long)cta_counts[threadIdx.x]);
}

// Compressed cache: a hit row holds feature_len one-byte codes followed by an fp32 scale
// and is expanded to fp32 here; a miss row is a plain fp32 row of the host table.
// x^ = float(code) * scale, one multiplication, so the host replay is exact.
template <int CODEC>
__device__ __forceinline__ float decode_code(uint8_t b)
{
    if (CODEC == LEGION_CODEC_INT8) return (float)(int8_t)b;
    __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, __NV_E4M3);
    return __half2float(__half(h));
}

template <int CODEC>
__device__ __forceinline__ float4 decode_word(uint32_t packed, float scale)
{
    return make_float4(__fmul_rn(decode_code<CODEC>((uint8_t)(packed)), scale), __fmul_rn(decode_code<CODEC>((uint8_t)(packed >> 8)), scale),
                       __fmul_rn(decode_code<CODEC>((uint8_t)(packed >> 16)), scale), __fmul_rn(decode_code<CODEC>((uint8_t)(packed >> 24)), scale));
}

// The same shape as gather_vec_kernel: a lane looks one id up and fetches that row's scale, the warp copies R rows
// together, V words (128 V codes) of each per lane and step.  Bound by HBM (the fp32 rows written are four fifths of
// the bytes).  Eight words in flight per lane and, over all nodes of a batch, two CTAs per SM: 16 words and eight CTAs took
// the registers of the sampling kernels beside it (four batches of 800 seeds, 100 codes a row: 268 us against 234; one
// row after the other for rows of more than 128 codes was the alternative).
template <int CODEC, int V, int R>
__global__ void __launch_bounds__(256) gather_quant_kernel(GatherParams p)
{
    __shared__ int cta_counts[3];
    if (threadIdx.x < 3) cta_counts[threadIdx.x] = 0;
    __syncthreads();
    if (p.pub.o_ids != nullptr) publish_copy(p.pub);
    int off, n;
    segment_of(p.nc, p.nc_out, p.op_id, off, n);
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int f = p.feature_len, groups = f >> 2;
    const int rpw = rows_per_warp_for(n, n_warps, 8);
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * rpw < n; c += n_warps) {
        const int r = c * rpw + lane;
        const bool mine = lane < rpw && r < n;
        const int32_t id = mine ? __ldg(&p.ids[off + r]) : -1;
        int32_t gidx, host_row;
        int where;
        const uint8_t *src = resolve(p, id, gidx, where, host_row);
        if (mine) p.cache_index[off + r] = gidx;
        if (p.stats != nullptr) count_where(cta_counts, where, lane);
        const MissTicket ticket = miss_begin(p.miss, host_row, where, src, lane);
        const float my_scale = src != nullptr ? *reinterpret_cast<const float *>(src + f) : 0.0f;  // f is a multiple of 4
        const int rows_here = min(rpw, n - c * rpw);
        float *dst_base = reinterpret_cast<float *>(p.dst + (int64_t)(off + c * rpw) * p.row_bytes);
        for (int j0 = 0; j0 < rows_here; j0 += R) {
            const uint8_t *sp[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                sp[jj] = shfl_ptr(src, (j0 + jj) & 31);   // nullptr: invalid id, or a miss left to the miss kernel
                if (j0 + jj >= rows_here) sp[jj] = nullptr;
            }
            for (int g0 = 0; g0 < groups; g0 += 32 * V) {
                uint32_t packed[R][V];
#pragma unroll
                for (int jj = 0; jj < R; ++jj) {
#pragma unroll
                    for (int q = 0; q < V; ++q) {
                        const int g = g0 + lane + 32 * q;
                        if (sp[jj] != nullptr && g < groups) packed[jj][q] = *reinterpret_cast<const uint32_t *>(sp[jj] + g * 4);
                    }
                }
#pragma unroll
                for (int jj = 0; jj < R; ++jj) {
                    const float scale = __shfl_sync(kFull, my_scale, (j0 + jj) & 31);
#pragma unroll
                    for (int q = 0; q < V; ++q) {
                        const int g = g0 + lane + 32 * q;
                        if (sp[jj] != nullptr && g < groups)
                            __stcs(reinterpret_cast<float4 *>(dst_base + (int64_t)(j0 + jj) * f) + g, decode_word<CODEC>(packed[jj][q], scale));
                    }
                }
            }
        }
        miss_finish(p.miss, ticket, off + r, host_row, where, lane);
    }
    __syncthreads();
    if (p.stats != nullptr && threadIdx.x < 3 && cta_counts[threadIdx.x] != 0)
        atomicAdd(&p.stats[threadIdx.x], (unsigned long long)cta_counts[threadIdx.x]);
}

// Rows that miss the cache: one warp copies `R` rows of the miss list at a time from the pinned host
// table by zero-copy loads (16 bytes per lane, so a 512-byte row is four 128-byte reads on the
// host link).  Runs on its own stream with a grid of its own so that the link has thousands of
// reads in flight while the HBM-bound kernels of the next batch carry on.  The last CTA empties the
// list.  Measured alone on random 512-byte rows: 50.6 GB/s over a 1 GB table (0.91 of a pinned
// cudaMemcpy), 26 GB/s over 48 GB, where address translation of the scattered pages limits the link.
constexpr int kMissCtas = 148;     // CTAs of the host-link fetch (see launch_gather_misses)
constexpr int kMissThreads = 256;

struct MissParams {
    const int2 *miss_rows;
    int32_t *miss_count;
    int32_t *ticket;
    const uint8_t *host;
    int64_t n_nodes;
    uint8_t *dst;
    int32_t row_bytes;
    int32_t host_row_bytes;  // bytes of one row of the host table (compressed host tables: codes + scale, padded)
    int32_t *hist;           // counts of stretches to be zeroed for the next batch, or nullptr
};

// The miss list by rising table row, up to the order inside a stretch: place of an entry = entries of the stretches
// before its own + its number there.  Every CTA adds up all the counts for itself.
// Why: the host link's translations are shared by rows that lie close together and are asked for together.  Measured
// over a 4 GB table, 512-byte rows: 80,000 random rows 36.0 GB/s, sorted 47.6, by 4096 stretches 46.7, by 256 38.7;
// 20,000 rows 31.2, sorted 37.0, by 4096 stretches 36.8.
__global__ void __launch_bounds__(1024)
miss_order_kernel(const int2 *__restrict__ list, const int32_t *__restrict__ rank, const int32_t *__restrict__ count,
                  const int32_t *__restrict__ hist, int32_t shift, int32_t n_rows, int2 *out)
{
    static_assert(kMissStretches == 4096, "four counts per thread");
    __shared__ int32_t before[kMissStretches];
    __shared__ int32_t warp_sum[32];
    const int n = count[0];
    if ((int)(blockIdx.x * blockDim.x) >= n) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 h = reinterpret_cast<const int4 *>(hist)[threadIdx.x];
    const int mine = h.x + h.y + h.z + h.w;
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int at = incl - mine + __reduce_add_sync(kFull, lane < warp ? warp_sum[lane] : 0);
    int4 b;
    b.x = at; b.y = b.x + h.x; b.z = b.y + h.y; b.w = b.z + h.z;
    reinterpret_cast<int4 *>(before)[threadIdx.x] = b;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int2 e = list[i];
        out[before[miss_stretch(e.y, n_rows, shift)] + rank[i]] = e;
    }
}

// The list is complete and consumed: the last CTA to finish empties it for the next batch.
__device__ __forceinline__ void miss_list_done(const MissParams &p, int *s_last)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = atomicAdd(p.ticket, 1);
        *s_last = (t == (int)gridDim.x - 1);
    }
    __syncthreads();
    if (*s_last && threadIdx.x == 0) {
        p.miss_count[0] = 0;
        *p.ticket = 0;
    }
}

__device__ __forceinline__ void miss_zero_hist(const MissParams &p)
{
    if (p.hist != nullptr && blockIdx.x == 0)
        for (int t = threadIdx.x; t < kMissStretches; t += blockDim.x) p.hist[t] = 0;
}

// Host table stored as compressed rows (feature_len one-byte codes + fp32 scale): the fetch moves
// host_row_bytes per row over the host link instead of 4 * feature_len and decodes into the fp32 output row.
// Bound by the requests that the link takes (~380 a microsecond, whatever their size up to 128 bytes): NARROW rows (at most
// 32 vectors) are read by one 16-byte load per lane, scale included, which is as few requests as the row has 128-byte
// lines, and the words change lanes on the way to the output row; longer rows load the scale on its own.  Measured,
// 13,150 rows of 144 bytes: 110 -> 75 us, a batch of 8000 seeds 110 -> 81 us.
template <int CODEC, int R, bool NARROW>
__global__ void __launch_bounds__(1024) gather_miss_quant_kernel(MissParams p)
{
    __shared__ int s_last;
    miss_zero_hist(p);
    const int n = p.miss_count[0];
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int2 *list = p.miss_rows;
    const int f = p.row_bytes >> 2;
    const int groups = f >> 2;
    for (int m0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * R; m0 < n; m0 += n_warps * R) {
        const uint8_t *sp[R];
        float *dp[R];
#pragma unroll
        for (int jj = 0; jj < R; ++jj) {
            sp[jj] = nullptr;
            dp[jj] = nullptr;
            if (m0 + jj < n) {
                const int2 e = __ldg(&list[m0 + jj]);
                sp[jj] = p.host + ((int64_t)e.y % p.n_nodes) * (int64_t)p.host_row_bytes;
                dp[jj] = reinterpret_cast<float *>(p.dst + (int64_t)e.x * p.row_bytes);
            }
        }
        if constexpr (NARROW) {
            uint4 x[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj)
                x[jj] = sp[jj] != nullptr && lane * 16 < p.host_row_bytes ? *(reinterpret_cast<const uint4 *>(sp[jj]) + lane)
                                                                          : make_uint4(0u, 0u, 0u, 0u);
            // word g of a row is component g & 3 of lane g >> 2; the scale is word `groups`
            auto word = [&](const uint4 &v, int g) {
                const uint32_t a = __shfl_sync(kFull, v.x, g >> 2), b = __shfl_sync(kFull, v.y, g >> 2);
                const uint32_t c = __shfl_sync(kFull, v.z, g >> 2), d = __shfl_sync(kFull, v.w, g >> 2);
                return (g & 2) ? ((g & 1) ? d : c) : ((g & 1) ? b : a);
            };
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                const float scale = __uint_as_float(word(x[jj], groups));
                for (int g0 = 0; g0 < groups; g0 += 32) {
                    const int g = g0 + lane;
                    const uint32_t packed = word(x[jj], g < groups ? g : groups);
                    if (sp[jj] != nullptr && g < groups) __stcs(reinterpret_cast<float4 *>(dp[jj]) + g, decode_word<CODEC>(packed, scale));
                }
            }
        } else {
            float scale[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj)
                if (sp[jj] != nullptr) scale[jj] = *reinterpret_cast<const float *>(sp[jj] + f);
            for (int g0 = 0; g0 < groups; g0 += 32) {
                const int g = g0 + lane;
                uint32_t packed[R];
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr && g < groups) packed[jj] = *reinterpret_cast<const uint32_t *>(sp[jj] + g * 4);
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr && g < groups) __stcs(reinterpret_cast<float4 *>(dp[jj]) + g, decode_word<CODEC>(packed[jj], scale[jj]));
            }
        }
    }
    miss_list_done(p, &s_last);
}

template <int R>
__global__ void __launch_bounds__(1024) gather_miss_kernel(MissParams p)
{
    __shared__ int s_last;
    miss_zero_hist(p);
    const int n = p.miss_count[0];
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int2 *list = p.miss_rows;
    if ((p.row_bytes & 15) == 0) {
        const int row_vec = p.row_bytes >> 4;
        for (int m0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * R; m0 < n; m0 += n_warps * R) {
            const uint8_t *sp[R];
            uint8_t *dp[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                sp[jj] = nullptr;
                dp[jj] = nullptr;
                if (m0 + jj < n) {
                    const int2 e = __ldg(&list[m0 + jj]);
                    sp[jj] = p.host + ((int64_t)e.y % p.n_nodes) * (int64_t)p.row_bytes;
                    dp[jj] = p.dst + (int64_t)e.x * p.row_bytes;
                }
            }
            for (int q0 = 0; q0 < row_vec; q0 += 32) {
                uint4 v[R];
                const int idx = q0 + lane;
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr && idx < row_vec) v[jj] = *reinterpret_cast<const uint4 *>(sp[jj] + idx * 16);
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr && idx < row_vec) __stcs(reinterpret_cast<uint4 *>(dp[jj] + idx * 16), v[jj]);
            }
        }
    } else {
        const int row_words = p.row_bytes >> 2;
        for (int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < n; m += n_warps) {
            const int2 e = __ldg(&list[m]);
            const uint32_t *sp = reinterpret_cast<const uint32_t *>(p.host + ((int64_t)e.y % p.n_nodes) * (int64_t)p.row_bytes);
            uint32_t *dp = reinterpret_cast<uint32_t *>(p.dst + (int64_t)e.x * p.row_bytes);
            for (int w = lane; w < row_words; w += 32) __stcs(&dp[w], sp[w]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = atomicAdd(p.ticket, 1);
        s_last = (t == (int)gridDim.x - 1);
        if (s_last) {  // every CTA has read its count by now
            p.miss_count[0] = 0;
            *p.ticket = 0;
        }
    }
}

// ---- set-associative LRU cache ----------------------------------------------------------------------
// Lookup ("retrieve_and_touch"): a hit stamps the way with the batch clock.  Addressing: set = id % sets (one GPU),
// slot = set * ways + way.
struct LruParams {
    const int32_t *ids;
    int32_t *nc;
    int32_t op_id;
    int32_t *keys, *stamps;
    int64_t sets;
    int32_t ways;
    const BatchCtl *bctl;  // clock of the batch
    const uint8_t *rows;
    const uint8_t *host;
    int64_t n_nodes;
    uint8_t *dst;
    int64_t *cache_index;
    unsigned long long *stats;
    int32_t row_bytes;
    MissSink miss;
};

__device__ __forceinline__ int64_t lru_set(int32_t id, int64_t sets)
{
    return sets <= 0x7FFFFFFF ? (int64_t)((uint32_t)id % (uint32_t)sets) : (int64_t)id;  // an id is below 2^31
}

// Way of the set that holds `id`, or -1.  A lane probes the set of its own id: 8 ways are one 32-byte sector, read as
// two vectors, so that a warp has the keys of 32 ids under way at once.
__device__ __forceinline__ int lru_probe(const int32_t *set_keys, int ways, int32_t id)
{
    int hit = -1;
    if (ways >= 8) {
        for (int w0 = 0; w0 < ways; w0 += 8) {
            const int4 a = __ldcg(reinterpret_cast<const int4 *>(set_keys + w0)), b = __ldcg(reinterpret_cast<const int4 *>(set_keys + w0) + 1);
            const int32_t k[8] = { a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w };
#pragma unroll
            for (int w = 0; w < 8; ++w)
                if (k[w] == id && hit < 0) hit = w0 + w;
        }
        return hit;
    }
    for (int w = ways - 1; w >= 0; --w)
        if (__ldcg(&set_keys[w]) == id) hit = w;
    return hit;
}

// Bound by HBM for the rows; the probe used to be 8 dependent rounds of key loads per 32 ids.  Together with the insertion
// below: 1.9 x 10^5 rows of 512 bytes, 8 ways, 58% hits, 4.6 x 10^4 insertions, 1.19 -> 1.06 ms a batch, of which 1.0 ms are
// the fetch of the missed rows.
template <int VPL, int R>
__global__ void __launch_bounds__(256) gather_lru_kernel(LruParams p)
{
    __shared__ int cta_counts[3];
    if (threadIdx.x < 3) cta_counts[threadIdx.x] = 0;
    __syncthreads();
    int off, n;
    segment_of(p.nc, p.nc, p.op_id, off, n);
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int row_vec = p.row_bytes >> 4;
    const int clock = p.bctl->clock;
    const int rpw = rows_per_warp_for(n, n_warps, 8);
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * rpw < n; c += n_warps) {
        const int r = c * rpw + lane;
        const bool mine = lane < rpw && r < n;
        const int32_t id = mine ? __ldg(&p.ids[off + r]) : -1;
        int where = 3;
        const uint8_t *src = nullptr;
        int64_t slot = -1;
        if (id >= 0) {
            const int64_t first = lru_set(id, p.sets) * p.ways;
            const int way = lru_probe(p.keys + first, p.ways, id);
            if (way >= 0) {
                slot = first + way;
                p.stamps[slot] = clock;
                where = 0;
                src = p.rows + slot * (int64_t)p.row_bytes;
            } else if (p.host != nullptr) {
                where = 2;
                src = p.host + ((int64_t)id % p.n_nodes) * (int64_t)p.row_bytes;
            }
        }
        if (mine) p.cache_index[off + r] = slot;
        if (p.stats != nullptr) count_where(cta_counts, where, lane);
        const MissTicket ticket = miss_begin(p.miss, id, where, src, lane);
        const int rows_here = min(rpw, n - c * rpw);
        uint8_t *dst_base = p.dst + (int64_t)(off + c * rpw) * p.row_bytes;
        for (int j0 = 0; j0 < rows_here; j0 += R) {
            uint4 v[R][VPL];
            const uint8_t *sp[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                sp[jj] = shfl_ptr(src, (j0 + jj) & 31);
                if (j0 + jj >= rows_here) sp[jj] = nullptr;
            }
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
#pragma unroll
                for (int q = 0; q < VPL; ++q) {
                    int idx = lane + 32 * q;
                    if (sp[jj] != nullptr && idx < row_vec)
                        v[jj][q] = *reinterpret_cast<const uint4 *>(sp[jj] + idx * 16);
                }
            }
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
#pragma unroll
                for (int q = 0; q < VPL; ++q) {
                    int idx = lane + 32 * q;
                    if (sp[jj] != nullptr && idx < row_vec)
                        __stcs(reinterpret_cast<uint4 *>(dst_base + (int64_t)(j0 + jj) * p.row_bytes + idx * 16),
                               v[jj][q]);
                }
            }
        }
        miss_finish(p.miss, ticket, off + r, id, where, lane);
    }
    __syncthreads();
    if (p.stats != nullptr && threadIdx.x < 3 && cta_counts[threadIdx.x] != 0)
        atomicAdd(&p.stats[threadIdx.x], (unsigned long long)cta_counts[threadIdx.x]);
}

// Insertion phase, run once per batch after every gather (two launches):
//  claim : every missed id picks the way of its set with the smallest stamp (empty ways count
//          as -1, ways stamped in this batch are excluded, lowest way on ties) and bids for it
//          with its position in the id list (atomicMin);
//  commit: the lowest bidder writes key and stamp, copies its row from the batch's feature
//          buffer (already gathered) into the slot and takes its bid back for the next batch.
__global__ void lru_claim_kernel(const int32_t *__restrict__ ids, const int64_t *__restrict__ cache_index,
                                 const int32_t *__restrict__ nc, const int32_t *__restrict__ keys,
                                 const int32_t *__restrict__ stamps, int64_t sets, int ways,
                                 const BatchCtl *__restrict__ bctl, unsigned long long *claim,
                                 int64_t *victim /* per row: chosen slot or -1 */)
{
    const int clock = bctl->clock;
    const int n = nc[LEGION_INTRABATCH_CON * 3 + nc[LEGION_INTRABATCH_CON * 3 - 1]];  // all nodes of the batch
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int64_t v = -1;
        const int32_t id = ids[r];
        if (id >= 0 && cache_index[r] < 0) {
            const int64_t first = lru_set(id, sets) * ways;
            int best = -1, best_stamp = 0;
            auto offer = [&](int w, int32_t key, int32_t stamp) {
                const int32_t st = key == -1 ? -1 : stamp;
                if (st != clock && (best < 0 || st < best_stamp)) { best = w; best_stamp = st; }
            };
            if (ways >= 4) {
                for (int w = 0; w < ways; w += 4) {
                    const int4 k = *reinterpret_cast<const int4 *>(keys + first + w), t = *reinterpret_cast<const int4 *>(stamps + first + w);
                    offer(w, k.x, t.x); offer(w + 1, k.y, t.y); offer(w + 2, k.z, t.z); offer(w + 3, k.w, t.w);
                }
            } else {
                for (int w = 0; w < ways; ++w) offer(w, keys[first + w], stamps[first + w]);
            }
            if (best >= 0) {
                v = first + best;
                atomicMin(&claim[v], (unsigned long long)r);
            }
        }
        victim[r] = v;
    }
}

// A warp reads the choices and the bids of up to 32 rows at once and then copies the rows that won, four at a time.
// Bound by HBM: 2 * row_bytes per insertion and 8 (misses: 16) bytes per row.  (One row after the other per warp, each
// behind its choice and its bid, took 92 us for 1.9 x 10^5 rows and 4.6 x 10^4 insertions.)
__global__ void __launch_bounds__(256)
lru_commit_kernel(const int32_t *__restrict__ ids, const int32_t *__restrict__ nc, int32_t *keys,
                  int32_t *stamps, const BatchCtl *__restrict__ bctl, unsigned long long *claim,
                  const int64_t *__restrict__ victim, const uint8_t *__restrict__ features,
                  uint8_t *rows, int row_bytes, unsigned long long *stats)
{
    constexpr int R = 4;
    __shared__ int cta_inserts;
    if (threadIdx.x == 0) cta_inserts = 0;
    __syncthreads();
    const int clock = bctl->clock;
    const int n = nc[LEGION_INTRABATCH_CON * 3 + nc[LEGION_INTRABATCH_CON * 3 - 1]];  // all nodes of the batch
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int row_vec = row_bytes >> 4;
    const int rpw = rows_per_warp_for(n, n_warps, 8);
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * rpw < n; c += n_warps) {
        const int r = c * rpw + lane;
        int64_t v = lane < rpw && r < n ? victim[r] : -1;
        // a lower position may have won the way (and may have taken its bid back already)
        if (v >= 0 && __ldcg(&claim[v]) != (unsigned long long)r) v = -1;
        if (v >= 0) {
            claim[v] = ~0ull;
            keys[v] = ids[r];
            stamps[v] = clock;
        }
        unsigned won = __ballot_sync(kFull, v >= 0);
        if (lane == 0 && won != 0u) atomicAdd(&cta_inserts, __popc(won));
        while (won != 0u) {
            const uint4 *sp[R];
            uint4 *dp[R];
#pragma unroll
            for (int jj = 0; jj < R; ++jj) {
                const int j = won != 0u ? __ffs(won) - 1 : -1;
                won &= won - 1u;
                const int64_t slot = __shfl_sync(kFull, (long long)v, j & 31);
                sp[jj] = j >= 0 ? reinterpret_cast<const uint4 *>(features + (int64_t)(c * rpw + j) * row_bytes) : nullptr;
                dp[jj] = reinterpret_cast<uint4 *>(rows + slot * (int64_t)row_bytes);
            }
            for (int q = lane; q < row_vec; q += 32) {
                uint4 x[R];
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr) x[jj] = sp[jj][q];
#pragma unroll
                for (int jj = 0; jj < R; ++jj)
                    if (sp[jj] != nullptr) dp[jj][q] = x[jj];
            }
        }
    }
    __syncthreads();
    if (stats != nullptr && threadIdx.x == 0 && cta_inserts != 0) atomicAdd(&stats[3], (unsigned long long)cta_inserts);
}

// ---- launchers ------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(256) publish_kernel(Publish p) { publish_copy(p); }

template <int VPL, int R>
static void launch_vec(int grid, cudaStream_t s, const GatherParams &gp)
{
    gather_vec_kernel<VPL, R><<<grid, 256, 0, s>>>(gp);
}
// Widest element that divides the row and to which every row of the caches, the staging area and the output is aligned.
static void launch_flat(int grid, cudaStream_t s, const GatherParams &gp)
{
    uintptr_t a = (uintptr_t)gp.dst | (uintptr_t)gp.stage_rows | (uintptr_t)(uint32_t)gp.row_bytes;
    for (int k = 0; k <= LEGION_MAX_DEVICE; ++k) a |= (uintptr_t)gp.part[k];
    if ((a & 15) == 0) gather_flat_kernel<uint4, 4><<<grid, 256, 0, s>>>(gp);
    else if ((a & 7) == 0) gather_flat_kernel<uint2, 8><<<grid, 256, 0, s>>>(gp);
    else gather_flat_kernel<uint32_t, 8><<<grid, 256, 0, s>>>(gp);
}
template <int VPL, int R>
static void launch_lru(int grid, cudaStream_t s, const LruParams &lp)
{
    gather_lru_kernel<VPL, R><<<grid, 256, 0, s>>>(lp);
}

// 0: loads and stores through registers; 1: bulk asynchronous copies through shared memory.  The
// environment variable LEGION_GATHER_ENGINE sets the start value (legion_set_tunable overrides it).
static int gather_engine_from_env()
{
    const char *v = getenv("LEGION_GATHER_ENGINE");
    return (v != nullptr && v[0] == '1' && v[1] == 0) ? 1 : 0;
}
int g_gather_engine = gather_engine_from_env();
int g_gather_cps = 0;  // CTAs per SM of the hit gathers (0 = default); see legion_set_tunable
int g_gather_rows = 0; // rows in flight per warp for 512-byte-class rows (0 = default)

int g_gather_rpw = 0;  // rows per warp and chunk of the 512-byte-class gather (0 = default); see legion_set_tunable

// CTAs for the worst-case rows of this segment (the seeds, the new nodes of hop (op_id / 3), or all nodes) at
// `least` rows per warp, at most `cps` per SM.
static int segment_grid(const LegionPool *p, int32_t op_id, int64_t *rows_out, int least, int cps)
{
    int hop = op_id / LEGION_INTRABATCH_CON;  // 0 = seeds
    int64_t rows = p->batch_size;
    int64_t nodes = p->batch_size;
    for (int h = 0; h < hop; ++h) { rows = nodes * p->fanout[h]; nodes += rows; }
    if (op_id == kOpGatherAll) rows = p->max_nodes;
    if (rows_out) *rows_out = rows;
    int64_t chunks = (rows + least - 1) / least;
    int64_t g64 = (chunks + 7) / 8;
    int64_t cap = (int64_t)p->sm_count * (g_gather_cps > 0 ? g_gather_cps : cps);
    return (int)(g64 < 1 ? 1 : (g64 > cap ? cap : g64));
}

// Rows that a gather may list at worst from which on its list is fetched by rising table row.  What a batch lists is a
// thirtieth of its worst case, and launch and gain balance at about 2,500 rows.  Measured, us a batch with ordering against
// without, two pipes: 123 rows listed of at most 2,112: 31.4 against 28.3; 728 of 67,584: 45.7, 45.2; 2,379: 61.2, 61.1;
// 7,694 of 264,000: 122.0, 125.0; 10,465: 151.4, 155.9; 68,030: 755, 771.  Through the operators, which list and fetch op by
// op: 608 of at most 14,080 in the longest: 96.6 against 85.1.
constexpr int64_t kOrderedFrom = 1 << 14;

// Rows of a stretch of the table, as a power of two.
static int stretch_shift(int32_t n_rows)
{
    int shift = 0;
    while (((n_rows - 1) >> shift) >= kMissStretches) ++shift;
    return shift;
}

// List of the pipe's misses.  By stretches (miss_order_kernel in front of the fetch) where it can be long, `most` rows, and
// scattered: behind an LRU cache it is up to tens of thousands of rows over the whole table.
static MissSink miss_sink(LegionPool *p, const LegionCache *c, int64_t most)
{
    const int pipe = p->pipe;
    MissSink m;
    m.rows = p->miss_rows[pipe];
    m.count = p->miss_count[pipe];
    const bool by_stretch = c != nullptr && c->host_table != nullptr && c->kind == 1 && most >= kOrderedFrom;
    m.n_rows = c != nullptr ? (int32_t)c->n_nodes : 1;
    m.shift = stretch_shift(m.n_rows);
    m.hist = by_stretch ? p->miss_hist[pipe] : nullptr;
    m.rank = by_stretch ? p->miss_rank[pipe] : nullptr;
    p->miss_ordered[pipe] = by_stretch ? 1 : 0;
    return m;
}

template <int CODEC>
static void launch_quant(int grid, cudaStream_t s, const GatherParams &gp)
{
    if (gp.feature_len <= 128) gather_quant_kernel<CODEC, 1, 8><<<grid, 256, 0, s>>>(gp);
    else if (gp.feature_len <= 256) gather_quant_kernel<CODEC, 2, 8><<<grid, 256, 0, s>>>(gp);
    else gather_quant_kernel<CODEC, 4, 4><<<grid, 256, 0, s>>>(gp);
}

// Lookup + gather of every row that is served from GPU memory; rows served by the host table
// are listed for launch_gather_misses.
int launch_gather_hits(cudaStream_t s, LegionPool *p, LegionCache *c, int32_t op_id)
{
    const int pipe = p->pipe;
    int64_t most = 0;
    const int grid = segment_grid(p, op_id, &most, 32, 8);
    const int row_bytes = p->row_bytes_out;

    if (c != nullptr && c->kind == 1) {
        LG_ARG(c->row_bytes == row_bytes && row_bytes % 16 == 0, "lru cache rows must be a multiple of 16 bytes");
        LruParams lp;
        lp.ids = p->ids[pipe];
        lp.nc = p->pub_nc[pipe % p->slots];  // the hand-off slot's counters (the pipe's own unless it samples ahead)
        lp.op_id = op_id;
        lp.keys = c->keys;
        lp.stamps = c->stamps;
        lp.sets = c->sets;
        lp.ways = c->ways;
        lp.bctl = p->bctl[pipe];
        lp.rows = (const uint8_t *)c->rows;
        lp.host = (const uint8_t *)c->host_table;
        lp.n_nodes = c->n_nodes;
        lp.dst = (uint8_t *)p->features[pipe];
        lp.cache_index = p->cache_index[pipe];
        lp.stats = c->stats;
        lp.row_bytes = row_bytes;
        lp.miss = miss_sink(p, c, most);
        int vpl = (row_bytes / 16 + 31) / 32;
        LG_ARG(vpl >= 1 && vpl <= 4, "row size above 2048 bytes is not supported by the lru gather");
        switch (vpl) {
        case 1: launch_lru<1, 8>(grid, s, lp); break;
        case 2: launch_lru<2, 4>(grid, s, lp); break;
        case 3: launch_lru<3, 2>(grid, s, lp); break;
        default: launch_lru<4, 2>(grid, s, lp); break;
        }
        LG_LAUNCH_CHECK();
        return LEGION_OK;
    }

    GatherParams gp;
    gp.ids = p->ids[pipe];
    gp.nc = gp.nc_out = p->pub_nc[pipe % p->slots];  // the hand-off slot's counters (the pipe's own unless it samples ahead)
    gp.op_id = op_id;
    gp.lut = c ? c->lut : nullptr;
    gp.capacity = c ? (c->capacity > 0 ? c->capacity : 1) : 1;
    gp.kg = c ? c->kg : 1;
    gp.ki = c ? c->ki : 0;
    for (int k = 0; k <= LEGION_MAX_DEVICE; ++k) gp.part[k] = c ? (const uint8_t *)c->part[k] : nullptr;
    gp.host = c ? (const uint8_t *)c->host_table : nullptr;
    gp.n_nodes = c ? c->n_nodes : 1;
    gp.dst = (uint8_t *)p->features[pipe];
    gp.cache_index = reinterpret_cast<int32_t *>(p->cache_index[pipe]);
    gp.stats = c ? c->stats : nullptr;
    gp.row_bytes = row_bytes;
    gp.slot_bytes = c ? c->slot_bytes : row_bytes;
    gp.feature_len = row_bytes / 4;
    gp.miss = miss_sink(p, c, most);
    gp.err = p->ctl[pipe] + CTL_ERROR;
    // staged seed rows are only meaningful for a launch that starts at the seeds, over uncompressed rows
    const bool staged = p->stage_rows != nullptr && (op_id == kOpGatherAll || op_id == 1) && c != nullptr &&
                        c->codec == LEGION_CODEC_RAW && g_gather_engine == 0;
    gp.stage_rows = staged ? p->stage_rows : nullptr;
    gp.stage_pos = staged ? p->stage_pos : nullptr;
    gp.stage_base = staged ? p->stage_base : 0;
    gp.stage_n = staged ? p->stage_n : 0;
    gp.n_rows = -1;
    gp.rows_per_warp = 0;

    // The gather over a batch that was sampled ahead also hands its block structure over; a launch of its own for that
    // was 4 us of every batch.  The bulk-copy engine keeps the two apart.
    gp.pub.o_ids = nullptr;
    if (p->slots < p->pipes && op_id == kOpGatherAll) {
        const int slot = pipe % p->slots;
        gp.pub = Publish{ p->ids[pipe], p->labels[pipe], p->agg_src[pipe], p->agg_dst[pipe], p->node_counter[pipe], p->edge_counter[pipe],
                          p->pub_ids[slot], p->pub_labels[slot], p->pub_agg_src[slot], p->pub_agg_dst[slot], p->pub_nc[slot], p->pub_ec[slot] };
        if (g_gather_engine == 1) {
            publish_kernel<<<p->sm_count * 2, 256, 0, s>>>(gp.pub);
            LG_LAUNCH_CHECK();
            gp.pub.o_ids = nullptr;
        }
        gp.nc = p->node_counter[pipe];
    }

    // the bulk-copy engine has only ever read this GPU's own memory: a clique of more than one GPU keeps the register path
    if (g_gather_engine == 1 && gp.kg == 1 && (c == nullptr || c->codec == LEGION_CODEC_RAW) && row_bytes % 16 == 0 &&
        row_bytes <= 1024 && gp.slot_bytes == row_bytes) {
        // 32 rows per warp in shared memory: 64 KB per CTA for 512-byte rows, three CTAs per SM
        const size_t smem = (size_t)kBulkWarps * 32 * row_bytes;
        static bool attr_set[64] = { false };
        if (p->dev_id >= 0 && p->dev_id < 64 && !attr_set[p->dev_id]) {
            LG_CUDA(cudaFuncSetAttribute(gather_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
            attr_set[p->dev_id] = true;
        }
        int64_t rows = 0;
        segment_grid(p, op_id, &rows, 32, 8);
        int64_t want = (rows + 32 * kBulkWarps - 1) / (32 * kBulkWarps);
        int per_sm = (int)(200 * 1024 / (smem + 1024));
        if (per_sm < 1) per_sm = 1;
        if (g_gather_cps > 0 && g_gather_cps < per_sm) per_sm = g_gather_cps;
        int64_t cap = (int64_t)p->sm_count * per_sm;
        int bgrid = (int)(want < 1 ? 1 : (want > cap ? cap : want));
        gather_bulk_kernel<<<bgrid, kBulkWarps * 32, smem, s>>>(gp);
        LG_LAUNCH_CHECK();
        return LEGION_OK;
    }

    if (c != nullptr && c->codec != LEGION_CODEC_RAW) {
        LG_ARG(gp.feature_len % 4 == 0, "compressed rows need a feature length that is a multiple of 4");
        // (see gather_quant_kernel)
        const int qgrid = segment_grid(p, op_id, nullptr, 8, op_id == kOpGatherAll ? 2 : 8);
        if (c->codec == LEGION_CODEC_INT8) launch_quant<LEGION_CODEC_INT8>(qgrid, s, gp);
        else launch_quant<LEGION_CODEC_E4M3>(qgrid, s, gp);
        LG_LAUNCH_CHECK();
        return LEGION_OK;
    }
    if (row_bytes % 16 == 0 && row_bytes <= 2048) {
        int vpl = (row_bytes / 16 + 31) / 32;
        const int cps = vpl == 1 && op_id == kOpGatherAll ? 2 : 8;
        const int vec_grid = g_gather_rpw > 0 && vpl == 1 ? segment_grid(p, op_id, nullptr, g_gather_rpw, cps * 32 / g_gather_rpw)
                                                          : segment_grid(p, op_id, nullptr, 4, cps);
        gp.rows_per_warp = vpl == 1 ? g_gather_rpw : 0;
        switch (vpl) {
        case 1:
            // 8 rows (4 KB) in flight per warp measured best on 512-byte rows (2: 0.47-0.55 of the copy
            // peak, 4: 0.55-0.57, 8: 0.58-0.61, 16: 0.52-0.55, over 2-8 CTAs per SM)
            // The gather over all nodes of a batch runs beside the sampling kernels of the other pipes.  With two
            // CTAs per SM (each warp then copies two or three chunks, the next chunk's lookups in flight) it
            // leaves a third of the register file to them: the launch alone is as fast as with eight (46.1 against
            // 45.7 us at 2 x 10^5 rows), the batch is 3% shorter with the whole table cached (70.1 against 72.4 us).
            if (g_gather_rows == 4) launch_vec<1, 4>(vec_grid, s, gp);
            else if (g_gather_rows == 16) launch_vec<1, 16>(vec_grid, s, gp);
            else if (g_gather_rows == 2) launch_vec<1, 2>(vec_grid, s, gp);
            else launch_vec<1, 8>(vec_grid, s, gp);
            break;
        case 2: launch_vec<2, 2>(vec_grid, s, gp); break;
        case 3: launch_vec<3, 2>(vec_grid, s, gp); break;
        default: launch_vec<4, 2>(vec_grid, s, gp); break;
        }
    } else {
        LG_ARG(row_bytes % 4 == 0, "row size must be a multiple of 4 bytes");
        launch_flat(segment_grid(p, op_id, nullptr, 4, 8), s, gp);
    }
    LG_LAUNCH_CHECK();
    return LEGION_OK;
}

int g_miss_ctas = 0;     // 0 = default; see legion_set_tunable
int g_miss_threads = 0;  // 0 = default
int g_miss_rows = 0;     // rows a warp of the fetch keeps in flight (0 = default, 4)

// The rows the hit kernels listed so far, fetched from the pinned host table; empties the list.
// No-op when nothing can be on the list: without a host table, or when the cache holds every node and only this library
// has written its table (the launch alone, over an empty list, was 3 us of a batch).
bool cache_may_miss(const LegionCache *c)
{
    return c != nullptr && c->host_table != nullptr && (!c->holds_all || c->lut_given);
}

int launch_gather_misses(cudaStream_t s, LegionPool *p, LegionCache *c)
{
    if (!cache_may_miss(c)) return LEGION_OK;
    const int pipe = p->pipe;
    MissParams mp;
    mp.miss_rows = p->miss_rows[pipe];
    mp.miss_count = p->miss_count[pipe];
    mp.ticket = p->miss_count[pipe] + 4;
    mp.host = (const uint8_t *)c->host_table;
    mp.n_nodes = c->n_nodes;
    mp.dst = (uint8_t *)p->features[pipe];
    mp.row_bytes = p->row_bytes_out;
    mp.host_row_bytes = c->host_codec != LEGION_CODEC_RAW ? c->slot_bytes : p->row_bytes_out;

    // A static cache behind seed staging leaves a few thousand scattered rows per batch, which arrive at the
    // scattered-page rate of the link whatever is in flight, while every row in flight slows the kernels beside
    // the fetch: one row per warp and four warps per CTA measured best (6.5 k batches/s against 6.1 k with four
    // rows per warp and eight warps).  An LRU cache misses tens of thousands of rows per batch: its fetch
    // keeps the wider shape.
    const bool many = c->kind == 1;
    int64_t g64 = (p->max_nodes + 31) / 32;
    int cap = g_miss_ctas > 0 ? g_miss_ctas : kMissCtas;
    int threads = g_miss_threads > 0 ? g_miss_threads : (many ? kMissThreads : 128);
    const int rows = g_miss_rows > 0 ? g_miss_rows : (many ? 4 : 1);
    int grid = (int)(g64 < 1 ? 1 : (g64 > cap ? cap : g64));
    mp.hist = p->miss_ordered[pipe] ? p->miss_hist[pipe] : nullptr;
    if (p->miss_ordered[pipe]) {
        const int32_t n_rows = (int32_t)c->n_nodes;
        const int64_t og = (p->max_nodes + 1023) / 1024;
        miss_order_kernel<<<(int)(og > p->sm_count ? p->sm_count : og), 1024, 0, s>>>(p->miss_rows[pipe], p->miss_rank[pipe], p->miss_count[pipe],
                                                                                    p->miss_hist[pipe], stretch_shift(n_rows), n_rows, p->miss_sorted[pipe]);
        LG_LAUNCH_CHECK();
        mp.miss_rows = p->miss_sorted[pipe];
    }
    const bool narrow = mp.host_row_bytes <= 512 && ((uintptr_t)mp.host & 15) == 0;
    if (c->host_codec == LEGION_CODEC_INT8) {
        if (narrow) gather_miss_quant_kernel<LEGION_CODEC_INT8, 4, true><<<grid, threads, 0, s>>>(mp);
        else gather_miss_quant_kernel<LEGION_CODEC_INT8, 4, false><<<grid, threads, 0, s>>>(mp);
    } else if (c->host_codec == LEGION_CODEC_E4M3) {
        if (narrow) gather_miss_quant_kernel<LEGION_CODEC_E4M3, 4, true><<<grid, threads, 0, s>>>(mp);
        else gather_miss_quant_kernel<LEGION_CODEC_E4M3, 4, false><<<grid, threads, 0, s>>>(mp);
    }
    else if (rows == 1) gather_miss_kernel<1><<<grid, threads, 0, s>>>(mp);
    else if (rows == 2) gather_miss_kernel<2><<<grid, threads, 0, s>>>(mp);
    else if (rows == 8) gather_miss_kernel<8><<<grid, threads, 0, s>>>(mp);
    else gather_miss_kernel<4><<<grid, threads, 0, s>>>(mp);
    LG_LAUNCH_CHECK();
    return LEGION_OK;
}

int launch_gather(cudaStream_t s, LegionPool *p, LegionCache *c, int32_t op_id)
{
    int rc = launch_gather_hits(s, p, c, op_id);
    if (rc != LEGION_OK) return rc;
    return launch_gather_misses(s, p, c);
}

int launch_lru_insert(cudaStream_t s, LegionPool *p, LegionCache *c)
{
    if (c == nullptr || c->kind != 1) return LEGION_OK;
    const int pipe = p->pipe;
    const int cap = p->sm_count * 8;
    int64_t g_thread = (p->max_nodes + 255) / 256;
    int64_t g_warp = (p->max_nodes + 7) / 8;
    int grid_t = (int)(g_thread > cap ? cap : g_thread);
    int grid_w = (int)(g_warp > cap ? cap : g_warp);
    unsigned long long *claim = reinterpret_cast<unsigned long long *>(c->claim);
    lru_claim_kernel<<<grid_t, 256, 0, s>>>(p->ids[pipe], p->cache_index[pipe], p->node_counter[pipe], c->keys, c->stamps,
                                            c->sets, c->ways, p->bctl[pipe], claim, p->lru_victim[pipe]);
    LG_LAUNCH_CHECK();
    lru_commit_kernel<<<grid_w, 256, 0, s>>>(p->ids[pipe], p->node_counter[pipe], c->keys, c->stamps, p->bctl[pipe], claim,
                                             p->lru_victim[pipe], (const uint8_t *)p->features[pipe],
                                             (uint8_t *)c->rows, c->row_bytes, c->stats);
    LG_LAUNCH_CHECK();
    return LEGION_OK;
}

}  // namespace legion

// ---- gather without any allocation ---------------------------------------------------------------------
// legion_gather_rows_noalloc: the lookup + gather of one list of node ids (cached rows from the
// clique's partitions, the others from the pinned host table) for callers that must not allocate
// device memory when they call into this library: a trainer-side process whose framework allocator
// already owns the GPU's memory, or a serving loop that cannot afford the device-wide
// synchronisation, the fragmentation or the failure of a cudaMalloc in the middle of a step.  The
// entry points above take their scratch (cache_index, the miss list and its counters, the segment
// words the kernels read) from a LegionPool, which allocates; this one keeps the same scratch in a
// fixed array inside the library image.  Every GPU that loads the library holds that array
// (256 B + 12 B per row of LEGION_NOALLOC_MAX_ROWS, about 3 MB) until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[256 + 12 * (size_t)LEGION_NOALLOC_MAX_ROWS];

namespace legion {

// byte offsets inside the array
constexpr size_t kNaMissCount = 64;  // 8 int32: [0] entries of the miss list, [4] ticket
constexpr size_t kNaMissRows = 256;  // int2[LEGION_NOALLOC_MAX_ROWS]
constexpr size_t kNaCacheIndex = 256 + 8 * (size_t)LEGION_NOALLOC_MAX_ROWS;  // int32[LEGION_NOALLOC_MAX_ROWS]

}  // namespace legion

// In host code the name g_noalloc_scratch is only a stand-in for the device array: its device
// address is asked for once per device, with that device current, and kept here.
static void *g_noalloc_ptr[64] = { nullptr };
static cudaError_t noalloc_scratch_of(int dev_id, unsigned char **out)
{
    if (g_noalloc_ptr[dev_id] == nullptr) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev_id] = p;
    }
    *out = (unsigned char *)g_noalloc_ptr[dev_id];
    return cudaSuccess;
}

extern "C" int legion_gather_rows_noalloc(void *stream, int32_t dev_id, const int32_t *ids_dev, int64_t n_rows,
                                          const int32_t *lut_dev, int32_t capacity, int32_t kg, int32_t ki,
                                          const void *const *partitions, const void *host_table, int64_t n_nodes,
                                          int32_t row_bytes, void *out_dev)
{
    using namespace legion;
    LG_ARG(dev_id >= 0 && dev_id < 64, "dev_id out of range");
    LG_ARG(n_rows >= 0 && (n_rows == 0 || (ids_dev != nullptr && out_dev != nullptr)), "NULL pointer");
    if (n_rows > LEGION_NOALLOC_MAX_ROWS) {
        set_error("legion_gather_rows_noalloc: %lld rows are above the built-in scratch of %d rows; split the list or "
                  "use legion_feature_cache_lookup with a LegionPool",
                  (long long)n_rows, LEGION_NOALLOC_MAX_ROWS);
        return LEGION_E_LIMIT;
    }
    LG_ARG(row_bytes > 0 && row_bytes % 4 == 0, "row_bytes must be a positive multiple of 4");
    LG_ARG(kg >= 1 && kg <= LEGION_MAX_DEVICE && ki >= 0 && ki < kg, "bad clique size or member index");
    LG_ARG(lut_dev == nullptr || (capacity > 0 && partitions != nullptr), "a lookup table needs partitions");
    LG_ARG(n_nodes > 0, "n_nodes must be positive");
    LG_CUDA(cudaSetDevice(dev_id));
    unsigned char *scratch = nullptr;
    LG_CUDA(noalloc_scratch_of(dev_id, &scratch));
    if (n_rows == 0) return LEGION_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int32_t *miss_count = reinterpret_cast<int32_t *>(scratch + kNaMissCount);
    // The array is shared by every call and keeps what the last call left: a call that may list misses starts from an
    // empty list.  Without a host table nothing is listed, and the gather is the only launch.
    if (host_table != nullptr) LG_CUDA(cudaMemsetAsync(miss_count, 0, 32, s));

    GatherParams gp;
    gp.ids = ids_dev;
    gp.nc = gp.nc_out = nullptr;
    gp.pub.o_ids = nullptr;
    gp.op_id = 1;
    gp.n_rows = (int32_t)n_rows;
    gp.rows_per_warp = 0;
    gp.lut = lut_dev;
    gp.capacity = capacity > 0 ? capacity : 1;
    gp.kg = kg;
    gp.ki = ki;
    for (int k = 0; k <= LEGION_MAX_DEVICE; ++k)
        gp.part[k] = (lut_dev != nullptr && k < kg) ? (const uint8_t *)partitions[k] : nullptr;
    gp.host = (const uint8_t *)host_table;
    gp.n_nodes = n_nodes;
    gp.dst = (uint8_t *)out_dev;
    gp.cache_index = reinterpret_cast<int32_t *>(scratch + kNaCacheIndex);
    gp.stats = nullptr;
    gp.err = nullptr;
    gp.stage_rows = nullptr;
    gp.stage_pos = nullptr;
    gp.stage_base = gp.stage_n = 0;
    gp.row_bytes = row_bytes;
    gp.slot_bytes = row_bytes;
    gp.feature_len = row_bytes / 4;
    gp.miss = MissSink{ reinterpret_cast<int2 *>(scratch + kNaMissRows), miss_count, nullptr, nullptr, 0, 1 };
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_id);
    if (sms <= 0) sms = 148;
    const int64_t g64 = ((n_rows + 3) / 4 + 7) / 8;
    const int grid = (int)(g64 > (int64_t)sms * 8 ? (int64_t)sms * 8 : g64);
    if (row_bytes % 16 == 0 && row_bytes <= 2048) {
        int vpl = (row_bytes / 16 + 31) / 32;
        switch (vpl) {
        case 1: launch_vec<1, 8>(grid, s, gp); break;  // the shape the pool-based path launches
        case 2: launch_vec<2, 2>(grid, s, gp); break;
        case 3: launch_vec<3, 2>(grid, s, gp); break;
        default: launch_vec<4, 2>(grid, s, gp); break;
        }
    } else {
        launch_flat(grid, s, gp);
    }
    LG_LAUNCH_CHECK();
    if (host_table != nullptr) {
        MissParams mp;
        mp.miss_rows = gp.miss.rows;
        mp.hist = nullptr;
        mp.miss_count = miss_count;
        mp.ticket = miss_count + 4;
        mp.host = (const uint8_t *)host_table;
        mp.n_nodes = n_nodes;
        mp.dst = (uint8_t *)out_dev;
        mp.row_bytes = row_bytes;
        mp.host_row_bytes = row_bytes;
        int64_t m64 = (n_rows + 31) / 32;
        int mgrid = (int)(m64 < 1 ? 1 : (m64 > (int64_t)sms * 2 ? (int64_t)sms * 2 : m64));
        gather_miss_kernel<4><<<mgrid, 256, 0, s>>>(mp);
        LG_LAUNCH_CHECK();
    }
    return LEGION_OK;
}

// Launch-shape knobs for measurements.  "miss_ctas": CTAs of the host-link fetch (0 = one per SM).
extern "C" int legion_set_tunable(const char *name, int32_t value)
{
    using namespace legion;
    LG_ARG(name != nullptr, "name is NULL");
    if (strcmp(name, "miss_ctas") == 0) {
        LG_ARG(value >= 0 && value <= 4096, "miss_ctas out of range");
        g_miss_ctas = value;
        return LEGION_OK;
    }
    if (strcmp(name, "miss_threads") == 0) {
        LG_ARG(value == 0 || (value >= 32 && value <= 1024 && value % 32 == 0), "miss_threads must be a multiple of 32 up to 1024");
        g_miss_threads = value;
        return LEGION_OK;
    }
    if (strcmp(name, "miss_rows") == 0) {
        LG_ARG(value == 0 || value == 1 || value == 2 || value == 4 || value == 8, "miss_rows must be 0, 1, 2, 4 or 8");
        g_miss_rows = value;
        return LEGION_OK;
    }
    if (strcmp(name, "map_front_shift") == 0) {
        LG_ARG(value >= -1 && value <= 30, "map_front_shift must be -1 (automatic) or 0..30");
        g_map_front_shift = value;  // pools created afterwards
        return LEGION_OK;
    }
    if (strcmp(name, "pdl") == 0) {
        LG_ARG(value >= -1 && value <= 1, "pdl must be -1 (by the pool), 0 or 1");
        g_pdl = value;  // takes effect for runners created (graphs captured) afterwards
        return LEGION_OK;
    }
    if (strcmp(name, "scan_wait_limit") == 0) {
        LG_ARG(value >= -1 && value <= 1 << 30, "scan_wait_limit must be -1 .. 2^30");
        g_scan_wait_limit = value;  // ops issued and graphs captured afterwards
        return LEGION_OK;
    }
    if (strcmp(name, "gather_engine") == 0) {
        LG_ARG(value == 0 || value == 1, "gather_engine must be 0 (registers) or 1 (bulk copies)");
        g_gather_engine = value;
        return LEGION_OK;
    }
    if (strcmp(name, "gather_ctas_per_sm") == 0) {
        LG_ARG(value >= 0 && value <= 16, "gather_ctas_per_sm out of range");
        g_gather_cps = value;
        return LEGION_OK;
    }
    if (strcmp(name, "gather_rows_per_warp") == 0) {
        LG_ARG(value == 0 || value == 8 || value == 16 || value == 32, "gather_rows_per_warp must be 0, 8, 16 or 32");
        g_gather_rpw = value == 32 ? 0 : value;
        return LEGION_OK;
    }
    if (strcmp(name, "gather_rows_in_flight") == 0) {
        LG_ARG(value == 0 || value == 2 || value == 4 || value == 8 || value == 16, "gather_rows_in_flight must be 0, 2, 4, 8 or 16");
        g_gather_rows = value;
        return LEGION_OK;
    }
    set_error("legion_set_tunable: unknown name %s", name);
    return LEGION_E_ARG;
}
