// Batched many-table entry points: thousands of independent unordered_set / unordered_map objects of
// uneven sizes built and probed in one launch per operation.
//
// All tables of a batch share one device arena (each table's probe groups contiguous, the layout and
// geometry of a single table: include/stdgpu_gb300/detail/layout.cuh) and a device array of per-table
// views.  An operation takes the keys of all tables concatenated, with per-table offsets in device
// memory.  A small kernel turns the offsets into a tile list -- tile x covers 32 consecutive keys of
// one table -- as a prefix count of tiles per table; a persistent kernel then walks the tiles
// (tile -> table by binary search of the prefix), running the same warp steps as the single-table
// kernels on that table's view.  No host work depends on the sizes, so a sequence of batched calls
// can be captured in a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <vector>

#include "region_build.cuh"
#include "sg_internal.cuh"
#include "stdgpu_gb300.h"
#include "table_core.cuh"

namespace sg
{
namespace detail
{

// Exclusive scan over the tables t < n of count(t), handed to put(t, sum before t) for t <= n, by one block of 1024
// threads, four consecutive tables per thread at a time.  What bounds it is the chain from a round's loads to the
// next round's: 4 us for up to 4096 tables, 19 for 16384, 71 for 65536.  With a run of tables per thread, read twice
// and one after another, an insert of 3 keys each into 65536 tables takes 210 us instead of 126.
template <typename Count, typename Put>
SG_D void
scan_tables(int32_t n, Count count, Put put)
{
    constexpr int kPer = 4;
    __shared__ long long warp_sums[2][32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    long long carry = 0;
    int buf = 0;
    for (int64_t base = 0; base < n; base += kPer * 1024, buf ^= 1)
    {
        const int64_t t0 = base + kPer * static_cast<int64_t>(threadIdx.x);
        long long c[kPer];
        long long s = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            c[k] = t0 + k < n ? count(t0 + k) : 0;
            s += c[k];
        }
        long long incl = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const long long x = __shfl_up_sync(0xffffffffu, incl, d);
            incl += lane >= d ? x : 0;
        }
        if (lane == 31)
        {
            warp_sums[buf][warp] = incl;
        }
        __syncthreads(); // one per round: the next one fills the other buffer
        const bool more = base + kPer * 1024 < n;
        long long run = carry + incl - s;
        for (int w = 0; w < (more ? 32 : warp); ++w)
        {
            const long long x = warp_sums[buf][w];
            run += w < warp ? x : 0;
            carry += x;
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            if (t0 + k < n)
            {
                put(t0 + k, run);
            }
            run += c[k];
        }
        if (!more && threadIdx.x == 1023)
        {
            put(n, run);
        }
    }
}

SG_D long long
tiles_of(const int64_t* offsets, int64_t t, int tile)
{
    const int64_t cnt = offsets[t + 1] - offsets[t];
    return cnt > 0 ? (cnt + tile - 1) / tile : 0;
}

// Prefix of tile counts: prefix[t] = sum over u < t of ceil(n_u / 32); prefix[n] = all tiles.  Tables whose `todo`
// (nullable) is 0 have no tiles.
__global__ void __launch_bounds__(1024, 2)
k_batch_tiles(const int64_t* offsets, int32_t n, int64_t* prefix, bool has_keys, const uint8_t* todo)
{
    wait_for_stream();
    scan_tables(
            n,
            [&](int64_t t) -> long long {
                return has_keys && (todo == nullptr || todo[t] != 0) ? tiles_of(offsets, t, 32) : 0;
            },
            [&](int64_t t, long long x) { prefix[t] = x; });
}

// Table of tile x: the last t with prefix[t] <= x (binary search by lane 0, broadcast to the warp).
SG_D int32_t
tile_table(const int64_t* prefix, int32_t n, int64_t x)
{
    int32_t t = 0;
    if ((threadIdx.x & 31) == 0)
    {
        int32_t lo = 0, hi = n; // invariant: prefix[lo] <= x < prefix[hi]
        while (hi - lo > 1)
        {
            const int32_t mid = (lo + hi) >> 1;
            if (prefix[mid] <= x)
            {
                lo = mid;
            }
            else
            {
                hi = mid;
            }
        }
        t = lo;
    }
    return __shfl_sync(0xffffffffu, t, 0);
}

// ---------------------------------------------------------------- inserts into empty tables (region_build.cuh)

// A region of one table.
struct build_item
{
    int32_t table;
    uint32_t first; // groups
    uint32_t count;
    int32_t list; // its list, or -1 for a table's only region: the keys are read from the input
};

constexpr int kListPer = 4; // elements per thread and tile of the lists

// Counts of a call, behind the lists' lengths; all zero when it starts.
struct build_words
{
    unsigned int spilled; // keys offered to the spill list
    unsigned int taken;   // items that blocks have taken beyond their first
    unsigned int arrived; // blocks of k_batch_choose that are done
    unsigned int any;     // 1: a table is built
};

// A key that found no room in its region, for the probe kernel.  More of them than the buffer holds mark their
// tables todo.
struct spill_entry
{
    uint4 image; // the slot's bytes (16, 8 or 4 of them)
    int32_t table;
    int32_t pad[3];
};
constexpr unsigned int kSpillMax = 1u << 15;

struct spill_list
{
    unsigned int* count; // offered (may exceed kSpillMax)
    spill_entry* entry;
};

// First launch of an insert into a batch that may be empty: build[t] = 1 for a table that holds nothing and gets at
// least a key per group (a region is written whole, so fewer keys are cheaper to insert one by one) and not many more
// than it has slots; todo[t] = 1 for the others that get keys.  4096 tables of 8192, built and walked: 142 and 105 us
// at half a key per group, 152 and 150 at one, 179 and 257 at two; of 1000 (one region) 40 and 33, 40 and 49, 43 and
// 70.  A table of several regions with more keys than slots is left to the walk, since a list would overflow.  A
// table of one region is built by one block, whatever copies its keys hold, while that block gets at most twice an
// even share of the call's keys among `resident` blocks: 697 tables of 1000 with 5000 distinct keys each take 6680 us
// so, 9074 by the walk, and one table of 1000 with 2^22 copies of 500 keys takes 127 us by the walk, 9270 by one
// block.  Tables of several regions get lists (prefix: their tiles of `tile` elements; item_prefix: the regions of
// the tables before that are built), which leave no room for an element's index: with per-key flags they go to the
// probe kernel.  The last block to finish adds up the tables, unless none is built: 3 keys each into 65536 cleared
// tables of 2100 take 155 us, 520 when one block did all of it and each region had its block, 244 with no table ever
// built.
__global__ void __launch_bounds__(1024)
k_batch_choose(const dview* views, const int64_t* offsets, int32_t n, const int32_t* first_item, bool flags, int tile,
               int resident, uint8_t* build, uint8_t* todo, int64_t* prefix, int64_t* item_prefix, build_words* words)
{
    wait_for_stream();
    __shared__ unsigned int s_last;
    const bool alone = gridDim.x == 1;
    const int64_t twice = 2 * (offsets[n] - offsets[0]);
    bool any = false;
    for (int32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    {
        const dview v = views[t];
        const int64_t cnt = offsets[t + 1] - offsets[t];
        const int32_t regions = first_item[t + 1] - first_item[t];
        const bool ok = cnt >= v.num_groups &&
                        (cnt <= v.total || (regions == 1 && cnt * resident <= twice)) && regions > 0 &&
                        (regions == 1 || !flags) && v.hdr->size == 0 && v.hdr->tombstones == 0;
        build[t] = ok ? 1 : 0;
        todo[t] = cnt > 0 && !ok ? 1 : 0;
        any = any || ok;
    }
    any = __syncthreads_or(any) != 0;
    if (!alone)
    {
        if (threadIdx.x == 0)
        {
            if (any)
            {
                atomicOr(&words->any, 1u);
            }
            __threadfence();
            s_last = atomicAdd(&words->arrived, 1u) == gridDim.x - 1 ? 1u : 0u;
            __threadfence();
        }
        __syncthreads();
        if (s_last == 0u)
        {
            return;
        }
        // the last block has all tables' marks
        any = __ldcg(&words->any) != 0u;
    }
    if (!any)
    {
        if (threadIdx.x == 0)
        {
            prefix[n] = 0;
            item_prefix[n] = 0;
        }
        return;
    }
    // both sums in one scan: tiles in the upper half, items (fewer than 2^31) in the lower
    scan_tables(
            n,
            [&](int64_t t) -> long long {
                const uint8_t mark = alone ? build[t] : __ldcg(build + t);
                const long long regions = mark != 0 ? first_item[t + 1] - first_item[t] : 0;
                return (regions > 1 ? tiles_of(offsets, t, tile) << 32 : 0) + regions;
            },
            [&](int64_t t, long long x) {
                prefix[t] = x >> 32;
                item_prefix[t] = x & 0xffffffffll;
            });
}

// Second launch: the items that are built in `order` (nullable: the build looks at every item), and the keys of the
// tables that are built and have several regions, appended to the lists in their regions' slots.
template <int KIND, bool AOS>
__global__ void __launch_bounds__(kListThreads, 3)
k_batch_lists(const dview* views, const int64_t* offsets, const int64_t* prefix, int32_t n, const int32_t* first_item,
              const build_item* items, int32_t n_items, const uint8_t* build, const int64_t* item_prefix,
              build_item* order, unsigned int* fill, uint8_t* todo, const void* in0, const void* in1)
{
    wait_for_stream();
    if (order != nullptr && item_prefix[n] == 0)
    {
        return;
    }
    for (int32_t i = order != nullptr ? blockIdx.x * kListThreads + threadIdx.x : n_items; i < n_items;
         i += gridDim.x * kListThreads)
    {
        const build_item it = items[i];
        if (build[it.table] != 0)
        {
            order[item_prefix[it.table] + i - first_item[it.table]] = it;
        }
    }
    using C = kind_consts<KIND>;
    using E = typename slot_image<KIND>::type;
    constexpr int PER = kListPer;
    constexpr int64_t kTile = int64_t{ PER } * kListThreads;
    extern __shared__ __align__(128) unsigned char smem[];
    auto& s = *reinterpret_cast<list_tile<E, PER>*>(smem);
    __shared__ int32_t s_table;
    // a block takes consecutive tiles: one search, then the tables in order
    const int64_t tiles = prefix[n];
    const int64_t x_lo = tiles * blockIdx.x / gridDim.x, x_hi = tiles * (blockIdx.x + 1) / gridDim.x;
    if (x_lo == x_hi)
    {
        return;
    }
    if (threadIdx.x < 32)
    {
        const int32_t t = tile_table(prefix, n, x_lo);
        if (threadIdx.x == 0)
        {
            s_table = t;
        }
    }
    __syncthreads();
    int32_t tb = s_table;
    for (int64_t x = x_lo; x < x_hi; ++x)
    {
        while (prefix[tb + 1] <= x)
        {
            ++tb;
        }
        const dview t = views[tb];
        const int32_t i0 = first_item[tb];
        const int regions = first_item[tb + 1] - i0;
        const int64_t lo = offsets[tb] + (x - prefix[tb]) * kTile;
        const int64_t hi = offsets[tb + 1];
        E elem[PER];
        int rid[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j)
        {
            const int64_t i = lo + j * kListThreads + threadIdx.x;
            rid[j] = -1;
            if (i < hi)
            {
                typename C::K key;
                typename C::V val;
                load_input<KIND, AOS>(in0, in1, i, key, val);
                if (key >= C::tomb_key)
                {
                    if (special_insert<KIND>(t, key, val) != 0)
                    {
                        atomicAdd(&t.hdr->size, 1ull);
                    }
                }
                else
                {
                    elem[j] = pack_element<KIND>(key, val);
                    rid[j] = static_cast<int>(home_of<KIND>(t, key) >> kRegionGroupsLog2);
                }
            }
        }
        const bool lost = append_to_lists<E, PER>(
                s, regions, elem, rid, fill + i0,
                [&](int r, unsigned int k) {
                    return reinterpret_cast<E*>(t.slots + (static_cast<uint64_t>(r) << (kRegionGroupsLog2 + 7))) + k;
                },
                [&](int r) {
                    return min(t.num_groups - (static_cast<uint32_t>(r) << kRegionGroupsLog2), kRegionGroups) *
                           C::slots_per_group;
                });
        if (lost)
        {
            todo[tb] = 1;
        }
    }
}

// Third launch: the items that are built, one region at a time per block.  A batch of more items than blocks that are
// resident at once (ORDERED) gives the built ones in `items`, `built` of them, and the blocks take the next one from
// a counter: a block for each of its regions, built or not, made an insert of 3 keys each into 4096 cleared tables of
// 8192 take 46 us, 26 so.  Else each item has its block, which looks whether it is built: two reads less to wait for,
// 13.2 us against 14.2 for 697 tables of 817 regions.  Spilled keys go to the probe kernel one by one.  A table some
// of whose keys found no room in a list is marked todo: the probe kernel then runs over all its keys, which changes
// nothing for those stored here.
template <int KIND, bool AOS, bool ORDERED>
__global__ void __launch_bounds__(kRegionThreads, kRegionBlocks)
k_batch_build(const dview* views, const int64_t* offsets, const build_item* items, const int64_t* built,
              const uint8_t* build, unsigned int* next, const unsigned int* fill, uint8_t* todo, const void* in0,
              const void* in1, uint8_t* out_flags, spill_list spills)
{
    wait_for_stream();
    using C = kind_consts<KIND>;
    using K = typename C::K;
    using V = typename C::V;
    using E = typename slot_image<KIND>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned int s_next;
    const int64_t n_built = ORDERED ? *built : gridDim.x;
    for (int64_t w = blockIdx.x; w < n_built; w = ORDERED ? s_next : n_built)
    {
        const build_item it = items[w];
        const bool whole = it.list < 0;
        const dview t = views[it.table];
        const int64_t lo = offsets[it.table], hi = offsets[it.table + 1];
        const unsigned int listed = whole ? 0u : fill[it.list];
        if (!ORDERED && build[it.table] == 0)
        {
            return;
        }
        const region r{ reinterpret_cast<char*>(smem), it.first, it.count, whole };
        region_start<KIND>(t, r);
        __syncthreads();
        if (ORDERED && threadIdx.x == 0)
        {
            s_next = gridDim.x + atomicAdd(next, 1u); // there by the time the region is built
        }
        const E* const list = reinterpret_cast<const E*>(t.slots + (static_cast<uint64_t>(it.first) << 7));
        const int64_t count = whole ? hi - lo
                                            : static_cast<int64_t>(min(listed, it.count * C::slots_per_group));
        unsigned int done = 0, refused = 0;
        constexpr int kAhead = 4; // keys loaded before any is inserted
        for (int64_t base = threadIdx.x; base < count; base += kAhead * kRegionThreads)
        {
            K key[kAhead];
            V val[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j)
            {
                const int64_t i = base + j * kRegionThreads;
                if (i < count)
                {
                    if (whole)
                    {
                        load_input<KIND, AOS>(in0, in1, lo + i, key[j], val[j]);
                    }
                    else
                    {
                        unpack_element<KIND>(__ldcg(list + i), key[j], val[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kAhead; ++j)
            {
                const int64_t i = base + j * kRegionThreads;
                if (i >= count)
                {
                    break;
                }
                const int res = key[j] >= C::tomb_key
                                        ? special_insert<KIND>(t, key[j], val[j])
                                        : region_insert<KIND>(r, home_of<KIND>(t, key[j]) - it.first,
                                                              rot_of(static_cast<uint64_t>(key[j])), key[j], val[j]);
                done += (res == kRegionInserted);
                refused += (res == kRegionRefused);
                if (res == kRegionSpill)
                {
                    const unsigned int k = atomicAdd(spills.count, 1u);
                    if (k < kSpillMax)
                    {
                        spill_entry x{};
                        *reinterpret_cast<E*>(&x.image) = pack_element<KIND>(key[j], val[j]);
                        x.table = it.table;
                        spills.entry[k] = x;
                    }
                    else
                    {
                        todo[it.table] = 1;
                    }
                }
                if (out_flags != nullptr)
                {
                    out_flags[lo + i] = static_cast<uint8_t>(res == kRegionInserted);
                }
            }
        }
        __syncthreads(); // the list, which lies in the region's slots, is read
        region_write(t, r);
        unsigned int c[2] = { done, refused };
        unsigned long long* const dst[2] = { &t.hdr->size, &t.hdr->refused };
        region_add<2>(c, dst);
        __syncthreads(); // the region is written out, and the next item is there
    }
}

enum batch_op : int
{
    kOpInsertAos = 0,
    kOpInsertSoa = 1,
    kOpErase = 2,
    kOpFind = 3,
    kOpContains = 4
};

// Persistent walk over the tile list; each warp takes up to `tiles_per_step` consecutive tiles at a time (fewer when
// there are not that many for every warp).  Bound by the probes' instructions and L2 reads; what a step pays beyond
// its probes is the search for its first table, a dozen dependent loads.  25.8 M queries over 4096 tables: 449 us
// with 8 tiles a step, 483 with 4, 719 with 1, 564 with a search and a view per tile at 4 a step.
template <int KIND, int OP, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
k_batch(const dview* views, const int64_t* offsets, const int64_t* prefix, int32_t n, int tiles_per_step,
        const void* in0, const void* in1, void* out_vals, uint8_t* out_flags, const uint8_t* todo,
        spill_list spills)
{
    wait_for_stream();
    const tile_lanes L;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t tiles = prefix[n];
    unsigned long long retry = 0;
    const int64_t share = tiles / nwarps;
    tiles_per_step = share < tiles_per_step ? (share < 1 ? 1 : static_cast<int>(share)) : tiles_per_step;
    for (int64_t x0 = warp * tiles_per_step; x0 < tiles; x0 += nwarps * tiles_per_step)
    {
        const int64_t x1 = x0 + tiles_per_step < tiles ? x0 + tiles_per_step : tiles;
        // one search per step, then the tables in order; a table's counts are added once per step
        int32_t tb = tile_table(prefix, n, x0);
        int64_t next = prefix[tb + 1]; // first tile of the table after
        for (int64_t x = x0; x < x1;)
        {
            while (next <= x)
            {
                ++tb;
                next = prefix[tb + 1];
            }
            const dview t = views[tb];
            const int64_t end = offsets[tb + 1];
            int64_t i = offsets[tb] + (x - prefix[tb]) * 32 + L.lane;
            step_counts c;
            for (const int64_t stop = next < x1 ? next : x1; x < stop; ++x, i += 32)
            {
                const bool valid = i < end;
                if constexpr (OP == kOpInsertAos || OP == kOpInsertSoa)
                {
                    insert_step<KIND, OP == kOpInsertAos>(t, L, in0, in1, i, valid, out_flags, c);
                }
                else if constexpr (OP == kOpErase)
                {
                    erase_step<KIND>(t, L, in0, i, valid, out_flags, c);
                }
                else
                {
                    find_step<KIND, OP == kOpFind>(t, L, in0, i, valid, out_vals, out_flags);
                }
            }
            if constexpr (OP == kOpInsertAos || OP == kOpInsertSoa)
            {
                const unsigned int d = __reduce_add_sync(0xffffffffu, c.done);
                const unsigned int r = __reduce_add_sync(0xffffffffu, c.refused);
                const unsigned int u = __reduce_add_sync(0xffffffffu, c.reused);
                retry += c.retry;
                if (L.lane == 0)
                {
                    if (d != 0)
                    {
                        atomicAdd(&t.hdr->size, static_cast<unsigned long long>(d));
                    }
                    if (r != 0)
                    {
                        atomicAdd(&t.hdr->refused, static_cast<unsigned long long>(r));
                    }
                    if (u != 0)
                    {
                        atomicAdd(&t.hdr->tombstones, 0ull - u);
                    }
                }
            }
            else if constexpr (OP == kOpErase)
            {
                const unsigned int d = __reduce_add_sync(0xffffffffu, c.done);
                const unsigned int o = __reduce_add_sync(0xffffffffu, c.oob);
                if (L.lane == 0 && d != 0)
                {
                    atomicAdd(&t.hdr->size, 0ull - d);
                    atomicAdd(&t.hdr->tombstones, static_cast<unsigned long long>(d - o));
                }
            }
        }
    }
    if constexpr (OP == kOpInsertAos || OP == kOpInsertSoa)
    {
        // keys that found no room in their region, one per warp step (their tables differ); those of a table marked
        // todo are among the keys walked above, and a full table counts each refused key once
        const int64_t spilled = todo != nullptr ? min(*spills.count, kSpillMax) : 0u;
        for (int64_t e = warp; e < spilled; e += nwarps)
        {
            const spill_entry x = spills.entry[e];
            if (todo[x.table] != 0)
            {
                continue;
            }
            const dview t = views[x.table];
            typename kind_consts<KIND>::K key;
            typename kind_consts<KIND>::V val;
            unpack_element<KIND>(*reinterpret_cast<const typename slot_image<KIND>::type*>(&x.image), key, val);
            step_counts c;
            insert_kv_step<KIND>(t, L, key, val, 0, L.lane == 0, nullptr, c);
            retry += c.retry;
            if (L.lane == 0)
            {
                atomicAdd(c.done != 0 ? &t.hdr->size : &t.hdr->refused,
                          static_cast<unsigned long long>(c.done + c.refused));
            }
        }
    }
    if (retry != 0)
    {
        atomicOr(&views[0].hdr->error, kErrRetry);
    }
}

SG_D void
reset_header(table_header* h)
{
    h->size = 0;
    h->refused = 0;
    h->tombstones = 0;
    h->special_state[0] = 0;
    h->special_state[1] = 0;
    h->error = 0;
    h->count = 0;
}

// clear() of all tables after the arena is filled with the never-used marker in one stream of writes: the erased
// marker into each table's slots at or above total_count, and the headers (4 us for 4096 tables).  Blocks that walked
// pieces of 256 KB, each found by two dependent loads, took 164 us for 0.85 GB; clear, insert and contains of 4096
// tables went from 1107 to 1071 us.
template <int KIND>
__global__ void __launch_bounds__(256)
k_batch_reset(const dview* views, int32_t n)
{
    using C = kind_consts<KIND>;
    using K = typename C::K;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const dview t = views[i];
        // fewer than a group of them
        for (uint32_t s = t.total; s < t.num_groups * C::slots_per_group; ++s)
        {
            *reinterpret_cast<K*>(t.slots + static_cast<uint64_t>(s) * C::slot_bytes) = C::tomb_key;
        }
        reset_header(t.hdr);
    }
}

// clear() of all tables of a small arena in one launch: a region per block and turn, the group of the out-of-band keys
// with a table's last region, the header with its first.
template <int KIND>
__global__ void __launch_bounds__(256)
k_batch_clear(const dview* views, const build_item* items, int32_t n_items)
{
    wait_for_stream();
    using C = kind_consts<KIND>;
    for (int32_t i = blockIdx.x; i < n_items; i += gridDim.x)
    {
        const build_item it = items[i];
        const dview t = views[it.table];
        uint4* const units = reinterpret_cast<uint4*>(t.slots + (static_cast<uint64_t>(it.first) << 7));
        const uint32_t inside = it.count * (kGroupBytes / 16);
        const uint32_t all = inside + (it.first + it.count == t.num_groups ? kGroupBytes / 16 : 0u);
        for (uint32_t u = threadIdx.x; u < all; u += blockDim.x)
        {
            units[u] = u < inside ? cleared_unit<KIND>(t, it.first * C::slots_per_group + u * C::slots_per_lane)
                                  : make_uint4(~0u, ~0u, ~0u, ~0u);
        }
        if (it.first == 0u && threadIdx.x == 0)
        {
            reset_header(t.hdr);
        }
    }
}

__global__ void
k_batch_gather_sizes(const dview* views, int32_t n, long long* sizes)
{
    for (int32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    {
        sizes[t] = static_cast<long long>(views[t].hdr->size);
    }
}

} // namespace detail
} // namespace sg

using namespace sg::detail;

struct sg_table_batch
{
    int32_t kind;
    int32_t n;
    int32_t threads;       // launch shape of the walking kernels (autotuned)
    int32_t blocks_per_sm;
    int32_t tiles_per_step;
    int32_t sms;
    char* arena;
    table_header* headers;
    dview* views;            // device
    std::vector<dview> host_views;
    std::vector<int64_t> capacities, bucket_counts, totals;
    int64_t* prefix;         // device, n + 1
    long long* sizes_dev;    // device, n
    long long* sizes_host;   // pinned, n
    int64_t arena_bytes;
    unsigned int* locks;     // stripe locks of native device inserts, shared by the batch's tables
    // Inserts into empty tables: the regions, table by table; per table its first region (n + 1), the two marks of a
    // call and the prefix of its lists' tiles; per region the length of its list.  All in build_block.
    char* build_block;       // device
    build_item* items;       // device
    int64_t n_items;
    int32_t* first_item;     // device, n + 1
    uint8_t* marks;          // device, 2 n
    build_item* order;       // device, n_items: a call's items that are built
    unsigned int* fill;      // device, n_items, and the build_words behind them
    int64_t* list_prefix;    // device, n + 1
    spill_list spills;       // device
    bool in_regions;         // every table has its regions among the items
    bool torn;               // lists were queued into tables' slots, but the launch that builds from them was refused
    bool maybe_empty;        // cleared or created since the last insert: tries the build (the device decides per table)
};

size_t
fill_bytes(int64_t n_items)
{
    return sizeof(unsigned int) * static_cast<size_t>(n_items) + sizeof(build_words);
}

build_words*
words_of(unsigned int* fill, int64_t n_items)
{
    return reinterpret_cast<build_words*>(fill + n_items);
}

// A batch whose tables take no more than this together is cleared in one launch (k_batch_clear), which a launch less
// makes sooner; above it the fill's rate counts.  One launch, and a fill and a launch: 1 table of 1.7 KB 1.7 and 4.5 us
// (4.4 before there were two), of 53 KB 2.1 and 8.3 (4.4), 1000 of 5 KB 2.4 and 10.5 (4.4), 697 uneven ones of 9.6 MB
// 3.6 and 10.5, 600 of 335 KB (201 MB) 33 and 37; 2000 of them (671 MB) 106 and 99.
constexpr int64_t kClearArenaMax = int64_t{ 1 } << 28;

constexpr int64_t kBatchInsertLocks = int64_t{ 1 } << 16;

namespace
{

inline void
batch_geometry(int64_t capacity, int kind, int64_t* bucket_count, int64_t* total, int64_t* groups, int* bits)
{
    int64_t b = 0, e = 0;
    reference_geometry(capacity, &b, &e);
    const int spg = kGroupBytes / slot_bytes_of_kind(kind);
    *bucket_count = b;
    *total = b + e;
    *groups = (*total + spg - 1) / spg;
    *bits = log2_exact(b);
}

template <int KIND>
struct batch_launch
{
    template <int OP, int THREADS>
    static sg_status
    go(sg_table_batch* b, const int64_t* offsets, const void* in0, const void* in1, void* out_vals,
       uint8_t* out_flags, const uint8_t* todo, cudaStream_t s)
    {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<KIND, OP, THREADS>, THREADS, 0);
        per_sm = per_sm < 1 ? 1 : per_sm;
        const int want = b->blocks_per_sm > 0 ? (b->blocks_per_sm < per_sm ? b->blocks_per_sm : per_sm) : per_sm;
        SG_CUDA_TRY(launch_early(k_batch<KIND, OP, THREADS>, b->sms * want, THREADS, s, b->views, offsets, b->prefix,
                                 b->n, b->tiles_per_step, in0, in1, out_vals, out_flags, todo, b->spills));
        SG_LAUNCH_CHECK();
        return SG_OK;
    }

    template <int OP>
    static sg_status
    run_op(sg_table_batch* b, const int64_t* offsets, const void* in0, const void* in1, void* out_vals,
           uint8_t* out_flags, const uint8_t* todo, cudaStream_t s)
    {
        switch (b->threads)
        {
            case 128:
                return go<OP, 128>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            case 512:
                return go<OP, 512>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            default:
                return go<OP, 256>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
        }
    }

    static sg_status
    run(sg_table_batch* b, int op, const int64_t* offsets, const void* in0, const void* in1, void* out_vals,
        uint8_t* out_flags, const uint8_t* todo, cudaStream_t s)
    {
        switch (op)
        {
            case kOpInsertAos:
                return run_op<kOpInsertAos>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            case kOpInsertSoa:
                return run_op<kOpInsertSoa>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            case kOpErase:
                return run_op<kOpErase>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            case kOpFind:
                return run_op<kOpFind>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
            default:
                return run_op<kOpContains>(b, offsets, in0, in1, out_vals, out_flags, todo, s);
        }
    }

    // The tables of an insert that are built; the others are marked todo for the probe kernel.
    template <bool AOS>
    static sg_status
    build(sg_table_batch* b, const int64_t* offsets, const void* in0, const void* in1, uint8_t* out_flags,
          cudaStream_t s)
    {
        using Lists = list_tile<typename slot_image<KIND>::type, kListPer>;
        // once: a call to set an attribute takes a microsecond of the host's time
        static const cudaError_t shared_set = [] {
            constexpr cudaFuncAttribute kShared = cudaFuncAttributeMaxDynamicSharedMemorySize;
            cudaError_t e = cudaFuncSetAttribute(k_batch_lists<KIND, AOS>, kShared, static_cast<int>(sizeof(Lists)));
            e = e != cudaSuccess ? e
                                 : cudaFuncSetAttribute(k_batch_build<KIND, AOS, true>, kShared,
                                                        static_cast<int>(kRegionBytes));
            return e != cudaSuccess ? e
                                    : cudaFuncSetAttribute(k_batch_build<KIND, AOS, false>, kShared,
                                                           static_cast<int>(kRegionBytes));
        }();
        SG_CUDA_TRY(shared_set);
        uint8_t* const todo = b->marks + b->n;
        build_words* const words = words_of(b->fill, b->n_items);
        SG_CUDA_TRY(cudaMemsetAsync(b->fill, 0, fill_bytes(b->n_items), s));
        SG_CUDA_TRY(launch_early(k_batch_choose, grid_for(b->n, 1024, b->sms), 1024, s, b->views, offsets, b->n, b->first_item,
                                 out_flags != nullptr, kListPer * kListThreads, b->sms * kRegionBlocks, b->marks, todo,
                                 b->list_prefix, b->prefix, words));
        SG_LAUNCH_CHECK();
        static const int lists_grid = persistent_grid(k_batch_lists<KIND, AOS>, kListThreads, sizeof(Lists));
        static const int build_grid =
                persistent_grid(k_batch_build<KIND, AOS, true>, kRegionThreads, kRegionBytes);
        const bool ordered = b->n_items > build_grid;
        SG_CUDA_TRY(launch_early_shared(k_batch_lists<KIND, AOS>, lists_grid, kListThreads, sizeof(Lists), s, b->views,
                                        offsets, b->list_prefix, b->n, b->first_item, b->items,
                                        static_cast<int32_t>(b->n_items), b->marks, b->prefix,
                                        ordered ? b->order : nullptr, b->fill, todo, in0, in1));
        b->torn = true;
        SG_LAUNCH_CHECK();
        if (ordered)
        {
            SG_CUDA_TRY(launch_early_shared(k_batch_build<KIND, AOS, true>, build_grid, kRegionThreads, kRegionBytes, s,
                                            b->views, offsets, b->order, b->prefix + b->n, b->marks, &words->taken,
                                            b->fill, todo, in0, in1, out_flags, b->spills));
        }
        else
        {
            SG_CUDA_TRY(launch_early_shared(k_batch_build<KIND, AOS, false>, static_cast<int>(b->n_items),
                                            kRegionThreads, kRegionBytes, s, b->views, offsets, b->items, nullptr,
                                            b->marks, nullptr, b->fill, todo, in0, in1, out_flags, b->spills));
        }
        SG_LAUNCH_CHECK();
        b->torn = false;
        return SG_OK;
    }

    static sg_status
    init(sg_table_batch* b, cudaStream_t s)
    {
        if (b->in_regions && b->arena_bytes <= kClearArenaMax)
        {
            static const int grid = persistent_grid(k_batch_clear<KIND>, 256);
            SG_CUDA_TRY(launch_early(k_batch_clear<KIND>, static_cast<int>(std::min<int64_t>(b->n_items, grid)), 256, s,
                                     b->views, b->items, static_cast<int32_t>(b->n_items)));
            SG_LAUNCH_CHECK();
            return SG_OK;
        }
        SG_CUDA_TRY(cudaMemsetAsync(b->arena, 0xFF, static_cast<size_t>(b->arena_bytes), s));
        k_batch_reset<KIND><<<(b->n + 255) / 256, 256, 0, s>>>(b->views, b->n);
        SG_LAUNCH_CHECK();
        return SG_OK;
    }
};

template <int KIND>
sg_status
build_kind(sg_table_batch* b, bool aos, const int64_t* offsets, const void* in0, const void* in1, uint8_t* out_flags,
           cudaStream_t s)
{
    return aos ? batch_launch<KIND>::template build<true>(b, offsets, in0, in1, out_flags, s)
               : batch_launch<KIND>::template build<false>(b, offsets, in0, in1, out_flags, s);
}

sg_status
dispatch_build(sg_table_batch* b, bool aos, const int64_t* offsets, const void* in0, const void* in1,
               uint8_t* out_flags, cudaStream_t s)
{
    switch (b->kind)
    {
        case 0:
            return build_kind<0>(b, aos, offsets, in0, in1, out_flags, s);
        case 1:
            return build_kind<1>(b, aos, offsets, in0, in1, out_flags, s);
        case 2:
            return build_kind<2>(b, aos, offsets, in0, in1, out_flags, s);
        case 3:
            return build_kind<3>(b, aos, offsets, in0, in1, out_flags, s);
        case 4:
            return build_kind<4>(b, aos, offsets, in0, in1, out_flags, s);
        case 5:
            return build_kind<5>(b, aos, offsets, in0, in1, out_flags, s);
        default:
            return SG_ERR_BAD_ARG;
    }
}

sg_status
dispatch_op(sg_table_batch* b, int op, const int64_t* offsets, const void* in0, const void* in1, void* out_vals,
            uint8_t* out_flags, cudaStream_t s)
{
    if (b->torn)
    {
        return SG_ERR_CUDA; // until clear()
    }
    const bool insert = op == kOpInsertAos || op == kOpInsertSoa;
    const bool build = insert && b->maybe_empty && in0 != nullptr && b->n_items > 0;
    if (insert && in0 != nullptr)
    {
        b->maybe_empty = false;
    }
    if (build)
    {
        const sg_status st = dispatch_build(b, op == kOpInsertAos, offsets, in0, in1, out_flags, s);
        if (st != SG_OK)
        {
            return st;
        }
    }
    // the tables whose keys are walked (all, without a build)
    const uint8_t* todo = build ? b->marks + b->n : nullptr;
    // a NULL key array (all ranges empty, as an empty tensor gives) walks no tile
    SG_CUDA_TRY(launch_early(k_batch_tiles, 1, 1024, s, offsets, b->n, b->prefix, in0 != nullptr, todo));
    SG_LAUNCH_CHECK();
    switch (b->kind)
    {
        case 0:
            return batch_launch<0>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        case 1:
            return batch_launch<1>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        case 2:
            return batch_launch<2>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        case 3:
            return batch_launch<3>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        case 4:
            return batch_launch<4>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        case 5:
            return batch_launch<5>::run(b, op, offsets, in0, in1, out_vals, out_flags, todo, s);
        default:
            return SG_ERR_BAD_ARG;
    }
}

sg_status
dispatch_init(sg_table_batch* b, cudaStream_t s)
{
    switch (b->kind)
    {
        case 0:
            return batch_launch<0>::init(b, s);
        case 1:
            return batch_launch<1>::init(b, s);
        case 2:
            return batch_launch<2>::init(b, s);
        case 3:
            return batch_launch<3>::init(b, s);
        case 4:
            return batch_launch<4>::init(b, s);
        case 5:
            return batch_launch<5>::init(b, s);
        default:
            return SG_ERR_BAD_ARG;
    }
}

bool
args_ok(const sg_table_batch* b, const void* in0, const int64_t* offsets)
{
    (void)in0; // NULL keys are allowed: the call then walks no tile
    return b != nullptr && offsets != nullptr;
}

} // namespace

extern "C" {

sg_status
sg_batch_create(int32_t kind, int32_t n_tables, const int64_t* capacities, void* stream, sg_table_batch** out)
{
    if (out == nullptr || capacities == nullptr || n_tables <= 0 || kind < SG_SET_U32 || kind > SG_MAP_U32_U64)
    {
        return SG_ERR_BAD_ARG;
    }
    *out = nullptr;
    auto* b = new (std::nothrow) sg_table_batch{};
    if (b == nullptr)
    {
        return SG_ERR_OOM;
    }
    b->kind = kind;
    b->n = n_tables;
    b->threads = 256;
    b->blocks_per_sm = 0;
    b->tiles_per_step = 1;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
    b->capacities.assign(capacities, capacities + n_tables);
    std::vector<int64_t> group_offset(n_tables + 1, 0);
    std::vector<int> bits(n_tables);
    std::vector<int64_t> groups(n_tables);
    b->bucket_counts.resize(n_tables);
    b->totals.resize(n_tables);
    for (int32_t t = 0; t < n_tables; ++t)
    {
        if (capacities[t] <= 0)
        {
            delete b;
            return SG_ERR_BAD_ARG;
        }
        batch_geometry(capacities[t], kind, &b->bucket_counts[t], &b->totals[t], &groups[t], &bits[t]);
        if (b->totals[t] >= (int64_t{ 1 } << 31))
        {
            delete b;
            return SG_ERR_BAD_ARG;
        }
        group_offset[t + 1] = group_offset[t] + groups[t] + 1; // + tail group of out-of-band keys
    }
    b->arena_bytes = group_offset[n_tables] * kGroupBytes;
    b->in_regions = true;
    std::vector<build_item> items;
    std::vector<int32_t> first_item(n_tables + 1, 0);
    for (int32_t t = 0; t < n_tables; ++t)
    {
        const int64_t regions = (groups[t] + kRegionGroups - 1) / kRegionGroups;
        // (larger tables have no regions: their inserts fill the chip on their own)
        b->in_regions = b->in_regions && regions <= kListRegions;
        for (int64_t k = 0; regions <= kListRegions && k < regions; ++k)
        {
            const int64_t g = k * kRegionGroups;
            items.push_back(build_item{ t, static_cast<uint32_t>(g),
                                        static_cast<uint32_t>(std::min<int64_t>(groups[t] - g, kRegionGroups)),
                                        regions == 1 ? -1 : static_cast<int32_t>(items.size()) });
        }
        first_item[t + 1] = static_cast<int32_t>(items.size());
    }
    b->n_items = static_cast<int64_t>(items.size());
    cudaError_t e = sg::detail::dev_malloc(&b->arena, static_cast<size_t>(b->arena_bytes));
    if (e == cudaSuccess)
    {
        e = sg::detail::dev_malloc(&b->headers, sizeof(table_header) * n_tables);
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::dev_malloc(&b->views, sizeof(dview) * n_tables);
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::dev_malloc(&b->prefix, sizeof(int64_t) * (n_tables + 1));
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::dev_malloc(&b->sizes_dev, sizeof(long long) * n_tables);
    }
    if (e == cudaSuccess)
    {
        e = cudaMallocHost(&b->sizes_host, sizeof(long long) * n_tables);
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::dev_malloc(&b->locks, sizeof(unsigned int) * kBatchInsertLocks);
    }
    // what inserts into empty tables need, in one block (a batch of 64 tables of 1000 is created and destroyed in
    // 766 us; 852 with seven allocations here instead of one): the items and the tables' first ones, copied from the
    // host as one piece, then the arrays of a call.  Only regions that are not all of their table spill.
    size_t build_bytes = 0;
    const auto piece = [&build_bytes](size_t bytes) {
        const size_t at = build_bytes;
        build_bytes += (bytes + 255) / 256 * 256;
        return at;
    };
    const bool lists = std::any_of(items.begin(), items.end(), [](const build_item& it) { return it.list >= 0; });
    const size_t at_items = piece(sizeof(build_item) * items.size());
    const size_t at_first = piece(sizeof(int32_t) * first_item.size());
    const size_t from_host = build_bytes;
    const size_t at_order = piece(sizeof(build_item) * items.size());
    const size_t at_fill = piece(fill_bytes(b->n_items));
    const size_t at_prefix = piece(sizeof(int64_t) * (static_cast<size_t>(n_tables) + 1));
    const size_t at_marks = piece(2 * static_cast<size_t>(n_tables));
    const size_t at_spills = piece(lists ? sizeof(spill_entry) * kSpillMax : 0);
    std::vector<char> host_block(from_host);
    if (!items.empty())
    {
        std::memcpy(host_block.data() + at_items, items.data(), sizeof(build_item) * items.size());
        std::memcpy(host_block.data() + at_first, first_item.data(), sizeof(int32_t) * first_item.size());
        if (e == cudaSuccess)
        {
            e = sg::detail::dev_malloc(&b->build_block, build_bytes);
        }
        if (e == cudaSuccess)
        {
            b->items = reinterpret_cast<build_item*>(b->build_block + at_items);
            b->first_item = reinterpret_cast<int32_t*>(b->build_block + at_first);
            b->order = reinterpret_cast<build_item*>(b->build_block + at_order);
            b->fill = reinterpret_cast<unsigned int*>(b->build_block + at_fill);
            b->list_prefix = reinterpret_cast<int64_t*>(b->build_block + at_prefix);
            b->marks = reinterpret_cast<uint8_t*>(b->build_block + at_marks);
            b->spills.count = &words_of(b->fill, b->n_items)->spilled;
            b->spills.entry = reinterpret_cast<spill_entry*>(b->build_block + at_spills);
        }
    }
    if (e == cudaSuccess)
    {
        e = cudaMemsetAsync(b->locks, 0, sizeof(unsigned int) * kBatchInsertLocks, as_stream(stream));
    }
    if (e != cudaSuccess)
    {
        sg_batch_destroy(b);
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? SG_ERR_OOM : SG_ERR_CUDA;
    }
    b->host_views.resize(n_tables);
    for (int32_t t = 0; t < n_tables; ++t)
    {
        b->host_views[t] = dview{ b->arena + group_offset[t] * kGroupBytes, b->headers + t,
                                  static_cast<uint32_t>(groups[t]), static_cast<uint32_t>(b->totals[t]), bits[t] };
    }
    cudaStream_t s = as_stream(stream);
    e = cudaMemcpyAsync(b->views, b->host_views.data(), sizeof(dview) * n_tables, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !items.empty())
    {
        e = cudaMemcpyAsync(b->build_block, host_block.data(), from_host, cudaMemcpyHostToDevice, s);
    }
    if (e == cudaSuccess)
    {
        e = cudaStreamSynchronize(s); // host vectors above are released on return
    }
    if (e != cudaSuccess)
    {
        sg_batch_destroy(b);
        return SG_ERR_CUDA;
    }
    const sg_status st = dispatch_init(b, s);
    if (st != SG_OK)
    {
        sg_batch_destroy(b);
        return st;
    }
    b->maybe_empty = true;
    *out = b;
    return SG_OK;
}

sg_status
sg_batch_destroy(sg_table_batch* b)
{
    if (b == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaDeviceSynchronize();
    sg::detail::dev_free(b->arena);
    sg::detail::dev_free(b->headers);
    sg::detail::dev_free(b->views);
    sg::detail::dev_free(b->prefix);
    sg::detail::dev_free(b->sizes_dev);
    sg::detail::dev_free(b->locks);
    sg::detail::dev_free(b->build_block);
    if (b->sizes_host != nullptr)
    {
        cudaFreeHost(b->sizes_host);
    }
    delete b;
    return SG_OK;
}

sg_status
sg_batch_configure(sg_table_batch* b, int32_t threads_per_block, int32_t blocks_per_sm, int32_t tiles_per_step)
{
    if (b == nullptr || (threads_per_block != 128 && threads_per_block != 256 && threads_per_block != 512) ||
        blocks_per_sm < 0 || tiles_per_step < 1 || tiles_per_step > 64)
    {
        return SG_ERR_BAD_ARG;
    }
    b->threads = threads_per_block;
    b->blocks_per_sm = blocks_per_sm;
    b->tiles_per_step = tiles_per_step;
    return SG_OK;
}

sg_status
sg_batch_clear(sg_table_batch* b, void* stream)
{
    if (b == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    const sg_status st = dispatch_init(b, as_stream(stream));
    b->maybe_empty = b->maybe_empty || st == SG_OK;
    b->torn = b->torn && st != SG_OK;
    return st;
}

sg_status
sg_batch_insert(sg_table_batch* b, const void* values, const int64_t* offsets, uint8_t* out_inserted, void* stream)
{
    if (!args_ok(b, values, offsets))
    {
        return SG_ERR_BAD_ARG;
    }
    return dispatch_op(b, kOpInsertAos, offsets, values, nullptr, nullptr, out_inserted, as_stream(stream));
}

sg_status
sg_batch_insert_kv(sg_table_batch* b, const void* keys, const void* mapped, const int64_t* offsets,
                   uint8_t* out_inserted, void* stream)
{
    if (!args_ok(b, keys, offsets))
    {
        return SG_ERR_BAD_ARG;
    }
    return dispatch_op(b, kOpInsertSoa, offsets, keys, mapped, nullptr, out_inserted, as_stream(stream));
}

sg_status
sg_batch_erase(sg_table_batch* b, const void* keys, const int64_t* offsets, uint8_t* out_erased, void* stream)
{
    if (!args_ok(b, keys, offsets))
    {
        return SG_ERR_BAD_ARG;
    }
    return dispatch_op(b, kOpErase, offsets, keys, nullptr, nullptr, out_erased, as_stream(stream));
}

sg_status
sg_batch_find(sg_table_batch* b, const void* keys, const int64_t* offsets, void* out_mapped, uint8_t* out_found,
              void* stream)
{
    if (!args_ok(b, keys, offsets))
    {
        return SG_ERR_BAD_ARG;
    }
    const bool is_map = b->kind >= SG_MAP_U64_U32;
    return dispatch_op(b, kOpFind, offsets, keys, nullptr, is_map ? out_mapped : nullptr, out_found,
                       as_stream(stream));
}

sg_status
sg_batch_contains(sg_table_batch* b, const void* keys, const int64_t* offsets, uint8_t* out_flags, void* stream)
{
    if (!args_ok(b, keys, offsets) || (keys != nullptr && out_flags == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    return dispatch_op(b, kOpContains, offsets, keys, nullptr, nullptr, out_flags, as_stream(stream));
}

sg_status
sg_batch_sizes(sg_table_batch* b, void* stream, int64_t* out_sizes)
{
    if (b == nullptr || out_sizes == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaStream_t s = as_stream(stream);
    // by way of device memory: thousands of stores into host memory take the kernel longer than the copy
    k_batch_gather_sizes<<<(b->n + 255) / 256, 256, 0, s>>>(b->views, b->n, b->sizes_dev);
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(cudaMemcpyAsync(b->sizes_host, b->sizes_dev, sizeof(long long) * b->n, cudaMemcpyDeviceToHost, s));
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    for (int32_t t = 0; t < b->n; ++t)
    {
        out_sizes[t] = static_cast<int64_t>(b->sizes_host[t]);
    }
    return SG_OK;
}

sg_status
sg_batch_view_of(const sg_table_batch* b, int32_t table, sg_unordered_view* out)
{
    if (b == nullptr || out == nullptr || table < 0 || table >= b->n)
    {
        return SG_ERR_BAD_ARG;
    }
    const dview& v = b->host_views[table];
    out->slots = v.slots;
    out->header = v.hdr;
    out->num_groups = v.num_groups;
    out->total_count = v.total;
    out->bucket_count = b->bucket_counts[table];
    out->bucket_bits = v.bits;
    out->kind = b->kind;
    out->insert_locks = b->locks;
    out->lock_mask = kBatchInsertLocks - 1;
    return SG_OK;
}

sg_status
sg_batch_info(const sg_table_batch* b, int64_t* out_storage_bytes, int32_t* out_n_tables)
{
    if (b == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    if (out_storage_bytes != nullptr)
    {
        *out_storage_bytes = b->arena_bytes;
    }
    if (out_n_tables != nullptr)
    {
        *out_n_tables = b->n;
    }
    return SG_OK;
}

} // extern "C"
