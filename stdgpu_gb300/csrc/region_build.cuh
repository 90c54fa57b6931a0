// Bulk insert into a table that holds nothing, built in shared memory.
//
// The probe kernels insert with one read of a 128-byte group and one compare-and-swap per key in L2 or DRAM: two
// round trips and about 19 warp instructions per key, which keeps them well below the memory's rate when a table is
// filled.  Here the keys are first written, region by region of whole probe groups, into the regions' own slots (the
// table is empty, so its slots are free to hold the lists); then a block takes a region, starts it in its shared
// memory as clear() leaves it, inserts the region's list there and writes the region out in whole lines.
//
// Only for tables known to hold nothing (no key, no erased slot): every slot below total_count is never used, a key
// goes to the first never-used slot of its home group in the key's rotated order, else of the next group, which is the
// rule of the probe kernels (insert_kv_place), and no slot has to be looked at twice.  A key whose groups are full up
// to the region's end is left to the probe kernels (a spill).
#ifndef SG_REGION_BUILD_CUH
#define SG_REGION_BUILD_CUH

#include <cuda_runtime.h>

#include <cstdint>

#include "table_core.cuh"

namespace sg
{
namespace detail
{

// 256 groups: 32 KB of shared memory and 256 threads, 6 blocks per SM.  Building the 4096 tables of the batched case
// (0.85 GB of slots) took 276 us so, 308 us with twice the region and block, 259 us with half of them, but then the
// lists' launch took 211 us instead of 199 and every table had twice the regions to keep.
constexpr uint32_t kRegionGroupsLog2 = 8;
constexpr int kRegionThreads = 256;
constexpr int kRegionBlocks = 1536 / kRegionThreads; // per SM
constexpr int kListThreads = 512;
constexpr uint32_t kRegionGroups = 1u << kRegionGroupsLog2;
constexpr size_t kRegionBytes = size_t{ kRegionGroups } * kGroupBytes;

// Groups [first, first + count) of a table, in the block's shared memory.
struct region
{
    char* smem;
    uint32_t first;
    uint32_t count;
    bool whole; // the table's every group: the probe sequence wraps inside the region
};

enum region_result : int
{
    kRegionPresent = 0,
    kRegionInserted = 1,
    kRegionRefused = 2, // the whole table is full
    kRegionSpill = 3    // no free slot up to the region's end
};

template <typename K>
SG_D K
shared_cas(char* p, K expected, K desired)
{
    if constexpr (sizeof(K) == 8)
    {
        return static_cast<K>(atomicCAS(reinterpret_cast<unsigned long long*>(p),
                                        static_cast<unsigned long long>(expected),
                                        static_cast<unsigned long long>(desired)));
    }
    else
    {
        return static_cast<K>(atomicCAS(reinterpret_cast<unsigned int*>(p), static_cast<unsigned int>(expected),
                                        static_cast<unsigned int>(desired)));
    }
}

// Inserts key into the region from its home group first + l on.  The claim is a compare-and-swap of the key word; the
// mapped value is stored after it (nothing reads values before the region is written out).  Copies of one key walk
// the same slots, and a slot once taken stays so, so one copy is inserted.
template <int KIND>
SG_D int
region_insert(const region& r, uint32_t l, uint32_t rot, typename kind_consts<KIND>::K key,
              typename kind_consts<KIND>::V val)
{
    using C = kind_consts<KIND>;
    using K = typename C::K;
    constexpr uint32_t G = C::slots_per_group;
    for (uint32_t probes = 0; probes < r.count; ++probes)
    {
        char* const group = r.smem + (l << 7);
#pragma unroll 1
        for (uint32_t k = 0; k < G; ++k)
        {
            char* const slot = group + ((rot + k) & (G - 1)) * C::slot_bytes;
            const K cur = shared_cas<K>(slot, C::empty_key, key);
            if (cur == C::empty_key)
            {
                if constexpr (kind_traits<KIND>::is_map)
                {
                    *reinterpret_cast<typename C::V*>(slot + kind_traits<KIND>::val_offset) = val;
                }
                return kRegionInserted;
            }
            if (cur == key)
            {
                return kRegionPresent;
            }
        }
        if (++l == r.count)
        {
            if (!r.whole)
            {
                return kRegionSpill;
            }
            l = 0;
        }
    }
    return kRegionRefused;
}

// The 16-byte unit whose first slot is s0 as clear() leaves it: never-used slots, and erased markers at or above
// total_count.
template <int KIND>
SG_D uint4
cleared_unit(const dview& t, uint32_t s0)
{
    using C = kind_consts<KIND>;
    using K = typename C::K;
    uint4 d = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (s0 + C::slots_per_lane > t.total)
    {
        char* bytes = reinterpret_cast<char*>(&d);
        for (int s = 0; s < C::slots_per_lane; ++s)
        {
            if (s0 + s >= t.total)
            {
                *reinterpret_cast<K*>(bytes + s * C::slot_bytes) = C::tomb_key;
            }
        }
    }
    return d;
}

// The region as clear() leaves it.
template <int KIND>
SG_D void
region_start(const dview& t, const region& r)
{
    using C = kind_consts<KIND>;
    uint4* const smem = reinterpret_cast<uint4*>(r.smem);
    const uint32_t first_slot = r.first * C::slots_per_group;
    const bool whole_slots = first_slot + r.count * C::slots_per_group <= t.total;
    for (uint32_t u = threadIdx.x; u < r.count * (kGroupBytes / 16); u += blockDim.x)
    {
        smem[u] = whole_slots ? make_uint4(~0u, ~0u, ~0u, ~0u)
                              : cleared_unit<KIND>(t, first_slot + u * C::slots_per_lane);
    }
}

// The region to the table.
SG_D void
region_write(const dview& t, const region& r)
{
    const uint4* const smem = reinterpret_cast<const uint4*>(r.smem);
    uint4* const out = reinterpret_cast<uint4*>(t.slots + (static_cast<uint64_t>(r.first) << 7));
    for (uint32_t u = threadIdx.x; u < r.count * (kGroupBytes / 16); u += blockDim.x)
    {
        out[u] = smem[u];
    }
}

// Sums of 32-bit counts over the block, added to *dst[k] by one thread each.
template <int N>
SG_D void
region_add(unsigned int (&v)[N], unsigned long long* const (&dst)[N])
{
    __shared__ unsigned int sum[N];
    if (threadIdx.x < N)
    {
        sum[threadIdx.x] = 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        const unsigned int s = __reduce_add_sync(0xffffffffu, v[k]);
        if ((threadIdx.x & 31) == 0 && s != 0u)
        {
            atomicAdd(&sum[k], s);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        if (threadIdx.x == k && sum[k] != 0u)
        {
            atomicAdd(dst[k], static_cast<unsigned long long>(sum[k]));
        }
    }
}

// ---------------------------------------------------------------- lists of a tile's elements
// A block's tile of up to PER x kListThreads elements, element j * kListThreads + threadIdx.x being item j of the
// thread, sorted by region in shared memory and appended to the regions' lists, so that each list's stores are runs.
// regions <= kListRegions.

constexpr int kListRegions = 1024;

template <typename E, int PER>
struct list_tile
{
    E stage[PER * kListThreads];
    uint16_t rid[PER * kListThreads];
    unsigned int cnt[kListRegions];  // elements of the tile per region
    unsigned int off[kListRegions];  // where they start in the stage
    unsigned int base[kListRegions]; // and in the region's list
    unsigned int warp[kListThreads / 32];
};

// rid[j] < 0: no element.  fill[r]: elements offered to list r (may exceed its capacity); at(r, k) the address of
// element k of list r; cap(r) its capacity.  Returns whether an element found no room (it is not stored).
template <typename E, int PER, typename At, typename Cap>
SG_D bool
append_to_lists(list_tile<E, PER>& s, int regions, const E (&elem)[PER], const int (&rid)[PER], unsigned int* fill,
                At at, Cap cap)
{
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    __syncthreads(); // the previous tile's stage is written out
    for (int r = threadIdx.x; r < regions; r += kListThreads)
    {
        s.cnt[r] = 0u;
    }
    __syncthreads();
    unsigned int rank[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j)
    {
        rank[j] = rid[j] >= 0 ? atomicAdd(&s.cnt[rid[j]], 1u) : 0u;
    }
    __syncthreads();
    // exclusive scan of the counts, two per thread, and a reservation in each list
    static_assert(kListRegions <= 2 * kListThreads, "two counts per thread");
    unsigned int c[2], sum = 0u;
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
        const int r = 2 * static_cast<int>(threadIdx.x) + k;
        c[k] = r < regions ? s.cnt[r] : 0u;
        sum += c[k];
    }
    unsigned int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
    {
        const unsigned int x = __shfl_up_sync(0xffffffffu, incl, d);
        incl += lane >= d ? x : 0u;
    }
    if (lane == 31)
    {
        s.warp[warp] = incl;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
        const int r = 2 * static_cast<int>(threadIdx.x) + k;
        if (c[k] != 0u)
        {
            s.base[r] = atomicAdd(fill + r, c[k]);
        }
    }
    __syncthreads();
    unsigned int run = incl - sum, count = 0u;
#pragma unroll
    for (int w = 0; w < kListThreads / 32; ++w)
    {
        run += w < warp ? s.warp[w] : 0u;
        count += s.warp[w];
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
        const int r = 2 * static_cast<int>(threadIdx.x) + k;
        if (r < regions)
        {
            s.off[r] = run;
            run += c[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j)
    {
        if (rid[j] >= 0)
        {
            const unsigned int pos = s.off[rid[j]] + rank[j];
            s.stage[pos] = elem[j];
            s.rid[pos] = static_cast<uint16_t>(rid[j]);
        }
    }
    __syncthreads();
    bool lost = false;
    for (unsigned int e = threadIdx.x; e < count; e += kListThreads)
    {
        const int r = s.rid[e];
        const unsigned int k = s.base[r] + (e - s.off[r]);
        if (k < cap(r))
        {
            *at(r, k) = s.stage[e];
        }
        else
        {
            lost = true;
        }
    }
    return lost;
}

} // namespace detail
} // namespace sg

#endif
