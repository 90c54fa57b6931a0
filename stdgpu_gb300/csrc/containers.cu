// vector<T>::push_back, deque<T>::push_back / pop_front and bitset::count for GB300.
//
// vector / deque replace the reference's per-element global atomic plus slot
// spin lock (src/stdgpu/impl/vector_detail.cuh:181-238,
// src/stdgpu/impl/deque_detail.cuh:202-258, 388-446).  A vector reserves once
// per tile of up to 8192 elements (a counter that every warp hits once saturates
// near 0.5 G updates a second on one address); a deque's mixed call counts its
// pushes first, which settles every element's ticket without a reservation.
//
// The deque is a ring of tickets: push k and pop k use slot k mod capacity; a
// per-slot turn counter (the k-th push stores k+1 after writing the element,
// the k-th pop stores k+capacity after reading it) orders a pop after the push
// of the same ticket and a push after the pop one lap earlier.  Only small rings
// and mixed calls of more elements than slots order their launches by the turn
// words.  Those waits are bounded: a wait that runs out sets an error bit and the operation reports
// failure instead of spinning on.
//
// bitset::count (src/stdgpu/impl/bitset_detail.cuh:388-404, count_block_bits
// :130-160) is a two-pass reduction: 16-byte loads and popc per thread, one
// partial per block, then one block sums the partials.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <new>

#include "sg_internal.cuh"
#include "stdgpu_gb300.h"
#include "stdgpu_gb300/detail/layout.cuh"

namespace sg
{
namespace detail
{

constexpr int kCThreads = 256;
SG_D unsigned
lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <typename T>
SG_D T
ld_stream(const T* p)
{
    return __ldcs(p);
}

// A ring slot's turn word read without ordering (a fence_gpu after the reads orders what follows), and
// stored without ordering (a fence_gpu before the stores orders what precedes).
SG_D unsigned
load_turn_relaxed(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

SG_D void
store_turn_relaxed(unsigned* p, unsigned v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

SG_D void
fence_gpu()
{
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

// ---------------------------------------------------------------- block reservations
//
// A block takes a tile of kItems x kCThreads elements, element tile + j * kCThreads + threadIdx.x being
// item j of the thread.  Each warp ballots its items and writes one count per (item, warp) into shared
// memory in element order; one warp scans the kItems * kWarps counts, so every element learns its rank
// among the tile's selected elements and the tile makes one reservation on the shared counter.

constexpr int kItems = 8;
constexpr int kWarps = kCThreads / 32;
constexpr int kCounts = kItems * kWarps; // 64: two per lane of the scanning warp
constexpr int64_t kTileElems = int64_t{ kItems } * kCThreads;
static_assert(kCounts == 64, "the scan gives each lane two counts");

// Exclusive scan of cnt[0, 64) in place by one warp; returns the total to every lane.
SG_D unsigned
scan_counts(unsigned* cnt, int lane)
{
    const unsigned a = cnt[2 * lane];
    const unsigned b = cnt[2 * lane + 1];
    unsigned s = a + b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
    {
        const unsigned t = __shfl_up_sync(0xffffffffu, s, d);
        if (lane >= d)
        {
            s += t;
        }
    }
    const unsigned excl = s - a - b;
    cnt[2 * lane] = excl;
    cnt[2 * lane + 1] = excl + a;
    return __shfl_sync(0xffffffffu, s, 31);
}

// True in every thread of the last block to arrive here (`arrived` 0 before the launch, and again after it): that
// block's threads see what all blocks wrote before they arrived.
SG_D bool
last_block(unsigned int* arrived)
{
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
        if (last)
        {
            *arrived = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    return last;
}

// Bit j set when byte j of x is not zero.
SG_D unsigned
nonzero_bytes(unsigned x)
{
    return ((__vsetne4(x, 0u) * 0x10204080u) >> 28) & 0xFu;
}

// ---------------------------------------------------------------- vector

// Control word of a vector's launches, behind the sync words of its device calls.
struct vector_control
{
    unsigned int arrived; // last_block
};
constexpr size_t kControlOffset = 64;
constexpr size_t kSyncBytes = 256;

// Size and device-call state at the end of a bulk call: the size clamped into [0, capacity] after `minus`
// elements are taken from its back, the device calls' epoch advanced and the size it starts from recorded.
SG_D void
vector_call_ends(long long* size, int64_t cap, int64_t minus, sg_vector_sync* sync, uint32_t epoch)
{
    long long s = __ldcg(size);
    s = s < 0 ? 0 : (s > cap ? cap : s);
    s = s > minus ? s - minus : 0;
    *size = s;
    sync->base_size = s;
    sync->epoch = epoch;
}

// Bulk push_back: element i pushes values[i] where pred[i] != 0 (every element without pred).  A warp takes ROWS
// rows of 32 elements: its lanes read the predicate bytes of consecutive elements, so a lane soon holds a whole
// row's mask; the block makes one reservation on the size for all its rows, and only then are the selected values
// read, eight rows of loads in flight.  A reservation past capacity fails the elements there, as the reference's
// push_back fails past capacity() (its size is clamped when read, vector_detail.cuh:484-511).
//
// What bounds it: at 32 rows (8192 elements per reservation) the memory; below that the reservations, updates of one
// address that complete at about 0.5 G a second.  2^26 threads, 8-byte elements, 30 % pushed, with flags:
// 130 us, 179 us with one reservation per 1024 elements and the values read before it (4-byte elements 99 / 179).
// Launches below kVecLargeTile take 4 rows (1024 elements per block), which spreads them over more SMs.
template <typename T, int ROWS>
__global__ void __launch_bounds__(kCThreads)
k_vector_push_back(T* data, long long* size, int64_t cap, const T* values, const uint8_t* pred, int64_t n,
                   uint8_t* out_pushed, sg_vector_sync* sync, uint32_t epoch, vector_control* ctl)
{
    wait_for_stream();
    static_assert(ROWS == 4 || ROWS == 32, "a lane reads 4 or 32 predicate bytes");
    constexpr int64_t kWarpElems = ROWS * 32;
    constexpr int64_t kTile = kWarpElems * kWarps;
    __shared__ unsigned warp_total[2][kWarps];
    __shared__ long long s_base[2];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const bool words = (reinterpret_cast<uintptr_t>(pred) % ROWS == 0 || reinterpret_cast<uintptr_t>(pred) % 16 == 0) &&
                       pred != nullptr;
    int buf = 0;
    for (int64_t tile = static_cast<int64_t>(blockIdx.x) * kTile; tile < n;
         tile += static_cast<int64_t>(gridDim.x) * kTile, buf ^= 1)
    {
        const int64_t first = tile + warp * kWarpElems; // the warp's first element
        const int64_t mine = first + lane * ROWS;       // the lane's first predicate byte
        unsigned bits = 0u;                             // of the elements mine .. mine + ROWS
        if (pred != nullptr && words && mine + ROWS <= n)
        {
            if constexpr (ROWS == 32)
            {
                const uint4 a = __ldcs(reinterpret_cast<const uint4*>(pred + mine));
                const uint4 b = __ldcs(reinterpret_cast<const uint4*>(pred + mine) + 1);
                bits = nonzero_bytes(a.x) | nonzero_bytes(a.y) << 4 | nonzero_bytes(a.z) << 8 |
                       nonzero_bytes(a.w) << 12 | nonzero_bytes(b.x) << 16 | nonzero_bytes(b.y) << 20 |
                       nonzero_bytes(b.z) << 24 | nonzero_bytes(b.w) << 28;
            }
            else
            {
                bits = nonzero_bytes(__ldcs(reinterpret_cast<const unsigned*>(pred + mine)));
            }
        }
        else
        {
            for (int j = 0; j < ROWS; ++j)
            {
                bits |= static_cast<unsigned>(mine + j < n && (pred == nullptr || pred[mine + j] != 0)) << j;
            }
        }
        // lane r (r < ROWS): the mask of row r
        unsigned row;
        if constexpr (ROWS == 32)
        {
            row = bits;
        }
        else
        {
            row = 0u;
#pragma unroll
            for (int k = 0; k < 8; ++k)
            {
                row |= __shfl_sync(0xffffffffu, bits, ((lane * 8) & 31) + k) << (4 * k);
            }
            row = lane < ROWS ? row : 0u;
        }
        const unsigned c = static_cast<unsigned>(__popc(row));
        unsigned incl = c;
#pragma unroll
        for (int d = 1; d < ROWS; d <<= 1)
        {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d)
            {
                incl += t;
            }
        }
        if (lane == ROWS - 1)
        {
            warp_total[buf][warp] = incl;
        }
        __syncthreads();
        unsigned before = 0u;
        unsigned total = 0u;
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
        {
            const unsigned x = warp_total[buf][w];
            before += w < warp ? x : 0u;
            total += x;
        }
        if (threadIdx.x == 0)
        {
            // one reservation for the tile (vector_detail.cuh:186-195)
            s_base[buf] = total > 0 ? static_cast<long long>(atomicAdd(reinterpret_cast<unsigned long long*>(size),
                                                                       static_cast<unsigned long long>(total)))
                                    : 0;
        }
        __syncthreads();
        const long long base = s_base[buf] + before;
        const unsigned row_before = incl - c;
        constexpr int kFlight = ROWS < 8 ? ROWS : 8;
#pragma unroll 1
        for (int r0 = 0; r0 < ROWS; r0 += kFlight)
        {
            T vals[kFlight];
            unsigned masks[kFlight];
#pragma unroll
            for (int k = 0; k < kFlight; ++k)
            {
                masks[k] = __shfl_sync(0xffffffffu, row, r0 + k);
                if ((masks[k] >> lane) & 1u)
                {
                    vals[k] = ld_stream(values + first + (r0 + k) * 32 + lane);
                }
            }
#pragma unroll
            for (int k = 0; k < kFlight; ++k)
            {
                const long long pos = base + __shfl_sync(0xffffffffu, row_before, r0 + k) +
                                      __popc(masks[k] & lanemask_lt());
                const bool ok = ((masks[k] >> lane) & 1u) && pos < cap;
                if (ok)
                {
                    data[pos] = vals[k];
                }
                const int64_t i = first + (r0 + k) * 32 + lane;
                if (out_pushed != nullptr && i < n)
                {
                    out_pushed[i] = static_cast<uint8_t>(ok);
                }
            }
        }
        // no barrier: the next tile fills the other buffer, and the one after passes two barriers that every
        // warp reaches only after reading this tile's totals
    }
    if (last_block(&ctl->arrived) && threadIdx.x == 0)
    {
        vector_call_ends(size, cap, 0, sync, epoch);
    }
}

// ---------------------------------------------------------------- deque

SG_D long long
atomic_add_ll(long long* p, long long v)
{
    return static_cast<long long>(
            atomicAdd(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v)));
}

// Reserves up to `want` units of `counter` below `bound` (grow) or above zero (!grow): a preemptive read,
// one add, and an undo of what did not fit (deque_detail.cuh:207-217 push_back, :393-404 pop_front).
SG_D long long
reserve(long long* counter, long long bound, long long want, bool grow)
{
    const long long cur = *reinterpret_cast<volatile long long*>(counter);
    if (grow ? cur >= bound : cur <= 0)
    {
        return 0;
    }
    const long long old = atomic_add_ll(counter, grow ? want : -want);
    const long long room = grow ? bound - old : old;
    const long long take = room <= 0 ? 0 : (room < want ? room : want);
    if (take < want)
    {
        atomic_add_ll(counter, grow ? take - want : want - take);
    }
    return take;
}

// Mixed launch: element i pushes values[i] when is_push[i] != 0, else pops.  Each
// tile reserves its pushes and its pops once; the tile's pushes take consecutive tickets in element
// order, and so do its pops.
// resident blocks per SM the mixed deque launch is compiled for (its fast path keeps 8 tickets per thread in
// registers); measured for 2^26 mixed ops: 4 blocks 1.60 ms, 5 blocks 1.40 ms, 6 blocks 1.27 ms, and the
// one-by-one protocol alone (every element's turn waited for and released in turn) 1.60 ms
#ifndef SG_DEQUE_MIN_BLOCKS
#define SG_DEQUE_MIN_BLOCKS 6
#endif
// 0: every element takes the one-by-one path (for comparison)
#ifndef SG_DEQUE_FAST
#define SG_DEQUE_FAST 1
#endif

// What a mixed call does, settled on the device by k_deque_plan; behind the sync words of the device calls.  pushes
// and arrived are 0 between calls.
struct deque_control
{
    unsigned long long pushes;  // of the call
    unsigned long long push_t0; // first ticket of its pushes
    unsigned long long pop_t0;  // and of its pops
    long long push_ok;          // pushes that succeed, the first in element order
    long long pop_ok;           // pops that succeed
    long long held;             // of these, pops of elements stored before the call
    unsigned int arrived;       // last_block
    unsigned int apart;         // 1: no push and pop of the call meet at a slot
};

// Device-call state at the end of a bulk call: the tickets it leaves, the epoch advanced; dirty: the turn words are
// not kept (k_deque_rebuild_turns makes them before a launch that waits on them).
SG_D void
deque_call_ends(const deque_counters* c, sg_deque_sync* sync, uint32_t epoch, uint32_t dirty)
{
    sync->base_begin = c->begin;
    sync->base_end = c->end;
    sync->epoch = epoch;
    sync->dirty = dirty;
}

constexpr int kPlanTile = 2048; // elements per warp of the plan, per block of the move
static_assert(kPlanTile == kTileElems, "one count per tile of the move");

// First launch of a mixed call of at most `capacity` elements: pushes per tile of 2048 elements, turned by the last
// block into the pushes before each tile; that block then settles the call.  The order it stands for runs pushes
// while there is room and pops while there are elements, in turn, so a push fails only where the deque ends full and
// a pop only where it ends empty; pushes take the tickets from `end` on and pops those from `begin` on, in element
// order.  The launches that follow need neither turn words nor reservations; the last one moves the counters, so a
// call that breaks off between its launches leaves the deque as it was.
// counts: room for a word per tile (the turn words' array, which is marked dirty).
__global__ void __launch_bounds__(kCThreads)
k_deque_plan(const uint8_t* is_push, int64_t n, unsigned* counts, const deque_counters* c, int64_t cap,
             sg_deque_sync* sync, deque_control* ctl)
{
    wait_for_stream();
    __shared__ unsigned long long s_block;
    __shared__ unsigned s_warp[kWarps];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int64_t tiles = (n + kPlanTile - 1) / kPlanTile;
    const bool vec = reinterpret_cast<uintptr_t>(is_push) % 16 == 0;
    if (threadIdx.x == 0)
    {
        s_block = 0;
    }
    __syncthreads();
    unsigned long long mine = 0;
    for (int64_t tile = static_cast<int64_t>(blockIdx.x) * kWarps + warp; tile < tiles;
         tile += static_cast<int64_t>(gridDim.x) * kWarps)
    {
        const int64_t first = tile * kPlanTile;
        unsigned count = 0;
        if (vec && first + kPlanTile <= n)
        {
            const uint4* p = reinterpret_cast<const uint4*>(is_push + first);
#pragma unroll
            for (int k = 0; k < kPlanTile / 512; ++k)
            {
                const uint4 x = p[k * 32 + lane];
                count += __popc(__vsetne4(x.x, 0u)) + __popc(__vsetne4(x.y, 0u)) + __popc(__vsetne4(x.z, 0u)) +
                         __popc(__vsetne4(x.w, 0u));
            }
        }
        else
        {
            for (int64_t i = first + lane; i < n && i < first + kPlanTile; i += 32)
            {
                count += is_push[i] != 0;
            }
        }
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0)
        {
            counts[tile] = count;
            mine += count;
        }
    }
    if (lane == 0 && mine != 0)
    {
        atomicAdd(&s_block, mine);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_block != 0)
    {
        atomicAdd(&ctl->pushes, s_block);
    }
    if (!last_block(&ctl->arrived))
    {
        return;
    }
    // exclusive scan of the counts, kScan consecutive ones per thread at a time
    constexpr int kScan = 4;
    unsigned carry = 0;
    for (int64_t base = 0; base < tiles; base += kScan * kCThreads)
    {
        const int64_t k = base + kScan * static_cast<int64_t>(threadIdx.x);
        unsigned v[kScan];
        unsigned sum = 0;
#pragma unroll
        for (int j = 0; j < kScan; ++j)
        {
            v[j] = k + j < tiles ? __ldcg(counts + k + j) : 0u;
            sum += v[j];
        }
        unsigned incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d)
            {
                incl += t;
            }
        }
        if (lane == 31)
        {
            s_warp[warp] = incl;
        }
        __syncthreads();
        unsigned run = carry + incl - sum;
        for (int w = 0; w < kWarps; ++w)
        {
            const unsigned x = s_warp[w];
            run += w < warp ? x : 0u;
            carry += x;
        }
#pragma unroll
        for (int j = 0; j < kScan; ++j)
        {
            if (k + j < tiles)
            {
                counts[k + j] = run;
            }
            run += v[j];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        const long long pushes = static_cast<long long>(__ldcg(&ctl->pushes));
        const long long pops = n - pushes;
        const long long held = c->avail;
        const long long room = cap - held;
        ctl->pushes = 0;
        const long long net = held + pushes - pops; // elements left if all succeed
        const long long push_ok = net > cap ? pushes - (net - cap) : pushes;
        const long long pop_ok = net < 0 ? pops + net : pops;
        ctl->push_ok = push_ok;
        ctl->pop_ok = pop_ok;
        ctl->held = pop_ok < held ? pop_ok : held;
        ctl->push_t0 = c->end;
        ctl->pop_t0 = c->begin;
        ctl->apart = push_ok <= room && pop_ok <= held ? 1u : 0u;
        sync->dirty = 1u; // the counts lie where the turn words were
    }
}

// Before a launch that waits on turn words, when the last call did not keep them: every slot's word from the tickets
// -- a slot holding ticket t (t in [begin, end)) gets t + 1, a free slot the ticket of the next push_back that maps
// to it.
__global__ void
k_deque_rebuild_turns(unsigned* seq, const deque_counters* c, const sg_deque_sync* sync, int64_t cap)
{
    wait_for_stream();
    if (*reinterpret_cast<const volatile uint32_t*>(&sync->dirty) == 0u)
    {
        return;
    }
    const unsigned long long b = c->begin;
    const unsigned long long e = c->end;
    const unsigned long long ucap = static_cast<unsigned long long>(cap);
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < cap; i += stride)
    {
        const unsigned long long ui = static_cast<unsigned long long>(i);
        const unsigned long long from_b = (ui + ucap - b % ucap) % ucap; // tickets t = b + from_b map to slot i
        unsigned v;
        if (from_b < e - b)
        {
            v = static_cast<unsigned>(b + from_b + 1ull);
        }
        else
        {
            v = static_cast<unsigned>(e + (ui + ucap - e % ucap) % ucap);
        }
        seq[i] = v;
    }
}

// The launches after the plan: element i moves its element.  Its rank among the pushes (or pops) before it is its
// tile's count, its warp's and its row's, so tickets follow the element order and a row's pushes and pops go to
// consecutive slots.  An operation moves flag, value or popped value, slot and outcome, 25 bytes: 422 MB in 105 us at
// 2^24 operations, 0.6 of the measured copy rate, with 68 % of the issue slots taken; neither is full, since each load
// waits for its rank, which waits for the flags.
// kMoveFirst: pops of elements stored before the call, every outcome, and the pushes too when they meet no pop
// at a slot (the other two launches then return at once); else kMovePush and kMoveLate follow, pushes
// and then the pops of elements that the call pushed.
// 2^24 mixed operations on 8-byte elements in steady state: 116 us in all (124 before launch_early), 303 us when
// every slot's turn word was read, waited on and written (and the outputs filled before); from an empty deque, where
// each pop depends on a push of the call, 262 us against 779 us.
enum move_phase : int
{
    kMoveFirst = 0,
    kMovePush = 1,
    kMoveLate = 2
};

// Compiled for 8 resident blocks per SM, two rows in flight at a time: 124 us (as plain launches, like the rest of
// this line); 7 blocks and 4 rows 126, 7 and 8 rows 139, 6 and 8 rows 144 us (ranks in 64 bits 153), the 4 blocks that
// 64 registers allow 162 us: the loads wait for the flags and the counts, and other warps fill that wait better than
// more loads per warp.
template <typename T, int PHASE>
__global__ void __launch_bounds__(kCThreads, 8)
k_deque_move(T* data, const unsigned* before, unsigned ucap, const uint8_t* is_push, const T* values, unsigned n,
             T* out_popped, uint8_t* out_ok, bool zero_rest, const deque_control* ctl, deque_counters* c,
             sg_deque_sync* sync, uint32_t epoch)
{
    wait_for_stream();
    if (PHASE == kMoveLate && blockIdx.x == 0 && threadIdx.x == 0)
    {
        // nothing of the call reads the counters any more
        c->end += static_cast<unsigned long long>(ctl->push_ok);
        c->begin += static_cast<unsigned long long>(ctl->pop_ok);
        c->size += ctl->push_ok - ctl->pop_ok;
        c->avail += ctl->push_ok - ctl->pop_ok;
        deque_call_ends(c, sync, epoch, 1u);
    }
    const bool apart = ctl->apart != 0u;
    if (PHASE != kMoveFirst && apart)
    {
        return;
    }
    __shared__ unsigned s_warp[2][kWarps];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned push_pos = static_cast<unsigned>(ctl->push_t0 % ucap);
    const unsigned pop_pos = static_cast<unsigned>(ctl->pop_t0 % ucap);
    const unsigned push_ok = static_cast<unsigned>(ctl->push_ok);
    const unsigned pop_ok = static_cast<unsigned>(ctl->pop_ok);
    const unsigned held = static_cast<unsigned>(ctl->held);
    int buf = 0;
    for (unsigned tile = blockIdx.x; tile * kPlanTile < n; tile += gridDim.x, buf ^= 1)
    {
        const unsigned first = tile * kPlanTile + warp * (kItems * 32) + lane;
        unsigned masks[kItems]; // pushes of row j
        unsigned total = 0;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
        {
            const unsigned i = first + j * 32;
            masks[j] = __ballot_sync(0xffffffffu, i < n && is_push[i] != 0);
            total += __popc(masks[j]);
        }
        if (lane == 0)
        {
            s_warp[buf][warp] = total;
        }
        __syncthreads();
        unsigned rank = before[tile]; // pushes before the tile, then before the row
        for (int w = 0; w < warp; ++w)
        {
            rank += s_warp[buf][w];
        }
        // rows in flight together; more of them cost the registers that a second resident warp would use
        constexpr int kRows = 2;
#pragma unroll
        for (int j0 = 0; j0 < kItems; j0 += kRows)
        {
            T v[kRows];
            unsigned pos[kRows];
            unsigned done = 0u; // bit j: row j0 + j's item succeeds
            unsigned move = 0u; // bit j: and moves its element in this launch
#pragma unroll
            for (int j = 0; j < kRows; ++j)
            {
                const unsigned i = first + (j0 + j) * 32;
                const unsigned mask = masks[j0 + j];
                const bool push = (mask >> lane) & 1u;
                const unsigned pushes = rank + __popc(mask & lanemask_lt()); // before element i
                const unsigned r = push ? pushes : i - pushes;
                const bool ok = i < n && r < (push ? push_ok : pop_ok);
                const bool now = PHASE == kMoveFirst ? (push ? apart : r < held)
                                                     : (PHASE == kMovePush ? push : !push && r >= held);
                const unsigned p = (push ? push_pos : pop_pos) + r;
                pos[j] = p >= ucap ? p - ucap : p;
                v[j] = T{};
                done |= static_cast<unsigned>(ok) << j;
                if (ok && now)
                {
                    move |= 1u << j;
                    v[j] = push ? ld_stream(values + i) : __ldcg(data + pos[j]);
                }
                rank += __popc(mask);
            }
#pragma unroll
            for (int j = 0; j < kRows; ++j)
            {
                const unsigned i = first + (j0 + j) * 32;
                const bool push = (masks[j0 + j] >> lane) & 1u;
                const bool moves = (move >> j) & 1u;
                if (push && moves)
                {
                    data[pos[j]] = v[j];
                }
                // a pop of an element that the call pushed is written by the last launch
                if (out_popped != nullptr && i < n &&
                    (PHASE == kMoveFirst ? zero_rest || (!push && moves) : !push && moves))
                {
                    out_popped[i] = push ? T{} : v[j];
                }
                if (PHASE == kMoveFirst && out_ok != nullptr && i < n)
                {
                    out_ok[i] = static_cast<uint8_t>((done >> j) & 1u);
                }
            }
        }
        // no barrier: the next tile fills the other count buffer
    }
}

template <typename T>
__global__ void __launch_bounds__(kCThreads, SG_DEQUE_MIN_BLOCKS)
k_deque_ops(T* data, unsigned* seq, deque_counters* c, int64_t cap, const uint8_t* is_push, const T* values,
            int64_t n, T* out_popped, uint8_t* out_ok, bool zero_rest, deque_control* ctl, sg_deque_sync* sync,
            uint32_t epoch)
{
    wait_for_stream();
    __shared__ unsigned cpush[kCounts];
    __shared__ unsigned cpop[kCounts];
    __shared__ unsigned mpush[kCounts]; // the ballots, so the wait loop below indexes no local array
    __shared__ unsigned mpop[kCounts];
    __shared__ long long s_push_ok, s_pop_ok;
    __shared__ unsigned long long s_push_t0, s_pop_t0;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    for (int64_t tile = static_cast<int64_t>(blockIdx.x) * kTileElems; tile < n;
         tile += static_cast<int64_t>(gridDim.x) * kTileElems)
    {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
        {
            const int64_t i = tile + j * kCThreads + threadIdx.x;
            const bool in = i < n;
            const bool push = in && is_push[i] != 0;
            if (in && zero_rest && out_popped != nullptr)
            {
                out_popped[i] = T{}; // a pop that succeeds writes over it below, in this thread
            }
            const unsigned pm = __ballot_sync(0xffffffffu, push);
            const unsigned qm = __ballot_sync(0xffffffffu, in && !push);
            if (lane == 0)
            {
                cpush[j * kWarps + warp] = __popc(pm);
                cpop[j * kWarps + warp] = __popc(qm);
                mpush[j * kWarps + warp] = pm;
                mpop[j * kWarps + warp] = qm;
            }
        }
        __syncthreads();
        if (warp < 2)
        {
            const bool grow = warp == 0;
            const unsigned total = scan_counts(grow ? cpush : cpop, lane);
            if (lane == 0)
            {
                const long long ok = total > 0 ? reserve(grow ? &c->size : &c->avail, cap, total, grow) : 0;
                unsigned long long t0 = 0;
                if (ok > 0)
                {
                    t0 = atomicAdd(grow ? &c->end : &c->begin, static_cast<unsigned long long>(ok));
                    atomic_add_ll(grow ? &c->avail : &c->size, grow ? ok : -ok);
                }
                if (grow)
                {
                    s_push_ok = ok;
                    s_push_t0 = t0;
                }
                else
                {
                    s_pop_ok = ok;
                    s_pop_t0 = t0;
                }
            }
        }
        __syncthreads();
        const long long push_ok = s_push_ok;
        const long long pop_ok = s_pop_ok;
        const unsigned long long push_t0 = s_push_t0;
        const unsigned long long pop_t0 = s_pop_t0;
        // The thread's tickets: slot and low 32 bits of the ticket (a push waits for turn tk and leaves
        // tk + 1, a pop waits for tk + 1 and leaves tk + capacity; capacity < 2^31).  All turns are read at
        // once (relaxed, then one fence); when every one of them is already there -- the usual case, each
        // slot's previous operation having finished in an earlier tile or launch -- the elements are moved,
        // one fence orders those moves before the turns, and the turns are stored.  Otherwise the thread
        // takes its elements one by one with bounded waits, each releasing its turn at once, since one of
        // its elements may wait for a turn another of them leaves.
        unsigned pos[kItems];
        unsigned tk32[kItems];
        unsigned pushes = 0u; // bit j: item j is a push with a ticket
        unsigned pops = 0u;   // bit j: item j is a pop with a ticket
        bool ready = true;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
        {
            const unsigned bit = 1u << lane;
            const unsigned pm = mpush[j * kWarps + warp];
            const unsigned qm = mpop[j * kWarps + warp];
            pos[j] = 0u;
            tk32[j] = 0u;
            unsigned want = 0u;
            bool live = false;
            if (pm & bit)
            {
                const long long r = cpush[j * kWarps + warp] + __popc(pm & lanemask_lt());
                if (r < push_ok)
                {
                    const unsigned long long tk = push_t0 + static_cast<unsigned long long>(r);
                    pos[j] = static_cast<unsigned>(tk % static_cast<unsigned long long>(cap));
                    tk32[j] = static_cast<unsigned>(tk);
                    want = tk32[j];
                    pushes |= 1u << j;
                    live = true;
                }
            }
            else if (qm & bit)
            {
                const long long r = cpop[j * kWarps + warp] + __popc(qm & lanemask_lt());
                if (r < pop_ok)
                {
                    const unsigned long long tk = pop_t0 + static_cast<unsigned long long>(r);
                    pos[j] = static_cast<unsigned>(tk % static_cast<unsigned long long>(cap));
                    tk32[j] = static_cast<unsigned>(tk);
                    want = tk32[j] + 1u;
                    pops |= 1u << j;
                    live = true;
                }
            }
            if (live)
            {
                const unsigned cur = load_turn_relaxed(seq + pos[j]); // independent loads, all in flight
                ready = ready & (cur == want) & (SG_DEQUE_FAST != 0);
            }
        }
        if (ready)
        {
            fence_gpu(); // the turns read above come before the element accesses below
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                const int64_t i = tile + j * kCThreads + threadIdx.x;
                if (pushes & (1u << j))
                {
                    data[pos[j]] = ld_stream(values + i);
                }
                else if (pops & (1u << j))
                {
                    const T v = __ldcg(data + pos[j]);
                    if (out_popped != nullptr)
                    {
                        out_popped[i] = v;
                    }
                }
                if (i < n && out_ok != nullptr)
                {
                    out_ok[i] = static_cast<uint8_t>(((pushes | pops) >> j) & 1u);
                }
            }
            fence_gpu(); // the element accesses above come before the turns that hand the slots on
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                if (pushes & (1u << j))
                {
                    store_turn_relaxed(seq + pos[j], tk32[j] + 1u);
                }
                else if (pops & (1u << j))
                {
                    store_turn_relaxed(seq + pos[j], tk32[j] + static_cast<unsigned>(cap));
                }
            }
        }
        else
        {
            // One by one in the order of their turns: a push of ticket t before the pop of t, which comes
            // before the push of t + capacity.  Every wait is for a turn that precedes the element's own,
            // so a thread never waits for one of its own later elements (a pop and the push of the same
            // ticket can fall to one thread when the deque runs near empty inside a tile, and a push and
            // the pop one lap earlier when the ring wraps inside a tile).
            unsigned done = 0u;
            const unsigned live = pushes | pops;
#pragma unroll 1
            for (int step = 0; step < kItems; ++step)
            {
                int sel = -1;
                unsigned sel_tk = 0u;
                unsigned sel_pos = 0u;
                bool sel_pop = false;
#pragma unroll
                for (int j = 0; j < kItems; ++j)
                {
                    const bool pj = (pops >> j) & 1u;
                    // order key: ticket, then push before pop (tickets compared modulo 2^32)
                    const bool before = sel < 0 || static_cast<int>(tk32[j] - sel_tk) < 0 ||
                                        (tk32[j] == sel_tk && !pj && sel_pop);
                    if ((((live & ~done) >> j) & 1u) && before)
                    {
                        sel = j;
                        sel_tk = tk32[j];
                        sel_pos = pos[j];
                        sel_pop = pj;
                    }
                }
                if (sel < 0)
                {
                    break;
                }
                done |= 1u << sel;
                const int64_t i = tile + static_cast<int64_t>(sel) * kCThreads + threadIdx.x;
                const unsigned want = sel_pop ? sel_tk + 1u : sel_tk;
                bool ok = false;
                if (wait_turn(seq + sel_pos, want, &c->error))
                {
                    if (sel_pop)
                    {
                        const T v = *reinterpret_cast<volatile T*>(data + sel_pos);
                        store_turn(seq + sel_pos, sel_tk + static_cast<unsigned>(cap));
                        if (out_popped != nullptr)
                        {
                            out_popped[i] = v;
                        }
                    }
                    else
                    {
                        data[sel_pos] = values[i];
                        store_turn(seq + sel_pos, sel_tk + 1u);
                    }
                    ok = true;
                }
                if (out_ok != nullptr)
                {
                    out_ok[i] = static_cast<uint8_t>(ok);
                }
            }
            // elements without a ticket (refused, or past n)
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                const int64_t i = tile + j * kCThreads + threadIdx.x;
                if (!((live >> j) & 1u) && i < n && out_ok != nullptr)
                {
                    out_ok[i] = 0u;
                }
            }
        }
        __syncthreads(); // the counts and reservations are rewritten by the next tile
    }
    if (last_block(&ctl->arrived) && threadIdx.x == 0)
    {
        deque_call_ends(c, sync, epoch, 0u);
    }
}

// A launch of one kind of operation: element i acts as the i-th of a sequence of calls (push_front of values[0..n)
// leaves values[n-1] at the front, pop_back pops the back element first; the reference runs them concurrently with
// the other end under per-slot locks, src/stdgpu/impl/deque_detail.cuh:202-446).  The first min(n, room) elements
// succeed.  Nothing else runs on the deque during the launch; every block reads the counters as the call found
// them, and the last one to finish moves them.
// keep: the ring keeps its turn words between calls (kTurnsKeptMax): a push_back or pop_front waits, bounded, for its
// slot's turn, and every operation leaves the word that the launches that follow expect (a front push the word of a
// push_back of its ticket, a back pop the one that lets push_back reuse its ticket).  Larger rings leave them out.
enum deque_end : int
{
    kPushFront = 0,
    kPopBack = 1,
    kPushBack = 2,
    kPopFront = 3
};

template <typename T, int OP>
__global__ void __launch_bounds__(kCThreads)
k_deque_end_ops(T* data, deque_counters* c, int64_t cap, const T* values, int64_t n, T* out_popped, uint8_t* out_ok,
                bool zero_rest, unsigned* seq, bool keep, sg_deque_sync* sync, uint32_t epoch, deque_control* ctl)
{
    wait_for_stream();
    constexpr bool push = OP == kPushFront || OP == kPushBack;
    constexpr bool up = OP == kPushBack || OP == kPopFront; // tickets go up from t0, else down from t0 - 1
    const unsigned long long ucap = static_cast<unsigned long long>(cap);
    const unsigned long long begin = __ldcg(&c->begin), end = __ldcg(&c->end);
    const long long room = push ? cap - __ldcg(&c->size) : __ldcg(&c->avail);
    const long long k = room <= 0 ? 0 : (room < n ? room : n);
    const unsigned long long t0 = OP == kPushFront || OP == kPopFront ? begin : end;
    const int64_t base = static_cast<int64_t>((up ? t0 : t0 - 1ull) % ucap);
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const uint32_t dirty = *reinterpret_cast<const volatile uint32_t*>(&sync->dirty);
    if (keep)
    {
        for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
        {
            bool ok = i < k;
            T v{};
            if (ok)
            {
                int64_t p = up ? base + i : base - i;
                p = p >= cap ? p - cap : (p < 0 ? p + cap : p);
                const unsigned tk = static_cast<unsigned>(up ? t0 + static_cast<unsigned long long>(i)
                                                             : t0 - 1ull - static_cast<unsigned long long>(i));
                if (up && dirty == 0u)
                {
                    ok = wait_turn(seq + p, push ? tk : tk + 1u, &c->error);
                }
                if (ok)
                {
                    if constexpr (push)
                    {
                        data[p] = values[i];
                    }
                    else
                    {
                        v = __ldcg(data + p);
                    }
                    seq[p] = push ? tk + 1u : (OP == kPopFront ? tk + static_cast<unsigned>(cap) : tk);
                }
            }
            if (!push && out_popped != nullptr && (ok || zero_rest))
            {
                out_popped[i] = v;
            }
            if (out_ok != nullptr)
            {
                out_ok[i] = static_cast<uint8_t>(ok);
            }
        }
    }
    constexpr int kFlight = 4;
    for (int64_t i0 = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; !keep && i0 < n;
         i0 += kFlight * stride)
    {
        T v[kFlight];
        int64_t pos[kFlight];
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
        {
            const int64_t i = i0 + j * stride;
            v[j] = T{};
            if (i < k) // k <= capacity: the slot index wraps at most once
            {
                int64_t p = up ? base + i : base - i;
                p = p >= cap ? p - cap : (p < 0 ? p + cap : p);
                pos[j] = p;
                v[j] = push ? ld_stream(values + i) : __ldcg(data + p);
            }
        }
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
        {
            const int64_t i = i0 + j * stride;
            if (i >= n)
            {
                break;
            }
            const bool ok = i < k;
            if (push && ok)
            {
                data[pos[j]] = v[j];
            }
            if (!push && out_popped != nullptr && (ok || zero_rest))
            {
                out_popped[i] = v[j];
            }
            if (out_ok != nullptr)
            {
                out_ok[i] = static_cast<uint8_t>(ok);
            }
        }
    }
    if (last_block(&ctl->arrived) && threadIdx.x == 0)
    {
        const unsigned long long uk = static_cast<unsigned long long>(k);
        c->begin = OP == kPushFront ? begin - uk : (OP == kPopFront ? begin + uk : begin);
        c->end = OP == kPushBack ? end + uk : (OP == kPopBack ? end - uk : end);
        c->size += push ? k : -k;
        c->avail += push ? k : -k;
        deque_call_ends(c, sync, epoch, keep ? dirty : 1u);
    }
}

// vector::pop_back for n elements (src/stdgpu/impl/vector_detail.cuh:240-299): element i takes the i-th
// element from the back.  Every block reads the size as the call found it (clamped into [0, capacity]: a push
// launch may leave it above); the last one to finish lowers it.
template <typename T>
__global__ void __launch_bounds__(kCThreads)
k_vector_pop_back(const T* data, long long* size, int64_t cap, int64_t n, T* out_values, uint8_t* out_ok,
                  sg_vector_sync* sync, uint32_t epoch, vector_control* ctl)
{
    wait_for_stream();
    long long sz = __ldcg(size);
    sz = sz < 0 ? 0 : (sz > cap ? cap : sz);
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        const long long pos = sz - 1 - i;
        const bool ok = pos >= 0;
        if (ok && out_values != nullptr)
        {
            out_values[i] = data[pos];
        }
        if (out_ok != nullptr)
        {
            out_ok[i] = static_cast<uint8_t>(ok);
        }
    }
    if (last_block(&ctl->arrived) && threadIdx.x == 0)
    {
        vector_call_ends(size, cap, n, sync, epoch);
    }
}

// clear(), and the end of the calls that the host drives (insert, erase).
__global__ void
k_vector_call_ends(long long* size, int64_t cap, bool clear, sg_vector_sync* sync, uint32_t epoch, vector_control* ctl)
{
    wait_for_stream();
    if (clear)
    {
        *ctl = vector_control{}; // whatever launches that overlapped against the rules left there
        *size = 0;
    }
    vector_call_ends(size, cap, 0, sync, epoch);
}

// keep: the turn words too (slot i is free for ticket i, modulo 2^32)
__global__ void
k_deque_reset(unsigned* seq, deque_counters* c, int64_t cap, bool keep, sg_deque_sync* sync, uint32_t epoch,
              deque_control* ctl)
{
    wait_for_stream();
    if (keep)
    {
        for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < cap;
             i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        {
            seq[i] = static_cast<unsigned>(i);
        }
    }
    if (blockIdx.x != 0 || threadIdx.x != 0)
    {
        return;
    }
    // tickets start at capacity x 2^32: a multiple of the capacity (so ticket mod capacity is the slot)
    // and of 2^32 (so the 32-bit turn words start at the slot index), far enough from zero for
    // push_front to move begin down
    c->size = 0;
    c->begin = static_cast<unsigned long long>(cap) << 32;
    c->end = static_cast<unsigned long long>(cap) << 32;
    c->error = 0;
    c->avail = 0;
    *ctl = deque_control{};
    deque_call_ends(c, sync, epoch, keep ? 0u : 1u);
}

template <typename T>
__global__ void
k_deque_copy_out(const T* data, const deque_counters* c, int64_t cap, T* out)
{
    const long long n = c->size;
    const unsigned long long b = c->begin;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        out[i] = data[(b + static_cast<unsigned long long>(i)) % static_cast<unsigned long long>(cap)];
    }
}

// Up to 32 words of device memory into pinned host memory: sooner there than by a copy of a few bytes (size() of a
// vector or deque).
__global__ void
k_read_words(const unsigned long long* src, unsigned long long* host, int words)
{
    wait_for_stream();
    if (static_cast<int>(threadIdx.x) < words)
    {
        host[threadIdx.x] = __ldcg(src + threadIdx.x);
    }
}

// ---------------------------------------------------------------- bitset::count

constexpr int kCountThreads = 512;

__global__ void __launch_bounds__(kCountThreads)
k_bitset_count(const uint32_t* blocks, int64_t nbits, unsigned long long* partials)
{
    wait_for_stream();
    const int64_t nwords = (nbits + 31) / 32;
    const int64_t full_words = nbits / 32; // words with all 32 bits counted
    const bool aligned = (reinterpret_cast<uintptr_t>(blocks) & 15u) == 0;
    const int64_t nvec = aligned ? full_words / 4 : 0;
    const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    unsigned long long sum = 0;
    const uint4* v4 = reinterpret_cast<const uint4*>(blocks);
    // 4 independent 16-byte loads in flight per thread
    int64_t k = tid;
    for (; k + 3 * stride < nvec; k += 4 * stride)
    {
        const uint4 a = __ldcs(v4 + k);
        const uint4 b = __ldcs(v4 + k + stride);
        const uint4 c = __ldcs(v4 + k + 2 * stride);
        const uint4 d = __ldcs(v4 + k + 3 * stride);
        sum += __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);
        sum += __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
        sum += __popc(c.x) + __popc(c.y) + __popc(c.z) + __popc(c.w);
        sum += __popc(d.x) + __popc(d.y) + __popc(d.z) + __popc(d.w);
    }
    for (; k < nvec; k += stride)
    {
        const uint4 a = __ldcs(v4 + k);
        sum += __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);
    }
    // remaining full words, then the masked tail word (count_block_bits::block_mask)
    for (int64_t w = nvec * 4 + tid; w < nwords; w += stride)
    {
        uint32_t x = blocks[w];
        if (w >= full_words)
        {
            const int rem = static_cast<int>(nbits - w * 32);
            x &= (1u << rem) - 1u;
        }
        sum += __popc(x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    __shared__ unsigned long long red[kCountThreads / 32];
    if ((threadIdx.x & 31) == 0)
    {
        red[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long s = 0;
        for (int w = 0; w < kCountThreads / 32; ++w)
        {
            s += red[w];
        }
        partials[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(1024)
k_sum_partials(const unsigned long long* partials, int n, unsigned long long* out)
{
    wait_for_stream();
    unsigned long long s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
    {
        s += partials[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    __shared__ unsigned long long red[32];
    if ((threadIdx.x & 31) == 0)
    {
        red[threadIdx.x >> 5] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long t = 0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w)
        {
            t += red[w];
        }
        *out = t;
    }
}

int
count_grid()
{
    static const int g = persistent_grid(k_bitset_count, kCountThreads);
    return g;
}

// ---------------------------------------------------------------- allocation-free bitset::count
// The same count with its scratch in a fixed array compiled into the library instead of memory the
// library allocates: one partial sum per CTA, each CTA owning a fixed chunk of the blocks, so the
// array's length bounds the largest input.  The array lives in every GPU that loads the library until
// the process exits; all calls on a device share it, so calls that overlap on the GPU race.

constexpr int kNoAllocPartials = 8192;                                   // 64 KiB of partial sums
constexpr int64_t kNoAllocChunkWords = 65536;                            // 32-bit blocks per CTA (256 KiB)
constexpr int64_t kNoAllocMaxBits = kNoAllocPartials * kNoAllocChunkWords * 32; // 2^34 bits

static __device__ __align__(256) unsigned long long g_noalloc_partials[kNoAllocPartials];

__global__ void __launch_bounds__(kCountThreads)
k_bitset_count_chunked(const uint32_t* blocks, int64_t nbits, unsigned long long* partials)
{
    const int64_t nwords = (nbits + 31) / 32;
    const int64_t full_words = nbits / 32;
    const int64_t lo = static_cast<int64_t>(blockIdx.x) * kNoAllocChunkWords;
    const int64_t hi = lo + kNoAllocChunkWords < nwords ? lo + kNoAllocChunkWords : nwords;
    unsigned long long sum = 0;
    const bool aligned = (reinterpret_cast<uintptr_t>(blocks) & 15u) == 0;
    int64_t w = lo;
    if (aligned)
    {
        // whole 16-byte vectors of full words inside the chunk
        const int64_t vhi = lo + ((min(hi, full_words) - lo) / 4) * 4;
        const uint4* v4 = reinterpret_cast<const uint4*>(blocks + lo);
        const int64_t nv = (vhi - lo) / 4;
        for (int64_t k = threadIdx.x; k < nv; k += blockDim.x)
        {
            const uint4 a = __ldcs(v4 + k);
            sum += __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);
        }
        w = vhi;
    }
    for (int64_t x = w + threadIdx.x; x < hi; x += blockDim.x)
    {
        uint32_t b = blocks[x];
        if (x >= full_words)
        {
            b &= (1u << static_cast<int>(nbits - x * 32)) - 1u;
        }
        sum += __popc(b);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    __shared__ unsigned long long red[kCountThreads / 32];
    if ((threadIdx.x & 31) == 0)
    {
        red[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long t = 0;
        for (int k = 0; k < kCountThreads / 32; ++k)
        {
            t += red[k];
        }
        partials[blockIdx.x] = t; // every entry the sum kernel reads is written by this call
    }
}

} // namespace detail
} // namespace sg

using namespace sg::detail;

namespace
{

// Orders the bulk calls on one vector or deque on the device as the host made them, also when they are queued on
// different streams: a call's launches share counters and words that the next call's launches use too.
struct call_order
{
    cudaEvent_t done = nullptr;       // the end of the last call
    unsigned long long stream = 0ull; // and the id of its stream
    bool any = false;
};

// Lives from before a call's first launch to after its last one.  Calls under stream capture are left to the order
// of the graphs they go into.  It costs half a microsecond of the host's time a call, most of it for the event; on the
// device nothing before a launch_early (ten push_back and pop_front of 64 elements 67.2 us with and without) and a
// microsecond or so before another kernel (a pass of 2^24 mixed operations, a pop and the caller's own kernels 285 us,
// 286 with it).
class ordered_call
{
public:
    ordered_call(call_order& order, cudaStream_t s)
        : _order(order)
        , _s(s)
    {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        unsigned long long id = 0ull;
        if (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone ||
            cudaStreamGetId(s, &id) != cudaSuccess)
        {
            cudaGetLastError();
            return;
        }
        if (order.any && order.stream != id)
        {
            _error = cudaStreamWaitEvent(s, order.done, 0);
        }
        order.stream = id;
        _record = true;
    }

    ~ordered_call()
    {
        if (_record && cudaEventRecord(_order.done, _s) == cudaSuccess)
        {
            _order.any = true;
        }
    }

    ordered_call(const ordered_call&) = delete;
    ordered_call& operator=(const ordered_call&) = delete;

    cudaError_t
    error() const
    {
        return _error;
    }

private:
    call_order& _order;
    cudaStream_t _s;
    cudaError_t _error = cudaSuccess;
    bool _record = false;
};

} // namespace

struct sg_vector
{
    int32_t elem_bytes;
    int64_t capacity;
    void* data;
    long long* size;
    long long* host;
    uint16_t* slot_state;   // device calls' per-slot words (sg_vector_sync)
    sg_vector_sync* sync;
    uint32_t epoch;         // host copy of sync->epoch
    call_order order;
    object_allocator oa;            // the vector's own allocator (sg_vector_create_with_allocator), or none
    void (*release_ctx)(void* ctx); // called with oa.ctx when the vector is destroyed (nullable)
};

struct sg_deque
{
    int32_t elem_bytes;
    int64_t capacity;
    void* data;
    unsigned* seq;
    deque_counters* counters;
    deque_counters* host;
    uint16_t* slot_state; // device calls' per-slot words (sg_deque_sync)
    sg_deque_sync* sync;
    uint32_t epoch;       // host copy of sync->epoch
    call_order order;
    object_allocator oa;            // the deque's own allocator (sg_deque_create_with_allocator), or none
    void (*release_ctx)(void* ctx); // called with oa.ctx when the deque is destroyed (nullable)
};

namespace
{

// Per-device scratch of bitset::count: one partial per block plus the result word.
struct count_scratch
{
    unsigned long long* partials = nullptr;
    unsigned long long* host = nullptr;
    int blocks = 0;
};

std::mutex g_count_mutex;
count_scratch g_count_scratch[64];

} // namespace

namespace
{

// The device calls' epoch at the end of a bulk call: 1 .. 32767 (slot words are cleared when it wraps).
template <typename Object>
sg_status
next_epoch(Object* d, cudaStream_t s)
{
    uint32_t e = d->epoch + 1;
    if (e > 32767u)
    {
        SG_CUDA_TRY(cudaMemsetAsync(d->slot_state, 0, static_cast<size_t>(d->capacity) * sizeof(uint16_t), s));
        e = 1;
    }
    d->epoch = e;
    return SG_OK;
}

// Rings of at most this many slots keep their turn words from call to call and order every mixed launch by them: two
// launches instead of four.  Neither route is better for every call there: 16384 mixed operations on a ring of 2^16
// take 21 us by the turn words and 18 by the plan in steady state, 20 and 24 from empty, where pops follow the call's
// own pushes; on a ring of 2^14 4096 of them take 21 and 18, 18 and 24.  Above the line the plan wins both as calls
// grow: 2^18 operations 18 and 23 us, 25 and 39; 2^22 42 and 74, 80 and 155.  Larger rings make the words for the
// launches that wait on them, those of more elements than the ring has slots.
constexpr int64_t kTurnsKeptMax = int64_t{ 1 } << 16;

deque_control*
control_of(const sg_deque* d)
{
    return reinterpret_cast<deque_control*>(reinterpret_cast<char*>(d->sync) + kControlOffset);
}

vector_control*
control_of(const sg_vector* v)
{
    return reinterpret_cast<vector_control*>(reinterpret_cast<char*>(v->sync) + kControlOffset);
}

template <typename T, int OP>
sg_status
deque_end_launch(sg_deque* d, const void* values, int64_t n, void* out_popped, uint8_t* out_ok, bool zero_rest,
                 cudaStream_t s)
{
    static const int mg = persistent_grid(k_deque_end_ops<T, OP>, kCThreads);
    SG_CUDA_TRY(launch_early(k_deque_end_ops<T, OP>, grid_for(n, kCThreads, mg), kCThreads, s, static_cast<T*>(d->data),
                             d->counters, d->capacity, static_cast<const T*>(values), n, static_cast<T*>(out_popped),
                             out_ok, zero_rest, d->seq, d->capacity <= kTurnsKeptMax, d->sync, d->epoch,
                             control_of(d)));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

template <int OP>
sg_status
deque_end_ops(sg_deque* d, const void* values, int64_t n, void* out_popped, uint8_t* out_ok, bool zero_rest,
              void* stream)
{
    if (d == nullptr || n < 0 || ((OP == kPushFront || OP == kPushBack) && n > 0 && values == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    if (n == 0)
    {
        return SG_OK;
    }
    cudaStream_t s = as_stream(stream);
    const ordered_call call(d->order, s);
    SG_CUDA_TRY(call.error());
    const sg_status st = next_epoch(d, s);
    if (st != SG_OK)
    {
        return st;
    }
    return d->elem_bytes == 4
                   ? deque_end_launch<uint32_t, OP>(d, values, n, out_popped, out_ok, zero_rest, s)
                   : deque_end_launch<unsigned long long, OP>(d, values, n, out_popped, out_ok, zero_rest, s);
}

// A mixed call: the plan and the moves; by turn words on a small ring, or with more elements than slots, whose pushes
// and pops may pass through a slot several times.
template <typename T>
sg_status
deque_mixed(sg_deque* d, const uint8_t* is_push, const void* values, int64_t n, void* out_popped, uint8_t* out_ok,
            bool zero_rest, cudaStream_t s)
{
    T* const data = static_cast<T*>(d->data);
    const T* const in = static_cast<const T*>(values);
    T* const out = static_cast<T*>(out_popped);
    if (d->capacity <= kTurnsKeptMax || n > d->capacity)
    {
        static const int mr = persistent_grid(k_deque_rebuild_turns, kCThreads);
        SG_CUDA_TRY(launch_early(k_deque_rebuild_turns, grid_for(d->capacity, kCThreads, mr), kCThreads, s, d->seq,
                                 d->counters, d->sync, d->capacity));
        SG_LAUNCH_CHECK();
        static const int mo = persistent_grid(k_deque_ops<T>, kCThreads);
        SG_CUDA_TRY(launch_early(k_deque_ops<T>, grid_for(n, static_cast<int>(kTileElems), mo), kCThreads, s, data,
                                 d->seq, d->counters, d->capacity, is_push, in, n, out, out_ok, zero_rest,
                                 control_of(d), d->sync, d->epoch));
        SG_LAUNCH_CHECK();
        return SG_OK;
    }
    const int64_t tiles = (n + kPlanTile - 1) / kPlanTile;
    static const int mp = persistent_grid(k_deque_plan, kCThreads);
    SG_CUDA_TRY(launch_early(k_deque_plan, grid_for(tiles, kWarps, mp), kCThreads, s, is_push, n, d->seq, d->counters,
                             d->capacity, d->sync, control_of(d)));
    SG_LAUNCH_CHECK();
    // at most `capacity` elements, below 2^31: 32-bit ranks
    const unsigned ucap = static_cast<unsigned>(d->capacity);
    const unsigned un = static_cast<unsigned>(n);
    static const int m0 = persistent_grid(k_deque_move<T, kMoveFirst>, kCThreads);
    static const int m1 = persistent_grid(k_deque_move<T, kMovePush>, kCThreads);
    static const int m2 = persistent_grid(k_deque_move<T, kMoveLate>, kCThreads);
    SG_CUDA_TRY(launch_early(k_deque_move<T, kMoveFirst>, grid_for(tiles, 1, m0), kCThreads, s, data, d->seq, ucap,
                             is_push, in, un, out, out_ok, zero_rest, control_of(d), d->counters, d->sync, d->epoch));
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(launch_early(k_deque_move<T, kMovePush>, grid_for(tiles, 1, m1), kCThreads, s, data, d->seq, ucap,
                             is_push, in, un, out, out_ok, zero_rest, control_of(d), d->counters, d->sync, d->epoch));
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(launch_early(k_deque_move<T, kMoveLate>, grid_for(tiles, 1, m2), kCThreads, s, data, d->seq, ucap,
                             is_push, in, un, out, out_ok, zero_rest, control_of(d), d->counters, d->sync, d->epoch));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

sg_status
deque_ops(sg_deque* d, const uint8_t* is_push, const void* values, int64_t n, void* out_popped, uint8_t* out_ok,
          bool zero_rest, void* stream)
{
    if (d == nullptr || n < 0)
    {
        return SG_ERR_BAD_ARG;
    }
    if (n == 0)
    {
        return SG_OK;
    }
    cudaStream_t s = as_stream(stream);
    if (is_push == nullptr)
    {
        // all push_back; nothing is popped
        if (zero_rest && out_popped != nullptr)
        {
            SG_CUDA_TRY(cudaMemsetAsync(out_popped, 0, static_cast<size_t>(n) * d->elem_bytes, s));
        }
        return deque_end_ops<kPushBack>(d, values, n, nullptr, out_ok, false, stream);
    }
    const ordered_call call(d->order, s);
    SG_CUDA_TRY(call.error());
    const sg_status st = next_epoch(d, s);
    if (st != SG_OK)
    {
        return st;
    }
    return d->elem_bytes == 4
                   ? deque_mixed<uint32_t>(d, is_push, values, n, out_popped, out_ok, zero_rest, s)
                   : deque_mixed<unsigned long long>(d, is_push, values, n, out_popped, out_ok, zero_rest, s);
}

// Ends a bulk call on v that the host drives, or clears it.
sg_status
vector_call_ends(sg_vector* v, bool clear, cudaStream_t s)
{
    const sg_status st = next_epoch(v, s);
    if (st != SG_OK)
    {
        return st;
    }
    SG_CUDA_TRY(launch_early(k_vector_call_ends, 1, 1, s, v->size, v->capacity, clear, v->sync, v->epoch,
                             control_of(v)));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

// Launches of at least this many elements reserve once per 8192 of them (k_vector_push_back, 32 rows), smaller ones
// once per 1024 (4 rows): from here on there is a block of that size for every SM.  4-byte elements with flags, 4 and
// 32 rows: 2^16 elements 7-9 and 9 us, 2^20 10 and 11, 2^21 13 and 11, 2^23 27 and 19, 2^24 46 and 31.
constexpr int64_t kVecLargeTile = int64_t{ 1 } << 21;

template <typename T, int ROWS>
sg_status
push_back_launch(sg_vector* v, const void* values, const uint8_t* pred, int64_t n, uint8_t* out_pushed, cudaStream_t s)
{
    static const int mg = persistent_grid(k_vector_push_back<T, ROWS>, kCThreads);
    SG_CUDA_TRY(launch_early(k_vector_push_back<T, ROWS>, grid_for(n, ROWS * kCThreads, mg), kCThreads, s,
                             static_cast<T*>(v->data), v->size, v->capacity, static_cast<const T*>(values), pred, n,
                             out_pushed, v->sync, v->epoch, control_of(v)));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

} // namespace

extern "C" {

static sg_status
create_vector(int32_t elem_bytes, int64_t capacity, const object_allocator& oa, sg_vector** out)
{
    if (out == nullptr || (elem_bytes != 4 && elem_bytes != 8) || capacity <= 0)
    {
        return SG_ERR_BAD_ARG;
    }
    *out = nullptr;
    auto* v = new (std::nothrow) sg_vector{};
    if (v == nullptr)
    {
        return SG_ERR_OOM;
    }
    v->elem_bytes = elem_bytes;
    v->capacity = capacity;
    v->oa = oa;
    cudaError_t e = sg::detail::obj_malloc(v->oa, &v->data, static_cast<size_t>(capacity) * elem_bytes);
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(v->oa, &v->size, sizeof(long long));
    }
    if (e == cudaSuccess)
    {
        e = cudaMemset(v->size, 0, sizeof(long long));
    }
    if (e == cudaSuccess)
    {
        e = cudaMallocHost(&v->host, sizeof(long long));
    }
    if (e == cudaSuccess)
    {
        e = cudaEventCreateWithFlags(&v->order.done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(v->oa, &v->slot_state, static_cast<size_t>(capacity) * sizeof(uint16_t));
    }
    if (e == cudaSuccess)
    {
        e = cudaMemset(v->slot_state, 0, static_cast<size_t>(capacity) * sizeof(uint16_t));
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(v->oa, &v->sync, kSyncBytes);
    }
    if (e == cudaSuccess)
    {
        e = cudaMemset(v->sync, 0, kSyncBytes);
    }
    if (e == cudaSuccess)
    {
        const sg_vector_sync init{ 1u, 0u, 0 };
        v->epoch = 1;
        e = cudaMemcpy(v->sync, &init, sizeof(init), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess)
    {
        sg_vector_destroy(v);
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? SG_ERR_OOM : SG_ERR_CUDA;
    }
    *out = v;
    return SG_OK;
}

sg_status
sg_vector_create(int32_t elem_bytes, int64_t capacity, sg_vector** out)
{
    return create_vector(elem_bytes, capacity, object_allocator{}, out);
}

sg_status
sg_vector_create_with_allocator(int32_t elem_bytes, int64_t capacity, const sg_allocator* allocator, sg_vector** out)
{
    if (allocator == nullptr || allocator->alloc == nullptr || allocator->release == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    const sg_status st =
            create_vector(elem_bytes, capacity, object_allocator{ allocator->alloc, allocator->release, allocator->ctx }, out);
    if (st == SG_OK)
    {
        (*out)->release_ctx = allocator->release_ctx;
    }
    return st;
}

sg_status
sg_vector_destroy(sg_vector* v)
{
    if (v == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaDeviceSynchronize();
    sg::detail::obj_free(v->oa, v->data);
    sg::detail::obj_free(v->oa, v->size);
    sg::detail::obj_free(v->oa, v->slot_state);
    sg::detail::obj_free(v->oa, v->sync);
    if (v->host != nullptr)
    {
        cudaFreeHost(v->host);
    }
    if (v->order.done != nullptr)
    {
        cudaEventDestroy(v->order.done);
    }
    if (v->release_ctx != nullptr)
    {
        v->release_ctx(v->oa.ctx);
    }
    delete v;
    return SG_OK;
}

sg_status
sg_vector_push_back(sg_vector* v, const void* values, const uint8_t* pred, int64_t n, uint8_t* out_pushed,
                    void* stream)
{
    if (v == nullptr || n < 0 || (n > 0 && values == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    if (n == 0)
    {
        return SG_OK;
    }
    cudaStream_t s = as_stream(stream);
    const ordered_call call(v->order, s);
    SG_CUDA_TRY(call.error());
    const sg_status st = next_epoch(v, s);
    if (st != SG_OK)
    {
        return st;
    }
    if (n >= kVecLargeTile)
    {
        return v->elem_bytes == 4 ? push_back_launch<uint32_t, 32>(v, values, pred, n, out_pushed, s)
                                  : push_back_launch<unsigned long long, 32>(v, values, pred, n, out_pushed, s);
    }
    return v->elem_bytes == 4 ? push_back_launch<uint32_t, 4>(v, values, pred, n, out_pushed, s)
                              : push_back_launch<unsigned long long, 4>(v, values, pred, n, out_pushed, s);
}

sg_status
sg_vector_size(sg_vector* v, void* stream, int64_t* out_size)
{
    if (v == nullptr || out_size == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaStream_t s = as_stream(stream);
    SG_CUDA_TRY(launch_early(k_read_words, 1, 32, s, reinterpret_cast<const unsigned long long*>(v->size),
                             reinterpret_cast<unsigned long long*>(v->host), 1));
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    long long x = *v->host;
    *out_size = x < 0 ? 0 : (x > v->capacity ? v->capacity : x);
    return SG_OK;
}

sg_status
sg_vector_clear(sg_vector* v, void* stream)
{
    if (v == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    const ordered_call call(v->order, as_stream(stream));
    SG_CUDA_TRY(call.error());
    return vector_call_ends(v, true, as_stream(stream));
}

sg_status
sg_vector_pop_back(sg_vector* v, int64_t n, void* out_values, uint8_t* out_ok, void* stream)
{
    if (v == nullptr || n < 0)
    {
        return SG_ERR_BAD_ARG;
    }
    if (n == 0)
    {
        return SG_OK;
    }
    cudaStream_t s = as_stream(stream);
    const ordered_call call(v->order, s);
    SG_CUDA_TRY(call.error());
    const sg_status st = next_epoch(v, s);
    if (st != SG_OK)
    {
        return st;
    }
    const int g = grid_for(n, kCThreads, 4096);
    if (v->elem_bytes == 4)
    {
        SG_CUDA_TRY(launch_early(k_vector_pop_back<uint32_t>, g, kCThreads, s, static_cast<const uint32_t*>(v->data),
                                 v->size, v->capacity, n, static_cast<uint32_t*>(out_values), out_ok, v->sync, v->epoch,
                                 control_of(v)));
    }
    else
    {
        SG_CUDA_TRY(launch_early(k_vector_pop_back<unsigned long long>, g, kCThreads, s,
                                 static_cast<const unsigned long long*>(v->data), v->size, v->capacity, n,
                                 static_cast<unsigned long long*>(out_values), out_ok, v->sync, v->epoch,
                                 control_of(v)));
    }
    SG_LAUNCH_CHECK();
    return SG_OK;
}

sg_status
sg_vector_insert(sg_vector* v, const void* values, int64_t n, void* stream)
{
    if (v == nullptr || n < 0 || (n > 0 && values == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    const ordered_call call(v->order, as_stream(stream));
    SG_CUDA_TRY(call.error());
    int64_t size = 0;
    const sg_status st = sg_vector_size(v, stream, &size);
    if (st != SG_OK)
    {
        return st;
    }
    if (size + n > v->capacity)
    {
        return SG_ERR_FULL; // nothing inserted (vector_detail.cuh:372-410 refuses the whole range)
    }
    cudaStream_t s = as_stream(stream);
    SG_CUDA_TRY(cudaMemcpyAsync(static_cast<char*>(v->data) + size * v->elem_bytes, values,
                                static_cast<size_t>(n) * v->elem_bytes, cudaMemcpyDeviceToDevice, s));
    *v->host = size + n;
    SG_CUDA_TRY(cudaMemcpyAsync(v->size, v->host, sizeof(long long), cudaMemcpyHostToDevice, s));
    const sg_status e = vector_call_ends(v, false, s);
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    return e;
}

sg_status
sg_vector_erase(sg_vector* v, int64_t n, void* stream)
{
    if (v == nullptr || n < 0)
    {
        return SG_ERR_BAD_ARG;
    }
    const ordered_call call(v->order, as_stream(stream));
    SG_CUDA_TRY(call.error());
    int64_t size = 0;
    const sg_status st = sg_vector_size(v, stream, &size);
    if (st != SG_OK)
    {
        return st;
    }
    if (n > size)
    {
        return SG_ERR_BAD_ARG; // nothing erased (vector_detail.cuh:418-450 refuses a range past the start)
    }
    cudaStream_t s = as_stream(stream);
    *v->host = size - n;
    SG_CUDA_TRY(cudaMemcpyAsync(v->size, v->host, sizeof(long long), cudaMemcpyHostToDevice, s));
    const sg_status e = vector_call_ends(v, false, s);
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    return e;
}

sg_status
sg_vector_view_of(const sg_vector* v, sg_vector_view* out)
{
    if (v == nullptr || out == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    out->data = v->data;
    out->size = v->size;
    out->capacity = v->capacity;
    out->elem_bytes = v->elem_bytes;
    out->pad = 0;
    out->slot_state = v->slot_state;
    out->sync = v->sync;
    return SG_OK;
}

static sg_status
create_deque(int32_t elem_bytes, int64_t capacity, const object_allocator& oa, sg_deque** out)
{
    if (out == nullptr || (elem_bytes != 4 && elem_bytes != 8) || capacity <= 0 || capacity >= (int64_t{ 1 } << 31))
    {
        return SG_ERR_BAD_ARG;
    }
    *out = nullptr;
    auto* d = new (std::nothrow) sg_deque{};
    if (d == nullptr)
    {
        return SG_ERR_OOM;
    }
    d->elem_bytes = elem_bytes;
    d->capacity = capacity;
    d->oa = oa;
    cudaError_t e = sg::detail::obj_malloc(d->oa, &d->data, static_cast<size_t>(capacity) * elem_bytes);
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(d->oa, &d->seq, static_cast<size_t>(capacity) * sizeof(unsigned));
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(d->oa, &d->counters, sizeof(deque_counters));
    }
    if (e == cudaSuccess)
    {
        e = cudaMallocHost(&d->host, sizeof(deque_counters));
    }
    if (e == cudaSuccess)
    {
        e = cudaEventCreateWithFlags(&d->order.done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(d->oa, &d->slot_state, static_cast<size_t>(capacity) * sizeof(uint16_t));
    }
    if (e == cudaSuccess)
    {
        e = cudaMemset(d->slot_state, 0, static_cast<size_t>(capacity) * sizeof(uint16_t));
    }
    if (e == cudaSuccess)
    {
        e = sg::detail::obj_malloc(d->oa, &d->sync, kSyncBytes);
    }
    if (e == cudaSuccess)
    {
        e = cudaMemset(d->sync, 0, kSyncBytes);
    }
    if (e != cudaSuccess)
    {
        sg_deque_destroy(d);
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? SG_ERR_OOM : SG_ERR_CUDA;
    }
    sg_status st = sg_deque_clear(d, nullptr);
    if (st != SG_OK)
    {
        sg_deque_destroy(d);
        return st;
    }
    *out = d;
    return SG_OK;
}

sg_status
sg_deque_create(int32_t elem_bytes, int64_t capacity, sg_deque** out)
{
    return create_deque(elem_bytes, capacity, object_allocator{}, out);
}

sg_status
sg_deque_create_with_allocator(int32_t elem_bytes, int64_t capacity, const sg_allocator* allocator, sg_deque** out)
{
    if (allocator == nullptr || allocator->alloc == nullptr || allocator->release == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    const sg_status st =
            create_deque(elem_bytes, capacity, object_allocator{ allocator->alloc, allocator->release, allocator->ctx }, out);
    if (st == SG_OK)
    {
        (*out)->release_ctx = allocator->release_ctx;
    }
    return st;
}

sg_status
sg_deque_destroy(sg_deque* d)
{
    if (d == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaDeviceSynchronize();
    sg::detail::obj_free(d->oa, d->data);
    sg::detail::obj_free(d->oa, d->seq);
    sg::detail::obj_free(d->oa, d->counters);
    sg::detail::obj_free(d->oa, d->slot_state);
    sg::detail::obj_free(d->oa, d->sync);
    if (d->host != nullptr)
    {
        cudaFreeHost(d->host);
    }
    if (d->order.done != nullptr)
    {
        cudaEventDestroy(d->order.done);
    }
    if (d->release_ctx != nullptr)
    {
        d->release_ctx(d->oa.ctx);
    }
    delete d;
    return SG_OK;
}

sg_status
sg_deque_clear(sg_deque* d, void* stream)
{
    if (d == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaStream_t s = as_stream(stream);
    const ordered_call call(d->order, s);
    SG_CUDA_TRY(call.error());
    const sg_status st = next_epoch(d, s);
    if (st != SG_OK)
    {
        return st;
    }
    const bool keep = d->capacity <= kTurnsKeptMax;
    SG_CUDA_TRY(launch_early(k_deque_reset, keep ? grid_for(d->capacity, kCThreads, 256) : 1, kCThreads, s, d->seq,
                             d->counters, d->capacity, keep, d->sync, d->epoch, control_of(d)));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

sg_status
sg_deque_push_front(sg_deque* d, const void* values, int64_t n, uint8_t* out_ok, void* stream)
{
    return deque_end_ops<kPushFront>(d, values, n, nullptr, out_ok, false, stream);
}

sg_status
sg_deque_pop_back(sg_deque* d, int64_t n, void* out_popped, uint8_t* out_ok, void* stream)
{
    return deque_end_ops<kPopBack>(d, nullptr, n, out_popped, out_ok, false, stream);
}

sg_status
sg_deque_ops(sg_deque* d, const uint8_t* is_push, const void* values, int64_t n, void* out_popped, uint8_t* out_ok,
             void* stream)
{
    return deque_ops(d, is_push, values, n, out_popped, out_ok, false, stream);
}

sg_status
sg_deque_ops_zero(sg_deque* d, const uint8_t* is_push, const void* values, int64_t n, void* out_popped,
                  uint8_t* out_ok, void* stream)
{
    return deque_ops(d, is_push, values, n, out_popped, out_ok, true, stream);
}

sg_status
sg_deque_pop_front(sg_deque* d, int64_t n, void* out_popped, uint8_t* out_ok, void* stream)
{
    return deque_end_ops<kPopFront>(d, nullptr, n, out_popped, out_ok, true, stream);
}

sg_status
sg_deque_size(sg_deque* d, void* stream, int64_t* out_size)
{
    if (d == nullptr || out_size == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaStream_t s = as_stream(stream);
    static_assert(sizeof(deque_counters) % 8 == 0 && sizeof(deque_counters) <= 32 * 8, "one warp copies the counters");
    SG_CUDA_TRY(launch_early(k_read_words, 1, 32, s, reinterpret_cast<const unsigned long long*>(d->counters),
                             reinterpret_cast<unsigned long long*>(d->host),
                             static_cast<int>(sizeof(deque_counters) / 8)));
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    const long long x = d->host->size;
    *out_size = x < 0 ? 0 : (x > d->capacity ? d->capacity : x);
    return (d->host->error & kDequeErrWait) != 0u ? SG_ERR_RETRY_EXHAUSTED : SG_OK;
}

sg_status
sg_deque_copy_out(sg_deque* d, void* out, void* stream, int64_t* out_n)
{
    if (d == nullptr || out == nullptr || out_n == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    cudaStream_t s = as_stream(stream);
    int64_t n = 0;
    sg_status st = sg_deque_size(d, stream, &n);
    if (st != SG_OK)
    {
        return st;
    }
    if (n > 0)
    {
        const int grid = grid_for(n, kCThreads, 4096);
        if (d->elem_bytes == 4)
        {
            k_deque_copy_out<uint32_t><<<grid, kCThreads, 0, s>>>(static_cast<const uint32_t*>(d->data), d->counters,
                                                                  d->capacity, static_cast<uint32_t*>(out));
        }
        else
        {
            k_deque_copy_out<unsigned long long><<<grid, kCThreads, 0, s>>>(
                    static_cast<const unsigned long long*>(d->data), d->counters, d->capacity,
                    static_cast<unsigned long long*>(out));
        }
        SG_LAUNCH_CHECK();
        SG_CUDA_TRY(cudaStreamSynchronize(s));
    }
    *out_n = n;
    return SG_OK;
}

sg_status
sg_deque_view_of(const sg_deque* d, sg_deque_view* out)
{
    if (d == nullptr || out == nullptr)
    {
        return SG_ERR_BAD_ARG;
    }
    out->data = d->data;
    out->seq = d->seq;
    out->counters = d->counters;
    out->capacity = d->capacity;
    out->elem_bytes = d->elem_bytes;
    out->pad = 0;
    out->slot_state = d->slot_state;
    out->sync = d->sync;
    return SG_OK;
}

sg_status
sg_bitset_count(const uint32_t* blocks, int64_t nbits, void* stream, int64_t* out_count)
{
    if (out_count == nullptr || nbits < 0 || (nbits > 0 && blocks == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    if (nbits == 0)
    {
        *out_count = 0;
        return SG_OK;
    }
    int dev = 0;
    SG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
    {
        return SG_ERR_NO_DEVICE;
    }
    cudaStream_t s = as_stream(stream);
    std::lock_guard<std::mutex> lock(g_count_mutex);
    count_scratch& sc = g_count_scratch[dev];
    if (sc.partials == nullptr)
    {
        const int blocks_max = count_grid();
        SG_CUDA_TRY(cudaMalloc(&sc.partials, static_cast<size_t>(blocks_max + 1) * sizeof(unsigned long long)));
        SG_CUDA_TRY(cudaMallocHost(&sc.host, sizeof(unsigned long long)));
        sc.blocks = blocks_max;
    }
    const int64_t nvec = (nbits + 127) / 128;
    const int grid = grid_for(nvec, kCountThreads * 4, sc.blocks);
    SG_CUDA_TRY(launch_early(k_bitset_count, grid, kCountThreads, s, blocks, nbits, sc.partials));
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(launch_early(k_sum_partials, 1, 1024, s, sc.partials, grid, sc.host)); // straight into the pinned result
    SG_LAUNCH_CHECK();
    SG_CUDA_TRY(cudaStreamSynchronize(s));
    *out_count = static_cast<int64_t>(*sc.host);
    return SG_OK;
}

} // extern "C"

namespace
{

// Device address of the fixed scratch array, looked up once per device with that device current.
std::mutex g_noalloc_mutex;
unsigned long long* g_noalloc_ptr[64] = {};

sg_status
noalloc_scratch(unsigned long long** out)
{
    int dev = 0;
    SG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
    {
        return SG_ERR_NO_DEVICE;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_ptr[dev] == nullptr)
    {
        void* p = nullptr;
        // the symbol name in host code is a host-side stand-in; the kernels need its device address
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess || p == nullptr)
        {
            cudaGetLastError();
            return SG_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = static_cast<unsigned long long*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return SG_OK;
}

} // namespace

extern "C" {

sg_status
sg_bitset_count_noalloc(const uint32_t* blocks, int64_t nbits, int64_t* out_count, void* stream)
{
    if (out_count == nullptr || nbits < 0 || (nbits > 0 && blocks == nullptr))
    {
        return SG_ERR_BAD_ARG;
    }
    if (nbits > kNoAllocMaxBits)
    {
        return SG_ERR_BAD_ARG; // more chunks than the fixed scratch array holds partial sums for
    }
    unsigned long long* scratch = nullptr;
    sg_status st = noalloc_scratch(&scratch);
    if (st != SG_OK)
    {
        return st;
    }
    cudaStream_t s = as_stream(stream);
    const int64_t nwords = (nbits + 31) / 32;
    const int chunks = static_cast<int>((nwords + kNoAllocChunkWords - 1) / kNoAllocChunkWords);
    if (chunks > 0)
    {
        k_bitset_count_chunked<<<chunks, kCountThreads, 0, s>>>(blocks, nbits, scratch);
        SG_LAUNCH_CHECK();
    }
    SG_CUDA_TRY(launch_early(k_sum_partials, 1, 1024, s, scratch, chunks,
                             reinterpret_cast<unsigned long long*>(out_count)));
    SG_LAUNCH_CHECK();
    return SG_OK;
}

} // extern "C"
