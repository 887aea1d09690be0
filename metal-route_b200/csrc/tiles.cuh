// tiles.cuh — label arithmetic and the tile work queue shared by the relax kernels.
//
// Labels are u64 = dist << 32 | hops (device.cuh).  The queue is the
// asynchronous schedule's: a ticketed ring of (field, tile) items plus one
// state word per tile, so a tile is queued at most once and held by one worker
// (a CTA or a warp) at a time.
#pragma once

#include "device.cuh"
#include "kernels.h"

namespace mrc {

// Label extended by a run of `h` steps whose prices sum to `d` (kMax = blocked or
// saturated); a dist reaching 0xFFFFFFFF is unreachable.  With 32-bit wrapping
// addition, td or d equal to kMax always gives nd < td or nd == kMax, so those
// two tests cover the blocked operands too.
__device__ __forceinline__ u64 ext2(u64 t, uint32_t d, uint32_t h) {
    const uint32_t td = (uint32_t)(t >> 32);
    const uint32_t nd = td + d;
    const bool bad = (nd < td) | (nd == kMax);
    return bad ? kInf : (((u64)nd << 32) | (uint32_t)((uint32_t)t + h));
}

// Saturating sum of step prices; kMax absorbs (an operand equal to kMax gives
// s == kMax or s < a under wrapping addition).
__device__ __forceinline__ uint32_t dsum(uint32_t a, uint32_t b) {
    const uint32_t s = a + b;
    return s < a ? kMax : s;
}

// The word of a step price in the layer kernel's planes, exact for every price below
// 2^31 - 1: price << kLayerHopBits | 1 where that stays below 2^29 (a packed word),
// else the price itself with the top bit set; kPackedInf for no step, kPriceLook for a
// price to be formed from the board's words.
constexpr uint32_t kPriceLook = 0xFFFFFFFFu, kPricePlain = 1u << 31;
__device__ __forceinline__ uint32_t plane_word(uint32_t p) {
    if (p < (1u << (29 - kLayerHopBits))) return (p << kLayerHopBits) | 1u;
    return p == kMax ? kPackedInf : p < kPriceLook - kPricePlain ? kPricePlain | p : kPriceLook;
}
// The price of a word; `look` forms one that no word holds.
template <class Look>
__device__ __forceinline__ uint32_t plane_price(uint32_t word, Look look) {
    if (word < kPackedInf) return word >> kLayerHopBits;
    return word == kPackedInf ? kMax : word == kPriceLook ? look() : word & (kPricePlain - 1u);
}

__device__ __forceinline__ u64 umin64(u64 a, u64 b) { return a < b ? a : b; }

// Work queue of the queue forms.  count[0] = tickets handed to pushers (tail),
// head[0] = tickets handed to poppers, count[1] = items queued or in flight (or,
// goal-directed, unfinished fields).  tags[0, list_cap), list_cap a power of two, is
// the ring: one 64-bit word per slot, lap << 56 | field << 28 | tile, so an item is
// published and taken with one store and one load (zeroed before launch; laps count
// 1..255).  A tile is queued at most once at a time (its tstamp word is the queued
// flag), so at most list_cap items are queued at once.  Nothing keeps a slot for a worker that
// holds its ticket and has not read it yet, though, while other tiles go round the ring: that
// is a margin, not a handshake.  A ring has kMinRing slots at least, more than three
// times the workers of any launch (2368 warps of the warp schedule), so a worker would
// have to miss three items of every other worker, microseconds each, between two polls,
// which lie at most 128 ns apart; an item lost that way would end the launch with
// kStatusBarrier.
constexpr uint32_t kQueueSpinLimit = 1u << 25;  // polls of one wait (seconds with the backoff below)
constexpr u64 kSlotItem = (1ull << 56) - 1;     // the item bits of a slot word; all ones: the launch is over

__device__ __forceinline__ u64 queue_lap(const RelaxArgs &a, uint32_t h) {
    return (u64)((h >> (31 - __clz((int)a.list_cap))) % 255u + 1u) << 56;
}
// Publishes item (fi, u) under ticket h; what the item relies on was ordered before.
__device__ __forceinline__ void queue_store(const RelaxArgs &a, uint32_t h, u64 item) {
    __stcg(a.tags + (h & (a.list_cap - 1u)), queue_lap(a, h) | item);
}
__device__ __forceinline__ u64 queue_item(uint32_t fi, uint32_t u) { return ((u64)fi << 28) | u; }

// Tile states in the tstamp word: 0 idle, 1 queued, 2 held by a worker,
// 3 held and improved again meanwhile (the holder continues it in place, or
// queues it once more, when it finishes, so improvements that arrive during a
// relaxation share one re-activation and no tile is ever relaxed by two
// workers at once).
constexpr uint32_t kTileIdle = 0, kTileQueued = 1, kTileHeld = 2, kTileHeldDirty = 3;

// `live`: the count of items queued or in flight, the launch's (count[1]) or, in
// a goal-directed launch, the field's (count[1] then counts unfinished fields).
__device__ __forceinline__ void async_enqueue(const RelaxArgs &a, uint32_t fi, uint32_t u, uint32_t *live) {
    atomicAdd(live, 1u);  // in flight before it is visible
    const uint32_t h = atomicAdd(&a.ctl->count[0], 1u);
    __threadfence();
    queue_store(a, h, queue_item(fi, u));
}

__device__ __forceinline__ void async_push(const RelaxArgs &a, uint32_t fi, uint32_t tile_off, uint32_t u,
                                           uint32_t *live) {
    uint32_t *st = a.tstamp + tile_off + u;
    for (int tries = 0; tries < 1024; ++tries) {
        const uint32_t old = atomicCAS(st, kTileIdle, kTileQueued);
        if (old == kTileIdle) {
            async_enqueue(a, fi, u, live);
            return;
        }
        if (old == kTileQueued || old == kTileHeldDirty) return;  // it will read our labels
        if (atomicCAS(st, kTileHeld, kTileHeldDirty) == kTileHeld) return;
        // the holder finished in between: try again from idle
    }
    atomicOr(&a.ctl->status, kStatusQueueOverflow);  // the state kept changing under us
}

// Called by the holder after its write-back and pushes: release the tile, or
// queue it again if a neighbour improved it while it was held.
__device__ __forceinline__ void async_release(const RelaxArgs &a, uint32_t fi, uint32_t tile_off, uint32_t t) {
    uint32_t *st = a.tstamp + tile_off + t;
    if (atomicCAS(st, kTileHeld, kTileIdle) == kTileHeldDirty) {
        atomicExch(st, kTileQueued);
        async_enqueue(a, fi, t, &a.ctl->count[1]);
    }
}

// Whether the launch has failed: a limit was passed, or a wait ran out.
__device__ __forceinline__ bool launch_failed(const RelaxArgs &a) {
    return *(volatile const uint32_t *)&a.ctl->status != 0u;
}

// A CTA's count of activations not yet added to the launch's, once it is to leave.
constexpr unsigned long long kLeaveLaunch = ~0ull;

// Adds a worker's activations and sweeps to the launch's.  False: the launch has
// failed, by too many activations or otherwise, and the worker leaves it.  A
// queue that never runs dry keeps its workers from waiting, and so from reading the
// status word in async_pop; they read it here, every kCountBatch activations.
__device__ __forceinline__ bool count_flush(const RelaxArgs &a, unsigned long long acts, unsigned long long sweeps) {
    if (atomicAdd(&a.ctl->activations, acts) + acts > a.activation_limit)
        atomicOr(&a.ctl->status, kStatusActivationLimit);
    atomicAdd(&a.ctl->sweeps, sweeps);
    return !launch_failed(a);
}

// Next item for the calling worker (one thread) as field << 32 | tile, or kInf when
// no work is left.  The wait is bounded: kQueueSpinLimit polls, then
// kStatusBarrier and an exit.  Each waiter polls its own slot; the shared words
// (the in-flight count, the status) are read every kCheck-th poll, and the sleep
// between polls doubles up to 128 ns: a longer one delays every hop of a lone
// field, whose next item goes to the CTA that has waited longest.
template <uint32_t kCheck = 16>
__device__ __forceinline__ u64 async_pop(const RelaxArgs &a) {
    Ctl *c = a.ctl;
    const uint32_t h = atomicAdd(&c->head[0], 1u);
    const volatile u64 *slot = a.tags + (h & (a.list_cap - 1u));
    const u64 lap = queue_lap(a, h);
    for (uint32_t spins = 0;; ++spins) {
        const u64 v = *slot;
        if ((v & ~kSlotItem) == lap) {
            __threadfence();
            const u64 item = v & kSlotItem;
            return item == kSlotItem ? kInf : ((item >> 28) << 32) | (item & 0xFFFFFFFu);
        }
        if (spins % kCheck == kCheck - 1u) {
            if (*(volatile const uint32_t *)&c->count[1] == 0u) return kInf;  // nothing queued or running
            if (launch_failed(a)) return kInf;
        }
        if (spins > kQueueSpinLimit) {
            atomicOr(&c->status, kStatusBarrier);
            return kInf;
        }
        __nanosleep(spins < 32u ? 20u : spins < 64u ? 64u : 128u);
    }
}

// Planes of step prices into a cell: from -x, +x, -y, +y, the layer below, the
// layer above (the order of the price planes and of a staged tile's planes).
enum { kInNegX = 0, kInPosX = 1, kInNegY = 2, kInPosY = 3, kInBelow = 4, kInAbove = 5 };

// Exact price of the step into cell c (at l, y, x) from direction `dir`, with
// the net's own pads, endpoints, via exemptions and directed-price overrides (the staging rules of the
// CTA-wide relax kernel without price planes, negotiated.rs:2914-2966 and :3010-3043).
static __device__ __noinline__ uint32_t exact_in_price(const DevBoard &b, const DevField &f, const uint32_t *pads, int dir, uint32_t c,
                                   uint32_t l, uint32_t y, uint32_t x) {
    const uint8_t fc = b.flags ? __ldg(b.flags + c) : 0;
    const uint32_t ec = cell_enter(b, f, pads, c, fc);
    if (ec == kMax) return kMax;
    const uint32_t plane = b.w * b.h;
    if (dir == kInBelow || dir == kInAbove) {
        const bool below = dir == kInBelow;
        if (below ? l == 0 : l + 1 >= b.layers) return kMax;
        const uint32_t k = below ? l - 1 : l;
        if (!((b.via_mask >> k) & 1u)) return kMax;
        const uint32_t p = below ? c - plane : c + plane;
        const uint8_t fp = b.flags ? __ldg(b.flags + p) : 0;
        if ((cell_tile_flags(f, pads, c, fc) | cell_tile_flags(f, pads, p, fp)) & kViaBlocked) return kMax;
        return capmul(__ldg(b.via_edge + k), ec);
    }
    uint32_t p, base;
    uint8_t out_bit, in_bit;
    if (dir == kInNegX) {
        if (x == 0) return kMax;
        p = c - 1;
        base = b.directed ? field_directed(b, f, c, 1) : __ldg(b.x_edge + x - 1);
        out_bit = kEdgePosX;
        in_bit = kEdgeNegX;
    } else if (dir == kInPosX) {
        if (x + 1 >= b.w) return kMax;
        p = c + 1;
        base = b.directed ? field_directed(b, f, c, 2) : __ldg(b.x_edge + x);
        out_bit = kEdgeNegX;
        in_bit = kEdgePosX;
    } else if (dir == kInNegY) {
        if (y == 0) return kMax;
        p = c - b.w;
        base = b.directed ? field_directed(b, f, c, 0) : __ldg(b.y_edge + y - 1);
        out_bit = kEdgePosY;
        in_bit = kEdgeNegY;
    } else {
        if (y + 1 >= b.h) return kMax;
        p = c + b.w;
        base = b.directed ? field_directed(b, f, c, 3) : __ldg(b.y_edge + y);
        out_bit = kEdgeNegY;
        in_bit = kEdgePosY;
    }
    const uint8_t fp = b.flags ? __ldg(b.flags + p) : 0;
    if ((fp & out_bit) | (fc & in_bit)) return kMax;
    if (b.directed && base == kMax) return kMax;
    return capmul(base, ec);
}

}  // namespace mrc
