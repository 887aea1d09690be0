// relax.cu — the batched field + canonical path kernels.
//
// relax_rounds_kernel: one cooperative persistent launch solves every field
// (net x window) of a batch.  Each field's labels live in HBM as u64
// (dist << 32 | hops), window-packed like the reference's ragged layout
// (metal/src/lib.rs:833-871).  Windows are cut into tiles of 32 x TH cells over
// every layer.  Work proceeds in bulk-synchronous rounds over a shared list of
// active (field, tile) items: a CTA stages a tile plus a one-cell halo ring in
// shared memory, relaxes it to local convergence with directional sweeps (the
// edge-aware row / column / layer-stack sweeps of gpu.rs:259-430, run on-chip
// instead of one dispatch per round), writes it back and queues each neighbour
// whose halo it now improves for the next round.  A field is final when no
// tile of it is queued; the launch ends when the whole list drains.
//
// Tiles of one field run concurrently in different CTAs.  That is safe because
// labels only decrease, every label is one aligned 64-bit word (a halo read is
// an old or a new label, never a torn mix), labels are read through L2
// (ld.global.cg) so no SM sees a stale L1 line, and a tile is processed by at
// most one CTA per round.  A neighbour read before it improves is re-queued by
// that neighbour's own push check, so no improvement is lost.
//
// path kernels: the path length is hops[dst] + 1 (every canonical predecessor
// has exactly one fewer hop), so offsets come from one device scan and one warp
// per net walks dst -> src choosing the lowest-CellIdx predecessor whose label
// and step reproduce the current label (metal/src/lib.rs:308-396).
#include <cuda_runtime.h>

#include <algorithm>

#include "cta_tile.cuh"
#include "device.cuh"
#include "kernels.h"
#include "tiles.cuh"

namespace mrc {

constexpr uint32_t kBarrierSpinLimit = 1u << 25;  // ~ seconds with the backoff below

// Grid-wide barrier for a cooperative launch.  The wait is bounded: after
// kBarrierSpinLimit polls it records kStatusBarrier and returns, and every CTA
// leaves the round loop once the status word is non-zero.
__device__ void grid_barrier(Ctl *c, uint32_t nblocks, uint32_t spin_limit = kBarrierSpinLimit) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        volatile uint32_t *gen_p = &c->bar_gen;
        const uint32_t gen = *gen_p;
        const uint32_t arrived = atomicAdd(&c->bar_count, 1u) + 1u;
        if (arrived == nblocks) {
            atomicExch(&c->bar_count, 0u);
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        } else {
            uint32_t spins = 0;
            while (*gen_p == gen) {
                if (++spins > spin_limit) {
                    atomicOr(&c->status, kStatusBarrier);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t ld_status(const Ctl *c) { return *(volatile const uint32_t *)&c->status; }


template <int TH, int NT, bool OV>
__global__ void __launch_bounds__(NT) relax_rounds_kernel(RelaxArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ u64 s_item;
    Ctl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x;
    const uint32_t cap = a.list_cap;
    // ---- round 0: every field's source tile ---------------------------------
    for (uint32_t fi = blockIdx.x * blockDim.x + tid; fi < a.n_fields; fi += gridDim.x * blockDim.x) {
        const DevField f = a.fields[fi];
        const DevBoard b = a.boards[f.board];
        const uint32_t plane = b.w * b.h;
        const uint32_t sr = f.src % plane, sx = sr % b.w, sy = sr / b.w;
        const uint8_t sfl = b.flags ? b.flags[f.src] : 0;
        if (sx >= f.x0 && sx < f.x0 + f.ww && sy >= f.y0 && sy < f.y0 + f.wh &&
            cell_enter(b, f, a.pads, f.src, sfl) != kMax) {
            const uint32_t t = ((sy - f.y0) / TH) * field_ntx(f) + (sx - f.x0 + f.xa) / kTW;
            a.tstamp[f.tile_off + t] = 1u;
            const uint32_t idx = atomicAdd(&ctl->count[0], 1u);
            a.lists[idx] = ((u64)fi << 32) | t;
        }
    }
    grid_barrier(ctl, gridDim.x);

    for (uint32_t round = 0;; ++round) {
        const uint32_t cur = round % 3, old = (round + 2) % 3;
        const uint32_t n = *(volatile uint32_t *)&ctl->count[cur];
        if (n == 0 || ld_status(ctl)) break;
        if (round >= a.round_limit) {
            if (blockIdx.x == 0 && tid == 0) atomicOr(&ctl->status, kStatusRoundLimit);
            break;
        }
        if (blockIdx.x == 0 && tid == 0) {
            ctl->count[old] = 0;
            ctl->head[old] = 0;
            ctl->rounds = round + 1;
        }
        for (;;) {
            if (tid == 0) {
                const uint32_t idx = atomicAdd(&ctl->head[cur], 1u);
                s_item = idx < n ? __ldcg(a.lists + (size_t)cur * cap + idx) : kInf;
            }
            __syncthreads();
            const u64 item = s_item;
            if (item == kInf) break;
            process_item<TH, false, OV, false>(a, (uint32_t)(item >> 32), (uint32_t)item, round, smem_raw, nullptr);
        }
        grid_barrier(ctl, gridDim.x);
    }
}

// Asynchronous form: no rounds.  Every CTA pops items from one ticketed queue
// and pushes the neighbours it improves; the launch ends when no item is
// queued or in flight.  The label arena is +inf-initialised (every label is
// valid from the start), and a tile is held by one CTA at a time: improvements
// that reach a held tile mark it dirty and its holder queues it once more.
// 64 registers a thread: four 256-thread CTAs per SM
template <int TH, int NT, bool OV>
__global__ void __launch_bounds__(NT, 65536 / (NT * 64)) relax_async_kernel(RelaxArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ u64 s_item;
    __shared__ unsigned long long s_cnt[2];  // activations and sweeps not yet added to the launch's
    if (threadIdx.x == 0) s_cnt[0] = s_cnt[1] = 0;
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) s_item = s_cnt[0] == kLeaveLaunch ? kInf : async_pop(a);
        __syncthreads();
        const u64 item = s_item;
        if (item == kInf) break;
        process_item<TH, true, OV, false>(a, (uint32_t)(item >> 32), (uint32_t)item, 0, smem_raw, s_cnt);
    }
    if (threadIdx.x == 0) {
        if (s_cnt[0] && s_cnt[0] != kLeaveLaunch) atomicAdd(&a.ctl->activations, s_cnt[0]);
        if (s_cnt[1]) atomicAdd(&a.ctl->sweeps, s_cnt[1]);
    }
}

// Seeds of the asynchronous form: the source label and the source tile of
// every field whose source is inside its window and enterable.
template <int TH>
__global__ void async_seed_kernel(RelaxArgs a) {
    for (uint32_t fi = blockIdx.x * blockDim.x + threadIdx.x; fi < a.n_fields; fi += gridDim.x * blockDim.x) {
        const DevField f = a.fields[fi];
        const DevBoard b = a.boards[f.board];
        const uint32_t plane = b.w * b.h;
        const uint32_t sl = f.src / plane, sr = f.src % plane, sx = sr % b.w, sy = sr / b.w;
        const uint8_t sfl = b.flags ? b.flags[f.src] : 0;
        if (sx >= f.x0 && sx < f.x0 + f.ww && sy >= f.y0 && sy < f.y0 + f.wh &&
            cell_enter(b, f, a.pads, f.src, sfl) != kMax) {
            a.lab[f.lab_off + ((uint64_t)sl * f.wh + (sy - f.y0)) * f.ww + (sx - f.x0)] = 0;
            const uint32_t t = ((sy - f.y0) / TH) * field_ntx(f) + (sx - f.x0 + f.xa) / kTW;
            __threadfence();
            uint32_t *live = &a.ctl->count[1];
            if (a.goal) {  // goal-directed: the launch counts fields, the field its items
                const BoardGoal bg = *b.goal;
                const uint32_t dl = f.dst / plane, dr = f.dst % plane, dx = dr % b.w, dy = dr / b.w;
                const uint32_t e = goal_weight(bg, f), each = ~bg.inv_min_dir;
                const uint32_t f0 = min(dsum(dsum(goal_rest(b.directed ? nullptr : b.x_sum, each, e, sx, dx),
                                                  goal_rest(b.directed ? nullptr : b.y_sum, each, e, sy, dy)),
                                             goal_rest(b.via_sum, 0, e, sl, dl)), kCap);
                // First threshold: room for two vias, a detour of two cells, and a share
                // of the bound.  A path through random prices avoids the dear ones: its
                // mean step lies about a third of the way from the cheapest to the mean
                // price (congestion board: path cost 1.38 x the bound where mean /
                // cheapest is 2.3; negotiation board 1.01 x at 1.1).  Relax us with a share
                // of 0, 0.17, 0.25, 0.35, 0.45 and 0.6 of that distance: two congestion
                // boards 1906, 1617, 1420, 1449, 1449, 1520 and 2047, 1690, 1540, 1503,
                // 1537, 1575; negotiation boards of 1280 x 1153 x 6 and 640 x 500 x 4 1487,
                // 1520, 1571, 1530, 1545, 1578 and 761, 666, 676, 662, 670, 668; 512 uneven
                // instances 750 at each.  With a zero bound nothing waits.
                float spread = 1.0f;  // mean over cheapest price
                if (bg.n_cost && ~bg.inv_min_cost) spread *= (float)bg.sum_cost / (float)bg.n_cost / (float)~bg.inv_min_cost;
                if (b.directed && bg.n_dir && each) spread *= (float)bg.sum_dir / (float)bg.n_dir / (float)each;
                spread = fminf(fmaxf(0.35f * (spread - 1.0f), 0.0f), 2.0f);
                const u64 room = (u64)((double)spread * f0) + 2ull * capmul(b.min_via, e) +
                                 4ull * capmul(b.directed ? each : b.min_gap, e);
                FieldGoal g{};
                g.ub = kMax;
                g.f0 = f0;
                g.thr = (f0 == 0 || f0 + room >= kCap) ? kMax : (uint32_t)(f0 + room);
                a.goal[fi] = g;
                __threadfence();
                atomicAdd(live, 1u);
                live = &a.goal[fi].active;
            }
            async_push(a, fi, f.tile_off, t, live);
        }
    }
}

// Label of a window cell after the relax launch (unvisited tiles are unreached).
__device__ __forceinline__ u64 field_label(const PathArgs &a, const DevField &f, uint32_t lx, uint32_t ly,
                                           uint32_t l) {
    if (!a.arena_filled) {
        const uint32_t t = (ly >> (__ffs((int)a.tile_h) - 1)) * field_ntx(f) + (lx + f.xa) / kTW;  // tile heights are powers of two
        if (!a.tvisit[f.tile_off + t]) return kInf;
    }
    return a.lab[f.lab_off + ((uint64_t)l * f.wh + ly) * f.ww + lx];
}

// Per field: search cost and path length (hops[dst] + 1), then an exclusive
// scan into path offsets.  Single CTA; loops over the fields in chunks.
__global__ void __launch_bounds__(1024) path_offsets_kernel(PathArgs a) {
    __shared__ unsigned long long warp_sums[32];
    __shared__ unsigned long long carry;
    // phase 1: cost and length of every field, stored at its output slot
    for (uint32_t i = threadIdx.x; i < a.n_fields; i += blockDim.x) {
        const DevField f = a.fields[i];
        const DevBoard b = a.boards[f.board];
        const uint32_t plane = b.w * b.h;
        const uint32_t dl = f.dst / plane, dr = f.dst % plane;
        const uint32_t dx = dr % b.w, dy = dr / b.w;
        uint32_t cost = kMax, len = 0;
        if (dx >= f.x0 && dx < f.x0 + f.ww && dy >= f.y0 && dy < f.y0 + f.wh) {
            const u64 v = field_label(a, f, dx - f.x0, dy - f.y0, dl);
            cost = (uint32_t)(v >> 32);
            if (cost != kMax) len = (uint32_t)v + 1u;
            // a simple path never has more cells than its window
            if ((uint64_t)len > (uint64_t)f.ww * f.wh * b.layers) {
                atomicOr(a.status, kStatusPathBroken);
                len = 0;
            }
        }
        a.costs[f.out] = cost;
        a.lens[f.out] = len;
    }
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    // phase 2: exclusive scan of the lengths in output order
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (uint32_t base = 0; base < a.n_fields; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const unsigned long long v = (i < a.n_fields) ? (unsigned long long)a.lens[i] : 0ull;
        unsigned long long x = v;
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31) warp_sums[wid] = x;
        __syncthreads();
        if (wid == 0) {
            unsigned long long w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0ull;
            for (int o = 1; o < 32; o <<= 1) {
                unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, w, o);
                if (lane >= (uint32_t)o) w += y;
            }
            warp_sums[lane] = w;
        }
        __syncthreads();
        const unsigned long long excl = carry + (wid ? warp_sums[wid - 1] : 0ull) + x - v;
        if (i < a.n_fields) a.offsets[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) a.offsets[a.n_fields] = carry;
}

// Step price of the move p -> cur for the walk and the plain form.
// kind: 0 = p is cur's lower layer, 1 = -y, 2 = -x, 3 = +x, 4 = +y, 5 = upper layer.
__device__ __forceinline__ uint32_t global_step(const DevBoard &b, const DevField &f, const uint32_t *pads,
                                                uint32_t p, uint32_t cur, int kind) {
    const uint8_t fc = b.flags ? b.flags[cur] : 0, fp = b.flags ? b.flags[p] : 0;
    const uint32_t ec = cell_enter(b, f, pads, cur, fc);
    if (ec == kMax) return kMax;
    const uint32_t plane = b.w * b.h;
    const uint32_t r = cur % plane, x = r % b.w, y = r / b.w, l = cur / plane;
    if (kind == 0 || kind == 5) {
        const uint32_t k = kind == 0 ? l - 1 : l;
        if (!((b.via_mask >> k) & 1u)) return kMax;
        const uint8_t tc = cell_tile_flags(f, pads, cur, fc), tp = cell_tile_flags(f, pads, p, fp);
        if ((tc | tp) & kViaBlocked) return kMax;
        return capmul(__ldg(b.via_edge + k), ec);
    }
    uint8_t out_bit, in_bit;
    uint32_t base;
    if (kind == 1) {  // p at -y: p moves +y
        out_bit = kEdgePosY;
        in_bit = kEdgeNegY;
        base = b.directed ? field_directed(b, f, cur, 0) : __ldg(b.y_edge + y - 1);
    } else if (kind == 2) {  // p at -x: p moves +x
        out_bit = kEdgePosX;
        in_bit = kEdgeNegX;
        base = b.directed ? field_directed(b, f, cur, 1) : __ldg(b.x_edge + x - 1);
    } else if (kind == 3) {  // p at +x: p moves -x
        out_bit = kEdgeNegX;
        in_bit = kEdgePosX;
        base = b.directed ? field_directed(b, f, cur, 2) : __ldg(b.x_edge + x);
    } else {  // p at +y: p moves -y
        out_bit = kEdgeNegY;
        in_bit = kEdgePosY;
        base = b.directed ? field_directed(b, f, cur, 3) : __ldg(b.y_edge + y);
    }
    if ((fp & out_bit) | (fc & in_bit)) return kMax;
    if (b.directed && base == kMax) return kMax;
    return capmul(base, ec);
}

// global_step for the path walk with every load issued before any is used
// (the flags of both cells, the enter cost and the base price), so a step costs
// one memory round trip instead of a chain of dependent ones.
// own: cur's tile holds directed-price overrides of this field.
__device__ __forceinline__ uint32_t walk_step(const DevBoard &b, const DevField &f, const uint32_t *pads,
                                              uint32_t p, uint32_t cur, uint32_t x, uint32_t y, uint32_t l, int kind,
                                              bool own) {
    const uint8_t fc = b.flags ? __ldg(b.flags + cur) : 0, fp = b.flags ? __ldg(b.flags + p) : 0;
    const uint32_t cc = __ldg(b.cost + cur);
    uint32_t base = 0;
    if (kind == 0) base = __ldg(b.via_edge + l - 1);
    else if (kind == 5) base = __ldg(b.via_edge + l);
    else if (b.directed) {
        const int slot = kind == 1 ? 0 : kind == 2 ? 1 : kind == 3 ? 2 : 3;
        base = own ? field_directed(b, f, cur, slot)
                   : __ldg(reinterpret_cast<const uint32_t *>(b.directed + cur) + slot);
    }
    else if (kind == 1) base = __ldg(b.y_edge + y - 1);
    else if (kind == 2) base = __ldg(b.x_edge + x - 1);
    else if (kind == 3) base = __ldg(b.x_edge + x);
    else base = __ldg(b.y_edge + y);
    // cell_enter on the loaded values
    uint32_t ec;
    if (fc & kTraceNode) ec = kMax;
    else if (cc != kMax) ec = cc;
    else ec = (cur == f.src || cur == f.dst || sorted_has(pads + f.pad_off, f.n_pads, cur)) ? 1u : kMax;
    if (ec == kMax) return kMax;
    if (kind == 0 || kind == 5) {
        const uint32_t k = kind == 0 ? l - 1 : l;
        if (!((b.via_mask >> k) & 1u)) return kMax;
        const uint8_t tc = cell_tile_flags(f, pads, cur, fc), tp = cell_tile_flags(f, pads, p, fp);
        if ((tc | tp) & kViaBlocked) return kMax;
        return capmul(base, ec);
    }
    uint8_t out_bit, in_bit;
    if (kind == 1) {
        out_bit = kEdgePosY;
        in_bit = kEdgeNegY;
    } else if (kind == 2) {
        out_bit = kEdgePosX;
        in_bit = kEdgeNegX;
    } else if (kind == 3) {
        out_bit = kEdgeNegX;
        in_bit = kEdgePosX;
    } else {
        out_bit = kEdgeNegY;
        in_bit = kEdgePosY;
    }
    if ((fp & out_bit) | (fc & in_bit)) return kMax;
    if (b.directed && base == kMax) return kMax;
    return capmul(base, ec);
}

// Neighbour `kind` of (x, y, l): 0 the layer below, 1 -y, 2 -x, 3 +x, 4 +y,
// 5 the layer above (ascending CellIdx); kind 5 - k is the opposite of k.
__device__ __forceinline__ void walk_offset(int kind, int &x, int &y, int &l) {
    if (kind == 0) l -= 1;
    else if (kind == 1) y -= 1;
    else if (kind == 2) x -= 1;
    else if (kind == 3) x += 1;
    else if (kind == 4) y += 1;
    else l += 1;
}

// Label of window cell (x, y, l) (absolute coordinates inside the window), or
// +inf when its tile was never visited.
__device__ __forceinline__ u64 walk_label(const PathArgs &a, const DevField &f, uint32_t ntx, uint32_t tile_shift,
                                          int x, int y, int l) {
    const uint32_t lx = (uint32_t)x - f.x0, ly = (uint32_t)y - f.y0;
    const u64 raw = a.lab[f.lab_off + ((uint64_t)(uint32_t)l * f.wh + ly) * f.ww + lx];
    if (a.arena_filled) return raw;
    return a.tvisit[f.tile_off + (ly >> tile_shift) * ntx + (lx + f.xa) / kTW] ? raw : kInf;
}

__device__ __forceinline__ bool walk_inside(const DevField &f, const DevBoard &b, int x, int y, int l) {
    return l >= 0 && l < (int)b.layers && x >= (int)f.x0 && x < (int)(f.x0 + f.ww) && y >= (int)f.y0 &&
           y < (int)(f.y0 + f.wh);
}

// Is the neighbour `kind` of target t = (tx, ty, tl) a predecessor of t, i.e.
// its label extended by the step into t equals `need`?  Its cell and label are
// returned for the caller to carry forward.
// (px, py, pl) is that neighbour, computed by the caller.
__device__ __forceinline__ bool walk_try(const PathArgs &a, const DevField &f, const DevBoard &b, uint32_t ntx,
                                         uint32_t tile_shift, int tx, int ty, int tl, uint32_t t, u64 need, int kind,
                                         int px, int py, int pl, uint32_t *q, u64 *lq) {
    if (!walk_inside(f, b, px, py, pl)) return false;
    *q = ((uint32_t)pl * b.h + (uint32_t)py) * b.w + (uint32_t)px;
    *lq = walk_label(a, f, ntx, tile_shift, px, py, pl);
    bool own = false;
    if (a.tover && f.n_over)
        own = a.tover[f.tile_off + (((uint32_t)ty - f.y0) >> tile_shift) * ntx + ((uint32_t)tx - f.x0 + f.xa) / kTW] != 0;
    const uint32_t st = walk_step(b, f, a.pads, *q, t, (uint32_t)tx, (uint32_t)ty, (uint32_t)tl, kind, own);
    return *lq != kInf && extend(*lq, st) == need;
}

// One warp per field: lanes 0..5 test the six neighbours of the current cell
// (ascending CellIdx) and the lowest qualifying one is the canonical
// predecessor.  Each step issues all of its loads at once (the candidate's
// label and tile flag, and the step inputs) and carries the winner's label and
// coordinates forward, so no step divides a cell index.
__global__ void __launch_bounds__(256) path_walk_kernel(PathArgs a) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (warp >= a.n_fields) return;
    const DevField f = a.fields[warp];
    const uint32_t len = a.lens[f.out];
    if (len == 0) return;
    const DevBoard b = a.boards[f.board];
    const uint32_t plane = b.w * b.h;
    const uint32_t ntx = field_ntx(f);
    const uint32_t tile_shift = (uint32_t)(__ffs((int)a.tile_h) - 1);  // tile heights are powers of two
    uint32_t *out = a.cells + a.offsets[f.out];
    uint32_t cur = f.dst;
    int cx, cy, cl;
    {
        const uint32_t r = cur % plane;
        cx = (int)(r % b.w);
        cy = (int)(r / b.w);
        cl = (int)(cur / plane);
    }
    u64 need = walk_label(a, f, ntx, tile_shift, cx, cy, cl);
    int ox = 0, oy = 0, oz = 0;  // this lane's neighbour offset (lanes 0-5), a loop constant
    if (lane < 6) walk_offset((int)lane, ox, oy, oz);
    for (uint32_t pos = len - 1;; --pos) {
        if (lane == 0) out[pos] = cur;
        if (pos == 0) {
            if (lane == 0 && cur != f.src) atomicOr(a.status, kStatusPathBroken);
            return;
        }
        bool ok = false;
        uint32_t p = 0;
        u64 lp = kInf;
        const int px = cx + ox, py = cy + oy, pz = cl + oz;
        if (lane < 6) {
            ok = walk_try(a, f, b, ntx, tile_shift, cx, cy, cl, cur, need, (int)lane, px, py, pz, &p, &lp);
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
        if (m == 0) {
            if (lane == 0) atomicOr(a.status, kStatusPathBroken);
            return;
        }
        const uint32_t win = __ffs(m) - 1;
        cur = __shfl_sync(0xFFFFFFFFu, p, win);
        need = __shfl_sync(0xFFFFFFFFu, lp, win);
        cx = __shfl_sync(0xFFFFFFFFu, px, win);
        cy = __shfl_sync(0xFFFFFFFFu, py, win);
        cl = __shfl_sync(0xFFFFFFFFu, pz, win);
    }
}

// Complete u32 distance field of every field (MRC_FLAG_KEEP_FIELDS).
// The fields come in ascending lab_off order and are emitted in output slot order,
// so that they are downloaded as one block.
__global__ void emit_fields_kernel(PathArgs a, uint32_t *out, uint64_t total) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = a.n_fields;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (a.fields[mid].lab_off <= i) lo = mid;
            else hi = mid;
        }
        const DevField f = a.fields[lo];
        // a window has at most 2^32 cells (the CellIdx domain): 32-bit index math
        const uint32_t li = (uint32_t)(i - f.lab_off);
        const uint32_t rr = li / f.ww, lx = li - rr * f.ww;
        const uint32_t l = rr / f.wh, ly = rr - l * f.wh;
        out[f.out_off + li] = (uint32_t)(field_label(a, f, lx, ly, l) >> 32);
    }
}

// ---- the plain form: one Jacobi round over one field ----------------------
__global__ void plain_round_kernel(PlainArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const DevField f = a.field;
    const DevBoard b = a.board;
    const uint64_t wcells = (uint64_t)f.ww * f.wh * b.layers;
    if (i >= wcells) return;
    const uint32_t lx = (uint32_t)(i % f.ww);
    const uint64_t r = i / f.ww;
    const uint32_t ly = (uint32_t)(r % f.wh), l = (uint32_t)(r / f.wh);
    const uint32_t x = f.x0 + lx, y = f.y0 + ly;
    const uint32_t cur = (l * b.h + y) * b.w + x;
    const u64 old = a.in[i];
    u64 best = old;
    if (!(cur == f.src && best == 0)) {
        const int64_t plane_l = (int64_t)f.ww * f.wh;
        const int64_t off[6] = {-plane_l, -(int64_t)f.ww, -1, 1, (int64_t)f.ww, plane_l};
        const bool has[6] = {l > 0, ly > 0, lx > 0, lx + 1 < f.ww, ly + 1 < f.wh, l + 1 < b.layers};
        const int64_t goff[6] = {-(int64_t)b.w * b.h, -(int64_t)b.w, -1, 1, (int64_t)b.w, (int64_t)b.w * b.h};
        for (int k = 0; k < 6; ++k) {
            if (!has[k]) continue;
            const uint64_t j = (uint64_t)((int64_t)i + off[k]);
            const u64 lp = a.in[j];
            if (lp == kInf) continue;
            const uint32_t p = (uint32_t)((int64_t)cur + goff[k]);
            const u64 cand = extend(lp, global_step(b, f, a.pads, p, cur, k));
            if (cand < best) best = cand;
        }
    }
    a.out[i] = best;
    if (best != old) *a.changed = 1u;
}

// OR Grid::via_forbidden into the flag byte as kStaticVia.
__global__ void combine_flags_kernel(uint8_t *flags, const uint8_t *via_forbidden, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (via_forbidden[i]) flags[i] |= kStaticVia;
}

// ---- gather of page-locked host buffers into HBM ---------------------------
// One launch moves many host spans of one instance set to their places in a
// device block: the SMs read the host memory through its device mapping (PCIe
// reads, 16 bytes a thread, several in flight), so thousands of small and large
// spans cost one launch instead of one copy call each.  The spans are cut into
// 64 KiB chunks and the blocks stride over the chunks.

constexpr uint64_t kGatherChunk = 64u << 10;

// 0x80 in each nonzero byte of w, 0 elsewhere
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
    return (((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
}
static_assert(kStaticVia == 0x40, "the via-mask bit is the nonzero mark shifted by one");

__device__ __forceinline__ uint32_t flag_word(uint32_t board, uint32_t via) { return board | (nonzero_bytes(via) >> 1); }

__global__ void __launch_bounds__(256) host_gather_kernel(const HostSpan *spans, const uint64_t *chunk_start,
                                                          uint32_t n_spans, uint64_t n_chunks) {
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        // the span holding chunk c: the last s with chunk_start[s] <= c
        uint32_t lo = 0, hi = n_spans - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (chunk_start[mid] <= c) lo = mid; else hi = mid - 1;
        }
        const HostSpan sp = spans[lo];
        const uint64_t off = (c - chunk_start[lo]) * kGatherChunk;
        const uint64_t len = min(kGatherChunk, sp.bytes - off);
        const unsigned char *src = static_cast<const unsigned char *>(sp.src) + off;
        const unsigned char *src2 = static_cast<const unsigned char *>(sp.src2) + off;
        unsigned char *dst = static_cast<unsigned char *>(sp.dst) + off;
        const bool have_src = sp.src != nullptr, have_src2 = sp.src2 != nullptr;
        const uintptr_t align = (uintptr_t)dst | (have_src ? (uintptr_t)src : 0) | (have_src2 ? (uintptr_t)src2 : 0);
        uint64_t done = 0;
        if ((align & 15) == 0) {
            const uint64_t n16 = len / 16;
            constexpr int U = 4;
            for (uint64_t i0 = 0; i0 < n16; i0 += (uint64_t)U * blockDim.x) {
                uint4 a[U], b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * blockDim.x + threadIdx.x;
                    a[u] = make_uint4(0, 0, 0, 0);
                    b[u] = make_uint4(0, 0, 0, 0);
                    if (i < n16) {
                        if (have_src) a[u] = reinterpret_cast<const uint4 *>(src)[i];
                        if (sp.kind == 1 && have_src2) b[u] = reinterpret_cast<const uint4 *>(src2)[i];
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * blockDim.x + threadIdx.x;
                    if (i >= n16) continue;
                    if (sp.kind == 1)
                        a[u] = make_uint4(flag_word(a[u].x, b[u].x), flag_word(a[u].y, b[u].y), flag_word(a[u].z, b[u].z),
                                          flag_word(a[u].w, b[u].w));
                    reinterpret_cast<uint4 *>(dst)[i] = a[u];
                }
            }
            done = n16 * 16;
        } else if ((align & 3) == 0 && sp.kind == 0) {
            const uint64_t n4 = len / 4;
            constexpr int U = 8;
            for (uint64_t i0 = 0; i0 < n4; i0 += (uint64_t)U * blockDim.x) {
                uint32_t a[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * blockDim.x + threadIdx.x;
                    a[u] = (i < n4 && have_src) ? reinterpret_cast<const uint32_t *>(src)[i] : 0u;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * blockDim.x + threadIdx.x;
                    if (i < n4) reinterpret_cast<uint32_t *>(dst)[i] = a[u];
                }
            }
            done = n4 * 4;
        }
        for (uint64_t i = done + threadIdx.x; i < len; i += blockDim.x) {
            uint8_t v = have_src ? src[i] : 0;
            if (sp.kind == 1 && have_src2 && src2[i]) v |= kStaticVia;
            dst[i] = v;
        }
    }
}

// ---- host-side launch helpers ---------------------------------------------

cudaError_t host_gather_launch(const HostSpan *spans, const uint64_t *chunk_start, uint32_t n_spans, uint64_t n_chunks,
                               uint32_t sms, cudaStream_t st) {
    if (!n_spans || !n_chunks) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>(n_chunks, (uint64_t)sms * 8);
    host_gather_kernel<<<(uint32_t)blocks, 256, 0, st>>>(spans, chunk_start, n_spans, n_chunks);
    return cudaGetLastError();
}

uint64_t host_gather_chunks(uint64_t bytes) { return (bytes + kGatherChunk - 1) / kGatherChunk; }

cudaError_t combine_flags_launch(uint8_t *flags, const uint8_t *via_forbidden, uint64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 4096);
    combine_flags_kernel<<<(uint32_t)blocks, 256, 0, st>>>(flags, via_forbidden, n);
    return cudaGetLastError();
}

size_t relax_smem_bytes(uint32_t layers, uint32_t tile_h, bool directed) {
    (void)directed;  // directed prices are folded into the step planes
    return tile_layout(layers, tile_h).total;
}

namespace {
template <int TH>
const void *relax_fn_th(bool wide, bool async) {
    if (async)
        return wide ? (const void *)relax_async_kernel<TH, 256, false> : (const void *)relax_async_kernel<TH, 128, false>;
    return wide ? (const void *)relax_rounds_kernel<TH, 256, false> : (const void *)relax_rounds_kernel<TH, 128, false>;
}

const void *relax_fn(uint32_t tile_h, uint32_t threads, bool async, bool over) {
    if (over) {  // the override variants exist for the 8 x 256 configuration only
        if (tile_h != kOverTileH || threads != kOverThreads) return nullptr;
        if (async) return (const void *)relax_async_kernel<kOverTileH, kOverThreads, true>;
        return (const void *)relax_rounds_kernel<kOverTileH, kOverThreads, true>;
    }
    const bool wide = threads >= 256;
    switch (tile_h) {
        case 8: return relax_fn_th<8>(wide, async);
        case 16: return relax_fn_th<16>(wide, async);
        case 32: return relax_fn_th<32>(wide, async);
        default: return relax_fn_th<64>(wide, async);
    }
}

const void *seed_fn(uint32_t tile_h) {
    switch (tile_h) {
        case 8: return (const void *)async_seed_kernel<8>;
        case 16: return (const void *)async_seed_kernel<16>;
        case 32: return (const void *)async_seed_kernel<32>;
        default: return (const void *)async_seed_kernel<64>;
    }
}
}  // namespace

cudaError_t relax_configure(uint32_t tile_h, uint32_t threads, size_t smem, bool async, bool over) {
    const void *fn = relax_fn(tile_h, threads, async, over);
    if (!fn) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

cudaError_t relax_occupancy(uint32_t tile_h, uint32_t threads, size_t smem, int *blocks_per_sm, bool async,
                            bool over) {
    const void *fn = relax_fn(tile_h, threads, async, over);
    if (!fn) return cudaErrorInvalidValue;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, (int)threads, smem);
}

cudaError_t seed_launch(const RelaxArgs &a, cudaStream_t st) {
    if (!a.n_fields) return cudaSuccess;
    RelaxArgs copy = a;
    void *args[] = {&copy};
    return cudaLaunchKernel(seed_fn(a.tile_h), dim3((a.n_fields + 255) / 256), dim3(256), args, 0, st);
}

cudaError_t relax_launch(const RelaxArgs &a, uint32_t grid, uint32_t threads, size_t smem, cudaStream_t st,
                         bool async, bool over) {
    const void *fn = relax_fn(a.tile_h, threads, async, over);
    if (!fn) return cudaErrorInvalidValue;
    RelaxArgs copy = a;
    void *args[] = {&copy};
    if (async) {
        // seeds, then the queue-driven kernel (a plain launch: no grid barrier,
        // and a CTA only takes a ticket while it is resident)
        cudaError_t e = seed_launch(a, st);
        if (e != cudaSuccess) return e;
        return cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, smem, st);
    }
    // Cooperative (all CTAs co-resident, checked by the CUDA runtime against occupancy);
    // the attribute form is also what stream capture records as a graph node.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

// Tile-staged walk, for batches of the layer kernel whose nets carry no price
// overrides.  One CTA per field.  The CTA stages the labels of a window of 32 x
// walk_rows(L) cells over all layers, with a one-cell ring, relative to the current
// cell (D, H): word = (D - dist) << kLayerHopBits | (H - hops), so q is a predecessor of c
// by a step of price word p exactly when word(q) == word(c) + p.  All threads then look
// for the canonical (lowest CellIdx) predecessor of every cell of the window, reading a
// price only where a neighbour's label is lower, and keep it as the offset to that
// neighbour in shared memory; the walk itself is one thread following offsets, a
// shared-memory load a step, until it leaves the window.  A window with a cell that may
// be on the path and is further back than a word holds (large prices) is staged once
// more, and the rest of the path after it, in words of 64 bits.  Cells priced for the
// net itself (own pads, via pads) are looked up with exact prices; a step from more of
// them than the list holds is taken from HBM.
//
// Bound by a window's two round trips to HBM (labels, prices), some 3 us, and the
// number of windows; a step inside one costs about 50 cycles.  Testing the six
// neighbours step by step in one warp took about 0.5 us a step, and 6 us where the
// prices are the net's own.  Longest of 256 paths on 512x512x4: 267 -> 162 us;
// 640 instances with pads: 820 -> 147 us.  512 threads, so that the rows of a
// window and the prices of its cells are one round of loads each (256: 211 us).
//
// Origin of the walk tile along one axis of extent e for a walk at c heading in
// direction d (-1, 0, +1): a few cells behind c, so most of the tile lies ahead.
// A walk heading diagonally then leaves a tile through one side instead of two.
__device__ __forceinline__ int walk_origin(int c, int d, int e) {
    const int back = e / 8;
    return d > 0 ? c - back : d < 0 ? c - (e - 1 - back) : c - e / 2;
}

__device__ __forceinline__ int walk_dir(int from, int to) { return to > from ? 1 : to < from ? -1 : 0; }

// The exact step price, out of line: the tiled walk needs it only on the
// endpoints' stacks and for nets with own pads, so its loads and branches stay
// out of the common step's code.
// It reads the board and field records from global memory (L1-resident after
// the first call) so the caller's copies stay in registers.
__device__ __noinline__ uint32_t walk_step_exact(const DevBoard *b, const DevField *f, const uint32_t *pads,
                                                 uint32_t p, uint32_t cur, uint32_t x, uint32_t y, uint32_t l,
                                                 int kind) {
    return walk_step(*b, *f, pads, p, cur, x, y, l, kind, false);
}

constexpr int kWalkThreads = 512;
constexpr uint32_t kWalkSteps = 512;     // steps recorded per window
constexpr uint32_t kWalkUnroll = 8;      // steps taken between two looks at whether the walk goes on
constexpr uint32_t kWalkSpec = 256;      // cells of a window priced for the net itself

// Words of a window's labels.  Of a cell that is not on the path: kNone, from which, and to
// which, no step leads.
struct WalkWord {  // 32 bits; only for windows all of whose cells are in range
    using type = uint32_t;
    static constexpr uint32_t kNone = kMax, kHops = (1u << kLayerHopBits) - 1u;
    static __device__ __forceinline__ bool in(uint32_t dist, uint32_t hops) {
        return dist < (1u << (29 - kLayerHopBits)) && hops <= kHops;
    }
    static __device__ __forceinline__ type make(uint32_t dist, uint32_t hops) { return (dist << kLayerHopBits) | hops; }
    static __device__ __forceinline__ type none() { return kNone; }
    static __device__ __forceinline__ uint32_t dist(type w) { return w >> kLayerHopBits; }
    static __device__ __forceinline__ uint32_t hops(type w) { return w & kHops; }
    static __device__ __forceinline__ bool is(type w) { return w != kNone; }
    // may q precede c, by a step of some price
    static __device__ __forceinline__ bool asks(type c, type q) { return q != kNone && q > c; }
    // does it, by a step of price word p (one that does costs less than a plain price)
    static __device__ __forceinline__ bool by(type c, type q, uint32_t p) { return q == c + p && p < kPackedInf; }
};
struct WalkWide {  // 64 bits
    using type = uint2;  // hops, dist
    static __device__ __forceinline__ bool in(uint32_t, uint32_t) { return true; }
    static __device__ __forceinline__ type make(uint32_t dist, uint32_t hops) { return make_uint2(hops, dist); }
    static __device__ __forceinline__ type none() { return make_uint2(kMax, 0u); }
    static __device__ __forceinline__ uint32_t dist(type w) { return w.y; }
    static __device__ __forceinline__ uint32_t hops(type w) { return w.x; }
    static __device__ __forceinline__ bool is(type w) { return w.x != kMax; }
    static __device__ __forceinline__ bool asks(type c, type q) { return q.x == c.x + 1u && q.y >= c.y; }
    static __device__ __forceinline__ bool by(type c, type q, uint32_t p) {
        const uint32_t want = q.y - c.y;
        return p == (want < (1u << (29 - kLayerHopBits)) ? (want << kLayerHopBits) | 1u : want | kPricePlain);
    }
};

__global__ void __launch_bounds__(kWalkThreads, 2) path_walk_tiled_kernel(PathArgs a) {
    extern __shared__ __align__(16) unsigned char wsm[];
    __shared__ uint32_t s_path[kWalkSteps + kWalkUnroll];          // cells walked in this window (indices into it)
    __shared__ uint32_t s_spec[kWalkSpec], s_code[kWalkSpec];
    __shared__ uint32_t s_nspec, s_n, s_ok, s_next[3];  // s_ok, s_next: after a step from HBM, the cell and its label
    const DevField f = a.fields[blockIdx.x];
    const uint32_t len = a.lens[f.out];
    if (len == 0) return;  // the same for the whole CTA
    const DevBoard b = a.boards[f.board];
    const uint32_t L = b.layers, WH = walk_rows(L), W = kTW, PW = W + 2, PL = (WH + 2) * PW;  // ring included
    const uint32_t plane = b.w * b.h, tid = threadIdx.x, lane = tid & 31;
    const int wx0 = (int)f.x0, wy0 = (int)f.y0, wx1 = (int)(f.x0 + f.ww), wy1 = (int)(f.y0 + f.wh);
    const u64 *lab = a.lab + f.lab_off;
    const uint32_t wp = planes_pitch(b.w);
    const uint64_t NP = (uint64_t)wp * b.h * L;
    bool wide = b.goal->wide != 0;  // windows in 64-bit words
    uint32_t *out = a.cells + a.offsets[f.out];
    const uint32_t src_xy = f.src % plane;
    const int sx = (int)(src_xy % b.w), sy = (int)(src_xy / b.w);  // the walk heads for the source
    // the current cell and its label (the same in every thread)
    uint32_t pos = len - 1;
    int cx, cy, cl;
    {
        const uint32_t r = f.dst % plane;
        cx = (int)(r % b.w);
        cy = (int)(r / b.w);
        cl = (int)(f.dst / plane);
    }
    u64 need = __ldcg(lab + ((uint64_t)(uint32_t)cl * f.wh + (uint32_t)(cy - wy0)) * f.ww + (uint32_t)(cx - wx0));
    if (tid == 0) {
        out[pos] = f.dst;
        s_nspec = s_n = 0;
    }
    int dx = walk_dir(cx, sx), dy = walk_dir(cy, sy);
    while (pos) {
        const int tx0 = walk_origin(cx, dx, (int)W), ty0 = walk_origin(cy, dy, (int)WH);
        // Stages the window, looks up its predecessors and walks as far as it goes; false:
        // a cell is out of the words' range.
        auto window = [&](auto words) -> bool {
            using Q = decltype(words);
            const uint32_t D = (uint32_t)(need >> 32), H = (uint32_t)need;
            auto *word = reinterpret_cast<typename Q::type *>(wsm);
            int16_t *delta = reinterpret_cast<int16_t *>(word + L * PL);
            bool far = false;
            __syncthreads();  // every thread is past the previous window
            // ---- labels of the window and its ring: a warp per row, several rows in flight
            // word of the cell in column xx, row yy (ring included) of layer l, from its label
            auto put = [&](uint32_t i, u64 v, int gx, int gy, int l) {
                // cells of the path have no larger dist than (D, H), and fewer hops by
                // at least their distance in cells
                const uint32_t d = (uint32_t)(v >> 32), h = (uint32_t)v;
                const uint32_t away = (uint32_t)(abs(gx - cx) + abs(gy - cy) + abs(l - cl));
                const bool can = d <= D && h <= H && H - h >= away;
                const bool in = Q::in(D - d, H - h);
                word[i] = can && in ? Q::make(D - d, H - h) : Q::none();
                far |= can && !in;
                delta[i] = 0;
            };
            auto label = [&](int gx, int gy, uint32_t l) -> u64 {
                if (gx < wx0 || gx >= wx1 || gy < wy0 || gy >= wy1) return kInf;
                return __ldcg(lab + ((uint64_t)l * f.wh + (uint32_t)(gy - wy0)) * f.ww + (uint32_t)(gx - wx0));
            };
            const uint32_t rows = L * (WH + 2), wid = tid >> 5, nw = blockDim.x >> 5;
            // the last two columns, their loads issued with the rows'
            const uint32_t eq = tid >> 1, ex = W + (tid & 1u), el = eq / (WH + 2);
            const int egx = tx0 + (int)ex - 1, egy = ty0 + (int)(eq - el * (WH + 2)) - 1;
            const u64 ev = eq < rows ? label(egx, egy, el) : kInf;
            constexpr uint32_t kRows = 8;
            for (uint32_t r0 = wid; r0 < rows; r0 += kRows * nw) {
                u64 v[kRows];
#pragma unroll
                for (uint32_t k = 0; k < kRows; ++k) {
                    const uint32_t q = r0 + k * nw, l = q / (WH + 2), yy = q - l * (WH + 2);
                    v[k] = q < rows ? label(tx0 + (int)lane - 1, ty0 + (int)yy - 1, l) : kInf;
                }
#pragma unroll
                for (uint32_t k = 0; k < kRows; ++k) {
                    const uint32_t q = r0 + k * nw, l = q / (WH + 2), yy = q - l * (WH + 2);
                    if (q < rows) put(q * PW + lane, v[k], tx0 + (int)lane - 1, ty0 + (int)yy - 1, (int)l);
                }
            }
            if (eq < rows) put(eq * PW + ex, ev, egx, egy, (int)el);
            for (uint32_t e = tid + blockDim.x; e < 2 * rows; e += blockDim.x) {  // (more than 14 layers)
                const uint32_t q = e >> 1, xx = W + (e & 1u), l = q / (WH + 2), yy = q - l * (WH + 2);
                const int gx = tx0 + (int)xx - 1, gy = ty0 + (int)yy - 1;
                put(q * PW + xx, label(gx, gy, l), gx, gy, (int)l);
            }
            // cells priced for the net itself: own pads; a via pad's cell and the cells below and above it
            for (uint32_t k = tid; k < f.n_pads + 3 * f.n_vpads; k += blockDim.x) {
                const uint32_t m = k - f.n_pads;
                const uint32_t c = __ldg(a.pads + (k < f.n_pads ? f.pad_off + k : f.vpad_off + m / 3));
                const uint32_t l = c / plane + (k < f.n_pads ? 0u : m % 3 - 1u), r = c % plane, gy = r / b.w, gx = r - gy * b.w;
                const uint32_t xx = gx - (uint32_t)tx0, yy = gy - (uint32_t)ty0;
                if (l >= L || xx >= W || yy >= WH) continue;
                const uint32_t i = atomicAdd(&s_nspec, 1u);
                if (i < kWalkSpec) {
                    s_spec[i] = l * PL + (yy + 1) * PW + xx + 1;
                    s_code[i] = 7;
                }
            }
            if (__syncthreads_or(far)) {
                if (tid == 0) s_nspec = 0;
                return false;
            }
            // ---- the predecessor of every cell: neighbours in ascending CellIdx ----
            const int off[6] = {-(int)PL, -(int)PW, -1, 1, (int)PW, (int)PL};
            constexpr uint32_t in_plane[6] = {kInBelow, kInNegY, kInNegX, kInPosX, kInPosY, kInAbove};
            constexpr uint32_t kCells = 4;  // cells of one thread whose prices are in flight together
            for (uint32_t r0 = wid; r0 < L * WH; r0 += kCells * nw) {
                uint32_t p[kCells][6], most = 0;
#pragma unroll
                for (uint32_t k = 0; k < kCells; ++k) {
                    const uint32_t q = r0 + k * nw, l = q / WH, yy = q % WH;
                    const uint32_t at = l * PL + (yy + 1) * PW + lane + 1;
                    const auto wc = q < L * WH ? word[at] : Q::none();
                    const uint32_t *pr = b.planes + ((uint64_t)l * b.h + (uint32_t)(ty0 + (int)yy)) * wp + (uint32_t)(tx0 + (int)lane);
#pragma unroll
                    for (int n = 0; n < 6; ++n) {
                        p[k][n] = kPackedInf;
                        if (!Q::is(wc) || (n == 0 && l == 0) || (n == 5 && l + 1 == L)) continue;
                        if (Q::asks(wc, word[(int)at + off[n]])) p[k][n] = __ldg(pr + in_plane[n] * NP);
                    }
                }
#pragma unroll
                for (uint32_t k = 0; k < kCells; ++k) {
                    const uint32_t q = r0 + k * nw, l = q / WH, yy = q % WH;
                    const uint32_t at = l * PL + (yy + 1) * PW + lane + 1;
                    if (q >= L * WH) continue;
                    const auto wc = word[at];
                    int dl = 0;
#pragma unroll
                    for (int n = 5; n >= 0; --n) {
                        if (p[k][n] == kPackedInf) continue;  // (a price was read only where one is asked for)
                        if (Q::by(wc, word[(int)at + off[n]], p[k][n])) dl = off[n];
                        most = max(most, p[k][n]);
                    }
                    if (dl) delta[at] = (int16_t)dl;
                }
                if constexpr (sizeof(typename Q::type) == 8) {
                    if (most != kPriceLook) continue;
                    // prices that no word holds: formed from the board's words
#pragma unroll 1
                    for (uint32_t k = 0; k < kCells; ++k) {
                        const uint32_t q = r0 + k * nw, l = q / WH, yy = q % WH;
                        const uint32_t at = l * PL + (yy + 1) * PW + lane + 1;
                        if (q >= L * WH) continue;
                        const auto wc = word[at];
                        int dl = 0;
#pragma unroll 1
                        for (int n = 5; n >= 0; --n) {
                            const int o = n == 0 ? -(int)PL : n == 1 ? -(int)PW : n == 2 ? -1 : n == 3 ? 1 : n == 4 ? (int)PW : (int)PL;
                            if (!Q::is(wc) || (n == 0 && l == 0) || (n == 5 && l + 1 == L) || !Q::asks(wc, word[(int)at + o])) continue;
                            int px = tx0 + (int)lane, py = ty0 + (int)yy, pz = (int)l;
                            const uint32_t gx = (uint32_t)px, gy = (uint32_t)py;
                            walk_offset(n, px, py, pz);
                            if (walk_step_exact(a.boards + f.board, a.fields + blockIdx.x, a.pads,
                                                ((uint32_t)pz * b.h + (uint32_t)py) * b.w + (uint32_t)px,
                                                (l * b.h + gy) * b.w + gx, gx, gy, l, n) == Q::dist(word[(int)at + o]) - Q::dist(wc))
                                dl = o;
                        }
                        delta[at] = (int16_t)dl;
                    }
                }
            }
            if (s_nspec) {  // the same for the whole CTA
                __syncthreads();
                const uint32_t ns = min(s_nspec, kWalkSpec);
                for (uint32_t i = tid; i < 6 * ns; i += blockDim.x) {
                    const uint32_t e = i / 6, at = s_spec[e];
                    const int kind = (int)(i % 6);
                    const uint32_t l = at / PL, q = at - l * PL, yy = q / PW, xx = q - yy * PW;
                    const auto wc = word[at];
                    if (!Q::is(wc) || (kind == 0 && l == 0) || (kind == 5 && l + 1 == L)) continue;
                    int px = tx0 + (int)xx - 1, py = ty0 + (int)yy - 1, pz = (int)l;
                    const uint32_t gx = (uint32_t)px, gy = (uint32_t)py;
                    const int off = kind == 0 ? -(int)PL : kind == 1 ? -(int)PW : kind == 2 ? -1 : kind == 3 ? 1
                                  : kind == 4 ? (int)PW : (int)PL;
                    const auto wq = word[(int)at + off];
                    if (!Q::asks(wc, wq) || Q::hops(wq) != Q::hops(wc) + 1u) continue;
                    walk_offset(kind, px, py, pz);
                    const uint32_t st = walk_step_exact(a.boards + f.board, a.fields + blockIdx.x, a.pads,
                                                        ((uint32_t)pz * b.h + (uint32_t)py) * b.w + (uint32_t)px,
                                                        (l * b.h + gy) * b.w + gx, gx, gy, l, kind);
                    if (st == Q::dist(wq) - Q::dist(wc)) atomicMin(&s_code[e], (uint32_t)kind + 1u);
                }
                __syncthreads();
                for (uint32_t e = tid; e < ns; e += blockDim.x) {
                    const uint32_t c = s_code[e];
                    delta[s_spec[e]] = (int16_t)(c == 1 ? -(int)PL : c == 2 ? -(int)PW : c == 3 ? -1 : c == 4 ? 1
                                               : c == 5 ? (int)PW : c == 6 ? (int)PL : 0);
                }
                // more such cells than the list holds: none of the window's steps is taken from it
                if (s_nspec > kWalkSpec) {
                    __syncthreads();
                    if (tid == 0) delta[(uint32_t)cl * PL + (uint32_t)(cy - ty0 + 1) * PW + (uint32_t)(cx - tx0 + 1)] = 0;
                }
            }
            __syncthreads();
            // ---- the walk ---------------------------------------------------------
            if (tid == 0) {
                uint32_t at = (uint32_t)cl * PL + (uint32_t)(cy - ty0 + 1) * PW + (uint32_t)(cx - tx0 + 1), n = 0;
                const uint32_t most = min(pos, kWalkSteps);
                // an offset is 0 on the ring and where no predecessor was found: the walk
                // then stays where it is, so several steps go by before it is looked at
                for (;;) {
                    uint32_t moved = 0;
#pragma unroll
                    for (uint32_t k = 0; k < kWalkUnroll; ++k) {
                        const int d = delta[at];
                        at = (uint32_t)((int)at + d);
                        s_path[n + k] = at;
                        moved += d != 0;
                    }
                    n += moved;
                    if (moved < kWalkUnroll || n >= most) break;
                }
                s_n = min(n, most);
                s_nspec = 0;  // for the next window
            }
            __syncthreads();
            const uint32_t n = s_n;
            if (n) {
                for (uint32_t k = tid; k < n; k += blockDim.x) {
                    const uint32_t at = s_path[k], l = at / PL, q = at - l * PL, yy = q / PW, xx = q - yy * PW;
                    out[pos - 1 - k] = (l * b.h + (uint32_t)(ty0 + (int)yy - 1)) * b.w + (uint32_t)(tx0 + (int)xx - 1);
                }
                const uint32_t at = s_path[n - 1], l = at / PL, q = at - l * PL, yy = q / PW, xx = q - yy * PW;
                const auto w = word[at];
                cx = tx0 + (int)xx - 1;
                cy = ty0 + (int)yy - 1;
                cl = (int)l;
                need = ((u64)(D - Q::dist(w)) << 32) | (H - Q::hops(w));
                pos -= n;
            }
            return true;
        };
        if (!wide) wide = !window(WalkWord{});
        if (wide) window(WalkWide{});
        if (s_n == 0) {
            // one step from HBM with exact prices
            if (tid < 32) {
                bool ok = false;
                uint32_t p = 0;
                u64 lp = kInf;
                int px = cx, py = cy, pz = cl;
                const uint32_t cur = ((uint32_t)cl * b.h + (uint32_t)cy) * b.w + (uint32_t)cx;
                if (lane < 6) walk_offset((int)lane, px, py, pz);
                if (lane < 6 && walk_inside(f, b, px, py, pz)) {
                    p = ((uint32_t)pz * b.h + (uint32_t)py) * b.w + (uint32_t)px;
                    lp = __ldcg(lab + ((uint64_t)(uint32_t)pz * f.wh + (uint32_t)(py - wy0)) * f.ww + (uint32_t)(px - wx0));
                    const uint32_t st = walk_step_exact(a.boards + f.board, a.fields + blockIdx.x, a.pads, p, cur,
                                                        (uint32_t)cx, (uint32_t)cy, (uint32_t)cl, (int)lane);
                    ok = lp != kInf && extend(lp, st) == need;
                }
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
                const uint32_t win = m ? __ffs(m) - 1 : 0;
                p = __shfl_sync(0xFFFFFFFFu, p, win);
                lp = __shfl_sync(0xFFFFFFFFu, lp, win);
                if (lane == 0) {
                    s_ok = m;
                    s_next[0] = p;
                    s_next[1] = (uint32_t)(lp >> 32);
                    s_next[2] = (uint32_t)lp;
                    if (m) out[pos - 1] = p;
                    else atomicOr(a.status, kStatusPathBroken);
                }
            }
            __syncthreads();
            if (s_ok == 0) return;
            const uint32_t p = s_next[0], r = p % plane;
            cx = (int)(r % b.w);
            cy = (int)(r / b.w);
            cl = (int)(p / plane);
            need = ((u64)s_next[1] << 32) | s_next[2];
            --pos;
        }
        // the side the path left the window by, else towards the source
        dx = cx < tx0 ? -1 : cx >= tx0 + (int)W ? 1 : walk_dir(cx, sx);
        dy = cy < ty0 ? -1 : cy >= ty0 + (int)WH ? 1 : walk_dir(cy, sy);
    }
    if (tid == 0 && ((uint32_t)cl * b.h + (uint32_t)cy) * b.w + (uint32_t)cx != f.src) atomicOr(a.status, kStatusPathBroken);
}

namespace {
// One warp per field: every override cell inside the window flags its tile.
__global__ void mark_over_tiles_kernel(const DevField *fields, uint32_t n_fields, const DevBoard *boards,
                                       uint32_t tile_h, uint8_t *tover) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t fi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; fi < n_fields; fi += warps) {
        const DevField f = fields[fi];
        if (!f.n_over) continue;
        const DevBoard b = boards[f.board];
        const uint32_t plane = b.w * b.h, ntx = field_ntx(f);
        for (uint32_t k = lane; k < f.n_over; k += 32) {
            const uint32_t c = b.over_cells[f.over_off + k], r = c % plane, x = r % b.w, y = r / b.w;
            if (x < f.x0 || x >= f.x0 + f.ww || y < f.y0 || y >= f.y0 + f.wh) continue;
            tover[f.tile_off + ((y - f.y0) / tile_h) * ntx + (x - f.x0 + f.xa) / kTW] = 1;
        }
    }
}
}  // namespace

cudaError_t mark_over_tiles_launch(const DevField *fields, uint32_t n_fields, const DevBoard *boards, uint32_t tile_h,
                                   uint8_t *tover, cudaStream_t st) {
    if (!n_fields) return cudaSuccess;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>(((uint64_t)n_fields * 32 + 255) / 256, 148ull * 16);
    mark_over_tiles_kernel<<<blocks, 256, 0, st>>>(fields, n_fields, boards, tile_h, tover);
    return cudaGetLastError();
}

cudaError_t path_launch(const PathArgs &a, cudaStream_t st) {
    path_offsets_kernel<<<1, 1024, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (a.n_fields && a.walk_smem) {
        e = cudaFuncSetAttribute(path_walk_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)a.walk_smem);
        if (e != cudaSuccess) return e;
        path_walk_tiled_kernel<<<a.n_fields, kWalkThreads, a.walk_smem, st>>>(a);
    } else if (a.n_fields) {
        const uint32_t warps_per_block = 8;
        path_walk_kernel<<<(a.n_fields + warps_per_block - 1) / warps_per_block, 32 * warps_per_block, 0, st>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t fields_launch(const PathArgs &a, uint32_t *out, uint64_t total, cudaStream_t st) {
    if (total == 0 || a.n_fields == 0) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>((total + 255) / 256, 8192);
    emit_fields_kernel<<<(uint32_t)blocks, 256, 0, st>>>(a, out, total);
    return cudaGetLastError();
}

cudaError_t plain_round_launch(const PlainArgs &a, uint64_t wcells, cudaStream_t st) {
    const uint32_t threads = 256;
    plain_round_kernel<<<(uint32_t)((wcells + threads - 1) / threads), threads, 0, st>>>(a);
    return cudaGetLastError();
}

// Self-test of the bounded wait: one CTA waits at the grid barrier for a CTA
// that does not exist, so the wait must give up after `spins` polls, record
// kStatusBarrier and return with the context intact.
__global__ void wait_selftest_kernel(Ctl *c, uint32_t spins) { grid_barrier(c, gridDim.x + 1, spins); }

cudaError_t wait_selftest_launch(Ctl *c, uint32_t spins, cudaStream_t st) {
    wait_selftest_kernel<<<1, 32, 0, st>>>(c, spins);
    return cudaGetLastError();
}

}  // namespace mrc
