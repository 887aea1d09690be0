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
#include "tma.cuh"

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
    __shared__ unsigned long long s_cnt[2];  // this CTA's activations and sweeps not yet added to the launch's
    if (threadIdx.x == 0) s_cnt[0] = s_cnt[1] = 0;
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) s_item = async_pop(a);
        __syncthreads();
        const u64 item = s_item;
        if (item == kInf) break;
        process_item<TH, true, OV, false>(a, (uint32_t)(item >> 32), (uint32_t)item, 0, smem_raw, s_cnt);
    }
    if (threadIdx.x == 0) {
        if (s_cnt[0]) atomicAdd(&a.ctl->activations, s_cnt[0]);
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
                const BoardGoal *bg = b.goal;
                const uint32_t *hx = b.goal_sums, *hy = hx + b.w, *hv = hy + b.h;
                const uint32_t dl = f.dst / plane, dr = f.dst % plane, dx = dr % b.w, dy = dr / b.w;
                const uint32_t e = f.n_pads ? min(bg->min_cost, 1u) : bg->min_cost;
                auto rest = [&](const uint32_t *p, uint32_t u, uint32_t v) {
                    return capmul(p[u] > p[v] ? p[u] - p[v] : p[v] - p[u], e);
                };
                const uint32_t f0 = min(dsum(dsum(rest(hx, sx, dx), rest(hy, sy, dy)), rest(hv, sl, dl)), kCap);
                // first threshold: room for two vias, a detour of two cells, and the
                // board's spread of prices; with a zero bound nothing waits
                const u64 room = (u64)((double)bg->spread * f0) + 2ull * capmul(bg->min_via, e) +
                                 4ull * capmul(bg->min_step, e);
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
// `fields_by_offset` lists the fields in ascending lab_off order.
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
        out[i] = (uint32_t)(field_label(a, f, lx, ly, l) >> 32);
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

// Tile-staged walk, for batches whose boards carry price planes and a TMA map
// (the CTA queue form) and whose nets carry no price overrides.  One CTA per
// field stages a walk tile of 32 x WH cells over all layers — the labels with a
// one-cell ring by plain loads, the six price planes by WH / tile_h TMA loads of
// the relax kernel's box — and warp 0 walks inside it from shared memory,
// re-staging when the path leaves the tile.  A step then costs shared-memory
// reads instead of a round trip to L2 or HBM.  The step prices are the planes'
// except on the stacks of the net's endpoints, and for every step of a net with
// own or via pads, where walk_step prices exactly; the choice among the
// candidates is path_walk_kernel's.
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

__global__ void __launch_bounds__(256) path_walk_tiled_kernel(PathArgs a) {
    extern __shared__ __align__(128) unsigned char wsm[];
    __shared__ __align__(8) uint64_t s_mbar;
    __shared__ int s_tile[2];   // walk tile origin (board x, y)
    __shared__ uint32_t s_done;
    const DevField f = a.fields[blockIdx.x];
    const uint32_t len = a.lens[f.out];
    if (len == 0) return;  // the same for the whole CTA
    const DevBoard b = a.boards[f.board];
    const uint32_t L = b.layers, TH = a.tile_h, WH = walk_tile_rows(TH), nload = WH / TH;
    const uint32_t plane = b.w * b.h;
    uint32_t *pl = reinterpret_cast<uint32_t *>(wsm);
    u64 *lab = reinterpret_cast<u64 *>(wsm + walk_smem_planes(L, TH));
    const uint32_t box_words = 6 * L * TH * kPlaneTmaBoxW;
    const bool exact_all = (f.n_pads | f.n_vpads) != 0 || b.goal->wide;
    const uint32_t src_xy = f.src % plane, dst_xy = f.dst % plane;
    const int sx = (int)(src_xy % b.w), sy = (int)(src_xy / b.w);  // the walk heads for the source
    const int dstx = (int)(dst_xy % b.w), dsty = (int)(dst_xy / b.w);
    const int wx0 = (int)f.x0, wy0 = (int)f.y0, wx1 = (int)(f.x0 + f.ww), wy1 = (int)(f.y0 + f.wh);
    const uint32_t lane = threadIdx.x & 31;
    uint32_t *out = a.cells + a.offsets[f.out];
    // walk state (warp 0)
    uint32_t cur = f.dst, pos = len - 1;
    int cx = (int)((f.dst % plane) % b.w), cy = (int)((f.dst % plane) / b.w), cl = (int)(f.dst / plane);
    u64 need = a.lab[f.lab_off + ((uint64_t)(uint32_t)cl * f.wh + (uint32_t)(cy - wy0)) * f.ww + (uint32_t)(cx - wx0)];
    uint32_t phase = 0;
    // Per-lane constants of a step: the neighbour offset of kind `lane` (lanes 0-5),
    // the in-price plane of the move from it into the current cell, and the
    // relax tile height as a shift (tile heights are powers of two).
    int ox = 0, oy = 0, oz = 0;
    if (lane < 6) walk_offset((int)lane, ox, oy, oz);
    const uint32_t pin = lane == 0 ? kInBelow : lane == 1 ? kInNegY : lane == 2 ? kInNegX
                       : lane == 3 ? kInPosX : lane == 4 ? kInPosY : kInAbove;
    const uint32_t th_shift = (uint32_t)__ffs((int)TH) - 1u;
    if (threadIdx.x == 0) {
        mbar_init(&s_mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_tile[0] = walk_origin(cx, walk_dir(cx, sx), (int)kTW);
        s_tile[1] = walk_origin(cy, walk_dir(cy, sy), (int)WH);
        s_done = 0;
    }
    for (;;) {
        __syncthreads();
        const int tx0 = s_tile[0], ty0 = s_tile[1];
        const uint32_t xo = (uint32_t)tx0 & 3u;
        if (threadIdx.x == 0) {
            fence_proxy_async_smem();
            mbar_expect_tx(&s_mbar, nload * box_words * 4u);
            for (uint32_t j = 0; j < nload; ++j)
                tma_load_4d(pl + j * box_words, b.tmap, tx0 & ~3, ty0 + (int)(j * TH), 0, 0, &s_mbar);
        }
        // labels of the tile and its ring (+inf outside the window), kStageBatch
        // loads in flight per thread before any is stored
        const uint32_t nl = L * (WH + 2) * 34;
        constexpr uint32_t kStageBatch = 8;
        for (uint32_t i0 = threadIdx.x; i0 < nl; i0 += kStageBatch * blockDim.x) {
            u64 v[kStageBatch];
#pragma unroll
            for (uint32_t k = 0; k < kStageBatch; ++k) {
                const uint32_t i = i0 + k * blockDim.x;
                const uint32_t sx = i % 34, r = i / 34, sy = r % (WH + 2), l = r / (WH + 2);
                const int gx = tx0 + (int)sx - 1, gy = ty0 + (int)sy - 1;
                v[k] = kInf;
                if (i < nl && gx >= wx0 && gx < wx1 && gy >= wy0 && gy < wy1)
                    v[k] = __ldcg(a.lab + f.lab_off + ((uint64_t)l * f.wh + (uint32_t)(gy - wy0)) * f.ww +
                                  (uint32_t)(gx - wx0));
            }
#pragma unroll
            for (uint32_t k = 0; k < kStageBatch; ++k)
                if (i0 + k * blockDim.x < nl) lab[i0 + k * blockDim.x] = v[k];
        }
        // bounded wait for the planes (a load that never lands breaks the path)
        for (uint32_t spins = 0; !mbar_try_wait(&s_mbar, phase & 1u); ++spins) {
            if (spins > kTmaSpinLimit) {
                if (threadIdx.x == 0) {
                    atomicOr(a.status, kStatusPathBroken);
                    s_done = 1;
                }
                break;
            }
        }
        ++phase;
        __syncthreads();
        if (s_done) return;
        if (threadIdx.x < 32) {
            for (;;) {
                if (lane == 0) out[pos] = cur;
                if (pos == 0) {
                    if (lane == 0) {
                        if (cur != f.src) atomicOr(a.status, kStatusPathBroken);
                        s_done = 1;
                    }
                    break;
                }
                bool ok = false;
                uint32_t p = 0;
                u64 lp = kInf;
                const int px = cx + ox, py = cy + oy, pz = cl + oz;
                if (lane < 6 && walk_inside(f, b, px, py, pz)) {
                    p = ((uint32_t)pz * b.h + (uint32_t)py) * b.w + (uint32_t)px;
                    lp = lab[((uint32_t)pz * (WH + 2) + (uint32_t)(py - ty0 + 1)) * 34 + (uint32_t)(px - tx0 + 1)];
                    uint32_t st;
                    if (exact_all || (cx == sx && cy == sy) || (cx == dstx && cy == dsty)) {
                        st = walk_step_exact(a.boards + f.board, a.fields + blockIdx.x, a.pads, p, cur, (uint32_t)cx,
                                             (uint32_t)cy, (uint32_t)cl, (int)lane);
                    } else {
                        // in-price plane `pin` at cur, from the TMA box of cur's relax-tile rows
                        const uint32_t yy = (uint32_t)(cy - ty0), j = yy >> th_shift;
                        st = pl[j * box_words + ((pin * L + (uint32_t)cl) * TH + (yy & (TH - 1u))) * kPlaneTmaBoxW +
                                (uint32_t)(cx - tx0) + xo];
                        st = st >= kPackedInf ? kMax : st >> a.hop_bits;
                    }
                    ok = lp != kInf && extend(lp, st) == need;
                }
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
                if (m == 0) {
                    if (lane == 0) {
                        atomicOr(a.status, kStatusPathBroken);
                        s_done = 1;
                    }
                    break;
                }
                const uint32_t win = __ffs(m) - 1;
                cur = __shfl_sync(0xFFFFFFFFu, p, win);
                need = __shfl_sync(0xFFFFFFFFu, lp, win);
                cx = __shfl_sync(0xFFFFFFFFu, px, win);
                cy = __shfl_sync(0xFFFFFFFFu, py, win);
                cl = __shfl_sync(0xFFFFFFFFu, pz, win);
                --pos;
                if (cx < tx0 || cx >= tx0 + (int)kTW || cy < ty0 || cy >= ty0 + (int)WH) {
                    if (lane == 0) {  // the path left the tile: stage one ahead of cur
                        const int dx = cx < tx0 ? -1 : cx >= tx0 + (int)kTW ? 1 : walk_dir(cx, sx);
                        const int dy = cy < ty0 ? -1 : cy >= ty0 + (int)WH ? 1 : walk_dir(cy, sy);
                        s_tile[0] = walk_origin(cx, dx, (int)kTW);
                        s_tile[1] = walk_origin(cy, dy, (int)WH);
                    }
                    break;
                }
            }
        }
        __syncthreads();
        if (s_done) return;
    }
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
        path_walk_tiled_kernel<<<a.n_fields, 256, a.walk_smem, st>>>(a);
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
