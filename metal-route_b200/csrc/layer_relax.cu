// layer_relax.cu — the queue-driven relax kernel with a warp per layer and packed labels.
//
// A CTA holds one 32 x TH tile over all L layers of a field, warp l its layer l:
// lane x keeps the TH labels of column x in registers.  TH is 8, or 16 where the
// batch's longest chains of tiles bound it (batch_layout has the rule).  Inside an activation a
// label is one word, (dist - least staged dist) << HB | (hops - least staged
// hops) in 32 bits, and a step price is (price << HB) | 1, so the lexicographic min-plus step
// of (dist, hops) is one add-and-min instruction (__viaddmin_u32) where 64-bit
// labels with saturation take about ten.  kBig is +inf: label + price stays below
// 2^32, and a min with a label at most kBig clamps the sum.  A sweep is:
//   columns  each lane runs its column down and up in registers (the halo rows in
//            two more registers), no data exchanged;
//   rows     through shared memory (one store and two 16-byte loads a lane): four
//            lanes a row, eight cells each, eight rows at a time, joined by a two-step
//            scan; the warp
//            repeats columns and rows until its plane is closed, with no CTA barrier;
//   stacks   a thread per (y, x) runs the layers up and down; only here the warps
//            of a tile meet.
// What changed is found by comparing registers (old and new label of the own
// column), so there are no dirty-line or fell marks.
//
// The packing is exact or not used: a tile whose staged labels spread too far, or
// whose largest final label comes within one price of kBig (the only way a sum
// could have been clamped), or with a final label at the last value of the hops, or with
// a price that does not fit, does not fit 32-bit words.  (Words are sums dist 2^HB +
// hops, so a word is the lexicographic least label as long as that label's hops fit,
// whatever other paths carried into the dist; and the first label of a best path that
// doesn't fit follows one whose hops are the last value.)  It is relaxed from the labels
// in HBM, which this kernel has not touched by then:
//   on boards whose prices make that likely (BOTH) in 64-bit words, 40 bits of dist and 24
//   of hops, which hold every price and sum; labels whose dist saturates are not kept.
//   A field that few tiles of fit goes there straight away (RelaxArgs::misfits).
//   Relax, us, on 32-bit words with exact_item alone, so, and on 64-bit labels throughout
//   before 32-bit words came in: 256 nets of 512 x 512 x 4 at 2500 times their prices
//   7000, 4000, 4530; 64 nets of 640 x 500 x 4 2900, 1780, 2320; 128 nets of 300 x 280 x 4
//   at gaps of 40 000 1690, 1100, 1270;
//   elsewhere, and with hops past 24 bits, by exact_item.
//
// Bound by the chain of activations (a queue hop, the label loads, the sweeps, the
// write-back) on small batches and by instruction issue on large ones.
#include <cuda_runtime.h>

#include <algorithm>

#include "cta_tile.cuh"
#include "device.cuh"
#include "kernels.h"
#include "tiles.cuh"
#include "tma.cuh"

namespace mrc {
namespace {

// The words of a tile: labels and prices, dist << kHops | hops relative to the least staged
// ones.  kBig is +inf; staged labels, final labels and prices lie below kNarrow.  kNone is the
// price of no step.
template <class W>
struct Words;
template <>
struct Words<uint32_t> {
    static constexpr int kHops = (int)kLayerHopBits;
    static constexpr uint32_t kBig = kPackedInf, kNarrow = 1u << 29, kNone = kBig;
    // Pitch of a row of labels: 16-byte aligned, and the rows' segments and the columns
    // of a warp fall on distinct banks.
    static constexpr uint32_t kPitch = kPlaneTmaBoxW;
    static __device__ __forceinline__ uint32_t addmin(uint32_t a, uint32_t b, uint32_t c) { return __viaddmin_u32(a, b, c); }
    static __device__ __forceinline__ uint32_t price(uint32_t staged) { return staged; }  // a packed word
};
template <>
struct Words<u64> {
    static constexpr int kHops = 24;
    static constexpr u64 kBig = 1ull << 62, kNarrow = 1ull << 61, kNone = ((u64)kMax << kHops) | 1u;
    static constexpr uint32_t kPitch = 34;  // (36 costs the third CTA of 16-row and of 8-layer tiles)
    static __device__ __forceinline__ u64 addmin(u64 a, u64 b, u64 c) { return min(a + b, c); }
    static __device__ __forceinline__ u64 price(uint32_t staged) { return ((u64)staged << kHops) | 1u; }  // a plain price
};
constexpr uint32_t kPitch = kPlaneTmaBoxW;  // of a row of prices
constexpr uint32_t kSpecCap = 512;      // cells of a tile priced for the net itself
// A field's tiles go straight to 64-bit words from this count of misfits on; one counts
// as much as kMisfitWeight of those that fit.  (8, 16 or 32: no difference on boards of
// large prices, nor with a dear corner.)
constexpr int kMisfitWeight = 4, kMisfits = 32;
constexpr int kPlaneIters = 2;          // column and row passes of a plane between two meetings

// Shared memory: the prices, then the labels.
__host__ __device__ inline size_t layer_lab_off(uint32_t L, uint32_t TH) { return (size_t)6 * L * TH * kPitch * 4; }

struct LayerShared {
    u64 item;
    uint64_t mbar;  // completion of the price-plane TMA loads
    unsigned long long cnt[2];  // activations and sweeps not yet added to the launch's
    uint32_t n_spec, near_pad, wide, dmin, hmin, hmax, ub, thr, more;
    uint32_t push;              // bits: left, right, top, bottom improved
    uint32_t park[4];           // GD: the smallest f that waits to enter each
    uint32_t hy[kLayerTallH + 2];  // GD: remaining price along y, rows -1 .. TH
    uint32_t spec[kSpecCap];
    int misfits;                // of the field so far (RelaxArgs::misfits)
};

// The item on prices formed per tile and labels in HBM's form, from the start (the hold is
// taken again, which drops a dirty mark, but the labels are read after it).
template <int TH, bool OV, bool GD>
__device__ __noinline__ uint32_t exact_item(const RelaxArgs &a, uint32_t fi, uint32_t t, unsigned char *smem_raw,
                                            unsigned long long *cnt) {
    __builtin_assume(__isShared(smem_raw));
    __builtin_assume(__isShared(cnt));
    return process_item<TH, true, OV, GD, true>(a, fi, t, 0, smem_raw, cnt);
}

// The exact price, on the records in global memory (so that the caller's copies
// stay in registers).
__device__ __noinline__ uint32_t exact_price(const DevBoard *b, const DevField *f, const uint32_t *pads, uint32_t dir,
                                             uint32_t l, uint32_t y, uint32_t x) {
    return exact_in_price(*b, *f, pads, (int)dir, (l * b->h + y) * b->w + x, l, y, x);
}

// The staged form of price p: packed, or plain in a tile of 64-bit words.
template <class W>
__device__ __forceinline__ uint32_t staged_price(uint32_t p, uint32_t *wide) {
    if constexpr (sizeof(W) == 8) return p;
    if (p < (Words<uint32_t>::kNarrow >> kLayerHopBits)) return (p << kLayerHopBits) | 1u;
    if (p != kMax) *wide = 1;
    return kPackedInf;
}

// The stacks of rows y = y0, y0 + step, ...: the layers upward, then downward.  NL is
// the layer count at compile time, so that all labels and prices of a stack are
// loaded before any is used.
template <class W, int NL, int TH>
__device__ __forceinline__ void stack_rows(W *lab, const uint32_t *st, uint32_t y0, uint32_t step) {
    using X = Words<W>;
    constexpr uint32_t LS = TH * X::kPitch, PS = TH * kPitch, SP = NL * PS;  // words from a layer, from a plane, to the next
#pragma unroll 1
    for (uint32_t y = y0; y < TH; y += step) {
        W *q = lab + y * X::kPitch;
        const uint32_t *pu = st + kInBelow * SP + y * kPitch, *pd = st + kInAbove * SP + y * kPitch;
        W c[NL];
        uint32_t up[NL], down[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            c[l] = q[l * LS];
            if (l) up[l] = pu[l * PS];
            if (l + 1 < NL) down[l] = pd[l * PS];
        }
#pragma unroll
        for (int l = 1; l < NL; ++l) c[l] = X::addmin(c[l - 1], X::price(up[l]), c[l]);
#pragma unroll
        for (int l = NL - 2; l >= 0; --l) c[l] = X::addmin(c[l + 1], X::price(down[l]), c[l]);
#pragma unroll
        for (int l = 0; l < NL; ++l) q[l * LS] = c[l];
    }
}

template <class W, int LM, int TH>
__device__ __forceinline__ void stack_pass_layers(W *lab, const uint32_t *st, uint32_t L, uint32_t y0, uint32_t step) {
    using X = Words<W>;
    switch (L) {
        case 2: return stack_rows<W, 2, TH>(lab, st, y0, step);
        case 3: return stack_rows<W, 3, TH>(lab, st, y0, step);
        case 4: return stack_rows<W, 4, TH>(lab, st, y0, step);
    }
    if constexpr (LM > 4) {
        switch (L) {
            case 5: return stack_rows<W, 5, TH>(lab, st, y0, step);
            case 6: return stack_rows<W, 6, TH>(lab, st, y0, step);
            case 7: return stack_rows<W, 7, TH>(lab, st, y0, step);
            case 8: return stack_rows<W, 8, TH>(lab, st, y0, step);
        }
    }
    if constexpr (LM > 8) {  // 9 layers and more, in shared memory
        const uint32_t LS = TH * X::kPitch, PS = TH * kPitch, SP = L * PS;
        for (uint32_t y = y0; y < TH; y += step) {
            W *q = lab + y * X::kPitch;
            const uint32_t *pu = st + kInBelow * SP + y * kPitch, *pd = st + kInAbove * SP + y * kPitch;
            W c = q[0];
            for (uint32_t l = 1; l < L; ++l) q[l * LS] = c = X::addmin(c, X::price(pu[l * PS]), q[l * LS]);
            for (uint32_t l = L - 1; l-- > 0;) q[l * LS] = c = X::addmin(c, X::price(pd[l * PS]), q[l * LS]);
        }
    }
}

// Labels of one layer of the tiles beyond `sides` of the tile at (x, y) of a ww x wh
// window into L2: one 128-byte line a lane, three lines a row of eight.
template <int TH>
__device__ __noinline__ void prefetch_neighbours(const u64 *lab, uint32_t sides, uint32_t lane, int x, int y,
                                                 uint32_t ww, uint32_t wh) {
    for (; sides; sides &= sides - 1u) {
        const uint32_t k = __ffs(sides) - 1u;  // left, right, top, bottom
        const int lx = x + (k == 0 ? -(int)kTW : k == 1 ? (int)kTW : 0) + (int)(lane & 3u) * 16;
        const int ly = y + (k == 2 ? -TH : k == 3 ? TH : 0) + (int)(lane >> 2);
        if ((lane & 3u) < 3u && lx < (int)ww && ly < (int)wh)
            prefetch_l2(lab + (uint64_t)(uint32_t)ly * ww + (uint32_t)max(lx, 0));
    }
}

// What became of an item.  Of the first two thread 0 alone knows.
enum : uint32_t {
    kMoreInFlight = 0,
    kLastInFlight = 1,  // of the launch or (GD) of its field
    kMisfit = 2,        // not done: these words don't hold the tile
    kWontFit = 3        // not tried, nor the price planes waited for
};

// Relaxes one held-to-be item in words W.  BOTH: a tile that 32-bit words don't hold is
// held, with its prices in shared memory, or (`wait`) on their way there, when it gets to
// 64-bit ones (WIDE).  Else such a tile is exact_item's.
template <class W, int LM, int TH, bool OV, bool GD, bool BOTH>
__device__ __forceinline__ uint32_t layer_item(const RelaxArgs &a, uint32_t fi, uint32_t t, unsigned char *smem_raw,
                                               LayerShared &sh, uint32_t &phase, bool wait = true) {
    using X = Words<W>;
    constexpr bool WIDE = sizeof(W) == 8;
    constexpr int HB = X::kHops, RG = TH / 8, NB = 2 + RG;  // row groups, border cells of a lane
    constexpr uint32_t kHopMask = (1u << HB) - 1u, LP = X::kPitch;
    // (static: lambdas that capture them by reference would put them in memory)
    static constexpr W kBig = X::kBig, kNarrow = X::kNarrow, kNone = X::kNone;
    static constexpr uint32_t kFar = (uint32_t)(kNarrow >> HB < kMax ? kBig >> HB : kMax);  // dists from here on don't fit
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wl = tid >> 5;
    const uint32_t r = lane >> 2, seg = lane & 3u;  // row layout: row (of each group of 8) and segment of 8 cells
    const DevField f = a.fields[fi];
    const DevBoard b = a.boards[f.board];
    const uint32_t L = b.layers;
    const uint32_t ntx = field_ntx(f), nty = (f.wh + TH - 1) / TH;
    const uint32_t tyi = t / ntx, txi = t - tyi * ntx;
    const int tx0 = (int)(f.x0 - f.xa + txi * kTW), ty0 = (int)(f.y0 + tyi * TH);
    const uint32_t tw = min(kTW, f.ww + f.xa - txi * kTW), th = min((uint32_t)TH, f.wh - tyi * TH);
    const uint32_t xlo = txi == 0 ? f.xa : 0u;
    uint32_t *st = reinterpret_cast<uint32_t *>(smem_raw);
    W *lab = reinterpret_cast<W *>(smem_raw + layer_lab_off(L, TH));
    uint32_t *live = GD ? &a.goal[fi].active : &a.ctl->count[1];
    uint32_t *state = a.tstamp + f.tile_off + t;
    const bool mine = wl < L;                            // this warp has a layer
    const bool col_in = mine && lane >= xlo && lane < tw;  // this lane has a column of the window
    uint2 lim0;
    if (!WIDE && tid == 0) {
        // hold the tile before reading any label: a neighbour that improves our
        // halo after this point marks it dirty, and we carry it on
        atomicExch(state, kTileHeld);
        // every thread is past the previous item: the planes of this tile go
        // global -> shared while the labels are read
        fence_proxy_async_smem();
        mbar_expect_tx(&sh.mbar, 6u * L * TH * kPitch * 4u);
        tma_load_4d(st, b.tmap, tx0, ty0, 0, 0, &sh.mbar);
        if constexpr (GD) {
            a.tpark[f.tile_off + t] = kMax;  // what waited is in the labels read from here on
            lim0 = __ldcg(reinterpret_cast<const uint2 *>(a.goal + fi));
        }
    }
    // is a price in or around this tile too large?  (the last warp looks: the first one
    // has the hold to wait for)
    if (!WIDE && wl + 1u == (blockDim.x >> 5) && __ldg(&b.goal->wide)) {
        // a lane per 8 x 8 cells: the tile and its ring touch 6 x 4 at most
        const uint32_t bx = (uint32_t)max(tx0 - 1, 0) / 8u + lane % 6u, by = (uint32_t)max(ty0 - 1, 0) / 8u + lane / 6u;
        if (bx <= ((uint32_t)tx0 + kTW) / 8u && by <= ((uint32_t)ty0 + TH) / 8u && bx * 8u < b.w && by * 8u < b.h &&
            __ldg(b.dear + by * dear_pitch(b.w) + bx))
            *(volatile uint32_t *)&sh.wide = 1;
    }
    int misfits = 0;
    if (BOTH && !WIDE && tid == 0) misfits = (int)__ldcg(a.misfits + fi);
    // GD: remaining price along each axis
    uint32_t hxl = 0, hxls = 0;  // of this lane's column, and of its halo column, on this layer
    bool dst_here = false, dst_mine = false;
    uint32_t dst_row = 0;
    if constexpr (GD) {
        const uint32_t plane = b.w * b.h, dst_l = f.dst / plane, dr = f.dst - dst_l * plane, dst_y = dr / b.w,
                       dst_x = dr - dst_y * b.w;
        const uint32_t e = goal_weight(*b.goal, f), each = ~b.goal->inv_min_dir;
        auto rest = [&](const uint32_t *sums, int at, uint32_t n, uint32_t to) {
            return goal_rest(sums, each, e, (uint32_t)min(max(at, 0), (int)n - 1), to);
        };
        const uint32_t *px = b.directed ? nullptr : b.x_sum, *py = b.directed ? nullptr : b.y_sum, *pv = b.via_sum;
        const uint32_t hl = rest(pv, (int)wl, L, dst_l);
        hxl = dsum(rest(px, tx0 + (int)lane, b.w, dst_x), hl);
        hxls = dsum(rest(px, seg == 0 ? tx0 - 1 : tx0 + (int)kTW, b.w, dst_x), hl);
        if (wl == 0 && lane < TH + 2) sh.hy[lane] = rest(py, ty0 + (int)lane - 1, b.h, dst_y);
        dst_here = dst_x >= (uint32_t)tx0 + xlo && dst_x < (uint32_t)tx0 + tw && dst_y >= (uint32_t)ty0 &&
                   dst_y < (uint32_t)ty0 + th;
        dst_row = dst_y - (uint32_t)ty0;
        dst_mine = dst_here && wl == dst_l && lane == dst_x - (uint32_t)tx0;
    }
    if (!WIDE && tid == 0) {
        if (BOTH) sh.misfits = misfits;
        __threadfence();  // the hold before the labels
        if constexpr (GD) {
            sh.ub = lim0.x;   // an older (larger) bound of the target is still a bound
            sh.thr = lim0.y;  // the threshold only moves while no item of the field is in flight
        }
    }
    __syncthreads();
    // the planes: a bounded wait for the TMA load.  A load that never lands sets the
    // status, and the CTA leaves before the write-back
    auto wait_planes = [&]() {
        for (uint32_t spins = 0; !mbar_try_wait(&sh.mbar, phase & 1u); ++spins) {
            if (spins == kTmaSpinLimit) {
                if (tid == 0) atomicOr(&a.ctl->status, kStatusQueueOverflow);
            } else if (spins > 2 * kTmaSpinLimit) {
                *(volatile unsigned long long *)&sh.cnt[0] = kLeaveLaunch;
                *(volatile uint32_t *)&sh.wide = 1;
                break;
            }
        }
        ++phase;
    };
    if (BOTH && !WIDE && sh.misfits >= kMisfits) return kWontFit;  // nor did this field's other tiles

    const u64 *glab = a.lab + f.lab_off;
    const int64_t row0 = ((int64_t)wl * f.wh + (ty0 - (int)f.y0)) * (int64_t)f.ww + (tx0 - (int)f.x0);
    W price[NB];                               // prices into the neighbour tiles' border cells
    const bool top = tyi > 0, bottom = tyi + 1 < nty;
    // border cells of a lane: 0 the top and 1 the bottom of its column, 2 + g its end of
    // row r of group g
    bool side[RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        side[g] = mine && r + 8u * g < th && ((seg == 0 && txi > 0) || (seg == 3 && txi + 1 < ntx));
        price[2 + g] = kNone;
    }
    price[0] = price[1] = kNone;
    // exact price of the move over border cell k
    auto beyond_price = [&](int k) -> uint32_t {
        const uint32_t gx = k < 2 ? (uint32_t)tx0 + lane : seg == 0 ? (uint32_t)tx0 - 1 : (uint32_t)tx0 + kTW;
        const uint32_t gy = k == 0 ? (uint32_t)ty0 - 1 : k == 1 ? (uint32_t)ty0 + TH : (uint32_t)ty0 + r + 8u * (k - 2);
        const uint32_t dir = k == 0 ? kInPosY : k == 1 ? kInNegY : seg == 0 ? kInPosX : kInNegX;
        return exact_price(a.boards + f.board, a.fields + fi, a.pads, dir, wl, gy, gx);
    };
    bool last = false;
    for (uint32_t cont = 0;; ++cont) {
        // ---- labels of the column, the halo rows and the halo columns ----------
        u64 v[TH], vh[NB];
#pragma unroll
        for (int y = 0; y < TH; ++y) {
            v[y] = kInf;
            if (col_in && y < (int)th) v[y] = __ldcg(glab + row0 + (int64_t)y * f.ww + lane);
        }
        vh[0] = col_in && top ? __ldcg(glab + row0 - (int64_t)f.ww + lane) : kInf;
        vh[1] = col_in && bottom ? __ldcg(glab + row0 + (int64_t)TH * f.ww + lane) : kInf;
#pragma unroll
        for (int g = 0; g < RG; ++g)
            vh[2 + g] = side[g] ? __ldcg(glab + row0 + (int64_t)(r + 8u * g) * f.ww + (seg == 0 ? -1 : (int)kTW)) : kInf;
        if (cont == 0) {
            const uint32_t wp = planes_pitch(b.w);
            const uint64_t NP = (uint64_t)wp * b.h * L;
            const uint32_t *pl = b.planes + ((uint64_t)wl * b.h + (uint32_t)ty0) * wp + (uint32_t)tx0;
            auto border = [&](uint32_t dir, int64_t at, int k) -> W {
                const uint32_t p = __ldg(pl + dir * NP + at);
                if constexpr (!WIDE) return p;
                else return X::price(plane_price(p, [&] { return beyond_price(k); }));
            };
            if (col_in && top) price[0] = border(kInPosY, (int64_t)lane - wp, 0);
            if (col_in && bottom) price[1] = border(kInNegY, (int64_t)lane + (int64_t)TH * wp, 1);
#pragma unroll
            for (int g = 0; g < RG; ++g)
                if (side[g])
                    price[2 + g] = border(seg == 0 ? kInPosX : kInNegX, (int64_t)(r + 8u * g) * wp + (seg == 0 ? -1 : (int)kTW), 2 + g);
            // cells of this tile whose prices depend on the net: its own pads, its via pads
            for (uint32_t k = tid; k < f.n_pads + f.n_vpads; k += blockDim.x) {
                const bool q = k >= f.n_pads;
                const uint32_t c = __ldg(a.pads + (q ? f.vpad_off + k - f.n_pads : f.pad_off + k));
                const uint32_t plane = b.w * b.h, l = c / plane, rr = c - l * plane, gy = rr / b.w, gx = rr - gy * b.w;
                const uint32_t x = gx - (uint32_t)tx0, y = gy - (uint32_t)ty0;
                if (x + 1u <= kTW + 1u && y + 1u <= TH + 1u) sh.near_pad = 1;  // in the tile or its ring
                if (x < xlo || x >= tw || y >= th) continue;
                const uint32_t i = atomicAdd(&sh.n_spec, 1u);
                if (i < kSpecCap) sh.spec[i] = (q ? 1u << 31 : 0u) | (l << 16) | (y << 8) | x;
                else sh.wide = 1;
            }
        }
        {
            uint32_t dm = kMax, hm = kMax, hM = 0;
            auto see = [&](u64 q) {
                const uint32_t d = (uint32_t)(q >> 32), h = (uint32_t)q;
                dm = min(dm, d);
                hm = min(hm, h);
                if (d != kMax) hM = max(hM, h);
            };
#pragma unroll
            for (int y = 0; y < TH; ++y) see(v[y]);
#pragma unroll
            for (int k = 0; k < NB; ++k) see(vh[k]);
            dm = __reduce_min_sync(0xFFFFFFFFu, dm);
            hm = __reduce_min_sync(0xFFFFFFFFu, hm);
            hM = __reduce_max_sync(0xFFFFFFFFu, hM);
            if (lane == 0 && dm != kMax) {
                atomicMin(&sh.dmin, dm);
                atomicMin(&sh.hmin, hm);
                atomicMax(&sh.hmax, hM);
            }
        }
        __syncthreads();
        const uint32_t dbase = sh.dmin, hbase = sh.hmin;
        // staged hops stay below the dist bits, and no dist of the tile can saturate
        bool bad = dbase != kMax && (sh.hmax - hbase >= kHopMask || (!WIDE && dbase > kMax - kFar));
        uint32_t ub = kMax;
        W w[TH], w0[TH], lim[TH], there[NB];  // there: staged labels beyond the border
        if constexpr (GD) ub = sh.ub;
        // The word from which on no label counts: +inf, or a dist that saturates (64-bit
        // words, which hold sums past it)
        const W none = WIDE ? (W)(kMax - dbase) << HB : kBig;
        // GD: the word from which on a label at a cell with remaining price h is past
        // the bound `top`: (top - dbase - h + 1) << HB between 0 and that
        auto limit = [&](uint32_t top, uint32_t h) -> W {
            if (!GD || top == kMax) return none;
            const uint32_t room = top >= dbase ? top - dbase + 1u : 0u;
            return (W)min(max(room, h) - h, WIDE ? kMax - dbase : kFar) << HB;
        };
        auto pack = [&](u64 q, W past) -> W {
            const uint32_t d = (uint32_t)(q >> 32);
            const W v = ((W)min(d - dbase, kFar) << HB) | (((uint32_t)q - hbase) & kHopMask);
            if (!WIDE && d != kMax && v >= kNarrow && (v < past || past == kBig)) bad = true;  // it matters and does not fit
            return d == kMax || v >= min(past, kNarrow) ? kBig : v;
        };
        auto set_limits = [&]() {
#pragma unroll
            for (int y = 0; y < TH; ++y) lim[y] = GD ? limit(ub, dsum(hxl, sh.hy[y + 1])) : none;
        };
        set_limits();
#pragma unroll
        for (int y = 0; y < TH; ++y) w0[y] = w[y] = pack(v[y], lim[y]);
        // GD: remaining price from the cell beyond border cell k
        auto beyond = [&](int k) -> uint32_t {
            if (!GD) return 0u;
            return k == 0 ? dsum(hxl, sh.hy[0]) : k == 1 ? dsum(hxl, sh.hy[TH + 1]) : dsum(hxls, sh.hy[r + 8u * (k - 2) + 1]);
        };
#pragma unroll
        for (int k = 0; k < NB; ++k) there[k] = pack(vh[k], limit(ub, beyond(k)));
        if (cont == 0) {
            if constexpr (!WIDE) {
                wait_planes();
                if (mine && (tw < kTW || th < TH || xlo)) {  // no step enters a cell past the window
                    for (uint32_t y = 0; y < TH; ++y) {
                        if (col_in && y < th) continue;
                        for (uint32_t p = 0; p < 6; ++p) st[((p * L + wl) * TH + y) * kPitch + lane] = kPackedInf;
                    }
                }
            } else {  // the prices as they are
                if (wait) wait_planes();
                if (mine) {
#pragma unroll 1
                    for (uint32_t q = 0; q < 6u * TH; ++q) {
                        const uint32_t p = q / TH, y = q % TH;
                        uint32_t &v = st[((p * L + wl) * TH + y) * kPitch + lane];
                        v = !col_in || y >= th ? kMax : plane_price(v, [&] {
                            return exact_price(a.boards + f.board, a.fields + fi, a.pads, p, wl, (uint32_t)ty0 + y, (uint32_t)tx0 + lane);
                        });
                    }
                }
                __syncthreads();
            }
            const uint32_t ns = min(sh.n_spec, kSpecCap);
            const bool over = OV && f.n_over && a.tover[f.tile_off + t];
            for (uint32_t i = tid; i < 6 * ns; i += blockDim.x) {
                const uint32_t e = sh.spec[i / 6], p0 = i % 6;
                uint32_t l = (e >> 16) & 0xFFu, p = p0;
                const uint32_t y = (e >> 8) & 0xFFu, x = e & 0xFFu;
                if (e >> 31) {  // a via pad: the via steps at its cell and at the cells below and above it
                    l = l + p0 / 2 - 1u;
                    if (l >= L) continue;
                    p = (p0 & 1u) ? kInAbove : kInBelow;
                }
                const uint32_t gy = (uint32_t)ty0 + y, gx = (uint32_t)tx0 + x;
                st[((p * L + l) * TH + y) * kPitch + x] =
                    staged_price<W>(exact_price(a.boards + f.board, a.fields + fi, a.pads, p, l, gy, gx), &sh.wide);
            }
            if (over) {  // cells where this net's own directed prices differ from the board's
                const uint32_t *oc = b.over_cells + f.over_off;
                for (uint32_t j = tid; j < L * th; j += blockDim.x) {
                    const uint32_t l = j / th, y = j - l * th, gy = (uint32_t)ty0 + y;
                    const uint32_t lo_c = (l * b.h + gy) * b.w + (uint32_t)tx0 + xlo, hi_c = lo_c - xlo + tw;
                    for (uint32_t k = over_lower_bound(oc, f.n_over, lo_c); k < f.n_over; ++k) {
                        const uint32_t c = __ldg(oc + k);
                        if (c >= hi_c) break;
                        const uint32_t gx = c - (l * b.h + gy) * b.w;
                        for (uint32_t p = kInNegX; p <= kInPosY; ++p)
                            st[((p * L + l) * TH + y) * kPitch + gx - (uint32_t)tx0] =
                                staged_price<W>(exact_price(a.boards + f.board, a.fields + fi, a.pads, p, l, gy, gx),
                                                &sh.wide);
                    }
                }
            }
            if (WIDE || ns || over) __syncthreads();
        }

        // ---- relax to local convergence --------------------------------------
        W *colp = lab + (wl * TH) * LP + lane;              // this lane's column, row y at + y * LP
        W *rowp = lab + (wl * TH + r) * LP + seg * 8;       // this lane's row segment, of group g at + g * 8 * LP
        const uint32_t *stc = st + (wl * TH) * kPitch + lane;          // prices of the column, plane p at + p * L * TH * kPitch
        const uint32_t *str = st + (wl * TH + r) * kPitch + seg * 8;   // prices of the row segment
        const uint32_t SP = L * TH * kPitch;
        bool plane = false;  // this warp's plane is open (warp-uniform)
        if (mine && (WIDE || !*(volatile uint32_t *)&sh.wide)) {  // (else its words don't add)
            bool any = false;
#pragma unroll
            for (int k = 0; k < NB; ++k) any |= there[k] != kBig;
#pragma unroll
            for (int y = 0; y < TH; ++y) {
                any |= w[y] < lim[y];
                colp[y * LP] = w[y];
            }
            plane = __any_sync(0xFFFFFFFFu, any);
        }
        bool stk = plane;    // labels that the stacks have not seen
        uint32_t sweep = 0;
        const uint32_t sweep_limit = L * kTW * TH + 4;
        for (;;) {
            if (plane) {
                for (int it = 0;; ++it) {
                    // columns
                    bool ch = false;
                    {
                        W u[TH], prev = there[0];
#pragma unroll
                        for (int y = 0; y < TH; ++y)
                            prev = u[y] = X::addmin(prev, X::price(stc[kInNegY * SP + y * kPitch]), w[y]);
                        prev = there[1];
#pragma unroll
                        for (int y = TH - 1; y >= 0; --y) {
                            prev = u[y] = X::addmin(prev, X::price(stc[kInPosY * SP + y * kPitch]), u[y]);
                            ch |= u[y] < min(w[y], lim[y]);
                            w[y] = u[y];
                        }
                    }
                    ch = __any_sync(0xFFFFFFFFu, ch);
                    stk |= ch;
                    if (it > 0 && !ch) {  // the rows were closed by the last row pass
                        plane = false;
                        break;
                    }
                    // rows
                    __syncwarp();
#pragma unroll
                    for (int y = 0; y < TH; ++y) colp[y * LP] = w[y];
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < RG; ++g) {
                        W *rp = rowp + g * 8 * LP;
                        const uint32_t *sg = str + g * 8 * kPitch;
                        const W hs = there[2 + g];
                        W u[8], P[8];
                        uint32_t p[8];
#pragma unroll
                        for (int i = 0; i < 8; i += 16 / (int)sizeof(W)) *reinterpret_cast<uint4 *>(u + i) = *reinterpret_cast<const uint4 *>(rp + i);
                        const uint4 *pf = reinterpret_cast<const uint4 *>(sg + kInNegX * SP);
                        *reinterpret_cast<uint4 *>(p) = pf[0];
                        *reinterpret_cast<uint4 *>(p + 4) = pf[1];
                        // forward: the halo column enters the first segment's chain
                        if (seg == 0) u[0] = X::addmin(hs, X::price(p[0]), u[0]);
                        P[0] = X::price(p[0]);
#pragma unroll
                        for (int i = 1; i < 8; ++i) {
                            u[i] = X::addmin(u[i - 1], X::price(p[i]), u[i]);
                            P[i] = X::addmin(P[i - 1], X::price(p[i]), kBig);
                        }
                        W A = u[7], D = P[7];
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            const W Ap = __shfl_up_sync(0xFFFFFFFFu, A, o, 4);
                            const W Dp = __shfl_up_sync(0xFFFFFFFFu, D, o, 4);
                            if (seg >= (uint32_t)o) {
                                A = X::addmin(Ap, D, A);
                                D = X::addmin(Dp, D, kBig);
                            }
                        }
                        W C = __shfl_up_sync(0xFFFFFFFFu, A, 1, 4);
                        if (seg == 0) C = kBig;
#pragma unroll
                        for (int i = 0; i < 8; ++i) u[i] = X::addmin(C, P[i], u[i]);
                        // backward over the forward results
                        const uint4 *pq = reinterpret_cast<const uint4 *>(sg + kInPosX * SP);
                        *reinterpret_cast<uint4 *>(p) = pq[0];
                        *reinterpret_cast<uint4 *>(p + 4) = pq[1];
                        if (seg == 3) u[7] = X::addmin(hs, X::price(p[7]), u[7]);
                        P[7] = X::price(p[7]);
#pragma unroll
                        for (int i = 6; i >= 0; --i) {
                            u[i] = X::addmin(u[i + 1], X::price(p[i]), u[i]);
                            P[i] = X::addmin(P[i + 1], X::price(p[i]), kBig);
                        }
                        A = u[0];
                        D = P[0];
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            const W Ap = __shfl_down_sync(0xFFFFFFFFu, A, o, 4);
                            const W Dp = __shfl_down_sync(0xFFFFFFFFu, D, o, 4);
                            if (seg + (uint32_t)o < 4u) {
                                A = X::addmin(Ap, D, A);
                                D = X::addmin(Dp, D, kBig);
                            }
                        }
                        C = __shfl_down_sync(0xFFFFFFFFu, A, 1, 4);
                        if (seg == 3) C = kBig;
#pragma unroll
                        for (int i = 0; i < 8; ++i) u[i] = X::addmin(C, P[i], u[i]);
#pragma unroll
                        for (int i = 0; i < 8; i += 16 / (int)sizeof(W)) *reinterpret_cast<uint4 *>(rp + i) = *reinterpret_cast<const uint4 *>(u + i);
                    }
                    __syncwarp();
                    ch = false;
#pragma unroll
                    for (int y = 0; y < TH; ++y) {
                        const W n = colp[y * LP];
                        ch |= n < min(w[y], lim[y]);
                        w[y] = n;
                    }
                    plane = __any_sync(0xFFFFFFFFu, ch);
                    stk |= plane;
                    if (!plane || it + 1 == kPlaneIters) break;
                }
            }
            ++sweep;
            if constexpr (GD) {  // the target's own tile tightens its bound from sweep to sweep
                if (dst_mine && !bad) {
                    W q = kBig;
#pragma unroll
                    for (int y = 0; y < TH; ++y)
                        if (y == (int)dst_row) q = w[y];
                    if (q < none && dbase + (uint32_t)(q >> HB) < sh.ub) {  // this lane alone writes it
                        sh.ub = dbase + (uint32_t)(q >> HB);
                        *(volatile uint32_t *)&a.goal[fi].ub = sh.ub;
                    }
                }
            }
            if (!__syncthreads_or(stk || plane)) break;
            if (GD && dst_here) {
                ub = *(volatile uint32_t *)&sh.ub;
                set_limits();
            }
            if (sweep > sweep_limit) {
                if (tid == 0) atomicOr(&a.ctl->status, kStatusRoundLimit);
                break;
            }
            stk = false;
            if (L == 1) continue;
            // the plane's labels are in shared memory, as of the last row pass or the
            // start; a column pass that ended the loop changed nothing
            stack_pass_layers<W, LM, TH>(lab + lane, st + lane, L, wl, blockDim.x >> 5);
            __syncthreads();
            if (mine) {
                bool ch = false;
#pragma unroll
                for (int y = 0; y < TH; ++y) {
                    const W n = colp[y * LP];
                    ch |= n < min(w[y], lim[y]);
                    w[y] = n;
                }
                plane |= __any_sync(0xFFFFFFFFu, ch);
            }
        }

        // ---- is the packing exact for this tile? -------------------------------
        if (mine) {
            W over = ~(W)0;      // least label from kNarrow on (kBig is at kNarrow)
            uint32_t hops = 0;   // most hops
#pragma unroll
            for (int y = 0; y < TH; ++y) {
                if (!WIDE) over = X::addmin(w[y], (W)0 - kNarrow, over);
                hops = max(hops, (uint32_t)w[y] & kHopMask);
            }
            bad |= over < kNarrow || hops == kHopMask;
        }
        if (__syncthreads_or(bad || *(volatile uint32_t *)&sh.wide)) {
            if constexpr (BOTH) {
                return kMisfit;
            } else {
                if (*(volatile unsigned long long *)&sh.cnt[0] == kLeaveLaunch) return kMoreInFlight;  // without its prices
                return exact_item<TH, OV, GD>(a, fi, t, smem_raw, sh.cnt);
            }
        }
        if constexpr (GD) ub = *(volatile uint32_t *)&sh.ub;

        // ---- write back the labels that fell -----------------------------------
        if (mine) {
            u64 *out = a.lab + f.lab_off + row0 + lane;
#pragma unroll
            for (int y = 0; y < TH; ++y)
                if (w[y] < min(w0[y], lim[y]))
                    out[(int64_t)y * f.ww] = ((u64)(dbase + (uint32_t)(w[y] >> HB)) << 32) | (hbase + ((uint32_t)w[y] & kHopMask));
            // ---- neighbours this tile can improve --------------------------------
            // own: our label at a border cell; price: of the move into the neighbour
            // beyond; there: the neighbour's staged label.
            W own[NB];
            bool better[NB], wait[NB];  // improved; GD: improved, past the threshold
            uint32_t ex[NB];            // dist of an exactly priced improvement
            const uint32_t thr = GD ? sh.thr : kMax;
            own[0] = w[0];
            own[1] = w[TH - 1];
#pragma unroll
            for (int g = 0; g < RG; ++g)
                own[2 + g] = side[g] ? lab[(wl * TH + r + 8u * g) * LP + (seg == 0 ? 0u : kTW - 1)] : kBig;
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const W cand = own[k] + price[k];  // (no price or label: at least kBig, as `there` at most, or `none`)
                better[k] = cand < there[k];
                wait[k] = false;
                ex[k] = kMax;
                if constexpr (GD || WIDE) better[k] &= cand < limit(ub, beyond(k));
                if constexpr (GD) wait[k] = better[k] && cand >= limit(thr, beyond(k));
            }
            if (sh.near_pad || (OV && f.n_over)) {  // its own pads, or its own prices, beyond the border
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    const bool ok = (k == 0 ? col_in && top : k == 1 ? col_in && bottom : side[k < 2 ? 0 : k - 2]) && own[k] < none;
                    bool exact = price[k] == kNone;
                    if constexpr (OV) {
                        const uint32_t nb = k == 0 ? t - ntx : k == 1 ? t + ntx : seg == 0 ? t - 1 : t + 1;
                        exact |= ok && f.n_over && a.tover[f.tile_off + nb];
                    }
                    if (!ok || !exact) continue;
                    auto label = [&](W q) { return ((u64)(dbase + (uint32_t)(q >> HB)) << 32) | (hbase + ((uint32_t)q & kHopMask)); };
                    const u64 c64 = ext2(label(own[k]), beyond_price(k), 1);
                    const u64 q64 = there[k] >= none ? kInf : label(there[k]);
                    ex[k] = (uint32_t)(c64 >> 32);
                    const uint32_t fx = min(dsum(ex[k], beyond(k)), kCap);
                    better[k] = c64 < q64 && (!GD || fx <= ub);
                    wait[k] = GD && better[k] && fx > thr;
                }
            }
            bool side_now = false, any_wait = false;
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                better[k] &= !wait[k];
                any_wait |= wait[k];
                if (k >= 2) side_now |= better[k];
            }
            uint32_t sides = (__any_sync(0xFFFFFFFFu, side_now && seg == 0) ? 1u : 0u) |
                             (__any_sync(0xFFFFFFFFu, side_now && seg == 3) ? 2u : 0u) |
                             (__any_sync(0xFFFFFFFFu, better[0]) ? 4u : 0u) | (__any_sync(0xFFFFFFFFu, better[1]) ? 8u : 0u);
            if (lane == 0 && sides) atomicOr(&sh.push, sides);
            if (GD && __any_sync(0xFFFFFFFFu, any_wait)) {
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    if (!wait[k]) continue;
                    const uint32_t d = ex[k] != kMax ? ex[k] : dbase + (uint32_t)((own[k] + price[k]) >> HB);
                    atomicMin(&sh.park[k < 2 ? k + 2 : seg == 0 ? 0 : 1], min(dsum(d, beyond(k)), kCap));
                }
            }
        }
        __syncthreads();
        if (tid < 32) {
            // Lanes 0-3: the neighbours this tile improves; lane 4: the tile itself,
            // released, or, if a neighbour improved it meanwhile, held again and
            // carried on, or queued once more.  The lanes go through each round trip
            // together: the states, then the count of items in flight (this item out,
            // the pushed ones in) beside the tickets, then the slots.
            const uint32_t u = lane == 0 ? t - 1 : lane == 1 ? t + 1 : lane == 2 ? t - ntx : lane == 3 ? t + ntx : t;
            const bool push = lane < 4 && ((sh.push >> lane) & 1u), park = GD && lane < 4 && !push && sh.park[lane & 3u] != kMax;
            uint32_t *us = a.tstamp + f.tile_off + u;
            bool queued = false;  // this lane has an item to publish
            uint32_t more = 0;
            __threadfence();      // the labels before the states
            if (push || lane == 4) {
                uint32_t old = atomicCAS(us, push ? kTileIdle : kTileHeld, push ? kTileQueued : kTileIdle);
                if (push) {
                    for (int tries = 0; old == kTileHeld; ++tries) {  // held: mark it dirty, or find it released
                        if (atomicCAS(us, kTileHeld, kTileHeldDirty) == kTileHeld) break;
                        old = atomicCAS(us, kTileIdle, kTileQueued);
                        if (tries == 1024) {
                            atomicOr(&a.ctl->status, kStatusQueueOverflow);
                            break;
                        }
                    }
                    queued = old == kTileIdle;  // else its holder, or the next one, reads our labels
                } else if (old != kTileHeld) {  // held and dirty
                    more = cont + 1 < kContinueLimit;
                    queued = !more;
                    atomicExch(us, more ? kTileHeld : kTileQueued);
                }
            }
            if (park) atomicMin(a.tpark + f.tile_off + u, sh.park[lane & 3u]);
            if (__any_sync(0xFFFFFFFFu, park || more)) __threadfence();  // before the count; before the labels are read again
            more = __shfl_sync(0xFFFFFFFFu, more, 4);
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, queued), n = __popc(mask);
            uint32_t got = 0;
            if ((lane == 0 && (n || !more)) || (lane == 1 && n))
                got = atomicAdd(lane == 0 ? live : &a.ctl->count[0], lane == 0 ? n + more - 1u : n);
            const uint32_t in_flight = __shfl_sync(0xFFFFFFFFu, got, 0), h0 = __shfl_sync(0xFFFFFFFFu, got, 1);
            if (queued) queue_store(a, h0 + __popc(mask & ((1u << lane) - 1u)), queue_item(fi, u));
            last = !more && in_flight + n == 1u;
            if (lane == 0) {
                sh.more = more;
                sh.dmin = sh.hmin = kMax;
                sh.hmax = 0;
                if (BOTH && !WIDE && sh.misfits > 0) atomicSub(a.misfits + fi, 1);  // one that fits
                sh.cnt[1] += sweep;
                if (++sh.cnt[0] == kCountBatch) {
                    sh.cnt[0] = count_flush(a, sh.cnt[0], sh.cnt[1]) ? 0 : kLeaveLaunch;
                    sh.cnt[1] = 0;
                }
            }
            __syncwarp();
            if (lane < 4) sh.park[lane] = kMax;
            if (lane == 0) sh.push = 0;
        } else if constexpr (LM > 4) {
            // Meanwhile the other warps send for the labels of the tiles being queued,
            // so that they are in L2 when a CTA takes them (layer 0 with layer 1).  Only
            // with more than four layers, where it takes 10 % off (1280x1153x6 1.78 ->
            // 1.60 ms, 640 uneven instances 707 -> 657 us); on four layers the tile's
            // registers are short and it costs 2 % (512x512x4 1.44 -> 1.48 ms).
            const uint32_t sides = *(volatile uint32_t *)&sh.push;
            for (uint32_t l = wl == 1 ? 0u : wl; l <= wl && l < L; ++l)
                prefetch_neighbours<TH>(glab + (int64_t)l * f.wh * f.ww, sides, lane, tx0 - (int)f.x0, ty0 - (int)f.y0, f.ww, f.wh);
        }
        __syncthreads();
        if (!sh.more) break;
    }
    return last ? kLastInFlight : kMoreInFlight;
}

// The item in 64-bit words, or, where they don't hold it, without any; what the 32-bit
// form found out about the tile is forgotten.
template <int LM, int TH, bool OV, bool GD>
__device__ __noinline__ uint32_t wide_item(const RelaxArgs &a, uint32_t fi, uint32_t t, unsigned char *smem_raw,
                                           LayerShared &sh, uint32_t phase, bool wait) {
    __builtin_assume(__isShared(smem_raw));
    __builtin_assume(__isShared(&sh));
    if (sh.cnt[0] == kLeaveLaunch) return kMoreInFlight;  // without its prices
    if (threadIdx.x == 0) {
        if (!wait) atomicAdd(a.misfits + fi, kMisfitWeight);
        sh.n_spec = sh.near_pad = sh.wide = 0;
        sh.dmin = sh.hmin = kMax;
        sh.hmax = 0;
    }
    __syncthreads();
    return layer_item<u64, LM, TH, OV, GD, true>(a, fi, t, smem_raw, sh, phase, wait);
}

// The launch is over: an end word for every ticket that a CTA of the launch holds
// or will take.
__device__ __forceinline__ void end_launch(const RelaxArgs &a) {
    const uint32_t tail = *(volatile const uint32_t *)&a.ctl->count[0];
    for (uint32_t k = threadIdx.x; k < gridDim.x; k += blockDim.x) queue_store(a, tail + k, kSlotItem);
}

// A goal-directed field with nothing in flight: queue the waiting tiles that can
// still matter, or end the field.  The calling CTA is the field's only worker.
// Without a target label the threshold grows (twice the distance above the
// bound, at least to the smallest f that waits; everything after kGoalPhases
// releases); with one, every f up to the target's dist goes.
// Returns whether the launch is over: it was the last field, or the launch has failed.
__device__ __noinline__ bool field_release(const RelaxArgs &a, uint32_t fi) {
    const uint32_t TH = a.tile_h;
    __shared__ uint32_t s_min;
    const DevField f = a.fields[fi];
    FieldGoal *fg = a.goal + fi;
    const uint32_t ntiles = field_ntx(f) * ((f.wh + TH - 1) / TH);
    uint32_t *park = a.tpark + f.tile_off;
    for (;;) {
        __threadfence();
        if (threadIdx.x == 0) s_min = kMax;
        if (__syncthreads_or(threadIdx.x == 0 && launch_failed(a))) return true;  // its tiles may never be released
        const uint32_t ub = *(volatile const uint32_t *)&fg->ub;
        uint32_t m = kMax;
        for (uint32_t i = threadIdx.x; i < ntiles; i += 4 * blockDim.x) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) v[k] = i + k * blockDim.x < ntiles ? __ldcg(park + i + k * blockDim.x) : kMax;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) m = min(m, v[k]);
        }
        m = __reduce_min_sync(0xFFFFFFFFu, m);
        if ((threadIdx.x & 31) == 0 && m != kMax) atomicMin(&s_min, m);
        __syncthreads();
        m = s_min;
        if (m == kMax || m > ub) {  // nothing waits that could matter: the field is final
            __syncthreads();
            if (threadIdx.x == 0) s_min = atomicSub(&a.ctl->count[1], 1u);
            __syncthreads();
            return s_min == 1u;
        }
        uint32_t thr = kMax;
        const uint32_t f0 = __ldcg(&fg->f0), phases = __ldcg(&fg->phases);
        if (ub == kMax && phases + 1 < kGoalPhases) {
            const uint32_t was = *(volatile const uint32_t *)&fg->thr, slack = was - f0;
            thr = max(dsum(was, slack), dsum(m, slack / 2));
        }
        if (threadIdx.x == 0) atomicAdd(&fg->active, 1u);  // this CTA, until every release is queued
        __syncthreads();
        if (threadIdx.x == 0) {
            *(volatile uint32_t *)&fg->thr = thr;
            fg->phases = phases + 1;
            __threadfence();
        }
        __syncthreads();
        const uint32_t lim = min(thr, ub);
        const uint32_t lane = threadIdx.x & 31u;
        for (uint32_t i0 = threadIdx.x - lane; i0 < ntiles; i0 += blockDim.x) {
            const uint32_t i = i0 + lane, v = i < ntiles ? __ldcg(park + i) : kMax;
            const bool go = v != kMax && v <= lim && atomicCAS(a.tstamp + f.tile_off + i, kTileIdle, kTileQueued) == kTileIdle;
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, go), n = __popc(mask);
            if (!n) continue;
            uint32_t got = 0;
            if (lane < 2) got = atomicAdd(lane == 0 ? &fg->active : &a.ctl->count[0], n);
            const uint32_t live = __shfl_sync(0xFFFFFFFFu, got, 0), h0 = __shfl_sync(0xFFFFFFFFu, got, 1);
            // (live is used so that its round trip ends before the items are visible)
            if (go && live != kMax) queue_store(a, h0 + __popc(mask & ((1u << lane) - 1u)), queue_item(fi, i));
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            s_min = atomicSub(&fg->active, 1u) - 1u;
        }
        __syncthreads();
        if (s_min != 0) return false;  // the field's other workers carry it on
        __syncthreads();
    }
}

constexpr u64 kReleaseField = kInf - 1;  // in place of an item: this CTA finished the last one in flight

template <int LM, int TH, bool OV, bool GD, bool BOTH>
__global__ void __launch_bounds__(LM * 32, LM == 4 ? (TH == 8 ? 5 : 3) : LM == 8 ? 3 : 1) relax_layer_kernel(const __grid_constant__ RelaxArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ LayerShared sh;
    uint32_t phase = 0, fi = 0;
    bool last = false;
    if (threadIdx.x == 0) {
        sh.cnt[0] = sh.cnt[1] = 0;
        mbar_init(&sh.mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) {
            sh.item = sh.cnt[0] == kLeaveLaunch ? kInf : last ? kReleaseField : async_pop<64>(a);
            sh.n_spec = sh.near_pad = sh.wide = 0;
            sh.dmin = sh.hmin = kMax;
            sh.hmax = 0;
            sh.push = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) sh.park[k] = kMax;
        }
        __syncthreads();
        const u64 item = sh.item;
        if (item == kInf) break;
        if (item == kReleaseField) {  // nothing in flight: of the field (GD), of the launch
            if (!GD || field_release(a, fi)) {
                end_launch(a);
                break;
            }
            last = false;
        } else {
            fi = (uint32_t)(item >> 32);
            uint32_t r = layer_item<uint32_t, LM, TH, OV, GD, BOTH>(a, fi, (uint32_t)item, smem_raw, sh, phase);
            if constexpr (BOTH) {
                if (r >= kMisfit) {
                    const bool wait = r == kWontFit;
                    r = wide_item<LM, TH, OV, GD>(a, fi, (uint32_t)item, smem_raw, sh, phase, wait);
                    phase += wait;
                    if (r == kMisfit && sh.cnt[0] != kLeaveLaunch)
                        r = exact_item<TH, OV, GD>(a, fi, (uint32_t)item, smem_raw, sh.cnt);
                }
            }
            last = r == kLastInFlight;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (sh.cnt[0] && sh.cnt[0] != kLeaveLaunch) atomicAdd(&a.ctl->activations, sh.cnt[0]);
        if (sh.cnt[1]) atomicAdd(&a.ctl->sweeps, sh.cnt[1]);
    }
}

template <int LM, int TH, bool BOTH>
const void *layer_fn_lm(bool over, bool goal) {
    if constexpr (TH == kLayerTileH) {
        if (over)
            return goal ? (const void *)relax_layer_kernel<LM, TH, true, true, BOTH> : (const void *)relax_layer_kernel<LM, TH, true, false, BOTH>;
    } else if (over) {
        return nullptr;
    }
    return goal ? (const void *)relax_layer_kernel<LM, TH, false, true, BOTH> : (const void *)relax_layer_kernel<LM, TH, false, false, BOTH>;
}

template <bool BOTH>
const void *layer_fn_words(uint32_t max_layers, uint32_t tile_h, bool over, bool goal) {
    if (tile_h == kLayerTallH) return max_layers <= kLayerTallMax ? layer_fn_lm<4, kLayerTallH, BOTH>(over, goal) : nullptr;
    return max_layers <= 4   ? layer_fn_lm<4, kLayerTileH, BOTH>(over, goal)
           : max_layers <= 8  ? layer_fn_lm<8, kLayerTileH, BOTH>(over, goal)
           : max_layers <= 16 ? layer_fn_lm<16, kLayerTileH, BOTH>(over, goal)
                              : layer_fn_lm<kLayerMax, kLayerTileH, BOTH>(over, goal);
}

const void *layer_fn(uint32_t max_layers, uint32_t tile_h, bool over, bool goal, bool both) {
    return both ? layer_fn_words<true>(max_layers, tile_h, over, goal) : layer_fn_words<false>(max_layers, tile_h, over, goal);
}

}  // namespace

size_t layer_smem_bytes(uint32_t max_layers, uint32_t tile_h) {
    const size_t words = layer_lab_off(max_layers, tile_h) + (size_t)max_layers * tile_h * Words<u64>::kPitch * 8;
    return std::max(words, tile_layout(max_layers, tile_h).total);  // exact_item's tile is staged in the same block
}

cudaError_t layer_configure(uint32_t max_layers, uint32_t tile_h, size_t smem, bool over, bool goal, bool both, int *blocks_per_sm) {
    const void *fn = layer_fn(max_layers, tile_h, over, goal, both);
    if (!fn) return cudaErrorInvalidValue;
    // the most any layer count of this kernel takes: a batch of more layers may
    // already be laid out, and is launched after this call
    const uint32_t most = max_layers <= 4 ? 4u : max_layers <= 8 ? 8u : max_layers <= 16 ? 16u : kLayerMax;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)layer_smem_bytes(most, tile_h));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, (int)max_layers * 32, smem);
}

cudaError_t layer_launch(const RelaxArgs &a, uint32_t grid, size_t smem, cudaStream_t st, bool over, bool goal, bool both) {
    const cudaError_t e = seed_launch(a, st);
    if (e != cudaSuccess) return e;
    RelaxArgs copy = a;
    void *args[] = {&copy};
    return cudaLaunchKernel(layer_fn(a.max_layers, a.tile_h, over, goal, both), dim3(grid), dim3(a.max_layers * 32), args, smem, st);
}

}  // namespace mrc
