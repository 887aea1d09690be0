// layer_relax.cu — the queue-driven relax kernel with a warp per layer and 32-bit labels.
//
// A CTA holds one 32 x TH tile over all L layers of a field, warp l its layer l:
// lane x keeps the TH labels of column x in registers.  TH is 8, or 16 where the
// batch's longest chains of tiles bound it (batch_layout has the rule).  Inside an activation a
// label is one word, (dist - least staged dist) << HB | (hops - least staged
// hops), and a step price is (price << HB) | 1, so the lexicographic min-plus step
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
// could have been clamped), or with a final label at the last value of the hops, is
// relaxed on 64-bit labels instead (wide_item), from the labels in HBM, which this
// kernel has not touched by then.  (Words are sums dist 2^HB + hops, so a word is
// the lexicographic least label as long as that label's hops fit, whatever other
// paths carried into the dist; and the first label of a best path that doesn't fit
// follows one whose hops are the last value.)  So is every tile
// of a board with a finite price of 2^(29 - HB) or more.
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

constexpr uint32_t kBig = kPackedInf;   // +inf
constexpr uint32_t kNarrow = 1u << 29;  // staged labels, final labels and prices lie below
// Pitch of a row of labels or prices: 16-byte aligned, and the rows' segments and
// the columns of a warp fall on distinct banks.
constexpr uint32_t kPitch = kPlaneTmaBoxW;
constexpr uint32_t kSpecCap = 512;      // cells of a tile priced for the net itself
constexpr int kPlaneIters = 2;          // column and row passes of a plane between two meetings

__host__ __device__ inline size_t layer_st_off(uint32_t L, uint32_t TH) {
    return ((size_t)L * TH * kPitch * 4 + 127) & ~(size_t)127;
}

struct LayerShared {
    u64 item;
    uint64_t mbar;  // completion of the price-plane TMA loads
    unsigned long long cnt[2];  // activations and sweeps not yet added to the launch's
    uint32_t n_spec, near_pad, wide, dmin, hmin, hmax, ub, thr, more;
    uint32_t push;              // bits: left, right, top, bottom improved
    uint32_t park[4];           // GD: the smallest f that waits to enter each
    uint32_t hy[kLayerTallH + 2];  // GD: remaining price along y, rows -1 .. TH
    uint32_t spec[kSpecCap];
};

// The 64-bit form of one item, from the start (the hold is taken again, which
// drops a dirty mark, but the labels are read after it).
template <int TH, bool OV, bool GD>
__device__ __noinline__ bool wide_item(const RelaxArgs &a, uint32_t fi, uint32_t t, unsigned char *smem_raw,
                                       unsigned long long *cnt) {
    return process_item<TH, true, OV, GD, true>(a, fi, t, 0, smem_raw, cnt);
}

// The exact price, on the records in global memory (so that the caller's copies
// stay in registers).
__device__ __noinline__ uint32_t exact_price(const DevBoard *b, const DevField *f, const uint32_t *pads, uint32_t dir,
                                             uint32_t l, uint32_t y, uint32_t x) {
    return exact_in_price(*b, *f, pads, (int)dir, (l * b->h + y) * b->w + x, l, y, x);
}

template <int HB>
__device__ __forceinline__ uint32_t pack_price(uint32_t p, uint32_t *wide) {
    if (p < (kNarrow >> HB)) return (p << HB) | 1u;
    if (p != kMax) *wide = 1;
    return kBig;
}

// The stacks of rows y = y0, y0 + step, ...: the layers upward, then downward.  NL is
// the layer count at compile time, so that all labels and prices of a stack are
// loaded before any is used.
template <int NL, int TH>
__device__ __forceinline__ void stack_rows(uint32_t *lab, const uint32_t *st, uint32_t y0, uint32_t step) {
    constexpr uint32_t LS = TH * kPitch, SP = NL * LS;  // words from a layer, from a plane, to the next
#pragma unroll 1
    for (uint32_t y = y0; y < TH; y += step) {
        uint32_t *q = lab + y * kPitch;
        const uint32_t *pu = st + kInBelow * SP + y * kPitch, *pd = st + kInAbove * SP + y * kPitch;
        uint32_t c[NL], up[NL], down[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            c[l] = q[l * LS];
            if (l) up[l] = pu[l * LS];
            if (l + 1 < NL) down[l] = pd[l * LS];
        }
#pragma unroll
        for (int l = 1; l < NL; ++l) c[l] = __viaddmin_u32(c[l - 1], up[l], c[l]);
#pragma unroll
        for (int l = NL - 2; l >= 0; --l) c[l] = __viaddmin_u32(c[l + 1], down[l], c[l]);
#pragma unroll
        for (int l = 0; l < NL; ++l) q[l * LS] = c[l];
    }
}

template <int LM, int TH>
__device__ __forceinline__ void stack_pass_layers(uint32_t *lab, const uint32_t *st, uint32_t L, uint32_t y0,
                                                  uint32_t step) {
    switch (L) {
        case 2: return stack_rows<2, TH>(lab, st, y0, step);
        case 3: return stack_rows<3, TH>(lab, st, y0, step);
        case 4: return stack_rows<4, TH>(lab, st, y0, step);
    }
    if constexpr (LM > 4) {
        switch (L) {
            case 5: return stack_rows<5, TH>(lab, st, y0, step);
            case 6: return stack_rows<6, TH>(lab, st, y0, step);
            case 7: return stack_rows<7, TH>(lab, st, y0, step);
            case 8: return stack_rows<8, TH>(lab, st, y0, step);
        }
    }
    if constexpr (LM > 8) {  // 9 .. 16 layers, in shared memory
        const uint32_t LS = TH * kPitch, SP = L * LS;
        for (uint32_t y = y0; y < TH; y += step) {
            uint32_t *q = lab + y * kPitch;
            const uint32_t *pu = st + kInBelow * SP + y * kPitch, *pd = st + kInAbove * SP + y * kPitch;
            uint32_t c = q[0];
            for (uint32_t l = 1; l < L; ++l) q[l * LS] = c = __viaddmin_u32(c, pu[l * LS], q[l * LS]);
            for (uint32_t l = L - 1; l-- > 0;) q[l * LS] = c = __viaddmin_u32(c, pd[l * LS], q[l * LS]);
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

// Relaxes one held-to-be item; thread 0 returns whether it was the last one in
// flight, of the launch or (GD) of its field.
template <int LM, int TH, bool OV, bool GD>
__device__ __forceinline__ bool layer_item(const RelaxArgs &a, uint32_t fi, uint32_t t, unsigned char *smem_raw,
                                           LayerShared &sh, uint32_t &phase) {
    constexpr int HB = (int)kLayerHopBits, RG = TH / 8, NB = 2 + RG;  // row groups, border cells of a lane
    constexpr uint32_t kHopMask = (1u << HB) - 1u;
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
    uint32_t *lab = reinterpret_cast<uint32_t *>(smem_raw);
    uint32_t *st = reinterpret_cast<uint32_t *>(smem_raw + layer_st_off(L, TH));
    uint32_t *live = GD ? &a.goal[fi].active : &a.ctl->count[1];
    uint32_t *state = a.tstamp + f.tile_off + t;
    const bool mine = wl < L;                            // this warp has a layer
    const bool col_in = mine && lane >= xlo && lane < tw;  // this lane has a column of the window
    uint2 lim0;
    if (tid == 0) {
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
    const uint32_t board_wide = __ldg(&b.goal->wide);
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
    if (tid == 0) {
        __threadfence();  // the hold before the labels
        if constexpr (GD) {
            sh.ub = lim0.x;   // an older (larger) bound of the target is still a bound
            sh.thr = lim0.y;  // the threshold only moves while no item of the field is in flight
        }
    }
    __syncthreads();

    const u64 *glab = a.lab + f.lab_off;
    const int64_t row0 = ((int64_t)wl * f.wh + (ty0 - (int)f.y0)) * (int64_t)f.ww + (tx0 - (int)f.x0);
    uint32_t price[NB];                        // prices into the neighbour tiles' border cells
    const bool top = tyi > 0, bottom = tyi + 1 < nty;
    // border cells of a lane: 0 the top and 1 the bottom of its column, 2 + g its end of
    // row r of group g
    bool side[RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        side[g] = mine && r + 8u * g < th && ((seg == 0 && txi > 0) || (seg == 3 && txi + 1 < ntx));
        price[2 + g] = kBig;
    }
    price[0] = price[1] = kBig;
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
            if (col_in && top) price[0] = __ldg(pl + kInPosY * NP + lane - wp);
            if (col_in && bottom) price[1] = __ldg(pl + kInNegY * NP + lane + (uint64_t)TH * wp);
#pragma unroll
            for (int g = 0; g < RG; ++g)
                if (side[g])
                    price[2 + g] = __ldg(pl + (seg == 0 ? kInPosX : kInNegX) * NP + (uint64_t)(r + 8u * g) * wp +
                                         (seg == 0 ? -1 : (int)kTW));
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
        bool bad = dbase != kMax && (sh.hmax - hbase >= kHopMask || dbase > kMax - (kBig >> HB));
        uint32_t ub = kMax;
        uint32_t w[TH], w0[TH], lim[TH], there[NB];  // there: staged labels beyond the border
        if constexpr (GD) ub = sh.ub;
        // GD: the word from which on a label at a cell with remaining price h is past
        // the bound `top`: (top - dbase - h + 1) << HB between 0 and kBig
        auto limit = [&](uint32_t top, uint32_t h) -> uint32_t {
            if (!GD || top == kMax) return kBig;
            const uint32_t room = top >= dbase ? top - dbase + 1u : 0u;
            return min(max(room, h) - h, kBig >> HB) << HB;
        };
        auto pack = [&](u64 q, uint32_t past) {
            const uint32_t d = (uint32_t)(q >> 32);
            const uint32_t v = (min(d - dbase, kBig >> HB) << HB) | (((uint32_t)q - hbase) & kHopMask);
            if (d != kMax && v >= kNarrow && (v < past || past == kBig)) bad = true;  // it matters and does not fit
            return d == kMax || v >= min(past, kNarrow) ? kBig : v;
        };
        auto set_limits = [&]() {
#pragma unroll
            for (int y = 0; y < TH; ++y) lim[y] = GD ? limit(ub, dsum(hxl, sh.hy[y + 1])) : kBig;
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
            // the planes: a bounded wait for the TMA load.  A load that never lands sets
            // the status, and the CTA leaves before the write-back
            for (uint32_t spins = 0; !mbar_try_wait(&sh.mbar, phase & 1u); ++spins) {
                if (spins == kTmaSpinLimit) {
                    if (tid == 0) atomicOr(&a.ctl->status, kStatusQueueOverflow);
                } else if (spins > 2 * kTmaSpinLimit) {
                    *(volatile unsigned long long *)&sh.cnt[0] = kLeaveLaunch;
                    bad = true;
                    break;
                }
            }
            ++phase;
            if (board_wide) {
                if (__syncthreads_or(bad && *(volatile unsigned long long *)&sh.cnt[0] == kLeaveLaunch)) return false;
                // everybody is past the load and the staged words
                return wide_item<TH, OV, GD>(a, fi, t, smem_raw, sh.cnt);
            }
            if (mine && (tw < kTW || th < TH || xlo)) {  // no step enters a cell past the window
                for (uint32_t y = 0; y < TH; ++y) {
                    if (col_in && y < th) continue;
                    for (uint32_t p = 0; p < 6; ++p) st[((p * L + wl) * TH + y) * kPitch + lane] = kBig;
                }
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
                    pack_price<HB>(exact_price(a.boards + f.board, a.fields + fi, a.pads, p, l, gy, gx), &sh.wide);
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
                                pack_price<HB>(exact_price(a.boards + f.board, a.fields + fi, a.pads, p, l, gy, gx),
                                               &sh.wide);
                    }
                }
            }
            if (ns || over) __syncthreads();
        }

        // ---- relax to local convergence --------------------------------------
        uint32_t *colp = lab + (wl * TH) * kPitch + lane;              // this lane's column, row y at + y * kPitch
        uint4 *rowp = reinterpret_cast<uint4 *>(lab + (wl * TH + r) * kPitch + seg * 8);  // group g at + g * 2 * kPitch
        const uint32_t *stc = st + (wl * TH) * kPitch + lane;          // prices of the column, plane p at + p * L * TH * kPitch
        const uint32_t *str = st + (wl * TH + r) * kPitch + seg * 8;   // prices of the row segment
        const uint32_t SP = L * TH * kPitch;
        bool plane = false;  // this warp's plane is open (warp-uniform)
        if (mine) {
            bool any = false;
#pragma unroll
            for (int k = 0; k < NB; ++k) any |= there[k] != kBig;
#pragma unroll
            for (int y = 0; y < TH; ++y) {
                any |= w[y] < lim[y];
                colp[y * kPitch] = w[y];
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
                        uint32_t u[TH], prev = there[0];
#pragma unroll
                        for (int y = 0; y < TH; ++y)
                            prev = u[y] = __viaddmin_u32(prev, stc[kInNegY * SP + y * kPitch], w[y]);
                        prev = there[1];
#pragma unroll
                        for (int y = TH - 1; y >= 0; --y) {
                            prev = u[y] = __viaddmin_u32(prev, stc[kInPosY * SP + y * kPitch], u[y]);
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
                    for (int y = 0; y < TH; ++y) colp[y * kPitch] = w[y];
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < RG; ++g) {
                        uint4 *rp = rowp + g * 2 * kPitch;
                        const uint32_t *sg = str + g * 8 * kPitch, hs = there[2 + g];
                        uint32_t u[8], p[8], P[8];
                        *reinterpret_cast<uint4 *>(u) = rp[0];
                        *reinterpret_cast<uint4 *>(u + 4) = rp[1];
                        const uint4 *pf = reinterpret_cast<const uint4 *>(sg + kInNegX * SP);
                        *reinterpret_cast<uint4 *>(p) = pf[0];
                        *reinterpret_cast<uint4 *>(p + 4) = pf[1];
                        // forward: the halo column enters the first segment's chain
                        if (seg == 0) u[0] = __viaddmin_u32(hs, p[0], u[0]);
                        P[0] = p[0];
#pragma unroll
                        for (int i = 1; i < 8; ++i) {
                            u[i] = __viaddmin_u32(u[i - 1], p[i], u[i]);
                            P[i] = __viaddmin_u32(P[i - 1], p[i], kBig);
                        }
                        uint32_t A = u[7], D = P[7];
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            const uint32_t Ap = __shfl_up_sync(0xFFFFFFFFu, A, o, 4);
                            const uint32_t Dp = __shfl_up_sync(0xFFFFFFFFu, D, o, 4);
                            if (seg >= (uint32_t)o) {
                                A = __viaddmin_u32(Ap, D, A);
                                D = __viaddmin_u32(Dp, D, kBig);
                            }
                        }
                        uint32_t C = __shfl_up_sync(0xFFFFFFFFu, A, 1, 4);
                        if (seg == 0) C = kBig;
#pragma unroll
                        for (int i = 0; i < 8; ++i) u[i] = __viaddmin_u32(C, P[i], u[i]);
                        // backward over the forward results
                        const uint4 *pq = reinterpret_cast<const uint4 *>(sg + kInPosX * SP);
                        *reinterpret_cast<uint4 *>(p) = pq[0];
                        *reinterpret_cast<uint4 *>(p + 4) = pq[1];
                        if (seg == 3) u[7] = __viaddmin_u32(hs, p[7], u[7]);
                        P[7] = p[7];
#pragma unroll
                        for (int i = 6; i >= 0; --i) {
                            u[i] = __viaddmin_u32(u[i + 1], p[i], u[i]);
                            P[i] = __viaddmin_u32(P[i + 1], p[i], kBig);
                        }
                        A = u[0];
                        D = P[0];
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            const uint32_t Ap = __shfl_down_sync(0xFFFFFFFFu, A, o, 4);
                            const uint32_t Dp = __shfl_down_sync(0xFFFFFFFFu, D, o, 4);
                            if (seg + (uint32_t)o < 4u) {
                                A = __viaddmin_u32(Ap, D, A);
                                D = __viaddmin_u32(Dp, D, kBig);
                            }
                        }
                        C = __shfl_down_sync(0xFFFFFFFFu, A, 1, 4);
                        if (seg == 3) C = kBig;
#pragma unroll
                        for (int i = 0; i < 8; ++i) u[i] = __viaddmin_u32(C, P[i], u[i]);
                        rp[0] = *reinterpret_cast<uint4 *>(u);
                        rp[1] = *reinterpret_cast<uint4 *>(u + 4);
                    }
                    __syncwarp();
                    ch = false;
#pragma unroll
                    for (int y = 0; y < TH; ++y) {
                        const uint32_t n = colp[y * kPitch];
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
                    uint32_t q = kBig;
#pragma unroll
                    for (int y = 0; y < TH; ++y)
                        if (y == (int)dst_row) q = w[y];
                    if (q < kBig && dbase + (q >> HB) < sh.ub) {  // this lane alone writes it
                        sh.ub = dbase + (q >> HB);
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
            stack_pass_layers<LM, TH>(lab + lane, st + lane, L, wl, blockDim.x >> 5);
            __syncthreads();
            if (mine) {
                bool ch = false;
#pragma unroll
                for (int y = 0; y < TH; ++y) {
                    const uint32_t n = colp[y * kPitch];
                    ch |= n < min(w[y], lim[y]);
                    w[y] = n;
                }
                plane |= __any_sync(0xFFFFFFFFu, ch);
            }
        }

        // ---- is the packing exact for this tile? -------------------------------
        if (mine) {
            uint32_t over = kMax, hops = 0;  // least label from kNarrow on (kBig is at kNarrow), most hops
#pragma unroll
            for (int y = 0; y < TH; ++y) {
                over = __viaddmin_u32(w[y], 0u - kNarrow, over);
                hops = max(hops, w[y] & kHopMask);
            }
            bad |= over < kNarrow || hops == kHopMask;
        }
        if (__syncthreads_or(bad || *(volatile uint32_t *)&sh.wide)) {
            if (*(volatile unsigned long long *)&sh.cnt[0] == kLeaveLaunch) return false;  // without its prices
            return wide_item<TH, OV, GD>(a, fi, t, smem_raw, sh.cnt);
        }
        if constexpr (GD) ub = *(volatile uint32_t *)&sh.ub;

        // ---- write back the labels that fell -----------------------------------
        if (mine) {
            u64 *out = a.lab + f.lab_off + row0 + lane;
#pragma unroll
            for (int y = 0; y < TH; ++y)
                if (w[y] < min(w0[y], lim[y]))
                    out[(int64_t)y * f.ww] = ((u64)(dbase + (w[y] >> HB)) << 32) | (hbase + (w[y] & kHopMask));
            // ---- neighbours this tile can improve --------------------------------
            // own: our label at a border cell; price: of the move into the neighbour
            // beyond; there: the neighbour's staged label.
            uint32_t own[NB];
            bool better[NB], wait[NB];  // improved; GD: improved, past the threshold
            uint32_t ex[NB];            // dist of an exactly priced improvement
            const uint32_t thr = GD ? sh.thr : kMax;
            own[0] = w[0];
            own[1] = w[TH - 1];
#pragma unroll
            for (int g = 0; g < RG; ++g)
                own[2 + g] = side[g] ? lab[(wl * TH + r + 8u * g) * kPitch + (seg == 0 ? 0u : kTW - 1)] : kBig;
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const uint32_t cand = own[k] + price[k];  // (no price or label: at least kBig, as `there` at most)
                better[k] = cand < there[k];
                wait[k] = false;
                ex[k] = kMax;
                if constexpr (GD) {
                    better[k] &= cand < limit(ub, beyond(k));
                    wait[k] = better[k] && cand >= limit(thr, beyond(k));
                }
            }
            if (sh.near_pad || (OV && f.n_over)) {  // its own pads, or its own prices, beyond the border
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    const bool ok = (k == 0 ? col_in && top : k == 1 ? col_in && bottom : side[k < 2 ? 0 : k - 2]) && own[k] < kBig;
                    bool exact = price[k] == kBig;
                    if constexpr (OV) {
                        const uint32_t nb = k == 0 ? t - ntx : k == 1 ? t + ntx : seg == 0 ? t - 1 : t + 1;
                        exact |= ok && f.n_over && a.tover[f.tile_off + nb];
                    }
                    if (!ok || !exact) continue;
                    const uint32_t gx = k < 2 ? (uint32_t)tx0 + lane : seg == 0 ? (uint32_t)tx0 - 1 : (uint32_t)tx0 + kTW;
                    const uint32_t gy = k == 0 ? (uint32_t)ty0 - 1 : k == 1 ? (uint32_t)ty0 + TH : (uint32_t)ty0 + r + 8u * (k - 2);
                    const uint32_t dir = k == 0 ? kInPosY : k == 1 ? kInNegY : seg == 0 ? kInPosX : kInNegX;
                    const uint32_t p = exact_price(a.boards + f.board, a.fields + fi, a.pads, dir, wl, gy, gx);
                    const u64 c64 = ext2(((u64)(dbase + (own[k] >> HB)) << 32) | (hbase + (own[k] & kHopMask)), p, 1);
                    const u64 q64 = there[k] >= kBig ? kInf : ((u64)(dbase + (there[k] >> HB)) << 32) |
                                                                  (hbase + (there[k] & kHopMask));
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
                    const uint32_t d = ex[k] != kMax ? ex[k] : dbase + ((own[k] + price[k]) >> HB);
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
    return last;
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

template <int LM, int TH, bool OV, bool GD>
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
            last = layer_item<LM, TH, OV, GD>(a, fi, (uint32_t)item, smem_raw, sh, phase);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (sh.cnt[0] && sh.cnt[0] != kLeaveLaunch) atomicAdd(&a.ctl->activations, sh.cnt[0]);
        if (sh.cnt[1]) atomicAdd(&a.ctl->sweeps, sh.cnt[1]);
    }
}

template <int LM, int TH>
const void *layer_fn_lm(bool over, bool goal) {
    if constexpr (TH == kLayerTileH) {
        if (over)
            return goal ? (const void *)relax_layer_kernel<LM, TH, true, true> : (const void *)relax_layer_kernel<LM, TH, true, false>;
    } else if (over) {
        return nullptr;
    }
    return goal ? (const void *)relax_layer_kernel<LM, TH, false, true> : (const void *)relax_layer_kernel<LM, TH, false, false>;
}

const void *layer_fn(uint32_t max_layers, uint32_t tile_h, bool over, bool goal) {
    if (tile_h == kLayerTallH) return max_layers <= kLayerTallMax ? layer_fn_lm<4, kLayerTallH>(over, goal) : nullptr;
    return max_layers <= 4   ? layer_fn_lm<4, kLayerTileH>(over, goal)
           : max_layers <= 8 ? layer_fn_lm<8, kLayerTileH>(over, goal)
                             : layer_fn_lm<16, kLayerTileH>(over, goal);
}

}  // namespace

size_t layer_smem_bytes(uint32_t max_layers, uint32_t tile_h) {
    const size_t narrow = layer_st_off(max_layers, tile_h) + (size_t)6 * max_layers * tile_h * kPitch * 4;
    return std::max(narrow, tile_layout(max_layers, tile_h).total);  // a wide tile is staged in the same block
}

cudaError_t layer_configure(uint32_t max_layers, uint32_t tile_h, size_t smem, bool over, bool goal, int *blocks_per_sm) {
    const void *fn = layer_fn(max_layers, tile_h, over, goal);
    if (!fn) return cudaErrorInvalidValue;
    // the most any layer count of this kernel takes: a batch of more layers may
    // already be laid out, and is launched after this call
    const uint32_t most = max_layers <= 4 ? 4u : max_layers <= 8 ? 8u : 16u;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)layer_smem_bytes(most, tile_h));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, (int)max_layers * 32, smem);
}

cudaError_t layer_launch(const RelaxArgs &a, uint32_t grid, size_t smem, cudaStream_t st, bool over, bool goal) {
    const cudaError_t e = seed_launch(a, st);
    if (e != cudaSuccess) return e;
    RelaxArgs copy = a;
    void *args[] = {&copy};
    return cudaLaunchKernel(layer_fn(a.max_layers, a.tile_h, over, goal), dim3(grid), dim3(a.max_layers * 32), args, smem, st);
}

}  // namespace mrc
