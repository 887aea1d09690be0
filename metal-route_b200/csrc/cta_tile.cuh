// cta_tile.cuh — one (field, tile) item relaxed by a whole CTA on 64-bit labels.
//
// The tile of the bulk-synchronous rounds and of the queue form with prices
// formed per tile (relax.cu); the layer kernel (layer_relax.cu) falls back to it
// for tiles whose labels or prices do not fit its 32-bit words.
#pragma once

#include <algorithm>

#include "device.cuh"
#include "kernels.h"
#include "tiles.cuh"

namespace mrc {

constexpr uint32_t kTW = 32;  // tile width (one warp across a row)
constexpr int kLaneCells = 4;  // cells per lane in the row / column passes
// Shared-memory row pitches of the staged tile: labels (u64) per 34-cell row
// (32 + halo), step prices (u32) per 32-cell row.  (Padding them to 35 / 33
// removes bank conflicts of the row passes but measured no faster, and the
// extra bytes cost a resident CTA per SM on 8-layer tiles.)
constexpr uint32_t kLabPitch = 34;
constexpr uint32_t kStPitch = 32;
constexpr uint32_t kFlPitch = 36;  // flag bytes per staged row (34 used)
constexpr int kStageUnroll = 4;    // cells whose loads one thread issues together
constexpr uint32_t kNone = 0xFFFFFFFFu;


// Asynchronous 4-byte global -> shared copy (cp.async, L1-allocating) and its
// completion wait.
__device__ __forceinline__ void cp_async4(uint32_t *smem, const uint32_t *gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }


// Step-price planes of a staged tile: the move into cell c from its neighbour
// at -x, +x, -y, +y, the layer below and the layer above.
enum { kFromNegX = 0, kFromPosX = 1, kFromNegY = 2, kFromPosY = 3, kFromBelow = 4, kFromAbove = 5 };

// GD: goal-directed, labels whose bound f = dist + remaining price exceeds `ub`
// are not kept.
template <int TH, bool GD>
struct Tile {
    u64 *lab;        // [L][TH+2][34] labels with a one-cell halo ring
    uint32_t *st;    // [6][L][TH][32] step prices into interior cells
    uint8_t *rowd;   // [L][TH] row needs a sweep
    uint8_t *cold;   // [L][32] column needs a sweep
    uint8_t *stackd; // [TH][32] layer stack needs a sweep
    uint32_t *fellw; // [L][TH] bit x: the label of (l, y, x) fell in this activation
    uint8_t *fl;     // [L][TH+2][kFlPitch] board flag bytes of the tile and its halo
    uint32_t L;
    const uint32_t *hx, *hy, *hl;  // GD: remaining price along each axis, by staged column, staged row and layer
    uint32_t ub;                   // GD: no cheapest path has a larger f
    // f of a label with this dist at staged (l, sy, sx): at most kCap, and equal to
    // the dist's own saturation rule (a sum that reaches kMax is unreachable)
    __device__ __forceinline__ uint32_t bound(uint32_t dist, uint32_t l, uint32_t sy, uint32_t sx) const {
        return min(dsum(dsum(dist, hx[sx]), dsum(hy[sy], hl[l])), kCap);
    }
    // is a label worth keeping (interior cell)
    __device__ __forceinline__ bool within(u64 lab_v, uint32_t l, uint32_t y, uint32_t x) const {
        if constexpr (GD) return bound((uint32_t)(lab_v >> 32), l, y + 1, x + 1) <= ub;
        else return true;
    }
    __device__ __forceinline__ uint32_t li(uint32_t l, uint32_t sy, uint32_t sx) const {
        return (l * (TH + 2) + sy) * kLabPitch + sx;
    }
    __device__ __forceinline__ uint32_t si(uint32_t plane, uint32_t l, uint32_t y, uint32_t x) const {
        return ((plane * L + l) * TH + y) * kStPitch + x;
    }
    __device__ __forceinline__ void fell(uint32_t l, uint32_t y, uint32_t x) const {
        atomicOr(&fellw[l * TH + y], 1u << x);
    }
    // a label of interior cell (l, y, x) fell: every other line through it must be swept again
    __device__ __forceinline__ void touched_by_row(uint32_t l, uint32_t y, uint32_t x) const {
        cold[l * 32 + x] = 1;
        stackd[y * 32 + x] = 1;
        fell(l, y, x);
    }
    __device__ __forceinline__ void touched_by_col(uint32_t l, uint32_t y, uint32_t x) const {
        rowd[l * TH + y] = 1;
        stackd[y * 32 + x] = 1;
        fell(l, y, x);
    }
    __device__ __forceinline__ void touched_by_stack(uint32_t l, uint32_t y, uint32_t x) const {
        rowd[l * TH + y] = 1;
        cold[l * 32 + x] = 1;
        fell(l, y, x);
    }
};

// Line passes over lines of K*S cells, S consecutive lanes per line (K cells
// each), skipping lines whose dirty flag is clear.  Each lane runs its
// segment's local chain, the S lanes combine their transfer functions
// f(t) = min(A, t (+) (D, H)) with a Kogge-Stone scan (H, the hop count, is the
// group's cell count), and every cell takes min(local, incoming (+) prefix).
// `halo(line, &before, &after)` gives the label indices outside both ends;
// `keep(line, pos, label)` says whether a lower label is worth storing and
// `touch(line, pos)` marks the crossing lines of a cell whose label fell.
// Both directions of a line run in one pass: the forward scan, then, on its
// results still in registers, the backward scan (mirror image: shuffles down,
// the halo after the last cell).  A 1-D line is closed by one forward and one
// backward scan, so one load and one store of each label serve both.  `cell(line, pos, &lab,
// &step_fwd, &step_bwd)`: step_fwd prices the move into the cell from its
// predecessor in traversal order, step_bwd the move from its successor.
template <int K, int S, class CellFn, class HaloFn, class KeepFn, class TouchFn>
__device__ __forceinline__ bool seg_pass(u64 *lab, const uint32_t *st, uint8_t *dirty, uint32_t nlines, CellFn cell,
                                          HaloFn halo, KeepFn keep, TouchFn touch) {
    bool changed = false;
    const uint32_t lanes_total = nlines * S;
    for (uint32_t base = 0; base < lanes_total; base += blockDim.x) {
        if (base + (threadIdx.x & ~31u) >= lanes_total) break;
        const uint32_t tl = base + threadIdx.x;
        const uint32_t line = tl / S, seg = tl % S;
        const bool mine = dirty[line] != 0;
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, mine);
        if (!mine) continue;
        if (seg == 0) dirty[line] = 0;
        u64 v[K], u[K];
        uint32_t spf[K], spb[K], P[K], li[K];
#pragma unroll
        for (int i = 0; i < K; ++i) {
            uint32_t sf, sb;
            cell(line, seg * K + i, &li[i], &sf, &sb);
            v[i] = lab[li[i]];
            spf[i] = st[sf];
            spb[i] = st[sb];
        }
        uint32_t hf, hb;
        halo(line, &hf, &hb);
        // forward
        u[0] = v[0];
        P[0] = spf[0];
#pragma unroll
        for (int i = 1; i < K; ++i) {
            u[i] = umin64(v[i], ext2(u[i - 1], spf[i], 1));
            P[i] = dsum(P[i - 1], spf[i]);
        }
        {
            u64 A = u[K - 1];
            uint32_t D = P[K - 1];
#pragma unroll
            for (int o = 1; o < S; o <<= 1) {
                const u64 Ap = __shfl_up_sync(mask, A, o, S);
                const uint32_t Dp = __shfl_up_sync(mask, D, o, S);
                if (seg >= (uint32_t)o) {
                    A = umin64(A, ext2(Ap, D, (uint32_t)(K * o)));
                    D = dsum(Dp, D);
                }
            }
            const u64 hl = lab[hf];
            u64 C = hl;
            if (S > 1) {
                const u64 Fa = __shfl_up_sync(mask, A, 1, S);
                const uint32_t Fd = __shfl_up_sync(mask, D, 1, S);
                if (seg > 0) C = umin64(Fa, ext2(hl, Fd, K * seg));
            }
            if (C != kInf) {
#pragma unroll
                for (int i = 0; i < K; ++i) u[i] = umin64(u[i], ext2(C, P[i], (uint32_t)i + 1u));
            }
        }
        // backward over the forward results; segment sb = S-1-seg counts from the far end
        {
            const uint32_t sbk = (uint32_t)(S - 1) - seg;
            P[K - 1] = spb[K - 1];
#pragma unroll
            for (int i = K - 2; i >= 0; --i) {
                u[i] = umin64(u[i], ext2(u[i + 1], spb[i], 1));
                P[i] = dsum(P[i + 1], spb[i]);
            }
            u64 A = u[0];
            uint32_t D = P[0];
#pragma unroll
            for (int o = 1; o < S; o <<= 1) {
                const u64 Ap = __shfl_down_sync(mask, A, o, S);
                const uint32_t Dp = __shfl_down_sync(mask, D, o, S);
                if (sbk >= (uint32_t)o) {
                    A = umin64(A, ext2(Ap, D, (uint32_t)(K * o)));
                    D = dsum(Dp, D);
                }
            }
            const u64 hr = lab[hb];
            u64 C = hr;
            if (S > 1) {
                const u64 Fa = __shfl_down_sync(mask, A, 1, S);
                const uint32_t Fd = __shfl_down_sync(mask, D, 1, S);
                if (sbk > 0) C = umin64(Fa, ext2(hr, Fd, K * sbk));
            }
            if (C != kInf) {
#pragma unroll
                for (int i = 0; i < K; ++i) u[i] = umin64(u[i], ext2(C, P[i], (uint32_t)(K - i)));
            }
        }
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (u[i] < v[i] && keep(line, seg * K + i, u[i])) {
                lab[li[i]] = u[i];
                touch(line, seg * K + i);
                changed = true;
            }
        }
    }
    return changed;
}


// Flags of a window cell as a via endpoint: blocked by the board via node bit or
// by the static via mask unless the net lists the cell as a via pad.
// Own-pad and via-exemption lookups against the shared-memory copy of the
// field's sorted lists when they fit (kPadCache / kVPadCache), else HBM.
constexpr uint32_t kPadCache = 128, kVPadCache = 32;
__device__ __forceinline__ bool own_pad(const uint32_t *s, uint32_t cap, const uint32_t *g, uint32_t n,
                                        uint32_t key) {
    return n <= cap ? sorted_has(s, n, key) : sorted_has(g, n, key);
}

__device__ __forceinline__ bool via_blocked(const DevField &f, const uint32_t *pads, uint32_t gcell, uint8_t gf) {
    return (cell_tile_flags(f, pads, gcell, gf) & kViaBlocked) != 0;
}

template <int TH, bool GD>
__device__ __forceinline__ bool stack_pass(const Tile<TH, GD> &t);

// With 8-row tiles and 4 cells per lane, the row lanes of a layer (8 rows x 8
// lanes) and its column lanes (32 columns x 2 lanes) fall on the same pair of
// warps (2p, 2p+1), in every iteration of a pass.  Between the row and column
// passes those 64 threads synchronise alone (named barrier 1 + p) instead of
// the whole CTA.
__device__ __forceinline__ void pair_barrier() {
    asm volatile("bar.sync %0, 64;" ::"r"(1u + (threadIdx.x >> 6)) : "memory");
}

// The row and the column pass of a sweep on their own (the reversed sweep's).
template <int TH, bool GD>
__device__ __forceinline__ bool row_pass(const Tile<TH, GD> &t) {
    constexpr int KC = kLaneCells, SR = 32 / KC;  // cells per lane, lanes per row
    return seg_pass<KC, SR>(
        t.lab, t.st, t.rowd, t.L * TH,
        [&](uint32_t line, uint32_t pos, uint32_t *li, uint32_t *sf, uint32_t *sb) {
            const uint32_t l = line / TH, y = line % TH;
            *li = t.li(l, y + 1, pos + 1);
            *sf = t.si(kFromNegX, l, y, pos);
            *sb = t.si(kFromPosX, l, y, pos);
        },
        [&](uint32_t line, uint32_t *hf, uint32_t *hb) {
            *hf = t.li(line / TH, line % TH + 1, 0);
            *hb = t.li(line / TH, line % TH + 1, 33);
        },
        [&](uint32_t line, uint32_t pos, u64 v) { return t.within(v, line / TH, line % TH, pos); },
        [&](uint32_t line, uint32_t pos) { t.touched_by_row(line / TH, line % TH, pos); });
}

template <int TH, bool GD>
__device__ __forceinline__ bool col_pass(const Tile<TH, GD> &t) {
    constexpr int KC = kLaneCells, SC = TH / KC;  // cells per lane, lanes per column
    return seg_pass<KC, SC>(
        t.lab, t.st, t.cold, t.L * 32,
        [&](uint32_t line, uint32_t pos, uint32_t *li, uint32_t *sf, uint32_t *sb) {
            const uint32_t l = line / 32, x = line % 32;
            *li = t.li(l, pos + 1, x + 1);
            *sf = t.si(kFromNegY, l, pos, x);
            *sb = t.si(kFromPosY, l, pos, x);
        },
        [&](uint32_t line, uint32_t *hf, uint32_t *hb) {
            *hf = t.li(line / 32, 0, line % 32 + 1);
            *hb = t.li(line / 32, TH + 1, line % 32 + 1);
        },
        [&](uint32_t line, uint32_t pos, u64 v) { return t.within(v, line / 32, pos, line % 32); },
        [&](uint32_t line, uint32_t pos) { t.touched_by_col(line / 32, pos, line % 32); });
}

// rows <-> columns: only the warps of the same layers exchange data
// (WHOLE: the CTA's width is not a multiple of 64, so everybody meets)
template <int TH, bool WHOLE>
__device__ __forceinline__ void plane_barrier() {
    if constexpr (TH == 8 && kLaneCells == 4 && !WHOLE) {
        pair_barrier();
    } else {
        __syncthreads();
    }
}

// One sweep of a staged tile: rows (8 lanes x 4 cells), columns (TH/4 lanes x
// 4 cells), layer stacks (one thread each), each forward then backward, only
// over lines whose dirty flag is set.
template <int TH, bool GD>
__device__ __forceinline__ bool relax_tile(const Tile<TH, GD> &t) {
    constexpr int KC = kLaneCells;          // cells per lane in a line pass
    constexpr int SR = 32 / KC, SC = TH / KC;  // lanes per row / per column
    const uint32_t L = t.L;
    bool ch = false;
    ch |= seg_pass<KC, SR>(
        t.lab, t.st, t.rowd, L * TH,
        [&](uint32_t line, uint32_t pos, uint32_t *li, uint32_t *sf, uint32_t *sb) {
            const uint32_t l = line / TH, y = line % TH;
            *li = t.li(l, y + 1, pos + 1);
            *sf = t.si(kFromNegX, l, y, pos);
            *sb = t.si(kFromPosX, l, y, pos);
        },
        [&](uint32_t line, uint32_t *hf, uint32_t *hb) {
            *hf = t.li(line / TH, line % TH + 1, 0);
            *hb = t.li(line / TH, line % TH + 1, 33);
        },
        [&](uint32_t line, uint32_t pos, u64 v) { return t.within(v, line / TH, line % TH, pos); },
        [&](uint32_t line, uint32_t pos) { t.touched_by_row(line / TH, line % TH, pos); });
    // rows -> columns: only the warps of the same layers exchange data
    if constexpr (TH == 8 && kLaneCells == 4) {
        pair_barrier();
    } else {
        __syncthreads();
    }
    ch |= seg_pass<KC, SC>(
        t.lab, t.st, t.cold, L * 32,
        [&](uint32_t line, uint32_t pos, uint32_t *li, uint32_t *sf, uint32_t *sb) {
            const uint32_t l = line / 32, x = line % 32;
            *li = t.li(l, pos + 1, x + 1);
            *sf = t.si(kFromNegY, l, pos, x);
            *sb = t.si(kFromPosY, l, pos, x);
        },
        [&](uint32_t line, uint32_t *hf, uint32_t *hb) {
            *hf = t.li(line / 32, 0, line % 32 + 1);
            *hb = t.li(line / 32, TH + 1, line % 32 + 1);
        },
        [&](uint32_t line, uint32_t pos, u64 v) { return t.within(v, line / 32, pos, line % 32); },
        [&](uint32_t line, uint32_t pos) { t.touched_by_col(line / 32, pos, line % 32); });
    if (L > 1) {
        __syncthreads();
        ch |= stack_pass(t);
    }
    return ch;
}

// Columns first, then rows and stacks: the queue form's order (fewer sweeps per
// activation than rows first on its 32 x 8 tiles).
template <int TH, bool WHOLE, bool GD>
__device__ __forceinline__ bool relax_tile_cols_first(const Tile<TH, GD> &t) {
    bool ch = col_pass(t);
    plane_barrier<TH, WHOLE>();
    ch |= row_pass(t);
    if (t.L > 1) {
        __syncthreads();
        ch |= stack_pass(t);
    }
    return ch;
}

// The same passes in the opposite order (stacks, columns, rows); the rounds
// form alternates the two orders between sweeps.
template <int TH, bool GD>
__device__ __forceinline__ bool relax_tile_rev(const Tile<TH, GD> &t) {
    bool ch = false;
    if (t.L > 1) {
        ch = stack_pass(t);
        __syncthreads();
    }
    ch |= col_pass(t);
    plane_barrier<TH, false>();
    ch |= row_pass(t);
    return ch;
}

// Layer stacks: one thread per (y, x) column of the tile, upward then downward.
// Stacks of up to kStackRegs layers are held in registers between the two
// directions (one load and at most one store per label); taller ones run from
// shared memory.
constexpr uint32_t kStackRegs = 4;

template <int TH, bool GD>
__device__ __forceinline__ bool stack_pass(const Tile<TH, GD> &t) {
    const uint32_t L = t.L;
    bool ch = false;
    for (uint32_t r = threadIdx.x; r < TH * 32; r += blockDim.x) {
        if (!t.stackd[r]) continue;
        t.stackd[r] = 0;
        const uint32_t y = r / 32, x = r % 32;
        if (L <= kStackRegs) {
            u64 v[kStackRegs];
            uint32_t fell = 0;  // bit l: the label of layer l fell
#pragma unroll
            for (uint32_t l = 0; l < kStackRegs; ++l)
                if (l < L) v[l] = t.lab[t.li(l, y + 1, x + 1)];
            u64 prev = kInf;
#pragma unroll
            for (uint32_t l = 0; l < kStackRegs; ++l) {
                if (l < L) {
                    const u64 w = ext2(prev, l ? t.st[t.si(kFromBelow, l, y, x)] : kMax, 1);
                    if (w < v[l] && t.within(w, l, y, x)) {
                        v[l] = w;
                        fell |= 1u << l;
                    }
                    prev = v[l];
                }
            }
            prev = kInf;
#pragma unroll
            for (int l = (int)kStackRegs - 1; l >= 0; --l) {
                if ((uint32_t)l < L) {
                    const u64 w = ext2(prev, (uint32_t)l + 1 < L ? t.st[t.si(kFromAbove, (uint32_t)l, y, x)] : kMax, 1);
                    if (w < v[l] && t.within(w, (uint32_t)l, y, x)) {
                        v[l] = w;
                        fell |= 1u << l;
                    }
                    prev = v[l];
                }
            }
#pragma unroll
            for (uint32_t l = 0; l < kStackRegs; ++l) {
                if ((fell >> l) & 1u) {
                    t.lab[t.li(l, y + 1, x + 1)] = v[l];
                    t.touched_by_stack(l, y, x);
                    ch = true;
                }
            }
            continue;
        }
        u64 prev = kInf;
        for (uint32_t l = 0; l < L; ++l) {
            const uint32_t c = t.li(l, y + 1, x + 1);
            const u64 cur = t.lab[c];
            const u64 w = umin64(cur, ext2(prev, l ? t.st[t.si(kFromBelow, l, y, x)] : kMax, 1));
            if (w < cur && t.within(w, l, y, x)) {
                t.lab[c] = w;
                t.touched_by_stack(l, y, x);
                ch = true;
            }
            prev = w;
        }
        prev = kInf;
        for (int l = (int)L - 1; l >= 0; --l) {
            const uint32_t c = t.li((uint32_t)l, y + 1, x + 1);
            const u64 cur = t.lab[c];
            const u64 w =
                umin64(cur, ext2(prev, (uint32_t)l + 1 < L ? t.st[t.si(kFromAbove, (uint32_t)l, y, x)] : kMax, 1));
            if (w < cur && t.within(w, (uint32_t)l, y, x)) {
                t.lab[c] = w;
                t.touched_by_stack((uint32_t)l, y, x);
                ch = true;
            }
            prev = w;
        }
    }
    return ch;
}

// One (field, tile) item: stage the tile and its halo, relax it to local
// convergence, write it back and queue the neighbours it improves.
// Shared-memory layout of one staged tile (relax_smem_bytes sizes it the same way).
struct TileLayout {
    size_t st, rowd, fellw, fl, total;
};
__host__ __device__ inline TileLayout tile_layout(uint32_t L, uint32_t TH) {
    TileLayout o;
    o.st = ((size_t)L * (TH + 2) * kLabPitch * 8 + 127) & ~(size_t)127;
    o.rowd = o.st + (size_t)6 * L * TH * kStPitch * 4;
    o.fellw = (o.rowd + (size_t)L * TH + (size_t)L * kTW + (size_t)TH * kTW + 3) & ~(size_t)3;
    o.fl = o.fellw + (size_t)L * TH * 4;
    o.total = o.fl + (size_t)L * (TH + 2) * kFlPitch;
    return o;
}

// A field's directed-price overrides inside its tile (a negotiation net's own
// prices on its own footprint): they replace the raw directed words in the
// planes laid out as Tile::si, before the step prices are formed.  Out of line:
// it runs only for overriding fields and keeps the staging's registers free.
static __device__ __noinline__ void stage_overrides(const DevBoard &b, const DevField &f, uint32_t *st, uint32_t L,
                                                    uint32_t TH, int tx0, int ty0, uint32_t tw, uint32_t th) {
    const uint32_t *oc = b.over_cells + f.over_off;
    auto si = [&](int p, uint32_t l, uint32_t y, uint32_t x) { return (((uint32_t)p * L + l) * TH + y) * kStPitch + x; };
    for (uint32_t j = threadIdx.x; j < L * th; j += blockDim.x) {
        const uint32_t l = j / th, y = j - l * th;
        const uint32_t lo_c = (l * b.h + (uint32_t)ty0 + y) * b.w + (uint32_t)tx0, hi_c = lo_c + tw;
        for (uint32_t k = over_lower_bound(oc, f.n_over, lo_c); k < f.n_over; ++k) {
            const uint32_t c = __ldg(oc + k);
            if (c >= hi_c) break;
            const uint32_t x = c - lo_c;
            const uint4 d = __ldg(b.over_price + f.over_off + k);
            st[si(kFromNegX, l, y, x)] = d.y;
            st[si(kFromPosX, l, y, x)] = d.z;
            st[si(kFromNegY, l, y, x)] = d.x;
            st[si(kFromPosY, l, y, x)] = d.w;
        }
    }
}

// OV: the batch carries per-net directed-price overrides (negotiation with a
// clearance; always 8-row tiles); without it none of the override lookups is
// compiled in.  GD: goal-directed (FieldGoal).  Returns true when this item was
// the last one in flight, of the launch or (GD) of its field.
// WHOLE: see plane_barrier.
template <int TH, bool ASYNC, bool OV, bool GD, bool WHOLE = false>
__device__ __forceinline__ bool process_item(const RelaxArgs &a, uint32_t fi, uint32_t t, uint32_t round,
                                             unsigned char *smem_raw, unsigned long long *s_cnt) {
    const uint32_t SW = kTW + 2, SH = TH + 2;
    Tile<TH, GD> tile;
    __shared__ uint32_t s_push[4];
    __shared__ uint32_t s_park[4];                    // GD: smallest f that enters each neighbour above the threshold
    __shared__ uint32_t s_hx[kTW + 2], s_hy[TH + 2], s_hl[32], s_lim[2];
    __shared__ uint32_t s_vis[5];  // self, left, right, top, bottom
    __shared__ uint32_t s_pads[kPadCache], s_vpads[kVPadCache];
    Ctl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x;
    const uint32_t cap = a.list_cap;
    const DevField f = a.fields[fi];
    const DevBoard b = a.boards[f.board];
    const uint32_t L = b.layers;  // the shared tile is laid out for this board's layers
    const uint32_t nsm = L * SH * SW;  // staged cells (pitch kLabPitch in smem)
    const uint32_t ntx = field_ntx(f), nty = (f.wh + TH - 1) / TH;
    const uint32_t txi = t % ntx, tyi = t / ntx;
    const int tx0 = (int)(f.x0 - f.xa + txi * kTW), ty0 = (int)(f.y0 + tyi * TH);
    const TileLayout lay = tile_layout(L, TH);
    tile.lab = reinterpret_cast<u64 *>(smem_raw);
    tile.st = reinterpret_cast<uint32_t *>(smem_raw + lay.st);
    tile.rowd = smem_raw + lay.rowd;
    tile.cold = tile.rowd + L * TH;
    tile.stackd = tile.cold + L * kTW;
    tile.fellw = reinterpret_cast<uint32_t *>(smem_raw + lay.fellw);
    const uint32_t fell_words = L * TH;  // words of fell marks to clear
    tile.fl = smem_raw + lay.fl;
    tile.L = L;
    const uint32_t tw = min(kTW, f.ww + f.xa - txi * kTW), th = min(TH, f.wh - tyi * TH);  // (first columns may lie before the window)
    const int wx0 = (int)f.x0, wy0 = (int)f.y0, wx1 = (int)(f.x0 + f.ww), wy1 = (int)(f.y0 + f.wh);
    const u64 *lab = a.lab + f.lab_off;
    uint32_t *live = GD ? &a.goal[fi].active : &ctl->count[1];  // the count this item and its pushes are in
    bool last = false;
    if constexpr (ASYNC) {
        // hold the tile before reading any label: a neighbour that improves our
        // halo after this point marks it dirty, and we queue it again when done
        if (tid == 0) {
            atomicExch(a.tstamp + f.tile_off + t, kTileHeld);
            if constexpr (GD) a.tpark[f.tile_off + t] = kMax;  // what waited is in the labels read from here on
            __threadfence();
        }
    } else if (tid < 5) {
        uint32_t u = kNone;
        if (tid == 0) u = t;
        else if (tid == 1 && txi > 0) u = t - 1;
        else if (tid == 2 && txi + 1 < ntx) u = t + 1;
        else if (tid == 3 && tyi > 0) u = t - ntx;
        else if (tid == 4 && tyi + 1 < nty) u = t + ntx;
        s_vis[tid] = u == kNone ? 0u : __ldcg(a.tvisit + f.tile_off + u);
    }
    if (tid < 4) s_push[tid] = 0;
    // GD: the field's limits and the remaining price along each axis
    const uint32_t dst_r = f.dst % (b.w * b.h), dst_x = dst_r % b.w, dst_y = dst_r / b.w, dst_l = f.dst / (b.w * b.h);
    const bool dst_here = dst_x >= (uint32_t)tx0 && dst_x < (uint32_t)tx0 + kTW && dst_y >= (uint32_t)ty0 &&
                          dst_y < (uint32_t)ty0 + TH && dst_x < f.x0 + f.ww && dst_y < f.y0 + f.wh;
    const uint32_t dst_li = dst_here ? tile.li(dst_l, dst_y - ty0 + 1, dst_x - tx0 + 1) : 0u;
    if constexpr (GD) {
        if (tid < 4) s_park[tid] = kMax;
        if (tid == 0) {
            const uint2 lim = __ldcg(reinterpret_cast<const uint2 *>(a.goal + fi));
            s_lim[0] = lim.x;  // an older (larger) bound of the target is still a bound
            s_lim[1] = lim.y;  // the threshold only moves while no item of the field is in flight
        }
        const uint32_t e = goal_weight(*b.goal, f), each = ~b.goal->inv_min_dir;
        auto rest = [&](const uint32_t *sums, int at, int n, uint32_t to) {
            return goal_rest(sums, each, e, (uint32_t)min(max(at, 0), n - 1), to);
        };
        const uint32_t *hx = b.directed ? nullptr : b.x_sum, *hy = b.directed ? nullptr : b.y_sum, *hv = b.via_sum;
        for (uint32_t i = tid; i < SW + SH + L; i += blockDim.x) {
            if (i < SW) s_hx[i] = rest(hx, tx0 + (int)i - 1, (int)b.w, dst_x);
            else if (i < SW + SH) s_hy[i - SW] = rest(hy, ty0 + (int)(i - SW) - 1, (int)b.h, dst_y);
            else s_hl[i - SW - SH] = rest(hv, (int)(i - SW - SH), (int)L, dst_l);
        }
        tile.hx = s_hx;
        tile.hy = s_hy;
        tile.hl = s_hl;
    }
    if (f.n_pads <= kPadCache)
        for (uint32_t i = tid; i < f.n_pads; i += blockDim.x) s_pads[i] = __ldg(a.pads + f.pad_off + i);
    if (f.n_vpads <= kVPadCache)
        for (uint32_t i = tid; i < f.n_vpads; i += blockDim.x) s_vpads[i] = __ldg(a.pads + f.vpad_off + i);
    const uint32_t *gpads = a.pads + f.pad_off, *gvpads = a.pads + f.vpad_off;
    auto is_own_pad = [&](uint32_t c) {
        return c == f.src || c == f.dst || own_pad(s_pads, kPadCache, gpads, f.n_pads, c);
    };
    auto via_blk = [&](uint32_t c, uint8_t gf) {
        if (gf & kViaNode) return true;
        return (gf & kStaticVia) != 0 && !own_pad(s_vpads, kVPadCache, gvpads, f.n_vpads, c);
    };
    // Dirty lines start clear; staging marks exactly the lines that hold a
    // finite label (in the tile, or at their ends in the halo ring): a line of
    // +inf labels with +inf ends cannot change until a crossing line lowers one
    // of its cells, and that pass marks it.
    for (uint32_t i = tid; i < L * TH + L * kTW + TH * kTW; i += blockDim.x) tile.rowd[i] = 0;
    for (uint32_t i = tid; i < fell_words; i += blockDim.x) tile.fellw[i] = 0;
    __syncthreads();
    if constexpr (GD) tile.ub = s_lim[0];

    // ---- step prices into every interior cell: phase 1 -----------------
    // Per interior cell its cost (parked in the below-plane) and its four
    // planar base prices go global -> shared with asynchronous copies issued
    // first, so they overlap the label and flag loads below.  The board is
    // read-only during the launch, so the L1-allocating cp.async is safe for it
    // (labels, which other CTAs write, keep their L2-only loads).
    {
        const uint32_t ncell = L * TH * kTW;
        for (uint32_t i = tid; i < ncell; i += blockDim.x) {
            const uint32_t x = i % kTW, r = i / kTW, y = r % TH, l = r / TH;
            const int gx = tx0 + (int)x, gy = ty0 + (int)y;
            uint32_t *d0 = &tile.st[tile.si(kFromNegX, l, y, x)], *d1 = &tile.st[tile.si(kFromPosX, l, y, x)];
            uint32_t *d2 = &tile.st[tile.si(kFromNegY, l, y, x)], *d3 = &tile.st[tile.si(kFromPosY, l, y, x)];
            uint32_t *dc = &tile.st[tile.si(kFromBelow, l, y, x)];
            if (gx >= wx0 && gx < wx1 && gy < wy1) {
                const uint32_t gc = (l * b.h + (uint32_t)gy) * b.w + (uint32_t)gx;
                cp_async4(dc, b.cost + gc);
                if (b.directed) {
                    const uint32_t *dp = reinterpret_cast<const uint32_t *>(b.directed + gc);
                    cp_async4(d0, dp + 1);  // from -x
                    cp_async4(d1, dp + 2);  // from +x
                    cp_async4(d2, dp + 0);  // from -y
                    cp_async4(d3, dp + 3);  // from +y
                } else {
                    *d0 = gx > wx0 ? __ldg(b.x_edge + gx - 1) : kMax;
                    *d1 = gx + 1 < wx1 ? __ldg(b.x_edge + gx) : kMax;
                    *d2 = gy > wy0 ? __ldg(b.y_edge + gy - 1) : kMax;
                    *d3 = gy + 1 < wy1 ? __ldg(b.y_edge + gy) : kMax;
                }
            } else {
                *d0 = *d1 = *d2 = *d3 = *dc = kMax;
            }
        }
        cp_async_commit();
    }

    // ---- stage labels and flag bytes (tile + halo ring) ---------------
    // Every thread issues the loads of kStageUnroll cells before it
    // stores any of them, so several L2 requests per thread are in
    // flight (labels through L2 with ld.global.cg).
    const uint32_t plane = b.w * b.h;
    for (uint32_t i0 = tid; i0 < nsm; i0 += kStageUnroll * blockDim.x) {
        u64 lv[kStageUnroll];
        uint8_t fv[kStageUnroll];
#pragma unroll
        for (int k = 0; k < kStageUnroll; ++k) {
            const uint32_t i = i0 + k * blockDim.x;
            lv[k] = kInf;
            fv[k] = 0;
            if (i >= nsm) continue;
            const uint32_t sx = i % SW, r = i / SW, sy = r % SH, l = r / SH;
            const int gx = tx0 + (int)sx - 1, gy = ty0 + (int)sy - 1;
            if (gx >= wx0 && gx < wx1 && gy >= wy0 && gy < wy1) {
                const bool hx = sx == 0 || sx == SW - 1, hy = sy == 0 || sy == SH - 1;
                uint32_t owner;  // which tile's label this smem cell holds
                if (hx && hy) owner = 5;  // corner: never read
                else if (sx == 0) owner = 1;
                else if (sx == SW - 1) owner = 2;
                else if (sy == 0) owner = 3;
                else if (sy == SH - 1) owner = 4;
                else owner = 0;
                const uint32_t gcell = (l * b.h + (uint32_t)gy) * b.w + (uint32_t)gx;
                const uint64_t lc = ((uint64_t)l * f.wh + (uint32_t)(gy - wy0)) * f.ww + (uint32_t)(gx - wx0);
                if constexpr (ASYNC) {
                    if (owner < 5) lv[k] = __ldcg(lab + lc);  // the arena starts at +inf
                } else {
                    if (owner < 5 && s_vis[owner]) lv[k] = __ldcg(lab + lc);
                    else if (owner == 0 && gcell == f.src) lv[k] = 0;  // first visit of the source tile
                }
                if (b.flags) fv[k] = __ldg(b.flags + gcell);
            }
        }
#pragma unroll
        for (int k = 0; k < kStageUnroll; ++k) {
            const uint32_t i = i0 + k * blockDim.x;
            if (i >= nsm) continue;
            const uint32_t sx = i % SW, r = i / SW, sy = r % SH, l = r / SH;
            tile.lab[tile.li(l, sy, sx)] = lv[k];
            tile.fl[(l * SH + sy) * kFlPitch + sx] = fv[k];
            if (lv[k] != kInf && (!GD || tile.bound((uint32_t)(lv[k] >> 32), l, sy, sx) <= tile.ub)) {
                const bool row_in = sy >= 1 && sy <= TH, col_in = sx >= 1 && sx <= kTW;
                if (row_in) tile.rowd[l * TH + sy - 1] = 1;
                if (col_in) tile.cold[l * kTW + sx - 1] = 1;
                if (row_in && col_in) tile.stackd[(sy - 1) * kTW + sx - 1] = 1;
            }
        }
    }
    {
        cp_async_wait_all();  // the board words copied before the label loop
        __syncthreads();
        // this net's own directed prices (negotiation overrides) replace the
        // board's words before the step prices are formed
        if (OV && f.n_over && a.tover[f.tile_off + t]) {
            stage_overrides(b, f, tile.st, L, TH, tx0, ty0, tw, th);
            __syncthreads();
        }
        // Phase 2: every step price from the staged bytes (own pads and via
        // exemptions are the only global reads left).
        for (uint32_t i = tid; i < L * TH * kTW; i += blockDim.x) {
            const uint32_t x = i % kTW, r = i / kTW, y = r % TH, l = r / TH;
            const int gx = tx0 + (int)x, gy = ty0 + (int)y;
            uint32_t s0 = kMax, s1 = kMax, s2 = kMax, s3 = kMax, s4 = kMax, s5 = kMax;
            if (gx >= wx0 && gx < wx1 && gy < wy1) {
                const uint32_t gc = (l * b.h + (uint32_t)gy) * b.w + (uint32_t)gx;
                const uint8_t *flr = tile.fl + (l * SH + y + 1) * kFlPitch + x + 1;  // this cell
                const uint8_t fc = flr[0];
                const uint32_t cost = tile.st[tile.si(kFromBelow, l, y, x)];
                uint32_t ec;  // cell_enter on staged values
                if (fc & kTraceNode) ec = kMax;
                else if (cost != kMax) ec = cost;
                else ec = is_own_pad(gc) ? 1u : kMax;
                if (ec != kMax) {
                    const bool dir = b.directed != nullptr;
                    auto planar = [&](uint32_t base, uint8_t fp, uint8_t out_bit, uint8_t in_bit) -> uint32_t {
                        if (dir && base == kMax) return kMax;  // blocked directed edge
                        if ((fp & out_bit) | (fc & in_bit)) return kMax;
                        return capmul(base, ec);
                    };
                    if (gx > wx0) s0 = planar(tile.st[tile.si(kFromNegX, l, y, x)], flr[-1], kEdgePosX, kEdgeNegX);
                    if (gx + 1 < wx1) s1 = planar(tile.st[tile.si(kFromPosX, l, y, x)], flr[1], kEdgeNegX, kEdgePosX);
                    if (gy > wy0)
                        s2 = planar(tile.st[tile.si(kFromNegY, l, y, x)], flr[-(int)kFlPitch], kEdgePosY, kEdgeNegY);
                    if (gy + 1 < wy1)
                        s3 = planar(tile.st[tile.si(kFromPosY, l, y, x)], flr[kFlPitch], kEdgeNegY, kEdgePosY);
                    if (L > 1) {
                        const bool vc = via_blk(gc, fc);
                        if (l > 0 && ((b.via_mask >> (l - 1)) & 1u) && !vc) {
                            const uint8_t fq = flr[-(int)(SH * kFlPitch)];
                            if (!via_blk(gc - plane, fq)) s4 = capmul(__ldg(b.via_edge + l - 1), ec);
                        }
                        if (l + 1 < L && ((b.via_mask >> l) & 1u) && !vc) {
                            const uint8_t fq = flr[SH * kFlPitch];
                            if (!via_blk(gc + plane, fq)) s5 = capmul(__ldg(b.via_edge + l), ec);
                        }
                    }
                }
            }
            tile.st[tile.si(kFromNegX, l, y, x)] = s0;
            tile.st[tile.si(kFromPosX, l, y, x)] = s1;
            tile.st[tile.si(kFromNegY, l, y, x)] = s2;
            tile.st[tile.si(kFromPosY, l, y, x)] = s3;
            tile.st[tile.si(kFromBelow, l, y, x)] = s4;
            tile.st[tile.si(kFromAbove, l, y, x)] = s5;
        }
    }
    __syncthreads();

    // ---- relax to local convergence ---------------------------------
    // Queue form: a tile that a neighbour improved while this CTA held it is
    // continued here (up to kContinueLimit times): its halo ring is read again
    // and the sweeps resume on the staged tile, without a release, a queue
    // round trip and a full re-staging.  Each continuation counts as an
    // activation.
    const uint32_t sweep_limit = L * kTW * TH + 4;
    __shared__ uint32_t s_more;
    for (uint32_t cont = 0;; ++cont) {
        uint32_t sweep = 0;
        for (;;) {
            // the rounds form alternates the pass order between sweeps (fewer
            // sweeps on the one-activation tiles it runs); the queue form runs
            // columns first, where alternation costs sweeps
            bool ch;
            if constexpr (GD) {  // the target's own tile tightens its bound from sweep to sweep
                if (dst_here) tile.ub = min(tile.ub, (uint32_t)(tile.lab[dst_li] >> 32));
            }
            if constexpr (!ASYNC) ch = (sweep & 1) ? relax_tile_rev(tile) : relax_tile(tile);
            else ch = relax_tile_cols_first<TH, WHOLE>(tile);
            ++sweep;
            const int any = __syncthreads_or(ch ? 1 : 0);
            if (!any) break;
            if (sweep > sweep_limit) {
                if (tid == 0) atomicOr(&ctl->status, kStatusRoundLimit);
                break;
            }
        }

        if constexpr (GD) {
            if (dst_here) {
                tile.ub = min(tile.ub, (uint32_t)(tile.lab[dst_li] >> 32));
                if (tid == 0 && tile.ub < s_lim[0]) {  // held by this CTA alone: no other writer
                    s_lim[0] = tile.ub;
                    *(volatile uint32_t *)&a.goal[fi].ub = tile.ub;
                }
            }
        }

        // ---- write back and find neighbours this tile can improve -------
        u64 *labw = a.lab + f.lab_off;
        // the tile is held by this CTA alone (both schedules), so plain stores;
        // indices are split by the compile-time tile shape (cells past a ragged
        // window edge are skipped).  Only labels that fell are stored, unless the
        // arena holds nothing valid for this tile yet (first visit, rounds form).
        const bool all_labels = !ASYNC && !s_vis[0];
        for (uint32_t i = tid; i < L * TH * kTW; i += blockDim.x) {
            const uint32_t tx = i % kTW, r = i / kTW, ty = r % TH, l = r / TH;
            if (tx >= tw || ty >= th) continue;
            if (!all_labels && !((tile.fellw[l * TH + ty] >> tx) & 1u))
                continue;
            const uint64_t lc = ((uint64_t)l * f.wh + (uint32_t)(ty0 - wy0) + ty) * f.ww + (uint32_t)(tx0 - wx0 + (int)tx);
            labw[lc] = tile.lab[tile.li(l, ty + 1, tx + 1)];
        }
        // borders: 0 = left (-x), 1 = right (+x), 2 = top (-y), 3 = bottom (+y)
        const uint32_t nb = 2 * L * TH + 2 * L * kTW;
        for (uint32_t i = tid; i < nb; i += blockDim.x) {
            uint32_t side, l, k;
            if (i < 2 * L * TH) {
                side = i >= L * TH;
                const uint32_t r = i - side * L * TH;
                l = r / TH;
                k = r % TH;
                if (k >= th) continue;
            } else {
                const uint32_t j = i - 2 * L * TH;
                const uint32_t hi = j >= L * kTW;
                side = 2 + hi;
                const uint32_t r = j - hi * L * kTW;
                l = r / kTW;
                k = r % kTW;
                if (k >= tw) continue;
            }
            bool exists;
            uint32_t bsx, bsy, nsx, nsy, dir;
            uint8_t out_bit, in_bit;
            if (side == 0) {
                exists = txi > 0;
                bsx = 1; bsy = k + 1; nsx = 0; nsy = bsy;
                dir = 2; out_bit = kEdgeNegX; in_bit = kEdgePosX;
            } else if (side == 1) {
                exists = txi + 1 < ntx;
                bsx = tw; bsy = k + 1; nsx = tw + 1; nsy = bsy;
                dir = 1; out_bit = kEdgePosX; in_bit = kEdgeNegX;
            } else if (side == 2) {
                exists = tyi > 0;
                bsx = k + 1; bsy = 1; nsx = bsx; nsy = 0;
                dir = 3; out_bit = kEdgeNegY; in_bit = kEdgePosY;
            } else {
                exists = tyi + 1 < nty;
                bsx = k + 1; bsy = th; nsx = bsx; nsy = th + 1;
                dir = 0; out_bit = kEdgePosY; in_bit = kEdgeNegY;
            }
            if (!exists || s_push[side]) continue;
            const u64 lb = tile.lab[tile.li(l, bsy, bsx)];
            if (lb == kInf) continue;
            // the neighbour tile holds cells this net prices with its own overrides
            bool nb_over = false;
            if constexpr (OV) {
                const uint32_t u = side == 0 ? t - 1 : side == 1 ? t + 1 : side == 2 ? t - ntx : t + ntx;
                nb_over = f.n_over && a.tover[f.tile_off + u];
            }
            const uint32_t gn = (l * b.h + (uint32_t)(ty0 + (int)nsy - 1)) * b.w + (uint32_t)(tx0 + (int)nsx - 1);
            const uint8_t fb = tile.fl[(l * SH + bsy) * kFlPitch + bsx];
            const uint8_t fn = tile.fl[(l * SH + nsy) * kFlPitch + nsx];
            // the neighbour's enter cost and in-price, both loaded before either is used
            const uint32_t gx_n = (uint32_t)(tx0 + (int)nsx - 1), gy_n = (uint32_t)(ty0 + (int)nsy - 1);
            const uint32_t cn = __ldg(b.cost + gn);
            uint32_t base;
            if (b.directed)
                base = nb_over ? field_directed(b, f, gn, (int)dir)
                               : __ldg(reinterpret_cast<const uint32_t *>(b.directed + gn) + dir);
            else if (side == 0) base = __ldg(b.x_edge + gx_n);
            else if (side == 1) base = __ldg(b.x_edge + gx_n - 1);
            else if (side == 2) base = __ldg(b.y_edge + gy_n);
            else base = __ldg(b.y_edge + gy_n - 1);
            uint32_t en = kMax;  // cell_enter of the neighbour
            if (!(fn & kTraceNode)) en = cn != kMax ? cn : (is_own_pad(gn) ? 1u : kMax);
            if (en == kMax) continue;
            uint32_t step = kMax;  // planar_step_g on the loaded values
            if (!((fb & out_bit) | (fn & in_bit)) && !(b.directed && base == kMax)) step = capmul(base, en);
            const u64 cand = ext2(lb, step, 1);
            if (cand < tile.lab[tile.li(l, nsy, nsx)]) {
                if constexpr (GD) {
                    const uint32_t fv = tile.bound((uint32_t)(cand >> 32), l, nsy, nsx);
                    if (fv > tile.ub) continue;
                    if (fv > s_lim[1]) {
                        atomicMin(&s_park[side], fv);
                        continue;
                    }
                }
                s_push[side] = 1;
            }
        }
        __syncthreads();
        if (tid < 5) {
            __threadfence();  // labels before the visited flag and the queue entries
            if (tid == 4) {
                if constexpr (ASYNC) {
                    // the work counters are per CTA (s_cnt), added to the launch's
                    // every kCountBatch activations and when the CTA exits, so this
                    // thread makes no round trip to L2 here (kLeaveLaunch: the CTA
                    // leaves a failed launch after this item)
                    s_cnt[1] += sweep;
                    if (++s_cnt[0] == kCountBatch) {
                        s_cnt[0] = count_flush(a, s_cnt[0], s_cnt[1]) ? 0 : kLeaveLaunch;
                        s_cnt[1] = 0;
                    }
                } else {
                    if (!s_vis[0]) atomicExch(a.tvisit + f.tile_off + t, 1u);
                    atomicAdd(&ctl->activations, 1ull);
                    atomicAdd(&ctl->sweeps, (unsigned long long)sweep);
                }
            } else if (s_push[tid]) {
                const uint32_t u = tid == 0 ? t - 1 : tid == 1 ? t + 1 : tid == 2 ? t - ntx : t + ntx;
                if constexpr (ASYNC) {
                    async_push(a, fi, f.tile_off, u, live);
                } else {
                    const uint32_t want = round + 2;  // stamp s = queued for round s-1
                    if (atomicMax(a.tstamp + f.tile_off + u, want) < want) {
                        const uint32_t nxt = (round + 1) % 3;
                        const uint32_t idx = atomicAdd(&ctl->count[nxt], 1u);
                        if (idx < cap) {
                            a.lists[(size_t)nxt * cap + idx] = ((u64)fi << 32) | u;
                        } else {
                            atomicOr(&ctl->status, kStatusQueueOverflow);
                        }
                    }
                }
            } else if (GD && s_park[tid] != kMax) {
                const uint32_t u = tid == 0 ? t - 1 : tid == 1 ? t + 1 : tid == 2 ? t - ntx : t + ntx;
                atomicMin(a.tpark + f.tile_off + u, s_park[tid]);
                __threadfence();  // before this item leaves the field's count
            }
        }
        __syncthreads();
        if constexpr (!ASYNC) {
            break;
        } else {
            if (tid == 0) {
                // its own pushes are counted (the barrier above): release the tile
                // with one atomic, or, if a neighbour improved it meanwhile, hold it
                // again and continue, or queue it once more past the limit
                __threadfence();
                uint32_t *stw = a.tstamp + f.tile_off + t;
                s_more = 0;
                if (atomicCAS(stw, kTileHeld, kTileIdle) != kTileHeld) {  // held and dirty
                    if (cont + 1 < kContinueLimit) {
                        atomicExch(stw, kTileHeld);
                        s_more = 1;
                    } else {
                        atomicExch(stw, kTileQueued);
                        async_enqueue(a, fi, t, live);
                    }
                }
                if (!s_more) {  // this item leaves the in-flight count
                    const uint32_t left = atomicSub(live, 1u) - 1u;
                    if (left == 0) s_more = 2;
                }
            }
            __syncthreads();
            if (s_more != 1) {
                last = s_more == 2;
                break;
            }
            __threadfence();  // the neighbours' labels were written before they marked this tile
            if (tid < 4) s_push[tid] = 0;
            if (GD && tid < 4) s_park[tid] = kMax;
            for (uint32_t i = tid; i < fell_words; i += blockDim.x) tile.fellw[i] = 0;
            // the halo ring again: an improved cell marks the line that ends at it
            const uint32_t nr = 2 * L * TH + 2 * L * kTW;
            for (uint32_t i = tid; i < nr; i += blockDim.x) {
                uint32_t l, sx, sy;
                bool row;
                if (i < 2 * L * TH) {
                    const uint32_t side = i >= L * TH, r = i - side * L * TH;
                    l = r / TH;
                    sy = r % TH + 1;
                    if (sy > th || (side ? txi + 1 >= ntx : txi == 0)) continue;
                    sx = side ? tw + 1 : 0;
                    row = true;
                } else {
                    const uint32_t k = i - 2 * L * TH, side = k >= L * kTW, r = k - side * L * kTW;
                    l = r / kTW;
                    sx = r % kTW + 1;
                    if (sx > tw || (side ? tyi + 1 >= nty : tyi == 0)) continue;
                    sy = side ? th + 1 : 0;
                    row = false;
                }
                const int gx = tx0 + (int)sx - 1, gy = ty0 + (int)sy - 1;
                if (gx < wx0) continue;
                const u64 v = __ldcg(lab + ((uint64_t)l * f.wh + (uint32_t)(gy - wy0)) * f.ww + (uint32_t)(gx - wx0));
                u64 &cur = tile.lab[tile.li(l, sy, sx)];
                if (v < cur) {
                    cur = v;
                    if (GD && tile.bound((uint32_t)(v >> 32), l, sy, sx) > tile.ub) continue;
                    if (row) tile.rowd[l * TH + sy - 1] = 1;
                    else tile.cold[l * kTW + sx - 1] = 1;
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();  // (queue form: the tile was released, or queued again, inside the loop)
    return last;
}

}  // namespace mrc
