// Tile geometry of the fused forward kernels: which queries a work item holds, the key box of
// their neighbourhoods and how many chunks it takes; per-row windows inside that box.
#pragma once
#include "tc_plan.cuh"

namespace natten {
namespace fwdgeom {

using namespace tc;
using namespace tcplan;

// Geometry of one work item (a tile of 128 queries of one (batch, head)).
struct FwdTile {
    int b, h, hk;
    int rg[3], origin[3], Lp[3], lo[3], nc[3], x0[3], sx[3], nq[3], nqf[3];
    int nnb, nch;          // nch == 0 in a published header: no more tiles
    int mapped;            // the row maps of the tables are valid
};

// Walks the work items of a lane (w0, w0 + step, ...) without divisions: tile index inside the
// (batch, head), head and batch are advanced incrementally.
struct Cursor {
    unsigned w, bx, dq, dr;
    int h, b;
    __device__ __forceinline__ void init(const TcParams& P, unsigned w0, unsigned step)
    {
        w = w0;
        const unsigned hb = w0 / P.per_head;
        bx = w0 - hb * P.per_head;
        const unsigned heads = (unsigned)P.Hq >> P.pack_log;     // h counts groups of 1 << pack_log heads
        b = (int)(hb / heads);
        h = (int)(hb - (unsigned)b * heads);
        dq = step / P.per_head;
        dr = step - dq * P.per_head;
    }
    __device__ __forceinline__ void advance(const TcParams& P, unsigned step)
    {
        w += step;
        bx += dr;
        int dh = (int)dq;
        if (bx >= P.per_head) { bx -= P.per_head; ++dh; }
        h += dh;
        while (h >= P.Hq >> P.pack_log) { h -= P.Hq >> P.pack_log; ++b; }
    }
};

// Rows of the cursor's tile that exist in the output, by one warp: f(output row) for each.  (Position x0 + sx * i of the sub-grid is
// query i of an axis; a dilation group without queries has x0 < 0.)
template <typename F>
__device__ __forceinline__ void for_each_row(const TcParams& P, const Cursor& cur, int lane, F&& f)
{
    int rg[3], origin[3];
    tile_of_block(P, cur.bx, rg, origin);
#pragma unroll 1
    for (int r = lane; r < kTileRows; r += 32) {
        int qi[3];
        row_offsets(P, r, qi);
        bool in_tensor = true;
        long long oflat = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int x0 = P.qx0[a][rg[a]], pa = rg[a] + P.dil[a] * (x0 + P.qstep[a] * (origin[a] + qi[a]));
            in_tensor = in_tensor && x0 >= 0 && pa < P.L[a];
            oflat = oflat * P.O[a] + (P.st[a] == 1 ? pa : pa / P.st[a]);
        }
        if (in_tensor) f(((long long)cur.b * P.otot + oflat) * P.Hq + (cur.h << P.pack_log) + (r & ((1 << P.pack_log) - 1)));
    }
}

// What a softmax thread needs to know about its row is separable: along every axis the query's coordinate alone decides its
// position, whether it exists and its window.  The geometry warp writes one entry per (axis, coordinate of the tile) a tile ahead,
// tile[0] + tile[1] + tile[2] of them instead of 128 rows x 3 axes.  A slot: FwdTile, row maps, axis entries.
constexpr int kMapOff = 160, kEntOff = kMapOff + 8 * kTileRows, kTabBytes = kEntOff + 16 * (kTileRows + 2);
static_assert(sizeof(FwdTile) <= kMapOff, "no room for the tile in front of its tables");

// The cursor's work item (tile bx of (batch, head)) into the head of a slot, by one warp, an axis per lane; returns whether it holds a
// query of the sample.  origin[] counts queries of the dilation group; query i of an axis sits at sub-grid index x0 + sx * i (every
// index when the output stride is 1).  rows16: chunks of 16-column rows.
__device__ __forceinline__ bool publish_tile(const TcParams& P, const Cursor& cur, int chunk_log, bool rows16, int lane, FwdTile* H)
{
    const int a = lane < 2 ? lane : 2;
    int rg, origin, Lp, nq, nqf, lo = 0, nc = 1;
    bool active = lane_geometry(P, cur.bx, cur.b, a, rg, origin, Lp);
    const int sx = P.qstep[a];
    int x0 = P.qx0[a][rg];
    const int lpf = (int)fast_div((unsigned)(P.L[a] - rg + P.dil[a] - 1), P.dil_mul[a]);
    if (x0 < 0) {
        nq = 0; nqf = 0; x0 = 0;
    } else if (sx == 1) {
        nq = Lp;
        nqf = rg < P.L[a] ? lpf : 0;
    } else {
        nq = x0 < Lp ? (Lp - x0 + sx - 1) / sx : 0;
        nqf = x0 < lpf ? (lpf - x0 + sx - 1) / sx : 0;
    }
    active = __all_sync(0xffffffffu, active && origin < nq);
    if (!active) return false;
    {
        const int lastq = origin + P.tile[a] - 1 < nq - 1 ? origin + P.tile[a] - 1 : nq - 1;
        const int xf = x0 + sx * origin, xl = x0 + sx * lastq;
        lo = P.causal[a] ? xf - (P.K[a] - 1) : window_start(xf, Lp, P.K[a], 1);
        const int hi = P.causal[a] ? xl : window_start(xl, Lp, P.K[a], 1) + P.K[a] - 1;
        nc = chunks_along(P, a, hi - lo + 1);
    }
    const int nnb = __shfl_sync(0xffffffffu, nc, 0) * __shfl_sync(0xffffffffu, nc, 1) * __shfl_sync(0xffffffffu, nc, 2);
    if (lane < 3) {
        H->rg[lane] = rg; H->origin[lane] = origin; H->Lp[lane] = Lp; H->lo[lane] = lo; H->nc[lane] = nc;
        H->x0[lane] = x0; H->sx[lane] = sx; H->nq[lane] = nq; H->nqf[lane] = nqf;
    }
    if (lane == 2) {
        H->b = cur.b;
        const int h = cur.h << P.pack_log;
        H->h = h;
        H->hk = (int)fast_div((unsigned)h, P.group_mul);
        H->nnb = nnb;
        H->nch = nnb + ((P.n_extra + (1 << chunk_log) - 1) >> chunk_log);    // then the additional tokens, one chunk at a time
        H->mapped = rows16 && nc == 1 && nnb <= 16;
    }
    return true;
}

// The slot's tables, by one warp.  An entry is for a query coordinate of the tile along an axis: window [f, e) in the box, output
// position, flags (bit 0 query of the sample, bit 1 position of the tensor).
// `mapped`: chunks of 16-column rows, one chunk along the innermost axis and at most 16 chunks in all.  Then which of
// a chunk's four rows lie in a query's window depends on its two outer coordinates: a map per pair of them, four bits a chunk
// (every row of the window lands in one row of one chunk), and the window's columns as bits beside the flags.
__device__ __forceinline__ void write_tables(const TcParams& P, int lane, uint8_t* slot)
{
    const FwdTile* T = reinterpret_cast<const FwdTile*>(slot);
    int4* ent = reinterpret_cast<int4*>(slot + kEntOff);
    const int t0 = P.tile[0], t01 = t0 + P.tile[1], all = t01 + P.tile[2];
    const bool mapped = T->mapped;
#pragma unroll 1
    for (int i = lane; i < all; i += 32) {
        const int a = i < t0 ? 0 : i < t01 ? 1 : 2;
        const int qa = T->origin[a] + i - (a == 0 ? 0 : a == 1 ? t0 : t01), xq = T->x0[a] + T->sx[a] * qa, pa = T->rg[a] + P.dil[a] * xq;
        const int lo = T->lo[a], Lp = T->Lp[a], K = P.K[a], st = P.st[a];
        const int first = P.causal[a] ? xq - (K - 1) : window_start(xq, Lp, K, 1);
        int4 en = make_int4((first > 0 ? first : 0) - lo, (first + K < Lp ? first + K : Lp) - lo, st == 1 ? pa : pa / st,
                            (qa < T->nq[a] ? 1 : 0) | (qa < T->nqf[a] ? 2 : 0));
        if (a == 2 && mapped) {
            int jl, jh;
            chunk_range(P, 2, 0, en.x, en.y, jl, jh);
            if (jh > jl) en.w |= (low_bits(jh) & ~low_bits(jl)) << 16;
        }
        ent[i] = en;
    }
    __syncwarp();
    if (!mapped) return;
    unsigned long long* map = reinterpret_cast<unsigned long long*>(slot + kMapOff);
    for (int r = lane; r < t0 * P.tile[1]; r += 32) {
        const int4 e0 = ent[r >> P.tile1_log], e1 = ent[t0 + (r & (P.tile[1] - 1))];
        map[r] = (e0.w & e1.w & 1) ? row_map(P, T->nc[1], e0.x, e0.y, e1.x, e1.y) : 0ull;
    }
}

// A thread's row from the tables: its output row, whether it is a query of the sample / a row of the tensor, its window as a
// box-relative range [f, e) per axis, and the maps.
__device__ __forceinline__ long long row_from_tables(const TcParams& P, const uint8_t* slot, int row, int (&f)[3], int (&e)[3],
                                                     bool& valid_q, bool& in_tensor, unsigned long long& rowmap, uint32_t& colbits)
{
    const FwdTile* T = reinterpret_cast<const FwdTile*>(slot);
    const int4* ent = reinterpret_cast<const int4*>(slot + kEntOff);
    const int head = row & ((1 << P.pack_log) - 1), pos = row >> P.pack_log, r01 = pos >> P.tile2_log;
    const int4 e0 = ent[r01 >> P.tile1_log], e1 = ent[P.tile[0] + (r01 & (P.tile[1] - 1))],
               e2 = ent[P.tile[0] + P.tile[1] + (pos & (P.tile[2] - 1))];
    const int flags = e0.w & e1.w & e2.w;
    valid_q = flags & 1;
    in_tensor = flags & 2;
    f[0] = e0.x; f[1] = e1.x; f[2] = e2.x;
    e[0] = valid_q ? e0.y : e0.x;
    e[1] = valid_q ? e1.y : e1.x;
    e[2] = valid_q ? e2.y : e2.x;
    rowmap = T->mapped ? reinterpret_cast<const unsigned long long*>(slot + kMapOff)[r01] : 0ull;
    colbits = T->mapped && valid_q ? (uint32_t)e2.w >> 16 : 0u;
    const long long oflat = ((long long)e0.z * P.O[1] + e1.z) * P.O[2] + e2.z;
    return ((long long)T->b * P.otot + oflat) * P.Hq + T->h + head;
}

} // namespace fwdgeom
} // namespace natten
