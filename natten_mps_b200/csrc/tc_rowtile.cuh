// Row tiles of the fused backward on tensor cores, both sides: geometry of one work item (128 rows of one
// (batch, head) and the box of columns their windows or inverse windows cover) and the tables that the geometry
// warp publishes one tile ahead.
#pragma once
#include "tc_plan.cuh"

namespace natten {
namespace rowtile {

using namespace tc;
using namespace tcplan;

constexpr int kCols = 64;                   // columns per chunk
constexpr int kAxisEntries = 130;           // entries of a tile's axis table: tile[0] + tile[1] + tile[2] <= 128 + 1 + 1

__device__ __forceinline__ int ws1(int p, int L, int K) { return window_start(p, L, K, 1); }

// What a compute thread needs to know about its row of a tile is separable: along every axis the row's
// coordinate alone decides its position in the tensor, whether it exists, and its valid column range.  The
// geometry warp writes one entry per (axis, coordinate of the tile) one tile ahead, tile[0] + tile[1] + tile[2]
// entries instead of 128 rows x 3 axes; a compute thread combines the three entries of its row.
// x, y: valid column range [f, e) along the axis, relative to the column box; z: position along the axis in the tensor;
// w: bit 0 inside the (sub-grid of the) sample, bit 1 inside the tensor.
using AxisEntry = int4;
struct TileHead {
    int total, nbox, nc[3];            // total == 0: no more tiles
    int nchunks, boxlo[3], Lp[3];      // chunks of the column box, its origin, sub-grid extents
    int b, hy;                         // batch and head of the rows
    int rg[3], origin[3];              // dilation residues and origin of the row tile
    int mapped;                        // the row maps are valid
};
// A slot: head, row maps, axis entries.
constexpr int kHeadBytes = 96, kMapBytes = 8 * kTileRows, kTabBytes = kHeadBytes + kMapBytes + 16 * kAxisEntries;
static_assert(sizeof(TileHead) <= kHeadBytes, "the tile head has 96 bytes in front of the tables");

// Batch and (first) head of a work item's rows, and its block index among the tiles of that head.
template <bool kKeySide>
__device__ __forceinline__ unsigned split_work(const TcParams& P, unsigned work, int& b, int& hy)
{
    const unsigned hb = work / P.per_head, heads = (unsigned)(kKeySide ? P.Hkv : P.Hq >> P.pack_log);
    b = (int)(hb / heads);
    hy = (int)(hb - (unsigned)b * heads) << (kKeySide ? 0 : P.pack_log);
    return work - hb * P.per_head;
}

// The work item into the head of a slot, by one warp, an axis per lane; returns whether it holds a row of the sample.
// rows16: chunks of 16-column rows.
template <bool kKeySide>
__device__ __forceinline__ bool publish_tile(const TcParams& P, unsigned work, bool rows16, int lane, TileHead* H)
{
    int b, hy, rg, origin, Lp;
    const unsigned bx = split_work<kKeySide>(P, work, b, hy);
    const int a = lane < 2 ? lane : 2;
    if (!__all_sync(0xffffffffu, lane_geometry(P, bx, b, a, rg, origin, Lp))) return false;
    const int last = origin + P.tile[a] - 1 < Lp - 1 ? origin + P.tile[a] - 1 : Lp - 1;
    int boxlo, hi;
    if (kKeySide) {
        int t;
        inverse_range(origin, Lp, P.K[a], P.causal[a], boxlo, t, /*exact=*/false);
        inverse_range(last, Lp, P.K[a], P.causal[a], t, hi, /*exact=*/false);
    } else {
        boxlo = P.causal[a] ? origin - (P.K[a] - 1) : ws1(origin, Lp, P.K[a]);
        hi = P.causal[a] ? last : ws1(last, Lp, P.K[a]) + P.K[a] - 1;
    }
    const int nc = chunks_along(P, a, hi - boxlo + 1);
    const int nchunks = __shfl_sync(0xffffffffu, nc, 0) * __shfl_sync(0xffffffffu, nc, 1) * __shfl_sync(0xffffffffu, nc, 2);
    if (lane < 3) {
        H->nc[lane] = nc; H->boxlo[lane] = boxlo; H->Lp[lane] = Lp; H->rg[lane] = rg; H->origin[lane] = origin;
    }
    if (lane == 2) {
        H->b = b;
        H->hy = hy;
        H->nchunks = nchunks;
        H->nbox = nchunks * (kKeySide ? P.group : 1);
        H->total = H->nbox + (kKeySide ? 0 : ((P.n_extra + kCols - 1) >> 6));
        H->mapped = rows16 && nc == 1 && nchunks <= 16;
    }
    return true;
}

// The slot's tables, by one warp.  mapped: chunks of 16-column rows, one along the innermost axis, at most 16 in the box.  Then
// which of a chunk's four rows lie in a row's range depends on its two outer coordinates: a map per pair of them, four bits a chunk.
template <bool kKeySide>
__device__ __forceinline__ void write_tables(const TcParams& P, int lane, uint8_t* slot)
{
    const TileHead* H = reinterpret_cast<const TileHead*>(slot);
    AxisEntry* ent = reinterpret_cast<AxisEntry*>(slot + kHeadBytes + kMapBytes);
    const int t0 = P.tile[0], t01 = t0 + P.tile[1], all = t01 + P.tile[2];
#pragma unroll 1
    for (int i = lane; i < all; i += 32) {
        const int a = i < t0 ? 0 : i < t01 ? 1 : 2;
        const int xa = H->origin[a] + i - (a == 0 ? 0 : a == 1 ? t0 : t01), Lp = H->Lp[a], lo = H->boxlo[a], K = P.K[a];
        AxisEntry en;
        en.z = H->rg[a] + P.dil[a] * xa;
        en.w = (xa < Lp ? 1 : 0) | (en.z < P.L[a] ? 2 : 0);
        if (kKeySide) {
            int qlo, qhi;
            inverse_range(xa, Lp, K, P.causal[a], qlo, qhi);
            en.x = qlo - lo;
            en.y = qhi + 1 - lo;
        } else {
            const int first = P.causal[a] ? xa - (K - 1) : ws1(xa, Lp, K);
            en.x = (first > 0 ? first : 0) - lo;
            en.y = (first + K < Lp ? first + K : Lp) - lo;
        }
        ent[i] = en;
    }
    __syncwarp();
    if (!H->mapped) return;
    unsigned long long* map = reinterpret_cast<unsigned long long*>(slot + kHeadBytes);
    for (int r = lane; r < t0 * P.tile[1]; r += 32) {
        const AxisEntry e0 = ent[r >> P.tile1_log], e1 = ent[t0 + (r & (P.tile[1] - 1))];
        map[r] = (e0.w & e1.w & 1) ? row_map(P, H->nc[1], e0.x, e0.y, e1.x, e1.y) : 0ull;
    }
}

} // namespace rowtile
} // namespace natten
