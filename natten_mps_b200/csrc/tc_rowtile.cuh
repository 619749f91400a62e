// Row tiles of the persistent tensor-core kernels (fused backward, both sides; double-buffered fused forward):
// geometry of one work item (128 rows of one (batch, head) and the box of columns their windows or inverse
// windows cover) and the tables a helper warp publishes one tile ahead.
#pragma once
#include "tc_plan.cuh"

namespace natten {
namespace rowtile {

using namespace tc;
using namespace tcplan;

constexpr int kCols = 64;                   // columns per chunk
constexpr int kAxisEntries = 130;           // entries of a tile's axis table: tile[0] + tile[1] + tile[2] <= 128 + 1 + 1

__device__ __forceinline__ int ws1(int p, int L, int K) { return window_start(p, L, K, 1); }

// Geometry of one work item: a tile of 128 rows (queries | keys) of one (batch, head).
struct BwdTile {
    int b, hy;                 // batch; head of the row tensors (query head | kv head)
    int rg[3], origin[3], Lp[3], boxlo[3], nc[3];
    int nchunks;               // chunks of the column box
    int nbox, total;           // column passes: box chunks x query heads of the group, then additional tokens
    bool active;
};

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

template <bool kKeySide>
__device__ __forceinline__ void bwd_tile_setup(const TcParams& P, unsigned work, BwdTile& T)
{
    const unsigned hb = work / P.per_head;
    const unsigned bx = work - hb * P.per_head;
    const unsigned H = (unsigned)(kKeySide ? P.Hkv : P.Hq >> P.pack_log);
    T.b = (int)(hb / H);
    T.hy = (int)(hb - (unsigned)T.b * H) << (kKeySide ? 0 : P.pack_log);
    T.active = cta_geometry(P, bx, T.b, T.rg, T.origin, T.Lp);
    T.nchunks = 1;
    if (T.active) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int last = T.origin[a] + P.tile[a] - 1 < T.Lp[a] - 1 ? T.origin[a] + P.tile[a] - 1 : T.Lp[a] - 1;
            int hi;
            if (kKeySide) {
                int t;
                inverse_range(T.origin[a], T.Lp[a], P.K[a], P.causal[a], T.boxlo[a], t, /*exact=*/false);
                inverse_range(last, T.Lp[a], P.K[a], P.causal[a], t, hi, /*exact=*/false);
            } else {
                T.boxlo[a] = P.causal[a] ? T.origin[a] - (P.K[a] - 1) : ws1(T.origin[a], T.Lp[a], P.K[a]);
                hi = P.causal[a] ? last : ws1(last, T.Lp[a], P.K[a]) + P.K[a] - 1;
            }
            T.nc[a] = chunks_along(P, a, hi - T.boxlo[a] + 1);
            T.nchunks *= T.nc[a];
        }
    }
    T.nbox = T.nchunks * (kKeySide ? P.group : 1);
    T.total = T.nbox + (kKeySide ? 0 : ((P.n_extra + kCols - 1) >> 6));
}

// The work item into the head of a slot, by one warp (what bwd_tile_setup gives, an axis per lane); returns whether it is active.
// rows16: chunks of 16-column rows.
template <bool kKeySide>
__device__ __forceinline__ bool publish_tile(const TcParams& P, unsigned work, bool rows16, int lane, TileHead* H)
{
    const unsigned hb = work / P.per_head, heads = (unsigned)(kKeySide ? P.Hkv : P.Hq >> P.pack_log);
    const int b = (int)(hb / heads), hy = (int)(hb - (unsigned)b * heads) << (kKeySide ? 0 : P.pack_log), a = lane < 2 ? lane : 2;
    int rg, origin, Lp;
    if (!__all_sync(0xffffffffu, lane_geometry(P, work - hb * P.per_head, b, a, rg, origin, Lp))) return false;
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
