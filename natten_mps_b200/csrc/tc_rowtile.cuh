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
    const unsigned H = (unsigned)(kKeySide ? P.Hkv : P.Hq);
    T.b = (int)(hb / H);
    T.hy = (int)(hb - (unsigned)T.b * H);
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

// Entry of the tile's row coordinate i along axis a.
template <bool kKeySide>
__device__ __forceinline__ AxisEntry axis_entry(const TcParams& P, const BwdTile& X, int a, int i)
{
    const int xa = X.origin[a] + i, pa = X.rg[a] + P.dil[a] * xa;
    AxisEntry en;
    en.z = pa;
    en.w = (xa < X.Lp[a] ? 1 : 0) | (pa < P.L[a] ? 2 : 0);
    if (kKeySide) {
        int qlo, qhi;
        inverse_range(xa, X.Lp[a], P.K[a], P.causal[a], qlo, qhi);
        en.x = qlo - X.boxlo[a];
        en.y = qhi + 1 - X.boxlo[a];
    } else {
        const int first = P.causal[a] ? xa - (P.K[a] - 1) : ws1(xa, X.Lp[a], P.K[a]);
        en.x = (first > 0 ? first : 0) - X.boxlo[a];
        en.y = (first + P.K[a] < X.Lp[a] ? first + P.K[a] : X.Lp[a]) - X.boxlo[a];
    }
    return en;
}

// One warp writes a tile's tables.  mapped: chunks of 16-column rows, one along the innermost axis, at most 16 in the box.  Then
// which of a chunk's four rows lie in a row's range depends on its two outer coordinates: a map per pair of them, four bits a chunk.
template <bool kKeySide>
__device__ __forceinline__ void write_tables(const TcParams& P, const BwdTile& X, bool mapped, int lane, uint8_t* slot)
{
    AxisEntry* ent = reinterpret_cast<AxisEntry*>(slot + kHeadBytes + kMapBytes);
    int base = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int i = lane; i < P.tile[a]; i += 32) ent[base + i] = axis_entry<kKeySide>(P, X, a, i);
        base += P.tile[a];
    }
    if (!mapped) return;
    unsigned long long* map = reinterpret_cast<unsigned long long*>(slot + kHeadBytes);
    for (int r = lane; r < P.tile[0] * P.tile[1]; r += 32) {
        const AxisEntry e0 = axis_entry<kKeySide>(P, X, 0, r >> P.tile1_log), e1 = axis_entry<kKeySide>(P, X, 1, r & (P.tile[1] - 1));
        map[r] = (e0.w & e1.w & 1) ? row_map(P, X.nc[1], e0.x, e0.y, e1.x, e1.y) : 0ull;
    }
}

} // namespace rowtile
} // namespace natten
