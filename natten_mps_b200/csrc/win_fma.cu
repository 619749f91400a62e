// Window kernels in full fp32 arithmetic: fused attention for float32 tensors and the split operators for every type
// whose head dim the tensor-core kernels do not take (sums always in fp32; 16-bit tensors are widened when they are
// staged).
//
// Bound: the multiply-adds and the shared-memory reads that feed them.  A warp of the general SIMT kernels reads a whole
// row from memory for every (query, key) pair; here four queries share every key row that is read, from shared memory:
//   * a query (or key) row is spread over LPQ = D / 8 lanes, 8 channels each; a group of LPQ lanes holds FOUR rows that
//     are neighbours along a1 (rank 1: along a2), 32 / LPQ groups sit next to each other along a2;
//   * the column box of the CTA's rows is staged in shared memory in chunks, fp32, 16-byte pieces swizzled so that the
//     eight lanes of a phase touch different banks;
//   * per column a lane reads its 8 channels (two 16-byte reads), multiplies them with its four rows (packed fp32 pairs),
//     the four partial sums are reduced over the group so that lane i ends up with row i's (3 shuffles for 4 lanes), it
//     alone does the scalar work of that row (mask, exponential), and four shuffles hand the results back.
// A pass over the columns of K = 7 x 7 costs 23 shared-memory cycles for 32 pairs of which 70 % are needed.
//
// Measured, 56 x 56, 7 x 7, 4 heads of 32, batch 4, against the general SIMT kernels: float32 forward 31 us (185), dQ 37 (236),
// dK and dV 65 (304); split operators in bf16: scores 24 (93), apply 24 (93), gather 30 (115); in float32: 25 (96), 23 (469),
// 28 (152).
// What bounds them there: too few warps.  448 CTAs have 444 (forward, dQ), 296 (dK and dV, 245 to 255 registers) or 592 (split)
// places, 7 to 12 warps on an SM.  Schedulers issue in 47, 43, 38 % of the active cycles (forward, dQ, dK and dV) and in 49, 38,
// 39 % (scores, apply, gather); the largest stalls are the latency of dependent instructions and the barriers around a chunk, whose
// loads nothing overlaps, in apply and gather that of the weights.  DRAM is at 3 to 9 %.  The weights are
// half of the gather: 32 lanes read 32 sectors, which the few KB of L1 beside the staged columns do not keep.
//
// Rows are queries and columns keys, or the other way round (key side: dK, dV; columns = the queries that attend to a key,
// a contiguous range per axis).  Fixed order of summation everywhere, no atomics.
#include "simt_kernels.cuh"

#include "tc_kernels.cuh"
#include "tc_plan.cuh"

#include <algorithm>
#include <cfloat>
#include <type_traits>

namespace natten {
namespace {

using tcplan::fast_div;
using tcplan::fast_exp2;
using tcplan::fma2;
using tcplan::hi_of;
using tcplan::inverse_range;
using tcplan::kernel_axis_ok;
using tcplan::lo_of;
using tcplan::mul2;
using tcplan::pack2;

constexpr int kWarpsF = 4;
constexpr int kThreadsF = 32 * kWarpsF;
// Pairs of weights a lane fetches ahead.  With more the gather spills more at the 128 registers that four CTAs leave a thread: 56 x 56, 7 x 7,
// head dim 32, bf16, two gathers 61.4 us with 2, 71.5 with 4, 84 with 8 (apply 49.1, 49.8, 53.1); three CTAs with 7: 94.7 and 59.6.
// With 4 in nine shapes of ranks 1 to 3 (windows of 27 to 255, head dims 32 to 128, float32 and bf16): gathers 4 to 28 % slower, applies
// 1 to 9 % (two of 36 faster: head dim 32 in float32, 9 x 9 on 96 x 100 2 %, window 255 of 4097 4 %).
constexpr int kAheadF = 2;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

// A tensor as the kernels see it: element strides of batch, token, head.
struct TensorF {
    const void* p;
    long long bs, ts, hs;
};

struct FmaParams {
    int L[3], K[3], dil[3], causal[3];
    int tile1, tile2, ww;                // rows of a CTA along a1 and a2; warps along a2 (the others along a1)
    int ntile[3];                        // CTA tiles per axis and dilation group
    int chunk_rows, chunk_cols;          // columns staged at a time
    int rank, B, Hq, Hkv, group;
    long long ltot;
    int ktot;
    float scale, scale_log2;
    TensorF row1, row2, col1, col2;      // row tensors (queries | keys), column tensors (keys | queries)
};

template <bool kKeySide>
__device__ __forceinline__ void range_of(const FmaParams& P, int a, int x, int Lp, int& f, int& e, bool exact = true)
{
    if (kKeySide) {
        int lo, hi;
        inverse_range(x, Lp, P.K[a], P.causal[a], lo, hi, exact);
        f = lo;
        e = hi + 1;
    } else {
        const int first = P.causal[a] ? x - (P.K[a] - 1) : window_start(x, Lp, P.K[a], 1);
        f = first > 0 ? first : 0;
        e = first + P.K[a] < Lp ? first + P.K[a] : Lp;
    }
}

// A CTA's rows and column box.
struct TileF {
    int rg[3], o[3], Lp[3], lo[3], n[3];
};
template <bool kKeySide>
__device__ __forceinline__ bool tile_of(const FmaParams& P, unsigned bx, TileF& T)
{
    const int tile[3] = {1, P.tile1, P.tile2};
    bool active = true;
#pragma unroll
    for (int a = 2; a >= 0; --a) {
        const unsigned q = bx / (unsigned)P.ntile[a];
        T.o[a] = (int)(bx - q * P.ntile[a]) * tile[a];
        bx = q;
    }
#pragma unroll
    for (int a = 2; a >= 0; --a) {
        const unsigned q = bx / (unsigned)P.dil[a];
        T.rg[a] = (int)(bx - q * P.dil[a]);
        bx = q;
        T.Lp[a] = (P.L[a] - T.rg[a] + P.dil[a] - 1) / P.dil[a];
        if (T.o[a] >= T.Lp[a]) active = false;
    }
    if (!active) return false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // along a0 there is one row, and nothing but this box says which columns are its own (a key that no query attends to,
        // the last one of an even kernel, has none); along a1 and a2 each row has its own range in RowsF
        const int last = min(T.o[a] + tile[a], T.Lp[a]) - 1;
        int t, hi;
        range_of<kKeySide>(P, a, T.o[a], T.Lp[a], T.lo[a], t, a == 0);
        range_of<kKeySide>(P, a, last, T.Lp[a], t, hi, a == 0);
        T.n[a] = hi - T.lo[a];
    }
    return true;
}
__device__ __forceinline__ long long flat_of(const FmaParams& P, const TileF& T, int x0, int x1, int x2)
{
    return ((long long)(T.rg[0] + P.dil[0] * x0) * P.L[1] + (T.rg[1] + P.dil[1] * x1)) * P.L[2] + (T.rg[2] + P.dil[2] * x2);
}

// Eight values of a tensor row as four packed pairs.
template <typename T> __device__ __forceinline__ void widen8(const uint4& r, uint64_t (&x)[4])
{
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 f;
        if constexpr (std::is_same<T, __half>::value) f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        else f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        x[i] = pack2(f.x, f.y);
    }
}
template <typename T> __device__ __forceinline__ void load8(const T* p, uint64_t (&x)[4])
{
    if constexpr (std::is_same<T, float>::value) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 4);
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    } else {
        widen8<T>(*reinterpret_cast<const uint4*>(p), x);
    }
}
template <typename T> __device__ __forceinline__ void store8(T* p, const uint64_t (&x)[4])
{
    if constexpr (std::is_same<T, float>::value) {
        *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x[0], x[1]);
        *reinterpret_cast<ulonglong2*>(p + 4) = make_ulonglong2(x[2], x[3]);
    } else {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = tcplan::cvt_pack<std::is_same<T, __nv_bfloat16>::value>(lo_of(x[i]), hi_of(x[i]));
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
template <typename T> __device__ __forceinline__ float widen(T v)
{
    if constexpr (std::is_same<T, float>::value) return v;
    else if constexpr (std::is_same<T, __half>::value) return __half2float(v);
    else return __bfloat162float(v);
}
template <typename T> __device__ __forceinline__ T narrow(float v)
{
    if constexpr (std::is_same<T, float>::value) return v;
    else if constexpr (std::is_same<T, __half>::value) return __float2half_rn(v);
    else return __float2bfloat16_rn(v);
}

// Lane layout and shared-memory layout for head dim D.
template <int D, bool LINE> struct LaneF {
    static constexpr int LPQ = D / 8, GP = 32 / LPQ;     // lanes per row, groups of four rows per warp
    // physical piece of logical piece j of staged column x (rows of an even number of columns): neighbouring groups (columns one
    // apart; rank 1: four) or, for longer rows, the two halves of a 256-byte span read from different halves of the banks
    static __device__ __forceinline__ int piece(int j, int x) { return D == 32 ? j ^ ((LINE ? x >> 2 : x) & 1) : j ^ ((j >> 3) & 1); }
};

// Stage columns [y0, y1) x [s0, s1) (box-relative) at a0 position x0 of one tensor: [row][col][D] fp32.
template <typename T, int D, bool LINE>
__device__ __forceinline__ void stage_cols(const FmaParams& P, const TileF& Ti, const TensorF& t, int b, int h, int x0, int y0, int y1,
                                           int s0, int s1, float* dst)
{
    using LF = LaneF<D, LINE>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nc = s1 - s0;
    const T* base = static_cast<const T*>(t.p) + b * t.bs + h * t.hs;
    constexpr int V = std::is_same<T, float>::value ? 4 : 8;             // channels per 16-byte load
    constexpr int kLoads = D / V;
    for (int y = y0 + warp; y < y1; y += kWarpsF) {
        const long long pos = flat_of(P, Ti, x0, Ti.lo[1] + y, Ti.lo[2] + s0);
        const T* src = base + pos * t.ts;
        float* row = dst + (size_t)(y - y0) * P.chunk_cols * D;
        if constexpr (V == 4) {
            for (int i = lane; i < nc * kLoads; i += 32) {
                const int x = i / kLoads, j = i % kLoads;
                const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(row + x * D + 4 * LF::piece(j, x)));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src + (long long)x * P.dil[2] * t.ts + V * j) : "memory");
            }
        } else {
            for (int i0 = lane; i0 < nc * kLoads; i0 += 128) {           // four loads in flight (clamped, no branch between them)
                uint4 raw[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = min(i0 + 32 * u, nc * kLoads - 1);
                    raw[u] = *reinterpret_cast<const uint4*>(src + (long long)(i / kLoads) * P.dil[2] * t.ts + V * (i % kLoads));
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + 32 * u, x = i / kLoads, j = i % kLoads;
                    if (i >= nc * kLoads) break;
                    uint64_t v[4];
                    widen8<T>(raw[u], v);
                    float* d = row + x * D;
                    *reinterpret_cast<ulonglong2*>(d + 4 * LF::piece(2 * j, x)) = make_ulonglong2(v[0], v[1]);
                    *reinterpret_cast<ulonglong2*>(d + 4 * LF::piece(2 * j + 1, x)) = make_ulonglong2(v[2], v[3]);
                }
            }
        }
    }
}
__device__ __forceinline__ void staged()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// This lane's 8 channels (logical pieces 2c, 2c + 1) of a staged column.
template <int D, bool LINE>
__device__ __forceinline__ void read_col(const float* base, int cell, int c, uint64_t (&v)[4])
{
    using LF = LaneF<D, LINE>;
    const float* p = base + cell * D;
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p + 4 * LF::piece(2 * c, cell));
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(p + 4 * LF::piece(2 * c + 1, cell));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ float dot8(const uint64_t (&a)[4], const uint64_t (&b)[4])
{
    uint64_t s = mul2(a[0], b[0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) s = fma2(a[i], b[i], s);
    return lo_of(s) + hi_of(s);
}
// Partial sums of four rows over the group's lanes -> lane c gets the total of row c & 3.
template <int LPQ> __device__ __forceinline__ float reduce4(float s0, float s1, float s2, float s3, int c)
{
    const bool b0 = c & 1, b1 = c & 2;
    float k0 = b0 ? s1 : s0, k1 = b0 ? s3 : s2;
    k0 += __shfl_xor_sync(0xffffffffu, b0 ? s0 : s1, 1);
    k1 += __shfl_xor_sync(0xffffffffu, b0 ? s2 : s3, 1);
    float k = b1 ? k1 : k0;
    k += __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
#pragma unroll
    for (int m = 4; m < LPQ; m <<= 1) k += __shfl_xor_sync(0xffffffffu, k, m);
    return k;
}
// The value of row j, from the lane that has it.
__device__ __forceinline__ float row_value(float v, int lane, int c, int j) { return __shfl_sync(0xffffffffu, v, (lane - c) | j); }
__device__ __forceinline__ uint64_t twice(float v) { return pack2(v, v); }
// Bits 0 .. 3: does the column at hand belong to rows 0 .. 3 of the group?  (ok: to the lane's own row.)
__device__ __forceinline__ uint32_t rows_with(bool ok, int lane, int c) { return __ballot_sync(0xffffffffu, ok) >> (lane - c); }
// acc += w * x where `on` is not zero
__device__ __forceinline__ void add_if(uint32_t on, uint64_t (&acc)[4], uint64_t w, const uint64_t (&x)[4])
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %9, 0;\n\t"
        "@p fma.rn.f32x2 %0, %8, %4, %0;\n\t@p fma.rn.f32x2 %1, %8, %5, %1;\n\t"
        "@p fma.rn.f32x2 %2, %8, %6, %2;\n\t@p fma.rn.f32x2 %3, %8, %7, %3;\n\t}"
        : "+l"(acc[0]), "+l"(acc[1]), "+l"(acc[2]), "+l"(acc[3])
        : "l"(x[0]), "l"(x[1]), "l"(x[2]), "l"(x[3]), "l"(w), "r"(on));
}

// A lane's view of its group's four rows.
template <int D, bool LINE, bool kKeySide> struct RowsF {
    using LF = LaneF<D, LINE>;
    int lane, c, g, x1, x2;              // first row of the group
    int f1, f2;                          // own row (c & 3): its columns, box-relative ...
    unsigned n1, n2;
    int r0, r1, c0, c1;                  // the group's: rows of columns (warp-uniform) and columns; empty: none
    int nmax;                            // most columns of any group of the warp

    __device__ __forceinline__ void init(const FmaParams& P, const TileF& T)
    {
        const int warp = threadIdx.x >> 5;
        lane = threadIdx.x & 31;
        c = lane % LF::LPQ;
        g = lane / LF::LPQ;
        const int wx = warp % P.ww, wy = warp / P.ww;
        x1 = T.o[1] + (LINE ? 0 : 4 * wy);
        x2 = T.o[2] + (LINE ? 4 : 1) * (LF::GP * wx + g);
        const int j = c & 3;
        f1 = f2 = 0;
        n1 = n2 = 0u;
        if (exists(T, j)) {
            int e;
            range_of<kKeySide>(P, 1, row1(j), T.Lp[1], f1, e);
            n1 = e > f1 ? (unsigned)(e - f1) : 0u;
            range_of<kKeySide>(P, 2, row2(j), T.Lp[2], f2, e);
            n2 = e > f2 ? (unsigned)(e - f2) : 0u;
            f1 -= T.lo[1];
            f2 -= T.lo[2];
        }
        // unions over the rows that exist (bounds never decrease with the row)
        r0 = r1 = c0 = c1 = 0;
        if (x1 < T.Lp[1]) {
            int t;
            range_of<kKeySide>(P, 1, x1, T.Lp[1], r0, t, false);
            range_of<kKeySide>(P, 1, min(row1(3), T.Lp[1] - 1), T.Lp[1], t, r1, false);
            r0 -= T.lo[1];
            r1 -= T.lo[1];
        }
        if (x2 < T.Lp[2]) {
            int t;
            range_of<kKeySide>(P, 2, x2, T.Lp[2], c0, t, false);
            range_of<kKeySide>(P, 2, min(row2(3), T.Lp[2] - 1), T.Lp[2], t, c1, false);
            c0 -= T.lo[2];
            c1 -= T.lo[2];
        }
    }
    __device__ __forceinline__ int row1(int j) const { return x1 + (LINE ? 0 : j); }
    __device__ __forceinline__ int row2(int j) const { return x2 + (LINE ? j : 0); }
    __device__ __forceinline__ bool exists(const TileF& T, int j) const { return row1(j) < T.Lp[1] && row2(j) < T.Lp[2]; }
    __device__ __forceinline__ long long flat(const FmaParams& P, const TileF& T, int j) const { return flat_of(P, T, T.o[0], row1(j), row2(j)); }

    // this lane's 8 channels of the four rows (zero where there is no row)
    template <typename T> __device__ __forceinline__ void load_rows(const FmaParams& P, const TileF& Ti, const TensorF& t, int b, int h,
                                                                    uint64_t (&x)[4][4]) const
    {
        const T* base = static_cast<const T*>(t.p) + b * t.bs + h * t.hs + 8 * c;
#pragma unroll
        for (int j = 0; j < 4; ++j)                          // clamped, so that the loads need no branch
            load8<T>(base + flat_of(P, Ti, Ti.o[0], min(row1(j), Ti.Lp[1] - 1), min(row2(j), Ti.Lp[2] - 1)) * t.ts, x[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (!exists(Ti, j))
#pragma unroll
                for (int i = 0; i < 4; ++i) x[j][i] = 0ull;
    }
    // acc[row] += a * xa + b * xb over the group's rows, a and b from the lane that has the row (zero where it does not attend
    // to the column).  kExact: the columns that a row does not attend to are left out, whatever they hold; see exact_if_tainted.
    template <bool kExact>
    __device__ __forceinline__ void add_pair(uint64_t (&acc)[4][4], bool ok_a, float a, const uint64_t (&xa)[4], bool ok_b, float b,
                                             const uint64_t (&xb)[4]) const
    {
        const uint32_t in_a = kExact ? rows_with(ok_a, lane, c) : 0u, in_b = kExact ? rows_with(ok_b, lane, c) : 0u;
        a = ok_a ? a : 0.f;
        b = ok_b ? b : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) add_row<kExact>(j, acc[j], in_a, a, xa, in_b, b, xb);
    }
    template <bool kExact>
    __device__ __forceinline__ void add_row(int j, uint64_t (&acc)[4], uint32_t in_a, float a, const uint64_t (&xa)[4], uint32_t in_b,
                                            float b, const uint64_t (&xb)[4]) const
    {
        const uint64_t a2 = twice(row_value(a, lane, c, j)), b2 = twice(row_value(b, lane, c, j));
        if constexpr (kExact) {
            add_if(in_a & (1u << j), acc, a2, xa);
            add_if(in_b & (1u << j), acc, b2, xb);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = fma2(b2, xb[i], fma2(a2, xa[i], acc[i]));
        }
    }
    // Walk the staged chunk [y0, y1) x [s0, s1) two columns at a time (independent chains for the scheduler): neighbours along
    // a1 (rank 1: along a2), of which a group's union has an even number when the kernel size is odd.
    // body(shared-memory column of the first, of the second, whether each belongs to the lane's own row, box-relative row and column
    // of the first; the second is one row further, rank 1: one column)
    template <typename F> __device__ __forceinline__ void walk(const FmaParams& P, int y0, int y1, int s0, int s1, F&& body) const
    {
        walk_ahead<1>(P, y0, y1, s0, s1, [](int, bool, bool, int, int) {},
                      [&](int, int xa, int xb, bool ok_a, bool ok_b, int y, int x) { body(xa, xb, ok_a, ok_b, y, x); });
    }
    // The same with up to N pairs of columns announced together: ahead(u, ok_a, ok_b, y, x) for each of them, then
    // body(u, ...) for each (what a lane has to fetch for its row is in flight by then).
    template <int N, typename G, typename F>
    __device__ __forceinline__ void walk_ahead(const FmaParams& P, int y0, int y1, int s0, int s1, G&& ahead, F&& body) const
    {
        const int a = max(c0, s0), n = min(c1, s1) - a;
        int most = n > 0 ? n : 0;
#pragma unroll
        for (int m = 16; m >= LF::LPQ; m >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, m));
        const int from = max(r0, y0), to = min(r1, y1), last = s1 - 1 - s0;
        constexpr int kStep = LINE ? 2 : 1;                  // columns along a2 per pair
        for (int y = from; y < to; y += 3 - kStep) {
            const int yb = min(y + 1, to - 1);
            const bool row_a = (unsigned)(y - f1) < n1, row_b = LINE ? row_a : y + 1 < to && (unsigned)(y + 1 - f1) < n1;
            const int cell_a = (y - y0) * P.chunk_cols, cell_b = LINE ? cell_a : (yb - y0) * P.chunk_cols;
            for (int t0 = 0; t0 < most; t0 += N * kStep) {
                auto ok = [&](int t, bool row) { return row && t < n && (unsigned)(a + t - f2) < n2; };
                if constexpr (N > 1) {
#pragma unroll
                    for (int u = 0; u < N; ++u) {
                        const int t = t0 + u * kStep;
                        ahead(u, ok(t, row_a), ok(t + kStep - 1, row_b), y, a + t);
                    }
                }
#pragma unroll
                for (int u = 0; u < N; ++u) {
                    const int t = t0 + u * kStep;
                    if (t >= most) break;
                    body(u, cell_a + min(a + t - s0, last), cell_b + min(a + t + kStep - 1 - s0, last), ok(t, row_a), ok(t + kStep - 1, row_b),
                         y, a + t);
                }
            }
        }
    }
};

// Walks the CTA's column box in chunks: before(x0, y0, y1, s0, s1) stages one, then every warp visits it.
template <typename Stage, typename Visit>
__device__ __forceinline__ void for_chunks(const FmaParams& P, const TileF& T, Stage&& stage, Visit&& visit)
{
    for (int i0 = 0; i0 < T.n[0]; ++i0)
        for (int y0 = 0; y0 < T.n[1]; y0 += P.chunk_rows)
            for (int s0 = 0; s0 < T.n[2]; s0 += P.chunk_cols) {
                const int y1 = min(y0 + P.chunk_rows, T.n[1]), s1 = min(s0 + P.chunk_cols, T.n[2]);
                __syncthreads();
                stage(T.lo[0] + i0, y0, y1, s0, s1);
                staged();
                visit(T.lo[0] + i0, y0, y1, s0, s1);
            }
}

__device__ __forceinline__ void clear(uint64_t (&acc)[4][4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0ull;
}
// Not 0: some value is NaN or Inf.
__device__ __forceinline__ int tainted(const uint64_t (&acc)[4][4])
{
    uint64_t t = 0ull;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) t = fma2(acc[j][i], 0ull, t);
    return lo_of(t) + hi_of(t) == 0.f ? 0 : 1;
}
// Runs pass(false), and pass(true) over it if that left a NaN or Inf in the CTA's sums (taint()).  Four rows share every column,
// and the plain pass gives a row that does not attend to it a weight of zero, which a NaN or Inf turns into NaN; the exact pass
// leaves it out.  Exact arithmetic throughout (a vote, and a predicate per row and column) took a float32 training step of
// 56 x 56, 7 x 7, 4 heads of 32, batch 4 from 155 to 199 us; the test at the end takes it to 158.
template <typename Pass, typename Taint> __device__ __forceinline__ void exact_if_tainted(Pass&& pass, Taint&& taint)
{
    pass(std::false_type{});
    if (__syncthreads_or(taint())) pass(std::true_type{});
}

// ---------------------------------------------------------------------------------------------------------------
// fused forward.  Row i's stabiliser lives in lane i of its group: the first score it meets; moved (everything
// accumulated so far is rescaled, a warp-uniform branch) only when a score exceeds it by 2^30.
// ---------------------------------------------------------------------------------------------------------------
template <typename T, int D, bool LINE>
__global__ void __launch_bounds__(kThreadsF, 3)
fma_fwd_kernel(const __grid_constant__ FmaParams P, T* __restrict__ out, float* __restrict__ lse)
{
    using LF = LaneF<D, LINE>;
    extern __shared__ __align__(16) float sm[];
    const int h = blockIdx.y, b = blockIdx.z, hk = h / P.group;
    TileF Ti;
    if (!tile_of<false>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, false> R;
    R.init(P, Ti);
    uint64_t q[4][4], acc[4][4];
    R.template load_rows<T>(P, Ti, P.row1, b, h, q);
    float m, l;
    float* vs = sm + P.chunk_rows * P.chunk_cols * D;
    exact_if_tainted([&](auto exact) {
        constexpr bool kExact = decltype(exact)::value;
        clear(acc);
        m = -FLT_MAX;                                        // finite: masked scores (-inf) minus it stay -inf
        l = 0.f;
        for_chunks(P, Ti,
            [&](int x0, int y0, int y1, int s0, int s1) {
                stage_cols<T, D, LINE>(P, Ti, P.col1, b, hk, x0, y0, y1, s0, s1, sm);
                stage_cols<T, D, LINE>(P, Ti, P.col2, b, hk, x0, y0, y1, s0, s1, vs);
            },
            [&](int, int y0, int y1, int s0, int s1) {
                R.walk(P, y0, y1, s0, s1, [&](int xa, int xb, bool ok_a, bool ok_b, int, int) {
                    uint64_t ka[4], kb[4], va[4], vb[4];
                    read_col<D, LINE>(sm, xa, R.c, ka);
                    read_col<D, LINE>(sm, xb, R.c, kb);
                    float sa = reduce4<LF::LPQ>(dot8(q[0], ka), dot8(q[1], ka), dot8(q[2], ka), dot8(q[3], ka), R.c) * P.scale_log2;
                    float sb = reduce4<LF::LPQ>(dot8(q[0], kb), dot8(q[1], kb), dot8(q[2], kb), dot8(q[3], kb), R.c) * P.scale_log2;
                    read_col<D, LINE>(vs, xa, R.c, va);
                    read_col<D, LINE>(vs, xb, R.c, vb);
                    sa = ok_a ? sa : -INFINITY;
                    sb = ok_b ? sb : -INFINITY;
                    const float top = fmaxf(sa, sb);
                    if (__any_sync(0xffffffffu, top > m + 30.f)) {
                        const bool grow = top > m + 30.f;
                        const float fac = grow ? fast_exp2(m - top) : 1.f;
                        if (grow) m = top;
                        l *= fac;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint64_t f2 = twice(row_value(fac, R.lane, R.c, j));
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[j][i] = mul2(acc[j][i], f2);
                        }
                    }
                    const float pa = fast_exp2(sa - m), pb = fast_exp2(sb - m);
                    l += pa + pb;
                    R.template add_pair<kExact>(acc, ok_a, pa, va, ok_b, pb, vb);
                });
            });
    }, [&] { return tainted(acc); });
    const float inv = 1.f / l;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint64_t f2 = twice(row_value(inv, R.lane, R.c, j));
        if (!R.exists(Ti, j)) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = mul2(acc[j][i], f2);
        store8<T>(out + (((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hq + h) * D + 8 * R.c, acc[j]);
    }
    if (R.c < 4 && R.exists(Ti, R.c))
        lse[((long long)b * P.ltot + R.flat(P, Ti, R.c)) * P.Hq + h] = (m + log2f(l)) * kLn2;
}

// ---------------------------------------------------------------------------------------------------------------
// fused backward, query side: dQ, and delta = rowsum(out * dout) - dlse for the key side
// ---------------------------------------------------------------------------------------------------------------
template <typename T, int D, bool LINE>
__global__ void __launch_bounds__(kThreadsF, 3)
fma_bwd_q_kernel(const __grid_constant__ FmaParams P, const T* __restrict__ out, const float* __restrict__ lse,
                 const float* __restrict__ dlse, float* __restrict__ delta, T* __restrict__ dq)
{
    using LF = LaneF<D, LINE>;
    extern __shared__ __align__(16) float sm[];
    const int h = blockIdx.y, b = blockIdx.z, hk = h / P.group;
    TileF Ti;
    if (!tile_of<false>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, false> R;
    R.init(P, Ti);
    uint64_t q[4][4], go[4][4], acc[4][4];
    float lse2 = 0.f, dl = 0.f;
    {
        const TensorF ot{out, P.ltot * P.Hq * D, (long long)P.Hq * D, D};
        R.template load_rows<T>(P, Ti, ot, b, h, q);
        R.template load_rows<T>(P, Ti, P.row2, b, h, go);
        dl = reduce4<LF::LPQ>(dot8(q[0], go[0]), dot8(q[1], go[1]), dot8(q[2], go[2]), dot8(q[3], go[3]), R.c);
        const int j = R.c & 3;
        if (R.exists(Ti, j)) {
            const long long row = ((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hq + h;
            lse2 = lse[row] * kLog2e;
            if (dlse) dl -= dlse[row];
            if (R.c < 4) delta[row] = dl;
        }
    }
    R.template load_rows<T>(P, Ti, P.row1, b, h, q);
    float* vs = sm + P.chunk_rows * P.chunk_cols * D;
    exact_if_tainted([&](auto exact) {
        constexpr bool kExact = decltype(exact)::value;
        clear(acc);
        for_chunks(P, Ti,
            [&](int x0, int y0, int y1, int s0, int s1) {
                stage_cols<T, D, LINE>(P, Ti, P.col1, b, hk, x0, y0, y1, s0, s1, sm);
                stage_cols<T, D, LINE>(P, Ti, P.col2, b, hk, x0, y0, y1, s0, s1, vs);
            },
            [&](int, int y0, int y1, int s0, int s1) {
                R.walk(P, y0, y1, s0, s1, [&](int xa, int xb, bool ok_a, bool ok_b, int, int) {
                    auto one = [&](int x, uint64_t (&k)[4]) {
                        uint64_t v[4];
                        read_col<D, LINE>(sm, x, R.c, k);
                        read_col<D, LINE>(vs, x, R.c, v);
                        const float s = reduce4<LF::LPQ>(dot8(q[0], k), dot8(q[1], k), dot8(q[2], k), dot8(q[3], k), R.c);
                        const float dp = reduce4<LF::LPQ>(dot8(go[0], v), dot8(go[1], v), dot8(go[2], v), dot8(go[3], v), R.c);
                        return fast_exp2(fmaf(s, P.scale_log2, -lse2)) * (dp - dl) * P.scale;
                    };
                    uint64_t ka[4], kb[4];
                    const float da = one(xa, ka), db = one(xb, kb);
                    R.template add_pair<kExact>(acc, ok_a, da, ka, ok_b, db, kb);
                });
            });
    }, [&] { return tainted(acc); });
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (R.exists(Ti, j)) store8<T>(dq + (((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hq + h) * D + 8 * R.c, acc[j]);
}

// ---------------------------------------------------------------------------------------------------------------
// fused backward, key side: dK and dV over the queries that attend to the keys, one query head of the group at a time
// ---------------------------------------------------------------------------------------------------------------
template <typename T, int D, bool LINE>
__global__ void __launch_bounds__(kThreadsF, 2)
fma_bwd_k_kernel(const __grid_constant__ FmaParams P, const float* __restrict__ lse, const float* __restrict__ delta,
                 T* __restrict__ dk, T* __restrict__ dv)
{
    using LF = LaneF<D, LINE>;
    extern __shared__ __align__(16) float sm[];
    const int hk = blockIdx.y, b = blockIdx.z;
    TileF Ti;
    if (!tile_of<true>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, true> R;
    R.init(P, Ti);
    uint64_t k[4][4], v[4][4], ak[4][4], av[4][4];
    R.template load_rows<T>(P, Ti, P.row1, b, hk, k);
    R.template load_rows<T>(P, Ti, P.row2, b, hk, v);
    const int cells = P.chunk_rows * P.chunk_cols;
    float* gs = sm + cells * D;
    float2* stats = reinterpret_cast<float2*>(gs + cells * D);       // lse * log2(e), delta of the chunk's queries
    exact_if_tainted([&](auto exact) {
        constexpr bool kExact = decltype(exact)::value;
        clear(ak);
        clear(av);
        for (int h = hk * P.group; h < (hk + 1) * P.group; ++h)
            for_chunks(P, Ti,
                [&](int x0, int y0, int y1, int s0, int s1) {
                    stage_cols<T, D, LINE>(P, Ti, P.col1, b, h, x0, y0, y1, s0, s1, sm);
                    stage_cols<T, D, LINE>(P, Ti, P.col2, b, h, x0, y0, y1, s0, s1, gs);
                    for (int y = y0 + (threadIdx.x >> 5); y < y1; y += kWarpsF)
                        for (int x = s0 + (threadIdx.x & 31); x < s1; x += 32) {
                            const long long row = ((long long)b * P.ltot + flat_of(P, Ti, x0, Ti.lo[1] + y, Ti.lo[2] + x)) * P.Hq + h;
                            stats[(y - y0) * P.chunk_cols + (x - s0)] = make_float2(lse[row] * kLog2e, delta[row]);
                        }
                },
                [&](int, int y0, int y1, int s0, int s1) {
                    R.walk(P, y0, y1, s0, s1, [&](int xa, int xb, bool ok_a, bool ok_b, int, int) {
                        auto one = [&](int x, bool ok, uint64_t (&q)[4], uint64_t (&go)[4], float& p, float& ds) {
                            read_col<D, LINE>(sm, x, R.c, q);
                            read_col<D, LINE>(gs, x, R.c, go);
                            const float2 st = stats[x];
                            const float s = reduce4<LF::LPQ>(dot8(k[0], q), dot8(k[1], q), dot8(k[2], q), dot8(k[3], q), R.c);
                            const float dp = reduce4<LF::LPQ>(dot8(v[0], go), dot8(v[1], go), dot8(v[2], go), dot8(v[3], go), R.c);
                            p = fast_exp2(fmaf(s, P.scale_log2, -st.x));
                            ds = p * (dp - st.y) * P.scale;
                            p = ok ? p : 0.f;
                            ds = ok ? ds : 0.f;
                        };
                        uint64_t qa[4], qb[4], ga[4], gb[4];
                        float pa, pb, da, db;
                        one(xa, ok_a, qa, ga, pa, da);
                        one(xb, ok_b, qb, gb, pb, db);
                        const uint32_t in_a = kExact ? rows_with(ok_a, R.lane, R.c) : 0u, in_b = kExact ? rows_with(ok_b, R.lane, R.c) : 0u;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            R.template add_row<kExact>(j, av[j], in_a, pa, ga, in_b, pb, gb);
                            R.template add_row<kExact>(j, ak[j], in_a, da, qa, in_b, db, qb);
                        }
                    });
                });
    }, [&] { return tainted(ak) | tainted(av); });
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (R.exists(Ti, j)) {
            const long long o = (((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hkv + hk) * D + 8 * R.c;
            store8<T>(dk + o, ak[j]);
            store8<T>(dv + o, av[j]);
        }
}

// ---------------------------------------------------------------------------------------------------------------
// split operators.  A window's slot is linear in the column: slot = (k0 * K1 + k1) * K2 + k2 with k = column - first column
// of the window (which a causal axis may place before the tensor).
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ int first_of(const FmaParams& P, int a, int x, int Lp)
{
    return P.causal[a] ? x - (P.K[a] - 1) : window_start(x, Lp, P.K[a], 1);
}
// Slot of box column (a0 position i0, y, x) in the own row's window = base + y * K2 + x for the a0 position at hand.
struct SlotF {
    int base, per0;
    template <typename Rows> __device__ __forceinline__ void init(const FmaParams& P, const TileF& T, const Rows& R)
    {
        const int j = R.c & 3;
        per0 = P.K[1] * P.K[2];
        base = -first_of(P, 0, T.o[0], T.Lp[0]) * per0 + (T.lo[1] - first_of(P, 1, R.row1(j), T.Lp[1])) * P.K[2] +
               (T.lo[2] - first_of(P, 2, R.row2(j), T.Lp[2]));
    }
    __device__ __forceinline__ int at(int i0) const { return base + i0 * per0; }
};
// Writes the warp's `n` rows of ktot values from shared memory, eight rows at a time (a row is too short and too oddly aligned
// for wider accesses).  at(i): element offset of row i's values, -1 none.
template <typename T, typename At>
__device__ __forceinline__ void write_rows(const FmaParams& P, T* global, const T* shared, int n, At&& at)
{
    const int lane = threadIdx.x & 31, ktot = P.ktot;
    for (int i0 = 0; i0 < n; i0 += 8) {
        long long off[8];
        {
            const int i = i0 + (lane & 7);                  // lanes 0 .. 7 work out a row each
            const long long o = i < n ? at(i) : -1;
#pragma unroll
            for (int u = 0; u < 8; ++u) off[u] = __shfl_sync(0xffffffffu, o, u);
        }
        for (int s = lane; s < ktot; s += 32) {
            T v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = shared[(i0 + u < n ? i0 + u : 0) * ktot + s];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (off[u] >= 0) global[off[u] + s] = v[u];
        }
    }
}
// Element offset of the slots of row i (0 .. 4 * GP - 1) of the warp's block, -1: no such row.
template <int D, bool LINE>
__device__ __forceinline__ long long warp_row(const FmaParams& P, const TileF& T, int i, int b, int h)
{
    using LF = LaneF<D, LINE>;
    const int warp = threadIdx.x >> 5, wx = warp % P.ww, wy = warp / P.ww;
    const int x1 = T.o[1] + (LINE ? 0 : 4 * wy + (i & 3)), x2 = T.o[2] + (LINE ? 4 * LF::GP * wx + i : LF::GP * wx + (i >> 2));
    if (x1 >= T.Lp[1] || x2 >= T.Lp[2]) return -1;
    return (((long long)b * P.ltot + flat_of(P, T, T.o[0], x1, x2)) * P.Hq + h) * P.ktot;
}
// Bias window start of the relative position bias at position p of an axis (odd kernels).
__device__ __forceinline__ int bias_start(int p, int L, int K, int d)
{
    const int nh = K / 2;
    if (d <= 1) return nh + (p < nh ? nh - p : (p + nh >= L ? L - p - 1 - nh : 0));
    return p - nh * d < 0 ? K - 1 - p / d : (p + nh * d >= L ? (L - p - 1) / d : nh);
}

// out[row, slot] = scale * <x[row], y[column]>  (+ bias): logits, or the gradient of the attention weights.  The rows' slots
// are collected in shared memory and leave in whole rows.
template <typename T, int D, bool LINE, bool kBias>
__global__ void __launch_bounds__(kThreadsF, 4)
fma_scores_kernel(const __grid_constant__ FmaParams P, T* __restrict__ out, float fill, const T* __restrict__ rpb)
{
    using LF = LaneF<D, LINE>;
    extern __shared__ __align__(16) float sm[];
    const int h = blockIdx.y, b = blockIdx.z, hk = h / P.group, warp = threadIdx.x >> 5;
    TileF Ti;
    if (!tile_of<false>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, false> R;
    R.init(P, Ti);
    SlotF S;
    S.init(P, Ti, R);
    uint64_t q[4][4];
    R.template load_rows<T>(P, Ti, P.row1, b, h, q);
    T* tile = reinterpret_cast<T*>(sm + P.chunk_rows * P.chunk_cols * D) + warp * 4 * LF::GP * P.ktot;
    T* mine = tile + (4 * R.g + (R.c & 3)) * P.ktot;
    for (int i = R.lane; i < 4 * LF::GP * P.ktot; i += 32) tile[i] = narrow<T>(fill);
    __syncwarp();
    // bias entry of slot (k0, k1, k2): ((pb0 + k0) * (2 K1 - 1) + pb1 + k1) * (2 K2 - 1) + pb2 + k2, as entry + y * w2 + x
    int entry = 0, w2 = 0, w1 = 0;
    if constexpr (kBias) {
        const int j = R.c & 3, x1 = R.row1(j), x2 = R.row2(j);
        w2 = 2 * P.K[2] - 1;
        w1 = (2 * P.K[1] - 1) * w2;
        const int p0 = Ti.rg[0] + P.dil[0] * Ti.o[0], p1 = Ti.rg[1] + P.dil[1] * x1, p2 = Ti.rg[2] + P.dil[2] * x2;
        entry = (bias_start(p0, P.L[0], P.K[0], P.dil[0]) - first_of(P, 0, Ti.o[0], Ti.Lp[0])) * w1 +
                (bias_start(p1, P.L[1], P.K[1], P.dil[1]) + Ti.lo[1] - first_of(P, 1, x1, Ti.Lp[1])) * w2 +
                bias_start(p2, P.L[2], P.K[2], P.dil[2]) + Ti.lo[2] - first_of(P, 2, x2, Ti.Lp[2]);
        rpb += (long long)h * (2 * P.K[0] - 1) * w1;
    }
    for_chunks(P, Ti,
        [&](int x0, int y0, int y1, int s0, int s1) { stage_cols<T, D, LINE>(P, Ti, P.col1, b, hk, x0, y0, y1, s0, s1, sm); },
        [&](int x0, int y0, int y1, int s0, int s1) {
            const int at = S.at(x0);
            R.walk(P, y0, y1, s0, s1, [&](int xa, int xb, bool ok_a, bool ok_b, int y, int x) {
                uint64_t ka[4], kb[4];
                read_col<D, LINE>(sm, xa, R.c, ka);
                read_col<D, LINE>(sm, xb, R.c, kb);
                float sa = reduce4<LF::LPQ>(dot8(q[0], ka), dot8(q[1], ka), dot8(q[2], ka), dot8(q[3], ka), R.c) * P.scale;
                float sb = reduce4<LF::LPQ>(dot8(q[0], kb), dot8(q[1], kb), dot8(q[2], kb), dot8(q[3], kb), R.c) * P.scale;
                const int slot = at + y * P.K[2] + x, step = LINE ? 1 : P.K[2];
                if constexpr (kBias) {
                    const T* e = rpb + entry + x0 * w1 + y * w2 + x;
                    if (ok_a) sa += widen(e[0]);
                    if (ok_b) sb += widen(e[LINE ? 1 : w2]);
                }
                if (R.c < 4) {
                    if (ok_a) mine[slot] = narrow<T>(sa);
                    if (ok_b) mine[slot + step] = narrow<T>(sb);
                }
            });
        });
    __syncwarp();
    write_rows(P, out, tile, 4 * LF::GP, [&](int i) { return warp_row<D, LINE>(P, Ti, i, b, h); });
}

// out[row] = scale * sum over slots of w[row, slot] * y[column]: values weighted by attention, or the gradient of the queries.
template <typename T, int D, bool LINE>
__global__ void __launch_bounds__(kThreadsF, 4)
fma_apply_kernel(const __grid_constant__ FmaParams P, const T* __restrict__ w, T* __restrict__ out)
{
    extern __shared__ __align__(16) float sm[];
    const int h = blockIdx.y, b = blockIdx.z, hk = h / P.group;
    TileF Ti;
    if (!tile_of<false>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, false> R;
    R.init(P, Ti);
    SlotF S;
    S.init(P, Ti, R);
    const int own = R.c & 3;
    const T* mine = w + (R.exists(Ti, own) ? (((long long)b * P.ltot + R.flat(P, Ti, own)) * P.Hq + h) * P.ktot : 0ll);
    uint64_t acc[4][4];
    exact_if_tainted([&](auto exact) {
        constexpr bool kExact = decltype(exact)::value;
        clear(acc);
        for_chunks(P, Ti,
            [&](int x0, int y0, int y1, int s0, int s1) { stage_cols<T, D, LINE>(P, Ti, P.col1, b, hk, x0, y0, y1, s0, s1, sm); },
            [&](int x0, int y0, int y1, int s0, int s1) {
                const int at = S.at(x0);
                T wa8[kAheadF], wb8[kAheadF];
                R.template walk_ahead<kAheadF>(P, y0, y1, s0, s1, [&](int u, bool ok_a, bool ok_b, int y, int x) {
                    const int slot = at + y * P.K[2] + x;
                    wa8[u] = mine[ok_a ? slot : 0];
                    wb8[u] = mine[ok_b ? slot + (LINE ? 1 : P.K[2]) : 0];
                }, [&](int u, int xa, int xb, bool ok_a, bool ok_b, int, int) {
                    const float wa = widen(wa8[u]), wb = widen(wb8[u]);
                    uint64_t va[4], vb[4];
                    read_col<D, LINE>(sm, xa, R.c, va);
                    read_col<D, LINE>(sm, xb, R.c, vb);
                    R.template add_pair<kExact>(acc, ok_a, wa, va, ok_b, wb, vb);
                });
            });
    }, [&] { return tainted(acc); });
    const uint64_t sc2 = twice(P.scale);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (R.exists(Ti, j)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[j][i] = mul2(acc[j][i], sc2);
            store8<T>(out + (((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hq + h) * D + 8 * R.c, acc[j]);
        }
}

// dst[key] = scale * sum over the queries that attend to it of w[query, slot of the key] * x[query]: the gradient of the
// values, or of the keys.  Every weight is read once, by the lane that owns the key, kAheadF pairs at a time.
template <typename T, int D, bool LINE>
__global__ void __launch_bounds__(kThreadsF, 4)
fma_gather_kernel(const __grid_constant__ FmaParams P, const T* __restrict__ w, T* __restrict__ dst)
{
    extern __shared__ __align__(16) float sm[];
    const int hk = blockIdx.y, b = blockIdx.z;
    TileF Ti;
    if (!tile_of<true>(P, blockIdx.x, Ti)) return;
    RowsF<D, LINE, true> R;
    R.init(P, Ti);
    const int n1 = R.row1(R.c & 3), n2 = R.row2(R.c & 3);
    uint64_t acc[4][4];
    exact_if_tainted([&](auto exact) {
        constexpr bool kExact = decltype(exact)::value;
        clear(acc);
        for (int h = hk * P.group; h < (hk + 1) * P.group; ++h)
            for_chunks(P, Ti,
                [&](int x0, int y0, int y1, int s0, int s1) { stage_cols<T, D, LINE>(P, Ti, P.col1, b, h, x0, y0, y1, s0, s1, sm); },
                [&](int x0, int y0, int y1, int s0, int s1) {
                    // element of w: row of query (y, x), slot of the own key in its window (offsets within a sample fit 32 bits)
                    const int w2 = P.dil[2] * P.Hq * P.ktot, w1 = P.dil[1] * P.L[2] * P.Hq * P.ktot;
                    const T* base = w + (((long long)b * P.ltot + flat_of(P, Ti, x0, Ti.lo[1], Ti.lo[2])) * P.Hq + h) * P.ktot;
                    const int own = ((Ti.o[0] - first_of(P, 0, x0, Ti.Lp[0])) * P.K[1] + n1) * P.K[2] + n2;
                    T wa8[kAheadF], wb8[kAheadF];
                    R.template walk_ahead<kAheadF>(P, y0, y1, s0, s1, [&](int u, bool ok_a, bool ok_b, int y, int x) {
                        const int at = own + x * w2 - first_of(P, 2, Ti.lo[2] + x, Ti.Lp[2]);
                        if (LINE) {
                            wa8[u] = base[ok_a ? at : 0];
                            wb8[u] = base[ok_b ? own + (x + 1) * w2 - first_of(P, 2, Ti.lo[2] + x + 1, Ti.Lp[2]) : 0];
                        } else {
                            wa8[u] = base[ok_a ? at + y * w1 - P.K[2] * first_of(P, 1, Ti.lo[1] + y, Ti.Lp[1]) : 0];
                            wb8[u] = base[ok_b ? at + (y + 1) * w1 - P.K[2] * first_of(P, 1, Ti.lo[1] + y + 1, Ti.Lp[1]) : 0];
                        }
                    }, [&](int u, int xa, int xb, bool ok_a, bool ok_b, int, int) {
                        const float wa = widen(wa8[u]), wb = widen(wb8[u]);
                        uint64_t va[4], vb[4];
                        read_col<D, LINE>(sm, xa, R.c, va);
                        read_col<D, LINE>(sm, xb, R.c, vb);
                        R.template add_pair<kExact>(acc, ok_a, wa, va, ok_b, wb, vb);
                    });
                });
    }, [&] { return tainted(acc); });
    const uint64_t sc2 = twice(P.scale);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (R.exists(Ti, j)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[j][i] = mul2(acc[j][i], sc2);
            store8<T>(dst + (((long long)b * P.ltot + R.flat(P, Ti, j)) * P.Hkv + hk) * D + 8 * R.c, acc[j]);
        }
}

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------
// As much of the column box at a time as the CTAs that registers allow on an SM can have of its 227 KB: three of the forward and of
// dQ, two of the key side.  Every chunk is a barrier that nothing overlaps.  Measured, 56 x 56, 7 x 7, 4 heads of 32, batch 4, with
// 32, 48, 64, 72, 100 KB: forward 35.6, 34.3, 35.3, 30.2, 33.7 us (the last with two CTAs); dQ 42.9, 42.5, 43.5, 37.5, 42.1;
// dK and dV 80.6, 75.7, 75.5, 72.5, 67.0.  Against 64 KB for all, in nine shapes of ranks 1 to 3: forward and dQ equal or up to 15 %
// faster at head dim 32, equal to 4 % at 64 and 128; dK and dV 2 to 18 % (head dims 32 | 64 | 128, 56 x 56: 72 -> 65, 114 -> 111,
// 193 -> 179 us; 12 x 24 x 26, 3 x 3 x 3, 64: 169 -> 127; where the box then fits in one chunk 2 x: 48 x 60, 13 x 13, 128: 544 -> 286).
// Slower: 8 x 28 x 28, 3 x 5 x 5, 32: 123 -> 128; 88 x 106, 5 x 35, dilation 2 x 1, 1 head of 32: 235 -> 270 (undilated 208 -> 180; 3 x 35
// on 64 x 64, 64: 382 -> 199).
constexpr int kQueryChunk = 72 * 1024, kKeyChunk = 100 * 1024;

// Rows of a warp are 4 x (256 / D) (rank 1: one row of 1024 / D).  `tensors`: column tensors staged side by side,
// `extra`: further shared-memory bytes per staged column, `budget`: bytes of a chunk.
bool make_fma(const Geo& g, FmaParams& p, bool key_side, int tensors, int extra, size_t fixed, int budget, dim3& grid, size_t& smem)
{
    if ((g.D != 32 && g.D != 64 && g.D != 128) || g.n_extra || g.extents || g.B == 0) return false;
    const int pad = 3 - g.rank;
    for (int a = 0; a < 3; ++a) {
        const int s = a - pad;
        p.L[a] = s >= 0 ? g.L[s] : 1;
        p.K[a] = s >= 0 ? g.K[s] : 1;
        p.dil[a] = s >= 0 ? g.dil[s] : 1;
        p.causal[a] = s >= 0 ? g.causal[s] : 0;
        if (s >= 0 && (g.st[s] != 1 || !kernel_axis_ok(g, s))) return false;
    }
    p.rank = g.rank; p.B = g.B; p.Hq = g.Hq; p.Hkv = g.Hkv; p.group = g.group;
    p.ltot = g.ltot; p.ktot = g.ktot;
    p.scale = (float)g.scale;
    p.scale_log2 = (float)(g.scale * 1.4426950408889634);
    const int gp = 256 / g.D, inverse = key_side ? 1 : 0;
    if (g.rank == 1) {
        p.ww = kWarpsF;
        p.tile1 = 1;
        p.tile2 = 4 * gp * kWarpsF;
    } else {
        // warps side by side or stacked: fewest columns staged and rows of columns walked over the whole grid
        const int lp1 = (p.L[1] + p.dil[1] - 1) / p.dil[1], lp2 = (p.L[2] + p.dil[2] - 1) / p.dil[2];
        long long best = -1;
        for (int ww = kWarpsF; ww >= 1; ww /= 2) {
            const int t1 = 4 * (kWarpsF / ww), t2 = gp * ww;
            const long long n = (long long)((lp1 + t1 - 1) / t1) * ((lp2 + t2 - 1) / t2) *
                                ((t1 - 1 + p.K[1]) * (long long)(t2 - 1 + p.K[2]) + 2LL * kWarpsF * (3 + p.K[1]) * p.K[2]);
            if (best < 0 || n < best) { best = n; p.ww = ww; p.tile1 = t1; p.tile2 = t2; }
        }
    }
    long long tiles = 1;
    const int tile[3] = {1, p.tile1, p.tile2};
    for (int a = 0; a < 3; ++a) {
        p.ntile[a] = ((p.L[a] + p.dil[a] - 1) / p.dil[a] + tile[a] - 1) / tile[a];
        tiles *= (long long)p.ntile[a] * p.dil[a];
    }
    const int heads = key_side ? g.Hkv : g.Hq;
    if (tiles > 0x7fffffffll || heads > 65535 || g.B > 65535) return false;
    grid = dim3((unsigned)tiles, (unsigned)heads, (unsigned)g.B);
    // Chunk: whole rows of the box where two of them fit in the budget, else pieces of one row.
    const int cell = g.D * 4 * tensors + extra;
    auto longest = [&](int a) {                              // of a CTA's box along axis a, clamped edges included
        const int lp = (p.L[a] + p.dil[a] - 1) / p.dil[a];
        return std::min(lp, tile[a] - 1 + p.K[a] + inverse * (p.causal[a] ? 0 : p.K[a]));
    };
    p.chunk_cols = (longest(2) + 7) / 8 * 8;                 // a multiple of what the swizzle looks at
    if (p.chunk_cols * cell > budget / 2) p.chunk_cols = std::max(8, std::min(p.chunk_cols, budget / cell / 8 * 8));
    p.chunk_rows = std::max(1, std::min(longest(1), budget / (p.chunk_cols * cell)));
    if (p.chunk_rows < longest(1) && p.chunk_rows > 1) p.chunk_rows &= ~1;       // rows are taken in pairs
    smem = (size_t)p.chunk_rows * p.chunk_cols * cell + fixed;
    return smem <= kMaxDynamicSmem;
}

// Rows readable 16 bytes at a time.
bool vec_rows(const void* p, const long long s[3], int elt)
{
    return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && s[0] * elt % 16 == 0 && s[1] * elt % 16 == 0 && s[2] * elt % 16 == 0;
}
TensorF tensor_of(const void* p, const long long s[3]) { return TensorF{p, s[0], s[1], s[2]}; }
TensorF dense(const void* p, const Geo& g, int heads, int D)
{
    return TensorF{p, g.ltot * heads * (long long)D, (long long)heads * D, D};
}
template <typename F> void with_dim(int D, F&& f)
{
    if (D == 32) f(std::integral_constant<int, 32>{});
    else if (D == 64) f(std::integral_constant<int, 64>{});
    else f(std::integral_constant<int, 128>{});
}
template <typename F> void with_line(const Geo& g, F&& f)
{
    if (g.rank == 1) f(std::true_type{});
    else f(std::false_type{});
}
template <typename K> cudaError_t prepare_kernel(K kernel, size_t smem)
{
    return smem > 48 * 1024 ? ensure_dynamic_smem((const void*)kernel, kMaxDynamicSmem) : cudaSuccess;
}

} // namespace

int fma_fused_fwd(int dtype, const Geo& g, const void* q, const void* k, const void* v, void* out, void* lse, cudaStream_t s)
{
    if (dtype != 0 || g.Dv != g.D || !vec_rows(q, g.qs, 4) || !vec_rows(k, g.ks, 4) || !vec_rows(v, g.vs, 4) ||
        (reinterpret_cast<uintptr_t>(out) & 15u))
        return -2;
    FmaParams p;
    dim3 grid;
    size_t smem;
    if (!make_fma(g, p, false, 2, 0, 0, kQueryChunk, grid, smem)) return -2;
    p.row1 = tensor_of(q, g.qs);
    p.col1 = tensor_of(k, g.ks);
    p.col2 = tensor_of(v, g.vs);
    cudaError_t err = cudaSuccess;
    with_dim(g.D, [&](auto dim) {
        with_line(g, [&](auto line) {
            auto* kernel = fma_fwd_kernel<float, decltype(dim)::value, decltype(line)::value>;
            if ((err = prepare_kernel(kernel, smem)) != cudaSuccess) return;
            kernel<<<grid, kThreadsF, smem, s>>>(p, (float*)out, (float*)lse);
            err = cudaGetLastError();
        });
    });
    simt_count_launch(1);
    return (int)err;
}

int fma_fused_bwd(int dtype, const Geo& g, const void* q, const void* k, const void* v, const void* out, const void* lse,
                  const void* dout, const void* dlse, void* dq, void* dk, void* dv, void* workspace, cudaStream_t s)
{
    if (dtype != 0 || g.Dv != g.D || !vec_rows(q, g.qs, 4) || !vec_rows(k, g.ks, 4) || !vec_rows(v, g.vs, 4)) return -2;
    for (const void* p : {out, dout, (const void*)dq, (const void*)dk, (const void*)dv})
        if (reinterpret_cast<uintptr_t>(p) & 15u) return -2;
    FmaParams pq, pk;
    dim3 gq, gk;
    size_t sq, sk;
    if (!make_fma(g, pq, false, 2, 0, 0, kQueryChunk, gq, sq) || !make_fma(g, pk, true, 2, 8, 0, kKeyChunk, gk, sk)) return -2;
    float* delta = static_cast<float*>(workspace);
    pq.row1 = tensor_of(q, g.qs);
    pq.row2 = dense(dout, g, g.Hq, g.D);
    pq.col1 = tensor_of(k, g.ks);
    pq.col2 = tensor_of(v, g.vs);
    pk.row1 = pq.col1;
    pk.row2 = pq.col2;
    pk.col1 = pq.row1;
    pk.col2 = pq.row2;
    cudaError_t err = cudaSuccess;
    with_dim(g.D, [&](auto dim) {
        with_line(g, [&](auto line) {
            constexpr int D = decltype(dim)::value;
            auto* kq = fma_bwd_q_kernel<float, D, decltype(line)::value>;
            auto* kk = fma_bwd_k_kernel<float, D, decltype(line)::value>;
            if ((err = prepare_kernel(kq, sq)) != cudaSuccess || (err = prepare_kernel(kk, sk)) != cudaSuccess) return;
            kq<<<gq, kThreadsF, sq, s>>>(pq, (const float*)out, (const float*)lse, (const float*)dlse, delta, (float*)dq);
            kk<<<gk, kThreadsF, sk, s>>>(pk, (const float*)lse, delta, (float*)dk, (float*)dv);
            err = cudaGetLastError();
        });
    });
    simt_count_launch(2);
    return (int)err;
}

namespace {
int elt_of(int dtype) { return dtype == 0 ? 4 : 2; }
template <typename F> void with_type(int dtype, F&& f)
{
    if (dtype == 0) f(float{});
    else if (dtype == 1) f(__half{});
    else f(__nv_bfloat16{});
}
// geometry of a split call on head dim g.D with a scale of its own
bool make_split(int dtype, const Geo& g, FmaParams& p, bool key_side, float scale, size_t fixed, dim3& grid, size_t& smem)
{
    // four CTAs share an SM while the rows' slots leave room for it
    const int budget = 54 * 1024 - (int)std::min<size_t>(fixed, 30 * 1024);
    if (dtype > 2 || !make_fma(g, p, key_side, 1, 0, fixed, budget, grid, smem)) return false;
    p.scale = scale;
    return smem <= 110 * 1024;
}
} // namespace

// Enough (query, head) rows for these kernels?  The general kernels spread a small problem over more blocks; theirs is a time
// per pair, and a block of these kernels lives as long as its window is large, however few blocks there are, so the two meet
// at a number of rows that hardly depends on the window.  Microseconds here | general, head dim 32:
//   scores, 16 bits   7 x 7: 3136 rows 13.0 | 10.2, 6400 14.4 | 15.6, 12544 13.3 | 28.2;  13 x 13: 3136 27 | 25, 6400 33 | 42;
//                     3 x 5 x 5: 4704 19.6 | 17.5, 6400 19.8 | 22.5;  33: 2000 11.6 | 6.6, 8000 11.8 | 15.2
//   scores, float32   7 x 7: 1600 10.9 | 7.6, 3136 11.1 | 10.5;  13 x 13: 1600 22.4 | 16.2, 3136 23.8 | 25.9 (larger head dims:
//                     the general kernel's time grows faster, so the line is on the safe side)
//   apply, 16 bits    7 x 7: 6400 15.3 | 15.5, 12544 15.3 | 28.7;  13 x 13: 6400 43 | 41, 12544 35 | 83;
//                     3 x 5 x 5: 6400 25 | 22, 12800 27 | 42;  33: 8000 11.6 | 15.3
//   gather, 16 bits   7 x 7: 6400 25.7 | 22.1, 12544 25.6 | 36.9;  13 x 13: 6400 73 | 56, 12544 87 | 101;
//                     3 x 5 x 5: 6400 53 | 39, 12800 57 | 60;  3 x 3: 3136 8.4 | 7.3, 12544 8.8 | 18.8
//   apply and gather, float32   784 rows 13.2 | 33 and 22.4 | 30;  3 x 3: 3136 6.2 | 10.7 and 6.7 | 9.3
bool enough_rows(const Geo& g, long long least) { return g.B * g.ltot * g.Hq >= least; }

// The same three products as tc_scores / tc_apply / tc_gather (tc_kernels.cuh), in fp32; unit stride.
int fma_scores(int dtype, const Geo& g, const void* x, const long long xs[3], const void* y, const long long ys[3], float scale,
               bool neg_inf, void* out, cudaStream_t s, const void* rpb)
{
    const int rows = 4 * 256 / g.D * kWarpsF;
    FmaParams p;
    dim3 grid;
    size_t smem;
    if (dtype > 2 || !enough_rows(g, dtype == 0 ? 3000 : 8000) || !vec_rows(x, xs, elt_of(dtype)) || !vec_rows(y, ys, elt_of(dtype)) ||
        !make_split(dtype, g, p, false, scale, (size_t)rows * g.ktot * elt_of(dtype), grid, smem))
        return -2;
    if (rpb) {
        if (g.Hq != g.Hkv) return -2;
        for (int a = 0; a < g.rank; ++a)
            if (g.causal[a] || (g.K[a] & 1) == 0) return -2;
    }
    p.row1 = tensor_of(x, xs);
    p.col1 = tensor_of(y, ys);
    cudaError_t err = cudaSuccess;
    with_type(dtype, [&](auto type) {
        with_dim(g.D, [&](auto dim) {
            with_line(g, [&](auto line) {
                using T = decltype(type);
                auto* kernel = rpb ? fma_scores_kernel<T, decltype(dim)::value, decltype(line)::value, true>
                                   : fma_scores_kernel<T, decltype(dim)::value, decltype(line)::value, false>;
                if ((err = prepare_kernel(kernel, smem)) != cudaSuccess) return;
                kernel<<<grid, kThreadsF, smem, s>>>(p, (T*)out, neg_inf ? -INFINITY : 0.f, (const T*)rpb);
                err = cudaGetLastError();
            });
        });
    });
    simt_count_launch(1);
    return (int)err;
}

int fma_apply(int dtype, const Geo& g, const void* w, const void* y, const long long ys[3], float scale, void* out, cudaStream_t s)
{
    FmaParams p;
    dim3 grid;
    size_t smem;
    if (dtype > 2 || !enough_rows(g, dtype == 0 ? 800 : 8000) || !vec_rows(y, ys, elt_of(dtype)) || (reinterpret_cast<uintptr_t>(out) & 15u) ||
        !make_split(dtype, g, p, false, scale, 0, grid, smem))
        return -2;
    p.col1 = tensor_of(y, ys);
    cudaError_t err = cudaSuccess;
    with_type(dtype, [&](auto type) {
        with_dim(g.D, [&](auto dim) {
            with_line(g, [&](auto line) {
                using T = decltype(type);
                auto* kernel = fma_apply_kernel<T, decltype(dim)::value, decltype(line)::value>;
                if ((err = prepare_kernel(kernel, smem)) != cudaSuccess) return;
                kernel<<<grid, kThreadsF, smem, s>>>(p, (const T*)w, (T*)out);
                err = cudaGetLastError();
            });
        });
    });
    simt_count_launch(1);
    return (int)err;
}

int fma_gather(int dtype, const Geo& g, const void* w, const void* x, const long long xs[3], float scale, void* dst, cudaStream_t s)
{
    FmaParams p;
    dim3 grid;
    size_t smem;
    if (dtype > 2 || !enough_rows(g, dtype == 0 ? 800 : 12000) || !vec_rows(x, xs, elt_of(dtype)) ||
        (reinterpret_cast<uintptr_t>(dst) & 15u) || g.ltot * g.Hq * g.ktot >= (1ll << 31) ||                // 32-bit offsets
        !make_split(dtype, g, p, true, scale, 0, grid, smem))
        return -2;
    p.col1 = tensor_of(x, xs);
    cudaError_t err = cudaSuccess;
    with_type(dtype, [&](auto type) {
        with_dim(g.D, [&](auto dim) {
            with_line(g, [&](auto line) {
                using T = decltype(type);
                auto* kernel = fma_gather_kernel<T, decltype(dim)::value, decltype(line)::value>;
                if ((err = prepare_kernel(kernel, smem)) != cudaSuccess) return;
                kernel<<<grid, kThreadsF, smem, s>>>(p, (const T*)w, (T*)dst);
                err = cudaGetLastError();
            });
        });
    });
    simt_count_launch(1);
    return (int)err;
}

} // namespace natten
