// Fused neighbourhood-attention forward for head dims up to 128 on tcgen05 tensor cores (sm_100a),
// built from small persistent CTAs: four of them share an SM up to head dim 64 (two where there are few tiles), two above it, each working
// on one tile of 128 queries at a time (tiles blockIdx.x, + gridDim.x, ...).
//
// Per tile the union of the queries' neighbourhoods is a box of keys walked in chunks of 64 keys
// (additional tokens follow as extra chunks):
//   S = Q K^T                    tcgen05.mma (N = 64), Q / K tiles staged by TMA, S in TMEM
//   P = exp2(S*scale*log2e - m)  one thread per query row; the row's 64 scores are read from TMEM in
//                                16-column pieces (a piece that is empty for the whole warp is skipped),
//                                masked, and written back as 16-bit P over the scores they came from
//   O += P V                     tcgen05.mma with A = P from TMEM, V tile read MN-major, O in TMEM
// The chunk rows are interleaved (chunk c holds the key rows c, c + n, c + 2n, ... of the box), so every
// chunk carries a share of every warp's window and the four warps of a tile finish a chunk together.
// A row's stabiliser m is fixed at the first valid columns it meets and only moves if a later score
// exceeds it by 2^60 (2^14 for fp16); O, the row sum and the probabilities already stored for the
// chunk are then rescaled.  Up to head dim 64 four independent CTAs per SM give the schedulers sixteen
// softmax warps in different phases of their tiles, which is what hides the TMEM / barrier / MMA latencies
// (128 TMEM columns and 55 KB of shared memory per CTA).  Above it only two CTAs fit (256 columns, 103 KB),
// so the scores get two buffers there: S(c + 1) is computed while the threads work on S(c).
//
// Eight warps: four of softmax (a warpgroup), one that issues the products, one that loads, one for the geometry, one idle (a
// register split goes by warpgroups).  What bounds it is the chain of a chunk, not an issue rate: S -> softmax -> P -> the
// issuing warp -> P V and the next S, about 2800 cycles of which the softmax is 1500; four tiles in flight per SM share the
// gaps.  Counters at 64 x 64, 7 x 7: issue slots 49 %, tensor pipe active in 26 % of the cycles, DRAM 26 %; head dim 128, window 255:
// 40, 29, 21 %.  So whatever is not the chain is kept off the issuing warp and the softmax warps.  Measured on one B200 (us), one warp that
// loaded, issued and did the geometry | loads and geometry apart (kernel alone): 64 x 64, 7 x 7, 8 heads of 64, batch 8,
// bf16 61.7 | 50.2; 128 x 128, 13 x 13, dilation 2, batch 4 196 | 174; 16 x 32 x 32, 3 x 7 x 7, causal frames, batch 2 137 | 117 (103 with
// its chunks interleaved, see make_plan); 135 x 241, 7 x 9, 6 heads of 32, batch 2, fp16 80 | 68; 8191 causal, window 255, 16 heads of
// 128 on 4, batch 2 98 | 84.6 (74 with heads packed, see make_packed_plan).
//
// TMEM columns: head dim 64: S [0,64) (P over [0,32)), O [64,128);
//               head dim 128: S of even chunks [0,64), of odd chunks [64,128), O [128,256).
#include "tc_kernels.cuh"

#include "tc_fwd_geom.cuh"
#include "tc_plan.cuh"

#include <type_traits>

namespace natten {

using namespace tc;
using namespace tcplan;
using namespace fwdgeom;

namespace {

constexpr int kKeys = 64;                   // keys per chunk
constexpr int kKeysLog = 6;
constexpr int kStages = 2;
constexpr int kThreads = 256;               // 4 softmax warps; one that issues the products, one that loads, one for the geometry
constexpr uint32_t kColS = 0;
// Up to this many tiles an SM, head dims up to 64 run with two score buffers and two CTAs an SM, too: there is nothing else to fill a
// chunk's gaps.  7 x 7, one buffer | two: 28 x 28, 8 heads of 32 (56 tiles) 12.2 | 10.6 us, 16 heads of 64 (112) 13.8 | 11.9; batch 2,
// 16 heads of 32 (224) 14.0 | 12.8; 48 x 60, 6 heads of 64 (270) 15.2 | 13.6.  Above it the second buffer costs a second wave.
constexpr unsigned kFewTiles = 2;

// Shared memory and TMEM of one CTA for head dim DH: four CTAs per SM with 128 TMEM columns each, or two with 256 and two score buffers
// (head dim 128, and 64 where there are few tiles).  Tiles are stored as blocks of 64 channels (128-byte rows, 128-byte swizzle).
template <int DH, bool TWO_S>
struct FwdSmall {
    static constexpr int kHalves = DH / 64;
    static constexpr int kQHalf = kTileRows * 128;          // [128 x 64] 16-bit
    static constexpr int kKVHalf = kKeys * 128;             // [64 x 64] 16-bit
    static constexpr int kQBytes = kQHalf * kHalves;
    static constexpr int kKVBytes = kKVHalf * kHalves;
    static constexpr int kOffQ = 0, kOffK = kQBytes, kOffV = kQBytes + kStages * kKVBytes;
    static constexpr int kBar = kQBytes + 2 * kStages * kKVBytes;
    static constexpr int kTab = kBar + 208;
    static constexpr int kSmemTotal = kTab + 2 * kTabBytes;
    // Two score buffers where TMEM has the room: S(c + 1) is computed while the threads turn S(c) into probabilities.  With four CTAs
    // an SM (one buffer, 128 columns each) the CTAs fill each other's gaps instead.
    static constexpr bool kTwoS = TWO_S;
    static constexpr uint32_t kTmemCols = kTwoS ? 256 : 128;        // S, O, rounded up to a power of two
    static constexpr int kPerSm = kTwoS ? 2 : 4;
    // 65536 / kPerSm / kThreads registers a thread at launch, 64 or 128; the helpers hand what they do not need to the softmax
    // warps, which spill with less than 88 (32 | 96, where the helpers spill: 64 x 64, 7 x 7 53.7 us instead of 49.8)
    static constexpr int kHelperRegs = kTwoS ? 104 : 40, kSoftmaxRegs = kTwoS ? 152 : 88;
    // There K has to be a chunk ahead of V, so the two are loaded and freed apart; with one score buffer they come and go together.
    static constexpr bool kSplitKV = kTwoS;
    static constexpr uint32_t kColO = kTwoS ? 128 : 64;
};

// kShort: the last 32 of the DH channels are padding.
template <int DH, bool BF16, int kInner, bool kShort, bool TWO_S>
__global__ void __launch_bounds__(kThreads, FwdSmall<DH, TWO_S>::kPerSm)
tc_fwd_small_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmEK,
                    const __grid_constant__ CUtensorMap tmEV, const __grid_constant__ TcParams P,
                    uint16_t* __restrict__ out, float* __restrict__ lse)
{
    using FS = FwdSmall<DH, TWO_S>;
    constexpr int kHalves = FS::kHalves, kQHalf = FS::kQHalf, kKVHalf = FS::kKVHalf, kQBytes = FS::kQBytes, kKVBytes = FS::kKVBytes;
    constexpr int kOffQ = FS::kOffQ, kOffK = FS::kOffK, kOffV = FS::kOffV, kBar = FS::kBar, kTab = FS::kTab;
    constexpr uint32_t kTmemCols = FS::kTmemCols, kColO = FS::kColO;
    constexpr bool kTwoS = FS::kTwoS, kSplitKV = FS::kSplitKV;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int prior_abort = *reinterpret_cast<volatile int*>(P.status);

    const uint32_t sbase = smem_u32(smem);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kBar + 192);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBar + 200);
    const uint32_t bar_q = sbase + kBar + 0;            // Q tile landed
    const uint32_t bar_qfree = sbase + kBar + 8;        // last Q K^T of the tile finished: Q may be overwritten
    const uint32_t bar_k = sbase + kBar + 16;           // [2] K chunk landed
    const uint32_t bar_v = sbase + kBar + 32;           // [2] V chunk landed
    const uint32_t bar_kfree = sbase + kBar + 48;       // [2] Q K^T of the chunk finished: its K may be overwritten
    const uint32_t bar_vfree = sbase + kBar + 64;       // [2] P V of the chunk finished: its V may be overwritten
    const uint32_t bar_s = sbase + kBar + 80;           // [2] S of the chunk is in TMEM (one score buffer: and every earlier product is done)
    const uint32_t bar_p = sbase + kBar + 96;           // [2] every thread stored its P
    const uint32_t bar_o = sbase + kBar + 112;          // last P V of the tile finished
    const uint32_t bar_head = sbase + kBar + 120;       // [2] geometry of the CTA's t-th tile published
    const uint32_t bar_tab_full = sbase + kBar + 136;   // [2] ... and its tables
    const uint32_t bar_tab_empty = sbase + kBar + 152;  // [2] ... read by the softmax threads and the other helpers
    // chunk n (counted over the CTA's whole run) -> its score columns, barriers and wait parity
    auto s_cols = [&](unsigned n) -> uint32_t { return kTwoS ? 64u * (n & 1u) : 0u; };
    auto bar_s_of = [&](unsigned n) -> uint32_t { return bar_s + (kTwoS ? 8u * (n & 1u) : 0u); };
    auto bar_p_of = [&](unsigned n) -> uint32_t { return bar_p + (kTwoS ? 8u * (n & 1u) : 0u); };
    auto par_of = [&](unsigned n) -> uint32_t { return kTwoS ? ((n >> 1) & 1u) : (n & 1u); };
    auto tab_slot = [&](unsigned t) { return reinterpret_cast<FwdTile*>(smem + kTab + (t & 1) * kTabBytes); };

    if (warp == 4) {
        if (lane == 0) {
            // swizzled tiles need a 1024-byte aligned base; once any CTA has given up, the rest bail out
            *abort_flag = ((sbase & 1023u) || prior_abort) ? 1 : 0;
            mbar_init(bar_q, 1);
            mbar_init(bar_qfree, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(bar_k + 8 * i, 1);
                mbar_init(bar_v + 8 * i, 1);
                mbar_init(bar_kfree + 8 * i, 1);
                mbar_init(bar_vfree + 8 * i, 1);
                mbar_init(bar_s + 8 * i, 1);
                mbar_init(bar_p + 8 * i, 128);
                mbar_init(bar_head + 8 * i, 1);
                mbar_init(bar_tab_full + 8 * i, 32);
                mbar_init(bar_tab_empty + 8 * i, 130);
            }
            mbar_init(bar_o, 1);
            mbar_init_fence();
            fence_async_smem();
        }
        __syncwarp();
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    } else if (warp == 5 && lane == 0) {
        prefetch_map(&tmQ);
        prefetch_map(&tmK);
        prefetch_map(&tmV);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const unsigned nwork = P.work_q;
    if (warp >= 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FS::kHelperRegs));
        if (warp == 4) {
            // =====================================================================
            // MMA issue.  The whole warp walks the CTA's tiles; the tensor-core instructions execute on one elected lane.  What it
            // does between a chunk's last probability and the next chunk's scores is on the chain of every chunk, so the loads
            // and the geometry are other warps', descriptors are ready and the next chunk's operands have been waited for.
            // =====================================================================
            if (!gave_up(abort_flag)) {
                constexpr uint32_t idesc_qk = instr_desc(BF16 ? 1 : 0, kKeys, 0, 0);
                constexpr uint32_t idesc_pv = instr_desc(BF16 ? 1 : 0, DH, 0, 1);
                const uint64_t dq0 = smem_desc(sbase + kOffQ, 16, 1024);
                const uint64_t dk_even = smem_desc(sbase + kOffK, 16, 1024), dk_odd = smem_desc(sbase + kOffK + kKVBytes, 16, 1024);
                const uint64_t dv_even = smem_desc(sbase + kOffV, kKVHalf, 1024), dv_odd = smem_desc(sbase + kOffV + kKVBytes, kKVHalf, 1024);
                const uint32_t leader = elect_one();
                bool ok = true;
                unsigned n_qk = 0, n_pv = 0;
                for (unsigned t = 0;; ++t) {
                    ok = warp_wait(bar_head + 8 * (t & 1), (t >> 1) & 1, abort_flag, P.wait_budget);
                    if (!ok) break;
                    const FwdTile* H = tab_slot(t);
                    const int nch = H->nch;
                    int nnb = 0, lo[3] = {0, 0, 0}, Lp[3] = {0, 0, 0}, nc[3] = {1, 1, 1};
                    bool padded = false;             // some chunk reaches past the sample's extent: those rows are zeroed
                    if (P.extents) {
                        nnb = H->nnb;
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            lo[a] = H->lo[a]; Lp[a] = H->Lp[a]; nc[a] = H->nc[a];
                            padded = padded || lo[a] + chunk_coord(P, a, nc[a] - 1, P.cb[a] - 1) >= Lp[a];
                        }
                    }
                    __syncwarp();                    // every lane has read the header
                    if (leader) mbar_arrive(bar_tab_empty + 8 * (t & 1));
                    if (nch == 0) break;
                    auto zero_padding = [&](int c, uint8_t* tile) {
                        if (c >= nnb) return;
                        const int c2 = c % nc[2], c1 = c / nc[2] % nc[1], c0 = c / nc[2] / nc[1];
                        const int box0[3] = {lo[0] + chunk_coord(P, 0, c0, 0), lo[1] + chunk_coord(P, 1, c1, 0), lo[2] + chunk_coord(P, 2, c2, 0)};
                        if (leader) zero_rows_past_extent(P, box0, Lp, kKeys, kHalves, kKVHalf, tile, tile);
                    };
                    auto wait_k = [&](int c) {       // chunk c's K has landed (and ends where the sample ends)
                        const unsigned s = n_qk & 1u;
                        ok = ok && mbar_wait(bar_k + 8 * s, (n_qk >> 1) & 1, abort_flag, P.wait_budget);
                        if (ok && padded) zero_padding(c, smem + kOffK + s * kKVBytes);
                    };
                    auto issue_qk = [&](bool last) {
                        const uint64_t dk0 = (n_qk & 1u) ? dk_odd : dk_even;
#pragma unroll
                        for (int ks = 0; ks < (kShort ? DH / 16 - 2 : DH / 16); ++ks) {     // 32 bytes per k-step inside a 64-channel block
                            mma_ss_e(tmem + kColS + s_cols(n_qk), dq0 + ((((ks / 4) * kQHalf) + (ks % 4) * 32) >> 4),
                                     dk0 + ((((ks / 4) * kKVHalf) + (ks % 4) * 32) >> 4), idesc_qk, ks > 0, leader);
                        }
                        mma_commit_e(bar_s_of(n_qk), leader);
                        if (kSplitKV) mma_commit_e(bar_kfree + 8 * (n_qk & 1u), leader);
                        if (last) mma_commit_e(bar_qfree, leader);        // last scores of the tile: Q may go once they are done
                        ++n_qk;
                    };
                    ok = mbar_wait(bar_q, t & 1, abort_flag, P.wait_budget);
                    wait_k(0);
                    tc_fence_after();
                    if (ok) issue_qk(nch == 1);
                    for (int c = 0; c < nch; ++c) {
                        const bool more = c + 1 < nch;
                        if (more) wait_k(c + 1);
                        // two score buffers: S(c + 1) goes into the other buffer while the threads work on S(c); that
                        // buffer's P(c - 1) is read by a product issued earlier from this warp, so the order holds
                        if (kTwoS && more && ok) { tc_fence_after(); issue_qk(c + 2 == nch); }
                        const unsigned sv = n_pv & 1u;
                        if (kSplitKV) ok = ok && mbar_wait(bar_v + 8 * sv, (n_pv >> 1) & 1, abort_flag, P.wait_budget);
                        if (ok && padded) zero_padding(c, smem + kOffV + sv * kKVBytes);
                        ok = ok && mbar_wait(bar_p_of(n_pv), par_of(n_pv), abort_flag, P.wait_budget);      // P(c) stored over S(c)
                        if (!ok) break;
                        tc_fence_after();
                        // V read MN-major: 16 key rows per k-step; P sits as 16-bit pairs in the first 32 S columns
                        const uint64_t dv0 = sv ? dv_odd : dv_even;
#pragma unroll
                        for (int ks = 0; ks < kKeys / 16; ++ks)
                            mma_ts_e(tmem + kColO, tmem + kColS + s_cols(n_pv) + 8 * ks, dv0 + 128 * ks, idesc_pv, (c > 0 || ks > 0) ? 1u : 0u, leader);
                        mma_commit_e(bar_vfree + 8 * sv, leader);
                        if (!kTwoS && more) issue_qk(c + 2 == nch);      // after P(c) has been read (issue order): over it
                        if (!more) mma_commit_e(bar_o, leader);
                        ++n_pv;
                    }
                    // the lanes agree once a tile, not at every wait: nothing in between is for the whole warp, and a vote there is on
                    // every chunk's chain (8 lengths up to 16384, window 255, 16 heads of 128 on 4: key side 601 us without any, 606
                    // like this, 611 with a vote in every wait)
                    if (!__all_sync(0xffffffffu, ok)) break;
                }
            }
        } else if (warp == 5) {
            // =====================================================================
            // Loads: Q of a tile, then its chunks; both run ahead across tile boundaries as far as the buffers allow.
            // =====================================================================
            if (!gave_up(abort_flag)) {
                bool ok = true;
                unsigned n = 0;                                  // chunks loaded
                for (unsigned t = 0;; ++t) {
                    ok = warp_wait(bar_head + 8 * (t & 1), (t >> 1) & 1, abort_flag, P.wait_budget);
                    if (!ok) break;
                    const FwdTile* H = tab_slot(t);
                    const int b = H->b, h = H->h, hk = H->hk, nnb = H->nnb, nch = H->nch, nc1 = H->nc[1], nc2 = H->nc[2];
                    const int X0 = H->rg[0] + P.dil[0] * H->lo[0], X1 = H->rg[1] + P.dil[1] * H->lo[1], X2 = H->rg[2] + P.dil[2] * H->lo[2];
                    const int Q0 = H->rg[0] + P.dil[0] * (H->x0[0] + H->sx[0] * H->origin[0]),
                              Q1 = H->rg[1] + P.dil[1] * (H->x0[1] + H->sx[1] * H->origin[1]),
                              Q2 = H->rg[2] + P.dil[2] * (H->x0[2] + H->sx[2] * H->origin[2]);
                    __syncwarp();                                // every lane has read the header
                    if (lane == 0) mbar_arrive(bar_tab_empty + 8 * (t & 1));
                    if (nch == 0) break;
                    if (t > 0) ok = warp_wait(bar_qfree, (t - 1) & 1, abort_flag, P.wait_budget);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(bar_q, kQBytes + ((P.inject == 1 && t == 0) ? 16u : 0u));
#pragma unroll
                        for (int hf = 0; hf < kHalves; ++hf)
                            tma_load_rows(sbase + kOffQ + hf * kQHalf, &tmQ, bar_q, P, h, 64 * hf, Q2, Q1, Q0, b);
                    }
                    int c0 = 0, c1 = 0, c2 = 0;
                    for (int c = 0; c < nch; ++c, ++n) {
                        const unsigned s = n & 1u, parity = ((n >> 1) - 1) & 1;
                        const bool box = c < nnb;                // else additional tokens (rows past n_extra are zero-filled)
                        const int x0 = box ? X0 + P.dil[0] * chunk_coord(P, 0, c0, 0) : 0, x1 = box ? X1 + P.dil[1] * chunk_coord(P, 1, c1, 0) : 0,
                                  x2 = box ? X2 + P.dil[2] * chunk_coord(P, 2, c2, 0) : (c - nnb) * kKeys;
                        if (++c2 == nc2) { c2 = 0; if (++c1 == nc1) { c1 = 0; ++c0; } }
                        if (n >= (unsigned)kStages) ok = warp_wait((kSplitKV ? bar_kfree : bar_vfree) + 8 * s, parity, abort_flag, P.wait_budget);
                        if (!ok) break;
                        const uint32_t full_k = bar_k + 8 * s, full_v = (kSplitKV ? bar_v : bar_k) + 8 * s;
                        if (lane == 0) {
                            mbar_expect_tx(full_k, kSplitKV ? kKVBytes : 2 * kKVBytes);
#pragma unroll
                            for (int hf = 0; hf < kHalves; ++hf)
                                tma_load_heads(sbase + kOffK + s * kKVBytes + hf * kKVHalf, box ? &tmK : &tmEK, full_k, P, hk, 64 * hf, x2, x1, x0, b);
                        }
                        __syncwarp();
                        if (kSplitKV && n >= (unsigned)kStages) ok = warp_wait(bar_vfree + 8 * s, parity, abort_flag, P.wait_budget);
                        if (!ok) break;
                        if (lane == 0) {
                            if (kSplitKV) mbar_expect_tx(full_v, kKVBytes);
#pragma unroll
                            for (int hf = 0; hf < kHalves; ++hf)
                                tma_load_heads(sbase + kOffV + s * kKVBytes + hf * kKVHalf, box ? &tmV : &tmEV, full_v, P, hk, 64 * hf, x2, x1, x0, b);
                        }
                        __syncwarp();
                    }
                    if (!ok) break;
                }
            }
        } else if (warp == 6) {
            // =====================================================================
            // Geometry: the CTA's tiles (blockIdx.x, + gridDim.x, ...), each one's tables as soon as its slot is free.  Rows of padding
            // tiles (per-sample extents) are zeroed here.
            // =====================================================================
            if (!gave_up(abort_flag)) {
                auto zero_rows = [&](const Cursor& at) {     // rows of a padding tile that exist in the output are zero
                    for_each_row(P, at, lane, [&](long long out_row) {
                        uint4* o4 = reinterpret_cast<uint4*>(out + out_row * P.dreal);
#pragma unroll
                        for (int i = 0; i < DH / 8; ++i)
                            if (8 * i < P.dreal) o4[i] = make_uint4(0, 0, 0, 0);
                        lse[out_row] = 0.f;
                    });
                };
                bool ok = true, found = true;
                Cursor cur;
                cur.init(P, blockIdx.x, gridDim.x);
                for (unsigned t = 0; ok && found; ++t) {
                    if (t >= 2) ok = warp_wait(bar_tab_empty + 8 * (t & 1), ((t >> 1) - 1) & 1, abort_flag, P.wait_budget);
                    if (!ok) break;
                    FwdTile* H = tab_slot(t);
                    found = false;
                    while (cur.w < nwork && !found) {
                        found = publish_tile(P, cur, kKeysLog, kInner == 16, lane, H);
                        if (!found && P.extents) zero_rows(cur);
                        cur.advance(P, gridDim.x);
                    }
                    if (!found && lane == 0) H->nch = 0;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_head + 8 * (t & 1));
                    if (found) write_tables(P, lane, reinterpret_cast<uint8_t*>(H));
                    mbar_arrive(bar_tab_full + 8 * (t & 1));
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FS::kSoftmaxRegs));
        // =====================================================================
        // softmax warps: thread = one query row, the chunk's 64 columns in 16-column pieces
        // =====================================================================
        const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
        constexpr float kGrow = BF16 ? 60.f : 14.f;      // exponent headroom of the stored probabilities
        constexpr float kGrowSum = BF16 ? 1.152921504606847e18f : 16384.f;      // 2^kGrow: a piece's row sum below it has no probability above it
        // With 16-column inner rows every piece is one inner row of the chunk: a piece is either inside the
        // row's window along the outer axes or not (one bit), and which of its 16 columns are valid is the
        // same for every piece.  The column mask then lives in the addends of the scale-and-shift, one
        // register per column: -m*scale*log2e inside the window, -inf outside.
        constexpr bool kRows16 = kInner == 16;
        bool ok = true;
        unsigned n = 0;                      // chunks processed so far (all tiles of this CTA)
        uint32_t scol = trow + kColS;        // TMEM address of this row's scores of the current chunk
        float m = -INFINITY, l = 0.f;
        float add[16];
        uint32_t add_cols = 0u;              // column mask the addends were built for
#pragma unroll
        for (int i = 0; i < 16; ++i) add[i] = -INFINITY;
        auto refresh_add = [&](uint32_t cols) {
            const float nmb = (m == -INFINITY) ? 0.f : -m * P.scale_log2;
#pragma unroll
            for (int i = 0; i < 16; ++i) add[i] = ((cols >> i) & 1u) ? nmb : -INFINITY;
            add_cols = cols;
        };
        // rare: a score far above the stabiliser.  Move it; rescale O, the row sum and the probabilities this
        // chunk has stored so far (every earlier product has finished).  `grow`: this row is the cause.
        auto rescale = [&](bool grow, float xmax, int c, int pc, uint32_t stored) {
            const float fac = grow ? fast_exp2(-xmax) : 1.f;
            if (c > 0) {
                // with two score buffers S(c) was issued before P V of chunk c - 1: wait for that product itself
                if (kTwoS) {
                    ok = mbar_wait(bar_vfree + 8 * ((n - 1) & 1u), par_of(n - 1), abort_flag, P.wait_budget) && ok;
                    tc_fence_after();
                }
#pragma unroll 1
                for (int part = 0; part < DH / 16; ++part) {
                    uint32_t o[16];
                    tmem_ld16(trow + kColO + 16 * part, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * fac);
                    tmem_st16(trow + kColO + 16 * part, o);
                }
            }
#pragma unroll 1
            for (int pp = 0; pp < pc; ++pp) {
                if (!((stored >> pp) & 1u)) continue;
                uint32_t old[8];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(old[0]), "=r"(old[1]), "=r"(old[2]), "=r"(old[3]), "=r"(old[4]), "=r"(old[5]),
                               "=r"(old[6]), "=r"(old[7])
                             : "r"(scol + 8 * pp) : "memory");
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float lo, hi;
                    if (BF16) {
                        lo = __uint_as_float(old[i] << 16);
                        hi = __uint_as_float(old[i] & 0xFFFF0000u);
                    } else {
                        const __half2 h2 = *reinterpret_cast<const __half2*>(&old[i]);
                        lo = __low2float(h2);
                        hi = __high2float(h2);
                    }
                    old[i] = cvt_pack<BF16>(lo * fac, hi * fac);
                }
                tmem_st8(scol + 8 * pp, old);
            }
            l *= fac;
            if (grow) m += xmax / P.scale_log2;
        };

        for (unsigned t = 0;; ++t) {
            ok = mbar_wait(bar_tab_full + 8 * (t & 1), (t >> 1) & 1, abort_flag, P.wait_budget) && ok;
            if (!__all_sync(0xffffffffu, ok)) break;
            const FwdTile* H = tab_slot(t);
            const int nch = H->nch;
            if (nch == 0) break;
            // ---- this thread's query row, from the geometry warp's tables ----
            const int nnb = H->nnb, nc1 = H->nc[1], nc2 = H->nc[2];
            const bool mapped = kRows16 && H->mapped;
            int f[3], e[3];
            bool valid_q, in_tensor;
            unsigned long long rowmap;
            uint32_t colbits;                    // 16-column rows: one bit per column
            const long long out_row = row_from_tables(P, reinterpret_cast<const uint8_t*>(H), warp * 32 + lane, f, e, valid_q, in_tensor, rowmap, colbits);
            mbar_arrive(bar_tab_empty + 8 * (t & 1));
            m = -INFINITY;
            l = 0.f;
            add_cols = 0xffffffffu;              // the addends belong to the previous tile's stabiliser
            int ci[3] = {0, 0, 0};
            const bool line = line_chunks(P);    // chunks are runs of the innermost axis (1-D windows): cheap validity words
            int jl[3] = {0, 0, 0}, jh[3] = {0, 0, 0};
            uint32_t rowbits = 0u, dirty = 7u;   // 16-column rows: one bit per piece
            for (int c = 0; c < nch; ++c, ++n) {
                // ---- validity of this row's columns in this chunk ----
                // jl/jh (columns of the chunk inside the row's window, per axis) only change along the axes whose
                // chunk index moved since the last chunk: `dirty` has a bit per axis.
                const bool extra = c >= nnb;   // additional tokens: every live row sees the first n_extra columns
                uint32_t words[2] = {0u, 0u};    // generic form: one bit per column
                if (extra) {
#pragma unroll
                    for (int pc = 0; pc < 2; ++pc)
                        words[pc] = valid_q ? low_bits(P.n_extra - ((c - nnb) * kKeys + 32 * pc)) : 0u;
                } else if (mapped) {
                    rowbits = (uint32_t)(rowmap >> (4 * c)) & 15u;
                } else {
                    if (kInner == 0 && line) {
#pragma unroll
                        for (int pc = 0; pc < 2; ++pc) words[pc] = line_word(P, pc, ci, f, e);
                    } else {
#pragma unroll
                        for (int a = 0; a < 3; ++a)
                            if ((dirty >> a) & 1u) chunk_range(P, a, ci[a], f[a], e[a], jl[a], jh[a]);
                        if constexpr (kInner > 0) {
                            // inner rows of the chunk (kInner columns each) are numbered r = j0 * cb1 + j1
                            if (dirty & 3u) {
                                const uint32_t m1 = jh[1] > jl[1] ? (low_bits(jh[1]) & ~low_bits(jl[1])) : 0u;
                                rowbits = 0u;
                                for (int j0 = jl[0]; j0 < jh[0]; ++j0) rowbits |= m1 << (j0 << P.cb1_log);
                            }
                            if (dirty & 4u) colbits = jh[2] > jl[2] ? (low_bits(jh[2]) & ~low_bits(jl[2])) : 0u;
                            if constexpr (!kRows16) {
#pragma unroll
                                for (int pc = 0; pc < 2; ++pc) words[pc] = ((rowbits >> pc) & 1u) ? colbits : 0u;
                            }
                        } else {
#pragma unroll
                            for (int pc = 0; pc < 2; ++pc) words[pc] = piece_word_ranges(P, pc, jl, jh);
                        }
                    }
                    dirty = 0u;
                }
                const bool fast = kRows16 && !extra;
                if (fast && colbits != add_cols) refresh_add(colbits);
                uint32_t mine = 0u, act = 0u;    // pieces inside this row's window, inside that of any row of the warp
                if (fast) {
                    mine = colbits != 0u ? rowbits & 15u : 0u;
                    act = __reduce_or_sync(0xffffffffu, mine);
                }

                scol = trow + kColS + s_cols(n);
                ok = ok && mbar_wait(bar_s_of(n), par_of(n), abort_flag, P.wait_budget);     // one score buffer: every earlier product has finished, too
                tc_fence_after();
                if (!__all_sync(0xffffffffu, ok)) { words[0] = 0u; words[1] = 0u; act = 0u; dirty = 7u; }

                uint32_t stored = 0u;            // pieces of this chunk that hold probabilities (bit per piece)
                // one 16-column piece on the general path: scores s, validity bits wd -> probabilities pk
                auto generic_piece = [&](int pc, uint32_t (&s)[16], uint32_t wd, uint32_t (&pk)[8]) {
                    if (m == -INFINITY && wd != 0u) {           // first valid columns of this row: fix the stabiliser
                        float mm = -INFINITY;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if ((wd >> i) & 1u) mm = fmaxf(mm, __uint_as_float(s[i]));
                        m = mm;
                        add_cols = 0xffffffffu;                 // the addends of the fast path are stale now
                    }
                    const float mb = (m == -INFINITY) ? 0.f : m * P.scale_log2;
                    // A piece that lies inside every row's window (most pieces of a long 1-D window) needs no
                    // masks and no running maximum: two columns per packed instruction, and the row sum tells
                    // whether any probability may have outgrown its stabiliser (then the general form redoes it).
                    bool done = false;
                    if (__all_sync(0xffffffffu, wd == 0xFFFFu)) {
                        const uint64_t sc2 = pack2(P.scale_log2, P.scale_log2), nb2 = pack2(-mb, -mb);
                        uint64_t rr = 0ull;
                        uint32_t pq[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const uint64_t xx = fma2(pack2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), sc2, nb2);
                            const float p0 = fast_exp2(lo_of(xx)), p1 = fast_exp2(hi_of(xx));
                            rr = add2(rr, pack2(p0, p1));
                            pq[i] = cvt_pack<BF16>(p0, p1);
                        }
                        const float rs = lo_of(rr) + hi_of(rr);
                        if (!__any_sync(0xffffffffu, !(rs <= kGrowSum))) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) pk[i] = pq[i];
                            l += rs;
                            stored |= 1u << pc;
                            done = true;
                        }
                    }
                    if (!done) {
                        float x[16], xmax = -INFINITY;
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            x[i] = fmaf(__uint_as_float(s[i]), P.scale_log2, -mb);
                            if (!((wd >> i) & 1u)) x[i] = -INFINITY;
                            xmax = fmaxf(xmax, x[i]);
                        }
                        const bool grow = xmax > kGrow;
                        if (__any_sync(0xffffffffu, grow)) {
                            rescale(grow, xmax, c, pc, stored);
                            if (grow) {
                                add_cols = 0xffffffffu;
#pragma unroll
                                for (int i = 0; i < 16; ++i) x[i] -= xmax;
                            }
                        }
                        float r0 = 0.f, r1 = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float p0 = fast_exp2(x[2 * i]), p1 = fast_exp2(x[2 * i + 1]);
                            r0 += p0;
                            r1 += p1;
                            pk[i] = cvt_pack<BF16>(p0, p1);
                        }
                        l += r0 + r1;
                        stored |= 1u << pc;
                    }
                };
                if (fast) {
                    // one 16-column row: scores s -> probabilities over the scores they came from (piece pc lands in columns this
                    // thread has already read)
                    auto row_piece = [&](int pc, uint32_t (&s)[16], uint32_t (&pk)[8]) {
                        const bool rowok = (mine >> pc) & 1u;
                        if (m == -INFINITY && rowok) {           // first valid columns of this row: fix the stabiliser
                            float mm = -INFINITY;
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                if ((colbits >> i) & 1u) mm = fmaxf(mm, __uint_as_float(s[i]));
                            m = mm;
                            refresh_add(colbits);
                        }
                        // No running maximum in the common case: the probabilities are formed at once and their
                        // row sum tells whether one of them may have outgrown the stabiliser; only then are the
                        // exponents looked at one by one (and, if it is so, everything rescaled and redone).
                        const uint64_t sc2 = pack2(P.scale_log2, P.scale_log2);
                        const uint32_t keep = rowok ? 0xffffffffu : 0u;     // rows outside their window store zeros
                        uint64_t rr = 0ull;                                 // two partial row sums
#pragma unroll
                        for (int i = 0; i < 8; ++i) {                       // two columns per packed fp32 fma
                            const uint64_t xx = fma2(pack2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), sc2, pack2(add[2 * i], add[2 * i + 1]));
                            const float p0 = fast_exp2(lo_of(xx)), p1 = fast_exp2(hi_of(xx));
                            rr = add2(rr, pack2(p0, p1));
                            pk[i] = cvt_pack<BF16>(p0, p1) & keep;
                        }
                        if (__any_sync(0xffffffffu, rowok && !(lo_of(rr) + hi_of(rr) <= kGrowSum))) {
                            float x[16], xmax = -INFINITY;
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                x[i] = fmaf(__uint_as_float(s[i]), P.scale_log2, add[i]);
                                xmax = fmaxf(xmax, x[i]);
                            }
                            const bool grow = rowok && xmax > kGrow;
                            if (__any_sync(0xffffffffu, grow)) {
                                rescale(grow, xmax, c, pc, stored);
                                if (grow) {
                                    refresh_add(colbits);
#pragma unroll
                                    for (int i = 0; i < 16; ++i) x[i] -= xmax;
                                }
                            }
                            rr = 0ull;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const float p0 = fast_exp2(x[2 * i]), p1 = fast_exp2(x[2 * i + 1]);
                                rr = add2(rr, pack2(p0, p1));
                                pk[i] = cvt_pack<BF16>(p0, p1) & keep;
                            }
                        }
                        if (rowok) l += lo_of(rr) + hi_of(rr);
                        stored |= 1u << pc;
                    };
#pragma unroll 1
                    for (int pc = 0; pc < 4; ++pc) {
                        uint32_t pk[8];
                        if ((act >> pc) & 1u) {
                            uint32_t s[16];
                            tmem_ld16(scol + 16 * pc, s);
                            tmem_ld_wait();
                            row_piece(pc, s, pk);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) pk[i] = 0u;
                        }
                        tmem_st8(scol + 8 * pc, pk);
                    }
                } else {
#pragma unroll 1
                    for (int pc = 0; pc < 4; ++pc) {
                        uint32_t pk[8];
                        const uint32_t wd = ((pc & 2) ? words[1] : words[0]) >> (16 * (pc & 1)) & 0xFFFFu;
                        if (__any_sync(0xffffffffu, wd != 0u)) {
                            uint32_t s[16];
                            tmem_ld16(scol + 16 * pc, s);
                            tmem_ld_wait();
                            generic_piece(pc, s, wd, pk);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) pk[i] = 0u;
                        }
                        // P over the scores it came from: piece pc lands in columns this thread has already read
                        tmem_st8(scol + 8 * pc, pk);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(bar_p_of(n));
                if (!mapped) {
                    ++ci[2];
                    dirty = 4u;
                    if (ci[2] == nc2) {
                        ci[2] = 0; ++ci[1]; dirty = nc2 > 1 ? 6u : 2u;
                        if (ci[1] == nc1) { ci[1] = 0; ++ci[0]; dirty = 1u | (nc1 > 1 ? 2u : 0u) | (nc2 > 1 ? 4u : 0u); }
                    }
                }
            }

            // ---- normalise and write out ----
            ok = mbar_wait(bar_o, t & 1, abort_flag, P.wait_budget) && ok;
            tc_fence_after();
            {
                const bool live = valid_q && ok;
                const float inv = (live && l > 0.f) ? 1.f / l : 0.f;
                // A thread holds a row, but 32 rows written 16 bytes at a time are 32 lines per store instruction (the stores of
                // the tile kept the load / store unit busy for 4200 cycles, 15 % of the kernel).  Four lanes exchange their
                // 16-byte pieces of 32 channels, so that a store writes 64 bytes of each of eight rows.
                const long long my_row = in_tensor ? out_row : -1;
                long long rows4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) rows4[i] = __shfl_sync(0xffffffffu, my_row, (lane & ~3) | i);
                const int piece = lane & 3;
#pragma unroll
                for (int part = 0; part < DH / 32; ++part) {
                    if (32 * part >= P.dreal) break;             // padded channels are not part of the output
                    uint32_t o[32], w[4][4];
                    tmem_ld32(trow + kColO + 32 * part, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            w[i][j] = live ? cvt_pack<BF16>(__uint_as_float(o[8 * i + 2 * j]) * inv, __uint_as_float(o[8 * i + 2 * j + 1]) * inv) : 0u;
                    transpose4(w, piece);                        // w[i]: this lane's piece of row i of the four
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (rows4[i] >= 0 && 32 * part + 8 * piece < P.dreal)
                            reinterpret_cast<uint4*>(out + rows4[i] * P.dreal)[4 * part + piece] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
                }
                // natural-log lse of scale * logits
                if (in_tensor)
                    lse[out_row] = (live && l > 0.f) ? (m * P.scale_log2 + log2f(l)) * 0.6931471805599453f : 0.f;
            }
            // the next tile's first P V is issued only after this thread has stored its next P
            tc_fence_before();
        }
    }

    if (*abort_flag) abort_grace_sleep();       // loads of a wait that gave up may still be landing
    tc_fence_before();
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
        if (lane == 0 && *abort_flag) raise_status(P);
    }
}

} // namespace

int tc_fused_fwd_small(int dtype, const Geo& g, const void* q, const void* k, const void* v, const void* ek,
                       const void* ev, void* out, void* lse, cudaStream_t s)
{
    if (g.D > 128) return -2;
    if (!tc_eligible(dtype, g, q, k, v, /*allow_stride=*/true)) return -2;
    if (g.n_extra > 0 && ((reinterpret_cast<uintptr_t>(ek) | reinterpret_cast<uintptr_t>(ev)) & 15u)) return -2;
    Plan plan;
    if (const int rc = make_packed_plan(g, plan, kKeys, /*with_stride=*/true, /*interleave=*/true, /*backward=*/false)) return rc;
    const bool bf16 = dtype == 2;
    CUtensorMap mq, mk, mv, mek, mev;
    if (!encode_map(&mq, q, bf16, plan.p, g.Hq, g.D, g.qs, plan.box_q, /*query_lattice=*/true, /*interleaved=*/false, /*rows=*/true) ||
        !encode_map(&mk, k, bf16, plan.p, g.Hkv, g.D, g.ks, plan.box_kv, false, /*interleaved=*/true) ||
        !encode_map(&mv, v, bf16, plan.p, g.Hkv, g.Dv, g.vs, plan.box_kv, false, /*interleaved=*/true))
        return -2;
    mek = mk; mev = mv;                      // placeholders when there are no additional tokens
    if (g.n_extra > 0 && (!encode_extra_map(&mek, ek, bf16, g.B, g.n_extra, g.Hkv, g.D, kKeys, plan.p.split_heads) ||
                          !encode_extra_map(&mev, ev, bf16, g.B, g.n_extra, g.Hkv, g.Dv, kKeys, plan.p.split_heads)))
        return -2;
    if (plan.p.work_q == 0 || g.B == 0) return 0;
    cudaError_t err = cudaSuccess;
    auto launch_as = [&](auto dh, auto bf, auto inner, auto shorter, auto two_s) {
        constexpr int kDh = decltype(dh)::value;
        using FS = FwdSmall<kDh, decltype(two_s)::value>;
        auto* kernel = tc_fwd_small_kernel<kDh, decltype(bf)::value, decltype(inner)::value, decltype(shorter)::value, decltype(two_s)::value>;
        const unsigned grid = persistent_grid(plan.p.work_q, FS::kPerSm);
        err = ensure_dynamic_smem((const void*)kernel, FS::kSmemTotal);
        if (err != cudaSuccess) return;
        kernel<<<grid, kThreads, FS::kSmemTotal, s>>>(mq, mk, mv, mek, mev, plan.p, (uint16_t*)out, (float*)lse);
    };
    auto launch = [&](auto dh, auto bf, auto inner, auto shorter) {
        if constexpr (decltype(dh)::value == 64) {
            if (plan.p.work_q > kFewTiles * (unsigned)sm_count()) return launch_as(dh, bf, inner, shorter, std::false_type{});
        }
        launch_as(dh, bf, inner, shorter, std::true_type{});
    };
    auto by_short = [&](auto dh, auto bf, auto inner) {
        if (g.D <= decltype(dh)::value - 32) launch(dh, bf, inner, std::true_type{});
        else launch(dh, bf, inner, std::false_type{});
    };
    auto by_inner = [&](auto dh, auto bf) {
        if (plan.p.cb[2] == 16) by_short(dh, bf, std::integral_constant<int, 16>{});
        else if (plan.p.cb[2] == 32) by_short(dh, bf, std::integral_constant<int, 32>{});
        else by_short(dh, bf, std::integral_constant<int, 0>{});
    };
    auto by_type = [&](auto dh) {
        if (bf16) by_inner(dh, std::true_type{});
        else by_inner(dh, std::false_type{});
    };
    if (g.D <= 64) by_type(std::integral_constant<int, 64>{});
    else by_type(std::integral_constant<int, 128>{});
    if (err == cudaSuccess) err = cudaGetLastError();
    tc_count_launch();
    return err == cudaSuccess ? 0 : (int)err;
}

// launches of the tensor-core kernels, counted on the host by every launcher
static unsigned long long g_tc_launches = 0;
void tc_count_launch() { ++g_tc_launches; }
unsigned long long tc_launch_count() { return g_tc_launches; }

} // namespace natten
