// Relative position bias for the split QK operator.
//
//   logits[b, pos, h, slot] += rpb[h, pb(pos_0) + slot_0, pb(pos_1) + slot_1, ...]
//
// with rpb of shape [H, 2*K_0 - 1, (2*K_1 - 1, (2*K_2 - 1))] and pb() the bias window start of the
// reference (src/natten_mps/utils/window.py:119-135; used by src/natten_mps/compat/v014.py:66-183):
// in the interior pb = K/2 and slot j looks at relative offset j - K/2; at the edges the window is
// clamped and pb moves so that the same relative offsets keep the same bias entries.
// The bias is added to the finished logits in one pass over them (masked slots hold -inf and stay
// -inf); its gradient is a fixed-order reduction of dlogits, one block per bias entry, so it is
// bit-reproducible.  Unit stride, non-causal (what the reference's bias operators cover).
#include "rpb.cuh"

#include "device_cache.cuh"
#include "tc_kernels.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace natten {
namespace {

__host__ __device__ __forceinline__ int pb_start(int index, int length, int kernel_size, int dilation)
{
    const int nh = kernel_size / 2;
    if (dilation <= 1) {
        int pb = nh;
        if (index < nh) pb += nh - index;
        else if (index + nh >= length) pb += length - index - 1 - nh;
        return pb;
    }
    if (index - nh * dilation < 0) return kernel_size - 1 - index / dilation;
    if (index + nh * dilation >= length) return (length - index - 1) / dilation;
    return nh;
}

template <typename T> struct Acc { using type = float; };
template <> struct Acc<double> { using type = double; };
template <typename T> __device__ __forceinline__ typename Acc<T>::type ld(const T* p) { return (typename Acc<T>::type)(*p); }
template <> __device__ __forceinline__ float ld<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T, typename A> __device__ __forceinline__ T st(A v) { return (T)v; }
template <> __device__ __forceinline__ __half st<__half, float>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 st<__nv_bfloat16, float>(float v) { return __float2bfloat16_rn(v); }

// Bias index of (position, slot) on every axis -> flat index into one head's bias table.
__device__ __forceinline__ long long bias_index(const Geo& g, long long pos_flat, int slot)
{
    int pos[3] = {0, 0, 0}, sl[3] = {0, 0, 0};
    for (int a = g.rank - 1; a >= 0; --a) {
        pos[a] = (int)(pos_flat % g.L[a]);
        pos_flat /= g.L[a];
        sl[a] = slot % g.K[a];
        slot /= g.K[a];
    }
    long long idx = 0;
    for (int a = 0; a < g.rank; ++a)
        idx = idx * (2 * g.K[a] - 1) + pb_start(pos[a], g.L[a], g.K[a], g.dil[a]) + sl[a];
    return idx;
}

template <typename T>
__global__ void __launch_bounds__(256)
rpb_add_kernel(const __grid_constant__ Geo g, const T* __restrict__ rpb, T* __restrict__ logits, long long total,
               long long table)
{
    using A = typename Acc<T>::type;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int slot = (int)(i % g.ktot);
    const long long row = i / g.ktot;               // (b * ltot + pos) * Hq + h
    const int h = (int)(row % g.Hq);
    const long long pos = (row / g.Hq) % g.ltot;
    const A bias = ld(rpb + h * table + bias_index(g, pos, slot));
    logits[i] = st<T, A>(ld(logits + i) + bias);
}

// One block per (head, bias entry): sums dlogits over every (batch, position) whose window maps a slot
// onto this entry, threads striding over (batch, position) and a tree reduction in a fixed order.
template <typename T>
__global__ void __launch_bounds__(256)
rpb_grad_kernel(const __grid_constant__ Geo g, const T* __restrict__ dlogits, T* __restrict__ drpb, long long table)
{
    using A = typename Acc<T>::type;
    __shared__ A red[256];
    const int h = blockIdx.y;
    long long e = blockIdx.x;
    int want[3] = {0, 0, 0};
    for (int a = g.rank - 1; a >= 0; --a) { want[a] = (int)(e % (2 * g.K[a] - 1)); e /= (2 * g.K[a] - 1); }
    A acc = 0;
    const long long n = (long long)g.B * g.ltot;
    for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        long long p = t % g.ltot;
        const long long b = t / g.ltot;
        int slot = 0;
        bool hit = true;
        int pos[3] = {0, 0, 0};
        for (int a = g.rank - 1; a >= 0; --a) { pos[a] = (int)(p % g.L[a]); p /= g.L[a]; }
        for (int a = 0; a < g.rank; ++a) {
            const int s = want[a] - pb_start(pos[a], g.L[a], g.K[a], g.dil[a]);
            if (s < 0 || s >= g.K[a]) hit = false;
            slot = slot * g.K[a] + s;
        }
        if (hit) {
            acc += ld(dlogits + ((b * g.ltot + t % g.ltot) * g.Hq + h) * g.ktot + slot);
        }
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) drpb[h * table + blockIdx.x] = st<T, A>(red[0]);
}

// The same sums in one pass over dlogits: a cluster of CTAs per head, every warp walks its share of the positions with one
// slot per lane and adds into a table of its own in shared memory (for one position every slot has a different entry, so
// no two lanes meet); the tables are then added up in a fixed order, first inside the CTA, then over the cluster through
// distributed shared memory.  Bound by the latency of the loads (kAhead positions of a warp are in flight).  The
// one-block-per-entry kernel above decodes every position for every entry of the table: 208 us for the 56 x 56, 7 x 7,
// 4 heads, batch 4 bias in bf16, 33 us here with 8 CTAs a head, 21 us with 16.
constexpr int kGradWarps = 16;
template <typename T, int kRegs>
__global__ void __launch_bounds__(kGradWarps * 32)
rpb_grad_pass_kernel(const __grid_constant__ Geo g, const T* __restrict__ dlogits, T* __restrict__ drpb, int table)
{
    namespace cg = cooperative_groups;
    extern __shared__ float tables[];                       // [kGradWarps][table], then [ktot] slot offsets
    int* slot_entry = reinterpret_cast<int*>(tables + (size_t)kGradWarps * table);
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kGradWarps * table; i += blockDim.x) tables[i] = 0.f;
    for (int j = threadIdx.x; j < g.ktot; j += blockDim.x) {
        int rem = j, off = 0, mul = 1;
        for (int a = g.rank - 1; a >= 0; --a) { off += (rem % g.K[a]) * mul; rem /= g.K[a]; mul *= 2 * g.K[a] - 1; }
        slot_entry[j] = off;
    }
    __syncthreads();
    float* mine = tables + (size_t)warp * table;
    // A warp takes runs of kRun positions along the last axis; the other axes' share of the first table entry is worked out
    // once per run.  Away from the clamped edges every position uses the same entries: those sums stay in registers (kRegs
    // slots a lane) and only the others touch the table.
    constexpr int kRun = 16, kAhead = kRegs > 2 ? 4 : 8;
    const int last = g.rank - 1, Ln = g.L[last], Kn = g.K[last], dn = g.dil[last];
    const int runs_per_row = (Ln + kRun - 1) / kRun, runs = (int)((long long)g.B * (g.ltot / Ln)) * runs_per_row;
    int inner_outer = 0, inner;
    for (int a = 0; a < last; ++a) inner_outer = inner_outer * (2 * g.K[a] - 1) + g.K[a] / 2;
    inner = inner_outer * (2 * Kn - 1) + Kn / 2;
    float acc[kRegs];
#pragma unroll
    for (int r = 0; r < kRegs; ++r) acc[r] = 0.f;
    for (int u = rank * kGradWarps + warp; u < runs; u += gridDim.x * kGradWarps) {
        const int row = u / runs_per_row, x0 = (u - row * runs_per_row) * kRun, x1 = x0 + kRun < Ln ? x0 + kRun : Ln;
        int rem = row, outer = 0, mul = 1;                  // batch and the outer axes
        for (int a = last - 1; a >= 0; --a) {
            const int q = rem / g.L[a];
            outer += pb_start(rem - q * g.L[a], g.L[a], g.K[a], g.dil[a]) * mul;
            mul *= 2 * g.K[a] - 1;
            rem = q;
        }
        const T* src = dlogits + ((long long)row * Ln * g.Hq + h) * g.ktot;
        const long long step = (long long)g.Hq * g.ktot;
        for (int x = x0; x < x1; x += kAhead) {
            T raw[kAhead][kRegs];                           // clamped addresses, no branches: the loads go out together
#pragma unroll
            for (int i = 0; i < kAhead; ++i)
#pragma unroll
                for (int r = 0; r < kRegs; ++r) raw[i][r] = src[min(x + i, x1 - 1) * step + min(lane + 32 * r, g.ktot - 1)];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int base = outer * (2 * Kn - 1) + pb_start(min(x + i, x1 - 1), Ln, Kn, dn);
                if (x + i >= x1) break;
                if (base == inner) {
#pragma unroll
                    for (int r = 0; r < kRegs; ++r) acc[r] += ld(&raw[i][r]);          // lanes past the window: never written out
                } else {
#pragma unroll
                    for (int r = 0; r < kRegs; ++r)
                        if (lane + 32 * r < g.ktot) mine[base + slot_entry[lane + 32 * r]] += ld(&raw[i][r]);
                    __syncwarp();                           // the next position may meet this entry in another lane
                }
                for (int j = lane + 32 * kRegs; j < g.ktot; j += 32) mine[base + slot_entry[j]] += ld(src + (x + i) * step + j);
                __syncwarp();
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kRegs; ++r)
        if (lane + 32 * r < g.ktot) mine[inner + slot_entry[lane + 32 * r]] += acc[r];
    __syncthreads();
    for (int i = threadIdx.x; i < table; i += blockDim.x) {
        float acc = 0.f;
        for (int w = 0; w < kGradWarps; ++w) acc += tables[(size_t)w * table + i];
        tables[i] = acc;                                    // row 0 of column i: read by this thread only
    }
    cluster.sync();
    for (int i = rank * blockDim.x + threadIdx.x; i < table; i += gridDim.x * blockDim.x) {
        float acc = 0.f;
        for (int r = 0; r < (int)gridDim.x; ++r) acc += *cluster.map_shared_rank(tables + i, r);
        drpb[(long long)h * table + i] = st<T, float>(acc);
    }
    cluster.sync();                                         // nobody leaves while its table is being read
}

// false: does not apply (no room for a cluster of eight, table too large for shared memory, too many positions for 32-bit
// indices, or so few values that the other kernel's many blocks are done sooner: 10 us against 13 at 39 K values)
template <typename T>
bool rpb_grad_pass(const Geo& g, const void* dlogits, void* drpb, long long table, cudaStream_t s, cudaError_t& err)
{
    const size_t smem = (size_t)kGradWarps * table * 4 + (size_t)g.ktot * 4;
    const long long positions = (long long)g.B * g.ltot;
    if (table > 8192 || smem > 200 * 1024 || positions > 0x7fff0000ll || g.Hq > 65535 || positions * g.Hq * g.ktot < 100000) return false;
    const int inject = tc_debug_inject();
    const unsigned limit = inject == 2 ? 8 : inject == 3 ? 0 : 16;
    // One cluster per head: 16 CTAs while the clusters of all heads find room side by side, else 8.  With two CTAs on an SM
    // (up to 64 slots) 12 heads of 7 x 7 on 56 x 56, batch 4, take 28 us with 16 and 33 with 8, 16 heads 43.5 and 43.9.  With
    // one, seven clusters of 16 fit: 7 and 8 heads of 13 x 13 on 40 x 40, batch 2, take 15.4 and 28.9 with 16, 24.4 with 8;
    // 23 x 23, 47.8 and 92.6 with 16, 86.4 with 8.
    auto launch = [&](auto* kernel) {
        err = ensure_dynamic_smem((const void*)kernel, kMaxDynamicSmem);
        if (err == cudaSuccess) err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (err != cudaSuccess) return true;
        for (unsigned ctas = 16; ctas >= 8; ctas /= 2) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = ctas;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(ctas, (unsigned)g.Hq);
            cfg.blockDim = dim3(kGradWarps * 32);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = s;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (ctas > limit || cluster_room((const void*)kernel, cfg) < (ctas > 8 ? g.Hq : 1)) continue;
            err = cudaLaunchKernelEx(&cfg, kernel, g, (const T*)dlogits, (T*)drpb, (int)table);
            return true;
        }
        return false;
    };
    return g.ktot <= 64 ? launch(rpb_grad_pass_kernel<T, 2>) : launch(rpb_grad_pass_kernel<T, 6>);
}

long long table_size(const Geo& g)
{
    long long t = 1;
    for (int a = 0; a < g.rank; ++a) t *= 2 * g.K[a] - 1;
    return t;
}

bool supported(const Geo& g)
{
    for (int a = 0; a < g.rank; ++a)
        if (g.st[a] != 1 || g.causal[a] || (g.K[a] & 1) == 0) return false;     // even kernels index past the table
    return g.extents == nullptr && g.n_extra == 0 && g.Hq == g.Hkv;
}

} // namespace

int rpb_add(int dtype, const Geo& g, const void* rpb, void* logits, cudaStream_t s)
{
    if (!supported(g)) return -2;
    const long long total = (long long)g.B * g.ltot * g.Hq * g.ktot;
    if (total == 0) return 0;
    const long long table = table_size(g);
    const unsigned blocks = (unsigned)((total + 255) / 256);
    switch (dtype) {
        case 0: rpb_add_kernel<float><<<blocks, 256, 0, s>>>(g, (const float*)rpb, (float*)logits, total, table); break;
        case 1: rpb_add_kernel<__half><<<blocks, 256, 0, s>>>(g, (const __half*)rpb, (__half*)logits, total, table); break;
        case 2: rpb_add_kernel<__nv_bfloat16><<<blocks, 256, 0, s>>>(g, (const __nv_bfloat16*)rpb, (__nv_bfloat16*)logits, total, table); break;
        case 3: rpb_add_kernel<double><<<blocks, 256, 0, s>>>(g, (const double*)rpb, (double*)logits, total, table); break;
        default: return -1;
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? 0 : (int)err;
}

int rpb_grad(int dtype, const Geo& g, const void* dlogits, void* drpb, cudaStream_t s)
{
    if (!supported(g)) return -2;
    const long long table = table_size(g);
    if (table > 0x7fffffffll || g.Hq > 65535) return -2;
    cudaError_t err = cudaSuccess;
    if ((dtype == 0 && rpb_grad_pass<float>(g, dlogits, drpb, table, s, err)) ||
        (dtype == 1 && rpb_grad_pass<__half>(g, dlogits, drpb, table, s, err)) ||
        (dtype == 2 && rpb_grad_pass<__nv_bfloat16>(g, dlogits, drpb, table, s, err)))
        return (int)err;
    const dim3 grid((unsigned)table, (unsigned)g.Hq);
    switch (dtype) {
        case 0: rpb_grad_kernel<float><<<grid, 256, 0, s>>>(g, (const float*)dlogits, (float*)drpb, table); break;
        case 1: rpb_grad_kernel<__half><<<grid, 256, 0, s>>>(g, (const __half*)dlogits, (__half*)drpb, table); break;
        case 2: rpb_grad_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(g, (const __nv_bfloat16*)dlogits, (__nv_bfloat16*)drpb, table); break;
        case 3: rpb_grad_kernel<double><<<grid, 256, 0, s>>>(g, (const double*)dlogits, (double*)drpb, table); break;
        default: return -1;
    }
    err = cudaGetLastError();
    return err == cudaSuccess ? 0 : (int)err;
}

} // namespace natten
