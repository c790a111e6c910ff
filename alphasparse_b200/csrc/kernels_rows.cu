// Rows by themselves: a warp or a CTA takes a whole row, the formats whose chunks of a row lie one after the other (warp or CTA per row
// chunk, and chunks with their sums in shared memory), where rows are short enough.
//
// What bounds them on matrices of a few microseconds is a chain of dependent loads and the number of launches, not bytes. The chunks'
// own kernels add up in y by `red`, so y is cleared by a kernel of its own before (1.8 us of the host, 2 us on the device), or they lay out sums in
// shared memory and look up which rows those belong to behind a barrier. Here an entry of a list says where a row's elements
// begin and which row of y it is; that, the values and the columns are read before the wait for the kernel before, and then one gather,
// one reduction and one store are left. Microseconds a call, by chunks / by rows, 40..120 elements a row, random columns, fp64: a warp per row
// chunk, 600 rows 5.3 / 2.6, 7,003 rows 7.6 / 4.4, 20,000 rows 14.7 / 9.5; chunks in shared memory 5.8 / 2.6, 11.1 / 4.4, 21.2 / 9.5; a CTA per row
// chunk, 123 rows of 1000..3000 6.4 / 3.8. From about a million non-zeros on, one L2 request a gather is the bound here too.
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "launch.h"
#include "sums.h"

namespace asp
{
typedef unsigned int u32;

namespace
{
template <class T>
__device__ __forceinline__ T ld_once(const T *p)
{
    T v;
    if constexpr (sizeof(T) == 8) asm volatile("ld.global.cs.b64 %0, [%1];" : "=d"(v) : "l"(p));
    else if constexpr (sizeof(T) == 2)
    {
        unsigned short t;
        asm volatile("ld.global.cs.u16 %0, [%1];" : "=h"(t) : "l"(p));
        v = (T)t;
    }
    else if constexpr (sizeof(T) == 1)
    {
        u32 t;
        asm volatile("ld.global.cs.u8 %0, [%1];" : "=r"(t) : "l"(p));
        v = (T)t;
    }
    else
    {
        u32 t;
        asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(t) : "l"(p));
        v = *reinterpret_cast<const T *>(&t);
    }
    return v;
}
// Sum of products with more than the values' bits, so that these kernels are no further from the exact result than the column-tiled layout that
// they are chosen before: fp32 in fp64 (the products are exact there), fp64 with the roundings that it leaves out (sums.h). Ordinary sums were 0.6 to 1.0e-7 and
// 1.1 to 1.5e-16 from the exact result (2-norm); these are 2.5e-8 and 4.7e-17,
// for up to 1.2 us more where 1.8 M products in fp64 take 13 operations each (5.2 -> 6.4 us; the layout 8.5).
template <class VT>
struct Sum;
template <>
struct Sum<float>
{
    double s = 0;
    __device__ __forceinline__ void add(float v, float x) { s = fma((double)v, (double)x, s); }
    __device__ __forceinline__ void add(const Sum &o) { s += o.s; }
    __device__ __forceinline__ Sum from(int lanes) const
    {
        Sum o;
        o.s = __shfl_xor_sync(0xffffffffu, s, lanes);
        return o;
    }
    __device__ __forceinline__ float value() const { return (float)s; }
};
template <>
struct Sum<double> : TwoSum
{
    __device__ __forceinline__ Sum from(int lanes) const
    {
        Sum o;
        o.hi = __shfl_xor_sync(0xffffffffu, hi, lanes);
        o.lo = __shfl_xor_sync(0xffffffffu, lo, lanes);
        return o;
    }
};
// of G neighbouring lanes, in each of them
template <int G, class VT>
__device__ __forceinline__ void total(Sum<VT> &s)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s.add(s.from(o));
}

// a thread's part of the row [begin, end): elements begin + t, begin + t + step, ..., four at a time; behind the end the last element is
// read again and left out. `wait` is called by every thread whose row has elements, before its first gather.
template <class VT, class CT, class W>
__device__ __forceinline__ Sum<VT> row_part(const RowArgs &a, u32 begin, u32 end, u32 t, u32 step, W &wait)
{
    constexpr int U = 4;
    const VT *const val = (const VT *)a.val, *const x = (const VT *)a.x;
    const CT *const col = (const CT *)a.col;
    Sum<VT> sum;
    for (u32 base = begin; base < end; base = end - base > U * step ? base + U * step : end)
    {
        const u32 left = end - base - 1; // of the elements from `base` on, the last one
        CT c[U];
        VT v[U], p[U];
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = ld_once(col + base + min(t + u * step, left));
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = ld_once(val + base + min(t + u * step, left));
        wait();
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = ld_x(x + c[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (t + u * step <= left) sum.add(v[u], p[u]);
    }
    return sum;
}

template <class VT, class CT>
__global__ void __launch_bounds__(256) k_row_warp(RowArgs a)
{
    const u32 lane = threadIdx.x & 31, w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); // (threads would not fit into 32 bits)
    WaitOnce wait;
    if (w < a.n)
    {
        const uint2 r = __ldg(a.rows + w);
        const u32 end = __ldg(&a.rows[w + 1].x);
        Sum<VT> s = row_part<VT, CT>(a, r.x, end, lane, 32, wait);
        total<32>(s);
        wait();
        if (lane == 0) ((VT *)a.y)[r.y] = s.value();
    }
    wait();
}

// Row-grouped: G lanes take a row, each one TLB of it (whose elements are e.w apart; the TLBs of neighbouring rows lie side by side). By
// strips, where a CTA takes 32 to 128 rows and its sums go through shared memory / by rows: 4,096 rows of 16 elements, fp32, 3.15 / 2.6 to 2.9 us, 78,000 rows of
// 5 6.5 / 4.9, fp64 8.4 / 4.6, 50,000 rows of 16 7.0 / 4.9. (Reading the rows' offsets before the wait in the strips' kernel: 3.17 -> 3.23.) G is the least that takes an average row at once: 2 to 32.
template <class VT, class CT, int G>
__global__ void __launch_bounds__(128) k_row_tlbs(RowArgs a)
{
    constexpr int U = 4;
    const VT *const val = (const VT *)a.val, *const x = (const VT *)a.x;
    const CT *const col = (const CT *)a.col;
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x, g = t / G, sub = t % G;
    WaitOnce wait;
    Sum<VT> s;
    u32 row = 0;
    if (g < a.n)
    {
        const uint4 e = __ldg(a.tlbs + g);
        const u32 n = e.z & 0xffffu, size = e.z >> 16;
        row = e.y;
        for (u32 i = sub; i < n; i += G)
            for (u32 k = 0; k < size; k += U)
            {
                CT c[U];
                VT v[U], p[U];
#pragma unroll
                for (int u = 0; u < U; u++) c[u] = ld_once(col + e.x + i + min(k + u, size - 1) * e.w);
#pragma unroll
                for (int u = 0; u < U; u++) v[u] = ld_once(val + e.x + i + min(k + u, size - 1) * e.w);
                wait();
#pragma unroll
                for (int u = 0; u < U; u++) p[u] = ld_x(x + c[u]);
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (k + u < size) s.add(v[u], p[u]);
            }
    }
    total<G>(s);
    wait();
    if (g < a.n && sub == 0) ((VT *)a.y)[row] = s.value();
}

// ELL- and SELL-like: 32 rows side by side, of whose TLBs W warps take every W-th element, so that a TLB of up to 4 W is one trip instead of a
// trip for every four. W is 4, 8 or 16 (TLBs of up to 16, up to 32, more). A row a thread, four TLBs a thread / by W warps, finite elements: 7,500 rows
// of 27, fp64, SELL 9.5 us / 2.5, ELL 7.7 / 2.5; 60,000 rows of 27 11.5 / 5.7, 9.2 / 5.8; 30,000 rows of 60 24 / 6.4, 20 / 6.4 (the column-tiled layout
// 8.5, and it takes 3 ms to build). Beyond what L2 holds the longer streams of the others win: 60,000 rows of 81, fp64, layout 14.6, this 16.0.
template <class VT, class CT, int W>
__global__ void __launch_bounds__(32 * W) k_row_strips(RowArgs a)
{
    constexpr int U = 4;
    __shared__ Sum<VT> part[W][32];
    const VT *const val = (const VT *)a.val, *const x = (const VT *)a.x;
    const CT *const col = (const CT *)a.col;
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint4 e = __ldg(a.strips + blockIdx.x);
    const u32 size = e.z & 0xffffu, n = e.z >> 16;
    const bool on = lane < n;
    u32 row = a.first_row + e.y + lane;
    if (a.place && on) row = __ldg(a.place + e.y + lane);
    WaitOnce wait;
    Sum<VT> s;
    for (u32 k = w; k < size; k += U * W)
    {
        CT c[U];
        VT v[U], p[U];
        const u32 at = e.x + (on ? lane : 0u);
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = ld_once(col + at + min(k + u * W, size - 1) * e.w);
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = ld_once(val + at + min(k + u * W, size - 1) * e.w);
        wait();
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = ld_x(x + c[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k + u * W < size) s.add(v[u], p[u]);
    }
    wait();
    part[w][lane] = s;
    __syncthreads();
    if (w != 0 || !on) return;
#pragma unroll
    for (int i = 1; i < W; i++) s.add(part[i][lane]);
    ((VT *)a.y)[row] = s.value();
}

// CSR5-like: element e of the matrix is element e % S of a thread that has S of them one after the other, and a warp's threads lie side by
// side; G lanes take a row's elements in turn, a CTA a long row's. Neighbouring elements lie 128 bytes apart, so this makes three requests to
// L2 for each: for small matrices only. Two kernels, y's shared rows cleared and added up / this: R-MAT scale 11 (20,000 elements) 5.4 us an SpMV /
// 2.7, scale 14 (200,000) 6.1 / 4.1, 22,500 rows of 24 to 27 5.5 to 6 / 3.0. Long rows by their lanes, eight trips instead of two: scale 13 4.4, so 2.9.
const u32 kRunThreads = 256; // 1024 elements of a long row a trip
template <class VT, class CT, int G>
__global__ void __launch_bounds__(kRunThreads) k_row_runs(RowArgs a)
{
    constexpr int U = 4;
    __shared__ Sum<VT> part[kRunThreads / 32];
    const VT *const val = (const VT *)a.val, *const x = (const VT *)a.x;
    const CT *const col = (const CT *)a.col;
    const bool hub = blockIdx.x < a.hubs;
    const u32 step = hub ? kRunThreads : (u32)G, sub = hub ? threadIdx.x : threadIdx.x % G;
    const u32 g = hub ? blockIdx.x : a.hubs + (blockIdx.x - a.hubs) * (kRunThreads / G) + threadIdx.x / G;
    const u32 S = a.size;
    uint4 r = make_uint4(0, 0, 0, 0);
    if (g < a.n) r = __ldg(a.runs + g);
    WaitOnce wait;
    Sum<VT> s;
    for (u32 i = sub; i < r.z; i += U * step)
    {
        u32 at[U];
        CT c[U];
        VT v[U], p[U];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const u32 e = r.x + min(i + u * step, r.z - 1), thread = e / S;
            at[u] = thread / 32 * (32 * S) + (e - thread * S) * 32 + thread % 32;
        }
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = ld_once(col + at[u]);
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = ld_once(val + at[u]);
        wait();
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = ld_x(x + c[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * step < r.z) s.add(v[u], p[u]);
    }
    wait();
    if (hub)
    {
        total<32>(s);
        if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = s;
        __syncthreads();
        if (threadIdx.x >= 32) return;
        s = threadIdx.x < kRunThreads / 32 ? part[threadIdx.x] : Sum<VT>();
        total<32>(s);
        if (threadIdx.x == 0) ((VT *)a.y)[r.y] = s.value();
        return;
    }
    total<G>(s);
    if (g < a.n && sub == 0) ((VT *)a.y)[r.y] = s.value();
}

template <class VT, class CT>
__global__ void __launch_bounds__(1024) k_row_cta(RowArgs a)
{
    __shared__ Sum<VT> part[32];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint2 r = __ldg(a.rows + blockIdx.x);
    const u32 end = __ldg(&a.rows[blockIdx.x + 1].x);
    WaitOnce wait;
    Sum<VT> s = row_part<VT, CT>(a, r.x, end, threadIdx.x, blockDim.x, wait);
    total<32>(s);
    wait();
    if (lane == 0) part[warp] = s;
    __syncthreads();
    if (warp != 0) return;
    s = lane < warps ? part[lane] : Sum<VT>();
    total<32>(s);
    if (lane == 0) ((VT *)a.y)[r.y] = s.value();
}

template <class VT, class CT>
cudaError_t launch(const RowArgs &a, cudaStream_t st)
{
    const auto tlbs = [&](auto kernel, u32 lanes) { return launch_pdl(kernel, dim3((unsigned)(((unsigned long long)a.n * lanes + 127) / 128)), dim3(128), 0, st, a); };
    switch (a.tlbs ? a.lanes : 0)
    {
    case 2: return tlbs(k_row_tlbs<VT, CT, 2>, 2);
    case 4: return tlbs(k_row_tlbs<VT, CT, 4>, 4);
    case 8: return tlbs(k_row_tlbs<VT, CT, 8>, 8);
    case 16: return tlbs(k_row_tlbs<VT, CT, 16>, 16);
    case 32: return tlbs(k_row_tlbs<VT, CT, 32>, 32);
    default: break;
    }
    if (a.tlbs) return cudaErrorInvalidValue;
    if (a.runs)
    {
        const auto runs = [&](auto kernel, u32 lanes) { return launch_pdl(kernel, dim3(a.hubs + ((a.n - a.hubs) * lanes + kRunThreads - 1) / kRunThreads), dim3(kRunThreads), 0, st, a); };
        return a.lanes == 4 ? runs(k_row_runs<VT, CT, 4>, 4) : a.lanes == 8 ? runs(k_row_runs<VT, CT, 8>, 8) : runs(k_row_runs<VT, CT, 16>, 16);
    }
    if (a.strips)
    {
        if (a.lanes == 4) return launch_pdl(k_row_strips<VT, CT, 4>, dim3(a.n), dim3(128), 0, st, a);
        if (a.lanes == 8) return launch_pdl(k_row_strips<VT, CT, 8>, dim3(a.n), dim3(256), 0, st, a);
        return launch_pdl(k_row_strips<VT, CT, 16>, dim3(a.n), dim3(512), 0, st, a);
    }
    if (a.cta == 0) return launch_pdl(k_row_warp<VT, CT>, dim3((a.n + 7) / 8), dim3(256), 0, st, a);
    return launch_pdl(k_row_cta<VT, CT>, dim3(a.n), dim3(a.cta), 0, st, a);
}
template <class VT>
cudaError_t launch_v(int col_width, const RowArgs &a, cudaStream_t st)
{
    switch (col_width)
    {
    case 1: return launch<VT, unsigned char>(a, st);
    case 2: return launch<VT, unsigned short>(a, st);
    case 4: return launch<VT, u32>(a, st);
    default: return cudaErrorInvalidValue;
    }
}
} // namespace

cudaError_t launch_own_rows(int val_is_f64, int col_width, const RowArgs &a, cudaStream_t st)
{
    return val_is_f64 ? launch_v<double>(col_width, a, st) : launch_v<float>(col_width, a, st);
}
} // namespace asp
