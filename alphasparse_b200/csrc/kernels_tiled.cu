// Column-tiled SpMV for matrices whose gathers of x are scattered.
//
// A gather of x through L1 costs one request to L2 for every cache line that a warp's 32 lanes touch, and an SM issues one
// such request per clock: with random columns that is one clock per non-zero and SM (290 G non-zeros/s on 148 SMs), two to
// four times what the matrix's bytes take at the memory's rate. Shared memory serves 9 to 12 random lanes per clock. So the
// columns are cut into tiles that fit in shared memory; a CTA loads a tile of x once (coalesced) and runs through its part of
// the tile's non-zeros, 2 + sizeof(value) bytes each (the column inside the tile has 16 bits):
//   piece  up to 32 non-zeros of one row in one tile
//   slice  64 pieces, two per lane, of about the same length (sorted inside windows of 1024 pieces); stored step by step,
//          a step = one non-zero of every piece
//   steps  one linear stream, cut evenly among the CTAs (one per SM) and inside them among the warps (32, or 16 in fp64), in the middle of
//          slices too: what a warp has summed when its slice or its share ends is added to its row by `red`
//   parts  a row that gets there in many parts would collect a rounding error with each (fp32, 80 elements over 25 tiles: 1.0e-7
//          from the 64-bit result, the formats' own kernels 0.72e-7): the sums of such rows are 64-bit ones in memory of the
//          group, which k_rows turns into y and leaves as zeros for the next call (0.42e-7). In fp64 tiles and warps
//          take `copies` sums of a row in turn, which k_rows adds up with their roundings. A piece is summed with more than the value's bits, too.
// The stream is read two batches deep into registers. 159 KB of shared memory per tile leave the L1 enough lines for the
// loads in flight: with 224 KB the same stream is read at 4.2 instead of 5 TB/s. (k_tiled_units takes 32 KB more: 2 KB a warp, in
// which the sums of a unit's rows are laid out.)
// Where rows have few elements in a tile (1 to 7) and lie side by side, there are units instead of slices (k_tiled_units): a slice
// puts pieces of one length together, so that its `red` goes to 32 rows anywhere among 1024, ten lines of sums or more, each of which is a
// request to L2, and that is what bounds it. A unit is 256 elements of a tile in order, eight a lane. Every lane adds up the runs of its
// elements, what reaches over lanes is added by a scan, and the sums leave in the order of the rows: two to three lines a `red`. That
// takes more instructions an element (31 against 21), so long runs stay with slices; the figures are where the rule is (tiled_build.cpp).
// A tile is loaded by cp.async, every thread's ten pieces in flight at once. Through registers, five at a time, nothing else runs for
// 5 us of an SpMV over R-MAT scale 21 (ten SpMVs: 504 -> 476 us; by bulk copies 482).
// Measured, fp32 (against the formats' own kernels): 200,000 rows of 40..120 non-zeros, random columns among 1 M: 31 us
// (76 us, row-grouped; 38 us in slices); 9,001 rows of 1000..3000: 25 us (77 us, long-row).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "launch.h"
#include "sums.h"
#include "tiled.h"

namespace asp
{
typedef unsigned long long u64;
typedef unsigned int u32;

namespace
{
template <class VT>
struct Pair;
template <>
struct Pair<float>
{
    typedef float2 type;
};
template <>
struct Pair<double>
{
    typedef double2 type;
};

// Sum of the products of a piece. fp32: the products of a batch in fp32 (four at most), the batches in fp64. fp64: the sum and
// the rounding errors that it left out (sums.h); 13 operations a product of the 64 that an SM does per clock in fp64, of which a
// non-zero takes one.
template <class VT>
struct Sum;
template <>
struct Sum<float>
{
    float part = 0;
    double sum = 0;
    __device__ __forceinline__ void add(float v, float x) { part += v * x; }
    __device__ __forceinline__ void batch()
    {
        sum += (double)part;
        part = 0;
    }
    __device__ __forceinline__ double take()
    {
        const double s = sum + (double)part;
        sum = 0;
        part = 0;
        return s;
    }
};
template <>
struct Sum<double> : TwoSum
{
    __device__ __forceinline__ void batch() {}
    __device__ __forceinline__ double take()
    {
        const double s = value();
        hi = lo = 0;
        return s;
    }
};

// x may have been written by the kernel before: read through L2 (as cp.async.cg does), in program order after the wait
__device__ __forceinline__ float ld_x1(const float *p)
{
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_x1(const double *p)
{
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

template <class VT>
__global__ void __launch_bounds__(256) k_clear(VT *y, u64 n)
{
    grid_release();
    grid_wait();
    const u64 stride = (u64)gridDim.x * blockDim.x;
    const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    constexpr u64 V = 16 / sizeof(VT);
    const u64 head = ((16 - ((uintptr_t)y & 15)) & 15) / sizeof(VT), h = head < n ? head : n, body = (n - h) / V;
    uint4 *b = reinterpret_cast<uint4 *>(y + h);
    for (u64 i = t; i < body; i += stride) b[i] = make_uint4(0, 0, 0, 0);
    if (t < h) y[t] = 0;
    if (t < n - h - body * V) y[h + body * V + t] = 0;
}

// row += v for the 32 pieces of a warp. Pieces of a long row lie next to one another, and a `red` of many lanes to one
// address is served lane by lane: those are summed in the warp first (R-MAT with hub rows: 72 -> 60 us an SpMV).
template <class VT>
__device__ __forceinline__ void add_rows(VT *y, double *sum, u32 row, double v, u32 lane)
{
    const u32 next = __shfl_down_sync(0xffffffffu, row, 1);
    const u32 goes_on = __ballot_sync(0xffffffffu, lane < 31 && row == next);
    bool head = true;
    if (goes_on != 0)
    {
        const u32 from = goes_on >> lane;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const double o = __shfl_down_sync(0xffffffffu, v, d);
            const u32 m = (1u << d) - 1u;
            if ((from & m) == m) v += o;
        }
        head = lane == 0 || ((goes_on >> (lane - 1)) & 1u) == 0;
    }
    if (!head || row == kTiledNoRow) return;
    if (row & kTiledInParts) atomicAdd(sum + (row & ~kTiledInParts), v); // result unused: red.global.add
    else atomicAdd(y + row, (VT)v);
}

// a CTA's tile of x, and a zero after it
template <u32 NT, class VT>
__device__ __forceinline__ void load_tile(const TiledArgs &a, VT *xs, u32 tile, u32 tile_cols)
{
    const VT *xp = (const VT *)a.x + (u64)tile * tile_cols;
    const u64 left = a.n_cols - (u64)tile * tile_cols;
    const u32 n = left < tile_cols ? (u32)left : tile_cols;
    constexpr u32 V = 16 / sizeof(VT);
    u32 i = 0;
    if (((uintptr_t)xp & 15) == 0)
    {
        // straight to shared memory, all of a thread's 16-byte pieces in flight at once
        const u32 n4 = n / V, to = (u32)__cvta_generic_to_shared(xs);
        for (u32 j = threadIdx.x; j < n4; j += NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + j * 16), "l"((const char *)xp + (size_t)j * 16) : "memory");
        i = n4 * V;
    }
    for (i += threadIdx.x; i < n; i += NT) xs[i] = ld_x1(xp + i);
    if (threadIdx.x == 0) xs[tile_cols] = 0;
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <class VT, int U, u32 W>
__global__ void __launch_bounds__(W * 32, 1) k_tiled(TiledArgs a, u32 tile_cols)
{
    typedef typename Pair<VT>::type P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    VT *xs = reinterpret_cast<VT *>(smem_raw);
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    VT *const y = (VT *)a.y;
    bool first = true;
    u32 visit = blockIdx.x;
    do
    {
        const uint4 k = __ldg(a.work + (size_t)visit * W + warp);
        u32 step = k.x, slice = k.z;
        const u32 end = k.y, tile = k.w & 0xffffu;
        visit = k.w >> 16;
        double *const sum = a.sum + (size_t)((tile + warp) & (a.copies - 1)) * a.sum_stride;
        const P *vp = reinterpret_cast<const P *>(a.val) + (size_t)step * 32 + lane;
        const u32 *cp = reinterpret_cast<const u32 *>(a.col) + (size_t)step * 32 + lane;
        P v[U];
        u32 c[U];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            v[u] = __ldcs(vp + u * 32);
            c[u] = __ldcs(cp + u * 32);
        }
        const uint2 *rp = reinterpret_cast<const uint2 *>(a.row) + (size_t)slice * 32 + lane;
        u32 s_end = __ldg(a.end + slice), s_next = __ldg(a.end + slice + 1);
        uint2 row = __ldg(rp), row_next = __ldg(rp + 32);
        if (first)
        {
            // nothing above depends on what ran before
            grid_release();
            grid_wait();
            first = false;
        }
        else
            __syncthreads(); // the tile before has been read
        load_tile<W * 32>(a, xs, tile, tile_cols);
        __syncthreads();
        Sum<VT> acc0, acc1;
        while (step < end)
        {
            P nv[U];
            u32 nc[U];
            vp += U * 32;
            cp += U * 32;
#pragma unroll
            for (int u = 0; u < U; u++)
            {
                nv[u] = __ldcs(vp + u * 32);
                nc[u] = __ldcs(cp + u * 32);
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (step < end)
                {
                    acc0.add(v[u].x, xs[c[u] & 0xffffu]);
                    acc1.add(v[u].y, xs[c[u] >> 16]);
                    step++;
                    if (step == s_end || step == end)
                    {
                        add_rows(y, sum, row.x, acc0.take(), lane);
                        add_rows(y, sum, row.y, acc1.take(), lane);
                        slice++;
                        rp += 32;
                        s_end = s_next;
                        row = row_next;
                        s_next = __ldg(a.end + slice + 1);
                        row_next = __ldg(rp + 32);
                    }
                }
#pragma unroll
            for (int u = 0; u < U; u++)
            {
                v[u] = nv[u];
                c[u] = nc[u];
            }
            acc0.batch();
            acc1.batch();
        }
    } while (visit != 0);
}

// ---- units: where rows have few elements in a tile (fp32)
const u32 kUnitSmem = kTiledTileBytes + kTiledUnitWarps * kTiledStage * 8;

// MODE: rows are added up in y (0), have sums (1), or some have (2)
template <int MODE>
__global__ void __launch_bounds__(kTiledUnitWarps * 32, 1) k_tiled_units(TiledArgs a, u32 tile_cols)
{
    constexpr u32 S = kTiledLane, U = kTiledUnit, NV = S / 4, NC = S / 8, NT = kTiledUnitWarps * 32, R = S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *const xs = reinterpret_cast<float *>(smem_raw);
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *const stage = reinterpret_cast<double *>(smem_raw + kTiledTileBytes) + warp * kTiledStage; // row j of the unit: stage[j + 1]
    float *const y = (float *)a.y;
    bool first = true;
    u32 visit = blockIdx.x;
    do
    {
        const uint4 k = __ldg(a.work + (size_t)visit * kTiledUnitWarps + warp);
        u32 unit = k.x;
        const u32 end = k.y, tile = k.z;
        visit = k.w;
        double *const sum = a.sum + (size_t)((tile + warp) & (a.copies - 1)) * a.sum_stride;
        float4 qv[NV];
        uint4 qc[NC];
        u32 word = 0, rows[R];
        // rows of the unit in `row`: [s0, s1), of the next one [s1, s2)
        u32 s0 = __ldg(a.seg + unit), s1 = __ldg(a.seg + unit + 1), s2 = __ldg(a.seg + unit + 2);
        auto fetch = [&](u32 u, u32 from, u32 to) {
            const float4 *vp = reinterpret_cast<const float4 *>(a.val) + (size_t)u * (U / 4) + lane;
            const uint4 *cp = reinterpret_cast<const uint4 *>(a.col) + (size_t)u * (U / 8) + lane;
#pragma unroll
            for (u32 i = 0; i < NV; i++) qv[i] = __ldcs(vp + i * 32);
#pragma unroll
            for (u32 i = 0; i < NC; i++) qc[i] = __ldcs(cp + i * 32);
            word = __ldcs(a.word + (size_t)u * 32 + lane);
#pragma unroll
            for (u32 i = 0; i < R; i++)
            {
                if (from + i * 32 >= to) break;
                if (from + i * 32 + lane < to) rows[i] = __ldcs(a.row + from + i * 32 + lane);
            }
        };
        if (unit < end) fetch(unit, s0, s1);
        if (first)
        {
            // nothing above depends on what ran before
            grid_release();
            grid_wait();
            first = false;
        }
        else
            __syncthreads(); // the tile before has been read
        load_tile<NT>(a, xs, tile, tile_cols);
        __syncthreads();
        while (unit < end)
        {
            float v[S], x[S];
            u32 row[R];
            const u32 F = word, n_rows = s1 - s0;
#pragma unroll
            for (u32 i = 0; i < NV; i++) v[4 * i] = qv[i].x, v[4 * i + 1] = qv[i].y, v[4 * i + 2] = qv[i].z, v[4 * i + 3] = qv[i].w;
#pragma unroll
            for (u32 i = 0; i < NC; i++)
            {
                const u32 c[4] = {qc[i].x, qc[i].y, qc[i].z, qc[i].w};
#pragma unroll
                for (u32 j = 0; j < 4; j++)
                {
                    x[i * 8 + 2 * j] = xs[c[j] & 0xffffu];
                    x[i * 8 + 2 * j + 1] = xs[c[j] >> 16];
                }
            }
#pragma unroll
            for (u32 i = 0; i < R; i++) row[i] = rows[i];
            unit++;
            s0 = s1;
            s1 = s2;
            s2 = __ldg(a.seg + unit + 2);
            if (unit < end) fetch(unit, s0, s1);
            // Every start stores what the lane has summed since the one before and goes on from zero. Before its first start that is
            // the end of a row of lanes before: it goes where that row's sum will be, and comes back.
            double *const mine = stage + (F >> 16);
            double *to = mine;
            double acc = 0; // (exact products)
#pragma unroll
            for (u32 j = 0; j < S; j++)
            {
                if (F & (1u << j))
                {
                    *to++ = acc;
                    acc = 0;
                }
                acc = fma((double)v[j], (double)x[j], acc);
            }
            const bool starts = (F & 0xffffu) != 0;
            double sc = starts ? *mine : acc;
            __syncwarp(); // the lane before, whose last row ends there, stores the whole sum over it
            // lane l: the sum up to the next lane in which a row starts; rounds as long as there are so many lanes without a start
            const u32 none = ~__ballot_sync(0xffffffffu, starts);
            for (u32 d = 1, c = none; c != 0; c &= c >> d, d *= 2)
            {
                const double o = __shfl_down_sync(0xffffffffu, sc, d);
                if (lane + d < 32 && (c >> lane & 1u)) sc += o;
            }
            const double more = __shfl_down_sync(0xffffffffu, sc, 1);
            if (starts) *to = lane == 31 ? acc : acc + more;
            __syncwarp();
#pragma unroll
            for (u32 i = 0; i < R; i++)
            {
                if (i * 32 >= n_rows) break;
                const u32 j = i * 32 + lane, r = row[i];
                if (j >= n_rows) continue;
                // (results unused: red.global.add)
                if (MODE == 1 || (MODE == 2 && (r & kTiledInParts))) atomicAdd(sum + (r & ~kTiledInParts), stage[j + 1]);
                else atomicAdd(y + r, (float)stage[j + 1]);
            }
            __syncwarp();
        }
    } while (visit != 0);
}

__device__ __forceinline__ double ld_sum(const double *p)
{
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

// the rows in many parts: y = their sums, which are zero afterwards (for the next k_tiled)
template <class VT, int G>
__global__ void __launch_bounds__(256) k_rows(const u32 *rows, double *sum, u64 stride, VT *y, u32 n)
{
    constexpr int U = G < 4 ? 4 / G : 1; // rows in flight
    const u32 threads = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    grid_release();
    grid_wait();
    for (u32 r = t; r < n; r += threads * U)
    {
        double s[U][G];
        u32 to[U];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const u32 q = r + u * threads < n ? r + u * threads : r;
            to[u] = rows ? __ldg(rows + q) : q;
#pragma unroll
            for (int g = 0; g < G; g++) s[u][g] = ld_sum(sum + g * stride + q);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (r + u * threads < n)
            {
#pragma unroll
                for (int g = 0; g < G; g++) sum[g * stride + r + u * threads] = 0;
                double hi = s[u][0], lo = 0; // the sum of the copies, and what its roundings leave out
#pragma unroll
                for (int g = 1; g < G; g++)
                {
                    const double v = s[u][g], t = hi + v, b = t - hi;
                    lo += (hi - (t - b)) + (v - b);
                    hi = t;
                }
                y[to[u]] = (VT)(G > 1 && isfinite(hi) ? hi + lo : hi);
            }
    }
}

// steps read ahead: 48 KB (fp32), 40 KB (fp64) in flight per SM
constexpr auto kSlices = k_tiled<float, 4, kTiledWarps>;
constexpr auto kSlices64 = k_tiled<double, 2, kTiledWarps>, kSlices64Few = k_tiled<double, 4, kTiledFewWarps>;

template <class VT>
cudaError_t clear(VT *y, u64 n, unsigned n_sm, cudaStream_t st)
{
    // a few 16-byte stores per thread
    const u64 want = (n * sizeof(VT) / 16 + 1023) / 1024;
    return launch_pdl(k_clear<VT>, dim3((unsigned)(want < 1 ? 1 : want < 4ull * n_sm ? want : 4ull * n_sm)), dim3(256), 0, st, y, n);
}

template <class VT>
cudaError_t launch_sums(const TiledArgs &a, unsigned n_sm, cudaStream_t st)
{
    if (a.direct)
    {
        const cudaError_t e = clear((VT *)a.y, a.n_rows, n_sm, st);
        if (e != cudaSuccess) return e;
    }
    const auto tiled = [&](auto kernel, u32 warps, u32 smem) { return launch_pdl(kernel, dim3(n_sm), dim3(warps * 32), smem, st, a, (u32)tiled_tile_cols(sizeof(VT) == 8)); };
    if (!a.word) return tiled(sizeof(VT) == 4 ? kSlices : a.warps == kTiledFewWarps ? kSlices64Few : kSlices64, a.warps, kTiledTileBytes);
    if (sizeof(VT) == 8) return cudaErrorInvalidValue; // (units are fp32)
    if (!a.direct) return tiled(k_tiled_units<1>, kTiledUnitWarps, kUnitSmem);
    return a.n_parts == 0 ? tiled(k_tiled_units<0>, kTiledUnitWarps, kUnitSmem) : tiled(k_tiled_units<2>, kTiledUnitWarps, kUnitSmem);
}

template <class VT>
cudaError_t launch_rows(const TiledArgs &a, unsigned n_sm, cudaStream_t st)
{
    // one trip per thread up to a full device: a trip waits once for its rows' sums (16 copies, 4000 rows, four trips a thread: 10 us)
    const u32 per_cta = 256 * (a.copies < 4 ? 4 / a.copies : 1);
    const u64 want = ((u64)a.n_parts + per_cta - 1) / per_cta;
    const dim3 grid((unsigned)(want < 8ull * n_sm ? want : 8ull * n_sm)), block(256);
    const auto rows = [&](auto kernel) { return launch_pdl(kernel, grid, block, 0, st, a.parts, a.sum, (u64)a.sum_stride, (VT *)a.y, (u32)a.n_parts); };
    if (a.copies == 1) return rows(k_rows<VT, 1>);
    if constexpr (sizeof(VT) == 8)
    {
        if (a.copies == 2) return rows(k_rows<VT, 2>);
        if (a.copies == 4) return rows(k_rows<VT, 4>);
        if (a.copies == 8) return rows(k_rows<VT, 8>);
        if (a.copies == 16) return rows(k_rows<VT, 16>);
    }
    return cudaErrorInvalidValue;
}
} // namespace

cudaError_t launch_clear(int val_is_f64, void *y, unsigned long long n, unsigned n_sm, cudaStream_t st)
{
    return val_is_f64 ? clear((double *)y, n, n_sm, st) : clear((float *)y, n, n_sm, st);
}

namespace
{
cudaError_t allow(const void *f, u32 smem) { return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }
} // namespace

cudaError_t tiled_setup(int val_is_f64)
{
    if (val_is_f64)
    {
        const cudaError_t e = allow((const void *)kSlices64, kTiledTileBytes);
        return e == cudaSuccess ? allow((const void *)kSlices64Few, kTiledTileBytes) : e;
    }
    cudaError_t e = allow((const void *)kSlices, kTiledTileBytes);
    for (const void *f : {(const void *)k_tiled_units<0>, (const void *)k_tiled_units<1>, (const void *)k_tiled_units<2>})
        if (e == cudaSuccess) e = allow(f, kUnitSmem);
    return e;
}

cudaError_t launch_tiled_sums(int val_is_f64, const TiledArgs &a, unsigned n_sm, cudaStream_t st)
{
    return val_is_f64 ? launch_sums<double>(a, n_sm, st) : launch_sums<float>(a, n_sm, st);
}

cudaError_t launch_tiled_rows(int val_is_f64, const TiledArgs &a, unsigned n_sm, cudaStream_t st)
{
    return val_is_f64 ? launch_rows<double>(a, n_sm, st) : launch_rows<float>(a, n_sm, st);
}
} // namespace asp
