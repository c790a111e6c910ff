// Block-value template (no counterpart among the reference's ten reduce templates): blocked ELL over
// dense R x C blocks, produced by the `block_value R C` operator.
//
// The reference's formats store one column index per non-zero. A matrix assembled from small dense blocks
// (finite elements with several unknowns per node: 3 x 3 blocks for 3-D elasticity) repeats that index R*C
// times per block and gathers every x value R times. Here a block carries ONE block-column index, its R*C
// values, and each thread gathers the C values of x once per block:
//   bytes per stored non-zero  12 -> 8 + 4 / (R*C)   (fp64, 3 x 3: 8.44)
//   gathers per stored non-zero 1 -> 1 / R
//
// Layout (NB = block rows padded to a multiple of 2, W = blocks per block row, padded with zero blocks):
//   block column of slot k of block row b     idx[k * NB + b]
//   element (i, j) of that block              val[((k * R + i) * C + j) * NB + b]
// so that the loads of a warp are contiguous in every slot, values and indices alike.
//
// A lane owns one block row (fp64) or two (fp32): 8 bytes of a value slice either way, and few enough registers for the
// warps that keep the memory busy. Its slots come one after the other, and each would wait for its index, its values and its
// x in turn; instead the indices and values of D slots are under way, and the x of the next slot is fetched before this
// one's products. SPLIT warps share the slots of a block row where the matrix has too few of them to fill the device, and
// add their sums up in shared memory.
// Measured, 27 blocks of 3 x 3 a row, fp64 (two block rows a lane, one batch after the other: before): 98,304 block rows
// 61.5 -> 36 us (31.5 us by bytes), 11,068 x 20 36 -> 5 us; 1,048,576 x 9 128 -> 115 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernel_args.h"
#include "kernels.h"
#include "launch.h"

namespace asp
{
typedef unsigned long long u64;
typedef unsigned int u32;

namespace
{
// adjacent values / indices, streamed (touched once per SpMV)
__device__ __forceinline__ void ld_vals(const double *p, double (&v)[1])
{
    asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v[0]) : "l"(p));
}
__device__ __forceinline__ void ld_vals(const float *p, float (&v)[2])
{
    asm volatile("ld.global.cs.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p));
}
__device__ __forceinline__ void ld_idx(const u32 *p, u32 (&v)[1])
{
    asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(v[0]) : "l"(p));
}
__device__ __forceinline__ void ld_idx(const u32 *p, u32 (&v)[2])
{
    asm volatile("ld.global.cs.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p));
}
template <class VT, int R, int C, int D, int SPLIT>
__global__ void __launch_bounds__(SPLIT == 8 ? 256 : 128) k_block_ell(KArgs a)
{
    constexpr int V = 8 / sizeof(VT); // block rows of a lane
    constexpr int WARPS = SPLIT == 8 ? 8 : 4;
    __shared__ VT part[SPLIT > 1 ? WARPS * V * R * 32 : 1];
    const VT *__restrict__ x = (const VT *)a.x + a.first_col;
    VT *__restrict__ y = (VT *)a.y + a.first_row;
    const u64 NB = a.n_tlb;       // padded block rows (even)
    const u32 W = a.tlb_size;     // block slots per block row
    const u64 rows = a.effective; // rows of the sub-matrix (the last block row may be partial)
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = warp % SPLIT;
    const u64 group = (u64)blockIdx.x * (blockDim.x / (32 * SPLIT)) + warp / SPLIT;
    const u64 at = (group * 32 + lane) * V;
    const bool in = at < NB;
    const u64 b0 = in ? at : 0; // (lanes past the last block row load the first one's and store nothing)
    const u32 k0 = W * sub / SPLIT, n = W * (sub + 1) / SPLIT - k0;
    const u32 *ip = (const u32 *)a.col + (u64)k0 * NB + b0;
    const VT *vp = (const VT *)a.val + (u64)k0 * (R * C) * NB + b0;
    VT acc[V][R];
#pragma unroll
    for (int s = 0; s < V; s++)
#pragma unroll
        for (int i = 0; i < R; i++) acc[s][i] = 0;
    u32 bc[D][V];
    VT v[D][R * C][V], xv[D][V][C];
    auto load = [&](int d, const u32 *i, const VT *p) {
        ld_idx(i, bc[d]);
#pragma unroll
        for (int e = 0; e < R * C; e++) ld_vals(p + (u64)e * NB, v[d][e]);
    };
    auto gather = [&](int d) {
#pragma unroll
        for (int s = 0; s < V; s++)
#pragma unroll
            for (int j = 0; j < C; j++) xv[d][s][j] = ld_x(x + (u64)bc[d][s] * C + j);
    };
#pragma unroll
    for (int d = 0; d < D; d++)
        if ((u32)d < n) load(d, ip + (u64)d * NB, vp + (u64)d * (R * C) * NB);
    grid_wait(); // the first indices and values are on their way
    grid_release();
    if (n > 0) gather(0);
    ip += (u64)D * NB;
    vp += (u64)D * (R * C) * NB;
    for (u32 k = 0; k < n; k += D)
    {
#pragma unroll
        for (int d = 0; d < D; d++)
            if (k + d < n)
            {
                if (k + d + 1 < n) gather((d + 1) % D);
#pragma unroll
                for (int s = 0; s < V; s++)
#pragma unroll
                    for (int i = 0; i < R; i++)
#pragma unroll
                        for (int j = 0; j < C; j++) acc[s][i] += v[d][i * C + j][s] * xv[d][s][j];
                if (k + d + D < n) load(d, ip, vp);
                ip += NB;
                vp += (u64)(R * C) * NB;
            }
    }
    if constexpr (SPLIT > 1)
    {
        // the first warp of every SPLIT adds up what the others found
        VT *mine = part + warp * (V * R * 32) + lane;
        if (sub != 0)
        {
#pragma unroll
            for (int q = 0; q < V * R; q++) mine[q * 32] = acc[q / R][q % R];
        }
        __syncthreads();
        if (sub != 0) return;
#pragma unroll
        for (int o = 1; o < SPLIT; o++)
#pragma unroll
            for (int q = 0; q < V * R; q++) acc[q / R][q % R] += mine[o * (V * R * 32) + q * 32];
    }
    if (!in) return;
#pragma unroll
    for (int s = 0; s < V; s++)
#pragma unroll
        for (int i = 0; i < R; i++)
            if ((b0 + s) * R + i < rows) y[(b0 + s) * R + i] = acc[s][i];
}

template <class VT, int R, int C, int D>
cudaError_t launch_split(const KArgs &a, unsigned block, cudaStream_t st)
{
    // Warps that cover the block rows, against the 20 to 24 a SM that the registers allow (about 3300 on 148 SMs). The rules lie
    // where the next split was no longer faster: 2,000 block rows x 27 want 8 parts (10 -> 4 us), 30,000 want 2 in fp64
    // (24.5 -> 16.4 us) and 4 in fp32 (22 -> 10 us), 65,000 and more fill the device in fp64 without. In fp32 a slot is half the
    // bytes and its time is latency for longer: 200,000 block rows x 27 are still faster in 4 parts (51 -> 43 us).
    const u64 groups = (a.n_tlb * sizeof(VT) / 8 + 31) / 32;
    const u32 W = a.tlb_size;
    const bool f32 = sizeof(VT) == 4;
    int split = 1;
    if (groups < 250 && W >= 16) split = 8;
    else if ((groups < 600 && W >= 8) || (f32 && groups < 4000 && W >= 24)) split = 4;
    else if (groups < 1800 && W >= 12) split = 2;
    const unsigned per_cta = split == 8 ? 1 : split > 1 ? 4 / split : block / 32;
    const u64 grid = (groups + per_cta - 1) / per_cta;
    if (grid > 2147483647ull) return cudaErrorInvalidValue;
    switch (split)
    {
    case 8: return launch_pdl(k_block_ell<VT, R, C, D, 8>, dim3((unsigned)grid), dim3(256), 0, st, a);
    case 4: return launch_pdl(k_block_ell<VT, R, C, D, 4>, dim3((unsigned)grid), dim3(128), 0, st, a);
    case 2: return launch_pdl(k_block_ell<VT, R, C, D, 2>, dim3((unsigned)grid), dim3(128), 0, st, a);
    default: return launch_pdl(k_block_ell<VT, R, C, D, 1>, dim3((unsigned)grid), dim3(block), 0, st, a);
    }
}

template <class VT>
cudaError_t launch_rc(int r, int c, const KArgs &a, unsigned block, cudaStream_t st)
{
    // slots under way: about 20 values a lane, fewer for 4 x 4 blocks
    if (r == 3 && c == 3) return launch_split<VT, 3, 3, 2>(a, block, st);
    if (r == 2 && c == 2) return launch_split<VT, 2, 2, 4>(a, block, st);
    if (r == 4 && c == 4) return launch_split<VT, 4, 4, 2>(a, block, st);
    return cudaErrorInvalidValue;
}
} // namespace

bool block_ell_supported(int r, int c) { return (r == 2 && c == 2) || (r == 3 && c == 3) || (r == 4 && c == 4); }

cudaError_t launch_block_ell(int val_is_f64, int r, int c, const KArgs &a, unsigned block, cudaStream_t st)
{
    if (block > 128 || block < 32 || block % 32 != 0) return cudaErrorInvalidValue;
    return val_is_f64 ? launch_rc<double>(r, c, a, block, st) : launch_rc<float>(r, c, a, block, st);
}

} // namespace asp
